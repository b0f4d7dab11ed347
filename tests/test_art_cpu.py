"""nart_b200.art without a GPU."""
import numpy as np
import pytest

from nart_b200 import _lib, art


@pytest.mark.parametrize("status", [_lib.ERR_CUDA, _lib.ERR_NOMEM])
def test_empty_io_without_page_locked_memory(monkeypatch, status):
    """Page-locked memory is limited; ordinary arrays serve as well."""
    monkeypatch.setattr(_lib.lib, "b200_malloc_host", lambda ptr, size: status)
    a = art._pinned_zeros((2, 3, 4), "float32")
    assert a.shape == (2, 3, 4) and a.dtype == np.float32 and a.flags.writeable and not a.any()
