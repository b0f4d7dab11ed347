// The one-tile-per-CTA convolution kernel for launches that do not fill the GPU (conv_small_sm100.cu): its arguments,
// and how a launch is cut for it.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200 {

struct alignas(64) SmallMaps {
    CUtensorMap a[4];   // activations, one per (row parity, column parity) of a strided conv
    CUtensorMap b;      // weights [kpad][R*S*C], boxes of bn rows
    CUtensorMap ones;   // 16 rows, the first all ones: the window-sum column of a weight zero point other than 128
};

struct SmallArgs {
    int n, oh, ow, cout;
    int r, s, pad_h, pad_w, stride_h, stride_w;
    int tw_sh, th_sh, tn;              // M-tile box (ow, oh, image) of 128 pixels: log2, log2, images
    int tiles_w, tiles_h, n_tiles_n;
    int bk, kblocks, cchunks;          // k-block bytes per pixel, k-blocks of a tile, k-blocks per tap
    int cpad, last_steps;              // weights' pitch per tap; 32-byte steps of a tap's last k-block that hold channels
    int bn;                            // output channels per tile
    int split;                         // CTAs (one cluster) that share a tile's k-blocks: 1, 2, 4 or 8
    int slots;                         // k-blocks in flight
    int a_wide;                        // see IgemmArgs::a_wide
    uint32_t idesc, tmem_cols;
    int form;                          // EpiForm, and its constants (see IgemmArgs)
    const int32_t *off32;              // [n_cls][kpad]
    const int32_t *mul, *shift;        // [kpad]
    int ushift, rnd_hi;
    const uint8_t *row_cls, *col_cls;  // [oh], [ow]
    int n_col_cls, n_cls, kpad;
    int ozp, qmax, relu_lo;
    uint32_t out_flip;                 // 0x80808080 for int8 outputs, else 0
    int wzp_d;                         // weight zero point - 128; not 0: the tile has the window-sum column
    uint8_t *y;
    const uint8_t *res;                // not nullptr: sum = eltwise SUM of y and res (constants as in IgemmArgs)
    uint8_t *sum;
    int r_m[2], r_add[2], r_b[2];
    int r_s0, r_ozp, r_lo;
    int *status;
    const uint8_t *next_ro;            // see IgemmArgs::next_ro
    uint32_t next_ro_bytes;
};

// How to cut m_tiles x (k output channels) x kblocks for this kernel: channels per tile and CTAs per tile.  False where
// the persistent kernel, with bn_p channels per tile, is the better one.
bool conv_small_pick(int m_tiles, int k, int kblocks, int bk, bool wzp, int bn_p, int *bn, int *split);
// Completes bn-dependent fields (slots, idesc, tmem_cols) and launches.
size_t conv_small_smem(SmallArgs &a, bool act_signed);
int conv_small_launch(const SmallMaps &maps, const SmallArgs &a, int m_tiles, size_t smem, size_t bytes, cudaStream_t st);
int conv_small_warm();

}  // namespace b200
