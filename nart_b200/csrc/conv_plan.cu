// conv_2d / ip plans: the one-time work the reference does (or repeats) in prepare and run --
// zero-point subtraction of the weights, scale decomposition, bias preload
// (art/modules/quant/src/op/conv_2d.c:95-147, conv_2d_uint8_impl.c:61-124 of ModelTC/NART) --
// done once here: weights repacked for the kernels, per-channel (mult, shift) tables, folded
// bias.  b200_conv2d_run then only launches.
#include <cmath>
#include <cstdlib>
#include <mutex>
#include <string.h>

#include <vector>

#include "common.cuh"
#include "kernels.h"

using namespace b200;

namespace {

template <typename T>
int upload(const std::vector<T> &v, T **dev)
{
    *dev = nullptr;
    if (v.empty())
        return B200_OK;
    B200_CUDA_TRY(cudaMalloc((void **)dev, v.size() * sizeof(T)));
    B200_CUDA_TRY(cudaMemcpy(*dev, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice));
    return B200_OK;
}

// The weights and tables of the CUDA-core kernel: one block that w_dev owns, one copy, or two where the weights are large (an allocation
// and a copy cost 8 us, moving 64 KB on the host 5).  Each part takes what an allocation of its own would, so that the plans' tensor-core weights,
// which every SM reads, lie where they did (1x1 24 -> 144 on 56 x 56, batch 32: 8.4 .. 9.7 us by their place).
int upload_direct(const std::vector<int8_t> &w, const std::vector<int32_t> &bias, const std::vector<uint32_t> &mult, const std::vector<int32_t> &shift, ConvDirectPlan *d)
{
    const size_t each = (bias.size() * 4 + 511) / 512 * 512, behind = (w.size() + 511) / 512 * 512, lead = w.size() <= (64u << 10) ? behind : 0;
    std::vector<uint8_t> image(lead + 3 * each);
    if (lead != 0)
        memcpy(image.data(), w.data(), w.size());
    memcpy(&image[lead], bias.data(), bias.size() * 4);
    memcpy(&image[lead + each], mult.data(), mult.size() * 4);
    memcpy(&image[lead + 2 * each], shift.data(), shift.size() * 4);
    uint8_t *block = nullptr;
    B200_CUDA_TRY(cudaMalloc((void **)&block, behind + 3 * each));
    d->w_dev = reinterpret_cast<int8_t *>(block);
    d->bias_fold_dev = reinterpret_cast<int32_t *>(block + behind);
    d->mult_dev = reinterpret_cast<uint32_t *>(block + behind + each);
    d->shift_dev = reinterpret_cast<int32_t *>(block + behind + 2 * each);
    if (lead == 0)
        B200_CUDA_TRY(cudaMemcpy(block, w.data(), w.size(), cudaMemcpyHostToDevice));
    B200_CUDA_TRY(cudaMemcpy(block + behind - lead, image.data(), image.size(), cudaMemcpyHostToDevice));
    return B200_OK;
}

// A plan's scratch tensors (they grow with the batch, so the first run allocates them).  Small ones come from a pool per device
// that keeps up to 64 MB of what was given back: mapping fresh device memory costs 0.3 .. 2.6 ms, taking it from the pool
// some 10 us.
constexpr size_t kScratchKeep = (size_t)64 << 20;
struct ScratchPool {
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;      // for allocations that belong to no stream of a caller
};
// The current device's
int scratch_pool(ScratchPool *out)
{
    static std::mutex mu;
    static ScratchPool pools[64];
    int device = 0;
    B200_CUDA_TRY(cudaGetDevice(&device));
    if (device >= 64)
        return fail(B200_ERR_UNSUPPORTED, "conv: no scratch pool for device %d", device);
    std::lock_guard<std::mutex> lock(mu);
    ScratchPool &q = pools[device];
    if (!q.stream)
        B200_CUDA_TRY(cudaStreamCreateWithFlags(&q.stream, cudaStreamNonBlocking));
    if (!q.pool) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        cudaMemPool_t pool = nullptr;
        B200_CUDA_TRY(cudaMemPoolCreate(&pool, &props));
        uint64_t keep = kScratchKeep;
        B200_CUDA_TRY(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
        q.pool = pool;
    }
    *out = q;
    return B200_OK;
}
int pool_alloc(uint8_t **p, size_t bytes, cudaMemPool_t pool, cudaStream_t st)
{
    *p = nullptr;
    const cudaError_t e = cudaMallocFromPoolAsync((void **)p, bytes, pool, st);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        *p = nullptr;
        return fail(B200_ERR_NOMEM, "conv: scratch of %zu bytes", bytes);
    }
    B200_CUDA_TRY(e);
    return B200_OK;
}
int scratch_alloc(uint8_t **p, size_t bytes)
{
    ScratchPool q;
    if (bytes > kScratchKeep || scratch_pool(&q) != B200_OK)
        return b200_malloc((void **)p, bytes);
    B200_TRY(pool_alloc(p, bytes, q.pool, q.stream));
    B200_CUDA_TRY(cudaStreamSynchronize(q.stream));
    return B200_OK;
}
// (cudaFree does not wait for the users of pool memory: `device`, the plan's own, need not be the current one)
cudaError_t scratch_free(uint8_t *p, int device)
{
    if (!p)
        return cudaSuccess;
    const DeviceGuard on(device);
    const cudaError_t e = cudaDeviceSynchronize();
    const cudaError_t f = cudaFree(p);
    return e != cudaSuccess ? e : f;
}

void destroy_conv(b200_conv *cv)
{
    if (!cv)
        return;
    cudaFree(cv->direct.w_dev);
    cudaFree(cv->direct.w_dw_dev);
    cudaFree(cv->direct.w_dw3_dev);
    cudaFree(cv->direct.w_dw3p_dev);
    cudaFree(cv->direct.q_dw3_dev);
    cudaFree(cv->direct.q_dw3p_dev);
    if (cv->igemm)
        conv_igemm_destroy(cv->igemm);
    if (cv->grouped)
        conv_igemm_destroy(cv->grouped);
    scratch_free(cv->scratch, cv->device);
    scratch_free(cv->padded, cv->device);
    scratch_free(cv->home, cv->device);
    delete cv;
}

// The channel-padded copy of the activations, and the rows it is lowered to, for n images
struct PaddedBytes {
    size_t padded, lowered;
    PaddedBytes(const b200_conv *cv, int32_t n)
        : padded((size_t)n * cv->g.h * cv->g.w * cv->pad_c), lowered(cv->lowered ? (size_t)n * cv->g.h * cv->g.ow * (kLowerWindow * 4) : 0) {}
    size_t lowered_at() const { return (padded + 255) & ~(size_t)255; }
    size_t total() const { return lowered_at() + lowered; }
};

// The launches of a plan on the tensor cores
int conv_run_igemm(b200_conv *cv, const uint8_t *x, int32_t n, uint8_t *y, uint8_t *padded, uint8_t *lowered, cudaStream_t st)
{
    const ConvGeom &g = cv->pad_c ? cv->g_pad : cv->g;
    if (cv->pad_c) {
        B200_TRY(conv_pad_channels_launch(x, padded, (size_t)n * g.h * g.w, cv->g.c, cv->pad_c, (uint8_t)g.izp, st));
        x = padded;
    }
    if (cv->lowered && conv_runs_grouped(cv, x, n))
        return conv_igemm_launch(cv->grouped, x, n, y, st);
    if (cv->lowered) {
        B200_TRY(conv_lower_rows_launch(g, x, n, lowered, st));
        x = lowered;
    }
    return conv_igemm_launch(cv->igemm, x, n, y, st);
}

// A padded plan without an owner who orders its runs.  The stream that runs it first keeps a scratch buffer in the plan; a
// run on another stream takes one from the pool for its own launches, and a run under capture leaves the graph a buffer of the
// graph's own (an allocation node), as a captured address must outlive the plan's growth.  All of it is ordered by the
// stream: no run waits for the device.  B200_ERR_NOMEM: nothing has been launched.
int conv_run_padded(b200_conv *cv, const uint8_t *x, int32_t n, uint8_t *y, cudaStream_t st)
{
    const PaddedBytes need(cv, n);
    ScratchPool q;
    B200_TRY(scratch_pool(&q));
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    unsigned long long id = 0;      // unique among all streams the process ever has, unlike the handle
    B200_CUDA_TRY(cudaStreamIsCapturing(st, &capture));
    if (capture == cudaStreamCaptureStatusNone)         // (not permitted under capture)
        B200_CUDA_TRY(cudaStreamGetId(st, &id));
    if (capture != cudaStreamCaptureStatusNone || (cv->home_taken && cv->home_stream != id)) {
        uint8_t *block = nullptr;
        B200_TRY(pool_alloc(&block, need.total(), q.pool, st));
        const int rc = conv_run_igemm(cv, x, n, y, block, block + need.lowered_at(), st);
        const cudaError_t e = cudaFreeAsync(block, st);
        B200_TRY(rc);
        B200_CUDA_TRY(e);
        return B200_OK;
    }
    if (cv->home_bytes < need.total()) {
        uint8_t *old = cv->home;
        cv->home = nullptr;
        cv->home_bytes = 0;
        if (old)
            B200_CUDA_TRY(cudaFreeAsync(old, st));
        B200_TRY(pool_alloc(&cv->home, need.total(), q.pool, st));
        cv->home_bytes = need.total();
    }
    cv->home_taken = true;
    cv->home_stream = id;
    return conv_run_igemm(cv, x, n, y, cv->home, cv->home + need.lowered_at(), st);
}

// A conv as one on groups of m neighbouring pixels, where the lines of the image are whole groups of a multiple of 16 bytes: its
// output pixel is the m / stride neighbouring output pixels whose windows start in one group, side by side as they lie in
// memory, its window the groups that theirs reach.  Part of the weights is zero (7x7 on 4 channels, stride 2: 128 output
// channels and 7 x 3 groups of 16 for 64 and 7 x 7 pixels of 4), but the image is read as it is.  flat: 1x1, all of an image is one line.
// Left out: lines of no whole number of groups, as a group would hold pixels of two lines; weight zero points, as the window-sum column
// would sum the pixels of all the group's windows; and signed activations, for which nothing has been measured.
int create_grouped(const ConvGeom &g, int m, bool flat, const std::vector<int8_t> &w, const int32_t *bias, const std::vector<uint32_t> &mult,
                   const std::vector<int32_t> &shift, ConvIgemmPlan **out)
{
    *out = nullptr;
    ConvGeom q = g;
    if (flat) {
        if ((long long)g.h * g.w > INT32_MAX)
            return B200_ERR_UNSUPPORTED;
        q.w = q.ow = g.h * g.w;
        q.h = q.oh = 1;
    }
    if (q.w % m != 0 || m % g.stride_w != 0 || g.wzp_d != 0 || g.act_signed)
        return B200_ERR_UNSUPPORTED;
    const int per = m / g.stride_w;
    auto group = [m](int px) { return (px >= 0 ? px : px - (m - 1)) / m; };
    const int first = group(-g.pad_w), last = group((per - 1) * g.stride_w + g.s - 1 - g.pad_w);
    const bool quads = m * g.c == 16;
    if (q.ow % per != 0 || (long long)per * g.k * m * g.c * g.r * (last - first + 1) > (1 << 20))      // (mostly zeros by then)
        return B200_ERR_UNSUPPORTED;
    q.c = m * g.c; q.w /= m; q.ow /= per; q.k = per * g.k; q.s = last - first + 1; q.pad_w = -first; q.stride_w = 1;
    if (quads && q.s > 8)
        return B200_ERR_UNSUPPORTED;
    std::vector<int8_t> wq((size_t)q.k * q.c * q.r * q.s, 0);
    std::vector<int32_t> bq(bias ? q.k : 0), sq(q.k);
    std::vector<uint32_t> mq(q.k);
    for (int k = 0; k < g.k; ++k) {
        for (int o = 0; o < per; ++o) {
            const int kq = o * g.k + k;
            if (bias)
                bq[kq] = bias[k];
            mq[kq] = mult[k];
            sq[kq] = shift[k];
            for (int rr = 0; rr < g.r; ++rr)        // a row of the window lies in the groups as it does in the image
                memcpy(&wq[((size_t)kq * q.r + rr) * q.s * q.c + (size_t)(o * g.stride_w - g.pad_w - first * m) * g.c],
                       &w[((size_t)k * g.r + rr) * g.s * g.c], (size_t)g.s * g.c);
        }
    }
    return conv_igemm_create(q, wq, bias ? bq.data() : nullptr, mq.data(), sq.data(), out, false, 0, quads);
}

// The images from which on a launch has a tile of groups of m pixels for every SM
int tile_an_sm(const ConvGeom &g, int m)
{
    const int per = m / g.stride_w;
    return (int)(((size_t)sm_count() * 128 * per + (size_t)g.oh * g.ow - 1) / ((size_t)g.oh * g.ow));
}

// Scratch tensors that serve every run of the plan: a copy with padded channels for n_padded images, a lowered one's rows for n_lowered
int reserve_owned(b200_conv *conv, int32_t n_padded, int32_t n_lowered)
{
    auto grow = [conv](uint8_t *&buf, size_t &have, size_t need) -> int {
        if (need <= have)
            return B200_OK;
        const DeviceGuard on(conv->device);
        B200_CUDA_TRY(scratch_free(buf, conv->device));
        buf = nullptr;
        have = 0;
        B200_TRY(scratch_alloc(&buf, need));
        have = need;
        return B200_OK;
    };
    if (conv->lowered)
        B200_TRY(grow(conv->scratch, conv->scratch_bytes, PaddedBytes(conv, n_lowered).lowered));
    if (conv->pad_c)
        B200_TRY(grow(conv->padded, conv->padded_bytes, PaddedBytes(conv, n_padded).padded));
    return B200_OK;
}

// A run on groups needs no rows, but the plan's scratch grows with the batch whatever route a run takes: after it, a smaller batch
// or an unaligned view of as many images neither allocates (it may be under capture) nor moves the rows that a captured graph knows.
// Without memory for more rows the plan keeps those it has and does not ask again.
int reserve_beside_groups(b200_conv *conv, int32_t n, cudaStream_t st)
{
    const size_t need = PaddedBytes(conv, n).lowered;
    if (need <= conv->scratch_bytes || need >= conv->scratch_declined)
        return B200_OK;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    B200_CUDA_TRY(cudaStreamIsCapturing(st, &capture));
    if (capture != cudaStreamCaptureStatusNone)
        return B200_OK;
    const DeviceGuard on(conv->device);
    uint8_t *rows = nullptr;
    const int rc = scratch_alloc(&rows, need);
    if (rc == B200_ERR_NOMEM) {
        conv->scratch_declined = need;
        return B200_OK;
    }
    B200_TRY(rc);
    const cudaError_t e = scratch_free(conv->scratch, conv->device);
    conv->scratch = rows;
    conv->scratch_bytes = need;
    B200_CUDA_TRY(e);
    return B200_OK;
}

}  // namespace

bool b200::conv_runs_grouped(const b200_conv *cv, const uint8_t *x, int32_t n)
{
    return cv->grouped && cv->algo == B200_CONV_ALGO_IGEMM && !cv->fused_residual && ((uintptr_t)x & 15) == 0 && n >= cv->grouped_from && n <= cv->grouped_to;
}

NextRead b200::conv_weights_read(const b200_conv *cv)
{
    NextRead r;
    if (cv->algo == B200_CONV_ALGO_IGEMM)
        conv_igemm_weights(cv->igemm, &r.plain, &r.plain_bytes);
    if (cv->grouped && cv->algo == B200_CONV_ALGO_IGEMM && !cv->fused_residual) {
        conv_igemm_weights(cv->grouped, &r.grouped, &r.grouped_bytes);
        r.from = cv->grouped_from;
        r.to = cv->grouped_to;
    }
    return r;
}

extern "C" {

int b200_conv2d_create(
    const b200_conv_params *p, const uint8_t *weights, const int32_t *bias, b200_conv_t **out)
{
    if (!p || !weights || !out)
        return fail(B200_ERR_INVALID, "conv: NULL argument");
    *out = nullptr;
    if (p->c <= 0 || p->h <= 0 || p->w <= 0 || p->k <= 0 || p->r <= 0 || p->s <= 0 || p->group <= 0
        || p->stride_h <= 0 || p->stride_w <= 0 || p->pad_h < 0 || p->pad_w < 0)
        return fail(B200_ERR_INVALID, "conv: non-positive dimension");
    if (p->c % p->group || p->k % p->group)
        return fail(B200_ERR_INVALID, "conv: c=%d and k=%d must be multiples of group=%d", p->c, p->k, p->group);
    if (p->h + 2 * p->pad_h < p->r || p->w + 2 * p->pad_w < p->s)
        return fail(B200_ERR_INVALID, "conv: kernel larger than the padded input");
    if (p->obits < 1 || p->obits > 8)
        return fail(B200_ERR_INVALID, "conv: obits=%d outside 1..8", (int)p->obits);
    if (!p->walpha || (p->n_walpha != 1 && p->n_walpha != p->k))
        return fail(B200_ERR_INVALID, "conv: n_walpha must be 1 or k");
    if (!(p->ialpha > 0.f) || !(p->oalpha > 0.f))
        return fail(B200_ERR_INVALID, "conv: ialpha and oalpha must be positive");
    if (p->algo != B200_CONV_ALGO_AUTO && p->algo != B200_CONV_ALGO_DIRECT && p->algo != B200_CONV_ALGO_IGEMM)
        return fail(B200_ERR_INVALID, "conv: unknown algo %d", p->algo);
    if (p->act_type != B200_ACT_U8 && p->act_type != B200_ACT_S8)
        return fail(B200_ERR_INVALID, "conv: unknown act_type %d", p->act_type);
    const bool s8 = p->act_type == B200_ACT_S8;
    if (s8 && p->obits == 8 && !p->s8_wrap)
        return fail(
            B200_ERR_UNSUPPORTED,
            "conv: int8 activations with obits = 8 clip at +-255 and then wrap into int8 in the reference "
            "(quant_helper.h:43-47); set s8_wrap to reproduce that, or use obits <= 7");
    if (s8 && p->obits == 8 && p->algo == B200_CONV_ALGO_IGEMM)
        return fail(B200_ERR_UNSUPPORTED, "conv: the wrapping int8 output exists on the CUDA-core path only");

    b200_conv *cv = new b200_conv();
    ConvGeom &g = cv->g;
    g.c = p->c; g.h = p->h; g.w = p->w; g.k = p->k; g.r = p->r; g.s = p->s;
    g.pad_h = p->pad_h; g.pad_w = p->pad_w; g.stride_h = p->stride_h; g.stride_w = p->stride_w;
    g.group = p->group;
    g.oh = (p->h + 2 * p->pad_h - p->r) / p->stride_h + 1;   // art/src/op.c:547-555
    g.ow = (p->w + 2 * p->pad_w - p->s) / p->stride_w + 1;
    g.izp = p->izp; g.ozp = p->ozp; g.qmax = (1 << p->obits) - 1;
    g.relu_lo = p->relu ? p->ozp : 0;
    g.wzp_d = (int)p->wzp - 128;
    g.act_signed = 0;
    g.s8_wrap = 0;
    if (s8) {
        const int m = (1 << p->obits) - 1;     // ssaturate_int_by_bits: +-(2^obits - 1)
        g.act_signed = 1;
        g.s8_wrap = p->obits == 8 ? 1 : 0;
        g.izp = 128; g.ozp = 128; g.wzp_d = 0;
        g.qmax = g.s8_wrap ? 255 : 128 + m;
        // the wrapping form works on the signed value itself (floor 0 or -255), the clipping one on value + 128
        g.relu_lo = g.s8_wrap ? (p->relu ? 0 : -255) : (p->relu ? 128 : 128 - m);
    }
    cv->oalpha = p->oalpha;
    cudaGetDevice(&cv->device);

    const int cg = g.c / g.group, taps = g.r * g.s;
    const size_t wcount = (size_t)g.k * cg * taps;
    // int32 accumulation wraps modulo 2^32 in every order, like the reference's int32 GEMM
    // (gemm/default/gemm.c:306-355), so no bound on the reduction length is needed.
    // Any stored byte minus 128 is an int8; a weight zero point other than 128 is carried as
    // wzp_d = wzp - 128 and applied through the sum of the activations (ConvGeom::wzp_d).
    std::vector<int8_t> w_s8(wcount);   // [k][r][s][cg], value = stored - 128
    const int minus = s8 ? 0 : 128;
    for (int k = 0; k < g.k; ++k) {
        const uint8_t *src = weights + (size_t)k * cg * taps;
        int8_t *dst = &w_s8[(size_t)k * cg * taps];
        if (taps == 1 || cg == 1) {
            for (int i = 0; i < cg * taps; ++i)
                dst[i] = (int8_t)(src[i] - minus);
            continue;
        }
        for (int t = 0; t < taps; ++t)
            for (int c = 0; c < cg; ++c)
                dst[(size_t)t * cg + c] = (int8_t)(src[(size_t)c * taps + t] - minus);
    }

    std::vector<uint32_t> mult(g.k);
    std::vector<int32_t> shift(g.k);
    for (int k = 0; k < g.k; ++k) {
        float wa = p->walpha[p->n_walpha == 1 ? 0 : k];
        if (!(wa > 0.f)) {
            destroy_conv(cv);
            return fail(B200_ERR_INVALID, "conv: walpha[%d] must be positive", k);
        }
        float scale = p->ialpha * wa / p->oalpha;   // conv_2d_uint8_impl.c:75, fp32, left to right
        uint32_t m;
        int8_t s;
        get_quant_scale(scale, 32, &m, &s);
        if (m == 0 || s < 1 || s > 62) {
            destroy_conv(cv);
            return fail(
                B200_ERR_UNSUPPORTED, "conv: scale %g of channel %d gives shift %d outside 1..62", (double)scale, k, (int)s);
        }
        mult[k] = m;
        shift[k] = s;
    }

    // ---- direct-kernel tables (always built: the accumulator-dumping entry uses them) --------
    const int cg4 = (cg + 3) / 4 * 4;
    std::vector<int8_t> w_pack((size_t)g.k * taps * cg4, 0);
    std::vector<int32_t> bias_fold(g.k), tap_sum(taps);
    for (int k = 0; k < g.k; ++k) {
        weights_to_pitch(&w_s8[(size_t)k * cg * taps], cg, taps, &w_pack[(size_t)k * taps * cg4], cg4, tap_sum.data());
        long long wsum = 0;
        for (int t = 0; t < taps; ++t)
            wsum += tap_sum[t];
        long long bf = (long long)(bias ? bias[k] : 0) - (long long)g.izp * wsum;
        bias_fold[k] = (int32_t)(uint32_t)(unsigned long long)bf;   // modulo 2^32
    }
    cv->direct.cg4 = cg4;
    int rc = upload_direct(w_pack, bias_fold, mult, shift, &cv->direct);
    if (rc == B200_OK && g.group == g.c && g.group == g.k && g.c % 16 == 0) {
        std::vector<int8_t> w_dw((size_t)taps * g.c);
        for (int c = 0; c < g.c; ++c)
            for (int t = 0; t < taps; ++t)
                w_dw[(size_t)t * g.c + c] = w_s8[(size_t)c * taps + t];
        rc = upload(w_dw, &cv->direct.w_dw_dev);
        // the dp4a form of the 3x3 case (conv_depthwise3x3_kernel)
        bool fast = g.r == 3 && g.s == 3 && g.qmax == 255 && g.wzp_d == 0;
        for (int k = 0; k < g.k && fast; ++k)
            fast = shift[k] >= 33 && shift[k] <= 53;
        if (rc == B200_OK && fast) {
            std::vector<uint32_t> w3((size_t)(g.c / 4) * 3 * 4, 0);
            std::vector<int4> q3(g.c);
            for (int c = 0; c < g.c; ++c) {
                for (int grp = 0; grp < 3; ++grp) {
                    uint32_t word = 0;
                    for (int j = 0; j < 4; ++j) {
                        const int t = grp * 4 + j;
                        if (t < 9)
                            word |= (uint32_t)(uint8_t)w_s8[(size_t)c * 9 + t] << (8 * j);
                    }
                    w3[((size_t)(c / 4) * 3 + grp) * 4 + (c % 4)] = word;
                }
                // (acc + bias_fold) * mult, rounded shift, + ozp  ==  (acc * mult + off64) >> shift
                const long long off64 = (long long)bias_fold[c] * (long long)mult[c] + (1ll << (shift[c] - 1))
                    + ((long long)g.ozp << shift[c]);
                q3[c] = make_int4((int)(uint32_t)(unsigned long long)off64, (int)(off64 >> 32), (int)mult[c], shift[c] - 32);
            }
            rc = upload(w3, &cv->direct.w_dw3_dev);
            if (rc == B200_OK) rc = upload(q3, &cv->direct.q_dw3_dev);
            // its fp32 requantize: every accumulator below 2^22, every result within the 16 bits it is clamped in (see
            // conv_depthwise3x3_strip_kernel: half steps below zero).  Taps are 0 .. 255, so a channel's negative and positive
            // weights bound its accumulators; 22 of 272 layers of MobileNetV2 with random weights miss a bound by their number.
            const bool strip = g.stride_w == 1 || g.stride_w == 2;
            bool fp = strip;
            for (int k = 0; k < g.k; ++k) {
                int neg = 0, pos = 0;
                for (int t = 0; t < 9; ++t) {
                    const int w = w_s8[(size_t)k * 9 + t];
                    (w < 0 ? neg : pos) += w;
                }
                const long long lo = bias_fold[k] + 255ll * neg, hi = bias_fold[k] + 255ll * pos;
                fp = fp && lo > -(1 << 22) && hi < (1 << 22) && ldexp((double)lo * mult[k], -shift[k]) > -16380.0
                    && ldexp((double)hi * mult[k], -shift[k]) + g.ozp < 32760.0;
            }
            if (rc == B200_OK && strip) {
                // one kernel row against 3 + stride_w neighbouring input pixels (conv_depthwise3x3_strip_kernel)
                const int nv = g.stride_w == 2 ? 3 : 2;
                std::vector<uint32_t> w3p((size_t)(g.c / 4) * 3 * nv * 4, 0);
                for (int c = 0; c < g.c; ++c)
                    for (int rr = 0; rr < 3; ++rr) {
                        uint32_t wb[3];
                        for (int j = 0; j < 3; ++j)
                            wb[j] = (uint32_t)(uint8_t)w_s8[(size_t)c * 9 + rr * 3 + j];
                        uint32_t *dst = &w3p[((size_t)(c / 4) * 3 + rr) * nv * 4 + (c % 4)];
                        dst[0] = wb[0] | (wb[1] << 8) | (wb[2] << 16);                   // left pixel: inputs 0..2
                        if (g.stride_w == 1) {
                            dst[4] = (wb[0] << 8) | (wb[1] << 16) | (wb[2] << 24);       // right pixel: inputs 1..3
                        } else {
                            dst[4] = (wb[0] << 16) | (wb[1] << 24);                      // right pixel: inputs 2, 3 ...
                            dst[8] = wb[2] << (8 * (c % 4));                             // ... and 4, at the channel's byte
                        }
                    }
                rc = upload(w3p, &cv->direct.w_dw3p_dev);
                std::vector<uint32_t> qf(fp ? (size_t)g.c * 2 : 0);
                for (int c = 0; c < g.c && fp; ++c) {
                    const float m = ldexpf((float)mult[c], -shift[c]);      // exact: mult has 24 significant bits
                    qf[(size_t)(c / 4) * 8 + c % 4] = 0x4B400000u + (uint32_t)bias_fold[c];
                    memcpy(&qf[(size_t)(c / 4) * 8 + 4 + c % 4], &m, 4);
                }
                if (rc == B200_OK) rc = upload(qf, &cv->direct.q_dw3p_dev);
            }
        }
    }
    if (rc != B200_OK) {
        destroy_conv(cv);
        return rc;
    }

    // ---- tensor-core plan ---------------------------------------------------------------------
    char why[256] = "";
    const bool ig_ok = conv_igemm_supported(g, why, sizeof(why)) != 0 && !g.s8_wrap;
    // Channel counts that are no multiple of 16 (the pixel stride of a TMA map) run on a copy padded to one, or to
    // the four channels of the row lowering below: the copy costs a pass over the input, the CUDA-core kernel
    // twenty (1x1 24 -> 144 channels on 56 x 56, batch 32: 129 us against 9).  Padding channels have zero weights and
    // hold the byte izp, so that their (x - izp) is zero in the window sums of a weight zero point as well.
    ConvGeom gt = g;                        // what the tensor cores see
    const std::vector<int8_t> *wt = &w_s8;
    std::vector<int8_t> w_pad;
    auto can_lower = [](const ConvGeom &q) {
        return q.group == 1 && q.c == 4 && q.s <= kLowerWindow && q.k >= 16 && q.stride_h <= 2 && q.h >= q.stride_h && !q.act_signed;
    };
    bool tc_ok = ig_ok;
    if (!ig_ok && !can_lower(g) && g.group == 1 && g.c % 16 != 0 && !g.s8_wrap && p->algo == B200_CONV_ALGO_AUTO) {
        gt.c = 4;
        if (g.c >= 4 || !can_lower(gt))
            gt.c = (g.c + 15) / 16 * 16;
        if (gt.c != 4)
            tc_ok = conv_igemm_supported(gt, why, sizeof(why)) != 0;
        if (gt.c == 4 || tc_ok) {
            cv->pad_c = gt.c;
            cv->g_pad = gt;
            w_pad.assign((size_t)g.k * gt.c * taps, 0);
            for (size_t i = 0; i < (size_t)g.k * taps; ++i)
                memcpy(&w_pad[i * gt.c], &w_s8[i * g.c], g.c);
            wt = &w_pad;
        }
    }
    // A 4-channel image with a short kernel row is no contraction the tensor cores can take as it
    // is (4 bytes per tap).  Gathering, for every input row and output column, the 8-pixel window
    // the kernel row slides over gives a 32-channel tensor [n][h][ow][8 pixels x 4 channels] on
    // which the same conv is an r x 1 kernel with stride (stride_h, 1): that is dense enough.
    // Window cells outside the image hold the byte izp, whose contribution the epilogue's
    // zero-point term removes exactly; cells past the kernel width get zero weights.
    rc = B200_ERR_UNSUPPORTED;
    if (p->algo == B200_CONV_ALGO_DIRECT) {
    } else if (!tc_ok && can_lower(gt)) {
        ConvGeom gl = gt;
        gl.c = kLowerWindow * 4;
        gl.w = g.ow;
        gl.s = 1;
        gl.pad_w = 0;
        gl.stride_w = 1;
        std::vector<int8_t> w_low((size_t)g.k * gl.c * g.r, 0);   // [k][r][1][32]
        for (size_t i = 0; i < (size_t)g.k * g.r; ++i)
            memcpy(&w_low[i * gl.c], &(*wt)[i * g.s * 4], (size_t)g.s * 4);
        rc = conv_igemm_create(gl, w_low, bias, mult.data(), shift.data(), &cv->igemm, true, g.s);
        if (rc == B200_OK) {
            cv->lowered = true;
            cv->g_low = gl;
            // The image in groups of four pixels instead, on launches of a tile of groups an SM: 7x7, 64 channels, 224 x 224,
            // batch 256: 175 -> 104 us, batch 8: 12.1 -> 8.3.  Smaller launches lower: alone they are faster on groups too (batch 1 5.0 against
            // 6.0 us), but not behind the other kernels of a network (ResNet-18, batch 1: 100.7 us, 102.2 on groups; batch 2: 111.2, 111.7;
            // batch 4: 121.7, 120.6).
            create_grouped(gt, 4, false, *wt, bias, mult, shift, &cv->grouped);     // (declined: all are lowered)
            cv->grouped_from = tile_an_sm(gt, 4);
            // for callers of b200_conv2d_run_static_scratch: everything that entry point would otherwise do
            // once per device (kernel set-up, the static array's address) happens here, where allocation is
            // allowed; a failure only matters to that entry point, which reports it itself
            if (conv_igemm_warm() != B200_OK || conv_static_scratch_prepare() != B200_OK)
                cudaGetLastError();
        }
    } else if (tc_ok) {
        rc = conv_igemm_create(gt, *wt, bias, mult.data(), shift.data(), &cv->igemm);
    } else if (p->algo == B200_CONV_ALGO_IGEMM) {
        rc = fail(B200_ERR_UNSUPPORTED, "conv: implicit-GEMM path declined: %s", why);
    }
    const bool flat = taps == 1 && g.stride_h == 1 && g.stride_w == 1 && g.pad_h == 0 && g.pad_w == 0;
    if (rc == B200_OK && !cv->pad_c && !cv->lowered && g.stride_w == 1 && g.stride_h == 1) {
        // Few output channels: what a tile costs beside its outputs -- an MMA takes 54 cycles for 128 pixels by 32 bytes whether it has 16
        // or 32 channels, 61 for 64, and an epilogue its waits -- is shared by the m pixels of a group.  1x1: up to four pixels and 128
        // columns (32 -> 16 on 112 x 112, batch 256: 60.2 -> 26.6 us; 64 -> 64 on 56 x 56: 24.3 -> 19.2; with 256 columns 20.5; 144 -> 32: 44.0 -> 24.8;
        // 256 -> 64, batch 64: 11.9 -> 12.4, too many zeros), 192 for 16 channels, which leave half of an operand row empty (16 -> 96 on
        // 112 x 112, batch 64: 30.8 -> 28.6).  Larger windows: pairs, up to 64 columns (16 -> 32, 3x3, 112 x 112, batch 128: 54.3 -> 32.6; 64 -> 64 on
        // 56 x 56: 47.3 -> 52.9), 128 up to 32 channels (32 -> 64 on 112 x 112: 36.6 -> 35.4).  On launches of a tile of groups an SM.
        const bool one = taps == 1;
        auto worth = [&](int m) {
            const int columns = m * g.k, depth = m * g.c;
            if ((flat ? (long long)g.h * g.w : g.w) % m != 0 || (!flat && g.ow % m != 0))
                return false;
            if (one)
                return columns <= (g.c == 16 ? 192 : 128) && depth <= (columns <= 64 ? 512 : 384);
            return m == 2 && columns <= (g.c <= 32 ? 128 : 64) && depth <= 128;
        };
        const int m = worth(4) ? 4 : worth(2) ? 2 : 0;
        if (m != 0) {
            create_grouped(g, m, flat, w_s8, bias, mult, shift, &cv->grouped);
            cv->grouped_from = tile_an_sm(g, m);
        }
    }
    if (rc == B200_OK && cv->pad_c > 4) {
        // Without the copy: groups of two or four pixels whose channels are a multiple of 16.  The zero weights cost `factor`
        // times the multiply-adds, at half of what the tensor cores do on dense ones, the copy three passes over the activations and a
        // launch (2.5 us).  24 -> 144 on 56 x 56, batch 32: 10.8 us with the copy, 8.5 on groups; 3x3 20 -> 100 on 28 x 28, batch 16: 11.1, 9.0;
        // 3x3 12 -> 52 on 58 x 58, batch 93, which keeps the copy: 41.8, 42.8.
        const int m = g.c % 8 == 0 && !(flat && g.c == 8) ? 2 : g.c % 4 == 0 ? 4 : 0;
        if (m != 0) {
            create_grouped(g, m, flat, w_s8, bias, mult, shift, &cv->grouped);
            const double factor = flat ? m : m * ((g.s - 1 + m - 1) / m + 1.0) / g.s;
            const double pixels = (double)g.oh * g.ow;
            const double gain = (double)g.h * g.w * (g.c + 2 * cv->pad_c) / 5e6 - pixels * 2.0 * (factor - 1.0) * g.c * taps * g.k / 1e9;    // us an image
            if (gain < 0.0)
                cv->grouped_to = (int)std::min(std::ceil(2.5 / -gain) - 1.0, (double)INT32_MAX);
        }
    }
    if (rc == B200_OK) {
        cv->algo = B200_CONV_ALGO_IGEMM;
        // what a first run under capture could not set up; a failure only matters to a run, which reports it itself
        ScratchPool q;
        int *status = nullptr;
        if (cv->pad_c && (scratch_pool(&q) != B200_OK || conv_igemm_warm() != B200_OK || status_word_ptr(&status) != B200_OK))
            cudaGetLastError();
    } else {
        cv->pad_c = 0;
        if (rc != B200_ERR_UNSUPPORTED || p->algo == B200_CONV_ALGO_IGEMM) {
            destroy_conv(cv);
            return rc;
        }   // declined under AUTO: the CUDA-core kernel runs it
    }
    *out = cv;
    return B200_OK;
}

int b200_ip_create(
    int32_t c, int32_t h, int32_t w, int32_t k, float ialpha, uint8_t izp, const float *walpha,
    int32_t n_walpha, uint8_t wzp, float oalpha, uint8_t ozp, uint8_t obits,
    const uint8_t *weights, const int32_t *bias, b200_conv_t **conv)
{
    // ip.cpp:133-209: y[n][k] = requant(bias[k] + sum_j (x[n][j] - izp) * (w[k][j] - wzp)) over the
    // flattened c*h*w input -- a convolution whose kernel is the whole image.
    b200_conv_params p;
    memset(&p, 0, sizeof(p));
    p.c = c; p.h = h; p.w = w; p.k = k; p.r = h; p.s = w;
    p.pad_h = p.pad_w = 0; p.stride_h = p.stride_w = 1; p.group = 1;
    p.ialpha = ialpha; p.izp = izp; p.wzp = wzp; p.ozp = ozp; p.obits = obits; p.oalpha = oalpha;
    p.walpha = walpha; p.n_walpha = n_walpha; p.relu = 0; p.algo = B200_CONV_ALGO_AUTO;
    return b200_conv2d_create(&p, weights, bias, conv);
}

int b200_ip_create_s8(
    int32_t c, int32_t h, int32_t w, int32_t k, float ialpha, const float *walpha, int32_t n_walpha,
    float oalpha, uint8_t obits, int32_t s8_wrap, const int8_t *weights, const int32_t *bias,
    b200_conv_t **conv)
{
    b200_conv_params p;
    memset(&p, 0, sizeof(p));
    p.c = c; p.h = h; p.w = w; p.k = k; p.r = h; p.s = w;
    p.pad_h = p.pad_w = 0; p.stride_h = p.stride_w = 1; p.group = 1;
    p.ialpha = ialpha; p.obits = obits; p.oalpha = oalpha;
    p.walpha = walpha; p.n_walpha = n_walpha; p.relu = 0; p.algo = B200_CONV_ALGO_AUTO;
    p.act_type = B200_ACT_S8; p.s8_wrap = s8_wrap;
    return b200_conv2d_create(&p, reinterpret_cast<const uint8_t *>(weights), bias, conv);
}

int b200_conv2d_out_dims(const b200_conv_t *conv, int32_t *oh, int32_t *ow)
{
    if (!conv || !oh || !ow)
        return fail(B200_ERR_INVALID, "conv: NULL argument");
    *oh = conv->g.oh;
    *ow = conv->g.ow;
    return B200_OK;
}

int b200_conv2d_algo(const b200_conv_t *conv) { return conv ? conv->algo : B200_ERR_INVALID; }

int b200_conv2d_describe(const b200_conv_t *conv, char *buf, size_t len)
{
    if (!conv || !buf || len == 0)
        return fail(B200_ERR_INVALID, "conv(describe): bad argument");
    if (conv->algo == B200_CONV_ALGO_IGEMM && conv->igemm) {
        const bool grouped = conv->ran_grouped;
        conv_igemm_describe(grouped ? conv->grouped : conv->igemm, buf, len);
        if (conv->lowered) {
            size_t used = strlen(buf);
            snprintf(buf + used, len - used, grouped ? ", on four-pixel groups of the image" : ", on the row-lowered image");
        }
        if (grouped && !conv->lowered) {
            size_t used = strlen(buf);
            snprintf(buf + used, len - used, ", on groups of pixels");
        } else if (conv->pad_c) {
            size_t used = strlen(buf);
            snprintf(buf + used, len - used, ", channels padded to %d", conv->pad_c);
        }
    } else {
        snprintf(buf, len, "CUDA cores (dp4a)%s", conv->g.group == conv->g.c && conv->g.group == conv->g.k ? ", depthwise" : "");
    }
    return B200_OK;
}

int b200_conv2d_run(b200_conv_t *conv, const uint8_t *x, int32_t n, uint8_t *y, b200_stream_t stream)
{
    if (!conv || n < 0 || (n > 0 && (!x || !y)))
        return fail(B200_ERR_INVALID, "conv: bad argument");
    if (n == 0)
        return B200_OK;
    if (conv->fused_residual)
        return fail(B200_ERR_INVALID, "conv: this plan has a residual add, run it with b200_conv2d_run_residual");
    cudaStream_t st = as_stream(stream);
    if (conv->algo != B200_CONV_ALGO_IGEMM)
        return conv_direct_launch(conv->g, conv->direct, x, n, y, nullptr, st);
    // Channel counts that AUTO pads would otherwise run on the CUDA cores, which take outputs at any address, any size and need
    // no memory; the tensor-core path stores 16 bytes at a time.
    if (conv->pad_c && (((uintptr_t)y & 15) != 0 || !conv_pad_channels_fits((size_t)n * conv->g.h * conv->g.w, conv->pad_c)))
        return conv_direct_launch(conv->g, conv->direct, x, n, y, nullptr, st);
    std::lock_guard<std::mutex> lock(conv->mu);
    const bool grouped = conv_runs_grouped(conv, conv->pad_c && conv->lowered ? nullptr : x, n);     // (a padded copy is aligned)
    conv->ran_grouped = grouped;
    if (grouped && !(conv->pad_c && conv->lowered)) {
        if (conv->lowered && !conv->one_owner)
            B200_TRY(reserve_beside_groups(conv, n, st));
        return conv_igemm_launch(conv->grouped, x, n, y, st);
    }
    if (conv->pad_c && !conv->one_owner) {
        const int rc = conv_run_padded(conv, x, n, y, st);
        return rc == B200_ERR_NOMEM ? conv_direct_launch(conv->g, conv->direct, x, n, y, nullptr, st) : rc;
    }
    B200_TRY(reserve_owned(conv, n, grouped ? 0 : n));   // grow-only scratch: the first call at a larger batch allocates (and synchronizes)
    return conv_run_igemm(conv, x, n, y, conv->padded, conv->scratch, st);
}

int b200_conv2d_reserve(b200_conv_t *conv, int32_t n)
{
    if (!conv || n < 0)
        return fail(B200_ERR_INVALID, "conv(reserve): bad argument");
    std::lock_guard<std::mutex> lock(conv->mu);
    if (!conv->pad_c || conv->one_owner) {
        // a case's tensors are aligned: launches on groups need neither the rows nor (their pixels are the conv's own) the copy
        const bool groups = conv->one_owner && conv->grouped;
        const int rc = reserve_owned(conv, groups && !conv->lowered && n <= conv->grouped_to ? 0 : n, groups ? std::min(n, conv->grouped_from - 1) : n);
        if (rc != B200_ERR_NOMEM || !conv->pad_c)
            return rc;
        conv->algo = B200_CONV_ALGO_DIRECT;         // needs no scratch
        conv->pad_c = 0;
        conv->lowered = false;
        return B200_OK;
    }
    const size_t need = PaddedBytes(conv, n).total();
    if (need <= conv->home_bytes)
        return B200_OK;
    const DeviceGuard on(conv->device);
    ScratchPool q;
    B200_TRY(scratch_pool(&q));
    B200_CUDA_TRY(scratch_free(conv->home, conv->device));
    conv->home = nullptr;
    conv->home_bytes = 0;
    B200_TRY(pool_alloc(&conv->home, need, q.pool, q.stream));
    B200_CUDA_TRY(cudaStreamSynchronize(q.stream));
    conv->home_bytes = need;
    return B200_OK;
}

int b200_conv2d_fuse_residual_add(
    b200_conv_t *conv, int32_t conv_input, const float *ialpha, const uint8_t *izp,
    const float *coeff, float oalpha, uint8_t ozp, uint8_t obits, int32_t relu)
{
    if (!conv || !ialpha || !izp || conv_input < 0 || conv_input > 1)
        return fail(B200_ERR_INVALID, "conv(fuse): bad argument");
    if (conv->algo != B200_CONV_ALGO_IGEMM || conv->lowered || conv->pad_c || !conv->igemm)
        return fail(B200_ERR_UNSUPPORTED, "conv(fuse): only plans on the tensor-core path take a residual add");
    if (conv->g.wzp_d != 0)
        return fail(B200_ERR_UNSUPPORTED, "conv(fuse): a weight zero point other than 128 and a fused residual add do not combine");
    if (conv->g.act_signed)
        return fail(B200_ERR_UNSUPPORTED, "conv(fuse): the residual add is a uint8 op (eltwise.c reads uint8 only)");
    if (conv->fused_residual)
        return fail(B200_ERR_INVALID, "conv(fuse): the plan already has a residual add");
    if (izp[conv_input] != (uint8_t)conv->g.ozp || ialpha[conv_input] != conv->oalpha)
        return fail(B200_ERR_UNSUPPORTED, "conv(fuse): the eltwise input's scale / zero point are not the conv's output ones");
    EltwiseArgs e;
    bool fast = false;
    B200_TRY(eltwise_prepare(2, ialpha, izp, coeff, oalpha, ozp, obits, relu, &e, &fast));
    if (!fast)
        return fail(B200_ERR_UNSUPPORTED, "conv(fuse): the eltwise rounding term does not fold (or obits != 8)");
    B200_TRY(conv_igemm_set_residual(conv->igemm, e, conv_input));
    conv->fused_residual = true;
    return B200_OK;
}

int b200_conv2d_run_residual(
    b200_conv_t *conv, const uint8_t *x, int32_t n, const uint8_t *res, uint8_t *y, b200_stream_t stream)
{
    if (!conv || n < 0 || (n > 0 && (!x || !y || !res)))
        return fail(B200_ERR_INVALID, "conv(residual): bad argument");
    if (!conv->fused_residual)
        return fail(B200_ERR_INVALID, "conv(residual): the plan has no residual add (b200_conv2d_fuse_residual_add)");
    if (n == 0)
        return B200_OK;
    conv->ran_grouped = false;
    return conv_igemm_launch(conv->igemm, x, n, y, as_stream(stream), nullptr, res);
}

int b200_conv2d_run_acc(
    b200_conv_t *conv, const uint8_t *x, int32_t n, uint8_t *y, int32_t *acc, b200_stream_t stream)
{
    if (!conv || !x || !y || !acc || n < 0)
        return fail(B200_ERR_INVALID, "conv: bad argument");
    return conv_direct_launch(conv->g, conv->direct, x, n, y, acc, as_stream(stream));
}

int b200_conv2d_destroy(b200_conv_t *conv)
{
    destroy_conv(conv);
    return B200_OK;
}

}  // extern "C"
