// NHWC uint8 max / average pooling with the reference CPU module's integer requantize
// (art/modules/quant/src/op/pool.c:96-249 of ModelTC/NART).  CUDA-core, HBM-bound: one thread
// owns VEC consecutive channels of one output pixel and reads one VEC-byte vector per tap, so a
// warp reads contiguous runs of the channel axis.
#include <math.h>

#include "common.cuh"
#include "kernels.h"

namespace b200 {

template <int VEC> struct VecT;
template <> struct VecT<16> { using type = uint4; };
template <> struct VecT<4> { using type = uint32_t; };
template <> struct VecT<1> { using type = uint8_t; };

template <int VEC>
__device__ __forceinline__ void load_words(const uint8_t *p, uint32_t (&wv)[(VEC + 3) / 4])
{
    if constexpr (VEC == 16) {
        uint4 q = __ldg(reinterpret_cast<const uint4 *>(p));
        wv[0] = q.x; wv[1] = q.y; wv[2] = q.z; wv[3] = q.w;
    } else if constexpr (VEC == 4) {
        wv[0] = __ldg(reinterpret_cast<const uint32_t *>(p));
    } else {
        wv[0] = __ldg(p);
    }
}

template <int VEC>
__device__ __forceinline__ void store_words(uint8_t *p, const uint32_t (&wv)[(VEC + 3) / 4])
{
    if constexpr (VEC == 16) {
        *reinterpret_cast<uint4 *>(p) = make_uint4(wv[0], wv[1], wv[2], wv[3]);
    } else if constexpr (VEC == 4) {
        *reinterpret_cast<uint32_t *>(p) = wv[0];
    } else {
        *p = (uint8_t)wv[0];
    }
}

// Byte-wise unsigned maximum without the emulated SIMD-in-a-word intrinsics (__vmaxu4 expands to
// about eight integer instructions on this architecture): the four bytes of a word are spread over
// two words of two 16-bit lanes each (one byte-permute apiece), maxima run on those with the native
// max.u16x2, and one byte-permute packs the result.
struct U16x4 {
    uint32_t lo, hi;   // bytes 0, 1 and bytes 2, 3 of the word, zero-extended to 16 bits
};
__device__ __forceinline__ U16x4 spread_bytes(uint32_t w) { return { __byte_perm(w, 0, 0x4140), __byte_perm(w, 0, 0x4342) }; }
__device__ __forceinline__ uint32_t pack_bytes(const U16x4 &v) { return __byte_perm(v.lo, v.hi, 0x6420); }
__device__ __forceinline__ uint32_t max_u16x2(uint32_t a, uint32_t b)
{
    uint32_t d;
    asm("max.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ U16x4 max_u16x4(const U16x4 &a, const U16x4 &b) { return { max_u16x2(a.lo, b.lo), max_u16x2(a.hi, b.hi) }; }

// MAX: running byte-wise maximum starting from 0 (pool.c:140-148), then a 256-entry table that
// holds sat_u(rshift_rn(mult16 * (max - izp), shift) + ozp) for every possible maximum, built on
// the host with the exact arithmetic.
template <int VEC>
__global__ void __launch_bounds__(256) pool_max_kernel(
    const uint8_t *__restrict__ x, uint8_t *__restrict__ y, PoolGeom g, const uint8_t *__restrict__ lut_g)
{
    __shared__ uint8_t lut[256];
    lut[threadIdx.x] = lut_g[threadIdx.x];   // written once, at preparation
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    constexpr int W = (VEC + 3) / 4;
    const int cv = g.c / VEC;
    const size_t total = (size_t)g.n * g.oh * g.ow * cv;
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (size_t)gridDim.x * blockDim.x) {
        int ci = (int)(idx % cv);
        size_t pix = idx / cv;
        int ox = (int)(pix % g.ow);
        int oy = (int)((pix / g.ow) % g.oh);
        int n = (int)(pix / ((size_t)g.ow * g.oh));
        int hs = oy * g.stride_h - g.pad_h, ws = ox * g.stride_w - g.pad_w;
        int he = min(hs + g.kernel_h, g.h), we = min(ws + g.kernel_w, g.w);
        hs = max(hs, 0);
        ws = max(ws, 0);
        U16x4 run[W];
#pragma unroll
        for (int j = 0; j < W; ++j)
            run[j] = { 0u, 0u };
        for (int iy = hs; iy < he; ++iy)
            for (int ix = ws; ix < we; ++ix) {
                uint32_t v[W];
                load_words<VEC>(x + (((size_t)n * g.h + iy) * g.w + ix) * g.c + (size_t)ci * VEC, v);
#pragma unroll
                for (int j = 0; j < W; ++j)
                    run[j] = max_u16x4(run[j], spread_bytes(v[j]));
            }
        uint32_t mx[W], o[W];
#pragma unroll
        for (int j = 0; j < W; ++j)
            mx[j] = pack_bytes(run[j]);
#pragma unroll
        for (int j = 0; j < W; ++j) {
            if constexpr (VEC == 1)
                o[j] = lut[mx[j] & 0xff];
            else
                o[j] = pack4(
                    lut[mx[j] & 0xff], lut[(mx[j] >> 8) & 0xff], lut[(mx[j] >> 16) & 0xff],
                    lut[mx[j] >> 24]);
        }
        store_words<VEC>(y + pix * g.c + (size_t)ci * VEC, o);
    }
}

// Small windows of a compile-time size KH x KW and horizontal stride SW, with 32-bit index arithmetic: one
// thread owns 4 * W channels of TWO output pixels side by side and loads the union of their windows
// (KH x (KW + SW) vectors) in one unrolled batch, so that all of a thread's loads are in flight together
// and the columns the two windows share are loaded, and reduced, once.  Taps outside the image read as 0:
// the value the running maximum starts from, and nothing to a sum.  Reductions run on 16-bit lanes down
// each column first, then across the columns of each output.
//   MAX        the maximum goes through the 256-entry table (IDENT: it maps every byte to itself)
//   AVE        at most 9 bytes a lane; the requantize of pool_avg_kernel in 32 bits (pool_launch checks that
//              its terms fit).  3x3 stride 2 on 64 channels of 112 x 112, batch 32: 33.6 us a pixel per thread.
// W = 4 where channels and addresses allow 16-byte vectors, else 1.
enum PoolPairOp { kPairMaxIdent, kPairMaxLut, kPairAve };

template <int W>
__device__ __forceinline__ void load_vec(const uint32_t *p, uint32_t (&v)[W])
{
    if constexpr (W == 4) {
        const uint4 q = __ldg(reinterpret_cast<const uint4 *>(p));
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else {
        v[0] = __ldg(p);
    }
}

template <int KH, int KW, int SW, PoolPairOp OP, int W>
__global__ void __launch_bounds__(256) pool_pair_kernel(
    const uint32_t *__restrict__ x, uint32_t *__restrict__ y, PoolGeom g, const uint8_t *__restrict__ lut_g, PoolAvgTab tab,
    uint32_t total)
{
    __shared__ uint8_t lut[256];
    __shared__ int2 mult_shift[PoolAvgTab::kMax][PoolAvgTab::kMax];   // indexed at run time: not as parameters
    if (OP == kPairMaxLut) {
        lut[threadIdx.x] = lut_g[threadIdx.x];
        __syncthreads();
    }
    if (OP == kPairAve) {
        if (threadIdx.x == 0) {
#pragma unroll
            for (int i = 0; i < PoolAvgTab::kMax * PoolAvgTab::kMax; ++i)
                mult_shift[i / PoolAvgTab::kMax][i % PoolAvgTab::kMax]
                    = make_int2(tab.mult[i / PoolAvgTab::kMax][i % PoolAvgTab::kMax], tab.shift[i / PoolAvgTab::kMax][i % PoolAvgTab::kMax]);
        }
        __syncthreads();
    }
    pdl_wait();
    pdl_trigger();
    constexpr int UW = KW + SW;   // columns of the union of the two windows
    const uint32_t cw = (uint32_t)g.c >> 2, cv = cw / W, owp = ((uint32_t)g.ow + 1) >> 1;
    for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
        const uint32_t ci = idx % cv;
        uint32_t pix = idx / cv;
        const uint32_t oxp = pix % owp;
        pix /= owp;
        const uint32_t oy = pix % (uint32_t)g.oh, n = pix / (uint32_t)g.oh;
        const int hs = (int)oy * g.stride_h - g.pad_h;
        const int ws = (int)oxp * 2 * SW - g.pad_w;
        const uint32_t *img = x + (size_t)n * (uint32_t)g.h * (uint32_t)g.w * cw + ci * W;
        uint32_t q[KH][UW][W];
#pragma unroll
        for (int r = 0; r < KH; ++r)
#pragma unroll
            for (int j = 0; j < UW; ++j) {
                const int iy = hs + r, ix = ws + j;
#pragma unroll
                for (int i = 0; i < W; ++i)
                    q[r][j][i] = 0;
                if ((unsigned)iy < (unsigned)g.h && (unsigned)ix < (unsigned)g.w)
                    load_vec<W>(img + ((uint32_t)iy * (uint32_t)g.w + (uint32_t)ix) * cw, q[r][j]);
            }
        auto join = [](const U16x4 &a, const U16x4 &b) {
            if constexpr (OP == kPairAve)
                return U16x4{ a.lo + b.lo, a.hi + b.hi };       // no carry between the lanes: sums stay below 2^16
            else
                return max_u16x4(a, b);
        };
        U16x4 s0[W], s1[W];
#pragma unroll
        for (int i = 0; i < W; ++i) {
            U16x4 col[UW];
#pragma unroll
            for (int j = 0; j < UW; ++j) {
                col[j] = spread_bytes(q[0][j][i]);
#pragma unroll
                for (int r = 1; r < KH; ++r)
                    col[j] = join(col[j], spread_bytes(q[r][j][i]));
            }
            s0[i] = col[0];
            s1[i] = col[SW];
#pragma unroll
            for (int j = 1; j < KW; ++j) {
                s0[i] = join(s0[i], col[j]);
                s1[i] = join(s1[i], col[SW + j]);
            }
        }
        uint32_t m0[W], m1[W];
        if constexpr (OP == kPairAve) {
            // valid taps, and the multiplier and shift of the window as the far edge (with its padding) cuts it
            const int vh = min(hs + KH, g.h) - max(hs, 0), dh = max(hs + KH - (g.h + g.pad_h), 0);
#pragma unroll
            for (int o = 0; o < 2; ++o) {
                const int wo = ws + o * SW;
                const int vw = min(wo + KW, g.w) - max(wo, 0), dw = min(max(wo + KW - (g.w + g.pad_w), 0), PoolAvgTab::kMax - 1);
                const int mult = mult_shift[dh][dw].x, sh = mult_shift[dh][dw].y;
                const int add = (1 << (sh - 1)) - mult * (max(vh, 0) * max(vw, 0) * g.izp);
#pragma unroll
                for (int i = 0; i < W; ++i) {
                    const U16x4 &s = o ? s1[i] : s0[i];
                    const int r0 = ((mult * (int)(s.lo & 0xffff) + add) >> sh) + g.ozp, r1 = ((mult * (int)(s.lo >> 16) + add) >> sh) + g.ozp;
                    const int r2 = ((mult * (int)(s.hi & 0xffff) + add) >> sh) + g.ozp, r3 = ((mult * (int)(s.hi >> 16) + add) >> sh) + g.ozp;
                    (o ? m1[i] : m0[i]) = pack_sat_u8x4(min(r0, g.qmax), min(r1, g.qmax), min(r2, g.qmax), min(r3, g.qmax));
                }
            }
        } else {
#pragma unroll
            for (int i = 0; i < W; ++i) {
                m0[i] = pack_bytes(s0[i]);
                m1[i] = pack_bytes(s1[i]);
                if (OP == kPairMaxLut) {
                    m0[i] = pack4(lut[m0[i] & 0xff], lut[(m0[i] >> 8) & 0xff], lut[(m0[i] >> 16) & 0xff], lut[m0[i] >> 24]);
                    m1[i] = pack4(lut[m1[i] & 0xff], lut[(m1[i] >> 8) & 0xff], lut[(m1[i] >> 16) & 0xff], lut[m1[i] >> 24]);
                }
            }
        }
        uint32_t *out = y + ((n * (uint32_t)g.oh + oy) * (uint32_t)g.ow + oxp * 2) * cw + ci * W;
        const bool second = oxp * 2 + 1 < (uint32_t)g.ow;
        if constexpr (W == 4) {
            *reinterpret_cast<uint4 *>(out) = make_uint4(m0[0], m0[1], m0[2], m0[3]);
            if (second)
                *reinterpret_cast<uint4 *>(out + cw) = make_uint4(m1[0], m1[1], m1[2], m1[3]);
        } else {
            out[0] = m0[0];
            if (second)
                out[cw] = m1[0];
        }
    }
}

template <int KH, int KW, int SW, PoolPairOp OP, int W>
static int pool_pair_launch(const uint8_t *x, uint8_t *y, const PoolGeom &g, const uint8_t *lut_dev, const PoolAvgTab &tab, size_t bytes,
                            cudaStream_t st)
{
    const size_t total = (size_t)g.n * g.oh * ((g.ow + 1) / 2) * (g.c / (4 * W));
    return launch_kernel(pool_pair_kernel<KH, KW, SW, OP, W>, dim3(resident_grid<pool_pair_kernel<KH, KW, SW, OP, W>, 256>((total + 255) / 256)),
                         dim3(256), 0, st, bytes, 1, reinterpret_cast<const uint32_t *>(x), reinterpret_cast<uint32_t *>(y), g, lut_dev, tab,
                         (uint32_t)total);
}

template <int KH, int KW, int SW>
static int pool_pair_pick(int method, int vec, const uint8_t *x, uint8_t *y, const PoolGeom &g, const uint8_t *lut_dev, const PoolAvgTab &tab,
                          size_t bytes, cudaStream_t st)
{
#define B200_PAIR(OP) return vec == 16 ? pool_pair_launch<KH, KW, SW, OP, 4>(x, y, g, lut_dev, tab, bytes, st) \
                                       : pool_pair_launch<KH, KW, SW, OP, 1>(x, y, g, lut_dev, tab, bytes, st)
    if (method == 1)
        B200_PAIR(kPairAve);
    if (g.lut_identity)
        B200_PAIR(kPairMaxIdent);
    B200_PAIR(kPairMaxLut);
#undef B200_PAIR
}

// AVE: sum of (x - izp) over the in-image part of the window; the multiplier and shift depend on
// the padded window size (pool.c:217-221) and come from a small host-built table indexed by how
// many rows / columns the window loses at the far edge.  The sums run on 16-bit lanes: pool_prepare
// admits at most 257 taps, 65535 a lane.
// LANES > 1: that many neighbouring lanes share an output, taking every LANES-th round of taps, for launches with few
// outputs and large windows, whose time is one thread's chain of loads (2048 channels of one 7x7 map: 10.8 us with one).
template <int VEC, int LANES = 1, bool ROWS = false>
__global__ void __launch_bounds__(256) pool_avg_kernel(
    const uint8_t *__restrict__ x, uint8_t *__restrict__ y, PoolGeom g, PoolAvgTab tab)
{
    pdl_wait();
    pdl_trigger();
    constexpr int W = (VEC + 3) / 4;
    const uint32_t cv = (uint32_t)(g.c / VEC);
    const size_t total = (size_t)g.n * g.oh * g.ow * cv;
    const int sub = threadIdx.x & (LANES - 1);
    // (LANES > 1 is launched with whole warps of work only, so that all lanes reach the shuffles)
    for (size_t idx = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / LANES; idx < total;
         idx += (size_t)gridDim.x * blockDim.x / LANES) {
        int ci = (int)(idx % cv);
        size_t pix = idx / cv;
        int ox = (int)(pix % g.ow);
        int oy = (int)((pix / g.ow) % g.oh);
        int n = (int)(pix / ((size_t)g.ow * g.oh));
        int hs = oy * g.stride_h - g.pad_h, ws = ox * g.stride_w - g.pad_w;
        int he = min(hs + g.kernel_h, g.h + g.pad_h), we = min(ws + g.kernel_w, g.w + g.pad_w);
        int dh = g.kernel_h - (he - hs), dw = g.kernel_w - (we - ws);   // rows / columns lost
        int mult = tab.mult[dh][dw], shift = tab.shift[dh][dw];
        hs = max(hs, 0);
        ws = max(ws, 0);
        he = min(he, g.h);
        we = min(we, g.w);
        U16x4 sum[W];
#pragma unroll
        for (int j = 0; j < W; ++j)
            sum[j] = { 0u, 0u };
        const int wd = max(we - ws, 0), cnt = max(he - hs, 0) * wd;
        // eight taps per round, loaded before any is used: a large window (the global average of a 7x7 map is 49 taps)
        // keeps several loads in flight
        constexpr int UNR = 8;
        auto add = [&](const uint32_t (&v)[UNR][W]) {
#pragma unroll
            for (int u = 0; u < UNR; ++u)
#pragma unroll
                for (int j = 0; j < W; ++j) {
                    const U16x4 b = spread_bytes(v[u][j]);
                    sum[j].lo += b.lo;
                    sum[j].hi += b.hi;
                }
        };
        if constexpr (ROWS) {
            for (int iy = hs; iy < he; ++iy) {
                const uint8_t *row = x + (((size_t)n * g.h + iy) * g.w) * g.c + (size_t)ci * VEC;
                for (int ix = ws; ix < we; ix += UNR) {
                    uint32_t v[UNR][W];
#pragma unroll
                    for (int u = 0; u < UNR; ++u) {
#pragma unroll
                        for (int j = 0; j < W; ++j)
                            v[u][j] = 0;
                        if (ix + u < we)
                            load_words<VEC>(row + (size_t)(ix + u) * g.c, v[u]);
                    }
                    add(v);
                }
            }
        } else {
            const uint8_t *base = x + (((size_t)n * g.h + hs) * g.w + ws) * g.c + (size_t)ci * VEC;
            int ty = 0, tx = 0;
            if (LANES > 1 && wd > 0) {
                ty = sub * UNR / wd;
                tx = sub * UNR - ty * wd;
            }
            for (int t = sub * UNR; t < cnt; t += UNR * LANES) {
                uint32_t v[UNR][W];
#pragma unroll
                for (int u = 0; u < UNR; ++u) {
#pragma unroll
                    for (int j = 0; j < W; ++j)
                        v[u][j] = 0;
                    if (t + u < cnt) {
                        load_words<VEC>(base + (size_t)(ty * g.w + tx) * g.c, v[u]);
                        if (++tx == wd) {
                            tx = 0;
                            ++ty;
                        }
                    }
                }
                add(v);
                if (LANES > 1 && t + UNR * LANES < cnt) {
                    const int at = t + UNR * LANES;
                    ty = at / wd;
                    tx = at - ty * wd;
                }
            }
        }
#pragma unroll
        for (int m = 1; m < LANES; m *= 2)
#pragma unroll
            for (int j = 0; j < W; ++j) {
                sum[j].lo += __shfl_xor_sync(0xffffffffu, sum[j].lo, m);
                sum[j].hi += __shfl_xor_sync(0xffffffffu, sum[j].hi, m);
            }
        uint32_t o[W];
#pragma unroll
        for (int j = 0; j < W; ++j)
            o[j] = 0;
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
            const uint32_t lanes = j % 4 < 2 ? sum[j / 4].lo : sum[j / 4].hi;
            int s = (int)((lanes >> (16 * (j % 2))) & 0xffff) - cnt * g.izp;
            // (int32)mult * sum is an int32 product in the reference; rshift_rn then runs on the
            // sign-extended value.
            long long p = (long long)(mult * s);
            int v = (int)(rshift_rn64(p, shift) + g.ozp);
            v = min(max(v, 0), g.qmax);
            o[j / 4] |= (uint32_t)v << (8 * (j % 4));
        }
        if (sub == 0)
            store_words<VEC>(y + pix * g.c + (size_t)ci * VEC, o);
    }
}

static int pool_out_dim(int in, int kernel, int pad, int stride, int ceil_mode, int any_pad)
{
    // art/src/op.c:934-956: double arithmetic, then one step back if the last window would start
    // at or beyond in + pad (only when some padding is set).
    double v = (in + pad * 2.0 - kernel) / stride + 1;
    int o = (int)(ceil_mode ? ceil(v) : floor(v));
    if (any_pad && (o - 1) * stride >= in + pad)
        --o;
    return o;
}

int pool_prepare(
    int h, int w, int method, int kernel_h, int kernel_w, int pad_h, int pad_w, int stride_h,
    int stride_w, int ceil_mode, float ialpha, uint8_t izp, float oalpha, uint8_t ozp,
    uint8_t obits, PoolGeom *g, uint8_t lut[256], PoolAvgTab *tab)
{
    if (h <= 0 || w <= 0 || kernel_h <= 0 || kernel_w <= 0 || stride_h <= 0 || stride_w <= 0
        || pad_h < 0 || pad_w < 0 || obits < 1 || obits > 8 || (method != 0 && method != 1))
        return fail(B200_ERR_INVALID, "pool: bad geometry");
    if (!(ialpha > 0.f) || !(oalpha > 0.f))
        return fail(B200_ERR_INVALID, "pool: scales must be positive");
    int any_pad = pad_h || pad_w;
    g->h = h; g->w = w;
    g->oh = pool_out_dim(h, kernel_h, pad_h, stride_h, ceil_mode, any_pad);
    g->ow = pool_out_dim(w, kernel_w, pad_w, stride_w, ceil_mode, any_pad);
    if (g->oh <= 0 || g->ow <= 0)
        return fail(B200_ERR_INVALID, "pool: empty output");
    g->kernel_h = kernel_h; g->kernel_w = kernel_w; g->pad_h = pad_h; g->pad_w = pad_w;
    g->stride_h = stride_h; g->stride_w = stride_w;
    g->izp = izp; g->ozp = ozp; g->qmax = (1 << obits) - 1;
    g->lut_identity = 0;
    g->avg32 = 1;
    const int qmax = g->qmax;
    if (method == 0) {
        uint32_t m16;
        int8_t sh;
        get_quant_scale(ialpha / oalpha, -16, &m16, &sh);
        if (sh < 1 || sh > 62)
            return fail(B200_ERR_UNSUPPORTED, "pool: shift %d outside 1..62", (int)sh);
        for (int q = 0; q < 256; ++q) {
            int32_t prod = (int32_t)m16 * (q - (int)izp);
            int32_t r = (int32_t)(rshift_rn_host(prod, sh) + ozp);
            lut[q] = (uint8_t)(r > qmax ? qmax : (r < 0 ? 0 : r));
        }
        g->lut_identity = 1;
        for (int q = 0; q < 256; ++q)
            if (lut[q] != q)
                g->lut_identity = 0;
    } else {
        // the windows at the far edge may be cut by `in + pad` (ceil mode): index the table by the
        // number of rows / columns cut
        int max_dh = 0, max_dw = 0;
        for (int oy = 0; oy < g->oh; ++oy) {
            int hs = oy * stride_h - pad_h;
            int d = hs + kernel_h - (h + pad_h);
            if (d > max_dh) max_dh = d;
        }
        for (int ox = 0; ox < g->ow; ++ox) {
            int ws = ox * stride_w - pad_w;
            int d = ws + kernel_w - (w + pad_w);
            if (d > max_dw) max_dw = d;
        }
        if (max_dh >= PoolAvgTab::kMax || max_dw >= PoolAvgTab::kMax)
            return fail(B200_ERR_UNSUPPORTED, "pool: window cut by %d/%d rows/cols at the edge", max_dh, max_dw);
        if ((long long)kernel_h * kernel_w * 255 * 32768 >= (1ll << 31))
            return fail(B200_ERR_UNSUPPORTED, "pool: average window too large for the int32 product");
        for (int dh = 0; dh < PoolAvgTab::kMax; ++dh)
            for (int dw = 0; dw < PoolAvgTab::kMax; ++dw) {
                tab->mult[dh][dw] = 0;
                tab->shift[dh][dw] = 1;
                if (dh > max_dh || dw > max_dw)
                    continue;
                uint32_t pool_size = (uint32_t)((kernel_h - dh) * (kernel_w - dw));
                if (pool_size == 0)
                    continue;
                uint32_t m;
                int8_t sh;
                get_quant_scale(ialpha / oalpha / pool_size, 16, &m, &sh);   // pool.c:221
                if (sh < 1 || sh > 62)
                    return fail(B200_ERR_UNSUPPORTED, "pool: shift %d outside 1..62", (int)sh);
                tab->mult[dh][dw] = (int)m;
                tab->shift[dh][dw] = sh;
                if (sh > 30 || (long long)kernel_h * kernel_w * 255 * m + (1ll << (sh - 1)) >= (1ll << 31))
                    g->avg32 = 0;
            }
    }
    return B200_OK;
}

int pool_launch(
    const uint8_t *x, uint8_t *y, int n, int c, int method, const PoolGeom &g0, const uint8_t *lut_dev,
    const PoolAvgTab &tab, cudaStream_t st)
{
    PoolGeom g = g0;
    g.n = n;
    g.c = c;
    if (n == 0)
        return B200_OK;
    int vec = (c % 16 == 0 && (((uintptr_t)x | (uintptr_t)y) & 15) == 0) ? 16
        : (c % 4 == 0 && (((uintptr_t)x | (uintptr_t)y) & 3) == 0)       ? 4
                                                                           : 1;
    const size_t bytes = (size_t)n * c * (g.h * g.w + g.oh * g.ow);
    // two outputs per thread, unrolled window, 32-bit indices: the common window shapes
    // (words of the input and, where the padding makes it the larger one, of the output; threads, with room for a grid past the end)
    if (vec >= 4 && (size_t)n * g.h * g.w * (c / 4) < 0xffffffffull && (size_t)n * g.oh * g.ow * (c / 4) < 0xffffffffull
        && (size_t)n * g.oh * ((g.ow + 1) / 2) * (c / vec) < 0xffffffffull - 256ull * 65536ull && (method == 0 || g.avg32)) {
        if (g.kernel_h == 3 && g.kernel_w == 3 && g.stride_w == 2)
            return pool_pair_pick<3, 3, 2>(method, vec, x, y, g, lut_dev, tab, bytes, st);
        if (g.kernel_h == 3 && g.kernel_w == 3 && g.stride_w == 1)
            return pool_pair_pick<3, 3, 1>(method, vec, x, y, g, lut_dev, tab, bytes, st);
        if (g.kernel_h == 2 && g.kernel_w == 2 && g.stride_w == 2)
            return pool_pair_pick<2, 2, 2>(method, vec, x, y, g, lut_dev, tab, bytes, st);
    }
    // an average whose 16-byte vectors would leave the SMs a few warps each goes by words: four times the threads for a chain of
    // loads (2048 channels of one 7x7 window, batch 256: 221 vectors an SM).  Beyond that the vectors win: 7x7 stride 7 on 256
    // channels of 56 x 56, batch 64, 443 an SM: 23.1 us by words, 15.5; 7x7 on 64 of 71 x 71, batch 8, 913: 36.4 and 19.6.
    if (method == 1 && vec == 16 && (size_t)n * g.oh * g.ow * (c / 16) < (size_t)sm_count() * 256)
        vec = 4;
    const size_t outs = (size_t)n * g.oh * g.ow * (c / vec), blocks = (outs + 255) / 256;
    if (method == 1 && vec == 4 && outs % 4 == 0 && outs * 8 <= (size_t)sm_count() * 2048 && g.kernel_h * g.kernel_w >= 16)
        return launch_kernel(pool_avg_kernel<4, 8>, dim3((unsigned)((outs * 8 + 255) / 256)), dim3(256), 0, st, bytes, 1, x, y, g, tab);
    if (method == 0) {
        if (vec == 16) return launch_kernel(pool_max_kernel<16>, dim3(resident_grid<pool_max_kernel<16>, 256>(blocks)), dim3(256), 0, st, bytes, 1, x, y, g, lut_dev);
        if (vec == 4) return launch_kernel(pool_max_kernel<4>, dim3(resident_grid<pool_max_kernel<4>, 256>(blocks)), dim3(256), 0, st, bytes, 1, x, y, g, lut_dev);
        return launch_kernel(pool_max_kernel<1>, dim3(resident_grid<pool_max_kernel<1>, 256>(blocks)), dim3(256), 0, st, bytes, 1, x, y, g, lut_dev);
    } else {
#define B200_AVG(...) return launch_kernel(pool_avg_kernel<__VA_ARGS__>, dim3(resident_grid<pool_avg_kernel<__VA_ARGS__>, 256>(blocks)), dim3(256), 0, st, bytes, 1, x, y, g, tab)
        // A window's taps as one sequence take the fewest rounds of loads, which counts while a launch is one thread's chain of
        // them; row by row they take fewer instructions, which counts once the GPU is full and where rows fill their rounds of
        // eight (7x7 stride 1, 7 channels of 56 x 56, batch 64: 65.3 and 52.9 us; 40 channels of 14 x 14: 6.8 and 8.8).
        // Sixteen channels a thread are bound by neither: 29.2 and 31.2 us (256 channels of 28 x 28, batch 32).
        const bool rows = (g.kernel_w + 7) / 8 * 7 <= g.kernel_w && outs >= (size_t)sm_count() * (vec == 1 ? 1024 : 4096);
        if (vec == 16) B200_AVG(16);
        if (vec == 4 && rows) B200_AVG(4, 1, true);
        if (vec == 4) B200_AVG(4);
        if (rows) B200_AVG(1, 1, true);
        B200_AVG(1);
#undef B200_AVG
    }
}

}  // namespace b200

using namespace b200;

extern "C" {

int b200_pool_out_dims(
    int32_t h, int32_t w, int32_t kernel_h, int32_t kernel_w, int32_t pad_h, int32_t pad_w,
    int32_t stride_h, int32_t stride_w, int32_t ceil_mode, int32_t *oh, int32_t *ow)
{
    if (!oh || !ow || stride_h <= 0 || stride_w <= 0)
        return fail(B200_ERR_INVALID, "pool_out_dims: bad argument");
    int any_pad = pad_h || pad_w;
    *oh = pool_out_dim(h, kernel_h, pad_h, stride_h, ceil_mode, any_pad);
    *ow = pool_out_dim(w, kernel_w, pad_w, stride_w, ceil_mode, any_pad);
    return B200_OK;
}

int b200_pool_u8(
    const uint8_t *x, int32_t n, int32_t c, int32_t h, int32_t w, int32_t method, int32_t kernel_h,
    int32_t kernel_w, int32_t pad_h, int32_t pad_w, int32_t stride_h, int32_t stride_w,
    int32_t ceil_mode, float ialpha, uint8_t izp, float oalpha, uint8_t ozp, uint8_t obits,
    uint8_t *y, b200_stream_t stream)
{
    if (!x || !y || n < 0 || c <= 0)
        return fail(B200_ERR_INVALID, "pool: bad argument");
    PoolGeom g;
    PoolAvgTab tab;
    uint8_t lut[256];
    B200_TRY(pool_prepare(
        h, w, method, kernel_h, kernel_w, pad_h, pad_w, stride_h, stride_w, ceil_mode, ialpha, izp,
        oalpha, ozp, obits, &g, lut, &tab));
    cudaStream_t st = as_stream(stream);
    const uint8_t *lut_dev = nullptr;
    if (method == 0)
        B200_TRY(lut_cache_get(lut, &lut_dev));   // uploaded once per distinct table, then reused
    return pool_launch(x, y, n, c, method, g, lut_dev, tab, st);
}

}  // extern "C"
