// Bandwidth-bound uint8 ops around the quantized convolution: quantize / dequantize with the
// NCHW <-> NHWC transpose fused in, plain layout changes, eltwise SUM (add) and relu.  All are
// CUDA-core kernels measured against HBM bandwidth: every global access is a full-sector,
// coalesced or 16-byte vector access.
#include "common.cuh"
#include "kernels.h"

namespace b200 {

// ---------------------------------------------------------------------------------------------
// [N][C][P] (P = H*W, the reference's NCHW) to and from [N][P][Cpad] (NHWC), the element conversion
// (quantize, dequantize or none) on the way.  A thread owns 32 channels of one pixel: on the NCHW side
// neighbouring threads read or write neighbouring elements of every channel plane, whatever P is, and
// on the NHWC side a thread's 32 bytes are one sector.  Nothing passes through shared memory.  Pixels
// are numbered through all images of the batch, so that small maps fill their blocks too.
// ---------------------------------------------------------------------------------------------
constexpr int TC = 32;          // channels per thread
constexpr int kLayoutThreads = 256;

struct QuantizeFn {
    // op_quantize_run_u8 (quantize.c:145-157) with saturate_float_by_bits (quant_helper.h:38-41):
    // t = (x - beta) / alpha in fp32 with beta = -(alpha * zp); the reference then truncates
    // (double)t + 0.5, which for 0 <= t <= qmax equals floor(t) + (t - floor(t) >= 0.5), exact in
    // fp32.  __fsub_rn/__fdiv_rn keep the two roundings separate (no contraction).
    float alpha, beta;
    int qmax;
    // The divide bounds the op (1.9 TB/s at 25.7 M elements).  u = x * inv + (zp + 0.5) differs from
    // t + 0.5 by less than 2^-13 for t in -1 .. 256: the roundings of inv, beta, x - beta, t and of the
    // multiply-add are at most 2^-24 of numbers below 512 each.  So floor(u) is the answer unless u lies
    // within 2^-12 of an integer, and only those (one element in 2000 of evenly spread data) are divided.
    float inv, half_zp;
    bool fast;                  // alpha is far from the ends of the fp32 range (else inv and u mean nothing)
    __device__ __forceinline__ uint8_t operator()(float x) const
    {
        float t = __fdiv_rn(__fsub_rn(x, beta), alpha);
        if (t > (float)qmax)
            return (uint8_t)qmax;
        if (t < 0.f)
            return 0;
        if (!(t == t))
            return 0;  // NaN: undefined in the reference
        float f = floorf(t);
        int v = (int)f + ((t - f) >= 0.5f ? 1 : 0);
        return (uint8_t)v;
    }
    __device__ __forceinline__ uint32_t word(float a, float b, float c, float d) const
    {
        const float x[4] = { a, b, c, d };
        uint32_t r[4];
        bool sure = fast;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            // (maximum and minimum return the number where one operand is NaN: 0 comes out, as above)
            const float u = fminf(fmaxf(__fmaf_rn(x[i], inv, half_zp), 0.5f), (float)qmax + 0.5f);
            const float big = __fadd_rz(u, 8388608.f);          // 2^23 + floor(u): the integer in the low bits
            const float centre = __fsub_rn(big, 8388607.5f);    // floor(u) + 0.5
            sure = sure && fabsf(__fsub_rn(u, centre)) < 0.5f - 0x1p-12f;
            r[i] = __float_as_uint(big);
        }
        if (!sure) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                r[i] = (*this)(x[i]);
        }
        return __byte_perm(__byte_perm(r[0], r[1], 0x0040), __byte_perm(r[2], r[3], 0x0040), 0x5410);
    }
};

struct DequantizeFn {
    // op_dequantize_run_u8 (dequantize.c:111-123): ((int16)q - zp) * alpha, int -> float multiply.
    float alpha;
    int zp;
    __device__ __forceinline__ float operator()(uint8_t q) const
    {
        return __fmul_rn((float)((int)q - zp), alpha);
    }
};

struct QuantizeS8Fn {
    // op_quantize_run_i8 (quantize.c:159-185): clip(round(x * alpha), -l, l) with alpha = (float)(1. / oalpha)
    // (formed on the host), the float product rounded half away from zero -- roundf of the float equals the
    // reference's round() of the same value widened to double -- and the clip done on the rounded value.
    float alpha;
    int l;
    __device__ __forceinline__ uint8_t operator()(float x) const
    {
        const float r = roundf(__fmul_rn(x, alpha));
        if (!(r == r))
            return 0;  // NaN: undefined in the reference
        const int v = (int)fminf(fmaxf(r, (float)-l), (float)l);
        return (uint8_t)(int8_t)v;
    }
    __device__ __forceinline__ uint32_t word(float a, float b, float c, float d) const
    {
        return pack4((*this)(a), (*this)(b), (*this)(c), (*this)(d));
    }
};

struct DequantizeS8Fn {
    // op_dequantize_run_i8 (dequantize.c:124-136): the int8 value as float, times alpha
    float alpha;
    __device__ __forceinline__ float operator()(uint8_t q) const { return __fmul_rn((float)(int)(int8_t)q, alpha); }
};

struct IdentityFn {
    __device__ __forceinline__ uint8_t operator()(uint8_t q) const { return q; }
    __device__ __forceinline__ uint32_t word(uint8_t a, uint8_t b, uint8_t c, uint8_t d) const { return pack4(a, b, c, d); }
};

// in: [N][C][P] of TIn  ->  out: [N][P][c_pad] of uint8; channels c..c_pad-1 are written `fill`.
// STORE: bytes per store (16 or 4, which divide c_pad and the address, or 1).
template <typename TIn, typename Fn, int STORE>
__global__ void __launch_bounds__(kLayoutThreads) nchw_to_nhwc_kernel(
    const TIn *__restrict__ in, uint8_t *__restrict__ out, int C, uint32_t P, int c_pad, int fill, uint32_t pixels, uint32_t groups, Fn fn)
{
    pdl_wait();
    pdl_trigger();
    // the channel groups of a pixel block are neighbouring blocks: they share the NHWC side's lines
    const uint32_t block = blockIdx.x / groups, gp = block * kLayoutThreads + threadIdx.x;
    if (gp >= pixels)
        return;
    const int c0 = (int)(blockIdx.x - block * groups) * TC;
    const uint32_t img = gp / P, p = gp - img * P;
    const TIn *src = in + ((size_t)img * C + c0) * P + p;
    uint8_t *dst = out + (size_t)gp * c_pad + c0;
    if (c0 + TC <= C && STORE != 1) {
        TIn v[TC];
#pragma unroll
        for (int c = 0; c < TC; ++c)
            v[c] = __ldg(src + (size_t)c * P);
        uint32_t wv[TC / 4];
#pragma unroll
        for (int j = 0; j < TC / 4; ++j)
            wv[j] = fn.word(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        if (STORE == 16) {
            reinterpret_cast<uint4 *>(dst)[0] = make_uint4(wv[0], wv[1], wv[2], wv[3]);
            reinterpret_cast<uint4 *>(dst)[1] = make_uint4(wv[4], wv[5], wv[6], wv[7]);
        } else {
            // rows at word addresses only: the words change hands inside the warp, so that eight lanes write the
            // 32 bytes of one pixel and not 32 lanes a word each of 32 pixels (16 M elements of 236 channels: 27.5 us so)
            __shared__ uint32_t tile[kLayoutThreads / 32][32][TC / 4 + 1];
            uint32_t (*t)[TC / 4 + 1] = tile[threadIdx.x / 32];
            const unsigned lane = threadIdx.x & 31;
            const unsigned live = min(32u, pixels - (gp - lane));         // the lanes that are here: a prefix of the warp
            const unsigned active = 0xffffffffu >> (32 - live);
#pragma unroll
            for (int j = 0; j < TC / 4; ++j)
                t[lane][j] = wv[j];
            __syncwarp(active);
            uint8_t *first = out + (size_t)(gp - lane) * c_pad + c0;      // the warp's first pixel
            for (unsigned i = lane; i < live * (TC / 4); i += live)
                *reinterpret_cast<uint32_t *>(first + (size_t)(i / (TC / 4)) * c_pad + (i % (TC / 4)) * 4) = t[i / (TC / 4)][i % (TC / 4)];
        }
        return;
    }
    // the last, narrower group of channels, and rows that no word store fits
    const int cend = min(TC, c_pad - c0);
#pragma unroll 4
    for (int c = 0; c < cend; c += 4) {
        TIn v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
            v[i] = c0 + c + i < C ? __ldg(src + (size_t)(c + i) * P) : TIn(0);
        uint32_t wv = fn.word(v[0], v[1], v[2], v[3]);
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (c0 + c + i >= C)
                wv = (wv & ~(0xffu << (8 * i))) | ((uint32_t)fill << (8 * i));
        if (STORE != 1) {
            *reinterpret_cast<uint32_t *>(dst + c) = wv;
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (c + i < cend)
                    dst[c + i] = (uint8_t)(wv >> (8 * i));
        }
    }
}

// in: [N][P][c_pad] uint8 -> out: [N][C][P] of TOut (channels >= C are dropped).
// LOAD: bytes per load, as STORE above.
template <typename TOut, typename Fn, int LOAD>
__global__ void __launch_bounds__(kLayoutThreads) nhwc_to_nchw_kernel(
    const uint8_t *__restrict__ in, TOut *__restrict__ out, int C, uint32_t P, int c_pad, uint32_t pixels, uint32_t groups, Fn fn)
{
    pdl_wait();
    pdl_trigger();
    // the channel groups of a pixel block are neighbouring blocks: they share the NHWC side's lines
    const uint32_t block = blockIdx.x / groups, gp = block * kLayoutThreads + threadIdx.x;
    if (gp >= pixels)
        return;
    const int c0 = (int)(blockIdx.x - block * groups) * TC;
    const uint32_t img = gp / P, p = gp - img * P;
    const uint8_t *src = in + (size_t)gp * c_pad + c0;
    TOut *dst = out + ((size_t)img * C + c0) * P + p;
    if (c0 + TC <= C && LOAD != 1) {
        uint32_t wv[TC / 4];
        if (LOAD == 16) {
            const uint4 a = __ldg(reinterpret_cast<const uint4 *>(src)), b = __ldg(reinterpret_cast<const uint4 *>(src) + 1);
            wv[0] = a.x; wv[1] = a.y; wv[2] = a.z; wv[3] = a.w; wv[4] = b.x; wv[5] = b.y; wv[6] = b.z; wv[7] = b.w;
        } else {
#pragma unroll
            for (int j = 0; j < TC / 4; ++j)
                wv[j] = __ldg(reinterpret_cast<const uint32_t *>(src) + j);
        }
#pragma unroll
        for (int c = 0; c < TC; ++c)
            dst[(size_t)c * P] = fn((uint8_t)(wv[c / 4] >> (8 * (c % 4))));
        return;
    }
    const int cend = min(TC, C - c0);
#pragma unroll 4
    for (int c = 0; c < cend; c += 4) {
        uint32_t wv = 0;
        if (LOAD != 1) {
            wv = __ldg(reinterpret_cast<const uint32_t *>(src + c));
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (c + i < cend)
                    wv |= (uint32_t)__ldg(src + c + i) << (8 * i);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (c + i < cend)
                dst[(size_t)(c + i) * P] = fn((uint8_t)(wv >> (8 * i)));
    }
}

// The kernels number pixels with 32 bits: larger batches go in several launches.  run(first image, images) does one.
template <typename Run>
static int in_image_slices(int n, int P, int channels, Run run)
{
    const size_t groups = ((size_t)channels + TC - 1) / TC;
    const size_t blocks = 0x7fffffffull / groups;                       // of kLayoutThreads pixels
    const size_t most = blocks * kLayoutThreads < 0xffffff00ull ? blocks * kLayoutThreads : 0xffffff00ull;
    const size_t images = (size_t)P > most ? 0 : most / P;
    if (images == 0)
        return fail(B200_ERR_UNSUPPORTED, "layout: more than 2^31 blocks an image");
    for (size_t i = 0; i < (size_t)n; i += images)
        B200_TRY(run(i, (size_t)n - i < images ? (size_t)n - i : images));
    return B200_OK;
}

template <typename TIn, typename Fn>
static int nchw_to_nhwc_launch(const TIn *x0, uint8_t *y0, int n, int c, int P, int c_pad, int fill, Fn fn, cudaStream_t st)
{
    return in_image_slices(n, P, c_pad, [=](size_t first, size_t images) {
        const TIn *x = x0 + first * c * P;
        uint8_t *y = y0 + first * c_pad * P;
        const size_t pixels = images * P, groups = ((size_t)c_pad + TC - 1) / TC;
        const dim3 grid((unsigned)((pixels + kLayoutThreads - 1) / kLayoutThreads * groups));
        const size_t bytes = pixels * (c * sizeof(TIn) + c_pad);
        const bool a16 = c_pad % 16 == 0 && ((uintptr_t)y & 15) == 0, a4 = c_pad % 4 == 0 && ((uintptr_t)y & 3) == 0;
        if (a16)
            return launch_kernel(nchw_to_nhwc_kernel<TIn, Fn, 16>, grid, dim3(kLayoutThreads), 0, st, bytes, 1, x, y, c, P, c_pad, fill, pixels, groups, fn);
        if (a4)
            return launch_kernel(nchw_to_nhwc_kernel<TIn, Fn, 4>, grid, dim3(kLayoutThreads), 0, st, bytes, 1, x, y, c, P, c_pad, fill, pixels, groups, fn);
        return launch_kernel(nchw_to_nhwc_kernel<TIn, Fn, 1>, grid, dim3(kLayoutThreads), 0, st, bytes, 1, x, y, c, P, c_pad, fill, pixels, groups, fn);
    });
}

template <typename TOut, typename Fn>
static int nhwc_to_nchw_launch(const uint8_t *x0, TOut *y0, int n, int c, int P, int c_pad, Fn fn, cudaStream_t st)
{
    return in_image_slices(n, P, c, [=](size_t first, size_t images) {
        const uint8_t *x = x0 + first * c_pad * P;
        TOut *y = y0 + first * c * P;
        const size_t pixels = images * P, groups = ((size_t)c + TC - 1) / TC;
        const dim3 grid((unsigned)((pixels + kLayoutThreads - 1) / kLayoutThreads * groups));
        const size_t bytes = pixels * (c * sizeof(TOut) + c_pad);
        const bool a16 = c_pad % 16 == 0 && ((uintptr_t)x & 15) == 0, a4 = c_pad % 4 == 0 && ((uintptr_t)x & 3) == 0;
        if (a16)
            return launch_kernel(nhwc_to_nchw_kernel<TOut, Fn, 16>, grid, dim3(kLayoutThreads), 0, st, bytes, 1, x, y, c, P, c_pad, pixels, groups, fn);
        if (a4)
            return launch_kernel(nhwc_to_nchw_kernel<TOut, Fn, 4>, grid, dim3(kLayoutThreads), 0, st, bytes, 1, x, y, c, P, c_pad, pixels, groups, fn);
        return launch_kernel(nhwc_to_nchw_kernel<TOut, Fn, 1>, grid, dim3(kLayoutThreads), 0, st, bytes, 1, x, y, c, P, c_pad, pixels, groups, fn);
    });
}

// Flat variants (no layout change): 4 elements per thread, as vectors where both addresses allow it (VEC).
template <typename Fn, bool VEC>
__global__ void quantize_flat_kernel(const float *__restrict__ in, uint8_t *__restrict__ out, size_t count, Fn fn)
{
    pdl_wait();
    pdl_trigger();
    size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (VEC && i + 4 <= count) {
        float4 v = *reinterpret_cast<const float4 *>(in + i);
        *reinterpret_cast<uint32_t *>(out + i) = fn.word(v.x, v.y, v.z, v.w);
    } else {
        const size_t end = i + 4 < count ? i + 4 : count;
        for (; i < end; ++i)
            out[i] = fn(in[i]);
    }
}

// word: a status word that leaves for the host with this launch (see status_publish_launch), or nullptr
template <typename Fn, bool VEC>
__global__ void dequantize_flat_kernel(const uint8_t *__restrict__ in, float *__restrict__ out, size_t count, Fn fn, int *word, int *host)
{
    pdl_wait();
    pdl_trigger();
    if (word != nullptr && blockIdx.x == 0 && threadIdx.x == 0)
        status_publish(word, host);
    size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (VEC && i + 4 <= count) {
        uint32_t q = *reinterpret_cast<const uint32_t *>(in + i);
        *reinterpret_cast<float4 *>(out + i) = make_float4(
            fn((uint8_t)q), fn((uint8_t)(q >> 8)), fn((uint8_t)(q >> 16)), fn((uint8_t)(q >> 24)));
    } else {
        const size_t end = i + 4 < count ? i + 4 : count;
        for (; i < end; ++i)
            out[i] = fn(in[i]);
    }
}

template <typename Fn>
static int quantize_flat_launch(const float *x, uint8_t *y, size_t count, Fn fn, cudaStream_t st)
{
    const dim3 grid((unsigned)(((count + 3) / 4 + 255) / 256));
    if ((((uintptr_t)x & 15) | ((uintptr_t)y & 3)) == 0)
        return launch_kernel(quantize_flat_kernel<Fn, true>, grid, dim3(256), 0, st, count * 5, 1, x, y, count, fn);
    return launch_kernel(quantize_flat_kernel<Fn, false>, grid, dim3(256), 0, st, count * 5, 1, x, y, count, fn);
}
template <typename Fn>
static int dequantize_flat_launch(const uint8_t *x, float *y, size_t count, Fn fn, cudaStream_t st, int *word = nullptr, int *host = nullptr)
{
    const dim3 grid((unsigned)(((count + 3) / 4 + 255) / 256));
    if ((((uintptr_t)x & 3) | ((uintptr_t)y & 15)) == 0)
        return launch_kernel(dequantize_flat_kernel<Fn, true>, grid, dim3(256), 0, st, count * 5, 1, x, y, count, fn, word, host);
    return launch_kernel(dequantize_flat_kernel<Fn, false>, grid, dim3(256), 0, st, count * 5, 1, x, y, count, fn, word, host);
}

// ---------------------------------------------------------------------------------------------
// eltwise SUM (eltwise.c:137-174): per input i, term_i = rshift_rn((x_i - zp_i) * m_i, b_i) with
// b_i = s_i - s0; t = sum term_i; y = sat_u(rshift_rn(t, s0) + ozp).  With
// rshift_rn(v, b) = (v + 2^(b-1)) >> b the term is (x_i * m_i + add_i) >> b_i where
// add_i = 2^(b_i-1) - zp_i * m_i is built on the host, one multiply-add and one shift per input.
// m_i < 2^22, so every intermediate fits int32 for b_i <= 30.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ int elt_finish(int t, const EltwiseArgs &a)
{
    int v = ((t + a.round0) >> a.s0) + a.ozp;
    return sat_relu(v, a.qmax, a.relu_lo);
}

// FAST: obits == 8 and the final rounding term 2^(s0-1) << b[0] fits into add[0] (folded there by
// the host, exact because it is a multiple of 2^b[0]); then y = sat_u8(max((t >> s0) + ozp, relu_lo))
// and the saturation comes with the pack.  64 bytes per input per thread and iteration.
// PLAIN (with FAST): ozp == 0 and no floor above 0, so y = sat_u8(t >> s0) and the pack does the rest.
// VPT: 16-byte vectors per input and thread (2: 0.80 ms, 4: 0.78 ms, 8: 0.79 ms for the 16 adds of ResNet-50 at
// batch 256).  One where four would leave SMs without a block: the time is then one thread's.
template <int N_IN, bool FAST, bool PLAIN = false, bool REV = false, int VPT = 4>
__global__ void __launch_bounds__(256) eltwise_sum_kernel(EltwiseArgs a, uint8_t *__restrict__ y, size_t count)
{
    pdl_wait();
    pdl_trigger();
    const size_t nvec = count / 16;
    // a block works on tiles of 256 * VPT vectors; vector u of a thread lies 256 vectors after vector
    // u - 1, so that every load and store instruction of a warp covers 512 contiguous bytes
    auto load = [&](uint32_t (&xin)[N_IN][4], size_t v) {
#pragma unroll
        for (int i = 0; i < N_IN; ++i) {
            const uint4 q = __ldg(reinterpret_cast<const uint4 *>(a.x[i]) + v);
            xin[i][0] = q.x; xin[i][1] = q.y; xin[i][2] = q.z; xin[i][3] = q.w;
        }
    };
    auto sum = [&](const uint32_t (&xin)[N_IN][4]) {
        uint32_t o[4];
#pragma unroll
        for (int wd = 0; wd < 4; ++wd) {
            int r[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                int t = 0;
#pragma unroll
                for (int i = 0; i < N_IN; ++i) {
                    const int xv = (int)__byte_perm(xin[i][wd], 0, 0x4440 | e);   // byte e, zero-extended
                    t += (xv * a.m[i] + a.add[i]) >> a.b[i];
                }
                r[e] = PLAIN ? (t >> a.s0) : (FAST ? max((t >> a.s0) + a.ozp, a.relu_lo) : elt_finish(t, a));
            }
            o[wd] = FAST ? pack_sat_u8x4(r[0], r[1], r[2], r[3]) : pack4(r[0], r[1], r[2], r[3]);
        }
        return make_uint4(o[0], o[1], o[2], o[3]);
    };
    const size_t ntile = nvec / (256 * VPT);
    for (size_t tile_i = blockIdx.x; tile_i < ntile; tile_i += gridDim.x) {
        const size_t tile = REV ? ntile - 1 - tile_i : tile_i;   // REV: from the last tile to the first
        const size_t v0 = tile * (256 * VPT) + threadIdx.x;
        uint32_t xin[VPT][N_IN][4];
#pragma unroll
        for (int u = 0; u < VPT; ++u)
            load(xin[u], v0 + u * 256);
        uint4 o[VPT];
#pragma unroll
        for (int u = 0; u < VPT; ++u)
            o[u] = sum(xin[u]);
#pragma unroll
        for (int u = 0; u < VPT; ++u)
            reinterpret_cast<uint4 *>(y)[v0 + u * 256] = o[u];
    }
    // the vectors behind the last whole tile: fewer than 256 * VPT, over as many blocks as they fill
    for (size_t v = ntile * (256 * VPT) + (size_t)blockIdx.x * 256 + threadIdx.x; v < nvec; v += (size_t)gridDim.x * 256) {
        uint32_t xin[N_IN][4];
        load(xin, v);
        reinterpret_cast<uint4 *>(y)[v] = sum(xin);
    }
    // the last, incomplete vector: fewer than 16 bytes
    if (blockIdx.x == 0 && threadIdx.x < count - nvec * 16) {
        const size_t e = nvec * 16 + threadIdx.x;
        int t = 0;
#pragma unroll
        for (int i = 0; i < N_IN; ++i)
            t += ((int)a.x[i][e] * a.m[i] + a.add[i]) >> a.b[i];
        int v = FAST ? min(max((t >> a.s0) + a.ozp, 0), 255) : elt_finish(t, a);
        y[e] = (uint8_t)(FAST ? max(v, a.relu_lo) : v);
    }
}

// relu (relu.c:76-115): v = max(x, izp); y = sat_u(rshift_rn((v - izp) * m, s) + ozp), (m, s) from
// get_quant_scale(ialpha / oalpha, 24).  A 256-entry table built on the host with the exact
// 64-bit arithmetic turns the op into a byte lookup; the table sits in shared memory.
__global__ void __launch_bounds__(256) lut_u8_kernel(
    const uint8_t *__restrict__ x, uint8_t *__restrict__ y, size_t count, const uint8_t *__restrict__ lut_g)
{
    __shared__ uint8_t lut[256];
    lut[threadIdx.x] = lut_g[threadIdx.x];   // written once, at preparation
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    const size_t nvec = count / 16;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x; v < nvec; v += stride) {
        uint4 q = __ldg(reinterpret_cast<const uint4 *>(x) + v);
        uint32_t in[4] = { q.x, q.y, q.z, q.w }, o[4];
#pragma unroll
        for (int wd = 0; wd < 4; ++wd)
            o[wd] = pack4(
                lut[in[wd] & 0xff], lut[(in[wd] >> 8) & 0xff], lut[(in[wd] >> 16) & 0xff],
                lut[in[wd] >> 24]);
        reinterpret_cast<uint4 *>(y)[v] = make_uint4(o[0], o[1], o[2], o[3]);
    }
    if (blockIdx.x == 0)
        for (size_t e = nvec * 16 + threadIdx.x; e < count; e += blockDim.x)
            y[e] = lut[x[e]];
}

int relu_build_lut(
    float ialpha, uint8_t izp, float oalpha, uint8_t ozp, uint8_t obits, uint8_t lut[256])
{
    if (obits < 1 || obits > 8)
        return fail(B200_ERR_INVALID, "relu: obits outside 1..8");
    if (!(oalpha > 0.f) || !(ialpha > 0.f))
        return fail(B200_ERR_INVALID, "relu: scales must be positive");
    uint32_t m;
    int8_t s;
    get_quant_scale(ialpha / oalpha, 24, &m, &s);
    if (s < 1 || s > 62)
        return fail(B200_ERR_UNSUPPORTED, "relu: shift %d outside 1..62", (int)s);
    const int qmax = (1 << obits) - 1;
    for (int q = 0; q < 256; ++q) {
        int v = q >= izp ? q : izp;
        uint32_t prod = (uint32_t)(v - (int)izp) * m;   // relu.c:106, unsigned 32-bit product
        int32_t r = (int32_t)(rshift_rn_host((int64_t)prod, s) + ozp);
        lut[q] = (uint8_t)(r > qmax ? qmax : (r < 0 ? 0 : r));
    }
    return B200_OK;
}

int lut_u8_launch(const uint8_t *x, uint8_t *y, size_t count, const uint8_t *lut_dev, cudaStream_t st)
{
    if ((((uintptr_t)x | (uintptr_t)y) & 15) != 0)
        return fail(B200_ERR_INVALID, "relu: buffers must be 16-byte aligned");
    if (count == 0)
        return B200_OK;
    const int grid = resident_grid<lut_u8_kernel, 256>((count / 16 + 1 + 255) / 256);
    return launch_kernel(lut_u8_kernel, dim3(grid), dim3(256), 0, st, 2 * count, 1, x, y, count, lut_dev);
}

}  // namespace b200

namespace b200 {

// Host side of eltwise SUM: the per-input multipliers, addends and shifts of the kernel's
// arithmetic (see the comment above EltwiseArgs' kernel) from the reference's scale decomposition.
// *fast_out: obits == 8 and the final rounding term folded into the first input's addend.
int eltwise_prepare(
    int n_in, const float *ialpha, const uint8_t *izp, const float *coeff, float oalpha, uint8_t ozp,
    uint8_t obits, int relu, EltwiseArgs *out, bool *fast_out)
{
    if (n_in > kMaxEltIn)
        return fail(B200_ERR_UNSUPPORTED, "eltwise: at most %d inputs, got %d", kMaxEltIn, n_in);
    if (!(oalpha > 0.f))
        return fail(B200_ERR_INVALID, "eltwise: oalpha must be positive");
    EltwiseArgs &a = *out;
    uint32_t m[kMaxEltIn];
    int8_t s[kMaxEltIn];
    int s0 = 127;
    for (int i = 0; i < n_in; ++i) {
        float scale = (coeff ? coeff[i] : 1.0f) * ialpha[i] / oalpha;
        if (!(scale > 0.f))
            return fail(B200_ERR_INVALID, "eltwise: scale of input %d must be positive", i);
        get_quant_scale(scale, 23, &m[i], &s[i]);
        if (s[i] < s0)
            s0 = s[i];
    }
    s0 -= 1;  // eltwise.c:150
    if (s0 < 1 || s0 > 30)
        return fail(B200_ERR_UNSUPPORTED, "eltwise: final shift %d outside 1..30 (scale ratio too extreme)", s0);
    for (int i = 0; i < kMaxEltIn; ++i) {
        a.x[i] = nullptr; a.m[i] = 0; a.add[i] = 0; a.b[i] = 1;
    }
    for (int i = 0; i < n_in; ++i) {
        int b = (int)s[i] - s0;
        if (b < 1 || b > 30)
            return fail(B200_ERR_UNSUPPORTED, "eltwise: per-input shift %d outside 1..30", b);
        a.m[i] = (int)m[i];
        a.b[i] = b;
        const long long add = (1ll << (b - 1)) - (long long)izp[i] * (long long)m[i];
        // the kernels form x * m + add in int32 where the reference's rshift_rn works on int64
        // (quant_helper.h:55-58): decline what would not fit (shifts of 25 and more with a small zero point)
        const long long hi = 255ll * (long long)m[i] + add, lo = add;
        if (hi >= (1ll << 31) || lo < -(1ll << 31))
            return fail(B200_ERR_UNSUPPORTED, "eltwise: input %d needs more than 32 bits before its shift of %d (scale ratio too extreme)", i, b);
        a.add[i] = (int)add;
    }
    {
        long long worst = 1ll << (s0 - 1);
        for (int i = 0; i < n_in; ++i)
            worst += ((255ll * a.m[i]) >> a.b[i]) + 1;
        if (worst >= (1ll << 31))
            return fail(B200_ERR_UNSUPPORTED, "eltwise: the int32 sum could overflow");
    }
    a.n_in = n_in;
    a.rev = 0;
    a.s0 = s0;
    a.round0 = 1 << (s0 - 1);
    a.ozp = ozp;
    a.qmax = (1 << obits) - 1;
    a.relu_lo = relu ? ozp : 0;
    // fold the final rounding term into the first input's addend when that stays inside int32
    bool fast = a.qmax == 255;
    {
        long long folded = (long long)a.add[0] + ((long long)a.round0 << a.b[0]);
        long long worst = folded < 0 ? -folded : folded;
        worst += 255ll * a.m[0];
        if (fast && worst < (1ll << 31))
            a.add[0] = (int)folded;
        else
            fast = false;
    }
    *fast_out = fast;
    return B200_OK;
}

}  // namespace b200

namespace b200 {

// Images of up to four channels (the network input, C = 3) into 4-channel NHWC pixels: a thread
// reads four consecutive pixels of every plane (one word each) and writes four pixels (16 bytes).
// The pixel count of a plane must be a multiple of 4 and the planes word aligned.  Four such quads
// per thread and round, a grid stride apart, with all their loads issued before the first is used:
// one quad per round keeps 12 bytes per thread in flight, too few to cover the memory latency.
__global__ void __launch_bounds__(256) nchw_to_nhwc_c4_kernel(
    const uint8_t *__restrict__ x, uint4 *__restrict__ y, int c, uint32_t quads_per_image, uint32_t total, uint8_t fill)
{
    constexpr int UNR = 4;
    pdl_wait();
    pdl_trigger();
    const uint32_t fill4 = (uint32_t)fill * 0x01010101u;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t idx0 = blockIdx.x * blockDim.x + threadIdx.x; idx0 < total; idx0 += UNR * stride) {
        uint32_t p[UNR][4];
#pragma unroll
        for (int u = 0; u < UNR; ++u) {
            const uint32_t idx = idx0 + u * stride;
            const uint32_t img = idx / quads_per_image, q = idx - img * quads_per_image;
            const uint32_t *planes = reinterpret_cast<const uint32_t *>(x) + (size_t)img * c * quads_per_image + q;
#pragma unroll
            for (int ch = 0; ch < 4; ++ch)
                p[u][ch] = (ch < c && idx < total) ? __ldg(planes + (size_t)ch * quads_per_image) : fill4;
        }
#pragma unroll
        for (int u = 0; u < UNR; ++u) {
            const uint32_t idx = idx0 + u * stride;
            // 4x4 byte transpose: word j of the result holds byte j of every plane
            const uint32_t t0 = __byte_perm(p[u][0], p[u][1], 0x5140), t1 = __byte_perm(p[u][2], p[u][3], 0x5140);
            const uint32_t t2 = __byte_perm(p[u][0], p[u][1], 0x7362), t3 = __byte_perm(p[u][2], p[u][3], 0x7362);
            if (idx < total)
                y[idx] = make_uint4(__byte_perm(t0, t1, 0x5410), __byte_perm(t0, t1, 0x7632),
                                    __byte_perm(t2, t3, 0x5410), __byte_perm(t2, t3, 0x7632));
        }
    }
}

}  // namespace b200

using namespace b200;

extern "C" {

int b200_quantize_u8(
    const float *x, uint8_t *y, int32_t n, int32_t c, int32_t h, int32_t w, float oalpha,
    uint8_t ozp, uint8_t obits, int32_t nhwc, b200_stream_t stream)
{
    if (!x || !y || n < 0 || c <= 0 || h <= 0 || w <= 0 || obits < 1 || obits > 8)
        return fail(B200_ERR_INVALID, "quantize: bad argument");
    if (!(oalpha > 0.f))
        return fail(B200_ERR_INVALID, "quantize: oalpha must be positive");
    if (n == 0)
        return B200_OK;
    QuantizeFn fn;
    fn.alpha = oalpha;
    fn.beta = -(oalpha * (float)ozp);
    fn.qmax = (1 << obits) - 1;
    fn.inv = 1.f / oalpha;
    fn.half_zp = (float)ozp + 0.5f;
    fn.fast = oalpha > 1e-30f && oalpha < 1e30f;
    const int P = h * w;
    if (nhwc && !(c == 1 || P == 1)) {
        return nchw_to_nhwc_launch(x, y, n, c, P, c, 0, fn, as_stream(stream));
    } else {
        return quantize_flat_launch(x, y, (size_t)n * c * P, fn, as_stream(stream));
    }
}

int b200_dequantize_u8(
    const uint8_t *x, float *y, int32_t n, int32_t c, int32_t h, int32_t w, float ialpha,
    uint8_t izp, int32_t nhwc, b200_stream_t stream)
{
    if (!x || !y || n < 0 || c <= 0 || h <= 0 || w <= 0)
        return fail(B200_ERR_INVALID, "dequantize: bad argument");
    if (n == 0)
        return B200_OK;
    DequantizeFn fn;
    fn.alpha = ialpha;
    fn.zp = izp;
    const int P = h * w;
    if (nhwc && !(c == 1 || P == 1)) {
        return nhwc_to_nchw_launch(x, y, n, c, P, c, fn, as_stream(stream));
    } else {
        return dequantize_flat_launch(x, y, (size_t)n * c * P, fn, as_stream(stream));
    }
}

}  // extern "C"

// b200_dequantize_u8 of one pixel an image, which also moves the current device's status word to *host
int b200::dequantize_and_publish(const uint8_t *x, float *y, size_t count, float ialpha, uint8_t izp, int *host, cudaStream_t st)
{
    int *word = nullptr;
    B200_TRY(status_word_ptr(&word));
    DequantizeFn fn;
    fn.alpha = ialpha;
    fn.zp = izp;
    return dequantize_flat_launch(x, y, count, fn, st, word, host);
}

extern "C" {

int b200_quantize_s8(
    const float *x, int8_t *y8, int32_t n, int32_t c, int32_t h, int32_t w, float oalpha, uint8_t obits,
    int32_t nhwc, b200_stream_t stream)
{
    if (!x || !y8 || n < 0 || c <= 0 || h <= 0 || w <= 0 || obits < 2 || obits > 8)
        return fail(B200_ERR_INVALID, "quantize(int8): bad argument (obits 2..8)");
    if (!(oalpha > 0.f))
        return fail(B200_ERR_INVALID, "quantize(int8): oalpha must be positive");
    if (n == 0)
        return B200_OK;
    uint8_t *y = reinterpret_cast<uint8_t *>(y8);
    QuantizeS8Fn fn;
    fn.alpha = (float)(1. / (double)oalpha);
    fn.l = (1 << (obits - 1)) - 1;
    const int P = h * w;
    if (nhwc && !(c == 1 || P == 1)) {
        return nchw_to_nhwc_launch(x, y, n, c, P, c, 0, fn, as_stream(stream));
    } else {
        return quantize_flat_launch(x, y, (size_t)n * c * P, fn, as_stream(stream));
    }
}

int b200_dequantize_s8(
    const int8_t *x8, float *y, int32_t n, int32_t c, int32_t h, int32_t w, float ialpha, int32_t nhwc,
    b200_stream_t stream)
{
    if (!x8 || !y || n < 0 || c <= 0 || h <= 0 || w <= 0)
        return fail(B200_ERR_INVALID, "dequantize(int8): bad argument");
    if (n == 0)
        return B200_OK;
    const uint8_t *x = reinterpret_cast<const uint8_t *>(x8);
    DequantizeS8Fn fn;
    fn.alpha = ialpha;
    const int P = h * w;
    if (nhwc && !(c == 1 || P == 1)) {
        return nhwc_to_nchw_launch(x, y, n, c, P, c, fn, as_stream(stream));
    } else {
        return dequantize_flat_launch(x, y, (size_t)n * c * P, fn, as_stream(stream));
    }
}

int b200_nchw_to_nhwc_u8(
    const uint8_t *x, uint8_t *y, int32_t n, int32_t c, int32_t h, int32_t w, int32_t c_pad,
    uint8_t fill, b200_stream_t stream)
{
    if (!x || !y || n < 0 || c <= 0 || h <= 0 || w <= 0 || c_pad < c)
        return fail(B200_ERR_INVALID, "nchw_to_nhwc: bad argument");
    if (n == 0)
        return B200_OK;
    const int P = h * w;
    if (c_pad == 4 && P % 4 == 0 && (((uintptr_t)x) & 3) == 0 && (((uintptr_t)y) & 15) == 0
        && (size_t)n * (P / 4) < 0xf0000000ull) {   // 32-bit indices, with room for the unrolled rounds past the end
        const uint32_t quads = (uint32_t)(P / 4), total = (uint32_t)n * quads;
        const int blocks = resident_grid<nchw_to_nhwc_c4_kernel, 256>(((size_t)total + 1023) / 1024);   // four quads per thread and round
        B200_TRY((launch_kernel(nchw_to_nhwc_c4_kernel, dim3(blocks), dim3(256), 0, as_stream(stream), (size_t)total * 28, 1, x, reinterpret_cast<uint4 *>(y), c, quads, total, fill)));
            return B200_OK;
    }
    return nchw_to_nhwc_launch(x, y, n, c, P, c_pad, fill, IdentityFn(), as_stream(stream));
}

int b200_nhwc_to_nchw_u8(
    const uint8_t *x, uint8_t *y, int32_t n, int32_t c, int32_t h, int32_t w, int32_t c_pad,
    b200_stream_t stream)
{
    if (!x || !y || n < 0 || c <= 0 || h <= 0 || w <= 0 || c_pad < c)
        return fail(B200_ERR_INVALID, "nhwc_to_nchw: bad argument");
    if (n == 0)
        return B200_OK;
    const int P = h * w;
    return nhwc_to_nchw_launch(x, y, n, c, P, c_pad, IdentityFn(), as_stream(stream));
}

int b200_eltwise_sum_u8(
    const uint8_t *const *xs, int32_t n_in, size_t count, const float *ialpha, const uint8_t *izp,
    const float *coeff, float oalpha, uint8_t ozp, uint8_t obits, int32_t relu, uint8_t *y,
    b200_stream_t stream)
{
    if (!xs || !ialpha || !izp || !y || n_in < 1 || obits < 1 || obits > 8)
        return fail(B200_ERR_INVALID, "eltwise: bad argument");
    EltwiseArgs a;
    bool fast = false;
    B200_TRY(eltwise_prepare(n_in, ialpha, izp, coeff, oalpha, ozp, obits, relu, &a, &fast));
    return eltwise_launch(a, fast, xs, y, count, 0, as_stream(stream));
}

}  // extern "C"

namespace b200 {

int eltwise_launch(const EltwiseArgs &prepared, bool fast, const uint8_t *const *xs, uint8_t *y, size_t count, int reverse,
                   cudaStream_t st)
{
    EltwiseArgs a = prepared;
    const int n_in = a.n_in;
    a.rev = reverse ? 1 : 0;
    for (int i = 0; i < n_in; ++i) {
        if (((uintptr_t)xs[i] & 15) != 0)
            return fail(B200_ERR_INVALID, "eltwise: input %d is not 16-byte aligned", i);
        a.x[i] = xs[i];
    }
    if (((uintptr_t)y & 15) != 0)
        return fail(B200_ERR_INVALID, "eltwise: output is not 16-byte aligned");
    if (count == 0)
        return B200_OK;
    const bool few = count < (size_t)sm_count() * (256 * 64);
    const size_t tile = few ? 256 * 16 : 256 * 64;    // bytes per block and round
    const size_t want = (count + tile - 1) / tile;
#define B200_ELT_LAUNCH(...) \
    return launch_kernel(eltwise_sum_kernel<__VA_ARGS__>, dim3(resident_grid<eltwise_sum_kernel<__VA_ARGS__>, 256>(want)), dim3(256), 0, st, (n_in + 1) * count, 1, a, y, count)
    if (fast && n_in == 2 && few)
        B200_ELT_LAUNCH(2, true, false, false, 1);
    if (fast) {
        switch (n_in) {
        case 1: B200_ELT_LAUNCH(1, true);
        case 2:
            if (a.ozp == 0 && a.relu_lo <= 0)
                B200_ELT_LAUNCH(2, true, true);
            if (a.rev)
                B200_ELT_LAUNCH(2, true, false, true);
            B200_ELT_LAUNCH(2, true);
        case 3: B200_ELT_LAUNCH(3, true);
        default: B200_ELT_LAUNCH(4, true);
        }
    }
    switch (n_in) {
    case 1: B200_ELT_LAUNCH(1, false);
    case 2: B200_ELT_LAUNCH(2, false);
    case 3: B200_ELT_LAUNCH(3, false);
    default: B200_ELT_LAUNCH(4, false);
    }
#undef B200_ELT_LAUNCH
}

}  // namespace b200

using namespace b200;

extern "C" {

int b200_relu_u8(
    const uint8_t *x, size_t count, float ialpha, uint8_t izp, float oalpha, uint8_t ozp,
    uint8_t obits, uint8_t *y, b200_stream_t stream)
{
    if (!x || !y)
        return fail(B200_ERR_INVALID, "relu: bad argument");
    uint8_t lut[256];
    B200_TRY(relu_build_lut(ialpha, izp, oalpha, ozp, obits, lut));
    if (count == 0)
        return B200_OK;
    const uint8_t *lut_dev = nullptr;
    B200_TRY(lut_cache_get(lut, &lut_dev));   // uploaded once per distinct table, then reused
    return lut_u8_launch(x, y, count, lut_dev, as_stream(stream));
}

}  // extern "C"
