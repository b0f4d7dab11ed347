// CUDA-core convolution kernels (dp4a) for the shapes that are not dense contractions: grouped and
// depthwise convs, tiny channel counts (the 3-channel stem), and any shape the tensor-core path
// declines.  Arithmetic follows op_conv_2d_u8xu8_run of the reference CPU module
// (art/modules/quant/src/op/conv_2d_uint8_impl.c:39-165 of ModelTC/NART):
//   acc = bias[k] + sum (x - izp) * (w - wzp),  taps outside the image contribute 0,
//   y   = sat_u(rshift_rn(acc * mult_k, shift_k) + ozp, obits).
// The kernels multiply the raw uint8 activation by the signed weight (dp4a.u32.s32) and read an
// out-of-image tap as the byte `izp`; with bias_fold[k] = bias[k] - izp * sum(w[k]) this gives the
// same int32 accumulator.
#include "common.cuh"
#include "kernels.h"

namespace b200 {

__device__ __forceinline__ int dp4a_us(uint32_t a, uint32_t b, int c)
{
    int d;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

// ---------------------------------------------------------------------------------------------
// Generic tiled kernel.  Block = 256 threads = 32 output pixels x 8 quads of output channels
// (32 channels of one group).  The reduction runs over "items" = 4-channel words of
// [r][s][cg4]; the weights of the block's 32 channels are staged through shared memory in
// chunks of 64 items as [item][channel] so that a quad reads one 16-byte vector per item.
// ---------------------------------------------------------------------------------------------
constexpr int DK = 32;       // output channels per block
constexpr int DP = 32;       // output pixels per block
constexpr int DCHUNK = 64;   // items per shared-memory stage

template <bool WORD_LOADS>
__global__ void __launch_bounds__(256) conv_direct_kernel(
    ConvGeom g, int cg4, const uint8_t *__restrict__ x, const uint32_t *__restrict__ wq,
    const int32_t *__restrict__ bias_fold, const uint32_t *__restrict__ mult,
    const int32_t *__restrict__ shift, uint8_t *__restrict__ y, int32_t *__restrict__ acc_out, int n)
{
    __shared__ __align__(16) uint32_t wsm[DCHUNK][DK];
    const int tid = threadIdx.x;
    const int kq = tid & 7;
    const int pl = tid >> 3;
    const int kg = g.k / g.group, cg = g.c / g.group;
    const int ktiles = (kg + DK - 1) / DK;
    const int grp = blockIdx.y / ktiles;
    const int kt = blockIdx.y % ktiles;
    const int k_in_g0 = kt * DK;               // first channel of the tile inside the group
    const int kvalid = min(DK, kg - k_in_g0);  // channels of this tile that exist
    const int k0 = grp * kg + k_in_g0;
    const size_t npix = (size_t)n * g.oh * g.ow;
    const size_t pix = (size_t)blockIdx.x * DP + pl;
    const bool pvalid = pix < npix;
    int ox = 0, oy = 0, img = 0;
    if (pvalid) {
        ox = (int)(pix % g.ow);
        oy = (int)((pix / g.ow) % g.oh);
        img = (int)(pix / ((size_t)g.ow * g.oh));
    }
    const int iy0 = oy * g.stride_h - g.pad_h, ix0 = ox * g.stride_w - g.pad_w;
    const int cwords = cg4 / 4;
    const int items = g.r * g.s * cwords;
    const uint32_t izp4 = (uint32_t)g.izp * 0x01010101u;
    const uint32_t x_flip = g.act_signed ? 0x80808080u : 0u;   // int8 bytes seen as uint8 with zero point 128
    const uint8_t *ximg = x + (size_t)img * g.h * g.w * g.c + (size_t)grp * cg;

    pdl_wait();
    pdl_trigger();
    int acc[4] = { 0, 0, 0, 0 };
    // wzp != 128: sum of the bytes the products see (out-of-image taps read izp, like the products),
    // with the bytes past the group's last channel masked out of the last word
    int xsum = 0;
    const uint32_t last_ones = 0x01010101u >> (8 * (cg4 - cg));
    for (int item0 = 0; item0 < items; item0 += DCHUNK) {
        const int nitem = min(DCHUNK, items - item0);
        __syncthreads();
        for (int i = tid; i < DCHUNK * DK; i += 256) {
            int it = i / DK, kl = i % DK;
            uint32_t v = 0;
            if (it < nitem && kl < kvalid)
                v = __ldg(wq + (size_t)(k0 + kl) * items + item0 + it);
            wsm[it][kl] = v;
        }
        __syncthreads();
        if (pvalid) {
            int tap = item0 / cwords, cw = item0 % cwords;
            for (int it = 0; it < nitem; ++it) {
                int rr = tap / g.s, ss = tap % g.s;
                int iy = iy0 + rr, ix = ix0 + ss;
                uint32_t xv = izp4;
                if (iy >= 0 && iy < g.h && ix >= 0 && ix < g.w) {
                    const uint8_t *px = ximg + ((size_t)iy * g.w + ix) * g.c + cw * 4;
                    if (WORD_LOADS) {
                        xv = __ldg(reinterpret_cast<const uint32_t *>(px));
                    } else {
                        xv = 0;
#pragma unroll
                        for (int b = 0; b < 4; ++b)
                            if (cw * 4 + b < cg)
                                xv |= (uint32_t)__ldg(px + b) << (8 * b);
                    }
                    xv ^= x_flip;   // (bytes past the group's last channel meet zero weights)
                }
                uint4 wv = *reinterpret_cast<const uint4 *>(&wsm[it][kq * 4]);
                acc[0] = dp4a_us(xv, wv.x, acc[0]);
                acc[1] = dp4a_us(xv, wv.y, acc[1]);
                acc[2] = dp4a_us(xv, wv.z, acc[2]);
                acc[3] = dp4a_us(xv, wv.w, acc[3]);
                if (g.wzp_d != 0)
                    xsum = (int)__dp4a(xv, cw == cwords - 1 ? last_ones : 0x01010101u, (unsigned)xsum);
                if (++cw == cwords) {
                    cw = 0;
                    ++tap;
                }
            }
        }
    }
    if (!pvalid)
        return;
    int q[4] = { 0, 0, 0, 0 };
    int nk = min(4, kvalid - kq * 4);
    for (int j = 0; j < 4; ++j) {
        if (j >= nk)
            break;
        int k = k0 + kq * 4 + j;
        int a = acc[j] + bias_fold[k];
        if (g.wzp_d != 0)   // sum (x - izp) over all taps (the out-of-image ones give 0) times -(wzp - 128)
            a -= g.wzp_d * (xsum - g.izp * g.r * g.s * cg);
        if (acc_out)
            acc_out[pix * g.k + k] = a;
        if (g.s8_wrap) {
            // ssaturate_int_by_bits(v, 8): clip at +-255, then the int8 return type keeps the low byte
            const int v = requant_raw(a, mult[k], shift[k], 0);
            q[j] = max(min(v, 255), g.relu_lo) & 0xff;
        } else {
            q[j] = sat_relu(requant_raw(a, mult[k], shift[k], g.ozp), g.qmax, g.relu_lo) ^ (g.act_signed ? 0x80 : 0);
        }
    }
    uint8_t *py = y + pix * g.k + k0 + kq * 4;
    if (nk == 4 && (((uintptr_t)y | (size_t)g.k | (size_t)k0) & 3) == 0) {
        *reinterpret_cast<uint32_t *>(py) = pack4(q[0], q[1], q[2], q[3]);
    } else {
        for (int j = 0; j < nk; ++j)
            py[j] = (uint8_t)q[j];
    }
}

// ---------------------------------------------------------------------------------------------
// Depthwise kernel (group == c == k, c % 16 == 0).  A thread owns 16 consecutive channels of one
// output pixel: one 16-byte activation vector and one 16-byte weight vector per tap, products
// formed per channel.  Weights are [r][s][c] int8.  HBM-bound: each activation byte is read once
// from DRAM (neighbouring taps hit L1/L2), each output byte written once.
// ---------------------------------------------------------------------------------------------
template <bool WZP>
__global__ void __launch_bounds__(256) conv_depthwise_kernel(
    ConvGeom g, const uint8_t *__restrict__ x, const int8_t *__restrict__ w_rsc,
    const int32_t *__restrict__ bias_fold, const uint32_t *__restrict__ mult,
    const int32_t *__restrict__ shift, uint8_t *__restrict__ y, int n)
{
    pdl_wait();
    pdl_trigger();
    const int cv = g.c / 16;
    const size_t total = (size_t)n * g.oh * g.ow * cv;
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (size_t)gridDim.x * blockDim.x) {
        const int ci = (int)(idx % cv);
        const size_t pix = idx / cv;
        const int ox = (int)(pix % g.ow);
        const int oy = (int)((pix / g.ow) % g.oh);
        const int img = (int)(pix / ((size_t)g.ow * g.oh));
        const int iy0 = oy * g.stride_h - g.pad_h, ix0 = ox * g.stride_w - g.pad_w;
        int acc[16];
        {
            const int4 *b4 = reinterpret_cast<const int4 *>(bias_fold + ci * 16);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                int4 b = __ldg(b4 + j);
                acc[4 * j] = b.x; acc[4 * j + 1] = b.y; acc[4 * j + 2] = b.z; acc[4 * j + 3] = b.w;
            }
        }
        // WZP: every channel is its own group, so the correction -(wzp - 128) * sum (x - izp) is per
        // channel: fold it into the weight, w - wzp = s8 - wzp_d, with izp at the out-of-image taps
        // (x - izp = 0 there) and the constant izp * taps * wzp_d added back
        if (WZP) {
#pragma unroll
            for (int j = 0; j < 16; ++j)
                acc[j] += g.izp * g.r * g.s * g.wzp_d;
        }
        for (int rr = 0; rr < g.r; ++rr) {
            const int iy = iy0 + rr;
            for (int ss = 0; ss < g.s; ++ss) {
                const int ix = ix0 + ss;
                uint4 wv = __ldg(reinterpret_cast<const uint4 *>(w_rsc + ((size_t)(rr * g.s + ss) * g.c) + ci * 16));
                uint4 xv;
                if (iy >= 0 && iy < g.h && ix >= 0 && ix < g.w) {
                    xv = __ldg(reinterpret_cast<const uint4 *>(
                        x + (((size_t)img * g.h + iy) * g.w + ix) * g.c + ci * 16));
                } else {
                    uint32_t z = (uint32_t)g.izp * 0x01010101u;
                    xv = make_uint4(z, z, z, z);
                }
                const uint32_t xw[4] = { xv.x, xv.y, xv.z, xv.w };
                const uint32_t ww[4] = { wv.x, wv.y, wv.z, wv.w };
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    int xb = (int)((xw[j / 4] >> (8 * (j % 4))) & 0xff);
                    int wb = (int)(int8_t)((ww[j / 4] >> (8 * (j % 4))) & 0xff);
                    if (WZP)
                        wb -= g.wzp_d;   // 9 bits: fine in the 32-bit multiply
                    acc[j] += xb * wb;
                }
            }
        }
        uint32_t o[4];
#pragma unroll
        for (int wd = 0; wd < 4; ++wd) {
            int q[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                int k = ci * 16 + wd * 4 + e;
                q[e] = sat_relu(requant_raw(acc[wd * 4 + e], __ldg(mult + k), __ldg(shift + k), g.ozp), g.qmax, g.relu_lo);
            }
            o[wd] = pack4(q[0], q[1], q[2], q[3]);
        }
        *reinterpret_cast<uint4 *>(y + pix * g.k + ci * 16) = make_uint4(o[0], o[1], o[2], o[3]);
    }
}

// ---------------------------------------------------------------------------------------------
// Depthwise 3x3 on dp4a.  A thread owns four consecutive channels of one output pixel.  The nine
// tap words (four channels each) are transposed four at a time with byte permutes into words that
// hold four taps of ONE channel, which dp4a multiplies with the matching weight word
// [c/4][tap group][channel]: 8 permutes + 4 dp4a per 16 multiply-adds instead of 16 extractions
// and 16 multiply-adds.  The requantize is the folded form of the tensor-core epilogue:
// y = sat_u8(max((acc * mult + off64) >> shift, floor)), the host having checked shift >= 33.
// Neighbouring threads read neighbouring words of a pixel and write neighbouring output words.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void transpose4x4(uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t (&ch)[4])
{
    const uint32_t t0 = __byte_perm(a, b, 0x5140), t1 = __byte_perm(c, d, 0x5140);   // a0 b0 a1 b1 | c0 d0 c1 d1
    const uint32_t t2 = __byte_perm(a, b, 0x7362), t3 = __byte_perm(c, d, 0x7362);   // a2 b2 a3 b3 | c2 d2 c3 d3
    ch[0] = __byte_perm(t0, t1, 0x5410);
    ch[1] = __byte_perm(t0, t1, 0x7632);
    ch[2] = __byte_perm(t2, t3, 0x5410);
    ch[3] = __byte_perm(t2, t3, 0x7632);
}

__global__ void __launch_bounds__(256) conv_depthwise3x3_kernel(
    ConvGeom g, const uint32_t *__restrict__ x, const uint4 *__restrict__ w3, const int4 *__restrict__ q3,
    uint32_t *__restrict__ y, int n)
{
    pdl_wait();
    pdl_trigger();
    const uint32_t cq = (uint32_t)g.c / 4;
    const uint32_t total = (uint32_t)n * g.oh * g.ow * cq;      // the launcher checks that it fits 32 bits
    const uint32_t izp4 = (uint32_t)g.izp * 0x01010101u;
    for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
        const uint32_t ci = idx % cq;
        const uint32_t pix = idx / cq;
        const int ox = (int)(pix % (uint32_t)g.ow);
        const uint32_t rowi = pix / (uint32_t)g.ow;
        const int oy = (int)(rowi % (uint32_t)g.oh);
        const uint32_t img = rowi / (uint32_t)g.oh;
        const int iy0 = oy * g.stride_h - g.pad_h, ix0 = ox * g.stride_w - g.pad_w;
        // word offsets fit 32 bits (checked by the launcher)
        const uint32_t row_pitch = (uint32_t)g.w * cq;
        const uint32_t *xc = x + (img * (uint32_t)g.h * row_pitch + ci);
        uint32_t t[9];
        if (iy0 >= 0 && iy0 + 2 < g.h && ix0 >= 0 && ix0 + 2 < g.w) {
            const uint32_t *p0 = xc + ((uint32_t)iy0 * row_pitch + (uint32_t)ix0 * cq);
#pragma unroll
            for (int rr = 0; rr < 3; ++rr)
#pragma unroll
                for (int ss = 0; ss < 3; ++ss)
                    t[rr * 3 + ss] = __ldg(p0 + (rr * row_pitch + ss * cq));
        } else {
#pragma unroll
            for (int rr = 0; rr < 3; ++rr)
#pragma unroll
                for (int ss = 0; ss < 3; ++ss) {
                    const int iy = iy0 + rr, ix = ix0 + ss;
                    t[rr * 3 + ss] = (iy >= 0 && iy < g.h && ix >= 0 && ix < g.w)
                        ? __ldg(xc + ((uint32_t)iy * row_pitch + (uint32_t)ix * cq)) : izp4;
                }
        }
        const uint4 wa = __ldg(w3 + (size_t)ci * 3), wb = __ldg(w3 + (size_t)ci * 3 + 1), wc = __ldg(w3 + (size_t)ci * 3 + 2);
        uint32_t ch[4];
        int acc[4];
        transpose4x4(t[0], t[1], t[2], t[3], ch);
        acc[0] = dp4a_us(ch[0], wa.x, 0); acc[1] = dp4a_us(ch[1], wa.y, 0);
        acc[2] = dp4a_us(ch[2], wa.z, 0); acc[3] = dp4a_us(ch[3], wa.w, 0);
        transpose4x4(t[4], t[5], t[6], t[7], ch);
        acc[0] = dp4a_us(ch[0], wb.x, acc[0]); acc[1] = dp4a_us(ch[1], wb.y, acc[1]);
        acc[2] = dp4a_us(ch[2], wb.z, acc[2]); acc[3] = dp4a_us(ch[3], wb.w, acc[3]);
        // the ninth tap: byte j of the word against byte 0 of the weight word
        acc[0] = dp4a_us(t[8] & 0xffu, wc.x, acc[0]); acc[1] = dp4a_us((t[8] >> 8) & 0xffu, wc.y, acc[1]);
        acc[2] = dp4a_us((t[8] >> 16) & 0xffu, wc.z, acc[2]); acc[3] = dp4a_us(t[8] >> 24, wc.w, acc[3]);
        int q[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int4 c4 = __ldg(q3 + (size_t)ci * 4 + j);
            const long long off = (long long)(((unsigned long long)(uint32_t)c4.y << 32) | (uint32_t)c4.x);
            const long long prod = (long long)acc[j] * c4.z + off;
            q[j] = max((int)(prod >> 32) >> c4.w, g.relu_lo);
        }
        y[idx] = pack_sat_u8x4(q[0], q[1], q[2], q[3]);
    }
}

// ---------------------------------------------------------------------------------------------
// Depthwise 3x3 with horizontal stride S (1 or 2): a thread computes two output pixels side by
// side, in ROWS output rows (one unless the vertical stride is S too), for four channels.  The two windows of a row cover 3 + S neighbouring input
// pixels per kernel row.  One transpose of the first four of those words gives, per channel, a
// word (x0, x1, x2, x3) that serves both pixels: dp4a against (w0, w1, w2, 0) is the left pixel's
// kernel row; the right pixel's is (0, w0, w1, w2) for S == 1, and for S == 2 (0, 0, w0, w1) plus
// the fifth word against w2 placed at the channel's own byte (no extraction).  Neighbouring output rows
// share 3 - S of their input rows.
//
// Its instructions bound it, most of them on the integer pipe (63 % of issue slots at 22 % of the warps): with 2 x 2 outputs per thread, 64-bit
// divisions and a wide integer requantize it took 24 instructions per output byte (144 channels of 56 x 56,
// batch 64: 35.7 us, 1.6 TB/s).  So weights and constants are read once for ROWS rows, indices are divided by
// multiplication, and the requantize is fp32, exactly, two values per instruction: the accumulator starts at
// bits(1.5 * 2^23) + bias, which makes its bits the float 1.5 * 2^23 + acc (|acc| < 2^22, checked when the table
// is built); mult * 2^-shift is a float m (24 significant bits); acc * m + (zero point less floor + 1/2) is formed by one
// multiply-add rounded toward zero, which never crosses an integer, and 2^23 is added, again toward zero: the low
// bits are then floor(acc * m + 1/2) + zero point less floor for every result of 0 or more, and for every negative one the
// low 16 bits are a negative 16-bit number (below 2^23 a float's last bit is a half: results stay within -2^14 .. 2^15,
// checked as well).  Both bounds run on pairs of those, and the floor goes back onto the packed bytes.
// (A thread that walks whole columns, every input row loaded and transposed once, is no faster: its accumulators in
// flight and weights leave 16 to 20 warps per SM, and its row loop's bookkeeping costs what the shared rows save.)
// Weight table: [c/4][3 kernel rows][2 + (S == 2)][4 channels] words.  Requantize table: [c/4] 4 start values, 4 floats.
// FP false, for scales whose results leave those bounds: the integers of conv_depthwise3x3_kernel, four constants a channel.
// (144 channels of 56 x 56, batch 64: 37.1 us with 2 rows, 75.4 pixel by pixel.)
// ---------------------------------------------------------------------------------------------
struct DwArgs {
    int c4, h, w, oh, ow, pad_h, pad_w;
    int stride_h, relu_lo;
    FastDiv by_c4, by_pairs, by_strips;         // channel words, pixel pairs of a row, strips of ROWS rows
    uint32_t total, izp4;
    float add;                                  // zero point less floor + 1/2
    uint32_t top2, lo4;                         // ceiling less floor, twice; floor, four times
};

// The low halves of two of fp_requant_pair's results in one word
__device__ __forceinline__ uint32_t requant_pair(int a0, int a1, int m0, int m1, float add)
{
    int q0, q1;
    fp_requant_pair(a0, a1, m0, m1, add, q0, q1);
    return __byte_perm(q0, q1, 0x5410);
}
// Both halves to 0 .. those of `top`: with the floor subtracted before and added to the packed bytes, one instruction for the two
// bounds.  (With that and the rows in one test, 11.0 million warp instructions for 12.2: 144 channels of 56 x 56, batch 64:
// 18.4 -> 18.2 us, batch 256: 60.0 -> 58.3; 960 of 7 x 7: 10.0 -> 9.6.)
__device__ __forceinline__ uint32_t clamp_s16x2(uint32_t v, uint32_t top)
{
    uint32_t d;
    asm("min.relu.s16x2 %0, %1, %2;" : "=r"(d) : "r"(v), "r"(top));
    return d;
}

template <int ROWS, int S, bool FP>
__global__ void __launch_bounds__(128) conv_depthwise3x3_strip_kernel(
    const __grid_constant__ DwArgs g, const uint32_t *__restrict__ x, const uint4 *__restrict__ w3p, const uint4 *__restrict__ qf,
    const int4 *__restrict__ q3, uint32_t *__restrict__ y)
{
    constexpr int IN_ROWS = 3 + (ROWS - 1) * S, IN_COLS = 3 + S, NV = S == 2 ? 3 : 2;
    const uint32_t idx = blockIdx.x * 128 + threadIdx.x;
    if (idx >= g.total) {
        pdl_wait();
        return;
    }
    const uint32_t pp = g.by_c4.div(idx), ci = idx - pp * g.c4;
    const uint32_t rowi = g.by_pairs.div(pp), oxp = pp - rowi * g.by_pairs.d;
    const uint32_t img = g.by_strips.div(rowi), strip = rowi - img * g.by_strips.d;
    const int ox = (int)oxp * 2, oy = (int)strip * ROWS;
    uint4 wv[3][NV];
#pragma unroll
    for (int rr = 0; rr < 3; ++rr)
#pragma unroll
        for (int v = 0; v < NV; ++v)
            wv[rr][v] = __ldg(w3p + ((size_t)ci * 3 + rr) * NV + v);
    uint4 start = make_uint4(0, 0, 0, 0), mb = start;
    int4 q[4];
    if (FP) {
        start = __ldg(qf + ci * 2);
        mb = __ldg(qf + ci * 2 + 1);
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            q[j] = __ldg(q3 + ci * 4 + j);
    }
    pdl_wait();
    pdl_trigger();
    const int iy0 = oy * (ROWS == 1 ? g.stride_h : S) - g.pad_h, ix0 = ox * S - g.pad_w;
    // byte offsets of 32 bits from the tensor's start (the launcher checks that it ends below 4 GB)
    auto at = [&](uint32_t off) { return __ldg(reinterpret_cast<const uint32_t *>(reinterpret_cast<const char *>(x) + off)); };
    const uint32_t col_pitch = (uint32_t)g.c4 * 4, row_pitch = (uint32_t)g.w * col_pitch;
    const uint32_t x0 = (img * (uint32_t)g.h + (uint32_t)iy0) * row_pitch + (uint32_t)ix0 * col_pitch + ci * 4;   // modulo 2^32
    uint32_t t[IN_ROWS][IN_COLS];
    if (ix0 >= 0 && ix0 + IN_COLS - 1 < g.w && iy0 >= -1 && iy0 + IN_ROWS - 2 < g.h) {
        // the strip's first and last rows may lie outside the image, nothing else
        const bool top = iy0 >= 0, bottom = iy0 + IN_ROWS - 1 < g.h;
#pragma unroll
        for (int rr = 0; rr < IN_ROWS; ++rr)
#pragma unroll
            for (int ss = 0; ss < IN_COLS; ++ss)
                t[rr][ss] = (rr > 0 || top) && (rr < IN_ROWS - 1 || bottom) ? at(x0 + rr * row_pitch + ss * col_pitch) : g.izp4;
    } else {
#pragma unroll
        for (int rr = 0; rr < IN_ROWS; ++rr)
#pragma unroll
            for (int ss = 0; ss < IN_COLS; ++ss) {
                const int iy = iy0 + rr, ix = ix0 + ss;
                t[rr][ss] = (iy >= 0 && iy < g.h && ix >= 0 && ix < g.w) ? at(x0 + rr * row_pitch + ss * col_pitch) : g.izp4;
            }
    }
    int acc[ROWS][2][4];
#pragma unroll
    for (int o = 0; o < ROWS; ++o)
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            acc[o][p][0] = (int)start.x; acc[o][p][1] = (int)start.y; acc[o][p][2] = (int)start.z; acc[o][p][3] = (int)start.w;
        }
    const int m0 = (int)mb.x, m1 = (int)mb.y, m2 = (int)mb.z, m3 = (int)mb.w;       // bits of floats
    const uint32_t out_row = (uint32_t)g.ow * col_pitch;
    const uint32_t out = ((img * (uint32_t)g.oh + (uint32_t)oy) * (uint32_t)g.ow + (uint32_t)ox) * col_pitch + ci * 4;
    const bool second = ox + 1 < g.ow;
#pragma unroll
    for (int ir = 0; ir < IN_ROWS; ++ir) {
        uint32_t ch[4];
        transpose4x4(t[ir][0], t[ir][1], t[ir][2], t[ir][3], ch);
#pragma unroll
        for (int o = 0; o < ROWS; ++o) {
            const int kr = ir - o * S;     // kernel row this input row meets in output row o
            if (kr < 0 || kr > 2)
                continue;
            const uint4 w0 = wv[kr][0], w1 = wv[kr][1];
            acc[o][0][0] = dp4a_us(ch[0], w0.x, acc[o][0][0]); acc[o][0][1] = dp4a_us(ch[1], w0.y, acc[o][0][1]);
            acc[o][0][2] = dp4a_us(ch[2], w0.z, acc[o][0][2]); acc[o][0][3] = dp4a_us(ch[3], w0.w, acc[o][0][3]);
            acc[o][1][0] = dp4a_us(ch[0], w1.x, acc[o][1][0]); acc[o][1][1] = dp4a_us(ch[1], w1.y, acc[o][1][1]);
            acc[o][1][2] = dp4a_us(ch[2], w1.z, acc[o][1][2]); acc[o][1][3] = dp4a_us(ch[3], w1.w, acc[o][1][3]);
            if (S == 2) {
                const uint4 w2 = wv[kr][NV - 1];
                const uint32_t x4 = t[ir][IN_COLS - 1];
                acc[o][1][0] = dp4a_us(x4, w2.x, acc[o][1][0]); acc[o][1][1] = dp4a_us(x4, w2.y, acc[o][1][1]);
                acc[o][1][2] = dp4a_us(x4, w2.z, acc[o][1][2]); acc[o][1][3] = dp4a_us(x4, w2.w, acc[o][1][3]);
            }
            if (kr == 2 && (o == 0 || oy + o < g.oh)) {
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    uint32_t out4;
                    if (FP) {
                        const uint32_t lo = clamp_s16x2(requant_pair(acc[o][p][0], acc[o][p][1], m0, m1, g.add), g.top2);
                        const uint32_t hi = clamp_s16x2(requant_pair(acc[o][p][2], acc[o][p][3], m2, m3, g.add), g.top2);
                        out4 = __byte_perm(lo, hi, 0x6420) + g.lo4;
                    } else {
                        int r[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const long long off = (long long)(((unsigned long long)(uint32_t)q[j].y << 32) | (uint32_t)q[j].x);
                            r[j] = max((int)(((long long)acc[o][p][j] * q[j].z + off) >> 32) >> q[j].w, g.relu_lo);
                        }
                        out4 = pack_sat_u8x4(r[0], r[1], r[2], r[3]);
                    }
                    if (p == 0 || second)
                        *reinterpret_cast<uint32_t *>(reinterpret_cast<char *>(y) + out + o * out_row + p * col_pitch) = out4;
                }
            }
        }
    }
}

template <int ROWS, int S, bool FP = true>
static int depthwise3x3_strip_launch(const ConvGeom &g, const ConvDirectPlan &p, const uint8_t *x, int n, uint8_t *y, cudaStream_t st)
{
    DwArgs a;
    a.c4 = g.c / 4; a.h = g.h; a.w = g.w; a.oh = g.oh; a.ow = g.ow; a.pad_h = g.pad_h; a.pad_w = g.pad_w;
    const uint32_t pairs = (uint32_t)(g.ow + 1) / 2, strips = (uint32_t)(g.oh + ROWS - 1) / ROWS;
    a.stride_h = g.stride_h; a.relu_lo = g.relu_lo;
    a.by_c4 = FastDiv((uint32_t)a.c4);
    a.by_pairs = FastDiv(pairs);
    a.by_strips = FastDiv(strips);
    a.total = (uint32_t)n * strips * pairs * (uint32_t)a.c4;
    a.izp4 = (uint32_t)g.izp * 0x01010101u;
    const int lo = g.relu_lo > 0 ? g.relu_lo : 0;
    a.add = (float)(g.ozp - lo) + 0.5f;
    a.top2 = (uint32_t)(255 - lo) * 0x00010001u;
    a.lo4 = (uint32_t)lo * 0x01010101u;
    return launch_kernel(
        conv_depthwise3x3_strip_kernel<ROWS, S, FP>, dim3((a.total + 127) / 128), dim3(128), 0, st, (size_t)n * g.c * (g.h * g.w + g.oh * g.ow), 1,
        a, reinterpret_cast<const uint32_t *>(x), reinterpret_cast<const uint4 *>(p.w_dw3p_dev), reinterpret_cast<const uint4 *>(p.q_dw3p_dev),
        p.q_dw3_dev, reinterpret_cast<uint32_t *>(y));
}

// ---------------------------------------------------------------------------------------------
// Row lowering for the tensor-core path of 4-channel images (see kernels.h).  One thread builds
// one 32-byte window: eight 4-byte pixels, two 16-byte stores.  Neighbouring threads read
// overlapping windows, so the image is fetched from DRAM once.
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) conv_lower_rows_kernel(
    const uint32_t *__restrict__ x, uint4 *__restrict__ out, int n, int h, int w, int ow, int stride_w, int pad_w,
    uint32_t izp4)
{
    pdl_wait();
    pdl_trigger();
    const size_t total = (size_t)n * h * ow;
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (size_t)gridDim.x * blockDim.x) {
        const int ox = (int)(idx % ow);
        const size_t rowi = idx / ow;                       // n * h + ih
        const uint32_t *xrow = x + rowi * w;
        const int px0 = ox * stride_w - pad_w;
        uint32_t v[kLowerWindow];
#pragma unroll
        for (int j = 0; j < kLowerWindow; ++j) {
            const int px = px0 + j;
            v[j] = (px >= 0 && px < w) ? __ldg(xrow + px) : izp4;
        }
        // halves swapped where bit 2 of ox is set: the 32-byte swizzle, applied here in global memory
        const int sw = (ox >> 2) & 1;
        out[idx * 2 + sw] = make_uint4(v[0], v[1], v[2], v[3]);
        out[idx * 2 + (sw ^ 1)] = make_uint4(v[4], v[5], v[6], v[7]);
    }
}

int conv_lower_rows_launch(const ConvGeom &g, const uint8_t *x, int n, uint8_t *out, cudaStream_t st)
{
    if (n == 0)
        return B200_OK;
    if (g.c != 4 || (((uintptr_t)x) & 3) != 0 || (((uintptr_t)out) & 15) != 0)
        return fail(B200_ERR_INVALID, "conv(lower): needs a 4-channel, word-aligned input");
    const size_t total = (size_t)n * g.h * g.ow;
    const int blocks = resident_grid<conv_lower_rows_kernel, 256>((total + 255) / 256);
    return launch_kernel(
        conv_lower_rows_kernel, dim3((unsigned)blocks), dim3(256), 0, st, total * (kLowerWindow * 4), 1,
        reinterpret_cast<const uint32_t *>(x), reinterpret_cast<uint4 *>(out), n, g.h, g.w, g.ow, g.stride_w, g.pad_w,
        (uint32_t)g.izp * 0x01010101u);
}

// ---------------------------------------------------------------------------------------------
// Channel padding ahead of the tensor-core path.  One thread builds 16 bytes (or the 4 of a pixel of four
// channels) of one pixel; where a pixel is no whole number of words, they come out of two neighbouring
// aligned words each, and only words that hold a valid byte are read.
// ---------------------------------------------------------------------------------------------
template <int WORDS>
__global__ void __launch_bounds__(256) conv_pad_channels_kernel(
    const uint8_t *__restrict__ x, uint32_t *__restrict__ y, int c, FastDiv by_vecs, uint32_t total, uint32_t fill4)
{
    const uint32_t idx = blockIdx.x * 256 + threadIdx.x;
    pdl_wait();
    pdl_trigger();
    if (idx >= total)
        return;
    const uint32_t pix = by_vecs.div(idx), c0 = (idx - pix * by_vecs.d) * (WORDS * 4);
    const uint8_t *src = x + (size_t)pix * c + c0;
    const int valid = min(WORDS * 4, c - (int)c0);       // at least one: the padding is less than a vector
    const int skew = (int)((uintptr_t)src & 3);
    const uint32_t *w = reinterpret_cast<const uint32_t *>(src - skew);
    uint32_t in[WORDS + 1];
#pragma unroll
    for (int i = 0; i <= WORDS; ++i)
        in[i] = i * 4 < skew + valid ? __ldg(w + i) : 0;
    uint32_t o[WORDS];
#pragma unroll
    for (int i = 0; i < WORDS; ++i) {
        o[i] = __funnelshift_r(in[i], in[i + 1], 8 * skew);
        const int left = valid - 4 * i;                 // bytes of this word that exist
        if (left < 4) {
            const uint32_t keep = left <= 0 ? 0u : 0xffffffffu >> (32 - 8 * left);
            o[i] = (o[i] & keep) | (fill4 & ~keep);
        }
    }
    if constexpr (WORDS == 4)
        reinterpret_cast<uint4 *>(y)[idx] = make_uint4(o[0], o[1], o[2], o[3]);
    else
        y[idx] = o[0];
}

static int pad_vectors(int c_pad) { return c_pad == 4 ? 1 : c_pad / 16; }
bool conv_pad_channels_fits(size_t pixels, int c_pad) { return pixels * pad_vectors(c_pad) < 0x7fffff00ull; }

int conv_pad_channels_launch(const uint8_t *x, uint8_t *y, size_t pixels, int c, int c_pad, uint8_t fill, cudaStream_t st)
{
    const int vecs = pad_vectors(c_pad);
    const size_t total = pixels * vecs;
    if (!conv_pad_channels_fits(pixels, c_pad))
        return fail(B200_ERR_UNSUPPORTED, "conv(pad): tensor too large");
    const dim3 grid((unsigned)((total + 255) / 256));
    const uint32_t fill4 = (uint32_t)fill * 0x01010101u;
    const size_t bytes = pixels * (c + c_pad);
    if (c_pad == 4)
        return launch_kernel(conv_pad_channels_kernel<1>, grid, dim3(256), 0, st, bytes, 1, x, reinterpret_cast<uint32_t *>(y), c, FastDiv(vecs), (uint32_t)total, fill4);
    return launch_kernel(conv_pad_channels_kernel<4>, grid, dim3(256), 0, st, bytes, 1, x, reinterpret_cast<uint32_t *>(y), c, FastDiv(vecs), (uint32_t)total, fill4);
}

int conv_direct_launch(
    const ConvGeom &g, const ConvDirectPlan &p, const uint8_t *x, int n, uint8_t *y, int32_t *acc_out,
    cudaStream_t st)
{
    if (n == 0)
        return B200_OK;
    const size_t npix = (size_t)n * g.oh * g.ow;
    const int kg = g.k / g.group, cg = g.c / g.group;
    const size_t bytes = (size_t)n * g.h * g.w * g.c + npix * g.k;
    const bool depthwise = p.w_dw_dev && !acc_out && !g.act_signed && ((((uintptr_t)x | (uintptr_t)y) & 15) == 0);
    const bool dw3 = depthwise && p.w_dw3_dev && p.q_dw3_dev && npix * (size_t)(g.c / 4) < 0xffffffffull
        && (size_t)n * g.h * g.w * (size_t)(g.c / 4) < 0xffffffffull;
    if (dw3 && p.w_dw3p_dev && npix * (size_t)g.c < 0xffffff00ull && (size_t)n * g.h * g.w * g.c < 0xffffff00ull) {
        // Rows per thread: as many as leave every SM about a thousand threads, of the heights that fit the map
        // (144 channels of 56 x 56, batch 256: 80.6 us with 4 rows, 71.2 with 7, 60.3 with 14; 960 of 7 x 7: 10.3 with 7,
        // 13.1 with 14; stride 2 to 28 x 28: 41.4 with 2, 34.4 with 4, 35.0 with 7).
        const bool fp = p.q_dw3p_dev != nullptr;
        if (g.stride_w != g.stride_h) {
            if (g.stride_w == 1)
                return fp ? depthwise3x3_strip_launch<1, 1>(g, p, x, n, y, st) : depthwise3x3_strip_launch<1, 1, false>(g, p, x, n, y, st);
            return fp ? depthwise3x3_strip_launch<1, 2>(g, p, x, n, y, st) : depthwise3x3_strip_launch<1, 2, false>(g, p, x, n, y, st);
        }
        if (!fp)
            return g.stride_w == 1 ? depthwise3x3_strip_launch<2, 1, false>(g, p, x, n, y, st) : depthwise3x3_strip_launch<2, 2, false>(g, p, x, n, y, st);
        const size_t per_row = (size_t)n * ((g.ow + 1) / 2) * (g.c / 4), few = (size_t)sm_count() * 1024;
        auto strips = [&](int rows) { return (size_t)((g.oh + rows - 1) / rows); };
        if (g.stride_w == 1) {
            if (strips(14) * 14 * 7 <= strips(7) * 7 * 8 && per_row * strips(14) >= few)
                return depthwise3x3_strip_launch<14, 1>(g, p, x, n, y, st);
            if (per_row * strips(7) >= few)
                return depthwise3x3_strip_launch<7, 1>(g, p, x, n, y, st);
            return depthwise3x3_strip_launch<2, 1>(g, p, x, n, y, st);
        }
        if (g.oh <= 7 && per_row >= few)
            return depthwise3x3_strip_launch<7, 2>(g, p, x, n, y, st);
        if (per_row * strips(4) >= few)
            return depthwise3x3_strip_launch<4, 2>(g, p, x, n, y, st);
        return depthwise3x3_strip_launch<1, 2>(g, p, x, n, y, st);
    } else if (dw3) {
        const size_t total = npix * (g.c / 4);
        const int grid = resident_grid<conv_depthwise3x3_kernel, 256>((total + 255) / 256);
        return launch_kernel(
            conv_depthwise3x3_kernel, dim3(grid), dim3(256), 0, st, bytes, 1, g, reinterpret_cast<const uint32_t *>(x), reinterpret_cast<const uint4 *>(p.w_dw3_dev), p.q_dw3_dev,
            reinterpret_cast<uint32_t *>(y), n);
    } else if (depthwise) {
        size_t total = npix * (g.c / 16);
        size_t blocks = (total + 255) / 256;
        size_t cap = (size_t)sm_count() * 8;
        int grid = (int)(blocks < cap ? blocks : cap);
        if (g.wzp_d != 0)
            return launch_kernel(conv_depthwise_kernel<true>, dim3(grid), dim3(256), 0, st, bytes, 1, g, x, p.w_dw_dev, p.bias_fold_dev, p.mult_dev, p.shift_dev, y, n);
        return launch_kernel(conv_depthwise_kernel<false>, dim3(grid), dim3(256), 0, st, bytes, 1, g, x, p.w_dw_dev, p.bias_fold_dev, p.mult_dev, p.shift_dev, y, n);
    } else {
        const int ktiles = (kg + DK - 1) / DK;
        size_t gx = (npix + DP - 1) / DP;
        if (gx > 0x7fffffffull || (size_t)g.group * ktiles > 65535)
            return fail(B200_ERR_UNSUPPORTED, "conv(direct): grid too large");
        dim3 grid((unsigned)gx, (unsigned)(g.group * ktiles));
        const bool word = (g.c % 4 == 0) && (cg % 4 == 0) && (((uintptr_t)x & 3) == 0);
        const uint32_t *wq = reinterpret_cast<const uint32_t *>(p.w_dev);
        if (word)
            return launch_kernel(
                conv_direct_kernel<true>, grid, dim3(256), 0, st, bytes, 1, g, p.cg4, x, wq, p.bias_fold_dev, p.mult_dev, p.shift_dev, y, acc_out, n);
        return launch_kernel(
            conv_direct_kernel<false>, grid, dim3(256), 0, st, bytes, 1, g, p.cg4, x, wq, p.bias_fold_dev, p.mult_dev, p.shift_dev, y, acc_out, n);
    }
}

}  // namespace b200
