// Implicit-GEMM int8 convolution on the 5th-generation tensor cores (sm_100a):
//   D[pixels, Cout] (int32, TMEM) += A[pixels, R*S*C] (uint8 activations) x B[Cout, R*S*C]^T (int8)
// with tcgen05.mma kind::i8, operands staged by TMA into swizzled shared memory, accumulators in
// tensor memory, and the reference's zero-point correction, bias, requantize and ReLU clamp
// fused into the epilogue (art/modules/quant/src/op/conv_2d_uint8_impl.c:107-164 of ModelTC/NART).
//
// GEMM view.  An M tile is 128 output pixels arranged as a TW x TH x TN box of
// (ow, oh, image); for filter tap (r, s) and a BK-channel slice the A operand is the box of input
// pixels one tiled TMA load fetches from the NHWC tensor (coordinates may run outside the image:
// TMA fills zeros).  Strided convs address the input through one tensor map per (row, column)
// parity so that every load stays a plain dense box.  B is the weight matrix repacked once to
// [Cout][R][S][C] int8.  K is walked tap by tap, BK channels at a time.
//
// Zero point.  The MMA multiplies the raw uint8 activation, and TMA pads with the byte 0, whereas
// the reference pads with the real value 0, i.e. the byte izp.  With
//   raw = sum_{valid taps} x * w      true = sum_{valid taps} (x - izp) * w = raw - izp * sum_{valid} w
// the correction depends only on which taps are inside the image, i.e. on the output pixel's
// border class.  The host builds off[class][k] = bias[k] - izp * sum_{taps valid in class} w[k].
//
// Warp roles (576 threads, one CTA per SM, persistent over tiles):
//   warp 0      TMA producer (one elected lane)
//   warp 1      tensor-memory allocation, MMA issue (one elected lane)
//   warps 2..17 epilogue, two groups of 8 warps (two per tensor-memory lane quarter) or, for narrow
//               channel tiles with a short mainloop, four groups of 4 warps; group i
//               owns accumulator stage i: tcgen05.ld -> requantize -> pack -> swizzled smem -> TMA store
//   warps 18, 19  the producer and the MMA issuer of a second pipeline (MODE 1)
// One accumulator stage per group in tensor memory lets the epilogue of tile i overlap the mainloop
// of the next tiles and their epilogues (the other groups).  MODE 3 runs on clusters of two CTAs that
// share every MMA (tcgen05 cta_group::2, M = 256), each CTA loading its own operands with plain TMA
// loads; the other instantiations launch without clusters.  No load is multicast.  Every wait is bounded:
// when one runs out the kernel records a code in the status word, all roles leave their loops,
// tensor memory is freed and the kernel returns.
#pragma once

#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "conv_boxes.h"
#include "kernels.h"
#include "sm100_ptx.cuh"

namespace b200 {

constexpr int kMaxAccStages = 4;              // accumulator stages in tensor memory = epilogue groups: 2 or 4
#ifndef B200_EPI_WARPS
#define B200_EPI_WARPS 16
#endif
constexpr int kEpiWarps = B200_EPI_WARPS;     // split into 2 groups of 8 warps or 4 groups of 4
constexpr int kThreads = 64 + kEpiWarps * 32;
constexpr int kRing1Warp = 2 + kEpiWarps;       // MODE 1: the second pipeline's producer, and behind it its MMA issuer
constexpr int kThreads2 = kThreads + 64;
constexpr int kTileM = 128;
constexpr int kMaxStages = 8;
constexpr int kGroupBytes = 32 * 1024;        // target size of one pipeline stage (a group of k-blocks)
constexpr int kMaxGroup = 10;

// device status codes (which wait gave up)
constexpr int kErrProducerWait = 0x101;
constexpr int kErrMmaFullWait = 0x102;
constexpr int kErrMmaTmemWait = 0x103;
constexpr int kErrEpilogueWait = 0x104;

struct alignas(64) IgemmMaps {
    CUtensorMap a[4];   // activations, one per (row parity, column parity) of a strided conv
    CUtensorMap b;      // weights [Cout][R*S*C]
    CUtensorMap y[2];   // output NHWC, one per column segment of the staging buffer
    CUtensorMap ones;   // 16 rows, the first all ones (HAS_WZP)
};

struct IgemmArgs {
    // problem
    int n, oh, ow, cout;
    int r, s, pad_h, pad_w, stride_h, stride_w;
    int c;               // input channels, rounded up to a multiple of 32: the weights' pitch per tap
    int cchunks;         // k-blocks per tap
    int last_steps;      // 32-byte steps of a tap's last k-block that hold channels (the rest of its box is padding)
    // tiling
    int tw, th, tn;      // M-tile box (ow, oh, image), tw*th*tn == 128, each a power of two
    int tw_sh, th_sh;    // log2(tw), log2(th)
    int tiles_w, tiles_h, tiles_n, n_tiles_n;   // tile counts along ow, oh, image and Cout
    int step_nt, step_w, step_h, step_n;        // mixed-radix digits of the grid size (see TileWalker)
    int bk;              // channels per k-block (32, 64, 128) == swizzle span of the operands
    int bn;              // output channels per tile (multiple of 16, <= 256)
    int stages;          // smem pipeline depth
    int groups;          // epilogue groups (2 or 4); group i takes every groups-th tile of the CTA
    int acc_stages;      // accumulator stages in tensor memory (a multiple of groups, at most 4)
    int kgroup;          // k-blocks per pipeline stage (divides the k-blocks of a tile): one barrier round trip per group
    int b_resident;      // 1: all k-blocks of B stay in shared memory (one channel tile, weights fit)
    int a_wide;          // 1: 32-channel rows stored pre-swizzled; A is fetched as whole rows of pixels
    int seg_w[2];        // column segments of a tile: widths in bytes (the second may be 0), see epilogue_segments
    uint32_t idesc;      // tcgen05 instruction descriptor
    uint32_t tmem_cols;  // columns to allocate (power of two >= 2*bn)
    // epilogue (see EpiForm)
    const int32_t *off32;    // [n_cls][kpad] accumulator offsets (form kEpiFp: plus the bits of 1.5 * 2^23)
    const int32_t *mul;      // [kpad] fp32 bits, uniform-shift multiplier or multiplier, by form
    const int32_t *shift;    // [kpad] (form kEpiGeneric)
    const uint8_t *row_cls;  // [oh]
    const uint8_t *col_cls;  // [ow]
    int n_col_cls, n_cls, kpad;
    int ozp, qmax, relu_lo;
    uint32_t out_flip;       // 0x80808080 for int8 outputs, else 0
    int ushift, rnd_hi;      // form kEpiInt: S - 32; high word of 2^(S-1) + (ozp << S) (the low one is 0)
    int use_tma_store;       // 0: plain stores (Cout not a multiple of 16)
    uint8_t *y;
    int *status;
    // fused residual add (eltwise SUM of this conv's output and `res`, see EltwiseArgs): index 0 is
    // the conv's own output, index 1 the residual tensor (NHWC, the dims of y); res == nullptr: off
    const uint8_t *res;
    int r_m[2], r_add[2], r_b[2];
    int r_s0, r_ozp, r_lo;
    // weight zero point other than 128 (HAS_WZP): acc -= wzp_d * sum of x over the pixel's window before the
    // requantize; the MMA forms that sum in a 17th..32nd column behind the tile's channels (weight row of ones)
    int wzp_d;
    // 1: the M tiles are visited from the last image / row / column tile down to the first, so that a layer
    // starts on the part of its input that the layer before wrote last (and that still sits in L2)
    int rev;
    // Read-only bytes the launch after this one starts on (the next layer's repacked weights): every CTA asks
    // for its slice to be brought into L2 while this layer runs, so that the next launch's first weight loads
    // do not all miss at once.  nullptr / 0: none.
    const uint8_t *next_ro;
    uint32_t next_ro_bytes;
    // CTA pair (MODE 3): two CTAs of a cluster share every MMA (tcgen05 cta_group::2, M = 256): CTA r of the
    // pair owns M tile 2 * pm + r of pair tile pm and loads that tile's activations and half r of the
    // weight tile; the pair tiles are walked as (nt fastest, pm) with the digits step_nt, step_pm of the
    // number of clusters.
    int pm_tiles;            // pair tiles along M: ceil(m_tiles / 2)
    int step_pm;
};
// MODES 4 and 5: one box of activations for all taps of a channel chunk (and parity plane), box_bytes of shared memory each; the
// groups of eight accumulator rows lie box_group pixels apart in it
struct IgemmBoxArgs : IgemmArgs {
    HaloTiles halo;
    uint32_t box_bytes;
    int box_group;
    int a_pitch;             // shared memory a pixel takes: bk bytes; 16 with
    int quads;               // 1: pixels of 16 channels, several neighbours an operand row (see ConvIgemmPlan::quads)
};

// How accumulators become output bytes.  For the reference's  y = sat(rshift_rn((acc + off) * mult, shift) + ozp)
//   kEpiFp       floor((acc + off) * m + 1/2) + ozp with m = mult * 2^-shift, exactly, in fp32 (off32 carries the bits of
//                1.5 * 2^23, so that one integer add makes the float; see conv_depthwise3x3_strip_kernel for the rest).
//                For layers whose accumulators stay below 2^22 whatever the input: reductions of a few hundred bytes, where
//                the epilogue sets the pace.  Two values per fp32 instruction.
//   kEpiInt      every channel's shift brought to the layer's smallest one, S, by dropping low zero bits of its
//                multiplier (an fp32 scale leaves at least 7): ((acc + off) * mult_u + 2^(S-1) + (ozp << S)) >> S
//   kEpiGeneric  64-bit shifts per channel, for shifts below 33 and layers no single shift serves
// The constants of a tile's channels sit in shared memory, two per channel, read four at a time; the offsets of
// layers with several border classes are read through L1 from the class's row.
// (64 -> 256 channels 1x1 on 56 x 56, batch 256: 95.3 us with the two integer constants as kernel parameters, 78.4 fp32;
// 128 -> 512 on 28 x 28: 54.7 us with a 64-bit addend and a shift per channel in shared memory, 41.1 fp32.)
enum EpiForm { kEpiFp, kEpiInt, kEpiGeneric };
// One kernel per form and kind of offsets and clamp: side by side in one kernel they spill (96 registers a thread).
//   One / Many  one border class (offsets in shared memory) or several
//   Full        floor, ceiling below 255 and output flip; else the floor relu_lo and the pack's own ceiling
enum EpiVariant { kEpiFpOne, kEpiFpOneFull, kEpiFpMany, kEpiFpManyFull, kEpiIntOne, kEpiIntOneFull, kEpiIntMany, kEpiIntManyFull, kEpiAny, kEpiVariants };

// Tile index -> (Cout tile, ow tile, oh tile, image tile), Cout tile fastest.  A persistent CTA
// visits tiles blockIdx.x, blockIdx.x + gridDim.x, ...: the digits advance by the mixed-radix
// digits of gridDim.x (computed on the host) with carries, so no role divides inside its loop.
struct TileWalker {
    int nt, twi, thi, tni;
    int pm = 0, rank = -1;   // CTA-pair mode (rank >= 0): pair tile index along M and this CTA's rank in its pair
    __device__ __forceinline__ void decode_pair(const IgemmArgs &g)
    {
        int mt = 2 * pm + rank;          // an M tile past the last one decodes to an image index past the batch
        twi = mt % g.tiles_w;
        mt /= g.tiles_w;
        thi = mt % g.tiles_h;
        tni = mt / g.tiles_h;
    }
    __device__ __forceinline__ void init_pair(const IgemmArgs &g, int pair_tile, int cta_rank)
    {
        rank = cta_rank;
        nt = pair_tile % g.n_tiles_n;
        pm = pair_tile / g.n_tiles_n;
        decode_pair(g);
    }
    __device__ __forceinline__ void init(const IgemmArgs &g, int tile)
    {
        nt = tile % g.n_tiles_n;
        int mt = tile / g.n_tiles_n;
        twi = mt % g.tiles_w;
        mt /= g.tiles_w;
        thi = mt % g.tiles_h;
        tni = mt / g.tiles_h;
    }
    __device__ __forceinline__ void advance(const IgemmArgs &g)
    {
        if (rank >= 0) {
            nt += g.step_nt;
            int carry = 0;
            if (nt >= g.n_tiles_n) { nt -= g.n_tiles_n; carry = 1; }
            pm += g.step_pm + carry;
            decode_pair(g);
            return;
        }
        nt += g.step_nt;
        int carry = 0;
        if (nt >= g.n_tiles_n) { nt -= g.n_tiles_n; carry = 1; }
        twi += g.step_w + carry;
        carry = 0;
        if (twi >= g.tiles_w) { twi -= g.tiles_w; carry = 1; }
        thi += g.step_h + carry;
        carry = 0;
        if (thi >= g.tiles_h) { thi -= g.tiles_h; carry = 1; }
        tni += g.step_n + carry;
    }
    // tile coordinates as the roles use them (reversed traversal mirrors every M digit)
    __device__ __forceinline__ int wi(const IgemmArgs &g) const { return g.rev ? g.tiles_w - 1 - twi : twi; }
    __device__ __forceinline__ int hi(const IgemmArgs &g) const { return g.rev ? g.tiles_h - 1 - thi : thi; }
    // (an M tile past the end -- the odd tail of a CTA pair -- keeps its out-of-range image index)
    __device__ __forceinline__ int ni(const IgemmArgs &g) const { return (g.rev && tni < g.tiles_n) ? g.tiles_n - 1 - tni : tni; }
};

// The named barrier of one epilogue group.
__device__ __forceinline__ void epi_bar_sync(int group, int group_threads)
{
    asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(group_threads) : "memory");
}

// ---- epilogue arithmetic ------------------------------------------------------------------------
struct EpiConsts {
    int ozp, qmax, relu_lo, ushift, rnd_hi;
    float add;                 // ozp + 1/2
    uint32_t out_flip;
    int r_m0, r_add0, r_b0, r_m1, r_add1, r_b1, r_s0, r_ozp, r_lo;   // fused residual add
};

constexpr int kFpMagic = 0x4B400000;    // bits of 1.5 * 2^23
constexpr int kFpOne = 0x4B000000;      // bits of 2^23

// (volatile: the constants of later columns are not loaded ahead, there are no registers for them)
__device__ __forceinline__ int4 lds4(uint32_t addr)
{
    int4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ void sts4(uint32_t addr, uint4 v)
{
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

__device__ __forceinline__ uint32_t lds1(uint32_t addr)
{
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}

// n bytes of a staged row to global memory, whatever the alignment of dst, by `lanes` neighbouring lanes (`sub` is this one's
// number): aligned words, funnel-shifted out of two staged ones, and the bytes before and behind them.
// load(off): the staged word at byte off, a multiple of 4.
__device__ __forceinline__ int copy_lanes(int n) { return n <= 16 ? 4 : n <= 32 ? 8 : n <= 64 ? 16 : 32; }
template <typename Load>
__device__ __forceinline__ void copy_row(uint8_t *dst, int n, int sub, int lanes, Load load)
{
    const int head = min((int)((0u - (uint32_t)(uintptr_t)dst) & 3u), n), words = (n - head) >> 2, tail = (n - head) & 3;
    for (int w = sub; w < words; w += lanes) {
        const uint32_t a = load(4 * w), b = head ? load(4 * w + 4) : 0u;
        *reinterpret_cast<uint32_t *>(dst + head + 4 * w) = __funnelshift_r(a, b, 8 * head);
    }
    if (sub < head)
        dst[sub] = (uint8_t)(load(0) >> (8 * sub));
    const int back = lanes - 1 - sub;
    if (back < tail) {
        const int off = head + 4 * words + back;
        dst[off] = (uint8_t)(load(off & ~3) >> (8 * (off & 3)));
    }
}

// eltwise SUM of the four bytes of y (a conv's output) and x (the residual), as eltwise_sum_kernel forms it
__device__ __forceinline__ uint32_t add_residual(const uint32_t y, const uint32_t x, const EpiConsts &ec)
{
    int q[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int a = (int)__byte_perm(y, 0, 0x4440 | i), b = (int)__byte_perm(x, 0, 0x4440 | i);
        const int t = ((a * ec.r_m0 + ec.r_add0) >> ec.r_b0) + ((b * ec.r_m1 + ec.r_add1) >> ec.r_b1);
        q[i] = max((t >> ec.r_s0) + ec.r_ozp, ec.r_lo);
    }
    return pack_sat_u8x4(q[0], q[1], q[2], q[3]);
}

// N accumulator columns of this thread's row, requantized and packed.  mul, shift: shared addresses of the columns'
// constants; the offsets are in shared memory (OFF_SHARED: off_s) or global memory (off_g).
template <int FORM, bool OFF_SHARED, bool FULL, bool WZP, int N>
__device__ __forceinline__ void epi_pack(const uint32_t (&v)[N], const uint32_t off_s, const int32_t *off_g, const uint32_t mul, const uint32_t shift,
                                         const EpiConsts &ec, const int wz, uint32_t (&packed)[N / 4])
{
#pragma unroll
    for (int q4 = 0; q4 < N / 4; ++q4) {
        const int4 o = OFF_SHARED ? lds4(off_s + q4 * 16) : __ldg(reinterpret_cast<const int4 *>(off_g + q4 * 4));
        const int4 m = lds4(mul + q4 * 16);
        int a[4] = { (int)v[q4 * 4] + o.x, (int)v[q4 * 4 + 1] + o.y, (int)v[q4 * 4 + 2] + o.z, (int)v[q4 * 4 + 3] + o.w };
        const int mm[4] = { m.x, m.y, m.z, m.w };
        if (WZP) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                a[i] += wz;
        }
        int q[4];
        if constexpr (FORM == kEpiFp) {
            fp_requant_pair(a[0], a[1], mm[0], mm[1], ec.add, q[0], q[1]);
            fp_requant_pair(a[2], a[3], mm[2], mm[3], ec.add, q[2], q[3]);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                q[i] = FULL ? q[i] - kFpOne : __viaddmax_s32(q[i], -kFpOne, ec.relu_lo);
        } else if constexpr (FORM == kEpiInt) {
            const long long rnd = (long long)((unsigned long long)(uint32_t)ec.rnd_hi << 32);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                q[i] = (int)(((long long)a[i] * mm[i] + rnd) >> 32) >> ec.ushift;
                if (!FULL)
                    q[i] = max(q[i], ec.relu_lo);
            }
        } else {
            const int4 sh = lds4(shift + q4 * 16);
            const int ss[4] = { sh.x, sh.y, sh.z, sh.w };
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                // narrowed to int32 as the reference narrows before saturating
                q[i] = (int)(((long long)a[i] * mm[i] + (1ll << (ss[i] - 1)) + ((long long)ec.ozp << ss[i])) >> ss[i]);
            }
        }
        if (FULL) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                q[i] = max(min(q[i], ec.qmax), ec.relu_lo);
        }
        packed[q4] = pack_sat_u8x4(q[0], q[1], q[2], q[3]);
        if (FULL)
            packed[q4] ^= ec.out_flip;
    }
}

// Sixteen columns of the persistent kernel's tables: offsets, multipliers and shifts `pitch` bytes apart; rv: the
// residual's bytes (RES).
template <int FORM, bool ONE, bool FULL, bool WZP, bool RES>
__device__ __forceinline__ uint4 epi_half(const uint32_t (&v)[16], const uint32_t tab, const uint32_t pitch, const int32_t *off,
                                          const EpiConsts &ec, const int wz, const uint4 rv)
{
    uint32_t p[4];
    epi_pack<FORM, ONE, FULL, WZP>(v, tab, off, tab + pitch, tab + 2 * pitch, ec, wz, p);
    if (RES) {
        p[0] = add_residual(p[0], rv.x, ec);
        p[1] = add_residual(p[1], rv.y, ec);
        p[2] = add_residual(p[2], rv.z, ec);
        p[3] = add_residual(p[3], rv.w, ec);
    }
    return make_uint4(p[0], p[1], p[2], p[3]);
}


// The n16 groups of sixteen columns of one segment for this thread's row: the tensor-memory read of the next group is in
// flight while one is requantized (two register sets).  row_out: shared address of the row in the staging buffer, whose
// 16-byte chunks lie XOR-swizzled with sw16 / 16 as the TMA store's swizzle mode expects.  The accumulator stage goes back to
// the MMA warp (tempty: 0 = not yet) after the last read.
template <int FORM, bool ONE, bool FULL, bool WZP, bool RES>
__device__ __forceinline__ void epi_segment(uint32_t t_col, const int n16, uint32_t tab, const uint32_t pitch, const int32_t *off,
                                            const EpiConsts &ec, const int wz, const uint8_t *res, const uint32_t row_out, const uint32_t sw16,
                                            const uint32_t tempty, const bool remote)
{
    uint32_t va[16], vb[16];
    auto residual = [&](int h) { return RES && res ? __ldg(reinterpret_cast<const uint4 *>(res) + h) : make_uint4(0, 0, 0, 0); };
    auto drained = [&]() {
        if (tempty != 0) {
            tc_fence_before();
            __syncwarp();
            if ((threadIdx.x & 31) == 0) {
                if (remote)
                    mbar_arrive_cluster(tempty);
                else
                    mbar_arrive(tempty);
            }
        }
    };
    tmem_ld16(t_col, va);
#pragma unroll 1
    for (int h = 0; h < n16; h += 2, tab += 128) {
        const uint4 ra = residual(h);
        tmem_ld_wait();
        if (h + 1 < n16)
            tmem_ld16(t_col + (h + 1) * 16, vb);
        else
            drained();
        sts4(row_out + ((uint32_t)(h << 4) ^ sw16), epi_half<FORM, ONE, FULL, WZP, RES>(va, tab, pitch, off + h * 16, ec, wz, ra));
        if (h + 1 < n16) {
            const uint4 rb = residual(h + 1);
            tmem_ld_wait();
            if (h + 2 < n16)
                tmem_ld16(t_col + (h + 2) * 16, va);
            else
                drained();
            sts4(row_out + ((uint32_t)((h + 1) << 4) ^ sw16), epi_half<FORM, ONE, FULL, WZP, RES>(vb, tab + 64, pitch, off + h * 16 + 16, ec, wz, rb));
        }
    }
}

// ---- one offset row for all pixels: fragment layout ----------------------------------------------------------------
// A thread that holds a whole row of the tile reads the constants of every column, and 32 lanes that read the same 16 bytes
// still fill 512 bytes of registers: 2300 cycles of shared-memory traffic for a tile of 256 columns, which bound the layers
// with a short reduction.  Here a thread holds two columns of every eight, of four rows: a quarter of the constants.  They
// lie in pairs of columns, { offset, offset, multiplier, multiplier }.  The weight tile's rows are in an order that gives a
// thread four neighbouring channels of every sixteen, one word of the staging buffer: accumulator column 8 j + 2 q + e is
// channel 4 q + 2 j + e (the tensor map of the weights does that, see encode_weights).
// 1x1 256 -> 1024, 14x14, batch 256: 26.1 -> 23.0 us; 64 -> 256, 56x56, bound by instruction issue: 63.2 -> 63.7.
__device__ __forceinline__ void sts1(uint32_t addr, uint32_t v) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
template <int FORM, bool FULL>
__device__ __forceinline__ void requant2(uint32_t v0, uint32_t v1, const int4 &k, const EpiConsts &ec, int &q0, int &q1)
{
    const int a0 = (int)v0 + k.x, a1 = (int)v1 + k.y;
    if constexpr (FORM == kEpiFp) {
        fp_requant_pair(a0, a1, k.z, k.w, ec.add, q0, q1);
        q0 = FULL ? q0 - kFpOne : __viaddmax_s32(q0, -kFpOne, ec.relu_lo);
        q1 = FULL ? q1 - kFpOne : __viaddmax_s32(q1, -kFpOne, ec.relu_lo);
    } else {
        const long long rnd = (long long)((unsigned long long)(uint32_t)ec.rnd_hi << 32);
        q0 = (int)(((long long)a0 * k.z + rnd) >> 32) >> ec.ushift;
        q1 = (int)(((long long)a1 * k.w + rnd) >> 32) >> ec.ushift;
        if (!FULL) {
            q0 = max(q0, ec.relu_lo);
            q1 = max(q1, ec.relu_lo);
        }
    }
    if (FULL) {
        q0 = max(min(q0, ec.qmax), ec.relu_lo);
        q1 = max(min(q1, ec.qmax), ec.relu_lo);
    }
}
template <int FORM, bool FULL>
__device__ __forceinline__ uint32_t requant4(uint32_t v0, uint32_t v1, uint32_t v2, uint32_t v3, const int4 &k0, const int4 &k1, const EpiConsts &ec)
{
    int q[4];
    requant2<FORM, FULL>(v0, v1, k0, ec, q[0], q[1]);
    requant2<FORM, FULL>(v2, v3, k1, ec, q[2], q[3]);
    const uint32_t out = pack_sat_u8x4(q[0], q[1], q[2], q[3]);
    return FULL ? out ^ ec.out_flip : out;
}
// 8 X columns: two halves of sixteen rows.  row_out: shared address of this thread's first row (lane / 4), col its chunk of
// sixteen columns there; pitch8: bytes of eight rows.
template <int FORM, bool FULL, int X>
__device__ __forceinline__ void frag_half(const uint32_t (&v)[4 * X], const int4 (&k)[X], const EpiConsts &ec, uint32_t row_out, uint32_t pitch8,
                                          uint32_t chunk, uint32_t sw16, uint32_t in_chunk)
{
#pragma unroll
    for (int j = 0; j < X; j += 2) {
        const uint32_t at = row_out + (((chunk + (j >> 1)) << 4) ^ sw16) + in_chunk;
        sts1(at, requant4<FORM, FULL>(v[4 * j], v[4 * j + 1], v[4 * j + 4], v[4 * j + 5], k[j], k[j + 1], ec));
        sts1(at + pitch8, requant4<FORM, FULL>(v[4 * j + 2], v[4 * j + 3], v[4 * j + 6], v[4 * j + 7], k[j], k[j + 1], ec));
    }
}
template <int FORM, bool FULL>
__device__ __forceinline__ void frag_segment(uint32_t t_col, const int n16, uint32_t tab, const EpiConsts &ec, uint32_t row_out, const uint32_t pitch8,
                                             const uint32_t sw16, const uint32_t tempty, const bool remote)
{
    constexpr uint32_t kHalf = 16u << 16;           // sixteen lanes of tensor memory
    const uint32_t q = threadIdx.x & 3, in_chunk = 4 * q;
    tab += q * 32;
    auto drained = [&]() {
        if (tempty != 0) {
            tc_fence_before();
            __syncwarp();
            if ((threadIdx.x & 31) == 0) {
                if (remote)
                    mbar_arrive_cluster(tempty);
                else
                    mbar_arrive(tempty);
            }
        }
    };
    uint32_t va[16], vb[16];
    const int n32 = n16 >> 1;
    if (n32 > 0)
        tmem_ld_frag<4>(t_col, va);
#pragma unroll 1
    for (int h = 0; h < n32; ++h, tab += 256) {
        int4 k[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            k[j] = lds4(tab + (j >> 1) * 128 + (j & 1) * 16);
        tmem_ld_wait();
        tmem_ld_frag<4>(t_col + h * 32 + kHalf, vb);
        frag_half<FORM, FULL, 4>(va, k, ec, row_out, pitch8, 2 * h, sw16, in_chunk);
        tmem_ld_wait();
        if (h + 1 < n32)
            tmem_ld_frag<4>(t_col + h * 32 + 32, va);
        else if (!(n16 & 1))
            drained();
        frag_half<FORM, FULL, 4>(vb, k, ec, row_out + 2 * pitch8, pitch8, 2 * h, sw16, in_chunk);
    }
    if (n16 & 1) {
        uint32_t v0[8], v1[8];
        tmem_ld_frag<2>(t_col + n32 * 32, v0);
        tmem_ld_frag<2>(t_col + n32 * 32 + kHalf, v1);
        const int4 k[2] = { lds4(tab), lds4(tab + 16) };
        tmem_ld_wait();
        drained();
        frag_half<FORM, FULL, 2>(v0, k, ec, row_out, pitch8, 2 * n32, sw16, in_chunk);
        frag_half<FORM, FULL, 2>(v1, k, ec, row_out + 2 * pitch8, pitch8, 2 * n32, sw16, in_chunk);
    }
}

// ---- shared memory layout (dynamic, base aligned to 1024) ---------------------------------------
//   [stages x A tile (128 x bk)] [stages x B tile (bn x bk)] [2 x output staging 128 x bn]
//   [per epilogue group: offsets, multipliers, shifts, bn x 4 each] [barriers][tmem address][abort flag]
struct SmemLayout {
    uint32_t a, b, out, tables, bars, tmem_slot, abort_flag, total;
};
// b_slots: B tiles held in shared memory -- one per pipeline stage, or every k-block of the layer
// when the weights stay resident.
// box_bytes: what an A slot takes where that is no tile (MODES 4 and 5).
__host__ __device__ inline SmemLayout smem_layout(int a_slots, int b_slots, int bk, int bn, int groups, int bn_b = 0, uint32_t box_bytes = 0)
{
    if (bn_b == 0)
        bn_b = bn;      // rows of a B tile in this CTA's shared memory (half of bn in a CTA pair)
    SmemLayout L;
    uint32_t o = 0;
    L.a = o;
    o += (uint32_t)a_slots * (box_bytes ? box_bytes : (uint32_t)kTileM * bk);
    L.b = o;
    uint32_t b_tile = ((uint32_t)bn_b * bk + 1023u) & ~1023u;
    o += (uint32_t)b_slots * b_tile;
    L.out = o;
    o += (uint32_t)groups * kTileM * bn;   // one output staging buffer per epilogue group
    o = (o + 1023u) & ~1023u;
    L.tables = o;                      // per epilogue group: off[bn], mul[bn], shift[bn] (int32)
    o += (uint32_t)groups * bn * 12;
    o = (o + 15u) & ~15u;
    L.bars = o;
    o += (2 * kMaxStages + 2 * kMaxAccStages + 1) * 8;
    L.tmem_slot = o;
    o += 8;
    L.abort_flag = o;
    o += 8;
    L.total = o;
    return L;
}

// Rows p0 .. p0 + 31 of a staged segment (shared address seg_out, w bytes a row) to global memory, for channel counts the TMA
// store cannot address (Cout % 16 != 0).  valid: the rows inside the output; n0, oh0, ow0, k0: the tile's first pixel and the
// segment's first channel.
__device__ __forceinline__ void store_ragged(const IgemmArgs &g, uint32_t seg_out, int w, int p0, unsigned valid, int n0, int oh0, int ow0, int k0)
{
    const int lane = threadIdx.x & 31, n = min(w, g.cout - k0);
    if (n <= 0)
        return;
    auto row_at = [&](int pr, uint8_t *&dst, uint32_t &src, uint32_t &psw) {
        const int prow = p0 + pr;
        const int plw = prow & (g.tw - 1), plh = (prow >> g.tw_sh) & (g.th - 1), pln = prow >> (g.tw_sh + g.th_sh);
        dst = g.y + (((size_t)(n0 + pln) * g.oh + (oh0 + plh)) * g.ow + (ow0 + plw)) * g.cout + k0;
        psw = (w == 128 ? prow & 7 : w == 64 ? (prow >> 1) & 3 : w == 32 ? (prow >> 2) & 1 : 0) << 4;
        src = seg_out + (uint32_t)(prow * w);
    };
    if ((g.cout & 7) == 0 && (reinterpret_cast<uintptr_t>(g.y) & 7) == 0) {
        // the rows as one run of eight-byte words, four a lane in flight (1x1 96 -> 24, 56x56, batch 256: 43.7 -> 27.9 us)
        const int wpp = n >> 3, total = 32 * wpp;
        const uint32_t rcp = (65536u + (uint32_t)wpp - 1) / (uint32_t)wpp;      // exact for indexes below 1152, wpp <= 32
        for (int i0 = lane; i0 < total; i0 += 128) {
            uint32_t lo[4], hi[4];
            uint8_t *dst[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int idx = i0 + 32 * u, pr = (int)(((uint32_t)idx * rcp) >> 16), off = (idx - pr * wpp) * 8;
                uint32_t src, psw;
                dst[u] = nullptr;
                if (idx < total && ((valid >> pr) & 1)) {
                    row_at(pr, dst[u], src, psw);
                    dst[u] += off;
                    asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(lo[u]), "=r"(hi[u]) : "r"(src + ((uint32_t)off ^ psw)));
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (dst[u])
                    *reinterpret_cast<uint2 *>(dst[u]) = make_uint2(lo[u], hi[u]);
        }
        return;
    }
    // else pixel by pixel, the lanes side by side along its channels
    const int lanes = copy_lanes(n);
    for (int pr = lane / lanes; pr < 32; pr += 32 / lanes) {
        if (!((valid >> pr) & 1))
            continue;
        uint8_t *dst;
        uint32_t src, psw;
        row_at(pr, dst, src, psw);
        copy_row(dst, n, lane & (lanes - 1), lanes, [&](int off) { return lds1(src + ((uint32_t)off ^ psw)); });
    }
}

// HAS_RES: the instantiation whose epilogue can add a residual tensor; plans without a fused add run the
// other one, which carries none of that code.
// MODE 0: tile by tile.  MODE 1: two pipelines, each with its own producer, MMA issuer and half of the stages, take the CTA's
// tiles in turn: the producer's and the issuer's chains of instructions set the pace of short k-blocks.  MODE 2: the CTA's tiles go in pairs that share every weight k-block: a stage holds the activation
// tiles of both and ONE weight tile.  MODE 3: CTA pairs.  MODE 4: one box of activations for all taps, weights resident; MODE 5:
// the same in two pipelines.  A box per tap brings every pixel r * s times, and the producer's and issuer's chains with it; one box leaves
// the MMAs (54 cycles at least for 128 pixels by 32 bytes, 61 with 64 channels, wherever a swizzle atom the operand starts) and the epilogue.
// 3x3 64 -> 64 on 56 x 56: batch 256 49.3 -> 47.0 us, 32 11.2 -> 10.2; 32 -> 64 on 112 x 112, batch 64: 48.7 -> 36.4; with a weight zero
// point, which has one pipeline with a box per tap, 83 -> 48.7 and 82.9 -> 36.8.
// RAGGED: the instantiation that can store channel counts the TMA store cannot address (modes 0 and 1 run without it where
// they need not, which is worth 2 % to the layers their epilogue bounds).
template <int EPI, bool HAS_RES, bool HAS_WZP, int MODE, bool RAGGED = true>
__global__ void __launch_bounds__(MODE == 1 || MODE == 5 ? kThreads2 : kThreads, 1) conv_igemm_i8_kernel(const __grid_constant__ IgemmMaps maps, const __grid_constant__ std::conditional_t<MODE == 4 || MODE == 5, IgemmBoxArgs, IgemmArgs> g)
{
    extern __shared__ uint8_t smem_raw[];
    // the swizzle patterns are functions of the absolute shared address: align the base to 1024
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t base = (raw_addr + 1023u) & ~1023u;
    uint8_t *smem = smem_raw + (base - raw_addr);
    const int kblocks_all = g.r * g.s * g.cchunks;
    const int slots = g.stages * g.kgroup;
    constexpr bool PAIR = MODE == 3;
    uint32_t cta_rank = 0;
    if (PAIR)
        asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(cta_rank));
    const bool leader = !PAIR || cta_rank == 0;
    constexpr int kOnes = HAS_WZP ? 16 : 0;      // rows of B, and accumulator columns, behind the tile's channels
    const int bnl = PAIR ? g.bn >> 1 : g.bn + kOnes;     // rows of B this CTA holds
    constexpr bool HALO = MODE == 4 || MODE == 5, RINGS = MODE == 1 || MODE == 5;
    uint32_t box_bytes = 0;
    if constexpr (HALO)
        box_bytes = g.box_bytes;
    const SmemLayout L = smem_layout(MODE == 2 ? 2 * slots : slots, g.b_resident ? kblocks_all : slots, g.bk, g.bn, g.groups, bnl, box_bytes);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);      // uniform, and known to be
    const int lane = threadIdx.x & 31;
    const uint32_t a_tile_bytes = (uint32_t)kTileM * g.bk;
    const uint32_t b_tile_bytes = ((uint32_t)bnl * g.bk + 1023u) & ~1023u;
    const uint32_t bar0 = base + L.bars;
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (kMaxStages + s); };
    auto tfull_bar = [&](int s) { return bar0 + 8u * (2 * kMaxStages + s); };
    auto tempty_bar = [&](int s) { return bar0 + 8u * (2 * kMaxStages + kMaxAccStages + s); };
    const uint32_t bres_bar = bar0 + 8u * (2 * kMaxStages + 2 * kMaxAccStages);   // resident weights have landed
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(smem + L.tmem_slot);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + L.abort_flag);

    if (threadIdx.x == 0) {
        for (int s = 0; s < g.stages; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        mbar_init(bres_bar, 1);
        for (int s = 0; s < g.acc_stages; ++s) {
            mbar_init(tfull_bar(s), 1);
            // one arrival per warp of the stage's epilogue group (of both CTAs of a pair: the leading CTA's
            // barrier tells its MMA warp that the accumulator halves of both are free)
            mbar_init(tempty_bar(s), (kEpiWarps / g.groups) * (PAIR ? 2 : 1));
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        prefetch_map(&maps.a[0]);
        prefetch_map(&maps.b);
        prefetch_map(&maps.y[0]);
    }
    if (warp == 1) {
        if (PAIR) {
            tmem_alloc_pair(base + L.tmem_slot, g.tmem_cols);
            tmem_relinquish_pair();
        } else {
            tmem_alloc(base + L.tmem_slot, g.tmem_cols);
            tmem_relinquish();
        }
    }
    tc_fence_before();
    __syncthreads();
    if (PAIR)
        cluster_sync_all();     // the peer's barriers are initialised before anything arrives on them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (threadIdx.x == 2 * 32 && g.next_ro_bytes != 0) {
        // this CTA's slice of the next launch's read-only operand, in 16-byte granules
        const uint32_t granules = g.next_ro_bytes >> 4;
        const uint32_t per = (granules + gridDim.x - 1) / gridDim.x;
        const uint32_t first = blockIdx.x * per;
        if (first < granules) {
            const uint32_t cnt = min(per, granules - first);
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(g.next_ro + ((size_t)first << 4)), "r"(cnt << 4) : "memory");
        }
    }

    const int m_tiles = g.tiles_w * g.tiles_h * g.tiles_n;
    // the tile sequence of this CTA: tile0, tile0 + tstride, ...  (a CTA pair walks pair tiles together)
    const int total_tiles = PAIR ? g.pm_tiles * g.n_tiles_n : m_tiles * g.n_tiles_n;
    const int tile0 = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
    const int tstride = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
    auto walker_init = [&](TileWalker &w) {
        if (PAIR)
            w.init_pair(g, tile0, (int)cta_rank);
        else
            w.init(g, tile0);
    };
    const int cchunks = g.cchunks;
    const int kblocks = g.r * g.s * cchunks;
    constexpr bool one_class = EPI == kEpiFpOne || EPI == kEpiFpOneFull || EPI == kEpiIntOne || EPI == kEpiIntOneFull;
    constexpr bool frag = one_class && !HAS_RES && !HAS_WZP;     // (the host permutes the weight rows by the same rule)
    auto load_weights = [&](uint32_t dst, uint32_t bar, int kc, int row) {
        if constexpr (frag && PAIR)
            tma_load_5d_pair(dst, &maps.b, bar, kc, 0, 0, 0, row >> 4);
        else if constexpr (frag)
            tma_load_5d(dst, &maps.b, bar, kc, 0, 0, 0, row >> 4);
        else if constexpr (PAIR)
            tma_load_2d_pair(dst, &maps.b, bar, kc, row);
        else
            tma_load_2d(dst, &maps.b, bar, kc, row);
    };

    // this warp's pipeline (MODE 1), its stages and its first tile
    constexpr int tile_step = RINGS || MODE == 2 ? 2 : 1;
    const int ring = RINGS && warp >= kRing1Warp ? 1 : 0, ring_stages = RINGS ? g.stages >> 1 : g.stages;
    const int ring_tile0 = tile0 + ring * tstride, stage0 = ring * ring_stages;
    if (warp == 0 || (RINGS && warp == kRing1Warp)) {
        // ================= TMA producer =================
        // The warp walks the k-blocks of this CTA's tiles in order, one elected lane issues: wait for the stage of the next group of k-blocks, post
        // the group's byte count, issue its loads.  The chain of instructions of one k-block bounds the mainloop (its MMAs take
        // 64 .. 512 cycles), so addresses and coordinates advance by counters: chunk -> tap -> tile, with what depends on the
        // tap or the tile worked out when that changes.
        //
        // Two tiles per stage (MODE 2): a k-block is the activation tiles of both and the one weight tile they share (the host
        // has checked that).
        if (ring_tile0 < total_tiles) {
            const uint32_t bk = g.bk, kgroup = g.kgroup;
            // a CTA pair: the leading CTA's barrier counts the bytes of both CTAs
            const uint32_t tx_bytes = (a_tile_bytes + (g.b_resident ? 0u : (uint32_t)bnl * bk)) * kgroup * (PAIR ? 2u : 1u);
            const uint32_t a_slot = a_tile_bytes * (MODE == 2 ? 2 : 1), b_slot = b_tile_bytes;
            // weights are written once, at preparation: they need not wait for the launch before this one
            if (g.b_resident && ring == 0) {
                // one channel tile and weights that fit: every k-block of B is loaded once and stays
                if (elect_one())
                    mbar_expect_tx(bres_bar, (uint32_t)kblocks * bnl * bk);
                __syncwarp();
                uint32_t dst = base + L.b;
                for (int tap = 0; tap < g.r * g.s; ++tap)
                    for (int c = 0; c < cchunks; ++c, dst += b_slot) {
                        const int kc = tap * g.c + c * (int)bk;
                        if (elect_one()) {
                            load_weights(dst, bres_bar, kc, 0);
                            if (HAS_WZP)
                                tma_load_2d(dst + g.bn * bk, &maps.ones, bres_bar, kc, 0);
                        }
                    }
            }
            if constexpr (HALO) {
                const HaloTiles &h = g.halo;
                const uint32_t bars0 = full_bar(stage0), a_dst0 = base + L.a + (uint32_t)stage0 * g.box_bytes;
                uint32_t fb = bars0, a_dst = a_dst0, phase = 1;
                int stage = 0;
                TileWalker tw;
                walker_init(tw);
                if (ring == 1)
                    tw.advance(g);
                pdl_wait();
                bool ok = true;
                for (int tile = ring_tile0; ok && tile < total_tiles; tile += tile_step * tstride) {
                    const int x0 = tw.wi(g) << g.tw_sh, y0 = tw.hi(g) << g.th_sh, n0 = tw.ni(g);
                    for (int c = 0; ok && c < cchunks; ++c)
                        for (int pl = 0; pl < h.planes; ++pl) {
                            if (!mbar_wait_warp(fb + 8u * kMaxStages, phase, abort_flag)) {
                                if (lane == 0)
                                    atomicCAS(g.status, 0, kErrProducerWait);
                                *abort_flag = 1;
                                ok = false;
                                break;
                            }
                            if (elect_one()) {
                                mbar_expect_tx(fb, (uint32_t)(h.rows[pl] * g.a_pitch));
                                if (g.quads)
                                    tma_load_3d(a_dst, &maps.a[pl], fb, (x0 + h.dx) * 2, y0 + h.dy[pl], n0);
                                else
                                    tma_load_4d(a_dst, &maps.a[pl], fb, c * (int)bk, x0 + h.dx, y0 + h.dy[pl], n0);
                            }
                            __syncwarp();
                            fb += 8;
                            a_dst += g.box_bytes;
                            if (++stage == ring_stages) {
                                stage = 0;
                                fb = bars0;
                                a_dst = a_dst0;
                                phase ^= 1;
                            }
                        }
                    for (int i = 0; i < tile_step; ++i)
                        tw.advance(g);
                }
            } else {
            const int groups = kblocks / (int)kgroup;
            const int sh_h = g.stride_h - 1, sh_w = g.stride_w - 1;         // strides are 1 or 2
            const int c_end = cchunks * (int)bk, c_pitch = g.c, taps_w = g.s, pad_w = g.pad_w, pad_h = g.pad_h;
            const uint32_t bars0 = full_bar(stage0), bars_end = full_bar(stage0 + ring_stages);
            const uint32_t a_dst0 = base + L.a + (uint32_t)(stage0 * g.kgroup) * a_slot, b_dst0 = base + L.b + (uint32_t)(stage0 * g.kgroup) * b_slot;
            uint32_t fb = bars0, a_dst = a_dst0, b_dst = b_dst0, phase = 1;
            uint32_t fb_lead = PAIR ? cluster_addr(fb, 0) : 0u;
            const uint32_t fb_lead0 = fb_lead;
            constexpr uint32_t to_empty = 8u * kMaxStages;
            int tile = ring_tile0;
            TileWalker tw, tw2;
            walker_init(tw);
            if (MODE == 1 && ring == 1)
                tw.advance(g);
            if (MODE == 2)
                tw2 = tw;
            const bool load_b = !g.b_resident, a_wide = MODE != 2 && MODE != 3 && g.a_wide;
            // Groups of several k-blocks, up to 32 a tile: lane i knows where k-block i lies (offsets from the tile's first pixel,
            // map, channel, weight column), and the warp takes four entries at a time by shuffles.  The counters below are one
            // chain of instructions, ~190 cycles a k-block.  (3x3 64 -> 64, 56x56, batch 256: 51.2 -> 49.4 us)
            // An offset has seven bits: -64 from the padding up to 31 from at most 32 taps.
            const bool table = (MODE == 0 || MODE == 1) && kgroup > 1 && kblocks <= 32 && pad_h <= 64 && pad_w <= 64;
            uint32_t tab = 0;
            int tab_kc = 0;
            if (table) {
                const int kb = min(lane, kblocks - 1), tap = kb / cchunks, c = (kb - tap * cchunks) * (int)bk;
                const int trr = tap / taps_w, tss = tap - trr * taps_w;
                const int tdh = trr - pad_h, tph = tdh & sh_h, tdw = tss - pad_w, tpw = tdw & sh_w;
                tab = (uint32_t)(((tdw - tpw) >> sh_w) + 64) | (uint32_t)(((tdh - tph) >> sh_h) + 64) << 7 | (uint32_t)(tph * 2 + tpw) << 14 | (uint32_t)(c >> 5) << 16;
                tab_kc = tap * c_pitch + c;
            }
            pdl_wait();
            for (bool ok = true; ok && tile < total_tiles;) {
                const int x0 = tw.wi(g) << g.tw_sh, y0 = tw.hi(g) << g.th_sh, n0 = tw.ni(g) * g.tn;
                const int b_row = tw.nt * g.bn + (PAIR ? (int)cta_rank * bnl : 0);
                bool second = false;
                int dx2 = 0, dy2 = 0, n2 = 0;
                if (MODE == 2) {
                    tw2.advance(g);
                    second = tile + tstride < total_tiles;
                    dx2 = (tw2.wi(g) << g.tw_sh) - x0;
                    dy2 = (tw2.hi(g) << g.th_sh) - y0;
                    n2 = tw2.ni(g) * g.tn;
                }
                const uint32_t tx = tx_bytes + (MODE == 2 && second ? a_tile_bytes : 0u);       // (MODE 2: kgroup is 1)
                // k-blocks left of the group, of the tap; position of the tap
                int cc = 0, kc = 0, kc0 = 0, rr = 0, ss = 0;
                // input row of output row oh for this tap: ih = oh*stride + d, d = rr - pad
                //   = stride * (oh + (d - p) / stride) + p with p = d mod stride (0 <= p < stride)
                int dh = -pad_h, ph = dh & sh_h, yh = y0 + ((dh - ph) >> sh_h);
                int dw = -pad_w, pw = dw & sh_w, xw = x0 + ((dw - pw) >> sh_w);
                const CUtensorMap *amap = &maps.a[ph * 2 + pw];
                for (int grp = 0; grp < groups; ++grp) {
                    if (!mbar_wait_warp(fb + to_empty, phase, abort_flag)) {
                        if (lane == 0)
                            atomicCAS(g.status, 0, kErrProducerWait);
                        *abort_flag = 1;
                        ok = false;
                        break;
                    }
                    if ((!PAIR || leader) && elect_one())
                        mbar_expect_tx(fb, tx);
                    if (table) {
                        const int kb0 = grp * (int)kgroup;
                        for (int j0 = 0; j0 < (int)kgroup; j0 += 4) {
                            uint32_t e[4];
                            int ekc[4];
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                const int i = kb0 + min(j0 + u, (int)kgroup - 1);
                                e[u] = __shfl_sync(0xffffffffu, tab, i);
                                ekc[u] = load_b ? __shfl_sync(0xffffffffu, tab_kc, i) : 0;
                            }
                            if (elect_one()) {
#pragma unroll
                                for (int u = 0; u < 4; ++u)
                                    if (j0 + u < (int)kgroup) {
                                        const CUtensorMap *m = &maps.a[(e[u] >> 14) & 3];
                                        const int x = x0 + (int)(e[u] & 127) - 64, y = y0 + (int)((e[u] >> 7) & 127) - 64;
                                        const uint32_t a_at = a_dst + (uint32_t)(j0 + u) * a_slot, b_at = b_dst + (uint32_t)(j0 + u) * b_slot;
                                        if (a_wide)
                                            tma_load_3d(a_at, m, fb, x << 2, y, n0);
                                        else
                                            tma_load_4d(a_at, m, fb, (int)(e[u] >> 16) << 5, x, y, n0);
                                        if (load_b) {
                                            load_weights(b_at, fb, ekc[u], b_row);
                                            if (HAS_WZP)
                                                tma_load_2d(b_at + g.bn * bk, &maps.ones, fb, ekc[u], 0);
                                        }
                                    }
                            }
                            __syncwarp();
                        }
                        a_dst += kgroup * a_slot;
                        b_dst += kgroup * b_slot;
                    } else
                    for (int j = 0; j < (int)kgroup; ++j) {
                        if (elect_one()) {
                            if (PAIR) {
                                tma_load_4d_pair(a_dst, amap, fb_lead, cc, xw, yh, n0);
                                load_weights(b_dst, fb_lead, kc, b_row);
                            } else {
                                if (a_wide)                     // rows of tw pixels x 32 bytes, in 8-byte elements
                                    tma_load_3d(a_dst, amap, fb, xw << 2, yh, n0);
                                else
                                    tma_load_4d(a_dst, amap, fb, cc, xw, yh, n0);
                                if (MODE == 2 && second)        // the pair's second tile: same tap, its own pixels
                                    tma_load_4d(a_dst + a_tile_bytes, amap, fb, cc, xw + dx2, yh + dy2, n2);
                                if (load_b) {
                                    load_weights(b_dst, fb, kc, b_row);
                                    if (HAS_WZP)
                                        tma_load_2d(b_dst + g.bn * bk, &maps.ones, fb, kc, 0);
                                }
                            }
                        }
                        a_dst += a_slot;
                        b_dst += b_slot;
                        cc += bk;
                        kc += bk;
                        if (cc >= c_end) {
                            cc = 0;
                            kc = kc0 += c_pitch;
                            ++ss;
                            if (ss == taps_w) {
                                ss = 0;
                                ++rr;
                                dh = rr - pad_h, ph = dh & sh_h, yh = y0 + ((dh - ph) >> sh_h);
                            }
                            dw = ss - pad_w, pw = dw & sh_w, xw = x0 + ((dw - pw) >> sh_w);
                            amap = &maps.a[ph * 2 + pw];
                        }
                    }
                    fb += 8;
                    fb_lead += 8;
                    if (fb == bars_end) {
                        fb = bars0;
                        fb_lead = fb_lead0;
                        a_dst = a_dst0;
                        b_dst = b_dst0;
                        phase ^= 1;
                    }
                }
                tile += tile_step * tstride;
                tw.advance(g);
                if (tile_step == 2)
                    tw.advance(g);
                if (MODE == 2)
                    tw2.advance(g);
            }
            }
        }
        __syncwarp();
        // every load is on its way: the next launch's blocks may come (a block per SM that waits for longer
        // would keep the SM from the launches of other streams)
        if (ring == 0)
            pdl_trigger();
    } else if (warp == 1 || (RINGS && warp == kRing1Warp + 1)) {
        // ================= MMA issuer =================
        // The warp walks, one elected lane issues.  Descriptors of one operand differ only in the start-address field, so only their low words are
        // computed.  In a CTA pair the leading CTA's warp issues for both; the peer's has nothing to do.
        if (leader) {
            const int kgroup = g.kgroup, ksteps_full = g.bk / 32, last_steps = g.last_steps;
            int stage = stage0;
            uint32_t phase = 0;
            int as = ring;
            uint32_t aphase = 0;
            bool ok = true;
            const uint64_t adesc0 = make_smem_desc(base + L.a, g.bk);
            const uint32_t desc_hi = (uint32_t)(adesc0 >> 32);        // the same for A and B
            const uint32_t a_step = (a_tile_bytes >> 4) * (MODE == 2 ? 2 : 1), b_step = b_tile_bytes >> 4;   // descriptor address units
            const uint32_t a_lo0 = (uint32_t)adesc0 + (uint32_t)(stage0 * kgroup) * a_step;
            const uint32_t b_lo0 = (uint32_t)make_smem_desc(base + L.b, g.bk) + (g.b_resident ? 0u : (uint32_t)(stage0 * kgroup) * b_step);
            uint32_t a_lo = a_lo0, b_lo = b_lo0;
            const int groups = kblocks / kgroup;
            const uint32_t idesc = g.idesc, acc_cols = (uint32_t)(g.bn + kOnes);
            const bool resident = g.b_resident;
            auto give_up = [&](int code) {
                if (lane == 0)
                    atomicCAS(g.status, 0, code);
                *abort_flag = 1;
                ok = false;
            };
            if (resident && ring_tile0 < total_tiles && !mbar_wait_warp(bres_bar, 0, abort_flag))
                give_up(kErrMmaFullWait);
            for (int tile = ring_tile0; tile < total_tiles && ok; tile += tile_step * tstride) {
                // (MODE 2: the last step may lack the second tile)
                const bool second = MODE == 2 && tile + tstride < total_tiles;
                if (!mbar_wait_warp(tempty_bar(as), aphase ^ 1, abort_flag) || (second && !mbar_wait_warp(tempty_bar(as + 1), aphase ^ 1, abort_flag))) {
                    give_up(kErrMmaTmemWait);
                    break;
                }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)as * acc_cols;
                uint32_t accumulate = 0;
                int chunk = 0;        // k-block of the tap
                if constexpr (HALO) {
                    const HaloTiles &h = g.halo;
                    const uint32_t a_hi = halo_desc_hi(desc_hi, g.box_group, g.a_pitch, g.quads);
                    const uint32_t a_col = (uint32_t)g.a_pitch >> 4, a_row = (uint32_t)(h.pitch * g.a_pitch) >> 4;
                    const uint32_t b_tap = (uint32_t)cchunks * b_step, b_row = h.tap_row * b_tap;
                    const uint32_t box_step = g.box_bytes >> 4;
                    for (int c = 0; ok && c < cchunks; ++c) {
                        const int ksteps = c + 1 == cchunks ? last_steps : ksteps_full;
                        for (int pl = 0; pl < h.planes; ++pl) {
                            if (!mbar_wait_warp(full_bar(stage), phase, abort_flag)) {
                                give_up(kErrMmaFullWait);
                                break;
                            }
                            tc_fence_after();
                            // the taps of the plane, up to three of a row at a time
                            uint32_t a0 = (uint32_t)adesc0 + (uint32_t)stage * box_step, b0 = b_lo0 + (uint32_t)c * b_step + h.tap0[pl] * b_tap;
                            const int th = h.taps_h[pl], tw = h.taps_w;
                            for (int i = 0; i < th; ++i, a0 += a_row, b0 += b_row) {
                                uint32_t a = a0, b = b0;
                                for (int j = 0; j < tw; j += 3, a += 3 * a_col, b += 3 * b_tap) {
                                    auto tap = [&](uint32_t ta, uint32_t tb, uint32_t acc) {
                                        mma_i8_ab(d_tmem, ta, tb, a_hi, desc_hi, idesc, acc);
                                        if (ksteps >= 2)
                                            mma_i8_ab(d_tmem, ta + 2, tb + 2, a_hi, desc_hi, idesc, 1);
                                        if (ksteps >= 3)
                                            mma_i8_ab(d_tmem, ta + 4, tb + 4, a_hi, desc_hi, idesc, 1);
                                        if (ksteps == 4)
                                            mma_i8_ab(d_tmem, ta + 6, tb + 6, a_hi, desc_hi, idesc, 1);
                                    };
                                    if (elect_one()) {
                                        tap(a, b, accumulate);
                                        if (j + 1 < tw)
                                            tap(a + a_col, b + b_tap, 1);
                                        if (j + 2 < tw)
                                            tap(a + 2 * a_col, b + 2 * b_tap, 1);
                                    }
                                    __syncwarp();
                                    accumulate = 1;
                                }
                            }
                            if (elect_one()) {
                                mma_commit(empty_bar(stage));
                                if (c + 1 == cchunks && pl + 1 == h.planes)
                                    mma_commit(tfull_bar(as));
                            }
                            __syncwarp();
                            if (++stage == stage0 + ring_stages) {
                                stage = stage0;
                                phase ^= 1;
                            }
                        }
                    }
                    if (!ok)
                        break;
                    as += tile_step;
                    if (as >= g.acc_stages) {
                        as -= g.acc_stages;
                        aphase ^= 1;
                    }
                    continue;
                }
                if (resident)
                    b_lo = b_lo0;
                for (int grp = 0; grp < groups; ++grp) {
                    if (!mbar_wait_warp(full_bar(stage), phase, abort_flag)) {
                        give_up(kErrMmaFullWait);
                        break;
                    }
                    tc_fence_after();
                    for (int j = 0; j < kgroup; ++j, a_lo += a_step, b_lo += b_step) {
                        // a k-block is up to 4 MMAs of K = 32 bytes: +2 (16-byte units) inside the swizzle atom
                        int ksteps = ksteps_full;
                        if (++chunk == cchunks) {
                            chunk = 0;
                            ksteps = last_steps;
                        }
                        auto block = [&](uint32_t d, uint32_t a) {
                            auto mma = [&](int k, uint32_t acc) {
                                if (PAIR)
                                    mma_i8_pair(d, a + 2 * k, b_lo + 2 * k, desc_hi, idesc, acc);
                                else
                                    mma_i8(d, a + 2 * k, b_lo + 2 * k, desc_hi, idesc, acc);
                            };
                            mma(0, accumulate);
                            if (ksteps >= 2)
                                mma(1, 1);
                            if (ksteps >= 3)
                                mma(2, 1);
                            if (ksteps == 4)
                                mma(3, 1);
                        };
                        if (elect_one()) {
                            block(d_tmem, a_lo);
                            if (MODE == 2 && second)
                                block(d_tmem + acc_cols, a_lo + (a_tile_bytes >> 4));
                        }
                        __syncwarp();
                        accumulate = 1;
                    }
                    if (elect_one()) {
                        if (PAIR) {
                            // the stage is free again in both CTAs once these MMAs are done: one commit per CTA
                            mma_commit_pair(cluster_addr(empty_bar(stage), 0));
                            mma_commit_pair(cluster_addr(empty_bar(stage), 1));
                        } else
                            mma_commit(empty_bar(stage));   // frees the smem stage when the group's MMAs are done
                        if (grp + 1 == groups) {            // accumulator complete
                            if (PAIR) {                     // both CTAs' halves of it
                                mma_commit_pair(cluster_addr(tfull_bar(as), 0));
                                mma_commit_pair(cluster_addr(tfull_bar(as), 1));
                            } else
                                mma_commit(tfull_bar(as));
                            if (MODE == 2 && second)
                                mma_commit(tfull_bar(as + 1));
                        }
                    }
                    __syncwarp();
                    if (++stage == stage0 + ring_stages) {
                        stage = stage0;
                        phase ^= 1;
                        a_lo = a_lo0;
                        if (!resident)
                            b_lo = b_lo0;
                    }
                }
                if (!ok)
                    break;
                as += tile_step;
                if (as >= g.acc_stages) {
                    as -= g.acc_stages;
                    aphase ^= 1;
                }
            }
        }
        __syncwarp();
    } else {
        // ================= epilogue (warps 2..17) =================
        // Two independent groups of 8 warps; group i owns accumulator stage i, i.e. every second
        // tile of this CTA, with its own staging buffer, tables and named barriers, so that one
        // group's waits and barriers overlap the other group's arithmetic.
        const int group_warps = kEpiWarps / g.groups;      // 8 or 4: a multiple of four, one or two warps per lane quarter
        const int group_threads = group_warps * 32;
        const int group = (warp - 2) / group_warps;
        const int gw = (warp - 2) % group_warps;     // warp inside the group
        const int et = gw * 32 + lane;               // thread inside the group
        const int quarter = warp & 3;                // TMEM lanes 32*quarter .. +31 belong to this warp
        const int sub_warp = gw >> 2;                // which of the group's warps of that quarter
        const int row = quarter * 32 + lane;         // accumulator row = pixel of the tile
        int32_t *s_off = reinterpret_cast<int32_t *>(smem + L.tables + (size_t)group * g.bn * 12);
        int32_t *s_mul = s_off + g.bn, *s_shift = s_mul + g.bn;
        // one offset row for all pixels (1x1 and unpadded convs), in shared memory
        constexpr int form = EPI <= kEpiFpManyFull ? kEpiFp : EPI <= kEpiIntManyFull ? kEpiInt : kEpiGeneric;
        constexpr bool full = EPI == kEpiAny || (EPI & 1) != 0;
        const uint32_t out_bytes = (uint32_t)kTileM * g.bn;
        // this thread's pixel inside a tile (tw, th are powers of two)
        const int lw = row & (g.tw - 1), lh = (row >> g.tw_sh) & (g.th - 1), ln = row >> (g.tw_sh + g.th_sh);
        int as = group;                              // accumulator stage of this group's current tile
        uint32_t aphase = 0;
        int cur_nt = -1;
        bool store_pending = false;
        uint8_t *s_out = smem + L.out + (size_t)group * out_bytes;

        const EpiConsts ec = { g.ozp, g.qmax, g.relu_lo, g.ushift, g.rnd_hi, (float)g.ozp + 0.5f, g.out_flip,
                               g.r_m[0], g.r_add[0], g.r_b[0], g.r_m[1], g.r_add[1], g.r_b[1], g.r_s0, g.r_ozp, g.r_lo };

        // A tile's columns lie in the staging buffer as one or two segments, each a dense [pixel][width] box.  Each
        // warp owns its 32 rows of the segments it computes (all of them where it is alone on its lane quarter,
        // else the one of its number) and stores them with its own TMA store of the quarter box: no barrier between
        // the warps of a group on the way of a tile.  Group barriers remain only where the shared tables are reloaded.
        const int wpq = group_warps >> 2;                       // warps per lane quarter: 1 or 2
        const int seg0 = wpq == 1 ? 0 : sub_warp, seg1 = wpq == 1 ? (g.seg_w[1] ? 2 : 1) : (g.seg_w[sub_warp & 1] ? seg0 + 1 : seg0);
        // XOR mask of this row's 16-byte chunks in a segment of the given width (a power of two: TMA's swizzle; an odd
        // number of chunks spreads over the banks by itself)
        auto swizzle = [&](int w) { return w == 128 ? row & 7 : w == 64 ? (row >> 1) & 3 : w == 32 ? (row >> 2) & 1 : 0; };
        const int p0 = quarter * 32;                            // first pixel of this warp's rows inside a tile
        const int qlw = p0 & (g.tw - 1), qlh = (p0 >> g.tw_sh) & (g.th - 1), qln = p0 >> (g.tw_sh + g.th_sh);
        pdl_wait();            // the output may be what the launch before this one still reads
        bool failed = false;   // a wait ran out: skip the work of the remaining tiles, keep meeting the group barriers

        TileWalker tw;
        walker_init(tw);
        for (int i = 0; i < group; ++i)
            tw.advance(g);
        // a CTA pair's accumulator stages are handed back on the leading CTA's barrier
        auto tempty_arrive = [&](int stage_idx) {
            if (PAIR && !leader)
                mbar_arrive_cluster(cluster_addr(tempty_bar(stage_idx), 0));
            else
                mbar_arrive(tempty_bar(stage_idx));
        };
        for (int tile = tile0 + group * tstride; tile < total_tiles; tile += g.groups * tstride) {
            const int nt = tw.nt;
            const int ow0 = tw.wi(g) << g.tw_sh, oh0 = tw.hi(g) << g.th_sh, n0 = tw.ni(g) * g.tn;
            const int k0 = nt * g.bn;
            const int ow = ow0 + lw, oh = oh0 + lh, img = n0 + ln;
            const bool pix_valid = ow < g.ow && oh < g.oh && img < g.n;
            const uint8_t *res_row = g.res;
            if ((HAS_RES && g.res != nullptr) && pix_valid)
                res_row += (((size_t)img * g.oh + oh) * g.ow + ow) * g.cout + k0;
            int wz_t = 0;       // wzp != 128: this pixel's correction, the same for every channel
            int cls = 0;
            if (!one_class)
                cls = (int)g.row_cls[min(oh, g.oh - 1)] * g.n_col_cls + (int)g.col_cls[min(ow, g.ow - 1)];

            // per-channel tables change with the channel tile: the group meets before (everyone is
            // past the previous tile's reads) and after the reload
            if (nt != cur_nt) {
                epi_bar_sync(group, group_threads);
                for (int j = et; j < g.bn; j += group_threads) {
                    if (frag) {         // pairs of columns: { offset, offset, multiplier, multiplier }
                        const int at = (j >> 1) * 4 + (j & 1);
                        s_off[at] = g.off32[k0 + j];
                        s_off[at + 2] = g.mul[k0 + j];
                        continue;
                    }
                    s_mul[j] = g.mul[k0 + j];
                    if (EPI == kEpiAny)
                        s_shift[j] = g.shift[k0 + j];
                    if (one_class)
                        s_off[j] = g.off32[k0 + j];
                }
                epi_bar_sync(group, group_threads);
                cur_nt = nt;
            }
            if (!failed) {
                // this warp's previous store must have finished reading its part of the staging buffer
                if (store_pending) {
                    if (lane == 0)
                        tma_store_wait_read();
                    __syncwarp();
                }
                if (!__all_sync(0xffffffffu, mbar_wait(tfull_bar(as), aphase, abort_flag))) {
                    if (lane == 0) {
                        atomicCAS(g.status, 0, kErrEpilogueWait);
                        *abort_flag = 1;
                    }
                    failed = true;
                }
            }
            if (!failed) {
                tc_fence_after();
                const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(as * (g.bn + kOnes));
                if (HAS_WZP) {
                    uint32_t xs;
                    tmem_ld1(t_row + g.bn, xs);
                    tmem_ld_wait();
                    wz_t = -g.wzp_d * (int)xs;
                }
                const int32_t *off_row = g.off32 + (size_t)cls * g.kpad + k0;
                const uint32_t tab = smem_u32(s_off), pitch = (uint32_t)g.bn * 4;
                const uint32_t tempty = PAIR && !leader ? cluster_addr(tempty_bar(as), 0) : tempty_bar(as);
                const bool has_res = HAS_RES && g.res != nullptr;
                if (seg0 == seg1) {
                    tc_fence_before();
                    if (lane == 0)
                        tempty_arrive(as);
                }
                for (int seg = seg0; seg < seg1; ++seg) {
                    const int w = g.seg_w[seg], c0 = seg ? g.seg_w[0] : 0;
                    if constexpr (frag) {
                        const int frow = p0 + (lane >> 2);
                        const uint32_t fsw = w == 128 ? frow & 7 : w == 64 ? (frow >> 1) & 3 : w == 32 ? (frow >> 2) & 1 : 0;
                        frag_segment<form, full>(t_row + c0, w >> 4, tab + c0 * 8, ec, smem_u32(s_out) + (uint32_t)(kTileM * c0 + frow * w), 8 * w, fsw << 4,
                                                 seg + 1 == seg1 ? tempty : 0u, PAIR && !leader);
                    } else {
                        const uint32_t row_out = smem_u32(s_out) + (uint32_t)(kTileM * c0 + row * w);
                        epi_segment<form, one_class, full, HAS_WZP, HAS_RES>(
                            t_row + c0, w >> 4, tab + c0 * 4, pitch, off_row + c0, ec, wz_t, has_res && pix_valid ? res_row + c0 : nullptr, row_out,
                            (uint32_t)swizzle(w) << 4, seg + 1 == seg1 ? tempty : 0u, PAIR && !leader);
                    }
                }

                if (!RAGGED || g.use_tma_store) {
                    fence_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        for (int seg = seg0; seg < seg1; ++seg) {
                            const int c0 = seg ? g.seg_w[0] : 0;
                            if (k0 + c0 < g.cout)       // (the store clips what lies past Cout inside a segment)
                                tma_store_4d(&maps.y[seg], smem_u32(s_out + (size_t)kTileM * c0 + p0 * g.seg_w[seg]),
                                             k0 + c0, ow0 + qlw, oh0 + qlh, n0 + qln);
                        }
                        tma_store_commit();
                    }
                    store_pending = true;
                } else {
                    __syncwarp();
                    const unsigned valid = __ballot_sync(0xffffffffu, pix_valid);
                    for (int seg = seg0; seg < seg1; ++seg) {
                        const int c0 = seg ? g.seg_w[0] : 0;
                        store_ragged(g, smem_u32(s_out) + (uint32_t)(kTileM * c0), g.seg_w[seg], p0, valid, n0, oh0, ow0, k0 + c0);
                    }
                    __syncwarp();
                }
            }
            as += g.groups;                          // the group's next tile: stage (as + groups) mod acc_stages
            if (as >= g.acc_stages) {
                as -= g.acc_stages;
                aphase ^= 1;
            }
            for (int i = 0; i < g.groups; ++i)
                tw.advance(g);
        }
        if (store_pending && lane == 0)
            tma_store_wait_all();
    }

    // ---- common exit: every role gets here (all waits are bounded) ---------------------------------
    tc_fence_before();
    __syncthreads();
    if (PAIR)
        cluster_sync_all();     // neither CTA leaves (or gives tensor memory back) while its peer still works on the pair
    if (warp == 1) {
        tc_fence_after();
        if (PAIR)
            tmem_dealloc_pair(tmem_base, g.tmem_cols);
        else
            tmem_dealloc(tmem_base, g.tmem_cols);
    }
}


// The kernels, by EpiVariant; nullptr where a combination is not built.  The instantiations are spread over
// conv_igemm_inst_*.cu, which compile side by side.
typedef void (*IgemmKernel)(const IgemmMaps, const IgemmArgs);
IgemmKernel igemm_kernel_mode0(int epi);
IgemmKernel igemm_kernel_mode1(int epi);
IgemmKernel igemm_kernel_ragged(int epi, bool two_pipelines);
IgemmKernel igemm_kernel_mode2(int epi);
IgemmKernel igemm_kernel_mode3(int epi);                // none for variants that only short reductions have
typedef void (*IgemmBoxKernel)(const IgemmMaps, const IgemmBoxArgs);
IgemmBoxKernel igemm_kernel_mode4(int epi, bool wzp);
IgemmBoxKernel igemm_kernel_mode5(int epi, bool wzp);
IgemmKernel igemm_kernel_wzp(int epi);                  // a weight zero point other than 128
IgemmKernel igemm_kernel_residual(int epi);             // a residual add: none for the Full variants and kEpiAny

}  // namespace b200
