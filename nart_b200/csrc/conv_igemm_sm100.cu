// Host side of the implicit-GEMM convolution (kernels: conv_igemm_kernel.cuh, conv_small_sm100.cu): plans -- weights
// repacked, tiling, epilogue form and constants -- and launches, with their tensor maps.
#include <atomic>
#include <cuda.h>
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <cstdlib>
#include <vector>

#include "common.cuh"
#include "conv_igemm_kernel.cuh"
#include "conv_small.h"
#include "kernels.h"
#include "sm100_ptx.cuh"

namespace b200 {

namespace {

constexpr int kErrSelfTestWait = 0x1ff;   // wait_expiry_probe_kernel

// The give-up path of the bounded waits, on its own: one warp waits, through the same mbar_wait the
// convolution's roles use, on a barrier that nothing will ever arrive at, with the caller's (short)
// limit.  When the limit is reached the wait returns false, the code goes to the status word and the
// kernel ends normally -- no trap, nothing left waiting.
__global__ void __launch_bounds__(32) wait_expiry_probe_kernel(int *status, long long limit_cycles)
{
    __shared__ __align__(8) unsigned long long bar;
    __shared__ int abort_flag;
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&bar), 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    const bool ok = mbar_wait(smem_u32(&bar), 0, &abort_flag, limit_cycles);
    if (!__all_sync(0xffffffffu, ok) && threadIdx.x == 0) {
        atomicCAS(status, 0, kErrSelfTestWait);
        abort_flag = 1;
    }
}

// The tensor pipe's own rate for this kernel's instruction: every SM issues `mmas` MMAs of the shape the
// 256-wide tiles use (kind::i8, M128 x N256 x K32, u8 x s8 -> s32) back to back on operands that stay in
// shared memory (pseudo-random bytes: all-zero operands would draw less power and run at other clocks),
// alternating between two accumulators every 32 MMAs.  No loads, no epilogue: the number it gives is the
// ceiling the convolution's mainloop is measured against.
constexpr int kPeakGroup = 32;   // MMAs per commit
__global__ void __launch_bounds__(128, 1) mma_i8_peak_kernel(int mmas, int *status)
{
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t base = (raw_addr + 1023u) & ~1023u;
    uint8_t *smem = smem_raw + (base - raw_addr);
    constexpr uint32_t kA = 128 * 128, kB = 256 * 128;
    __shared__ __align__(8) unsigned long long bars[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    for (uint32_t i = threadIdx.x; i < (kA + kB) / 4; i += blockDim.x)
        reinterpret_cast<uint32_t *>(smem)[i] = (i + blockIdx.x) * 2654435761u;
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&bars[0]), 1);
        mbar_init(smem_u32(&bars[1]), 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    fence_async_smem();
    if (threadIdx.x < 32) {
        tmem_alloc(smem_u32(&tmem_slot), 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_slot;
    if (threadIdx.x < 32) {
        const uint32_t lead = threadIdx.x == 0 ? 1u : 0u;
        const uint64_t adesc = make_smem_desc(base, 128), bdesc = make_smem_desc(base + kA, 128);
        const uint32_t desc_hi = (uint32_t)(adesc >> 32), a_lo = (uint32_t)adesc, b_lo = (uint32_t)bdesc;
        const uint32_t idesc = (2u << 4) | (0u << 7) | (1u << 10) | ((256u >> 3) << 17) | ((128u >> 4) << 24);
        const int groups = mmas / kPeakGroup;
        uint32_t phase[2] = { 0, 0 };
        bool ok = true;
        for (int gi = 0; gi < groups && ok; ++gi) {
            const int b = gi & 1;
            if (gi >= 2) {     // the group two back has drained: at most two groups are queued
                if (!mbar_wait(smem_u32(&bars[b]), phase[b], &abort_flag)) {
                    if (lead)
                        atomicCAS(status, 0, kErrSelfTestWait);
                    ok = false;
                    break;
                }
                phase[b] ^= 1;
            }
            const uint32_t d = tmem_base + (uint32_t)b * 256u;
            if (elect_one()) {
#pragma unroll 4
                for (int j = 0; j < kPeakGroup; ++j)
                    mma_i8(d, a_lo + 2 * (j & 3), b_lo + 2 * (j & 3), desc_hi, idesc, j ? 1u : 0u);
                mma_commit(smem_u32(&bars[b]));
            }
        }
        // the last groups must have finished before tensor memory goes back
        for (int t = groups < 2 ? 0 : groups - 2; t < groups && ok; ++t) {
            const int b = t & 1;
            if (!mbar_wait(smem_u32(&bars[b]), phase[b], &abort_flag)) {
                if (lead)
                    atomicCAS(status, 0, kErrSelfTestWait);
                ok = false;
            }
            phase[b] ^= 1;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x < 32) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

// ---- host side -------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(
    CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
    const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
    CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn()
{
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess
            && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

CUtensorMapSwizzle swizzle_for(int bytes)
{
    return bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
        : bytes == 64   ? CU_TENSOR_MAP_SWIZZLE_64B
        : bytes == 32   ? CU_TENSOR_MAP_SWIZZLE_32B
                        : CU_TENSOR_MAP_SWIZZLE_NONE;
}

int encode(CUtensorMap *m, void *base, int rank, const cuuint64_t *dims, const cuuint64_t *strides_bytes,
           const cuuint32_t *box, CUtensorMapSwizzle sw, CUtensorMapDataType dtype = CU_TENSOR_MAP_DATA_TYPE_UINT8)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn)
        return fail(B200_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
    cuuint32_t estr[5] = { 1, 1, 1, 1, 1 };
    CUresult r = CUDA_SUCCESS;
    for (int round = 0; round < 2; ++round) {
        r = fn(m, dtype, (cuuint32_t)rank, base, dims, strides_bytes, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        int device = 0;
        if (r != CUDA_ERROR_INVALID_CONTEXT || cudaGetDevice(&device) != cudaSuccess || cudaSetDevice(device) != cudaSuccess)
            break;      // else this is the thread's first call to CUDA: its context is current now
    }
    if (r != CUDA_SUCCESS)
        return fail(B200_ERR_CUDA, "cuTensorMapEncodeTiled failed with CUresult %d (rank %d, dims %llu %llu, box %u %u)",
                    (int)r, rank, (unsigned long long)dims[0], (unsigned long long)dims[1], box[0], box[1]);
    return B200_OK;
}

}  // namespace

struct ConvIgemmPlan {
    ConvGeom g;
    int groups = 2, acc_stages = 2;
    int cpad = 0;                   // input channels rounded up to a multiple of 32
    int bk = 0, bn = 0, stages = 0, kgroup = 1, kpad = 0, b_resident = 0, a_wide = 0, rings = 1, pair = 0;
    // Two CTAs of a cluster per MMA (kernel MODE 3).  Whether a launch uses it depends on the batch: the pair
    // wins 3-6 % once every cluster walks many tiles and loses a little on short launches (cluster launch,
    // two cluster-wide syncs), so the plan carries both configurations and build_launch picks.
    int pair_ok = 0, pair_want = -1, stages_pair = 0;
    int max_clusters = 0;           // co-resident CTA pairs of that kernel on this device
    // Pixels of 16 channels of which an operand row holds as many neighbours as the window has columns, rounded up to 2, 4 or 8: the
    // pixels of a box lie 16 bytes apart and rows of 32 to 128 bytes overlap, which the unswizzled layout can say.  A row of
    // the window is then one tap (taps_w is 1).
    int quads = 0, taps_w = 0;
    // One box of activations for all taps (kernel MODE 4), its tiles and its stages (0: not possible)
    HaloTiles halo;
    int stages_halo = 0, box_group = 8, halo_want = -1;
    uint32_t box_bytes = 0;
    int n_row_cls = 0, n_col_cls = 0;
    int seg_w[2] = { 0, 0 };        // see epilogue_segments
    int form = kEpiGeneric, variant = kEpiAny, ushift = 0, rnd_hi = 0;      // see EpiForm, EpiVariant
    uint8_t *block_dev = nullptr;   // the device memory behind all of these
    int8_t *w_dev = nullptr;        // [kpad][r][s][c]
    int32_t *off32_dev = nullptr;   // [n_cls][kpad] accumulator offsets
    int32_t *off_form_dev = nullptr;    // the same plus kFpMagic (kEpiFp)
    int32_t *mul_form_dev = nullptr;    // [kpad]
    int32_t *shift_dev = nullptr;   // [kpad]
    uint8_t *row_cls_dev = nullptr, *col_cls_dev = nullptr;
    int rev = 0;                    // reversed tile traversal (conv_igemm_set_reverse)
    NextRead next;                  // what the next launch reads first (conv_igemm_set_next_readonly)
    size_t w_bytes = 0;             // size of w_dev
    // fused residual add (conv_igemm_set_residual)
    bool has_res = false;
    int r_m[2] = { 0, 0 }, r_add[2] = { 0, 0 }, r_b[2] = { 1, 1 };
    int r_s0 = 1, r_ozp = 0, r_lo = 0;
    int small_bn = 0, small_split = 0;
    bool small_ok = true;           // one tile per CTA where a launch leaves SMs without a tile
    int8_t *ones_dev = nullptr;     // wzp != 128: [16][r][s][c], the first row ones where the window has a channel
    bool attr_set = false;
    // Launch configurations by buffers and batch (callers that rotate through a handful of buffers): found again
    // without encoding tensor maps.
    struct Launch {
        const uint8_t *x;
        const uint8_t *res;
        const uint8_t *sum_res;     // ConvSum
        uint8_t *sum;
        bool summed;
        uint8_t *y;
        int n;
        int *status;
        bool small;                 // the one-tile-per-CTA kernel (conv_small_sm100.cu): smaps, sargs, m_tiles
        int cta_pair;
        bool halo;
        int m_tiles;
        IgemmKernel kernel;
        IgemmBoxKernel box_kernel;
        dim3 grid;
        size_t smem;
        SmallMaps smaps;
        SmallArgs sargs;
        IgemmMaps maps;
        IgemmBoxArgs args;
    };
    static constexpr size_t kMaxSaved = 8;
    std::vector<Launch> saved;
    size_t next_saved = 0, last = 0;
    const Launch *last_launch() const { return last < saved.size() ? &saved[last] : nullptr; }
};

// Cuts a tile's `bn` columns into at most two staging segments: one per warp of a lane quarter, or up to two that a
// lone warp handles.  A segment's row is one 16-byte chunk times 2, 4 or 8 -- TMA's swizzles keep its rows off each
// other's banks -- or times an odd number, where rows spread over the banks by themselves and are stored unswizzled.
static void epilogue_segments(int bn, int warps_per_quarter, int (&w)[2])
{
    const int t = bn / 16;
    auto good = [](int c) { return c % 2 == 1 || c == 0 || c == 2 || c == 4 || c == 8; };
    int a = t;
    if (warps_per_quarter == 2 || !good(t))
        for (a = (t + 1) / 2; !good(a) || !good(t - a); ++a) {}
    w[0] = a * 16;
    w[1] = (t - a) * 16;
}

// One filter's weights [taps][c] to [taps][pitch], with the sum of each tap.
void weights_to_pitch(const int8_t *w, int c, int taps, int8_t *dst, int pitch, int32_t *sums)
{
    for (int t = 0; t < taps; ++t) {
        const int8_t *src = w + (size_t)t * c;
        memcpy(dst + (size_t)t * pitch, src, c);
        int32_t sum = 0;
        for (int i = 0; i < c; ++i)
            sum += src[i];
        sums[t] = sum;
    }
}

int conv_igemm_supported(const ConvGeom &g, char *why, size_t why_len)
{
    const char *msg = nullptr;
    if (g.group != 1) msg = "group != 1";
    else if (g.c % 16 != 0) msg = "input channels not a multiple of 16";   // the pixel stride of a TMA map
    else if (g.k < 16) msg = "fewer than 16 output channels";
    else if (g.stride_h > 2 || g.stride_w > 2) msg = "stride > 2";
    else if (g.h < g.stride_h || g.w < g.stride_w) msg = "input smaller than the stride";
    else if ((long long)g.r * g.s * ((g.c + 31) / 32) >= 32768) msg = "more than 32767 k-blocks per tile";
    if (msg) {
        snprintf(why, why_len, "%s", msg);
        return 0;
    }
    return 1;
}

// Distinct sets of in-image taps along one axis: cls[o] = class of output coordinate o, and
// valid[class][t] = whether tap t falls inside the image.  The taps of a coordinate that do are neighbours: two numbers a class.
static void tap_classes(int out, int in, int kernel, int pad, int stride, std::vector<uint8_t> &cls,
                        std::vector<std::vector<char>> &valid)
{
    cls.resize(out);
    valid.clear();
    std::vector<std::pair<int, int>> spans;         // [first, end) of the taps inside, per class
    size_t id = 0;
    for (int o = 0; o < out; ++o) {
        const long long at = (long long)o * stride - pad;
        std::pair<int, int> span((int)std::max(0ll, -at), (int)std::min((long long)kernel, in - at));
        if (span.first >= span.second)
            span = { 0, 0 };
        if (id >= spans.size() || spans[id] != span) {
            id = 0;
            while (id < spans.size() && spans[id] != span)
                ++id;
            if (id == spans.size()) {
                spans.push_back(span);
                valid.emplace_back(kernel, 0);
                std::fill(valid[id].begin() + span.first, valid[id].begin() + span.second, 1);
            }
        }
        int last = o;
        if (span.first == 0 && span.second == kernel)       // all up to the other border
            last = (int)std::min((long long)out - 1, ((long long)in - kernel + pad) / stride);
        std::fill(cls.begin() + o, cls.begin() + last + 1, (uint8_t)id);
        o = last;
    }
}

int conv_igemm_create(
    const ConvGeom &g, const std::vector<int8_t> &w_s8, const int32_t *bias, const uint32_t *mult,
    const int32_t *shift, ConvIgemmPlan **out, bool a_row_swizzled, int window, bool quads)
{
    if (a_row_swizzled && !(g.c == 32 && g.s == 1 && g.stride_w == 1 && g.pad_w == 0 && g.w == g.ow))
        return fail(B200_ERR_INVALID, "conv(igemm): pre-swizzled rows need 32 channels and an r x 1 kernel");
    // The epilogue adds the accumulator offset in 64-bit arithmetic, where the reference's int32
    // accumulator would wrap; and its folded addend needs shift <= 53 to stay inside int64.
    {
        long long max_bias = 0;
        for (int k = 0; k < g.k && bias; ++k) {
            long long b = bias[k] < 0 ? -(long long)bias[k] : (long long)bias[k];
            if (b > max_bias)
                max_bias = b;
        }
        const long long wmag = 128ll + (g.wzp_d < 0 ? -g.wzp_d : g.wzp_d);   // |s8| plus the zero-point correction
        if (max_bias + (long long)g.r * g.s * g.c * 255ll * wmag >= (1ll << 31))
            return fail(B200_ERR_UNSUPPORTED, "conv(igemm): the int32 accumulator could wrap");
        for (int k = 0; k < g.k; ++k)
            if (shift[k] > 53)
                return fail(B200_ERR_UNSUPPORTED, "conv(igemm): shift %d of channel %d exceeds 53", shift[k], k);
    }
    ConvIgemmPlan *p = new ConvIgemmPlan();
    p->g = g;
    if (const char *e = getenv("B200_IGEMM_SMALL")) {           // tuning aid: 0, or <channels per tile>x<CTAs per tile>
        int bn = 0, split = 0;
        if (sscanf(e, "%dx%d", &bn, &split) == 2) {
            if ((bn == 16 || bn == 32 || bn == 64 || bn == 128) && (split == 1 || split == 2 || split == 4 || split == 8) && bn / split >= 8) {
                p->small_bn = bn;
                p->small_split = split;
            }
        } else if (atoi(e) == 0) {
            p->small_ok = false;
        }
    }
    p->saved.reserve(ConvIgemmPlan::kMaxSaved);   // launches never grow it: a later run touches no heap
    p->a_wide = a_row_swizzled ? 1 : 0;
    p->quads = quads ? 1 : 0;
    p->taps_w = quads ? 1 : g.s;
    const int mma_taps = g.r * p->taps_w;
    // K of an 8-bit MMA is 32 bytes: the channel count is rounded up to a multiple of 32 in the
    // repacked weights (zero weights); on the activation side the TMA box runs past the tensor's
    // channel extent and reads zeros there
    p->cpad = quads ? (g.s <= 2 ? 32 : g.s <= 4 ? 64 : 128) : (g.c + 31) / 32 * 32;
    // The k-block: 32, 64 or 128 channels.  The last block of a tap may run past the channels (TMA zero fill; its empty
    // MMA steps are left out), which costs shared memory but no traffic, and every block costs a barrier round trip:
    // 80 channels are one block of 128, 224 two, 160 and 192 three of 64.
    {
        int best = 1 << 30;
        for (int bk = 128; bk >= 32; bk /= 2) {
            const int cost = (p->cpad + bk - 1) / bk * (bk + 32);
            if (cost < best) {
                best = cost;
                p->bk = bk;
            }
        }
    }
    const int cchunks = (p->cpad + p->bk - 1) / p->bk;
    const int ones = g.wzp_d ? 16 : 0;      // rows of B and accumulator columns behind a tile's channels (window sums)
    // output-channel tile: a multiple of 16 up to 256 that wastes little of Cout
    {
        const int k16 = (g.k + 15) / 16 * 16;
        const int widest = 256 - ones;
        if (k16 <= widest) {
            p->bn = k16;
        } else {
            int best = widest, best_waste = 1 << 30;
            for (int bn = widest; bn >= 128; bn -= 16) {
                int tiles = (g.k + bn - 1) / bn;
                int waste = tiles * bn - g.k;
                if (waste < best_waste) {
                    best_waste = waste;
                    best = bn;
                }
            }
            p->bn = best;
        }
    }
    // a 1x1 output map (an inner product run as a full-image conv) has one row per image, far too few
    // row tiles to fill the SMs at any usual batch: narrow channel tiles spread the weight matrix over
    // many CTAs instead (2048 -> 1000 at batch 256: 8 CTAs and 0.035 ms at 256 wide, 64 CTAs and < 0.02 ms at 32)
    if (g.oh == 1 && g.ow == 1 && g.k >= 32)
        p->bn = 32;
    if (const char *e = getenv("B200_IGEMM_BN")) {   // tuning aid: channel-tile width, a multiple of 16 up to 256
        int v = atoi(e);
        if (v >= 16 && v <= 256 - ones && v % 16 == 0 && v <= (g.k + 15) / 16 * 16)
            p->bn = v;
    }
    const int n_tiles_n = (g.k + p->bn - 1) / p->bn;
    p->kpad = n_tiles_n * p->bn;
    // pipeline depth from the shared memory left after the staging buffer
    {
        const int kblocks = mma_taps * cchunks;
        // weights resident when there is one channel tile and they leave room for >= 3 A stages
        // four epilogue groups (four tiles in flight behind the mainloop) when the tiles are narrow:
        // their per-tile latency chain, not their arithmetic, sets the epilogue rate
        p->groups = (p->bn <= 64 || (p->bn <= 128 - ones && kblocks * p->bk <= 256)) ? 4 : 2;
        if (const char *e = getenv("B200_IGEMM_GROUPS")) {   // tuning aid: 2, or 4 when four accumulators fit
            int v = atoi(e);
            if (v == 2 || (v == 4 && 4 * (p->bn + ones) <= 512))
                p->groups = v;
        }
        epilogue_segments(p->bn, (kEpiWarps / p->groups) / 4, p->seg_w);
        p->acc_stages = 4 * (p->bn + ones) <= 512 ? 4 : p->groups;
        if (const char *e = getenv("B200_IGEMM_ACC")) {
            int v = atoi(e);
            if ((v == 2 || v == 4) && v * (p->bn + ones) <= 512 && v >= p->groups)
                p->acc_stages = v;
        }
        p->b_resident = n_tiles_n == 1 && smem_layout(3, kblocks, p->bk, p->bn, p->groups, p->bn + ones).total + 1024 <= 227 * 1024;
        // Narrow k-blocks (few bytes per barrier round trip) travel in groups: the largest divisor of
        // the tile's k-blocks that keeps a stage at or under kGroupBytes.
        const int kb_bytes = kTileM * p->bk + (p->b_resident ? 0 : (p->bn + ones) * p->bk);
        int kgroup = 1;
        for (int d = 1; d <= kblocks; ++d)
            if (kblocks % d == 0 && d * kb_bytes <= kGroupBytes && d <= kMaxGroup)
                kgroup = d;
        if (const char *e = getenv("B200_IGEMM_KGROUP")) {   // tuning aid: a divisor of the k-blocks, else ignored
            int v = atoi(e);
            if (v >= 1 && v <= kMaxGroup && kblocks % v == 0)
                kgroup = v;
        }
        int stages = kMaxStages;
        auto fits = [&](int st, int kg) {
            return smem_layout(st * kg, p->b_resident ? kblocks : st * kg, p->bk, p->bn, p->groups, p->bn + ones).total + 1024 <= 227 * 1024;
        };
        while (kgroup > 1 && !fits(3, kgroup)) {   // keep at least three stages in flight
            int d = kgroup - 1;
            while (kblocks % d != 0)
                --d;
            kgroup = d;
        }
        while (stages > 2 && (!fits(stages, kgroup) || stages * kgroup > 32))
            --stages;
        // a deep ring lets the producer run several tiles ahead when a tile has few k-blocks
        // Two pipelines (the kernel's MODE 1) where the k-blocks are short: an MMA of a tile this narrow takes 64 cycles or
        // less, and one producer thread needs ~300 cycles for a k-block (3x3 64-channel layer, 56x56, batch 256: 84 -> 51 us).
        // Tiles of 80 channels and more with a short reduction wait for their epilogue (16 -> 96, 112x112: 110 us, with two 119).
        p->rings = (p->bn <= 128 && (p->bn <= 64 || kblocks * p->bk > 256) && stages >= 4 && !ones) ? 2 : 1;
        if (const char *e = getenv("B200_IGEMM_RINGS")) {   // tuning aid: 1, or 2 when the ring has four stages or more
            int v = atoi(e);
            if (v == 1 || (v == 2 && stages >= 4 && !ones))
                p->rings = v;
        }
        if (p->rings == 2)
            stages &= ~1;
        // Pair mode (see the kernel's MODE 2): wide k-blocks of a layer with one channel tile, where the
        // operand loads from L2 set the pace: two tiles per stage share one weight tile.
        // (3x3 128-channel layer 0.047 -> 0.043 ms.  256-wide tiles lose: their two accumulators fill the
        // tensor memory, so the next pair's mainloop cannot overlap this pair's epilogue: 0.039 -> 0.044 ms.)
        const bool pair_off = getenv("B200_IGEMM_PAIR") && atoi(getenv("B200_IGEMM_PAIR")) == 0;   // tuning aid
        if (!pair_off && !ones && !p->b_resident && kgroup == 1 && !p->a_wide && !quads && n_tiles_n == 1 && p->bn <= 128) {
            int st = kMaxStages;
            auto fits2 = [&](int n) { return smem_layout(2 * n, n, p->bk, p->bn, p->groups).total + 1024 <= 227 * 1024; };
            while (st > 2 && !fits2(st))
                --st;
            if (fits2(st)) {
                p->pair = 1;
                p->rings = 1;
                stages = st;
            }
        }
        // CTA pair (the kernel's MODE 3): two CTAs of a cluster run every MMA together (cta_group::2, M = 256),
        // each loading its own activation tile and half of the weight tile.  A 256-wide MMA of one CTA reads
        // 12 KB of operands from shared memory while TMA writes the next 12 KB into it, which is more than the
        // shared memory moves per MMA time; the pair halves the weight bytes per SM on both sides.  For the
        // layers whose mainloop sets the pace: 256-wide tiles with at least 1 KB of reduction per pixel.
        {
            const char *e = getenv("B200_IGEMM_CTA_PAIR");     // tuning aid: 0 never, 1 wherever possible
            p->pair_want = e ? atoi(e) : -1;
            const bool can = !p->b_resident && !p->a_wide && !quads && !p->pair && p->bn % 32 == 0 && p->bn >= 64 && g.wzp_d == 0;
            const bool automatic = p->bn == 256 && kblocks * p->bk >= 1024;
            if (can && (p->pair_want == 1 || (p->pair_want == -1 && automatic))) {
                auto fits_p = [&](int st, int kg) {
                    return smem_layout(st * kg, st * kg, p->bk, p->bn, p->groups, p->bn / 2).total + 1024 <= 227 * 1024;
                };
                int st = kMaxStages;
                while (st > 2 && (!fits_p(st, kgroup) || st * kgroup > 32))
                    --st;
                if (fits_p(st, kgroup) && p->rings == 1) {
                    p->pair_ok = 1;
                    p->stages_pair = st;
                }
            }
        }
        p->stages = stages;
        p->kgroup = kgroup;
        // One box for all taps.  Tiles of eight by sixteen pixels, or of whole lines where a power of two holds a line
        // and its ring: the shapes whose 32-pixel quarters are boxes of the output.
        const HaloWindow win(g.r, p->taps_w, g.stride_h, g.stride_w, g.pad_h, g.pad_w, quads ? g.s : 0, quads ? p->bk / 16 : 1);
        if (const char *e = getenv("B200_IGEMM_HALO"))      // tuning aid: 0 never, 1 wherever possible
            p->halo_want = atoi(e);
        if (win.fits() && !p->a_wide && n_tiles_n == 1 && g.k % 16 == 0 && (quads || p->halo_want != 0)) {
            int line = 8;
            while (line < g.ow + win.ring_w)
                line *= 2;
            const long long by_cols = (long long)((g.ow + 7) / 8) * ((g.oh + 15) / 16);
            const long long by_lines = line <= kTileM ? (g.oh + kTileM / line - 1) / (kTileM / line) : by_cols + 1;
            for (int form = 0; form < 2 && p->stages_halo == 0; ++form) {      // the one of fewer tiles, or the other if only that fits
                const bool lines = (by_lines <= by_cols) == (form == 0);
                if (lines && line > kTileM)
                    break;
                HaloTiles &h = p->halo;
                memset(&h, 0, sizeof(h));
                h.tw = lines ? line : 8;
                h.th = kTileM / h.tw;
                h.pitch = lines ? line : 8 + win.ring_w;
                p->box_group = lines ? 8 : h.pitch;
                halo_planes(win, p->box_group, &h);
                p->box_bytes = ((uint32_t)(h.span * (quads ? 16 : p->bk)) + 1023u) & ~1023u;
                int st = kMaxStages;
                while (st > 0 && smem_layout(st, kblocks, p->bk, p->bn, p->groups, p->bn + ones, p->box_bytes).total + 1024 > 227 * 1024)
                    --st;
                if (st >= 2)
                    p->stages_halo = st >= 4 ? st & ~1 : st;       // (two pipelines from four on)
            }
        }
    }
    if (quads && !p->stages_halo) {         // (there is no other way to read these pixels)
        delete p;
        return fail(B200_ERR_UNSUPPORTED, "conv(igemm): no box of this image fits shared memory");
    }
    if (!quads && smem_layout((p->pair ? 2 : 1) * p->stages * p->kgroup, p->b_resident ? mma_taps * cchunks : p->stages * p->kgroup, p->bk, p->bn, p->groups, p->bn + ones).total + 1024 > 227 * 1024) {
        delete p;
        return fail(B200_ERR_UNSUPPORTED, "conv(igemm): tile does not fit shared memory");
    }

    const int taps = g.r * g.s;
    // ---- weights [kpad][r][s][c] ---------------------------------------------------------------
    std::vector<int8_t> wp((size_t)p->kpad * mma_taps * p->cpad, 0);
    std::vector<int32_t> wtap((size_t)g.k * taps);       // sum over channels per (k, tap)
    if (quads) {        // [kpad][r][pixels of a row][16]
        std::vector<int8_t> row((size_t)taps * 16);
        for (int k = 0; k < g.k; ++k) {
            weights_to_pitch(&w_s8[(size_t)k * g.c * taps], g.c, taps, row.data(), 16, &wtap[(size_t)k * taps]);
            for (int rr = 0; rr < g.r; ++rr)
                memcpy(&wp[((size_t)k * g.r + rr) * p->cpad], &row[(size_t)rr * g.s * 16], (size_t)g.s * 16);
        }
    } else {
        for (int k = 0; k < g.k; ++k)
            weights_to_pitch(&w_s8[(size_t)k * g.c * taps], g.c, taps, &wp[(size_t)k * taps * p->cpad], p->cpad, &wtap[(size_t)k * taps]);
    }
    // ---- border classes and offsets ---------------------------------------------------------------
    std::vector<uint8_t> row_cls, col_cls;
    std::vector<std::vector<char>> row_valid, col_valid;
    tap_classes(g.oh, g.h, g.r, g.pad_h, g.stride_h, row_cls, row_valid);
    tap_classes(g.ow, g.w, g.s, g.pad_w, g.stride_w, col_cls, col_valid);
    p->n_row_cls = (int)row_valid.size();
    p->n_col_cls = (int)col_valid.size();
    if (p->n_row_cls > 255 || p->n_col_cls > 255) {
        delete p;
        return fail(B200_ERR_UNSUPPORTED, "conv(igemm): too many border classes");
    }
    std::vector<int32_t> off32_all((size_t)p->n_row_cls * p->n_col_cls * p->kpad, 0);
    std::vector<long long> reach(g.k, 0);            // a bound of |accumulator + offset| per channel, whatever the input
    for (int rc = 0; rc < p->n_row_cls; ++rc)
        for (int cc = 0; cc < p->n_col_cls; ++cc)
            for (int k = 0; k < g.k; ++k) {
                long long sum = 0;
                for (int rr = 0; rr < g.r; ++rr)
                    if (row_valid[rc][rr])
                        for (int ss = 0; ss < g.s; ++ss)
                            if (col_valid[cc][ss])
                                sum += wtap[(size_t)k * taps + rr * g.s + ss];
                // int8 activations reach the tensor cores as signed bytes and TMA pads with a true zero: no correction
                long long v = (long long)(bias ? bias[k] : 0) - (long long)(g.act_signed ? 0 : g.izp) * sum;
                if (ones) {
                    // the window-sum column holds the raw bytes: sum (x - izp) over the in-image taps is that less izp for each
                    int taps_in = 0;
                    for (int rr = 0; rr < g.r; ++rr)
                        for (int ss = 0; ss < g.s; ++ss)
                            taps_in += row_valid[rc][rr] && col_valid[cc][ss] ? 1 : 0;
                    v += (long long)g.wzp_d * g.izp * taps_in * (window ? window * 4 : g.c);
                }
                const long long off32 = (long long)(int32_t)(uint32_t)(unsigned long long)v;
                off32_all[((size_t)rc * p->n_col_cls + cc) * p->kpad + k] = (int32_t)off32;
                reach[k] = std::max(reach[k], off32 < 0 ? -off32 : off32);
            }
    for (int k = 0; k < g.k; ++k) {
        const int8_t *row = &w_s8[(size_t)k * g.c * taps];
        int mag = 0;                            // (fits: at most 128 x 32767 k-blocks x 128 channels)
        for (int i = 0; i < g.c * taps; ++i)
            mag += row[i] < 0 ? -row[i] : row[i];
        reach[k] += 255ll * mag + 255ll * (g.wzp_d < 0 ? -g.wzp_d : g.wzp_d) * g.c * taps;
    }
    std::vector<int32_t> shiftp(p->kpad, 33);
    for (int k = 0; k < g.k; ++k) {
        shiftp[k] = shift[k];
    }
    // The form of the epilogue's arithmetic (EpiForm).
    std::vector<int32_t> mulp(p->kpad, 0), off_form = off32_all;
    {
        bool fp = true, uni = true;
        int smin = 127;
        for (int k = 0; k < g.k; ++k) {
            smin = shift[k] < smin ? shift[k] : smin;
            fp = fp && reach[k] < (1 << 22) && ldexp((double)reach[k] * mult[k], -shift[k]) < (double)(1 << 22);
        }
        uni = smin >= 33;
        for (int k = 0; k < g.k && uni; ++k) {
            const int d = shift[k] - smin;
            uni = d <= 7 && (mult[k] & ((1u << d) - 1u)) == 0;
        }
        const char *e = getenv("B200_IGEMM_EPI");       // tuning aid: 1 no fp32, 2 neither fp32 nor uniform shift
        const int least = e ? atoi(e) : 0;
        p->form = fp && least < 1 ? kEpiFp : uni && least < 2 ? kEpiInt : kEpiGeneric;
        const int full = g.act_signed || g.qmax != 255 ? 1 : 0, many = p->n_row_cls * p->n_col_cls > 1 ? 2 : 0;
        p->variant = p->form == kEpiGeneric ? kEpiAny : (p->form == kEpiFp ? kEpiFpOne : kEpiIntOne) + many + full;
        if (p->form == kEpiInt) {
            p->ushift = smin - 32;
            p->rnd_hi = (int)((1ll << (smin - 33)) + ((long long)g.ozp << (smin - 32)));
        }
        for (int k = 0; k < g.k; ++k) {
            if (p->form == kEpiFp) {
                const float m = ldexpf((float)mult[k], -shift[k]);      // exact: 24 significant bits
                memcpy(&mulp[k], &m, 4);
            } else {
                mulp[k] = (int32_t)(p->form == kEpiInt ? mult[k] >> (shift[k] - smin) : mult[k]);
            }
        }
        if (p->form == kEpiFp)
            for (int32_t &o : off_form)
                o += kFpMagic;
    }
    if (p->pair_ok && !igemm_kernel_mode3(p->variant))      // built for long reductions only
        p->pair_ok = 0;
    std::vector<int8_t> one_row;
    if (ones) {
        one_row.assign((size_t)16 * taps * p->cpad, 0);
        for (int t = 0; t < taps; ++t)
            for (int c = 0; c < (window ? window * 4 : g.c); ++c)
                one_row[(size_t)t * p->cpad + c] = 1;
    }
    p->w_bytes = wp.size();
    // one device block for the weights and all tables: an allocation and a copy each cost more than the small tables hold
    struct { const void *src; size_t bytes; void **dst; } parts[] = {
        { wp.data(), wp.size(), (void **)&p->w_dev },
        { one_row.data(), one_row.size(), (void **)&p->ones_dev },
        { mulp.data(), mulp.size() * 4, (void **)&p->mul_form_dev },
        { off_form.data(), p->form == kEpiFp ? off_form.size() * 4 : 0, (void **)&p->off_form_dev },
        { off32_all.data(), off32_all.size() * 4, (void **)&p->off32_dev },
        { shiftp.data(), shiftp.size() * 4, (void **)&p->shift_dev },
        { row_cls.data(), row_cls.size(), (void **)&p->row_cls_dev },
        { col_cls.data(), col_cls.size(), (void **)&p->col_cls_dev },
    };
    size_t small = 0;       // what goes behind the weights
    for (auto &q : parts)
        small += q.src == wp.data() ? 0 : (q.bytes + 255) / 256 * 256;
    const size_t behind = (wp.size() + 255) / 256 * 256;
    // copied together, small weights with them: a copy costs what moving 50 KB on the host does
    const size_t lead = wp.size() <= (64u << 10) ? behind : 0;
    std::vector<uint8_t> tables(lead + small);
    auto upload_all = [&]() -> int {
        B200_CUDA_TRY(cudaMalloc((void **)&p->block_dev, behind + small));
        size_t at = 0;
        for (auto &q : parts) {
            if (q.src == wp.data()) {
                *q.dst = p->block_dev;
                if (lead != 0)
                    memcpy(tables.data(), wp.data(), wp.size());
                continue;
            }
            if (q.bytes == 0)
                continue;
            memcpy(&tables[lead + at], q.src, q.bytes);
            *q.dst = p->block_dev + behind + at;
            at += (q.bytes + 255) / 256 * 256;
        }
        if (lead == 0)
            B200_CUDA_TRY(cudaMemcpy(p->block_dev, wp.data(), wp.size(), cudaMemcpyHostToDevice));
        B200_CUDA_TRY(cudaMemcpy(p->block_dev + behind - lead, tables.data(), lead + at, cudaMemcpyHostToDevice));
        return B200_OK;
    };
    const int rc = upload_all();
    if (rc != B200_OK) {
        conv_igemm_destroy(p);
        return rc;
    }
    *out = p;
    return B200_OK;
}

void conv_igemm_destroy(ConvIgemmPlan *p)
{
    if (!p)
        return;
    cudaFree(p->block_dev);
    delete p;
}

// Chooses the M-tile box (tw, th, tn), powers of two with product 128, that covers the output with
// the fewest tiles; ties go to the wider box.
static void choose_tile(int ow, int oh, int n, int *tw, int *th, int *tn, int min_a = 0, int max_a = 7)
{
    long long best = -1;
    for (int a = min_a; a <= max_a; ++a)
        for (int b = 0; a + b <= 7; ++b) {
            int w = 1 << a, h = 1 << b, nn = 1 << (7 - a - b);
            long long tiles = (long long)((ow + w - 1) / w) * ((oh + h - 1) / h) * ((n + nn - 1) / nn);
            if (best < 0 || tiles < best || (tiles == best && w > *tw)) {
                best = tiles;
                *tw = w;
                *th = h;
                *tn = nn;
            }
        }
}

void conv_igemm_describe(const ConvIgemmPlan *p, char *buf, size_t len)
{
    const ConvIgemmPlan::Launch *l = p->last_launch();      // the tiling depends on the batch of the run
    auto prefetch = [&](uint32_t bytes) {
        const size_t used = strlen(buf);
        if (bytes != 0)
            snprintf(buf + used, len - used, ", prefetches %u bytes", bytes);
    };
    if (l && l->small) {
        snprintf(buf, len, "tcgen05 igemm: bn=%d bk=%d slots=%d split=%d one tile per %s", l->sargs.bn, p->bk, l->sargs.slots, l->sargs.split,
                 l->sargs.split > 1 ? "cluster" : "CTA");
        prefetch(l->sargs.next_ro_bytes);
        return;
    }
    const bool cta_pair = l && l->cta_pair;
    const char *mode = l && l->halo ? "one box for all taps" : cta_pair ? "cta-pair (cta_group::2, M=256)" : p->pair ? "tile pairs on one weight tile"
        : p->pair_ok ? "tile by tile (cta pairs on long launches)"
        : p->rings == 2 ? "two pipelines" : "tile by tile";
    snprintf(buf, len, "tcgen05 igemm: bn=%d bk=%d stages=%d kgroup=%d groups=%d acc_stages=%d %s%s%s%s", p->bn, p->bk,
             l ? l->args.stages : p->stages, l ? l->args.kgroup : p->kgroup, p->groups, p->acc_stages, mode, (l ? l->args.b_resident : p->b_resident) ? ", weights resident" : "",
             p->form == kEpiFp ? ", fp32 epilogue" : p->form == kEpiInt ? ", uniform-shift epilogue" : ", generic requantize",
             p->rev ? ", reversed" : "");
    if (l)
        prefetch(l->args.next_ro_bytes);
}

void conv_igemm_set_reverse(ConvIgemmPlan *p, int reverse)
{
    if (p->rev != (reverse ? 1 : 0)) {
        p->rev = reverse ? 1 : 0;
        p->saved.clear();      // they carry the old direction
    }
}

void conv_igemm_weights(const ConvIgemmPlan *p, const uint8_t **ptr, size_t *bytes)
{
    *ptr = reinterpret_cast<const uint8_t *>(p->w_dev);
    *bytes = p->w_bytes;
}

void conv_igemm_set_next_readonly(ConvIgemmPlan *p, const NextRead &next)
{
    p->next = next;
    p->saved.clear();
}

// The bulk prefetch of a launch of n images, in its unit of 16 bytes; more than 64 MiB would only evict what the layers between need.
static void next_read(const ConvIgemmPlan *p, int n, const uint8_t **ptr, uint32_t *bytes)
{
    const bool grouped = n >= p->next.from && n <= p->next.to;
    const uint8_t *w = grouped ? p->next.grouped : p->next.plain;
    const size_t size = grouped ? p->next.grouped_bytes : p->next.plain_bytes;
    const bool fits = w && ((uintptr_t)w & 15) == 0 && size <= (64u << 20);
    *ptr = fits ? w : nullptr;
    *bytes = fits ? (uint32_t)(size & ~(size_t)15) : 0u;
}

int conv_igemm_set_residual(ConvIgemmPlan *p, const EltwiseArgs &e, int conv_input)
{
    // the fused form exists for the straight-line epilogue only: high-word requantize, 8-bit output,
    // whole 32-channel chunks stored through TMA
    if (p->form == kEpiGeneric || p->g.qmax != 255 || p->g.k % 32 != 0 || p->bn % 32 != 0)
        return fail(B200_ERR_UNSUPPORTED, "conv(igemm): residual add needs the fast requantize form and Cout %% 32 == 0");
    p->pair_ok = 0;     // the kernel variant with the residual add runs one CTA per tile
    if (e.n_in != 2 || e.qmax != 255 || conv_input < 0 || conv_input > 1)
        return fail(B200_ERR_UNSUPPORTED, "conv(igemm): residual add takes a two-input, 8-bit eltwise SUM");
    const int other = 1 - conv_input;
    p->r_m[0] = e.m[conv_input]; p->r_add[0] = e.add[conv_input]; p->r_b[0] = e.b[conv_input];
    p->r_m[1] = e.m[other]; p->r_add[1] = e.add[other]; p->r_b[1] = e.b[other];
    p->r_s0 = e.s0; p->r_ozp = e.ozp; p->r_lo = e.relu_lo;
    p->has_res = true;
    p->saved.clear();      // they carry the old constants
    return B200_OK;
}

// Tensor maps of the activations for M tiles of tw x th x tn pixels.
static int encode_activations(const ConvIgemmPlan *p, const uint8_t *x, int n, int tw, int th, int tn, CUtensorMap (&maps)[4])
{
    const ConvGeom &g = p->g;
    for (int ph = 0; ph < g.stride_h; ++ph)
        for (int pw = 0; pw < g.stride_w; ++pw) {
            // input pixels (ph + stride_h * i, pw + stride_w * j): a dense 4-D tensor (c, j, i, image)
            if (ph >= g.h || pw >= g.w) {
                maps[ph * 2 + pw] = maps[0];
                continue;
            }
            if (p->a_wide) {
                // rows of this parity as a 3-D tensor (ow * 32 bytes in 8-byte elements, row, image);
                // no swizzle: the bytes are already laid out as the MMA's 32-byte swizzle wants them
                cuuint64_t dims[3] = { (cuuint64_t)g.w * 4, (cuuint64_t)((g.h - ph + g.stride_h - 1) / g.stride_h), (cuuint64_t)n };
                cuuint64_t strides[2] = { (cuuint64_t)g.stride_h * g.w * 32, (cuuint64_t)g.h * g.w * 32 };
                cuuint32_t box[3] = { (cuuint32_t)tw * 4, (cuuint32_t)th, (cuuint32_t)tn };
                void *base = (void *)(x + (size_t)ph * g.w * 32);
                B200_TRY(encode(&maps[ph * 2 + pw], base, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_DATA_TYPE_UINT64));
                continue;
            }
            cuuint64_t dims[4] = { (cuuint64_t)g.c, (cuuint64_t)((g.w - pw + g.stride_w - 1) / g.stride_w),
                                   (cuuint64_t)((g.h - ph + g.stride_h - 1) / g.stride_h), (cuuint64_t)n };
            cuuint64_t strides[3] = { (cuuint64_t)g.stride_w * g.c, (cuuint64_t)g.stride_h * g.w * g.c,
                                      (cuuint64_t)g.h * g.w * g.c };
            cuuint32_t box[4] = { (cuuint32_t)p->bk, (cuuint32_t)tw, (cuuint32_t)th, (cuuint32_t)tn };
            void *base = (void *)(x + ((size_t)ph * g.w + pw) * g.c);
            B200_TRY(encode(&maps[ph * 2 + pw], base, 4, dims, strides, box, swizzle_for(p->bk)));
        }
    for (int i = 0; i < 4; ++i)
        if (i / 2 >= g.stride_h || i % 2 >= g.stride_w)
            maps[i] = maps[0];
    return B200_OK;
}

// Per axis: the least and the largest offset, in pixels of the parity, of the taps of one parity; false where there is none.
static bool tap_span(int kernel, int stride, int pad, int parity, int *lo, int *hi)
{
    *lo = 1 << 20;
    *hi = -(1 << 20);
    for (int t = 0; t < kernel; ++t) {
        const int d = t - pad, p = d & (stride - 1), o = (d - p) / stride;
        if (p == parity) {
            *lo = o < *lo ? o : *lo;
            *hi = o > *hi ? o : *hi;
        }
    }
    return *lo <= *hi;
}

HaloWindow::HaloWindow(int r_, int s_, int stride_h_, int stride_w_, int pad_h_, int pad_w_, int row_pixels, int width_)
    : r(r_), s(s_), stride_h(stride_h_), stride_w(stride_w_), pad_h(pad_h_), pad_w(pad_w_), width(width_)
{
    int lo, hi;
    for (int p = 0; p < stride_h; ++p)
        if (tap_span(r, stride_h, pad_h, p, &lo, &hi) && hi - lo > ring_h)
            ring_h = hi - lo;
    ring_w = row_pixels > 0 ? row_pixels - 1 : s - 1;
}

void halo_planes(const HaloWindow &win, int group, HaloTiles *out)
{
    HaloTiles &h = *out;
    h.planes = 0;
    h.span = 0;
    h.tap_row = win.stride_h * win.s;
    h.taps_w = win.s;
    h.col_parity = (uint8_t)(win.pad_w & (win.stride_w - 1));
    int x1;
    tap_span(win.s, win.stride_w, win.pad_w, h.col_parity, &h.dx, &x1);
    for (int ph = 0; ph < win.stride_h; ++ph) {
        int y0, y1, r0 = 0;
        if (!tap_span(win.r, win.stride_h, win.pad_h, ph, &y0, &y1))
            continue;
        while (((r0 - win.pad_h) & (win.stride_h - 1)) != ph)       // the first tap of this parity; the others follow a stride apart
            ++r0;
        const int pl = h.planes++;
        h.dy[pl] = y0;
        h.rows[pl] = h.pitch * (h.th + y1 - y0);
        h.row_parity[pl] = (uint8_t)ph;
        h.taps_h[pl] = (win.r - r0 + win.stride_h - 1) / win.stride_h;
        h.tap0[pl] = r0 * win.s;
        // an operand is sixteen groups of eight rows from its first one on (of `width` pixels each)
        const int last = (h.taps_h[pl] - 1) * h.pitch + h.taps_w - 1;
        h.span = std::max(h.span, std::max(h.rows[pl], last + 15 * group + 8 + win.width - 1));
    }
}

// The same for the boxes of HaloTiles, a map per plane.
static int encode_boxes(const ConvIgemmPlan *p, const uint8_t *x, int n, const HaloTiles &h, CUtensorMap (&maps)[4])
{
    const ConvGeom &g = p->g;
    for (int i = 0; i < h.planes; ++i) {
        const int ph = h.row_parity[i], pw = h.col_parity;
        if (p->quads) {         // whole lines of the image, in 8-byte elements
            cuuint64_t dims[3] = { (cuuint64_t)g.w * 2, (cuuint64_t)((g.h - ph + g.stride_h - 1) / g.stride_h), (cuuint64_t)n };
            cuuint64_t strides[2] = { (cuuint64_t)g.stride_h * g.w * 16, (cuuint64_t)g.h * g.w * 16 };
            cuuint32_t box[3] = { (cuuint32_t)h.pitch * 2, (cuuint32_t)(h.rows[i] / h.pitch), 1 };
            B200_TRY(encode(&maps[i], (void *)(x + (size_t)ph * g.w * 16), 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_DATA_TYPE_UINT64));
            continue;
        }
        cuuint64_t dims[4] = { (cuuint64_t)g.c, (cuuint64_t)((g.w - pw + g.stride_w - 1) / g.stride_w),
                               (cuuint64_t)((g.h - ph + g.stride_h - 1) / g.stride_h), (cuuint64_t)n };
        cuuint64_t strides[3] = { (cuuint64_t)g.stride_w * g.c, (cuuint64_t)g.stride_h * g.w * g.c, (cuuint64_t)g.h * g.w * g.c };
        cuuint32_t box[4] = { (cuuint32_t)p->bk, (cuuint32_t)h.pitch, (cuuint32_t)(h.rows[i] / h.pitch), 1 };
        B200_TRY(encode(&maps[i], (void *)(x + ((size_t)ph * g.w + pw) * g.c), 4, dims, strides, box, swizzle_for(p->bk)));
    }
    for (int i = h.planes; i < 4; ++i)
        maps[i] = maps[0];
    return B200_OK;
}

// Tensor map of [rows][r*s*c] weights in boxes of `box_rows` rows and one k-block.
// frag: the row order of the fragment epilogue (frag_segment): row 8 j + 2 q + e of every sixteen is channel 4 q + 2 j + e.
static int encode_weights(const ConvIgemmPlan *p, const int8_t *w, int rows, int box_rows, CUtensorMap *map, bool frag = false)
{
    const int ktot = p->g.r * p->taps_w * p->cpad;
    if (frag) {
        cuuint64_t dims[5] = { (cuuint64_t)ktot, 2, 4, 2, (cuuint64_t)(rows / 16) };
        cuuint64_t strides[4] = { (cuuint64_t)ktot, 4 * (cuuint64_t)ktot, 2 * (cuuint64_t)ktot, 16 * (cuuint64_t)ktot };
        cuuint32_t box[5] = { (cuuint32_t)p->bk, 2, 4, 2, (cuuint32_t)(box_rows / 16) };
        return encode(map, const_cast<int8_t *>(w), 5, dims, strides, box, swizzle_for(p->bk));
    }
    cuuint64_t dims[2] = { (cuuint64_t)ktot, (cuuint64_t)rows };
    cuuint64_t strides[1] = { (cuuint64_t)ktot };
    cuuint32_t box[2] = { (cuuint32_t)p->bk, (cuuint32_t)box_rows };
    return encode(map, const_cast<int8_t *>(w), 2, dims, strides, box, swizzle_for(p->bk));
}

// Fills l.smaps / l.sargs if the launch is one for conv_small_kernel; l.small says so.
static int build_small(ConvIgemmPlan *p, const uint8_t *x, int n, uint8_t *y, int *status, int tw, int th, int tn, const ConvSum *ws, ConvIgemmPlan::Launch &l)
{
    const ConvGeom &g = p->g;
    SmallArgs &a = l.sargs;
    memset(&a, 0, sizeof(a));
    a.tiles_w = (g.ow + tw - 1) / tw;
    a.tiles_h = (g.oh + th - 1) / th;
    const int m_tiles = a.tiles_w * a.tiles_h * ((n + tn - 1) / tn);
    a.cchunks = (p->cpad + p->bk - 1) / p->bk;
    a.cpad = p->cpad;
    a.last_steps = (p->cpad - (a.cchunks - 1) * p->bk) / 32;
    a.kblocks = g.r * g.s * a.cchunks;
    a.bk = p->bk;
    if (p->small_bn && p->small_split <= a.kblocks) {              // tuning aid
        a.bn = p->small_bn;
        a.split = p->small_split;
    } else if (!conv_small_pick(m_tiles, g.k, a.kblocks, a.bk, g.wzp_d != 0, p->bn, &a.bn, &a.split)) {
        return B200_OK;
    }
    a.n = n; a.oh = g.oh; a.ow = g.ow; a.cout = g.k;
    a.r = g.r; a.s = g.s; a.pad_h = g.pad_h; a.pad_w = g.pad_w; a.stride_h = g.stride_h; a.stride_w = g.stride_w;
    for (a.tw_sh = 0; (1 << a.tw_sh) < tw; ++a.tw_sh) {}
    for (a.th_sh = 0; (1 << a.th_sh) < th; ++a.th_sh) {}
    a.tn = tn;
    a.n_tiles_n = (g.k + a.bn - 1) / a.bn;
    a.a_wide = p->a_wide;
    a.form = p->form;
    a.off32 = p->off_form_dev ? p->off_form_dev : p->off32_dev; a.mul = p->mul_form_dev; a.shift = p->shift_dev;
    a.ushift = p->ushift; a.rnd_hi = p->rnd_hi;
    a.row_cls = p->row_cls_dev; a.col_cls = p->col_cls_dev;
    a.n_col_cls = p->n_col_cls; a.n_cls = p->n_row_cls * p->n_col_cls; a.kpad = p->kpad;
    a.ozp = g.ozp; a.qmax = g.qmax; a.relu_lo = g.relu_lo; a.out_flip = g.act_signed ? 0x80808080u : 0u;
    a.wzp_d = g.wzp_d;
    a.y = y;
    a.status = status;
    next_read(p, n, &a.next_ro, &a.next_ro_bytes);
    if (ws && g.k % 16 == 0 && !g.act_signed) {         // (other channel counts leave through staged rows)
        const int ci = ws->conv_input, other = 1 - ci;
        const EltwiseArgs &e = *ws->elt;
        a.res = ws->res;
        a.sum = ws->sum;
        a.r_m[0] = e.m[ci]; a.r_add[0] = e.add[ci]; a.r_b[0] = e.b[ci];
        a.r_m[1] = e.m[other]; a.r_add[1] = e.add[other]; a.r_b[1] = e.b[other];
        a.r_s0 = e.s0; a.r_ozp = e.ozp; a.r_lo = e.relu_lo;
        l.summed = true;
    }
    const size_t smem = conv_small_smem(a, g.act_signed != 0);
    if (smem > 227 * 1024)
        return B200_OK;
    B200_TRY(encode_activations(p, x, n, tw, th, tn, l.smaps.a));
    B200_TRY(encode_weights(p, p->w_dev, p->kpad, a.bn, &l.smaps.b));
    l.smaps.ones = l.smaps.b;
    if (p->ones_dev)
        B200_TRY(encode_weights(p, p->ones_dev, 16, 16, &l.smaps.ones));
    l.smem = smem;
    l.m_tiles = m_tiles;
    l.small = true;
    return B200_OK;
}

static int build_launch(ConvIgemmPlan *p, const uint8_t *x, int n, uint8_t *y, int *status_word, const uint8_t *res, const ConvSum *ws, ConvIgemmPlan::Launch &l)
{
    const ConvGeom &g = p->g;
    if ((((uintptr_t)x | (uintptr_t)y) & 15) != 0)
        return fail(B200_ERR_INVALID, "conv(igemm): x and y must be 16-byte aligned");
    l.x = x; l.res = res; l.y = y; l.n = n; l.status = status_word;
    l.sum_res = ws ? ws->res : nullptr; l.sum = ws ? ws->sum : nullptr; l.summed = false;
    l.small = false;
    l.cta_pair = 0;
    l.halo = false;
    IgemmBoxArgs &a = l.args;
    memset(&a, 0, sizeof(a));
    if (status_word)
        a.status = status_word;       // caller-provided word (the allocation-free entry point)
    else
        B200_TRY(status_word_ptr(&a.status));
    a.n = n; a.oh = g.oh; a.ow = g.ow; a.cout = g.k;
    a.r = g.r; a.s = p->taps_w; a.pad_h = g.pad_h; a.pad_w = g.pad_w; a.stride_h = g.stride_h; a.stride_w = g.stride_w;
    a.c = p->cpad;
    if (p->a_wide)   // whole swizzle atoms (8 pixels) per row segment, at most 256 8-byte elements
        choose_tile(g.ow, g.oh, n, &a.tw, &a.th, &a.tn, 3, 6);
    else
        choose_tile(g.ow, g.oh, n, &a.tw, &a.th, &a.tn);
    a.tiles_w = (g.ow + a.tw - 1) / a.tw;
    a.tiles_h = (g.oh + a.th - 1) / a.th;
    a.tiles_n = (n + a.tn - 1) / a.tn;
    a.n_tiles_n = p->kpad / p->bn;
    const int sms = sm_count();
    if (!p->attr_set) {
        B200_TRY(conv_igemm_warm());
        p->attr_set = true;
    }
    if (!res && p->small_ok && !p->quads && !(p->pair_ok && p->pair_want == 1)) {
        B200_TRY(build_small(p, x, n, y, a.status, a.tw, a.th, a.tn, ws, l));
        if (l.small)
            return B200_OK;
    }
    if (p->pair_ok) {
        if (p->max_clusters == 0) {
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
            cfg.gridDim = dim3((unsigned)(sms & ~1));
            cfg.blockDim = dim3(kThreads);
            cfg.dynamicSmemBytes = smem_layout(p->stages_pair * p->kgroup, p->stages_pair * p->kgroup, p->bk, p->bn, p->groups, p->bn / 2).total + 1024;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            int nc = 0;
            if (cudaOccupancyMaxActiveClusters(&nc, igemm_kernel_mode3(p->variant), &cfg) != cudaSuccess || nc < 1) {
                cudaGetLastError();
                nc = sms / 2;
            }
            p->max_clusters = nc < sms / 2 ? nc : sms / 2;
        }
        const int pair_tiles = (a.tiles_w * a.tiles_h * a.tiles_n + 1) / 2 * (p->kpad / p->bn);
        // a pair tile for every cluster at least (one buffer, queued: 3x3 256 -> 256, 14x14, batch 256: 26.5 -> 25.8 us; 3x3 s2
        // 512 -> 512: 34.1 -> 31.1)
        l.cta_pair = (p->pair_want == 1 || pair_tiles >= p->max_clusters) ? 1 : 0;
    }
    if (p->stages_halo && !res && !l.cta_pair) {
        const HaloTiles &h = p->halo;
        const long long boxes = (long long)((g.ow + h.tw - 1) / h.tw) * ((g.oh + h.th - 1) / h.th) * n;
        // Windows of stride 1, whose taps all share one box.  What the tiles waste beside the image decides: they hold one image's
        // pixels, and lines end in them.  Up to a fifth the box wins 4 .. 50 % (64 -> 64 on 56 x 56, batch 64: 16.6 -> 15.8 us, 32 -> 64 on 112 x 112:
        // 48.7 -> 36.6, 96 -> 96 on 40 x 40: 18.3 -> 14.9); with k-blocks of 128 channels up to a third (128 -> 128 on 14 x 14, batch 256:
        // 12.4 -> 11.5; 64 -> 64 there 8.04 -> 7.84, on 27 x 35 11.7 -> 12.7), and up to a half where a window-sum column leaves one pipeline
        // to a box per tap (24.6 -> 16.3; on 14 x 14 10.1 -> 8.2).  Tiles of more than 128 channels wait for their epilogue (32 -> 256 on 30 x 30:
        // 13.8 -> 14.9); with a stride a box holds few taps (64 -> 128, stride 2: 9.8 -> 10.8).
        const long long tiles = (long long)a.tiles_w * a.tiles_h * a.tiles_n;
        l.halo = p->quads || p->halo_want == 1
            || (h.planes == 1 && (p->bn <= 128 || g.wzp_d != 0) && boxes * 100 <= tiles * (g.wzp_d != 0 ? 150 : p->bk == 128 ? 133 : 120));
        if (l.halo) {
            a.tw = h.tw; a.th = h.th; a.tn = 1;
            a.tiles_w = (g.ow + a.tw - 1) / a.tw;
            a.tiles_h = (g.oh + a.th - 1) / a.th;
            a.tiles_n = n;
            a.halo = h;
            a.box_bytes = p->box_bytes;
            a.box_group = p->box_group;
            a.quads = p->quads;
            a.a_pitch = p->quads ? 16 : p->bk;
        }
    }
    a.bk = p->bk; a.bn = p->bn; a.stages = l.cta_pair ? p->stages_pair : p->stages; a.kgroup = p->kgroup; a.groups = p->groups; a.acc_stages = p->acc_stages;
    a.cchunks = (p->cpad + p->bk - 1) / p->bk;
    a.last_steps = (p->cpad - (a.cchunks - 1) * p->bk) / 32;
    a.b_resident = p->b_resident; a.a_wide = p->a_wide;
    for (a.tw_sh = 0; (1 << a.tw_sh) < a.tw; ++a.tw_sh) {}
    for (a.th_sh = 0; (1 << a.th_sh) < a.th; ++a.th_sh) {}
    // instruction descriptor: D = S32 (2 at bit 4), A = unsigned 8-bit (0 at bit 7), B = signed 8-bit
    // (1 at bit 10), both K-major, N >> 3 at bit 17, M >> 4 at bit 24
    a.idesc = (2u << 4) | ((g.act_signed ? 1u : 0u) << 7) | (1u << 10) | ((uint32_t)((p->bn + (g.wzp_d ? 16 : 0)) >> 3) << 17)
        | ((uint32_t)((l.cta_pair ? 2 * kTileM : kTileM) >> 4) << 24);
    uint32_t cols = 32;
    const int ones = g.wzp_d ? 16 : 0;       // accumulator columns behind the channels
    while (cols < (uint32_t)(p->acc_stages * (p->bn + ones)))
        cols <<= 1;
    a.tmem_cols = cols;
    a.off32 = p->off_form_dev ? p->off_form_dev : p->off32_dev; a.mul = p->mul_form_dev; a.shift = p->shift_dev;
    a.seg_w[0] = p->seg_w[0]; a.seg_w[1] = p->seg_w[1];
    a.ushift = p->ushift; a.rnd_hi = p->rnd_hi;
    a.row_cls = p->row_cls_dev; a.col_cls = p->col_cls_dev;
    a.n_col_cls = p->n_col_cls; a.n_cls = p->n_row_cls * p->n_col_cls; a.kpad = p->kpad;
    a.ozp = g.ozp; a.qmax = g.qmax; a.relu_lo = g.relu_lo;
    a.out_flip = g.act_signed ? 0x80808080u : 0u;
    a.rev = p->rev;
    next_read(p, n, &a.next_ro, &a.next_ro_bytes);
    a.use_tma_store = (g.k % 16 == 0) ? 1 : 0;
    a.y = y;
    a.res = res;
    for (int i = 0; i < 2; ++i) {
        a.r_m[i] = p->r_m[i]; a.r_add[i] = p->r_add[i]; a.r_b[i] = p->r_b[i];
    }
    a.r_s0 = p->r_s0; a.r_ozp = p->r_ozp; a.r_lo = p->r_lo;
    a.wzp_d = g.wzp_d;

    // ---- tensor maps -------------------------------------------------------------------------------
    if (l.halo)
        B200_TRY(encode_boxes(p, x, n, p->halo, l.maps.a));
    else
        B200_TRY(encode_activations(p, x, n, a.tw, a.th, a.tn, l.maps.a));
    const bool frag = !res && !g.wzp_d && p->n_row_cls * p->n_col_cls == 1 && p->variant != kEpiAny;   // as the kernel's `frag`
    B200_TRY(encode_weights(p, p->w_dev, p->kpad, l.cta_pair ? p->bn / 2 : p->bn, &l.maps.b, frag));   // a CTA of a pair loads half the rows
    l.maps.ones = l.maps.b;
    if (p->ones_dev)
        B200_TRY(encode_weights(p, p->ones_dev, 16, 16, &l.maps.ones));
    if (a.use_tma_store) {
        cuuint64_t dims[4] = { (cuuint64_t)g.k, (cuuint64_t)g.ow, (cuuint64_t)g.oh, (cuuint64_t)n };
        cuuint64_t strides[3] = { (cuuint64_t)g.k, (cuuint64_t)g.ow * g.k, (cuuint64_t)g.oh * g.ow * g.k };
        // one store covers the 32 pixels of a tensor-memory lane quarter: a sub-box of the tile
        cuuint32_t qw = a.tw >= 32 ? 32 : a.tw;
        cuuint32_t qh = a.tw >= 32 ? 1 : (a.tw * a.th >= 32 ? 32 / a.tw : a.th);
        cuuint32_t qn = a.tw * a.th >= 32 ? 1 : 32 / (a.tw * a.th);
        for (int i = 0; i < 2; ++i) {
            const int w = p->seg_w[i] ? p->seg_w[i] : p->seg_w[0];
            cuuint32_t box[4] = { (cuuint32_t)w, qw, qh, qn };
            B200_TRY(encode(&l.maps.y[i], y, 4, dims, strides, box, swizzle_for(w)));
        }
    } else {
        l.maps.y[0] = l.maps.y[1] = l.maps.b;
    }
    if (l.halo) {
        a.stages = p->stages_halo;
        a.kgroup = 1;
        a.b_resident = 1;
    }
    l.box_kernel = !l.halo ? nullptr : (a.stages >= 4 ? igemm_kernel_mode5 : igemm_kernel_mode4)(p->variant, g.wzp_d != 0);
    l.kernel = res ? igemm_kernel_residual(p->variant)
        : g.wzp_d ? igemm_kernel_wzp(p->variant)
        : l.cta_pair ? igemm_kernel_mode3(p->variant)
        : p->pair ? igemm_kernel_mode2(p->variant)
        : !a.use_tma_store ? igemm_kernel_ragged(p->variant, p->rings == 2)
        : p->rings == 2 ? igemm_kernel_mode1(p->variant) : igemm_kernel_mode0(p->variant);
    if (!l.kernel && !l.box_kernel)
        return fail(B200_ERR_UNSUPPORTED, "conv(igemm): no kernel of epilogue variant %d for this launch", p->variant);
    const int total_tiles = a.tiles_w * a.tiles_h * a.tiles_n * a.n_tiles_n;
    l.grid = dim3((unsigned)(total_tiles < sms ? total_tiles : sms));
    l.smem = smem_layout((p->pair ? 2 : 1) * a.stages * p->kgroup, p->b_resident ? g.r * p->taps_w * a.cchunks : a.stages * p->kgroup, p->bk, p->bn, p->groups,
                         l.cta_pair ? p->bn / 2 : p->bn + ones).total + 1024;
    if (l.halo)
        l.smem = smem_layout(a.stages, g.r * p->taps_w * a.cchunks, p->bk, p->bn, p->groups, p->bn + ones, p->box_bytes).total + 1024;
    if (l.cta_pair) {
        // pair tiles (two neighbouring M tiles, one channel tile) over the CTA pairs that fit the device at once
        a.pm_tiles = (a.tiles_w * a.tiles_h * a.tiles_n + 1) / 2;
        const int pair_tiles = a.pm_tiles * a.n_tiles_n;
        const int clusters = pair_tiles < p->max_clusters ? pair_tiles : p->max_clusters;
        l.grid = dim3((unsigned)(2 * clusters));
        a.step_nt = clusters % a.n_tiles_n;
        a.step_pm = clusters / a.n_tiles_n;
    } else
    {
        int gsz = (int)l.grid.x;
        a.step_nt = gsz % a.n_tiles_n;
        gsz /= a.n_tiles_n;
        a.step_w = gsz % a.tiles_w;
        gsz /= a.tiles_w;
        a.step_h = gsz % a.tiles_h;
        a.step_n = gsz / a.tiles_h;
    }
    return B200_OK;
}

int conv_igemm_launch(ConvIgemmPlan *p, const uint8_t *x, int n, uint8_t *y, cudaStream_t st, int *status_word, const uint8_t *res,
                      const ConvSum *with_sum, bool *summed)
{
    if (summed)
        *summed = false;
    if (n == 0)
        return B200_OK;
    if (p->g.wzp_d != 0 && res != nullptr)
        return fail(B200_ERR_UNSUPPORTED, "conv(igemm): a fused residual add and a weight zero point other than 128 do not combine");
    if (res != nullptr && !p->has_res)
        return fail(B200_ERR_INVALID, "conv(igemm): a residual tensor was given but no residual add is set");
    if (res == nullptr && p->has_res)
        return fail(B200_ERR_INVALID, "conv(igemm): this conv was fused with a residual add and needs the residual tensor");
    if (res != nullptr && (((uintptr_t)res) & 15) != 0)
        return fail(B200_ERR_INVALID, "conv(igemm): the residual tensor must be 16-byte aligned");
    auto matches = [&](const ConvIgemmPlan::Launch &l) { return l.x == x && l.y == y && l.n == n && l.status == status_word && l.res == res
               && l.sum_res == (with_sum ? with_sum->res : nullptr) && l.sum == (with_sum ? with_sum->sum : nullptr); };
    if (p->last >= p->saved.size() || !matches(p->saved[p->last])) {
        size_t i = 0;
        while (i < p->saved.size() && !matches(p->saved[i]))
            ++i;
        if (i == p->saved.size()) {
            ConvIgemmPlan::Launch l;
            B200_TRY(build_launch(p, x, n, y, status_word, res, with_sum, l));
            if (p->saved.size() < ConvIgemmPlan::kMaxSaved) {
                p->saved.push_back(l);
            } else {
                i = p->next_saved;
                p->saved[i] = l;
                p->next_saved = (i + 1) % ConvIgemmPlan::kMaxSaved;
            }
        }
        p->last = i;
    }
    const ConvIgemmPlan::Launch &l = p->saved[p->last];
    const size_t bytes = (size_t)n * ((size_t)p->g.h * p->g.w * p->g.c + (size_t)p->g.oh * p->g.ow * p->g.k) + p->w_bytes;
    if (summed)
        *summed = l.small && l.summed;
    if (l.small)
        return conv_small_launch(l.smaps, l.sargs, l.m_tiles, l.smem, bytes, st);
    const bool two_rings = l.halo ? l.args.stages >= 4 : !l.cta_pair && !res && p->g.wzp_d == 0 && !p->pair && p->rings == 2;
    if (l.halo)
        return launch_kernel(l.box_kernel, l.grid, dim3(two_rings ? kThreads2 : kThreads), l.smem, st, bytes, 1, l.maps, l.args);
    return launch_kernel(l.kernel, l.grid, dim3(two_rings ? kThreads2 : kThreads), l.smem, st, bytes, l.cta_pair ? 2 : 1, l.maps, static_cast<const IgemmArgs &>(l.args));
}

// Everything the first launch of any plan would otherwise do once per process or device: the driver
// entry point of the tensor-map encoder and the kernels' shared-memory attribute (which also loads
// this module's code onto the current device).  Called at plan creation, while allocation is allowed.
int conv_igemm_warm()
{
    if (!encode_fn())
        return fail(B200_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
    // once per device: the attributes belong to the loaded module (256 devices and more are set up on every call)
    static std::atomic<bool> done[256];
    int device = 0;
    B200_CUDA_TRY(cudaGetDevice(&device));
    if (device < 256 && done[device].load(std::memory_order_acquire))
        return B200_OK;
    B200_TRY(conv_small_warm());
    for (int epi = 0; epi < kEpiVariants; ++epi)
        for (IgemmKernel k : { igemm_kernel_mode0(epi), igemm_kernel_mode1(epi), igemm_kernel_ragged(epi, false), igemm_kernel_ragged(epi, true),
                               igemm_kernel_mode2(epi), igemm_kernel_mode3(epi),
                               igemm_kernel_wzp(epi), igemm_kernel_residual(epi) })
            if (k)
                B200_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    for (int epi = 0; epi < kEpiVariants; ++epi)
        for (bool wzp : { false, true })
            for (IgemmBoxKernel k : { igemm_kernel_mode4(epi, wzp), igemm_kernel_mode5(epi, wzp) })
                B200_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    if (device < 256)
        done[device].store(true, std::memory_order_release);
    return B200_OK;
}

int mma_i8_peak_launch(int mmas_per_sm, float *ms, double *ops, cudaStream_t st)
{
    int *status = nullptr;
    B200_TRY(status_word_ptr(&status));
    const int mmas = mmas_per_sm / kPeakGroup * kPeakGroup;
    const size_t smem = 128 * 128 + 256 * 128 + 1024;
    B200_CUDA_TRY(cudaFuncSetAttribute(mma_i8_peak_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    cudaEvent_t e0, e1;
    B200_CUDA_TRY(cudaEventCreate(&e0));
    B200_CUDA_TRY(cudaEventCreate(&e1));
    const int sms = sm_count();
    B200_CUDA_TRY(cudaEventRecord(e0, st));
    mma_i8_peak_kernel<<<sms, 128, smem, st>>>(mmas, status);
    cudaError_t le = cudaGetLastError();
    B200_CUDA_TRY(cudaEventRecord(e1, st));
    cudaError_t se = cudaEventSynchronize(e1);
    float t = 0.f;
    if (le == cudaSuccess && se == cudaSuccess)
        se = cudaEventElapsedTime(&t, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    B200_CUDA_TRY(le);
    B200_CUDA_TRY(se);
    *ms = t;
    *ops = (double)sms * (double)mmas * 2.0 * 128.0 * 256.0 * 32.0;
    return B200_OK;
}

int wait_expiry_probe_launch(long long limit_cycles, cudaStream_t st)
{
    int *status = nullptr;
    B200_TRY(status_word_ptr(&status));
    wait_expiry_probe_kernel<<<1, 32, 0, st>>>(status, limit_cycles);
    B200_CUDA_TRY(cudaGetLastError());
    return B200_OK;
}

}  // namespace b200
