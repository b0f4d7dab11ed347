// Implicit-GEMM int8 convolution for launches that do not fill the GPU: a batch of one or a few images, the
// last stages of a network at a serving batch, an inner product.  Same arithmetic and operands as the persistent
// kernel (conv_igemm_sm100.cu); what differs is what bounds it.  There the tensor pipe and the epilogue set the
// pace; here a launch is one chain -- launch, first TMA round trip, MMAs, accumulator, store -- and its length is the
// time.  On one image the persistent kernel walked all k-blocks of 256 channels x 3x3 on two CTAs (14.4 us) and of
// 512 channels on two (22.8 us): 72 and 144 MMAs one after the other at 64 cycles or more each, 3 to 6 stages of
// operands in flight.  So:
//   * one tile per CTA, narrow channel tiles, and the k-blocks of a tile split over a cluster of up to eight CTAs
//     (int32 sums: any order gives the same bits).  The partial accumulators meet in a reduce-scatter over distributed
//     shared memory: CTA r of the cluster receives and finishes channels [r * bn / split, (r + 1) * bn / split);
//   * every k-block of a CTA has a slot of its own where they fit, the weights' loads are issued before
//     griddepcontrol.wait, and constants reach shared memory while the operands are on their way;
//   * 320 threads and as little shared memory as that needs, so that the next launch's CTAs are resident beside these.
// Roles: warp 0 TMA (one elected lane), warp 1 tensor memory and MMAs, warps 2-9 epilogue, two per lane quarter.  The
// epilogue is the persistent kernel's arithmetic (EpiForm); requantizing channel by channel with a shift each, as this kernel
// first did, took 0.9 us per 16 channels of a tile, most of a 64-channel launch's time.
#include <stdlib.h>

#include "common.cuh"
#include "conv_igemm_kernel.cuh"
#include "conv_small.h"
#include "kernels.h"
#include "sm100_ptx.cuh"

namespace b200 {

namespace {

constexpr int kSmallEpiThreads = 256;
constexpr int kSmallThreads = 64 + kSmallEpiThreads;
constexpr int kSmallM = 128;            // pixels per tile
constexpr int kSmallSlots = 16;
constexpr int kSmallClsCols = 4096;     // border classes x channels that are staged in shared memory; more are read in place

constexpr int kErrSmallProducer = 0x201, kErrSmallFull = 0x202, kErrSmallEpilogue = 0x203;

struct SmallLayout {
    uint32_t b, b_tile, red, xred, mult, shift, off, stage, stage_pitch, bars, tmem_slot, abort_flag, total;
};
__host__ __device__ inline SmallLayout small_layout(const SmallArgs &g)
{
    SmallLayout L;
    uint32_t o = (uint32_t)g.slots * kSmallM * g.bk;
    L.b = o;
    L.b_tile = ((uint32_t)(g.bn + (g.wzp_d ? 16 : 0)) * g.bk + 1023u) & ~1023u;
    o += g.slots * L.b_tile;
    L.red = o;                                              // [split][channel quad][128][4] partial accumulators
    o += g.split > 1 ? (uint32_t)g.bn * kSmallM * 4 : 0;
    L.xred = o;                                             // [split][128] partial window sums
    o += g.split > 1 && g.wzp_d ? (uint32_t)g.split * kSmallM * 4 : 0;
    L.mult = o;
    o += g.bn * 4;
    L.shift = o;
    o += g.bn * 4;
    L.off = o;
    o += g.n_cls * g.bn <= kSmallClsCols ? (uint32_t)g.n_cls * g.bn * 4 : 0;
    o = (o + 15u) & ~15u;
    // Cout % 16 != 0: the tile's bytes pass through shared memory, so that whole words reach global memory (a byte store
    // per channel and pixel took 20 us for 218 channels of 6776 pixels)
    L.stage = o;
    L.stage_pitch = (uint32_t)(g.bn / g.split) + 16;
    o += g.cout % 16 != 0 ? kSmallM * L.stage_pitch : 0;
    L.bars = o;                                             // full[slots], empty[slots], accumulator
    o += (2 * kSmallSlots + 1) * 8;
    L.tmem_slot = o;
    o += 8;
    L.abort_flag = o;
    o += 8;
    L.total = o + 1024;                                     // the base is aligned to 1024
    return L;
}

__device__ __forceinline__ void st_cluster4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d)
{
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void st_cluster(uint32_t addr, uint32_t v)
{
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

// Where a CTA's tables lie (shared addresses), and this thread's border class's offsets.
struct SmallTables {
    uint32_t off_s, mul, shift;
    const int32_t *off_g;               // nullptr: staged at off_s
};

// N channels from accumulators `acc` (one pixel), the first at channel j of the tile: requantized, packed, stored at element
// `at` of the output, and with the residual added at the same element of its sum; or at the shared address `stage`.
template <int N, bool SUM>
__device__ __forceinline__ void store_channels(const uint32_t (&acc)[N], const SmallArgs &g, const EpiConsts &ec, const SmallTables &t, int xcorr,
                                               int j, size_t at, uint32_t stage)
{
    uint32_t w[N / 4], x[N / 4];
    if (SUM) {            // on its way while the accumulators are requantized (Cout is a multiple of 16 then)
        if constexpr (N == 16) {
            const uint4 v = __ldg(reinterpret_cast<const uint4 *>(g.res + at));
            x[0] = v.x, x[1] = v.y, x[2] = v.z, x[3] = v.w;
        } else {
            const uint2 v = __ldg(reinterpret_cast<const uint2 *>(g.res + at));
            x[0] = v.x, x[1] = v.y;
        }
    }
    if (t.off_g == nullptr) {
        if (g.form == kEpiFp)
            epi_pack<kEpiFp, true, true, true>(acc, t.off_s + j * 4, nullptr, t.mul + j * 4, t.shift + j * 4, ec, xcorr, w);
        else if (g.form == kEpiInt)
            epi_pack<kEpiInt, true, true, true>(acc, t.off_s + j * 4, nullptr, t.mul + j * 4, t.shift + j * 4, ec, xcorr, w);
        else
            epi_pack<kEpiGeneric, true, true, true>(acc, t.off_s + j * 4, nullptr, t.mul + j * 4, t.shift + j * 4, ec, xcorr, w);
    } else {
        if (g.form == kEpiFp)
            epi_pack<kEpiFp, false, true, true>(acc, 0, t.off_g + j, t.mul + j * 4, t.shift + j * 4, ec, xcorr, w);
        else if (g.form == kEpiInt)
            epi_pack<kEpiInt, false, true, true>(acc, 0, t.off_g + j, t.mul + j * 4, t.shift + j * 4, ec, xcorr, w);
        else
            epi_pack<kEpiGeneric, false, true, true>(acc, 0, t.off_g + j, t.mul + j * 4, t.shift + j * 4, ec, xcorr, w);
    }
    if (stage != 0) {
        if constexpr (N == 16)
            sts4(stage, make_uint4(w[0], w[1], w[2], w[3]));
        else
            asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(stage), "r"(w[0]), "r"(w[1]) : "memory");
        return;
    }
    auto store = [&](uint8_t *dst) {
        if constexpr (N == 16)
            *reinterpret_cast<uint4 *>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
        else
            *reinterpret_cast<uint2 *>(dst) = make_uint2(w[0], w[1]);
    };
    store(g.y + at);
    if (SUM) {
#pragma unroll
        for (int q = 0; q < N / 4; ++q)
            w[q] = add_residual(w[q], x[q], ec);
        store(g.sum + at);
    }
}

// SUM: the instantiation that also forms a residual add (ConvSum); the other one carries none of that code.
template <bool SUM>
__global__ void __launch_bounds__(kSmallThreads) conv_small_kernel(const __grid_constant__ SmallMaps maps, const __grid_constant__ SmallArgs g)
{
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t base = (raw_addr + 1023u) & ~1023u;
    uint8_t *smem = smem_raw + (base - raw_addr);
    const SmallLayout L = small_layout(g);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;     // (the warp: known to be uniform)
    const uint32_t bars = base + L.bars;
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (kSmallSlots + s); };
    const uint32_t acc_bar = bars + 8u * (2 * kSmallSlots);
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(smem + L.tmem_slot);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + L.abort_flag);

    const int split = g.split;
    const int rank = split > 1 ? (int)(blockIdx.x % (unsigned)split) : 0;    // clusters are consecutive blocks
    const int tile = (int)(blockIdx.x / (unsigned)split);
    const int nt = tile % g.n_tiles_n;
    int mt = tile / g.n_tiles_n;
    const int twi = mt % g.tiles_w;
    mt /= g.tiles_w;
    const int thi = mt % g.tiles_h, tni = mt / g.tiles_h;
    const int kb0 = rank * g.kblocks / split, kb1 = (rank + 1) * g.kblocks / split;
    const int k0 = nt * g.bn;

    if (threadIdx.x == 0) {
        for (int s = 0; s < g.slots; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        mbar_init(acc_bar, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x == 64) {
        prefetch_map(&maps.a[0]);
        prefetch_map(&maps.b);
    }
    if (warp == 1) {
        tmem_alloc(base + L.tmem_slot, g.tmem_cols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    if (split > 1)
        cluster_sync_all();         // the peers run: their shared memory may be written
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t a_tile = (uint32_t)kSmallM * g.bk;

    if (warp == 0) {
        // ================= TMA =================
        // in order: the weights of the first `slots` k-blocks (constant, the launch before this one does not matter to them),
        // and behind its wait the k-blocks one by one; uniform loops around elect_one(), see there
        {
            const uint32_t tx = a_tile + (uint32_t)(g.bn + (g.wzp_d ? 16 : 0)) * g.bk;
            const int sh_h = g.stride_h - 1, sh_w = g.stride_w - 1;
            auto load_b = [&](int slot, int kc) {
                const uint32_t b_dst = base + L.b + slot * L.b_tile;
                if (elect_one()) {
                    mbar_expect_tx(full_bar(slot), tx);
                    tma_load_2d(b_dst, &maps.b, full_bar(slot), kc, k0);
                    if (g.wzp_d)
                        tma_load_2d(b_dst + g.bn * g.bk, &maps.ones, full_bar(slot), kc, 0);
                }
            };
            const int tap0 = kb0 / g.cchunks, chunk0 = kb0 - tap0 * g.cchunks;
            int chunk = chunk0, tap_c = tap0 * g.cpad;
            auto advance = [&] {
                if (++chunk == g.cchunks) {
                    chunk = 0;
                    tap_c += g.cpad;
                    return true;
                }
                return false;
            };
            for (int kb = kb0, slot = 0; slot < g.slots && kb < kb1; ++kb, ++slot) {
                load_b(slot, tap_c + chunk * g.bk);
                advance();
            }
            pdl_wait();
            chunk = chunk0;
            tap_c = tap0 * g.cpad;
            int rr = tap0 / g.s, ss = tap0 - rr * g.s, slot = 0;
            uint32_t phase = 1;
            for (int kb = kb0; kb < kb1; ++kb) {
                if (kb >= kb0 + g.slots) {
                    if (!mbar_wait_warp(empty_bar(slot), phase, abort_flag)) {
                        if (lane == 0)
                            atomicCAS(g.status, 0, kErrSmallProducer);
                        *abort_flag = 1;
                        break;
                    }
                    load_b(slot, tap_c + chunk * g.bk);
                }
                // see the producer of conv_igemm_i8_kernel
                const int dh = rr - g.pad_h, ph = dh & sh_h, dw = ss - g.pad_w, pw = dw & sh_w;
                const int yh = (thi << g.th_sh) + ((dh - ph) >> sh_h), xw = (twi << g.tw_sh) + ((dw - pw) >> sh_w), n0 = tni * g.tn;
                const CUtensorMap *amap = &maps.a[ph * 2 + pw];
                if (elect_one()) {
                    if (g.a_wide)
                        tma_load_3d(base + slot * a_tile, amap, full_bar(slot), xw << 2, yh, n0);
                    else
                        tma_load_4d(base + slot * a_tile, amap, full_bar(slot), chunk * g.bk, xw, yh, n0);
                }
                if (advance() && ++ss == g.s) {
                    ss = 0;
                    ++rr;
                }
                if (++slot == g.slots) {
                    slot = 0;
                    phase ^= 1;
                }
            }
        }
        __syncwarp();
        pdl_trigger();
    } else if (warp == 1) {
        // ================= MMA =================
        const uint64_t adesc0 = make_smem_desc(base, g.bk), bdesc0 = make_smem_desc(base + L.b, g.bk);
        const uint32_t desc_hi = (uint32_t)(adesc0 >> 32);
        int slot = 0, chunk = kb0 % g.cchunks;
        uint32_t phase = 0, accumulate = 0;
        bool ok = true;
        for (int kb = kb0; kb < kb1; ++kb) {
            if (!mbar_wait_warp(full_bar(slot), phase, abort_flag)) {
                if (lane == 0)
                    atomicCAS(g.status, 0, kErrSmallFull);
                *abort_flag = 1;
                ok = false;
                break;
            }
            tc_fence_after();
            const uint32_t a_lo = (uint32_t)adesc0 + slot * (a_tile >> 4), b_lo = (uint32_t)bdesc0 + slot * (L.b_tile >> 4);
            const int ksteps = chunk == g.cchunks - 1 ? g.last_steps : g.bk / 32;
            chunk = chunk == g.cchunks - 1 ? 0 : chunk + 1;
            if (elect_one()) {
                mma_i8(tmem_base, a_lo, b_lo, desc_hi, g.idesc, accumulate);
                if (ksteps >= 2)
                    mma_i8(tmem_base, a_lo + 2, b_lo + 2, desc_hi, g.idesc, 1);
                if (ksteps >= 3)
                    mma_i8(tmem_base, a_lo + 4, b_lo + 4, desc_hi, g.idesc, 1);
                if (ksteps == 4)
                    mma_i8(tmem_base, a_lo + 6, b_lo + 6, desc_hi, g.idesc, 1);
                if (kb + g.slots < kb1)
                    mma_commit(empty_bar(slot));
            }
            __syncwarp();
            accumulate = 1;
            if (++slot == g.slots) {
                slot = 0;
                phase ^= 1;
            }
        }
        if (ok && elect_one())
            mma_commit(acc_bar);
    }

    // ================= epilogue (warps 2..9) =================
    const int quarter = warp & 3;                       // tensor-memory lanes of this warp
    const int half = (warp - 2) >> 2;                   // which of the two warps of the quarter
    const int row = quarter * 32 + lane;
    const int bnl = g.bn / split;                       // channels this CTA finishes
    const bool off_staged = g.n_cls * g.bn <= kSmallClsCols;
    const int lw = row & ((1 << g.tw_sh) - 1), lh = (row >> g.tw_sh) & ((1 << g.th_sh) - 1), ln = row >> (g.tw_sh + g.th_sh);
    const int ow = (twi << g.tw_sh) + lw, oh = (thi << g.th_sh) + lh, img = tni * g.tn + ln;
    const bool pix_valid = ow < g.ow && oh < g.oh && img < g.n;
    const size_t at = (((size_t)img * g.oh + oh) * g.ow + ow) * g.cout + k0;
    const EpiConsts ec = { g.ozp, g.qmax, g.relu_lo, g.ushift, g.rnd_hi, (float)g.ozp + 0.5f, g.out_flip,
                           g.r_m[0], g.r_add[0], g.r_b[0], g.r_m[1], g.r_add[1], g.r_b[1], g.r_s0, g.r_ozp, g.r_lo };
    SmallTables t = { base + L.off, base + L.mult, base + L.shift, nullptr };
    const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const uint32_t stage = g.cout % 16 != 0 ? base + L.stage + (uint32_t)row * L.stage_pitch : 0u;
    bool ok = true;
    if (warp >= 2) {
        int *s_mult = reinterpret_cast<int *>(smem + L.mult), *s_shift = reinterpret_cast<int *>(smem + L.shift);
        int32_t *s_off = reinterpret_cast<int32_t *>(smem + L.off);
        const int et = threadIdx.x - 64;
        if (et == 0 && g.next_ro_bytes != 0) {
            const uint32_t granules = g.next_ro_bytes >> 4, per = (granules + gridDim.x - 1) / gridDim.x, from = blockIdx.x * per;
            if (from < granules)
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(g.next_ro + ((size_t)from << 4)), "r"(min(per, granules - from) << 4) : "memory");
        }
        for (int j = et; j < g.bn; j += kSmallEpiThreads) {
            const bool in = k0 + j < g.kpad;
            s_mult[j] = in ? __ldg(g.mul + k0 + j) : 0;
            s_shift[j] = in ? __ldg(g.shift + k0 + j) : 33;
        }
        if (off_staged)
            for (int i = et; i < g.n_cls * g.bn; i += kSmallEpiThreads) {
                const int c = i / g.bn, j = i - c * g.bn;
                s_off[i] = k0 + j < g.kpad ? __ldg(g.off32 + (size_t)c * g.kpad + k0 + j) : 0;
            }
        const int cls = (int)__ldg(g.row_cls + min(oh, g.oh - 1)) * g.n_col_cls + (int)__ldg(g.col_cls + min(ow, g.ow - 1));
        if (off_staged)
            t.off_s += (uint32_t)(cls * g.bn) * 4;
        else
            t.off_g = g.off32 + (size_t)cls * g.kpad + k0;
        asm volatile("bar.sync 1, 256;" ::: "memory");
        ok = __all_sync(0xffffffffu, mbar_wait(acc_bar, 0, abort_flag));
        if (!ok && lane == 0) {
            atomicCAS(g.status, 0, kErrSmallEpilogue);
            *abort_flag = 1;
        }
        tc_fence_after();
        pdl_wait();                                     // the output may be what the launch before this one still reads
        if (ok && split == 1) {
            int xcorr = 0;
            if (g.wzp_d) {
                uint32_t xs;
                tmem_ld1(t_row + g.bn, xs);
                tmem_ld_wait();
                xcorr = -g.wzp_d * (int)xs;
            }
            for (int c0 = half * 16; c0 < g.bn && k0 + c0 < g.cout; c0 += 32) {
                uint32_t v[16];
                tmem_ld16(t_row + c0, v);
                tmem_ld_wait();
                if (pix_valid)
                    store_channels<16, SUM>(v, g, ec, t, xcorr, c0, at + c0, stage ? stage + c0 : 0u);
                __syncwarp();
            }
        } else if (ok) {
            // this CTA's partial sums to the CTAs that finish them, four channels of 32 neighbouring pixels a store
            for (int c0 = half * 16; c0 < g.bn; c0 += 32) {
                uint32_t v[16];
                tmem_ld16(t_row + c0, v);
                tmem_ld_wait();
#pragma unroll
                for (int h = 0; h < 16; h += 8) {       // bn / split is a multiple of 8
                    const int owner = (c0 + h) / bnl, ch = ((c0 + h) - owner * bnl) >> 2;
                    const uint32_t to = cluster_addr(base + L.red + (uint32_t)(((rank * (bnl >> 2) + ch) * kSmallM + row) * 16), (uint32_t)owner);
                    st_cluster4(to, v[h], v[h + 1], v[h + 2], v[h + 3]);
                    st_cluster4(to + kSmallM * 16, v[h + 4], v[h + 5], v[h + 6], v[h + 7]);
                }
            }
            if (g.wzp_d && half == 0) {
                uint32_t xs;
                tmem_ld1(t_row + g.bn, xs);
                tmem_ld_wait();
                for (int o = 0; o < split; ++o)
                    st_cluster(cluster_addr(base + L.xred + (uint32_t)(rank * kSmallM + row) * 4, (uint32_t)o), xs);
            }
        }
    }
    if (split > 1) {
        __syncthreads();
        cluster_sync_all();
        if (warp >= 2 && ok && pix_valid) {
            int xcorr = 0;
            if (g.wzp_d) {
                const int *xred = reinterpret_cast<const int *>(smem + L.xred);
                for (int s = 0; s < split; ++s)
                    xcorr -= xred[s * kSmallM + row];
                xcorr *= g.wzp_d;
            }
            const int c1 = rank * bnl;                  // first channel of this CTA's share
            for (int j = half * 8; j < bnl && k0 + c1 + j < g.cout; j += 16) {
                uint32_t acc[8] = { 0, 0, 0, 0, 0, 0, 0, 0 };
                const uint32_t from = base + L.red + (uint32_t)(((j >> 2) * kSmallM + row) * 16);
#pragma unroll 4
                for (int s = 0; s < split; ++s) {
                    const int4 a = lds4(from + (uint32_t)(s * kSmallM * bnl) * 4);
                    const int4 b = lds4(from + (uint32_t)(s * kSmallM * bnl) * 4 + kSmallM * 16);
                    acc[0] += a.x; acc[1] += a.y; acc[2] += a.z; acc[3] += a.w;
                    acc[4] += b.x; acc[5] += b.y; acc[6] += b.z; acc[7] += b.w;
                }
                store_channels<8, SUM>(acc, g, ec, t, xcorr, c1 + j, at + c1 + j, stage ? stage + j : 0u);
            }
        }
    }
    if (stage != 0 && warp >= 2) {
        asm volatile("bar.sync 1, 256;" ::: "memory");      // both warps of a quarter have staged their channels
        const int c1 = rank * bnl, n = min(bnl, g.cout - k0 - c1);
        const unsigned valid = __ballot_sync(0xffffffffu, pix_valid && ok);
        if (n > 0) {
            const int lanes = copy_lanes(n), step = 32 / lanes;
            for (int pr = half * step + lane / lanes; pr < 32; pr += 2 * step) {
                if (!((valid >> pr) & 1))
                    continue;
                const int prow = quarter * 32 + pr;
                const int plw = prow & ((1 << g.tw_sh) - 1), plh = (prow >> g.tw_sh) & ((1 << g.th_sh) - 1), pln = prow >> (g.tw_sh + g.th_sh);
                uint8_t *dst = g.y + (((size_t)(tni * g.tn + pln) * g.oh + (thi << g.th_sh) + plh) * g.ow + (twi << g.tw_sh) + plw) * g.cout + k0 + c1;
                const uint32_t src = base + L.stage + (uint32_t)prow * L.stage_pitch;
                copy_row(dst, n, lane & (lanes - 1), lanes, [&](int off) { return lds1(src + off); });
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, g.tmem_cols);
    }
}

}  // namespace

bool conv_small_pick(int m_tiles, int k, int kblocks, int bk, bool wzp, int bn_p, int *bn_out, int *split_out)
{
    // Microseconds on this GPU, fitted to sweeps over both kernels' tilings of ResNet-50's and MobileNetV2's layers at
    // batches 1 to 32.  What counts: a k-block's rows through the SM's TMA unit (0.25 us for 128 rows of 64 bytes, 0.37 of
    // 128), the epilogue behind the last MMA, and the cluster's exchange of partial sums.
    const int sms = sm_count(), extra = wzp ? 16 : 0, k16 = (k + 15) / 16 * 16;
    const double row = 0.13 + 0.0019 * bk;
    double best;
    {   // the persistent kernel: a round's loads and the epilogue of the round before it overlap
        const int rounds = (m_tiles * ((k + bn_p - 1) / bn_p) + sms - 1) / sms;
        const double load = kblocks * row * (bn_p > 128 ? 1.4 : 1.1), epi = 0.008 * bn_p;
        best = 3.4 + rounds * (load > epi ? load : epi) + (load > epi ? epi : load);
    }
    bool small = false;
    for (int bn = 16; bn <= 128; bn *= 2) {
        if (bn > 16 && bn / 2 >= k16)
            break;
        const int tiles = m_tiles * ((k + bn - 1) / bn);
        for (int split = 1; split <= 8 && split <= kblocks && bn / split >= 8; split *= 2) {
            const int ctas = tiles * split, kb = (kblocks + split - 1) / split;
            // two CTAs share an SM where both fit its shared memory; clusters of four and eight leave SMs of a GPC over
            const int slots = kb < 4 ? kb : 4;
            const bool two = split == 1 && slots * (kSmallM + bn + extra) * bk <= 104 * 1024;
            if (ctas > (split == 8 ? sms * 2 / 3 : split == 4 ? sms * 7 / 8 : two ? 2 * sms : sms))
                continue;
            const double load = kb * (row + 0.0003 * (bn + extra));
            const double epi = split > 1 ? 0.6 + 0.012 * bn + 0.7 * ctas / sms + (split == 8 ? 0.5 : 0.0) : bn > 32 ? 0.0125 * (bn - 32) : 0.0;
            const double cost = ctas > sms ? 3.2 + (load + epi) * ctas / sms : 2.3 + load + epi;
            if (cost < best) {
                best = cost;
                small = true;
                *bn_out = bn;
                *split_out = split;
            }
        }
    }
    return small;
}

size_t conv_small_smem(SmallArgs &a, bool act_signed)
{
    const int kb = (a.kblocks + a.split - 1) / a.split, n = a.bn + (a.wzp_d ? 16 : 0);
    a.idesc = (2u << 4) | ((act_signed ? 1u : 0u) << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kSmallM >> 4) << 24);
    a.tmem_cols = 32;
    while (a.tmem_cols < (uint32_t)n)
        a.tmem_cols <<= 1;
    a.slots = kb < kSmallSlots ? kb : kSmallSlots;
    while (a.slots > 4 && small_layout(a).total > 110 * 1024)       // two CTAs per SM: this launch's and the next one's
        --a.slots;
    while (a.slots > 1 && small_layout(a).total > 227 * 1024)
        --a.slots;
    // A CTA waits for tensor memory (512 columns an SM) while its cluster waits for it, so CTAs of clusters must never fill an
    // SM's columns against each other: two clusters could each hold what the other's peer waits for.  Three CTAs fit an
    // SM's registers, and 128 columns each fit.  Those of 256 (a window-sum column beside 128 channels) ask for more than half
    // of the shared memory, so that an SM holds one of them at most.  (CTAs without a cluster give theirs back by themselves.)
    const size_t total = small_layout(a).total, half_sm = 116 * 1024;
    return a.split > 1 && a.tmem_cols > 128 && total < half_sm ? half_sm : total;
}

int conv_small_launch(const SmallMaps &maps, const SmallArgs &a, int m_tiles, size_t smem, size_t bytes, cudaStream_t st)
{
    return launch_kernel(a.res ? conv_small_kernel<true> : conv_small_kernel<false>, dim3((unsigned)(m_tiles * a.n_tiles_n * a.split)), dim3(kSmallThreads), smem, st, bytes, a.split, maps, a);
}

int conv_small_warm()
{
    for (auto k : { conv_small_kernel<false>, conv_small_kernel<true> })
        B200_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    return B200_OK;
}

}  // namespace b200
