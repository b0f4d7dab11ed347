// Shared host/device helpers of the sm_100a quantized-convolution backend: status reporting
// for the C-ABI, and the device restatement of the reference CPU module's integer requantize
// arithmetic (art/modules/quant/include/art/quant/quant_helper.h:29-118 of ModelTC/NART).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "nart_b200.h"

namespace b200 {

// ---- host: error plumbing ------------------------------------------------------------------
void set_error(const char *fmt, ...);
int fail(int status, const char *fmt, ...);

#define B200_CUDA_TRY(expr)                                                                    \
    do {                                                                                       \
        cudaError_t _e = (expr);                                                               \
        if (_e != cudaSuccess) {                                                               \
            cudaGetLastError(); /* a non-sticky error must not surface at a later, unrelated call */ \
            return ::b200::fail(                                                               \
                B200_ERR_CUDA, "%s failed: %s (%s:%d)", #expr, cudaGetErrorString(_e), __FILE__, \
                __LINE__);                                                                     \
        }                                                                                      \
    } while (0)

#define B200_TRY(expr)           \
    do {                         \
        int _s = (expr);         \
        if (_s != B200_OK)       \
            return _s;           \
    } while (0)

inline cudaStream_t as_stream(b200_stream_t s) { return reinterpret_cast<cudaStream_t>(s); }

// Per-device int the kernels with bounded waits write a code into when a wait runs out.
int status_word_ptr(int **dev_ptr);
// Queues a kernel that moves the current device's status word to *host (pinned) and clears it.
int status_publish_launch(int *host, cudaStream_t st);
__device__ __forceinline__ void status_publish(int *word, int *host)
{
    const int v = *word;
    *host = v;
    if (v != 0)
        *word = 0;
}

// Device copy of a 256-byte lookup table, uploaded the first time this table is seen on the current device
// and cached for the life of the process (runtime.cu).
int lut_cache_get(const uint8_t lut[256], const uint8_t **dev_ptr);

// Division of 32-bit numbers below 2^31 by a launch constant, after Granlund and Montgomery, "Division by invariant integers
// using multiplication" (PLDI 1994): one high multiplication, one shift (the multiplier is rounded up, 2^(31 + l) / d
// with 2^(l-1) < d <= 2^l, whose error stays below one part in 2^31).
struct FastDiv {
    uint32_t d = 1, mul = 0x80000000u, shift = 0;
    FastDiv() = default;
    explicit FastDiv(uint32_t divisor) : d(divisor)
    {
        uint32_t l = 0;
        while ((1ull << l) < divisor)
            ++l;
        mul = (uint32_t)(((1ull << (31 + l)) + divisor - 1) / divisor);
        shift = l;
    }
#ifdef __CUDACC__
    __device__ __forceinline__ uint32_t div(uint32_t n) const { return (uint32_t)(((uint64_t)n * mul) >> 31) >> shift; }
#endif
};

// Another device as the current one for the time of a scope.
struct DeviceGuard {
    int before = -1;
    explicit DeviceGuard(int device)
    {
        int now = device;
        if (cudaGetDevice(&now) == cudaSuccess && now != device && cudaSetDevice(device) == cudaSuccess)
            before = now;
    }
    ~DeviceGuard()
    {
        if (before >= 0)
            cudaSetDevice(before);
    }
    DeviceGuard(const DeviceGuard &) = delete;
};

// Number of SMs of the current device (cached).
int sm_count();

// Grid of a grid-stride kernel: the blocks that are resident at one time (occupancy x SMs), or
// fewer when there is less work.  A larger grid would run a second, partly filled wave.
template <auto Kernel, int Threads>
int resident_grid(size_t blocks_wanted)
{
    static const int per_sm = [] {
        int occ = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, Kernel, Threads, 0) != cudaSuccess || occ < 1)
            occ = 1;
        return occ;
    }();
    const size_t cap = (size_t)sm_count() * per_sm;
    const size_t blocks = blocks_wanted < cap ? blocks_wanted : cap;
    return (int)(blocks < 1 ? 1 : blocks);
}

// ---- programmatic dependent launch ------------------------------------------------------------
// Kernels are launched through launch_kernel, as a rule with the programmatic-serialization
// attribute, and run pdl_wait() before they touch memory that another launch of its stream may
// write or read: its blocks become resident, and its prologue runs, while the launch before it drains.
// pdl_wait() returns when that launch has completed and its writes are visible; since that launch
// waited for the one before it in the same way, everything earlier in the stream has completed too.
// pdl_trigger() lets the next launch of the stream become resident.  Kernels trigger after their own wait,
// so that one launch at most is resident ahead of its turn, and the convolutions only once their last
// loads are issued: blocks that wait take their SM's shared memory and registers from others (ResNet-50 at
// batch 1 0.635 ms with the trigger at entry, 0.594 ms so, 0.712 ms without the attribute).
// A kernel that allocates tensor memory triggers after it holds it: a later launch that got there
// first would keep it from this one while waiting for it.
// The case runner bounds the bytes a launch may move to get the attribute (PdlLimit): with batches in
// flight on several streams, blocks that are resident ahead of their turn take SMs from the other
// streams' kernels, which costs more than the launch it hides once the kernels are long.
inline thread_local size_t t_pdl_limit = SIZE_MAX;
struct PdlLimit {
    size_t before = t_pdl_limit;
    explicit PdlLimit(size_t bytes) { t_pdl_limit = bytes; }
    ~PdlLimit() { t_pdl_limit = before; }
};
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// bytes: what the launch moves.  cluster_x > 1: launched as clusters of that many blocks along x.
template <typename... KArgs, typename... Args>
inline int launch_kernel(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, size_t bytes, int cluster_x, Args &&...args)
{
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = (unsigned)cluster_x; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    const bool pdl = bytes < t_pdl_limit;
    cfg.attrs = pdl ? at : at + 1;
    cfg.numAttrs = (pdl ? 1 : 0) + (cluster_x > 1 ? 1 : 0);
    B200_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...));
    return B200_OK;
}

// Host restatement of quant_helper.h:60-118 (see b200_get_quant_scale).
void get_quant_scale(float x, int bits, uint32_t *mult, int8_t *shift);
// Host restatement of quant_helper.h:55-58.
inline int64_t rshift_rn_host(int64_t x, int bits)
{
    int64_t y = x >> (bits - 1);
    return (y + ((y & 1) << 1)) >> 1;
}

// ---- device: requantize ----------------------------------------------------------------------
// rshift_rn(x, b) of the reference is ((x >> (b-1)) + (((x >> (b-1)) & 1) << 1)) >> 1 on int64,
// which equals floor((x + 2^(b-1)) / 2^b) whenever x + 2^(b-1) does not overflow (here
// |x| < 2^62).  For b >= 33 the low 32 bits of x cannot change the floor, so the high word of
// the product is enough:  floor((hi*2^32 + lo + 2^(b-1)) / 2^b) = (hi + 2^(b-33)) >> (b-32).
//
// Returns the value the reference passes to saturate_int_by_bits: the rounded shift plus the
// output zero point, narrowed to int32 (conv_2d_uint8_impl.c:159-164).
__device__ __forceinline__ int requant_raw(int acc, uint32_t mult, int shift, int ozp)
{
    if (shift >= 33) {
        return ((__mulhi(acc, (int)mult) + (1 << (shift - 33))) >> (shift - 32)) + ozp;
    }
    long long p = (long long)acc * (long long)mult;
    return (int)(((p + (1ll << (shift - 1))) >> shift) + (long long)ozp);
}

// saturate_int_by_bits (quant_helper.h:33-36) followed, when relu_lo >= 0, by the clamp at the
// output zero point that the reference's relu op performs for equal scales (relu.c:103-109).
__device__ __forceinline__ int sat_relu(int v, int qmax, int relu_lo)
{
    v = min(max(v, 0), qmax);
    return max(v, relu_lo);
}

__device__ __forceinline__ uint32_t pack4(int a, int b, int c, int d)
{
    return (uint32_t)a | ((uint32_t)b << 8) | ((uint32_t)c << 16) | ((uint32_t)d << 24);
}

// sat_u8 of four int32 values packed little-endian (byte 0 = a): cvt.pack.sat.u8.s32 converts two
// values with saturation to 0..255 and merges them above the low half of a third operand.
__device__ __forceinline__ uint32_t pack_sat_u8x4(int a, int b, int c, int d)
{
    uint32_t hi, out;
    asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(hi) : "r"(d), "r"(c), "r"(0));
    asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(out) : "r"(b), "r"(a), "r"(hi));
    return out;
}

// 64-bit rounded shift, 1 <= b <= 62.
__device__ __forceinline__ long long rshift_rn64(long long x, int b)
{
    return (x + (1ll << (b - 1))) >> b;
}

// The bits of 2^23 + floor(((a0, a1) - 1.5 * 2^23) * (m0, m1) + add)
__device__ __forceinline__ void fp_requant_pair(int a0, int a1, int m0, int m1, float add, int &q0, int &q1)
{
    asm("{\n\t.reg .b64 a, m, c, d;\n\t"
        "mov.b64 a, {%2, %3};\n\t"
        "mov.b64 c, {%6, %6};\n\t"
        "add.rn.f32x2 a, a, c;\n\t"
        "mov.b64 m, {%4, %5};\n\t"
        "mov.b64 d, {%7, %7};\n\t"
        "fma.rz.f32x2 a, a, m, d;\n\t"
        "mov.b64 c, {%8, %8};\n\t"
        "add.rz.f32x2 a, a, c;\n\t"
        "mov.b64 {%0, %1}, a;\n\t}"
        : "=r"(q0), "=r"(q1)
        : "r"(a0), "r"(a1), "r"(m0), "r"(m1), "f"(-12582912.f), "f"(add), "f"(8388608.f));
}

}  // namespace b200
