// Shared device/host helpers for the B200 (sm_100a) backend of the mynah-asr hot path.
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

namespace mb {

// ----------------------------------------------------------------- host errors
void set_error(const char *fmt, ...);
const char *last_error();

// (the error also comes off the thread: the next call's cudaGetLastError would report it as its own)
#define MB_CUDA(call)                                                                    \
    do {                                                                                 \
        cudaError_t e_ = (call);                                                         \
        if (e_ != cudaSuccess) {                                                         \
            cudaGetLastError();                                                          \
            mb::set_error("%s:%d %s -> %s", __FILE__, __LINE__, #call, cudaGetErrorString(e_)); \
            return -1;                                                                   \
        }                                                                                \
    } while (0)

#define MB_CUDA_NULL(call)                                                               \
    do {                                                                                 \
        cudaError_t e_ = (call);                                                         \
        if (e_ != cudaSuccess) {                                                         \
            cudaGetLastError();                                                          \
            mb::set_error("%s:%d %s -> %s", __FILE__, __LINE__, #call, cudaGetErrorString(e_)); \
            return nullptr;                                                              \
        }                                                                                \
    } while (0)

// While one lives, its thread's queries, allocations and frees leave a recording alone that another thread of the process
// makes in the global capture mode (they would end it with an error).
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    RelaxedCapture(const RelaxedCapture &) = delete;
    RelaxedCapture &operator=(const RelaxedCapture &) = delete;
};

// CUDA keeps function attributes and the SM count per device; a process may drive several devices.
// PerDevice remembers, for every device, the largest value configured so far (0 = nothing yet).
static constexpr int MB_MAX_DEVICES = 64;
struct PerDevice {
    size_t v[MB_MAX_DEVICES];
    // true when the current device has less than `want` on record; *dev receives the current device
    bool below(size_t want, int *dev) const;
    void record(int dev, size_t want);
};
int device_sm_count();      // SM count of the current device (cached per device; 148 if the query fails)

static inline int cdiv(int a, int b) { return (a + b - 1) / b; }
static inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// Device status word codes written by kernels whose bounded waits ran out.
// ST_RANGE: a value that had to become an fp16 (hi, lo) operand pair was not finite or reached 65504 in
// magnitude (the planes cannot hold it), so the result is not to be trusted.
enum { ST_OK = 0, ST_TIMEOUT_PRODUCER = 1, ST_TIMEOUT_MMA = 2, ST_TIMEOUT_EPILOGUE = 3, ST_RANGE = 4 };

// A matrix stored as two fp16 planes: value = hi + lo * 2^-11 (22 significant bits).
// The residual is kept pre-scaled by 2^11 so that it has the magnitude of hi and never
// falls into the fp16 subnormal range. GEMM operands are always read in this form so
// that the tensor cores can reproduce f32-grade products with three fp16 MMAs:
// hi*hi into one accumulator, lo*hi + hi*lo into a second one that the epilogue adds
// back scaled by 2^-11.
struct H16 {
    __half *hi;
    __half *lo;
};

#ifdef __CUDACC__
// ---- chained launches (programmatic dependent launch) --------------------------------------------------------
// A decoder position is some fifty small kernels, each waiting for the one before. Launched with `chain`, a kernel's
// blocks may be placed on the SMs while its predecessor in the stream is still running; the kernel calls
// chain_trigger() when it starts (its successor may be placed) and chain_wait() before it touches any memory a
// predecessor writes or reads: chain_wait() returns once every earlier kernel of the stream has finished and its
// writes are visible. What comes before chain_wait() may only read constants (weights) and set up the block.
// Both calls are no-ops in a kernel launched the ordinary way.
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... KArgs, typename... Args>
static inline cudaError_t launch_kernel(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, bool chain,
                                        int cluster_x, Args... args) {
    cudaLaunchConfig_t lc = {};
    lc.gridDim = grid; lc.blockDim = block; lc.dynamicSmemBytes = smem; lc.stream = st;
    cudaLaunchAttribute at[2];
    int n = 0;
    if (cluster_x > 1) {
        at[n].id = cudaLaunchAttributeClusterDimension;
        at[n].val.clusterDim.x = (unsigned)cluster_x; at[n].val.clusterDim.y = 1; at[n].val.clusterDim.z = 1;
        n++;
    }
    if (chain) {
        at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[n].val.programmaticStreamSerializationAllowed = 1;
        n++;
    }
    lc.attrs = at; lc.numAttrs = (unsigned)n;
    return cudaLaunchKernelEx(&lc, kernel, KArgs(args)...);
}

// ------------------------------------------------------------- device helpers
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

static constexpr float H16_LO_SCALE = 2048.0f;          // 2^11
static constexpr float H16_LO_INV = 1.0f / 2048.0f;
// Returns false when v does not fit the planes (|v| >= 65504, inf or NaN): hi would be infinite and lo a NaN.
// Producers that own a status word report ST_RANGE then.
static constexpr float H16_MAX = 65504.0f;
__device__ __forceinline__ bool split_h16(float v, __half &hi, __half &lo) {
    hi = __float2half_rn(v);
    lo = __float2half_rn((v - __half2float(hi)) * H16_LO_SCALE);
    return fabsf(v) < H16_MAX;
}

// The same for two values, and for four: neighbours share the conversions.
__device__ __forceinline__ bool split_h16x2(float x, float y, uint32_t &hi, uint32_t &lo) {
    const __half2 h = __floats2half2_rn(x, y);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn((x - f.x) * H16_LO_SCALE, (y - f.y) * H16_LO_SCALE);
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = *reinterpret_cast<const uint32_t *>(&l);
    return (fabsf(x) < H16_MAX) & (fabsf(y) < H16_MAX);
}
__device__ __forceinline__ bool split_h16x4(float4 v, uint2 &hi, uint2 &lo) {
    return split_h16x2(v.x, v.y, hi.x, lo.x) & split_h16x2(v.z, v.w, hi.y, lo.y);
}

// 1 / d for normal d whose reciprocal is normal, by one step of Newton's iteration on the instruction's approximation (2^-23): the
// step squares the error, what is left is its last rounding. In place of __frcp_rn in the element-wise passes: the encoder over twelve
// ragged utterances in the single-product mode 4.47 -> 4.23 ms, over eight with int8 activations 7.05 -> 6.40, one minute on 24
// layers 11.90 -> 11.70.
__device__ __forceinline__ float reciprocal(float d) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    return fmaf(r, fmaf(-d, r, 1.0f), r);
}

// Sigmoid for the bulk element-wise passes (GLU, SiLU after the conv norm, the contractions' epilogues). Below -87 (1.6e-38) it is 0:
// the reciprocal would leave the normal range, and x * sigmoid(x) has to vanish for large x, too. NaN stays NaN. Largest
// relative error against float64 over four million arguments: 1.33e-7 for x >= 0, 3.84e-6 below (the exponential's).
__device__ __forceinline__ float sigmoid_fast(float x) {
    const float r = reciprocal(1.0f + __expf(-x));
    return x < -87.0f ? 0.0f : r;
}
__device__ __forceinline__ float silu_f(float x) { return x * sigmoid_fast(x); }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// --------------------------------------------------------------- mbarrier/TMA
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: gives up after ~2^31 clocks (about a second) and reports false.
// No wait in this library spins without a limit.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (clock64() - t0 > (1ll << 31)) return false;
    }
    return true;
}

// The same by a whole warp, with one answer for all lanes.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t *bar, uint32_t parity) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    const long long t0 = clock64();
    while (!__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) {
        if (__any_sync(0xffffffffu, clock64() - t0 > (1ll << 31))) return false;
    }
    return true;
}

__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap *m) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
// 2-D tiled TMA load into this CTA's own shared memory.
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *m, int x, int y, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

// The warp's number as a value that the compiler knows to be the same in all lanes, and one lane of a converged warp: what a warp
// computes for an instruction that one lane issues then stays in uniform registers, which tcgen05 and TMA take their operands from.
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0); }
__device__ __forceinline__ bool elect_one() {
    uint32_t on;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(on));
    return on != 0;
}

// ------------------------------------------------------------------- tcgen05
__device__ __forceinline__ void tc_alloc(uint32_t *slot, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)),
                 "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tc_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// D[tmem] (+)= A[smem] * B[smem]; fp16 inputs, f32 accumulators.
__device__ __forceinline__ void tc_mma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                           uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrive on an mbarrier once every MMA issued so far by this thread has finished.
__device__ __forceinline__ void tc_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     smem_u32(bar))
                 : "memory");
}
// 32 lanes x 32 consecutive f32 columns of TMEM -> 32 registers per thread.
__device__ __forceinline__ void tc_ld32(uint32_t taddr, float *v) {
    uint32_t *r = reinterpret_cast<uint32_t *>(v);
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
// 32 lanes x 16 consecutive f32 columns.
__device__ __forceinline__ void tc_ld16(uint32_t taddr, float *v) {
    uint32_t *r = reinterpret_cast<uint32_t *>(v);
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor for a K-major operand tile whose rows are
// 128 bytes (64 fp16) laid out by TMA with the 128-byte swizzle: eight-row
// groups are 1024 bytes apart (stride byte offset), descriptor version 1.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);          // start address
    d |= (uint64_t)0 << 16;                                // leading byte offset (unused, K-major swizzled)
    d |= (uint64_t)(1024u >> 4) << 32;                     // stride byte offset
    d |= (uint64_t)1 << 46;                                // descriptor version (sm_100)
    d |= (uint64_t)2 << 61;                                // layout: SWIZZLE_128B
    return d;
}
// Instruction descriptor: D f32, A/B fp16, both K-major, M x N tile.
__host__ __device__ constexpr uint32_t umma_idesc_f16(int M, int N) {
    return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
#endif  // __CUDACC__

}  // namespace mb
