// Shared device/host helpers for the sm_100a kernels of the RWKV-7 decode path.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include <mutex>

namespace ab {

// ---------------------------------------------------------------------------------------------
// Status codes returned by every extern "C" entry point (0 = success).
// ---------------------------------------------------------------------------------------------
enum Status : int {
    OK = 0,
    ERR_BAD_ARG = -1,      // null pointer, misaligned pointer, unsupported shape
    ERR_CUDA = -2,         // a CUDA runtime call failed; see ab_last_error()
    ERR_TOO_LARGE = -3,    // size exceeds a compiled-in limit
    ERR_DEVICE_WAIT = -4,  // a bounded device-side wait ran out (reported through the status word)
};

void set_error(const char* fmt, ...);
int check_cuda(cudaError_t e, const char* what);

#define AB_CHECK_ARG(cond, ...)                 \
    do {                                        \
        if (!(cond)) {                          \
            ab::set_error(__VA_ARGS__);         \
            return ab::ERR_BAD_ARG;             \
        }                                       \
    } while (0)

#define AB_CUDA(call)                                        \
    do {                                                     \
        int _s = ab::check_cuda((call), #call);              \
        if (_s != ab::OK) return _s;                         \
    } while (0)

// One-time set-up of a launcher (function attributes, device properties) is per DEVICE, not per process: a process
// may drive several GPUs, and cudaFuncSetAttribute applies to the current one only. `run` executes `f` the first time
// it is called with a given device current (under a lock: host threads may launch concurrently) and remembers success.
constexpr int AB_MAX_DEVICES = 64;
struct DeviceProps {
    int n_sm = 0;
    size_t smem_optin = 0;
};
struct PerDeviceOnce {
    std::mutex mu;
    bool done[AB_MAX_DEVICES] = {};
    DeviceProps props[AB_MAX_DEVICES];
    template <class F>
    int run(const DeviceProps** out, F f) {
        int dev = 0;
        AB_CUDA(cudaGetDevice(&dev));
        AB_CHECK_ARG(dev >= 0 && dev < AB_MAX_DEVICES, "device index %d not supported (at most %d devices per process)", dev, AB_MAX_DEVICES);
        std::lock_guard<std::mutex> lock(mu);
        if (!done[dev]) {
            int v = 0, m = 0;
            AB_CUDA(cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev));
            AB_CUDA(cudaDeviceGetAttribute(&m, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
            props[dev].n_sm = v;
            props[dev].smem_optin = (size_t)m;
            const int s = f(props[dev]);
            if (s != OK) return s;
            done[dev] = true;
        }
        if (out) *out = &props[dev];
        return OK;
    }
};

int current_sm_count();   // SMs of the current device

// Device-side status word: kernels OR a bit in when a bounded wait gives up.
// The host reads it with ab_device_status().
static __device__ unsigned int g_device_status = 0;
constexpr unsigned int DEV_WAIT_GEMV = 1u;
constexpr unsigned int DEV_WAIT_GEMM = 2u;
constexpr unsigned int DEV_WAIT_HEAD = 4u;
constexpr unsigned int DEV_BOUNDS = 16u;     // bounds-checked build only: a computed index fell outside its array (the access was skipped)
constexpr unsigned int DEV_BAD_TOKEN = 8u;   // a token id outside [0, vocab) reached a kernel (it was clamped, not followed)

#ifndef TAG_POLL_NS_VALUE
#define TAG_POLL_NS_VALUE 100u
#endif
constexpr unsigned TAG_POLL_NS = TAG_POLL_NS_VALUE;   // pause between two looks at a tagged word that is not there yet

// Bounds-checked build (-DAB_BOUNDS_CHECK, `python -m albatross_b200.build --bounds-check`): the stand-in for a memory
// checker where none can be run. AB_BC(cond) is `true` in the normal build and costs nothing; in the checked build it
// evaluates the range condition of the access it guards, and when the condition fails it records DEV_BOUNDS in the status
// word and yields false, so that the access is skipped instead of made: `if (AB_BC(i < n)) a[i] = v;`.
#ifdef AB_BOUNDS_CHECK
#define AB_BC(cond) ((cond) ? true : (atomicOr(&ab::g_device_status, ab::DEV_BOUNDS), false))
#else
#define AB_BC(cond) true
#endif

// ---------------------------------------------------------------------------------------------
// PTX wrappers
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// try_wait that lets the hardware park the thread for up to `ns` before it reports "not yet":
// polling in a tight loop floods the shared-memory pipe that the math loads need.
__device__ __forceinline__ bool mbar_try_wait_park(uint64_t* bar, uint32_t parity, uint32_t ns) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(ns)
        : "memory");
    return ok != 0;
}
// Bounded wait: returns false (and the caller records an error) instead of spinning for ever.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, uint32_t max_iters = (1u << 20)) {
    for (uint32_t i = 0; i < max_iters; ++i) {
        if (mbar_try_wait_park(bar, parity, 2000u)) return true;
        if (i > 4) __nanosleep(64);
    }
    return false;
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// 1-D bulk (TMA) copy global -> shared, completion counted in bytes on an mbarrier.
// dst, src 16-byte aligned; bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
// Same with an L2 eviction-priority hint (weights are streamed once: evict first).
__device__ __forceinline__ void bulk_g2s_hint(void* dst, const void* src, uint32_t bytes, uint64_t* bar,
                                              uint64_t policy) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::
            "r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar)), "l"(policy)
        : "memory");
}
__device__ __forceinline__ uint64_t policy_evict_first() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint64_t policy_evict_last() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}

// Before a stage of shared memory is handed back to a copy engine (bulk or tensor copies write through the asynchronous
// proxy): what this thread read of the stage has arrived in its registers. An arrival on a barrier does not say that by
// itself: loads that were issued before it but whose results nobody has used yet may still be on their way when the refill
// lands, and then deliver bytes of it. (Seen with fp16 weights, whose words went into tensor memory only after the arrival: one 16-byte
// piece of one weight row in some ten million was that of the slot's next content.) `used` combines a word of each load, so that
// the comparison cannot be made before all of them are there; the store it guards hardly ever happens and means nothing. (One
// predicated store: as a branch it cost the step of 8 sequences 3.3 us of 174, so it costs 0.8.)
__device__ __forceinline__ void loads_returned(uint32_t used, uint32_t* nobody) {
    asm volatile("{\n .reg .pred p;\n setp.eq.u32 p, %0, 0x9e3779b9;\n @p st.volatile.shared.u32 [%1], %0;\n}" ::"r"(used), "r"(smem_u32(nobody)) : "memory");
}

// Programmatic dependent launch: wait for the preceding grid in the stream / let the next one start.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// 4-way int8 dot products. a: signed bytes; b: signed (ss) or unsigned (su) bytes.
__device__ __forceinline__ int dp4a_ss(uint32_t a, uint32_t b, int c) {
    int d;
    asm("dp4a.s32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ int dp4a_su(uint32_t a, uint32_t b, int c) {
    int d;
    asm("dp4a.s32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

// One byte holding two e2m1 codes (low nibble first) -> half2.
__device__ __forceinline__ __half2 e2m1x2_to_half2(uint32_t byte) {
    uint32_t out;
    asm("{\n .reg .b8 lo, hi;\n .reg .b16 t;\n cvt.u16.u32 t, %1;\n mov.b16 {lo, hi}, t;\n cvt.rn.f16x2.e2m1x2 %0, lo;\n}"
        : "=r"(out)
        : "r"(byte));
    return *reinterpret_cast<__half2*>(&out);
}
// Four bytes = eight e2m1 codes -> four half2 (byte i -> out[i], low nibble first): one unpack, four converts.
__device__ __forceinline__ void e2m1x8_to_half2x4(uint32_t word, uint32_t* out) {
    asm("{\n .reg .b8 b0, b1, b2, b3;\n mov.b32 {b0, b1, b2, b3}, %4;\n"
        " cvt.rn.f16x2.e2m1x2 %0, b0;\n cvt.rn.f16x2.e2m1x2 %1, b1;\n"
        " cvt.rn.f16x2.e2m1x2 %2, b2;\n cvt.rn.f16x2.e2m1x2 %3, b3;\n}"
        : "=r"(out[0]), "=r"(out[1]), "=r"(out[2]), "=r"(out[3])
        : "r"(word));
}
// Two e4m3 codes (16 bits) -> half2.
__device__ __forceinline__ __half2 e4m3x2_to_half2(uint32_t two) {
    uint32_t out;
    asm("{\n .reg .b16 t;\n cvt.u16.u32 t, %1;\n cvt.rn.f16x2.e4m3x2 %0, t;\n}" : "=r"(out) : "r"(two));
    return *reinterpret_cast<__half2*>(&out);
}
__device__ __forceinline__ float e4m3_to_float(uint32_t code) {
    return __low2float(e4m3x2_to_half2(code & 0xffu));
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// fp16 rounding points: the reference computes its glue in fp16 tensors, so each torch op rounds.
__device__ __forceinline__ float rh(float v) { return __half2float(__float2half_rn(v)); }
// Reciprocal, quotient and square root of operands that stay clear of the ends of the range, in straight-line code: several steps of
// the glue then run side by side. Each is the hardware's approximation, which PTX documents (rcp.approx and rsqrt.approx:
// relative error below 2^-22), and one Newton step whose residual a fused multiply-add computes with a
// single rounding (Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990):
//   reciprocal  r' = r + r (1 - d r)          from f(r) = 1/r - d:    1 - d r' = (1 - d r)^2
//   quotient    q' = q - r (d q - x)          q = x r, with r for 1 / d
//   root        s' = s + (r / 2) (x - s s)    s = x r, from f(s) = s^2 - x, with r for 1 / s
// With e the approximation's relative error the corrected value is within e^2 (2^-44) of the true one before the last operation rounds it:
// half a unit in the last place, but for results that lie within 2^-44 of the middle between two floats. Over all
// operands that reciprocal and root are given here, and all quotients of fp16 numerators by fp16 norms, the results are those of `1.f / d`,
// `x / d` and `sqrtf` (ab_glue_selftest goes through every one of them). Two blocks of the network, 4096 wide, with these and with the operators:
// 8 sequences one step 243 and 250 us, a prompt of 768 tokens 1360 and 1385, 5 of 37 tokens 384 and 398.
__device__ __forceinline__ float recip_(float d) {   // 1 <= d < 2^126, or NaN
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    return fmaf(r, fmaf(-d, r, 1.f), r);
}
__device__ __forceinline__ float quot_(float x, float d) {   // 1e-12 <= d <= 65504 or infinite; x finite, or infinite with d, or NaN
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    const float q = x * r;
    return d > 65504.f ? q : fmaf(-r, fmaf(d, q, -x), q);   // (signs like this: a numerator of -0 stays -0)
}
__device__ __forceinline__ float root_(float x) {   // 0, 2^-60 <= x < 2^60, infinite or NaN
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    const float s = x * r, y = fmaf(0.5f * r, fmaf(-s, s, x), s);
    return x > 0.f && x < 3e38f ? y : x;
}
__device__ __forceinline__ float sigmoidf_(float v) {   // (below -80 the result is 0 in fp16, and 1 is what it adds to in an exponent)
    return recip_(1.0f + __expf(v < -80.f ? 80.f : -v));
}

constexpr int HEAD = 64;

}  // namespace ab
