// Device-side building blocks shared by the SZx codec kernels.
//
// Everything here is bit-level arithmetic of the SZx stream format
// (szcompressor/SZx) restated for the GPU: IEEE patterns, the logical shifts of
// the reference's unsigned unions (szx/include/szx.h:56-68), big-endian header
// fields (szx/src/szx_BytesToolkit.cc:266-317,460-476) and the scans that place
// variable-length payloads.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace szxg {

constexpr int kWarp = 32;

// Programmatic dependent launch: a kernel launched by launch_after() may be
// scheduled while the kernel before it in the stream still runs; it waits here,
// before its first access to memory, until that kernel has finished, and then
// lets its own successor be scheduled.  (After a plain launch the wait returns
// at once.)
__device__ __forceinline__ void pdl_start() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// ------------------------------------------------------------------ element traits

template <typename T> struct Elem;
template <> struct Elem<float> {
    using U = uint32_t;
    static constexpr int W = 4;          // bytes per word
    static __device__ __forceinline__ U bits(float v) { return __float_as_uint(v); }
    static __device__ __forceinline__ float of(U u) { return __uint_as_float(u); }
    // leading identical bytes of the XOR, szx/src/szx_float.cc:96-101
    static __device__ __forceinline__ int lead(U x) {
        return x < (1u << 8) ? 3 : x < (1u << 16) ? 2 : x < (1u << 24) ? 1 : 0;
    }
    static __device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
    static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
};
template <> struct Elem<double> {
    using U = unsigned long long;
    static constexpr int W = 8;
    static __device__ __forceinline__ U bits(double v) { return (U)__double_as_longlong(v); }
    static __device__ __forceinline__ double of(U u) { return __longlong_as_double((long long)u); }
    // szx/src/szx_double.cc:80-85
    static __device__ __forceinline__ int lead(U x) {
        return x < (1ull << 40) ? 3 : x < (1ull << 48) ? 2 : x < (1ull << 56) ? 1 : 0;
    }
    static __device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
    static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
};

// ------------------------------------------------------------------ x86 NaN rules
//
// The reference runs on x86-64 SSE, where an arithmetic NaN result is the
// first NaN operand, quieted (the second when only it is NaN), an invalid
// operation (inf - inf, 0/0) gives the negative "indefinite" NaN, and
// float<->double conversions keep the payload.  CUDA returns one canonical
// NaN instead.  These helpers restore the x86 result; the hot loops call the
// plain operation and take the fix-up path only when a warp saw a NaN.
// max with NaN propagation (a NaN input gives a NaN), two and three inputs
// (the three-input form is sm_100 and later)
__device__ __forceinline__ float fmax_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float fmax3_nan(float a, float b, float c) {
    float r;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float nan_rule(float a, float b) {
    uint32_t ua = __float_as_uint(a), ub = __float_as_uint(b);
    if ((ua & 0x7FFFFFFFu) > 0x7F800000u) return __uint_as_float(ua | 0x00400000u);
    if ((ub & 0x7FFFFFFFu) > 0x7F800000u) return __uint_as_float(ub | 0x00400000u);
    return __uint_as_float(0xFFC00000u);
}
__device__ __forceinline__ double nan_rule(double a, double b) {
    unsigned long long ua = (unsigned long long)__double_as_longlong(a);
    unsigned long long ub = (unsigned long long)__double_as_longlong(b);
    if ((ua & 0x7FFFFFFFFFFFFFFFull) > 0x7FF0000000000000ull) return __longlong_as_double((long long)(ua | 0x0008000000000000ull));
    if ((ub & 0x7FFFFFFFFFFFFFFFull) > 0x7FF0000000000000ull) return __longlong_as_double((long long)(ub | 0x0008000000000000ull));
    return __longlong_as_double((long long)0xFFF8000000000000ull);
}
__device__ __forceinline__ float xsub(float a, float b) { float r = __fsub_rn(a, b); return r == r ? r : nan_rule(a, b); }
__device__ __forceinline__ float xadd(float a, float b) { float r = __fadd_rn(a, b); return r == r ? r : nan_rule(a, b); }
__device__ __forceinline__ float xmul(float a, float b) { float r = __fmul_rn(a, b); return r == r ? r : nan_rule(a, b); }
__device__ __forceinline__ float xdiv(float a, float b) { float r = __fdiv_rn(a, b); return r == r ? r : nan_rule(a, b); }
// The FP64 pipe of this GPU retires two lanes a clock on an SM (a warp
// instruction holds it for 16 clocks), 1/32 of what the integer pipe does, so
// double code spends it on the additions alone: tests, halving and conversions
// work on the bit pattern, with the plain operation for the rare patterns
// (infinities, NaNs, subnormals) they leave out.
// (the halves are taken by PTX moves: from casts the compiler recognises a
// test for infinity or NaN and makes a double comparison of it)
__device__ __forceinline__ uint32_t hi32(double v) {
    uint32_t r;
    asm("{\n\t.reg .b32 t;\n\tmov.b64 {t, %0}, %1;\n\t}" : "=r"(r) : "d"(v));
    return r;
}
__device__ __forceinline__ uint32_t lo32(double v) {
    uint32_t r;
    asm("{\n\t.reg .b32 t;\n\tmov.b64 {%0, t}, %1;\n\t}" : "=r"(r) : "d"(v));
    return r;
}
__device__ __forceinline__ double from_hi_lo(uint32_t hi, uint32_t lo) {
    return __longlong_as_double((long long)(((unsigned long long)hi << 32) | lo));
}
__device__ __forceinline__ bool inf_or_nan(double v) { return (hi32(v) & 0x7FF00000u) == 0x7FF00000u; }
__device__ __forceinline__ bool inf_or_nan(float v) { return (__float_as_uint(v) & 0x7F800000u) == 0x7F800000u; }
__device__ __forceinline__ bool is_zero(double v) { return ((hi32(v) << 1) | lo32(v)) == 0u; }
__device__ __forceinline__ bool is_zero(float v) { return v == 0.0f; }
__device__ __forceinline__ double xsub(double a, double b) {
    const double r = __dsub_rn(a, b);
    if (!inf_or_nan(r)) return r;
    return r == r ? r : nan_rule(a, b);
}
__device__ __forceinline__ double xadd(double a, double b) {
    const double r = __dadd_rn(a, b);
    if (!inf_or_nan(r)) return r;
    return r == r ? r : nan_rule(a, b);
}
__device__ __forceinline__ double xmul(double a, double b) { double r = __dmul_rn(a, b); return r == r ? r : nan_rule(a, b); }
__device__ __forceinline__ double xdiv(double a, double b) { double r = __ddiv_rn(a, b); return r == r ? r : nan_rule(a, b); }
// x / 2 as a multiplication: both are the correctly rounded value of the same
// real number (subnormal results included), and a NaN x propagates the same
// way, so the result is bit-identical to the division at a fraction of its
// cost.
__device__ __forceinline__ float xhalf(float x) { return xmul(x, 0.5f); }
// (double: the exponent less one, where both x and the half are normal numbers)
__device__ __forceinline__ double xhalf(double x) {
    const uint32_t hi = hi32(x), e = (hi >> 20) & 0x7FFu;
    if (e - 2u <= 2044u) return from_hi_lo(hi - 0x00100000u, lo32(x));
    if (is_zero(x)) return x;
    return xmul(x, 0.5);
}
// cvtsd2ss / cvtss2sd
__device__ __forceinline__ float xd2f(double d) {
    const uint32_t hi = hi32(d), lo = lo32(d), e = (hi >> 20) & 0x7FFu;
    if (e - 897u <= 253u) {   // a normal float (or the overflow to infinity that rounding up makes of it)
        uint32_t u = __funnelshift_l(lo, hi, 3) - 0xC0000000u;       // exponent less 896, the top 23 fraction bits
        u += ((lo & 0x1FFFFFFFu) + 0x0FFFFFFFu + (u & 1u)) >> 29;    // to nearest, ties to even
        return __uint_as_float((u & 0x7FFFFFFFu) | (hi & 0x80000000u));
    }
    if (is_zero(d)) return __uint_as_float(hi);
    if (d == d) return __double2float_rn(d);
    unsigned long long b = (unsigned long long)__double_as_longlong(d);
    return __uint_as_float((uint32_t)(b >> 32 & 0x80000000u) | 0x7FC00000u | (uint32_t)(b >> 29 & 0x7FFFFFu));
}
__device__ __forceinline__ double xf2d(float f) {
    const uint32_t b = __float_as_uint(f), e = (b >> 23) & 0xFFu;
    if (e - 1u <= 253u) return from_hi_lo((b & 0x80000000u) | (((b & 0x7FFFFFFFu) >> 3) + 0x38000000u), b << 29);
    if ((b << 1) == 0u) return from_hi_lo(b, 0u);
    if (f == f) return (double)f;
    return __longlong_as_double((long long)(((unsigned long long)(b & 0x80000000u) << 32) | 0x7FF8000000000000ull |
                                            ((unsigned long long)(b & 0x7FFFFFu) << 29)));
}
template <typename T> __device__ __forceinline__ T widen_median(float m);
template <> __device__ __forceinline__ float widen_median<float>(float m) { return m; }
template <> __device__ __forceinline__ double widen_median<double>(float m) { return xf2d(m); }

// getExponent_float / getPrecisionReqLength_double, szx/src/szx_BytesToolkit.cc:335-387
__device__ __forceinline__ int exponent_f32(float v) { return (int)((__float_as_uint(v) & 0x7F800000u) >> 23) - 127; }
__device__ __forceinline__ int exponent_f64_of_f32(float v) {
    unsigned long long b = (unsigned long long)__double_as_longlong((double)v);
    return (int)((b & 0x7FF0000000000000ull) >> 52) - 1023;
}
// computeReqLength_float (szx/src/szx_float.cc:1708-1717) / _double
// (szx/src/szx_double.cc:2020-2031).  Returns reqLength; *zero_median set when
// the clamp at the word width zeroes the stored median.
// The bound's exponent (exponent_f64_of_f32(eb)) is a per-field constant:
// callers that place many blocks under one bound compute it once and use the
// eb_exp overloads.
template <typename T> __device__ __forceinline__ int req_length_e(int eb_exp, float radius, bool* zero_median);
template <> __device__ __forceinline__ int req_length_e<float>(int eb_exp, float radius, bool* zm) {
    int r = 10 + exponent_f32(radius) - eb_exp;
    *zm = false;
    if (r < 9) r = 9;
    if (r > 32) { r = 32; *zm = true; }
    return r;
}
template <> __device__ __forceinline__ int req_length_e<double>(int eb_exp, float radius, bool* zm) {
    int r = 12 + exponent_f32(radius) - eb_exp;
    *zm = false;
    if (r < 12) r = 12;
    if (r > 64) { r = 64; *zm = true; }
    return r;
}
template <typename T> __device__ __forceinline__ int req_length(float eb, float radius, bool* zero_median) {
    return req_length_e<T>(exponent_f64_of_f32(eb), radius, zero_median);
}
// Stored-byte counts of four values, max(R - lead, 0) per byte, for leads in
// 0..3 and R in 1..8 (what __vsubus4(R * 0x01010101, leads) returns) without
// the emulated SIMD instruction: R is raised by the bytes whose lead exceeds
// it (lead 3 when R <= 2, lead >= 2 when R == 1) so the subtraction never
// borrows across bytes.
__device__ __forceinline__ uint32_t stored_counts(int R, uint32_t ldb) {
    const uint32_t hi = (ldb >> 1) & 0x01010101u;   // lead >= 2
    const uint32_t l3 = ldb & hi;                   // lead == 3
    uint32_t up = R <= 2 ? l3 : 0u;
    if (R <= 1) up += hi;
    return (uint32_t)R * 0x01010101u + up - ldb;
}
__device__ __forceinline__ void split_reqlen(int reqLength, int* R, int* s) {
    int rb = reqLength & 7;
    *R = (reqLength >> 3) + (rb != 0);
    *s = rb ? 8 - rb : 0;
}

// 16 lead codes as stored (4 to a byte, MSB first), one bit of each pair set:
// moved to value order, value e's bit (its pair's low one) to position 2e+1
__device__ __forceinline__ uint32_t vorder(uint32_t m) { return __byte_perm(__brev(m), 0, 0x0123); }
// byte i of x, zero-extended
__device__ __forceinline__ uint32_t byte_of(uint32_t x, int i) { return __byte_perm(x, 0, 0x4440 | i); }

// ------------------------------------------------------------------ warp scans

__device__ __forceinline__ unsigned lane_id() { return threadIdx.x & 31; }

template <typename V>
__device__ __forceinline__ V warp_inclusive_sum(V v) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        V o = __shfl_up_sync(0xffffffffu, v, d);
        if ((int)lane_id() >= d) v += o;
    }
    return v;
}
template <typename V>
__device__ __forceinline__ V warp_sum(V v) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    return v;
}

// ------------------------------------------------------------------ decoupled look-back
//
// Single-pass exclusive prefix over tiles (Merrill & Garland, "Single-pass
// Parallel Prefix Scan with Decoupled Look-back", NVR-2016-002).  Tiles are
// taken in order from an atomic counter, so every predecessor is running or
// done and the look-back always ends; the spin is still capped and reports
// through *err instead of hanging.

constexpr unsigned kSpinLimit = 1u << 22;   // polls before giving up (~1 s with backoff)
// Every look-back below takes its poll limit as a last argument (default
// kSpinLimit); the failure-detection self-test (selftest.cu) passes a small
// one and withholds a tile, so the give-up path runs for real.  (The placement
// window has no waits of its own: it is read again kWinRepolls times, then one
// of them takes over.)

enum : int { kErrNone = 0, kErrLookback = 1, kErrCapacity = 2, kErrStream = 3 };

// Three 21-bit fields combined by max each (latest tile index + 1, 0 = none).
struct Max3x21Op {
    static __device__ __forceinline__ unsigned long long id() { return 0; }
    static __device__ __forceinline__ unsigned long long op(unsigned long long x, unsigned long long y) {
        unsigned long long r = 0;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            unsigned long long a = (x >> (21 * k)) & 0x1FFFFF, b = (y >> (21 * k)) & 0x1FFFFF;
            r |= (a > b ? a : b) << (21 * k);
        }
        return r;
    }
};

// ------------------------------------------------------------------ TMA bulk copies + mbarriers
//
// One thread arms an mbarrier with the byte count and issues a 1-D bulk copy
// (cp.async.bulk) global -> shared; consumers wait on the barrier's phase.
// Source, destination and size must be multiples of 16 bytes.

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// Raise the transaction count the current phase waits for, without arriving.
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, uint32_t bytes) {
    asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tma_load_1d(void* dst, const void* src, uint32_t bytes, unsigned long long* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: gives up (returns false) after kSpinLimit polls.
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, uint32_t parity) {
    for (unsigned i = 0; i < (1u << 22); i++) {
        if (mbar_try_wait(bar, parity)) return true;
        if (i > 16) __nanosleep(64);
    }
    return false;
}

__device__ __forceinline__ uint4 ld_volatile_v4(const uint32_t* p) {
    uint4 v;
    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p)
                 : "memory");
    return v;
}

// ------------------------------------------------------------------ inline-prefix look-back
//
// One 64-bit status word per tile: [63:62] flag (0 empty, 1 aggregate,
// 2 inclusive), [61:0] the tile's byte count (aggregate) or the inclusive
// prefix itself.  Resolving a tile is then one memory round trip per window
// of 128 predecessors (4 words per lane), with no second load for the prefix.
constexpr unsigned long long kS64Agg = 1ull << 62, kS64Inc = 2ull << 62, kS64Val = (1ull << 62) - 1;

// Status words are read and written with relaxed GPU-scope accesses: every
// party is on this GPU, and system scope (what `volatile` means) costs far
// more on a coherent CPU-GPU node.
__device__ __forceinline__ void st_volatile64(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_volatile64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void ld_volatile_v2x2(const unsigned long long* p, unsigned long long (&w)[4]) {
    unsigned long long a, b, c, d;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0,%1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0,%1}, [%2];" : "=l"(c), "=l"(d) : "l"(p + 2) : "memory");
    w[0] = a; w[1] = b; w[2] = c; w[3] = d;
}

// Lane 0 publishes the tile's aggregate (tile 0 publishes its inclusive value).
__device__ __forceinline__ void prefix_publish(unsigned long long* st, long long tile, unsigned long long agg) {
    if (lane_id() != 0) return;
    st_volatile64(&st[tile], (tile == 0 ? kS64Inc : kS64Agg) | (agg & kS64Val));
}

// Whole warp: exclusive prefix of `tile` (aggregate already published), then
// publish its inclusive value.  `st` holds ntiles + 4 zeroed words.
__device__ __forceinline__ unsigned long long prefix_resolve(unsigned long long* st, long long tile,
                                                            unsigned long long agg, int* err,
                                                            unsigned limit = kSpinLimit) {
    if (tile == 0) return 0;
    const unsigned lane = lane_id();
    unsigned long long pa = 0;
    long long g0 = ((tile - 1) >> 2) << 2;
    unsigned spins = 0;
    bool failed = false;
    while (true) {
        const long long g = g0 - 4 * (long long)lane;
        unsigned long long w[4];
        if (g >= 0) ld_volatile_v2x2(st + g, w);
        else { w[0] = w[1] = w[2] = w[3] = kS64Inc; }
        int inc_j = -1;
        bool ready = true;
        unsigned long long sa = 0;
#pragma unroll
        for (int j = 3; j >= 0; j--) {
            const unsigned long long f = w[j] & ~kS64Val;
            if (g + j < tile && inc_j < 0) {
                if (f == kS64Inc) { inc_j = j; sa += w[j] & kS64Val; }
                else { ready = ready && f != 0; sa += w[j] & kS64Val; }
            }
        }
        const unsigned inc_mask = __ballot_sync(0xffffffffu, inc_j >= 0);
        const unsigned stop = inc_mask ? (unsigned)__ffs(inc_mask) - 1 : 31u;
        const unsigned window = stop == 31u ? 0xffffffffu : ((1u << (stop + 1)) - 1);
        if (__ballot_sync(0xffffffffu, !ready) & window) {
            if (++spins > limit) { failed = true; break; }
            __nanosleep(spins < 64 ? 32 : 256);
            continue;
        }
        pa += warp_sum(lane <= stop ? sa : 0ull);
        if (inc_mask) break;
        g0 -= 128;
    }
    if (failed && lane == 0) atomicExch(err, kErrLookback);
    if (lane == 0) st_volatile64(&st[tile], kS64Inc | ((pa + agg) & kS64Val));
    return pa;
}

// The same by the whole CTA, WARPS windows of 128 predecessors in one memory
// round trip; every thread gets the prefix.  For grids of fewer than 128 *
// WARPS CTAs that hold one tile each: the tiles without an inclusive prefix are
// then fewer than the windows reach (read again until one is seen).  sm: WARPS
// words; a barrier lies between two calls.  st needs the alignment of its words
// only: a decoder's workspace may lie at any multiple of 8.
template <int WARPS>
__device__ __forceinline__ unsigned long long prefix_resolve_cta(unsigned long long* st, long long tile,
                                                                 unsigned long long agg, int* err,
                                                                 unsigned long long* sm,
                                                                 unsigned limit = kSpinLimit) {
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    const long long g0 = (((tile - 1) >> 2) << 2) - 128 * (long long)warp, g = g0 - 4 * (long long)lane;
    unsigned long long pa = 0;
    bool done = false;
    unsigned spins = 0;
    for (unsigned round = 0; !done && round < limit; round++) {   // (the same rounds in every thread)
        if (round) __syncthreads();   // (the sums of the round before are read)
        unsigned long long mine = kS64Inc;   // this warp's window: its sum, and kS64Inc where a prefix ends it
        while (tile > 0 && g0 >= 0) {
            unsigned long long w[4] = {kS64Inc, kS64Inc, kS64Inc, kS64Inc};
            if (g >= 0) {
                if (((uintptr_t)st & 15) == 0) {
                    ld_volatile_v2x2(st + g, w);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; j++) w[j] = ld_volatile64(st + g + j);
                }
            }
            bool inc = false, ready = true;
            unsigned long long sa = 0;
#pragma unroll
            for (int j = 3; j >= 0; j--) {
                const unsigned long long f = w[j] & ~kS64Val;
                if (g + j < tile && !inc) {
                    sa += w[j] & kS64Val;
                    inc = f == kS64Inc;
                    ready = ready && f != 0;
                }
            }
            const unsigned inc_mask = __ballot_sync(0xffffffffu, inc);
            const unsigned stop = inc_mask ? (unsigned)__ffs(inc_mask) - 1 : 31u;
            if (!(__ballot_sync(0xffffffffu, !ready) & (0xffffffffu >> (31 - stop)))) {
                mine = (inc_mask ? kS64Inc : 0ull) | (warp_sum(lane <= stop ? sa : 0ull) & kS64Val);
                break;
            }
            if (++spins > limit) {   // (its window counts as an empty prefix: the walk ends, the error stands)
                if (lane == 0) atomicExch(err, kErrLookback);
                break;
            }
            __nanosleep(spins < 64 ? 32 : 256);
        }
        if (lane == 0) sm[warp] = mine;
        __syncthreads();
        pa = 0;
#pragma unroll
        for (int k = 0; k < WARPS; k++) {
            const unsigned long long v = sm[k];
            if (!done) pa += v & kS64Val;
            done = done || (v & ~kS64Val) != 0;
        }
    }
    if (!done && threadIdx.x == 0) atomicExch(err, kErrLookback);
    if (threadIdx.x == 0 && tile > 0) st_volatile64(&st[tile], kS64Inc | ((pa + agg) & kS64Val));
    return pa;
}

// One pass of cta_copy_realign for a word phase of WS: 16 destination bytes
// are words WS .. WS+4 of two 16-byte staging chunks, shifted by rs bits.
// sp: shared address of the first of n full destination chunks' staging chunk.
template <int WS>
__device__ __forceinline__ void copy_realign_chunks(uint32_t sp, uint8_t* gp, uint32_t n, uint32_t rs, uint32_t tid,
                                                    uint32_t nthr) {
    sp += 16 * tid;
    gp += 16 * tid;
    for (uint32_t c = tid; c < n; c += nthr, sp += 16 * nthr, gp += 16 * nthr) {
        uint32_t a[8];
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(sp) : "memory");
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4+16];"
                     : "=r"(a[4]), "=r"(a[5]), "=r"(a[6]), "=r"(a[7]) : "r"(sp) : "memory");
        *(uint4*)gp = make_uint4(__funnelshift_r(a[WS], a[WS + 1], rs), __funnelshift_r(a[WS + 1], a[WS + 2], rs),
                                 __funnelshift_r(a[WS + 2], a[WS + 3], rs), __funnelshift_r(a[WS + 3], a[WS + 4], rs));
    }
}

// Copy n bytes from a 16-aligned staging buffer (data at offset 0, 32 bytes
// of slack behind it) to global dst of any alignment with threads tid = 0 ..
// nthr - 1 of the CTA (nthr a multiple of 32): 16-byte aligned stores, the
// staging bytes realigned with funnel shifts; byte copies at the ragged ends.
// The staging side is read as aligned 16-byte chunks (8 shared-memory
// wavefronts per warp and 512 bytes; five 4-byte reads at a 16-byte stride
// take 20): the phase between the two sides is the same for every chunk, so
// its word part is a branch of the whole CTA.
__device__ __forceinline__ void cta_copy_realign(const uint8_t* stg, uint32_t n, uint8_t* dst, uint32_t tid,
                                                 uint32_t nthr) {
    if (n == 0) return;
    const uint32_t head = (0u - (uint32_t)(uintptr_t)dst) & 15u;   // bytes before dst's first 16-byte boundary
    const uint32_t h = head < n ? head : n, full = (n - h) >> 4, tail = h + 16 * full;
    const uint32_t sp = smem_u32(stg), rs = (head & 3u) * 8u;
    uint8_t* gp = dst + h;
    switch (head >> 2) {
        case 0: copy_realign_chunks<0>(sp, gp, full, rs, tid, nthr); break;
        case 1: copy_realign_chunks<1>(sp, gp, full, rs, tid, nthr); break;
        case 2: copy_realign_chunks<2>(sp, gp, full, rs, tid, nthr); break;
        default: copy_realign_chunks<3>(sp, gp, full, rs, tid, nthr); break;
    }
    // lanes 0-15 the bytes before the first full chunk, lanes 16-31 those after the last
    if (tid < 32) {
        const uint32_t k = tid < 16 ? tid : tail + tid - 16;
        if (k < (tid < 16 ? h : n)) dst[k] = stg[k];
    }
}

// 16-byte asynchronous global -> shared copies (cp.async, the LSU path: they
// do not queue behind the TMA unit's bulk copies), L2 only.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem)), "l"(gmem) : "memory");
}
template <int BYTES>   // 4 or 8, for data that is not 16-byte aligned
__device__ __forceinline__ void cp_async_small(void* smem, const void* gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(smem)), "l"(gmem), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// wait until at most N of this thread's committed groups are still in flight
template <int N>
__device__ __forceinline__ void cp_async_wait_group() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void st_relaxed16(uint16_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u16 [%0], %1;" ::"l"(p), "h"((unsigned short)v) : "memory");
}

// Lane-predicated claim of the next tile: the reply is waited for where `next`
// is used, not at the end of a branch.
__device__ __forceinline__ void claim_tile(unsigned long long& next, unsigned long long* ctr, bool take) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p atom.relaxed.gpu.global.add.u64 %0, [%1], 1;\n\t}"
                 : "+l"(next)
                 : "l"(ctr), "r"((uint32_t)take)
                 : "memory");
}

// ------------------------------------------------------------------ placement window
//
// How the persistent encoders place a tile: its offset is the inclusive prefix
// of this CTA's previous tile (the anchor, known here) plus the byte counts of
// the tiles claimed between the two, read from 16-bit words (count + 1, 0: not
// yet published) that one warp copies into shared memory well before it needs
// them.  A tile without an anchor within kLbWin tiles of the same field, or
// with counts still missing after a few re-reads, falls back to the global
// look-back over the 64-bit status words (prefix_resolve), which every
// placement keeps valid by publishing its inclusive prefix.
//
// kLbWin (2 KiB of counts): a CTA's previous tile is one launch's CTAs back on
// average (456 or 608), further for a CTA that lags; 512 sent a third of the
// lagging CTAs' tiles to the global walk.
constexpr int kLbWin = 1024;
constexpr int kWinRepolls = 32;   // window re-reads before the global look-back walk
struct PlaceWin {   // shared memory; one warp's own
    __align__(16) uint16_t w16[kLbWin + 8];
    unsigned long long an_incl;   // the anchor's inclusive prefix
    int an_t, an_f, lo, ok;       // anchor tile (-1: none), its field; the window's first tile and state
    __device__ __forceinline__ void init() {   // one thread
        an_t = -1;
        an_f = -1;
        an_incl = 0;
        ok = 0;
    }
    __device__ __forceinline__ void anchor(int f, int t, unsigned long long incl) {   // lane 0
        an_t = t;
        an_f = f;
        an_incl = incl;
    }
    // whole warp: start copying the window of tile t of field f (counts agg)
    __device__ __forceinline__ void issue(const uint16_t* agg, int f, int t) {
        const int lane = (int)lane_id(), a = an_t;
        int state = 0, first = 0;
        if (t > 0 && a >= 0 && an_f == f && a < t && t - a - 1 <= kLbWin) {
            if (t - a == 1) {
                state = 2;
            } else {
                first = (a + 1) & ~7;
                const int units = (t - first + 7) >> 3;
                for (int u = lane; u < units; u += 32) cp_async16(&w16[8 * u], agg + first + 8 * u);
                state = 1;
            }
        }
        if (lane == 0) {
            lo = first;
            ok = state;
        }
        __syncwarp();
    }
    // whole warp: tile t's offset from the window, false when it has to come
    // from the global look-back
    __device__ __forceinline__ bool offset(const uint16_t* agg, int t, unsigned long long* base) {
        *base = 0;
        if (t == 0) return true;
        const int state = ok, at0 = an_t;
        const unsigned long long incl = an_incl;
        *base = incl;
        if (state == 2) return true;
        if (state != 1) return false;
        // Sum of the counts of tiles an_t + 1 .. t - 1, eight to a 16-byte
        // read and a redux across the warp; the words outside that range count
        // as 1, published and empty.
        const int lane = (int)lane_id(), l = lo, units = (t - l + 7) >> 3, first = at0 + 1 - l, last = t - l;
        cp_async_wait_all();
        __syncwarp();
        for (int attempt = 0;; attempt++) {
            uint32_t sum = 0, least = ~0u;
            for (int u = lane; u < units; u += 32) {
                const uint4 q = *(const uint4*)&w16[8 * u];
                uint32_t w[4] = {q.x, q.y, q.z, q.w};
                if (u == 0 || u == units - 1) {
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const int at = 8 * u + i, sh = 16 * (i & 1);
                        if (at < first || at >= last) w[i >> 1] = (w[i >> 1] & ~(0xFFFFu << sh)) | (1u << sh);
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    sum = __dp2a_lo(w[i], 0x0101u, sum);
                    least = __vminu2(least, w[i]);
                }
                sum -= 8;
            }
            if (__all_sync(0xffffffffu, (least & 0xFFFFu) != 0 && least >= 0x10000u)) {
                *base = incl + __reduce_add_sync(0xffffffffu, sum);
                return true;
            }
            if (attempt == kWinRepolls) return false;
            __nanosleep(64);
            const uint32_t* src = (const uint32_t*)(agg + l);
            __syncwarp();
            for (int u = lane; u < units; u += 32) *(uint4*)&w16[8 * u] = ld_volatile_v4(src + 4 * u);
            __syncwarp();
        }
    }
};
}  // namespace szxg
