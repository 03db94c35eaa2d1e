// Segment helpers shared by the blocked codec kernels: a block of up to G*E
// values is handled by a segment of G lanes of a warp (G a power of two),
// E = 16 float / 8 double values per lane: a run of consecutive values (codec)
// or chunks of 4 values dealt out in turn (constant blocks, fixed-rate sampling).
#pragma once
#include "common.cuh"

namespace szxg {

// Reductions and scans run inside segments with shuffle widths of G, so
// several blocks share one warp instruction and the per-block work is
// replicated G times, not 32.

template <typename T> struct EncCfg;
template <> struct EncCfg<float> { static constexpr int E = 16; };    // values per lane
template <> struct EncCfg<double> { static constexpr int E = 8; };

// high word of a double's order-preserving signed key (its own inverse)
__device__ __forceinline__ int dkey_hi(uint32_t h) { return (int)(h ^ ((uint32_t)((int)h >> 31) & 0x7FFFFFFFu)); }

template <int G, typename V>
__device__ __forceinline__ V seg_sum(V v) {
#pragma unroll
    for (int d = G / 2; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d, G);
    return v;
}
template <int G, typename V>
__device__ __forceinline__ V seg_inclusive_sum(V v) {
    const int sl = (int)(lane_id() & (G - 1));
#pragma unroll
    for (int d = 1; d < G; d <<= 1) {
        V o = __shfl_up_sync(0xffffffffu, v, d, G);
        if (sl >= d) v += o;
    }
    return v;
}

// Chunked lane layout.  A block is split into chunks of 4 values (one lead
// byte each); lane sl of a G-lane segment owns chunks sl, sl+G, sl+2G, ...
// so consecutive lanes touch consecutive chunks (no shared-memory bank
// conflicts) while each chunk stays contiguous for the XOR chain.
template <typename T, int G>
struct Chunks {
    static constexpr int E = EncCfg<T>::E;
    static constexpr int NC = E / 4;                  // chunks per lane
    // first value of the lane's k-th chunk
    static __device__ __forceinline__ int first(int sl, int k) { return 4 * (sl + k * G); }
};

// Run layout: lane sl owns the E consecutive values from E*sl on (64 bytes).
template <typename T, int G>
struct Runs {
    static constexpr int E = EncCfg<T>::E;
    static __device__ __forceinline__ int first(int sl, int k) { return E * sl + 4 * k; }
};

// Tiles of values in shared memory hold their 16-byte chunks swizzled: chunk c
// lies at chunk c ^ ((c >> 3) & 3), so that the eight lanes of a quarter warp
// that read one chunk each of eight consecutive 64-byte runs touch all 32
// banks (unswizzled, such a read is 4-way conflicted).
__device__ __forceinline__ uint32_t swz16(uint32_t c) { return c ^ ((c >> 3) & 3u); }
// byte offset of value i in a swizzled tile
template <typename T>
__device__ __forceinline__ uint32_t swz_off(uint32_t i) {
    constexpr uint32_t VN = 16 / sizeof(T);
    return swz16(i / VN) * 16 + (i % VN) * (uint32_t)sizeof(T);
}

// Run `row` (64 bytes) of a swizzled tile at shared address `tile`, a multiple
// of 64: the swizzle is one exclusive-or on the address per 16-byte chunk.
template <typename T>
__device__ __forceinline__ void load_run_full(uint32_t tile, uint32_t row, T (&v)[EncCfg<T>::E]) {
    const uint32_t p = tile + 64 * row + 8 * (row & 6u);   // chunk 0 of the run: chunk (row >> 1) & 3 of its 64 bytes
#pragma unroll
    for (int j = 0; j < 4; j++) {
        if constexpr (sizeof(T) == 4)
            asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];"
                         : "=f"(v[4 * j]), "=f"(v[4 * j + 1]), "=f"(v[4 * j + 2]), "=f"(v[4 * j + 3])
                         : "r"(p ^ (16u * j))
                         : "memory");
        else
            asm volatile("ld.shared.v2.f64 {%0,%1}, [%2];" : "=d"(v[2 * j]), "=d"(v[2 * j + 1]) : "r"(p ^ (16u * j)) : "memory");
    }
}

// A lane's run of the block that starts at value e0 of a swizzled tile.  vec:
// blocks start on 16-byte boundaries.  Values past the block's end are what
// lies there (the caller masks them); the reads stay inside a tile of
// G*E-value blocks.
template <typename T, int G>
__device__ __forceinline__ void load_run(const uint8_t* tile, uint32_t e0, bool vec, T (&v)[EncCfg<T>::E]) {
    constexpr int E = EncCfg<T>::E;
    constexpr uint32_t VN = 16 / sizeof(T);
    const uint32_t f = e0 + E * (lane_id() & (G - 1));
    if (vec) {
        const uint32_t c0 = f / VN;
#pragma unroll
        for (uint32_t j = 0; j < E / VN; j++) {
            const uint8_t* p = tile + swz16(c0 + j) * 16;
            if constexpr (sizeof(T) == 4) {
                const float4 q = *(const float4*)p;
                v[4 * j] = q.x; v[4 * j + 1] = q.y; v[4 * j + 2] = q.z; v[4 * j + 3] = q.w;
            } else {
                const double2 q = *(const double2*)p;
                v[2 * j] = q.x; v[2 * j + 1] = q.y;
            }
        }
    } else {
#pragma unroll
        for (int e = 0; e < E; e++) v[e] = *(const T*)(tile + swz_off<T>(f + e));
    }
}

template <typename T, int G>
__device__ __forceinline__ void load_chunks(const T* xs, int len, bool vec, T (&v)[EncCfg<T>::E]) {
    using C = Chunks<T, G>;
    const int sl = (int)(lane_id() & (G - 1));
#pragma unroll
    for (int k = 0; k < C::NC; k++) {
        const int f = C::first(sl, k);
        if (vec && f + 4 <= len) {
            if constexpr (sizeof(T) == 4) {
                const float4 q = *(const float4*)(xs + f);
                v[4 * k] = q.x; v[4 * k + 1] = q.y; v[4 * k + 2] = q.z; v[4 * k + 3] = q.w;
            } else {
                const double2 a = *(const double2*)(xs + f), b = *(const double2*)(xs + f + 2);
                v[4 * k] = a.x; v[4 * k + 1] = a.y; v[4 * k + 2] = b.x; v[4 * k + 3] = b.y;
            }
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) v[4 * k + i] = f + i < len ? xs[f + i] : (T)0;
        }
    }
}


template <typename T, int G>
__device__ __forceinline__ void store_chunks(T* ob, int len, bool vec, const T (&v)[EncCfg<T>::E]) {
    using C = Chunks<T, G>;
    const int sl = (int)(lane_id() & (G - 1));
#pragma unroll
    for (int k = 0; k < C::NC; k++) {
        const int f = C::first(sl, k);
        if (vec && f + 4 <= len) {
            if constexpr (sizeof(T) == 4) {
                *(float4*)(ob + f) = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
            } else {
                *(double2*)(ob + f) = make_double2(v[4 * k], v[4 * k + 1]);
                *(double2*)(ob + f + 2) = make_double2(v[4 * k + 2], v[4 * k + 3]);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (f + i < len) ob[f + i] = v[4 * k + i];
        }
    }
}

// Three-input forms (sm_100 and later): NaN inputs are ignored like fminf /
// fmaxf (fmax_nan / fmax3_nan, which propagate them, are in common.cuh).
__device__ __forceinline__ float fmin3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
// bytes [0, n) of a word set (n <= 0: none, n >= 4: all)
__device__ __forceinline__ uint32_t low_bytes_mask(int n) {
    return n >= 4 ? 0xFFFFFFFFu : (n <= 0 ? 0u : 0xFFFFFFFFu >> (32 - 8 * n));
}

// Segment-wide min/max with the reference's sequential semantics
// (szx/src/szx_float.cc:322-345): the first value reaching an extreme wins,
// NaNs are skipped unless the block's first value is NaN.  `special` is set
// (segment-uniform) when the block holds a NaN or an infinity, where the
// x86 NaN rules of the subtraction matter.  C: the lanes' layout (Chunks or
// Runs).
template <typename T, int G, bool FULL, typename C = Chunks<T, G>>
__device__ __forceinline__ void seg_minmax(const T (&v)[EncCfg<T>::E], int len, T& mn, T& mx, bool& special) {
    constexpr int E = C::E;
    const int sl = (int)(lane_id() & (G - 1));
    if constexpr (sizeof(T) == 4) {
        float lo = __builtin_huge_valf(), hi = -__builtin_huge_valf(), hn = -__builtin_huge_valf();
        if constexpr (FULL) {
#pragma unroll
            for (int e = 0; e < E; e += 2) {
                lo = fmin3(lo, v[e], v[e + 1]);
                hi = fmax3(hi, v[e], v[e + 1]);
                hn = fmax3_nan(hn, v[e], v[e + 1]);
            }
        } else {
#pragma unroll
            for (int e = 0; e < E; e++) {
                if (C::first(sl, e / 4) + (e & 3) < len) {
                    lo = fminf(lo, v[e]);
                    hi = fmaxf(hi, v[e]);
                    hn = fmax_nan(hn, v[e]);
                }
            }
        }
#pragma unroll
        for (int d = G / 2; d > 0; d >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, d, G));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, d, G));
        }
        mn = lo;
        mx = hi;
        // a NaN anywhere in the segment: one vote instead of a reduction
        const unsigned seg0 = lane_id() & ~(unsigned)(G - 1);
        const unsigned segmask = G == 32 ? 0xffffffffu : (((1u << G) - 1) << seg0);
        special = (__ballot_sync(0xffffffffu, isnan(hn)) & segmask) != 0 || isinf(lo) || isinf(hi);
    } else {
        // Order-preserving integer keys, high words first: the extremes of
        // the 32-bit high keys, then of the low words beside them -- 32-bit
        // operations throughout, about half of what 64-bit keys cost.  Any
        // infinity or NaN shows in the high extremes.
        int khn = 0x7FFFFFFF, khx = (int)0x80000000;
#pragma unroll
        for (int e = 0; e < E; e++) {
            const int k = dkey_hi(hi32(v[e]));
            const bool in = FULL || C::first(sl, e / 4) + (e & 3) < len;
            khn = in ? min(khn, k) : khn;
            khx = in ? max(khx, k) : khx;
        }
#pragma unroll
        for (int d = G / 2; d > 0; d >>= 1) {
            khn = min(khn, __shfl_xor_sync(0xffffffffu, khn, d, G));
            khx = max(khx, __shfl_xor_sync(0xffffffffu, khx, d, G));
        }
        const bool odd = khx >= 0x7FF00000 || khn <= (int)0x800FFFFF;
        if (!__any_sync(0xffffffffu, odd)) {
            uint32_t kln = 0xFFFFFFFFu, klx = 0u;
#pragma unroll
            for (int e = 0; e < E; e++) {
                const uint32_t h = hi32(v[e]), l = lo32(v[e]) ^ (uint32_t)((int)h >> 31);
                const int k = dkey_hi(h);
                const bool in = FULL || C::first(sl, e / 4) + (e & 3) < len;
                if (in && k == khn) kln = min(kln, l);
                if (in && k == khx) klx = max(klx, l);
            }
#pragma unroll
            for (int d = G / 2; d > 0; d >>= 1) {
                kln = min(kln, __shfl_xor_sync(0xffffffffu, kln, d, G));
                klx = max(klx, __shfl_xor_sync(0xffffffffu, klx, d, G));
            }
            mn = from_hi_lo((uint32_t)dkey_hi((uint32_t)khn), kln ^ (uint32_t)(khn >> 31));
            mx = from_hi_lo((uint32_t)dkey_hi((uint32_t)khx), klx ^ (uint32_t)(khx >> 31));
            special = false;
        } else {
        long long lo = 0x7FFFFFFFFFFFFFFFll, hi = (long long)0x8000000000000000ull;
        bool nan = false;
#pragma unroll
        for (int e = 0; e < E; e++) {
            const unsigned long long u = (unsigned long long)__double_as_longlong(v[e]);
            const bool in = FULL || C::first(sl, e / 4) + (e & 3) < len;
            const bool fin = (u & 0x7FFFFFFFFFFFFFFFull) <= 0x7FF0000000000000ull;
            const long long k = (long long)(u ^ ((unsigned long long)((long long)u >> 63) & 0x7FFFFFFFFFFFFFFFull));
            if (in && fin) {
                lo = k < lo ? k : lo;
                hi = k > hi ? k : hi;
            }
            nan |= in && !fin;
        }
#pragma unroll
        for (int d = G / 2; d > 0; d >>= 1) {
            const long long a = __shfl_xor_sync(0xffffffffu, lo, d, G), b = __shfl_xor_sync(0xffffffffu, hi, d, G);
            lo = a < lo ? a : lo;
            hi = b > hi ? b : hi;
        }
        auto inv = [](long long k) {
            const unsigned long long u = (unsigned long long)k;
            return __longlong_as_double((long long)(u ^ ((unsigned long long)(k >> 63) & 0x7FFFFFFFFFFFFFFFull)));
        };
        mn = inv(lo);
        mx = inv(hi);
        const unsigned nm = __ballot_sync(0xffffffffu, nan);
        const unsigned seg0 = lane_id() & ~(unsigned)(G - 1);
        const unsigned segmask = G == 32 ? 0xffffffffu : (((1u << G) - 1) << seg0);
        special = (nm & segmask) != 0 || isinf(mn) || isinf(mx);
        }
    }
    // a zero extreme takes the sign of the block's first zero; only warps
    // that met one pay for the search
    if (__any_sync(0xffffffffu, is_zero(mn) || is_zero(mx))) {
        int zi = 1 << 30;
        T zv = 0;
#pragma unroll
        for (int e = E - 1; e >= 0; e--) {
            const int idx = C::first(sl, e / 4) + (e & 3);
            if ((FULL || idx < len) && is_zero(v[e]) && idx < zi) { zi = idx; zv = v[e]; }
        }
        int best = zi;
#pragma unroll
        for (int d = G / 2; d > 0; d >>= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, d, G));
        const unsigned m = __ballot_sync(0xffffffffu, zi == best && zi < (1 << 30));
        const unsigned seg0 = lane_id() & ~(unsigned)(G - 1);
        const unsigned segmask = G == 32 ? 0xffffffffu : (((1u << G) - 1) << seg0);
        const unsigned mm = m & segmask;
        const T first = __shfl_sync(0xffffffffu, zv, mm ? __ffs(mm) - 1 : (int)seg0);
        if (mm) {
            if (is_zero(mn)) mn = first;
            if (is_zero(mx)) mx = first;
        }
    }
    // a NaN first value pins both extremes; only a block holding a NaN can have one
    if (__any_sync(0xffffffffu, special)) {
        const T x0 = __shfl_sync(0xffffffffu, v[0], 0, G);
        if (isnan(x0)) { mn = x0; mx = x0; }
    }
}


// Lead codes of a block's shifted words (szx/src/szx_float.cc:94-113,
// szx/src/szx_double.cc:78-97): per chunk of the lane, the leading identical
// bytes (capped at 3) of each value with its predecessor in block order
// (zero before the block), value i of the chunk in byte i.
template <typename T, int G>
__device__ __forceinline__ void seg_lead_bytes(const typename Elem<T>::U (&cur)[EncCfg<T>::E],
                                               uint32_t (&ldb)[EncCfg<T>::E / 4]) {
    using U = typename Elem<T>::U;
    constexpr int NC = EncCfg<T>::E / 4;
    const int sl = (int)(lane_id() & (G - 1));
    U wrap = 0;   // lane 0: the last lane's value of the previous round (zero before the block)
#pragma unroll
    for (int k = 0; k < NC; k++) {
        // value before this chunk: the previous lane's chunk k, or for lane 0
        // the last lane's chunk k-1 -- one rotation per round serves both
        const U rot = __shfl_sync(0xffffffffu, cur[4 * k + 3], (sl + G - 1) & (G - 1), G);
        const U prev = sl ? rot : wrap;
        wrap = rot;
        uint32_t b = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const U xr = cur[4 * k + i] ^ (i ? cur[4 * k + i - 1] : prev);
            uint32_t lz;
            if constexpr (sizeof(T) == 4) lz = (uint32_t)__clz(xr | 0xFFu) >> 3;
            else lz = (uint32_t)__clzll((long long)(xr | 0xFFFFFFFFFFull)) >> 3;
            b |= lz << (8 * i);
        }
        ldb[k] = b;
    }
}

// Differences of a run from the median, as bit patterns: floats two to an
// instruction (add.f32x2 rounds each half like the scalar addition of -med).
template <int N>
__device__ __forceinline__ void sub_run(const float (&v)[N], float med, uint32_t (&d)[N]) {
    const float nm = -med;
#pragma unroll
    for (int e = 0; e < N; e += 2)
        asm("{\n\t.reg .b64 a, b;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %4};\n\tadd.rn.f32x2 a, a, b;\n\t"
            "mov.b64 {%0, %1}, a;\n\t}"
            : "=r"(d[e]), "=r"(d[e + 1])
            : "f"(v[e]), "f"(v[e + 1]), "f"(nm));
}
template <int N>
__device__ __forceinline__ void sub_run(const double (&v)[N], double med, unsigned long long (&d)[N]) {
#pragma unroll
    for (int e = 0; e < N; e++) d[e] = Elem<double>::bits(__dsub_rn(v[e], med));
}

// Byte-wise appending to a payload in shared memory.  A lane appends its
// run's values one after the other: `last` holds the four bytes written last
// (the newest on top), so the word that a value completes is a funnel shift of
// (last, value) by the position's bit offset and the next `last` one by the
// value's bits -- no masks, no byte stores, and whole words leave with one
// predicated store each: ~8 instructions a float value, where a store per
// byte took ~15 and up to four stores.  The first word a lane completes
// carries stale bytes below the run's start; what belongs there (the lane
// before's last bytes, or the block's lead codes) has to be stored after it:
// finish(), the bytes of the run's last, partial word, comes after a
// synchronisation of all lanes whose runs may share a word.
struct RunOut {
    uint32_t last, q8, sp;   // last four bytes, bit position, shared address of the word being filled
    // run of bytes at offset q0 of a staging buffer (16-byte aligned shared memory)
    __device__ __forceinline__ void start(const uint8_t* stg, uint32_t q0) {
        last = 0;
        q8 = 8 * q0;
        sp = smem_u32(stg) + (q0 & ~3u);
    }
    __device__ __forceinline__ void append(uint32_t v, uint32_t n8) {   // the low n8 / 8 (0..4) bytes of v
        const uint32_t w = __funnelshift_l(last, v, q8);
        last = __funnelshift_rc(last, v, n8);
        const uint32_t q = q8 + n8;
        // predicated, not branched over: the position crosses a word boundary
        asm volatile("{\n\t.reg .pred p;\n\t.reg .b32 t;\n\tlop3.or.b32 t|p, %1, %2, -32, 0x28, 0;\n\t"
                     "@p st.shared.u32 [%0], %3;\n\t@p add.u32 %0, %0, 4;\n\t}"
                     : "+r"(sp)
                     : "r"(q), "r"(q8), "r"(w)
                     : "memory");
        q8 = q;
    }
    // the bytes of the last word from the run's start (if that lies in it) to its end
    __device__ __forceinline__ void finish(const uint8_t* stg, uint32_t q0) const {
        const uint32_t w = __funnelshift_l(last, 0u, q8);
        const uint32_t end = (q8 >> 3) & 3u, beg = (sp ^ smem_u32(stg + q0)) < 4u ? q0 & 3u : 0u;
#pragma unroll
        for (uint32_t j = 0; j < 3; j++)
            if (j >= beg && j < end) asm volatile("st.shared.u8 [%0], %1;" ::"r"(sp + j), "r"(w >> (8 * j)) : "memory");
    }
};

// 32-byte stores (sm_100 and later): a lane's 8 floats / 4 doubles at a
// 32-byte aligned address, so that lanes writing consecutive 64-byte runs fill
// whole 32-byte sectors.
__device__ __forceinline__ void st_v8(float* p, const float* v) {
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]),
                 "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
}
__device__ __forceinline__ void st_v8(double* p, const double* v) {
    asm volatile("st.global.v4.f64 [%0], {%1,%2,%3,%4};" ::"l"(p), "d"(v[0]), "d"(v[1]), "d"(v[2]), "d"(v[3])
                 : "memory");
}

// N words at any byte address, from the aligned words that hold them; the
// caller's bytes end at `end`.  False when the last aligned word passes it.
template <int N>
__device__ __forceinline__ bool load_words(const uint8_t* p, const uint8_t* end, uint32_t (&w)[N]) {
    const uint32_t sh = (uint32_t)((uintptr_t)p & 3);
    const uint32_t* q = (const uint32_t*)(p - sh);
    if ((const uint8_t*)(q + N + (sh != 0)) > end) return false;
    uint32_t a[N + 1];
#pragma unroll
    for (int i = 0; i < N; i++) a[i] = __ldg(q + i);
    a[N] = sh ? __ldg(q + N) : 0u;
#pragma unroll
    for (int i = 0; i < N; i++) w[i] = __funnelshift_r(a[i], a[i + 1], 8 * sh);
    return true;
}

// ------------------------------------------------------------------ runs, decoded

// Lead-byte tables (a lead byte holds 4 codes, MSB first): 8 * the four leads
// as bytes, value 0 in byte 0; at 256 + c the same with leads cut at 2.  A
// value stores max(R - lead, 0) bytes, so 8 * R less the entry is its stored
// bits, from the second table where R is 2 (the decoders turn R = 1 into it).
__device__ __forceinline__ void lead_table_init(uint32_t* lut) {
    for (int c = threadIdx.x; c < 256; c += blockDim.x) {
        uint32_t a = 0, b = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint32_t ld = (uint32_t)c >> (6 - 2 * i) & 3u;
            a |= 8 * ld << (8 * i);
            b |= 8 * (ld < 2 ? ld : 2u) << (8 * i);
        }
        lut[c] = a;
        lut[256 + c] = b;
    }
}

__device__ __forceinline__ uint32_t lds32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t lds8(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}

// The run decoder below takes R = 2 bytes a value at least, what this library's
// encoders write (reqLength from 9).  A value of one byte is one of two whose
// top byte is always its predecessor's, zero before the first: every lead one
// higher, cut at 2.  Four codes to a byte, any number of bytes.
__device__ __forceinline__ bool one_byte_req(int reqLength) { return reqLength <= 8; }
__device__ __forceinline__ uint32_t one_byte_codes(uint32_t c) { return 0x55555555u + ((c | c >> 1) & 0x55555555u); }
// Stored bytes of a value at lead 0; reqLength 1 .. 8 * sizeof(T).
__device__ __forceinline__ int run_bytes(int reqLength) { return reqLength <= 8 ? 2 : (reqLength + 7) >> 3; }
// A block's reqLength byte is taken as it comes, and decoded without reading
// outside the block's largest size: 0 as 8, one above the type's bits as all
// bytes shifted by what its low three bits say.
template <typename T>
__device__ __forceinline__ bool plain_req(int reqLength) { return (uint32_t)(reqLength - 9) <= 8u * sizeof(T) - 9u; }
template <typename T>
__device__ __forceinline__ int clamp_req(int reqLength) {
    constexpr int B = 8 * (int)sizeof(T);
    return reqLength == 0 ? 8 : (reqLength > B ? B - (-reqLength & 7) : reqLength);
}

// The lead codes of a run of up to E (at most 16) values as masks, value e's
// bit at position 2e + 1: values with lead <= 0, 1, 2, i.e. those that store
// byte lane W-1, W-2, W-3.
template <int E>
struct RunLeads {
    uint32_t v0, v1, v2, low;   // low: bytes every value stores below the top three
    int nv, R;
    // codes: 4 to a byte, MSB first, chunk k in byte k; nv values
    __device__ __forceinline__ RunLeads(uint32_t codes, int nv_, int R_) : nv(nv_), R(R_) {
        const uint32_t c2 = vorder(codes & 0x55555555u), c1 = vorder((codes >> 1) & 0x55555555u);
        const uint32_t valid = nv ? 0xAAAAAAAAu >> (32 - 2 * nv) : 0u;
        v0 = ~(c1 | c2) & valid;
        v1 = ~c1 & valid;
        v2 = R >= 3 ? ~(c1 & c2) & valid : 0u;
        low = R > 3 ? (uint32_t)(R - 3) : 0u;
    }
    // bytes the run stores
    __device__ __forceinline__ uint32_t bytes() const { return __popc(v0) + __popc(v1) + __popc(v2) + low * (uint32_t)nv; }
    // the top three bytes as the run leaves them (v, zero where it wrote none)
    // and a mask of the ones it wrote (w); q0: shared address of its first byte
    __device__ __forceinline__ void summary(uint32_t q0, uint32_t& v, uint32_t& w) const {
        v = 0;
        w = 0;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            if (k == 0 ? v0 : k == 1 ? v1 : v2) {
                v |= lds8(q0 + last_at(k)) << (16 - 8 * k);
                w |= 0xFFu << (16 - 8 * k);
            }
        }
    }
    // where in the run's bytes the last value that stored byte lane W-1-k put it (there is one)
    __device__ __forceinline__ uint32_t last_at(int k) const {
        const int top = 31 - __clz(k == 0 ? v0 : k == 1 ? v1 : v2);
        const uint32_t before = (1u << top) - 1u;
        return __popc(v0 & before) + __popc(v1 & before) + __popc(v2 & before) + low * (uint32_t)(top >> 1) +
               (uint32_t)(R - 1 - k);
    }
};

// One pass over a run: cur, the values' bits less the median, and v, their
// sums with it.  reqLength: 1 .. 8 * sizeof(T), R its run_bytes(); q0: shared
// address of the run's first stored byte (the reads start up to eight bytes
// before it); carry: the top 32 bits of the value before (three bytes of them
// count).  Returns whether a sum may be a NaN: the x86 rules then decide
// (nan_rule).  FULL: nv is E.
template <typename T, int E, bool FULL>
__device__ __forceinline__ bool run_decode(uint32_t codes, int nv, int R, int reqLength, uint32_t q0, uint32_t carry,
                                           T med, const uint32_t* lut_ld, typename Elem<T>::U (&cur)[E], T (&v)[E]) {
    using EL = Elem<T>;
    using U = typename EL::U;
    constexpr int W = EL::W;
    constexpr int NC = E / 4;
    uint32_t q8 = 8 * q0;   // bit address of the next stored byte
    const uint32_t* lut_cnt = lut_ld + (R == 2 ? 256 : 0);
    const uint32_t R8 = (uint32_t)R * 0x08080808u;
    unsigned long long nan2 = 0;
    if constexpr (sizeof(T) == 4) {
        const int down = 32 - reqLength;   // `run` ends in the value's required bits
        // (the shift by `down` is a multiplication: the integer pipe sets the pace, the FMA pipe has room)
        const uint32_t scale = 1u << down;
        uint32_t run = carry >> (32 - 8 * R);
        // the word before the one the position lies in, and that word
        uint32_t sp = q0 & ~3u;
        uint32_t wa = lds32(sp - 4), wb = lds32(sp);
#pragma unroll
        for (int k = 0; k < NC; k++) {
            uint32_t cnt8 = R8 - lut_cnt[byte_of(codes, k)];
            if constexpr (!FULL) cnt8 &= low_bytes_mask(nv - 4 * k);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t n8 = byte_of(cnt8, i);
                const uint32_t qn = q8 + n8;
                // (predicated: the position crosses into the next word)
                asm volatile("{\n\t.reg .pred p;\n\t.reg .b32 t;\n\tlop3.or.b32 t|p, %3, %4, -32, 0x28, 0;\n\t"
                             "@p mov.b32 %0, %1;\n\t@p ld.shared.u32 %1, [%2+4];\n\t@p add.u32 %2, %2, 4;\n\t}"
                             : "+r"(wa), "+r"(wb), "+r"(sp)
                             : "r"(qn), "r"(q8)
                             : "memory");
                q8 = qn;
                const uint32_t y = __funnelshift_r(wa, wb, q8);   // the four bytes before q8
                run = __funnelshift_lc(y, __funnelshift_rc(run, 0u, n8), n8);
                asm("mul.lo.u32 %0, %1, %2;" : "=r"(cur[4 * k + i]) : "r"(run), "r"(scale));
            }
        }
        // the sums, two to an instruction, and a word that is NaN if any sum is one (or an infinity)
        asm("mov.b64 %0, {%1, %1};" : "=l"(nan2) : "f"(0.0f));
#pragma unroll
        for (int e = 0; e < E; e += 2)
            asm("{\n\t.reg .b64 a, b, z;\n\tmov.b64 a, {%3, %4};\n\tmov.b64 b, {%5, %5};\n\tmov.b64 z, {%6, %6};\n\t"
                "add.rn.f32x2 a, a, b;\n\tfma.rn.f32x2 %2, a, z, %2;\n\tmov.b64 {%0, %1}, a;\n\t}"
                : "=f"(v[e]), "=f"(v[e + 1]), "+l"(nan2)
                : "r"(cur[e]), "r"(cur[e + 1]), "f"(med), "f"(0.0f));
    } else {
        const int s = 8 * R - reqLength;
        const U keep = ~(U)0 << (8 * (W - R));
        uint32_t prev = carry;   // the previous value's top 32 bits
#pragma unroll
        for (int k = 0; k < NC; k++) {
            const uint32_t code = byte_of(codes, k), ld8 = lut_ld[code];
            uint32_t cnt8 = R8 - lut_cnt[code];
            if constexpr (!FULL) cnt8 &= low_bytes_mask(nv - 4 * k);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                q8 += byte_of(cnt8, i);
                const uint32_t l8 = byte_of(ld8, i);
                const uint32_t a = (q8 >> 3) & ~3u;
                const uint32_t w0 = lds32(a - 8), w1 = lds32(a - 4), w2 = lds32(a);
                const uint32_t ylo = __funnelshift_r(w0, w1, q8), yhi = __funnelshift_r(w1, w2, q8);   // the eight bytes before q8
                const uint32_t hi = __funnelshift_r(yhi, __funnelshift_l(prev, 0u, l8), l8);
                const uint32_t lo = __funnelshift_r(ylo, yhi, l8);
                const U u = (((U)hi << 32) | lo) & keep;
                prev = hi;
                cur[4 * k + i] = u << s;
                v[4 * k + i] = EL::add(EL::of(cur[4 * k + i]), med);
            }
        }
    }
    // a NaN (or infinite) result anywhere
    if constexpr (sizeof(T) == 4) {
        const float a = __uint_as_float((uint32_t)nan2) + __uint_as_float((uint32_t)(nan2 >> 32));   // zero, or NaN
        return a != a;
    } else {
        // (integer test: a compare costs the FP64 pipe as much as the addition)
        bool bad = false;
#pragma unroll
        for (int e = 0; e < E; e++) bad |= inf_or_nan(v[e]);
        return bad;
    }
}

}  // namespace szxg
