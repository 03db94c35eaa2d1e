// Blocked layouts of the SZx stream (fastMode 2, 3, 4): encode and decode.
//
// Stream (mode 3, szx/src/szx_float.cc:1407-1489):
//   [1,1,1,1] | blockSize u64 BE | nbConstant u64 BE | O u16[nnc] | state bits
//   | constant medians f32 BE [nc] | payloads of the non-constant blocks
// mode 2 (szx/src/szx_float.cc:1059-1139): [1,1,1,0] | blockSize u8 | nbConstant
//   u64 BE | state bits | medians | payloads  (no size index)
// mode 4 (szx/src/szx_float.cc:1218-1405): mode-3 layout, medians native endian.
// Block payload (szx/src/szx_float.cc:49-252): reqLength u8 | median f32 BE |
//   2-bit lead codes MSB-first | mid bytes.
//
// GB300 design
// * Encode is ONE pass over the input.  Persistent CTAs take tiles of blocks
//   from an atomic counter and pipeline them over four shared-memory buffers
//   filled by cp.async.  A block is handled by a segment of G lanes, each with
//   a run of consecutive values (16 float / 8 double, 64 bytes, swizzled in
//   16-byte chunks so that neither the fill nor the runs meet bank conflicts);
//   a lane's stored bytes are then one run of the payload, written as whole
//   words.  One warp places a tile from its CTA's previous tile and a window
//   of byte counts while the others copy the tile before it out in aligned
//   16-byte stores.
// * The payload region is written at a fixed position (as if no block were
//   non-constant); the stream then starts 2*nnc (mode 3/4) or 4*nnc (mode 2)
//   bytes into the buffer, so that header, size index, state bits and
//   medians (compacted from per-block scratch by a small look-back kernel) end
//   exactly where the payload region begins.  Nothing is ever moved.
// * Decode scans the size index and the state bits once (payload offsets by
//   non-constant rank, rank at each 32-block state word); then a producer
//   warp per CTA stages each tile's payload range by a bulk copy into a ring
//   of buffers while eight consumer warps decode G lanes per block, the bytes
//   inherited from earlier lanes resolved by one "last writer" scan over the
//   lanes' summaries.
#include "common.cuh"
#include "kernels.h"
#include "segment.cuh"

namespace szxg {

// Encoder tiles: ~16 KiB of input per tile, as many warps as the tile has
// block groups (at least 4), 24 warps per SM.  An earlier form of the encoder
// took 0.396 ms for 512^3 fp32 with 8 KiB tiles in 4-warp CTAs (6 per SM)
// against 0.380 ms -- the extra look-backs and tile claims cost more than the
// extra barrier domains save.  Four CTAs of 8 warps with a three-buffer ring
// (64 registers) took 462 us against 281 us: the loads are issued too late and
// the double variants spill.
constexpr int kEncTileBytes = 16384;
constexpr int kEncWarpsPerSm = 24;
constexpr int kSizeThreads = 256;
constexpr int kIdxThreads = 256;
constexpr int kIdxItems = 8;   // items per thread in the index scans

// ------------------------------------------------------------------ encode
//
// Per-block state a segment keeps in registers from its statistics pass to
// its emission (szx/src/szx_float.cc:49-252 for one block).  A lane owns a run
// of E consecutive values (64 bytes), whose stored bytes are one run of the
// payload.
template <typename T, int G>
struct BlockEnc {
    using U = typename Elem<T>::U;
    static constexpr int E = EncCfg<T>::E;
    static constexpr int NC = E / 4;
    U ev[E];                         // the value's required bytes (reqLength bits), right-aligned
    uint32_t cnt8[NC];               // bits stored of each of the chunk's 4 values (byte i: value i)
    uint32_t codes;                  // lead byte of chunk k in byte k
    uint32_t excl;                   // mid bytes of earlier lanes
    int state;                       // 0 constant, 1 coded, 2 no block
    int reqLength;
    uint32_t med_bits;               // median as stored (payload or constant list)
    uint32_t size;                   // payload bytes of a coded block
};

struct EncArgs {
    BlkField one;                // the field when nf == 1
    const BlkField* fields;      // nf > 1: device table in ascending enc_tile0
    int nf;
    int bs;
    int omp_stats;               // mode-4 double statistics
    unsigned long long total_tiles;
    unsigned long long* tile_ctr;
    const uint32_t* tile_field;  // nf > 1: field of every launch-wide tile
    int* err;
};

// A double block is constant when radius <= (double)eb.  The radius is a
// non-negative number or a NaN, so the test is one on unsigned bit patterns:
// pattern < eb_key, with key 0 (never) for negative and NaN bounds; a NaN's
// pattern of either sign is above every bound's.
__device__ __forceinline__ unsigned long long eb_key_of(float eb) {
    if (!(eb >= 0.0f)) return 0ull;
    return (unsigned long long)__double_as_longlong(xf2d(fabsf(eb))) + 1ull;
}

// Extremes of a lane's block, for blocks without infinities, NaNs and (beside
// a zero extreme) negative zeros; true where the block has one of these and
// the exact rules below decide.
template <typename T, int G, bool FULL>
__device__ __forceinline__ bool enc_minmax_fast(const T (&v)[EncCfg<T>::E], int len, T& mn, T& mx) {
    constexpr int E = EncCfg<T>::E;
    const int f = E * (int)(lane_id() & (G - 1));
    bool odd;
    if constexpr (sizeof(T) == 4) {
        // (three-input forms where whole runs are compared; hn: NaN if any value is one)
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
                if (f + e < len) {
                    lo = fminf(lo, v[e]);
                    hi = fmaxf(hi, v[e]);
                    hn = fmax_nan(hn, v[e]);
                }
            }
        }
        odd = isnan(hn);
#pragma unroll
        for (int d = G / 2; d > 0; d >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, d, G));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, d, G));
        }
        mn = lo;
        mx = hi;
        odd = odd || (len > 0 && (inf_or_nan(lo) || inf_or_nan(hi)));
    } else {
        // Order-preserving integer keys, high words first: the extremes of
        // the 32-bit high keys, then of the low words beside them -- 32-bit
        // operations throughout, about half of what 64-bit keys cost.  Any
        // infinity or NaN shows in the high extremes.
        int khn = 0x7FFFFFFF, khx = (int)0x80000000;
#pragma unroll
        for (int e = 0; e < E; e++) {
            const int k = dkey_hi(hi32(v[e]));
            const bool in = FULL || f + e < len;
            khn = in ? min(khn, k) : khn;
            khx = in ? max(khx, k) : khx;
        }
#pragma unroll
        for (int d = G / 2; d > 0; d >>= 1) {
            khn = min(khn, __shfl_xor_sync(0xffffffffu, khn, d, G));
            khx = max(khx, __shfl_xor_sync(0xffffffffu, khx, d, G));
        }
        odd = khx >= 0x7FF00000 || khn <= (int)0x800FFFFF;
        uint32_t kln = 0xFFFFFFFFu, klx = 0u;
#pragma unroll
        for (int e = 0; e < E; e++) {
            const uint32_t h = hi32(v[e]), l = lo32(v[e]) ^ (uint32_t)((int)h >> 31);
            const int k = dkey_hi(h);
            const bool in = FULL || f + e < len;
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
    }
    // a zero extreme has the sign of the block's first zero: plus, unless there is a negative one
    if (__any_sync(0xffffffffu, is_zero(mn) || is_zero(mx))) {
#pragma unroll
        for (int e = 0; e < E; e++) {
            if constexpr (sizeof(T) == 4) odd = odd || __float_as_uint(v[e]) == 0x80000000u;
            else odd = odd || (hi32(v[e]) == 0x80000000u && lo32(v[e]) == 0u);
        }
    }
    return odd;
}

// Floats: what the extremes above leave open of the reference's sequential
// scan (szx/src/szx_float.cc:322-345).  They ignored the NaNs, as the scan does
// unless the block's first value is one; a zero extreme takes the sign of the
// first zero.  In registers, like the differences below: the loops over shared
// memory that doubles take cost 2^23 floats with NaNs in one of a hundred values
// 55 us a compress, 38.6 now (51.2 before the runs; 35.2 without NaNs), and their
// code spilled beside the float loop (2^27 values: 282 -> 275 us).
template <int G, bool FULL>
__device__ __forceinline__ void enc_minmax_rules(const float (&v)[EncCfg<float>::E], int len, float& mn, float& mx) {
    constexpr int E = EncCfg<float>::E;
    const int f = E * (int)(lane_id() & (G - 1));
    if (__any_sync(0xffffffffu, is_zero(mn) || is_zero(mx))) {
        int zi = 1 << 30;   // 2 * index + sign of the first zero
#pragma unroll
        for (int e = E - 1; e >= 0; e--)
            if (is_zero(v[e]) && (FULL || f + e < len)) zi = 2 * (f + e) + (int)(__float_as_uint(v[e]) >> 31);
#pragma unroll
        for (int d = G / 2; d > 0; d >>= 1) zi = min(zi, __shfl_xor_sync(0xffffffffu, zi, d, G));
        const float zero = __uint_as_float((uint32_t)zi << 31);
        if (is_zero(mn)) mn = zero;
        if (is_zero(mx)) mx = zero;
    }
    const float x0 = __shfl_sync(0xffffffffu, v[0], 0, G);
    if (len > 0 && isnan(x0)) mn = mx = x0;
}

// Doubles, with every rule of the scan
// (szx/src/szx_double.cc:973-1030), for the warps that met an odd value: NaNs
// are skipped unless the block's first value is one, a zero extreme has the
// sign of the first zero.  Values come from shared memory again, one at a
// time: this is the rare path, and small code beside the encoder's loop
// matters more than its speed.  Returns whether the block holds a NaN or an
// infinity.
template <typename T, int G>
__device__ __forceinline__ bool enc_minmax_exact(const uint8_t* tile, uint32_t e0, int len, T& mn, T& mx) {
    using U = typename Elem<T>::U;
    using K = typename std::make_signed<U>::type;   // order-preserving key of a non-NaN pattern
    constexpr int E = EncCfg<T>::E;
    constexpr int B = 8 * (int)sizeof(T) - 1;
    constexpr U MAG = (U)~(U)0 >> 1;
    const U inf = Elem<T>::bits((T)__builtin_huge_val());
    const int f = E * (int)(lane_id() & (G - 1));
    auto key = [](U u) { return (K)(u ^ ((U)((K)u >> B) & MAG)); };
    K lo = (K)MAG, hi = (K)~MAG;
    int zi = 1 << 30;   // 2 * index + sign of the first zero
    bool nan = false;
#pragma unroll 1
    for (int i = f; i < f + E && i < len; i++) {
        const U u = *(const U*)(tile + swz_off<T>(e0 + i)), m = u & MAG;
        if (m > inf) { nan = true; continue; }
        lo = min(lo, key(u));
        hi = max(hi, key(u));
        if (m == 0) zi = min(zi, 2 * i + (int)(u >> B));
    }
#pragma unroll 1
    for (int d = G / 2; d > 0; d >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, d, G));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, d, G));
        zi = min(zi, __shfl_xor_sync(0xffffffffu, zi, d, G));
        nan = __shfl_xor_sync(0xffffffffu, (int)nan, d, G) || nan;
    }
    U ulo = (U)lo ^ ((U)(lo >> B) & MAG), uhi = (U)hi ^ ((U)(hi >> B) & MAG);
    const U zero = (U)(zi & 1) << B;
    if ((ulo & MAG) == 0) ulo = zero;
    if ((uhi & MAG) == 0) uhi = zero;
    if (len > 0) {
        const U u = *(const U*)(tile + swz_off<T>(e0));
        if ((u & MAG) > inf) ulo = uhi = u;
    }
    mn = Elem<T>::of(ulo);
    mx = Elem<T>::of(uhi);
    return nan || (ulo & MAG) >= inf || (uhi & MAG) >= inf;
}
// A run's differences from the median under the x86 NaN rules, in place.
template <typename T, int G>
__device__ __forceinline__ void enc_diff_exact(uint8_t* tile, uint32_t e0, int len, T med) {
    constexpr int E = EncCfg<T>::E;
    const int f = E * (int)(lane_id() & (G - 1));
#pragma unroll 1
    for (int i = f; i < f + E && i < len; i++) {
        T* p = (T*)(tile + swz_off<T>(e0 + i));
        *p = xsub(*p, med);
    }
    __syncwarp();
}

// Statistics pass of one block by a G-lane segment: state, reqLength and
// median (szx/src/szx_float.cc:314-371), the shifted words, lead codes
// (szx/src/szx_float.cc:94-113) and stored-byte counts, all kept in registers.
//
// eb_key: the bound's rule for double radii (constant when the radius's bit
// pattern, as an unsigned number, is below it; see eb_key_of).
template <typename T, int G, bool FULL>
__device__ __forceinline__ void enc_block_stats(uint8_t* tile, uint32_t e0, int len, bool vec, float eb,
                                                int eb_exp, unsigned long long eb_key, int omp_stats,
                                                BlockEnc<T, G>& b) {
    using EL = Elem<T>;
    using U = typename EL::U;
    constexpr int W = EL::W;
    constexpr int E = EncCfg<T>::E;
    constexpr int NC = E / 4;
    const int sl = (int)(lane_id() & (G - 1));
    T v[E];
    if constexpr (FULL) load_run_full<T>(smem_u32(tile), e0 / E + sl, v);
    else load_run<T, G>(tile, e0, vec, v);
    T mn, mx;
    bool special = enc_minmax_fast<T, G, FULL>(v, len, mn, mx);
    if (__any_sync(0xffffffffu, special)) {
        if constexpr (sizeof(T) == 4) enc_minmax_rules<G, FULL>(v, len, mn, mx);
        else special = enc_minmax_exact<T, G>(tile, e0, len, mn, mx);
    }
    int state;
    float radius_f, median_f;
    if constexpr (sizeof(T) == 4) {
        const float range = xsub(mx, mn);
        radius_f = xhalf(range);
        median_f = xadd(mn, radius_f);
        state = (radius_f <= eb) ? 0 : 1;
    } else if (!omp_stats) {
        // szx/src/szx_double.cc:991-1003: double statistics, float median/radius
        const double range = xsub(mx, mn);
        const double radius = xhalf(range);
        const double median = xadd(mn, radius);
        state = (unsigned long long)__double_as_longlong(radius) < eb_key ? 0 : 1;
        radius_f = xd2f(radius);
        median_f = xd2f(median);
    } else {
        // computeStateMedianRadius_double2 (szx/src/szx_double.cc:1120-1135)
        const double range = xsub(mx, mn);
        radius_f = xd2f(xhalf(range));
        median_f = xd2f(xadd(mn, xf2d(radius_f)));
        state = (radius_f <= eb) ? 0 : 1;
    }
    bool zm;
    const int reqLength = req_length_e<T>(eb_exp, radius_f, &zm);
    int R, s;
    split_reqlen(reqLength, &R, &s);
    const uint32_t payload_med = zm ? 0u : __float_as_uint(median_f);
    T med;
    if constexpr (sizeof(T) == 4) med = __uint_as_float(payload_med);
    else med = xf2d(median_f);
    // differences from the median (szx/src/szx_float.cc:88-92); x86 NaN rules only where a NaN can arise
    U d[E];
    if (sizeof(T) == 8 && __any_sync(0xffffffffu, special)) {
        enc_diff_exact<T, G>(tile, e0, len, med);
        load_run<T, G>(tile, e0, vec, v);
#pragma unroll
        for (int e = 0; e < E; e++) d[e] = EL::bits(v[e]);
    } else {
        sub_run(v, med, d);
        if (sizeof(T) == 4 && __any_sync(0xffffffffu, special)) {
#pragma unroll
            for (int e = 0; e < E; e++)
                if (isnan(EL::of(d[e]))) d[e] = EL::bits(nan_rule(v[e], med));
        }
    }
    // Lead codes: leading identical bytes of the words shifted right by s with
    // the previous value's, capped at 3 -- (leading zeros of the XOR + s) / 8,
    // with a guard bit that ends the count at 24 - s.  Only the top 32 bits
    // decide; four leading-bit positions (31 - zeros) are packed in a word,
    // by multiplications the idle FMA pipe takes, before the division.
    auto top = [](U u) { return (uint32_t)(u >> (8 * W - 32)); };
    uint32_t prev = __shfl_up_sync(0xffffffffu, top(d[E - 1]), 1, G);
    if (sl == 0) prev = 0u;   // zero before the block
    const uint32_t guard = 0x80u << s, s4 = (uint32_t)(31 + s) * 0x01010101u;
    uint32_t codes = 0, mine = 0;
#pragma unroll
    for (int k = 0; k < NC; k++) {
        uint32_t lb[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint32_t h = top(d[4 * k + i]);
            asm("bfind.u32 %0, %1;" : "=r"(lb[i]) : "r"((h ^ prev) | guard));
            prev = h;
        }
        const uint32_t p = (lb[3] * 256u + lb[2]) * 65536u + (lb[1] * 256u + lb[0]);
        uint32_t ldb = ((s4 - p) >> 3) & 0x03030303u;
        // max(R - lead, 0) per value; R is at least 2 here, so only lead 3 at R = 2 needs raising
        uint32_t cnt4 = (uint32_t)R * 0x01010101u + (R == 2 ? (ldb >> 1) & ldb & 0x01010101u : 0u) - ldb;
        if constexpr (!FULL) {
            const uint32_t m = low_bytes_mask(len - (E * sl + 4 * k));
            ldb &= m;
            cnt4 &= m;
        }
        b.cnt8[k] = cnt4 << 3;
        mine = __dp4a(cnt4, 0x01010101u, mine);
        codes |= ((ldb * 0x40100401u) >> 24) << (8 * k);   // 4 leads -> one byte, MSB first
    }
    const uint32_t incl = seg_inclusive_sum<G>(mine);
    const uint32_t mid = __shfl_sync(0xffffffffu, incl, G - 1, G);
    b.excl = incl - mine;
    b.codes = codes;
    const int down = 8 * W - reqLength;   // drops the bits below the required ones
#pragma unroll
    for (int e = 0; e < E; e++) b.ev[e] = d[e] >> down;
    const int Lb = FULL ? G * NC : (len + 3) / 4;
    b.size = 5 + (uint32_t)Lb + mid;
    b.state = len ? state : 2;
    b.reqLength = reqLength;
    b.med_bits = state == 1 ? payload_med : __float_as_uint(median_f);
}

// Emission of the coded blocks of a warp (act: this segment has one) into the
// tile's staging buffer: every lane's whole words, then headers, lead bytes
// and the bytes of the words that lanes share.  Every byte of a block's
// [loc, loc + size) ends up as the stream wants it; bytes outside are not
// touched (a lane's first word starts at most 3 bytes early, inside the
// block's own header and lead bytes).  ~8 instructions and one 4-byte store
// per float value, where a store per byte took ~15 and up to four.
template <typename T, int G, bool FULL>
__device__ __forceinline__ void enc_block_emit(uint8_t* stg, uint32_t loc, int len, bool act, const BlockEnc<T, G>& b) {
    constexpr int E = EncCfg<T>::E;
    constexpr int NC = E / 4;
    const int sl = (int)(lane_id() & (G - 1));
    const int Lb = FULL ? G * NC : (len + 3) / 4;
    const uint32_t q0 = loc + 5 + (uint32_t)Lb + b.excl;
    RunOut o;
    o.start(stg, q0);
    if (act) {
#pragma unroll
        for (int k = 0; k < NC; k++) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t n8 = byte_of(b.cnt8[k], i);
                if constexpr (sizeof(T) == 4) {
                    o.append((uint32_t)b.ev[4 * k + i], n8);
                } else {
                    const uint32_t nl = n8 < 32u ? n8 : 32u;
                    o.append((uint32_t)b.ev[4 * k + i], nl);
                    o.append((uint32_t)(b.ev[4 * k + i] >> 32), n8 - nl);
                }
            }
        }
    }
    __syncwarp();
    if (act) {
        o.finish(stg, q0);
        uint8_t* p = stg + loc;
        // lead codes: 4 per byte, MSB first (szx/src/szx_TypeManager.cc:198-273)
#pragma unroll
        for (int k = 0; k < NC; k++)
            if (FULL || NC * sl + k < Lb) p[5 + NC * sl + k] = (uint8_t)(b.codes >> (8 * k));
        if (sl == 0) {
            p[0] = (uint8_t)b.reqLength;
            p[1] = (uint8_t)(b.med_bits >> 24);
            p[2] = (uint8_t)(b.med_bits >> 16);
            p[3] = (uint8_t)(b.med_bits >> 8);
            p[4] = (uint8_t)b.med_bits;
        }
    }
}

template <typename T, int G, int TBYTES = kEncTileBytes>
struct EncTile {
    static constexpr int E = EncCfg<T>::E;
    static constexpr int kBsMax = G * E;                               // largest block of this variant
    static constexpr int kBpw = 32 / G;                                // blocks per warp
    static constexpr int kRaw = TBYTES / (kBsMax * (int)sizeof(T));
    static constexpr int kBlocks = kRaw >= 64 ? 64 : (kRaw < 8 ? 8 : kRaw);   // blocks per tile
    static constexpr int kGroups = kBlocks / kBpw;                     // warps with blocks
    static constexpr int kWarps = kGroups > 4 ? kGroups : 4;
    static constexpr int kThreads = kWarps * 32;
    static constexpr int kMinCtas = kEncWarpsPerSm / kWarps;
    static constexpr int kIn = kBlocks * kBsMax * (int)sizeof(T);      // input bytes per buffer
    static constexpr int kMaxPay = 5 + (kBsMax + 3) / 4 + (int)sizeof(T) * kBsMax;
    // payloads of a tile + slack for the word-wise reads of the realigning copy
    // (a multiple of 64: a run's address is swizzled by exclusive-or)
    static constexpr int kStage = ((kBlocks * kMaxPay + 32 + 63) / 64) * 64;
    // a ring buffer holds a tile's input, then (in place) its payloads
    static constexpr int kBuf = kIn > kStage ? kIn : kStage;
    static constexpr int kDynSmem = 4 * kBuf;
    static_assert(kGroups <= 8 && kBlocks % kBpw == 0, "one block group per warp");
    static_assert(kBlocks <= 64, "a tile's sizes are scanned as two warp-wide halves");
    static_assert(kBlocks * kMaxPay < 65535, "a tile's byte count + 1 fits the 16-bit aggregate words");
    static_assert(kIn % 512 == 0 && kBuf % 64 == 0, "swizzled chunks stay inside the tile, runs on 64-byte boundaries");
    static_assert(kThreads % 32 == 0, "a thread's chunks keep one swizzle phase");
};

// One pass over the input.  A CTA works through its tiles T_j in a ring of
// four shared-memory buffers; iteration j, between two CTA barriers:
//   barrier (T_j's values are in)  |  cp.async of T_{j+1} into the buffer
//   T_{j-3} left; statistics of T_j's blocks (registers)  |  barrier  |  the
//   window copy for T_{j-1}; every warp scans T_j's block sizes for its own
//   blocks' offsets (warp 0 publishes T_j's byte count) and emits them into
//   T_j's buffer in place (its input is dead); then warp 0 places T_{j-1}
//   while the other warps copy T_{j-2} out, one of them T_j's block tables.
// Every global round trip of a tile -- input load, tile claim, look-back --
// thus has most of an iteration to complete, and nothing waits for warp 0.
// Tile ids come from an atomic counter, taken in increasing order two tiles
// ahead (the look-back stays deadlock-free with any number of resident CTAs).
// A segment of G lanes owns one block from its statistics to its emission.
//
// Bound by the instructions of the statistics and the emission (issue 65 %):
// 50 warp instructions per 32 floats, 124 per 32 doubles.  2^27 floats, REL
// 1e-3, blocks of 128: 275 us (512 MiB in, 129 us with the stream at the copy
// rate); 2^28 doubles in blocks of 64: 1355 us (490).  Before -- lanes over
// interleaved 4-value chunks, byte stores, doubles on the FP64 pipe (two lanes
// a clock and SM here), T_{j-2} placed by warp 0 while the others waited --
// 363 and 2791 us.
template <typename T, int G, bool MULTI, int TBYTES = kEncTileBytes>
__global__ void __launch_bounds__(EncTile<T, G, TBYTES>::kThreads, EncTile<T, G, TBYTES>::kMinCtas)
    k_blocked_encode(EncArgs a) {
    pdl_start();
    using TL = EncTile<T, G, TBYTES>;
    constexpr int TB = TL::kBlocks;
    constexpr int BPW = TL::kBpw;
    constexpr int NGRP = TB / BPW;
    extern __shared__ __align__(128) uint8_t dsm[];
    __shared__ uint32_t s_size[TB], s_med[TB];
    __shared__ uint8_t s_state[TB];
    __shared__ PlaceWin s_win;
    __shared__ uint32_t s_agg[4];
    __shared__ int s_tile[4];           // launch-wide tile index of each ring position (-1: none left)
    __shared__ int s_fld[4];            // its field
    __shared__ unsigned long long s_base[2];
    __shared__ int s_skip[2];
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int seg = lane / G, sl = lane & (G - 1);
    const uint32_t tile_elems = (uint32_t)(TB * a.bs);
    const bool vec = ((a.bs * (int)sizeof(T)) & 15) == 0;   // every block starts 16-byte aligned
    // field of a launch-wide tile: one load from the plan's tile map
    auto field_of = [&](int g) { return (int)a.tile_field[g]; };
    auto buf_ptr = [&](int r) { return dsm + r * TL::kBuf; };
    if (threadIdx.x == 0) {
        for (int r = 0; r < 2; r++) {
            const unsigned long long g = atomicAdd(a.tile_ctr, 1ull);
            s_tile[r] = g < a.total_tiles ? (int)g : -1;
            s_fld[r] = (MULTI && s_tile[r] >= 0) ? field_of(s_tile[r]) : 0;
        }
    }
    __syncthreads();
    // a field's members: from the kernel parameters for one field, from the table for a batch
    auto fld = [&](int f) -> const BlkField* { return MULTI ? a.fields + f : nullptr; };
#define FV(F_, m) (MULTI ? (F_)->m : a.one.m)

    auto tile_count = [&](const BlkField* F, int t) {
        if (t + 1 < (int)FV(F, enc_tiles)) return tile_elems;
        return (uint32_t)(FV(F, n) - (unsigned long long)t * tile_elems);
    };
    // all threads: the tile's values into ring buffer r, swizzled in 16-byte
    // chunks, by cp.async (one group; completed before the next iteration's
    // first barrier)
    auto issue = [&](int g, int f, int r) {
        const BlkField* F = fld(f);
        const int t = g - (int)FV(F, enc_tile0);
        const uint32_t cnt = tile_count(F, t);
        const uint8_t* src = (const uint8_t*)((const T*)FV(F, x) + (unsigned long long)t * tile_elems);
        uint8_t* dst = buf_ptr(r);
        if (((uintptr_t)src & 15) == 0) {
            constexpr uint32_t VN = 16 / sizeof(T);
            const uint32_t nch = cnt / VN;
            const uint8_t* sp = src + 16 * threadIdx.x;
            uint8_t* dp = dst + 16 * swz16(threadIdx.x);   // the threads' later chunks share its swizzle phase
            if (TL::kIn % (16 * TL::kThreads) == 0 && nch == TL::kIn / 16) {   // a whole tile of the largest blocks
#pragma unroll
                for (int k = 0; k < TL::kIn / 16 / TL::kThreads; k++)
                    cp_async16(dp + 16 * k * TL::kThreads, sp + 16 * k * TL::kThreads);
                return;
            }
            for (uint32_t c = threadIdx.x; c < nch; c += TL::kThreads) cp_async16(dst + 16 * swz16(c), src + 16 * c);
            const uint32_t i = nch * VN + threadIdx.x;
            if (i < cnt) cp_async_small<sizeof(T)>(dst + swz_off<T>(i), src + i * sizeof(T));
        } else {
            for (uint32_t i = threadIdx.x; i < cnt; i += TL::kThreads)
                cp_async_small<sizeof(T)>(dst + swz_off<T>(i), src + i * sizeof(T));
        }
    };
    auto block_len = [&](const BlkField* F, int t, int lb) {
        const unsigned long long b = (unsigned long long)t * TB + lb;
        if (b >= FV(F, nb)) return 0;
        const unsigned long long rem = FV(F, n) - b * (unsigned long long)a.bs;
        return rem < (unsigned long long)a.bs ? (int)rem : a.bs;
    };

    unsigned long long nnc_cta = 0;   // warp kMetaWarp lane 0, single field: non-constant blocks of this CTA's tiles
    if (threadIdx.x == 0) s_win.init();
    auto agg16_of = [&](const BlkField* F) {
        return (uint16_t*)(FV(F, st_enc) + enc_tile_words(FV(F, nb)));
    };
    // one warp: sizes, medians and state bits of tile t's blocks, by block
    constexpr int kMetaWarp = TL::kWarps - 2;
    auto meta = [&](const BlkField* F, int t) {
        const unsigned long long tb0 = (unsigned long long)t * TB;
        uint32_t m01[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int lb = lane + 32 * h;
            const bool in = lb < TB;
            const int st = in ? s_state[lb] : 2;
            if (in && st != 2) {
                FV(F, size_blk)[tb0 + lb] = (uint16_t)s_size[lb];
                FV(F, med_blk)[tb0 + lb] = s_med[lb];
            }
            m01[h] = __ballot_sync(0xffffffffu, in && st == 1);
        }
        if (lane == 0) {
            // state bits, MSB first (szx/src/szx_TypeManager.cc:16-40)
            uint8_t* sbp = FV(F, s_scr) + (unsigned long long)t * (TB / 8);
            const uint32_t r0 = __brev(m01[0]), r1 = __brev(m01[1]);
#pragma unroll
            for (int k = 0; k < TB / 8; k++) sbp[k] = (uint8_t)((k < 4 ? r0 : r1) >> (24 - 8 * (k & 3)));
            const unsigned long long k = (unsigned long long)(__popc(m01[0]) + __popc(m01[1]));
            if (!MULTI) nnc_cta += k;
            else if (k) atomicAdd(&FV(F, tot)->nnc, k);
        }
    };
    // warp 0: place tile t of field f, ring position r: its offset in the payload, the capacity check, the field's payload total
    auto place = [&](const BlkField* F, int f, int t, int r) {
        const uint32_t agg = s_agg[r];
        unsigned long long base;
        if (!s_win.offset(agg16_of(F), t, &base)) base = prefix_resolve(FV(F, st_enc), t, agg, a.err);   // (publishes)
        else if (t > 0 && lane == 0) st_volatile64(&FV(F, st_enc)[t], kS64Inc | ((base + agg) & kS64Val));
        if (lane == 0) {
            const bool cap_ok = base + agg <= FV(F, payload_cap);
            if (!cap_ok) atomicExch(a.err, kErrCapacity);
            if (t == (int)FV(F, enc_tiles) - 1) FV(F, tot)->payload_bytes = base + agg;
            s_base[r & 1] = base;
            s_skip[r & 1] = !cap_ok;
            s_win.anchor(f, t, base + agg);
        }
        __syncwarp();
    };
    // threads tid of nthr: the placed tile of ring position r to its place
    auto copy_out = [&](const BlkField* F, int r, uint32_t tid, uint32_t nthr) {
        if (!s_skip[r & 1]) cta_copy_realign(buf_ptr(r), s_agg[r], FV(F, payload) + s_base[r & 1], tid, nthr);
    };

    if (s_tile[0] >= 0) issue(s_tile[0], s_fld[0], 0);
    const bool taker = warp == TL::kWarps - 1 && lane == 0;
    int t1 = -1, t2 = -1;         // T_{j-1}, T_{j-2} (field-local), -1: none
    int eb_f = -1, eb_exp = 0;    // field whose bound is loaded, the bound's exponent
    float eb = 0.f;
    unsigned long long eb_key = 0;   // and its key for double radii
    int f1 = 0, f2 = 0;
    int j = 0;
    for (;; j++) {
        const int r = j & 3;
        // (after the last tile two more iterations place and copy out what is staged)
        cp_async_wait_all();   // T_j's values are in
        __syncthreads();   // ring position j+1 claimed, copy-out of T_{j-3} done
        {
            const int rn = (j + 1) & 3;
            const int gn = s_tile[rn];
            if (gn >= 0) issue(gn, s_fld[rn], rn);
        }
        const int g = s_tile[r];
        const bool live = g >= 0;
        if (!live && t1 < 0 && t2 < 0) break;
        const int f = live ? s_fld[r] : 0;
        const BlkField* F = fld(f);
        const int t = live ? g - (int)FV(F, enc_tile0) : -1;
        // the last warp takes the tile of ring position j+2; the reply is used at the iteration's end
        unsigned long long gc = ~0ull;
        claim_tile(gc, a.tile_ctr, taker && live);
        // ---- statistics of the tile's blocks, one block per segment
        const int lb = warp * BPW + seg;
        const bool mine = live && warp < NGRP;
        // every tile but a field's last holds whole blocks only
        const int len = !mine ? 0 : (t + 1 < (int)FV(F, enc_tiles) ? a.bs : block_len(F, t, lb));
        const bool full = __all_sync(0xffffffffu, len == TL::kBsMax);
        if (live && f != eb_f) {   // the field's bound and its exponent, once per field
            eb = FV(F, params) ? FV(F, params)->eb : FV(F, eb);
            eb_exp = exponent_f64_of_f32(eb);
            if constexpr (sizeof(T) == 8) eb_key = eb_key_of(eb);
            eb_f = f;
        }
        BlockEnc<T, G> b;
        if (mine) {
            const uint32_t e0 = (uint32_t)(lb * a.bs);
            if (full) enc_block_stats<T, G, true>(buf_ptr(r), e0, len, vec, eb, eb_exp, eb_key, a.omp_stats, b);
            else enc_block_stats<T, G, false>(buf_ptr(r), e0, len, vec, eb, eb_exp, eb_key, a.omp_stats, b);
            if (sl == 0) {
                s_state[lb] = (uint8_t)b.state;
                s_size[lb] = b.state == 1 ? b.size : 0;
                s_med[lb] = b.med_bits;
            }
        }
        __syncthreads();   // statistics in (T_j's input is dead)
        // warp 0: T_{j-1}'s look-back window, in flight during the emission
        if (warp == 0 && t1 >= 0) s_win.issue(agg16_of(fld(f1)), f1, t1);
        // every warp: the tile's block offsets (two warp-wide halves)
        const bool in0 = lane < TB;
        const uint32_t sz0 = in0 ? s_size[lane] : 0;
        const uint32_t i0 = warp_inclusive_sum(sz0);
        const uint32_t loc_lo = __shfl_sync(0xffffffffu, i0 - sz0, lb & 31);
        uint32_t i1 = i0, loc_hi = 0;   // tiles of up to 32 blocks have no second half
        if constexpr (TB > 32) {
            const bool in1 = lane + 32 < TB;
            const uint32_t sz1 = in1 ? s_size[lane + 32] : 0;
            i1 = warp_inclusive_sum(sz1) + __shfl_sync(0xffffffffu, i0, 31);
            loc_hi = __shfl_sync(0xffffffffu, i1 - sz1, lb & 31);
        }
        if (live && warp == 0) {
            const uint32_t agg = __shfl_sync(0xffffffffu, i1, 31);
            if (lane == 0) {
                s_agg[r] = agg;
                st_relaxed16(agg16_of(F) + t, agg + 1);
            }
            prefix_publish(FV(F, st_enc), t, agg);
        }
        if (mine) {
            const uint32_t loc = lb < 32 ? loc_lo : loc_hi;
            if (full) enc_block_emit<T, G, true>(buf_ptr(r), loc, len, b.state == 1, b);
            else enc_block_emit<T, G, false>(buf_ptr(r), loc, len, b.state == 1, b);
        }
        // T_{j-2} to its place by all warps but warp 0, which places T_{j-1} meanwhile
        if (warp == 0) {
            if (t1 >= 0) place(fld(f1), f1, t1, (j - 1) & 3);
        } else {
            if (live && warp == kMetaWarp) meta(F, t);
            if (t2 >= 0) copy_out(fld(f2), (j - 2) & 3, threadIdx.x - 32, TL::kThreads - 32);
        }
        if (taker) {
            const int rc = (j + 2) & 3;   // T_{j-2}'s position: its id was read two barriers ago
            s_tile[rc] = gc < a.total_tiles ? (int)gc : -1;
            s_fld[rc] = (MULTI && gc < a.total_tiles) ? field_of((int)gc) : 0;
        }
        t2 = t1;
        f2 = f1;
        t1 = t;
        f1 = f;
    }
    if (warp == kMetaWarp && lane == 0 && nnc_cta) atomicAdd(&a.one.tot->nnc, nnc_cta);
#undef FV
}

// Exact stream sizes of float fields in blocks of 128 at given bounds, without
// coding them: the encoder's statistics alone, every warp on its own over a
// contiguous range of 4-block steps (2 KiB, copied a step ahead into its own
// two buffers), no placement, no barriers.  An item is a field and a bound;
// acc[2 i] / [2 i + 1] gain its coded blocks' payload bytes and their number.
// (Four CTAs an SM, 64 registers: 263 us in the batch of 24 fields, 284 at two
// CTAs and the 120 registers it takes unasked.)
__global__ void __launch_bounds__(kSizeThreads, 4) k_blocked_sizes(const SizeItem* items, int ni,
                                                                unsigned long long steps, unsigned long long* acc) {
    constexpr int G = 8, BS = 128, STEP = 4 * BS;   // values per step
    __shared__ __align__(512) uint8_t buf[kSizeThreads / 32][2][STEP * 4];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, seg = lane / G, sl = lane & (G - 1);
    const unsigned long long w = (unsigned long long)blockIdx.x * (kSizeThreads / 32) + warp,
                             nw = (unsigned long long)gridDim.x * (kSizeThreads / 32);
    const unsigned long long u0 = steps * w / nw, u1 = steps * (w + 1) / nw;
    if (u0 >= u1) return;
    // item of step u0: the last one that starts at or before it
    int lo = 0, hi = ni - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (items[mid].step0 <= u0) lo = mid;
        else hi = mid - 1;
    }
    int it = lo, itl = lo;   // items of the step in work and of the step being copied
    SizeItem cur = items[it], nxt = cur;
    auto load = [&](unsigned long long u, int b) {
        while (itl + 1 < ni && items[itl + 1].step0 <= u) nxt = items[++itl];
        const unsigned long long v0 = (u - nxt.step0) * STEP;
        const uint32_t cnt = nxt.n - v0 < STEP ? (uint32_t)(nxt.n - v0) : (uint32_t)STEP;
        const float* src = nxt.x + v0;
        uint8_t* d = buf[warp][b];
        if (((uintptr_t)src & 15) == 0 && cnt == STEP) {
#pragma unroll
            for (int k = 0; k < STEP / 128; k++) cp_async16(d + 16 * swz16(lane) + 512 * k, src + 4 * lane + 128 * k);
        } else {
            for (uint32_t i = lane; i < cnt; i += 32) cp_async_small<4>(d + swz_off<float>(i), src + i);
        }
        cp_async_commit();
    };
    unsigned long long pay = 0;
    uint32_t nnc = 0;
    auto flush = [&]() {
        const unsigned long long p = warp_sum(pay);
        const uint32_t c = __reduce_add_sync(0xffffffffu, nnc);
        if (lane == 0 && c) {
            atomicAdd(&acc[2 * it], p);
            atomicAdd(&acc[2 * it + 1], (unsigned long long)c);
        }
        pay = 0;
        nnc = 0;
    };
    int eb_exp = exponent_f64_of_f32(cur.eb);
    load(u0, 0);
    for (unsigned long long u = u0; u < u1; u++) {
        const int b = (int)(u - u0) & 1;
        if (u + 1 < u1) {
            load(u + 1, b ^ 1);
            cp_async_wait_group<1>();
        } else {
            cp_async_wait_all();
        }
        __syncwarp();
        if (it + 1 < ni && items[it + 1].step0 <= u) {
            flush();
            while (it + 1 < ni && items[it + 1].step0 <= u) it++;
            cur = items[it];
            eb_exp = exponent_f64_of_f32(cur.eb);
        }
        const unsigned long long v = (u - cur.step0) * STEP + (unsigned long long)(seg * BS);
        const int len = v >= cur.n ? 0 : (cur.n - v < BS ? (int)(cur.n - v) : BS);
        BlockEnc<float, G> e;
        if (__all_sync(0xffffffffu, len == BS))
            enc_block_stats<float, G, true>(buf[warp][b], seg * BS, len, true, cur.eb, eb_exp, 0ull, 0, e);
        else
            enc_block_stats<float, G, false>(buf[warp][b], seg * BS, len, true, cur.eb, eb_exp, 0ull, 0, e);
        if (sl == 0 && e.state == 1) {
            pay += e.size;
            nnc++;
        }
        __syncwarp();   // (the buffer is copied into again by the next step)
    }
    flush();
}

cudaError_t launch_blocked_sizes(const SizeItem* d_items, int ni, unsigned long long steps, unsigned long long* d_acc,
                                 cudaStream_t s) {
    if (ni < 1 || steps == 0) return cudaErrorInvalidValue;
    static int per_sm[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!per_sm[dev]) {
        int occ = 0;
        cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_blocked_sizes, kSizeThreads, 0);
        if (e != cudaSuccess) return e;
        per_sm[dev] = occ < 1 ? 1 : occ;
    }
    const unsigned long long cap = (unsigned long long)sm_count() * per_sm[dev], want = (steps + 15) / 16;   // >= 2 steps a warp
    TraceScope tr("blocked_sizes", s);
    k_blocked_sizes<<<(unsigned)(want < cap ? want : cap), kSizeThreads, 0, s>>>(d_items, ni, steps, d_acc);
    return cudaGetLastError();
}

// Header, size index, state bits and medians (szx/src/szx_float.cc:1437-1483).
// The encoder leaves payload sizes and medians by block index; this kernel
// compacts them: an assemble tile covers kAsmWords state words (32 blocks
// each), the non-constant rank of its first block comes from an inline-prefix
// look-back over the tiles' popcounts, and each block then writes its size
// (non-constant, by rank) or its median (constant, by constant rank).  The
// sizes and medians are loaded before the look-back, not behind it: 2^20
// blocks 25.5 -> 20.5 us, 2^22 blocks 55 -> 38.  (The index's CTA-wide
// look-back: 22.4.)
constexpr int kAsmThreads = 256;
constexpr int kAsmWords = (int)(kAsmBlocksPerTile / 32);
constexpr int kAsmItems = (int)kAsmBlocksPerTile / kAsmThreads;   // blocks a thread

struct AsmArgs {
    BlkField one;                // the field when nf == 1
    const BlkField* fields;      // nf > 1: device table in ascending asm_tile0
    int nf;
    int layout;
    unsigned long long bs;
    unsigned long long total_tiles;
    unsigned long long* ctr;     // [0] tile counter, [1] finished CTAs
    int* err;
};

// Header of field F (szx/src/szx_float.cc:1437-1447) and its result record.
__device__ __forceinline__ void asm_header(const BlkField* F, int layout, unsigned long long bs, int status) {
    const unsigned long long nb = F->nb, nnc = F->tot->nnc, nc = nb - nnc, sb = (nb + 7) / 8;
    const bool ra = layout != kBlocked;
    const unsigned long long hdr = ra ? 20 : 13;
    const unsigned long long shift = ra ? 2 * nnc : 4 * nnc;
    uint8_t* s = F->out + shift;
    s[0] = 1; s[1] = 1; s[2] = 1; s[3] = ra ? 1 : 0;
    if (ra) {
        for (int k = 0; k < 8; k++) s[4 + k] = (uint8_t)(bs >> (56 - 8 * k));
        for (int k = 0; k < 8; k++) s[12 + k] = (uint8_t)(nc >> (56 - 8 * k));
    } else {
        s[4] = (uint8_t)bs;
        for (int k = 0; k < 8; k++) s[5 + k] = (uint8_t)(nc >> (56 - 8 * k));
    }
    StreamResult r;
    r.offset = shift;
    r.size = hdr + (ra ? 2 * nnc : 0) + sb + 4 * nc + F->tot->payload_bytes;
    r.nb_const = nc;
    r.eb = F->params ? F->params->eb : F->eb;
    r.status = status;
    *F->res = r;
}

__global__ void __launch_bounds__(kAsmThreads, 4) k_blocked_assemble(AsmArgs a) {
    pdl_start();
    __shared__ uint32_t s_word[kAsmWords], s_pre[kAsmWords];
    __shared__ uint32_t s_wsum[kAsmThreads / 32];
    __shared__ long long s_t;
    __shared__ int s_f;
    __shared__ unsigned long long s_base;
    __shared__ int s_last;
    __shared__ BlkField s_one;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool ra = a.layout != kBlocked;
    if (tid == 0 && a.nf == 1) s_one = a.one;
    for (;;) {
        if (tid == 0) {
            const long long g = (long long)atomicAdd(a.ctr, 1ull);
            int f = 0;
            if (a.nf > 1 && g < (long long)a.total_tiles) {
                int lo = 0, hi = a.nf - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if ((long long)a.fields[mid].asm_tile0 <= g) lo = mid;
                    else hi = mid - 1;
                }
                f = lo;
            }
            s_t = g;
            s_f = f;
        }
        __syncthreads();
        if (s_t >= (long long)a.total_tiles) break;
        const BlkField* F = a.nf == 1 ? &s_one : a.fields + s_f;
        const long long t = s_t - (long long)F->asm_tile0;
        const unsigned long long nb = F->nb, nnc = F->tot->nnc, sb = (nb + 7) / 8;
        const unsigned long long hdr = ra ? 20 : 13;
        uint8_t* O = F->out + (ra ? 2 * nnc : 4 * nnc) + hdr;
        uint8_t* R = O + (ra ? 2 * nnc : 0);
        uint8_t* M = R + sb;
        const bool o_aligned = ((uintptr_t)O & 1) == 0;
        const unsigned long long nw = (nb + 31) / 32;
        const unsigned long long w = (unsigned long long)t * kAsmWords + tid;
        uint32_t word = 0;
        if (tid < kAsmWords && w < nw) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const unsigned long long bi = 4 * w + j;
                const uint32_t byte = bi < sb ? (uint32_t)F->s_scr[bi] : 0u;
                word = (word << 8) | byte;
                if (bi < sb) R[bi] = (uint8_t)byte;
            }
        }
        const uint32_t pc = __popc(word);
        const uint32_t incl = warp_inclusive_sum(pc);
        if (lane == 31) s_wsum[warp] = incl;
        if (tid < kAsmWords) s_word[tid] = word;
        __syncthreads();
        // every block's size or median, in flight during the look-back
        const unsigned long long b0 = (unsigned long long)t * kAsmWords * 32;
        uint32_t val[kAsmItems];
#pragma unroll
        for (int k = 0; k < kAsmItems; k++) {
            const int lb = k * kAsmThreads + tid;
            const unsigned long long b = b0 + lb;
            val[k] = 0;
            if (b < nb) {
                if ((s_word[lb >> 5] >> (31 - (lb & 31))) & 1u) {
                    if (ra) val[k] = F->size_blk[b];
                } else {
                    val[k] = F->med_blk[b];
                }
            }
        }
        uint32_t wpre = 0, agg = 0;
#pragma unroll
        for (int k = 0; k < kAsmThreads / 32; k++) {
            const uint32_t v = s_wsum[k];
            wpre += k < warp ? v : 0u;
            agg += v;
        }
        if (tid < kAsmWords) s_pre[tid] = wpre + incl - pc;
        if (warp == 0) {
            prefix_publish(F->st_asm, t, agg);
            const unsigned long long base = prefix_resolve(F->st_asm, t, agg, a.err);
            if (lane == 0) s_base = base;
        }
        __syncthreads();
        const unsigned long long base = s_base;
#pragma unroll
        for (int k = 0; k < kAsmItems; k++) {
            const int lb = k * kAsmThreads + tid;
            const unsigned long long b = b0 + lb;
            if (b >= nb) break;
            const uint32_t wd = s_word[lb >> 5];
            const int bit = lb & 31;
            const unsigned long long rank = base + s_pre[lb >> 5] + (bit ? __popc(wd >> (32 - bit)) : 0);
            if ((wd >> (31 - bit)) & 1u) {
                if (ra) {
                    const uint16_t v = (uint16_t)val[k];
                    if (o_aligned) {
                        *(uint16_t*)(O + 2 * rank) = v;   // little-endian u16
                    } else {
                        O[2 * rank] = (uint8_t)v;
                        O[2 * rank + 1] = (uint8_t)(v >> 8);
                    }
                }
            } else {
                const uint32_t v = val[k];
                uint8_t* q = M + 4 * (b - rank);
                if (a.layout == kRandomAccessNative) {
                    q[0] = (uint8_t)v; q[1] = (uint8_t)(v >> 8); q[2] = (uint8_t)(v >> 16); q[3] = (uint8_t)(v >> 24);
                } else {
                    q[0] = (uint8_t)(v >> 24); q[1] = (uint8_t)(v >> 16); q[2] = (uint8_t)(v >> 8); q[3] = (uint8_t)v;
                }
            }
        }
        __syncthreads();
    }
    // the last CTA to finish writes every field's header and result record
    if (tid == 0) {
        __threadfence();
        s_last = atomicAdd(&a.ctr[1], 1ull) == (unsigned long long)gridDim.x - 1;
    }
    __syncthreads();
    if (s_last) {
        __threadfence();
        const int status = *(volatile int*)a.err;
        for (int f = tid; f < a.nf; f += kAsmThreads) asm_header(a.nf == 1 ? &s_one : a.fields + f, a.layout, a.bs, status);
    }
}

size_t blocked_bound(int layout, int dtype, size_t n, int bs) {
    size_t es = dtype == 0 ? 4 : 8;
    size_t nb = (n + bs - 1) / bs, sb = (nb + 7) / 8;
    size_t hdr = layout == kBlocked ? 13 : 20;
    return hdr + sb + 4 * nb + nb * (5 + ((size_t)bs + 3) / 4) + es * n + 64;
}

// ctas_per_sm: 0 as many as fit, else at most that many.
template <typename T, int G, int TBYTES = kEncTileBytes>
static cudaError_t run_encode(EncArgs a, const LaunchShape& shape, cudaStream_t s) {
    const int ctas_per_sm = shape.enc_ctas_per_sm;
    using TL = EncTile<T, G, TBYTES>;
    static bool attr_set[64] = {false};
    static int per_sm[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!attr_set[dev]) {
        // the ring needs the largest shared-memory carveout for 3 CTAs per SM
        cudaError_t e = cudaSuccess;
        for (auto k : {k_blocked_encode<T, G, false, TBYTES>, k_blocked_encode<T, G, true, TBYTES>}) {
            if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, TL::kDynSmem);
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        }
        int occ = 0;
        if (e == cudaSuccess)
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_blocked_encode<T, G, false, TBYTES>,
                                                              TL::kThreads, TL::kDynSmem);
        if (e != cudaSuccess) return e;
        per_sm[dev] = occ < 1 ? 1 : occ;
        attr_set[dev] = true;
    }
    const int cps = ctas_per_sm > 0 && ctas_per_sm < per_sm[dev] ? ctas_per_sm : per_sm[dev];
    const size_t g = (size_t)sm_count() * cps;
    const int grid = (int)(a.total_tiles < g ? a.total_tiles : g);
    TraceScope tr("blocked_encode", s);
    auto k = a.nf == 1 ? k_blocked_encode<T, G, false, TBYTES> : k_blocked_encode<T, G, true, TBYTES>;
    if (shape.after_kernel) return launch_after(k, grid, TL::kThreads, TL::kDynSmem, s, a);
    k<<<grid, TL::kThreads, TL::kDynSmem, s>>>(a);
    return cudaGetLastError();
}
// The one encoder tile variant a launch shape can pick besides the default:
// 8 KiB tiles (16 blocks, 4 warps, 6 CTAs per SM) for float blocks of 65..128
// values.
constexpr int kEncTileBytesSmall = 8192;

static int lanes_for_bs(int dtype, int bs) {
    const int per = dtype == 0 ? 16 : 8;   // values per lane
    const int need = (bs + per - 1) / per;
    return need <= 1 ? 1 : need <= 2 ? 2 : need <= 4 ? 4 : need <= 8 ? 8 : need <= 16 ? 16 : 32;
}

int blocked_tile_blocks(int dtype, int bs, int tile_variant) {
    const int G = lanes_for_bs(dtype, bs);
    if (tile_variant == 1 && dtype == 0 && G == 8) return EncTile<float, 8, kEncTileBytesSmall>::kBlocks;
    if (dtype == 0) {
        switch (G) {
            case 1: return EncTile<float, 1>::kBlocks;
            case 2: return EncTile<float, 2>::kBlocks;
            case 4: return EncTile<float, 4>::kBlocks;
            case 8: return EncTile<float, 8>::kBlocks;
            default: return EncTile<float, 16>::kBlocks;
        }
    }
    switch (G) {
        case 1: return EncTile<double, 1>::kBlocks;
        case 2: return EncTile<double, 2>::kBlocks;
        case 4: return EncTile<double, 4>::kBlocks;
        case 8: return EncTile<double, 8>::kBlocks;
        case 16: return EncTile<double, 16>::kBlocks;
        default: return EncTile<double, 32>::kBlocks;
    }
}

cudaError_t launch_blocked_encode_fields(int layout, int dtype, int bs, int nf, const BlkField& one,
                                         const BlkField* d_fields, const uint32_t* d_tile_field,
                                         unsigned long long enc_total, unsigned long long asm_total,
                                         unsigned long long* counters, int* err, cudaStream_t s,
                                         const LaunchShape& shape) {
    if (nf < 1 || enc_total == 0 || enc_total > 0x7FFFFFFFull || (nf > 1 && !d_tile_field)) return cudaErrorInvalidValue;
    EncArgs a;
    a.one = one;
    a.fields = d_fields;
    a.nf = nf;
    a.bs = bs;
    a.omp_stats = layout == kRandomAccessNative;
    a.total_tiles = enc_total;
    a.tile_ctr = &counters[0];
    a.tile_field = d_tile_field;
    a.err = err;
    cudaError_t e;
    const int G = lanes_for_bs(dtype, bs);
    if (dtype == 0) {
        switch (G) {
            case 1: e = run_encode<float, 1>(a, shape, s); break;
            case 2: e = run_encode<float, 2>(a, shape, s); break;
            case 4: e = run_encode<float, 4>(a, shape, s); break;
            case 8:
                e = shape.enc_tile_variant == 1
                        ? run_encode<float, 8, kEncTileBytesSmall>(a, shape, s)
                        : run_encode<float, 8>(a, shape, s);
                break;
            default: e = run_encode<float, 16>(a, shape, s); break;
        }
    } else {
        switch (G) {
            case 1: e = run_encode<double, 1>(a, shape, s); break;
            case 2: e = run_encode<double, 2>(a, shape, s); break;
            case 4: e = run_encode<double, 4>(a, shape, s); break;
            case 8: e = run_encode<double, 8>(a, shape, s); break;
            case 16: e = run_encode<double, 16>(a, shape, s); break;
            default: e = run_encode<double, 32>(a, shape, s); break;
        }
    }
    if (e != cudaSuccess) return e;
    AsmArgs m;
    m.one = one;
    m.fields = d_fields;
    m.nf = nf;
    m.layout = layout;
    m.bs = (unsigned long long)bs;
    m.total_tiles = asm_total;
    m.ctr = &counters[1];
    m.err = err;
    const size_t gmax = (size_t)sm_count() * 4;
    const int ag = (int)(asm_total < gmax ? (asm_total ? asm_total : 1) : gmax);
    TraceScope tr("blocked_assemble", s);
    return launch_after(k_blocked_assemble, ag, kAsmThreads, 0, s, m);
}

ClearList blocked_enc_clear(const Workspace& ws, size_t nb) {
    ClearList c{};
    c.p[0] = ws.st_word;
    c.bytes[0] = 8 * blocked_status_words(nb);
    c.p[1] = ws.totals;
    c.bytes[1] = kWsHeaderClear;
    c.n = 2;
    return c;
}

cudaError_t launch_blocked_encode(int layout, int dtype, const void* x, size_t n, int bs, bool use_params,
                                  float abs_eb, uint8_t* d_out, size_t cap, const Workspace& ws, cudaStream_t s,
                                  bool cleared, StreamResult* res_out) {
    if (n == 0 || bs < 1 || bs > 256) return cudaErrorInvalidValue;
    if (layout == kBlocked && bs > 255) return cudaErrorInvalidValue;
    const size_t nb = (n + bs - 1) / bs, sb = (nb + 7) / 8;
    const size_t hdr = layout == kBlocked ? 13 : 20;
    const size_t qfix = hdr + sb + 4 * nb;
    if (cap < qfix) return cudaErrorInvalidValue;
    cudaError_t e;
    // status words of both look-backs, then totals / result / error / counters
    if (!cleared && (e = launch_ws_clear(blocked_enc_clear(ws, nb), s)) != cudaSuccess) return e;
    const size_t tb = (size_t)blocked_tile_blocks(dtype, bs, 0);
    BlkField F;
    F.x = x; F.n = n; F.nb = nb;
    F.enc_tiles = (nb + tb - 1) / tb; F.enc_tile0 = 0;
    F.asm_tiles = (nb + kAsmBlocksPerTile - 1) / kAsmBlocksPerTile; F.asm_tile0 = 0;
    F.eb = abs_eb; F.pad = 0;
    F.params = use_params ? ws.params : nullptr;
    F.out = d_out;
    F.payload = d_out + qfix;
    F.payload_cap = cap - qfix;
    F.st_enc = ws.st_word;
    F.st_asm = ws.st_word + enc_status_words(nb);   // encoder's words first
    F.size_blk = ws.o_scr; F.med_blk = ws.m_scr; F.s_scr = ws.s_scr;
    F.tot = ws.totals;
    F.res = res_out ? res_out : ws.result;
    LaunchShape shape;
    shape.after_kernel = true;   // the clear, or the value-range pass
    return launch_blocked_encode_fields(layout, dtype, bs, 1, F, nullptr, nullptr, F.enc_tiles, F.asm_tiles,
                                        ws.counters, ws.err, s, shape);
}

// ------------------------------------------------------------------ decode

__device__ __forceinline__ unsigned long long be64(const uint8_t* p) {
    unsigned long long v = 0;
    for (int i = 0; i < 8; i++) v = (v << 8) | p[i];
    return v;
}

// Parse and validate the mode-3/4 header (szx/src/szxd_float.cc:402-434).
__device__ BlockedHdr parse_blocked(const uint8_t* s, unsigned long long len, unsigned long long n,
                                    unsigned long long bs_expect) {
    BlockedHdr r = {};
    r.n = n;
    r.ok = 0;
    if (len >= 20 && s[3] == 1) {
        r.bs = be64(s + 4);
        r.nc = be64(s + 12);
        if (r.bs >= 1 && r.bs <= 256 && (bs_expect == 0 || r.bs == bs_expect)) {
            r.nb = (n + r.bs - 1) / r.bs;
            r.sb = (r.nb + 7) / 8;
            if (r.nc <= r.nb) {
                r.nnc = r.nb - r.nc;
                r.o_off = 20;
                r.s_off = 20 + 2 * r.nnc;
                r.m_off = r.s_off + r.sb;
                r.q_off = r.m_off + 4 * r.nc;
                r.ok = r.q_off <= len;
            }
        }
    }
    return r;
}

// Parse and validate the mode-2 header (szx/src/szxd_float.cc:247-270).
__device__ BlockedHdr parse_m2(const uint8_t* s, unsigned long long len, unsigned long long n,
                               unsigned long long bs_expect) {
    BlockedHdr r = {};
    r.n = n;
    r.ok = 0;
    if (len >= 13 && s[3] == 0) {
        r.bs = s[4];
        r.nc = be64(s + 5);
        if (r.bs >= 1 && (bs_expect == 0 || r.bs == bs_expect)) {
            r.nb = (n + r.bs - 1) / r.bs;
            r.sb = (r.nb + 7) / 8;
            if (r.nc <= r.nb) {
                r.nnc = r.nb - r.nc;
                r.o_off = 13;
                r.s_off = 13;
                r.m_off = r.s_off + r.sb;
                r.q_off = r.m_off + 4 * r.nc;
                r.ok = r.q_off <= len;
            }
        }
    }
    return r;
}

// First kernel of a decode: the index kernel's counter and status words
// cleared, the header parsed (thread 0) into *h and the error word set.
__global__ void k_blocked_begin(ClearList c, const uint8_t* s, unsigned long long len, unsigned long long n,
                                unsigned long long bs_expect, int m2, BlockedHdr* h, int* err) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (tid == 0) {
        const BlockedHdr r = m2 ? parse_m2(s, len, n, bs_expect) : parse_blocked(s, len, n, bs_expect);
        *h = r;
        *err = r.ok ? kErrNone : kErrStream;
    }
    for (int r = 0; r < c.n; r++)
        for (size_t i = tid; i < c.bytes[r] / 4; i += (size_t)gridDim.x * blockDim.x) ((uint32_t*)c.p[r])[i] = 0u;
}

// The whole of it for a stream of at most kIdxSmallBlocks blocks: header,
// payload offsets and rank words by one CTA, without counter, status words or
// their clearing.  (The parse, clear and index kernels took three launches.)
constexpr int kIdxSmallThreads = 1024, kIdxSmallPer = 16;
constexpr size_t kIdxSmallBlocks = (size_t)kIdxSmallThreads * kIdxSmallPer;
__global__ void __launch_bounds__(kIdxSmallThreads) k_blocked_index_small(const uint8_t* s, unsigned long long len,
                                                                          unsigned long long n,
                                                                          unsigned long long bs_expect, int m2,
                                                                          BlockedHdr* hp, int* err,
                                                                          unsigned long long* P, uint32_t* RW) {
    __shared__ uint32_t s_w[2][32];
    __shared__ BlockedHdr s_h;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        const BlockedHdr r = m2 ? parse_m2(s, len, n, bs_expect) : parse_blocked(s, len, n, bs_expect);
        s_h = r;
        *hp = r;
        *err = r.ok ? kErrNone : kErrStream;
    }
    __syncthreads();
    const BlockedHdr h = s_h;
    if (!h.ok || h.nb > kIdxSmallBlocks) {
        if (h.ok && tid == 0) *err = kErrStream;   // (not reached: the host sized the launch by the same count)
        return;
    }
    // payload sizes of ranks 16 tid .. (no size index in fastMode 2), population of state word tid
    const uint32_t nnc = m2 ? 0u : (uint32_t)h.nnc, nw = (uint32_t)((h.nb + 31) / 32);
    uint32_t v[kIdxSmallPer], mine = 0, pc = 0;
#pragma unroll
    for (int i = 0; i < kIdxSmallPer; i++) {
        const uint32_t k = kIdxSmallPer * tid + i;
        v[i] = k < nnc ? (uint32_t)s[h.o_off + 2 * k] | (uint32_t)s[h.o_off + 2 * k + 1] << 8 : 0u;
        mine += v[i];
    }
    if ((uint32_t)tid < nw)
        for (int j = 0; j < 4; j++) {
            const uint32_t bi = 4 * tid + j;
            if (bi < h.sb) pc += __popc((uint32_t)s[h.s_off + bi]);
        }
    const uint32_t ia = warp_inclusive_sum(mine), ib = warp_inclusive_sum(pc);
    if (lane == 31) {
        s_w[0][warp] = ia;
        s_w[1][warp] = ib;
    }
    __syncthreads();
    if (warp < 2) {
        const uint32_t w = s_w[warp][lane];
        s_w[warp][lane] = warp_inclusive_sum(w) - w;
    }
    __syncthreads();
    unsigned long long run = (unsigned long long)s_w[0][warp] + ia - mine;   // < 16384 * 65536
#pragma unroll
    for (int i = 0; i < kIdxSmallPer; i++) {
        const uint32_t k = kIdxSmallPer * tid + i;
        if (k < nnc) P[k] = run;
        run += v[i];
        if (k + 1 == nnc) {
            P[nnc] = run;
            if (h.q_off + run > len) *err = kErrStream;
        }
    }
    if ((uint32_t)tid < nw) RW[tid] = s_w[1][warp] + ib - pc;
}

// Every stream of a batch: one thread per field.
__global__ void k_blocked_parse_fields(const DecField* F, int nf, unsigned long long bs) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nf) return;
    const DecField& D = F[f];
    const BlockedHdr r = parse_blocked(D.s, D.len, D.n, bs);
    *D.hdr = r;
    if (!r.ok) *D.err = kErrStream;
}

// CTA-wide exclusive sum over kIdxThreads threads.
__device__ __forceinline__ uint32_t cta_exclusive_sum(uint32_t v, uint32_t* total, uint32_t* smem /*[8]*/) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t incl = warp_inclusive_sum(v);
    if (lane == 31) smem[warp] = incl;
    __syncthreads();
    uint32_t wpre = 0, tot = 0;
#pragma unroll
    for (int w = 0; w < kIdxThreads / 32; w++) {
        const uint32_t x = smem[w];
        if (w < warp) wpre += x;
        tot += x;
    }
    *total = tot;
    return wpre + incl - v;
}

// Two independent exclusive scans:
//   family A: payload offsets  P[k] = sum O[0..k)          (k < nnc)
//   family B: rank words       RW[w] = popcount(state < 32w) (w < ceil(nb/32))
// One tile (kIdxPerTile items, kIdxItems consecutive ones a thread) of either,
// by the whole CTA.  st: the family's status words.
//
// Bound by latency: 2^20 blocks are 528 tiles, all resident, 2 + 8 MB of
// traffic.  With items loaded a byte at a time, results stored 8 bytes at a
// time and a look-back by one warp, 32 words and two dependent loads a round,
// it took 21.6 us (between events); words, 32-byte stores and inline prefixes
// alone 22.7, with the look-back over 1024 words at once 15.7.
__device__ __forceinline__ void index_tile(const uint8_t* s, const BlockedHdr& h, unsigned long long* P, uint32_t* RW,
                                           unsigned long long* st, bool famA, long long lt, unsigned long long len,
                                           int* err, uint32_t* sm, unsigned long long* s_base) {
    static_assert((unsigned long long)kIdxThreads * kIdxItems == kIdxPerTile && kIdxItems == 8, "index tile size");
    const unsigned long long nw = (h.nb + 31) / 32, items = famA ? h.nnc : nw;
    const unsigned long long first = (unsigned long long)lt * kIdxPerTile + threadIdx.x * kIdxItems;
    const bool all = first + kIdxItems <= items;
    uint32_t vals[kIdxItems];
    uint32_t w4[4], w8[8];
    if (famA && all && load_words<4>(s + h.o_off + 2 * first, s + len, w4)) {
#pragma unroll
        for (int i = 0; i < kIdxItems; i++) vals[i] = (w4[i >> 1] >> (16 * (i & 1))) & 0xFFFFu;
    } else if (!famA && 4 * (first + kIdxItems) <= h.sb && load_words<8>(s + h.s_off + 4 * first, s + len, w8)) {
#pragma unroll
        for (int i = 0; i < kIdxItems; i++) vals[i] = __popc(w8[i]);
    } else {
#pragma unroll
        for (int i = 0; i < kIdxItems; i++) {
            const unsigned long long k = first + i;
            uint32_t v = 0;
            if (famA) {
                if (k < h.nnc) v = (uint32_t)s[h.o_off + 2 * k] | ((uint32_t)s[h.o_off + 2 * k + 1] << 8);
            } else if (k < nw) {
                for (int j = 0; j < 4; j++) {
                    const unsigned long long bi = 4 * k + j;
                    v += bi < h.sb ? __popc((uint32_t)s[h.s_off + bi]) : 0;
                }
            }
            vals[i] = v;
        }
    }
    uint32_t mine = 0;
#pragma unroll
    for (int i = 0; i < kIdxItems; i++) mine += vals[i];
    uint32_t tot;
    const uint32_t ex = cta_exclusive_sum(mine, &tot, sm);
    if (threadIdx.x < 32) prefix_publish(st, lt, tot);
    // (a workspace need not be aligned to a sector)
    const bool wide = all && ((uintptr_t)(famA ? (const void*)P : (const void*)RW) & 31) == 0;
    const unsigned long long run0 = prefix_resolve_cta<kIdxThreads / 32>(st, lt, tot, err, s_base) + ex;
    if (famA) {
        unsigned long long run = run0;
        double q[kIdxItems];   // (a store's type: the offsets' bits)
#pragma unroll
        for (int i = 0; i < kIdxItems; i++) {
            const unsigned long long k = first + i;
            q[i] = __longlong_as_double((long long)run);
            if (!wide && k < h.nnc) P[k] = run;
            run += vals[i];
            if (k + 1 == h.nnc) {
                P[h.nnc] = run;
                if (h.q_off + run > len) atomicExch(err, kErrStream);
            }
        }
        if (wide) {
            st_v8((double*)(P + first), q);
            st_v8((double*)(P + first) + 4, q + 4);
        }
    } else {
        uint32_t run = (uint32_t)run0;
        float q[kIdxItems];
#pragma unroll
        for (int i = 0; i < kIdxItems; i++) {
            q[i] = __uint_as_float(run);
            if (!wide && first + i < nw) RW[first + i] = run;
            run += vals[i];
        }
        if (wide) st_v8((float*)(RW + first), q);
    }
    __syncthreads();
}

// The scans of one stream in one persistent launch (family A first).
__global__ void __launch_bounds__(kIdxThreads) k_blocked_index(const uint8_t* s, const BlockedHdr* hp,
                                                               unsigned long long* P, uint32_t* RW,
                                                               unsigned long long* stA, unsigned long long* stB,
                                                               unsigned long long* ctr, int* err,
                                                               unsigned long long len, int famA) {
    pdl_start();
    __shared__ uint32_t sm[8];
    __shared__ long long s_tile;
    __shared__ unsigned long long s_base[8];
    const BlockedHdr h = *hp;
    if (!h.ok) return;
    const unsigned long long nw = (h.nb + 31) / 32;
    const long long TA = famA ? (long long)((h.nnc + kIdxPerTile - 1) / kIdxPerTile) : 0;   // no size index in fastMode 2
    const long long TBt = (long long)((nw + kIdxPerTile - 1) / kIdxPerTile);
    for (;;) {
        if (threadIdx.x == 0) s_tile = (long long)atomicAdd(ctr, 1ull);
        __syncthreads();
        long long t = s_tile;
        if (t >= TA + TBt) break;
        const bool fa = t < TA;
        index_tile(s, h, P, RW, fa ? stA : stB, fa, fa ? t : t - TA, len, err, sm, s_base);
    }
}

// The scans of every stream of a batch: tiles in field order (each field's
// offset tiles, then its rank tiles) from one counter; a field whose header
// failed, and offset tiles past a field's real nnc, do nothing.
__global__ void __launch_bounds__(kIdxThreads) k_blocked_index_fields(const DecField* F, int nf,
                                                                      unsigned long long total,
                                                                      unsigned long long* ctr) {
    __shared__ uint32_t sm[8];
    __shared__ long long s_tile;
    __shared__ int s_f;
    __shared__ unsigned long long s_base[8];
    for (;;) {
        if (threadIdx.x == 0) {
            const long long g = (long long)atomicAdd(ctr, 1ull);
            int lo = 0, hi = nf - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if ((long long)F[mid].idx_tile0 <= g) lo = mid;
                else hi = mid - 1;
            }
            s_tile = g;
            s_f = lo;
        }
        __syncthreads();
        const long long g = s_tile;
        if (g >= (long long)total) break;
        const DecField& D = F[s_f];
        const BlockedHdr h = *D.hdr;
        const long long local = g - (long long)D.idx_tile0;
        const bool fa = local < (long long)D.idxA_tiles;
        const long long lt = fa ? local : local - (long long)D.idxA_tiles;
        const long long TA = (long long)((h.nnc + kIdxPerTile - 1) / kIdxPerTile);
        if (h.ok && (!fa || lt < TA)) {
            index_tile(D.s, h, D.P, D.RW, fa ? D.stA : D.stB, fa, lt, D.len, D.err, sm, s_base);
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------ decode, per block
//
// One block by a segment of G lanes; p: its payload (shared address).  Lane
// sl decodes the E consecutive values [E*sl, E*sl + E).
//
// A value's top `lead` bytes are its predecessor's (szx/src/szxd_float.cc:
// 431-470).  What a lane inherits from before its run is found first, from
// its lead codes alone: per top byte lane the last value that stored it and
// where, three byte loads, and a "last writer" scan over the G lanes.  Then one
// pass over the run finishes the values in order: the four (eight) payload
// bytes that END with a value's last one hold its stored bytes on top, so two
// funnel shifts put them under the bytes kept from the previous value -- no
// masks, and no second pass to merge what was inherited.
//
// FULL: every segment of the warp decodes a whole block of G*E values (no
// range checks); otherwise values at or past len are ignored.
// vec: 0 scalar stores, 1 16-byte stores, 2 32-byte stores (the output's
// alignment and the block's byte size allow them).
template <typename T, int G, bool FULL>
__device__ __forceinline__ void dec_segment(uint32_t p, int len, T* ob, int vec, const uint32_t* lut_ld) {
    using EL = Elem<T>;
    using U = typename EL::U;
    constexpr int E = EncCfg<T>::E;
    constexpr int NC = E / 4;
    const int sl = (int)(lane_id() & (G - 1));
    int reqLength = (int)lds8(p);
    const uint32_t mb = (lds8(p + 1) << 24) | (lds8(p + 2) << 16) | (lds8(p + 3) << 8) | lds8(p + 4);
    const int Lb = FULL ? G * NC : (len + 3) / 4;
    const int nv = FULL ? E : (len - E * sl < 0 ? 0 : (len - E * sl < E ? len - E * sl : E));   // the lane's values
    // the lane's lead bytes, chunk k in byte k
    const uint32_t lp = p + 5 + NC * sl;
    uint32_t codes = __funnelshift_r(lds32(lp & ~3u), lds32((lp & ~3u) + 4), 8 * lp);
    if constexpr (NC == 2) codes &= 0xFFFFu;
    int R = (reqLength + 7) >> 3;
    if (!__all_sync(0xffffffffu, plain_req<T>(reqLength))) {   // (one vote: no lane pays for what no encoder here writes)
        reqLength = clamp_req<T>(reqLength);
        R = run_bytes(reqLength);
        if (one_byte_req(reqLength)) codes = one_byte_codes(codes);
    }
    const RunLeads<E> leads(codes, nv, R);
    const uint32_t incl = seg_inclusive_sum<G>(leads.bytes());
    const uint32_t q0 = p + 5 + (uint32_t)Lb + incl - leads.bytes();   // the run's first byte
    uint32_t sv, sw;   // the top three bytes as the lane leaves them, and which of them it wrote
    leads.summary(q0, sv, sw);
#pragma unroll
    for (int d = 1; d < G; d <<= 1) {
        const uint32_t ov = __shfl_up_sync(0xffffffffu, sv, d, G), ow = __shfl_up_sync(0xffffffffu, sw, d, G);
        if (sl >= d) {
            sv = (ov & ~sw) | (sv & sw);
            sw |= ow;
        }
    }
    const uint32_t ex = __shfl_up_sync(0xffffffffu, sv, 1, G);
    const uint32_t carry = sl ? ex << 8 : 0u;   // top three bytes of a 32-bit word (zero before the block)
    const T med = widen_median<T>(__uint_as_float(mb));
    U cur[E];
    T v[E];
    const bool bad = run_decode<T, E, FULL>(codes, nv, R, reqLength, q0, carry, med, lut_ld, cur, v);
    if (__any_sync(0xffffffffu, bad && len > 0)) {
#pragma unroll
        for (int e = 0; e < E; e++) v[e] = xadd(EL::of(cur[e]), med);
    }
    // store the lane's E consecutive values (a segment called with len 0 --
    // a constant block, whose median is already stored -- stores nothing)
    const int f0 = E * sl;
    constexpr int V8 = 32 / (int)sizeof(T);   // values per 32-byte store
    if (vec == 2 && f0 + E <= len) {
#pragma unroll
        for (int k = 0; k < E / V8; k++) st_v8(ob + f0 + V8 * k, v + V8 * k);
    } else if (vec && f0 + E <= len) {
#pragma unroll
        for (int k = 0; k < NC; k++) {
            if constexpr (sizeof(T) == 4) {
                *(float4*)(ob + f0 + 4 * k) = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
            } else {
                *(double2*)(ob + f0 + 4 * k) = make_double2(v[4 * k], v[4 * k + 1]);
                *(double2*)(ob + f0 + 4 * k + 2) = make_double2(v[4 * k + 2], v[4 * k + 3]);
            }
        }
    } else {
#pragma unroll
        for (int e = 0; e < E; e++)
            if (f0 + e < len) ob[f0 + e] = v[e];
    }
}

// ------------------------------------------------------------------ decode, pipelined tiles
//
// One producer warp per CTA walks the CTA's tiles ahead of the decoders: it
// reads the tile's state bits and first rank, the payload offsets of its
// non-constant blocks and the medians of its constant blocks, checks them,
// and stages the tile's payload bytes (one contiguous range) into a ring of
// kDecStages shared-memory buffers with a bulk copy.  Eight consumer
// warps decode a tile per step, G lanes per block, and write the values with
// 32-byte stores.  Full/empty mbarriers hand the buffers back and forth; every
// wait is bounded and reports kErrLookback instead of hanging.
//
// Bound by the integer pipe for floats (2^27 values: 177 us, 129 us of
// traffic; 240 us before the run decoder) and by the FP64 add for doubles
// (2^28 values: 727 us, 427 us of FP64 pipe and 522 us of traffic; 1117 us
// before the NaN check left that pipe).
constexpr int kDecWarps = 8;
constexpr int kDecThreadsP = (kDecWarps + 1) * 32;
constexpr int kDecStages = 3;
// 4 CTAs of 9 warps per SM (56 registers, three ring stages of shared memory,
// or two of the largest blocks': 2^28 float64 in blocks of 256 took 1010 us
// with three stages, which left three resident CTAs to a grid of four)
constexpr int kDecCtasPerSm = 4;
constexpr int kSmemPerSm = 233472;   // bytes

template <typename T, int G>
struct DecTileV {
    static constexpr int E = EncCfg<T>::E;
    static constexpr int kBsMax = G * E;
    static constexpr int kBpw = 32 / G;
    static constexpr int kBlocks = kDecWarps * kBpw;     // one segment per consumer warp and tile
    static constexpr int kMaxPay = 5 + (kBsMax + 3) / 4 + (int)sizeof(T) * kBsMax;
    // a valid tile's payloads fit kBlocks * kMaxPay; one more kMaxPay + 32
    // keeps the reads of a corrupt block inside the buffer
    static constexpr int kFront = 16;   // the decoder reads up to eight bytes before a value
    static constexpr int kStage = (kFront + ((kBlocks + 1) * kMaxPay + 32) + 15) / 16 * 16;
    // two stages where three would leave shared memory for three CTAs an SM only
    static constexpr int kStatic = 2048 + 128 + 17 * kBlocks + 1024;   // lead tables, block tables, the reserved part
    static constexpr int kStages = kDecStages * kStage + kStatic <= kSmemPerSm / kDecCtasPerSm ? kDecStages : kDecStages - 1;
    static constexpr int kDynSmem = kStages * kStage;
};

struct DecArgs {
    const uint8_t* s;
    unsigned long long len;
    const BlockedHdr* hdr;
    const unsigned long long* P;   // payload offsets by non-constant rank, [nnc + 1]
    const uint32_t* RW;            // non-constant rank at each 32-block state word
    void* out;
    int native_medians;
    int* err;                      // one stream: its error word; a batch: the launch's (bounded waits)
    const DecField* fields;        // a batch: the field table (ascending dec_tile0), else unused
    const uint32_t* tile_field;    // a batch: field of every launch-wide decode tile
    int nf, bs;
    unsigned long long total_tiles;
};

enum : uint8_t { kBlkConst = 0, kBlkCoded = 1, kBlkNone = 2 };

template <typename T, int G, bool MULTI>
__global__ void __launch_bounds__(kDecThreadsP, kDecCtasPerSm) k_blocked_decode(DecArgs a) {
    pdl_start();
    using TL = DecTileV<T, G>;
    constexpr int TB = TL::kBlocks;
    constexpr int NS = TL::kStages;
    extern __shared__ __align__(128) uint8_t dsm[];
    __shared__ unsigned long long full[NS], empty[NS];
    __shared__ uint32_t s_info[NS][TB];    // coded: payload position in the stage; constant: median bits
    __shared__ uint8_t s_kind[NS][TB];
    __shared__ uint8_t s_ok[NS];
    __shared__ int s_fld[NS];              // a batch: the tile's field
    __shared__ uint16_t s_rank[TB];        // producer scratch: rank within the tile
    __shared__ uint32_t lut_ld[512];
    BlockedHdr h = {};
    if constexpr (!MULTI) {
        h = *a.hdr;
        if (!h.ok) return;
        if (h.bs > (unsigned long long)TL::kBsMax) {
            if (threadIdx.x == 0 && blockIdx.x == 0) atomicExch(a.err, kErrStream);
            return;
        }
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < NS; i++) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], kDecWarps);
        }
        mbar_fence_init();
    }
    lead_table_init(lut_ld);
    __syncthreads();
    const long long ntiles = MULTI ? (long long)a.total_tiles : (long long)((h.nb + TB - 1) / TB);
    const int bs = MULTI ? a.bs : (int)h.bs;
    // field of a launch-wide tile (batch): one load from the plan's tile map
    auto field_of = [&](long long g) { return (int)a.tile_field[g]; };

    // The producer's copy of a tile's payload range [sa, sa + nbytes) of the
    // stream [sbeg, send): one bulk copy of the 16-byte chunks it touches, and
    // plain copies of the ends where a chunk would pass the stream's.  Byte x
    // goes to stage + kFront + (x - (sa & ~15)).
    auto copy_range = [&](uint8_t* stage, const uint8_t* src, unsigned long long nbytes, const uint8_t* sbeg,
                          const uint8_t* send, int slot) {
        if (nbytes == 0) return;
        const uintptr_t sa = (uintptr_t)src, se = sa + nbytes, base = sa & ~(uintptr_t)15;
        const uintptr_t a0 = base < (uintptr_t)sbeg ? base + 16 : base;
        uintptr_t a1 = (se + 15) & ~(uintptr_t)15;
        if (a1 > (uintptr_t)send) a1 -= 16;
        if (a1 > a0 && lane == 0) {
            fence_proxy_async();
            mbar_expect_tx(&full[slot], (uint32_t)(a1 - a0));
            tma_load_1d(stage + TL::kFront + (a0 - base), (const void*)a0, (uint32_t)(a1 - a0), &full[slot]);
        }
        uint8_t* d = stage + TL::kFront;
        const uintptr_t head = a0 < se ? a0 : se, tail = a1 > head ? a1 : head;   // plain: [sa, head) and [tail, se)
        for (uintptr_t x = sa + lane; x < head; x += 32) d[x - base] = *(const uint8_t*)x;
        for (uintptr_t x = tail + lane; x < se; x += 32) d[x - base] = *(const uint8_t*)x;
    };
    if (!MULTI && TB <= 32 && warp == kDecWarps) {
        // ---------------------------------------------------------- producer, one stream, at most 32 blocks a tile
        // Pipelined: iteration i issues the loads of tile i+2's state bits and
        // rank word and of tile i+1's offsets and medians, and stages tile i
        // from what the iteration before loaded.  (Loaded when needed, the
        // three dependent round trips took 3.2 us of a tile's 3.9, and the
        // decoders waited for them.)  Lane l holds block l of the tile's
        // 32-block state word; the tile's blocks are lanes bit0 .. bit0 + TB - 1.
        const uint8_t* S = a.s;
        auto load_a = [&](long long t, uint32_t& st, uint32_t& rw) {
            const unsigned long long w = (unsigned long long)t * TB >> 5, bi = 4 * w + (lane >> 3);
            st = bi < h.sb ? (uint32_t)S[h.s_off + bi] : 0u;
            rw = a.RW[w];
        };
        // tile t's coded blocks (bit per block), first rank, and this lane's block lb = lane
        auto blocks_of = [&](long long t) { const unsigned long long left = h.nb - (unsigned long long)t * TB; return left < (unsigned long long)TB ? (int)left : TB; };
        auto load_b = [&](long long t, uint32_t st, uint32_t rw, uint32_t& mt, uint32_t (&x)[4], uint32_t& good) {
            const unsigned long long b0 = (unsigned long long)t * TB;
            const int bit0 = (int)(b0 & 31), nblk = blocks_of(t);
            const uint32_t m = __ballot_sync(0xffffffffu, (st >> (7 - (lane & 7))) & 1u);
            const uint32_t rank0 = rw + __popc(m & ((1u << bit0) - 1u));
            mt = m >> bit0 & (nblk < 32 ? (1u << nblk) - 1u : 0xFFFFFFFFu);
            const uint32_t r = __popc(mt & ((1u << lane) - 1u));
            good = rank0 + __popc(mt) <= h.nnc;
            x[0] = x[1] = x[2] = x[3] = 0;
            if (lane < nblk) {
                if (mt >> lane & 1u) {
                    if (good) {
                        const unsigned long long k = (unsigned long long)rank0 + r, p0 = a.P[k], p1 = a.P[k + 1];
                        x[0] = (uint32_t)p0; x[1] = (uint32_t)(p0 >> 32);
                        x[2] = (uint32_t)p1; x[3] = (uint32_t)(p1 >> 32);
                    }
                } else {
                    const unsigned long long b = b0 + lane, rk = (unsigned long long)rank0 + r, mo = h.m_off + 4 * (b - rk);
                    if (b >= rk && mo + 4 <= h.q_off) {
#pragma unroll
                        for (int c = 0; c < 4; c++) x[c] = S[mo + c];
                    } else {
                        good = 0;
                    }
                }
            }
        };
        long long t = blockIdx.x, i = 0;
        const long long gs = gridDim.x;
        uint32_t stA = 0, rwA = 0, mtB = 0, xB[4] = {0, 0, 0, 0}, goodB = 0;
        if (t < ntiles) {
            load_a(t, stA, rwA);
            load_b(t, stA, rwA, mtB, xB, goodB);
        }
        if (t + gs < ntiles) load_a(t + gs, stA, rwA);
        for (; t < ntiles; t += gs, i++) {
            uint32_t stN = 0, rwN = 0, mtN = 0, xN[4] = {0, 0, 0, 0}, goodN = 0;
            if (t + 2 * gs < ntiles) load_a(t + 2 * gs, stN, rwN);
            if (t + gs < ntiles) load_b(t + gs, stA, rwA, mtN, xN, goodN);
            const int slot = (int)(i % NS);
            if (i >= NS && !mbar_wait(&empty[slot], (uint32_t)((i / NS - 1) & 1))) {
                if (lane == 0) atomicExch(a.err, kErrLookback);
                break;
            }
            uint8_t* stage = dsm + slot * TL::kStage;
            const int nblk = blocks_of(t);
            const unsigned long long p0 = ((unsigned long long)xB[1] << 32) | xB[0], p1 = ((unsigned long long)xB[3] << 32) | xB[2];
            const int first = mtB ? __ffs(mtB) - 1 : 0, last = mtB ? 31 - __clz(mtB) : 0;
            const unsigned long long pa = __shfl_sync(0xffffffffu, p0, first), pb = __shfl_sync(0xffffffffu, p1, last);
            uint32_t ok = goodB;
            if (mtB && (pb < pa || pb - pa > (unsigned long long)TB * TL::kMaxPay || h.q_off + pb > a.len)) ok = 0;
            ok = __all_sync(0xffffffffu, ok);
            const unsigned long long nbytes = ok && mtB ? pb - pa : 0;
            const uint8_t* src = S + h.q_off + pa;
            const uint32_t ph = (uint32_t)((uintptr_t)src & 15);
            copy_range(stage, src, nbytes, S, S + a.len, slot);
            if (lane < TB) {
                const bool in = lane < nblk, coded = mtB >> lane & 1u;
                uint32_t info;
                if (coded) {
                    const unsigned long long rem = h.n - ((unsigned long long)t * TB + lane) * h.bs;
                    const int blen = rem < h.bs ? (int)rem : bs;
                    const unsigned long long minsz = 5 + (unsigned long long)((blen + 3) / 4);
                    if (p0 < pa || p1 > pb || p1 < p0 + minsz || p1 - p0 > (unsigned long long)TL::kMaxPay) ok = 0;
                    info = TL::kFront + ph + (uint32_t)(p0 - pa);
                } else {
                    info = a.native_medians ? (xB[0] | (xB[1] << 8) | (xB[2] << 16) | (xB[3] << 24))
                                            : ((xB[0] << 24) | (xB[1] << 16) | (xB[2] << 8) | xB[3]);
                }
                s_info[slot][lane] = info;
                s_kind[slot][lane] = !in ? kBlkNone : (coded ? kBlkCoded : kBlkConst);
            }
            ok = __all_sync(0xffffffffu, ok);
            __threadfence_block();
            __syncwarp();
            if (lane == 0) {
                s_ok[slot] = (uint8_t)ok;
                if (!ok) atomicExch(a.err, kErrStream);
                mbar_arrive(&full[slot]);
            }
            stA = stN; rwA = rwN;
            mtB = mtN; goodB = goodN;
#pragma unroll
            for (int c = 0; c < 4; c++) xB[c] = xN[c];
        }
        // copies still in flight finish before the CTA exits
        for (long long k = i > NS ? i - NS : 0; k < i; k++) mbar_wait(&full[k % NS], (uint32_t)((k / NS) & 1));
        return;
    }
    if (warp == kDecWarps) {
        // ---------------------------------------------------------- producer, any tile
        long long i = 0;
        for (long long t = blockIdx.x; t < ntiles; t += gridDim.x, i++) {
            const int slot = (int)(i % NS);
            if (i >= NS && !mbar_wait(&empty[slot], (uint32_t)((i / NS - 1) & 1))) {
                if (lane == 0) atomicExch(a.err, kErrLookback);
                break;
            }
            uint8_t* stage = dsm + slot * TL::kStage;
            // the tile's stream: the launch's, or its field's
            const uint8_t* S = a.s;
            unsigned long long L = a.len;
            const unsigned long long* P = a.P;
            const uint32_t* RW = a.RW;
            int* ferr = a.err;
            BlockedHdr hh = h;
            long long lt = t;
            if constexpr (MULTI) {
                const int f = field_of(t);
                const DecField* D = a.fields + f;
                S = D->s; L = D->len; P = D->P; RW = D->RW; ferr = D->err;
                hh = *D->hdr;
                lt = t - (long long)D->dec_tile0;
                if (lane == 0) s_fld[slot] = f;
            }
            const unsigned long long b0 = (unsigned long long)lt * TB;
            const unsigned long long rest = hh.ok ? hh.nb - b0 : 0;   // a batch's failed header: no blocks
            const int nblk = rest < (unsigned long long)TB ? (int)rest : TB;
            // rank of the tile's first block
            const unsigned long long w = b0 >> 5;
            const int bit0 = (int)(b0 & 31);
            uint32_t word = 0;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const unsigned long long bi = 4 * w + j;
                word = (word << 8) | (bi < hh.sb ? (uint32_t)S[hh.s_off + bi] : 0u);
            }
            const unsigned long long rank0 = hh.ok ? RW[w] + (bit0 ? __popc(word >> (32 - bit0)) : 0) : 0;
            // state of every block (loads independent of the rank above)
            uint32_t ok = 1, running = 0;
            for (int j = 0; j < TB; j += 32) {
                const int lb = j + lane;
                const unsigned long long b = b0 + lb;
                const bool in = lb < nblk;
                const uint32_t coded = in ? (S[hh.s_off + (b >> 3)] >> (7 - (b & 7))) & 1u : 0u;
                const unsigned m = __ballot_sync(0xffffffffu, coded);
                const uint32_t r = running + __popc(m & ((1u << lane) - 1));
                running += __popc(m);
                if (lb < TB) {
                    s_kind[slot][lb] = !in ? kBlkNone : (coded ? kBlkCoded : kBlkConst);
                    s_rank[lb] = (uint16_t)r;   // coded: rank among the tile's coded blocks; else among them before
                }
            }
            const uint32_t nnc_t = running;
            // the tile's payload range, then its copy at once: the rest of the
            // metadata is gathered while the copy is in flight
            unsigned long long pa = 0, pb = 0;
            if (rank0 + nnc_t > hh.nnc) ok = 0;
            if (ok && nnc_t) {
                pa = P[rank0];
                pb = P[rank0 + nnc_t];
                if (pb < pa || pb - pa > (unsigned long long)TB * TL::kMaxPay || hh.q_off + pb > L) ok = 0;
            }
            const uint8_t* src = S + hh.q_off + pa;
            const uint32_t ph = (uint32_t)((uintptr_t)src & 15);
            const unsigned long long nbytes = ok ? pb - pa : 0;
            __syncwarp();
            copy_range(stage, src, nbytes, S, S + L, slot);
            // medians of the constant blocks, payload offsets of the coded ones
            for (int j = 0; j < TB; j += 32) {
                const int lb = j + lane;
                if (lb >= nblk) continue;
                const unsigned long long b = b0 + lb;
                const uint32_t r = s_rank[lb];
                if (s_kind[slot][lb] == kBlkConst) {
                    const unsigned long long mo = hh.m_off + 4 * (b - (rank0 + r));
                    uint32_t mbits = 0;
                    if (b >= rank0 + r && mo + 4 <= hh.q_off) {
                        const uint8_t* mp = S + mo;
                        mbits = a.native_medians
                                    ? ((uint32_t)mp[0] | ((uint32_t)mp[1] << 8) | ((uint32_t)mp[2] << 16) |
                                       ((uint32_t)mp[3] << 24))
                                    : (((uint32_t)mp[0] << 24) | ((uint32_t)mp[1] << 16) | ((uint32_t)mp[2] << 8) |
                                       mp[3]);
                    } else {
                        ok = 0;
                    }
                    s_info[slot][lb] = mbits;
                } else if (nbytes) {
                    const unsigned long long k = rank0 + r;
                    const unsigned long long p0 = P[k], p1 = P[k + 1];
                    const unsigned long long rem = hh.n - b * hh.bs;
                    const int blen = rem < hh.bs ? (int)rem : bs;
                    const unsigned long long minsz = 5 + (unsigned long long)((blen + 3) / 4);
                    if (p0 < pa || p1 > pb || p1 < p0 + minsz || p1 - p0 > (unsigned long long)TL::kMaxPay) ok = 0;
                    s_info[slot][lb] = TL::kFront + ph + (uint32_t)(p0 - pa);
                } else {
                    ok = 0;   // a coded block without a valid payload range
                }
            }
            ok = __all_sync(0xffffffffu, ok);
            __threadfence_block();
            __syncwarp();
            if (lane == 0) {
                s_ok[slot] = (uint8_t)ok;
                if (!ok) atomicExch(ferr, kErrStream);
                mbar_arrive(&full[slot]);
            }
        }
        // copies still in flight finish before the CTA exits
        for (long long j = i > NS ? i - NS : 0; j < i; j++) mbar_wait(&full[j % NS], (uint32_t)((j / NS) & 1));
        return;
    }

    // -------------------------------------------------------------- consumers
    T* out = (T*)a.out;
    auto vec_of = [&](const T* o) {
        const uintptr_t al = (uintptr_t)o | (uintptr_t)(bs * (int)sizeof(T));
        return (al & 31) == 0 ? 2 : ((al & 15) == 0 ? 1 : 0);
    };
    int vec = vec_of(out);
    unsigned long long n = h.n;
    const int seg = lane / G;
    const int lb = warp * TL::kBpw + seg;
    long long i = 0;
    for (long long t = blockIdx.x; t < ntiles; t += gridDim.x, i++) {
        const int slot = (int)(i % NS);
        if (!mbar_wait(&full[slot], (uint32_t)((i / NS) & 1))) {
            if (lane == 0) atomicExch(a.err, kErrLookback);
            break;
        }
        long long lt = t;
        if constexpr (MULTI) {
            const DecField* D = a.fields + s_fld[slot];
            out = (T*)D->out;
            n = D->n;
            lt = t - (long long)D->dec_tile0;
            vec = vec_of(out);
        }
        const unsigned long long b = (unsigned long long)lt * TB + lb;
        const int kind = s_kind[slot][lb];
        const uint32_t info = s_info[slot][lb];
        int blen = 0;
        T* ob = out;
        if (kind != kBlkNone) {
            const unsigned long long off = b * (unsigned long long)bs, rem = n - off;
            blen = rem < (unsigned long long)bs ? (int)rem : bs;
            ob = out + off;
        }
        if (kind == kBlkConst) {
            const T m = widen_median<T>(__uint_as_float(info));
            T v[EncCfg<T>::E];
#pragma unroll
            for (int e = 0; e < EncCfg<T>::E; e++) v[e] = m;
            store_chunks<T, G>(ob, blen, vec, v);
        }
        const bool coded = kind == kBlkCoded && s_ok[slot];
        const uint32_t pay = smem_u32(dsm + slot * TL::kStage) + (coded ? info : (uint32_t)TL::kFront);
        // the whole warp takes one path: segments that decode nothing store nothing either way
        if (__all_sync(0xffffffffu, !coded || blen == TL::kBsMax))
            dec_segment<T, G, true>(pay, coded ? blen : 0, ob, vec, lut_ld);
        else
            dec_segment<T, G, false>(pay, coded ? blen : 0, ob, vec, lut_ld);
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[slot]);
    }
}

template <typename T, int G, bool MULTI>
static cudaError_t dec_attr() {
    static bool attr_set[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attr_set[dev]) {
        cudaError_t e = cudaFuncSetAttribute(k_blocked_decode<T, G, MULTI>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, DecTileV<T, G>::kDynSmem);
        if (e != cudaSuccess) return e;
        attr_set[dev] = true;
    }
    return cudaSuccess;
}

template <typename T, int G>
static cudaError_t run_decode(const uint8_t* s, size_t len, size_t nb, const Workspace& ws, void* out, int native,
                              cudaStream_t st) {
    using TL = DecTileV<T, G>;
    cudaError_t e = dec_attr<T, G, false>();
    if (e != cudaSuccess) return e;
    const size_t tiles = (nb + TL::kBlocks - 1) / TL::kBlocks;
    const size_t cap = (size_t)sm_count() * kDecCtasPerSm;
    const int grid = (int)(tiles < cap ? (tiles ? tiles : 1) : cap);
    DecArgs a = {};
    a.s = s; a.len = len; a.hdr = ws.bhdr; a.P = ws.p_off; a.RW = ws.rank_w; a.out = out;
    a.native_medians = native; a.err = ws.err;
    TraceScope tr("blocked_decode", st);
    return launch_after(k_blocked_decode<T, G, false>, grid, kDecThreadsP, TL::kDynSmem, st, a);
}

template <typename T, int G>
static cudaError_t run_decode_fields(const DecField* F, const uint32_t* tf, int nf, int bs, unsigned long long total,
                                     int native, int* lerr, int ctas_per_sm, cudaStream_t st) {
    using TL = DecTileV<T, G>;
    cudaError_t e = dec_attr<T, G, true>();
    if (e != cudaSuccess) return e;
    const int cps = ctas_per_sm > 0 && ctas_per_sm < kDecCtasPerSm ? ctas_per_sm : kDecCtasPerSm;
    const size_t cap = (size_t)sm_count() * cps;
    const int grid = (int)(total < cap ? (total ? total : 1) : cap);
    DecArgs a = {};
    a.native_medians = native; a.err = lerr;
    a.fields = F; a.tile_field = tf; a.nf = nf; a.bs = bs; a.total_tiles = total;
    TraceScope tr("blocked_decode_fields", st);
    k_blocked_decode<T, G, true><<<grid, kDecThreadsP, TL::kDynSmem, st>>>(a);
    return cudaGetLastError();
}

// Lanes per block as in the encoder: 16 (float) / 8 (double) values per lane.
static int dec_lanes(int dtype, int bs) {
    const int per = dtype == 0 ? 16 : 8;
    const int need = (bs + per - 1) / per;
    return need <= 1 ? 1 : need <= 2 ? 2 : need <= 4 ? 4 : need <= 8 ? 8 : need <= 16 ? 16 : 32;
}

int blocked_dec_tile_blocks(int dtype, int bs) { return kDecWarps * (32 / dec_lanes(dtype, bs)); }

// Per-field outcome of a batched decode; *err gets the first failing status.
__global__ void k_blocked_decode_finish(const DecField* F, int nf, int esize, StreamResult* res, const int* lerr,
                                        int* err) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nf) return;
    const DecField& D = F[f];
    int st = *D.err;
    if (!st) st = *lerr;
    StreamResult r;
    r.offset = 0;
    r.size = D.n * (unsigned long long)esize;
    r.nb_const = D.hdr->ok ? D.hdr->nc : 0;
    r.eb = 0.f;
    r.status = st;
    *(D.res ? D.res : res + f) = r;
    if (st) atomicCAS(err, 0, st);
}

cudaError_t launch_blocked_decode_fields(int layout, int dtype, int bs, int nf, const DecField* d_fields,
                                         const uint32_t* d_tile_field, unsigned long long idx_total,
                                         unsigned long long dec_total,
                                         unsigned long long* counters, StreamResult* res, int* err,
                                         cudaStream_t s, const LaunchShape& shape) {
    if (layout != kRandomAccess && layout != kRandomAccessNative) return cudaErrorInvalidValue;
    if (bs < 1 || bs > 256 || nf < 1) return cudaErrorInvalidValue;
    int* lerr = (int*)(counters + 3);
    {
        TraceScope tr("blocked_parse_fields", s);
        k_blocked_parse_fields<<<(nf + 127) / 128, 128, 0, s>>>(d_fields, nf, (unsigned long long)bs);
    }
    {
        const unsigned long long cap = (unsigned long long)sm_count() * 4;
        const int ig = (int)(idx_total < cap ? (idx_total ? idx_total : 1) : cap);
        TraceScope tr("blocked_index_fields", s);
        k_blocked_index_fields<<<ig, kIdxThreads, 0, s>>>(d_fields, nf, idx_total, &counters[0]);
    }
    const int native = layout == kRandomAccessNative;
    cudaError_t e;
    if (dtype == 0) {
        switch (dec_lanes(dtype, bs)) {
            case 1: e = run_decode_fields<float, 1>(d_fields, d_tile_field, nf, bs, dec_total, native, lerr, shape.dec_ctas_per_sm, s); break;
            case 2: e = run_decode_fields<float, 2>(d_fields, d_tile_field, nf, bs, dec_total, native, lerr, shape.dec_ctas_per_sm, s); break;
            case 4: e = run_decode_fields<float, 4>(d_fields, d_tile_field, nf, bs, dec_total, native, lerr, shape.dec_ctas_per_sm, s); break;
            case 8: e = run_decode_fields<float, 8>(d_fields, d_tile_field, nf, bs, dec_total, native, lerr, shape.dec_ctas_per_sm, s); break;
            default: e = run_decode_fields<float, 16>(d_fields, d_tile_field, nf, bs, dec_total, native, lerr, shape.dec_ctas_per_sm, s); break;
        }
    } else {
        switch (dec_lanes(dtype, bs)) {
            case 1: e = run_decode_fields<double, 1>(d_fields, d_tile_field, nf, bs, dec_total, native, lerr, shape.dec_ctas_per_sm, s); break;
            case 2: e = run_decode_fields<double, 2>(d_fields, d_tile_field, nf, bs, dec_total, native, lerr, shape.dec_ctas_per_sm, s); break;
            case 4: e = run_decode_fields<double, 4>(d_fields, d_tile_field, nf, bs, dec_total, native, lerr, shape.dec_ctas_per_sm, s); break;
            case 8: e = run_decode_fields<double, 8>(d_fields, d_tile_field, nf, bs, dec_total, native, lerr, shape.dec_ctas_per_sm, s); break;
            case 16: e = run_decode_fields<double, 16>(d_fields, d_tile_field, nf, bs, dec_total, native, lerr, shape.dec_ctas_per_sm, s); break;
            default: e = run_decode_fields<double, 32>(d_fields, d_tile_field, nf, bs, dec_total, native, lerr, shape.dec_ctas_per_sm, s); break;
        }
    }
    if (e != cudaSuccess) return e;
    k_blocked_decode_finish<<<(nf + 127) / 128, 128, 0, s>>>(d_fields, nf, dtype == 0 ? 4 : 8, res, lerr, err);
    return cudaGetLastError();
}

cudaError_t launch_blocked_decode(int layout, int dtype, const uint8_t* d_stream, size_t len, size_t n, int bs,
                                  void* d_out, const Workspace& ws, cudaStream_t s) {
    if (layout != kBlocked && layout != kRandomAccess && layout != kRandomAccessNative) return cudaErrorInvalidValue;
    if (bs < 1 || bs > 256 || n == 0) return cudaErrorInvalidValue;
    const bool m2 = layout == kBlocked;
    cudaError_t e;
    const size_t nb = (n + bs - 1) / bs;
    if (nb <= kIdxSmallBlocks) {
        TraceScope tr("blocked_index", s);
        k_blocked_index_small<<<1, kIdxSmallThreads, 0, s>>>(d_stream, len, n, (unsigned long long)bs, m2 ? 1 : 0,
                                                             ws.bhdr, ws.err, ws.p_off, ws.rank_w);
    } else {
        {
            // the index kernel's tile counter and both look-backs' status words
            const size_t ta = (nb + kIdxPerTile - 1) / kIdxPerTile, tb = ((nb + 31) / 32 + kIdxPerTile - 1) / kIdxPerTile;
            ClearList c{};
            c.p[0] = ws.counters;
            c.bytes[0] = sizeof(unsigned long long);
            c.p[1] = ws.st_word;
            c.bytes[1] = sizeof(unsigned long long) * ta;
            c.p[2] = ws.st2_word;
            c.bytes[2] = sizeof(unsigned long long) * tb;
            c.n = 3;
            TraceScope tr("blocked_parse", s);
            k_blocked_begin<<<(unsigned)((2 * ta + 255) / 256), 256, 0, s>>>(c, d_stream, len, n, (unsigned long long)bs,
                                                                            m2 ? 1 : 0, ws.bhdr, ws.err);
        }
        const size_t tiles = (m2 ? 0 : (nb + kIdxPerTile - 1) / kIdxPerTile) + ((nb + 31) / 32 + kIdxPerTile - 1) / kIdxPerTile;
        const size_t cap = (size_t)sm_count() * 4;
        TraceScope tr("blocked_index", s);
        if ((e = launch_after(k_blocked_index, (unsigned)(tiles < cap ? tiles : cap), kIdxThreads, 0, s, d_stream, ws.bhdr,
                              ws.p_off, ws.rank_w, ws.st_word, ws.st2_word, &ws.counters[0], ws.err,
                              (unsigned long long)len, m2 ? 0 : 1)) != cudaSuccess)
            return e;
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (m2 && (e = launch_m2_offsets(dtype, d_stream, len, n, bs, ws.m2, ws.m2_bytes, ws, s)) != cudaSuccess)
        return e;
    // bs comes from the stream header (read by the caller); the device header
    // is validated again by every kernel and a mismatch is reported, not used.
    const int native = layout == kRandomAccessNative;
    const int G = dec_lanes(dtype, bs);
    if (dtype == 0) {
        switch (G) {
            case 1: e = run_decode<float, 1>(d_stream, len, nb, ws, d_out, native, s); break;
            case 2: e = run_decode<float, 2>(d_stream, len, nb, ws, d_out, native, s); break;
            case 4: e = run_decode<float, 4>(d_stream, len, nb, ws, d_out, native, s); break;
            case 8: e = run_decode<float, 8>(d_stream, len, nb, ws, d_out, native, s); break;
            default: e = run_decode<float, 16>(d_stream, len, nb, ws, d_out, native, s); break;
        }
    } else {
        switch (G) {
            case 1: e = run_decode<double, 1>(d_stream, len, nb, ws, d_out, native, s); break;
            case 2: e = run_decode<double, 2>(d_stream, len, nb, ws, d_out, native, s); break;
            case 4: e = run_decode<double, 4>(d_stream, len, nb, ws, d_out, native, s); break;
            case 8: e = run_decode<double, 8>(d_stream, len, nb, ws, d_out, native, s); break;
            case 16: e = run_decode<double, 16>(d_stream, len, nb, ws, d_out, native, s); break;
            default: e = run_decode<double, 32>(d_stream, len, nb, ws, d_out, native, s); break;
        }
    }
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

}  // namespace szxg
