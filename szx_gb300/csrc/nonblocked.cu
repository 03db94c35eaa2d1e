// Non-blocked layout of the SZx stream (fastMode 1):
//   SZx_fast_compress_args_unpredictable_float, szx/src/szx_float.cc:1492-1699
//   (double: szx/src/szx_double.cc:1593-2011), decoded by
//   szx/src/szxd_float.cc:478-662 (double: szx/src/szxd_double.cc:683-1114).
//
//   [1,1,1,0] | reqLength u8 | median f32 BE | leadBytes u64 BE | 2-bit lead
//   codes for all N values | mid bytes
//
// One global median/radius (from the value-range pass) and ONE XOR chain over
// the whole array: each value's lead code depends only on its predecessor, so
// codes are data-parallel; mid-byte positions need a device-wide prefix sum
// (encoder: decoupled look-back over 4096-value tiles, placed from the CTA's
// own previous tile and a window of counts).  Decoding must also find,
// for every value, the last earlier value that stored each of the top three
// byte lanes -- possibly many tiles back.  The lead codes alone give every
// tile's byte count and its last writers, so the decoder needs no look-back:
// per-tile counts (k_nb_count), one scan of group totals (k_nb_scan), the
// carried bytes per tile (k_nb_carry), then the tiles decode independently.
//
// The stream is placed 15 bytes into the output buffer so the lead-code array
// (stream offset 17) starts 16-byte aligned.
#include "common.cuh"
#include "kernels.h"
#include "segment.cuh"

namespace szxg {

constexpr int kNbThreads = 256;
constexpr int kNbPer = 16;                        // values per thread
constexpr int kNbTile = kNbThreads * kNbPer;      // 4096 values per tile
constexpr unsigned long long kNbShift = 15;

// CTA-wide exclusive sum (256 threads), returns the total through *tot.  One
// barrier: the caller places another barrier between this call and the next
// one that writes `sm`.
__device__ __forceinline__ uint32_t cta_excl_sum32(uint32_t v, uint32_t* tot, uint32_t* sm /*[8]*/) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t incl = warp_inclusive_sum(v);
    if (lane == 31) sm[warp] = incl;
    __syncthreads();
    uint32_t pre = 0, t = 0;
#pragma unroll
    for (int w = 0; w < kNbThreads / 32; w++) {
        uint32_t x = sm[w];
        pre += w < warp ? x : 0;
        t += x;
    }
    *tot = t;
    return pre + incl - v;
}

template <typename T>
__device__ __forceinline__ void load16(const T* p, unsigned long long first, unsigned long long n, T (&v)[kNbPer]) {
    const bool full = first + kNbPer <= n;
    if (full && ((uintptr_t)(p + first) % 16) == 0) {
        const uint4* q = (const uint4*)(p + first);
#pragma unroll
        for (int i = 0; i < kNbPer * (int)sizeof(T) / 16; i++) {
            uint4 w = q[i];
            if constexpr (sizeof(T) == 4) {
                v[4 * i] = __uint_as_float(w.x); v[4 * i + 1] = __uint_as_float(w.y);
                v[4 * i + 2] = __uint_as_float(w.z); v[4 * i + 3] = __uint_as_float(w.w);
            } else {
                v[2 * i] = __longlong_as_double((long long)(((unsigned long long)w.y << 32) | w.x));
                v[2 * i + 1] = __longlong_as_double((long long)(((unsigned long long)w.w << 32) | w.z));
            }
        }
    } else {
#pragma unroll
        for (int e = 0; e < kNbPer; e++) v[e] = first + e < n ? p[first + e] : (T)0;
    }
}

template <typename T>
__device__ __forceinline__ void store16(T* p, unsigned long long first, unsigned long long n, const T (&v)[kNbPer]) {
    const bool full = first + kNbPer <= n;
    if (full && ((uintptr_t)(p + first) % 32) == 0) {   // whole 32-byte sectors
        constexpr int V8 = 32 / (int)sizeof(T);
#pragma unroll
        for (int i = 0; i < kNbPer / V8; i++) st_v8(p + first + V8 * i, v + V8 * i);
    } else if (full && ((uintptr_t)(p + first) % 16) == 0) {
        uint4* q = (uint4*)(p + first);
#pragma unroll
        for (int i = 0; i < kNbPer * (int)sizeof(T) / 16; i++) {
            uint4 w;
            if constexpr (sizeof(T) == 4) {
                w = make_uint4(__float_as_uint(v[4 * i]), __float_as_uint(v[4 * i + 1]), __float_as_uint(v[4 * i + 2]),
                               __float_as_uint(v[4 * i + 3]));
            } else {
                unsigned long long a = (unsigned long long)__double_as_longlong(v[2 * i]);
                unsigned long long b = (unsigned long long)__double_as_longlong(v[2 * i + 1]);
                w = make_uint4((uint32_t)a, (uint32_t)(a >> 32), (uint32_t)b, (uint32_t)(b >> 32));
            }
            q[i] = w;
        }
    } else {
#pragma unroll
        for (int e = 0; e < kNbPer; e++)
            if (first + e < n) p[first + e] = v[e];
    }
}

// ------------------------------------------------------------------ encode

struct NbEncArgs {
    const void* x;
    unsigned long long n, ntiles, cap;
    const CodecParams* params;
    uint8_t* out;
    unsigned long long* st;   // look-back status words [ntiles + 4], zeroed
    uint16_t* agg;            // counts + 1 [ntiles + 16], zeroed
    unsigned long long* tile_ctr;
    int* err;
    StreamResult* res;
};

// One pass over the input in tiles of kNbTile values taken from an atomic
// counter, one tile ahead.  Iteration j, between two CTA barriers: the values
// of T_j (loaded during the previous iteration), differences and lead codes
// (one XOR chain over the whole array: a thread's first value's predecessor is
// the previous thread's last, or the value before the tile), a CTA scan of the
// stored-byte counts | barrier | the tile's byte count published, the lead
// codes to their fixed place, the mid bytes into one of three shared staging
// buffers, the next tile's loads; then warp 0 places T_{j-1} (PlaceWin; its
// window was copied in during the emission) while the other warps copy T_{j-2}
// to its place | barrier | the bytes of the words that threads share.
// Bound by the instruction rate and the two barriers, 242 us at 2^27 float32
// values (512 MiB read, 129 us at the copy rate).  With the placement of
// T_{j-2} between the barriers, followed by a status word beside a prefix array
// and a fence, the seven other warps waited for warp 0 half the time: 395 us.
template <typename T>
constexpr int nb_stage_bytes() { return ((kNbTile * (int)sizeof(T) + 48) + 15) / 16 * 16; }

template <typename T>
__global__ void __launch_bounds__(kNbThreads, sizeof(T) == 4 ? 4 : 2) k_nb_encode(NbEncArgs a) {
    pdl_start();
    using EL = Elem<T>;
    using U = typename EL::U;
    constexpr int W = EL::W;
    extern __shared__ __align__(16) uint8_t nb_dyn[];   // three staging buffers of nb_stage_bytes<T>()
    auto stage = [&](int k) { return nb_dyn + ((unsigned)k % 3u) * nb_stage_bytes<T>(); };
    __shared__ PlaceWin s_win;
    __shared__ uint32_t s_sum[8];
    __shared__ int s_tile[2];
    __shared__ uint32_t s_total[3];
    __shared__ unsigned long long s_base[2];
    __shared__ int s_skip[2];
    const T* x = (const T*)a.x;
    const CodecParams P = *a.params;
    // szx/src/szx_float.cc:1514-1535 / szx_double.cc:1615-1636
    bool zm;
    const int reqLength = req_length<T>(P.eb, P.radius, &zm);
    int R, s;
    split_reqlen(reqLength, &R, &s);
    T med;
    if constexpr (sizeof(T) == 4) med = zm ? 0.0f : P.median;
    else med = xf2d(P.median);
    const uint32_t med_stored = zm ? 0u : __float_as_uint(P.median);
    const unsigned long long L = (a.n + 3) / 4;
    uint8_t* lead = a.out + kNbShift + 17;
    uint8_t* mid = lead + L;
    const unsigned long long mid_cap = a.cap - (kNbShift + 17 + L);
    const int lane = threadIdx.x & 31;
    const int down = 8 * W - reqLength;
    const uint32_t guard = 0x80u << s, s4 = (uint32_t)(31 + s) * 0x01010101u, R4 = (uint32_t)R * 0x01010101u;
    const int nt = (int)a.ntiles;
    // warp 0: tile t (count agg, iteration k) placed, the header and result with the last tile
    auto place = [&](int t, int k) {
        const uint32_t agg = s_total[(unsigned)k % 3u];
        unsigned long long base;
        if (!s_win.offset(a.agg, t, &base)) base = prefix_resolve(a.st, t, agg, a.err);   // (publishes)
        else if (t > 0 && lane == 0) st_volatile64(&a.st[t], kS64Inc | ((base + agg) & kS64Val));
        if (lane == 0) {
            s_win.anchor(0, t, base + agg);
            s_base[k & 1] = base;
            const bool ok = base + agg <= mid_cap;
            s_skip[k & 1] = !ok;
            if (!ok) atomicExch(a.err, kErrCapacity);
            if (t == nt - 1) {
                uint8_t* h = a.out + kNbShift;
                h[0] = 1; h[1] = 1; h[2] = 1; h[3] = 0;
                h[4] = (uint8_t)reqLength;
                h[5] = (uint8_t)(med_stored >> 24); h[6] = (uint8_t)(med_stored >> 16);
                h[7] = (uint8_t)(med_stored >> 8); h[8] = (uint8_t)med_stored;
                for (int q = 0; q < 8; q++) h[9 + q] = (uint8_t)(L >> (56 - 8 * q));
                StreamResult r;
                r.offset = kNbShift;
                r.size = 17 + L + base + agg;
                r.nb_const = 0;
                r.eb = P.eb;
                r.status = 0;
                *a.res = r;
            }
        }
        __syncwarp();
    };
    if (threadIdx.x == 0) {
        s_win.init();
        const unsigned long long g = atomicAdd(a.tile_ctr, 1ull);
        s_tile[0] = g < a.ntiles ? (int)g : -1;
    }
    __syncthreads();
    int tile = s_tile[0], t1 = -1, t2 = -1;   // T_j, T_{j-1}, T_{j-2}; -1: none
    const bool taker = threadIdx.x == kNbThreads - 32;   // the last warp claims the tiles
    T v[kNbPer];
    T before = (T)0;     // lane 0: the value before its first one
    auto fetch = [&](int t) {
        const unsigned long long first = (unsigned long long)t * kNbTile + threadIdx.x * kNbPer;
        load16<T>(x, first, a.n, v);
        before = (lane == 0 && first > 0 && first - 1 < a.n) ? x[first - 1] : (T)0;
    };
    if (tile >= 0) fetch(tile);
    // (after the last tile two more iterations place and copy out what is staged)
    for (int it = 0; tile >= 0 || t1 >= 0 || t2 >= 0; it++) {
        const bool live = tile >= 0;
        // the next tile's claim; the reply is used before the scan's barrier
        unsigned long long gc = ~0ull;
        claim_tile(gc, a.tile_ctr, taker && live);
        const unsigned long long first = (unsigned long long)tile * kNbTile + threadIdx.x * kNbPer;
        U d[kNbPer];
        T dprev = (T)0;
        // (no double subtractions in the two iterations after the last tile: they held the FP64 pipe as long as a tile's
        // do, 15.9 instead of 13.8 us for 2^18 doubles, a tile a CTA; for floats the branch spills)
        if (sizeof(T) == 4 || live) {
            dprev = EL::sub(before, med);
            sub_run(v, med, d);
        } else {
#pragma unroll
            for (int e = 0; e < kNbPer; e++) d[e] = 0;
        }
        U d_l0 = first > 0 ? EL::bits(dprev) : (U)0;   // lane 0: the value before its first one
        bool bad = lane == 0 && first > 0 && inf_or_nan(dprev);
        if constexpr (sizeof(T) == 4) {
            float hn = __uint_as_float(d[0]);
#pragma unroll
            for (int e = 1; e + 1 < kNbPer; e += 2) hn = fmax3_nan(hn, __uint_as_float(d[e]), __uint_as_float(d[e + 1]));
            bad = bad || isnan(fmax_nan(hn, __uint_as_float(d[kNbPer - 1])));
        } else {
#pragma unroll
            for (int e = 0; e < kNbPer; e++) bad = bad || inf_or_nan(EL::of(d[e]));
        }
        if (__any_sync(0xffffffffu, bad)) {
#pragma unroll
            for (int e = 0; e < kNbPer; e++) {
                // (doubles: the subtraction is done, an infinity among the differences stands)
                if constexpr (sizeof(T) == 4) d[e] = EL::bits(xsub(v[e], med));
                else if ((d[e] & 0x7FFFFFFFFFFFFFFFull) > 0x7FF0000000000000ull) d[e] = EL::bits(nan_rule(v[e], med));
            }
            if (lane == 0 && first > 0) d_l0 = EL::bits(xsub(before, med));
        }
        // lead codes from the top 32 bits, as in the blocked encoder
        auto top = [](U u) { return (uint32_t)(u >> (8 * W - 32)); };
        uint32_t prev = __shfl_up_sync(0xffffffffu, top(d[kNbPer - 1]), 1);
        if (lane == 0) prev = top(d_l0);
        const int rem = first >= a.n ? 0 : (a.n - first < kNbPer ? (int)(a.n - first) : kNbPer);   // values of this thread
        uint32_t codes = 0, mine = 0, cnt8[kNbPer / 4];
#pragma unroll
        for (int k = 0; k < kNbPer / 4; k++) {
            uint32_t lb[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t h = top(d[4 * k + i]);
                asm("bfind.u32 %0, %1;" : "=r"(lb[i]) : "r"((h ^ prev) | guard));
                prev = h;
            }
            const uint32_t p = (lb[3] * 256u + lb[2]) * 65536u + (lb[1] * 256u + lb[0]);
            const uint32_t keep = low_bytes_mask(rem - 4 * k);
            const uint32_t ldb = ((s4 - p) >> 3) & 0x03030303u & keep;
            // max(R - lead, 0) per value, R >= 2
            const uint32_t c4 = (R4 + (R == 2 ? (ldb >> 1) & ldb & 0x01010101u : 0u) - ldb) & keep;
            cnt8[k] = c4 << 3;
            mine = __dp4a(c4, 0x01010101u, mine);
            codes |= ((ldb * 0x40100401u) >> 24) << (8 * k);   // 4 leads -> one byte, MSB first
        }
        if (taker) s_tile[(it + 1) & 1] = gc < a.ntiles ? (int)gc : -1;
        uint32_t total;
        const uint32_t ex = cta_excl_sum32(mine, &total, s_sum);   // one barrier
        if (threadIdx.x < 32) {
            if (live) {
                if (lane == 0) {
                    s_total[(unsigned)it % 3u] = total;
                    st_relaxed16(a.agg + tile, total + 1);
                }
                prefix_publish(a.st, tile, total);
            }
            // T_{j-1}'s window, in flight during the emission
            if (t1 >= 0) s_win.issue(a.agg, 0, t1);
        }
        RunOut o;
        if (live) {
        // lead codes: 4 bytes per thread, at their fixed place
        const unsigned long long lb = first >> 2;
        if (lb + 4 <= L && ((uintptr_t)(lead + lb) & 3) == 0) *(uint32_t*)(lead + lb) = codes;
        else
            for (int j = 0; j < 4; j++)
                if (lb + j < L) lead[lb + j] = (uint8_t)(codes >> (8 * j));
        // mid bytes: each value's low (R - lead) bytes of its required bits, at
        // tile-local offsets: whole words now, the bytes of the words that
        // threads share after the barrier below
        o.start(stage(it), ex);
#pragma unroll
        for (int k = 0; k < kNbPer / 4; k++) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t n8 = byte_of(cnt8[k], i);
                const U ev = d[4 * k + i] >> down;
                if constexpr (sizeof(T) == 4) {
                    o.append((uint32_t)ev, n8);
                } else {
                    const uint32_t nl = n8 < 32u ? n8 : 32u;
                    o.append((uint32_t)ev, nl);
                    o.append((uint32_t)(ev >> 32), n8 - nl);
                }
            }
        }
        }
        // the next tile's values are in flight during the placement and the copy-out
        const int next = s_tile[(it + 1) & 1];
        if (next >= 0) fetch(next);
        if (threadIdx.x < 32) {
            if (t1 >= 0) place(t1, it - 1);
        } else if (t2 >= 0 && !s_skip[it & 1]) {
            cta_copy_realign(stage(it + 1), s_total[(unsigned)(it + 1) % 3u], mid + s_base[it & 1], threadIdx.x - 32,
                             kNbThreads - 32);
        }
        __syncthreads();   // T_j's whole words staged; T_{j-1}'s offset known, T_{j-2}'s buffer free
        if (live) o.finish(stage(it), ex);   // (read by T_j's copy-out, two iterations on)
        t2 = t1;
        t1 = tile;
        tile = next;
    }
}

size_t nonblocked_bound(int dtype, size_t n) {
    size_t es = dtype == 0 ? 4 : 8;
    return kNbShift + 17 + (n + 3) / 4 + es * n + 64;
}

ClearList nonblocked_enc_clear(const Workspace& ws, size_t n) {
    const size_t ntiles = (n + kNbTile - 1) / kNbTile;
    ClearList c{};
    c.p[0] = ws.st32;   // the 16-bit counts
    c.bytes[0] = (2 * (ntiles + 16) + 3) & ~size_t(3);
    c.p[1] = ws.totals;
    c.bytes[1] = kWsHeaderClear;
    c.p[2] = ws.st_word;
    c.bytes[2] = sizeof(unsigned long long) * (ntiles + 4);
    c.n = 3;
    return c;
}

cudaError_t launch_nonblocked_encode(int dtype, const void* x, size_t n, uint8_t* d_out, size_t cap,
                                     const Workspace& ws, cudaStream_t s, bool cleared, StreamResult* res_out) {
    if (n == 0 || cap < nonblocked_bound(dtype, n) - 64) return cudaErrorInvalidValue;
    const size_t ntiles = (n + kNbTile - 1) / kNbTile;
    if (ntiles > 0x7FFFFFFF) return cudaErrorInvalidValue;
    cudaError_t e;
    if (!cleared && (e = launch_ws_clear(nonblocked_enc_clear(ws, n), s)) != cudaSuccess) return e;
    NbEncArgs a;
    a.x = x; a.n = n; a.ntiles = ntiles; a.cap = cap; a.params = ws.params; a.out = d_out;
    a.st = ws.st_word;
    a.agg = (uint16_t*)ws.st32;
    a.tile_ctr = &ws.counters[0];
    a.err = ws.err;
    a.res = res_out ? res_out : ws.result;
    static int per_sm[2][64] = {{0}};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    int& occ = per_sm[dtype == 0 ? 0 : 1][dev];
    const size_t dyn = 3 * (size_t)(dtype == 0 ? nb_stage_bytes<float>() : nb_stage_bytes<double>());
    if (!occ) {
        if (dtype == 0) {
            e = cudaFuncSetAttribute(k_nb_encode<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
            if (e == cudaSuccess)
                e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_nb_encode<float>, kNbThreads, dyn);
        } else {
            e = cudaFuncSetAttribute(k_nb_encode<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
            if (e == cudaSuccess)
                e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_nb_encode<double>, kNbThreads, dyn);
        }
        if (e != cudaSuccess) return e;
        if (occ < 1) occ = 1;
    }
    size_t g = (size_t)sm_count() * occ;
    int grid = (int)(ntiles < g ? ntiles : g);
    {
        TraceScope tr("nonblocked_encode", s);
        return launch_after(dtype == 0 ? k_nb_encode<float> : k_nb_encode<double>, grid, kNbThreads, dyn, s, a);
    }
}

// ------------------------------------------------------------------ decode

// W: bytes of a value.  A reqLength above its bits is refused here, for every kernel of the decode (they test ok alone,
// and find the counting kernel's tables complete).
__device__ NonBlockedHdr parse_nb(const uint8_t* s, unsigned long long len, unsigned long long n, int W) {
    NonBlockedHdr r = {};
    r.n = n;
    r.ok = 0;
    if (len >= 17 && s[3] == 0) {
        unsigned long long L = 0;
        for (int k = 0; k < 8; k++) L = (L << 8) | s[9 + k];
        r.L = L;
        r.reqLength = s[4];
        r.median = __uint_as_float(((uint32_t)s[5] << 24) | ((uint32_t)s[6] << 16) | ((uint32_t)s[7] << 8) | s[8]);
        r.mid_off = 17 + L;
        r.ok = L == (n + 3) / 4 && r.mid_off <= len && r.reqLength >= 1 && r.reqLength <= 8 * W;
        r.mid_len = r.ok ? len - r.mid_off : 0;
    }
    return r;
}

__device__ __forceinline__ uint32_t lead_word(const uint8_t* lead, unsigned long long lb, unsigned long long L) {
    uint32_t w = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) w |= (lb + j < L ? (uint32_t)lead[lb + j] : 0u) << (8 * j);
    return w;
}

// Lead word of values [first, first + 16), as the two aligned words that hold
// it: joined by lead_join() where it is used, so that a word loaded ahead is
// not waited for.  (The codes start 17 bytes into the stream: at no word
// boundary where the stream itself starts at one.)
__device__ __forceinline__ void lead_load(const uint8_t* lead, unsigned long long first, unsigned long long L,
                                          uint32_t& a, uint32_t& b) {
    const unsigned long long lb = first >> 2;
    const uint32_t sh = (uint32_t)((uintptr_t)(lead + lb) & 3);
    if (lb + 8 <= L) {
        const uint32_t* q = (const uint32_t*)(lead + lb - sh);
        a = __ldg(q);
        b = __ldg(q + 1);
    } else {
        const uint32_t w = lead_word(lead, lb, L);
        a = w << (8 * sh);
        b = __funnelshift_l(w, 0u, 8 * sh);
    }
}
__device__ __forceinline__ uint32_t lead_join(const uint8_t* lead, uint32_t a, uint32_t b) {
    return __funnelshift_r(a, b, 8 * (uint32_t)((uintptr_t)lead & 3));   // (words lie whole words into the codes)
}

// Per tile (one warp): its mid-byte count (tcnt[t]) and, for each of the top
// three byte lanes, where in the tile's mid bytes the last value storing that
// lane put it (aux[3t+2], 3x21 bits, position+1, 0 = none).  A lane takes 8
// consecutive 16-code words, so the tile takes one warp scan.  A word costs its
// three masks, their population counts (a value stores max(R - lead, 0) bytes,
// the number of k < R with lead <= k) and the last word of each mask that is
// not empty.  (One word per lane and eight scans a tile: 59 us at 2^27 values;
// codes that start at no word boundary, the usual case, were read a byte at a
// time: 46 us, 33 as words.)
// The CTA's eight tiles form a group: aux[3t] / aux[3t+1] get the tile's
// exclusive prefix within its group (bytes; latest writer tiles, 3x21 bits,
// tile+1), gsum[g] / gwr[g] the group's totals.  Independent per group: no
// look-back.
template <typename T>
__global__ void __launch_bounds__(kNbThreads) k_nb_count(const uint8_t* __restrict__ s, unsigned long long len,
                                                         unsigned long long n, NonBlockedHdr* hp, int* err,
                                                         uint32_t* __restrict__ tcnt,
                                                         unsigned long long* __restrict__ aux,
                                                         unsigned long long* __restrict__ gsum,
                                                         unsigned long long* __restrict__ gwr) {
    constexpr int W = Elem<T>::W;
    constexpr int kTpg = kNbThreads / 32;   // tiles per group
    constexpr int kWords = kNbTile / (32 * kNbPer);   // words per lane
    __shared__ uint32_t s_cnt[kTpg];
    __shared__ unsigned long long s_own[kTpg];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const NonBlockedHdr h = parse_nb(s, len, n, W);   // (every thread: the same loads, from cache)
    if (blockIdx.x == 0 && threadIdx.x == 0) {     // for the kernels that follow
        *hp = h;
        *err = h.ok ? kErrNone : kErrStream;
    }
    if (!h.ok) return;
    const int R = run_bytes(h.reqLength);
    const unsigned long long ntiles = (h.n + kNbTile - 1) / kNbTile;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long tile = (long long)blockIdx.x * kTpg + warp;
    const uint8_t* lead = s + 17;
    uint32_t run = 0;
    int gpos[3] = {-1, -1, -1};
    if (tile < (long long)ntiles) {
        const unsigned long long first = (unsigned long long)tile * kNbTile + (unsigned long long)(kWords * kNbPer) * lane;
        uint32_t cw[kWords];
        const uint8_t* lp = lead + (first >> 2);
        if (first + kWords * kNbPer <= h.n && ((uintptr_t)lp & 15) == 0) {
            const uint4 a = __ldg((const uint4*)lp), b = __ldg((const uint4*)lp + 1);
            cw[0] = a.x; cw[1] = a.y; cw[2] = a.z; cw[3] = a.w;
            cw[4] = b.x; cw[5] = b.y; cw[6] = b.z; cw[7] = b.w;
        } else if (first + kWords * kNbPer > h.n || !load_words<kWords>(lp, s + len, cw)) {
#pragma unroll
            for (int j = 0; j < kWords; j++) cw[j] = lead_word(lead, (first >> 2) + 4 * j, h.L);
        }
        if (one_byte_req(h.reqLength)) {
#pragma unroll
            for (int j = 0; j < kWords; j++) cw[j] = one_byte_codes(cw[j]);
        }
        uint32_t mine = 0, lastw[3] = {0, 0, 0}, lastc[3] = {0, 0, 0};   // per byte lane: its last word and the bytes before it
        int lastn[3] = {0, 0, 0};
#pragma unroll
        for (int j = 0; j < kWords; j++) {
            const unsigned long long f = first + kNbPer * j;
            const int nv = f >= h.n ? 0 : (h.n - f < kNbPer ? (int)(h.n - f) : kNbPer);
            const RunLeads<kNbPer> l(cw[j], nv, R);
#pragma unroll
            for (int k = 0; k < 3; k++)
                if (k == 0 ? l.v0 : k == 1 ? l.v1 : l.v2) {
                    lastw[k] = cw[j];
                    lastc[k] = mine;
                    lastn[k] = nv;
                }
            mine += l.bytes();
        }
        const uint32_t incl = warp_inclusive_sum(mine);
        run = __shfl_sync(0xffffffffu, incl, 31);
#pragma unroll
        for (int k = 0; k < 3; k++)
            if (lastn[k]) {
                const RunLeads<kNbPer> l(lastw[k], lastn[k], R);
                gpos[k] = (int)(incl - mine + lastc[k] + l.last_at(k));
            }
    }
    unsigned long long own = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int p = __reduce_max_sync(0xffffffffu, gpos[k]);
        own |= (unsigned long long)(p + 1) << (21 * k);
    }
    if (lane == 0) {
        s_cnt[warp] = run;
        s_own[warp] = own;
    }
    __syncthreads();
    if (threadIdx.x < 32) {   // the group's prefixes: lane w holds tile w (0 past the last)
        const long long t = (long long)blockIdx.x * kTpg + lane;
        const bool in = lane < kTpg && t < (long long)ntiles;
        const unsigned long long o = in ? s_own[lane] : 0ull;
        const uint32_t c = in ? s_cnt[lane] : 0u;
        unsigned long long pa = c, pb = 0;
#pragma unroll
        for (int k = 0; k < 3; k++)
            if ((o >> (21 * k)) & 0x1FFFFF) pb |= (unsigned long long)(t + 1) << (21 * k);
#pragma unroll
        for (int d = 1; d < kTpg; d <<= 1) {
            const unsigned long long oa = __shfl_up_sync(0xffffffffu, pa, d), ob = __shfl_up_sync(0xffffffffu, pb, d);
            if (lane >= d) {
                pa += oa;
                pb = Max3x21Op::op(ob, pb);
            }
        }
        if (lane == kTpg - 1) {
            gsum[blockIdx.x] = pa;
            gwr[blockIdx.x] = pb;
        }
        const unsigned long long eb = __shfl_up_sync(0xffffffffu, pb, 1);
        if (in) {
            aux[3 * t] = pa - c;
            aux[3 * t + 1] = lane ? eb : 0ull;
            aux[3 * t + 2] = o;
            tcnt[t] = c;
        }
    }
}

// One CTA: exclusive scan, in place, of the group totals (gsum: bytes, a
// sum; gwr: latest writer tiles, combined by max), over chunks of
// kScanThreads * kScanPer groups carried from chunk to chunk.  A stream
// whose mid bytes run past its end is reported.
constexpr int kScanThreads = 512, kScanPer = 8;

__global__ void __launch_bounds__(kScanThreads) k_nb_scan(const NonBlockedHdr* hp, unsigned long long* gsum,
                                                          unsigned long long* gwr, int* err) {
    pdl_start();
    __shared__ unsigned long long s_a[kScanThreads / 32], s_b[kScanThreads / 32];
    const NonBlockedHdr h = *hp;
    if (!h.ok) return;
    const unsigned long long ntiles = (h.n + kNbTile - 1) / kNbTile;
    const unsigned long long ng = (ntiles + kNbThreads / 32 - 1) / (kNbThreads / 32);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned long long ca = 0, cb = 0;   // totals of the earlier chunks
    for (unsigned long long c0 = 0; c0 < ng; c0 += (unsigned long long)kScanThreads * kScanPer) {
        const unsigned long long g0 = c0 + (unsigned long long)threadIdx.x * kScanPer;
        unsigned long long va[kScanPer], vb[kScanPer];
        unsigned long long la = 0, lb = 0;
#pragma unroll
        for (int i = 0; i < kScanPer; i++) {
            va[i] = g0 + i < ng ? gsum[g0 + i] : 0ull;
            vb[i] = g0 + i < ng ? gwr[g0 + i] : 0ull;
            la += va[i];
            lb = Max3x21Op::op(lb, vb[i]);
        }
        unsigned long long ia = la, ib = lb;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned long long oa = __shfl_up_sync(0xffffffffu, ia, d);
            const unsigned long long ob = __shfl_up_sync(0xffffffffu, ib, d);
            if (lane >= d) {
                ia += oa;
                ib = Max3x21Op::op(ob, ib);
            }
        }
        if (lane == 31) {
            s_a[warp] = ia;
            s_b[warp] = ib;
        }
        __syncthreads();
        unsigned long long pa = ca, pb = cb, ta = ca, tb = cb;
        for (int w = 0; w < kScanThreads / 32; w++) {
            if (w < warp) {
                pa += s_a[w];
                pb = Max3x21Op::op(pb, s_b[w]);
            }
            ta += s_a[w];
            tb = Max3x21Op::op(tb, s_b[w]);
        }
        unsigned long long ea = __shfl_up_sync(0xffffffffu, ia, 1), eb = __shfl_up_sync(0xffffffffu, ib, 1);
        if (lane == 0) {
            ea = 0;
            eb = 0;
        }
        pa += ea;
        pb = Max3x21Op::op(pb, eb);
#pragma unroll
        for (int i = 0; i < kScanPer; i++) {
            if (g0 + i < ng) {
                gsum[g0 + i] = pa;
                gwr[g0 + i] = pb;
            }
            pa += va[i];
            pb = Max3x21Op::op(pb, vb[i]);
        }
        ca = ta;
        cb = tb;
        __syncthreads();   // s_a / s_b are read before the next chunk writes them
    }
    if (threadIdx.x == 0 && ca > h.mid_len) atomicExch(err, kErrStream);
}

// One thread per tile: the bytes that the top three byte lanes carry into the
// tile (the last earlier value that stored each lane), read from the stream
// and packed into aux[3t+1] (lane W-1-k at bits 8*(2-k)).  A tile's offset is
// its group's prefix (gsum) plus its offset in the group (aux[3t]); each
// thread rewrites only its own tile's aux[3t+1] and reads only the other two
// words of other tiles.
__global__ void k_nb_carry(const uint8_t* __restrict__ s, unsigned long long len, const NonBlockedHdr* hp,
                           unsigned long long* aux, const unsigned long long* gsum,
                           const unsigned long long* gwr) {
    pdl_start();
    constexpr int kTpg = kNbThreads / 32;
    const NonBlockedHdr h = *hp;
    if (!h.ok) return;
    const unsigned long long ntiles = (h.n + kNbTile - 1) / kNbTile;
    const unsigned long long t = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntiles) return;
    const unsigned long long lw = Max3x21Op::op(gwr[t / kTpg], aux[3 * t + 1]);
    uint32_t carry = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const unsigned long long t1 = (lw >> (21 * k)) & 0x1FFFFF;
        if (t1) {
            const unsigned long long u = t1 - 1;
            const unsigned long long p1 = (aux[3 * u + 2] >> (21 * k)) & 0x1FFFFF;
            const unsigned long long pos = h.mid_off + gsum[u / kTpg] + aux[3 * u] + (p1 - 1);
            const uint32_t byte = pos < len ? s[pos] : 0u;
            carry |= byte << (8 * (2 - k));
        }
    }
    aux[3 * t + 1] = carry;
}

// Decode, tiles taken in a fixed order (blockIdx.x, + gridDim.x, ...): a
// tile's offset, carried bytes and byte count are known before it starts, so
// the next tile's lead codes and per-tile words are loaded at the start of an
// iteration and its mid bytes copied with cp.async into the second staging
// buffer while the current tile decodes.
template <typename T>
constexpr int nb_dec_stage_bytes() { return ((kNbTile * (int)sizeof(T) + 64) + 15) / 16 * 16; }
constexpr uint32_t kNbFront = 16;   // bytes before a tile's (the run decoder reads up to eight back)

template <typename T>
__global__ void __launch_bounds__(kNbThreads, sizeof(T) == 4 ? 4 : 2)
    k_nb_decode(const uint8_t* __restrict__ s, unsigned long long len, const NonBlockedHdr* hp,
                const uint32_t* tcnt, const unsigned long long* aux,
                const unsigned long long* gsum, T* out) {
    pdl_start();
    constexpr int kTpg = kNbThreads / 32;
    using EL = Elem<T>;
    using U = typename EL::U;
    extern __shared__ __align__(16) uint8_t nb_dyn[];   // two staging buffers of nb_dec_stage_bytes<T>()
    __shared__ uint32_t s_sum[8];
    __shared__ uint32_t s_wv[8], s_wm[8];   // per warp: last written top bytes, their byte mask
    __shared__ uint32_t lut_ld[512];
    const NonBlockedHdr h = *hp;
    if (!h.ok) return;
    const int R = run_bytes(h.reqLength);
    const long long ntiles = (long long)((h.n + kNbTile - 1) / kNbTile);
    long long tile = blockIdx.x;
    if (tile >= ntiles) return;
    lead_table_init(lut_ld);   // (the first tile's barriers come before its use)
    const uint8_t* lead = s + 17;
    const uint8_t* mid = s + h.mid_off;
    const uint8_t* send = s + len;
    const T med = widen_median<T>(h.median);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto stage = [&](int k) { return nb_dyn + (k & 1) * nb_dec_stage_bytes<T>(); };
    // the tile's mid bytes [base, base + tot) into staging buffer k, 16-byte
    // chunks by cp.async, a chunk at either end of the stream byte by byte
    auto copy_in = [&](int k, unsigned long long base, uint32_t tot) {
        const uint8_t* src = mid + base;
        const uint32_t sh = (uint32_t)((uintptr_t)src & 15);
        const uint8_t* gbase = src - sh;
        const uint32_t nch = (sh + tot + 15) >> 4;
        uint8_t* stg = stage(k) + kNbFront;
        for (uint32_t c = threadIdx.x; c < nch; c += kNbThreads) {
            const uint8_t* lo = gbase + (c << 4);
            if (lo >= s && lo + 16 <= send) cp_async16(stg + (c << 4), lo);
            else
                for (int j = 0; j < 16; j++) stg[(c << 4) + j] = (lo + j >= s && lo + j < send) ? lo[j] : 0;
        }
        cp_async_commit();
    };
    // a tile's words: lead codes (per thread), group prefix + offset in the
    // group, carried bytes, byte count
    auto words = [&](long long t, uint32_t& ca, uint32_t& cb, unsigned long long& ga, unsigned long long& la,
                     uint32_t& cy, uint32_t& tot) {
        lead_load(lead, (unsigned long long)t * kNbTile + threadIdx.x * kNbPer, h.L, ca, cb);
        ga = gsum[t / kTpg];
        la = aux[3 * t];
        cy = (uint32_t)aux[3 * t + 1];
        tot = tcnt[t];
    };
    const long long G = gridDim.x;
    uint32_t cd0, cy0, tot0, cd1 = 0, cy1 = 0, tot1 = 0;
    unsigned long long ga0, la0, ga1 = 0, la1 = 0;
    uint32_t ca, cb = 0;
    words(tile, ca, cb, ga0, la0, cy0, tot0);
    cd0 = lead_join(lead, ca, cb);
    if (tile + G < ntiles) {
        words(tile + G, ca, cb, ga1, la1, cy1, tot1);
        cd1 = lead_join(lead, ca, cb);
    }
    copy_in(0, ga0 + la0, tot0);
    for (int it = 0;; it++) {
        const bool more = tile + G < ntiles;
        // the words of the tile after next, in flight during this tile
        uint32_t ca2 = 0, cb2 = 0, cy2 = 0, tot2 = 0;
        unsigned long long ga2 = 0, la2 = 0;
        if (tile + 2 * G < ntiles) words(tile + 2 * G, ca2, cb2, ga2, la2, cy2, tot2);
        uint32_t codes = cd0;
        const uint32_t carry = cy0;
        // (R first: with the one test the loop spills and takes 226 us at 2^27 values, not 210)
        if (R == 2 && one_byte_req(h.reqLength)) codes = one_byte_codes(codes);
        const unsigned long long base = ga0 + la0;
        const unsigned long long first = (unsigned long long)tile * kNbTile + threadIdx.x * kNbPer;
        const int nv = first >= h.n ? 0 : (h.n - first < kNbPer ? (int)(h.n - first) : kNbPer);
        const RunLeads<kNbPer> leads(codes, nv, R);
        const uint32_t mine = leads.bytes();
        uint32_t total;
        const uint32_t ex = cta_excl_sum32(mine, &total, s_sum);   // one barrier
        if (more) copy_in(it + 1, ga1 + la1, tot1);
        else cp_async_commit();   // an empty group: the wait below still means "this tile's copy"
        cp_async_wait_group<1>();
        __syncthreads();   // this tile's bytes are staged
        const uint32_t q0 = smem_u32(stage(it)) + kNbFront + (uint32_t)((uintptr_t)(mid + base) & 15) + ex;
        // (top bytes, byte mask) pairs: a later pair's masked bytes win,
        // masks accumulate -- one three-input logic op each
        uint32_t sv, sw;
        leads.summary(q0, sv, sw);
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t ov = __shfl_up_sync(0xffffffffu, sv, d), ow = __shfl_up_sync(0xffffffffu, sw, d);
            if (lane >= d) {
                sv = (ov & ~sw) | (sv & sw);
                sw |= ow;
            }
        }
        if (lane == 31) {
            s_wv[warp] = sv;
            s_wm[warp] = sw;
        }
        __syncthreads();
        uint32_t pv = carry;   // the carried bytes: all three lanes written before the tile
        for (int w = 0; w < warp; w++) {
            const uint32_t m = s_wm[w];
            pv = (pv & ~m) | (s_wv[w] & m);
        }
        const uint32_t ev = __shfl_up_sync(0xffffffffu, sv, 1), ew = __shfl_up_sync(0xffffffffu, sw, 1);
        if (lane) pv = (pv & ~ew) | (ev & ew);
        // (values past the end of the field are decoded like the others and never stored)
        U sp[kNbPer];
        T v[kNbPer];
        const bool bad = run_decode<T, kNbPer, true>(codes, nv, R, h.reqLength, q0, pv << 8, med, lut_ld, sp, v);
        if (__any_sync(0xffffffffu, bad)) {
#pragma unroll
            for (int e = 0; e < kNbPer; e++) v[e] = xadd(EL::of(sp[e]), med);
        }
        store16<T>(out, first, h.n, v);
        if (!more) break;
        // no barrier here: this tile's buffer is next written by the copy
        // issued after the next iteration's scan barrier, s_wsum after the
        // barrier that follows that copy
        tile += G;
        cd0 = cd1; ga0 = ga1; la0 = la1; cy0 = cy1; tot0 = tot1;
        cd1 = lead_join(lead, ca2, cb2); ga1 = ga2; la1 = la2; cy1 = cy2; tot1 = tot2;
    }
    cp_async_wait_all();
}

cudaError_t launch_nonblocked_decode(int dtype, const uint8_t* d_stream, size_t len, size_t n, void* d_out,
                                     const Workspace& ws, cudaStream_t s) {
    if (n == 0) return cudaErrorInvalidValue;
    const size_t ntiles = (n + kNbTile - 1) / kNbTile;
    if (ntiles >= (1u << 21) - 1) return cudaErrorInvalidValue;
    cudaError_t e;
    uint32_t* tcnt = ws.st32;   // [ntiles] tile byte counts
    const size_t ng = (ntiles + kNbThreads / 32 - 1) / (kNbThreads / 32);
    unsigned long long* gsum = ws.st_word;                     // [ng] group byte totals, then prefixes
    unsigned long long* gwr = ws.st_word + ws.status_tiles;    // [ng] group latest writers, then prefixes
    {
        TraceScope tr("nonblocked_count", s);
        if (dtype == 0) k_nb_count<float><<<(int)ng, kNbThreads, 0, s>>>(d_stream, len, n, ws.nhdr, ws.err, tcnt, ws.tile_aux, gsum, gwr);
        else k_nb_count<double><<<(int)ng, kNbThreads, 0, s>>>(d_stream, len, n, ws.nhdr, ws.err, tcnt, ws.tile_aux, gsum, gwr);
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    {
        TraceScope tr("nonblocked_scan", s);
        if ((e = launch_after(k_nb_scan, 1, kScanThreads, 0, s, ws.nhdr, gsum, gwr, ws.err)) != cudaSuccess) return e;
    }
    {
        TraceScope tr("nonblocked_carry", s);
        if ((e = launch_after(k_nb_carry, (unsigned)((ntiles + 255) / 256), 256, 0, s, d_stream, (unsigned long long)len,
                              ws.nhdr, ws.tile_aux, gsum, gwr)) != cudaSuccess)
            return e;
    }
    static int per_sm[2][64] = {{0}};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    int& occ = per_sm[dtype == 0 ? 0 : 1][dev];
    const size_t dyn = 2 * (size_t)(dtype == 0 ? nb_dec_stage_bytes<float>() : nb_dec_stage_bytes<double>());
    if (!occ) {
        if (dtype == 0) {
            e = cudaFuncSetAttribute(k_nb_decode<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
            if (e == cudaSuccess)
                e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_nb_decode<float>, kNbThreads, dyn);
        } else {
            e = cudaFuncSetAttribute(k_nb_decode<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
            if (e == cudaSuccess)
                e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_nb_decode<double>, kNbThreads, dyn);
        }
        if (e != cudaSuccess) return e;
        if (occ < 1) occ = 1;
    }
    const size_t g = (size_t)sm_count() * occ;
    const int grid = (int)(ntiles < g ? ntiles : g);
    {
        TraceScope tr("nonblocked_decode", s);
        if (dtype == 0)
            return launch_after(k_nb_decode<float>, grid, kNbThreads, dyn, s, d_stream, (unsigned long long)len, ws.nhdr, tcnt,
                                ws.tile_aux, gsum, (float*)d_out);
        return launch_after(k_nb_decode<double>, grid, kNbThreads, dyn, s, d_stream, (unsigned long long)len, ws.nhdr, tcnt,
                            ws.tile_aux, gsum, (double*)d_out);
    }
}

}  // namespace szxg
