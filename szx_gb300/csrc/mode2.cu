// Block boundaries of the fastMode-2 stream, found in parallel.
//
// Layout (szx/src/szx_float.cc:1059-1139, the FXR output as well):
//   [1,1,1,0] | blockSize u8 | nbConstant u64 BE | state bits | medians f32 BE
//   | payloads of the non-constant blocks, back to back, with no size index.
// A payload's length follows from its own first bytes: reqLength (-> R
// stored bytes per value), then ceil(n/4) lead bytes, then sum over values of
// max(R - lead, 0) mid bytes.  The reference decoder walks the chain serially
// (szx/src/szxd_float.cc:247-311).
//
// Here the payload region is cut into segments of 32 maximal blocks.  Pass 1
// (one CTA per segment, its bytes staged in shared memory) starts a walk at
// every position of the segment's first `maxsize` bytes (a block that began
// in the previous segment ends there); walks from positions that are not
// block starts read a reqLength outside the valid range within a step or two
// and stop, and the few that land on a true boundary follow the true chain
// from then on, so the walks that reach the end of a segment all leave it at
// the same offset: the next segment's entry.  Each walk also records how many
// blocks it passed, so the true chain's count per segment is read off at the
// entry, ranks are an exclusive scan of those counts, and pass 2 replays the
// true chain in every segment in parallel, writing each block's payload
// offset by rank.  The replay checks itself (segment exits must meet the next
// entries, the last block must end the stream); if anything disagrees, a
// one-thread serial walk rebuilds the offsets.  The offsets then feed the same
// tile decoder as the random-access layout.
//
// What bounds it: a chain of ~50 blocks per segment, each step one block size
// from its lead bytes.  Walking global memory a byte and a table look-up at a
// time took 434 us (pass 1) and 187 us (pass 2) for 2^26 float32 values; with
// the segment in shared memory and the lead sums taken 16 codes at a time by
// population counts, a step of a surviving walk is one word per lane and a
// redux across the warp.
#include <atomic>

#include "common.cuh"
#include "kernels.h"

namespace szxg {

namespace {

constexpr int kM2Threads = 256;
constexpr unsigned short kM2Dead = 0xFFFF;

struct M2Geom {
    unsigned long long len;    // stream bytes; the payload region is [q_off, len)
    unsigned long long seg;    // segment bytes
    unsigned long long nseg;   // segments covering the largest possible payload region
    int maxsize;               // largest payload of a full block
    int list;                  // words of a segment's block list
};

// Payload bytes of a block of blen values from the sums over its lead codes
// (l: of the codes, n3: how many are 3).  A value stores max(R - lead, 0)
// bytes; R is at least 2 (reqLength >= 9), so only lead 3 at R = 2 clips.
__device__ __forceinline__ uint32_t m2_size_of(int R, int blen, int l, int n3) {
    return (uint32_t)(5 + ((blen + 3) >> 2) + R * blen - l + (R == 2 ? n3 : 0));
}
// reqLength: float 9..32 (szx/src/szx_float.cc:1708-1717), double 12..64 (szx/src/szx_double.cc:2020-2031)
__device__ __forceinline__ bool m2_valid_req(int rl, int W) {
    return W == 4 ? (rl >= 9 && rl <= 32) : (rl >= 12 && rl <= 64);
}
__device__ __forceinline__ int m2_bytes_of(int rl) { return (rl >> 3) + ((rl & 7) != 0); }

// Sums over the lead codes of a 32-bit word: the codes (low half), the codes equal to 3 (high half).
__device__ __forceinline__ uint32_t m2_word_sums(uint32_t w) {
    return (uint32_t)(__popc(w & 0x55555555u) + 2 * __popc(w & 0xAAAAAAAAu)) |
           ((uint32_t)__popc(w & (w >> 1) & 0x55555555u) << 16);
}

// Mask of the lead codes that word i of a block's lead bytes holds (blen values).
__device__ __forceinline__ uint32_t m2_lead_mask(int i, int blen) {
    const int rest = blen - 16 * i;
    if (rest >= 16) return 0xFFFFFFFFu;
    if (rest <= 0) return 0u;
    const int fb = rest >> 2, rem = rest & 3;   // whole bytes, then rem codes (the top ones of their byte)
    return ((1u << (8 * fb)) - 1u) | (((0xFFu << (8 - 2 * rem)) & 0xFFu) << (8 * fb));
}

// A segment's bytes in shared memory.  Offsets are relative to the segment's
// start; byte x lies at buf + ph + x.
struct M2Seg {
    const uint8_t* buf;
    uint32_t ph, len;   // len: bytes of the payload region from the segment's start on (saturated)
    __device__ __forceinline__ uint32_t word(uint32_t x) const {   // the 4 bytes from x on
        const uint32_t o = ph + x;
        const uint32_t* w = (const uint32_t*)buf + (o >> 2);
        return __funnelshift_r(w[0], w[1], o << 3);
    }
};

// Stage the bytes [x0, x0 + n) of the payload region at P (inside the stream
// [s, send)) with the whole CTA; buf has room for n + 48 bytes.
__device__ __forceinline__ uint32_t m2_stage(uint8_t* buf, const uint8_t* src, uint32_t n, const uint8_t* s,
                                             const uint8_t* send) {
    const uint32_t ph = (uint32_t)((uintptr_t)src & 15);
    const uint8_t* g = src - ph;
    const uint32_t nch = (ph + n + 15) >> 4;
    for (uint32_t c = threadIdx.x; c < nch; c += blockDim.x) {
        const uint8_t* a = g + 16 * (size_t)c;
        if (a >= s && a + 16 <= send) cp_async16(buf + 16 * c, a);
        else
            for (int j = 0; j < 16; j++) buf[16 * c + j] = (a + j >= s && a + j < send) ? a[j] : 0;
    }
    cp_async_wait_all();
    __syncthreads();
    return ph;
}

// Step from the block at p (blen values): its payload bytes, kM2No when the
// bytes there cannot start a block, kM2Past when they could but the block
// would run past the region's end.
constexpr uint32_t kM2No = 0xFFFFFFFFu, kM2Past = 0xFFFFFFFEu;
__device__ __forceinline__ uint32_t m2_finish(uint32_t len, uint32_t p, int rl, int blen, uint32_t sums) {
    // (a size is at least the header and the lead bytes, whatever the sums: it
    // also runs past the end when the lead bytes themselves do)
    const uint32_t size = m2_size_of(m2_bytes_of(rl), blen, (int)(sums & 0xFFFFu), (int)(sums >> 16));
    return p + size > len ? kM2Past : size;
}
// by one thread
__device__ __forceinline__ uint32_t m2_step(const M2Seg& S, uint32_t p, int blen, int W) {
    if (p + 5 > S.len) return kM2No;
    const int rl = S.buf[S.ph + p];
    if (!m2_valid_req(rl, W)) return kM2No;
    uint32_t sums = 0;
    for (int i = 0; 16 * i < blen; i++) sums += m2_word_sums(S.word(p + 5 + 4 * i) & m2_lead_mask(i, blen));
    return m2_finish(S.len, p, rl, blen, sums);
}
// by a whole warp, one lead word per lane (blocks of at most 256 values: 16
// words); mask: m2_lead_mask(lane, blen)
__device__ __forceinline__ uint32_t m2_step_warp(const M2Seg& S, uint32_t p, int blen, uint32_t mask, int W) {
    if (p + 5 > S.len) return kM2No;
    const int rl = S.buf[S.ph + p];
    const uint32_t w = S.word(p + 5 + (mask ? 4 * lane_id() : 0u)) & mask;
    if (!m2_valid_req(rl, W)) return kM2No;
    return m2_finish(S.len, p, rl, blen, __reduce_add_sync(0xffffffffu, m2_word_sums(w)));
}
// by a whole warp from global memory (x: the segment's start, len: bytes of
// the payload region from there on)
__device__ __forceinline__ uint32_t m2_step_global(const uint8_t* x, uint32_t len, uint32_t p, int blen, uint32_t mask,
                                                   int W) {
    if (p + 5 > len) return kM2No;
    const int rl = x[p];
    uint32_t w = 0;
#pragma unroll
    for (int b = 0; b < 4; b++) {
        const uint32_t o = p + 5 + 4 * lane_id() + b;
        if ((mask >> (8 * b) & 0xFFu) && o < len) w |= (uint32_t)x[o] << (8 * b);
    }
    if (!m2_valid_req(rl, W)) return kM2No;
    return m2_finish(len, p, rl, blen, __reduce_add_sync(0xffffffffu, m2_word_sums(w & mask)));
}

// The serial walk's step, from global memory: lut[R][byte] holds a lead byte's stored bytes.
__device__ __forceinline__ long long m2_size(const uint8_t* P, unsigned long long L, unsigned long long p, int blen,
                                             int W, const uint8_t* lut /*[9][256]*/) {
    if (p + 5 > L) return -1;
    const int rl = P[p];
    if (!m2_valid_req(rl, W)) return -1;
    const int R = m2_bytes_of(rl);
    const int Lb = (blen + 3) >> 2;
    if (p + 5 + (unsigned long long)Lb > L) return -2;
    const uint8_t* q = P + p + 5;
    const uint8_t* t = lut + 256 * R;
    long long mid = 0;
    const int full = blen >> 2;
    for (int b = 0; b < full; b++) mid += t[q[b]];
    if (blen & 3) {
        const int code = q[full];
        for (int i = 0; i < (blen & 3); i++) {
            const int ld = (code >> (6 - 2 * i)) & 3;
            mid += R > ld ? R - ld : 0;
        }
    }
    const long long size = 5 + Lb + mid;
    return p + (unsigned long long)size > L ? -2 : size;
}

// lut[R][byte] = sum over the byte's 4 lead codes of max(R - lead, 0)
__device__ __forceinline__ void m2_lut_init(uint8_t* lut) {
    for (int i = threadIdx.x; i < 9 * 256; i += blockDim.x) {
        const int R = i >> 8, b = i & 255;
        int c = 0;
        for (int k = 0; k < 4; k++) {
            const int ld = (b >> (6 - 2 * k)) & 3;
            c += R > ld ? R - ld : 0;
        }
        lut[i] = (uint8_t)c;
    }
}

}  // namespace

// Pass 1: one CTA per segment.  The candidate starts (offsets c < maxsize) with
// a valid reqLength are gathered, and each is walked by one thread until it
// has passed kM2Reach maximal blocks; that ends nearly all walks that are not
// on a block start, and the rest of them mostly stand at the same place: the
// true chain's first block there.  From every distinct place one warp walks
// on to the segment's end; the blocks it passes from the first place are
// listed for the second pass.  (Periodic data can leave many places: those
// beyond kM2Places are walked to the end by their threads.)
constexpr int kM2Places = 32;
// Maximal blocks a walk has to pass before it counts.  With two, false walks
// still registered places in many segments (the second pass then missed the
// listed one and walked: 41 us); four let none through on the fields measured.
constexpr uint32_t kM2Reach = 4;
__global__ void __launch_bounds__(kM2Threads) k_m2_walk(const uint8_t* s, const BlockedHdr* hp, M2Geom g, int W,
                                                        unsigned short* cnt_tab, unsigned long long* exit_lo,
                                                        unsigned long long* exit_hi, uint32_t* lists) {
    pdl_start();
    extern __shared__ __align__(16) uint8_t m2_dyn[];
    __shared__ uint32_t s_lo, s_hi;
    __shared__ int s_n, s_places;
    __shared__ uint32_t s_place[kM2Places], s_more[kM2Places], s_exit[kM2Places];   // more: blocks to the end, kM2No: none
    const BlockedHdr h = *hp;
    const unsigned long long j = blockIdx.x;
    const int nthr = (int)blockDim.x;   // kM2Threads, or fewer where the candidates are few (m2_walk_threads)
    if (!h.ok) return;
    const uint8_t* P = s + h.q_off;
    const unsigned long long L = g.len - h.q_off, x0 = j * g.seg;
    const uint32_t seg = (uint32_t)g.seg, ms = (uint32_t)g.maxsize;
    unsigned short* tab = cnt_tab + j * (unsigned long long)ms;
    uint32_t* s_cand = (uint32_t*)(m2_dyn + ((seg + ms + 64 + 15) & ~15u));   // [ms]: c, later blocks << 16 | c
    uint32_t* s_pos = s_cand + ms;                                            // [ms]: where the walk stands
    if (threadIdx.x == 0) {
        s_lo = 0xFFFFFFFFu;
        s_hi = 0;
        s_n = 0;
        s_places = 0;
    }
    if (threadIdx.x < kM2Places) s_place[threadIdx.x] = 0u;
    const unsigned long long left = x0 < L ? L - x0 : 0;
    M2Seg S;
    S.buf = m2_dyn;
    S.len = left < 0x40000000ull ? (uint32_t)left : 0x40000000u;
    S.ph = m2_stage(m2_dyn, P + x0, S.len < seg + ms ? S.len : seg + ms, s, s + g.len);
    const int bs = (int)h.bs;
    const uint32_t end = seg < S.len ? seg : S.len;   // a walk is through when it stands here or beyond
    // candidates: a valid reqLength (the last four bytes of the region start no block)
    for (uint32_t c0 = 0; c0 < ms; c0 += (uint32_t)nthr) {
        const uint32_t c = c0 + threadIdx.x;
        const bool in = c < ms, ok = in && c + 5 <= S.len && m2_valid_req(S.buf[S.ph + c], W);
        if (in && !ok) tab[c] = kM2Dead;
        const unsigned m = __ballot_sync(0xffffffffu, ok);
        int at = 0;
        if (lane_id() == 0 && m) at = atomicAdd(&s_n, __popc(m));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (ok) s_cand[at + __popc(m & ((1u << lane_id()) - 1))] = c;
    }
    __syncthreads();
    const int n = s_n;
    // p after the blocks up to `to`, counted in k; false: the walk ended before
    auto walk = [&](uint32_t& p, uint32_t& k, uint32_t to) {
        while (p < to) {
            const uint32_t sz = m2_step(S, p, bs, W);
            if (sz == kM2No) return false;
            k++;
            p = sz == kM2Past ? S.len : p + sz;   // the stream's last block when it is short
        }
        return true;
    };
    const uint32_t t0 = kM2Reach * ms < end ? kM2Reach * ms : end;
    for (int i = threadIdx.x; i < n; i += nthr) {
        const uint32_t c = s_cand[i];
        uint32_t p = c, k = 0, pos = kM2No;
        if (walk(p, k, t0)) {
            pos = p;
            if (p < end) {
                // register the place once (a slot is claimed by its first walk)
                int slot = 0;
                for (; slot < kM2Places; slot++) {
                    const uint32_t o = atomicCAS(&s_place[slot], 0u, p);   // (places are beyond t0 > 0)
                    if (o == 0u) atomicAdd(&s_places, 1);
                    if (o == 0u || o == p) break;
                }
                if (slot == kM2Places) {
                    if (!walk(p, k, end)) pos = kM2No;
                    else pos = p;
                }
            }
        }
        s_cand[i] = k << 16 | c;
        s_pos[i] = pos;
    }
    __syncthreads();
    const int np = s_places;
    const uint32_t mask = m2_lead_mask((int)lane_id(), bs);
    uint32_t* list = lists + j * (unsigned long long)g.list;   // [0] the place, [1] blocks listed, then their offsets
    if (threadIdx.x == 0) list[0] = np ? s_place[0] : kM2No;
    for (int i = threadIdx.x >> 5; i < np; i += nthr / 32) {
        uint32_t p = s_place[i], k = 0;
        while (p < end) {
            if (i == 0 && lane_id() == 0) list[2 + k] = p;   // (a whole block's payload is at least its header and lead bytes)
            const uint32_t sz = m2_step_warp(S, p, bs, mask, W);
            k++;
            if (sz == kM2No) { p = kM2No; break; }
            p = sz == kM2Past ? S.len : p + sz;
        }
        if (lane_id() == 0) {
            s_more[i] = p == kM2No ? kM2No : k;
            s_exit[i] = p;
            if (i == 0) list[1] = k;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += nthr) {
        const uint32_t c = s_cand[i] & 0xFFFFu;
        uint32_t k = s_cand[i] >> 16, p = s_pos[i];
        bool alive = p != kM2No;
        if (alive && p < end) {
            int slot = 0;
            while (s_place[slot] != p) slot++;
            alive = s_more[slot] != kM2No;
            k += s_more[slot];
            p = s_exit[slot];
        }
        tab[c] = alive ? (unsigned short)k : kM2Dead;
        if (alive) {
            atomicMin(&s_lo, p);
            atomicMax(&s_hi, p);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        exit_lo[j] = s_lo == 0xFFFFFFFFu ? ~0ull : x0 + s_lo;
        exit_hi[j] = x0 + s_hi;
    }
}

// Entries and counts of the true chain per segment (one thread per segment).
__global__ void k_m2_link(const BlockedHdr* hp, M2Geom g, const unsigned short* cnt_tab,
                          const unsigned long long* exit_lo, const unsigned long long* exit_hi,
                          unsigned long long* entry, unsigned int* cnt, unsigned int* ambiguous, unsigned int* redo) {
    pdl_start();
    const unsigned long long j = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (j == 0) *redo = 0;
    const BlockedHdr h = *hp;
    if (!h.ok || j >= g.nseg) return;
    const unsigned long long L = g.len - h.q_off;
    unsigned long long e = 0;
    bool ok = true;
    unsigned int amb = 0;
    if (j > 0) {
        e = exit_lo[j - 1];
        ok = e != ~0ull;
        amb = ok && exit_hi[j - 1] != e;
    }
    ambiguous[j] = amb;
    unsigned int k = 0;
    if (ok && e >= j * g.seg && e - j * g.seg < (unsigned long long)g.maxsize && e < L) {
        const unsigned short v = cnt_tab[j * (unsigned long long)g.maxsize + (e - j * g.seg)];
        k = v == kM2Dead ? 0 : v;
    } else {
        e = ~0ull;
    }
    entry[j] = e;
    cnt[j] = k;
}

// Exclusive scan of the per-segment counts (one CTA, eight segments a thread
// and round).
constexpr int kM2ScanPer = 8;
__global__ void __launch_bounds__(1024) k_m2_scan(unsigned long long nseg, const unsigned int* cnt,
                                                  unsigned long long* base) {
    pdl_start();
    __shared__ unsigned long long s_w[32];
    unsigned long long carry = 0;
    for (unsigned long long j0 = 0; j0 < nseg; j0 += 1024 * kM2ScanPer) {
        const unsigned long long j = j0 + (unsigned long long)threadIdx.x * kM2ScanPer;
        unsigned int v[kM2ScanPer];
        unsigned long long mine = 0;
#pragma unroll
        for (int i = 0; i < kM2ScanPer; i++) {
            v[i] = j + i < nseg ? cnt[j + i] : 0;
            mine += v[i];
        }
        const unsigned long long incl = warp_inclusive_sum(mine);
        if ((threadIdx.x & 31) == 31) s_w[threadIdx.x >> 5] = incl;
        __syncthreads();
        if (threadIdx.x < 32) s_w[threadIdx.x] = warp_inclusive_sum(s_w[threadIdx.x]);
        __syncthreads();
        unsigned long long run = (threadIdx.x >= 32 ? s_w[(threadIdx.x >> 5) - 1] : 0) + carry + incl - mine;
#pragma unroll
        for (int i = 0; i < kM2ScanPer; i++) {
            if (j + i < nseg) base[j + i] = run;
            run += v[i];
        }
        carry += s_w[31];
        __syncthreads();
    }
}

// Pass 2: the true chain of each segment (one warp each), its payload offsets
// by rank (P[nnc] = end of the last block).  The few blocks from the entry to
// the place where pass 1's walks met are stepped through, the rest comes from
// pass 1's list; a chain that misses the place, and the stream's end, where
// the last block may be short, are walked.  Disagreements raise `redo`.
__global__ void __launch_bounds__(kM2Threads) k_m2_replay(const uint8_t* s, const BlockedHdr* hp, M2Geom g, int W,
                                                          const unsigned long long* entry,
                                                          const unsigned long long* base,
                                                          const unsigned int* ambiguous, const uint32_t* lists,
                                                          unsigned long long* Poff, unsigned int* redo) {
    pdl_start();
    const BlockedHdr h = *hp;
    if (!h.ok) return;
    const unsigned long long j = ((unsigned long long)blockIdx.x * kM2Threads + threadIdx.x) >> 5;
    if (j >= g.nseg) return;
    unsigned long long rank = base[j];
    if (rank >= h.nnc) return;   // the chain ended in an earlier segment
    const bool lead = lane_id() == 0;
    if (ambiguous[j] || entry[j] == ~0ull) {
        if (lead) atomicExch(redo, 1u);
        return;
    }
    const unsigned long long L = g.len - h.q_off, x0 = j * g.seg;   // (x0 < L: the segment has an entry)
    const uint8_t* x = s + h.q_off + x0;
    const unsigned long long left = L - x0;
    const uint32_t len = left < 0x40000000ull ? (uint32_t)left : 0x40000000u, seg = (uint32_t)g.seg;
    // the last block is short when n is not a multiple of bs and block nb-1 is non-constant
    const unsigned long long last_len = h.n - (h.nb - 1) * h.bs;
    const bool last_coded = (s[h.s_off + ((h.nb - 1) >> 3)] >> (7 - ((h.nb - 1) & 7))) & 1;
    const uint32_t* list = lists + j * (unsigned long long)g.list;
    const uint32_t place = list[0], more = place == kM2No ? 0u : list[1];   // (a place has at least one block)
    uint32_t p = (uint32_t)(entry[j] - x0);
    int blen = (int)h.bs;
    uint32_t mask = m2_lead_mask((int)lane_id(), blen);
    while (p < seg && rank < h.nnc) {
        if (p == place) {
            // the listed blocks of the chain, but the last of them, which is stepped over below
            const uint32_t m = more < h.nnc - rank ? more : (uint32_t)(h.nnc - rank);
            for (uint32_t i = lane_id(); i + 1 < m; i += 32) Poff[rank + i] = x0 + list[2 + i];
            rank += m - 1;
            p = list[2 + m - 1];
        }
        if (rank == h.nnc - 1 && last_coded) {
            blen = (int)last_len;
            mask = m2_lead_mask((int)lane_id(), blen);
        }
        const uint32_t sz = m2_step_global(x, len, p, blen, mask, W);
        if (sz >= kM2Past) {
            if (lead) atomicExch(redo, 1u);
            return;
        }
        if (lead) Poff[rank] = x0 + p;
        p += sz;
        rank++;
    }
    if (!lead) return;
    if (rank == h.nnc) {
        Poff[h.nnc] = x0 + p;
        if (x0 + p != L) atomicExch(redo, 1u);
    } else if (j + 1 < g.nseg && entry[j + 1] != x0 + p) {
        atomicExch(redo, 1u);
    }
}

// Fallback when the parallel passes disagree: the serial walk (one thread).
__global__ void k_m2_serial(const uint8_t* s, const BlockedHdr* hp, M2Geom g, int W, const unsigned int* redo,
                            unsigned long long* Poff, int* err) {
    pdl_start();
    __shared__ uint8_t lut[9 * 256];
    m2_lut_init(lut);
    __syncthreads();
    if (threadIdx.x != 0 || !*redo) return;
    const BlockedHdr h = *hp;
    if (!h.ok) return;
    const uint8_t* P = s + h.q_off;
    const unsigned long long L = g.len - h.q_off;
    const unsigned long long last_len = h.n - (h.nb - 1) * h.bs;
    const bool last_coded = (s[h.s_off + ((h.nb - 1) >> 3)] >> (7 - ((h.nb - 1) & 7))) & 1;
    unsigned long long p = 0;
    for (unsigned long long r = 0; r < h.nnc; r++) {
        const int blen = (r == h.nnc - 1 && last_coded) ? (int)last_len : (int)h.bs;
        const long long sz = m2_size(P, L, p, blen, W, lut);
        if (sz < 0) { atomicExch(err, kErrStream); return; }
        Poff[r] = p;
        p += (unsigned long long)sz;
    }
    Poff[h.nnc] = p;
    if (p != L) atomicExch(err, kErrStream);
}

namespace {

int m2_maxsize(int dtype, int bs) { return 5 + (bs + 3) / 4 + (dtype == 0 ? 4 : 8) * bs; }
// Threads of a segment's walk.  A segment of small blocks has few candidates and
// few bytes, and one warp a segment keeps up to 32 of them on an SM instead of
// eight: decode of 2^22 floats in blocks of 2 / 3 / 8 / 32 values 515 / 374 / 170
// / 88 us with 256 threads, 312 / 226 / 114 / 75 with 32; blocks of 64 (277
// bytes) 52 and 60, 24 doubles (203 bytes) 118 and 140.
unsigned m2_walk_threads(int maxsize) { return maxsize <= 160 ? 32u : (unsigned)kM2Threads; }
// Words of a segment's block list: place, count, and as many blocks of the smallest payload as a segment holds.
int m2_list_words(int dtype, int bs) { return 3 + 32 * m2_maxsize(dtype, bs) / (5 + (bs + 3) / 4); }

}  // namespace

// Segments for a stream of len bytes of n values in blocks of bs: the payload
// region is at most len - 13 - state bytes.
size_t m2_segments(int dtype, size_t n, int bs, size_t len) {
    const size_t nb = (n + bs - 1) / bs, sb = (nb + 7) / 8;
    const size_t pmax = len > 13 + sb ? len - 13 - sb : 0;
    return pmax / (32 * (size_t)m2_maxsize(dtype, bs)) + 1;
}

size_t m2_ws_bytes(int dtype, size_t n, int bs, size_t len) {
    if (bs < 1 || n == 0) return 256;
    const size_t ms = (size_t)m2_maxsize(dtype, bs);
    const size_t nseg = m2_segments(dtype, n, bs, len);
    auto a = [](size_t x) { return (x + 255) & ~(size_t)255; };
    return a(2 * nseg * ms) + 3 * a(8 * nseg) + 2 * a(4 * nseg) + a(4 * nseg * (size_t)m2_list_words(dtype, bs)) + 256;
}

// Payload offsets by non-constant rank for a fastMode-2 stream of len bytes
// (ws.p_off; P[nnc] = payload end), after the header is parsed into ws.bhdr.
cudaError_t launch_m2_offsets(int dtype, const uint8_t* d_stream, size_t len, size_t n, int bs, void* m2ws,
                              size_t m2wsb, const Workspace& ws, cudaStream_t s) {
    const int ms = m2_maxsize(dtype, bs);
    M2Geom g;
    g.len = len;
    g.maxsize = ms;
    g.seg = 32ull * ms;
    g.list = m2_list_words(dtype, bs);
    g.nseg = m2_segments(dtype, n, bs, len);
    if (m2wsb < m2_ws_bytes(dtype, n, bs, len)) return cudaErrorInvalidValue;
    auto a = [](size_t x) { return (x + 255) & ~(size_t)255; };
    uint8_t* b = (uint8_t*)m2ws;
    unsigned short* cnt_tab = (unsigned short*)b; b += a(2 * g.nseg * ms);
    unsigned long long* exit_lo = (unsigned long long*)b; b += a(8 * g.nseg);
    unsigned long long* exit_hi = (unsigned long long*)b; b += a(8 * g.nseg);
    unsigned long long* entry = (unsigned long long*)b; b += a(8 * g.nseg);
    unsigned int* cnt = (unsigned int*)b; b += a(4 * g.nseg);
    unsigned int* amb = (unsigned int*)b; b += a(4 * g.nseg);
    unsigned long long* base = exit_hi;   // reused after the link pass
    uint32_t* lists = (uint32_t*)b; b += a(4 * g.nseg * (size_t)g.list);
    unsigned int* redo = (unsigned int*)b;
    const int W = dtype == 0 ? 4 : 8;
    // shared memory of the walk: a segment, the block that may start at its
    // end, read slack, and the candidates
    const size_t dyn = (((size_t)g.seg + (size_t)ms + 64 + 15) & ~(size_t)15) + 8 * (size_t)ms;
    static std::atomic<bool> attr_set[64];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!attr_set[dev].load()) {
        constexpr int kMost = 33 * (5 + 64 + 8 * 256) + 80 + 8 * (5 + 64 + 8 * 256);   // blocks of 256 doubles
        if ((e = cudaFuncSetAttribute(k_m2_walk, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost)) != cudaSuccess ||
            (e = cudaFuncSetAttribute(k_m2_walk, cudaFuncAttributePreferredSharedMemoryCarveout,
                                      cudaSharedmemCarveoutMaxShared)) != cudaSuccess)
            return e;
        attr_set[dev].store(true);
    }
    {
        TraceScope tr("m2_walk", s);
        e = launch_after(k_m2_walk, (unsigned)g.nseg, m2_walk_threads(ms), dyn, s, d_stream, ws.bhdr, g, W, cnt_tab, exit_lo, exit_hi,
                         lists);
    }
    if (e == cudaSuccess)
        e = launch_after(k_m2_link, (unsigned)((g.nseg + 255) / 256), 256, 0, s, ws.bhdr, g, cnt_tab, exit_lo, exit_hi, entry,
                         cnt, amb, redo);
    if (e == cudaSuccess) e = launch_after(k_m2_scan, 1, 1024, 0, s, g.nseg, cnt, base);
    if (e == cudaSuccess) {
        TraceScope tr("m2_replay", s);
        e = launch_after(k_m2_replay, (unsigned)((g.nseg + kM2Threads / 32 - 1) / (kM2Threads / 32)), kM2Threads, 0, s,
                         d_stream, ws.bhdr, g, W, entry, base, amb, lists, ws.p_off, redo);
    }
    if (e == cudaSuccess) e = launch_after(k_m2_serial, 1, 256, 0, s, d_stream, ws.bhdr, g, W, redo, ws.p_off, ws.err);
    return e;
}

}  // namespace szxg
