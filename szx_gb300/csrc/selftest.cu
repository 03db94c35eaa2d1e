// Failure-detection self-test of the device-wide look-back scans.
//
// Every variable-length placement in this library (payload offsets of the
// encoders, the decoders' offset and rank scans) goes through a decoupled
// look-back: a tile waits for its predecessors' status words.  Tiles are
// taken in order, so in the codecs every predecessor is running and the wait
// ends; the waits are still bounded, and a tile that gives up records
// SZXG_ERR_LOOKBACK in the call's error word instead of hanging the GPU.
//
// SZxG_selftest_lookback runs the same look-back functions the codecs use over
// ntiles one-warp or one-CTA tiles (tile t contributes t + 1 bytes), with one tile
// `withheld` that never publishes, and a small poll limit.  The tile after the
// withheld one waits, gives up after `spinLimit` polls, and the call reports
// SZXG_ERR_LOOKBACK; with nothing withheld it returns every tile's exclusive
// prefix, t(t+1)/2.  Nothing faults, traps or waits without a limit.
#include <vector>

#include "../../include/szx_gb300.h"
#include "common.cuh"
#include "kernels.h"

namespace szxg {
namespace {

// scan 0: the 64-bit status words of the encoders' placement (prefix_resolve);
// scan 1: the placement window (PlaceWin) both encoders try first, anchored at
//         tile 1, and the same words behind it.
__global__ void k_selftest_lookback(int scan, unsigned long long* st64, uint16_t* counts, int ntiles, int withheld,
                                    unsigned limit, unsigned long long* prefix, int* err) {
    const long long tile = blockIdx.x;
    if (tile >= ntiles || tile == withheld) return;   // the withheld tile never publishes
    const unsigned long long agg = (unsigned long long)tile + 1;
    if (lane_id() == 0) st_relaxed16(counts + tile, (uint32_t)agg + 1);
    prefix_publish(st64, tile, agg);
    unsigned long long p = 0;
    bool placed = false;
    if (scan == 1) {
        __shared__ PlaceWin win;
        if (lane_id() == 0) {
            win.init();
            if (tile > 1 && withheld != 1) win.anchor(0, 1, 3);   // tiles 0 and 1: one byte and two
        }
        __syncwarp();
        win.issue(counts, 0, (int)tile);
        placed = win.offset(counts, (int)tile, &p);
        if (placed && tile > 0 && lane_id() == 0) st_volatile64(&st64[tile], kS64Inc | ((p + agg) & kS64Val));
    }
    if (!placed) p = prefix_resolve(st64, tile, agg, err, limit);
    if (lane_id() == 0) prefix[tile] = p;
}

// scan 2: the CTA-wide look-back of the decoders' index (prefix_resolve_cta),
//         256 threads a tile; scan 3: the same with the status words 8 bytes
//         behind a 16-byte boundary, where they are read one at a time.
constexpr int kSelfCta = 256;
__global__ void __launch_bounds__(kSelfCta) k_selftest_lookback_cta(unsigned long long* st64, int ntiles, int withheld,
                                                                    unsigned limit, unsigned long long* prefix,
                                                                    int* err) {
    __shared__ unsigned long long sm[kSelfCta / kWarp];
    const long long tile = blockIdx.x;
    if (tile >= ntiles || tile == withheld) return;
    const unsigned long long agg = (unsigned long long)tile + 1;
    if (threadIdx.x < kWarp) prefix_publish(st64, tile, agg);
    const unsigned long long p = prefix_resolve_cta<kSelfCta / kWarp>(st64, tile, agg, err, sm, limit);
    if (threadIdx.x == 0) prefix[tile] = p;
}

}  // namespace
}  // namespace szxg

using namespace szxg;

extern "C" int SZxG_selftest_lookback(int scan, int ntiles, int withheld, unsigned spinLimit,
                                      unsigned long long* prefix, void* stream) {
    if (scan < 0 || scan > 3 || ntiles < 1 || ntiles > 4096 || withheld >= ntiles || spinLimit < 1) {
        set_last_error(SZXG_ERR_ARG);
        return SZXG_ERR_ARG;
    }
    cudaStream_t s = (cudaStream_t)stream;
    const size_t n = (size_t)ntiles;
    auto a256 = [](size_t x) { return (x + 255) & ~size_t(255); };
    const size_t ocnt = a256(8 * (n + 8)), opre = ocnt + a256(2 * (n + 16)), oerr = opre + a256(8 * n), bytes = oerr + 256;
    unsigned char* b = nullptr;
    if (cudaMalloc(&b, bytes) != cudaSuccess) {
        cudaGetLastError();
        set_last_error(SZXG_ERR_CUDA);
        return SZXG_ERR_CUDA;
    }
    unsigned long long* st64 = (unsigned long long*)b;          // [n + 8]
    uint16_t* counts = (uint16_t*)(b + ocnt);                    // [n + 16]
    unsigned long long* d_prefix = (unsigned long long*)(b + opre);
    int* d_err = (int*)(b + oerr);
    int rc = SZXG_OK;
    cudaError_t e = cudaMemsetAsync(b, 0, bytes, s);
    if (e == cudaSuccess) {
        if (scan < 2)
            k_selftest_lookback<<<ntiles, kWarp, 0, s>>>(scan, st64, counts, ntiles, withheld, spinLimit, d_prefix, d_err);
        else   // (scan 3 starts a word later: the n + 8 words hold what is read past the last tile's all the same)
            k_selftest_lookback_cta<<<ntiles, kSelfCta, 0, s>>>(st64 + (scan == 3), ntiles, withheld, spinLimit, d_prefix,
                                                                d_err);
        e = cudaGetLastError();
    }
    int h_err = 0;
    std::vector<unsigned long long> h(n);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h_err, d_err, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(h.data(), d_prefix, 8 * n, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaFree(b);
    if (e != cudaSuccess) {
        cudaGetLastError();
        rc = SZXG_ERR_CUDA;
    } else {
        rc = h_err == kErrLookback ? SZXG_ERR_LOOKBACK : h_err ? SZXG_ERR_ARG : SZXG_OK;
        if (prefix)
            for (size_t i = 0; i < n; i++) prefix[i] = h[i];
    }
    set_last_error(rc);
    return rc;
}
