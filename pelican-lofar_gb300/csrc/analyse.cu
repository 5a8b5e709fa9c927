// K5: DedispersionAnalyser (lib/src/DedispersionAnalyser.cpp:30-203).
//
// For each DM row and each block of 2^P samples (a trailing partial block is
// dropped) the reference builds a dyadic boxcar tree, level n holding sums of
// 2^n samples formed as b_n[j] = b_{n-1}[2j] + b_{n-1}[2j+1] in FP32, and
// records every value at or above level n's threshold.  Events are listed
// after a dummy (0,0,1,0) by DM, block, level and position.
//
// Two launches.  The (DM, block) pairs in the reference's order are cut into
// tiles of 128.  analyse_count reads every sample once, a warp 128 adjacent
// samples at a time (16 bytes per lane), builds the tree in the lanes with the
// reference's pairing (bit-identical sums) and leaves each tile's number of
// events; the CTA that finishes last turns these into the tiles' places in the
// list.  analyse_emit does the few tiles that have events over again, a thread
// per pair, and writes them in order.
//
// Bound: HBM, one read of the window (134 MB for 2048 x 16384: 20 us at the
// measured copy rate).  Before, a thread read its own block's 256 bytes, four
// more launches scanned one count per pair, and the 6 MB of counts were
// allocated and given back on every pv_analyse call: 390 us for that call.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

#include "pv_common.cuh"

namespace {

constexpr int kMaxPow2 = 8;

struct Thresholds {
    float v[kMaxPow2 + 1];
};

template <int P>
__device__ __forceinline__ void load_block(float (&b)[1 << P], const float* __restrict__ src,
                                           bool vec4) {
    constexpr int M = 1 << P;
    if (M >= 4 && vec4) {
        const float4* s4 = reinterpret_cast<const float4*>(src);
#pragma unroll
        for (int q = 0; q < M / 4; ++q) {
            const float4 v = __ldg(s4 + q);
            b[4 * q] = v.x; b[4 * q + 1] = v.y; b[4 * q + 2] = v.z; b[4 * q + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int j = 0; j < M; ++j) b[j] = __ldg(src + j);
    }
}

// Level N of the tree: b[j] = b[2j] + b[2j+1] for j < 2^(P-N), then the
// threshold test; recursion keeps every index a compile-time constant so the
// block stays in registers.
template <int P, int N, typename F>
struct TreeLevel {
    __device__ __forceinline__ static void run(float (&b)[1 << P], const Thresholds& thr, F& emit) {
        constexpr int cur = (1 << P) >> N;
#pragma unroll
        for (int j = 0; j < cur; ++j) {
            b[j] = __fadd_rn(b[2 * j], b[2 * j + 1]);
            if (b[j] >= thr.v[N]) emit((1 << N) * j, 1 << N, b[j]);
        }
        TreeLevel<P, N + 1, F>::run(b, thr, emit);
    }
};
template <int P, typename F>
struct TreeLevel<P, P + 1, F> {
    __device__ __forceinline__ static void run(float (&)[1 << P], const Thresholds&, F&) {}
};

// Walks the tree of one block; calls emit(t_in_block, width, value) for each
// value at or above its threshold in the reference order.
template <int P, typename F>
__device__ __forceinline__ void walk_block(float (&b)[1 << P], const Thresholds& thr, F emit) {
    constexpr int M = 1 << P;
#pragma unroll
    for (int j = 0; j < M; ++j)
        if (b[j] >= thr.v[0]) emit(j, 1, b[j]);
    TreeLevel<P, 1, F>::run(b, thr, emit);
}

constexpr int kTilePairs = 128;      // (DM, block) pairs of a tile
constexpr int kCountThreads = 256;

// Device scratch of one call, laid out by tiles_in().
struct Tiles {
    long long* offset;  // [tiles] events before the tile's first
    int* count;         // [tiles]
    unsigned* done;     // CTAs of analyse_count finished; cleared by analyse_emit
};

// Runs in every CTA after it has stored its count: the last one to get here
// scans the counts of all tiles and leaves the total (with the dummy event).
__device__ __forceinline__ void finish_tiles(const Tiles& w, int ntiles, long long* total) {
    __shared__ bool last;
    __shared__ long long wsum[kCountThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        __threadfence();
        last = atomicAdd(w.done, 1u) == (unsigned)gridDim.x - 1;
        __threadfence();
    }
    __syncthreads();
    if (!last) return;
    const int per = (ntiles + kCountThreads - 1) / kCountThreads;
    const int first = min(tid * per, ntiles), end = min(first + per, ntiles);
    long long sum = 0;
    for (int i = first; i < end; ++i) sum += __ldcg(w.count + i);
    long long x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    long long at = x - sum;
    for (int k = 0; k < warp; ++k) at += wsum[k];
    for (int i = first; i < end; ++i) {
        w.offset[i] = at;
        at += __ldcg(w.count + i);
    }
    if (tid == kCountThreads - 1) *total = 1 + at;
}

// Rows of 16-byte aligned samples, blocks of 8 to 256.  Lane l holds samples
// 4l..4l+3 of a group of 128; a block of 2^P samples is 2^(P-2) lanes, and the
// levels above 2 add lane pairs (the upper lane of a pair gets the same sum,
// which is not counted).  For P == 8 a block is two groups.
template <int P>
__global__ void __launch_bounds__(kCountThreads) analyse_count_vec(const float* __restrict__ data, long long ld,
                                                                   int nblocks, long long npairs, Thresholds thr,
                                                                   Tiles w, int ntiles, long long* total) {
    constexpr int M = 1 << P, G = P == 8 ? 2 : 1;    // 128-sample groups that a warp takes together
    constexpr int LANES = P == 8 ? 32 : M / 4;       // lanes of a block within a group
    constexpr int NW = kCountThreads / 32;
    constexpr int GROUPS = kTilePairs * M / (128 * G);  // of a tile
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long g0 = (long long)blockIdx.x * kTilePairs;
    const int dm0 = (int)(g0 / nblocks), i0 = (int)(g0 - (long long)dm0 * nblocks);
    const int left = (int)min((long long)kTilePairs, npairs - g0);
    int n = 0;
    constexpr int UNROLL = GROUPS / NW >= 4 ? 4 : (GROUPS / NW >= 2 ? 2 : 1);
#pragma unroll 1
    for (int q0 = warp; q0 < GROUPS; q0 += NW * UNROLL) {
        float4 v[UNROLL][G];
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            const int q = q0 + u * NW;
            const int p = P == 8 ? q : (q * 128 + 4 * lane) / M;  // the lane's pair within the tile
            int i = i0 + p, dm = dm0;
            if (i >= nblocks) {
                const int r = i / nblocks;
                dm += r;
                i -= r * nblocks;
            }
            const float4* src = reinterpret_cast<const float4*>(data + (long long)dm * ld + (long long)i * M);
#pragma unroll
            for (int h = 0; h < G; ++h)
                v[u][h] = p < left ? __ldcs(src + h * 32 + (P == 8 ? lane : lane % LANES))
                                   : make_float4(NAN, NAN, NAN, NAN);  // never at a threshold
        }
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            float top[G];
#pragma unroll
            for (int h = 0; h < G; ++h) {
                const float4 x = v[u][h];
                n += (x.x >= thr.v[0]) + (x.y >= thr.v[0]) + (x.z >= thr.v[0]) + (x.w >= thr.v[0]);
                const float a = __fadd_rn(x.x, x.y), b = __fadd_rn(x.z, x.w);
                n += (a >= thr.v[1]) + (b >= thr.v[1]);
                float c = __fadd_rn(a, b);
                n += c >= thr.v[2];
#pragma unroll
                for (int k = 3; k <= (P == 8 ? 7 : P); ++k) {
                    const int bit = 1 << (k - 3);
                    const float o = __shfl_xor_sync(0xffffffffu, c, bit);
                    c = __fadd_rn(c, o);  // commutative: both lanes hold the lower + upper sum
                    n += (lane & (2 * bit - 1)) == 0 && c >= thr.v[k];
                }
                top[h] = c;
            }
            if (P == 8) n += lane == 0 && __fadd_rn(top[0], top[G - 1]) >= thr.v[8];
        }
    }
    n = __reduce_add_sync(0xffffffffu, n);
    __shared__ int part[NW];
    if (lane == 0) part[warp] = n;
    __syncthreads();
    if (tid == 0) {
        int t = 0;
        for (int k = 0; k < NW; ++k) t += part[k];
        w.count[blockIdx.x] = t;
    }
    finish_tiles(w, ntiles, total);
}

// Any alignment and block size: a thread per pair.
template <int P>
__global__ void __launch_bounds__(kCountThreads) analyse_count(const float* __restrict__ data, long long ld,
                                                               int nblocks, long long npairs, Thresholds thr,
                                                               Tiles w, int ntiles, long long* total) {
    const int tid = threadIdx.x;
    const long long g = (long long)blockIdx.x * kTilePairs + tid;
    int n = 0;
    if (tid < kTilePairs && g < npairs) {
        const int dm = (int)(g / nblocks), i = (int)(g % nblocks);
        float b[1 << P];
        load_block<P>(b, data + dm * ld + (long long)i * (1 << P), false);
        walk_block<P>(b, thr, [&](int, int, float) { ++n; });
    }
    __shared__ int sum;
    if (tid == 0) sum = 0;
    __syncthreads();
    n = __reduce_add_sync(0xffffffffu, n);
    if ((tid & 31) == 0 && n) atomicAdd(&sum, n);
    __syncthreads();
    if (tid == 0) w.count[blockIdx.x] = sum;
    finish_tiles(w, ntiles, total);
}

// CTA t writes tile t's events; CTA 0 the dummy event as well.  CTA 0 clears
// the counter of finished CTAs: after the count of its own call, so calls that
// overlapped (which spoils their own results) leave it at 0 all the same.
template <int P>
__global__ void __launch_bounds__(kTilePairs) analyse_emit(const float* __restrict__ data, long long ld, int nblocks,
                                                           long long npairs, Thresholds thr, bool vec4, Tiles w,
                                                           pv_event* __restrict__ ev, long long cap) {
    __shared__ int wsum[kTilePairs / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (blockIdx.x == 0 && tid == 0) {
        *w.done = 0;
        if (cap > 0) ev[0] = pv_event{0, 0, 1.0f, 0.0f};
    }
    if (w.count[blockIdx.x] == 0) return;
    const long long g = (long long)blockIdx.x * kTilePairs + tid;
    const int dm = (int)(g / nblocks), i = (int)(g % nblocks);
    const float* src = data + dm * ld + (long long)i * (1 << P);
    float b[1 << P];
    int n = 0;
    if (g < npairs) {
        load_block<P>(b, src, vec4);
        walk_block<P>(b, thr, [&](int, int, float) { ++n; });
    }
    int x = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    if (n == 0) return;
    long long o = 1 + w.offset[blockIdx.x] + x - n;
    for (int k = 0; k < warp; ++k) o += wsum[k];
    const int base = i * (1 << P);
    load_block<P>(b, src, vec4);
    walk_block<P>(b, thr, [&](int t, int width, float v) {
        if (o < cap) ev[o] = pv_event{dm, base + t, (float)width, v};
        ++o;
    });
}

__global__ void analyse_none(pv_event* ev, long long cap, long long* total) {
    if (cap > 0) ev[0] = pv_event{0, 0, 1.0f, 0.0f};
    *total = 1;
}

// Scratch bytes of the analyser for npairs (trial, block) pairs, rounded to
// 256: what is placed after it stays aligned.
constexpr long long tiles_of(long long npairs) {
    return npairs > 0 ? (npairs + kTilePairs - 1) / kTilePairs : 1;
}
constexpr size_t scratch_bytes_for(long long npairs) {
    return ((size_t)tiles_of(npairs) * (sizeof(int) + sizeof(long long)) + 16 + 255) / 256 * 256;
}
// The counter comes first, at the same place for every size.
Tiles tiles_in(void* p, long long npairs) {
    Tiles w;
    w.done = static_cast<unsigned*>(p);
    w.offset = reinterpret_cast<long long*>(static_cast<char*>(p) + 16);
    w.count = reinterpret_cast<int*>(w.offset + tiles_of(npairs));
    return w;
}

template <int P>
int run_analyse(const float* data, long long ld, int tdms, int nsamp, const Thresholds& thr, pv_event* ev,
                long long cap, long long* d_total, void* scratch, cudaStream_t s) {
    const int nblocks = nsamp >> P;
    const long long npairs = (long long)tdms * nblocks;
    if (npairs == 0) {
        analyse_none<<<1, 1, 0, s>>>(ev, cap, d_total);
        return pv::check_launch("analyse_none");
    }
    const Tiles w = tiles_in(scratch, npairs);
    const bool vec4 = (ld % 4 == 0) && ((reinterpret_cast<uintptr_t>(data) & 15) == 0);
    const int ntiles = (int)tiles_of(npairs);
    // blocks of fewer than 8 samples are too short for the lanes' tree to have a level
    if constexpr (P >= 3) {
        if (vec4)
            analyse_count_vec<P><<<ntiles, kCountThreads, 0, s>>>(data, ld, nblocks, npairs, thr, w, ntiles, d_total);
    }
    if (P < 3 || !vec4)
        analyse_count<P><<<ntiles, kCountThreads, 0, s>>>(data, ld, nblocks, npairs, thr, w, ntiles, d_total);
    PV_TRY(pv::check_launch("analyse_count"));
    analyse_emit<P><<<ntiles, kTilePairs, 0, s>>>(data, ld, nblocks, npairs, thr, vec4, w, ev, cap);
    return pv::check_launch("analyse_emit");
}

}  // namespace

namespace pv {

// Scratch bytes the analyser needs for tdms x nsamp at 2^bin_pow2 blocks.  It
// has to be cleared once; every call clears its counter at its end.
size_t analyse_scratch_bytes(int tdms, int nsamp, int bin_pow2) {
    return scratch_bytes_for((long long)tdms * (nsamp >> bin_pow2));
}

// Analyser with caller-provided scratch (analyse_scratch_bytes bytes);
// asynchronous: the event total (dummy included) lands in *d_total.
int analyse_launch(const float* data, long long ld, int tdms, int nsamp, float threshold,
                   float rms, int bin_pow2, pv_event* ev, long long cap, long long* d_total,
                   void* scratch, cudaStream_t s) {
    Thresholds thr{};
    PV_TRY(pv_analyser_thresholds(threshold, rms, bin_pow2, thr.v));
    switch (bin_pow2) {
#define PV_CASE(P) \
    case P: return run_analyse<P>(data, ld, tdms, nsamp, thr, ev, cap, d_total, scratch, s);
        PV_CASE(0) PV_CASE(1) PV_CASE(2) PV_CASE(3) PV_CASE(4) PV_CASE(5) PV_CASE(6) PV_CASE(7)
        PV_CASE(8)
#undef PV_CASE
        default:
            set_error("pv_analyse: power2ForBinning must be in 0..%d", kMaxPow2);
            return PV_ERR_ARG;
    }
}

}  // namespace pv

extern "C" int pv_analyser_thresholds(float threshold, float rms, int bin_pow2, float* h_thr) {
    if (bin_pow2 < 0 || bin_pow2 > kMaxPow2 || !h_thr) {
        pv::set_error("pv_analyser_thresholds: power2ForBinning must be in 0..%d", kMaxPow2);
        return PV_ERR_ARG;
    }
    // Level 0 is the float product; wider boxcars multiply it by ::sqrt of
    // the (float) width in double and round once (DedispersionAnalyser.cpp:121).
    const float base = threshold * rms;
    h_thr[0] = base;
    for (int n = 1; n <= bin_pow2; ++n)
        h_thr[n] = (float)((double)base * std::sqrt((double)(float)(1u << n)));
    return PV_OK;
}

extern "C" int pv_analyse(const float* d_data, long long ld, int tdms, int nsamp, float threshold,
                          float rms, int bin_pow2, pv_event* d_events, long long cap,
                          long long* h_count, void* stream) {
    if (!h_count || tdms < 0 || nsamp < 0 || ld < nsamp || (cap > 0 && !d_events) ||
        (tdms > 0 && nsamp > 0 && !d_data)) {
        pv::set_error("pv_analyse: invalid arguments");
        return PV_ERR_ARG;
    }
    if (bin_pow2 < 0 || bin_pow2 > kMaxPow2) {
        pv::set_error("pv_analyse: power2ForBinning must be in 0..%d", kMaxPow2);
        return PV_ERR_ARG;
    }
    cudaStream_t s = pv::as_stream(stream);
    pv::Scratch scratch;
    PV_TRY(pv::scratch_take(&scratch, pv::analyse_scratch_bytes(tdms, nsamp, bin_pow2), s));
    // the total goes straight to host memory
    long long* total = static_cast<long long*>(scratch.host);
    int rc = pv::analyse_launch(d_data, ld, tdms, nsamp, threshold, rms, bin_pow2, d_events, cap, total,
                                scratch.dev, s);
    if (rc == PV_OK) rc = pv::cuda_status(cudaStreamSynchronize(s), "synchronise");
    if (rc != PV_OK) {  // its kernels may not have run to their end
        pv::scratch_drop(scratch);
        return rc;
    }
    *h_count = *static_cast<volatile long long*>(total);
    pv::scratch_give(scratch);
    return PV_OK;
}

// ---------------------------------------------------------------------------
// pv_analyse_noalloc: the analyser with its scratch in a fixed device array
// ---------------------------------------------------------------------------
namespace {

constexpr size_t kNoAllocPairs = PV_ANALYSE_NOALLOC_MAX_PAIRS;
// the same formula as pv_analyse's scratch at the largest pair count: a call
// within the pair limit always fits
constexpr size_t kNoAllocScratch = scratch_bytes_for((long long)kNoAllocPairs);
static_assert(scratch_bytes_for((long long)kNoAllocPairs) >= scratch_bytes_for((long long)kNoAllocPairs - 1),
              "scratch grows with the pair count");
// Scratch (counts, offsets, counter) followed by the event total.
// Every GPU that loads the library keeps this array until the process exits.
__device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratch + 256];

constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mutex;
void* g_noalloc_addr[kMaxDevices] = {};

// Device address of g_noalloc_scratch on the current device.  The host-side
// name is only a stand-in, so the address is looked up once per device with
// that device current.
int noalloc_scratch(void** out) {
    int dev = 0;
    PV_CUDA(cudaGetDevice(&dev), "cudaGetDevice");
    if (dev < 0 || dev >= kMaxDevices) {
        pv::set_error("pv_analyse_noalloc: device %d out of range", dev);
        return PV_ERR_ARG;
    }
    std::lock_guard<std::mutex> lk(g_noalloc_mutex);
    if (!g_noalloc_addr[dev]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) {
            pv::set_error("pv_analyse_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
            return PV_ERR_CUDA;
        }
        g_noalloc_addr[dev] = p;
    }
    *out = g_noalloc_addr[dev];
    return PV_OK;
}

}  // namespace

extern "C" int pv_analyse_noalloc(const float* d_data, long long ld, int tdms, int nsamp,
                                  float threshold, float rms, int bin_pow2, pv_event* d_events,
                                  long long cap, long long* h_count, void* stream) {
    if (!h_count || tdms < 0 || nsamp < 0 || ld < nsamp || (cap > 0 && !d_events) ||
        (tdms > 0 && nsamp > 0 && !d_data)) {
        pv::set_error("pv_analyse_noalloc: invalid arguments");
        return PV_ERR_ARG;
    }
    if (bin_pow2 < 0 || bin_pow2 > kMaxPow2) {
        pv::set_error("pv_analyse_noalloc: power2ForBinning must be in 0..%d", kMaxPow2);
        return PV_ERR_ARG;
    }
    const long long pairs = (long long)tdms * (nsamp >> bin_pow2);
    if (pairs > (long long)kNoAllocPairs) {
        pv::set_error("pv_analyse_noalloc: %d trials x %d blocks of 2^%d samples = %lld pairs "
                      "exceeds the fixed scratch limit of %lld pairs; use pv_analyse",
                      tdms, nsamp >> bin_pow2, bin_pow2, pairs, (long long)kNoAllocPairs);
        return PV_ERR_ARG;
    }
    void* scratch = nullptr;
    PV_TRY(noalloc_scratch(&scratch));
    // Nothing in the scratch needs clearing: every count, offset and the total are written before they
    // are read, and each call leaves the counter at 0.
    long long* d_total = reinterpret_cast<long long*>(static_cast<char*>(scratch) + kNoAllocScratch);
    cudaStream_t s = pv::as_stream(stream);
    PV_TRY(pv::analyse_launch(d_data, ld, tdms, nsamp, threshold, rms, bin_pow2, d_events, cap,
                              d_total, scratch, s));
    PV_CUDA(cudaMemcpyAsync(h_count, d_total, sizeof(long long), cudaMemcpyDeviceToHost, s),
            "read event count");
    PV_CUDA(cudaStreamSynchronize(s), "synchronise");
    return PV_OK;
}
