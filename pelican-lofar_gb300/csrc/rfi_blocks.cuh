// The clipper in blocks of spectra: a few launches instead of a walk.
//
// Included by rfi.cu inside its anonymous namespace, after RfiState,
// RfiConfig, RfiBuffers, Geo and the reductions.
//
// What makes the clipper sequential is small.  A spectrum's channel sum, its
// good-channel counts and, while the histories fill, its band statistics
// depend on the running averages only through WHICH channels are clipped, and
// the running averages need nothing else of the spectrum (the RMS history
// takes |mean / meanOverRMS|, computeRMSfromMean).  So:
//
//  rfi_stats_kernel  one CTA per spectrum of the block: clips with the margin
//                    expected from the state before the block, sums what is
//                    left in the canonical order, and records the largest
//                    value kept and the smallest value clipped.
//  rfi_scan_kernel   one CTA per beam: the running averages of all spectra of
//                    the block, 512 at a time, from the recorded sums, and for
//                    every spectrum the proof that its exact margin clips the
//                    recorded channels (it lies between the two recorded
//                    values).  Where the proof fails, and where a spectrum is
//                    rejected, fills the last good spectrum or resets the
//                    histories, that one spectrum is done over by the whole
//                    CTA with the exact state.
//  rfi_apply_kernel  one CTA per spectrum: clips with the exact margin,
//                    flattens, normalises and stores.
//  rfi_kernel        the walk, for what the scan left to it.
//
// The margin moves over a block, and a channel whose value lies between the
// expected and the exact margin fails the proof: rare in quiet data, common
// with strong RFI whose values reach down to the margin while the averages
// drift.  At the first failure the scan works out, in FP32, the margins that
// the recorded sums predict for the rest of the block.  Where they would fail
// more records it writes them down and leaves the rest to a second
// rfi_stats_kernel, which clips the unproven spectra with them, and a second
// rfi_scan_kernel; so does a scan that meets more failures than predicted.
// Both return at once where the first scan was enough.
//
// The running averages x <- fl(fl(x - a) + b) are rounded at every step, and
// every bit of them is kept: while x stays in one binade, x is an integer
// multiple X of that binade's spacing, and rounding x - a to the nearest
// multiple is X - rn(a / spacing) unless a / spacing lies exactly half way
// (where the even neighbour depends on X).  So the rounded chain is a sum of
// integers, and a prefix sum gives all of them at once.  A half-way case, or
// a binade's end, is one of the spectra that are done over.
//
// A spectrum done over costs as much as a step of the walk or up to four times
// that.  Where most of a block's spectra need it (the histories filling under a
// bandpass with terms, spectra rejected one after another, averages that stay
// 0, histories of a few spectra) the scan may leave the rest of the block to
// the walk, which goes on from the state where the scan stopped (scan_leaves).
//
// Bound: reading the block (stats), again from L2 (apply) and writing it; the
// scan is bound by the FP64 unit (each FP64 instruction of a warp takes its
// sub-partition 64 cycles: 128 for a chain of two adds whatever the number of
// spectra in flight, which is why the prefix sum is in integers).

// One spectrum's record (rfi_stats_kernel).
struct __align__(16) SpecRec {
    float ssum;           // canonical sum of the kept channels / their count
    int total_good;
    int bad_bands;
    int nfill;            // kept channels without a last good value
    float keep_max;       // largest value kept, smallest clipped: of the spectrum when the bandpass
    float clip_min;       //   is flat, else of (value - dataModel) - bandpass at dm_g, p0_g
    float srms, md4;      // adaptive phase: smallest band RMS, fifth smallest band minimum
    float dm_g, p0_g;
    int adaptive;         // 1: taken for a spectrum of the adaptive phase
    int pad;
};
// What rfi_apply_kernel needs of a spectrum (rfi_scan_kernel).
struct __align__(16) SpecOut {
    float dm, margin, params0, mean_f;
    int sclip;
    int pad[3];
};
struct RfiWork {
    SpecRec* rec;  // [kRfiBlock]
    SpecOut* out;  // [kRfiBlock]
    int* fill_at;  // [nbins] spectrum of the block that filled the channel's last good value (-1: earlier)
    int* hdr;      // see kHdr*
    int* hard;     // kHdrHard of the last block for the host, in its memory
};

// Spectra per block: the block of a 3904-channel beam (32 MB) stays in L2
// between the two passes over it, and a scan is four groups of 512.
constexpr int kRfiBlock = 2048;
constexpr int kScanThreads = 512;
constexpr int kZeroList = 2048;
// RfiWork::hdr: before the block, num and the channels without a last good
// value; after the first scan, the spectrum it reached, whether the second
// pass is wanted and whether a spectrum of the block has filled channels; after
// the last scan, the spectra that are done (the rest is the walk's) and whether
// it left any or had many to do over one by one.
constexpr int kHdrNum = 0, kHdrZeros = 1, kHdrPos = 2, kHdrRedo = 3, kHdrFilled = 4, kHdrEnd = 5, kHdrHard = 6,
              kHdrWords = 8;
// Failed proofs that the first scan does over by itself.  Each costs a scan of
// one spectrum and a group begun again, a second pass 3 to 15 us of statistics:
// the forecast at the first failure tells (more failures than kForecastMax,
// itself included, want the pass), and where it was wrong kAloneMax does.
constexpr int kForecastMax = 2, kAloneMax = 4;
constexpr int kForecast = 4;  // spectra per thread of a forecast: a whole block at once
constexpr int kSerial = 256;  // spectra of a group whose averages are added one by one, at most

// Order-preserving map of a float's bits to int (NaN excluded by the callers).
__device__ __forceinline__ int ord_f(float f) {
    const int b = __float_as_int(f);
    return b ^ ((b >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float unord_f(int o) { return __int_as_float(o ^ ((o >> 31) & 0x7fffffff)); }

// RFI_Clipper.cpp:383-394 on good-channel counts.
__device__ __forceinline__ int count_bad_bands(const Geo& geo, const int (&good)[8], int total_good) {
    int bad = 0;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        if (good[b] < geo.band_good_min) ++bad;
        if (good[b] == 0) bad += 4;
    }
    if (total_good < geo.good_min) bad += 4;
    return bad;
}

// Sum, sum of squares and minimum of the channels p, p+P, ... of band b
// (RFI_Clipper.cpp:214-278); get(c) is channel c's value.
template <int P, typename G>
__device__ __forceinline__ void band_partial(const Geo& geo, int p, int b, G get, float (&s12)[2], float& lo) {
    const int first = b * geo.cpb, end = first + geo.cpb;  // nbins is a multiple of 8
    s12[0] = s12[1] = 0.0f;
    lo = 1e6f;
    for (int c = first > p ? p + (first - p + P - 1) / P * P : p; c < end; c += P) {
        const float v = get(c);
        lo = fminf(lo, v);
        s12[0] = __fadd_rn(s12[0], v);
        s12[1] = __fadd_rn(s12[1], __fmul_rn(v, v));
    }
}

// The partials of 32 adjacent threads by the canonical tree; lane 0 stores
// them as the warp partials of warp index w.
template <int K>
__device__ __forceinline__ void warp_tree_at(float (&v)[K], float* red, int w) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) {
            const float o = __shfl_down_sync(0xffffffffu, v[k], off);
            if (lane < off) v[k] = __fadd_rn(v[k], o);
        }
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < K; ++k) red[w * K + k] = v[k];
}

// Warp partials of every band of partial p's 32 threads: red [band][warp][2],
// redm [band][warp] (minima of the data).
template <int P, typename G>
__device__ __forceinline__ void band_warps(const Geo& geo, int p, G get, float* red, float* redm) {
    for (int b = 0; b < 8; ++b) {
        float s12[2], lo;
        band_partial<P>(geo, p, b, get, s12, lo);
        lo = lane_min(lo);
        warp_tree_at<2>(s12, red + b * 64, p >> 5);
        if ((threadIdx.x & 31) == 0) redm[b * 32 + (p >> 5)] = lo;
    }
}
// Warp 0: smallest band RMS and the bands' minima from the warp partials of
// one spectrum.
template <int NW>
__device__ __forceinline__ float band_totals(const Geo& geo, const float* red, const float* redm, float (&md)[8]) {
    float srms = 0.0f;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        float pa[2], pm[1];
        lane_partials<1, NW>(red + b * 64, pa, 0.0f);
        lane_partials<1, NW>(redm + b * 32, pm, 1e30f);
        const float s1 = lane_tree<NW>(pa[0]);
        const float s2 = lane_tree<NW>(pa[1]);
        md[b] = lane_min(pm[0]);
        const float a = __fdiv_rn(s2, (float)geo.cpb);
        const float m = __fdiv_rn(s1, (float)geo.cpb);
        const float sg = __fsqrt_rn(__fsub_rn(a, __fmul_rn(m, m)));
        srms = (b == 0 || sg < srms) ? sg : srms;
    }
    return srms;
}
__device__ __forceinline__ float fifth_smallest(float (&x)[8]) {
    for (int i = 1; i < 8; ++i)
        for (int j = i; j > 0 && x[j - 1] > x[j]; --j) {
            const float y = x[j];
            x[j] = x[j - 1];
            x[j - 1] = y;
        }
    return x[4];
}

// ---------------------------------------------------------------------------
// Statistics of every spectrum of a block.  KM > 0: at most KM channels per
// thread, kept in registers; 0: any number, read again where needed.  PLAIN:
// one polarisation (a spectrum's channels are adjacent) and a flat bandpass.
// ---------------------------------------------------------------------------
// The clipped channels of a record are those of (dm, margin, p0).  Flat, the
// test is monotone in the channel's value, so the two nearest values decide
// for all.  Otherwise (value - dataModel) - bandpass moves by d0 for killed
// channels (whose bandpass is 0) and by d1 for the others between the recorded
// and the exact state, and slack covers the roundings of both evaluations.
__device__ __forceinline__ bool rfi_proven(const RfiConfig& cfg, bool flat, const SpecRec& r, float dm, float margin,
                                           float p0) {
    bool ok = true;
    if (flat) {
        const float bpf = __fmul_rn(cfg.scale, p0);
        if (r.total_good > 0 && !(__fsub_rn(__fsub_rn(r.keep_max, dm), bpf) <= margin)) ok = false;
        if (r.total_good < cfg.nbins && !(__fsub_rn(__fsub_rn(r.clip_min, dm), bpf) > margin)) ok = false;
    } else {
        const float big = fabsf(cfg.scale) * (fmaxf(fabsf(r.p0_g), fabsf(p0)) + cfg.term_abs);
        const float d0 = r.dm_g - dm, d1 = d0 + cfg.scale * (r.p0_g - p0);
        const float slack = 9.5367431640625e-7f * (float)(cfg.deg + 4) *
                            (fabsf(margin) + fabsf(dm) + fabsf(r.dm_g) + fabsf(d0) + fabsf(d1) + big);
        if (r.total_good > 0 && !(r.keep_max + fmaxf(d0, d1) + slack < margin)) ok = false;
        if (r.total_good < cfg.nbins && !(r.clip_min - 1e-5f * fabsf(r.clip_min) + fminf(d0, d1) - slack > margin))
            ok = false;
    }
    return ok;
}

template <int P, int KM, bool PLAIN>
__device__ __forceinline__ void rfi_stats_body(const RfiConfig& cfg, const RfiBuffers& bufs, const RfiWork& w,
                                               const float* __restrict__ row, const Geo& geo, int i, bool second) {
    constexpr int NW = P / 32;
    __shared__ float red[8 * 64], redm[8 * 32];
    __shared__ int s_max[32], s_min[32], s_fill[32], cnt[8];
    __shared__ float s_guess[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nbins = cfg.nbins;
    const bool flat = PLAIN || (cfg.deg == 0 && bufs.killed == nullptr);
    auto at = [&](int c) -> long long { return PLAIN ? c : geo.off(c); };
    const RfiState* S = bufs.state;
    float dm = 0.0f, margin, p0, srms = 0.0f, md4 = 0.0f;
    int adaptive;
    if (second) {
        if (w.hdr[kHdrRedo] == 0 || i < w.hdr[kHdrPos]) return;
        const SpecRec r = w.rec[i];
        const SpecOut o = w.out[i];
        adaptive = r.adaptive;
        if (adaptive && !flat) return;
        if (rfi_proven(cfg, flat, r, o.dm, o.margin, o.params0)) return;
        dm = o.dm;
        margin = o.margin;
        p0 = o.params0;
        srms = r.srms;
        md4 = r.md4;
    } else {
        adaptive = S->rms_size + i < cfg.history ? 1 : 0;
        p0 = S->params0;
        margin = __fmul_rn(cfg.cr, (float)S->rms_run);
        if (adaptive && !flat) {  // every such spectrum is done by the scan
            if (tid == 0) w.rec[i].adaptive = 1;
            return;
        }
    }
    const float bpf = __fmul_rn(cfg.scale, p0);
    float v[KM > 0 ? KM : 1];
    if constexpr (KM > 0) {
#pragma unroll
        for (int k = 0; k < KM; ++k) {
            const int c = tid + k * P;
            v[k] = c < nbins ? row[at(c)] : 0.0f;
        }
    }
    if (tid < 8) cnt[tid] = 0;
    if (adaptive && !second) {
        band_warps<P>(geo, tid, [&](int c) { return row[at(c)]; }, red, redm);
        __syncthreads();
        if (warp == 0) {
            float md[8];
            srms = band_totals<NW>(geo, red, redm, md);
            md4 = fifth_smallest(md);
            // expected running RMS: the block's spectra so far taken to be like this one
            const int rs = S->rms_size;
            const float rg = ((float)S->rms_acc + (float)(i + 1) * srms) / (float)(rs + i + 1);
            if (lane == 0) {
                s_guess[0] = __fadd_rn(__fsub_rn(md4, fminf(1e6f, bpf)), __fmul_rn(cfg.mmm_f, rg));
                s_guess[1] = __fmul_rn(cfg.cr, rg);
            }
        }
        __syncthreads();
        dm = s_guess[0];
        margin = s_guess[1];
    }
    __syncthreads();
    const bool zeros = S->remaining_zeros != 0;
    float g[1] = {0.0f};
    int kmax = ord_f(-INFINITY), cmin = ord_f(INFINITY), nfill = 0;
    auto channel = [&](int c, float x) {
        const float stat = __fsub_rn(__fsub_rn(x, dm), flat ? bpf : bp_value(cfg, bufs, p0, c));
        const bool clip = stat > margin;
        const float key = flat ? x : stat;
        if (clip) {
            cmin = min(cmin, ord_f(key));
            atomicAdd(&cnt[geo.band(c)], 1);
        } else {
            g[0] = __fadd_rn(g[0], x);
            if (key == key) kmax = max(kmax, ord_f(key));
            if (zeros && bufs.last_good[c] == 0.0f && x != 0.0f) ++nfill;
        }
    };
    if constexpr (KM > 0) {
#pragma unroll
        for (int k = 0; k < KM; ++k) {
            const int c = tid + k * P;
            if (c < nbins) channel(c, v[k]);
        }
    } else {
        for (int c = tid; c < nbins; c += P) channel(c, row[at(c)]);
    }
    warp_tree_at<1>(g, red, warp);
    kmax = __reduce_max_sync(0xffffffffu, kmax);
    cmin = __reduce_min_sync(0xffffffffu, cmin);
    nfill = __reduce_add_sync(0xffffffffu, nfill);
    if (lane == 0) {
        s_max[warp] = kmax;
        s_min[warp] = cmin;
        s_fill[warp] = nfill;
    }
    __syncthreads();
    if (warp == 0) {
        float pc[1];
        lane_partials<1, NW>(red, pc, 0.0f);
        const float gsum = lane_tree<NW>(pc[0]);
        kmax = __reduce_max_sync(0xffffffffu, lane < NW ? s_max[lane] : ord_f(-INFINITY));
        cmin = __reduce_min_sync(0xffffffffu, lane < NW ? s_min[lane] : ord_f(INFINITY));
        nfill = __reduce_add_sync(0xffffffffu, lane < NW ? s_fill[lane] : 0);
        if (lane == 0) {
            int good[8], total = 0;
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                good[b] = geo.cpb - cnt[b];  // nbins is a multiple of 8
                total += good[b];
            }
            SpecRec r;
            r.ssum = __fdiv_rn(gsum, (float)total);
            r.total_good = total;
            r.bad_bands = count_bad_bands(geo, good, total);
            r.nfill = nfill;
            r.keep_max = unord_f(kmax);
            r.clip_min = unord_f(cmin);
            r.srms = srms;
            r.md4 = md4;
            r.dm_g = dm;
            r.p0_g = p0;
            r.adaptive = adaptive;
            r.pad = 0;
            w.rec[i] = r;
        }
    }
}

// ---------------------------------------------------------------------------
// Running averages as integers of one binade
// ---------------------------------------------------------------------------
struct Binade {  // x = X * 2^(e - bias - mantissa bits)
    long long X;
    int e;
    bool ok;
};
__device__ __forceinline__ Binade binade64(double x) {
    const long long b = __double_as_longlong(x);
    const int e = (int)((b >> 52) & 0x7ff);
    long long m = (b & 0xfffffffffffffLL) | (1LL << 52);
    return {b < 0 ? -m : m, e, e >= 64 && e < 0x7fe};
}
__device__ __forceinline__ double value64(long long X, int e) {
    const long long m = X < 0 ? -X : X;
    return __longlong_as_double((X < 0 ? (1LL << 63) : 0LL) | ((long long)e << 52) | (m & 0xfffffffffffffLL));
}
// (double)f and the float nearest to X * 2^(e - 1075), |X| in [2^52, 2^53),
// in integer instructions.
__device__ __forceinline__ double widen(float f) {
    const int b = __float_as_int(f), e = (b >> 23) & 0xff;
    if (e == 0 || e == 0xff) return (double)f;
    return __hiloint2double((b & (int)0x80000000) | ((e + 896) << 20) | ((b & 0x7fffff) >> 3), b << 29);
}
__device__ __forceinline__ float narrow(double x) {
    const long long b = __double_as_longlong(x);
    const int e = (int)((b >> 52) & 0x7ff) - 896;
    if (e < 1 || e > 253) return (float)x;
    const long long m = b & 0xfffffffffffffLL;
    int r = (e << 23) | (int)(m >> 29);
    const int rem = (int)(m & 0x1fffffff);
    if (rem > 0x10000000 || (rem == 0x10000000 && (r & 1))) ++r;  // a carry moves into the exponent
    return __int_as_float((b < 0 ? (int)0x80000000 : 0) | r);
}
// x strictly inside its binade: the neighbouring values on both sides have its spacing
__device__ __forceinline__ bool inside64(long long X) {
    const long long m = X < 0 ? -X : X;
    return m > (1LL << 52) && m < (1LL << 53);
}
__device__ __forceinline__ Binade binade32(float x) {
    const int b = __float_as_int(x);
    const int e = (b >> 23) & 0xff;
    const long long m = (b & 0x7fffff) | (1 << 23);
    return {b < 0 ? -m : m, e, e >= 40 && e < 0xfe};
}
__device__ __forceinline__ float value32(long long X, int e) {
    const int m = (int)(X < 0 ? -X : X);
    return __int_as_float((X < 0 ? (int)0x80000000 : 0) | (e << 23) | (m & 0x7fffff));
}
__device__ __forceinline__ bool inside32(long long X) {
    const long long m = X < 0 ? -X : X;
    return m > (1LL << 23) && m < (1LL << 24);
}
// a in spacings of the binade e of MB mantissa bits, rounded to nearest;
// false: half way, not finite, or too large for the sums of a group not to
// overflow (a quarter of the binade's lower end and more).
template <int MB>
__device__ __forceinline__ bool spacings(unsigned long long mag, bool neg, int ea, int e, long long& q) {
    const int sh = e - ea;
    q = 0;
    if (ea == (MB == 52 ? 0x7ff : 0xff) || sh < 2) return false;
    if (ea == 0 || sh > MB + 1) return true;  // below half a spacing
    const unsigned long long m = mag | (1ULL << MB);
    const unsigned long long rem = m & ((1ULL << sh) - 1), half = 1ULL << (sh - 1);
    long long r = (long long)(m >> sh);
    if (rem > half) ++r;
    q = neg ? -r : r;
    return rem != half;
}
__device__ __forceinline__ bool spacings64(double a, int e, long long& q) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(a);
    return spacings<52>(b & 0xfffffffffffffULL, (b >> 63) != 0, (int)((b >> 52) & 0x7ff), e, q);
}
__device__ __forceinline__ bool spacings32(float a, int e, long long& q) {
    const unsigned b = (unsigned)__float_as_int(a);
    return spacings<23>(b & 0x7fffffu, (b >> 31) != 0, (int)((b >> 23) & 0xff), e, q);
}

// Inclusive prefix sum over the CTA's threads.  wt: one word per warp, not in
// use by any other scan since the last barrier but one.
__device__ __forceinline__ long long block_scan(long long x, long long* wt) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wt[warp] = x;
    __syncthreads();
    long long t = lane < kScanThreads / 32 ? wt[lane] : 0;
#pragma unroll
    for (int o = 1; o < kScanThreads / 32; o <<= 1) {
        const long long y = __shfl_up_sync(0xffffffffu, t, o);
        if (lane >= o) t += y;
    }
    const long long before = __shfl_sync(0xffffffffu, t, warp == 0 ? 0 : warp - 1);
    return warp == 0 ? x : x + before;
}

// ---------------------------------------------------------------------------
// One CTA per beam: the state chain over a block's spectra.
// ---------------------------------------------------------------------------
struct ScanShared {
    RfiState st;
    long long wt[3][kScanThreads / 32];
    double E[kScanThreads];
    float rf[kScanThreads], mf[kScanThreads], pi[kScanThreads], pb[kScanThreads];
    int first_bad;
    float dm, margin;
    int fill, filled, rejected;
    float red[8 * 64], redm[8 * 32], redb[8 * 32];
    double fa[kSerial], fb[kSerial], fx[kSerial], ga[kSerial], gx[kSerial];
    int cnt[8];
    int zn;
    int zlist[kZeroList];
};

// The channels without a last good value.
__device__ __forceinline__ void list_zeros(ScanShared& sh, const RfiConfig& cfg, const RfiBuffers& bufs) {
    if (threadIdx.x == 0) sh.zn = 0;
    __syncthreads();
    for (int c = threadIdx.x; c < cfg.nbins; c += kScanThreads)
        if (bufs.last_good[c] == 0.0f) {
            const int k = atomicAdd(&sh.zn, 1);
            if (k < kZeroList) sh.zlist[k] = c;
        }
    __syncthreads();
}

// One spectrum with the exact state, by the whole CTA (RFI_Clipper.cpp:190-567
// without the data's own flattening and normalisation).
template <int P>
__device__ __forceinline__ void scan_one(ScanShared& sh, const RfiConfig& cfg, const RfiBuffers& bufs,
                                         const RfiWork& w, const float* __restrict__ row, const Geo& geo, int i) {
    constexpr int NW = P / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nbins = cfg.nbins, H = cfg.history;
    const bool flat = cfg.deg == 0 && bufs.killed == nullptr;
    const double inv_h = cfg.inv_h;
    const bool adaptive = sh.st.rms_size < H;
    const float p0 = sh.st.params0;
    const float bpf = __fmul_rn(cfg.scale, p0);
    auto bpv = [&](int c) { return flat ? bpf : bp_value(cfg, bufs, p0, c); };
    if (tid < 8) sh.cnt[tid] = 0;
    if (tid == 0) sh.filled = 0;
    if (adaptive) {
        for (int p = tid; p < P; p += kScanThreads) {
            band_warps<P>(geo, p, [&](int c) { return row[geo.off(c)]; }, sh.red, sh.redm);
            if (!flat)  // the bands' minima of the bandpass
                for (int b = 0; b < 8; ++b) {
                    float s12[2], lo;
                    band_partial<P>(geo, p, b, bpv, s12, lo);
                    lo = lane_min(lo);
                    if (lane == 0) sh.redb[b * 32 + (p >> 5)] = lo;
                }
        }
    }
    __syncthreads();
    RfiState st;  // warp 0: every lane the same
    if (warp == 0) {
        st = sh.st;
        float dm = 0.0f;
        if (adaptive) {
            float md[8];
            const float srms = band_totals<NW>(geo, sh.red, sh.redm, md);
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                float pb[1] = {fminf(1e6f, bpf)};
                if (!flat) {
                    lane_partials<1, NW>(sh.redb + b * 32, pb, 1e30f);
                    pb[0] = lane_min(pb[0]);
                }
                md[b] = __fsub_rn(md[b], pb[0]);
            }
            const float d4 = fifth_smallest(md);
            const int pos = wrap_h(st.rms_head + st.rms_size, H);
            if (lane == 0) bufs.rms_buf[pos] = (double)srms;
            st.rms_acc_prev = st.rms_acc;
            st.rms_acc = st.rms_acc + (double)srms;
            st.rms_size += 1;
            st.rms_run = st.rms_acc / (double)st.rms_size;
            if (st.rms_size == H) {
                st.mean_over_rms = st.mean_run / st.rms_run;
                st.inv_mor = 1.0 / st.mean_over_rms;
            }
            dm = __fadd_rn(d4, __fmul_rn(cfg.mmm_f, (float)st.rms_run));
        } else {
            const double front = bufs.rms_buf[st.rms_head];
            const double last = bufs.rms_buf[wrap_h(st.rms_head + H - 1, H)];
            st.rms_run = st.rms_run - front * inv_h;
            st.rms_run = st.rms_run + last * inv_h;
            __syncwarp();
            if (lane == 0) bufs.rms_buf[st.rms_head] = fabs(st.mean_run * st.inv_mor);
            st.rms_head = wrap_h(st.rms_head + 1, H);
        }
        if (lane == 0) {
            sh.dm = dm;
            sh.margin = __fmul_rn(cfg.cr, (float)st.rms_run);
        }
        __syncwarp();
    }
    __syncthreads();
    const float dm = sh.dm, margin = sh.margin;
    for (int p = tid; p < P; p += kScanThreads) {
        float g[1] = {0.0f};
        for (int c = p; c < nbins; c += P) {
            const float v = row[geo.off(c)];
            if (__fsub_rn(__fsub_rn(v, dm), bpv(c)) > margin) atomicAdd(&sh.cnt[geo.band(c)], 1);
            else g[0] = __fadd_rn(g[0], v);
        }
        warp_tree_at<1>(g, sh.red, p >> 5);
    }
    __syncthreads();
    if (warp == 0) {
        float pc[1];
        lane_partials<1, NW>(sh.red, pc, 0.0f);
        const float gsum = lane_tree<NW>(pc[0]);
        int good[8], total = 0;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            good[b] = geo.cpb - sh.cnt[b];
            total += good[b];
        }
        const float ssum = __fdiv_rn(gsum, (float)total);
        const int bad_bands = count_bad_bands(geo, good, total);
        // the newest entry before this spectrum's (0 when there is none)
        const double prev = st.mean_size > 0 ? bufs.mean_buf[(st.mean_head + st.mean_size - 1) % H] : 0.0;
        if (st.mean_size < H) {
            const int pos = wrap_h(st.mean_head + st.mean_size, H);
            __syncwarp();
            if (lane == 0) bufs.mean_buf[pos] = (double)ssum;
            st.mean_acc_prev = st.mean_acc;
            st.mean_acc = st.mean_acc + (double)ssum;
            st.mean_size += 1;
            st.mean_run = st.mean_acc / (double)st.mean_size;
        } else {
            const double front = bufs.mean_buf[st.mean_head];
            st.mean_run = st.mean_run - front * inv_h;
            st.mean_run = st.mean_run + prev * inv_h;
            __syncwarp();
            if (lane == 0) bufs.mean_buf[st.mean_head] = (double)ssum;
            st.mean_head = wrap_h(st.mean_head + 1, H);
        }
        const float tol = (float)((double)__fmul_rn(cfg.sr, st.bp_rms) * cfg.inv_sqrt_nbins);
        int sclip = 0, fill = 0;
        if (st.mean_size < 1000) {
            sclip = 1;
        } else if ((double)ssum - st.mean_run > (double)tol || bad_bands >= 4) {
            sclip = 1;
            st.bad_spectra += 1;
            // pop_back + push_back(back()): the newest entry takes the previous one's value
            const int mlast = wrap_h(st.mean_head + st.mean_size - 1, H);
            const int rlast = wrap_h(st.rms_head + st.rms_size - 1, H);
            const double rprev = st.rms_size > 1 ? bufs.rms_buf[(st.rms_head + st.rms_size - 2) % H] : 0.0;
            __syncwarp();
            if (lane == 0) {
                bufs.mean_buf[mlast] = prev;
                bufs.rms_buf[rlast] = rprev;
            }
            st.mean_acc = st.mean_acc_prev + prev;
            st.rms_acc = st.rms_acc_prev + rprev;
        } else if (st.remaining_zeros != 0) {
            fill = 1;
        }
        if (lane == 0) {
            w.rec[i].total_good = total;
            w.out[i] = SpecOut{dm, margin, p0, (float)st.mean_run, sclip, {0, 0, 0}};
            sh.fill = fill;
            sh.rejected = st.mean_size >= 1000 && sclip != 0 ? 1 : 0;
        }
    }
    __syncthreads();
    if (sh.fill) {  // RFI_Clipper.cpp:441-460: kept channels that have no last good value yet
        int n = 0;
        for (int c = tid; c < nbins; c += kScanThreads) {
            const float v = row[geo.off(c)];
            if (!(__fsub_rn(__fsub_rn(v, dm), bpv(c)) > margin) && bufs.last_good[c] == 0.0f && v != 0.0f) {
                bufs.last_good[c] = v;
                w.fill_at[c] = i;
                ++n;
            }
        }
        n = __reduce_add_sync(0xffffffffu, n);
        if (lane == 0 && n) atomicAdd(&sh.filled, n);
        __syncthreads();
    }
    if (warp == 0) {
        st.remaining_zeros -= sh.filled;
        // statistics (RFI_Clipper.cpp:535-560)
        if (st.num == 0) {
            const float frac = (float)(100.0 * (float)st.bad_spectra / (float)(10 * H));
            if (frac > 99.0f) {
                st.mean_size = st.rms_size = 0;
                st.mean_head = st.rms_head = 0;
                st.mean_acc = st.mean_acc_prev = st.rms_acc = st.rms_acc_prev = 0.0;
            }
            st.bad_spectra = 0;
        }
        // BandPass::setMean / setRMS (BandPass.cpp:44-74)
        const float mean_f = (float)st.mean_run;
        const float delta = __fsub_rn(mean_f, st.bp_mean);
        if (fabsf(delta) > 0.0f) {
            st.params0 = __fadd_rn(st.params0, __fdiv_rn(delta, cfg.scale));
            st.bp_mean = mean_f;
        }
        st.bp_rms = (float)st.rms_run;
        st.num = (st.num + 1) % (10 * H);
        if (lane == 0) sh.st = st;
    }
    if (sh.fill && sh.filled) list_zeros(sh, cfg, bufs);
    __syncthreads();
}

enum ScanMode {
    kParallel,  // prefix sums of integers
    kOneByOne,  // FP64 adds by one thread
    kPredict    // approximate, nothing committed
};

// x <- fl(fl(x - a) + b) over the group's m spectra: x after spectrum k and
// before it.  False: the integers do not give spectrum k's value (a half-way
// case, or outside x's binade).
__device__ __forceinline__ bool slide(ScanShared& sh, double x0, double a, double b, int k, int m, ScanMode mode,
                                      int which, double& x, double& before) {
    if (mode == kOneByOne) {
        if (k < m) {
            sh.fa[k] = a;
            sh.fb[k] = b;
        }
        __syncthreads();
        if (k == 0) {
            double y = x0;
            for (int j = 0; j < m; ++j) {
                y = y - sh.fa[j];
                y = y + sh.fb[j];
                sh.fx[j] = y;
            }
        }
        __syncthreads();
        x = k < m ? sh.fx[k] : 0.0;
        before = k == 0 ? x0 : (k < m ? sh.fx[k - 1] : 0.0);
        __syncthreads();
        return true;
    }
    const Binade z = binade64(x0);
    long long qa = 0, qb = 0;
    bool ok = z.ok;
    ok &= spacings64(a, z.e, qa) || k >= m;
    ok &= spacings64(b, z.e, qb) || k >= m;
    const long long X = z.X + block_scan(qb - qa, sh.wt[which]);
    if (mode == kPredict) {
        const double u = __longlong_as_double((long long)max(z.e - 52, 1) << 52);
        x = (double)X * u;
        before = (double)(X - qb + qa) * u;
        return true;
    }
    ok &= inside64(X) && inside64(X - qb);
    x = value64(X, z.e);
    before = k == 0 ? x0 : value64(X - qb + qa, z.e);
    return ok;
}

// Up to m spectra from spectrum i of the block; returns how many of them are
// proven and committed, and whether the integers stopped it (chain) or a
// failed proof (unproven).  kPredict: writes the expected margins of all m
// and moves the shared state on, but no history and nothing else.
__device__ __forceinline__ int scan_group(ScanShared& sh, const RfiConfig& cfg, const RfiBuffers& bufs,
                                          const RfiWork& w, const float* __restrict__ rows, long long spec_elems,
                                          const Geo& geo, int i, int m, bool filled, ScanMode mode, bool& chain,
                                          bool& unproven) {
    const int k = threadIdx.x;
    const int H = cfg.history;
    const bool act = k < m;
    const bool flat = cfg.deg == 0 && bufs.killed == nullptr;
    const double inv_h = cfg.inv_h;
    const RfiState& st = sh.st;
    const bool adaptive = st.rms_size < H;
    const bool predict = mode == kPredict;
    const int mhead = st.mean_head, rhead = st.rms_head, size0 = st.rms_size;
    SpecRec r{};
    if (act) r = w.rec[i + k];
    // a spectrum's entry of the mean history; predicted, a rejected one leaves the mean where it is
    const float loud = predict ? narrow(st.mean_run) + 1.01f * cfg.sr * st.bp_rms * (float)cfg.inv_sqrt_nbins : 0.0f;
    auto entry = [&](const SpecRec& q) {
        return predict && size0 >= 1000 && (q.ssum > loud || q.bad_bands >= 4) ? st.mean_run : widen(q.ssum);
    };
    const double V = entry(r);
    bool bad = false;
    double M, R, macc = 0.0, macc_prev = 0.0, racc = 0.0, racc_prev = 0.0, E = 0.0;
    if (k == 0) sh.first_bad = 4 * m;
    const bool other_phase = (r.adaptive != 0) != adaptive;  // the record is of the other phase
    if (!adaptive) {
        // mean: fl(fl(M - oldest / H) + newest / H); then the RMS history's
        // entry |mean before / meanOverRMS|, and the same for the RMS
        double a = 0.0, b = 0.0, Mp;
        if (act) {
            a = bufs.mean_buf[wrap_h(mhead + k, H)] * inv_h;
            if (k > 0) b = widen(w.rec[i + k - 1].ssum);
            else b = bufs.mean_buf[wrap_h(mhead + H - 1, H)];
            b = b * inv_h;
        }
        bad = !slide(sh, st.mean_run, a, b, k, m, mode, 0, M, Mp);
        E = fabs(Mp * st.inv_mor);
        sh.E[k] = E;
        __syncthreads();
        if (act) {
            a = bufs.rms_buf[wrap_h(rhead + k, H)] * inv_h;
            if (k > 0) b = sh.E[k - 1];
            else b = bufs.rms_buf[wrap_h(rhead + H - 1, H)];
            b = b * inv_h;
        }
        bad |= !slide(sh, st.rms_run, a, b, k, m, mode, 1, R, Mp);
    } else {
        const double srms = widen(r.srms);
        if (mode == kOneByOne) {
            if (act) {
                sh.fa[k] = srms;
                sh.fb[k] = V;
            }
            __syncthreads();
            // two warps of different sub-partitions
            if (k == 0) {
                double y = st.rms_acc;
                for (int j = 0; j < m; ++j) sh.fx[j] = y = y + sh.fa[j];
            }
            if (k == 32) {
                double y = st.mean_acc;
                for (int j = 0; j < m; ++j) sh.gx[j] = y = y + sh.fb[j];
            }
            __syncthreads();
            if (act) {
                racc = sh.fx[k];
                macc = sh.gx[k];
                racc_prev = k == 0 ? st.rms_acc : sh.fx[k - 1];
                macc_prev = k == 0 ? st.mean_acc : sh.gx[k - 1];
            }
        } else {
            bad = !slide(sh, st.rms_acc, 0.0, srms, k, m, mode, 0, racc, racc_prev);
            bad |= !slide(sh, st.mean_acc, 0.0, V, k, m, mode, 1, macc, macc_prev);
        }
        const double n = (double)(size0 + 1 + k);
        R = racc / n;
        M = macc / n;
    }
    const bool chain_bad = bad;
    const float Rf = narrow(R), Mf = narrow(M);
    sh.rf[k] = Rf;
    sh.mf[k] = Mf;
    __syncthreads();
    const float bp_rms = k == 0 ? st.bp_rms : sh.rf[k - 1];
    // params[0] of the bandpass: one rounded FP32 add per spectrum whose mean changed
    const float delta = __fsub_rn(Mf, k == 0 ? st.bp_mean : sh.mf[k - 1]);
    const bool step = act && fabsf(delta) > 0.0f;
    const float pinc = step ? __fdiv_rn(delta, cfg.scale) : 0.0f;
    float p_before, p_after;
    if (predict) {
        p_before = st.params0 + (k == 0 ? 0.0f : (sh.mf[k - 1] - st.bp_mean) / cfg.scale);
        p_after = st.params0 + (Mf - st.bp_mean) / cfg.scale;
    } else {
        const Binade bpz = binade32(st.params0);
        long long qp = 0;
        bool pbad = act && (!bpz.ok || !spacings32(pinc, bpz.e, qp));
        const long long Z = bpz.X + block_scan(qp, sh.wt[2]);
        pbad |= act && !inside32(Z);
        p_before = k == 0 ? st.params0 : value32(Z - qp, bpz.e);
        p_after = value32(Z, bpz.e);
        if (__syncthreads_or(pbad && !bad)) {
            // half-way sums or another binade: warp 0 adds them one by one
            sh.pi[k] = pinc;
            __syncthreads();
            if (k < 32) {
                float p = st.params0;
                for (int b = 0; b < m; b += 32) {
                    const float x = sh.pi[b + k];
                    float mine = 0.0f;
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const float y = __shfl_sync(0xffffffffu, x, j);
                        if (k == j) mine = p;
                        if (y != 0.0f) p = __fadd_rn(p, y);
                    }
                    sh.pb[b + k] = mine;
                }
            }
            __syncthreads();
            p_before = sh.pb[k];
            p_after = step ? __fadd_rn(p_before, pinc) : p_before;
        }
    }
    const int size = adaptive ? size0 + 1 + k : H;
    const float margin = __fmul_rn(cfg.cr, Rf);
    const float bpf = __fmul_rn(cfg.scale, p_before);
    const float dm = adaptive ? __fadd_rn(__fsub_rn(r.md4, fminf(1e6f, bpf)), __fmul_rn(cfg.mmm_f, Rf)) : 0.0f;
    const bool early = size < 1000;
    int f = m;
    chain = unproven = false;
    if (!predict) {
        const bool wrong = other_phase || !rfi_proven(cfg, flat, r, dm, margin, p_before);
        bad |= wrong;
        if (!early) {
            // Rejection compares V - mean with the tolerance in double: clear cases by their FP32
            // values (whose errors are below the bound subtracted), the others exactly.
            const float tolf = cfg.sr * bp_rms * (float)cfg.inv_sqrt_nbins;
            const float gap = 1e-6f * (fabsf(r.ssum) + fabsf(Mf) + fabsf(tolf));
            if (!(r.ssum - Mf < tolf - gap)) {
                const float tol = (float)((double)__fmul_rn(cfg.sr, bp_rms) * cfg.inv_sqrt_nbins);
                if (V - M > (double)tol) bad = true;
            }
            if (r.bad_bands >= 4) bad = true;
            if (act && !bad && st.remaining_zeros != 0 && r.nfill > 0) {
                if (!filled || sh.zn > kZeroList) {
                    bad = true;
                } else {  // the record counts channels that an earlier spectrum of the block has filled
                    const float* row = rows + (long long)(i + k) * spec_elems;
                    for (int z = 0; z < sh.zn; ++z) {
                        const int c = sh.zlist[z];
                        const float v = row[geo.off(c)];
                        const float bp = flat ? bpf : bp_value(cfg, bufs, p_before, c);
                        if (v != 0.0f && !(__fsub_rn(__fsub_rn(v, dm), bp) > margin)) {
                            bad = true;
                            break;
                        }
                    }
                }
            }
        }
        // the first spectrum that is not proven, and why: 0 the integers, 1 its record, 2 its own event
        const int why = chain_bad ? 0 : (wrong ? 1 : 2);
        const int mine = __reduce_min_sync(0xffffffffu, act && bad ? 4 * k + why : 4 * m);
        if ((k & 31) == 0 && mine < 4 * m) atomicMin(&sh.first_bad, mine);
        __syncthreads();
        f = sh.first_bad >> 2;
        chain = f < m && (sh.first_bad & 3) == 0;
        unproven = f < m && (sh.first_bad & 3) == 1;
    }
    const int num = st.num;
    __syncthreads();  // every read of the state is done
    if (k < f) {
        if (!predict) {
            if (!adaptive) {
                bufs.mean_buf[wrap_h(mhead + k, H)] = V;
                bufs.rms_buf[wrap_h(rhead + k, H)] = E;
            } else {
                bufs.mean_buf[wrap_h(mhead + size0 + k, H)] = V;
                bufs.rms_buf[wrap_h(rhead + size0 + k, H)] = widen(r.srms);
            }
        }
        w.out[i + k] = SpecOut{dm, margin, p_before, Mf, early ? 1 : 0, {0, 0, 0}};
        if (k == f - 1) {
            RfiState& s = sh.st;
            if (!adaptive) {
                s.mean_head = wrap_h(mhead + f, H);
                s.rms_head = wrap_h(rhead + f, H);
            } else {
                s.mean_size = s.rms_size = size0 + f;
                s.mean_acc = macc;
                s.mean_acc_prev = macc_prev;
                s.rms_acc = racc;
                s.rms_acc_prev = racc_prev;
            }
            s.mean_run = M;
            s.rms_run = R;
            s.bp_mean = Mf;
            s.bp_rms = Rf;
            s.params0 = p_after;
            s.num = (num + f) % (10 * H);
        }
    }
    __syncthreads();
    return f;
}

// FP32 prefix sums over kForecast * kScanThreads values, v[j] being number
// j * kScanThreads + thread: what lies before each (before) and up to it (v).
// wt: a word per warp and j, not in use since the last barrier.
__device__ __forceinline__ void block_scan_f(float (&v)[kForecast], float (&before)[kForecast], float* wt) {
    constexpr int NW = kScanThreads / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float x[kForecast];
#pragma unroll
    for (int j = 0; j < kForecast; ++j) x[j] = v[j];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
#pragma unroll
        for (int j = 0; j < kForecast; ++j) {
            const float y = __shfl_up_sync(0xffffffffu, x[j], o);
            if (lane >= o) x[j] += y;
        }
    if (lane == 31)
#pragma unroll
        for (int j = 0; j < kForecast; ++j) wt[j * NW + warp] = x[j];
    __syncthreads();
    static_assert(kForecast * NW == 64, "two warp totals a lane");
    const float t0 = wt[2 * lane], t1 = wt[2 * lane + 1];
    float t = t0 + t1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float y = __shfl_up_sync(0xffffffffu, t, o);
        if (lane >= o) t += y;
    }
    // t: the totals up to number 2 * lane + 1
#pragma unroll
    for (int j = 0; j < kForecast; ++j) {
        const int q = j * NW + warp;
        const float upto = __shfl_sync(0xffffffffu, t, q >> 1), odd = __shfl_sync(0xffffffffu, t1, q >> 1);
        const float own = __shfl_sync(0xffffffffu, t0, q >> 1);
        const float base = (q & 1) ? upto - odd : upto - odd - own;
        before[j] = base + (x[j] - v[j]);
        v[j] = base + x[j];
    }
}

// The expected margins of spectra i..n-1 with full histories, from the records
// and in FP32, written to RfiWork::out; returns how many records they do not
// prove.  exact: the shared state is the one before spectrum i (else the
// newest history entry is the record's before it).  The state and the
// histories stay as they are.  18k cycles for 2048 spectra; by the exact
// scan's groups, as the adaptive phase still does it, 48k.
__device__ __forceinline__ int scan_forecast(ScanShared& sh, const RfiConfig& cfg, const RfiBuffers& bufs,
                                             const RfiWork& w, int i, int n, bool exact) {
    const int tid = threadIdx.x;
    const int H = cfg.history;
    const RfiState& st = sh.st;
    const bool flat = cfg.deg == 0 && bufs.killed == nullptr;
    const float inv_h = narrow(cfg.inv_h), inv_mor = narrow(st.inv_mor), mean_first = narrow(st.mean_run);
    const float inv_scale = 1.0f / cfg.scale;
    // a rejected spectrum leaves the mean where it is
    const float loud = mean_first + 1.01f * cfg.sr * st.bp_rms * narrow(cfg.inv_sqrt_nbins);
    float mean0 = mean_first, rms0 = narrow(st.rms_run);
    int mhead = st.mean_head, rhead = st.rms_head;
    __syncthreads();
    if (tid == 0) sh.first_bad = 0;
    while (i < n) {
        const int m = min(min(kForecast * kScanThreads, n - i), H);
        float dm[kForecast], dr[kForecast], mb[kForecast], rb[kForecast], old[kForecast];
#pragma unroll
        for (int j = 0; j < kForecast; ++j) {
            const int k = j * kScanThreads + tid;
            dm[j] = old[j] = 0.0f;
            if (k < m) {
                float b;
                if (k > 0 || !exact) {
                    const SpecRec& q = w.rec[i + k - 1];
                    b = H >= 1000 && (q.ssum > loud || q.bad_bands >= 4) ? mean_first : q.ssum;
                } else {
                    b = narrow(bufs.mean_buf[wrap_h(mhead + H - 1, H)]);
                }
                dm[j] = (b - narrow(bufs.mean_buf[wrap_h(mhead + k, H)])) * inv_h;
                old[j] = narrow(bufs.rms_buf[wrap_h(rhead + k, H)]);
            }
        }
        block_scan_f(dm, mb, sh.rf);
#pragma unroll
        for (int j = 0; j < kForecast; ++j) {
            // the entry |mean / meanOverRMS| of the spectrum before, to one step of the mean
            const float b = fabsf((mean0 + mb[j]) * inv_mor);
            dr[j] = j * kScanThreads + tid < m ? (b - old[j]) * inv_h : 0.0f;
        }
        block_scan_f(dr, rb, sh.mf);
        int bad = 0;
#pragma unroll
        for (int j = 0; j < kForecast; ++j) {
            const int k = j * kScanThreads + tid;
            if (k >= m) continue;
            const float mean = mean0 + dm[j], rms = rms0 + dr[j], margin = cfg.cr * rms;
            const float p = st.params0 + (mean0 + mb[j] - st.bp_mean) * inv_scale;
            bad += rfi_proven(cfg, flat, w.rec[i + k], 0.0f, margin, p) ? 0 : 1;
            w.out[i + k] = SpecOut{0.0f, margin, p, mean, 0, {0, 0, 0}};
            if (k == m - 1) {
                sh.pi[0] = mean;
                sh.pi[1] = rms;
            }
        }
        bad = __reduce_add_sync(0xffffffffu, bad);
        if ((tid & 31) == 0 && bad) atomicAdd(&sh.first_bad, bad);
        __syncthreads();
        mean0 = sh.pi[0];
        rms0 = sh.pi[1];
        i += m;
        mhead = wrap_h(mhead + m, H);
        rhead = wrap_h(rhead + m, H);
        exact = false;
        __syncthreads();
    }
    return sh.first_bad;
}

// Spectra done over one by one in a scan so far, by why.
struct ScanAlone {
    int rejected, idle, other;  // idle: averages that are 0 (or not finite, or tiny)
    __device__ __forceinline__ int all() const { return rejected + idle + other; }
};

// Whether the walk would do spectra i..n-1 sooner: more of them are expected to
// be done over one by one than the walk's time is worth, as a part of them all.
// While the histories fill under a bandpass with terms every one is.  Rejected
// ones are counted in the records; others are taken to come on as often as
// since spectrum i0, which takes many to believe unless the block before was
// such a one.  us a spectrum by 64 / 512 / 1024 / 4096 / 8192 / 15616 channels:
// walked 2.4 2.9 4.1 6.2 6.7 8.7, all rejected 2.8 3.1 3.8 5.2 8.5 19, every
// fourth 9.2 9.2 9.8 11 14 20 for each rejected; with terms, walked 2.5 3.3 4.2
// 6.2 6.8 9.0 and averages of 0 3.2 3.6 4.8 8.8 16 38; the histories filling
// with terms, walked 5.9 6.8 8.7 14 15 19 and one by one 10 9.3 11 15 27 43.
__device__ __forceinline__ bool scan_leaves(const ScanShared& sh, const RfiConfig& cfg, const RfiWork& w, bool flat,
                                            int i0, int i, int n, const ScanAlone& alone) {
    const RfiState& st = sh.st;
    const int left = n - i, nbins = cfg.nbins;
    if (left <= 16) return false;
    if (!flat && st.rms_size < cfg.history) {
        const float part = nbins <= 128    ? 0.37f
                           : nbins <= 512  ? 0.45f
                           : nbins <= 1024 ? 0.65f
                           : nbins <= 4096 ? 0.85f
                           : nbins <= 8192 ? 0.45f
                                           : 0.35f;
        return (float)min(left, cfg.history - st.rms_size) >= part * (float)left;
    }
    const int done = alone.all();
    if (done < 8 || (done & (done - 1)) != 0) return false;  // looked into at 8, 16, 32, ...
    // parts of the spectra left from which on the walk is sooner (above 1: never)
    const float part_rejected = nbins <= 512 ? 0.3f : (nbins <= 4096 ? 2.0f : 0.45f);
    const float part_idle = nbins > 512 && nbins <= 4096 && !flat ? 0.8f : part_rejected;
    int rejected = 0;
    if (st.mean_size >= 1000) {
        const float loud = narrow(st.mean_run) + cfg.sr * st.bp_rms * narrow(cfg.inv_sqrt_nbins);
        for (int k = i; k < n; k += kScanThreads) {
            const int j = k + (int)threadIdx.x;
            rejected += __syncthreads_count(j < n && (w.rec[j].ssum > loud || w.rec[j].bad_bands >= 4));
        }
    }
    const bool many = alone.idle + alone.other >= (w.hdr[kHdrHard] != 0 ? 32 : 512);
    const float of_left = many ? (float)left / (float)(i - i0) : 0.0f;
    return ((float)rejected + of_left * (float)alone.other) / part_rejected + of_left * (float)alone.idle / part_idle >=
           (float)left;
}

template <int P>
__device__ __forceinline__ void rfi_scan_body(const RfiConfig& cfg, const RfiBuffers& bufs, const RfiWork& w,
                                              const float* __restrict__ rows, const Geo& geo, int n, bool second,
                                              bool may_leave) {
    __shared__ ScanShared sh;
    const int tid = threadIdx.x;
    const long long spec_elems = (long long)geo.nsub * geo.npol * geo.nchan;
    const bool flat = cfg.deg == 0 && bufs.killed == nullptr;
    const int H = cfg.history;
    if (second && w.hdr[kHdrRedo] == 0) return;
    int i = second ? w.hdr[kHdrPos] : 0;
    bool filled = second && w.hdr[kHdrFilled] != 0;
    if (tid == 0) {
        sh.st = *bufs.state;
        if (!second) {
            w.hdr[kHdrNum] = sh.st.num;
            w.hdr[kHdrZeros] = sh.st.remaining_zeros;
        }
        sh.zn = 0;
    }
    __syncthreads();
    if (sh.st.remaining_zeros != 0) {
        if (!second)
            for (int c = tid; c < cfg.nbins; c += kScanThreads) w.fill_at[c] = -1;
        else if (filled)
            list_zeros(sh, cfg, bufs);
    }
    const int i0 = i;
    ScanAlone by_itself{0, 0, 0};
    int alone = 0, streak = 0;     // spectra to do one by one before the next group
    int serial = 0, grow = 32;     // spectra of the next group if its averages are added one by one
    int failed = 0;
    bool redo = false;
    for (;;) {
        bool ask = false;
        while (i < n) {
            __syncthreads();
            const int rs = sh.st.rms_size, num = sh.st.num;
            // A group ends before the statistics' reset and before the histories are full; in the steady phase
            // its oldest entries are older than the group.
            int m = min(kScanThreads, n - i);
            if (num == 0) m = 0;
            else m = min(m, 10 * H - num);
            if (rs < H) m = flat ? min(m, H - 1 - rs) : 0;
            else m = min(m, H);
            // averages that are 0, not finite or tiny have no usable binade
            const RfiState& st = sh.st;
            const bool idle =
                !binade64(rs < H ? st.rms_acc : st.rms_run).ok || !binade64(rs < H ? st.mean_acc : st.mean_run).ok;
            if (idle) m = 0;
            if (alone > 0) {
                --alone;
                m = 0;
            }
            if (m > 0) {
                if (serial) m = min(m, serial);
                bool chain, unproven;
                const int f = scan_group(sh, cfg, bufs, w, rows, spec_elems, geo, i, m, filled,
                                         serial ? kOneByOne : kParallel, chain, unproven);
                i += f;
                if (chain) {  // past a half-way case; longer where they come again at once (x near a binade's end)
                    grow = f < 64 ? min(2 * grow, kSerial) : 32;
                    serial = grow;
                    continue;
                }
                serial = 0;
                if (f == m) {
                    streak = 0;
                    continue;
                }
                if (unproven && !second && n - i > kAloneMax) {
                    ++failed;
                    if ((failed == 1 && rs >= H) || failed > kAloneMax) {
                        ask = true;
                        break;
                    }
                }
                // groups that prove nothing are tried less and less often
                streak = f == 0 ? min(streak + 1, 6) : 0;
                alone = f == 0 ? (1 << streak) - 1 : 0;
            }
            if (may_leave && scan_leaves(sh, cfg, w, flat, i0, i, n, by_itself)) break;
            scan_one<P>(sh, cfg, bufs, w, rows + (long long)i * spec_elems, geo, i);
            filled |= sh.fill != 0 && sh.filled != 0;
            if (sh.rejected) ++by_itself.rejected;
            else if (idle) ++by_itself.idle;
            else ++by_itself.other;
            ++i;
        }
        if (!ask) break;
        redo = failed > kAloneMax;
        __syncthreads();
        if (tid == 0) *bufs.state = sh.st;  // before spectrum i; with a second pass the shared one moves on
        int at = i;
        while (at < n && sh.st.rms_size < H) {  // a second pass: approximately through the adaptive phase
            __syncthreads();
            const int rs = sh.st.rms_size;
            const int m = min(min(kScanThreads, n - at), max(H - 1 - rs, 1));
            bool c, u;
            scan_group(sh, cfg, bufs, w, rows, spec_elems, geo, at, m, false, kPredict, c, u);
            at += m;
            if (sh.st.rms_size >= H - 1 && tid == 0) {  // the histories are full
                sh.st.rms_size = sh.st.mean_size = H;
                sh.st.inv_mor = sh.st.rms_run / sh.st.mean_run;
            }
            __syncthreads();
        }
        if (at < n && scan_forecast(sh, cfg, bufs, w, at, n, at == i) > kForecastMax) redo = true;
        if (redo) break;
        alone = 1;
    }
    __syncthreads();
    if (tid == 0) {
        if (!redo) {
            *bufs.state = sh.st;
            w.hdr[kHdrEnd] = i;
            const int done = by_itself.all();
            const int hard = i < n || (done >= 32 && 10 * done >= 3 * (i - i0)) ? 1 : 0;
            if (w.hdr[kHdrHard] != hard) {
                w.hdr[kHdrHard] = hard;
                if (w.hard) *w.hard = hard;
            }
        }
        if (!second) {
            w.hdr[kHdrPos] = i;
            w.hdr[kHdrRedo] = redo ? 1 : 0;
            w.hdr[kHdrFilled] = filled ? 1 : 0;
        }
    }
}

// ---------------------------------------------------------------------------
// Clip, flatten, normalise and store every spectrum of a block
// (RFI_Clipper.cpp:313-342,441-532) with its exact state.
// ---------------------------------------------------------------------------
template <int P, int KM, bool PLAIN>
__device__ __forceinline__ void rfi_apply_body(const RfiConfig& cfg, const RfiBuffers& bufs, const RfiWork& w,
                                               float* __restrict__ row, const Geo& geo,
                                               unsigned char* __restrict__ flags, int i) {
    const int end = w.hdr[kHdrEnd];
    if (i >= end) return;
    const bool last = i == end - 1;
    constexpr int NW = P / 32;
    __shared__ float red[32 * 2];
    __shared__ float s_norm[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nbins = cfg.nbins, npol = PLAIN ? 1 : geo.npol;
    const bool flat = PLAIN || (cfg.deg == 0 && bufs.killed == nullptr);
    auto at = [&](int c) -> long long { return PLAIN ? c : geo.off(c); };
    const SpecOut o = w.out[i];
    const bool filling = w.hdr[kHdrZeros] != 0;
    const bool sclip = o.sclip != 0;
    const float bpf = __fmul_rn(cfg.scale, o.params0);
    const float bpd = __fadd_rn(bpf, o.dm);
    float s12[2] = {0.0f, 0.0f};
    float v[KM > 0 ? KM : 1];
    // the flattened channel
    auto flatten = [&](int c, float x) {
        const float bp = flat ? bpf : bp_value(cfg, bufs, o.params0, c);
        const bool clip = __fsub_rn(__fsub_rn(x, o.dm), bp) > o.margin;
        if (clip) {
            x = bufs.last_good[c];
            if (filling && w.fill_at[c] >= i) x = 0.0f;  // not filled yet at this spectrum
        }
        if (npol > 1 && (clip || sclip)) {  // every polarisation takes the last good value
            const long long off = geo.off(c);
            for (int p = 1; p < npol; ++p) row[off + (long long)p * geo.nchan] = sclip ? -0.2f : x;
        }
        if (flags) flags[c] = (clip ? 1 : 0) | (sclip ? 2 : 0);
        if (sclip) x = -0.2f;
        return __fsub_rn(x, flat ? bpd : __fadd_rn(bp, o.dm));
    };
    if constexpr (KM > 0) {
#pragma unroll
        for (int k = 0; k < KM; ++k) {
            const int c = tid + k * P;
            v[k] = c < nbins ? row[at(c)] : 0.0f;
        }
#pragma unroll
        for (int k = 0; k < KM; ++k) {
            const int c = tid + k * P;
            if (c < nbins) {
                v[k] = flatten(c, v[k]);
                s12[0] = __fadd_rn(s12[0], v[k]);
                s12[1] = __fadd_rn(s12[1], __fmul_rn(v[k], v[k]));
            }
        }
    } else {
        for (int c = tid; c < nbins; c += P) {
            const long long off = at(c);
            const float x = flatten(c, row[off]);
            row[off] = x;
            s12[0] = __fadd_rn(s12[0], x);
            s12[1] = __fadd_rn(s12[1], __fmul_rn(x, x));
        }
    }
    warp_tree_at<2>(s12, red, warp);
    __syncthreads();
    if (warp == 0) {
        float pf[2];
        lane_partials<1, NW>(red, pf, 0.0f);
        const float s1 = lane_tree<NW>(pf[0]);
        const float s2 = lane_tree<NW>(pf[1]);
        const float m = __fdiv_rn(s1, (float)nbins);
        const float ms = __fdiv_rn(s2, (float)nbins);
        float srms = __fsqrt_rn(__fsub_rn(ms, __fmul_rn(m, m)));
        if (srms == 0.0f) srms = 1.0f;
        if (lane == 0) {
            s_norm[0] = cfg.zero_dming == 1 ? m : o.mean_f;
            s_norm[1] = srms;
            if (last) bufs.state->rms_carry = (double)srms;
        }
    }
    __syncthreads();
    const float sub = s_norm[0], rms = s_norm[1], cr = cfg.cr;
    auto normalise = [&](float x) {
        if (sclip) return x;
        x = __fdiv_rn(__fsub_rn(x, sub), rms);
        return x > cr ? 0.0f : x;
    };
    if constexpr (KM > 0) {
#pragma unroll
        for (int k = 0; k < KM; ++k) {
            const int c = tid + k * P;
            if (c < nbins) row[at(c)] = normalise(v[k]);
        }
    } else {
        for (int c = tid; c < nbins; c += P) {
            const long long off = at(c);
            row[off] = normalise(row[off]);
        }
    }
}

// The running fraction of bad channels (RFI_Clipper.cpp:345-352,548-560), one
// FP32 add per spectrum in order, by one CTA beside those of the spectra.
template <int P>
__device__ __forceinline__ void rfi_fraction(const RfiConfig& cfg, const RfiBuffers& bufs, const RfiWork& w) {
    const int n = w.hdr[kHdrEnd];
    __shared__ __align__(16) float f[P];
    const int period = 10 * cfg.history, tid = threadIdx.x;
    // the statistics' reset is after the spectrum at which num is 0
    const int num = w.hdr[kHdrNum];
    long long reset = num == 0 ? 0 : period - num;
    float acc = bufs.state->frac_bad_channels;
    for (int b = 0; b < n; b += P) {
        const int cnt = min(P, n - b);
        f[tid] = tid < cnt ? __fdiv_rn((float)(cfg.nbins - w.rec[b + tid].total_good), (float)cfg.nbins) : 0.0f;
        __syncthreads();
        if (tid == 0) {
            for (int j = 0; j < cnt;) {
                const int stop = (int)min((long long)cnt, max(reset - b, (long long)j));
                for (; j + 4 <= stop && (j & 3) == 0; j += 4) {
                    const float4 y = *reinterpret_cast<const float4*>(f + j);
                    acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, y.x), y.y), y.z), y.w);
                }
                for (; j < stop; ++j) acc = __fadd_rn(acc, f[j]);
                if (j < cnt) {  // j is the spectrum of the reset
                    acc = 0.0f;
                    ++j;
                    reset += period;
                }
            }
        }
        __syncthreads();
    }
    if (tid == 0) bufs.state->frac_bad_channels = acc;
}
