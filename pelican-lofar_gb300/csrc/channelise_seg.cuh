// K1 fast path in two phases through shared memory (included by channelise.cu
// inside its anonymous namespace, after FirWindow): Stokes I of a
// dual-polarisation, 8-tap PPF with N = 16 or 32 channels, integrated over 1,
// 2, 4 or 8 blocks; or its complex spectra.
//
// A CTA of 128 threads takes one subband and 128/N streams of `range`
// consecutive blocks each, 8 blocks of every stream per phase:
//  FIR   a thread has two channels of one polarisation, adjacent (N = 16) or
//        16 apart (N = 32): coefficients and the 8-block window stay in
//        registers as packed pairs, raw samples are read eight blocks ahead,
//        and the FFT's stage of stride 16 runs on the sums before they go to
//        shared memory.
//  FFT   a thread has 16 channels of one block and polarisation: the last four
//        stages in registers with constant twiddles and no shuffles, then
//        |X|^2 or |Y|^2 back to shared memory, where the window's blocks are
//        added in order.
// Segments of 16 complex values are 144 bytes apart, so that 16-byte reads of
// neighbouring segments meet distinct banks.
//
// Every product, sum, butterfly and integration step is the one of
// channelise_kernel and chan_stokes_i_kernel: the results are bit-identical.
//
// Bound: the FP32 pipe (a packed operation takes it two cycles: 31 cycles per
// 32 complex samples, 16 of them the FIR) and issue (36 instructions, against
// 57 with the shuffled FFT of chan_stokes_i_kernel, whose four cross-lane
// stages multiply every lane by a twiddle).  244 subbands x 16 channels x
// 65536 blocks: 831 us against 1151, the FP32 pipe busy 51 % of the time, 15
// warps per SM.  122 x 32 x 16384: 256 against 330.  For 64 channels the same
// split (four channels per thread, or a 32-point FFT) needs more registers
// than three CTAs per SM have and was slower (404 against 358 us).
constexpr int kSegThreads = 128;
constexpr int kSegWords = 36;  // 16 complex values and 16 bytes

__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// a - b per half (a + (-1) * b rounds once: the same)
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
    return fma2(b, 0xbf800000bf800000ull, a);
}

// 16-point decimation-in-frequency FFT, output in bit-reversed places.  The
// twiddles exp(-2 pi i e / 16) to FP32 are the table's values.  Products with 1
// and -i are exact and left out, but for FULL (float voltages, which may be
// infinite: the product's infinity times 0 is then part of the result).
template <bool FULL>
struct Fft16 {
    unsigned long long v[16];
    template <int H>
    __device__ __forceinline__ void stage() {
#pragma unroll
        for (int lo = 0; lo < 16; ++lo) {
            if (lo & H) continue;
            const int e = (lo & (H - 1)) * (8 / H);
            const unsigned long long a = v[lo], b = v[lo + H];
            v[lo] = add2(a, b);
            const unsigned long long d = sub2(a, b);
            if (e == 0 && !(FULL && H >= 4)) {
                v[lo + H] = d;
            } else if (e == 4 && !(FULL && H >= 4)) {
                const float2 z = times_minus_i(upk2(d));
                v[lo + H] = pk2(z.x, z.y);
            } else {
                constexpr float c1 = 0x1.d906bcp-1f, c2 = 0x1.6a09e6p-1f, c3 = 0x1.87de2ap-2f;
                const float2 w = e == 0   ? make_float2(1.0f, -0.0f)
                                 : e == 4 ? make_float2(0.0f, -1.0f)
                                 : e == 1 ? make_float2(c1, -c3)
                                 : e == 2 ? make_float2(c2, -c2)
                                 : e == 3 ? make_float2(c3, -c1)
                                 : e == 5 ? make_float2(-c3, -c1)
                                 : e == 6 ? make_float2(-c2, -c2)
                                          : make_float2(-c1, -c3);
                const float2 z = twiddle_mul(upk2(d), w);
                v[lo + H] = pk2(z.x, z.y);
            }
        }
    }
    __device__ __forceinline__ void load(const float* seg) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(seg + 4 * k);
            v[2 * k] = x.x;
            v[2 * k + 1] = x.y;
        }
    }
    // Channels in order: row of 16 * M, this being segment k of M.
    template <int M>
    __device__ __forceinline__ void store(float* row, int k) const {
        if constexpr (M == 1) {
#pragma unroll
            for (int c = 0; c < 16; c += 2) {
                ulonglong2 x;
                x.x = v[brev4(c)];
                x.y = v[brev4(c + 1)];
                *reinterpret_cast<ulonglong2*>(row + 2 * c) = x;
            }
        } else {
            __syncwarp();  // the row's other segment has been read
#pragma unroll
            for (int c = 0; c < 16; ++c)
                *reinterpret_cast<unsigned long long*>(row + 2 * (M * c + k)) = v[brev4(c)];
        }
    }
    static constexpr __device__ int brev4(int c) {
        return (c & 1) << 3 | (c & 2) << 1 | (c & 4) >> 1 | (c & 8) >> 3;
    }
    __device__ __forceinline__ void run() {
        stage<8>();
        stage<4>();
        stage<2>();
        stage<1>();
    }
    __device__ __forceinline__ float power(int i) const {
        const float2 z = upk2(v[i]);
        return __fadd_rn(__fmul_rn(z.x, z.x), __fmul_rn(z.y, z.y));
    }
};

// The two raw samples of a FIR thread in one block: channels 2j, 2j + 1 (N =
// 16) or j, j + 16.
template <int N, bool I16>
struct SegRaw {
    using S = typename RawSample<I16>::type;
    S x[2];
    __device__ __forceinline__ void load(const void* row, long long i) {
        const S* p = static_cast<const S*>(row) + i;
        if constexpr (N == 16 && I16) {
            const int2 q = __ldcs(reinterpret_cast<const int2*>(p));
            x[0] = q.x;
            x[1] = q.y;
        } else if constexpr (N == 16) {
            const float4 q = __ldcs(reinterpret_cast<const float4*>(p));
            x[0] = make_float2(q.x, q.y);
            x[1] = make_float2(q.z, q.w);
        } else {
            x[0] = __ldcs(p);
            x[1] = __ldcs(p + 16);
        }
    }
    __device__ __forceinline__ float2 get(int k) const { return RawSample<I16>::f2(x[k]); }
};

// SPECTRA: J.out takes the complex spectra [block][sub][pol][N] instead.
template <int N, bool I16, bool SPECTRA>
__global__ void __launch_bounds__(kSegThreads, 4)
chan_stokes_seg_kernel(const pv::ChanJob* __restrict__ jobs, const __grid_constant__ pv::ChanJob one, int njobs,
                       const pv::BeamStep* __restrict__ bs) {
    constexpr int M = N / 16, T = kFastTaps, H = T - 1;
    constexpr int STREAMS = kSegThreads / N;  // of a CTA, N FIR threads each
    constexpr int SEGS = 8 * STREAMS * M;     // segments of a phase and polarisation
    constexpr int POL = SEGS * kSegWords + 4; // words between the polarisations
    constexpr int PF = I16 ? 8 : 4;           // raw loads run PF blocks ahead
    constexpr int LOGN = M == 1 ? 4 : 5;
    static_assert(SEGS == 16 * (kSegThreads / 32), "a warp has 16 segments of both polarisations");
    __shared__ __align__(16) float sm[2 * POL];
    int lo = 0, hi = njobs - 1;  // the job whose CTAs include this one
    while (jobs && lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (jobs[mid].unit_begin <= (long long)blockIdx.x) lo = mid;
        else hi = mid - 1;
    }
    const pv::ChanJob& J = jobs ? jobs[lo] : one;
    int par = 0;  // step parity of this beam: input buffer and history double buffer
    if (bs) {
        const pv::BeamStep& B = bs[J.beam];
        if (!B.active) return;
        par = (int)((B.written - B.base) & 1);
    }
    const int nblocks = J.nblocks, window = J.window, nu = J.nu, nsub = J.nsub, range = J.range;
    const long long local = (long long)blockIdx.x - J.unit_begin;
    const int s = (int)(local / J.nranges);
    const int first = (int)(local - (long long)s * J.nranges) * STREAMS * range;  // the CTA's first block
    const float2* hin = J.hist[par];
    float2* hout = J.hist[par ^ 1];
    const void* src = (par && J.in_odd) ? J.in_odd : J.in;

    const int tid = threadIdx.x, lane = tid & 31;
    const int stream = tid / N, r = tid % N, pol = r / (N / 2), j = r % (N / 2);
    const int c0 = N == 16 ? 2 * j : j, c1 = N == 16 ? c0 + 1 : c0 + 16;  // the thread's channels
    const int B0 = first + stream * range, B1 = min(B0 + range, nblocks);
    const long long row = (long long)s * 2 + pol;
    const void* in = static_cast<const char*>(src) + (row * nblocks * N + c0) * (I16 ? 4 : 8);

    unsigned long long cf[T];  // coefficient pairs
#pragma unroll
    for (int t = 0; t < T; ++t) cf[t] = pk2(J.coeffs[t * N + c0], J.coeffs[t * N + c1]);
    const float2 tw = M == 2 ? J.twiddle[j] : make_float2(1.0f, 0.0f);  // of the stage of stride 16
    // FIR window: slot b & 7 holds block b (B0 is a multiple of 8)
    unsigned long long re[T], im[T];
    auto set = [&](int q, float2 v, float2 w) {
        re[q] = pk2(v.x, w.x);
        im[q] = pk2(v.y, w.y);
    };
    SegRaw<N, I16> cur[PF];
#pragma unroll
    for (int q = 1; q < T; ++q) {
        const int b = B0 - T + q;
        float2 v = make_float2(0.0f, 0.0f), w = v;
        if (b >= 0 && b < nblocks) {
            cur[0].load(in, (long long)b * N);
            v = cur[0].get(0);
            w = cur[0].get(1);
        } else if (b < 0 && hin) {
            v = hin[(row * H + (H + b)) * N + c0];
            w = hin[(row * H + (H + b)) * N + c1];
        }
        set(q, v, w);
    }
#pragma unroll
    for (int q = 0; q < PF; ++q)
        if (B0 + q < B1) cur[q].load(in, (long long)(B0 + q) * N);

    const int last = min(range, nblocks - first);  // blocks of the CTA's longest stream
    for (int p0 = 0; p0 < last; p0 += 8) {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int b = B0 + p0 + q;
            const float2 x0 = cur[q % PF].get(0), x1 = cur[q % PF].get(1);
            if (b + PF < B1) cur[q % PF].load(in, (long long)(b + PF) * N);
            set(q, x0, x1);
            unsigned long long ar = 0ull, ai = 0ull;  // +0.0f pairs; oldest tap first
#pragma unroll
            for (int t = 0; t < T; ++t) {
                const int slot = (q + 1 + t) & (T - 1);
                ar = fma2(re[slot], cf[t], ar);
                ai = fma2(im[slot], cf[t], ai);
            }
            const float2 a = upk2(ar), i = upk2(ai);
            float2 y0 = make_float2(a.x, i.x), y1 = make_float2(a.y, i.y);
            float* seg = sm + pol * POL + (stream * 8 + q) * M * kSegWords + 2 * c0;
            if constexpr (N == 16) {
                *reinterpret_cast<float4*>(seg) = make_float4(y0.x, y0.y, y1.x, y1.y);
            } else {
                *reinterpret_cast<float2*>(seg) = make_float2(__fadd_rn(y0.x, y1.x), __fadd_rn(y0.y, y1.y));
                *reinterpret_cast<float2*>(seg + kSegWords) = dif_upper(y0, y1, tw);
            }
        }
        __syncthreads();
        const int seg0 = (tid >> 5) * 16;  // the warp's first segment
        // the warp's rows of N spectrum values, 16 bytes per lane
        auto copy_spectra = [&]() {
#pragma unroll
            for (int it = 0; it < 8; ++it) {
                const int sl = it * 4 + (lane >> 3), q = sl >> 4, sg = seg0 + (sl & 15);
                const int lb = sg / M, k = sg % M, at = k * 32 + (lane & 7) * 4;  // words into the row
                const int b = first + (lb >> 3) * range + p0 + (lb & 7);
                const float4 x = *reinterpret_cast<const float4*>(sm + q * POL + lb * M * kSegWords + at);
                if (b < nblocks)
                    *reinterpret_cast<float4*>(J.out + (((long long)b * nsub + s) * 2 + q) * 2 * N + at) = x;
            }
        };
        {
            float* seg = sm + (lane >> 4) * POL + (seg0 + (lane & 15)) * kSegWords;
            Fft16<!I16> f;
            f.load(seg);
            f.run();
            if constexpr (SPECTRA) {
                f.template store<M>(sm + (lane >> 4) * POL + (seg0 + (lane & 15)) / M * (M * kSegWords), (lane & 15) % M);
                __syncwarp();
                copy_spectra();
                __syncthreads();
                continue;
            }
            float p[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) p[i] = f.power(i);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                reinterpret_cast<float4*>(seg)[i] = make_float4(p[4 * i], p[4 * i + 1], p[4 * i + 2], p[4 * i + 3]);
        }
        __syncwarp();
        // the warp's 16 / M blocks in windows; a thread takes four adjacent places of one
        for (int g = lane; g < 64 / window; g += 32) {
            const int wi = g / (N / 4), qd = g % (N / 4);
            const int lb = seg0 / M + wi * window;
            const int b = first + (lb >> 3) * range + p0 + (lb & 7);  // the window's first block
            const int u = b / window;
            const float* px = sm + (lb * M + (qd >> 2)) * kSegWords + 4 * (qd & 3);
            float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            for (int t = 0; t < window; ++t, px += M * kSegWords) {
                const float4 x = *reinterpret_cast<const float4*>(px), y = *reinterpret_cast<const float4*>(px + POL);
                a[0] = __fadd_rn(a[0], __fadd_rn(x.x, y.x));
                a[1] = __fadd_rn(a[1], __fadd_rn(x.y, y.y));
                a[2] = __fadd_rn(a[2], __fadd_rn(x.z, y.z));
                a[3] = __fadd_rn(a[3], __fadd_rn(x.w, y.w));
            }
            if (u < nu) {
                float* o = J.out + ((long long)u * nsub + s) * N;
#pragma unroll
                for (int k = 0; k < 4; ++k) o[__brev((unsigned)(4 * qd + k)) >> (32 - LOGN)] = a[k];
            }
        }
        __syncthreads();
    }
    // the stream that ends the chunk carries its last 7 blocks to the next call
    if (hout && B0 < nblocks && B1 == nblocks) {
#pragma unroll
        for (int q = 0; q < H; ++q) {
            cur[0].load(in, (long long)(nblocks - H + q) * N);
            hout[(row * H + q) * N + c0] = cur[0].get(0);
            hout[(row * H + q) * N + c1] = cur[0].get(1);
        }
    }
}
