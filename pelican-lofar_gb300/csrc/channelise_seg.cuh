// K1 fast path in two phases through shared memory (included by channelise.cu
// inside its anonymous namespace, after FirWindow): Stokes I of a
// dual-polarisation, 8-tap PPF with N = 16, 32 or 64 channels, integrated over
// 1, 2, 4 or 8 blocks, from voltages or LOFAR packets; or its complex spectra.
//
// A CTA of 128 threads takes one subband and a few streams of `range`
// consecutive blocks each, 8 blocks of every stream per phase:
//  FIR   a thread has two channels of one polarisation, adjacent (N = 16) or
//        16 apart (N = 32), or four 16 apart (N = 64): coefficients and the
//        8-block window stay in registers as packed pairs, raw samples are
//        read eight blocks ahead, and the FFT's stages of stride >= 16 run on
//        the sums before they go to shared memory.
//  FFT   a thread has 16 channels of one block and polarisation (N = 64: of
//        both, one after the other): the last four stages in registers with
//        constant twiddles and no shuffles, then |X|^2 or |Y|^2 back to shared
//        memory, where the window's blocks are added in order.
// Segments of 16 complex values are 144 bytes apart, so that 16-byte reads of
// neighbouring segments meet distinct banks.
//
// Every product, sum, butterfly and integration step is the one of
// channelise_kernel and chan_stokes_i_kernel: the results are bit-identical.
//
// Bound: the FP32 pipe (a packed operation takes it two cycles: 31 cycles per
// 32 complex samples, 16 of them the FIR) and issue (36 instructions, against
// 57 with the shuffled FFT of chan_stokes_i_kernel, whose four cross-lane
// stages multiply every lane by a twiddle).  int16 voltages: 244 subbands x 16
// channels x 65536 blocks 811 us against 1150, the FP32 pipe busy 51 % of the
// time, 15 warps per SM (128 registers; 168 or 96 are slower); 122 x 32 x
// 16384 253 against 331; 61 x 64 x 16391 268 against 358, two CTAs of 250
// registers per SM (three of 168 spill: 451).
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

// Where a FIR thread finds its C channels of a block: sample k of block b at
// base + b * block + k * step (in raw samples).
struct SegSource {
    const void* base;
    long long block;
    int step;
};

template <int N, bool I16, bool PKT, int C>
struct SegRaw {
    using S = typename RawSample<I16>::type;
    S x[C];
    __device__ __forceinline__ void load(const SegSource& s, int b) {
        const S* p = static_cast<const S*>(s.base) + b * (PKT ? s.block : (long long)N);
        if constexpr (N == 16 && I16 && !PKT) {
            const int2 q = __ldcs(reinterpret_cast<const int2*>(p));
            x[0] = q.x;
            x[1] = q.y;
        } else if constexpr (N == 16 && !PKT) {
            const float4 q = __ldcs(reinterpret_cast<const float4*>(p));
            x[0] = make_float2(q.x, q.y);
            x[1] = make_float2(q.z, q.w);
        } else {
#pragma unroll
            for (int k = 0; k < C; ++k) x[k] = __ldcs(p + (PKT ? k * s.step : k * 16));
        }
    }
    __device__ __forceinline__ float2 get(int k) const { return RawSample<I16>::f2(x[k]); }
};

// SPECTRA: J.out takes the complex spectra [block][sub][pol][N] instead (16 and
// 32 channels).  PKT: the voltages are LOFAR packets (int16, 16 samples each,
// [subband][time][pol] after a 16-byte header; AdapterTimeSeriesDataSet.cpp:
// 246-288), read in place.
template <int N, bool I16, bool PKT, bool SPECTRA>
__global__ void __launch_bounds__(kSegThreads, N == 64 ? 2 : 4)
chan_stokes_seg_kernel(const pv::ChanJob* __restrict__ jobs, const __grid_constant__ pv::ChanJob one, int njobs,
                       const pv::BeamStep* __restrict__ bs) {
    constexpr int M = N / 16, T = kFastTaps, H = T - 1;
    constexpr int C = N == 64 ? 4 : 2;            // channels per FIR thread
    constexpr int TPS = 2 * N / C;                // FIR threads per stream
    constexpr int STREAMS = kSegThreads / TPS;    // of a CTA
    constexpr int SEGS = 8 * STREAMS * M;         // segments of a phase and polarisation
    constexpr int PER = SEGS / (kSegThreads / 32);  // of a warp: 16, or 32 of one polarisation after the other
    constexpr int POL = SEGS * kSegWords + 4;     // words between the polarisations
    constexpr int PF = I16 ? 8 : 4;               // raw loads run PF blocks ahead
    constexpr int LOGN = M == 1 ? 4 : (M == 2 ? 5 : 6);
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
    const int stream = tid / TPS, r = tid % TPS, pol = r / (N / C), j = r % (N / C);
    const int c0 = N == 16 ? 2 * j : j;  // the thread's channels: c0, c0 + 1, or c0 + 16 k
    auto chan = [&](int k) { return N == 16 ? c0 + k : c0 + 16 * k; };
    const int B0 = first + stream * range, B1 = min(B0 + range, nblocks);
    const long long row = (long long)s * 2 + pol;
    SegSource in;
    if constexpr (PKT) {  // block b is packets b * M .. of the subband's stream, channel c its sample c % 16 of packet c / 16
        const long long pw = J.pkt_bytes / 4;
        const int ps = s / J.pkt_nsub, ls = s - ps * J.pkt_nsub;
        in.base = static_cast<const int*>(src) + ps * ((long long)nblocks * M) * pw + 4 + (ls * 16 + c0) * 2 + pol;
        in.block = M * pw;
        in.step = N == 16 ? 2 : (int)pw;
    } else {
        in.base = static_cast<const char*>(src) + (row * nblocks * N + c0) * (I16 ? 4 : 8);
        in.block = N;
        in.step = 16;
    }

    unsigned long long cf[T][C / 2];  // coefficient pairs
#pragma unroll
    for (int t = 0; t < T; ++t)
#pragma unroll
        for (int k = 0; k < C / 2; ++k)
            cf[t][k] = pk2(J.coeffs[t * N + chan(2 * k)], J.coeffs[t * N + chan(2 * k + 1)]);
    float2 tw[3];  // of the stages of stride 32 and 16
    if constexpr (M >= 2) tw[0] = J.twiddle[j];
    if constexpr (M == 4) {
        tw[1] = J.twiddle[j + 16];
        tw[2] = J.twiddle[2 * j];
    }
    // FIR window: slot b & 7 holds block b (B0 is a multiple of 8)
    unsigned long long re[T][C / 2], im[T][C / 2];
    auto set = [&](int q, const float2 (&v)[C]) {
#pragma unroll
        for (int k = 0; k < C / 2; ++k) {
            re[q][k] = pk2(v[2 * k].x, v[2 * k + 1].x);
            im[q][k] = pk2(v[2 * k].y, v[2 * k + 1].y);
        }
    };
    SegRaw<N, I16, PKT, C> cur[PF];
#pragma unroll
    for (int q = 1; q < T; ++q) {
        const int b = B0 - T + q;
        float2 v[C];
#pragma unroll
        for (int k = 0; k < C; ++k) v[k] = make_float2(0.0f, 0.0f);
        if (b >= 0 && b < nblocks) {
            cur[0].load(in, b);
#pragma unroll
            for (int k = 0; k < C; ++k) v[k] = cur[0].get(k);
        } else if (b < 0 && hin) {
#pragma unroll
            for (int k = 0; k < C; ++k) v[k] = hin[(row * H + (H + b)) * N + chan(k)];
        }
        set(q, v);
    }
#pragma unroll
    for (int q = 0; q < PF; ++q)
        if (B0 + q < B1) cur[q].load(in, B0 + q);

    const int last = min(range, nblocks - first);  // blocks of the CTA's longest stream
    for (int p0 = 0; p0 < last; p0 += 8) {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int b = B0 + p0 + q;
            float2 x[C];
#pragma unroll
            for (int k = 0; k < C; ++k) x[k] = cur[q % PF].get(k);
            if (b + PF < B1) cur[q % PF].load(in, b + PF);
            set(q, x);
            float2 y[C];
#pragma unroll
            for (int k = 0; k < C / 2; ++k) {
                unsigned long long ar = 0ull, ai = 0ull;  // +0.0f pairs; oldest tap first
#pragma unroll
                for (int t = 0; t < T; ++t) {
                    const int slot = (q + 1 + t) & (T - 1);
                    ar = fma2(re[slot][k], cf[t][k], ar);
                    ai = fma2(im[slot][k], cf[t][k], ai);
                }
                const float2 a = upk2(ar), i = upk2(ai);
                y[2 * k] = make_float2(a.x, i.x);
                y[2 * k + 1] = make_float2(a.y, i.y);
            }
            auto fly = [&](int u, int w, float2 t) {
                const float2 a = y[u], c = y[w];
                y[u] = make_float2(__fadd_rn(a.x, c.x), __fadd_rn(a.y, c.y));
                y[w] = dif_upper(a, c, t);
            };
            if constexpr (M == 2) {
                fly(0, 1, tw[0]);
            } else if constexpr (M == 4) {
                fly(0, 2, tw[0]);
                fly(1, 3, tw[1]);
                fly(0, 1, tw[2]);
                fly(2, 3, tw[2]);
            }
            float* seg = sm + pol * POL + (stream * 8 + q) * M * kSegWords + 2 * c0;
            if constexpr (N == 16) {
                *reinterpret_cast<float4*>(seg) = make_float4(y[0].x, y[0].y, y[1].x, y[1].y);
            } else {
#pragma unroll
                for (int m = 0; m < M; ++m) *reinterpret_cast<float2*>(seg + m * kSegWords) = y[m];
            }
        }
        __syncthreads();
        const int seg0 = (tid >> 5) * PER;  // the warp's first segment
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
#pragma unroll
        for (int h = 0; h < PER / 16; ++h) {
            float* seg = PER == 16 ? sm + (lane >> 4) * POL + (seg0 + (lane & 15)) * kSegWords
                                   : sm + h * POL + (seg0 + lane) * kSegWords;
            Fft16<!I16> f;
            f.load(seg);
            f.run();
            if constexpr (SPECTRA) {
                f.template store<M>(sm + (lane >> 4) * POL + (seg0 + (lane & 15)) / M * (M * kSegWords),
                                    (lane & 15) % M);
                __syncwarp();
                copy_spectra();
            } else {
                float p[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) p[i] = f.power(i);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    reinterpret_cast<float4*>(seg)[i] =
                        make_float4(p[4 * i], p[4 * i + 1], p[4 * i + 2], p[4 * i + 3]);
            }
        }
        __syncwarp();
        // the warp's blocks in windows; a thread takes four adjacent places of one
        for (int g = lane; !SPECTRA && g < 4 * PER / window; g += 32) {
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
            cur[0].load(in, nblocks - H + q);
#pragma unroll
            for (int k = 0; k < C; ++k) hout[(row * H + q) * N + chan(k)] = cur[0].get(k);
        }
    }
}
