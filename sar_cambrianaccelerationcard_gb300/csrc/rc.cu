// rc.cu -- range compression and range upsampling on sm_103a.
//
// Implements code/SAR_BP/matlab/BPA_SAR.m:93-111 (matched filter
// ifft(fft(s).*conj(fft(h))) followed by 8x upsampling through mid-spectrum
// zero insertion) as two kernels:
//
//   rc_forward  (one CTA per pulse): zero-padded echo row -> shared memory ->
//               forward FFT -> multiply by the filter spectrum
//               G[k] = conj(H[k]) e^{-j2pi k D/N} / N -> spectrum scratch.
//               Also emits the per-pulse bound sum_k |Y[k]| (>= max |output|)
//               from which the FP16 storage scale is derived.
//   rc_inverse  (one or two upsampling phases r per CTA): the L*N-point
//               inverse of the zero-inserted spectrum evaluated at bins
//               b = L*i + r equals the N-point inverse of Y[k]*e^{+j2pi kappa r/(LN)}
//               (kappa = signed frequency), so a phase is one N-point inverse
//               FFT whose outputs are every L-th bin of the row.
//
// The FFT is a Stockham autosort transform with radix-32/16/8 stages (one
// radix-4 or radix-2 stage for the remaining factor), in place in shared
// memory (XOR-swizzled so every stage's accesses are free of bank conflicts)
// with a barrier between each stage's loads and stores.  The upsampling ramp
// is a power of E = e^{j 2 pi / (L N)}, from a two-level table in global memory,
// E^m = T_hi[m >> 8] * T_lo[m & 255] (computed in double precision on the host);
// the transform twiddles are powers of W = E^L from a second two-level table
// derived from it into shared memory at kernel start, so no FFT stage touches
// global memory.
//
// N = 32768 (shared memory holds 16384 points) is split by one radix-2 stage:
// the forward runs two CTAs per pulse on the half-size inputs x[n] + x[n+M] and
// (x[n] - x[n+M]) W_N^n, giving the even and odd spectral bins; the inverse folds
// the ramped spectrum modulo M = 16384 while loading it, Y[k] E^{kappa r} +
// Y[k+M] E^{kappa' r} for r < 2 L, which is upsampling by 2 L of an M-point
// transform and needs no exchange between CTAs.  (A 2-CTA cluster per phase that
// combined its halves through distributed shared memory: 768 pulses 1.61 ms,
// folded 1.30, 1.23 with the table and layout changes of fft_smem.cuh.)  Folding
// smaller transforms does not pay: 16384 points as 2 x 8192, two CTAs per SM,
// 3.39 against 2.87 ms for 4096 pulses, for a store then touches 32 lines and
// every fold adds a complex product per point.
//
// What bounds the inverse: the load/store path (shared wavefronts of the two
// passes, 48% of them at 8192 points the strided stores; 74% busy there) and, at
// 16384 points, that one 131 KB CTA per SM runs its load, butterfly and store
// phases one after the other.
#include "fft_smem.cuh"

namespace sarbp {
namespace {

template <int T>
__device__ __forceinline__ float block_sum(float v, float *red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) red[w] = v;
    __syncthreads();
    float t = 0.f;
    if (threadIdx.x < 32) {
        t = (l < T / 32) ? red[l] : 0.f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    }
    return t;  // valid in thread 0
}

// The FP16 storage scale from the bound on |output|: a power of two, so that
// stored magnitudes stay <= 2^14.
__device__ __forceinline__ float storage_scale(float bound) {
    return bound > 0.f && isfinite(bound) ? exp2f(ceilf(log2f(bound) - 14.f)) : 1.f;
}

// SCALE: also the per-pulse bound sum_k |Y[k]| and the FP16 storage scale
// from it (complex16 rows only).
template <int N, int T, bool SCALE>
__global__ void __launch_bounds__(T, (fft_min_blocks<N, T>())) rc_forward_kernel(int ns, int L, const float2 *__restrict__ echo,
                                                       const float2 *__restrict__ filt,
                                                       const float2 *__restrict__ etab,
                                                       float2 *__restrict__ spec,
                                                       float *__restrict__ scale) {
    extern __shared__ float2 sm[];
    __shared__ float red[32];
    const int p = blockIdx.x;
    // first-stage inputs straight from the echo row (zero padding past ns),
    // issued before the table loads so both latencies overlap
    using F = FirstIn<N, T>;
    float2 v[F::PER][F::R];
    const float2 *row = echo + (size_t)p * ns;
#pragma unroll
    for (int b = 0; b < F::PER; ++b)
#pragma unroll
        for (int r = 0; r < F::R; ++r) {
            const int i = F::point(b, r);
            v[b][r] = (F::live(b) && i < ns) ? __ldg(&row[i]) : make_float2(0.f, 0.f);
        }
    const Etab E = load_etab<N, T>(sm, etab, L);  // the first stage's barrier publishes the W tables
    float2 *out = spec + (size_t)p * N;
    float acc = 0.f;
    fft_io<N, T, false>(sm, E, v, [&](int k, float2 x) {
        const float2 y = cmul(x, __ldg(&filt[k]));
        out[k] = y;
        if constexpr (SCALE) acc += sqrtf(fmaf(y.x, y.x, y.y * y.y));
    });
    if constexpr (!SCALE) return;
    const float bound = block_sum<T>(acc, red);
    if (threadIdx.x == 0) scale[p] = storage_scale(bound);
}

// Points between the arrays of a CTA's G phases: in the last stage a half-warp loads
// 16 / G points of each, from disjoint banks.
template <int G>
constexpr int group_pad = G > 1 ? 16 / G : 0;
// The ramp factors into two levels (per thread, per phase) where every first-stage
// point of a thread is congruent to its index modulo T: all but the transforms of
// 64 to 256 points, which read E^{kappa r} point by point.
template <int N, int M, int T>
constexpr bool two_level_ramp = (N / 2) % T == 0 && N / T <= kRampMax && FirstIn<M, T>::NB % T == 0;
// STAGED copies the E table to shared memory, a spare slot per 8 entries.  At 16x
// upsampling the strides of W^m = E^{16 m} and of the point-by-point ramp put
// every lane on a line of its own, and gathers from global memory bound the
// transforms of 128 and 256 points: 8192 pulses, complex64 / FP16 rows, 253 / 226 us
// from global, 210 / 214 staged (128 points), 348 / 289 and 295 / 249 (256).  64
// points have too few gathers to pay for the copy (175 / 191 against 182 / 201); at 8x
// reading from global memory is the faster one (256 points: 140 -> 134 us).
template <int N>
constexpr bool staged_at_16x = N == 128 || N == 256;
constexpr int kStagedTable = 256 + 16;  // entries at 256 points and 16x
__device__ __forceinline__ int tslot(int i) { return i + (i >> 3); }
constexpr int kStagedSlots = kStagedTable + kStagedTable / 8;

// N-bin spectrum, M-point transforms (M divides N), G of them per CTA: CTA (p, r0)
// gives the bins (L N / M) i + r of the phases r = G r0 .. G r0 + G - 1, r < L N / M,
// each the M-point inverse of the spectrum times its ramp folded modulo M.  The
// G phases' bins are neighbours in the row, and the last stage's lanes store
// them together.
template <int N, int M, int T, int G, int STORE, bool STAGED>
__global__ void __launch_bounds__(G *T, (fft_min_blocks<G * M, G * T>()))
    rc_inverse_kernel(int L, int nbins, const float2 *__restrict__ spec, const float2 *__restrict__ etab,
                      const float *__restrict__ bound2, float *__restrict__ scale, void *__restrict__ out) {
    extern __shared__ float2 sm[];
    constexpr int FOLD = N / M, CS = M + group_pad<G>;
    const int LF = L * FOLD, per = LF / G;
    const int group = G > 1 ? threadIdx.x / T : 0, tid = G > 1 ? threadIdx.x % T : threadIdx.x;
    const int p = blockIdx.x / per;
    const int r0 = (blockIdx.x - p * per) * G, r = r0 + group;
    const float2 *in = spec + (size_t)p * N;
    const int LN = L * N;
    // first-stage inputs straight from the spectrum, issued before the tables
    using F = FirstIn<M, T>;
    float2 v[F::PER][F::R];
#pragma unroll
    for (int b = 0; b < F::PER; ++b)
#pragma unroll
        for (int q = 0; q < F::R; ++q)
            v[b][q] = F::live(b, tid) ? __ldg(&in[F::point(b, q, tid)]) : make_float2(0.f, 0.f);
    float2 *tables = sm + G * CS;
    constexpr bool kTwoLevel = two_level_ramp<N, M, T>;
    static_assert(kTwoLevel ? !STAGED : FOLD == 1 && G == 1 && N <= 256, "point-by-point ramp: small single transforms");
    float2 *et = tables + kWlo + kWhiMax + kRampMax;
    auto staged_e = [&](int m) { return cmul(et[tslot(256 + (m >> 8))], et[tslot(m & 255)]); };
    if (STAGED) {
        for (int i = threadIdx.x; i < 256 + LN / 256; i += T) et[tslot(i)] = __ldg(&etab[i]);
        __syncthreads();
        fill_w<M, T>(tables, L, staged_e);
    }
    const Etab E = STAGED ? Etab{etab, tables, tables + kWlo} : load_etab_at<M, T, G * T>(tables, etab, LF);
    // Ramp E^{kappa r}, kappa the signed frequency (MATLAB split floor((N+1)/2)
    // = N/2 for even N).  With k = tid + T i (every first-stage point of a
    // thread is congruent to tid mod T when M / R is a multiple of T) and N/2 a
    // multiple of T it factors into a per-thread E^{tid r} and a per-phase table
    // over i that also carries the E^{-N r} of the negative half.
    float2 *rt = tables + kWlo + kWhiMax + group * kRampMax;
    float2 base = make_float2(1.f, 0.f);
    if (kTwoLevel && r != 0) {
        if (tid < N / T) {
            const int i = tid;
            float2 w = E((T * i * r) & (LN - 1));
            if (T * i >= N / 2) w = cmul(w, E((LN - N * r) & (LN - 1)));
            rt[i] = w;
        }
        base = E((tid * r) & (LN - 1));
    }
    if (kTwoLevel) __syncthreads();  // the ramp table; the W tables are read behind the first stage's barrier
    if (r != 0) {
#pragma unroll
        for (int b = 0; b < F::PER; ++b)
#pragma unroll
            for (int q = 0; q < F::R; ++q) {
                const int k = F::point(b, q, tid);
                if (kTwoLevel) {
                    v[b][q] = cmul(v[b][q], rt[k / T]);
                } else {
                    const int m = ((k < N / 2 ? k : k - N) * r) & (LN - 1);  // LN is a power of two
                    v[b][q] = cmul(v[b][q], STAGED ? staged_e(m) : E(m));
                }
            }
#pragma unroll
        for (int f = 1; f < FOLD; ++f)
#pragma unroll
            for (int b = 0; b < F::PER; ++b)
#pragma unroll
                for (int q = 0; q < F::R; ++q) {
                    const int k = F::point(b, q, tid) + f * M;
                    v[b][q] = cfma(__ldg(&in[k]), rt[k / T], v[b][q]);
                }
        if (kTwoLevel) {
#pragma unroll
            for (int b = 0; b < F::PER; ++b)
#pragma unroll
                for (int q = 0; q < F::R; ++q) v[b][q] = cmul(v[b][q], base);
        }
    } else {
#pragma unroll
        for (int f = 1; f < FOLD; ++f)
#pragma unroll
            for (int b = 0; b < F::PER; ++b)
#pragma unroll
                for (int q = 0; q < F::R; ++q) v[b][q] = cadd(v[b][q], __ldg(&in[F::point(b, q, tid) + f * M]));
    }
    // outputs x of phase r0 + g: bin LF x + r0 + g, inside the row for x < live
    const int last = r0 + (G > 1 ? (int)(threadIdx.x % G) : 0);
    const int live = (nbins - last + LF - 1) / LF;
    auto run = [&](auto store) {
        if constexpr (G > 1)
            fft_io_group<M, T, true, G, CS>(sm, E, v, [&](int, int x, float2 y) { store(x, y); });
        else
            fft_io<M, T, true>(sm, E, v, store);
    };
    if (STORE == SARBP_STORE_C64) {
        float2 *o = reinterpret_cast<float2 *>(out) + (size_t)p * nbins + last;
        run([&](int x, float2 y) {
            if (x < live) o[(size_t)LF * x] = y;
        });
    } else {
        float sc;
        if (bound2) {  // the forward ran as two CTAs: combine their parts of the bound
            sc = storage_scale(__ldg(&bound2[2 * p]) + __ldg(&bound2[2 * p + 1]));
            if (r0 == 0 && threadIdx.x == 0) scale[p] = sc;
        } else {
            sc = scale[p];
        }
        const float inv = 1.f / sc;  // exact: scale is a power of two
        __half2 *o = reinterpret_cast<__half2 *>(out) + (size_t)p * nbins + last;
        run([&](int x, float2 y) {
            if (x < live) o[(size_t)LF * x] = __floats2half2_rn(y.x * inv, y.y * inv);
        });
    }
}

// N = 2M forward: CTA pair (h = 0, 1) per pulse; h = 0 yields X[2k], h = 1 X[2k+1].
// bound2[2p + h] receives the CTA's part of sum_k |Y[k]|.
template <int M, int T>
__global__ void __launch_bounds__(T) rc_forward2_kernel(int ns, int L, const float2 *__restrict__ echo,
                                                        const float2 *__restrict__ filt,
                                                        const float2 *__restrict__ etab,
                                                        float2 *__restrict__ spec, float *__restrict__ bound2) {
    extern __shared__ float2 sm[];
    __shared__ float red[32];
    const int h = blockIdx.x & 1, p = blockIdx.x >> 1;
    const Etab E = load_etab<M, T>(sm, etab, 2 * L);  // E tables published by its barrier
    const float2 *row = echo + (size_t)p * ns;
    using F = FirstIn<M, T>;
    float2 v[F::PER][F::R];
#pragma unroll
    for (int b = 0; b < F::PER; ++b)
#pragma unroll
        for (int q = 0; q < F::R; ++q) {
            const int i = F::point(b, q);
            const float2 x0 = (F::live(b) && i < ns) ? __ldg(&row[i]) : make_float2(0.f, 0.f);
            const float2 x1 = (F::live(b) && i + M < ns) ? __ldg(&row[i + M]) : make_float2(0.f, 0.f);
            if (h == 0) {
                v[b][q] = cadd(x0, x1);
            } else {
                float2 w = E(L * i);  // W_N^i = conj(E^{L i})
                w.y = -w.y;
                v[b][q] = cmul(csub(x0, x1), w);
            }
        }
    float2 *out = spec + (size_t)p * (2 * M);
    float acc = 0.f;
    fft_io<M, T, false>(sm, E, v, [&](int k, float2 x) {
        const int idx = 2 * k + h;
        const float2 y = cmul(x, __ldg(&filt[idx]));
        out[idx] = y;
        acc += sqrtf(fmaf(y.x, y.x, y.y * y.y));
    });
    const float bound = block_sum<T>(acc, red);
    if (threadIdx.x == 0) bound2[2 * p + h] = bound;
}

constexpr int kInvPoints = 16384;  // largest inverse transform of one CTA
// CTA sizes (threads) per transform length, measured on GB300 (ms for 4096
// pulses, forward + eight inverse transforms each).  8192 points: 1.886 at
// 1024 threads (one CTA per SM: its barriers are overlapped by nothing), 1.295
// at 512 (two CTAs per SM), 1.123 at 256 (two per SM, 32 points per thread:
// radix-32 stages 32-32-8).  16384 points (128 KB, one CTA per SM whatever the
// size): 3.077 at 1024 (16-16-16-4), 2.986 at 512 (32-32-16).  The 16384-point
// halves of the 32768-point split path: 4.35 at 1024, 4.29 at 512 (radix-16),
// 4.17 at 512 with radix-32 stages (2048 pulses).  4096 points: 16 per thread
// (256 threads, 16-16-16) against 8 (512, 8-8-8-8): 512 pulses 95 -> 73 us.
template <int N>
constexpr int threads_for() {
    return N >= 16384 ? 512 : (N >= 2048 ? 256 : (N >= 512 ? N / 8 : 64));
}

// Phases per CTA of the inverse, measured (2048 pulses, L = 8, forward and
// inverse, us at 1 / 2 / 4): 4096 points 301 / 246 / 254 (FP16 rows 270 / 261 / 262),
// 8192 points 603 / 572 (FP16 rows 630 / 644), 2048 points 167 / 171 / 171.  A
// phase's bins lie L bins apart, so a warp's store touches 16 lines of 128 bytes;
// two phases' neighbouring bins halve that, which pays while the shared-memory and
// store path bounds the kernel and the larger CTA costs no residency (two
// 16384-point phases do not fit one SM).
template <int N, int STORE>
constexpr int phases_for() {
    return N == 4096 || (N == 8192 && STORE == SARBP_STORE_C64) ? 2 : 1;
}
// Whether a launch takes pairs where the length has them (same bits either way).  Rows
// divide evenly: L % 2 == 0.  While single phases have an SM each, pairs only make
// each CTA longer (us, single / pairs: 16 pulses of 4096 points at 4x 15.9 / 18.0,
// FP16 19.0 / 21.1; of 8192 points 22.0 / 23.9).  At 8192 points a pair takes an SM
// alone, single phases share one three ways, so at 2x and 4x, with less of the store
// path to save, a second wave of pairs has to be half full (2x, 200 pulses 31.3 / 33.4,
// 304 pulses 35.4 / 33.4), and at 2x beyond two waves single phases win (4096 pulses
// 318 / 344; at 4x 691 / 643).
template <int N>
bool take_pairs(const RcPlan &p) {
    const long long pairs = (long long)p.np * p.L / 2, sms = current_sms();
    if (p.L % 2 || 2 * pairs <= sms) return false;
    if (N < 8192 || p.L > 4) return true;
    if (pairs > sms && 2 * pairs <= 3 * sms) return false;
    return p.L == 4 || pairs <= 2 * sms;
}
// With t_prepare set the launchers below configure their kernel and return
// without launching it (prepare_rc_kernels).
thread_local bool t_prepare = false;

template <int N>
cudaError_t fwd_n(const RcPlan &p, const float2 *echo, const float2 *filt, const float2 *etab,
                  float2 *spec, float *scale, cudaStream_t s) {
    constexpr int T = threads_for<N>();
    const size_t smem = sizeof(float2) * N + kTabSmem;
    // the FP16 scale only for complex16 rows (a scale array is ignored otherwise)
    auto k = p.storage == SARBP_STORE_C32H ? rc_forward_kernel<N, T, true> : rc_forward_kernel<N, T, false>;
    cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void *>(k));
    if (e != cudaSuccess || t_prepare) return e;
    k<<<p.np, T, smem, s>>>(p.ns, p.L, echo, filt, etab, spec, scale);
    return cudaGetLastError();
}

template <int N, int STORE, int G, bool STAGED = false>
cudaError_t inv_g(const RcPlan &p, const float2 *spec, const float2 *etab, const float *bound2, float *scale,
                  void *out, cudaStream_t s) {
    constexpr int M = N < kInvPoints ? N : kInvPoints, T = threads_for<M>();
    constexpr int slots = G * (M + group_pad<G>) + (G - 1) * kRampMax + (STAGED ? kStagedSlots : 0);
    const size_t smem = sizeof(float2) * slots + kTabSmem;
    auto k = rc_inverse_kernel<N, M, T, G, STORE, STAGED>;
    cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void *>(k));
    if (e != cudaSuccess || t_prepare) return e;
    k<<<p.np * (p.L * (N / M) / G), G * T, smem, s>>>(p.L, p.nbins, spec, etab, bound2, scale, out);
    return cudaGetLastError();
}
template <int N, int STORE>
cudaError_t inv_s(const RcPlan &p, const float2 *spec, const float2 *etab, const float *bound2, float *scale,
                  void *out, cudaStream_t s) {
    if constexpr (staged_at_16x<N>) {
        if (p.L == 16) return inv_g<N, STORE, 1, true>(p, spec, etab, bound2, scale, out, s);
    }
    if constexpr (phases_for<N, STORE>() == 2) {
        if (t_prepare) {  // both layouts: a later launch may have any number of pulses
            const cudaError_t e = inv_g<N, STORE, 2>(p, spec, etab, bound2, scale, out, s);
            if (e != cudaSuccess) return e;
        } else if (take_pairs<N>(p)) {
            return inv_g<N, STORE, 2>(p, spec, etab, bound2, scale, out, s);
        }
    }
    return inv_g<N, STORE, 1>(p, spec, etab, bound2, scale, out, s);
}
template <int N>
cudaError_t inv_n(const RcPlan &p, const float2 *spec, const float2 *etab, const float *bound2, float *scale,
                  void *out, cudaStream_t s) {
    return p.storage == SARBP_STORE_C64 ? inv_s<N, SARBP_STORE_C64>(p, spec, etab, bound2, scale, out, s)
                                        : inv_s<N, SARBP_STORE_C32H>(p, spec, etab, bound2, scale, out, s);
}

template <int M>
cudaError_t fwd2(const RcPlan &p, const float2 *echo, const float2 *filt, const float2 *etab, float2 *spec,
                 float *bound2, cudaStream_t s) {
    constexpr int T = threads_for<M>();
    const size_t smem = sizeof(float2) * M + kTabSmem;
    auto k = rc_forward2_kernel<M, T>;
    cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void *>(k));
    if (e != cudaSuccess || t_prepare) return e;
    k<<<2 * p.np, T, smem, s>>>(p.ns, p.L, echo, filt, etab, spec, bound2);
    return cudaGetLastError();
}

}  // namespace

bool rc_size_supported(int nfft) {
    return nfft >= 64 && nfft <= 32768 && (nfft & (nfft - 1)) == 0;
}

#define SARBP_RC_SWITCH(N_, CALL)      \
    switch (N_) {                      \
        case 64: return CALL(64);      \
        case 128: return CALL(128);    \
        case 256: return CALL(256);    \
        case 512: return CALL(512);    \
        case 1024: return CALL(1024);  \
        case 2048: return CALL(2048);  \
        case 4096: return CALL(4096);  \
        case 8192: return CALL(8192);  \
        case 16384: return CALL(16384); \
        default: return cudaErrorInvalidValue; \
    }

cudaError_t launch_rc_forward(const RcPlan &p, const float2 *echo, const float2 *filt,
                              const float2 *etab, float2 *spec, float *scale, cudaStream_t s) {
    if (p.np <= 0) return cudaSuccess;
    if (p.L < 1 || p.L > 16) return cudaErrorInvalidValue;
    if (p.nfft == 32768) {
        if (!p.bound2 && !t_prepare) return cudaErrorInvalidValue;
        return fwd2<16384>(p, echo, filt, etab, spec, p.bound2, s);
    }
#define SARBP_FWD(N) fwd_n<N>(p, echo, filt, etab, spec, scale, s)
    SARBP_RC_SWITCH(p.nfft, SARBP_FWD)
#undef SARBP_FWD
}

cudaError_t launch_rc_inverse(const RcPlan &p, const float2 *spec, const float2 *etab,
                              const float *scale, void *out, cudaStream_t s) {
    if (p.np <= 0) return cudaSuccess;
    if (p.L < 1 || p.L > 16) return cudaErrorInvalidValue;
    float *sc = const_cast<float *>(scale);
    if (p.nfft == 32768) {
        if (!p.bound2 && !t_prepare) return cudaErrorInvalidValue;
        return inv_n<32768>(p, spec, etab, p.bound2, sc, out, s);
    }
#define SARBP_INV(N) inv_n<N>(p, spec, etab, nullptr, sc, out, s)
    SARBP_RC_SWITCH(p.nfft, SARBP_INV)
#undef SARBP_INV
}

cudaError_t prepare_rc_kernels(const RcPlan &p) {
    if (p.L < 1 || p.L > 16) return cudaErrorInvalidValue;
    RcPlan q = p;
    q.np = 1;  // the launchers return early for empty plans
    t_prepare = true;
    cudaError_t e = launch_rc_forward(q, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr);
    if (e == cudaSuccess) e = launch_rc_inverse(q, nullptr, nullptr, nullptr, nullptr, nullptr);
    t_prepare = false;
    return e;
}

}  // namespace sarbp
