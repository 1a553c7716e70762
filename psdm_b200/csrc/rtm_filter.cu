// Frequency filter of recorded traces on the device: the reference's
// freq_filter (src/auxiliar.f90:498-531) with filters_function1D and its
// order-6 Butterworth response (src/filters.f90:50-232).  Each trace is
// placed at the end of a zero buffer 24 times its length, transformed,
// multiplied by the response (and by 1/n, the forward scaling of the
// reference's FFT), transformed back, and the real part of the last nt
// samples is kept.
//
// Only lags below nt of that circular convolution reach the samples that are
// kept, so a transform of N >= 2 nt - 1 points (a power of two) with the
// response's impulse response cut to those lags gives the same samples with
// a twelfth of the work.  filter_kernel does it in one pass, a block a trace:
// real transform, response and inverse in shared memory, so that a trace is
// read and written once.  480 traces of 2004 samples: 18.6 us, against 1.41 ms
// with batched cuFFT transforms of the padded traces (three passes over 92 MB
// buffers); the error against 64 bits is the same 9.5e-5, that of the
// reference's single-precision frequency sums.
// Traces of more than 16384 samples, whose transform does not fit a block's
// shared memory, take the cuFFT form (filter_traces).  The results agree
// with the reference's arithmetic to FP32 rounding, not bit for bit.

#include <cuda_runtime.h>
#include <cuComplex.h>
#include <cufft.h>

#include <cmath>
#include <complex>
#include <vector>

#include "../../include/psdm_rtm.h"
#include "rtm_internal.h"

namespace psdm {

// Butterworth response H[ts] (butterworth, filters.f90:129-232) for the
// filter filters_function1D sets up: order n = 6 (even), high-pass start
// fs = 40 Hz, band edges f1 and fc, f0 = sqrt(f1 fc), Q = f0 / (fc - f1),
// frequency step fe/ts accumulated in single precision as the reference does.
void butterworth_response(int ts, float fe, int typef, float f1, float fc, std::complex<float>* H) {
    using cf = std::complex<float>;
    const int n = 6;
    const float pi = 3.14159265f, fs = 40.f;
    const float f2 = fc;
    const float f0 = std::sqrt(f1 * f2);
    const float Q = f0 / (f2 - f1);
    const cf I(0.f, 1.f);
    std::vector<cf> Bn(ts, cf(1.f, 0.f));
    float f = 0.f;
    for (int j = 0; j < ts / 2 + 1; ++j) {
        for (int k = 1; k <= n / 2; ++k) {
            const float c = std::cos((float(2 * k + n - 1) * pi) / float(2 * n));
            cf s;
            if (typef == 1)
                s = (I * f) / fc;
            else if (typef == 2)
                s = fs / (I * f);
            else
                s = Q * ((I * f) / f0 + f0 / (I * f));
            Bn[j] = Bn[j] * (s * s - 2.f * s * c + 1.f);
        }
        f = f + fe / float(ts);
    }
    for (int j = 0; j < ts / 2 + 1; ++j) H[j] = cf(1.f, 0.f) / Bn[j];
    H[0] = typef == 1 ? cf(1.f, 0.f) : cf(0.f, 0.f);
    for (int j = 2; j <= ts / 2; ++j) H[ts / 2 + j - 1] = std::conj(H[ts / 2 + 1 - (j - 1) - 1]);
}

namespace {

// Real input rows of ts samples, the trace at the end of each.
__global__ void pad_traces(const float* tr, int nt, int ts, int num, float* x) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)ts * num) return;
    const int t = (int)(i % ts), r = (int)(i / ts);
    const int off = ts - nt;
    x[i] = t >= off ? tr[(size_t)r * nt + (t - off)] : 0.f;
}

// The non-negative half of the spectrum times H / ts (the forward scaling
// of the reference's transform).
__global__ void apply_response(cufftComplex* X, const cufftComplex* H, int nh, int num, float scale) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)nh * num) return;
    const cufftComplex h = H[i % nh], v = X[i];
    const float re = v.x * scale, im = v.y * scale;
    X[i] = make_cuComplex(re * h.x - im * h.y, re * h.y + im * h.x);
}

__global__ void unpad_traces(const float* x, int nt, int ts, int num, const int* keep, float* tr) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)nt * num) return;
    const int t = (int)(i % nt), r = (int)(i / nt);
    if (!keep[r]) return;  // an all-zero trace is left as it is (is_not_cero)
    tr[i] = x[(size_t)r * ts + (ts - nt) + t];
}

__global__ void nonzero_traces(const float* tr, int nt, int num, int* keep) {
    const int r = blockIdx.x;
    if (r >= num) return;
    int any = 0;
    for (int t = threadIdx.x; t < nt && !any; t += blockDim.x) any = tr[(size_t)r * nt + t] != 0.f;
    any = __syncthreads_or(any);
    if (threadIdx.x == 0) keep[r] = any;
}

}  // namespace

size_t filter_work_floats(int ts, int num) {
    const size_t real = ((size_t)ts * num + 3) & ~(size_t)3;  // complex half starts 16-byte aligned
    return real + (size_t)(ts / 2 + 1) * num * 2;
}

// ---- the one-pass form

namespace {

__device__ __forceinline__ float2 cmul(const float2& a, const float2& b) {
    return make_float2(fmaf(a.x, b.x, -__fmul_rn(a.y, b.y)), fmaf(a.x, b.y, __fmul_rn(a.y, b.x)));
}
__device__ __forceinline__ float2 cadd(const float2& a, const float2& b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(const float2& a, const float2& b) { return make_float2(a.x - b.x, a.y - b.y); }
// a times -i (forward) or i (inverse)
template <bool INV>
__device__ __forceinline__ float2 rot(const float2& a) {
    return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}
template <bool INV>
__device__ __forceinline__ void dft4(float2& a, float2& b, float2& c, float2& d) {
    const float2 s = cadd(a, c), t = csub(a, c), u = cadd(b, d), v = rot<INV>(csub(b, d));
    a = cadd(s, u);
    b = cadd(t, v);
    c = csub(s, u);
    d = csub(t, v);
}
template <bool INV, int R>
__device__ __forceinline__ void dft(float2 (&v)[R]) {
    if (R == 2) {
        const float2 t = v[0];
        v[0] = cadd(t, v[1]);
        v[1] = csub(t, v[1]);
    } else if (R == 4) {
        dft4<INV>(v[0], v[1], v[2], v[3]);
    } else {
        float2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
        dft4<INV>(e[0], e[1], e[2], e[3]);
        dft4<INV>(o[0], o[1], o[2], o[3]);
        const float r = 0.70710678118654752f;
        o[1] = cmul(o[1], make_float2(r, INV ? r : -r));
        o[2] = rot<INV>(o[2]);
        o[3] = cmul(o[3], make_float2(-r, INV ? r : -r));
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[k] = cadd(e[k], o[k]);
            v[k + 4] = csub(e[k], o[k]);
        }
    }
}

// Shared index of point i: a pad after every 16 points keeps the strided
// stores of the first stages off one bank.
__device__ __forceinline__ int padded(int i) { return i + (i >> 4); }

// One self-sorting stage of radix R over M points held E a thread: butterfly
// b = s p + q takes points b + k M / R and leaves q + s (R p + k), times
// W_M^(s p k) (tw: W_2M).
template <bool INV, int R, int E>
__device__ __forceinline__ void fft_stage(float2* z, const float2* __restrict__ tw, int M, int ls, int tid, int T) {
    constexpr int B = E / R;
    const int nb = M / R;
    float2 v[B][R];
#pragma unroll
    for (int u = 0; u < B; ++u) {
        const int b = tid + u * T;
        if (b >= nb) break;
#pragma unroll
        for (int k = 0; k < R; ++k) v[u][k] = z[padded(b + k * nb)];
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < B; ++u) {
        const int b = tid + u * T;
        if (b >= nb) break;
        const int p = b >> ls, q = b & ((1 << ls) - 1);
        dft<INV, R>(v[u]);
        z[padded(q + ((R * p) << ls))] = v[u][0];
#pragma unroll
        for (int k = 1; k < R; ++k) {
            float2 w = __ldg(tw + (((p * k) << ls) << 1));
            if (INV) w.y = -w.y;
            z[padded(q + ((R * p + k) << ls))] = cmul(v[u][k], w);
        }
    }
    __syncthreads();
}

template <bool INV, int E>
__device__ __forceinline__ void fft(float2* z, const float2* tw, int M, int logM, int tid, int T) {
    int ls = 0;
    for (; logM - ls >= 3; ls += 3) fft_stage<INV, 8, E>(z, tw, M, ls, tid, T);
    if (logM - ls == 2) fft_stage<INV, 4, E>(z, tw, M, ls, tid, T);
    if (logM - ls == 1) fft_stage<INV, 2, E>(z, tw, M, ls, tid, T);
}

// One trace a block: y = x * h on a circle of 2M points.  The real trace is
// transformed as M complex points (even samples + i odd samples); X(k) and
// X(M - k) are separated, multiplied by the response G (M + 1 bins, 1/M
// included) and put together again.  A trace of zeros is left as it is
// (is_not_cero).
template <int E>
__global__ void __launch_bounds__(1024) filter_kernel(float* tr, int nt, int M, int logM, const float2* __restrict__ tw,
                              const float2* __restrict__ G) {
    extern __shared__ float2 z[];
    const int tid = threadIdx.x, T = blockDim.x;
    float* x = tr + (size_t)blockIdx.x * nt;
    int any = 0;
    for (int n = tid; n < M; n += T) {
        const float a = 2 * n < nt ? x[2 * n] : 0.f, b = 2 * n + 1 < nt ? x[2 * n + 1] : 0.f;
        z[padded(n)] = make_float2(a, b);
        any |= a != 0.f || b != 0.f;
    }
    if (!__syncthreads_or(any)) return;
    fft<false, E>(z, tw, M, logM, tid, T);
    for (int k = tid; k <= M / 2; k += T) {
        const int m = (M - k) & (M - 1);
        const float2 a = z[padded(k)], c = z[padded(m)], w = __ldg(tw + k);
        const float2 e = make_float2(0.5f * (a.x + c.x), 0.5f * (a.y - c.y));
        const float2 o = make_float2(0.5f * (a.y + c.y), -0.5f * (a.x - c.x));  // (a - conj c) / 2i
        const float2 wo = cmul(w, o);
        const float2 gm = __ldg(G + M - k);
        const float2 y = cmul(cadd(e, wo), __ldg(G + k));
        const float2 ym = cmul(csub(e, wo), make_float2(gm.x, -gm.y));  // conj of Y(M - k)
        const float2 e2 = make_float2(0.5f * (y.x + ym.x), 0.5f * (y.y + ym.y));
        const float2 o2 = cmul(make_float2(0.5f * (y.x - ym.x), 0.5f * (y.y - ym.y)), make_float2(w.x, -w.y));
        z[padded(k)] = make_float2(e2.x - o2.y, e2.y + o2.x);  // e2 + i o2
        if (m != k) z[padded(m)] = make_float2(e2.x + o2.y, o2.x - e2.y);  // conj e2 + i conj o2
    }
    __syncthreads();
    fft<true, E>(z, tw, M, logM, tid, T);
    for (int n = tid; n < nt; n += T) {
        const float2 v = z[padded(n >> 1)];
        x[n] = (n & 1) ? v.y : v.x;
    }
}

// Sums of a spectrum at kOut outputs a block: 2 sum_k v[k].x cos(2 pi k j / n)
// and 2 sum_k v[k].y sin(2 pi k j / n), k from 0 to count - 1, k = 0 and `last`
// at half weight (of `last` only v.x counts).  A load of v serves kOut outputs,
// and the angles come from a rotation a thread that starts anew every kAnew
// terms, so that the sums are bound by double-precision arithmetic (six
// operations a term and output).  The first call of a band with traces of 2004
// / 8192 / 16384 samples: 0.26 / 1.3 / 3.6 ms, against 0.58 / 7.2 / 27.9 with a
// root read from a table for each term and the lags l and -l summed apart.
constexpr int kOut = 4, kAnew = 64, kSumThreads = 256;
__device__ __forceinline__ void trig_sums(const double2* __restrict__ v, int count, int last, int n, int j0,
                                          double2 (&sum)[kOut]) {
    __shared__ double part[kSumThreads / 32][2 * kOut];
    const int tid = threadIdx.x;
    double2 w[kOut], step[kOut], s[kOut];
    auto angle = [n](long long k, int j) {
        double2 r;
        sincospi(2.0 * (double)(k * j % n) / n, &r.y, &r.x);
        return r;
    };
#pragma unroll
    for (int r = 0; r < kOut; ++r) {
        step[r] = angle(kSumThreads, j0 + r);
        s[r] = make_double2(0.0, 0.0);
    }
    for (int k0 = tid; k0 < count; k0 += kAnew * kSumThreads) {
#pragma unroll
        for (int r = 0; r < kOut; ++r) w[r] = angle(k0, j0 + r);
        const int end = min(count, k0 + kAnew * kSumThreads);
        for (int k = k0; k < end; k += kSumThreads) {
            double2 g = v[k];
            if (k == 0 || k == last) {
                g.x *= 0.5;
                g.y = k == last ? 0.0 : 0.5 * g.y;
            }
#pragma unroll
            for (int r = 0; r < kOut; ++r) {
                const double x = w[r].x, y = w[r].y;
                s[r].x = fma(g.x, x, s[r].x);
                s[r].y = fma(g.y, y, s[r].y);
                w[r].x = fma(x, step[r].x, -(y * step[r].y));
                w[r].y = fma(x, step[r].y, y * step[r].x);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < kOut; ++r) {
        for (int o = 16; o > 0; o >>= 1) {
            s[r].x += __shfl_down_sync(0xffffffffu, s[r].x, o);
            s[r].y += __shfl_down_sync(0xffffffffu, s[r].y, o);
        }
        if ((tid & 31) == 0) {
            part[tid >> 5][2 * r] = s[r].x;
            part[tid >> 5][2 * r + 1] = s[r].y;
        }
    }
    __syncthreads();
    if (tid != 0) return;
#pragma unroll
    for (int r = 0; r < kOut; ++r) {
        sum[r] = make_double2(0.0, 0.0);
        for (int k = 0; k < kSumThreads / 32; ++k) {
            sum[r].x += part[k][2 * r];
            sum[r].y += part[k][2 * r + 1];
        }
        sum[r].x *= 2.0;
        sum[r].y *= 2.0;
    }
}

// Impulse response at the lags l and -l, l < nt, of the response H (bins 0 ..
// ts/2; of the last one only the real part counts) on a circle of ts points:
// (h(l) + h(-l)) / 2 and (h(-l) - h(l)) / 2.
__global__ void __launch_bounds__(kSumThreads) impulse_kernel(const double2* __restrict__ H, int ts, int nt, double2* h) {
    double2 sum[kOut];
    trig_sums(H, ts / 2 + 1, ts / 2, ts, blockIdx.x * kOut, sum);
    for (int r = 0; threadIdx.x == 0 && r < kOut; ++r)
        if (blockIdx.x * kOut + r < nt) h[blockIdx.x * kOut + r] = make_double2(sum[r].x / ts, sum[r].y / ts);
}

// Bins 0 .. M of that impulse response's transform of 2M points, / M.
__global__ void __launch_bounds__(kSumThreads) response_kernel(const double2* __restrict__ h, int nt, int M, float2* G) {
    double2 sum[kOut];
    trig_sums(h, nt, -1, 2 * M, blockIdx.x * kOut, sum);
    for (int r = 0; threadIdx.x == 0 && r < kOut; ++r)
        if (blockIdx.x * kOut + r <= M)
            G[blockIdx.x * kOut + r] = make_float2((float)(sum[r].x / M), (float)(sum[r].y / M));
}

// exp(-2 pi i j / n) in single precision
__global__ void twiddle_kernel(float2* tw, int n) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    double s, c;
    sincospi(2.0 * j / n, &s, &c);
    tw[j] = make_float2((float)c, (float)-s);
}

}  // namespace

int filter_points(int nt) {
    int M = 256;
    while (2 * M < 2 * nt - 1) M *= 2;
    return M <= kFilterMaxPoints ? M : 0;
}

void butterworth_response_f64(int ts, float fe, int typef, float f1, float fc, std::complex<double>* H) {
    // butterworth_response's parameters and frequencies (its single-precision
    // sums), the response itself in double: s is purely imaginary, s = i b
    constexpr int n = 6;
    const float pi = 3.14159265f, fs = 40.f, f0 = std::sqrt(f1 * fc), Q = f0 / (fc - f1);
    double c[n / 2];
    for (int k = 1; k <= n / 2; ++k) c[k - 1] = std::cos((float(2 * k + n - 1) * pi) / float(2 * n));
    float f = 0.f;
    for (int j = 0; j <= ts / 2; ++j) {
        const double x = f;
        const double b = typef == 1 ? x / fc : (typef == 2 ? -fs / x : (double)Q * (x / f0 - f0 / x));
        std::complex<double> B(1.0, 0.0);
        for (int k = 1; k <= n / 2; ++k) {
            const double re = 1.0 - b * b, im = -2.0 * b * c[k - 1];
            B = std::complex<double>(B.real() * re - B.imag() * im, B.real() * im + B.imag() * re);
        }
        const double q = B.real() * B.real() + B.imag() * B.imag();
        H[j] = std::complex<double>(B.real() / q, -B.imag() / q);
        f = f + fe / float(ts);
    }
    H[0] = typef == 1 ? 1.0 : 0.0;
}

size_t filter_design_bytes(int ts, int nt) { return ((size_t)ts / 2 + 1 + nt) * sizeof(double2); }

int design_filter(const void* d_H, void* work, int ts, int nt, int M, void* d_tw, void* d_G, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    double2* h = static_cast<double2*>(work);
    impulse_kernel<<<(nt + kOut - 1) / kOut, kSumThreads, 0, st>>>(static_cast<const double2*>(d_H), ts, nt, h);
    response_kernel<<<(M + kOut) / kOut, kSumThreads, 0, st>>>(h, nt, M, static_cast<float2*>(d_G));
    twiddle_kernel<<<(2 * M + 255) / 256, 256, 0, st>>>(static_cast<float2*>(d_tw), 2 * M);
    return (int)cudaGetLastError();
}

template <int E>
int launch_filter_t(float* d_tr, int nt, int num, int M, const void* d_tw, const void* d_G, cudaStream_t st) {
    int logM = 0;
    while ((1 << logM) < M) ++logM;
    const size_t bytes = (size_t)(M + M / 16) * sizeof(float2);
    if (bytes > 48 * 1024) {
        const cudaError_t rc = cudaFuncSetAttribute(filter_kernel<E>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                    (int)bytes);
        if (rc != cudaSuccess) return (int)rc;
    }
    filter_kernel<E><<<num, M / E, bytes, st>>>(d_tr, nt, M, logM, static_cast<const float2*>(d_tw),
                                                static_cast<const float2*>(d_G));
    return (int)cudaGetLastError();
}

int launch_filter(float* d_tr, int nt, int num, int M, const void* d_tw, const void* d_G, void* stream) {
    // 8 points a thread up to 1024 threads
    if (M <= 8192) return launch_filter_t<8>(d_tr, nt, num, M, d_tw, d_G, (cudaStream_t)stream);
    return launch_filter_t<16>(d_tr, nt, num, M, d_tw, d_G, (cudaStream_t)stream);
}

// ---- the cuFFT form

// The reference transforms the real trace as a complex one and keeps the real
// part of the inverse.  The product of a real trace's spectrum with the
// response is Hermitian in every bin but ts/2, where only its real part
// reaches the real output, so the half-spectrum transforms (real to complex,
// complex to real, which reads the real part of bin ts/2) give the same
// result at half the work.
int filter_traces(float* d_tr, int nt, int num, const void* d_H, float* d_x, int* d_keep, int ts, const int* plans,
                  void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    const int nh = ts / 2 + 1;
    float* x = d_x;
    cufftComplex* X = reinterpret_cast<cufftComplex*>(d_x + (((size_t)ts * num + 3) & ~(size_t)3));
    const size_t total = (size_t)ts * num;
    nonzero_traces<<<num, 256, 0, st>>>(d_tr, nt, num, d_keep);
    pad_traces<<<(int)((total + 255) / 256), 256, 0, st>>>(d_tr, nt, ts, num, x);
    if (cufftSetStream(plans[0], st) != CUFFT_SUCCESS || cufftSetStream(plans[1], st) != CUFFT_SUCCESS) return 1;
    if (cufftExecR2C(plans[0], x, X) != CUFFT_SUCCESS) return 2;
    apply_response<<<(int)(((size_t)nh * num + 255) / 256), 256, 0, st>>>(X, static_cast<const cufftComplex*>(d_H), nh,
                                                                          num, 1.f / float(ts));
    if (cufftExecC2R(plans[1], X, x) != CUFFT_SUCCESS) return 3;
    unpad_traces<<<(int)(((size_t)nt * num + 255) / 256), 256, 0, st>>>(x, nt, ts, num, d_keep, d_tr);
    return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

int make_fft_plans(int ts, int num, int* plans) {
    cufftHandle a, b;
    int n[1] = {ts};
    const int nh = ts / 2 + 1;
    if (cufftPlanMany(&a, 1, n, nullptr, 1, ts, nullptr, 1, nh, CUFFT_R2C, num) != CUFFT_SUCCESS) return 1;
    if (cufftPlanMany(&b, 1, n, nullptr, 1, nh, nullptr, 1, ts, CUFFT_C2R, num) != CUFFT_SUCCESS) {
        cufftDestroy(a);
        return 1;
    }
    plans[0] = a;
    plans[1] = b;
    return 0;
}

void destroy_fft_plans(int* plans) {
    cufftDestroy(plans[0]);
    cufftDestroy(plans[1]);
}

}  // namespace psdm

extern "C" int psdm_butterworth_response(int32_t ts, float fe, int32_t typef, float f1, float f2, float* H) {
    if (!H || ts < 2 || (ts & 1) || typef < 1 || typef > 3) {
        psdm::set_last_error("psdm_butterworth_response: null output, odd or short length, or typef not 1..3");
        return PSDM_ERR_ARG;
    }
    psdm::butterworth_response(ts, fe, typef, f1, f2, reinterpret_cast<std::complex<float>*>(H));
    return PSDM_OK;
}
