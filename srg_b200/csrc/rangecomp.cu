// rangecomp.cu -- range compression of decoded Sentinel-1 echo lines on the GPU.
//
// Follows sentinel/processsub.f90:86-123 in what it computes: the chirp
// replica of the decoded pulse parameters (processsub.f90:101-107, built on
// the host with the reference's types: t = (j-1)/samplefreq in FP32, the
// phase in FP64, each sample rounded to complex64 and divided by npts),
// its 32,768-point spectrum, and per line: the samples zero-padded to 32,768,
// forward FFT, times the conjugate replica spectrum, inverse FFT
// (unnormalised), the first nvalid = nsamps - npts samples kept.  The lines
// go through in blocks: one kernel pads a block, cuFFT transforms it, one
// kernel multiplies, cuFFT transforms back, one kernel writes the valid
// samples.  FFTs by cuFFT (the reference uses FFTW in single precision).
// Pulses of up to about 6,800 samples (Sentinel-1 IW: ~3,370) take the fused
// overlap-save kernel instead (rc_os_kernel below), same samples.
#include <cuda_runtime.h>
#include <cufft.h>

#include <climits>
#include <cmath>
#include <complex>
#include <cstring>
#include <mutex>
#include <vector>

#include "../../include/srg_bp.h"
#include "fft_conv.cuh"
#include "host_internal.h"

using namespace srg;
using namespace srg::detail;

namespace {

constexpr int kRangeFFT = 32768;  // ranfft (processsub.f90:38)
constexpr int kBlock = 256;       // lines per transform batch

#define CKR(call)                                                                      \
    do {                                                                               \
        cudaError_t e_ = (call);                                                       \
        if (e_ != cudaSuccess)                                                         \
            return fail(SRG_E_CUDA, "%s failed: %s", #call, cudaGetErrorString(e_));   \
    } while (0)
#define CKFR(call)                                                                     \
    do {                                                                               \
        cufftResult r_ = (call);                                                       \
        if (r_ != CUFFT_SUCCESS) return fail(SRG_E_CUDA, "%s failed: cufft %d", #call, (int)r_); \
    } while (0)

__global__ void rc_pad_kernel(const float2 *__restrict__ in, long long ld, int l0, int nlines, int nsamps,
                              float2 *__restrict__ buf) {
    const long long total = (long long)kBlock * kRangeFFT;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int l = (int)(i / kRangeFFT), n = (int)(i - (long long)l * kRangeFFT);
        float2 v = make_float2(0.f, 0.f);
        if (l0 + l < nlines && n < nsamps) v = in[(long long)(l0 + l) * ld + n];
        buf[i] = v;
    }
}

// spectrum times the conjugate replica spectrum
__global__ void rc_mul_kernel(float2 *__restrict__ buf, const float2 *__restrict__ ref) {
    const long long total = (long long)kBlock * kRangeFFT;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const float2 a = buf[i], r = ref[i & (kRangeFFT - 1)];
        buf[i] = make_float2(a.x * r.x + a.y * r.y, a.y * r.x - a.x * r.y);
    }
}

__global__ void rc_out_kernel(const float2 *__restrict__ buf, int l0, int nlines, int nvalid,
                              float2 *__restrict__ out, long long ldo) {
    const int nl = min(kBlock, nlines - l0);
    const long long total = (long long)nl * nvalid;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int l = (int)(i / nvalid), n = (int)(i - (long long)l * nvalid);
        out[(long long)(l0 + l) * ldo + n] = buf[(long long)l * kRangeFFT + n];
    }
}

// ---------------------------------------------------------------------------
// Fused matched filter by overlap-save.  The samples the reference keeps,
// y[n] = 32768 sum_{j < npts} conj(r[j]) x[n + j] for n < nvalid, are a
// linear correlation (the 32,768-point circular one never wraps into them),
// so 8,192-point transforms give them exactly up to rounding: a segment of
// 8,192 samples from s0 (zeros past the line) yields y[s0 .. s0 + L),
// L = 8192 - npts + 1.  A CTA (one per SM, persistent) takes (line, segment)
// items in turn: it loads the segment's samples once, convolves them in shared
// memory (fft_conv.cuh) with the filter H = (32768 / 8192) conj(DFT_8192(r))
// and writes its L outputs once: the lines cross HBM once each way, where the
// cuFFT path below takes five passes over 32,768-point rows.  A CTA takes two
// segments at once, 256 threads each, that share the twiddles (62 KB) in shared
// memory; the filter's spectrum (64 KB, once per segment) is read through L1.
// Bound by instruction issue (see fft_conv.cuh): 1,500 lines of 24,000 samples,
// pulse of 3,371, take 0.31 ms (0.45 with self-sorting transforms of one segment
// per 512-thread CTA), 700 lines of 29,001 with a pulse of 5,147 0.24 ms (0.58
// with cuFFT); error against 64 bits 1.8e-7 (2.0e-7 and 4.9e-7).  With fused
// butterflies (Plan::FUSED) 0.29 ms and 5 % more error, before the transforms'
// gain was taken out; with the spectrum in shared memory and half the twiddles
// turned from the others 0.30 and 10 % more; everything through L1 and two CTAs per
// SM 0.31, as two halves of 4,096 points at 16 points per thread 0.42.
using Seg = fftc::Plan<8192, 32, 16, 16, 32, false>;
constexpr int kOsM = Seg::M;                     // segment transform
// Segments per line up to which the kernel is the faster path: one takes
// 41 ns (of the whole chip), a line of the cuFFT path 0.84 us whatever its
// pulse.  Pulses of up to 6,400 samples stay within it on lines of any length.
constexpr int kOsMaxSegs = 20;
constexpr int kOsLines = 2;                      // segments of a CTA at once
constexpr int kOsThreads = kOsLines * Seg::T;
// pass 1's twiddles of every column in shared memory (exactly rounded: turned
// from the first columns' they cost 5 % more error); pass 2's are read through
// L1 (in shared memory as well they leave L1 too small for the spectrum: 0.33 ms)
constexpr int kOsTw1 = (Seg::RA - 1) * Seg::CA;
constexpr int kOsSmem = (kOsLines * Seg::BUF + kOsTw1) * (int)sizeof(float2);
struct SegTw1 {
    const float2 *t;
    __device__ __forceinline__ float2 operator()(int r, int j, int g) const {
        return t[(r - 1) * Seg::CA + j + g * Seg::T];
    }
};

__global__ void __launch_bounds__(kOsThreads, 1)
rc_os_kernel(const float2 *__restrict__ in, long long ld_in, int nsamps, int nvalid, int L,
             int nseg, int nitems, const float2 *__restrict__ H, const float2 *__restrict__ tw,
             float2 *__restrict__ out, long long ld_out) {
    extern __shared__ float2 os_sm[];
    const int j = threadIdx.x % Seg::T, slot = threadIdx.x / Seg::T;
    float2 *buf = os_sm + slot * Seg::BUF;
    float2 *t1 = os_sm + kOsLines * Seg::BUF;
    for (int i = threadIdx.x; i < kOsTw1; i += kOsThreads) t1[i] = __ldg(tw + i);
    __syncthreads();
    const SegTw1 tw1{t1};
    const float2 *tw2 = tw + kOsTw1;
    const fftc::Filter<Seg> filter{H};
    const int step = gridDim.x * kOsLines;
    for (int item = blockIdx.x * kOsLines + slot; item < nitems; item += step) {
        const int line = item / nseg, s0 = (item - line * nseg) * L;
        const float2 *x = in + (long long)line * ld_in + s0 + j;
        const int nin = nsamps - s0 - j;
        float2 v[Seg::EPT];
#pragma unroll
        for (int i = 0; i < Seg::EPT; ++i) {
            const int n = fftc::point_of<Seg>(i);
            v[i] = n < nin ? fftc::ld_stream(x + n) : make_float2(0.f, 0.f);
        }
        if (item + step < nitems) {  // the next segment into L2
            const int nl = (item + step) / nseg, ns = (item + step - nl * nseg) * L;
            const float2 *nx = in + (long long)nl * ld_in + ns;
            for (int c = 16 * j; c < min(kOsM, nsamps - ns); c += 16 * Seg::T)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(nx + c));
        }
        fftc::conv<Seg>(v, buf, j, slot, false, tw1, tw2, tw1, tw2, filter);
        float2 *y = out + (long long)line * ld_out + s0 + j;
        const int nout = min(L, nvalid - s0) - j;
#pragma unroll
        for (int i = 0; i < Seg::EPT; ++i) {
            const int n = fftc::point_of<Seg>(i);
            if (n < nout) y[n] = v[i];
        }
        fftc::line_sync<Seg>(slot, false);  // the buffer's reads are done
    }
}

// Forward DFT (sign -1, unnormalised) of a power-of-two length, in FP64 on
// the host: iterative radix-2 decimation in time.
void host_fft(std::vector<std::complex<double>> &a) {
    const int n = (int)a.size();
    for (int i = 1, j = 0; i < n; ++i) {
        int bit = n >> 1;
        for (; j & bit; bit >>= 1) j ^= bit;
        j ^= bit;
        if (i < j) std::swap(a[i], a[j]);
    }
    const double pi = 4.0 * std::atan2(1.0, 1.0);
    for (int len = 2; len <= n; len <<= 1) {
        for (int k = 0; k < len / 2; ++k) {
            const std::complex<double> w = std::polar(1.0, -2.0 * pi * k / len);
            for (int i = 0; i < n; i += len) {
                const std::complex<double> u = a[i + k], v = a[i + k + len / 2] * w;
                a[i + k] = u + v;
                a[i + k + len / 2] = u - v;
            }
        }
    }
}

struct RcCtx {
    std::mutex mu;
    cufftHandle plan_blk = 0, plan_one = 0;
    bool have_plans = false;
    DevBuf buf, ref;
    float key[4] = {NAN, NAN, NAN, NAN};  // replica parameters of `ref`
    // overlap-save path: filter spectrum, twiddle tables, their parameters
    DevBuf os_h, os_tw;
    bool os_ready = false;
    int os_ctas = 0;  // resident CTAs
    float os_key[4] = {NAN, NAN, NAN, NAN};
};
RcCtx g_rc[64];

// Samples of the replica of a pulse (processsub.f90:94), and whether n hold them.
int replica_points(float samplefreq, float pulselength, int n, int *npts) {
    if (n < 1 || !(samplefreq > 0) || !(pulselength > 0))
        return fail(SRG_E_ARG, "bad replica arguments");
    const float prod = pulselength * samplefreq;  // real*4 product
    *npts = (int)prod;                            // truncated, as the Fortran assignment
    if (*npts < 1 || *npts > n)
        return fail(SRG_E_ARG, "replica of %d samples does not fit %d", *npts, n);
    return SRG_OK;
}

int grid_of(long long n) { return (int)std::min<long long>((n + 255) / 256, 148LL * 32); }

}  // namespace

extern "C" {

int srg_range_replica(float samplefreq, float startfreq, float ramprate, float pulselength,
                      float *replica, int n, int *npts_out) {
    if (!replica) return fail(SRG_E_ARG, "bad replica arguments");
    int npts = 0;
    if (const int rc = replica_points(samplefreq, pulselength, n, &npts)) return rc;
    const double pi = 4.0 * std::atan2(1.0, 1.0);
    std::memset(replica, 0, sizeof(float) * 2 * (size_t)n);
    for (int j = 1; j <= npts; ++j) {
        const double t = (double)((float)(j - 1) / samplefreq);
        const double phase = 2.0 * pi * (double)startfreq * t + pi * (double)ramprate * t * t;
        replica[2 * (j - 1)] = (float)std::cos(phase) / (float)npts;
        replica[2 * (j - 1) + 1] = (float)std::sin(phase) / (float)npts;
    }
    if (npts_out) *npts_out = npts;
    return SRG_OK;
}

int srg_range_compress_device(const float *lines, long long ld_in, int nlines, int nsamps,
                              float samplefreq, float startfreq, float ramprate, float pulselength,
                              float *out, long long ld_out, int *nvalid_out, void *stream) {
    if (!lines || !out || nlines < 1 || nsamps < 1 || nsamps > kRangeFFT || ld_in < nsamps)
        return fail(SRG_E_ARG, "bad range-compression sizes: nlines=%d nsamps=%d (<= %d) ld=%lld",
                    nlines, nsamps, kRangeFFT, ld_in);
    int npts = 0;
    int rc = replica_points(samplefreq, pulselength, kRangeFFT, &npts);
    if (rc) return rc;
    const int nvalid = nsamps - npts;
    if (nvalid < 1) return fail(SRG_E_ARG, "pulse of %d samples leaves no valid sample of %d", npts, nsamps);
    if (ld_out < nvalid) return fail(SRG_E_ARG, "output row of %lld < %d valid samples", ld_out, nvalid);
    int dev = 0;
    CKR(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(SRG_E_ARG, "device %d out of range", dev);
    RcCtx &x = g_rc[dev];
    std::lock_guard<std::mutex> g(x.mu);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int L = kOsM - npts + 1, nseg = L > 0 ? (nvalid + L - 1) / L : 0;
    if (nseg > 0 && nseg <= kOsMaxSegs) {
        // fused overlap-save kernel (see rc_os_kernel)
        if ((rc = x.os_h.ensure(sizeof(float2) * kOsM)) ||
            (rc = x.os_tw.ensure(sizeof(float2) * (kOsTw1 + Seg::TW2))))
            return rc;
        if (!x.os_ready) {
            std::vector<float2> tw;
            const std::vector<float2> plan = fftc::tables<Seg>(0.0);
            const double tau = 8.0 * std::atan2(1.0, 1.0);
            for (int r = 1; r < Seg::RA; ++r)
                for (int d = 0; d < Seg::CA; ++d) {
                    const double a = tau * r * d / Seg::M;
                    tw.push_back(make_float2((float)std::cos(a), (float)-std::sin(a)));
                }
            tw.insert(tw.end(), plan.begin() + Seg::TW1, plan.end());
            int sms = 0;
            CKR(cudaFuncSetAttribute(rc_os_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kOsSmem));
            CKR(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
            CKR(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&x.os_ctas, rc_os_kernel, kOsThreads, kOsSmem));
            if (x.os_ctas < 1) return fail(SRG_E_UNSUPPORTED, "segment transform does not fit an SM");
            x.os_ctas *= sms;
            CKR(cudaMemcpyAsync(x.os_tw.p, tw.data(), sizeof(float2) * tw.size(), cudaMemcpyHostToDevice, st));
            CKR(cudaStreamSynchronize(st));  // `tw` is pageable host memory that goes out of scope
            x.os_ready = true;
        }
        const float key[4] = {samplefreq, startfreq, ramprate, pulselength};
        if (std::memcmp(key, x.os_key, sizeof key) != 0) {
            // H = (32768 / 8192) conj(DFT_8192(replica)), less the transforms' gain
            // (they return 1.0e-7 too little, half of the error against 64 bits), in
            // FP64 from the replica's complex64 samples
            std::vector<float> rep(2 * (size_t)kOsM);
            if ((rc = srg_range_replica(samplefreq, startfreq, ramprate, pulselength, rep.data(), kOsM,
                                        &npts)))
                return rc;
            std::vector<std::complex<double>> a(kOsM);
            for (int j = 0; j < npts; ++j) a[j] = std::complex<double>(rep[2 * j], rep[2 * j + 1]);
            host_fft(a);
            std::vector<float2> h(kOsM);
            const double scale = (double)kRangeFFT / kOsM / (1.0 + fftc::conv_gain<Seg>());
            for (int i = 0; i < Seg::EPT; ++i)
                for (int j = 0; j < Seg::T; ++j) {
                    const std::complex<double> b = a[fftc::spectrum_order<Seg>(i, j)];
                    h[i * Seg::T + j] = make_float2((float)(scale * b.real()), (float)(-scale * b.imag()));
                }
            CKR(cudaMemcpyAsync(x.os_h.p, h.data(), sizeof(float2) * kOsM, cudaMemcpyHostToDevice, st));
            CKR(cudaStreamSynchronize(st));  // `h` is pageable host memory that goes out of scope
            std::memcpy(x.os_key, key, sizeof key);
        }
        if ((long long)nlines * nseg > INT_MAX) return fail(SRG_E_ARG, "too many lines: %d", nlines);
        const int nitems = nlines * nseg;
        rc_os_kernel<<<std::min((nitems + kOsLines - 1) / kOsLines, x.os_ctas), kOsThreads, kOsSmem, st>>>(
            reinterpret_cast<const float2 *>(lines), ld_in, nsamps, nvalid, L, nseg, nitems,
            static_cast<const float2 *>(x.os_h.p), static_cast<const float2 *>(x.os_tw.p),
            reinterpret_cast<float2 *>(out), ld_out);
        CKR(cudaGetLastError());
        if (nvalid_out) *nvalid_out = nvalid;
        return SRG_OK;
    }
    if (!x.have_plans) {
        CKFR(cufftPlan1d(&x.plan_blk, kRangeFFT, CUFFT_C2C, kBlock));
        CKFR(cufftPlan1d(&x.plan_one, kRangeFFT, CUFFT_C2C, 1));
        x.have_plans = true;
    }
    if ((rc = x.buf.ensure(sizeof(float2) * (size_t)kBlock * kRangeFFT)) ||
        (rc = x.ref.ensure(sizeof(float2) * (size_t)kRangeFFT)))
        return rc;
    float2 *ref = static_cast<float2 *>(x.ref.p), *buf = static_cast<float2 *>(x.buf.p);
    const float key[4] = {samplefreq, startfreq, ramprate, pulselength};
    if (std::memcmp(key, x.key, sizeof key) != 0) {
        // replica spectrum (processsub.f90:101-108)
        std::vector<float> rep(2 * (size_t)kRangeFFT);
        if ((rc = srg_range_replica(samplefreq, startfreq, ramprate, pulselength, rep.data(), kRangeFFT,
                                    &npts)))
            return rc;
        CKR(cudaMemcpyAsync(ref, rep.data(), sizeof(float2) * kRangeFFT, cudaMemcpyHostToDevice, st));
        CKFR(cufftSetStream(x.plan_one, st));
        CKFR(cufftExecC2C(x.plan_one, reinterpret_cast<cufftComplex *>(ref),
                          reinterpret_cast<cufftComplex *>(ref), CUFFT_FORWARD));
        CKR(cudaStreamSynchronize(st));  // `rep` is pageable host memory that goes out of scope
        std::memcpy(x.key, key, sizeof key);
    }
    CKFR(cufftSetStream(x.plan_blk, st));
    for (int l0 = 0; l0 < nlines; l0 += kBlock) {
        rc_pad_kernel<<<grid_of((long long)kBlock * kRangeFFT), 256, 0, st>>>(
            reinterpret_cast<const float2 *>(lines), ld_in, l0, nlines, nsamps, buf);
        CKR(cudaGetLastError());
        CKFR(cufftExecC2C(x.plan_blk, reinterpret_cast<cufftComplex *>(buf),
                          reinterpret_cast<cufftComplex *>(buf), CUFFT_FORWARD));
        rc_mul_kernel<<<grid_of((long long)kBlock * kRangeFFT), 256, 0, st>>>(buf, ref);
        CKR(cudaGetLastError());
        CKFR(cufftExecC2C(x.plan_blk, reinterpret_cast<cufftComplex *>(buf),
                          reinterpret_cast<cufftComplex *>(buf), CUFFT_INVERSE));
        rc_out_kernel<<<grid_of((long long)kBlock * nvalid), 256, 0, st>>>(
            buf, l0, nlines, nvalid, reinterpret_cast<float2 *>(out), ld_out);
        CKR(cudaGetLastError());
    }
    if (nvalid_out) *nvalid_out = nvalid;
    return SRG_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// 2x oversampling of range lines (a finer line for the linear interpolation of
// the backprojection): even output samples are the input samples, odd ones an
// 8-tap Hann-windowed sinc at the half-sample point (taps normalised to unit
// DC gain, FP32); samples beyond the line read as 0.  2*nsamps - 1 samples
// per line.  No reference counterpart: the reference interpolates the
// original line linearly.
namespace {

// A CTA stages kOvSeg samples of a line and the four on either side in shared
// memory and writes their 2 kOvSeg outputs, 16 bytes per thread and store where
// the row allows it.  Bound by HBM (8 bytes read and 16 written per sample):
// 1,500 lines of 21,000 samples take 144 us (5.2 TB/s); one output per thread
// with its taps from global memory took 331.
constexpr int kOvSeg = 1024, kOvThreads = 256;
__global__ void __launch_bounds__(kOvThreads)
oversample2_kernel(const float2 *__restrict__ in, long long ld_in, int nlines, int nsamps, int nseg,
                   float2 *__restrict__ out, long long ld_out, float h0, float h1, float h2, float h3) {
    __shared__ float2 x[kOvSeg + 8];  // x[i]: sample k0 - 4 + i
    const float h[4] = {h0, h1, h2, h3};
    const long long items = (long long)nlines * nseg;
    for (long long item = blockIdx.x; item < items; item += gridDim.x) {
        const int l = (int)(item / nseg), k0 = (int)(item - (long long)l * nseg) * kOvSeg;
        const float2 *row = in + (long long)l * ld_in;
        for (int i = threadIdx.x; i < kOvSeg + 8; i += kOvThreads) {
            const int k = k0 - 4 + i;
            x[i] = k >= 0 && k < nsamps ? __ldg(row + k) : make_float2(0.f, 0.f);
        }
        __syncthreads();
        float2 *o = out + (long long)l * ld_out + 2 * k0;
        const bool pairs = (reinterpret_cast<unsigned long long>(o) & 15) == 0;
#pragma unroll
        for (int q = 0; q < kOvSeg / kOvThreads; ++q) {
            const int i = threadIdx.x + q * kOvThreads, k = k0 + i;  // samples k and between k, k + 1
            if (k >= nsamps) break;
            const float2 e = x[i + 4];
            float re = 0.f, im = 0.f;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const float2 sa = x[i + 4 - t], sb = x[i + 5 + t];
                re = fmaf(h[t], sa.x + sb.x, re);
                im = fmaf(h[t], sa.y + sb.y, im);
            }
            if (k + 1 == nsamps) {  // the line's last sample has none after it
                o[2 * i] = e;
            } else if (pairs) {
                reinterpret_cast<float4 *>(o)[i] = make_float4(e.x, e.y, re, im);
            } else {
                o[2 * i] = e;
                o[2 * i + 1] = make_float2(re, im);
            }
        }
        __syncthreads();
    }
}

}  // namespace

extern "C" {

void srg_oversample_taps(float taps[4]) {
    const double pi = 4.0 * std::atan2(1.0, 1.0);
    double h[4], s = 0.0;
    for (int t = 0; t < 4; ++t) {
        const double x = t + 0.5;
        const double sinc = std::sin(pi * x) / (pi * x);
        const double win = 0.5 * (1.0 + std::cos(pi * x / 4.0));
        h[t] = sinc * win;
        s += 2.0 * h[t];
    }
    for (int t = 0; t < 4; ++t) taps[t] = (float)(h[t] / s);
}

int srg_oversample_range_device(const float *in, long long ld_in, int nlines, int nsamps, float *out,
                                long long ld_out, void *stream) {
    if (!in || !out || nlines < 1 || nsamps < 2 || ld_in < nsamps || ld_out < 2LL * nsamps - 1)
        return fail(SRG_E_ARG, "bad oversampling sizes: nlines=%d nsamps=%d ld_in=%lld ld_out=%lld",
                    nlines, nsamps, ld_in, ld_out);
    float h[4];
    srg_oversample_taps(h);
    const int nseg = (nsamps - 1) / kOvSeg + 1;
    const long long items = (long long)nlines * nseg;
    oversample2_kernel<<<(int)std::min<long long>(items, 148LL * 64), kOvThreads, 0,
                         static_cast<cudaStream_t>(stream)>>>(
        reinterpret_cast<const float2 *>(in), ld_in, nlines, nsamps, nseg,
        reinterpret_cast<float2 *>(out), ld_out, h[0], h[1], h[2], h[3]);
    CKR(cudaGetLastError());
    return SRG_OK;
}

}  // extern "C"
