// crossmul.cu -- interferograms of co-registered complex64 images on the GPU.
//
// Follows int/crossmul.f90:95-185 in what it computes.  Per image line:
//   1. in * scale, zero-padded from na to nnn = the first 2^i >= na (i >= 1)
//      (crossmul.f90:69-73, 128-135);
//   2. forward FFT of nnn points (FFTW sign -1, unnormalised);
//   3. spectrum bins [0, nnn/2) to [0, nnn/2) and [nnn/2, nnn) to
//      [2nnn - nnn/2, 2nnn) of a zeroed 2nnn array (crossmul.f90:136-137);
//   4. inverse FFT of 2nnn points (sign +1), / nnn / 2 (crossmul.f90:139-141).
// Per pair and output sample (line L, column j), with u1, u2 the upsampled
// lines: igram = sum_k sum_i (u1 conj(u2))[2c] + (u1 conj(u2))[2c+1],
// c = j looksac + k, i over the looksdn input lines of L (crossmul.f90:155-172);
// amp likewise with (|u1|^2, |u2|^2), then (sqrt re, sqrt im) (:173); both
// zeroed where |sum of the raw input over the look window| <= 1e-6 in either
// image (crossmul.f90:112-125, 176-184).  Sums run in FP32 as the reference's
// complex*8 and in its order (reclaim, then down, then across), but that
// odd_stack_kernel forms the reclaim's sum as one chain of FMAs, the odd
// sample's products last.
//
// The transforms.  The forward and inverse transforms of steps 2-4 cancel at
// the even upsampled samples: u[2n] = x_s[n] / 2 (x_s = in * scale).  The odd
// ones are u[2n + 1] = the inverse nnn-point transform, evaluated half a
// sample on, of the spectrum with the bins from nnn/2 up negated, / nnn / 2: a
// circular convolution of the line, fused in shared memory (fft_conv.cuh,
// HalfSample).  So only odd samples are ever made:
//   * nnn = 64 .. 4,096, looks of one line down: odd_stack_kernel makes a line of each
//     image in turn and forms the pair with the image before from registers;
//     nothing but the images and the results crosses HBM.
//   * otherwise the odd samples go through a scratch array (8 bytes per
//     input sample) and crossmul_looks_kernel forms the looks: for nnn = 64 ..
//     8,192 from odd_kernel, for nnn = 16,384 .. 65,536 from odd_cluster_kernel
//     (a cluster of CTAs per line).
//   * nnn < 64 and nnn > 65,536 (lines of up to 32 or over 65,536 samples), and
//     a plan whose CTA or cluster the device has no room for: the transforms by
//     cuFFT over padded rows.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <cufft.h>

#include <cmath>
#include <mutex>
#include <vector>

#include "../../include/srg_bp.h"
#include "fft_conv.cuh"
#include "host_internal.h"

using namespace srg;
using namespace srg::detail;

namespace {
#define CKC(call)                                                                      \
    do {                                                                               \
        cudaError_t e_ = (call);                                                       \
        if (e_ != cudaSuccess)                                                         \
            return fail(SRG_E_CUDA, "%s failed: %s", #call, cudaGetErrorString(e_));   \
    } while (0)
#define CKF(call)                                                                      \
    do {                                                                               \
        cufftResult r_ = (call);                                                       \
        if (r_ != CUFFT_SUCCESS) return fail(SRG_E_CUDA, "%s failed: cufft %d", #call, (int)r_); \
    } while (0)

// in * scale, zero-padded to nnn, for nl lines
__global__ void pad_scale_kernel(const float2 *__restrict__ in, long long ld, int na, int nnn, int nl,
                                 float scale, float2 *__restrict__ out) {
    const long long total = (long long)nl * nnn;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int l = (int)(i / nnn), n = (int)(i - (long long)l * nnn);
        float2 v = make_float2(0.f, 0.f);
        if (n < na) {
            const float2 x = in[(long long)l * ld + n];
            v = make_float2(x.x * scale, x.y * scale);
        }
        out[i] = v;
    }
}

// nnn-point spectrum -> 2nnn array with the upper half of the bins at the top
__global__ void spread_kernel(const float2 *__restrict__ X, int nnn, int nl, float2 *__restrict__ up) {
    const int n2 = 2 * nnn, h = nnn / 2;
    const long long total = (long long)nl * n2;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int l = (int)(i / n2), m = (int)(i - (long long)l * n2);
        float2 v = make_float2(0.f, 0.f);
        if (m < h) v = X[(long long)l * nnn + m];
        else if (m >= n2 - h) v = X[(long long)l * nnn + (m - nnn)];
        up[i] = v;
    }
}


// a * conj(b)
__device__ __forceinline__ float2 cmul_conj(float2 a, float2 b) {
    return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}

// hypotf(m) <= 1e-6f: decided from the square where that is clear of the
// threshold's square by more than its rounding, which saves the hypotf of
// nearly every sample.
__device__ __forceinline__ bool empty_window(float2 m) {
    const float s = fmaf(m.x, m.x, m.y * m.y);
    if (s < 0.999e-12f) return true;
    if (s > 1.001e-12f) return false;
    return hypotf(m.x, m.y) <= 1.e-6f;
}

// One input column's share of an output sample: (u1 conj(u2)) and the powers
// at its even and odd upsampled samples.
__device__ __forceinline__ void column(float2 a0, float2 a1, float2 b0, float2 b1, float2 &g,
                                       float2 &p) {
    const float2 g0 = cmul_conj(a0, b0), g1 = cmul_conj(a1, b1);
    g = make_float2(g0.x + g1.x, g0.y + g1.y);
    p = make_float2((a0.x * a0.x + a0.y * a0.y) + (a1.x * a1.x + a1.y * a1.y),
                    (b0.x * b0.x + b0.y * b0.y) + (b1.x * b1.x + b1.y * b1.y));
}

// One thread per output sample (L, j); odd upsampled samples of column c at
// odd[l ldo + os c], to be multiplied by of.  Bound by its reads (the images
// and their odd samples once each: 32 bytes per input column of a pair).
__global__ void __launch_bounds__(256)
crossmul_looks_kernel(const float2 *__restrict__ odd1, const float2 *__restrict__ odd2, long long ldo,
                      int os, float of, const float2 *__restrict__ in1,
                      const float2 *__restrict__ in2, long long ld, float scale, int nout_lines,
                      int nout_cols, int looksac, int looksdn, int mask, float2 *__restrict__ igram,
                      float2 *__restrict__ amp) {
    const long long total = (long long)nout_lines * nout_cols;
    for (long long o = blockIdx.x * (long long)blockDim.x + threadIdx.x; o < total;
         o += (long long)gridDim.x * blockDim.x) {
        const int L = (int)(o / nout_cols), j = (int)(o - (long long)L * nout_cols);
        float2 ig = make_float2(0.f, 0.f), am = make_float2(0.f, 0.f);
        float2 m1 = make_float2(0.f, 0.f), m2 = make_float2(0.f, 0.f);
        for (int k = 0; k < looksac; ++k) {
            const int c = j * looksac + k;
            float2 gd = make_float2(0.f, 0.f), ad = make_float2(0.f, 0.f);
            float2 s1 = make_float2(0.f, 0.f), s2 = make_float2(0.f, 0.f);
#pragma unroll 4
            for (int i = 0; i < looksdn; ++i) {
                const long long l = (long long)L * looksdn + i;
                const float2 x1 = __ldg(in1 + l * ld + c), x2 = __ldg(in2 + l * ld + c);
                const float2 u1 = __ldg(odd1 + l * ldo + (long long)os * c),
                             u2 = __ldg(odd2 + l * ldo + (long long)os * c);
                const float2 a0 = make_float2(x1.x * scale * 0.5f, x1.y * scale * 0.5f);
                const float2 b0 = make_float2(x2.x * scale * 0.5f, x2.y * scale * 0.5f);
                float2 g, p;
                column(a0, make_float2(u1.x * of, u1.y * of), b0, make_float2(u2.x * of, u2.y * of), g, p);
                gd.x += g.x;
                gd.y += g.y;
                ad.x += p.x;
                ad.y += p.y;
                s1.x += x1.x;
                s1.y += x1.y;
                s2.x += x2.x;
                s2.y += x2.y;
            }
            ig.x += gd.x;
            ig.y += gd.y;
            am.x += ad.x;
            am.y += ad.y;
            m1.x += s1.x;
            m1.y += s1.y;
            m2.x += s2.x;
            m2.y += s2.y;
        }
        am = make_float2(sqrtf(am.x), sqrtf(am.y));
        if (mask && (empty_window(m1) || empty_window(m2))) {
            ig = make_float2(0.f, 0.f);
            am = make_float2(0.f, 0.f);
        }
        igram[o] = ig;
        amp[o] = am;
    }
}

// The same for looks of LAC = 2 or 4 columns and rows on 16-byte boundaries (even
// row strides): a thread's columns come in 16-byte loads and its columns' sums
// over the lines run side by side, added across in the same order.  Two images
// of 16,504 x 6,646 samples, 4 x 4 looks: 0.57 ms (6.3 TB/s), 0.81 with
// 8-byte loads at a stride of 32.
template <int LAC>
__global__ void __launch_bounds__(256)
crossmul_looks_vec_kernel(const float2 *__restrict__ odd1, const float2 *__restrict__ odd2,
                          long long ldo, float of, const float2 *__restrict__ in1,
                          const float2 *__restrict__ in2, long long ld, float scale, int nout_lines,
                          int nout_cols, int looksdn, int mask, float2 *__restrict__ igram,
                          float2 *__restrict__ amp) {
    constexpr int V = LAC / 2;
    const long long total = (long long)nout_lines * nout_cols;
    const float half = scale * 0.5f;
    for (long long o = blockIdx.x * (long long)blockDim.x + threadIdx.x; o < total;
         o += (long long)gridDim.x * blockDim.x) {
        const int L = (int)(o / nout_cols), j = (int)(o - (long long)L * nout_cols);
        float2 g[LAC], p[LAC], m1[LAC], m2[LAC];
#pragma unroll
        for (int k = 0; k < LAC; ++k) g[k] = p[k] = m1[k] = m2[k] = make_float2(0.f, 0.f);
#pragma unroll 2
        for (int i = 0; i < looksdn; ++i) {
            const long long l = (long long)L * looksdn + i;
            const float4 *r[4] = {reinterpret_cast<const float4 *>(in1 + l * ld + (long long)j * LAC),
                                  reinterpret_cast<const float4 *>(in2 + l * ld + (long long)j * LAC),
                                  reinterpret_cast<const float4 *>(odd1 + l * ldo + (long long)j * LAC),
                                  reinterpret_cast<const float4 *>(odd2 + l * ldo + (long long)j * LAC)};
            float4 q[4][V];
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int v = 0; v < V; ++v) q[a][v] = __ldg(r[a] + v);
#pragma unroll
            for (int k = 0; k < LAC; ++k) {
                auto at = [&](int a) {
                    const float4 w = q[a][k / 2];
                    return k & 1 ? make_float2(w.z, w.w) : make_float2(w.x, w.y);
                };
                const float2 x1 = at(0), x2 = at(1), u1 = at(2), u2 = at(3);
                float2 gg, pp;
                column(make_float2(x1.x * half, x1.y * half), make_float2(u1.x * of, u1.y * of),
                       make_float2(x2.x * half, x2.y * half), make_float2(u2.x * of, u2.y * of), gg, pp);
                g[k] = fftc::cadd(g[k], gg);
                p[k] = fftc::cadd(p[k], pp);
                m1[k] = fftc::cadd(m1[k], x1);
                m2[k] = fftc::cadd(m2[k], x2);
            }
        }
        float2 ig = make_float2(0.f, 0.f), am = ig, s1 = ig, s2 = ig;
#pragma unroll
        for (int k = 0; k < LAC; ++k) {
            ig = fftc::cadd(ig, g[k]);
            am = fftc::cadd(am, p[k]);
            s1 = fftc::cadd(s1, m1[k]);
            s2 = fftc::cadd(s2, m2[k]);
        }
        am = make_float2(sqrtf(am.x), sqrtf(am.y));
        if (mask && (empty_window(s1) || empty_window(s2))) ig = am = make_float2(0.f, 0.f);
        igram[o] = ig;
        amp[o] = am;
    }
}

// Transform plans by line length (nnn).  Threads of a CTA: kThreads, taking
// kThreads / T lines at once, or T where one line needs more.
using P64 = fftc::Plan<64, 16, 8, 4, 2>;
using P128 = fftc::Plan<128, 16, 16, 4, 2>;
using P256 = fftc::Plan<256, 16, 16, 8, 2>;
using P512 = fftc::Plan<512, 16, 16, 16, 2>;
using P1024 = fftc::Plan<1024, 16, 16, 16, 4>;
using P2048 = fftc::Plan<2048, 16, 16, 16, 8>;
using P4096 = fftc::Plan<4096, 16, 16, 16, 16>;
using P8192 = fftc::Plan<8192, 32, 16, 16, 32>;
constexpr int kThreads = 256;
template <class P>
__host__ __device__ constexpr int lines_per_cta() {
    return P::T >= kThreads ? 1 : kThreads / P::T;
}
template <class P>
__host__ __device__ constexpr int cta_threads() {
    return P::T * lines_per_cta<P>();
}

// Twiddle tables of a plan on the device, forward then half-sample inverse:
// kept in shared memory up to 4,096 points (32.6 KB a direction), read through
// L1 at 8,192, where the line itself takes 66 KB and two CTAs share an SM.
template <class P>
__host__ __device__ constexpr int table_entries() {  // one direction
    return P::TW1 + P::TW2;
}
template <class P>
__host__ __device__ constexpr bool tables_in_smem() {
    return P::M <= 4096;
}
template <class P>
__host__ __device__ constexpr int odd_smem() {
    return (int)sizeof(float2) *
           (lines_per_cta<P>() * P::BUF + (tables_in_smem<P>() ? 2 * table_entries<P>() : 0));
}
template <class P>
std::vector<float2> plan_tables() {
    std::vector<float2> all = fftc::tables<P>(0.0), inv = fftc::tables<P>(0.5);
    all.insert(all.end(), inv.begin(), inv.end());
    return all;
}

// What the odd samples are to be multiplied by for the transforms' gain
// (fft_conv.cuh), to the 1.2e-7 of a factor next to 1; C > 1: odd_cluster_kernel's.
template <class P, int C = 1>
__host__ __device__ constexpr float odd_correction() {
    constexpr double gain = fftc::conv_gain<P>() + fftc::half_sample_gain<P>() + fftc::dft_gain<C>();
    return (float)(1.0 / (1.0 + gain));
}

// The odd upsampled samples (unnormalised) of the line in v.
template <class P>
__device__ __forceinline__ void odd_samples(float2 (&v)[P::EPT], float2 *buf, int j, int slot,
                                            bool alone, const float2 *tab) {
    const float2 *inv = tab + table_entries<P>();
    fftc::conv<P>(v, buf, j, slot, alone, fftc::Tw1<P>{tab}, tab + P::TW1, fftc::Tw1<P>{inv},
                  inv + P::TW1, fftc::HalfSample<P>{});
}

template <class P, bool STREAM>
__device__ __forceinline__ void load_line(float2 (&v)[P::EPT], const float2 *__restrict__ x, int j,
                                          int na) {
    x += j;
    na -= j;
#pragma unroll
    for (int i = 0; i < P::EPT; ++i) {
        const int n = fftc::point_of<P>(i);
        v[i] = n < na ? (STREAM ? fftc::ld_stream(x + n) : __ldg(x + n)) : make_float2(0.f, 0.f);
    }
}

// Odd samples of every line of one or two images, of in * scale (multiplied
// first, as the reference does: a scale may bring samples into range that the
// sums of a line would leave) and not yet / nnn / 2, into odd[0], odd[1]
// ([nl][na]).  Launch and latency bound at small sizes: a 917 x 601 pair
// with looks takes 19 us in two launches (72 us in seven with cuFFT).  Persistent, kThreads / T lines of a CTA at once.
struct OddArgs {
    const float2 *in[2];
    float2 *odd[2];
};
template <class P>
__global__ void __launch_bounds__(cta_threads<P>(), 2)
odd_kernel(const __grid_constant__ OddArgs a, int nimg, long long ld, int na, int nl, float scale,
           const float2 *__restrict__ tabg) {
    extern __shared__ float2 xm_sm[];
    constexpr int LP = lines_per_cta<P>();
    const int slot = threadIdx.x / P::T, j = threadIdx.x % P::T;
    float2 *buf = xm_sm + slot * P::BUF;
    const float2 *tab = tabg;
    if constexpr (tables_in_smem<P>()) {
        float2 *t = xm_sm + LP * P::BUF;
        for (int i = threadIdx.x; i < 2 * table_entries<P>(); i += cta_threads<P>()) t[i] = __ldg(tabg + i);
        tab = t;
        __syncthreads();
    }
    const long long items = (long long)nimg * nl;
    for (long long base = (long long)blockIdx.x * LP; base < items; base += (long long)gridDim.x * LP) {
        const long long item = base + slot;
        const bool mine = item < items;
        const int k = mine && item >= nl ? 1 : 0;
        const long long l = mine ? item - (long long)k * nl : 0;
        float2 v[P::EPT];
        load_line<P, !tables_in_smem<P>()>(v, a.in[k] + l * ld, j, mine ? na : 0);
#pragma unroll
        for (int i = 0; i < P::EPT; ++i) v[i] = make_float2(v[i].x * scale, v[i].y * scale);
        odd_samples<P>(v, buf, j, slot, LP == 1, tab);
        float2 *out = a.odd[k] + l * na + j;
        const int nm = mine ? na - j : 0;
#pragma unroll
        for (int i = 0; i < P::EPT; ++i) {
            const int n = fftc::point_of<P>(i);
            if (n < nm) out[n] = v[i];
        }
        fftc::line_sync<P>(slot, LP == 1);  // the buffer's reads are done
    }
}

// The same for nnn = C M, M = 8,192: a line is too long for an SM, so a cluster
// of C CTAs takes it.  With w = exp(-2 pi i / nnn), the bins k = C m + q of the
// line's transform are the M-point transform of
//   a_q[n] = w^(q n) sum_c x[n + c M] exp(-2 pi i q c / C),
// which CTA q makes from global memory; the half-sample convolution of a_q
// (HalfSample: the upper half of the bins m is the upper half of the bins k),
// times exp(2 pi i q (n + 1/2) / nnn), is z_q, and
//   y[n + c M] = sum_q exp(2 pi i q c / C) z_q[n]:
// each CTA takes the n of M / C columns, reads the z_q there from all CTAs
// through distributed shared memory and writes C outputs per n.  So one
// exchange per line, of the line's size, and two CTAs of different lines share
// an SM.  Bound by instruction issue (53 % of the cycles) and the latency of
// its loads: two images of 16,504 x 6,646 samples take 3.75 ms, where padding,
// cuFFT's transforms of 32,768 and 65,536 points and the spread took 12.0; a
// cluster of two with 16,384 points each, alone on its SMs, took 5.3.  The
// grid is what the chip holds of clusters at once (with more, the last ones
// ran alone: 7.5 ms).  The items are the same in every CTA of a cluster, so all
// reach every cluster barrier.
// Table tabg: the plan's, then exp(-2 pi i q j / nnn) and exp(2 pi i q
// (j + 1/2) / nnn), [q][j], then exp(-2 pi i m / (nnn / T)), m < 32 C.
__device__ __forceinline__ float2 ld_cluster(unsigned addr) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr));
    return v;
}

template <int C>
__global__ void __launch_bounds__(P8192::T, 2)
odd_cluster_kernel(const __grid_constant__ OddArgs a, int nimg, long long ld, int na, int nl,
                   float scale, const float2 *__restrict__ tabg) {
    using P = P8192;
    namespace cg = cooperative_groups;
    extern __shared__ float2 xm_sm[];
    float2 *buf = xm_sm, *turn = xm_sm + P::BUF;  // turn[m] = exp(-2 pi i q m / (32 C))
    cg::cluster_group cl = cg::this_cluster();
    const int q = (int)cl.block_rank(), j = threadIdx.x;
    const float2 *own = tabg + 2 * table_entries<P>();
    const float2 *root = own + 2 * C * P::T;
    unsigned peer[C];  // shared-window addresses of the cluster's buffers
#pragma unroll
    for (int e = 0; e < C; ++e)
        asm("mapa.shared::cluster.u32 %0, %1, %2;"
            : "=r"(peer[e])
            : "r"((unsigned)__cvta_generic_to_shared(buf)), "r"(e));
    if (j < P::EPT) turn[j] = __ldg(root + (q * j) % (P::EPT * C));
    __syncthreads();
    const float2 pre = __ldg(own + q * P::T + j), post = __ldg(own + (C + q) * P::T + j);
    const long long items = (long long)nimg * nl;
    for (long long item = blockIdx.x / C; item < items; item += gridDim.x / C) {
        const int k = item >= nl ? 1 : 0;
        const long long l = item - (long long)k * nl;
        const float2 *x = a.in[k] + l * ld;
        float2 v[P::EPT];
        load_line<P, true>(v, x, j, na);
#pragma unroll
        for (int i = 0; i < P::EPT; ++i) v[i] = make_float2(v[i].x * scale, v[i].y * scale);
        if (item + gridDim.x / C < items) {  // this CTA's share of the next line into L2
            const long long ni = item + gridDim.x / C;
            const float2 *nx = ni >= nl ? a.in[1] + (ni - nl) * ld : a.in[0] + ni * ld;
            for (int c = 16 * (q * P::T + j); c < na; c += 16 * P::T * C)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(nx + c));
        }
#pragma unroll 1
        for (int c = 1; c < C; ++c) {
            if (c * P::M >= na) break;
            // scale exp(-2 pi i q c / C)
            const float2 w1 = __ldg(root + (q * c * P::EPT) % (P::EPT * C));
            const float2 wc = make_float2(w1.x * scale, w1.y * scale);
#pragma unroll
            for (int m0 = 0; m0 < P::EPT; m0 += 16) {  // in the order of the line
                if (m0 * P::T + c * P::M >= na) break;
                float2 b[16];
#pragma unroll
                for (int m = 0; m < 16; ++m) {
                    const int n = (m0 + m) * P::T + c * P::M;
                    b[m] = n < na - j ? fftc::ld_stream(x + j + n) : make_float2(0.f, 0.f);
                }
#pragma unroll
                for (int m = 0; m < 16; ++m) {  // point_of<P>(i) = (m0 + m) T
                    const int i = (m0 + m) % P::GA * P::RA + (m0 + m) / P::GA;
                    v[i] = fftc::cadd(v[i], fftc::cmul(b[m], wc));
                }
            }
        }
        if (q) {
#pragma unroll
            for (int i = 0; i < P::EPT; ++i)
                v[i] = fftc::cmul(v[i], fftc::cmul(pre, turn[fftc::point_of<P>(i) / P::T]));
        }
        // every CTA's reads of the line before are done
        if (item != blockIdx.x / C) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        odd_samples<P>(v, buf, j, 0, true, tabg);
        __syncthreads();  // the buffer's reads are done
#pragma unroll
        for (int i = 0; i < P::EPT; ++i) {
            if (q) v[i] = fftc::cmul(v[i], fftc::cmulc(post, turn[fftc::point_of<P>(i) / P::T]));
            buf[P::pad(j + fftc::point_of<P>(i))] = v[i];
        }
        cl.sync();
        float2 *out = a.odd[k] + l * na;
#pragma unroll
        for (int i = 0; i < P::EPT / C; ++i) {
            const int n = j + (q * (P::EPT / C) + i) * P::T;
            if (n >= na) break;
            float2 z[C];
#pragma unroll
            for (int e = 0; e < C; ++e) z[e] = ld_cluster(peer[e] + P::pad(n) * (int)sizeof(float2));
            fftc::dft<C, true>(z);
#pragma unroll
            for (int c = 0; c < C; ++c)
                if (n + c * P::M < na) out[n + c * P::M] = z[fftc::brev<C>(c)];
        }
        // this CTA's reads are done: the others may write their buffers again
        // (waited for behind the next line's loads)
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    }
    // no CTA leaves while another reads its buffer
    if (blockIdx.x / C < items) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// A whole stack with looks of one line down, nnn = M <= 4,096: per grid line each
// image's odd samples are made in turn and paired with those of the image
// before, still in the thread's registers (its even samples are read again
// from the input).  The images are read and the results written once.  Bound by
// instruction issue and latency (two CTAs of 256 threads per SM, by their
// registers): 32 images of 2,400 x 1,200 samples take 0.96 ms, 2.66 with
// self-sorting transforms of two lines per 512-thread CTA; of that, dealing
// the steps evenly gave 12 %, reading the even samples in batches of four and
// keeping each image's amplitudes another 10 %.
// Images of one launch (its pointers travel as a kernel parameter, 1.5 KB):
// longer stacks go in launches of up to kXmChunk images overlapping by one.
constexpr int kXmChunk = 64;
struct StackPtrs {
    const float2 *img[kXmChunk];
    float2 *ig[kXmChunk - 1], *am[kXmChunk - 1];
};
// The steps (line l, image k), l n + k, are dealt to `workers` lines of
// threads in contiguous runs of equal length, so that no SM waits for the
// last line of a whole stack; a run that starts inside a line makes the image
// before it once more.
constexpr int kBatch = 4;
// ACROSS: looks of `looksac` columns (one line down), nout per line.
template <class P, bool ACROSS>
__global__ void __launch_bounds__(cta_threads<P>(), 2)
odd_stack_kernel(const __grid_constant__ StackPtrs p, int n, long long ld, int na, int nlines,
                 int looksac, int nout, float scale, int mask, int workers,
                 const float2 *__restrict__ tabg) {
    extern __shared__ float2 xm_sm[];
    constexpr int LP = lines_per_cta<P>(), NT = cta_threads<P>();
    const int slot = threadIdx.x / P::T, j = threadIdx.x % P::T;
    float2 *buf = xm_sm + slot * P::BUF;
    float2 *tab = xm_sm + LP * P::BUF;
    for (int i = threadIdx.x; i < 2 * table_entries<P>(); i += NT) tab[i] = __ldg(tabg + i);
    __syncthreads();
    // results / nnn / 2: powers of two, applied to the input for the odd samples
    const float odd_scale = scale * (0.5f / (float)P::M * odd_correction<P>()), even_scale = scale * 0.5f;
    const long long steps = (long long)nlines * n;
    const int w = blockIdx.x * LP + slot;
    const long long s0 = w < workers ? steps * w / workers : 0;
    const long long s1 = w < workers ? steps * (w + 1) / workers : 0;
    long long l = s0 / n;
    int k = (int)(s0 - l * n);
    const int prime = k > 0 && s1 > s0 ? 1 : 0;
    k -= prime;
    // lines of one warp take the same number of turns (their barrier is the warp's)
    const int turns = P::T <= 32 ? (int)((steps + workers - 1) / workers) + 1 : (int)(s1 - s0) + prime;
    const int mine = (int)(s1 - s0) + prime;
    // the image before: odd samples, amplitudes, empty samples (bit i)
    float2 v[P::EPT], prev[P::EPT];
    float amp[P::EPT];
    unsigned empty = 0;
#pragma unroll
    for (int i = 0; i < P::EPT; ++i) {
        prev[i] = make_float2(0.f, 0.f);
        amp[i] = 0.f;
    }
    for (int t = 0; t < turns; ++t) {
        const int nm = t < mine ? na : 0;
        const long long row = t < mine ? l * ld : 0;
        load_line<P, false>(v, p.img[k] + row, j, nm);
#pragma unroll
        for (int i = 0; i < P::EPT; ++i) v[i] = make_float2(v[i].x * odd_scale, v[i].y * odd_scale);
        if (t + 1 < mine) {  // the next step's line into L2
            const float2 *nx = k + 1 < n ? p.img[k + 1] + row : p.img[0] + row + ld;
            for (int c = 16 * j; c < na; c += 16 * P::T)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(nx + c));
        }
        odd_samples<P>(v, buf, j, slot, LP == 1, tab);
        const bool pair = k > 0 && t >= prime;
        const float2 *x1 = p.img[pair ? k - 1 : k] + row, *x2 = p.img[k] + row;
        float2 *ig = p.ig[pair ? k - 1 : 0] + l * nout, *am = p.am[pair ? k - 1 : 0] + l * nout;
        if constexpr (!ACROSS) {
            const int nj = nm - j;
#pragma unroll
            for (int h = 0; h < P::EPT; h += kBatch) {  // a batch of loads in flight
                if (P::RA == P::EPT && h * P::T >= na) break;  // no column left
                float2 e1[kBatch], e2[kBatch];
#pragma unroll
                for (int i = 0; i < kBatch; ++i) {
                    const int c = fftc::point_of<P>(h + i);
                    e1[i] = e2[i] = make_float2(0.f, 0.f);
                    if (c < nj) {
                        e1[i] = __ldg(x1 + j + c);
                        e2[i] = __ldg(x2 + j + c);
                    }
                }
#pragma unroll
                for (int i = 0; i < kBatch; ++i) {
                    const int c = fftc::point_of<P>(h + i);
                    const bool none = mask && empty_window(e2[i]);
                    const float2 f1 = make_float2(e1[i].x * even_scale, e1[i].y * even_scale);
                    const float2 f2 = make_float2(e2[i].x * even_scale, e2[i].y * even_scale);
                    const float2 o1 = prev[h + i], o2 = v[h + i];
                    const float p2 =
                        sqrtf(fmaf(o2.x, o2.x, fmaf(o2.y, o2.y, fmaf(f2.x, f2.x, f2.y * f2.y))));
                    float2 g = make_float2(
                        fmaf(o1.x, o2.x, fmaf(o1.y, o2.y, fmaf(f1.x, f2.x, f1.y * f2.y))),
                        fmaf(o1.y, o2.x, fmaf(-o1.x, o2.y, fmaf(f1.y, f2.x, -f1.x * f2.y))));
                    float2 a = make_float2(amp[h + i], p2);
                    if (none || (empty >> (h + i) & 1)) g = a = make_float2(0.f, 0.f);
                    if (pair && c < nj) {
                        ig[j + c] = g;
                        am[j + c] = a;
                    }
                    amp[h + i] = p2;
                    empty = none ? empty | 1u << (h + i) : empty & ~(1u << (h + i));
                    prev[h + i] = o2;
                }
            }
        } else {
            // sums across the columns of a look, through the line's buffer:
            // the products first, then the powers
            fftc::line_sync<P>(slot, LP == 1);  // the buffer's reads are done
            float p2[P::EPT];
#pragma unroll
            for (int i = 0; i < P::EPT; ++i) {
                const int c = j + fftc::point_of<P>(i);
                const float2 o1 = prev[i], o2 = v[i];
                float2 f1 = make_float2(0.f, 0.f), f2 = f1;
                if (c < nm) {
                    f1 = __ldg(x1 + c);
                    f2 = __ldg(x2 + c);
                }
                f1 = make_float2(f1.x * even_scale, f1.y * even_scale);
                f2 = make_float2(f2.x * even_scale, f2.y * even_scale);
                p2[i] = fmaf(o2.x, o2.x, fmaf(o2.y, o2.y, fmaf(f2.x, f2.x, f2.y * f2.y)));
                buf[P::pad(c)] = make_float2(
                    fmaf(o1.x, o2.x, fmaf(o1.y, o2.y, fmaf(f1.x, f2.x, f1.y * f2.y))),
                    fmaf(o1.y, o2.x, fmaf(-o1.x, o2.y, fmaf(f1.y, f2.x, -f1.x * f2.y))));
                prev[i] = o2;
            }
            fftc::line_sync<P>(slot, LP == 1);
            float2 g[P::EPT / 2];
#pragma unroll
            for (int i = 0; i < P::EPT / 2; ++i) {
                const int o = j + i * P::T;
                g[i] = make_float2(0.f, 0.f);
                if (o < nout)
                    for (int e = 0; e < looksac; ++e) g[i] = fftc::cadd(g[i], buf[P::pad(o * looksac + e)]);
            }
            fftc::line_sync<P>(slot, LP == 1);
#pragma unroll
            for (int i = 0; i < P::EPT; ++i) buf[P::pad(j + fftc::point_of<P>(i))].x = p2[i];
            fftc::line_sync<P>(slot, LP == 1);
#pragma unroll
            for (int i = 0; i < P::EPT / 2; ++i) {
                const int o = j + i * P::T;
                if (o >= nout || nm == 0) continue;
                float s = 0.f;
                float2 m = make_float2(0.f, 0.f);
                for (int e = 0; e < looksac; ++e) {
                    s += buf[P::pad(o * looksac + e)].x;
                    m = fftc::cadd(m, __ldg(x2 + o * looksac + e));
                }
                s = sqrtf(s);
                const bool none = mask && empty_window(m);
                if (pair) {
                    const bool zero = none || (empty >> i & 1);
                    ig[o] = zero ? make_float2(0.f, 0.f) : g[i];
                    am[o] = zero ? make_float2(0.f, 0.f) : make_float2(amp[i], s);
                }
                amp[i] = s;
                empty = none ? empty | 1u << i : empty & ~(1u << i);
            }
        }
        if (++k == n) {
            k = 0;
            ++l;
        }
        fftc::line_sync<P>(slot, LP == 1);  // the buffer's reads are done
    }
}

struct Plan {
    int n = 0, batch = 0;
    cufftHandle h = 0;
    bool ok = false;
};

// The kernels and tables of one line length.
struct OwnPlan {
    int nnn;
    const void *odd;    // odd_kernel or odd_cluster_kernel
    const void *stack;  // odd_stack_kernel for single looks, or null
    const void *across; // the same for looks of several columns, one line down
    int threads, lines, smem, cluster;
    float correction;   // odd_correction
    std::vector<float2> (*tables)();
};
template <int C>
std::vector<float2> cluster_tables() {  // odd_cluster_kernel's
    std::vector<float2> t = plan_tables<P8192>();
    const double tau = 8.0 * std::atan2(1.0, 1.0), nnn = (double)C * P8192::M;
    auto add = [&](double x) { t.push_back(make_float2((float)std::cos(tau * x), (float)std::sin(tau * x))); };
    for (int q = 0; q < C; ++q)
        for (int j = 0; j < P8192::T; ++j) add(-(double)q * j / nnn);
    for (int q = 0; q < C; ++q)
        for (int j = 0; j < P8192::T; ++j) add(q * (j + 0.5) / nnn);
    for (int m = 0; m < P8192::EPT * C; ++m) add(-(double)m / (P8192::EPT * C));
    return t;
}
template <class P>
OwnPlan small_plan() {
    return {P::M, (const void *)odd_kernel<P>, (const void *)odd_stack_kernel<P, false>,
            (const void *)odd_stack_kernel<P, true>, cta_threads<P>(),
            lines_per_cta<P>(), odd_smem<P>(), 1, odd_correction<P>(), plan_tables<P>};
}
template <int C>
OwnPlan cluster_plan() {
    return {C * P8192::M, (const void *)odd_cluster_kernel<C>, nullptr, nullptr, P8192::T, 1,
            (int)sizeof(float2) * (P8192::BUF + P8192::EPT), C, odd_correction<P8192, C>(), cluster_tables<C>};
}
constexpr int kOwnPlans = 11;
const OwnPlan *own_plans() {
    static const OwnPlan plans[kOwnPlans] = {
        small_plan<P64>(), small_plan<P128>(), small_plan<P256>(), small_plan<P512>(),
        small_plan<P1024>(), small_plan<P2048>(), small_plan<P4096>(),
        {P8192::M, (const void *)odd_kernel<P8192>, nullptr, nullptr, P8192::T, 1, odd_smem<P8192>(), 1,
         odd_correction<P8192>(), plan_tables<P8192>},
        cluster_plan<2>(), cluster_plan<4>(), cluster_plan<8>()};
    return plans;
}
int own_plan_of(int nnn) {
    for (int i = 0; i < kOwnPlans; ++i)
        if (own_plans()[i].nnn == nnn) return i;
    return -1;
}

struct XmCtx {
    std::mutex mu;
    Plan fwd, inv;
    DevBuf pad, upA, upB;
    // per own plan: tables on the device, resident CTAs of the kernels
    DevBuf tab[kOwnPlans];
    int odd_ctas[kOwnPlans] = {}, stack_ctas[kOwnPlans] = {}, across_ctas[kOwnPlans] = {};
    bool ready[kOwnPlans] = {}, unfit[kOwnPlans] = {};  // unfit: does not fit the device's SMs
    bool own_off = false;  // srg_test_crossmul_own
};
XmCtx g_xm[64];

int plan_for(Plan &p, int n, int batch) {
    if (p.ok && p.n == n && p.batch == batch) return SRG_OK;
    if (p.ok) cufftDestroy(p.h);
    p.ok = false;
    CKF(cufftPlan1d(&p.h, n, CUFFT_C2C, batch));
    p.n = n;
    p.batch = batch;
    p.ok = true;
    return SRG_OK;
}

int grid_for(long long n) {
    long long g = (n + 255) / 256;
    return (int)std::min<long long>(g, 148LL * 32);
}

void cluster_config(const OwnPlan &p, int grid, cudaStream_t st, cudaLaunchConfig_t &cfg,
                    cudaLaunchAttribute &at) {
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)p.cluster;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(p.threads);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = p.cluster > 1 ? 1 : 0;
}

// Tables and launch limits of own plan `i` on the current device (made once),
// or unfit[i].
int ensure_plan(XmCtx &x, int i, int dev, cudaStream_t st) {
    if (x.ready[i] || x.unfit[i]) return SRG_OK;
    const OwnPlan &p = own_plans()[i];
    const std::vector<float2> t = p.tables();
    int rc = x.tab[i].ensure(sizeof(float2) * t.size());
    if (rc) return rc;
    int sms = 0;
    CKC(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    for (const void *fn : {p.odd, p.stack, p.across}) {
        if (!fn) continue;
        CKC(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, p.smem));
        int ctas = 0;
        if (p.cluster > 1) {  // clusters that the chip holds at once
            cudaLaunchConfig_t cfg{};
            cudaLaunchAttribute at{};
            cluster_config(p, sms * p.cluster, 0, cfg, at);
            if (cudaOccupancyMaxActiveClusters(&ctas, fn, &cfg) != cudaSuccess) {
                ctas = 0;  // a part of a device may be too small for the cluster
                cudaGetLastError();
            }
            ctas *= p.cluster;
        } else {
            CKC(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctas, fn, p.threads, p.smem));
            ctas *= sms;
        }
        if (ctas < 1) {
            x.unfit[i] = true;
            return SRG_OK;
        }
        (fn == p.odd ? x.odd_ctas : fn == p.stack ? x.stack_ctas : x.across_ctas)[i] = ctas;
    }
    CKC(cudaMemcpyAsync(x.tab[i].p, t.data(), sizeof(float2) * t.size(), cudaMemcpyHostToDevice, st));
    CKC(cudaStreamSynchronize(st));  // `t` is pageable host memory that goes out of scope
    x.ready[i] = true;
    return SRG_OK;
}

// odd samples of nimg (1 or 2) images by own plan `i`
int launch_odd(XmCtx &x, int i, OddArgs a, int nimg, long long ld, int na, int nl, float scale,
               cudaStream_t st) {
    const OwnPlan &p = own_plans()[i];
    const long long groups = ((long long)nimg * nl + p.lines - 1) / p.lines;
    const float2 *tab = static_cast<const float2 *>(x.tab[i].p);
    void *args[] = {&a, &nimg, &ld, &na, &nl, &scale, (void *)&tab};
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at{};
    cluster_config(p, (int)std::min<long long>(groups * p.cluster, x.odd_ctas[i]), st, cfg, at);
    CKC(cudaLaunchKernelExC(&cfg, p.odd, args));
    return SRG_OK;
}

// upsampled lines of one image into `up` (nl x 2nnn) by cuFFT
int upsample(XmCtx &x, const float2 *in, long long ld, int na, int nnn, int nl, float scale,
             float2 *up, cudaStream_t st) {
    float2 *pad = static_cast<float2 *>(x.pad.p);
    pad_scale_kernel<<<grid_for((long long)nl * nnn), 256, 0, st>>>(in, ld, na, nnn, nl, scale, pad);
    CKC(cudaGetLastError());
    CKF(cufftSetStream(x.fwd.h, st));
    CKF(cufftExecC2C(x.fwd.h, reinterpret_cast<cufftComplex *>(pad),
                     reinterpret_cast<cufftComplex *>(pad), CUFFT_FORWARD));
    spread_kernel<<<grid_for((long long)nl * 2 * nnn), 256, 0, st>>>(pad, nnn, nl, up);
    CKC(cudaGetLastError());
    CKF(cufftSetStream(x.inv.h, st));
    CKF(cufftExecC2C(x.inv.h, reinterpret_cast<cufftComplex *>(up),
                     reinterpret_cast<cufftComplex *>(up), CUFFT_INVERSE));
    return SRG_OK;
}

int check_args(long long ld, int na, int nlines, int looksac, int looksdn) {
    if (na < 1 || ld < na || nlines < 1 || looksac < 1 || looksdn < 1)
        return fail(SRG_E_ARG, "bad crossmul sizes: na=%d ld=%lld nlines=%d looks=%d x %d", na, ld,
                    nlines, looksac, looksdn);
    if (na / looksac < 1 || nlines / looksdn < 1)
        return fail(SRG_E_ARG, "looks %d x %d exceed the image %d x %d", looksac, looksdn, na, nlines);
    if (na > (1 << 24)) return fail(SRG_E_ARG, "line of %d samples exceeds 2^24", na);
    return SRG_OK;
}

int fft_length(int na) {  // crossmul.f90:69-73: first 2^i >= na, i = 1..24
    int n = 2;
    while (n < na) n *= 2;
    return n;
}

int run_stack(const float *const *slcs, int n, long long ld, int na, int nlines, int looksac,
              int looksdn, float scale, int mask, float *const *igrams, float *const *amps,
              void *stream) {
    int rc = check_args(ld, na, nlines, looksac, looksdn);
    if (rc) return rc;
    if (n < 2 || !slcs || !igrams || !amps) return fail(SRG_E_ARG, "need >= 2 images and outputs");
    for (int k = 0; k < n; ++k)
        if (!slcs[k]) return fail(SRG_E_ARG, "null image %d", k);
    for (int k = 0; k + 1 < n; ++k)
        if (!igrams[k] || !amps[k]) return fail(SRG_E_ARG, "null output of pair %d", k);
    int dev = 0;
    CKC(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(SRG_E_ARG, "device %d out of range", dev);
    XmCtx &x = g_xm[dev];
    std::lock_guard<std::mutex> g(x.mu);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int nnn = fft_length(na);
    const int nout_lines = nlines / looksdn, nout_cols = na / looksac;
    const int nl = nout_lines * looksdn;
    int own = x.own_off ? -1 : own_plan_of(nnn);
    if (own >= 0) {
        if ((rc = ensure_plan(x, own, dev, st))) return rc;
        if (x.unfit[own]) own = -1;  // cuFFT runs anywhere
    }
    if (own >= 0) {
        const OwnPlan &op = own_plans()[own];
        // (odd_stack_kernel takes scale / nnn / 2 as one factor, which must be a
        // normal number)
        if (op.stack && looksdn == 1 && (std::fabs(scale) >= 1e-30f || scale == 0.f)) {
            const void *fn = looksac == 1 ? op.stack : op.across;
            const int ctas = (looksac == 1 ? x.stack_ctas : x.across_ctas)[own];
            const float2 *tab = static_cast<const float2 *>(x.tab[own].p);
            for (int k0 = 0; k0 + 1 < n; k0 += kXmChunk - 1) {
                int m = std::min(kXmChunk, n - k0);
                // runs of at least four steps, or whole lines
                const long long want = std::max<long long>(nout_lines, (long long)nout_lines * m / 4);
                int workers = (int)std::min<long long>(want, (long long)ctas * op.lines);
                const int grid = (workers + op.lines - 1) / op.lines;
                StackPtrs p{};
                for (int k = 0; k < m; ++k) p.img[k] = reinterpret_cast<const float2 *>(slcs[k0 + k]);
                for (int k = 0; k + 1 < m; ++k) {
                    p.ig[k] = reinterpret_cast<float2 *>(igrams[k0 + k]);
                    p.am[k] = reinterpret_cast<float2 *>(amps[k0 + k]);
                }
                int lines = nout_lines, lac = looksac, cols = nout_cols;
                void *args[] = {&p, &m, &ld, &na, &lines, &lac, &cols, &scale, &mask, &workers, (void *)&tab};
                CKC(cudaLaunchKernel(fn, dim3(grid), dim3(op.threads), args, op.smem, st));
            }
            return SRG_OK;
        }
    } else if ((rc = plan_for(x.fwd, nnn, nl)) || (rc = plan_for(x.inv, 2 * nnn, nl)) ||
               (rc = x.pad.ensure((size_t)nl * nnn * sizeof(float2)))) {
        return rc;
    }
    // odd samples of two images in turn: [nl][na] from the library's own
    // transforms, every second sample of [nl][2 nnn] from cuFFT's
    const size_t up_bytes = (size_t)nl * (own >= 0 ? na : 2 * nnn) * sizeof(float2);
    if ((rc = x.upA.ensure(up_bytes)) || (rc = x.upB.ensure(up_bytes))) return rc;
    float2 *cur = static_cast<float2 *>(x.upA.p), *nxt = static_cast<float2 *>(x.upB.p);
    const int off = own >= 0 ? 0 : 1, os = own >= 0 ? 1 : 2;
    const long long ldo = own >= 0 ? na : 2LL * nnn;
    // the reference's divisions (by a power of two)
    const float of = 0.5f / (float)nnn * (own >= 0 ? own_plans()[own].correction : 1.f);
    for (int k = 0; k + 1 < n; ++k) {
        const float2 *a = reinterpret_cast<const float2 *>(slcs[k]);
        const float2 *b = reinterpret_cast<const float2 *>(slcs[k + 1]);
        const bool same = a == b;
        if (own >= 0) {
            OddArgs oa{};
            int m = 0;
            if (k == 0) {
                oa.in[m] = a;
                oa.odd[m++] = cur;
            }
            if (!same) {
                oa.in[m] = b;
                oa.odd[m++] = nxt;
            }
            if (m && (rc = launch_odd(x, own, oa, m, ld, na, nl, scale, st))) return rc;
        } else {
            if (k == 0 && (rc = upsample(x, a, ld, na, nnn, nl, scale, cur, st))) return rc;
            if (!same && (rc = upsample(x, b, ld, na, nnn, nl, scale, nxt, st))) return rc;
        }
        const float2 *o1 = cur + off, *o2 = (same ? cur : nxt) + off;
        float2 *ig = reinterpret_cast<float2 *>(igrams[k]), *am = reinterpret_cast<float2 *>(amps[k]);
        const int grid = grid_for((long long)nout_lines * nout_cols);
        const bool rows16 = own >= 0 && !((ld | ldo) & 1) &&
                            !((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15);
        if (rows16 && looksac == 4)
            crossmul_looks_vec_kernel<4><<<grid, 256, 0, st>>>(o1, o2, ldo, of, a, b, ld, scale, nout_lines,
                                                               nout_cols, looksdn, mask, ig, am);
        else if (rows16 && looksac == 2)
            crossmul_looks_vec_kernel<2><<<grid, 256, 0, st>>>(o1, o2, ldo, of, a, b, ld, scale, nout_lines,
                                                               nout_cols, looksdn, mask, ig, am);
        else
            crossmul_looks_kernel<<<grid, 256, 0, st>>>(o1, o2, ldo, os, of, a, b, ld, scale, nout_lines,
                                                        nout_cols, looksac, looksdn, mask, ig, am);
        CKC(cudaGetLastError());
        if (!same) std::swap(cur, nxt);
    }
    return SRG_OK;
}

}  // namespace

extern "C" {

int srg_test_crossmul_own(int use) {
    int dev = 0;
    CKC(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(SRG_E_ARG, "device %d out of range", dev);
    std::lock_guard<std::mutex> g(g_xm[dev].mu);
    g_xm[dev].own_off = !use;
    return SRG_OK;
}

int srg_crossmul_device(const float *slc1, const float *slc2, long long ld, int na, int nlines,
                        int looksac, int looksdn, float scale, int mask, float *igram, float *amp,
                        void *stream) {
    const float *s[2] = {slc1, slc2};
    float *ig[1] = {igram};
    float *am[1] = {amp};
    return run_stack(s, 2, ld, na, nlines, looksac, looksdn, scale, mask, ig, am, stream);
}

int srg_crossmul_stack_device(const float *const *slcs, int n, long long ld, int na, int nlines,
                              int looksac, int looksdn, float scale, int mask, float *const *igrams,
                              float *const *amps, void *stream) {
    return run_stack(slcs, n, ld, na, nlines, looksac, looksdn, scale, mask, igrams, amps, stream);
}

}  // extern "C"
