// fft_conv.cuh -- circular convolutions of complex64 lines by FFT in shared
// memory, for interferogram formation (crossmul.cu) and range compression
// (rangecomp.cu): forward transform, a multiplication of the spectrum,
// inverse transform, of M = 64 ... 8,192 points, each thread holding EPT
// (16 or 32) of them in registers between shared-memory exchanges.
//
// M = RA RB RC.  The forward transform is a decimation in frequency over the
// digits n = n0 RB RC + n1 RC + n2: a DFT over n0 (pass 1), times
// w_M^(k0 (n1 RC + n2)), a DFT over n1 (pass 2), times w_(RB RC)^(k1 n2), a DFT
// over n2.  Every pass writes where it read, so the spectrum ends in digit
// order (bin k = k0 + RA k1 + RA RB k2 at k0 RB RC + k1 RC + k2) and the
// inverse (a decimation in time) undoes the passes in turn, back to the
// natural order.  Two things follow, against transforms that sort
// themselves: a pass needs no barrier between its reads and its writes, and
// the last forward pass, the spectrum's multiplication and the first inverse
// pass work on the same RC contiguous points, in one thread's registers.  A
// line goes through shared memory four times (write and read) with four
// barriers and one more before the buffer is used again; the first pass reads
// global memory and the last one leaves its results in registers.
//
// What bounds it: instruction issue (per 16 points and pass about 208 FP32
// operations, a 16-point DFT in 148 and its twiddles in 60, and 40 others) at
// 55-65 % of the cycles: 16 warps per SM, by their 128 registers, do not cover
// all of the latency of shared memory and barriers.
//
// Buffer layout: index i + i / EPT, which puts the accesses of every pass
// (contiguous over threads, or EPT contiguous points per thread) on distinct
// banks.
//
// Twiddles are exactly rounded entries of tables [r - 1][column], contiguous
// over threads; where a thread has several columns of pass 1 and the caller
// keeps only the first ones' (Tw1: crossmul's 64 and 8,192 points), the others
// are turned from them, which adds a rounding.
#pragma once
#include <cuda_runtime.h>

#include <cmath>
#include <vector>

namespace srg {
namespace fftc {

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
// a * conj(b)
__device__ __forceinline__ float2 cmulc(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, a.y * b.y), fmaf(a.y, b.x, -a.x * b.y));
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }

// cos(2 pi q / 64), q = 0..16
__host__ __device__ constexpr double cos64(int q) {
    return q == 0    ? 1.0
           : q == 1  ? 0.995184726672196886
           : q == 2  ? 0.980785280403230449
           : q == 3  ? 0.956940335732208865
           : q == 4  ? 0.923879532511286756
           : q == 5  ? 0.881921264348355030
           : q == 6  ? 0.831469612302545237
           : q == 7  ? 0.773010453362736961
           : q == 8  ? 0.707106781186547524
           : q == 9  ? 0.634393284163645498
           : q == 10 ? 0.555570233019602225
           : q == 11 ? 0.471396736825997649
           : q == 12 ? 0.382683432365089772
           : q == 13 ? 0.290284677254462368
           : q == 14 ? 0.195090322016128268
           : q == 15 ? 0.098017140329560602
                     : 0.0;
}
__host__ __device__ constexpr double cos_turn64(int q) {  // cos(2 pi q / 64), any q >= 0
    const int m = q & 63;
    return m <= 16 ? cos64(m) : m <= 32 ? -cos64(32 - m) : m <= 48 ? -cos64(m - 32) : cos64(64 - m);
}
__host__ __device__ constexpr double sin_turn64(int q) { return cos_turn64(q + 48); }

// b * exp(-+2 pi i m / 64) (INV: +), m a constant after unrolling
template <bool INV>
__device__ __forceinline__ float2 rot64(float2 b, int m) {
    m &= 63;
    if (m == 0) return b;
    if (m == 16) return INV ? make_float2(-b.y, b.x) : make_float2(b.y, -b.x);
    if (m == 32) return make_float2(-b.x, -b.y);
    if (m == 48) return INV ? make_float2(b.y, -b.x) : make_float2(-b.y, b.x);
    constexpr float h = (float)cos64(8);
    if (m == 8)
        return INV ? make_float2((b.x - b.y) * h, (b.x + b.y) * h)
                   : make_float2((b.x + b.y) * h, (b.y - b.x) * h);
    if (m == 24)
        return INV ? make_float2((b.x + b.y) * -h, (b.x - b.y) * h)
                   : make_float2((b.y - b.x) * h, (b.x + b.y) * -h);
    const float c = (float)cos_turn64(m), s = (float)(INV ? sin_turn64(m) : -sin_turn64(m));
    return make_float2(fmaf(b.x, c, -b.y * s), fmaf(b.x, s, b.y * c));
}

// A sample of global memory, read through L1 without keeping a line there (the
// tables keep theirs).
__device__ __forceinline__ float2 ld_stream(const float2 *p) {
    float2 v;
    asm("ld.global.nc.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}

template <int R>
__host__ __device__ constexpr int brev(int i) {
    int o = 0;
    for (int b = 1, t = R >> 1; b < R; b <<= 1, t >>= 1)
        if (i & b) o |= t;
    return o;
}

// lo, hi = lo + w hi, lo - w hi, w = exp(-+2 pi i m / 64), 0 <= m < 32.  A
// rotation that is no quarter turn takes two FMAs for (x + r y, y - r x) with
// the ratio r of its sine and cosine (at most 1) and four for the sums scaled
// by the larger of the two: six operations and two roundings per result,
// against eight and three for the product and its sum and difference.  The
// ratio's own rounding shows in long sums, though: FUSED chooses.  Range
// compression goes without it (error against 64 bits 2.0e-7, 2.1e-7 with it, both
// before the gain below was taken out; 0.31 and 0.29 ms).  Crossmul takes it: its
// odd samples' error is no larger for it (1.37e-7 at 4,096 points and 1.43e-7
// without, the gain out, by the same operations on the CPU).
template <bool INV, bool FUSED>
__device__ __forceinline__ void butterfly(float2 &lo, float2 &hi, int m) {
    const float2 a = lo, b = hi;
    if (!FUSED || m % 16 == 0) {
        const float2 t = rot64<INV>(b, m);
        hi = csub(a, t);
        lo = cadd(a, t);
        return;
    }
    const double c = cos_turn64(m), s = INV ? -sin_turn64(m) : sin_turn64(m);
    float2 t;
    float k;
    if (m <= 8 || m >= 24) {
        const float r = (float)(s / c);
        t = make_float2(fmaf(r, b.y, b.x), fmaf(-r, b.x, b.y));
        k = (float)c;
    } else {
        const float r = (float)(c / s);
        t = make_float2(fmaf(r, b.x, b.y), fmaf(r, b.y, -b.x));
        k = (float)s;
    }
    hi = make_float2(fmaf(-k, t.x, a.x), fmaf(-k, t.y, a.y));
    lo = make_float2(fmaf(k, t.x, a.x), fmaf(k, t.y, a.y));
}

// R-point DFT (sign -, or + with INV; unnormalised) of v[0..R), in place:
// input in natural order, bin r of the result in v[brev<R>(r)].  Radix-2
// decimation in time over the bit-reversed view, so nothing is moved.
template <int R, bool INV, bool FUSED = true>
__device__ __forceinline__ void dft(float2 *v) {
#pragma unroll
    for (int h = 1; h < R; h <<= 1) {
#pragma unroll
        for (int i = 0; i < R; i += 2 * h) {
#pragma unroll
            for (int q = 0; q < h; ++q) {
                butterfly<INV, FUSED>(v[brev<R>(i + q)], v[brev<R>(i + q + h)], q * (32 / h));
            }
        }
    }
}

// The butterflies' constants are rounded, cos(pi / 8) to 3.1e-8 and cos(pi / 4)
// to 1.7e-8 below their values, so a rotation comes out short and a transform's
// results with it: by 1.0e-7 of themselves after a convolution of 4,096 points
// (whose error is 1.7e-7 with that and 1.4e-7 without), the same for every
// input.  The gains below (relative, to first order) let a caller take that out
// with a factor it multiplies by anyway: single looks of two convolved lines
// of 2,400 samples then err by 1.0e-7 against 64 bits instead of 1.5e-7.
//
// Gain of a rotation by 2 pi m / 64 with rounded constants (of butterfly
// <FUSED>, or rot64), less 1.
__host__ __device__ constexpr double rotation_gain(int m, bool fused) {
    const double c = cos_turn64(m), s = sin_turn64(m);
    if (m % 16 == 0) return 0.0;
    if (m % 16 == 8) return (float)cos64(8) / cos64(8) - 1.0;
    double cr = (float)c, sr = (float)s;
    if (fused && (m <= 8 || m >= 24)) sr = cr * (float)(s / c);
    else if (fused) cr = sr * (float)(c / s);
    return cr * c + sr * s - 1.0;
}
// Of an R-point DFT: half the points of a level are rotated.
template <int R, bool FUSED = true>
__host__ __device__ constexpr double dft_gain() {
    double g = 0.0;
    for (int h = 1; h < R; h <<= 1)
        for (int q = 0; q < h; ++q) g += rotation_gain(q * (32 / h), FUSED) / (2 * h);
    return g;
}

// Sizes of one transform and their tables.
template <int M_, int EPT_, int RA_, int RB_, int RC_, bool FUSED_ = true>
struct Plan {
    static constexpr bool FUSED = FUSED_;  // butterfly
    static constexpr int M = M_, EPT = EPT_, RA = RA_, RB = RB_, RC = RC_;
    static constexpr int T = M / EPT;            // threads of a line
    static constexpr int CA = M / RA;            // DFTs of pass 1
    static constexpr int GA = EPT / RA, GB = EPT / RB, GC = EPT / RC;  // DFTs per thread
    static constexpr int BUF = M + M / EPT;      // padded points of the buffer
    static constexpr int TW1 = (RA - 1) * T, TW2 = (RB - 1) * RC;     // table entries
    static_assert(RA * RB * RC == M && EPT % RA == 0 && EPT % RB == 0 && EPT % RC == 0, "digits");
    static __host__ __device__ __forceinline__ constexpr int pad(int i) { return i + i / EPT; }
    // pad(j + k) for a constant k; pj = pad(j).  Where EPT divides k the two
    // add up, and an access is a register plus an immediate.
    static __device__ __forceinline__ int pad_from(int pj, int j, int k) {
        return k % EPT == 0 ? pj + pad(k) : pad(j + k);
    }
    // pad(c / RC * RB RC + c mod RC + r RC), element r of DFT c of pass 2:
    // base(c) + step(r) where EPT divides RB RC
    static __device__ __forceinline__ int pass2(int c, int r) {
        if (RB * RC % EPT == 0) return c / RC * pad(RB * RC) + c % RC + pad(r * RC);
        return pad(c / RC * (RB * RC) + c % RC + r * RC);
    }
};

// Tables of a plan: tw1[(r - 1) T + d] = exp(-2 pi i r (d + shift) / M), d < T,
// tw2[(r - 1) RC + d] = exp(-2 pi i r (d + shift) / (RB RC)); the forward ones
// have shift 0; an inverse evaluated half a sample on has shift 1/2 (and
// takes their conjugates).  Where a thread has several DFTs of pass 1
// (columns j + g T), the other columns' twiddles are turned from column j's by
// a constant (Tw1).
template <class P>
inline std::vector<float2> tables(double shift) {
    const double tau = 8.0 * std::atan2(1.0, 1.0);
    std::vector<float2> t(P::TW1 + P::TW2);
    auto w = [&](double x) { return make_float2((float)std::cos(tau * x), (float)-std::sin(tau * x)); };
    for (int r = 1; r < P::RA; ++r)
        for (int d = 0; d < P::T; ++d) t[(r - 1) * P::T + d] = w(r * (d + shift) / P::M);
    for (int r = 1; r < P::RB; ++r)
        for (int d = 0; d < P::RC; ++d)
            t[P::TW1 + (r - 1) * P::RC + d] = w(r * (d + shift) / (P::RB * P::RC));
    return t;
}

template <class P>
struct Tw1 {
    const float2 *t;
    __device__ __forceinline__ float2 operator()(int r, int j, int g) const {
        // exp(-2 pi i r g T / M), T / M = 1 / EPT
        return rot64<false>(t[(r - 1) * P::T + j], r * g * (64 / P::EPT));
    }
};

// Thread j of a line holds point j + point_of(i) in v[i], before and after
// conv().
template <class P>
__device__ __forceinline__ constexpr int point_of(int i) {
    return (i / P::RA) * P::T + (i % P::RA) * P::CA;
}

// Barrier of the threads of one line; `slot` tells the lines of a CTA apart.
template <class P>
__device__ __forceinline__ void line_sync(int slot, bool alone) {
    if (P::T <= 32) __syncwarp();
    else if (alone) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"(slot + 1), "n"(P::T) : "memory");
}

// Multiplications of the spectrum in the middle pass: element i of thread j
// (bin digits k0 k1 = the row (j EPT + i) / RC, k2 = i mod RC).
// Half a sample on: exp(i pi k2 / RC), negated in the upper half of the bins
// (k2 >= RC / 2): with the half-sample inverse tables the inverse's value at
// n is the spectrum's trigonometric interpolant at n + 1/2, the upper half of
// the bins taken as the negative frequencies' images at the top of a doubled
// spectrum.
template <class P>
struct HalfSample {
    __device__ __forceinline__ float2 operator()(float2 z, int i, int) const {
        const int k2 = i % P::RC;
        const float2 a = rot64<true>(z, k2 * (32 / P::RC));
        return k2 < P::RC / 2 ? a : make_float2(-a.x, -a.y);
    }
};
// A filter's spectrum, entry [i][j] (spectrum_order).
template <class P>
struct Filter {
    const float2 *h;
    __device__ __forceinline__ float2 operator()(float2 z, int i, int j) const {
        return cmul(z, h[i * P::T + j]);
    }
};
// Gain of conv() with a multiplication of gain 0, and of HalfSample (dft_gain);
// the tables' entries err to both sides.
template <class P>
__host__ __device__ constexpr double conv_gain() {
    return 2.0 * (dft_gain<P::RA, P::FUSED>() + dft_gain<P::RB, P::FUSED>() + dft_gain<P::RC, P::FUSED>());
}
template <class P>
__host__ __device__ constexpr double half_sample_gain() {
    double g = 0.0;
    for (int k2 = 0; k2 < P::RC; ++k2) g += rotation_gain(k2 * (32 / P::RC), false) / P::RC;
    return g;
}
// Bin held as element i of thread j in the middle pass.
template <class P>
inline int spectrum_order(int i, int j) {
    const int p = j * P::EPT + i;
    const int k2 = p % P::RC, k1 = p / P::RC % P::RB, k0 = p / (P::RC * P::RB);
    return k0 + P::RA * (k1 + P::RB * k2);
}

// v: points j + point_of(i), replaced by the convolved line's at the same
// places.  buf: P::BUF points of this line's own.  tw1(r, j, g)
// (column d = j + g T), tw2: forward twiddles; iw1, iw2: those of the inverse (conjugated here).  The caller's next use of
// `buf` (by this function too) must be behind a line_sync.
template <class P, class Tw, class Mul>
__device__ __forceinline__ void conv(float2 (&v)[P::EPT], float2 *buf, int j, int slot, bool alone,
                                     const Tw &tw1, const float2 *tw2, const Tw &iw1,
                                     const float2 *iw2, const Mul &mul) {
    const int pj = P::pad(j);
    // pass 1, from registers
#pragma unroll
    for (int g = 0; g < P::GA; ++g) {
        dft<P::RA, false, P::FUSED>(v + g * P::RA);
#pragma unroll
        for (int r = 0; r < P::RA; ++r) {
            const float2 z = v[g * P::RA + brev<P::RA>(r)];
            buf[P::pad_from(pj, j, g * P::T + r * P::CA)] = r ? cmul(z, tw1(r, j, g)) : z;
        }
    }
    line_sync<P>(slot, alone);
    // pass 2: DFT c covers points k0 RB RC + n1 RC + n2, k0 = c / RC, n2 = c mod RC
#pragma unroll
    for (int g = 0; g < P::GB; ++g) {
        const int c = j + g * P::T, n2 = c % P::RC;
#pragma unroll
        for (int r = 0; r < P::RB; ++r) v[r] = buf[P::pass2(c, r)];
        dft<P::RB, false, P::FUSED>(v);
#pragma unroll
        for (int r = 0; r < P::RB; ++r) {
            const float2 z = v[brev<P::RB>(r)];
            buf[P::pass2(c, r)] = r ? cmul(z, tw2[(r - 1) * P::RC + n2]) : z;
        }
    }
    line_sync<P>(slot, alone);
    // middle: the last forward DFTs, the spectrum, the first inverse ones
    {
        float2 *row = buf + P::pad(j * P::EPT);
#pragma unroll
        for (int i = 0; i < P::EPT; ++i) v[i] = row[i];
#pragma unroll
        for (int g = 0; g < P::GC; ++g) {
            float2 *w = v + g * P::RC;
            dft<P::RC, false, P::FUSED>(w);
            float2 u[P::RC];
#pragma unroll
            for (int r = 0; r < P::RC; ++r) u[r] = mul(w[brev<P::RC>(r)], g * P::RC + r, j);
            dft<P::RC, true, P::FUSED>(u);
#pragma unroll
            for (int r = 0; r < P::RC; ++r) row[g * P::RC + r] = u[brev<P::RC>(r)];
        }
    }
    line_sync<P>(slot, alone);
    // inverse of pass 2
#pragma unroll
    for (int g = 0; g < P::GB; ++g) {
        const int c = j + g * P::T, n2 = c % P::RC;
#pragma unroll
        for (int r = 0; r < P::RB; ++r) {
            const float2 z = buf[P::pass2(c, r)];
            v[r] = r ? cmulc(z, iw2[(r - 1) * P::RC + n2]) : z;
        }
        dft<P::RB, true, P::FUSED>(v);
#pragma unroll
        for (int r = 0; r < P::RB; ++r) buf[P::pass2(c, r)] = v[brev<P::RB>(r)];
    }
    line_sync<P>(slot, alone);
    // inverse of pass 1, into registers in natural order
#pragma unroll
    for (int g = 0; g < P::GA; ++g) {
        float2 u[P::RA];
#pragma unroll
        for (int r = 0; r < P::RA; ++r) {
            const float2 z = buf[P::pad_from(pj, j, g * P::T + r * P::CA)];
            u[r] = r ? cmulc(z, iw1(r, j, g)) : z;
        }
        dft<P::RA, true, P::FUSED>(u);
#pragma unroll
        for (int r = 0; r < P::RA; ++r) v[g * P::RA + r] = u[brev<P::RA>(r)];
    }
}

}  // namespace fftc
}  // namespace srg
