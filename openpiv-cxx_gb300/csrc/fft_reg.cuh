// fft_reg.cuh -- radix-2 FFTs held entirely in one thread's registers.
//
// A thread owns N complex values (float2 v[N]) and transforms them without
// touching memory: every loop is fully unrolled, so array indices and twiddle
// indices are compile-time constants and v[] stays in registers.  Twiddles
// come from a __constant__ table (constant-bank operands of FFMA, no extra
// instruction); the trivial ones (1, -i, i) are folded away at compile time.
//
// Conventions: forward = exp(-2*pi*i*k*n/N), inverse = exp(+...), no 1/N
// scaling (as the reference's FFT class, openpiv/algos/fft.h:274-294).
#pragma once
#include <cuda_runtime.h>

namespace opiv {

// ---------------------------------------------------------------------------
// cos / sin of 2*pi*k/N evaluated at compile time.  The angle is reduced to
// [0, pi/4] exactly with integer arithmetic on k (quarter turns, then the
// complementary angle), then summed as a Taylor series (truncation < 1e-17
// for |x| <= pi/4).  This is plain mathematics, evaluated by the C++ front
// end; no device math library is involved.
constexpr double kPi = 3.141592653589793238462643383279502884;

constexpr double series_sin(double x)
{
    double x2 = x * x, term = x, sum = x;
    for (int n = 1; n < 14; ++n) {
        term *= -x2 / ((2.0 * n) * (2.0 * n + 1.0));
        sum += term;
    }
    return sum;
}

constexpr double series_cos(double x)
{
    double x2 = x * x, term = 1.0, sum = 1.0;
    for (int n = 1; n < 14; ++n) {
        term *= -x2 / ((2.0 * n - 1.0) * (2.0 * n));
        sum += term;
    }
    return sum;
}

// {cos, sin} of (pi/2) * r / N for 0 <= r <= N
constexpr void quarter(long r, long N, double& c, double& s)
{
    if (2 * r <= N) {
        const double x = (kPi / 2.0) * (double)r / (double)N;
        c = series_cos(x);
        s = series_sin(x);
    } else {
        const double x = (kPi / 2.0) * (double)(N - r) / (double)N;
        c = series_sin(x);
        s = series_cos(x);
    }
}

constexpr void cis_2pi(long k, long N, double& c, double& s)
{
    k %= N;
    if (k < 0) k += N;
    const long q = (4 * k) / N;          // quarter turn index
    const long r = 4 * k - q * N;        // remainder, in units of 1/(4N) turn
    double qc = 0, qs = 0;
    quarter(r, N, qc, qs);
    switch (q) {
    case 0: c = qc; s = qs; break;
    case 1: c = -qs; s = qc; break;
    case 2: c = -qc; s = -qs; break;
    default: c = qs; s = -qc; break;
    }
}

// exp(-2*pi*i*k/64) for k < 64; length-N transforms use entry k*(64/N).
constexpr int kTwMax = 64;
struct TwiddleTable {
    float re[kTwMax];
    float im[kTwMax];
};

constexpr TwiddleTable make_twiddles()
{
    TwiddleTable t{};
    for (int k = 0; k < kTwMax; ++k) {
        double c = 0, s = 0;
        cis_2pi(k, kTwMax, c, s);
        t.re[k] = (float)c;
        t.im[k] = (float)(-s);
    }
    return t;
}

static __constant__ TwiddleTable c_tw = make_twiddles();

// ---------------------------------------------------------------------------
// Packed FP32 pairs (one instruction for both components; each rounds as the
// scalar one does).
__device__ __forceinline__ float2 add2(float2 a, float2 b)
{
    float2 d;
    asm("{ .reg .b64 x, y; mov.b64 x, {%2, %3}; mov.b64 y, {%4, %5}; add.rn.f32x2 x, x, y; mov.b64 {%0, %1}, x; }"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b)
{
    float2 d;
    asm("{ .reg .b64 x, y; mov.b64 x, {%2, %3}; mov.b64 y, {%4, %5}; sub.rn.f32x2 x, x, y; mov.b64 {%0, %1}, x; }"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c)
{
    float2 d;
    asm("{ .reg .b64 x, y, z; mov.b64 x, {%2, %3}; mov.b64 y, {%4, %5}; mov.b64 z, {%6, %7}; "
        "fma.rn.f32x2 x, x, y, z; mov.b64 {%0, %1}, x; }"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}

// 4 conj(P) = ( 2 Im(Z Zm), |Z|^2 - |Zm|^2 ) of a bin of Z = FFT(a + i b) and
// its mirror Zm = Z[-k], P = B conj(A).  With s = Z + Zm and t = Z - Zm,
// 2 A = (s.x, t.y) and 2 B = (s.y, -t.x): formed from those, the rounding is
// that of A's and B's own product (squares of Z would round in units of
// |A|^2 + |B|^2, and one product serves both k and -k, so the two bins'
// roundings do not average out).
__device__ __forceinline__ float2 four_conj_p(float2 z, float2 m)
{
    const float2 s = add2(z, m), t = sub2(z, m);
    return make_float2(fmaf(s.x, s.y, -(t.x * t.y)), fmaf(s.x, t.x, s.y * t.y));
}

// ---------------------------------------------------------------------------
// Decimation in time in fused multiply-add form: with w = wx + i wy and
// t = wy / wx, w*b = wx * (b + i t b), so a +- w*b costs 2 FMAs for
// c = b + i t b and 4 FMAs for a +- wx*c: 6 instructions per twiddled
// butterfly instead of 8.  The factor with the larger magnitude is pulled
// out (wx when |wx| >= |wy|, else wy with w*b = wy * ((wx/wy) b + i b)), which
// keeps the ratio within [-1, 1].  The last four are two packed ones.  Tables
// are evaluated at compile time.
struct FmaTwiddles {
    float m[kTwMax];      // pulled-out factor: wx or wy of exp(-2 pi i k / 64)
    float r[kTwMax];      // ratio: wy / wx or wx / wy
    bool by_cos[kTwMax];  // |wx| >= |wy|
};

__host__ __device__ constexpr bool fma_by_cos(int k)
{
    // |cos| >= |sin| for angles within 45 degrees of the real axis
    const int q = k & (kTwMax / 2 - 1);   // k mod 32 (period pi for |cos|, |sin|)
    return q <= kTwMax / 8 || q >= 3 * kTwMax / 8;
}

constexpr FmaTwiddles make_fma_twiddles()
{
    FmaTwiddles t{};
    for (int k = 0; k < kTwMax; ++k) {
        double c = 0, s = 0;
        cis_2pi(k, kTwMax, c, s);
        const double wx = c, wy = -s;   // forward twiddle exp(-2 pi i k / 64)
        const bool bc = fma_by_cos(k);
        t.by_cos[k] = bc;
        t.m[k] = (float)(bc ? wx : wy);
        t.r[k] = (float)(bc ? wy / wx : wx / wy);
    }
    return t;
}

static __constant__ FmaTwiddles c_fma = make_fma_twiddles();

// a, b -> a + w b, a - w b with w = exp(-+2 pi i k / N)
template <int N, bool INV>
__device__ __forceinline__ void bfly_dit(float2& a, float2& b, int k)
{
    k &= (N - 1);
    if (k == 0) {
        const float2 t = b;
        b = sub2(a, t);
        a = add2(a, t);
        return;
    }
    if (4 * k == N) {   // w = -i (forward) or i (inverse)
        const float2 wb = INV ? make_float2(-b.y, b.x) : make_float2(b.y, -b.x);
        b = make_float2(a.x - wb.x, a.y - wb.y);
        a = make_float2(a.x + wb.x, a.y + wb.y);
        return;
    }
    const int q = k * (kTwMax / N);
    const float m = (INV && !fma_by_cos(q)) ? -c_fma.m[q] : c_fma.m[q];
    const float r = INV ? -c_fma.r[q] : c_fma.r[q];
    float2 c;
    if (fma_by_cos(q)) {    // w b = wx (bx - t by, by + t bx), t = wy / wx
        c = make_float2(fmaf(-r, b.y, b.x), fmaf(r, b.x, b.y));
    } else {                // w b = wy (s bx - by, s by + bx), s = wx / wy
        c = make_float2(fmaf(r, b.x, -b.y), fmaf(r, b.y, b.x));
    }
    b = fma2(make_float2(-m, -m), c, a);
    a = fma2(make_float2(m, m), c, a);
}

// Decimation in time, FMA form: bit-reversed input (v[i] holds
// x[bitrev(i)]), natural-order output.
template <int N, bool INV>
__device__ __forceinline__ void fft_dit_fma(float2 (&v)[N])
{
#pragma unroll
    for (int half = 1; half < N; half <<= 1) {
#pragma unroll
        for (int base = 0; base < N; base += 2 * half) {
#pragma unroll
            for (int j = 0; j < half; ++j)
                bfly_dit<N, INV>(v[base + j], v[base + j + half], j * (N / (2 * half)));
        }
    }
}

template <int N>
__host__ __device__ constexpr int bitrev(int i)
{
    int r = 0;
    for (int b = 1; b < N; b <<= 1) {
        r = (r << 1) | (i & 1);
        i >>= 1;
    }
    return r;
}

}  // namespace opiv
