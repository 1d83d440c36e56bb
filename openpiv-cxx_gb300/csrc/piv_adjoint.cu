// Adjoint of the window chain extract -> correlate -> find_peaks -> 3-point
// Gaussian fit -> vector, d(u, v) / d(pixel) for both frames.
//
// The integer peak (px, py) is piecewise constant in the pixels; u and v
// depend on them only through the sub-pixel fit (image_utils.impl.h:77-101)
//   fx = (ln l - ln r) / (2 (ln l + ln r - 2 ln c)),   u = W/2 - px - fx
// of five plane values c, l, r (row py) and u_, d (column px).  A plane
// value of FFT::cross_correlate (fft.h:188-206) at swapped position (x, y)
// is the circular correlation at lag (dx, dy) = (x - W/2, y - W/2):
//   R(dx, dy) = sum_p a[p] b[p + (dx, dy)],
// so dR/da[p] = b[p + lag], dR/db[q] = a[q - lag].  The kernel recomputes
// the five values as direct sums (no plane is stored), forms the partial
// derivatives of the fit, and either accumulates the vector-Jacobian
// product of per-window cotangents (gu, gv) into image gradients, or the
// propagated standard deviation of u and v for independent pixel noise.
//
// The five lags are the peak's and its four neighbours, so with frame B's
// window rotated by the peak's lag, b'[p] = b[p + lag], every sum and every
// derivative is a five-point stencil: of b' for d/da[p], of a (mirrored) for
// d/db[p + lag].  Lanes take columns; a warp holds its rows of a and b' in
// registers (each pixel loaded once, 64 independent loads a window), rows
// above and below are registers, columns left and right two shuffles.
// W = 16: the halves of a warp take the window's row halves; W = 32: one
// warp a window; W = 64: four warps a window, two columns a lane.
// A 2048 x 2048 float pair, 32 px windows at step 16 (16,129 windows), both
// outputs: 157 -> 50 us.  Re-reading the five taps of both frames for every
// pixel took sixteen loads a pixel where this takes two.  Bound by issue
// slots (65 % busy at 16 warps an SM: about 2,300 instructions a window, of
// them 640 FMAs, 192 shuffles, 64 loads and 64 gradient updates, and their
// addresses); 128 registers hold a 32 px window's two frames.
//
// REAL mode (FFT::cross_correlate_real, fft.h:208-227): the reference's
// two-for-one unpack leaves spectrum column k_x = 0 and rows k_y = 0, H/2 at
// zero (fft.h:163-183), so its plane is IFFT(M B conj A) with M the
// indicator of the other bins.  M is a projection that commutes with
// circular shifts, so M B conj A = (M B) conj (M A) and the plane is the
// plain circular correlation of the projected windows, P removing each
// row's mean (k_x = 0) and then, per column, the mean and the
// (-1)^y-weighted mean (k_y = 0, H/2); since a shifted P b already lies in
// P's range, the derivatives are the complex-mode ones on the projected
// windows, and P applies to the rotated window as well as to the window.
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>

#include "piv_kernels.h"

namespace opiv {
namespace {

constexpr int kWarps = 4;

// How a window lies in the lanes and warps.
template <int W>
struct layout {
    static constexpr int CPL = W == 64 ? 2 : 1;     // columns of a lane: x, x + 32
    static constexpr int LPR = W / CPL;             // lanes of a row
    static constexpr int WPW = W == 64 ? 4 : 1;     // warps of a window
    static constexpr int BANDS = 32 / LPR * WPW;    // row bands of a window
    static constexpr int RB = W / BANDS;            // rows of a band
    static constexpr int H = BANDS > 1 ? 1 : 0;     // rows held beyond a band's ends
    static constexpr int ROWS = RB + 2 * H;
};

// Left (D = -1) or right (D = 1) neighbours of a row, around its ends.
template <int W, int D>
__device__ __forceinline__ void beside(const float (&v)[layout<W>::CPL], int x, float (&out)[layout<W>::CPL])
{
    using L = layout<W>;
    float t[L::CPL];
#pragma unroll
    for (int c = 0; c < L::CPL; ++c) t[c] = __shfl_sync(0xffffffffu, v[c], (x + D) & (L::LPR - 1), L::LPR);
    if constexpr (L::CPL == 1) {
        out[0] = t[0];
    } else {
        const bool wrap = x == (D < 0 ? 0 : L::LPR - 1);   // the row's halves change places
        out[0] = wrap ? t[1] : t[0];
        out[1] = wrap ? t[0] : t[1];
    }
}

template <int W>
__device__ __forceinline__ float row_total(float s)
{
#pragma unroll
    for (int o = layout<W>::LPR / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// Totals of K values over a window's lanes (all bands), in every lane.
// sm: WPW * K floats; the caller's next use of it comes after a barrier.
template <int W, int K>
__device__ __forceinline__ void window_total(float (&v)[K], float* sm, int wib)
{
    using L = layout<W>;
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    if constexpr (L::WPW > 1) {
        if ((threadIdx.x & 31) == 0)
            for (int k = 0; k < K; ++k) sm[wib * K + k] = v[k];
        __syncthreads();
#pragma unroll
        for (int k = 0; k < K; ++k) {
            float s = 0.f;
            for (int i = 0; i < L::WPW; ++i) s += sm[i * K + k];
            v[k] = s;
        }
    }
}

// The projection P of REAL mode on a window's rows (bands and the rows
// beyond their ends).  y0: the band's first row.  sm: 2 * W * WPW floats.
template <int W>
__device__ __forceinline__ void project(float (&v)[layout<W>::ROWS][layout<W>::CPL], int x, int wib, float* sm)
{
    using L = layout<W>;
#pragma unroll
    for (int r = 0; r < L::ROWS; ++r) {
        float s = 0.f;
#pragma unroll
        for (int c = 0; c < L::CPL; ++c) s += v[r][c];
        s = row_total<W>(s) / (float)W;
#pragma unroll
        for (int c = 0; c < L::CPL; ++c) v[r][c] -= s;
    }
    // bands start on even rows: a row's sign follows its place in the band
    float s[L::CPL], t[L::CPL];
#pragma unroll
    for (int c = 0; c < L::CPL; ++c) {
        s[c] = t[c] = 0.f;
#pragma unroll
        for (int r = 0; r < L::RB; ++r) {
            s[c] += v[r + L::H][c];
            t[c] += (r & 1) ? -v[r + L::H][c] : v[r + L::H][c];
        }
        if constexpr (L::LPR < 32) {
            s[c] += __shfl_xor_sync(0xffffffffu, s[c], L::LPR);
            t[c] += __shfl_xor_sync(0xffffffffu, t[c], L::LPR);
        }
    }
    if constexpr (L::WPW > 1) {
        float2* p = reinterpret_cast<float2*>(sm);
        __syncthreads();   // the last use of sm is over
#pragma unroll
        for (int c = 0; c < L::CPL; ++c) p[wib * W + x + 32 * c] = make_float2(s[c], t[c]);
        __syncthreads();
#pragma unroll
        for (int c = 0; c < L::CPL; ++c) {
            s[c] = t[c] = 0.f;
            for (int i = 0; i < L::WPW; ++i) {
                const float2 q = p[i * W + x + 32 * c];
                s[c] += q.x;
                t[c] += q.y;
            }
        }
    }
#pragma unroll
    for (int c = 0; c < L::CPL; ++c) {
        s[c] /= (float)W;
        t[c] /= (float)W;
#pragma unroll
        for (int r = 0; r < L::ROWS; ++r) v[r][c] -= ((r - L::H) & 1) ? s[c] - t[c] : s[c] + t[c];
    }
}

// d(offset) / d(lo, hi, c) of one axis of the fit, negated (u = .. - fx);
// false (and zeros) where the fit has no derivative.
__device__ __forceinline__ bool fit_partials(float c, float lo, float hi, float& gc, float& glo, float& ghi)
{
    gc = glo = ghi = 0.f;
    if (!(c > 0.f && lo > 0.f && hi > 0.f)) return false;
    const float a = logf(lo), b = logf(hi);
    const float N = a - b, D = 2.f * (a + b - 2.f * logf(c));
    if (!(D != 0.f)) return false;
    const float D2 = D * D;
    glo = -(D - 2.f * N) / (lo * D2);
    ghi = (D + 2.f * N) / (hi * D2);
    gc = -4.f * N / (c * D2);
    return true;
}

template <int W, bool REAL, bool VJP, bool SIGMA, typename PixT>
__global__ void __launch_bounds__(32 * kWarps, 4)
piv_adjoint_kernel(const PivParams p, const int32_t* __restrict__ peaks, const float* __restrict__ cot,
                   float* grad_a, float* grad_b, size_t gpitch, float var_a, float var_b, float* sigma)
{
    using L = layout<W>;
    constexpr int m = W - 1;
    __shared__ __align__(8) float sm[L::WPW > 1 ? 2 * W * L::WPW : 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wib = warp % L::WPW;                       // warp of its window
    const int64_t w = (int64_t)blockIdx.x * (kWarps / L::WPW) + warp / L::WPW;
    if (w >= p.n_win) return;   // uniform over the window's warps
    const int32_t code = peaks[w];
    if (code < 0) {             // fewer than two peaks: the vector is zero, no gradient
        if (SIGMA && lane == 0 && wib == 0) {
            sigma[2 * w] = 0.f;
            sigma[2 * w + 1] = 0.f;
        }
        return;
    }
    const int px = (code & 0xFFFF) % W, py = (code & 0xFFFF) / W;
    const int lx = px - W / 2, ly = py - W / 2;
    const int gy = (int)((unsigned)w / (unsigned)p.gnx);
    const int bx = p.gx0 + ((int)w - gy * p.gnx) * p.gdx, by = p.gy0 + gy * p.gdy;
    const int x = lane & (L::LPR - 1);
    const int y0 = (wib * (32 / L::LPR) + lane / L::LPR) * L::RB;   // the band's first row
    const size_t pitch = p.pitch / sizeof(PixT);

    float a[L::ROWS][L::CPL], b[L::ROWS][L::CPL];
    {
        const PixT* fa = reinterpret_cast<const PixT*>(p.fa) + (size_t)by * pitch + bx;
        const PixT* fb = reinterpret_cast<const PixT*>(p.fb) + (size_t)by * pitch + bx;
#pragma unroll
        for (int r = 0; r < L::ROWS; ++r) {
            const int y = (y0 + r - L::H) & m;
#pragma unroll
            for (int c = 0; c < L::CPL; ++c) {
                a[r][c] = (float)__ldg(fa + (size_t)y * pitch + x + 32 * c);
                b[r][c] = (float)__ldg(fb + (size_t)((y + ly) & m) * pitch + ((x + 32 * c + lx) & m));
            }
        }
    }
    if constexpr (REAL) {
        project<W>(a, x, wib, sm);
        project<W>(b, x, wib, sm);
    }
    // row r of the band, r = -1 .. RB
    auto at = [](int r) { return L::H ? r + 1 : r & (L::RB - 1); };

    // the five plane values
    float R[5] = { 0.f, 0.f, 0.f, 0.f, 0.f };   // c, l, r, u, d
#pragma unroll
    for (int r = 0; r < L::RB; ++r) {
        float bl[L::CPL], br[L::CPL];
        beside<W, -1>(b[at(r)], x, bl);
        beside<W, 1>(b[at(r)], x, br);
#pragma unroll
        for (int c = 0; c < L::CPL; ++c) {
            const float av = a[at(r)][c];
            R[0] = fmaf(av, b[at(r)][c], R[0]);
            R[1] = fmaf(av, bl[c], R[1]);
            R[2] = fmaf(av, br[c], R[2]);
            R[3] = fmaf(av, b[at(r - 1)][c], R[3]);
            R[4] = fmaf(av, b[at(r + 1)][c], R[4]);
        }
    }
    if (REAL && L::WPW > 1) __syncthreads();   // the projection's sums are read
    window_total<W, 5>(R, sm, wib);

    // partial derivatives of u = W/2 - px - fx and v = W/2 - py - fy
    float gx[3], gv[3];   // by c, then l, r / u, d
    const bool okx = fit_partials(R[0], R[1], R[2], gx[0], gx[1], gx[2]);
    const bool oky = fit_partials(R[0], R[3], R[4], gv[0], gv[1], gv[2]);
    const float cu = VJP ? cot[2 * w] : 0.f, cv = VJP ? cot[2 * w + 1] : 0.f;
    float* ga = VJP ? grad_a + (size_t)by * gpitch + bx : nullptr;
    float* gb = VJP ? grad_b + (size_t)by * gpitch + bx : nullptr;

    if (!okx && !oky) {   // no derivative, whatever the pixels are (they may be infinite or NaN)
        const float z = fmaf(cu, 0.f, cv * 0.f);
        if (VJP && z != 0.f) {   // a cotangent that is not finite still shows
#pragma unroll 1
            for (int r = 0; r < L::RB; ++r)
                for (int c = 0; c < L::CPL; ++c) {
                    atomicAdd(ga + (size_t)(y0 + r) * gpitch + x + 32 * c, z);
                    atomicAdd(gb + (size_t)(y0 + r) * gpitch + x + 32 * c, z);
                }
        }
        if (SIGMA && lane == 0 && wib == 0) sigma[2 * w] = sigma[2 * w + 1] = __int_as_float(0x7fffffff);
        return;   // uniform over the window's warps
    }

    // per pixel: du/da[p] = sum_v gx[v] b[p + lag_v], du/db[q] = sum_v gx[v] a[q - lag_v]
    float var[2] = { 0.f, 0.f };
#pragma unroll
    for (int r = 0; r < L::RB; ++r) {
        const int y = y0 + r;
        float al[L::CPL], ar[L::CPL], bl[L::CPL], br[L::CPL];
        beside<W, -1>(a[at(r)], x, al);
        beside<W, 1>(a[at(r)], x, ar);
        beside<W, -1>(b[at(r)], x, bl);
        beside<W, 1>(b[at(r)], x, br);
#pragma unroll
        for (int c = 0; c < L::CPL; ++c) {
            const float ac = a[at(r)][c], bc = b[at(r)][c];
            const float dua = fmaf(gx[2], br[c], fmaf(gx[1], bl[c], gx[0] * bc));
            const float dva = fmaf(gv[2], b[at(r + 1)][c], fmaf(gv[1], b[at(r - 1)][c], gv[0] * bc));
            const float dub = fmaf(gx[2], al[c], fmaf(gx[1], ar[c], gx[0] * ac));
            const float dvb = fmaf(gv[2], a[at(r - 1)][c], fmaf(gv[1], a[at(r + 1)][c], gv[0] * ac));
            if (SIGMA) {
                var[0] = fmaf(var_a * dua, dua, fmaf(var_b * dub, dub, var[0]));
                var[1] = fmaf(var_a * dva, dva, fmaf(var_b * dvb, dvb, var[1]));
            }
            if (VJP) {
                atomicAdd(ga + (size_t)y * gpitch + x + 32 * c, fmaf(cu, dua, cv * dva));
                atomicAdd(gb + (size_t)((y + ly) & m) * gpitch + ((x + 32 * c + lx) & m), fmaf(cu, dub, cv * dvb));
            }
        }
    }
    if (SIGMA) {
        if (L::WPW > 1) __syncthreads();   // the plane values' totals are read
        window_total<W, 2>(var, sm, wib);
        if (lane == 0 && wib == 0) {
            const float nan = __int_as_float(0x7fffffff);
            sigma[2 * w] = okx ? sqrtf(var[0]) : nan;
            sigma[2 * w + 1] = oky ? sqrtf(var[1]) : nan;
        }
    }
}

struct outputs {
    const int32_t* peaks;
    const float* cot;
    float *grad_a, *grad_b;
    size_t gpitch;
    float var_a, var_b;
    float* sigma;
};

template <int W, bool REAL, typename PixT>
cudaError_t launch_t(const PivParams& p, const outputs& o, cudaStream_t s)
{
    const int64_t per_cta = kWarps / layout<W>::WPW;
    const unsigned blocks = (unsigned)((p.n_win + per_cta - 1) / per_cta);
    auto go = [&](auto kern) {
        kern<<<blocks, 32 * kWarps, 0, s>>>(p, o.peaks, o.cot, o.grad_a, o.grad_b, o.gpitch, o.var_a, o.var_b, o.sigma);
    };
    if (o.cot && o.sigma) go(piv_adjoint_kernel<W, REAL, true, true, PixT>);
    else if (o.cot) go(piv_adjoint_kernel<W, REAL, true, false, PixT>);
    else if (o.sigma) go(piv_adjoint_kernel<W, REAL, false, true, PixT>);
    return cudaGetLastError();
}

template <int W, bool REAL>
cudaError_t launch_dt(const PivParams& p, int dtype, const outputs& o, cudaStream_t s)
{
    switch (dtype) {
    case kU8: return launch_t<W, REAL, uint8_t>(p, o, s);
    case kU16: return launch_t<W, REAL, uint16_t>(p, o, s);
    case kF32: return launch_t<W, REAL, float>(p, o, s);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace

cudaError_t launch_piv_adjoint(const PivParams& p, int w, int dtype, int mode, const int32_t* peaks,
                               const float* cot, float* grad_a, float* grad_b, size_t gpitch,
                               float var_a, float var_b, float* sigma, cudaStream_t s)
{
    if (p.n_win <= 0) return cudaSuccess;
    const outputs o{ peaks, cot, grad_a, grad_b, gpitch, var_a, var_b, sigma };
    const bool real = mode == kModeReal;
    switch (w) {
    case 16: return real ? launch_dt<16, true>(p, dtype, o, s) : launch_dt<16, false>(p, dtype, o, s);
    case 32: return real ? launch_dt<32, true>(p, dtype, o, s) : launch_dt<32, false>(p, dtype, o, s);
    case 64: return real ? launch_dt<64, true>(p, dtype, o, s) : launch_dt<64, false>(p, dtype, o, s);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace opiv
