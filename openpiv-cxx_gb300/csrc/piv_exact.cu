// piv_exact.cu -- exact double-precision window kernel for sm_103a.
//
// Repeats the reference's double arithmetic operation for operation, so its
// correlation planes are bit-identical to OpenPIV-c++ built without fused
// multiply-add contraction:
//   * 2-D FFT = radix-2 DIT on every row, then every column (fft.h:87-119),
//     with the same butterfly graph as the recursive fft_inner
//     (fft.h:245-263): e + o*w, e - o*w, w = table[k * 2n/len], where the
//     table entries exp(-+i*pi*j/n) are computed on the host with the
//     reference's own expression (fft.h:274-294);
//   * complex product (a*c - b*d, b*c + a*d) (pixel_types.h:159-163), every
//     multiply and add rounded separately (__dmul_rn / __dadd_rn, no FMA);
//   * REAL mode: the partial two-for-one unpack of fft.h:163-183;
//   * swap_quadrants (image_utils.impl.h:367-386) as an index remap;
//   * find_peaks (image_utils.impl.h:42-74) with exact comparisons; among
//     equal values the first peak is the one std::sort puts first (its
//     introsort is replayed, sort_order.h);
//   * fit_simple_gaussian (impl:77-101) and the vector of main.cpp:220-236
//     in double.
//
// It serves two purposes: it re-decides the windows the FP32 kernel flagged
// as uncertain (after refine_window below, which settles nearly all of them
// from a few exact sums), and it is the device FP64 correlation used by the
// exact per-window API.  One CTA of 256 threads handles one window at a time;
// CTAs stride over the work list.  FP64 is slow on this part, so the hot path only sends
// the rare flagged windows here.

#include <atomic>
#include <cstdint>
#include <type_traits>
#include <cuda_runtime.h>

#include "offsets.cuh"
#include "piv_kernels.h"
#include "sort_order.h"

namespace opiv {

namespace {

constexpr int kThreads = 256;
constexpr int kMaxW = 64;

__device__ __forceinline__ double2 e_add(double2 a, double2 b)
{
    return make_double2(__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y));
}
__device__ __forceinline__ double2 e_sub(double2 a, double2 b)
{
    return make_double2(__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y));
}
// (a + ib)(c + id) = (a*c - b*d, b*c + a*d), pixel_types.h:159-163
__device__ __forceinline__ double2 e_mul(double2 p, double2 q)
{
    return make_double2(__dsub_rn(__dmul_rn(p.x, q.x), __dmul_rn(p.y, q.y)),
                        __dadd_rn(__dmul_rn(p.y, q.x), __dmul_rn(p.x, q.y)));
}
__device__ __forceinline__ double2 e_conj(double2 a) { return make_double2(a.x, -a.y); }

__device__ __forceinline__ double px_d(const uint8_t* p) { return (double)__ldg(p); }
__device__ __forceinline__ double px_d(const uint16_t* p) { return (double)__ldg(p); }
__device__ __forceinline__ double px_d(const float* p) { return (double)__ldg(p); }
__device__ __forceinline__ double px_d(const double* p) { return __ldg(p); }

// Radix-2 DIT transforms of all W lines of a W x W tile, in place, every
// thread of the block cooperating: rows when (s_line, s_elem) = (W, 1),
// columns when (1, W).  Per line this is the butterfly graph of fft_inner
// (bit-reversal, then stages len = 2 .. W combining e + o*w, e - o*w with
// w = tw[k * 2W/len]); spreading butterflies over threads changes no
// operation and no operand.  tw: table of W entries exp(-+i*pi*j/W).
__device__ void dit_lines(double2* X, int W, int lg, int s_line, int s_elem, const double2* tw)
{
    const int t = threadIdx.x, T = blockDim.x;
    for (int q = t; q < W * W; q += T) {
        const int line = q / W, i = q % W;
        const int j = (int)(__brev((unsigned)i) >> (32 - lg));
        if (i < j) {
            double2* x = X + line * s_line;
            const double2 v = x[i * s_elem];
            x[i * s_elem] = x[j * s_elem];
            x[j * s_elem] = v;
        }
    }
    __syncthreads();
    const int nb = W / 2;   // butterflies per line and stage
    for (int len = 2; len <= W; len <<= 1) {
        const int half = len >> 1, tstep = (2 * W) / len;
        for (int q = t; q < W * nb; q += T) {
            const int line = q / nb, b = q % nb;
            const int base = (b / half) * len, k = b % half;
            double2* x = X + line * s_line;
            const double2 e = x[(base + k) * s_elem];
            const double2 o = e_mul(x[(base + k + half) * s_elem], tw[k * tstep]);
            x[(base + k) * s_elem] = e_add(e, o);
            x[(base + k + half) * s_elem] = e_sub(e, o);
        }
        __syncthreads();
    }
}

// 2-D transform: every row, then every column (fft.h:104-116).
__device__ void fft2d(double2* X, int W, const double2* tw)
{
    int lg = 0;
    while ((1 << lg) < W) ++lg;
    dit_lines(X, W, lg, W, 1, tw);
    dit_lines(X, W, lg, 1, W, tw);
}

__device__ __forceinline__ void window_origin(const PivParams& p, int64_t w, int& bx, int& by)
{
    if (p.win_xy != nullptr) {
        bx = p.win_xy[2 * w];
        by = p.win_xy[2 * w + 1];
    } else {
        // a plan holds at most 2^31 - 1 windows
        const int gy = (int)((unsigned)w / (unsigned)p.gnx);
        bx = p.gx0 + ((int)w - gy * p.gnx) * p.gdx;
        by = p.gy0 + gy * p.gdy;
    }
}

// fit_simple_gaussian's axis function, image_utils.impl.h:86-94
__device__ __forceinline__ double gauss3(double l, double c, double r)
{
    const double num = log(l) - log(r);
    const double den = 2.0 * (log(l) + log(r) - 2.0 * log(c));
    if (den == 0.0) return 0.0;
    return num / den;
}

// One window w of pair p, by the whole CTA (A, B: 2 W^2 double2 of shared
// memory; row_count: W ints; total_cand: one int, both shared).
template <typename PixT>
__device__ __forceinline__ void exact_window(const PivParams& p, const int64_t w, const int W, const int mode,
                                             const int sy0, const int sy1, const int sx0, const int sx1,
                                             double2* A, double2* B, int* row_count, int* total_cand)
{
    const int t = threadIdx.x;
    const int N = W * W;
    const PixT* fa = reinterpret_cast<const PixT*>(p.fa);
    const PixT* fb = reinterpret_cast<const PixT*>(p.fb);
    const size_t pitch = p.pitch / sizeof(PixT);
    int bx, by, ox, oy;
    window_origin(p, w, bx, by);
    b_offset(p, W, bx, by, ox, oy);

    // ---- extract, convert (g_f by value), join / convert to complex
    for (int i = t; i < N; i += blockDim.x) {
        const int y = i / W, x = i % W;
        const double a = px_d(fa + (size_t)(by + y) * pitch + bx + x);
        const double b = px_d(fb + (size_t)(by + oy + y) * pitch + bx + ox + x);
        if (mode == kModeComplex) {
            A[i] = make_double2(a, 0.0);
            B[i] = make_double2(b, 0.0);
        } else {
            A[i] = make_double2(a, b);
        }
    }
    __syncthreads();

    fft2d(A, W, p.tw_fwd);
    if (mode == kModeComplex) {
        fft2d(B, W, p.tw_fwd);
        for (int i = t; i < N; i += blockDim.x) A[i] = e_mul(B[i], e_conj(A[i]));
    } else {
        // transform_real's unpack (fft.h:166-183) fused with the product;
        // each (k, -k) pair is owned by one thread.  Cells outside the
        // unpacked set (row 0, row W/2, column 0) become zero.
        const int npairs = (W / 2 - 1) * (W - 1);
        for (int q = t; q < npairs; q += blockDim.x) {
            const int h = 1 + q / (W - 1), x = 1 + q % (W - 1);
            const int k = h * W + x, m = (W - h) * W + (W - x);
            const double2 t1 = A[k], t2 = A[m];
            const double2 half = make_double2(0.5, 0.0);
            const double2 av = e_mul(half, e_add(t1, e_conj(t2)));
            double2 bv = e_mul(half, e_sub(t1, e_conj(t2)));
            bv = make_double2(bv.y, __dmul_rn(-1.0, bv.x));
            A[k] = e_mul(bv, e_conj(av));
            A[m] = e_mul(e_conj(bv), e_conj(e_conj(av)));
        }
        for (int i = t; i < N; i += blockDim.x) {
            const int y = i / W, x = i % W;
            if (y == 0 || y == W / 2 || x == 0) A[i] = make_double2(0.0, 0.0);
        }
        __syncthreads();
    }
    __syncthreads();
    fft2d(A, W, p.tw_rev);

    // ---- real part, quadrant swap -> plane in B[].x (row-major)
    for (int i = t; i < N; i += blockDim.x) {
        const int y = i / W, x = i % W;
        const int sy = (y + W / 2) % W, sx = (x + W / 2) % W;
        B[i].x = A[sy * W + sx].x;
    }
    __syncthreads();
    if (p.planes64 != nullptr)
        for (int i = t; i < N; i += blockDim.x) p.planes64[(size_t)w * N + i] = B[i].x;

    // ---- find_peaks: strict 4-neighbour maxima of the scanned rows, in
    // row-major scan order (the order the reference pushes them), then
    // std::sort's choice of the first one (sort_order.h) and the second
    // largest value (with multiplicity) for sn.
    peak_cand* cand = reinterpret_cast<peak_cand*>(A);   // A is free now
    int my_count = 0;
    const int y = t;
    const bool row_ok = t < W && y >= sy0 && y < sy1;
    if (row_ok) {
        for (int x = sx0; x < sx1; ++x) {
            const double c = B[y * W + x].x;
            if (B[y * W + x - 1].x < c && B[y * W + x + 1].x < c &&
                B[(y - 1) * W + x].x < c && B[(y + 1) * W + x].x < c)
                ++my_count;
        }
    }
    if (t < W) row_count[t] = my_count;
    __syncthreads();
    if (t == 0) {
        int acc = 0;
        for (int r = 0; r < W; ++r) {
            const int c = row_count[r];
            row_count[r] = acc;
            acc += c;
        }
        (*total_cand) = acc;
    }
    __syncthreads();
    if (row_ok) {
        int o = row_count[t];
        for (int x = sx0; x < sx1; ++x) {
            const double c = B[y * W + x].x;
            if (B[y * W + x - 1].x < c && B[y * W + x + 1].x < c &&
                B[(y - 1) * W + x].x < c && B[(y + 1) * W + x].x < c)
                cand[o++] = peak_cand{ c, y * W + x };
        }
    }
    __syncthreads();
    if (t == 0) {
        const int n = (*total_cand);
        const double ninf = -__longlong_as_double(0x7ff0000000000000ll);
        double g0 = ninf, g1 = ninf;   // two largest values, with multiplicity
        for (int i = 0; i < n; ++i) {
            const double c = cand[i].v;
            if (c > g0) { g1 = g0; g0 = c; }
            else if (c > g1) g1 = c;
        }
        int k = -1;
        if (n >= 2) {
            sort_order_head(cand, n);
            k = cand[0].key;
        }
        const int count = n >= 2 ? 2 : n;
        opiv_vector out{ 0.f, 0.f, 0.f, 0.f, 0.f };
        int32_t code = -1;
        if (count == 2) {
            const int px = k % W, py = k / W;
            const double c = B[py * W + px].x;
            const double lx = (double)px + gauss3(B[py * W + px - 1].x, c, B[py * W + px + 1].x);
            const double ly = (double)py + gauss3(B[(py - 1) * W + px].x, c, B[(py + 1) * W + px].x);
            const int mx = bx + W / 2, my = by + W / 2;
            out.x = (float)mx;
            out.y = (float)((double)p.img_h - (double)my);
            out.u = (float)((double)mx - ((double)bx + lx) - (double)ox);
            out.v = (float)((double)my - ((double)by + ly) - (double)oy);
            out.sn = (g1 > 0) ? (float)(g0 / g1) : 0.f;
            code = k | OPIV_PEAK_EXACT;
        }
        if (p.out_vec) p.out_vec[w] = out;
        if (p.out_peak) p.out_peak[w] = code;
        if (p.out_disp)
            p.out_disp[w] = count == 2 ? pack_disp(k % W - W / 2 + ox, k / W - W / 2 + oy)
                                       : pack_disp(ox, oy);
    }
    __syncthreads();
}

// ---- a flagged window from exact sums -----------------------------------------
// Nearly every window that the FP32 kernel cannot decide hangs on a handful
// of plane values: two peaks within its error bound, or a second peak or a
// fit whose value needs more digits.  Those values are direct correlation
// sums, sum_p a[p] b[p + lag]: whole numbers for 8/16-bit frames (at most
// 2^44, kept in 64 bits), FP64 sums for float frames.  So instead of three
// 2-D transforms in FP64 (about 160,000 FP64 operations for a 32 px window at
// two per cycle and SM: 40 us for one CTA at best), the CTA takes the cells
// of the FP32 plane that could be one of the two highest maxima within its
// error bound (the window's record), and evaluates those cells and their
// neighbours exactly.  In units of W^2 times a plane value,
// REAL mode's plane (spectrum column 0 and rows 0, W/2 left out) is
//   V = W^2 R - W (rows + columns + (-1)^dy alternating)
//         + Sa Sb + (-1)^dy Ta Tb,
// where rows and columns are the 1-D correlations of the windows' row and
// column sums, alternating that of the (-1)^y-weighted column sums, S and T
// the totals of the plain and the weighted sums: whole numbers again.
// Returns false, with nothing written, where the exact kernel has to decide:
// ties and signs within the reference's own FP64 rounding, more than
// kMaxCand candidates, windows with infinite or huge pixels.
// The launch's time with the FP64 transforms and with this: a 4096 x 4096
// pass of 32 px windows at step 8 (4 flagged) 111 -> 12 us; 2048 x 1536, 16 px
// at step 8 (78 flagged) 48 -> 9 us; 2048 x 2048, 64 px at step 16 (2 flagged)
// 360 -> 19 us; 15,625 of 15,625 32 px windows flagged 7125 -> 349 us (with room for
// the records of one in 32 before); none flagged 3 us.  What is left is a chain of dependent loads,
// block barriers and FP64 logarithms of one window.
struct refine_shared {
    long long val[5 * kMaxCand];   // or doubles: centre, left, right, up, down
    int key[kMaxCand];
    int ok;
};

template <typename T>
__device__ __forceinline__ T warp_total(T v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <typename PixT>
__device__ __forceinline__ bool refine_window(const PivParams& p, const int64_t w, const int W, const int mode,
                                              const flag_record& rec, unsigned char* smem, refine_shared& rs)
{
    constexpr bool kFloat = sizeof(PixT) == 4;
    using Px = typename std::conditional<kFloat, double, uint32_t>::type;
    using Acc = typename std::conditional<kFloat, double, long long>::type;
    const int t = threadIdx.x, T = blockDim.x, lane = t & 31, warp = t >> 5, warps = T >> 5;
    const int N = W * W, m = W - 1, lg = 31 - __clz(W);
    const float dlt = rec.dlt;
    const int n = rec.n;
    if (!(dlt > 1e-30f && dlt < 1e30f) || n > kMaxCand) return false;   // block-uniform

    Px* A = reinterpret_cast<Px*>(smem);
    Px* B = A + N;
    Acc* prof = reinterpret_cast<Acc*>(B + N);   // REAL: 6 W sums
    int bx, by, ox, oy;
    window_origin(p, w, bx, by);
    b_offset(p, W, bx, by, ox, oy);
    {
        const PixT* fa = reinterpret_cast<const PixT*>(p.fa);
        const PixT* fb = reinterpret_cast<const PixT*>(p.fb);
        const size_t pitch = p.pitch / sizeof(PixT);
        for (int i = t; i < N; i += T) {
            const int y = i >> lg, x = i & m;
            A[i] = (Px)__ldg(fa + (size_t)(by + y) * pitch + bx + x);
            B[i] = (Px)__ldg(fb + (size_t)(by + oy + y) * pitch + bx + ox + x);
        }
    }
    if (t < kMaxCand) rs.key[t] = rec.key[t] & (N - 1);
    __syncthreads();
    if (mode == kModeReal) {
        // row sums of a and b, column sums, (-1)^y-weighted column sums
        for (int i = t; i < 4 * W; i += T) {
            const Px* X = (i & 1) ? B : A;
            const int l = (i >> 1) & m;
            Acc s = 0, h = 0;
            if (i < 2 * W) {
                for (int x = 0; x < W; ++x) s += (Acc)X[l * W + x];
                prof[(i & 1) * W + l] = s;
            } else {
                for (int y = 0; y < W; ++y) {
                    const Acc v = (Acc)X[y * W + l];
                    s += v;
                    h += (y & 1) ? -v : v;
                }
                prof[(2 + (i & 1)) * W + l] = s;
                prof[(4 + (i & 1)) * W + l] = h;
            }
        }
        __syncthreads();
    }

    // exact values, one warp per value
    Acc* val = reinterpret_cast<Acc*>(rs.val);
    for (int q = warp; q < 5 * n; q += warps) {
        const int k = rs.key[q / 5], j = q % 5;
        const int dx = (k & m) + (j == 2) - (j == 1) - W / 2, dy = (k >> lg) + (j == 4) - (j == 3) - W / 2;
        Acc s = 0;
#pragma unroll 8
        for (int i = lane; i < N; i += 32) {
            const int y = i >> lg, x = i & m;
            const Px a = A[i], b = B[(((y + dy) & m) << lg) + ((x + dx) & m)];
            if constexpr (kFloat) s = fma(a, b, s);
            else s += (long long)((unsigned long long)a * b);
        }
        s *= N;
        if (mode == kModeReal) {
            const Acc sg = (dy & 1) ? -1 : 1;
            Acc c = 0, sa = 0, sb = 0, ta = 0, tb = 0;
            for (int i = lane; i < W; i += 32) {
                const int iy = (i + dy) & m, ix = (i + dx) & m;
                c += prof[i] * prof[W + iy] + prof[2 * W + i] * prof[3 * W + ix] +
                     sg * prof[4 * W + i] * prof[5 * W + ix];
                sa += prof[i];
                sb += prof[W + i];
                ta += prof[4 * W + i];
                tb += prof[5 * W + i];
            }
            s -= W * c;
            s = warp_total(s) + warp_total(sa) * warp_total(sb) + sg * warp_total(ta) * warp_total(tb);
        } else {
            s = warp_total(s);
        }
        if (lane == 0) val[q] = s;
    }
    __syncthreads();

    // the decision, by one warp (every lane alike up to the logarithms)
    if (warp == 0) {
        // dlt bounds the FP32 plane's rounding, in units of 4 W^2; the
        // reference's FP64 transforms round 2^29 times finer.  32 times that,
        // in units of W^2, also covers the sums here (two neighbouring whole
        // numbers are W^2 apart)
        const double eps = (double)dlt * 1.4901161193847656e-8;
        const Acc tol = kFloat ? (Acc)eps : (Acc)eps + 1;
        bool ok = true;
        int k0 = -1, found = 0;
        Acc v0 = 0, v1 = 0;
        for (int i = 0; i < n; ++i) {
            const Acc* v = val + 5 * i;
            const Acc c = v[0];
            bool peak = true, below = false;
            for (int j = 1; j < 5; ++j) {
                const Acc d = c - v[j];
                peak = peak && d > tol;
                below = below || d < -tol;
            }
            if (!peak) {
                ok = ok && below;
                continue;
            }
            if (found == 0 || c > v0) {
                v1 = v0;
                v0 = c;
                k0 = i;
            } else if (found == 1 || c > v1) {
                v1 = c;
            }
            ++found;
        }
        opiv_vector out{ 0.f, 0.f, 0.f, 0.f, 0.f };
        int32_t code = -1;
        int px = W / 2, py = W / 2;
        if (found >= 2) {
            const Acc x = val[5 * k0 + (lane < 5 ? lane : 0)];
            ok = ok && v0 - v1 > tol && (v1 > tol || v1 < -tol);
            ok = __all_sync(0xffffffffu, ok && (x > tol || x < -tol));
            const double lv = log((double)x);   // NaN where the reference's is
            const double lc = __shfl_sync(0xffffffffu, lv, 0);
            const double ll = __shfl_sync(0xffffffffu, lv, 1), lr = __shfl_sync(0xffffffffu, lv, 2);
            const double lu = __shfl_sync(0xffffffffu, lv, 3), ld = __shfl_sync(0xffffffffu, lv, 4);
            // the three quotients on three lanes: x offset, y offset, sn
            const double lo = lane == 1 ? lu : ll, hi = lane == 1 ? ld : lr;
            const double num = lane == 2 ? (double)v0 : lo - hi;
            const double den = lane == 2 ? (double)v1 : 2.0 * (lo + hi - 2.0 * lc);
            // a flatter peak than this magnifies the FP64 rounding too much
            ok = __all_sync(0xffffffffu, ok && !(fabs(den) < 1e-8));
            const double quot = num / den;
            const int key = rs.key[k0];
            px = key & m;
            py = key >> lg;
            const double lx = (double)px + __shfl_sync(0xffffffffu, quot, 0);
            const double ly = (double)py + __shfl_sync(0xffffffffu, quot, 1);
            const double sn = __shfl_sync(0xffffffffu, quot, 2);
            const int mx = bx + W / 2, my = by + W / 2;
            out.x = (float)mx;
            out.y = (float)(p.img_h - my);
            out.u = (float)((double)mx - ((double)bx + lx) - (double)ox);
            out.v = (float)((double)my - ((double)by + ly) - (double)oy);
            out.sn = v1 > 0 ? (float)sn : 0.f;
            code = key | OPIV_PEAK_EXACT;
        }
        if (lane == 0) {
            rs.ok = ok;
            if (ok) {
                if (p.out_vec) p.out_vec[w] = out;
                if (p.out_peak) p.out_peak[w] = code;
                if (p.out_disp) p.out_disp[w] = pack_disp(px - W / 2 + ox, py - W / 2 + oy);
            }
        }
    }
    __syncthreads();
    const bool ok = rs.ok;
    __syncthreads();   // read before the next window
    return ok;
}

// scan range in plane coordinates (find_peaks on the plane or on its
// centre view rect().dilate(0.5); rect.cpp:109-126)
__device__ __forceinline__ void scan_range(int W, int limit, int& sy0, int& sy1, int& sx0, int& sx1)
{
    int d0 = 0, vw = W;
    if (limit) {
        const int rw = (int)lround(0.5 * W);
        d0 = (W - rw) / 2;
        vw = rw;
    }
    sy0 = d0 + 1;
    sy1 = d0 + vw - 2;
    sx0 = d0 + 1;
    sx1 = d0 + vw - 1;
}

// LIST: the windows of flag_list (the pass after the FP32 kernel), exact
// sums first, for all of them or none (the list's order is the order of
// arrival, so the first flag_cap of more would be other windows each time); otherwise every window in FP64.
template <typename PixT, bool LIST>
__global__ void __launch_bounds__(kThreads)
piv_exact_kernel(const PivParams p, int W, int mode, int limit)
{
    extern __shared__ double2 sm[];
    __shared__ int row_count[kMaxW];
    __shared__ int total_cand;
    if (LIST) after_previous();
    const int64_t nwork = LIST ? (int64_t)min(p.flag_count[kFlagged], (unsigned int)p.flag_room) : p.n_win;
    int sy0, sy1, sx0, sx1;
    scan_range(W, limit, sy0, sy1, sx0, sx1);
    unsigned int settled = 0;
    unsigned long long* words = LIST ? reinterpret_cast<unsigned long long*>(p.flag_count) : nullptr;
    const unsigned long long settled_before = LIST ? words[kSettled / 2] : 0;
    for (int64_t item = blockIdx.x; item < nwork; item += gridDim.x) {
        const int64_t w = LIST ? (int64_t)p.flag_list[item] : item;
        if constexpr (LIST) {
            __shared__ refine_shared rs;
            if (nwork <= p.flag_cap &&
                refine_window<PixT>(p, w, W, mode, p.flag_recs[item], reinterpret_cast<unsigned char*>(sm), rs)) {
                ++settled;
                continue;
            }
        }
        exact_window<PixT>(p, w, W, mode, sy0, sy1, sx0, sx1, sm, sm + W * W, row_count, &total_cand);
    }
    if constexpr (LIST) {
        // the last CTA to finish leaves the counters as the next pass wants
        // them (every CTA has read the count by then), so that a pass is two
        // launches: a memset before them and a copy of the count after them
        // were half of a small pass's time (160 x 128 px: 25.8 -> 14.3 us)
        if (threadIdx.x == 0) {
            const uint64_t before = atomicAdd(words + kDone / 2, done_add(settled));
            if (last_done(before, gridDim.x)) {
                atomicAdd(words + kDone / 2, 0ull - gridDim.x);
                p.flag_count[kLastFlagged] = (unsigned int)nwork;
                words[kSettledBefore / 2] = settled_before;
                words[kSettled / 2] = all_settled(before, settled);
                p.flag_count[kFlagged] = 0u;
            }
        }
    }
}

// The exact pass of a work queue: every pair's flagged windows, one list
// (combined window numbers), CTAs striding over it.
template <typename PixT>
__global__ void __launch_bounds__(kThreads)
piv_exact_queue_kernel(const __grid_constant__ PivQueue q, int W, int mode, int limit)
{
    extern __shared__ double2 sm[];
    __shared__ int row_count[kMaxW];
    __shared__ int total_cand;
    __shared__ refine_shared rs;
    const int64_t nwork = (int64_t)(*q.flag_count);
    int sy0, sy1, sx0, sx1;
    scan_range(W, limit, sy0, sy1, sx0, sx1);
    for (int64_t item = blockIdx.x; item < nwork; item += gridDim.x) {
        const int g = q.flag_list[item];
        int lo = 0, hi = q.n_items - 1;   // pair of combined window g
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (q.first_win[mid] <= g) lo = mid;
            else hi = mid - 1;
        }
        const PivParams& p = q.items[lo];
        const int64_t w = (int64_t)(g - q.first_win[lo]);
        if (nwork <= p.flag_cap &&
            refine_window<PixT>(p, w, W, mode, p.flag_recs[item], reinterpret_cast<unsigned char*>(sm), rs))
            continue;
        exact_window<PixT>(p, w, W, mode, sy0, sy1, sx0, sx1, sm, sm + W * W, row_count, &total_cand);
    }
}

template <typename PixT, bool LIST>
cudaError_t launch_t(const PivParams& p, int w, int mode, int limit, int blocks, cudaStream_t s)
{
    const size_t smem = 2 * sizeof(double2) * (size_t)w * w;
    // the opt-in limit for the largest window, once per device
    static std::atomic<uint64_t> attr_done{ 0 };
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (!(attr_done.load() & bit)) {
        const cudaError_t e = cudaFuncSetAttribute(piv_exact_kernel<PixT, LIST>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)(2 * sizeof(double2) * 64 * 64));
        if (e != cudaSuccess) return e;
        attr_done.fetch_or(bit);
    }
    if (LIST)
        return launch_dependent(piv_exact_kernel<PixT, LIST>, (unsigned)blocks, kThreads, smem, s, p, w, mode, limit);
    piv_exact_kernel<PixT, LIST><<<blocks, kThreads, smem, s>>>(p, w, mode, limit);
    return cudaGetLastError();
}

// Threads per CTA of the queue's exact kernel: the kernel needs at least W
// threads (one per plane row in the peak scan).  16 px windows (8 KB of
// shared memory) run one warp each, so that about 28 share an SM instead of
// 8; larger windows are held to a few per SM by shared memory anyway.
inline int exact_queue_threads(int w) { return w <= 16 ? 32 : kThreads; }

template <typename PixT>
cudaError_t queue_t(const PivQueue& q, int w, int mode, int limit, int blocks, cudaStream_t s)
{
    const size_t smem = 2 * sizeof(double2) * (size_t)w * w;
    static std::atomic<uint64_t> attr_done{ 0 };
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (!(attr_done.load() & bit)) {
        const cudaError_t e = cudaFuncSetAttribute(piv_exact_queue_kernel<PixT>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)(2 * sizeof(double2) * 64 * 64));
        if (e != cudaSuccess) return e;
        attr_done.fetch_or(bit);
    }
    if (blocks <= 0) return cudaSuccess;
    piv_exact_queue_kernel<PixT><<<blocks, exact_queue_threads(w), smem, s>>>(q, w, mode, limit);
    return cudaGetLastError();
}

// ---- the per-window spectral API: FFT::transform, transform_real and
// auto_correlate (fft.h:87-186, :229-242) on a batch of windows, in the
// reference's double arithmetic (the same butterflies, twiddle tables,
// complex products and unpack as the correlation above).  One CTA per
// window (CTAs stride over the batch); X is one W x W double2 tile of
// shared memory.
template <int OP>
__global__ void __launch_bounds__(kThreads)
spectral_exact_kernel(const SpectralParams q)
{
    extern __shared__ double2 X[];
    const int W = q.w, N = W * W, t = threadIdx.x;
    for (int64_t w = blockIdx.x; w < q.n; w += gridDim.x) {
        const size_t o = (size_t)w * N;
        // transform: the input converted to complex (image::operator=,
        // image.h:136-145); transform_real: join_from_channels(a, b)
        // (image_utils.impl.h:288-315); auto_correlate: transform(a)
        for (int i = t; i < N; i += blockDim.x)
            X[i] = OP == kSpectralReal ? make_double2(q.in_ra[o + i], q.in_rb[o + i]) : q.in_c[o + i];
        __syncthreads();
        fft2d(X, W, q.tw);
        if (OP == kSpectralTransform) {
            for (int i = t; i < N; i += blockDim.x) q.out_a[o + i] = X[i];
        } else if (OP == kSpectralReal) {
            // the partial unpack of fft.h:163-183 into two zeroed spectra:
            // rows [1, H/2) x columns [1, W) and their mirrors
            for (int i = t; i < N; i += blockDim.x) {
                q.out_a[o + i] = make_double2(0.0, 0.0);
                q.out_b[o + i] = make_double2(0.0, 0.0);
            }
            __syncthreads();
            const int npairs = (W / 2 - 1) * (W - 1);
            for (int k = t; k < npairs; k += blockDim.x) {
                const int h = 1 + k / (W - 1), x = 1 + k % (W - 1);
                const int i = h * W + x, m = (W - h) * W + (W - x);
                const double2 t1 = X[i], t2 = X[m];
                const double2 half = make_double2(0.5, 0.0);
                const double2 av = e_mul(half, e_add(t1, e_conj(t2)));
                double2 bv = e_mul(half, e_sub(t1, e_conj(t2)));
                bv = make_double2(bv.y, __dmul_rn(-1.0, bv.x));
                q.out_a[o + i] = av;
                q.out_a[o + m] = e_conj(av);
                q.out_b[o + i] = bv;
                q.out_b[o + m] = e_conj(bv);
            }
        } else {
            // |A|^2 = (A * conj A).real (pixel_types.h:198), as a complex
            // image with zero imaginary parts; the unnormalised inverse;
            // its real part, quadrant-swapped (image_utils.impl.h:367-386)
            for (int i = t; i < N; i += blockDim.x) X[i] = make_double2(e_mul(X[i], e_conj(X[i])).x, 0.0);
            __syncthreads();
            fft2d(X, W, q.tw + W);
            for (int i = t; i < N; i += blockDim.x) {
                const int y = i / W, x = i % W;
                const int sy = (y + W / 2) % W, sx = (x + W / 2) % W;
                q.out_a[o + i] = make_double2(X[sy * W + sx].x, 0.0);
            }
        }
        __syncthreads();
    }
}

template <int OP>
cudaError_t spectral_t(const SpectralParams& q, int blocks, cudaStream_t s)
{
    const size_t smem = sizeof(double2) * (size_t)q.w * q.w;
    static std::atomic<uint64_t> attr_done{ 0 };
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (!(attr_done.load() & bit)) {
        const cudaError_t e = cudaFuncSetAttribute(spectral_exact_kernel<OP>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)(sizeof(double2) * kMaxW * kMaxW));
        if (e != cudaSuccess) return e;
        attr_done.fetch_or(bit);
    }
    spectral_exact_kernel<OP><<<blocks, kThreads, smem, s>>>(q);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_spectral_exact(const SpectralParams& q, int op, int blocks, cudaStream_t s)
{
    if (!exact_supports(q.w) || blocks <= 0 || q.n <= 0) return cudaErrorInvalidValue;
    switch (op) {
    case kSpectralTransform: return spectral_t<kSpectralTransform>(q, blocks, s);
    case kSpectralReal: return spectral_t<kSpectralReal>(q, blocks, s);
    case kSpectralAuto: return spectral_t<kSpectralAuto>(q, blocks, s);
    default: return cudaErrorInvalidValue;
    }
}

int exact_queue_max_ctas_per_sm(int w)
{
    int n = 0;
    const size_t smem = 2 * sizeof(double2) * (size_t)w * w;
    if (queue_t<uint16_t>(PivQueue{}, w, 0, 0, 0, nullptr) != cudaSuccess) return 1;   // attribute set-up only
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, piv_exact_queue_kernel<uint16_t>,
                                                      exact_queue_threads(w), smem) !=
        cudaSuccess)
        return 1;
    return n < 1 ? 1 : n;
}

cudaError_t launch_piv_exact_queue(const PivQueue& q, int w, int dtype, int mode, int limit, int blocks,
                                   cudaStream_t s)
{
    if (!exact_supports(w) || blocks <= 0) return cudaErrorInvalidValue;
    switch (dtype) {
    case kU8: return queue_t<uint8_t>(q, w, mode, limit, blocks, s);
    case kU16: return queue_t<uint16_t>(q, w, mode, limit, blocks, s);
    case kF32: return queue_t<float>(q, w, mode, limit, blocks, s);
    default: return cudaErrorInvalidValue;
    }
}

bool exact_supports(int w) { return w >= 4 && w <= kMaxW && (w & (w - 1)) == 0; }

cudaError_t launch_piv_exact(const PivParams& p, int w, int dtype, int mode, int limit,
                             bool use_list, int blocks, cudaStream_t s)
{
    if (!exact_supports(w) || blocks <= 0) return cudaErrorInvalidValue;
    switch (dtype) {
    case kU8:
        return use_list ? launch_t<uint8_t, true>(p, w, mode, limit, blocks, s)
                        : launch_t<uint8_t, false>(p, w, mode, limit, blocks, s);
    case kU16:
        return use_list ? launch_t<uint16_t, true>(p, w, mode, limit, blocks, s)
                        : launch_t<uint16_t, false>(p, w, mode, limit, blocks, s);
    case kF32:
        return use_list ? launch_t<float, true>(p, w, mode, limit, blocks, s)
                        : launch_t<float, false>(p, w, mode, limit, blocks, s);
    case kF64:   // the per-window API's double windows: never a list
        return use_list ? cudaErrorInvalidValue : launch_t<double, false>(p, w, mode, limit, blocks, s);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace opiv
