// piv_fp32_w64.cu -- fused FP32 PIV kernel for 64 x 64 windows (sm_103a).
//
// A 64-point row does not fit one lane's registers next to everything else,
// so one CTA of 256 threads takes a pair of windows through one 64 x 64
// float2 tile in shared memory.  z = a + i b of a window is transformed by
// radix-8 decimation-in-frequency passes (64 = 8^2), each thread taking two
// 8-point butterflies a pass; a pass's output goes back where its input came
// from, and the base-8 digit reversal that this leaves is absorbed in which
// rows or columns the next pass reads:
//   1  pixels from the frames, columns 8-point                 -> tile
//   2  columns 8-point;  3  rows 8-point                       tile -> tile
//   4  rows 8-point in registers, for both bins k and -k of the unpack:
//      a thread takes the butterflies of spectrum row k_y and of row -k_y, so
//      4 conj(P) = (2 Im(Z Zm), |Z|^2 - |Zm|^2) with Zm = Z[-k]
//      (P = B conj A, fft.h:188-227) needs nothing of another thread's.
//      The first window's products wait in 16 registers while the second
//      window goes through 1 to 4 in the same tile; then
//      Q = conj(4 P1) + i conj(4 P2) is formed at k and -k, and since a
//      butterfly's eight bins are what the inverse's first row pass takes,
//      that pass runs on them at once                          -> tile
//   5  rows 8-point;  6, 7  columns 8-point: plane 1 + i plane 2, natural order
// (one forward 2-D FFT of Q gives both planes).  REAL mode zeroes spectrum
// row 0, row W/2 and column 0 (fft.h:166-183), COMPLEX the DC bin, whose
// pedestal is added back.  find_peaks(plane, 2, 1) (image_utils.impl.h:42-74)
// is a scan of both planes at once, the fit (impl:77-101), the vector of
// main.cpp:220-236 and the certification run on one warp per window.
//
// The tile is transposed: its lines are image columns x (spectrum columns
// k_x), 65 float2 apart, elements along a line are y.  Sixteen threads
// reading sixteen neighbouring lines, sixteen neighbouring elements, or step
// 4's mirrored elements (two reversed groups of eight) all hit distinct
// banks; a warp's pixel loads are 32 neighbours of one image row; and an
// element's offset from its butterfly's first is a compile-time constant.
//
// 2048 x 2048, u16, step 16 (15,625 windows): 464 us with two tiles, seventeen
// trips through shared memory and a serial fit on one thread, 240 us with
// this (13,300 warp instructions a window where it took 21,600).  Packed FP32
// (add2, sub2, fma2) took 268 to 242 us of that: issue slots are 70 % busy
// (L1 and shared memory 81 %), so one instruction for both components pays
// although the FP32 pipe's rate is the same.  One tile (33 KB) and 64
// registers let four CTAs share an SM.

#include <atomic>
#include <cstdint>
#include <cuda_runtime.h>

#include "fft_reg.cuh"
#include "offsets.cuh"
#include "peak_scan.cuh"
#include "piv_kernels.h"

namespace opiv {
namespace w64 {

constexpr int W = 64;
constexpr int N = W * W;
constexpr int LD = W + 1;            // row stride (float2), odd: rows fall on distinct banks
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kCtasPerSm = 4;

// base-8 digit reversal of a 6-bit index (an involution)
__device__ __forceinline__ int dr(int v) { return ((v & 7) << 3) | (v >> 3); }

__device__ __forceinline__ float2 cmul(float2 a, float2 w)
{
    return make_float2(fmaf(a.x, w.x, -a.y * w.y), fmaf(a.x, w.y, a.y * w.x));
}

// In-place forward 8-point DFT, natural order in and out.
__device__ __forceinline__ void dft8(float2* x)
{
    constexpr float r = 0.70710678118654752f;   // cos(pi/4)
    const float2 a0 = add2(x[0], x[4]), a1 = sub2(x[0], x[4]), a2 = add2(x[2], x[6]), a3 = sub2(x[2], x[6]);
    const float2 a4 = add2(x[1], x[5]), a5 = sub2(x[1], x[5]), a6 = add2(x[3], x[7]), a7 = sub2(x[3], x[7]);
    // even outputs: 4-point DFT of (a0, a4, a2, a6)
    const float2 e0 = add2(a0, a2), e1 = sub2(a0, a2), e2 = add2(a4, a6), e3 = sub2(a4, a6);
    x[0] = add2(e0, e2);
    x[4] = sub2(e0, e2);
    x[2] = make_float2(e1.x + e3.y, e1.y - e3.x);   // e1 - i e3
    x[6] = make_float2(e1.x - e3.y, e1.y + e3.x);   // e1 + i e3
    // odd outputs: 4-point DFT of (a1, a5 w, -i a3, a7 w^3), w = exp(-i pi/4)
    const float2 b1 = make_float2((a5.x + a5.y) * r, (a5.y - a5.x) * r);
    const float2 b3 = make_float2((a7.y - a7.x) * r, -(a7.x + a7.y) * r);
    const float2 o0 = make_float2(a1.x + a3.y, a1.y - a3.x), o1 = make_float2(a1.x - a3.y, a1.y + a3.x);
    const float2 o2 = add2(b1, b3), o3 = sub2(b1, b3);
    x[1] = add2(o0, o2);
    x[5] = sub2(o0, o2);
    x[3] = make_float2(o1.x + o3.y, o1.y - o3.x);   // o1 - i o3
    x[7] = make_float2(o1.x - o3.y, o1.y + o3.x);   // o1 + i o3
}

// An 8-point butterfly over tile elements T[0], T[S], .. T[7 S].
template <int S>
__device__ __forceinline__ void load8(const float2* T, float2 (&x)[8])
{
#pragma unroll
    for (int m = 0; m < 8; ++m) x[m] = T[m * S];
}
template <int S>
__device__ __forceinline__ void store8(float2* T, const float2 (&x)[8])
{
#pragma unroll
    for (int m = 0; m < 8; ++m) T[m * S] = x[m];
}
// Output m of a first pass's butterfly j is scaled by exp(-2 pi i j m / 64):
// row j of the table, in four 16-byte loads (a warp's lanes share j).
constexpr int kTwRow = 8;
struct twiddles {
    float4 w[4];
    __device__ __forceinline__ twiddles(const float2* tw, int j)
    {
        const float4* q = reinterpret_cast<const float4*>(tw + j * kTwRow);
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = q[i];
    }
    __device__ __forceinline__ void scale(float2 (&x)[8]) const
    {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (i > 0) x[2 * i] = cmul(x[2 * i], make_float2(w[i].x, w[i].y));
            x[2 * i + 1] = cmul(x[2 * i + 1], make_float2(w[i].z, w[i].w));
        }
    }
};

// Passes over the whole tile: along its lines (lanes take lines, so a
// warp's j is uniform) or across them, elements 8 j + m or j + 8 m.
template <bool ALONG, bool BLOCK, bool TWIDDLE>
__device__ __forceinline__ void pass8(float2* T, const float2* tw)
{
    const int line = (int)threadIdx.x & 63;
#pragma unroll
    for (int it = 0; it < 2; ++it) {
        const int j = ((int)threadIdx.x >> 6) + 4 * it;
        float2 x[8];
        constexpr int E = ALONG ? 1 : LD, L = ALONG ? LD : 1;   // element and line strides
        float2* e = T + line * L + (BLOCK ? 8 * j : j) * E;
        load8<(BLOCK ? 1 : 8) * E>(e, x);
        dft8(x);
        if (TWIDDLE) twiddles(tw, j).scale(x);
        store8<(BLOCK ? 1 : 8) * E>(e, x);
    }
    __syncthreads();
}

// ---- the unpack's pairs of bins ------------------------------------------------
// A thread's butterflies: A at spectrum row ky, j (bins kx = j + 8 m) and B at
// row -ky, -j.  Bin m of A mirrors bin 7 - m of B, or (8 - m) & 7 where j = 0.
// Threads of warps 0 .. 5 take j = 1, 2, 3 and every row; warp 6 takes j = 0
// and warp 7 j = 4 with one row of each mirrored two (tile elements 1 .. 3,
// 36 .. 39, 8 .. 31), whose lane 0 holds the two that mirror themselves,
// ky = 0 (A) and W/2 (B).  In the tile's digit-reversed order -ky of the eight
// elements 8 g .. 8 g + 7 are the eight of group 8 - g, reversed (group 0:
// its own, reversed but for the first).
struct pair_slot {
    float im, d;   // 2 Im(Z Zm), |Z|^2 - |Zm|^2 at A's bin; at B's bin im, -d
};
__device__ __forceinline__ pair_slot product(float2 z, float2 m)
{
    const float2 p = four_conj_p(z, m);
    return pair_slot{ p.x, p.y };
}
// Q = conj(4 P1) + i conj(4 P2) at A's bin and at its mirror
__device__ __forceinline__ float2 q_at(pair_slot a, pair_slot b) { return make_float2(a.im - b.d, a.d + b.im); }
__device__ __forceinline__ float2 q_mirror(pair_slot a, pair_slot b) { return make_float2(a.im + b.d, b.im - a.d); }

__device__ __forceinline__ void pick(float2& a, float2& b, float2& c, bool rotate)
{   // (a, b, c) -> (c', a', b') = (b, c, a) when rotating
    const float2 x = a, y = b, z = c;
    a = rotate ? y : x;
    b = rotate ? z : y;
    c = rotate ? x : z;
}
// Lane 0 of warp 7: both rows mirror themselves with 7 - m; exchanging
// quarters makes its pairs those of the other threads, (X[m], Y[7 - m]) with
// X = A[0..3], B[0..3] and Y = B[4..7], A[4..7].
__device__ __forceinline__ void to_pairs(float2 (&A)[8], float2 (&B)[8], bool self)
{
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        pick(A[4 + i], B[i], B[4 + i], self);   // A[4+i] <- B[i], B[i] <- B[4+i], B[4+i] <- A[4+i]
    }
}
__device__ __forceinline__ void from_pairs(float2 (&A)[8], float2 (&B)[8], bool self)
{
#pragma unroll
    for (int i = 0; i < 4; ++i) pick(B[4 + i], B[i], A[4 + i], self);   // the inverse exchange
}

// Products of a window's bins, one slot per pair.
__device__ __forceinline__ void products(float2 (&A)[8], float2 (&B)[8], int j, bool self, pair_slot (&s)[8])
{
    if (j != 0) {
        if (j == 4) to_pairs(A, B, self);
#pragma unroll
        for (int m = 0; m < 8; ++m) s[m] = product(A[m], B[7 - m]);
    } else if (!self) {
#pragma unroll
        for (int m = 0; m < 8; ++m) s[m] = product(A[m], B[(8 - m) & 7]);
    } else {   // rows 0 and W/2 themselves: bins 0 and 4 are their own mirrors (d = 0), kept in one slot
        s[0] = pair_slot{ product(A[0], A[0]).im, product(A[4], A[4]).im };
        s[4] = pair_slot{ product(B[0], B[0]).im, product(B[4], B[4]).im };
#pragma unroll
        for (int m = 1; m < 4; ++m) {
            s[m] = product(A[m], A[8 - m]);
            s[4 + m] = product(B[m], B[8 - m]);
        }
    }
}
// Q at all bins of the two butterflies from both windows' products.
__device__ __forceinline__ void pack(const pair_slot (&s1)[8], const pair_slot (&s2)[8], int j, bool self,
                                     float2 (&A)[8], float2 (&B)[8])
{
    if (j != 0) {
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            A[m] = q_at(s1[m], s2[m]);
            B[7 - m] = q_mirror(s1[m], s2[m]);
        }
        if (j == 4) from_pairs(A, B, self);
    } else if (!self) {
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            A[m] = q_at(s1[m], s2[m]);
            B[(8 - m) & 7] = q_mirror(s1[m], s2[m]);
        }
    } else {
        A[0] = make_float2(s1[0].im, s2[0].im);
        A[4] = make_float2(s1[0].d, s2[0].d);
        B[0] = make_float2(s1[4].im, s2[4].im);
        B[4] = make_float2(s1[4].d, s2[4].d);
#pragma unroll
        for (int m = 1; m < 4; ++m) {
            A[m] = q_at(s1[m], s2[m]);
            A[8 - m] = q_mirror(s1[m], s2[m]);
            B[m] = q_at(s1[4 + m], s2[4 + m]);
            B[8 - m] = q_mirror(s1[4 + m], s2[4 + m]);
        }
    }
}

// Pixels a + i b to float, exactly (8/16-bit: into the mantissa of 2^23).
template <typename PixT>
__device__ __forceinline__ float2 widen(PixT a, PixT b)
{
    if constexpr (sizeof(PixT) <= 2)
        return sub2(make_float2(__uint_as_float(0x4B000000u | a), __uint_as_float(0x4B000000u | b)),
                    make_float2(8388608.f, 8388608.f));
    else
        return make_float2((float)a, (float)b);
}

__device__ __forceinline__ void window_origin(const PivParams& p, int w, int& bx, int& by)
{
    if (p.win_xy != nullptr) {
        bx = p.win_xy[2 * w];
        by = p.win_xy[2 * w + 1];
    } else {
        const int gy = (int)((unsigned)w / (unsigned)p.gnx);
        bx = p.gx0 + (w - gy * p.gnx) * p.gdx;
        by = p.gy0 + gy * p.gdy;
    }
}

extern __shared__ float2 w64_dyn_smem[];

// One task: windows 2 blk and 2 blk + 1 of pair p, run by the whole CTA.
template <int MODE, bool LIMIT, typename PixT, bool PLANES>
__device__ __forceinline__ void w64_task(const PivParams& p, const int blk)
{
    constexpr int D0 = LIMIT ? W / 4 : 0;
    constexpr int VW = LIMIT ? W / 2 : W;
    constexpr int SY0 = D0 + 1, SY1 = D0 + VW - 2;
    constexpr int SX0 = D0 + 1, SX1 = D0 + VW - 1;

    float2* T = w64_dyn_smem;
    __shared__ __align__(16) float2 tw[8 * kTwRow];
    __shared__ float s_energy[kWarps];
    __shared__ __align__(16) Top2 s_top[2][kWarps];
    __shared__ float s_ped[2];

    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int w0 = 2 * blk;
    if (w0 >= (int)p.n_win) return;
    const bool valid1 = w0 + 1 < (int)p.n_win;
    if (t < 64) {
        const int k = ((t >> 3) * (t & 7)) & 63;
        tw[(t >> 3) * kTwRow + (t & 7)] = make_float2(c_tw.re[k], c_tw.im[k]);
    }
    __syncthreads();

    // the thread's pair of row butterflies (step 4)
    const bool low = warp < 6;
    const int j = low ? 1 + (warp >> 1) : (warp == 6 ? 0 : 4);
    const int jb = (8 - j) & 7;
    const int ca = low ? t & 63 : lane >= 4 && lane < 8 ? 32 + lane : lane;   // tile element of ky, of -ky
    const bool self = !low && lane == 0;
    const int cb = self ? dr(W / 2) : dr((W - dr(ca)) & (W - 1));
    float2* const ea = T + 8 * j * LD + ca;
    float2* const eb = T + 8 * jb * LD + cb;

    float2 energy = make_float2(0.f, 0.f);
    int bad = 0;      // float windows: kBad bits, the second window's two up
    pair_slot first[8];
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
        float2 A[8], B[8];
        if (h == 0 || valid1) {   // CTA-uniform
            int bx, by, ox, oy;
            window_origin(p, w0 + h, bx, by);
            b_offset(p, W, bx, by, ox, oy);
            const size_t pitch = p.pitch / sizeof(PixT);
            const int x = t & 63;
            const PixT* fa = reinterpret_cast<const PixT*>(p.fa) + (size_t)by * pitch + bx + x;
            const PixT* fb = reinterpret_cast<const PixT*>(p.fb) + (size_t)(by + oy) * pitch + bx + ox + x;
            double sa = 0.0, sb = 0.0;
            const float2 before = energy;
#pragma unroll
            for (int it = 0; it < 2; ++it) {
                const int j1 = (t >> 6) + 4 * it;   // rows j1 + 8 m of column x
                const PixT *pa = fa + (size_t)j1 * pitch, *pb = fb + (size_t)j1 * pitch;
                float2 v[8];
#pragma unroll
                for (int m = 0; m < 8; ++m) {
                    const PixT a = __ldg(pa), b = __ldg(pb);
                    pa += 8 * pitch;
                    pb += 8 * pitch;
                    v[m] = widen(a, b);
                    energy = fma2(v[m], v[m], energy);
                    if (PLANES) {   // the per-window API's exact pedestal (double frames)
                        sa += (double)a;
                        sb += (double)b;
                    }
                }
                dft8(v);
                twiddles(tw, j1).scale(v);
                store8<8>(T + x * LD + j1, v);
            }
            if (PLANES) {
                double* red = reinterpret_cast<double*>(&s_top[0][0]);   // 2 kWarps doubles, free until the scan
                for (int o = 16; o > 0; o >>= 1) {
                    sa += __shfl_xor_sync(0xffffffffu, sa, o);
                    sb += __shfl_xor_sync(0xffffffffu, sb, o);
                }
                if (lane == 0) {
                    red[2 * warp] = sa;
                    red[2 * warp + 1] = sb;
                }
                __syncthreads();
                if (t == 0) {
                    sa = sb = 0.0;
                    for (int i = 0; i < kWarps; ++i) {
                        sa += red[2 * i];
                        sb += red[2 * i + 1];
                    }
                    p.peds[w0 + h] = (MODE == kModeComplex) ? sa * sb : 0.0;
                }
            }
            if constexpr (sizeof(PixT) >= 4) {
                const float e = energy.x + energy.y;
                if (__syncthreads_or(!(e < max_energy<PLANES>(W, kThreads)))) {
                    bad |= (__syncthreads_or(e != e) ? kBadNan : kBadHuge) << (2 * h);
                    energy = before;
                    for (int i = t >> 6; i < W; i += kThreads / W) T[x * LD + i] = make_float2(0.f, 0.f);
                    __syncthreads();
                }
            } else {
                __syncthreads();
            }
            pass8<true, true, false>(T, tw);
            pass8<false, false, true>(T, tw);
            load8<LD>(ea, A);
            load8<LD>(eb, B);
            dft8(A);
            dft8(B);
            if (MODE == kModeComplex) {   // the DC bin (sum a, sum b)
                if (self && j == 0) {
                    s_ped[h] = 4.f * A[0].x * A[0].y;
                    A[0] = make_float2(0.f, 0.f);
                }
            } else {                      // spectrum row 0, row W/2, column 0
                const float2 zero = make_float2(0.f, 0.f);
                // elements 0 and 4 are ky = 0 and W/2
                const bool zero_a = (ca & ~4) == 0, zero_b = (cb & ~4) == 0;
#pragma unroll
                for (int m = 0; m < 8; ++m) {
                    A[m] = zero_a || (m == 0 && j == 0) ? zero : A[m];
                    B[m] = zero_b || (m == 0 && j == 0) ? zero : B[m];
                }
                if (t == 0) s_ped[h] = 0.f;
            }
        } else {
#pragma unroll
            for (int m = 0; m < 8; ++m) A[m] = B[m] = make_float2(0.f, 0.f);
        }
        if (h == 0) {
            products(A, B, j, self, first);
            __syncthreads();   // the tile is read: the second window's rows may come
        } else {
            pair_slot second[8];
            products(A, B, j, self, second);
            pack(first, second, j, self, A, B);
            dft8(A);
            dft8(B);
            twiddles(tw, j).scale(A);
            twiddles(tw, jb).scale(B);
            store8<LD>(ea, A);
            store8<LD>(eb, B);
        }
    }
    {
        float e = energy.x + energy.y;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
        if (lane == 0) s_energy[warp] = e;
    }
    __syncthreads();
    pass8<false, false, false>(T, tw);
    pass8<true, true, true>(T, tw);
    pass8<true, false, false>(T, tw);

    // T[x * LD + y] = plane1(y, x) + i plane2(y, x), 4x scaled, before
    // the quadrant swap
    auto cell = [&](int ys, int xs) -> float2 {   // by swapped-plane coordinates
        return T[((xs + W / 2) & (W - 1)) * LD + ((ys + W / 2) & (W - 1))];
    };
    float total = 0.f;
#pragma unroll
    for (int i = 0; i < kWarps; ++i) total += s_energy[i];
    const float dlt = p.kappa * 5.9604645e-8f * 2.f * (float)N * total;

    if (PLANES)
        for (int h = 0; h < (valid1 ? 2 : 1); ++h)
            for (int i = t; i < N; i += kThreads) {
                const float2 v = cell(i >> 6, i & 63);
                p.planes[(size_t)(w0 + h) * N + i] =
                    (bad >> (2 * h)) & 3 ? __int_as_float(0x7fffffff) : 0.25f * (h ? v.y : v.x);
            }

    // ---- find_peaks on both planes at once: thread = (column, 16-row
    // block); its column rolls through registers
    Top2 s[2];
    s[0].init();
    s[1].init();
    {
        const int xs = t & 63, yb = (t >> 6) * 16;
        if (yb + 16 > SY0 && yb < SY1) {   // warp-uniform
            const float2* row = T + ((yb + W / 2) & (W - 1));
            const float2* cc0 = row + ((xs + W / 2) & (W - 1)) * LD;
            const float2* lf0 = row + ((xs + W / 2 - 1) & (W - 1)) * LD;
            const float2* rt0 = row + ((xs + W / 2 + 1) & (W - 1)) * LD;
            float2 up = cell(yb - 1, xs), cc = cc0[0];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const float2 dn = i < 15 ? cc0[i + 1] : cell(yb + 16, xs);
                const float2 lf = lf0[i], rt = rt0[i];
                const int ys = yb + i;
                if (ys >= SY0 && ys < SY1) {
                    s[0].add(cc.x, max4(up.x, dn.x, lf.x, rt.x), dlt, i);
                    s[1].add(cc.y, max4(up.y, dn.y, lf.y, rt.y), dlt, i);
                }
                up = cc;
                cc = dn;
            }
            s[0].key = (yb + s[0].key) * W + xs;   // unused where nothing was found
            s[1].key = (yb + s[1].key) * W + xs;
            if (xs < SX0 || xs >= SX1) {
                s[0].init();
                s[1].init();
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s[0].merge(s[0].across(o));
        s[1].merge(s[1].across(o));
    }
    if (lane < 2) s_top[lane][warp] = lane ? s[1] : s[0];
    __syncthreads();

    // ---- window h: warp h reduces, fits and writes
    if (warp < 2 && (warp == 0 || valid1)) {
        const int h = warp, w = w0 + h;
        Top2 g = s_top[h][lane & (kWarps - 1)];
#pragma unroll
        for (int o = kWarps / 2; o > 0; o >>= 1) g.merge(g.across(o));
        const float ped = s_ped[h];
        auto val = [&](int ys, int xs) -> float {
            const float2 v = cell(ys, xs);
            return h ? v.y : v.x;
        };
        const int bad_h = (bad >> (2 * h)) & 3;
        const bool has2 = bad_h == 0 && g.t1 > kNegInf;
        const int px = has2 ? g.key % W : W / 2, py = has2 ? g.key / W : W / 2;
        const float vc = val(py, px), vl = val(py, px - 1), vr = val(py, px + 1);
        const float vu = val(py - 1, px), vd = val(py + 1, px);
        // the six logarithms on six lanes: ln(L/R), ln(L/C), ln(R/C) and
        // ln(U/D), ln(U/C), ln(D/C), each as log1p((num - den) / (den + ped))
        const int q = lane < 6 ? lane : 0;
        const float an = q == 0 || q == 1 ? vl : q == 2 ? vr : q == 3 || q == 4 ? vu : vd;
        const float ad = q == 0 ? vr : q == 3 ? vd : vc;
        const float lg = log1pf((an - ad) / (ad + ped));
        const float lxr = __shfl_sync(0xffffffffu, lg, 0), lyd = __shfl_sync(0xffffffffu, lg, 3);
        const float denx = __shfl_sync(0xffffffffu, lg, 1) + __shfl_sync(0xffffffffu, lg, 2);
        const float deny = __shfl_sync(0xffffffffu, lg, 4) + __shfl_sync(0xffffffffu, lg, 5);
        int slot = -1;
        if (lane == 0) {
            int bx, by, ox, oy;
            window_origin(p, w, bx, by);
            b_offset(p, W, bx, by, ox, oy);
            opiv_vector out{ 0.f, 0.f, 0.f, 0.f, 0.f };
            int32_t code = -1;
            bool certain;
            if (bad_h != 0) {
                certain = bad_h == kBadNan;
            } else if (!has2) {
                certain = !(g.umax > kNegInf);
            } else {
                const float C = vc + ped, L = vl + ped, R = vr + ped, U = vu + ped, D = vd + ped;
                const float nan = __int_as_float(0x7fffffff);
                const bool okx = L > 0.f && C > 0.f && R > 0.f;
                const bool oky = U > 0.f && C > 0.f && D > 0.f;
                const float fx = okx ? lxr / (2.f * denx) : nan;
                const float fy = oky ? lyd / (2.f * deny) : nan;
                const float mx = fminf(fminf(L, R), C), my = fminf(fminf(U, D), C);
                const float ex = okx ? (denx == 0.f ? 3.4e38f
                                        : dlt * (1.f + 4.f * fabsf(fx)) / (mx * 2.f * fabsf(denx)))
                                     : (mx < -dlt ? 0.f : 3.4e38f);
                const float ey = oky ? (deny == 0.f ? 3.4e38f
                                        : dlt * (1.f + 4.f * fabsf(fy)) / (my * 2.f * fabsf(deny)))
                                     : (my < -dlt ? 0.f : 3.4e38f);
                const float p0 = g.t0 + ped, p1 = g.t1 + ped;
                const float sn_err = 0.5f * dlt * (1.f / fabsf(p0) + 1.f / fabsf(p1));
                certain = (g.umax < g.t1 - 2.f * dlt) && (g.t0 - g.t1 > dlt) && (fabsf(p1) > dlt) &&
                          (ex < kFitTol) && (ey < kFitTol) &&
                          (p1 <= 0.f || sn_err < kSnTol * fminf(1.f + p0 / p1, kSnCap));
                out.x = (float)(bx + W / 2);
                out.y = (float)(p.img_h - (by + W / 2));
                out.u = (float)(W / 2 - px - ox) - fx;
                out.v = (float)(W / 2 - py - oy) - fy;
                out.sn = (p1 > 0.f) ? p0 / p1 : 0.f;
                code = g.key;
            }
            p.out_vec[w] = out;
            if (p.out_peak) p.out_peak[w] = code;
            if (p.out_disp)
                p.out_disp[w] = has2 ? pack_disp(px - W / 2 + ox, py - W / 2 + oy) : pack_disp(ox, oy);
            if (!certain && p.flag_list) {
                const unsigned int at = atomicAdd(p.flag_count, 1u);
                if (at < (unsigned int)p.flag_room) p.flag_list[at] = (int32_t)w + p.flag_base;
                if (at < (unsigned int)p.flag_cap) slot = (int)at;
            }
        }
        // a flagged window hands its candidates on
        if (!PLANES) slot = __shfl_sync(0xffffffffu, slot, 0);
        if (!PLANES && slot >= 0)   // without a bound: to the FP64 transforms
            record_group<W, 32, true, SY0, SY1, SX0, SX1>(T, h, bad_h == 0 ? dlt : 0.f, p.flag_recs + slot);
    }
}

template <int MODE, bool LIMIT, typename PixT, bool PLANES>
__global__ void __launch_bounds__(kThreads, kCtasPerSm)
piv_w64_kernel(const PivParams p)
{
    after_previous();
    w64_task<MODE, LIMIT, PixT, PLANES>(p, (int)blockIdx.x);
}

// Persistent form over a device work queue: each CTA takes q.chunk tasks
// (window pairs) at a time until the pass's tasks (every image pair's) run
// out, claiming the next chunk while the current one runs (thread 0 keeps
// the atomic's result in a register until the next barrier).  No CTA waits
// for another.
// Copies pair j's descriptor from global memory into `dst` (shared) with
// the CTA's threads; all threads then read it from there.
__device__ __forceinline__ const PivParams& cta_item(const PivQueue& q, int j, PivParams* dst)
{
    constexpr int NQ = (int)(sizeof(PivParams) / 16);
    const uint4* src = reinterpret_cast<const uint4*>(q.items_g + j);
    if ((int)threadIdx.x < NQ) reinterpret_cast<uint4*>(dst)[threadIdx.x] = __ldg(src + threadIdx.x);
    __syncthreads();
    return *dst;
}

template <int MODE, bool LIMIT, typename PixT>
__global__ void __launch_bounds__(kThreads, kCtasPerSm)
piv_w64_queue_kernel(const __grid_constant__ PivQueue q)
{
    __shared__ unsigned int s_t0;
    __shared__ __align__(16) unsigned char s_item[sizeof(PivParams)];
    const int n_tasks = q.first_task[q.n_items];
    unsigned int next = 0;
    if (threadIdx.x == 0) next = atomicAdd(q.head, (unsigned int)q.chunk);
#pragma unroll 1
    for (;;) {
        if (threadIdx.x == 0) s_t0 = next;
        __syncthreads();
        const unsigned int t0 = s_t0;
        __syncthreads();   // every thread has read s_t0 before it is written again
        if (t0 >= (unsigned int)n_tasks) break;
        if (threadIdx.x == 0) next = atomicAdd(q.head, (unsigned int)q.chunk);
        const int t1 = min((int)t0 + q.chunk, n_tasks);
#pragma unroll 1
        for (int t = (int)t0; t < t1; ++t) {
            const int j = __ldg(q.task_item + t);
            __syncthreads();   // the previous task's tile and descriptor are no longer read
            const PivParams& p = cta_item(q, j, reinterpret_cast<PivParams*>(s_item));
            w64_task<MODE, LIMIT, PixT, false>(p, t - q.first_task[j]);
        }
    }
}

template <int MODE, bool LIMIT, typename PixT, bool PLANES>
cudaError_t launch_t(const PivParams& p, cudaStream_t s)
{
    const size_t smem = sizeof(float2) * W * LD;
    static std::atomic<uint64_t> attr_done{ 0 };   // one bit per device
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (!(attr_done.load() & bit)) {
        const cudaError_t e = cudaFuncSetAttribute(piv_w64_kernel<MODE, LIMIT, PixT, PLANES>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)smem);
        if (e != cudaSuccess) return e;
        attr_done.fetch_or(bit);
    }
    const int64_t blocks = (p.n_win + 1) / 2;
    return launch_dependent(piv_w64_kernel<MODE, LIMIT, PixT, PLANES>, (unsigned)blocks, kThreads, smem, s, p);
}

template <int MODE, bool LIMIT>
cudaError_t launch_dt(const PivParams& p, int dtype, bool planes, cudaStream_t s)
{
    if (planes) return dtype == kF64 ? launch_t<MODE, LIMIT, double, true>(p, s) : cudaErrorInvalidValue;
    switch (dtype) {
    case kU8: return launch_t<MODE, LIMIT, uint8_t, false>(p, s);
    case kU16: return launch_t<MODE, LIMIT, uint16_t, false>(p, s);
    case kF32: return launch_t<MODE, LIMIT, float, false>(p, s);
    default: return cudaErrorInvalidValue;
    }
}

// The same work list dispatched by the hardware: CTA b runs task b, no
// persistent loop.
template <int MODE, bool LIMIT, typename PixT>
__global__ void __launch_bounds__(kThreads, kCtasPerSm)
piv_w64_list_kernel(const __grid_constant__ PivQueue q)
{
    __shared__ __align__(16) unsigned char s_item[sizeof(PivParams)];
    const int t = (int)blockIdx.x;
    const int j = __ldg(q.task_item + t);
    const PivParams& p = cta_item(q, j, reinterpret_cast<PivParams*>(s_item));
    w64_task<MODE, LIMIT, PixT, false>(p, t - q.first_task[j]);
}

// blocks > 0: the persistent kernel on `blocks` CTAs; blocks == 0: the
// hardware-dispatched list kernel, one CTA per task
template <int MODE, bool LIMIT, typename PixT>
cudaError_t queue_t(const PivQueue& q, int blocks, int* max_ctas, cudaStream_t s)
{
    const size_t smem = sizeof(float2) * W * LD;
    auto kern = piv_w64_queue_kernel<MODE, LIMIT, PixT>;
    auto list = piv_w64_list_kernel<MODE, LIMIT, PixT>;
    static std::atomic<uint64_t> attr_done{ 0 };   // one bit per device
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (!(attr_done.load() & bit)) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(list, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        attr_done.fetch_or(bit);
    }
    if (max_ctas) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(max_ctas, kern, kThreads, smem);
    if (blocks < 0) return cudaErrorInvalidValue;
    if (blocks == 0) {
        const int n_tasks = q.first_task[q.n_items];
        if (n_tasks <= 0) return cudaSuccess;
        list<<<(unsigned)n_tasks, kThreads, smem, s>>>(q);
    } else {
        kern<<<(unsigned)blocks, kThreads, smem, s>>>(q);
    }
    return cudaGetLastError();
}

template <int MODE, bool LIMIT>
cudaError_t queue_dt(const PivQueue& q, int dtype, int blocks, int* max_ctas, cudaStream_t s)
{
    switch (dtype) {
    case kU8: return queue_t<MODE, LIMIT, uint8_t>(q, blocks, max_ctas, s);
    case kU16: return queue_t<MODE, LIMIT, uint16_t>(q, blocks, max_ctas, s);
    case kF32: return queue_t<MODE, LIMIT, float>(q, blocks, max_ctas, s);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace w64

// the 64 px kernel loads rows element-wise and needs no alignment flag
cudaError_t queue_piv_fp32_w64(const PivQueue& q, int dtype, int mode, int limit, bool, int blocks,
                               int* max_ctas, cudaStream_t s)
{
    if (mode == kModeComplex)
        return limit ? w64::queue_dt<kModeComplex, true>(q, dtype, blocks, max_ctas, s)
                     : w64::queue_dt<kModeComplex, false>(q, dtype, blocks, max_ctas, s);
    return limit ? w64::queue_dt<kModeReal, true>(q, dtype, blocks, max_ctas, s)
                 : w64::queue_dt<kModeReal, false>(q, dtype, blocks, max_ctas, s);
}

cudaError_t launch_piv_fp32_w64(const PivParams& p, int dtype, int mode, int limit, bool planes,
                                cudaStream_t s)
{
    if (p.n_win <= 0) return cudaSuccess;
    if (mode == kModeComplex)
        return limit ? w64::launch_dt<kModeComplex, true>(p, dtype, planes, s)
                     : w64::launch_dt<kModeComplex, false>(p, dtype, planes, s);
    return limit ? w64::launch_dt<kModeReal, true>(p, dtype, planes, s)
                 : w64::launch_dt<kModeReal, false>(p, dtype, planes, s);
}

}  // namespace opiv
