// peak_scan.cuh -- find_peaks(plane, 2, 1) (image_utils.impl.h:42-74) with an
// error bound, as the FP32 kernels run it: the running top two, the thresholds
// of certification, and the windows left out of a pair's transform.
#pragma once
#include <cuda_runtime.h>

#include "piv_kernels.h"

namespace opiv {

// A window is decided by an FP32 kernel only if the error bound of its
// sub-pixel fit stays below kFitTol pixels and the relative error bound of
// its sn below kSnTol * (1 + sn).  The parity tolerances are 1e-4 px and
// 1e-5 * (1 + sn): sn = p0 / p1 is a ratio of plane values, and plane values
// are specified to 1e-5 of the plane peak p0, which bounds the relative
// error of p1 by 1e-5 * p0 / p1 = 1e-5 * sn.  The thresholds sit 1.6x inside
// those tolerances (the rounding of the final FP32 logarithms, sums and
// ratio adds ~1e-6 px and ~2e-7 relative on top of the bounds).  At 3e-5 /
// 3e-6 three times as many 16 px windows went to the exact pass, nearly all
// of them for the sn bound.  The factor 1 + sn ends at kSnCap: a few windows
// of sn in the tens, whose second peak is little more than rounding, carried
// nearly all of a field's sn error (2048 x 1536 field of 16 px windows: 1e-6 of
// its norm, 1e-7 with the cap, 139 windows flagged where 78 were; REAL mode
// with the limited search up to 1.5e-3 and 4e-8).
constexpr float kFitTol = 6e-5f;
constexpr float kSnTol = 6e-6f;
constexpr float kSnCap = 4.f;
#define kNegInf (-__int_as_float(0x7f800000))

// A window whose lanes' energies (`lanes` of them) stay below this overflows
// nowhere: plane and spectrum values are at most 8 W^2 times its energy.
// Beyond, and where a pixel is NaN, the pair is transformed without it (one
// transform carries both planes, so it would take the other window with it):
// with a NaN pixel every plane value is NaN and there is no peak; otherwise
// FP64 decides.  The per-window planes (double windows) only ask for finite.
template <bool PLANES>
__host__ __device__ constexpr float max_energy(int w, int lanes)
{
    return PLANES ? 3.4e38f : 3e38f / (8.f * (float)(w * w) * (float)lanes);
}
enum { kBadHuge = 1, kBadNan = 2 };

// a three-source max and a max
__device__ __forceinline__ float max4(float a, float b, float c, float d)
{
    float m;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(fmaxf(c, d)));
    return m;
}

// Running top-2 of strict 4-neighbour maxima (find_peaks) plus the largest
// value whose strict-maximum decision is within dlt of flipping.
struct Top2 {
    float t0, t1, umax;
    int key;
    __device__ __forceinline__ void init()
    {
        t0 = t1 = umax = kNegInf;
        key = 0;
    }
    __device__ __forceinline__ void add(float c, float m, float dlt, int k)
    {
        const float dd = m - c;
        umax = fabsf(dd) <= dlt ? fmaxf(umax, c) : umax;
        const float v = dd < 0.f ? c : kNegInf;
        t1 = fmaxf(t1, fminf(t0, v));
        key = v > t0 ? k : key;
        t0 = fmaxf(t0, v);
    }
    // with another's (ties to the lowest row-major index)
    __device__ __forceinline__ void merge(const Top2& o)
    {
        const bool take = (o.t0 > t0) || (o.t0 == t0 && o.key < key);
        t1 = fmaxf(fmaxf(t1, o.t1), fminf(t0, o.t0));
        key = take ? o.key : key;
        t0 = fmaxf(t0, o.t0);
        umax = fmaxf(umax, o.umax);
    }
    __device__ __forceinline__ Top2 across(int o) const   // the lane o away
    {
        Top2 r;
        r.t0 = __shfl_xor_sync(0xffffffffu, t0, o);
        r.t1 = __shfl_xor_sync(0xffffffffu, t1, o);
        r.umax = __shfl_xor_sync(0xffffffffu, umax, o);
        r.key = __shfl_xor_sync(0xffffffffu, key, o);
        return r;
    }
};

// The record of a flagged window, by LANES lanes of a warp; every lane calls
// it, with its group's arguments (rec null: nothing is written).  tile: both
// planes before the quadrant swap, the window's in component h; lines W + 1
// apart, of rows, or of columns where COLS.  dlt: the bound, zero for none.
// Scanned: swapped rows SY0 .. SY1 - 1 and columns SX0 .. SX1 - 1.  The order of
// the cells follows the scan, whichever lane finds them.
template <int W, int LANES, bool COLS, int SY0, int SY1, int SX0, int SX1>
__device__ __forceinline__ void record_candidates(const float2* tile, int h, float dlt, flag_record* rec)
{
    constexpr int NX = SX1 - SX0, NC = (SY1 - SY0) * NX;
    const int lane = (int)threadIdx.x & 31, gl = lane % LANES;
    auto cell = [&](int y, int x) -> float {
        y = (y + W / 2) & (W - 1);
        x = (x + W / 2) & (W - 1);
        const float2 v = tile[COLS ? x * (W + 1) + y : y * (W + 1) + x];
        return h ? v.y : v.x;
    };
    auto rise = [&](int y, int x, float c) {   // highest neighbour minus the cell
        return max4(cell(y - 1, x), cell(y + 1, x), cell(y, x - 1), cell(y, x + 1)) - c;
    };
    // the two highest cells that are maxima whatever the rounding: nothing
    // below the second of them (less the bound) matters
    float s0 = kNegInf, s1 = kNegInf;
#pragma unroll(LANES == 32 ? 4 : 2)
    for (int b = 0; b < NC; b += LANES) {
        const int i = b + gl, y = SY0 + i / NX, x = SX0 + i % NX;   // past the last: other cells of the tile
        const float c = cell(y, x);
        const float v = i < NC && rise(y, x, c) < -dlt ? c : kNegInf;
        s1 = fmaxf(s1, fminf(s0, v));
        s0 = fmaxf(s0, v);
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) {
        const float q0 = __shfl_xor_sync(0xffffffffu, s0, o), q1 = __shfl_xor_sync(0xffffffffu, s1, o);
        s1 = fmaxf(fmaxf(s1, q1), fminf(s0, q0));
        s0 = fmaxf(s0, q0);
    }
    const float floor_c = s1 - dlt;
    int n = 0;
#pragma unroll(LANES == 32 ? 4 : 2)
    for (int b = 0; b < NC; b += LANES) {
        const int i = b + gl, y = SY0 + i / NX, x = SX0 + i % NX;
        const float c = cell(y, x);
        const bool high = i < NC && c >= floor_c;
        if (!__any_sync(0xffffffffu, high)) continue;
        const bool mine = high && rise(y, x, c) <= dlt;
        const unsigned group = __ballot_sync(0xffffffffu, mine) >> (lane - gl) & (0xffffffffu >> (32 - LANES));
        const int at = n + __popc(group & ((1u << gl) - 1u));
        if (mine && rec != nullptr && at < kMaxCand) rec->key[at] = (uint16_t)(y * W + x);
        n += __popc(group);
    }
    if (rec != nullptr && gl == 0) {
        rec->n = n;
        rec->dlt = dlt;
    }
}

// Few windows are flagged, so the records are functions of their own: the
// others' code stays small (4096 x 4096, 32 px at step 8: 707 us, 716 inlined).
// record_group: a window by LANES lanes (32 px: a warp has two windows, and the
// loop of record_warp costs the kernel 8 us there).  record_warp: one window after
// the other by the whole warp; a lane whose slot is not negative speaks for a
// window (16 px, 2048 x 1536 at step 8: 42.5 us; 45.7 by a window's own eight lanes,
// whose scan the pass waits for).
template <int W, int LANES, bool COLS, int SY0, int SY1, int SX0, int SX1>
__device__ __noinline__ void record_group(const float2* tile, int h, float dlt, flag_record* rec)
{
    record_candidates<W, LANES, COLS, SY0, SY1, SX0, SX1>(tile, h, dlt, rec);
}
template <int W, bool COLS, int SY0, int SY1, int SX0, int SX1>
__device__ __noinline__ void record_warp(const float2* tile, int h, float dlt, int slot, flag_record* recs)
{
    for (unsigned todo = __ballot_sync(0xffffffffu, slot >= 0); todo != 0; todo &= todo - 1) {
        const int from = __ffs((int)todo) - 1;
        record_candidates<W, 32, COLS, SY0, SY1, SX0, SX1>(
            reinterpret_cast<const float2*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(tile), from)),
            __shfl_sync(0xffffffffu, h, from), __shfl_sync(0xffffffffu, dlt, from),
            recs + __shfl_sync(0xffffffffu, slot, from));
    }
}

}  // namespace opiv
