// The tracer's ray: its start and its walk over the bordered heightmap.
#pragma once

#include "sgb_internal.cuh"

namespace sgb {

// The tracer reads the heightmap from a copy with a one-cell border of +inf
// ([H + 2][W + 2], cell (x, y) at (x + 1) + (y + 1) * (W + 2)).  A ray that
// steps off the grid meets the border, whose height test is always true, so
// the loop needs no per-axis step counts; the cell it stopped on tells a
// border stop (no hit, as the reference's bounds check) from a hit.  Heights
// inside the grid are the caller's, +inf included.  Each load's index is
// clamped into the copy (one unsigned min a step), so every load stays inside
// it whatever the float tests do; a ray never leaves the copy (the border
// ends it first), and one that did would end on the clamped border cell and
// return -1.  (The clamp measured 2.7% faster than a compare and branch.)
//
// With CONE, an upper ray also reads its direction's early-exit table
// (cone.cu) every kBoundEvery steps: a ray above the bound of a cell it has
// passed can hit nothing from there on (every later cell is reachable from
// that cell), so it ends with no hit, as the reference's range test would
// end it or as it would leave the grid.  (Reading the bound every step,
// packed with the height, cost more in loads than the steps it saved.)
constexpr int kBoundEvery = 12;   // steps between bound checks (4: +7.4%, 8: +1.4%, 16: +1.7% at 1024^2)

// A ray at one of its cells: the parameter t at which it entered it, its next
// crossing times and its height at t = 0.
struct Ray {
    float t, tMaxX, tMaxY, oz;
    int cell;
};

__device__ __forceinline__ void dda_step(Ray& r, int sx, int step_y, float dX, float dY)
{
    // one step, as selects: lanes that step on different axes stay
    // converged (measured 119.6 -> 116.5 ms at 1024^2 against branches)
    const bool xs = r.tMaxX < r.tMaxY;
    r.t = fminf(r.tMaxX, r.tMaxY);   // = xs ? tMaxX : tMaxY (equal when not xs and equal)
    r.cell += xs ? sx : step_y;
    const float nx = __fadd_rn(r.tMaxX, dX), ny = __fadd_rn(r.tMaxY, dY);
    r.tMaxX = xs ? nx : r.tMaxX;
    r.tMaxY = xs ? r.tMaxY : ny;
}

// The ray of (gx, gy, base_z) in direction d on its first tested cell; false
// when it can hit nothing (its first step leaves the grid, or its height is
// NaN or +inf).
__device__ __forceinline__ bool ray_start(int W, int H, int gx, int gy, float base_z, const DirEntry& d, Ray& r)
{
    // Cdir * 2.0f is exact, so these match the reference fused or not.
    const float ox = __fadd_rn((float)gx, __fmul_rn(d.cx, 2.0f));
    const float oy = __fadd_rn((float)gy, __fmul_rn(d.cy, 2.0f));
    r.oz = __fadd_rn(base_z, __fmul_rn(d.cz, 2.0f));
    int ix = __float2int_rd(ox);
    int iy = __float2int_rd(oy);
    const bool px = d.cx >= 0.0f;
    const bool py = d.cy >= 0.0f;
    r.tMaxX = __fdiv_rn(px ? __fsub_rn(__fadd_rn((float)ix, 1.0f), ox) : __fsub_rn(ox, (float)ix), d.ax);
    r.tMaxY = __fdiv_rn(py ? __fsub_rn(__fadd_rn((float)iy, 1.0f), oy) : __fsub_rn(oy, (float)iy), d.ay);
    // The first step checks both coordinates (the start cell, never tested,
    // may lie up to two cells outside the grid); after it the ray is inside
    // and moves one cell a step, so it stops on the border at the latest.
    if (r.tMaxX < r.tMaxY) { r.t = r.tMaxX; ix += px ? 1 : -1; r.tMaxX = __fadd_rn(r.tMaxX, d.dX); }
    else                   { r.t = r.tMaxY; iy += py ? 1 : -1; r.tMaxY = __fadd_rn(r.tMaxY, d.dY); }
    if ((unsigned)ix >= (unsigned)W || (unsigned)iy >= (unsigned)H) return false;
    // A start height of NaN or +inf gives no hit in the reference (every test
    // on it is false, or true only for the height range); it would also keep
    // the border test false, so it ends here.  -inf still stops on the border.
    if (r.oz != r.oz || r.oz == __int_as_float(0x7f800000)) return false;
    r.cell = (ix + 1) + (iy + 1) * (W + 2);
    return true;
}

// Walks ray r from its cell on: the 1-based id of the cell it hits, 0 for
// none, -1 for a ray that passed the border.
template <bool UP, bool CONE>
__device__ __forceinline__ int ray_walk(const float* __restrict__ gpad, const float* __restrict__ bound, int W, int H,
                                        float maxz, Ray& r, const DirEntry& d)
{
    const int Wp = W + 2;
    const int sx = d.cx >= 0.0f ? 1 : -1;
    const int step_y = d.cy >= 0.0f ? Wp : -Wp;
    const unsigned last = (unsigned)Wp * (unsigned)(H + 2) - 1u;
    float zr;
    // the reference tests the height range before the hit; both end the ray,
    // and which one it was is decided once, after the loop
    if constexpr (CONE) {
        for (;;) {
            // The bound of the cell the group of steps starts on also bounds
            // every cell after it, so its load has the whole group to arrive.
            const float b = __ldg(bound + min((unsigned)r.cell, last));
#pragma unroll
            for (int k = 0; k < kBoundEvery; ++k) {
                zr = __fmaf_rn(d.cz, r.t, r.oz);
                if (zr > maxz || __fsub_rn(__ldg(gpad + min((unsigned)r.cell, last)), zr) > 0.01f) goto stopped;
                dda_step(r, sx, step_y, d.dX, d.dY);
            }
            if (__fmaf_rn(d.cz, r.t, r.oz) > b) return (unsigned)r.cell > last ? -1 : 0;
        }
    } else {
        for (;;) {
            zr = __fmaf_rn(d.cz, r.t, r.oz);
            if ((UP ? (zr > maxz) : (zr < 0.0f)) || __fsub_rn(__ldg(gpad + min((unsigned)r.cell, last)), zr) > 0.01f)
                goto stopped;
            dda_step(r, sx, step_y, d.dX, d.dY);
        }
    }
stopped:
    if ((unsigned)r.cell > last) return -1;
    if (UP ? (zr > maxz) : (zr < 0.0f)) return 0;
    const int row = r.cell / Wp, q = r.cell - row * Wp;
    if (q == 0 || q > W || row == 0 || row > H) return 0;   // the border: the ray left the grid
    return (q - 1) + (row - 1) * W + 1;
}

}  // namespace sgb
