// Points placed in a dense grid's cells in FP32, with a bound of the error: the
// contact kernel and the BE step tell with it which points need no FP64.
#pragma once

#include "sdfo_internal.cuh"

namespace sdfo {

// A pose's map from body A's points to grid index coordinates, f = M x + t with
// M = R_B^T R_A / h and t = (R_B^T (r_A - r_B) - bmin) / h - 1/2.  x, M, t and
// three fused steps are each rounded to 2^-24 of at most |M|max |x|_1 + |t|max.
// The FP64 path adds R_B^T (r_A - r_B) and takes bmin off in the grid's own
// coordinates, whose rounding is that of their size, however small t is.  So f is
// within e0 + e1 |x|_1 of the FP64 path's value.
struct Place32
{
    float M[9], t[3], e0, e1;

    // `far`: the largest (|R_B^T (r_A - r_B)| + |bmin|) / h of an axis
    __device__ __forceinline__ void set_margin(double far)
    {
        float m = 0.f;
#pragma unroll
        for (int q = 0; q < 9; ++q) m = fmaxf(m, fabsf(M[q]));
        e1 = m * 0x1p-21f;
        e0 = fmaxf(fabsf(t[0]), fmaxf(fabsf(t[1]), fabsf(t[2]))) * 0x1p-21f + 0x1p-28f + (float)(far * 0x1p-50);
    }
};

enum : int
{
    kOutside32 = 0, // certainly outside the grid
    kInside32 = 1,  // certainly inside, in cell c at the fractions u -+ e
    kUnsure32 = 2   // only FP64 can tell
};

__device__ __forceinline__ int place32(const GridView& g, const Place32& f, float x, float y, float z, int c[3],
                                       float u[3], float& e)
{
    e = __fmaf_rn(fabsf(x) + fabsf(y) + fabsf(z), f.e1, f.e0);
    const int n[3] = {g.nx, g.ny, g.nz};
    bool out = false, cell = true;
    float edge = 1.f; // distance to the nearest cell boundary
#pragma unroll
    for (int a = 0; a < 3; ++a)
    {
        const float v = __fmaf_rn(f.M[3 * a], x, __fmaf_rn(f.M[3 * a + 1], y, __fmaf_rn(f.M[3 * a + 2], z, f.t[a])));
        out = out || v < -e || v > (float)(n[a] - 1) + e;
        // floor by rounding v - 1/2 at 1.5 2^23 (e < 1/4: |v| < 2^19); a point that
        // this rounds the other way lies on a boundary, which `edge` tells
        const float r = (v - 0.5f) + 12582912.f;
        c[a] = __float_as_int(r) - 0x4b400000;
        u[a] = v - (r - 12582912.f);
        edge = fminf(edge, fminf(u[a], 1.f - u[a]));
        cell = cell && (unsigned)c[a] < (unsigned)(n[a] - 1);
    }
    return out ? kOutside32 : cell && edge > e && e < 0.25f ? kInside32 : kUnsure32;
}

} // namespace sdfo
