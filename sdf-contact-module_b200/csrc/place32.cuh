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
    __device__ __forceinline__ void set_margin(float far)
    {
        float m = 0.f;
#pragma unroll
        for (int q = 0; q < 9; ++q) m = fmaxf(m, fabsf(M[q]));
        e1 = m * 0x1p-21f;
        e0 = fmaxf(fabsf(t[0]), fmaxf(fabsf(t[1]), fabsf(t[2]))) * 0x1p-21f + 0x1p-28f + far * 0x1p-50f;
    }
};

// True: certainly inside the grid, in cell c at the fractions u -+ e.  *out:
// certainly outside.  Neither: only FP64 can tell.
__device__ __forceinline__ bool place32(const GridView& g, const Place32& f, float x, float y, float z, int c[3],
                                        float u[3], float& e, bool& out)
{
    e = __fmaf_rn(fabsf(x) + fabsf(y) + fabsf(z), f.e1, f.e0);
    const int n[3] = {g.nx, g.ny, g.nz};
    out = false;
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
    }
    return !out && edge > e && e < 0.25f && (unsigned)c[0] < (unsigned)(n[0] - 1) &&
           (unsigned)c[1] < (unsigned)(n[1] - 1) && (unsigned)c[2] < (unsigned)(n[2] - 1);
}

// Bounds of the trilinear gap at a point from the cell's FP32 corner record: true
// with the gap in g -+ eps, else *out as place32.  A coordinate off by e moves the
// interpolant by at most e times the corners' spread per axis; corners rounded
// to FP32 and an interpolation in FP32 or FP64 are each off by less than 2^-20
// of the largest corner.
__device__ __forceinline__ bool gap32(const GridView& g, const Place32& f, float x, float y, float z, float& gap,
                                      float& eps, bool& out)
{
    int c[3];
    float u[3], e;
    if (!place32(g, f, x, y, z, c, u, e, out)) return false;
    const float4* q = g.cell8 + 2 * (c[0] + (int64_t)g.nx * (c[1] + (int64_t)g.ny * c[2]));
    const float4 p = __ldg(q), w = __ldg(q + 1);
    auto mix = [](float a0, float a1, float k) { return __fmaf_rn(k, a1 - a0, a0); };
    gap = mix(mix(mix(p.x, p.y, u[0]), mix(p.z, p.w, u[0]), u[1]),
              mix(mix(w.x, w.y, u[0]), mix(w.z, w.w, u[0]), u[1]), u[2]);
    const float lo = fminf(fminf(fminf(p.x, p.y), fminf(p.z, p.w)), fminf(fminf(w.x, w.y), fminf(w.z, w.w)));
    const float hi = fmaxf(fmaxf(fmaxf(p.x, p.y), fmaxf(p.z, p.w)), fmaxf(fmaxf(w.x, w.y), fmaxf(w.z, w.w)));
    eps = __fmaf_rn(4.f * e, hi - lo, 0x1p-19f * fmaxf(fabsf(lo), fabsf(hi)));
    return fabsf(gap) < INFINITY && eps < INFINITY;
}

} // namespace sdfo
