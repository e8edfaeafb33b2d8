// Warp-wide nearest-triangle search and binned parity rays over the
// reference-order tree: the fills' fast path, with the results of
// signed_nearest (build_common.cuh) bit for bit.
//
// What bounds the per-thread traversal: its threads diverge (6.4 of 32 lanes
// active on the hollow cylinder) and every node and most triangles cost FP64.
// Here a warp takes a compact patch of voxels (4 x 4 x 2) and walks the tree
// once for all its lanes (warp_nearest):
//   * node boxes and triangles are tested in FP32 with rigorous margins, a
//     subtree entered when any lane needs it, so the loop has no divergence
//     and every load is a broadcast;
//   * triangles that may be a lane's nearest go to a short list of the lane;
//     the reference's FP64 closest-point test runs on the few that are left
//     when the search ends.
// The search order differs from the reference's, so the smallest squared
// distance is found first and the triangle that the reference keeps among
// exactly equal ones is worked out afterwards (see flush_list).
//
// A patch about equally far from much of the mesh (the axis of a cylinder)
// enters hundreds of leaves, and one warp doing so outlasts the whole launch.
// Such a patch stops after kHeavyLeaves leaves; in a second launch a CTA takes
// it, its warps sharing out the subtrees.  Where there are no more pairs of
// patches than such CTAs, every search is latency, and kFewLeaves hands over
// sooner: 24 voxels along the longest side, 4,608 triangles of a cylinder 1.02 ->
// 0.76 ms for the build, 9,016 of a gear 1.37 -> 1.02, 20,480 of a ball 2.3 -> 2.0.
//
// The parity ray has one fixed direction.  The triangles are projected along
// it and binned on the plane; a voxel tests the triangles of its bin with FP32
// edge functions (conservative), and only the survivors with the reference's
// FP64 test.
//
// Voxels for which the argument of flush_list or of binned_ray_count does
// not hold (rounding at a box face) are marked and filled by the per-thread
// traversal in a third launch, as are whole meshes with more than
// kMaxUnbounded near-degenerate triangles, or whose long thin triangles crowd the
// ray's lists (kMaxCrowd): a 1,024-triangle pipe ten diameters long has 421
// entries where cylinders, gears and plates have 5 to 26, and its 64 x 64 x 128
// voxels took 0.73 ms here, 0.54 per thread.
//
// Measured (one B200, fill alone): 34,816-triangle hollow cylinder into
// 128 x 128 x 64 voxels 8.4 -> 2.0 ms; 327,680-triangle icosphere, 10.6 M
// voxels of a sparse 512^3 grid, 37.9 -> 8.1 ms.  Flat-faced parts gain nothing or
// lose a little, since a point near a plane has few candidates (builds of cubes,
// plates, rods and flat sheets of 768 to 12,288 triangles: 0.76 to 1.12 times the
// per-thread speed, the least for the smallest grids).  Bound now by instruction
// issue: 2.8 of 4 per cycle, about 34,000 per 64 voxels, of which a third FP32
// and a tenth FP64 (81,920 triangles, 256^3).  A triangle-box test ahead of the
// frame test changed nothing (7.2 against 7.3 ms).
#pragma once

#include <climits>

#include "build_common.cuh"

namespace sdfo {

namespace {

constexpr int kMaxUnbounded = 32;
constexpr int kWarpStack = 64;
constexpr int kLeafTris = 8;      // triangles of a leaf of the reference's tree, at most
constexpr int kLaneList = 8;      // triangles a lane keeps for the FP64 test
constexpr int kHeavyLeaves = 128; // leaves after which a patch is handed over,
constexpr int kFewLeaves = 16;    // where all patches fit the CTAs at once
constexpr int kHeavyWarps = 8;    // warps of the CTA that takes such a patch
constexpr int kHeavyBlocks = 3;   // such CTAs per SM
static_assert(kHeavyWarps <= kLaneList, "the warps' results are compared in a list");
constexpr int kPartDepth = 6;     // depth of the subtrees they share out
// Rays: a triangle goes to the finest level where it reaches at most this
// many cells, so the lists hold at most this many entries per triangle.
constexpr int kMaxCellsPerTri = 16;
constexpr int kMaxRayCells = 1024; // cells per side of the finest level
constexpr double kMaxCrowd = 128.0; // mean entries over the mesh's projected box

// state words of a WarpTree
enum : int
{
    kStateUnbounded = 0, // near-degenerate triangles
    kStateWild = 1,      // triangles whose rounding reaches past the plane
    kStateLevels = 2,    // bit l: level l holds triangles
    kStateMarked = 3,    // voxels left to the per-thread traversal
    kStateHeavy = 4,     // pairs of patches handed over
    kStateCrowd = 6,     // (64 bits) area of all list entries' cells, in finest cells
    kStateWords = 8
};

struct RayBins
{
    const float4* rec; // per slot: {ax, ay, bx, by}, {cx, cy, depth, tol}
    const int* off;    // CSR over the cells of all levels
    const int* ids;    // slots
    double e1[3], e2[3], o1, o2; // plane axes and lower corner
    double o3;         // the scene's middle along the ray
    double box_cells;  // area of the mesh's projected box, in finest cells
    double size;       // side of the plane's square
    double inv_cell;   // finest cells per unit length
    int g;             // finest cells per side (a power of two)
};

// What FP32 sees of the scene: points relative to its middle `o`, so that an
// offset from the origin costs no bits.  E: the half extent of mesh and grid
// about `o`; far: their largest coordinate.  FP64 differences to `o` are rounded
// to less than 2^-52 far.
struct Scene32
{
    double o[3], e, far;
};

struct WarpTreeView
{
    RefTreeView ref;
    double o[3];         // Scene32::o
    const float4* node4; // 4 float4 per node: both child boxes, child codes
    const float4* tri4;  // 5 float4 per slot: the triangle in its own frame (k_tri_frames)
    float bound_abs;     // warp_bound's absolute part, rounded up
    const int* unbounded; // slots of the near-degenerate triangles
    unsigned long long max_crowd; // of kStateCrowd
    int* heavy;          // first patches of the pairs handed over
    int max_leaves;      // leaves after which a pair is
    RayBins rays;
    int* state;
};

__device__ __forceinline__ bool warp_path_open(const WarpTreeView& t)
{
    return t.state[kStateUnbounded] <= kMaxUnbounded && t.state[kStateWild] == 0 &&
           *reinterpret_cast<const unsigned long long*>(t.state + kStateCrowd) <= t.max_crowd;
}

// Rounding of a point, a box or a distance that does not grow with the distance.
inline double scene_margin(const Scene32& c) { return std::ldexp(c.e, -20) + std::ldexp(c.far, -50); }

// {L.lo, L.hi, R.lo, R.hi} in FP32, rounded outward and widened by the margin,
// then the child codes: a node id, or ~id of a leaf.
__global__ void k_pack_node4(RefTreeView b, Scene32 sc, double margin, float4* __restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= b.nnodes) return;
    const int4 meta = __ldg(reinterpret_cast<const int4*>(b.nodes + i) + 3);
    if (meta.w > 0) return;
    const int ch[2] = {meta.x, meta.y};
    float f[12];
    int code[2];
    for (int k = 0; k < 2; ++k)
    {
        const RefNode& c = b.nodes[ch[k]];
        for (int a = 0; a < 3; ++a)
        {
            f[6 * k + a] = __double2float_rd(c.lo[a] - sc.o[a] - margin);
            f[6 * k + 3 + a] = __double2float_ru(c.hi[a] - sc.o[a] + margin);
        }
        code[k] = c.count > 0 ? ~ch[k] : ch[k];
    }
    float4* o = out + 4 * (int64_t)i;
    o[0] = make_float4(f[0], f[1], f[2], f[3]);
    o[1] = make_float4(f[4], f[5], f[6], f[7]);
    o[2] = make_float4(f[8], f[9], f[10], f[11]);
    o[3] = make_float4(__int_as_float(code[0]), __int_as_float(code[1]), 0.f, 0.f);
}

// Each triangle in slot order in its own frame: vertex a, the rows of the
// rotation to (along ab, in the plane across ab towards c, the normal), the
// length of ab, unit directions and lengths of ac and bc in the plane, and the
// part of TriPoint's error that does not depend on the point.
// Near-degenerate triangles get a negative length of ab: left out.
__device__ __forceinline__ void tri_frame(const RefTreeView& b, const Scene32& sc, float frame_m, int s,
                                          float4* __restrict__ out)
{
    const d3 v[3] = {tri_vertex(b, s, 0), tri_vertex(b, s, 1), tri_vertex(b, s, 2)};
    float4* o = out + 5 * (int64_t)s;
    if (b.tbox[2 * (int64_t)s].x == -INFINITY)
    {
        for (int k = 0; k < 5; ++k) o[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        o[3].x = -1.f;
        return;
    }
    auto unit = [](const d3& x, double& l) {
        l = sqrt(dot(x, x));
        return mk(x.x / l, x.y / l, x.z / l);
    };
    double lab, lac, lbc, ln;
    const d3 ac = sub(v[2], v[0]), bc = sub(v[2], v[1]);
    const d3 x = unit(sub(v[1], v[0]), lab);
    const d3 z = unit(cross(sub(v[1], v[0]), ac), ln);
    const d3 y = cross(z, x);
    const d3 uac = unit(ac, lac), ubc = unit(bc, lbc);
    o[0] = make_float4((float)(v[0].x - sc.o[0]), (float)(v[0].y - sc.o[1]), (float)(v[0].z - sc.o[2]), (float)x.x);
    o[1] = make_float4((float)x.y, (float)x.z, (float)y.x, (float)y.y);
    o[2] = make_float4((float)y.z, (float)z.x, (float)z.y, (float)z.z);
    o[3] = make_float4((float)lab, (float)dot(uac, x), (float)dot(uac, y), (float)lac);
    o[4] = make_float4((float)dot(ubc, x), (float)dot(ubc, y), (float)lbc,
                       __fmaf_ru(__double2float_ru(lab), 0x1p-20f, frame_m));
}

// ---------------------------------------------------------------------------
// ray bins
// ---------------------------------------------------------------------------
// The triangle on the plane, counter-clockwise: corners, reciprocal heights of
// its edges (0: flatter than `grow`) and its box grown by `grow`.
struct PlaneTri
{
    double x[3], y[3], inv[3], x0, x1, y0, y1, grow;
    __device__ PlaneTri(const double q[6], double g) : grow(g)
    {
        const bool turn = (q[2] - q[0]) * (q[5] - q[1]) - (q[3] - q[1]) * (q[4] - q[0]) < 0.0;
        x[0] = q[0];
        y[0] = q[1];
        x[1] = q[turn ? 4 : 2];
        y[1] = q[turn ? 5 : 3];
        x[2] = q[turn ? 2 : 4];
        y[2] = q[turn ? 3 : 5];
        x0 = fmin(x[0], fmin(x[1], x[2])) - g;
        x1 = fmax(x[0], fmax(x[1], x[2])) + g;
        y0 = fmin(y[0], fmin(y[1], y[2])) - g;
        y1 = fmax(y[0], fmax(y[1], y[2])) + g;
#pragma unroll
        for (int k = 0; k < 3; ++k)
        {
            const double d = y[k == 2 ? 0 : k + 1] - y[k];
            inv[k] = fabs(d) > g ? 1.0 / d : 0.0;
        }
    }
    // The x range of the grown triangle between the heights lo and hi: its
    // edges clipped to the strip grown by `grow`, grown in x (by far more than
    // the products are rounded).
    __device__ void strip(double lo, double hi, double& xl, double& xh) const
    {
        xl = DBL_MAX;
        xh = -DBL_MAX;
#pragma unroll
        for (int k = 0; k < 3; ++k)
        {
            const int e = k == 2 ? 0 : k + 1;
            const double a = y[k];
            if (fmax(a, y[e]) < lo - grow || fmin(a, y[e]) > hi + grow) continue;
            double t0 = 0.0, t1 = 1.0;
            if (inv[k] != 0.0)
            {
                t0 = fmin(fmax((lo - grow - a) * inv[k], 0.0), 1.0);
                t1 = fmin(fmax((hi + grow - a) * inv[k], 0.0), 1.0);
            }
            const double u = x[k] + t0 * (x[e] - x[k]), v = x[k] + t1 * (x[e] - x[k]);
            xl = fmin(xl, fmin(u, v));
            xh = fmax(xh, fmax(u, v));
        }
        xl -= grow;
        xh += grow;
    }
};

// The cells of a triangle's grown box on one level.
struct CellBox
{
    int x0, x1, y0, y1;
    __device__ CellBox(const RayBins& r, const PlaneTri& p, int level)
    {
        const double top = (double)r.g - 1.0;
        auto cell = [&](double v) { return (int)fmin(fmax(v * r.inv_cell, 0.0), top) >> level; };
        x0 = cell(p.x0);
        x1 = cell(p.x1);
        y0 = cell(p.y0);
        y1 = cell(p.y1);
    }
    __device__ int64_t count() const { return (int64_t)(x1 - x0 + 1) * (y1 - y0 + 1); }
};

// Calls f(cell) for the cells that the triangle may reach on one level, at
// most kMaxCellsPerTri of them, and returns their number (more: some left out).
template <class F>
__device__ __forceinline__ int for_cells(const RayBins& r, const PlaneTri& p, int level, F&& f)
{
    const CellBox b(r, p, level);
    const bool all = b.count() <= kMaxCellsPerTri;
    const double w = ldexp(1.0 / r.inv_cell, level), inv_w = ldexp(r.inv_cell, -level);
    int n = 0;
    for (int iy = b.y0; iy <= b.y1; ++iy)
    {
        int x0 = b.x0, x1 = b.x1;
        if (!all)
        {
            double xl, xh;
            p.strip(iy * w, (iy + 1) * w, xl, xh);
            if (!(xl <= xh)) continue;
            x0 = max(x0, (int)fmax(floor(xl * inv_w), 0.0));
            x1 = min(x1, (int)fmax(floor(xh * inv_w), 0.0));
        }
        for (int ix = x0; ix <= x1; ++ix)
        {
            if (++n > kMaxCellsPerTri) return n;
            f(iy * (r.g >> level) + ix);
        }
    }
    return n;
}

// The level of a triangle: the finest where its box covers at most
// kMaxCellsPerTri cells, or up to two levels finer for a thin triangle (less
// than 1/8 of its box) that reaches at most that many cells there.  Fans and
// long strips would otherwise crowd the cells of the coarse levels.
__device__ __forceinline__ int cell_level(const RayBins& r, const PlaneTri& p)
{
    int level = 0;
    while (CellBox(r, p, level).count() > kMaxCellsPerTri) ++level;
    const double area = (p.x[1] - p.x[0]) * (p.y[2] - p.y[0]) - (p.y[1] - p.y[0]) * (p.x[2] - p.x[0]);
    if (area < 0.25 * (p.x1 - p.x0) * (p.y1 - p.y0)) // area: twice the triangle's
        for (int l = max(level - 2, 0); l < level; ++l)
            if (for_cells(r, p, l, [](int) {}) <= kMaxCellsPerTri) return l;
    return level;
}

__device__ __forceinline__ int level_base(int g, int level)
{
    int base = 0;
    for (int l = 0; l < level; ++l) base += (g >> l) * (g >> l);
    return base;
}

// Triangle `s` on the plane.  Returns false when the reference's test can
// never count it (|det| below its eps).  `grow` bounds how far outside the
// triangle the FP64 test's rounding may still accept a point: with
// u, v >= -eps - err / |det|, err < 2^-48 E |e| (the test takes differences of
// points, whose rounding is relative to them), the accepted points lie within
// 3 (1e-12 + err / |det|) (|e1| + |e2|) of the triangle; `len` is the last factor.
__device__ bool project_triangle(const RefTreeView& b, const RayBins& r, const Scene32& sc, int s, double q[6],
                                 double depth[3], double& len, double& grow)
{
    const d3 dir = mk(b.dir[0], b.dir[1], b.dir[2]);
    d3 v[3];
    for (int k = 0; k < 3; ++k) v[k] = tri_vertex(b, s, k);
    const d3 e1 = sub(v[1], v[0]), e2 = sub(v[2], v[0]);
    const double det = dot(e1, cross(dir, e2)); // ray_hits' own det: it does not depend on the origin
    if (fabs(det) < 1.0e-12) return false;
    for (int k = 0; k < 3; ++k)
    {
        q[2 * k] = dot(v[k], mk(r.e1[0], r.e1[1], r.e1[2])) - r.o1;
        q[2 * k + 1] = dot(v[k], mk(r.e2[0], r.e2[1], r.e2[2])) - r.o2;
        depth[k] = dot(v[k], dir) - r.o3;
    }
    len = sqrt(dot(e1, e1)) + sqrt(dot(e2, e2));
    grow = 3.0 * (1.0e-12 + 0x1p-48 * sc.e * len / fabs(det)) * len + 0x1p-20 * r.size + 0x1p-44 * sc.far;
    return true;
}

// What there is per triangle (one thread each): its frame, its place in the list
// if it is near-degenerate (k_tri_boxes gives it an unbounded box: its computed
// distance may be anything, so FP32 bounds nothing; it stays out of the search,
// and every voxel takes the FP64 test of each), and for the rays its record, its
// level (-1: none) and the counts of its cells.
__global__ void k_tri_tables(RefTreeView b, RayBins r, Scene32 sc, float frame_m, float4* __restrict__ tri4,
                             int* __restrict__ unbounded, float4* __restrict__ rec, signed char* __restrict__ levels,
                             int* __restrict__ counts, int* __restrict__ state)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= b.n) return;
    tri_frame(b, sc, frame_m, s, tri4);
    if (b.tbox[2 * (int64_t)s].x == -INFINITY)
    {
        const int k = atomicAdd(state + kStateUnbounded, 1);
        if (k < kMaxUnbounded) unbounded[k] = s;
    }
    levels[s] = -1;
    double q[6], depth[3], len, grow;
    if (!project_triangle(b, r, sc, s, q, depth, len, grow)) return;
    // the plane has a margin of 2^-10 of its side about the mesh's box
    if (!(grow < 0x1p-11 * r.size))
    {
        atomicAdd(state + kStateWild, 1);
        return;
    }
    const PlaneTri p(q, grow);
    const int level = cell_level(r, p);
    // edge functions in FP32: coordinates are rounded by at most 2^-25 size,
    // differences are bounded by L for every origin in the triangle's cells,
    // and the rounding of the products sums to less than 40 2^-24 L size; the FP64
    // test accepts edge functions down to -(1e-12 |det| + err)
    const double L = (p.x1 - p.x0) + (p.y1 - p.y0) + 2.0 * ldexp(1.0 / r.inv_cell, level);
    const double tol = L * (r.size * 0x1p-17 + sc.far * 0x1p-44) + 0x1p-46 * sc.e * len;
    const double deep = fmax(depth[0], fmax(depth[1], depth[2])) + grow + 0x1p-18 * sc.e;
    rec[2 * (int64_t)s] = make_float4((float)p.x[0], (float)p.y[0], (float)p.x[1], (float)p.y[1]);
    rec[2 * (int64_t)s + 1] =
        make_float4((float)p.x[2], (float)p.y[2], __double2float_ru(deep), __double2float_ru(tol));
    levels[s] = (signed char)level;
    atomicOr(state + kStateLevels, 1 << level);
    const int base = level_base(r.g, level);
    const int reached = for_cells(r, p, level, [&](int c) { atomicAdd(counts + base + c, 1); });
    const unsigned lanes = __activemask();
    const unsigned area = __reduce_add_sync(lanes, (unsigned)reached << (2 * level));
    if ((int)(threadIdx.x & 31) == __ffs(lanes) - 1)
        atomicAdd(reinterpret_cast<unsigned long long*>(state + kStateCrowd), (unsigned long long)area);
}

// The lists' entries; counts go back to 0.
__global__ void k_ray_emit(RefTreeView b, RayBins r, Scene32 sc, const signed char* __restrict__ levels,
                           const int* __restrict__ off, int* __restrict__ counts, int* __restrict__ ids)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= b.n || levels[s] < 0) return;
    double q[6], depth[3], len, grow;
    project_triangle(b, r, sc, s, q, depth, len, grow);
    const int level = levels[s], base = level_base(r.g, level);
    for_cells(r, PlaneTri(q, grow), level,
              [&](int c) { ids[off[base + c] + atomicAdd(counts + base + c, -1) - 1] = s; });
}

// countRayIntersections by bins.  The reference tests a triangle when the
// ray crosses the boxes of its leaf and of all nodes above (rayIntersectsAabb
// in FP64).  Those boxes contain the triangle's own box, and the slab
// arithmetic is monotone in the box's sides, so a triangle whose own box
// passes is reached.  A hit whose own box does not pass clears *ok.
__device__ __forceinline__ int binned_ray_count(const WarpTreeView& t, const d3& p, bool* ok)
{
    const RayBins& r = t.rays;
    const d3 dir = mk(t.ref.dir[0], t.ref.dir[1], t.ref.dir[2]);
    const double q1 = dot(p, mk(r.e1[0], r.e1[1], r.e1[2])) - r.o1;
    const double q2 = dot(p, mk(r.e2[0], r.e2[1], r.e2[2])) - r.o2;
    if (!(q1 >= 0.0 && q1 < r.size && q2 >= 0.0 && q2 < r.size)) return 0;
    const float qx = (float)q1, qy = (float)q2, depth = (float)(dot(p, dir) - r.o3);
    const int cx = min((int)(q1 * r.inv_cell), r.g - 1), cy = min((int)(q2 * r.inv_cell), r.g - 1);
    int hits = 0, base = 0, gl = r.g;
    for (int levels = t.state[kStateLevels], l = 0; levels != 0; levels >>= 1, ++l)
    {
        if (levels & 1)
        {
            const int c = base + (cy >> l) * gl + (cx >> l);
            const int e = __ldg(r.off + c + 1);
            int k = __ldg(r.off + c);
            if (k < e)
            {
                // the next entry's record is on its way while one is tested
                int s = __ldg(r.ids + k), s1 = __ldg(r.ids + min(k + 1, e - 1));
                float4 m = __ldg(r.rec + 2 * (int64_t)s), n = __ldg(r.rec + 2 * (int64_t)s + 1);
                for (; k < e; ++k)
                {
                    const float4 m1 = __ldg(r.rec + 2 * (int64_t)s1), n1 = __ldg(r.rec + 2 * (int64_t)s1 + 1);
                    const int s2 = __ldg(r.ids + min(k + 2, e - 1));
                    const float c0 = (m.z - m.x) * (qy - m.y) - (m.w - m.y) * (qx - m.x);
                    const float c1 = (n.x - m.z) * (qy - m.w) - (n.y - m.w) * (qx - m.z);
                    const float c2 = (m.x - n.x) * (qy - n.y) - (m.y - n.y) * (qx - n.x);
                    // not behind the origin, and not outside an edge
                    if (!(depth > n.z) && !(fminf(c0, fminf(c1, c2)) < -n.w))
                    {
                        const d3 a = tri_vertex(t.ref, s, 0), b = tri_vertex(t.ref, s, 1), d = tri_vertex(t.ref, s, 2);
                        if (ray_hits(p, dir, a, b, d))
                        {
                            const double lo[3] = {fmin(a.x, fmin(b.x, d.x)), fmin(a.y, fmin(b.y, d.y)),
                                                  fmin(a.z, fmin(b.z, d.z))};
                            const double hi[3] = {fmax(a.x, fmax(b.x, d.x)), fmax(a.y, fmax(b.y, d.y)),
                                                  fmax(a.z, fmax(b.z, d.z))};
                            if (!ray_box_ref(p, t.ref.dir, lo, hi)) *ok = false;
                            ++hits;
                        }
                    }
                    s = s1;
                    s1 = s2;
                    m = m1;
                    n = n1;
                }
            }
        }
        base += gl * gl;
        gl >>= 1;
    }
    return hits;
}

// ---------------------------------------------------------------------------
// nearest triangle
// ---------------------------------------------------------------------------
// A lane's result for one point p.  sq: the smallest computed squared
// distance met so far; slot: of the triangles that attain it, the one the
// reference's search visits first; unsure: that cannot be told.
struct LaneNearest
{
    double sq;
    int slot;
    bool unsure;
};

// The reference's box distance to the triangle's own box is no more than sq.
__device__ __forceinline__ bool own_box_within(const d3& p, const d3& a, const d3& b, const d3& c, double sq)
{
    const double lo[3] = {fmin(a.x, fmin(b.x, c.x)), fmin(a.y, fmin(b.y, c.y)), fmin(a.z, fmin(b.z, c.z))};
    const double hi[3] = {fmax(a.x, fmax(b.x, c.x)), fmax(a.y, fmax(b.y, c.y)), fmax(a.z, fmax(b.z, c.z))};
    return box_dist_sq(p, lo, hi) <= sq;
}

// Of the slots list[0], list[32], .. list[32 (n - 1)] and `other` (< 0: none),
// the one that the reference's search (near child first, right only when
// strictly nearer) visits first at p: one descent, into the child visited
// first of those that hold any.
__device__ __forceinline__ int first_visited(const RefTreeView& t, const d3& p, const int* list, int n, int other)
{
    int node = 0, lo = 0, hi = t.n;
    for (;;)
    {
        const int4 meta = __ldg(reinterpret_cast<const int4*>(t.nodes + node) + 3);
        const int mid = meta.w > 0 ? hi : lo + (hi - lo) / 2; // a leaf: its slots in order
        int left = 0, right = 0, least = 0x7fffffff;
        for (int k = -1; k < n; ++k)
        {
            const int s = k < 0 ? other : list[32 * k];
            if (s < lo || s >= hi) continue;
            least = min(least, s);
            if (s < mid)
                ++left;
            else
                ++right;
        }
        if (left + right <= 1 || meta.w > 0) return least;
        bool go_left = left > 0;
        if (left > 0 && right > 0)
        {
            double llo[3], lhi[3], rlo[3], rhi[3];
            load_box(t.nodes + meta.x, llo, lhi);
            load_box(t.nodes + meta.y, rlo, rhi);
            go_left = !(box_dist_sq(p, rlo, rhi) < box_dist_sq(p, llo, lhi));
        }
        if (go_left)
        {
            node = meta.x;
            hi = mid;
        }
        else
        {
            node = meta.y;
            lo = mid;
        }
    }
}

// The FP64 tests of the listed triangles (entry k at list[32 k], its lower
// bound at low[32 k]) that can still matter; the list's space is used up.
//
// r.sq becomes the smallest computed squared distance so far, at the end over
// all triangles (the FP32 tests skip none that could reach it), so the
// reference's running best never falls below it.  The reference enters a node
// unless the node's box distance exceeds its best.  A node's box contains the
// own box of every triangle below it and the box distance is monotone in the
// box's sides, so a triangle whose own box distance is at most its computed
// squared distance is reached; of those that attain the smallest the reference
// keeps the first it reaches (strict update), which is the first in its
// visiting order.
__device__ __forceinline__ void flush_list(const WarpTreeView& t, const d3& p, int* list, const float* low, int n,
                                           float bound, LaneNearest& r)
{
    int ties = 0; // triangles at the front of the list that attain r.sq
    for (int k = 0; k < n; ++k)
    {
        if (low[32 * k] > bound) continue;
        const int s = list[32 * k];
        const d3 a = tri_vertex(t.ref, s, 0), b = tri_vertex(t.ref, s, 1), c = tri_vertex(t.ref, s, 2);
        const d3 d = sub(p, closest_point(p, a, b, c));
        const double sq = dot(d, d);
        if (sq < r.sq)
        {
            r.sq = sq;
            r.slot = -1;
            r.unsure = false;
            ties = 0;
        }
        if (sq == r.sq)
        {
            r.unsure = r.unsure || !own_box_within(p, a, b, c, sq);
            list[32 * ties++] = s;
        }
    }
    if (ties == 0) return;
    r.slot = ties == 1 && r.slot < 0 ? list[0] : first_visited(t.ref, p, list, ties, r.slot);
}

// The near-degenerate triangles after all others; the list's space is used up.
__device__ __forceinline__ void flush_unbounded(const WarpTreeView& t, const d3& p, int* list, float* low, LaneNearest& r)
{
    const int count = t.state[kStateUnbounded];
    for (int base = 0; base < count; base += kLaneList)
    {
        const int n = min(kLaneList, count - base);
        for (int k = 0; k < n; ++k)
        {
            list[32 * k] = __ldg(t.unbounded + base + k);
            low[32 * k] = 0.f;
        }
        flush_list(t, p, list, low, n, 0.f, r);
    }
}

// Lower bound of the squared distance to a box widened by the margin.
__device__ __forceinline__ float gap2(const float p[3], float lx, float ly, float lz, float hx, float hy, float hz)
{
    const float x = fmaxf(fmaxf(lx - p[0], p[0] - hx), 0.f);
    const float y = fmaxf(fmaxf(ly - p[1], p[1] - hy), 0.f);
    const float z = fmaxf(fmaxf(lz - p[2], p[2] - hz), 0.f);
    return __fmaf_rn(x, x, __fmaf_rn(y, y, z * z));
}

// Triangle s in FP32.  In the triangle's frame the squared distance is z^2
// plus the planar one.  Errors, in units of 2^-24: p and a are rounded to E per
// axis (and to 2^-52 far beforehand); their difference, the rotation, the
// segments of ab and ac and the root add less than 17 r, r = |x| + |y| + |z|; the
// segment of bc, 8 |ab|.  So the distance to the plane, to an edge's line or to a
// segment is known to within m = 2^-20 (E + r + |ab|) + 2^-50 far.
struct TriFrame
{
    float4 q0, q1, q2, q3, q4;
    __device__ __forceinline__ explicit TriFrame(const float4* q) : q0(q[0]), q1(q[1]), q2(q[2]), q3(q[3]), q4(q[4]) {}
    __device__ __forceinline__ bool left_out() const { return q3.x < 0.f; } // near-degenerate
};

// One point against one triangle: first the cheap lower bound by the
// triangle's plane and the lines of its edges (need()), then the distance.
struct TriPoint
{
    float x, y, z, m, eac, ebc, side;
    __device__ __forceinline__ TriPoint(const TriFrame& f, const float p[3])
    {
        const float dx = p[0] - f.q0.x, dy = p[1] - f.q0.y, dz = p[2] - f.q0.z;
        x = __fmaf_rn(f.q0.w, dx, __fmaf_rn(f.q1.x, dy, f.q1.y * dz));
        y = __fmaf_rn(f.q1.z, dx, __fmaf_rn(f.q1.w, dy, f.q2.x * dz));
        z = __fmaf_rn(f.q2.y, dx, __fmaf_rn(f.q2.z, dy, f.q2.w * dz));
        m = __fmaf_rn(fabsf(x) + fabsf(y) + fabsf(z), 0x1p-20f, f.q4.w);
        // signed distances outward of the edges ab, ac, bc
        eac = __fmaf_rn(f.q3.y, y, -(f.q3.z * x));
        ebc = __fmaf_rn(f.q4.y, x - f.q3.x, -(f.q4.x * y));
        side = fmaxf(-y, fmaxf(eac, ebc));
    }
    __device__ __forceinline__ bool need(const TriFrame& f, float bound) const
    {
        const float lz = fmaxf(fabsf(z) - m, 0.f), lo = fmaxf(side - m, 0.f);
        return !f.left_out() && !(__fmaf_rn(lz, lz, lo * lo) > bound);
    }
    // Bounds of the squared distance; false: the triangle cannot matter.
    // Otherwise `bound` is lowered to what this triangle attains: the distance
    // to its plane only where the point is inside its edges by more than their
    // error, else that to the nearest segment.  (At a needle's tip the edges'
    // signs are lost in rounding well outside the triangle.)
    __device__ __forceinline__ bool reaches(const WarpTreeView& t, const TriFrame& f, float& bound, float& low) const
    {
        // planar distance: 0 inside, else to the nearest of the three segments
        const float xb = x - f.q3.x;
        const float sab = x - fminf(fmaxf(x, 0.f), f.q3.x);
        const float tac = __fmaf_rn(f.q3.y, x, f.q3.z * y), sac = tac - fminf(fmaxf(tac, 0.f), f.q3.w);
        const float tbc = __fmaf_rn(f.q4.x, xb, f.q4.y * y), sbc = tbc - fminf(fmaxf(tbc, 0.f), f.q4.z);
        const float d2 = fminf(__fmaf_rn(sab, sab, y * y), fminf(__fmaf_rn(sac, sac, eac * eac),
                                                                __fmaf_rn(sbc, sbc, ebc * ebc)));
        const float d = sqrtf(__fmaf_rn(z, z, side > 0.f ? d2 : 0.f));
        low = fmaxf(d - m, 0.f);
        low *= low;
        if (f.left_out() || low > bound) return false;
        const float up = (side > 0.f || side < -m ? d : sqrtf(__fmaf_rn(z, z, d2))) + m;
        bound = fminf(bound, __fmaf_ru(__fmul_ru(up, up), 1.f + 0x1p-15f, t.bound_abs));
        return true;
    }
};

// Lists of a lane: entry k at list[32 k], low[32 k].  Drops the entries whose
// lower bound is above `bound`; returns how many are left.
__device__ __forceinline__ int compact_list(int* list, float* low, int n, float bound)
{
    int m = 0;
    for (int k = 0; k < n; ++k)
    {
        const float l = low[32 * k];
        const int s = list[32 * k];
        if (l > bound) continue;
        low[32 * m] = l;
        list[32 * m] = s;
        ++m;
    }
    return m;
}

// The FP32 search of a warp over two points per lane (every lane calls it;
// bound[k] < 0: nothing to find for point k).  One set of loads, votes and
// branches serves both points, which is most of what a node or a triangle
// costs.  Leaves in each lane's lists the triangles that may be nearest.
// PART false: returns false when the patches are to be handed over (too many
// leaves, or a list that stays full); the bounds then hold for a new search.
// PART true: the subtree `node` only, without a limit; empty(k) empties the
// list of point k.
template <bool PART, class Empty>
__device__ __forceinline__ bool warp_search(const WarpTreeView& t, int node, int* stack, float4* tris, const float pf[2][3],
                                            float bound[2], int n[2], int* list, float* low, int* status,
                                            Empty&& empty)
{
    const RefTreeView& b = t.ref;
    const int lane = (int)(threadIdx.x & 31);
    constexpr int kNext = kLaneList * 32; // the second point's list
    int sp = 0, leaves = 0;
    bool full = false;
    for (;;)
    {
        if (node >= 0)
        {
            const float4* nd = t.node4 + 4 * (int64_t)node;
            const float4 n0 = __ldg(nd), n1 = __ldg(nd + 1), n2 = __ldg(nd + 2), n3 = __ldg(nd + 3);
            const float dl = gap2(pf[0], n0.x, n0.y, n0.z, n0.w, n1.x, n1.y);
            const float dr = gap2(pf[0], n1.z, n1.w, n2.x, n2.y, n2.z, n2.w);
            const float el = gap2(pf[1], n0.x, n0.y, n0.z, n0.w, n1.x, n1.y);
            const float er = gap2(pf[1], n1.z, n1.w, n2.x, n2.y, n2.z, n2.w);
            const bool ml = __any_sync(0xffffffffu, !(dl > bound[0]) || !(el > bound[1]));
            const bool mr = __any_sync(0xffffffffu, !(dr > bound[0]) || !(er > bound[1]));
            const int cl = __float_as_int(n3.x), cr = __float_as_int(n3.y);
            if (ml && mr)
            {
                // most lanes' nearer child first
                const bool left = __popc(__ballot_sync(0xffffffffu, dl + el <= dr + er)) >= 16;
                if (sp < kWarpStack)
                {
                    if (lane == 0) stack[sp] = left ? cr : cl;
                    ++sp;
                }
                else if (lane == 0)
                    atomicOr(status, kStatusStackOverflow);
                node = left ? cl : cr;
                continue;
            }
            if (ml || mr)
            {
                node = ml ? cl : cr;
                continue;
            }
        }
        else
        {
            if (!PART && (leaves == t.max_leaves || __any_sync(0xffffffffu, full))) return false;
            ++leaves;
            const int4 meta = __ldg(reinterpret_cast<const int4*>(b.nodes + ~node) + 3);
            // the leaf's records (at most 8) in one go: one latency instead of
            // one per triangle
            const float4* src = t.tri4 + 5 * (int64_t)meta.z;
            if (lane < 5 * meta.w) tris[lane] = __ldg(src + lane);
            if (lane + 32 < 5 * meta.w) tris[lane + 32] = __ldg(src + lane + 32);
            __syncwarp();
            for (int s = meta.z; s < meta.z + meta.w; ++s)
            {
                const TriFrame f(tris + 5 * (s - meta.z));
                const TriPoint u(f, pf[0]), v(f, pf[1]);
                if (!__any_sync(0xffffffffu, u.need(f, bound[0]) || v.need(f, bound[1]))) continue;
#pragma unroll
                for (int k = 0; k < 2; ++k)
                {
                    float l;
                    if (!(k ? v : u).reaches(t, f, bound[k], l)) continue;
                    if (n[k] == kLaneList) n[k] = compact_list(list + k * kNext, low + k * kNext, n[k], bound[k]);
                    if (n[k] == kLaneList)
                    {
                        if constexpr (PART)
                            empty(k);
                        else
                        {
                            full = true;
                            continue;
                        }
                    }
                    list[k * kNext + 32 * n[k]] = s;
                    low[k * kNext + 32 * n[k]] = l;
                    ++n[k];
                }
            }
        }
        if (sp == 0) break;
        __syncwarp();
        --sp;
        node = stack[sp];
        __syncwarp();
    }
    return PART || !__any_sync(0xffffffffu, full);
}

// The subtree numbered `part` of 2^kPartDepth: the path from the root by the
// part's bits.  Returns its code (a node, ~id of a leaf) in *code; false: none
// (a leaf met on the way belongs to the part whose further bits are 0).
__device__ __forceinline__ bool part_root(const RefTreeView& b, int part, int* code)
{
    int node = 0;
    for (int d = 0;; ++d)
    {
        const int4 meta = __ldg(reinterpret_cast<const int4*>(b.nodes + node) + 3);
        if (meta.w > 0)
        {
            *code = ~node;
            return (part >> d) == 0;
        }
        if (d == kPartDepth) break;
        node = ((part >> d) & 1) ? meta.y : meta.x;
    }
    *code = node;
    return true;
}

// The signed result from the winning triangle and the ray's hits, as
// signed_nearest.
__device__ __forceinline__ void finish_signed(const WarpTreeView& t, const d3& p, const LaneNearest& w, int hits,
                                              SignedResult& r)
{
    const int slot = w.slot;
    const d3 a = tri_vertex(t.ref, slot, 0), b = tri_vertex(t.ref, slot, 1), c = tri_vertex(t.ref, slot, 2);
    int region;
    r.cp = closest_point(p, a, b, c, &region);
    r.fn = face_normal(a, b, c);
    const double dist = sqrt(w.sq);
    if (t.ref.pn)
    {
        d3 n = r.fn;
        if (region < kRegionFace)
        {
            const double* q = t.ref.pn + 18 * (int64_t)slot + 3 * region;
            n = mk(__ldg(q), __ldg(q + 1), __ldg(q + 2));
        }
        r.sd = dot(sub(p, r.cp), n) >= 0.0 ? dist : -dist;
        return;
    }
    if (hits > 0)
        r.sd = (hits % 2) == 1 ? -dist : dist;
    else
        r.sd = dot(sub(p, r.cp), r.fn) >= 0.0 ? dist : -dist;
}

constexpr int kFillThreads = 128;
// Resident CTAs per SM asked of the register allocator for the warp fills.
#ifndef SDFO_WARP_FILL_MIN_BLOCKS
#define SDFO_WARP_FILL_MIN_BLOCKS 6
#endif

// What a fill runs over: patches of 32 voxels, lane by lane.  A voxel left
// over has phi NaN in the query payload until it is filled.
//
// Dense: CTAs of one FillTile each, its warps compact patches of it (4 x 4 x 2
// voxels in the default 8 x 8 x 4 tile).
struct DenseJob
{
    WarpTreeView t;
    SpecD s;
    FillTile tile;
    int wx, wy, wz; // log2 extents of a warp's patch
    int gx, gy;     // tiles in x and y
    double* phi64;
    double* n64;
    double* w64;
    float4* phin;

    void shape(const FillTile& f)
    {
        tile = f;
        const dim3 g = f.grid(s);
        gx = (int)g.x;
        gy = (int)g.y;
        const int lz = 8 - f.lx - f.ly;
        wx = f.lx < 2 ? f.lx : 2;
        wy = f.ly < 2 ? f.ly : 2;
        wz = lz < 5 - wx - wy ? lz : 5 - wx - wy;
        while (wx + wy + wz < 5)
            if (wx < f.lx)
                ++wx;
            else
                ++wy;
    }
    int64_t patches() const { return 8 * (int64_t)gx * gy * tile.grid(s).z; }

    // Voxel `lane` of a patch; false: outside the grid.
    __device__ __forceinline__ bool voxel(int64_t patch, int lane, d3& c, int64_t& idx) const
    {
        const int w = (int)(patch & 7);
        const int64_t b = patch >> 3;
        const int bx = (int)(b % gx), by = (int)((b / gx) % gy), bz = (int)(b / ((int64_t)gx * gy));
        // patches that follow one another in a tile are neighbours in z
        const int nx = tile.lx - wx, nz = 8 - tile.lx - tile.ly - wz;
        const int i = bx * tile.x() + (((w >> nz) & ((1 << nx) - 1)) << wx) + (lane & ((1 << wx) - 1));
        const int j = by * tile.y() + ((w >> (nz + nx)) << wy) + ((lane >> wx) & ((1 << wy) - 1));
        const int k = bz * tile.z() + ((w & ((1 << nz) - 1)) << wz) + (lane >> (wx + wy));
        c = voxel_center(s, i, j, k);
        idx = i + (int64_t)s.n[0] * (j + (int64_t)s.n[1] * k);
        return i < s.n[0] && j < s.n[1] && k < s.n[2];
    }
    __device__ __forceinline__ void store(int64_t idx, const d3& c, const SignedResult& r) const
    {
        const d3 g = voxel_normal(c, r);
        phi64[idx] = r.sd;
        n64[3 * idx + 0] = g.x;
        n64[3 * idx + 1] = g.y;
        n64[3 * idx + 2] = g.z;
        w64[3 * idx + 0] = r.cp.x;
        w64[3 * idx + 1] = r.cp.y;
        w64[3 * idx + 2] = r.cp.z;
        phin[idx] = make_float4((float)r.sd, (float)g.x, (float)g.y, (float)g.z);
    }
    __device__ __forceinline__ void outside(int64_t) const {}
};

// Sparse: bricks of bd^3 voxels, 8^3 bricks in patches of 4 x 4 x 2; voxels
// outside the grid get phi 0, n (1, 0, 0) (SdfBuilder.cpp:925-965).
struct BrickJob
{
    WarpTreeView t;
    SpecD s;
    int bd;
    int bricks;
    const int32_t* ijk;
    float4* phin;

    int per_brick() const { return (bd * bd * bd + 31) / 32; }
    int64_t patches() const { return (int64_t)per_brick() * bricks; }

    __device__ __forceinline__ bool voxel(int64_t patch, int lane, d3& c, int64_t& idx) const
    {
        const int V = bd * bd * bd, per = (V + 31) / 32;
        const int blk = (int)(patch / per), w = (int)(patch % per);
        int local = 32 * w + lane;
        idx = -1;
        if (local >= V) return false;
        if (bd == 8)
        {
            const int x = (lane & 3) | (w & 4), y = ((lane >> 2) & 3) | ((w & 8) >> 1);
            local = x + 8 * (y + 8 * ((lane >> 4) | ((w & 3) << 1)));
        }
        const int i = ijk[3 * blk] * bd + local % bd, j = ijk[3 * blk + 1] * bd + (local / bd) % bd,
                  k = ijk[3 * blk + 2] * bd + local / (bd * bd);
        c = voxel_center(s, i, j, k);
        idx = (int64_t)blk * V + local;
        return i < s.n[0] && j < s.n[1] && k < s.n[2];
    }
    __device__ __forceinline__ void store(int64_t idx, const d3& c, const SignedResult& r) const
    {
        const d3 g = voxel_normal(c, r);
        phin[idx] = make_float4((float)r.sd, (float)g.x, (float)g.y, (float)g.z);
    }
    __device__ __forceinline__ void outside(int64_t idx) const
    {
        if (idx >= 0) phin[idx] = make_float4(0.f, 1.f, 0.f, 0.f);
    }
};

// Two patches per warp.
template <class Job>
__global__ void __launch_bounds__(kFillThreads, SDFO_WARP_FILL_MIN_BLOCKS)
    k_warp_fill(Job job, int64_t patches, int* status)
{
    constexpr int kWarps = kFillThreads / 32;
    __shared__ float4 tris[kWarps][5 * kLeafTris];
    __shared__ int stacks[kWarps][kWarpStack];
    __shared__ int lists[kWarps][2 * kLaneList * 32];
    __shared__ float lows[kWarps][2 * kLaneList * 32];
    const WarpTreeView& t = job.t;
    if (!warp_path_open(t)) return;
    const int warp = (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31);
    const int64_t patch = 2 * ((int64_t)blockIdx.x * kWarps + warp);
    if (patch >= patches) return;
    int* list = lists[warp] + lane;
    float* low = lows[warp] + lane;
    float pf[2][3], bound[2];
    int n[2] = {0, 0};
#pragma unroll
    for (int k = 0; k < 2; ++k)
    {
        d3 c = mk(0.0, 0.0, 0.0);
        int64_t idx = -1;
        const bool active = patch + k < patches && job.voxel(patch + k, lane, c, idx);
        if (!active) job.outside(idx);
        pf[k][0] = (float)(c.x - t.o[0]);
        pf[k][1] = (float)(c.y - t.o[1]);
        pf[k][2] = (float)(c.z - t.o[2]);
        bound[k] = active ? INFINITY : -1.f;
    }
    const bool done = warp_search<false>(t, t.ref.nnodes == 1 ? ~0 : 0, stacks[warp], tris[warp], pf, bound, n, list, low, status,
                                         [](int) {});
    if (!done && lane == 0) t.heavy[atomicAdd(t.state + kStateHeavy, 1)] = (int)patch;
#pragma unroll 1
    for (int k = 0; k < 2; ++k)
    {
        d3 c = mk(0.0, 0.0, 0.0);
        int64_t idx = -1;
        if (patch + k >= patches || !job.voxel(patch + k, lane, c, idx)) continue;
        const float bd = k ? bound[1] : bound[0];
        if (!done)
        {
            job.phin[idx] = make_float4(NAN, bd, 0.f, 0.f);
            continue;
        }
        LaneNearest w{DBL_MAX, -1, false};
        flush_list(t, c, list + k * kLaneList * 32, low + k * kLaneList * 32, k ? n[1] : n[0], bd, w);
        flush_unbounded(t, c, list + k * kLaneList * 32, low + k * kLaneList * 32, w);
        bool ok = w.slot >= 0 && !w.unsure;
        const int hits = ok && !t.ref.pn ? binned_ray_count(t, c, &ok) : 0;
        if (!ok)
        {
            job.phin[idx] = make_float4(NAN, 0.f, 0.f, 0.f);
            atomicAdd(t.state + kStateMarked, 1);
            continue;
        }
        SignedResult r;
        finish_signed(t, c, w, hits, r);
        job.store(idx, c, r);
    }
}

// The pairs of patches handed over, one per CTA.  Each warp searches parts of
// the tree for all 64 voxels, as they become free, and keeps its own nearest
// triangles; the warps' results are then compared.
template <class Job>
__global__ void __launch_bounds__(32 * kHeavyWarps, kHeavyBlocks) k_heavy_fill(Job job, int64_t patches, int* status)
{
    __shared__ float4 tris[kHeavyWarps][5 * kLeafTris];
    __shared__ int stacks[kHeavyWarps][kWarpStack];
    __shared__ int lists[kHeavyWarps][2 * kLaneList * 32];
    __shared__ float lows[kHeavyWarps][2 * kLaneList * 32];
    __shared__ double s_sq[kHeavyWarps][64];
    __shared__ int s_slot[kHeavyWarps][64]; // ~slot: unsure; kNoSlot: none
    __shared__ unsigned s_bound[64];
    __shared__ int s_next;
    constexpr int kNoSlot = 0x7fffffff;
    const WarpTreeView& t = job.t;
    if (!warp_path_open(t)) return;
    const int warp = (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31);
    int* list = lists[warp] + lane;
    float* low = lows[warp] + lane;
    const int pairs = t.state[kStateHeavy];
    for (int h = blockIdx.x; h < pairs; h += gridDim.x)
    {
        const int64_t patch = t.heavy[h];
        float pf[2][3], bound[2];
        int n[2] = {0, 0};
#pragma unroll
        for (int k = 0; k < 2; ++k)
        {
            d3 c = mk(0.0, 0.0, 0.0);
            int64_t idx = -1;
            const bool active = patch + k < patches && job.voxel(patch + k, lane, c, idx);
            pf[k][0] = (float)(c.x - t.o[0]);
            pf[k][1] = (float)(c.y - t.o[1]);
            pf[k][2] = (float)(c.z - t.o[2]);
            bound[k] = active ? job.phin[idx].y : -1.f;
            s_sq[warp][32 * k + lane] = DBL_MAX;
            s_slot[warp][32 * k + lane] = kNoSlot;
            if (warp == 0) s_bound[32 * k + lane] = __float_as_uint(INFINITY);
        }
        if (threadIdx.x == 0) s_next = 0;
        __syncthreads();
        // the listed triangles of point k into the warp's record
        auto empty = [&](int k) {
            d3 c = mk(0.0, 0.0, 0.0);
            int64_t idx = -1;
            if (patch + k >= patches || !job.voxel(patch + k, lane, c, idx)) return;
            const int kept = s_slot[warp][32 * k + lane];
            LaneNearest w{s_sq[warp][32 * k + lane], kept == kNoSlot ? -1 : kept < 0 ? ~kept : kept, kept < 0};
            flush_list(t, c, list + k * kLaneList * 32, low + k * kLaneList * 32, k ? n[1] : n[0],
                       k ? bound[1] : bound[0], w);
            s_sq[warp][32 * k + lane] = w.sq;
            s_slot[warp][32 * k + lane] = w.slot < 0 ? kNoSlot : w.unsure ? ~w.slot : w.slot;
            if (k)
                n[1] = 0;
            else
                n[0] = 0;
        };
        for (;;)
        {
            int part = 0, root = 0;
            if (lane == 0) part = atomicAdd(&s_next, 1);
            part = __shfl_sync(0xffffffffu, part, 0);
            if (part >= 1 << kPartDepth) break;
            if (!part_root(t.ref, part, &root)) continue;
#pragma unroll
            for (int k = 0; k < 2; ++k) // what the other warps know
                bound[k] = fminf(bound[k], __uint_as_float(*(volatile unsigned*)&s_bound[32 * k + lane]));
            warp_search<true>(t, root, stacks[warp], tris[warp], pf, bound, n, list, low, status, empty);
            __syncwarp();
#pragma unroll
            for (int k = 0; k < 2; ++k) // not negative: ordered as its bits
                if (bound[k] >= 0.f) atomicMin(&s_bound[32 * k + lane], __float_as_uint(bound[k]));
        }
#pragma unroll 1
        for (int k = 0; k < 2; ++k) empty(k);
        __syncthreads();
        if (threadIdx.x < 64)
        {
            const int v = (int)threadIdx.x;
            d3 c = mk(0.0, 0.0, 0.0);
            int64_t idx = -1;
            if (patch + (v >> 5) < patches && job.voxel(patch + (v >> 5), v & 31, c, idx))
            {
                LaneNearest w{DBL_MAX, -1, false};
                for (int q = 0; q < kHeavyWarps; ++q) w.sq = fmin(w.sq, s_sq[q][v]);
                // the slots that attain it, in the first warp's list space
                int ties = 0;
                int* mine = lists[v >> 5] + (v & 31);
                for (int q = 0; q < kHeavyWarps; ++q)
                {
                    const int kept = s_slot[q][v];
                    if (kept == kNoSlot || s_sq[q][v] != w.sq) continue;
                    w.unsure = w.unsure || kept < 0;
                    mine[32 * ties++] = kept < 0 ? ~kept : kept;
                }
                if (ties > 0) w.slot = ties == 1 ? mine[0] : first_visited(t.ref, c, mine, ties, -1);
                flush_unbounded(t, c, mine, lows[v >> 5] + (v & 31), w);
                bool ok = w.slot >= 0 && !w.unsure;
                const int hits = ok && !t.ref.pn ? binned_ray_count(t, c, &ok) : 0;
                if (ok)
                {
                    SignedResult r;
                    finish_signed(t, c, w, hits, r);
                    job.store(idx, c, r);
                }
                else
                {
                    job.phin[idx] = make_float4(NAN, 0.f, 0.f, 0.f);
                    atomicAdd(t.state + kStateMarked, 1);
                }
            }
        }
        __syncthreads();
    }
}

// The voxels left: by the per-thread traversal.
template <class Job>
__global__ void __launch_bounds__(256, SDFO_FILL_MIN_BLOCKS) k_rest_fill(Job job, int64_t patches, int* status)
{
    const WarpTreeView& t = job.t;
    const bool open = warp_path_open(t);
    if (open && t.state[kStateMarked] == 0) return;
    const int64_t patch = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (patch >= patches) return;
    d3 c = mk(0.0, 0.0, 0.0);
    int64_t idx = -1;
    if (!job.voxel(patch, (int)(threadIdx.x & 31), c, idx))
    {
        if (!open) job.outside(idx);
        return;
    }
    if (open && !isnan(job.phin[idx].x)) return;
    job.store(idx, c, signed_nearest(t.ref, c, status));
}

template <class Job>
void launch_warp_fill(const Job& job, int* status, cudaStream_t s)
{
    const int64_t patches = job.patches();
    if (patches <= 0) return;
    const unsigned blocks = (unsigned)((patches + 7) / 8);
    k_warp_fill<<<(unsigned)((patches + 2 * (kFillThreads / 32) - 1) / (2 * (kFillThreads / 32))), kFillThreads, 0, s>>>(
        job, patches, status);
    SDFO_CHECK_LAUNCH();
    k_heavy_fill<<<(unsigned)current_sm_count() * kHeavyBlocks, 32 * kHeavyWarps, 0, s>>>(job, patches, status);
    SDFO_CHECK_LAUNCH();
    k_rest_fill<<<blocks, 256, 0, s>>>(job, patches, status);
    SDFO_CHECK_LAUNCH();
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// Plane of the parity ray over the mesh's box: axes across the direction, the
// square about the projected box with a margin of 2^-10 of its side, and the
// cells: about sqrt(n) per side, so that lists stay around ten triangles.
inline RayBins ray_plane(const double dir[3], const double lo[3], const double hi[3], int64_t n)
{
    RayBins r{};
    // the axis least along dir, made orthogonal to it
    int least = 0;
    for (int a = 1; a < 3; ++a)
        if (std::fabs(dir[a]) < std::fabs(dir[least])) least = a;
    double len = 0.0;
    for (int a = 0; a < 3; ++a)
    {
        r.e1[a] = (a == least ? 1.0 : 0.0) - dir[least] * dir[a];
        len += r.e1[a] * r.e1[a];
    }
    for (int a = 0; a < 3; ++a) r.e1[a] /= std::sqrt(len);
    for (int a = 0; a < 3; ++a)
        r.e2[a] = dir[(a + 1) % 3] * r.e1[(a + 2) % 3] - dir[(a + 2) % 3] * r.e1[(a + 1) % 3];
    double mid[2] = {0.0, 0.0}, half[2] = {0.0, 0.0};
    for (int a = 0; a < 3; ++a)
    {
        const double m = 0.5 * (lo[a] + hi[a]), h = 0.5 * (hi[a] - lo[a]);
        mid[0] += m * r.e1[a];
        mid[1] += m * r.e2[a];
        half[0] += h * std::fabs(r.e1[a]);
        half[1] += h * std::fabs(r.e2[a]);
    }
    double side = 2.0 * std::max(half[0], half[1]);
    if (!(side > 0.0)) side = 1.0;
    r.size = side * (1.0 + 0x1p-9);
    r.o1 = mid[0] - 0.5 * r.size;
    r.o2 = mid[1] - 0.5 * r.size;
    r.g = 1;
    while (r.g < kMaxRayCells && (int64_t)r.g * r.g < n) r.g *= 2;
    r.inv_cell = (double)r.g / r.size;
    r.box_cells = 4.0 * half[0] * half[1] * r.inv_cell * r.inv_cell;
    return r;
}

inline int ray_cells(int g)
{
    int total = 0;
    for (; g > 0; g >>= 1) total += g * g;
    return total;
}

// The fast path's data of one reference-order tree.
struct DeviceWarpTree
{
    DeviceBuffer<unsigned char> mem; // one block: every free waits for the device
    DeviceBuffer<int> heavy;
    WarpTreeView v{};

    // `tree`: uploaded nodes, slot-order triangles and triangle boxes; lo, hi:
    // the mesh's box; far: the largest coordinate of mesh and grid.
    void build(const RefTreeView& tree, const double lo[3], const double hi[3], const sdfo_grid_info& grid, double far,
               cudaStream_t s)
    {
        const int n = tree.n, T = 256;
        Scene32 sc{};
        sc.far = far;
        for (int a = 0; a < 3; ++a)
        {
            const double l = std::min(lo[a], grid.bmin[a]), h = std::max(hi[a], grid.bmax[a]);
            v.o[a] = sc.o[a] = 0.5 * l + 0.5 * h;
            sc.e = std::max(sc.e, 0.5 * h - 0.5 * l);
        }
        const double margin = scene_margin(sc);
        v.ref = tree;
        v.rays = ray_plane(tree.dir, lo, hi, n);
        for (int a = 0; a < 3; ++a) v.rays.o3 += sc.o[a] * tree.dir[a];
        const int cells = ray_cells(v.rays.g);
        size_t temp = 0;
        SDFO_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, temp, (int*)nullptr, (int*)nullptr, cells + 1, s));
        size_t bytes = 0;
        auto part = [&](size_t b) {
            const size_t at = bytes;
            bytes += (b + 255) / 256 * 256;
            return at;
        };
        const size_t p_node4 = part(64 * (size_t)tree.nnodes), p_tri4 = part(80 * (size_t)n), p_rec = part(32 * (size_t)n),
                     p_ids = part(4 * (size_t)n * kMaxCellsPerTri), p_off = part(4 * ((size_t)cells + 1)),
                     p_levels = part((size_t)n), p_unbounded = part(4 * (size_t)kMaxUnbounded), p_scan = part(temp),
                     p_state = part(4 * (size_t)kStateWords), p_counts = part(4 * ((size_t)cells + 1));
        mem.reset(bytes);
        unsigned char* m = mem.get();
        float4 *node4 = (float4*)(m + p_node4), *tri4 = (float4*)(m + p_tri4), *rec = (float4*)(m + p_rec);
        int *ids = (int*)(m + p_ids), *off = (int*)(m + p_off), *unbounded = (int*)(m + p_unbounded),
            *state = (int*)(m + p_state), *counts = (int*)(m + p_counts);
        signed char* levels = (signed char*)(m + p_levels);
        SDFO_CUDA(cudaMemsetAsync(state, 0, bytes - p_state, s)); // state and counts
        k_tri_tables<<<(n + T - 1) / T, T, 0, s>>>(tree, v.rays, sc, (float)(margin * (1.0 + 0x1p-20)), tri4, unbounded,
                                                   rec, levels, counts, state);
        SDFO_CHECK_LAUNCH();
        k_pack_node4<<<(tree.nnodes + T - 1) / T, T, 0, s>>>(tree, sc, margin, node4);
        SDFO_CHECK_LAUNCH();
        SDFO_CUDA(cub::DeviceScan::ExclusiveSum(m + p_scan, temp, counts, off, cells + 1, s));
        k_ray_emit<<<(n + T - 1) / T, T, 0, s>>>(tree, v.rays, sc, levels, off, counts, ids);
        SDFO_CHECK_LAUNCH();
        v.node4 = node4;
        v.tri4 = tri4;
        // what the FP64 closest point of a well-conditioned triangle can be off by
        // beside 2^-16 of its squared distance: (2^-20 E)^2, and for coordinates
        // far from the origin, whose rounding is 2^-52 far, (2^-40 far)^2
        v.bound_abs = (float)((std::ldexp(sc.e * sc.e, -40) + std::ldexp(far * far, -80)) * (1.0 + 0x1p-15));
        v.rays.rec = rec;
        v.rays.off = off;
        v.rays.ids = ids;
        v.state = state;
        v.unbounded = unbounded;
        v.max_crowd = tree.pn ? ULLONG_MAX : (unsigned long long)std::min(kMaxCrowd * v.rays.box_cells, 1e18);
    }

    template <class Job>
    void fill(Job job, int* status, cudaStream_t s)
    {
        const int64_t pairs = (job.patches() + 1) / 2;
        heavy.reset((size_t)pairs);
        v.max_leaves = pairs <= kHeavyBlocks * (int64_t)current_sm_count() ? kFewLeaves : kHeavyLeaves;
        v.heavy = heavy.get();
        job.t = v;
        launch_warp_fill(job, status, s);
    }
};

} // namespace

} // namespace sdfo
