// Fused SDF penalty contact over quadrature points, batched over poses, with
// the forward-mode 6x6 pose Jacobian.
//
// Restates SDFContactEngine.evaluate (prototype/src/dynamics/contacts_sdf.py:
// 225-385).  Without a ContactCull every quadrature point is evaluated; with
// one, the engine's culling is applied as the reference does it: the point
// BVH's leaves overlapping the query box RA^T (bmin - rA) - m ..
// RA^T (bmax - rA) + m (m = max(narrow margin, 0.05); all points when the box
// encloses every point or no leaf overlaps it), then the narrow filter
// |Y_z| < narrow margin.  The same pass can produce measure_pair's
// ContactMeasure (contacts_sdf.py:171-214) over the BVH-kept points.  The
// force law:
//   Y = R_B^T (r_A + R_A X - r_B)                       (marker-free transform)
//   g, grad g = SDF(Y) (Trilinear or Tricubic)           (local, raw gradient)
//   active iff valid and k max(-g,0)^n > 1e-30
//   rg = R_B grad g, p = k max(-g,0)^n, fn = p rg
//   damping (c > 0, g < 0): fd = c (-(u_A - u_B).rg) rg
//   p_hat = p |grad g|, un = rg / |rg|, u_t = u - (u.un) un
//   ft = -mu p_hat u_t / sqrt(|u_t|^2 + reg^2)
//   F_A = sum w (fn + fd + ft), tau_A = sum w (x - r_A) x (fn + fd + ft)
// The Jacobian is d(F_A, tau_A)/d(dx, dtheta) for r_A += dx,
// R_A = exp([dtheta]x) R_A, propagated per point in forward mode through the
// interpolant's Hessian (no finite differences).
//
// Layout: one CTA per pose; the quadrature set (X, w) is shared by all poses
// and stays L1/L2-resident; the grid gather and interpolation are FP32; the
// per-point force law of active points, the Jacobian and the reductions
// (warp shuffles, then shared memory) are FP64.
//
// Most points of most poses are clear of the surface, where the law gives
// exactly nothing.  Dense grids keep one bit per cell that says whether the
// interpolated gap can be <= 0 there (GridView::touch); a first pass places
// every point in FP32 and lists those whose cell has the bit, or whose cell
// FP32 cannot tell (place32.cuh), and only the listed points take the FP64
// transform, the gather and the law, shared out over eight warps.  4096 poses of
// a 7,680-point ring about a block's face, a quarter of them in contact: forces
// and Jacobian 767 -> 308 us (one B200); bound by the latency of the few FP64
// steps of a pose, no longer by the 31 M gathers.
#include <climits>

#include "interp.cuh"
#include "place32.cuh"

namespace sdfo {
namespace {

// Threads per pose: kContactThreads, or kFewThreads when every pose has an SM to
// itself (no more poses than SMs; forces with touch bits, every measure): 33 poses
// of 7,680 points, forces and then the measure, 64 us with 256 threads, 53 with
// 512, of which 50 are the host's.
constexpr int kContactThreads = 256;
constexpr int kFewThreads = 512;
// Points are listed by spans of kJacSpan; then all warps share the span's list.
constexpr int kJacSpan = 4096;
// A pose's sums run in one order whatever the threads per pose, so that its forces
// do not depend on the other poses of the call.  Of a span's chunks of 32 points,
// number c belongs to list c mod 8, in order; with 512 threads warps w and w + 8
// list the first and the second half of list w.  Group k of 32 entries goes to
// force sum k mod kForceRows, one warp's registers, and column or group k of the
// Jacobian to sum k mod kJacRows.
constexpr int kForceRows = kContactThreads / 32;
constexpr int kJacRows = kFewThreads / 32;
// Groups of 32 points in contact up to which the Jacobian's columns are shared out
// over the warps, every column evaluating its points anew.  4,096 poses in light
// contact (about four groups): 0.58 ms with the columns shared out up to here, a
// quarter more up to eight groups; in deep contact, sharing out always took 6.1 ms
// against 5.1.
constexpr int kSplitGroups = 4;
// Points per thread in flight in the pass over the touch bits.
constexpr int kAhead = 4;

struct v3
{
    double x, y, z;
};
__device__ __forceinline__ v3 V(double x, double y, double z) { return {x, y, z}; }
__device__ __forceinline__ v3 operator+(v3 a, v3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ v3 operator-(v3 a, v3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ v3 operator*(double s, v3 a) { return {s * a.x, s * a.y, s * a.z}; }
// Products and sums are fused explicitly: the forward and the Jacobian kernels
// inline the same law, and left to the compiler its contraction differs between
// them in the last bit.
__device__ __forceinline__ double dot(v3 a, v3 b) { return fma(a.x, b.x, fma(a.y, b.y, __dmul_rn(a.z, b.z))); }
__device__ __forceinline__ v3 cross(v3 a, v3 b)
{
    return {fma(a.y, b.z, -__dmul_rn(a.z, b.y)), fma(a.z, b.x, -__dmul_rn(a.x, b.z)),
            fma(a.x, b.y, -__dmul_rn(a.y, b.x))};
}
__device__ __forceinline__ v3 add_scaled(v3 a, double s, v3 b) // a + s b
{
    return {fma(s, b.x, a.x), fma(s, b.y, a.y), fma(s, b.z, a.z)};
}
__device__ __forceinline__ v3 scaled(double s, v3 a)
{
    return {__dmul_rn(s, a.x), __dmul_rn(s, a.y), __dmul_rn(s, a.z)};
}
__device__ __forceinline__ v3 mul(const double R[9], v3 a)
{
    return {dot(V(R[0], R[1], R[2]), a), dot(V(R[3], R[4], R[5]), a), dot(V(R[6], R[7], R[8]), a)};
}
__device__ __forceinline__ v3 mulT(const double R[9], v3 a)
{
    return {dot(V(R[0], R[3], R[6]), a), dot(V(R[1], R[4], R[7]), a), dot(V(R[2], R[5], R[8]), a)};
}

template <int MODE, bool SPARSE, int BD, bool JAC>
__device__ __forceinline__ bool sample(const GridView& g, const double Y[3], float& gap, v3& grad,
                                       double Hl[6])
{
    const Cell c = cell_of(g, Y);
    if (!c.ok) return false;
    const float h[3] = {(float)g.voxel[0], (float)g.voxel[1], (float)g.voxel[2]};
    const float ih[3] = {g.ih[0], g.ih[1], g.ih[2]};
    Interp r;
    if (!SPARSE && MODE == SDFO_TRILINEAR && g.cell8 != nullptr)
    {
        float4 a, b;
        ld256(g.cell8 + 2 * dense_index(g, c.i0, c.j0, c.k0), a, b);
        const float phi[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        r = trilinear<JAC>(phi, c.u, c.v, c.w, ih);
    }
    else
    {
        float4 cs[8];
        if (!SPARSE && g.xpair != nullptr)
        {
            const int64_t base = dense_index(g, c.i0, c.j0, c.k0);
            const int64_t sy = g.nx, sz = (int64_t)g.nx * g.ny;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                ld256(g.xpair + 2 * (base + ((q & 1) ? sy : 0) + ((q & 2) ? sz : 0)), cs[2 * q],
                      cs[2 * q + 1]);
        }
        else
        {
            int64_t idx[8];
            if (!gather_corners<SPARSE, BD>(g, c, cs, idx)) return false;
        }
        if (MODE == SDFO_TRICUBIC)
        {
            r = tricubic<JAC>(cs, c.u, c.v, c.w, h, ih);
        }
        else
        {
            float phi[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) phi[q] = cs[q].x;
            r = trilinear<JAC>(phi, c.u, c.v, c.w, ih);
        }
    }
    gap = r.gap;
    grad = V(r.g[0], r.g[1], r.g[2]);
#pragma unroll
    for (int q = 0; q < 6; ++q) Hl[q] = r.H[q];
    return true;
}

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// Per-point contact state of one quadrature point at one pose.
struct PointState
{
    double p, gn, vn, udn, den, phat, dgdd, wq;
    v3 off, rg, gl, u, un, ut, fq;
    double Hl[6];
    bool damp, fric;
};

// Pose-level quantities shared by all points of a CTA.
struct PoseFrame
{
    v3 rA, rB, vA, wA, vB, wB, tl;
};

// The SDFContactEngine.evaluate force law of quadrature point i
// (contacts_sdf.py:256-385).  Returns 0 when the point is outside the grid,
// 1 when it is inside but exerts no force (k max(-g,0)^n <= 1e-30, or
// dropped by the narrow filter |Y_z| < narrow when narrow >= 0), 2 when it
// is active.  `gap` receives the gap of in-grid points; with need_gap false
// a point failing the narrow filter is not sampled (status 1, gap unset).
// HESS also records the interpolant's Hessian for the Jacobian.
template <int MODE, bool SPARSE, int BD, bool HESS>
__device__ __forceinline__ int point_state(const GridView& g, const float* __restrict__ qx,
                                           const float* __restrict__ qw, int i,
                                           const sdfo_body_state& sA, const sdfo_body_state& sB,
                                           const PoseFrame& f, const sdfo_contact_params& prm,
                                           double narrow, bool need_gap, PointState& st,
                                           double& gap_out)
{
    const v3 X = V(__ldg(qx + 3 * i), __ldg(qx + 3 * i + 1), __ldg(qx + 3 * i + 2));
    st.off = mul(sA.R, X);                   // x_w - r_A
    const v3 Yv = mulT(sB.R, st.off) + f.tl; // body-B local point
    const bool narrow_ok = !(narrow >= 0.0) || fabs(Yv.z) < narrow;
    if (!narrow_ok && !need_gap) return 1;
    const double Y[3] = {Yv.x, Yv.y, Yv.z};
    float gapf;
    if (!sample<MODE, SPARSE, BD, HESS>(g, Y, gapf, st.gl, st.Hl)) return 0;
    const double gap = gapf;
    gap_out = gap;
    if (!narrow_ok) return 1;
    const double delta = gap < 0.0 ? -gap : 0.0;
    const double dpow = prm.order == 2.0 ? delta * delta : prm.order == 1.0 ? delta : pow(delta, prm.order);
    st.p = prm.stiffness * dpow;
    if (!(st.p > 1e-30)) return 1;
    st.wq = (double)__ldg(qw + i);
    const v3 xw = f.rA + st.off;
    st.rg = mul(sB.R, st.gl);
    st.gn = sqrt(dot(st.gl, st.gl));
    st.fq = scaled(st.p, st.rg);
    const v3 uA = f.vA + cross(f.wA, st.off);
    const v3 uB = f.vB + cross(f.wB, xw - f.rB);
    st.u = uA - uB;
    st.damp = prm.damping > 0.0 && gap < 0.0;
    st.vn = dot(st.u, st.rg);
    if (st.damp) st.fq = add_scaled(st.fq, prm.damping * (-st.vn), st.rg);
    const double gsafe = st.gn > 1e-30 ? st.gn : 1e-30;
    st.un = scaled(1.0 / gsafe, st.rg);
    st.udn = dot(st.u, st.un);
    st.ut = add_scaled(st.u, -st.udn, st.un);
    st.den = sqrt(fma(prm.regularizer, prm.regularizer, dot(st.ut, st.ut)));
    st.phat = st.p * st.gn;
    st.fric = prm.friction * st.phat > 0.0;
    if (st.fric) st.fq = add_scaled(st.fq, -prm.friction * st.phat / st.den, st.ut);
    st.dgdd = -prm.stiffness * (prm.order == 2.0 ? 2.0 * delta
                                : prm.order == 1.0 ? 1.0
                                                   : prm.order * pow(delta, prm.order - 1.0));
    return 2;
}

// Entry `q` of M (0..8), of t (9..11), or set_margin's argument (12, in e0), for
// threads 0..12.
__device__ __forceinline__ void set_place_entry(const GridView& g, const sdfo_body_state& sA,
                                                const sdfo_body_state& sB, const v3& tl, int q, Place32& f)
{
    const double t[3] = {tl.x, tl.y, tl.z};
    if (q < 9)
    {
        const int a = q / 3, b = q % 3;
        f.M[q] = (float)((sB.R[a] * sA.R[b] + sB.R[3 + a] * sA.R[3 + b] + sB.R[6 + a] * sA.R[6 + b]) * g.ivoxel[a]);
    }
    else if (q < 12)
    {
        const int a = q - 9;
        f.t[a] = (float)(((a == 0 ? tl.x : a == 1 ? tl.y : tl.z) - g.bmin[a]) * g.ivoxel[a] - 0.5);
    }
    else if (q == 12)
    {
        double far = 0.0;
#pragma unroll
        for (int a = 0; a < 3; ++a) far = fmax(far, (fabs(t[a]) + fabs(g.bmin[a])) * g.ivoxel[a]);
        f.e0 = (float)far;
    }
}

enum : int
{
    kOutside = 0, // certainly outside the grid
    kClear = 1,   // certainly inside, in a cell that the surface does not reach
    kMayTouch = 2 // anything else: the FP64 path decides
};

__device__ __forceinline__ int touch_status(const GridView& g, const uint32_t* __restrict__ bits, const Place32& f,
                                            float x, float y, float z)
{
    int c[3];
    float u[3], e;
    bool out;
    const bool cell = place32(g, f, x, y, z, c, u, e, out);
    const int i = cell ? c[0] + g.nx * (c[1] + g.ny * c[2]) : 0;
    const uint32_t w = __ldg(bits + (i >> 5)); // no branch about it: loads of several points overlap
    return out ? kOutside : cell && !((w >> (i & 31)) & 1u) ? kClear : kMayTouch;
}

// Column j of the point's d(f, x f)/d(dx, dtheta), weighted by w.
__device__ __forceinline__ void jacobian_column(const PointState& st, const sdfo_body_state& sB,
                                                const PoseFrame& f, const sdfo_contact_params& prm,
                                                int j, double col[6])
{
    const double Hm[9] = {st.Hl[0], st.Hl[1], st.Hl[2], st.Hl[1], st.Hl[3],
                          st.Hl[4], st.Hl[2], st.Hl[4], st.Hl[5]};
    v3 dxw, doff;
    if (j < 3)
    {
        dxw = V(j == 0, j == 1, j == 2);
        doff = V(0.0, 0.0, 0.0);
    }
    else
    {
        doff = cross(V(j == 3, j == 4, j == 5), st.off);
        dxw = doff;
    }
    const v3 dYl = mulT(sB.R, dxw);
    const v3 dgl = V(Hm[0] * dYl.x + Hm[1] * dYl.y + Hm[2] * dYl.z,
                     Hm[3] * dYl.x + Hm[4] * dYl.y + Hm[5] * dYl.z,
                     Hm[6] * dYl.x + Hm[7] * dYl.y + Hm[8] * dYl.z);
    const double dg = dot(st.gl, dYl);
    const v3 drg = mul(sB.R, dgl);
    const double dp = st.dgdd * dg; // p = k delta^n, delta = -g
    v3 dfq = dp * st.rg + st.p * drg;
    const v3 du = cross(f.wA, doff) - cross(f.wB, dxw);
    if (st.damp)
    {
        const double dvn = dot(du, st.rg) + dot(st.u, drg);
        dfq = dfq + (-prm.damping) * (dvn * st.rg + st.vn * drg);
    }
    if (st.fric)
    {
        const double gsafe = st.gn > 1e-30 ? st.gn : 1e-30;
        const double dgn = st.gn > 1e-30 ? dot(st.gl, dgl) / st.gn : 0.0;
        const double dphat = dp * st.gn + st.p * dgn;
        const v3 dun = (1.0 / gsafe) * (st.gn > 1e-30 ? drg - dot(st.un, drg) * st.un : drg);
        const double dudn = dot(du, st.un) + dot(st.u, dun);
        const v3 dut = du - dudn * st.un - st.udn * dun;
        const double dden = dot(st.ut, dut) / st.den;
        dfq = dfq + (-prm.friction) * ((dphat / st.den) * st.ut + (st.phat / st.den) * dut -
                                       (st.phat * dden / (st.den * st.den)) * st.ut);
    }
    const v3 dtq = cross(doff, st.fq) + cross(st.off, dfq);
    col[0] = st.wq * dfq.x;
    col[1] = st.wq * dfq.y;
    col[2] = st.wq * dfq.z;
    col[3] = st.wq * dtq.x;
    col[4] = st.wq * dtq.y;
    col[5] = st.wq * dtq.z;
}

// One CTA per pose.  Without touch bits every thread evaluates its points (no
// Hessian) and accumulates F, tau, and with JAC the points in contact (typically
// a small fraction) are listed and evaluated again with the interpolant's
// Hessian for the six Jacobian columns; with touch bits all of that runs on
// the listed points alone.
// Resident CTAs per SM asked of the register allocator (256 threads each).  With
// the Jacobian two, without spills: at three, points in deep contact, evaluated
// for all six columns, ran 0.61 (sparse Tricubic) to 0.90 times as fast.
#ifndef SDFO_CONTACT_MIN_BLOCKS
#define SDFO_CONTACT_MIN_BLOCKS 3
#endif
#ifndef SDFO_CONTACT_JAC_MIN_BLOCKS
#define SDFO_CONTACT_JAC_MIN_BLOCKS 2
#endif

// Lexicographic (gap, key) minimum for measure_pair's argmin: the reference
// takes the first minimum in its point order, `key` is the point's position
// in that order.
struct MinRec
{
    double gap;
    int key;
    int i;
};

__device__ __forceinline__ bool less_rec(const MinRec& a, const MinRec& b)
{
    return a.gap < b.gap || (a.gap == b.gap && a.key < b.key);
}

__device__ __forceinline__ MinRec warp_min(MinRec r)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
    {
        MinRec q;
        q.gap = __shfl_down_sync(0xffffffffu, r.gap, o);
        q.key = __shfl_down_sync(0xffffffffu, r.key, o);
        q.i = __shfl_down_sync(0xffffffffu, r.i, o);
        if (less_rec(q, r)) r = q;
    }
    return r;
}

__device__ __forceinline__ int warp_isum(int v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// The pose's body states into shared memory, 18 doubles each, one per thread.
__device__ __forceinline__ void load_states(const sdfo_body_state* pose, const sdfo_body_state* body_b,
                                            sdfo_body_state& sA, sdfo_body_state& sB)
{
    static_assert(sizeof(sdfo_body_state) == 18 * sizeof(double), "a body state is 18 doubles");
    const int q = (int)threadIdx.x;
    if (q < 18)
        reinterpret_cast<double*>(&sA)[q] = __ldg(reinterpret_cast<const double*>(pose) + q);
    else if (q < 36)
        reinterpret_cast<double*>(&sB)[q - 18] = __ldg(reinterpret_cast<const double*>(body_b) + q - 18);
}

__device__ __forceinline__ PoseFrame pose_frame(const sdfo_body_state& sA, const sdfo_body_state& sB)
{
    PoseFrame f;
    f.rA = V(sA.r[0], sA.r[1], sA.r[2]);
    f.rB = V(sB.r[0], sB.r[1], sB.r[2]);
    f.vA = V(sA.v[0], sA.v[1], sA.v[2]);
    f.wA = V(sA.w[0], sA.w[1], sA.w[2]);
    f.vB = V(sB.v[0], sB.v[1], sB.v[2]);
    f.wB = V(sB.w[0], sB.w[1], sB.w[2]);
    f.tl = mulT(sB.R, f.rA - f.rB); // R_B^T (r_A - r_B)
    return f;
}

// Broad phase: AABB_BVH.query(bmin_local, bmax_local) (bvh.py:62-80).
struct BroadShared
{
    unsigned mask[kMaxCullLeaves / 32]; // leaves kept
    double box[6];
    int full;
};

// True: every point is kept (the mask is not set).  All threads call it.
template <int T>
__device__ __forceinline__ bool broad_phase(const ContactCull& cull, const sdfo_body_state& sA, const PoseFrame& f,
                                            BroadShared& s)
{
    if (!cull.enabled) return true;
    if (threadIdx.x == 0)
    {
        const v3 lo = mulT(sA.R, V(cull.bmin[0], cull.bmin[1], cull.bmin[2]) - f.rA);
        const v3 hi = mulT(sA.R, V(cull.bmax[0], cull.bmax[1], cull.bmax[2]) - f.rA);
        s.box[0] = lo.x - cull.box_margin;
        s.box[1] = lo.y - cull.box_margin;
        s.box[2] = lo.z - cull.box_margin;
        s.box[3] = hi.x + cull.box_margin;
        s.box[4] = hi.y + cull.box_margin;
        s.box[5] = hi.z + cull.box_margin;
        bool enc = true;
        for (int a = 0; a < 3; ++a) enc = enc && s.box[a] <= cull.root[a] && s.box[3 + a] >= cull.root[3 + a];
        s.full = enc ? 1 : 0;
    }
    for (int w = threadIdx.x; w < (cull.nleaves + 31) / 32; w += T) s.mask[w] = 0u;
    __syncthreads();
    if (s.full != 0) return true;
    bool any = false;
    for (int l = threadIdx.x; l < cull.nleaves; l += T)
    {
        const double* b = cull.leaf_box + 6 * (int64_t)l;
        const bool skip = b[3] < s.box[0] || b[4] < s.box[1] || b[5] < s.box[2] || b[0] > s.box[3] ||
                          b[1] > s.box[4] || b[2] > s.box[5];
        if (!skip)
        {
            atomicOr(&s.mask[l >> 5], 1u << (l & 31));
            any = true;
        }
    }
    return __syncthreads_or(any) == 0; // no leaf: every point (contacts_sdf.py:268-269)
}

// What a thread has measured.
struct Measured
{
    MinRec best{INFINITY, INT_MAX, -1};
    int nvalid = 0, nactive = 0;
    __device__ __forceinline__ void point(const ContactCull& cull, bool full, int i, double gap)
    {
        ++nvalid;
        if (gap < 0.0) ++nactive;
        const MinRec r{gap, full ? (cull.porig ? __ldg(cull.porig + i) : i) : i, i};
        if (less_rec(r, best)) best = r;
    }
};

template <int WARPS>
struct MeasureShared
{
    MinRec min[WARPS];
    int cnt[WARPS][2];
    int prefix;
};

// measure_pair's result from all threads' (contacts_sdf.py:171-214).
template <int MODE, bool SPARSE, int BD, int T>
__device__ __forceinline__ void write_measure(const GridView& g, const float* __restrict__ qx,
                                              const sdfo_body_state& sA, const sdfo_body_state& sB, const PoseFrame& f,
                                              const ContactCull& cull, bool full, const BroadShared& broad,
                                              MeasureShared<T / 32>& s, const Measured& mine,
                                              sdfo_contact_measure* __restrict__ out_at)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    {
        const MinRec r = warp_min(mine.best);
        const int nv = warp_isum(mine.nvalid), na = warp_isum(mine.nactive);
        if (lane == 0)
        {
            s.min[warp] = r;
            s.cnt[warp][0] = nv;
            s.cnt[warp][1] = na;
        }
        if (threadIdx.x == 0) s.prefix = 0;
    }
    __syncthreads();
    MinRec b = s.min[0];
    int nv = s.cnt[0][0], na = s.cnt[0][1];
#pragma unroll
    for (int w = 1; w < T / 32; ++w)
    {
        if (less_rec(s.min[w], b)) b = s.min[w];
        nv += s.cnt[w][0];
        na += s.cnt[w][1];
    }
    // position of the minimum in the broad phase's point list: the points of
    // the kept leaves before its own
    if (nv > 0 && !full)
    {
        const int lb = __ldg(cull.pleaf + b.i);
        int part = 0;
        for (int l = threadIdx.x; l < lb; l += T)
            if ((broad.mask[l >> 5] >> (l & 31)) & 1u) part += __ldg(cull.leaf_start + l + 1) - __ldg(cull.leaf_start + l);
        part = warp_isum(part);
        if (lane == 0 && part) atomicAdd(&s.prefix, part);
        __syncthreads();
    }
    if (threadIdx.x != 0) return;
    sdfo_contact_measure out;
    out.reserved0 = 0;
    out.active_count = na;
    out.valid_count = nv;
    if (nv == 0)
    {
        out.gap = INFINITY;
        out.penetration = 0.0;
        out.normal_velocity = 0.0;
        out.min_point_index = -1;
    }
    else
    {
        out.gap = b.gap;
        out.penetration = b.gap < 0.0 ? -b.gap : 0.0;
        out.min_point_index = full ? b.key : s.prefix + (b.i - __ldg(cull.leaf_start + __ldg(cull.pleaf + b.i)));
        // normal relative velocity at the minimum (contacts_sdf.py:199-211)
        const v3 X = V(__ldg(qx + 3 * b.i), __ldg(qx + 3 * b.i + 1), __ldg(qx + 3 * b.i + 2));
        const v3 off = mul(sA.R, X);
        const v3 Yv = mulT(sB.R, off) + f.tl;
        const double Y[3] = {Yv.x, Yv.y, Yv.z};
        float gapf;
        v3 gl;
        double Hl[6];
        sample<MODE, SPARSE, BD, false>(g, Y, gapf, gl, Hl);
        const double gn = sqrt(dot(gl, gl));
        const v3 un = gn > 1e-30 ? (1.0 / gn) * gl : V(0.0, 0.0, 1.0);
        v3 nw = mul(sB.R, un);
        const double nn = sqrt(dot(nw, nw));
        if (nn > 1e-30) nw = (1.0 / nn) * nw;
        const v3 xw = f.rA + off;
        const v3 uA = f.vA + cross(f.wA, off);
        const v3 uB = f.vB + cross(f.wB, xw - f.rB);
        out.normal_velocity = dot(uA - uB, nw);
    }
    *out_at = out;
}

// N lists of kJacSpan / N entries at most, taken one after the other: their
// lengths' inclusive prefix, lane by lane, and from it the place of entry e.  All
// lanes call both.  (Held in registers, sixteen lengths would spill in the loops
// of the force law.)
template <int N>
struct Lists
{
    int pre, total;
    __device__ __forceinline__ explicit Lists(const int* lengths)
    {
        const int lane = (int)(threadIdx.x & 31);
        pre = lane < N ? lengths[lane] : 0;
#pragma unroll
        for (int o = 1; o < N; o *= 2)
        {
            const int q = __shfl_up_sync(0xffffffffu, pre, o);
            if (lane >= o) pre += q;
        }
        total = __shfl_sync(0xffffffffu, pre, N - 1);
    }
    __device__ __forceinline__ int place(int e) const
    {
        int src = 0;
#pragma unroll
        for (int o = N / 2; o > 0; o /= 2)
            if (__shfl_sync(0xffffffffu, pre, src + o - 1) <= e) src += o;
        const int before = __shfl_sync(0xffffffffu, pre, src > 0 ? src - 1 : 0);
        return src * (kJacSpan / N) + e - (src > 0 ? before : 0);
    }
};

// The Jacobian of the points in contact, in kForceRows lists, into as many
// sums (kJacRows with touch bits).
template <int MODE, bool SPARSE, int BD, bool TOUCH, int T>
__device__ __forceinline__ void jacobian_pass(const GridView& g, const float* __restrict__ qx,
                                              const float* __restrict__ qw, const sdfo_body_state& sA,
                                              const sdfo_body_state& sB, const PoseFrame& f,
                                              const sdfo_contact_params& prm, double narrow, const int* list,
                                              const int* lengths, double (*sums)[36])
{
    constexpr int kWarps = T / 32, kRows = TOUCH ? kJacRows : kWarps;
    const int warp = (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31);
    const Lists<kForceRows> lists(lengths);
    auto add_column = [&](const double col[6], int row, int j) {
#pragma unroll
        for (int r = 0; r < 6; ++r)
        {
            const double sum = warp_sum(col[r]);
            if (lane == 0) sums[row][6 * r + j] += sum;
        }
    };
    auto in_contact = [&](int e, int at, PointState& st) {
        double gap = 0.0;
        return e < lists.total && point_state<MODE, SPARSE, BD, true>(g, qx, qw, list[at], sA, sB, f, prm, narrow, false,
                                                                      st, gap) == 2;
    };
    if (TOUCH && lists.total <= 32 * kSplitGroups)
    {
        // few points in contact: one column of 32 points at a time, so that more
        // warps have work
        for (int k = warp; 32 * (k / 6) < lists.total; k += kWarps) // warp-uniform
        {
            const int e = 32 * (k / 6) + lane, at = lists.place(e);
            double col[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
            PointState st;
            if (in_contact(e, at, st)) jacobian_column(st, sB, f, prm, k % 6, col);
            add_column(col, k % kRows, k % 6);
        }
        return;
    }
    for (int k = warp; 32 * k < lists.total; k += kWarps) // warp-uniform
    {
        const int e = 32 * k + lane, at = lists.place(e);
        PointState st;
        const bool mine = in_contact(e, at, st);
#pragma unroll 1
        for (int j = 0; j < 6; ++j)
        {
            double col[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
            if (mine) jacobian_column(st, sB, f, prm, j, col);
            add_column(col, k % kRows, j);
        }
    }
}

// The sum of N values `stride` apart, by halves.
template <int N>
__device__ __forceinline__ double row_sum(const double* p, int stride)
{
    double v[N];
#pragma unroll
    for (int w = 0; w < N; ++w) v[w] = p[w * stride];
#pragma unroll
    for (int h = N / 2; h > 0; h /= 2)
#pragma unroll
        for (int w = 0; w < h; ++w) v[w] += v[w + h];
    return v[0];
}

// EXT: the culled / measuring variant (ContactCull, measures); without it
// every point is evaluated and no measure is produced.
// TOUCH: `bits` are the mode's touch bits of a dense grid.  The first pass lists
// the points that may touch (with JAC alone: the points in contact), the second
// evaluates the list.
template <int MODE, bool SPARSE, int BD, bool JAC, bool EXT, bool TOUCH, int T, int MB>
__global__ void __launch_bounds__(T, MB)
    k_contact(GridView g, const float* __restrict__ qx, const float* __restrict__ qw, int nq,
              const sdfo_body_state* __restrict__ poses, const sdfo_body_state* __restrict__ body_b,
              sdfo_contact_params prm, double* __restrict__ ft, double* __restrict__ jac,
              ContactCull cull,
              sdfo_contact_measure* __restrict__ meas, const uint32_t* __restrict__ bits)
{
    constexpr int kWarps = T / 32;
    constexpr int kPerList = kJacSpan / kWarps, kPerAct = kJacSpan / kForceRows;
    constexpr int kRows = TOUCH ? kJacRows : kWarps; // sums of the Jacobian
    const int pose = blockIdx.x;
    __shared__ sdfo_body_state sA, sB;
    __shared__ double red[kForceRows][6];
    __shared__ double sjac[JAC ? kRows : 1][36];
    constexpr bool LIST = JAC || TOUCH;
    __shared__ int s_list[LIST ? kJacSpan : 1];
    __shared__ int s_act[TOUCH && JAC ? kJacSpan : 1];
    __shared__ int s_acnt[kForceRows];
    __shared__ Place32 s_touch;
    __shared__ int s_wcnt[kWarps];
    __shared__ BroadShared s_broad;
    __shared__ MeasureShared<kWarps> s_meas;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    load_states(poses + pose, body_b, sA, sB);
    if (JAC)
        for (int t = threadIdx.x; t < kRows * 36; t += T) (&sjac[0][0])[t] = 0.0;
    __syncthreads();
    const PoseFrame f = pose_frame(sA, sB);
    Place32 tf;
    if (TOUCH)
    {
        set_place_entry(g, sA, sB, f.tl, (int)threadIdx.x, s_touch);
        __syncthreads();
        tf = s_touch;
        tf.set_margin(s_touch.e0);
    }

    const bool full = EXT ? broad_phase<T>(cull, sA, f, s_broad) : true;
    const double narrow = EXT && cull.enabled ? cull.narrow_margin : -1.0;
    const bool want_force = ft != nullptr;
    const bool want_meas = EXT && meas != nullptr;
    double acc[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    Measured seen;

    // whether the broad phase keeps point i
    auto kept = [&](int i) {
        if (!EXT || full) return true;
        const int l = __ldg(cull.pleaf + i);
        return ((s_broad.mask[l >> 5] >> (l & 31)) & 1u) != 0;
    };
    auto add_force = [&](const PointState& st, double* sum) {
        const v3 tq = cross(st.off, st.fq);
        sum[0] = fma(st.wq, st.fq.x, sum[0]);
        sum[1] = fma(st.wq, st.fq.y, sum[1]);
        sum[2] = fma(st.wq, st.fq.z, sum[2]);
        sum[3] = fma(st.wq, tq.x, sum[3]);
        sum[4] = fma(st.wq, tq.y, sum[4]);
        sum[5] = fma(st.wq, tq.z, sum[5]);
    };

    // Spans of kJacSpan points (one span over all points when nothing is
    // listed).  First every point: by its touch bit, or by the forward law; each
    // warp lists its points, in point order, with no barrier.  Then the span's
    // list, one list after the other, is shared out by groups of 32 entries, so
    // all warps carry the FP64 work, and the sums run in a fixed order (repeated
    // runs are bit-identical).  Block-uniform trip counts: the barriers and warp
    // reductions below see every thread.
    for (int s0 = 0; s0 < nq; s0 += LIST ? kJacSpan : nq)
    {
    const int s1 = LIST ? min(nq, s0 + kJacSpan) : nq;
    // this warp's list: the place of its half in the order of all (see kForceRows)
    const int half = (warp % kForceRows) * (kWarps / kForceRows) + warp / kForceRows;
    int wcnt = 0; // its points (warp-uniform)
    // appends the lanes' points to a list of which `count` are filled
    auto append = [&](int* list, int& count, bool listed, int i) {
        const unsigned m = __ballot_sync(0xffffffffu, listed);
        if (listed) list[count + __popc(m & ((1u << lane) - 1u))] = i;
        count += __popc(m);
    };
    if constexpr (TOUCH)
    {
        // kAhead points per thread at a time: their loads, and then those of
        // their bits, are in flight together
        constexpr int kStride = 32 * kForceRows;
        const int base = s0 + 32 * (warp % kForceRows) + kJacSpan * kForceRows / kWarps * (warp / kForceRows) + lane;
        for (int j = 0; j < kPerList / 32 && base - lane + j * kStride < s1; j += kAhead)
        {
            float x[kAhead][3];
            bool in[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; ++u)
            {
                const int i = base + (j + u) * kStride;
                in[u] = i < s1 && kept(i);
#pragma unroll
                for (int a = 0; a < 3; ++a) x[u][a] = in[u] ? __ldg(qx + 3 * i + a) : 0.f;
            }
            int status[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; ++u) status[u] = touch_status(g, bits, tf, x[u][0], x[u][1], x[u][2]);
#pragma unroll
            for (int u = 0; u < kAhead; ++u)
            {
                if (want_meas && in[u] && status[u] == kClear) ++seen.nvalid;
                append(s_list + half * kPerList, wcnt, in[u] && status[u] == kMayTouch, base + (j + u) * kStride);
            }
        }
    }
    else
    {
        for (int i0 = s0; i0 < s1; i0 += T)
        {
            const int i = i0 + threadIdx.x;
            bool act = false;
            if (i < s1 && kept(i))
            {
                PointState st;
                double gap = 0.0;
                const int status =
                    point_state<MODE, SPARSE, BD, false>(g, qx, qw, i, sA, sB, f, prm, narrow, want_meas, st, gap);
                if (want_meas && status > 0) seen.point(cull, full, i, gap);
                act = status == 2 && want_force;
                if (act) add_force(st, acc);
            }
            if (LIST) append(s_list + warp * kPerList, wcnt, act, i);
        }
    }
    if (LIST)
    {
        if (lane == 0) s_wcnt[TOUCH ? half : warp] = wcnt;
        __syncthreads();
        if constexpr (TOUCH)
        {
            const Lists<kWarps> lists(s_wcnt);
            if (lists.total == 0)
            {
                __syncthreads();
                continue;
            }
            if (warp < kForceRows)
            {
                int acnt = 0;
                for (int k = warp; 32 * k < lists.total; k += kForceRows) // warp-uniform
                {
                    const int e = 32 * k + lane, at = lists.place(e);
                    bool act = false;
                    int idx = 0;
                    if (e < lists.total)
                    {
                        idx = s_list[at];
                        PointState st;
                        double gap = 0.0;
                        const int status = point_state<MODE, SPARSE, BD, false>(g, qx, qw, idx, sA, sB, f, prm, narrow,
                                                                                want_meas, st, gap);
                        if (want_meas && status > 0) seen.point(cull, full, idx, gap);
                        act = status == 2 && want_force;
                        if (act) add_force(st, acc);
                    }
                    if (JAC) append(s_act + warp * kPerAct, acnt, act, idx);
                }
                if (JAC && lane == 0) s_acnt[warp] = acnt;
            }
            if (JAC) __syncthreads();
        }
        if constexpr (JAC)
        {
            jacobian_pass<MODE, SPARSE, BD, TOUCH, T>(g, qx, qw, sA, sB, f, prm, narrow, TOUCH ? s_act : s_list,
                                                      TOUCH ? s_acnt : s_wcnt, sjac);
        }
        __syncthreads(); // s_list and s_wcnt are rewritten by the next span
    }
    }
    if (TOUCH && want_meas && __syncthreads_or(seen.best.gap <= 0.0) == 0)
    {
        // Clear of the surface: the least gap is not among the listed points
        // (elsewhere gaps are positive), so every point is measured.
        seen = Measured{};
        for (int i = threadIdx.x; i < nq; i += T)
            if (kept(i))
            {
                PointState st;
                double gap = 0.0;
                if (point_state<MODE, SPARSE, BD, false>(g, qx, qw, i, sA, sB, f, prm, narrow, true, st, gap) > 0)
                    seen.point(cull, full, i, gap);
            }
    }
    if (want_force && warp < kForceRows)
    {
#pragma unroll
        for (int q = 0; q < 6; ++q)
        {
            const double s = warp_sum(acc[q]);
            if (lane == 0) red[warp][q] = s;
        }
    }
    __syncthreads();
    if (want_force && threadIdx.x < 6)
    {
        ft[6 * (int64_t)pose + threadIdx.x] = row_sum<kForceRows>(&red[0][threadIdx.x], 6);
    }
    if (JAC && jac != nullptr && threadIdx.x < 36)
    {
        jac[36 * (int64_t)pose + threadIdx.x] = row_sum<kRows>(&sjac[0][threadIdx.x], 36);
    }
    if (want_meas)
        write_measure<MODE, SPARSE, BD, T>(g, qx, sA, sB, f, cull, full, s_broad, s_meas, seen, meas + pose);
}

// How a measure alone (no forces) meets its points.
enum : int
{
    kEveryPoint = 0, // FP64 for each
    kByBounds = 1,   // dense Trilinear: FP64 where FP32 bounds of the gap leave it open
    kByTouch = 2     // dense Tricubic: FP64 where the touch bits leave it open; if no
                     // gap is <= 0, for every point
};

// The least value of the warp's lanes (FP32 as ordered integers).
__device__ __forceinline__ float warp_least(float v)
{
    const int b = __float_as_int(v);
    const int m = __reduce_min_sync(0xffffffffu, b ^ ((b >> 31) & 0x7fffffff));
    return __int_as_float(m ^ ((m >> 31) & 0x7fffffff));
}

// measure_pair of every pose, without the forces (one CTA per pose).  Bound by
// the gather of every point and, for kEveryPoint, its FP64 transform.  kByBounds
// reads the cell record that the FP64 path would read, in FP32 alone, and takes
// the FP64 path only for points that may be the least (a warp shares the least
// upper bound met) or whose sign is open; so every point that attains the least
// gap is sampled, and gap, index and counts are those of sampling all.  4,096
// poses of a 7,680-point ring about a block, clear of it / in light / in deep
// contact, in the force kernel by touch bits and here (us): Trilinear 505 / 412 /
// 669 and 289 / 309 / 283; Tricubic 594 / 310 / 760 and 477 / 271 / 445.
template <int MODE, bool SPARSE, int BD, int HOW, int T, int MB>
__global__ void __launch_bounds__(T, MB)
    k_measure(GridView g, const float* __restrict__ qx, int nq, const sdfo_body_state* __restrict__ poses,
              const sdfo_body_state* __restrict__ body_b, ContactCull cull, sdfo_contact_measure* __restrict__ meas,
              const uint32_t* __restrict__ bits)
{
    const int pose = blockIdx.x;
    __shared__ sdfo_body_state sA, sB;
    __shared__ Place32 s_place;
    __shared__ BroadShared s_broad;
    __shared__ MeasureShared<T / 32> s_meas;
    load_states(poses + pose, body_b, sA, sB);
    __syncthreads();
    const PoseFrame f = pose_frame(sA, sB);
    Place32 at;
    if (HOW != kEveryPoint)
    {
        set_place_entry(g, sA, sB, f.tl, (int)threadIdx.x, s_place);
        __syncthreads();
        at = s_place;
        at.set_margin(s_place.e0);
    }
    const bool full = broad_phase<T>(cull, sA, f, s_broad);
    Measured seen;
    auto kept = [&](int i) {
        if (full) return true;
        const int l = __ldg(cull.pleaf + i);
        return ((s_broad.mask[l >> 5] >> (l & 31)) & 1u) != 0;
    };
    auto sample_point = [&](int i, float x, float y, float z) {
        const v3 Yv = mulT(sB.R, mul(sA.R, V(x, y, z))) + f.tl;
        const double Y[3] = {Yv.x, Yv.y, Yv.z};
        float gap;
        v3 gl;
        double Hl[6];
        if (sample<MODE, SPARSE, BD, false>(g, Y, gap, gl, Hl)) seen.point(cull, full, i, gap);
    };
    float least = INFINITY; // no gap above it is needed
    for (int i0 = 0; i0 < nq; i0 += T) // the same trips for every lane of a warp
    {
        const int i = i0 + (int)threadIdx.x;
        const bool in = i < nq && kept(i);
        float x = 0.f, y = 0.f, z = 0.f;
        if (in)
        {
            x = __ldg(qx + 3 * i);
            y = __ldg(qx + 3 * i + 1);
            z = __ldg(qx + 3 * i + 2);
        }
        bool open = in;
        if (HOW == kByBounds)
        {
            float gap = 0.f, eps = 0.f;
            bool out = false;
            const bool known = in && gap32(g, at, x, y, z, gap, eps, out);
            least = warp_least(known ? fminf(least, gap + eps) : least);
            const bool below = gap + eps < 0.f; // certainly active
            if (known && gap - eps > least && (gap - eps > 0.f || below))
            {
                ++seen.nvalid;
                if (below) ++seen.nactive;
                open = false;
            }
            open = open && !out;
        }
        if (HOW == kByTouch)
        {
            const int status = touch_status(g, bits, at, x, y, z);
            if (in && status == kClear) ++seen.nvalid;
            open = in && status == kMayTouch;
        }
        if (open) sample_point(i, x, y, z);
    }
    if (HOW == kByTouch && __syncthreads_or(seen.best.gap <= 0.0) == 0)
    {
        // clear of the surface: the least gap may be among the points left out
        seen = Measured{};
        for (int i = threadIdx.x; i < nq; i += T)
            if (kept(i)) sample_point(i, __ldg(qx + 3 * i), __ldg(qx + 3 * i + 1), __ldg(qx + 3 * i + 2));
    }
    write_measure<MODE, SPARSE, BD, T>(g, qx, sA, sB, f, cull, full, s_broad, s_meas, seen, meas + pose);
}

struct ContactLaunch
{
    const float* qx;
    const float* qw;
    int nq;
    const sdfo_body_state* pa;
    int np;
    const sdfo_body_state* pb;
    sdfo_contact_params prm;
    double* ft;
    double* jac;
    ContactCull cull;
    sdfo_contact_measure* meas;
};

template <int MODE, bool SPARSE, int BD, bool EXT, bool TOUCH, int T, int MB, int JAC_MB>
void launch5(const GridView& v, const ContactLaunch& c, const uint32_t* bits, cudaStream_t s)
{
    if (c.jac)
        k_contact<MODE, SPARSE, BD, true, EXT, TOUCH, T, JAC_MB><<<c.np, T, 0, s>>>(
            v, c.qx, c.qw, c.nq, c.pa, c.pb, c.prm, c.ft, c.jac, c.cull, c.meas, bits);
    else
        k_contact<MODE, SPARSE, BD, false, EXT, TOUCH, T, MB><<<c.np, T, 0, s>>>(
            v, c.qx, c.qw, c.nq, c.pa, c.pb, c.prm, c.ft, c.jac, c.cull, c.meas, bits);
}

template <int MODE, bool SPARSE, int BD, bool EXT, bool TOUCH>
void launch4(const GridView& v, const ContactLaunch& c, const uint32_t* bits, cudaStream_t s)
{
    constexpr int MB = SDFO_CONTACT_MIN_BLOCKS, JAC_MB = SDFO_CONTACT_JAC_MIN_BLOCKS;
    if constexpr (TOUCH)
    {
        if (c.np <= current_sm_count())
        {
            launch5<MODE, SPARSE, BD, EXT, TOUCH, kFewThreads, 1, 1>(v, c, bits, s);
            return;
        }
        // Trilinear Jacobians with touch bits gain by a third CTA per SM where there
        // are poses for it (4,096 poses, a quarter in light contact: 5 %), and lose
        // by its spills where there are not (149 poses in deep contact: 448 us with
        // two, 514 with three).
        if constexpr (MODE == SDFO_TRILINEAR)
            if (c.jac && c.np > 2 * current_sm_count())
            {
                launch5<MODE, SPARSE, BD, EXT, TOUCH, kContactThreads, MB, 3>(v, c, bits, s);
                return;
            }
    }
    launch5<MODE, SPARSE, BD, EXT, TOUCH, kContactThreads, MB, JAC_MB>(v, c, bits, s);
}

template <int MODE, bool SPARSE, int BD, bool TOUCH>
void launch3(const GridView& v, const ContactLaunch& c, const uint32_t* bits, cudaStream_t s)
{
    if (c.cull.enabled || c.meas)
        launch4<MODE, SPARSE, BD, true, TOUCH>(v, c, bits, s);
    else
        launch4<MODE, SPARSE, BD, false, TOUCH>(v, c, bits, s);
}

// Resident CTAs per SM asked of the register allocator for a measure (256 threads
// each): 4,096 clear poses, Trilinear 351 / 289 / 275 us at 3 / 4 / 5, Tricubic 539 /
// 477 / 529.
#ifndef SDFO_MEASURE_MIN_BLOCKS
#define SDFO_MEASURE_MIN_BLOCKS 4
#endif

template <int MODE, bool SPARSE, int BD, int HOW>
void launch_measure(const GridView& v, const ContactLaunch& c, const uint32_t* bits, cudaStream_t s)
{
    if (c.np <= current_sm_count())
        k_measure<MODE, SPARSE, BD, HOW, kFewThreads, 1><<<c.np, kFewThreads, 0, s>>>(v, c.qx, c.nq, c.pa, c.pb, c.cull,
                                                                                      c.meas, bits);
    else
        k_measure<MODE, SPARSE, BD, HOW, kContactThreads, SDFO_MEASURE_MIN_BLOCKS>
            <<<c.np, kContactThreads, 0, s>>>(v, c.qx, c.nq, c.pa, c.pb, c.cull, c.meas, bits);
}

template <int MODE>
void launch2(const GridView& v, const ContactLaunch& c, cudaStream_t s)
{
    if (c.meas && !c.ft)
    {
        // the touch bits and records of a grid that owns its payload
        const int64_t voxels = (int64_t)v.nx * v.ny * v.nz;
        const bool owned = v.layout == SDFO_LAYOUT_DENSE && v.touch && v.cell8 && voxels < (int64_t(1) << 31);
        if (v.layout != SDFO_LAYOUT_DENSE && v.bd == 8)
            launch_measure<MODE, true, 8, kEveryPoint>(v, c, nullptr, s);
        else if (v.layout != SDFO_LAYOUT_DENSE)
            launch_measure<MODE, true, 0, kEveryPoint>(v, c, nullptr, s);
        else if (!owned)
            launch_measure<MODE, false, 0, kEveryPoint>(v, c, nullptr, s);
        else if constexpr (MODE == SDFO_TRICUBIC)
            launch_measure<MODE, false, 0, kByTouch>(v, c, v.touch + touch_words(voxels), s);
        else
            launch_measure<MODE, false, 0, kByBounds>(v, c, nullptr, s);
        return;
    }
    if (v.layout == SDFO_LAYOUT_DENSE)
    {
        // The touch bits say where the gap can be <= 0; they leave out points
        // whose force is k 0^n, so the law needs n > 0.  Views have no bits.
        const int64_t voxels = (int64_t)v.nx * v.ny * v.nz;
        if (v.touch && c.prm.order > 0.0 && voxels < (int64_t(1) << 31))
            launch3<MODE, false, 0, true>(v, c, v.touch + (MODE == SDFO_TRICUBIC ? touch_words(voxels) : 0), s);
        else
            launch3<MODE, false, 0, false>(v, c, nullptr, s);
    }
    else if (v.bd == 8)
        launch3<MODE, true, 8, false>(v, c, nullptr, s);
    else
        launch3<MODE, true, 0, false>(v, c, nullptr, s);
}

} // namespace

void launch_contact(const GridView& v, int mode, const float* qx, const float* qw, int64_t nq,
                    const sdfo_body_state* pose_a, int64_t np, const sdfo_body_state* body_b,
                    const sdfo_contact_params& prm, double* ft, double* jac, cudaStream_t s,
                    const ContactCull* cull, sdfo_contact_measure* meas)
{
    if (np <= 0) return;
    ContactLaunch c{qx, qw, (int)nq, pose_a, (int)np, body_b, prm, ft, jac, ContactCull{}, meas};
    if (cull) c.cull = *cull;
    if (mode == SDFO_TRICUBIC)
        launch2<SDFO_TRICUBIC>(v, c, s);
    else
        launch2<SDFO_TRILINEAR>(v, c, s);
    SDFO_CHECK_LAUNCH();
}

} // namespace sdfo
