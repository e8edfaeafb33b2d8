// SDF construction on the device: LBVH over the triangles, closest-triangle
// and ray-parity traversal, dense fill + Hessian, sparse narrow-band
// activation / compaction / brick fill / Hessian.
//
// This translation unit is compiled with -fmad=false: every FP64 expression
// on the distance / sign path is evaluated in the order written, which is the
// reference's order (KdTree.h, SdfBuilder.cpp), so distances, witness points,
// normals and signs are bit-identical to the reference's FP64 arithmetic.
//
// Two acceleration structures (sdfo_set_bvh_mode):
//  * SDFO_BVH_REFERENCE (default): the reference's median-split tree
//    (KdTree.h:91-121, 188-242) built on the host with std::nth_element and
//    traversed on the device in the reference's near-first order with FP64
//    boxes.  Exactly equidistant triangles then resolve to the same triangle
//    as in the reference, which matters: for points the parity ray misses the
//    sign comes from that triangle's face normal (KdTree.h:156-163).
//  * SDFO_BVH_LBVH: a device-built linear BVH --
//      63-bit Morton codes of triangle centroids, radix-sorted (CUB),
//      Karras (2012) binary radix tree, one thread per internal node,
//      bottom-up FP64 box refit with per-node arrival counters,
//      packed 64-byte nodes holding both child boxes in FP32, rounded outward
//      and widened by a margin so FP32 culling is conservative.
//    Ties resolve to the lowest triangle index.
// Both decide every distance and every ray hit with the FP64 triangle tests.
// The fills over the reference-order tree run warp-wide (warp_tree.cuh), with
// the same results.
#include <atomic>
#include <climits>

#include "warp_tree.cuh"

namespace sdfo {

// ---------------------------------------------------------------------------
// host grid setup: SdfBuilder::setupGrid (SdfBuilder.cpp:994-1035)
// ---------------------------------------------------------------------------
namespace {
int snap_resolution(int n, int maxRes)
{
    // snapToStandardResolution (GridSpec.h:65-74)
    static const int levels[] = {8, 16, 32, 64, 128, 256, 512, 1024, 2048};
    for (int v : levels)
        if (v >= n || v >= maxRes) return std::min(v, maxRes);
    return maxRes;
}
} // namespace

sdfo_grid_info setup_grid(const double* verts, int64_t nv, const sdfo_build_params& p)
{
    double vmin[3] = {1e30, 1e30, 1e30}, vmax[3] = {-1e30, -1e30, -1e30};
    for (int64_t i = 0; i < nv; ++i)
        for (int a = 0; a < 3; ++a)
        {
            const double x = verts[3 * i + a];
            vmin[a] = x < vmin[a] ? x : vmin[a];
            vmax[a] = vmax[a] < x ? x : vmax[a];
        }
    const double d0 = vmax[0] - vmin[0], d1 = vmax[1] - vmin[1], d2 = vmax[2] - vmin[2];
    const double diag = std::sqrt(d0 * d0 + d1 * d1 + d2 * d2);
    const double pad = p.padding * diag;
    double bmin[3], size[3];
    for (int a = 0; a < 3; ++a)
    {
        bmin[a] = vmin[a] - pad;
        size[a] = (vmax[a] + pad) - bmin[a];
    }
    double h = p.voxel_size;
    if (h <= 0.0)
    {
        double longest = size[0];
        if (longest < size[1]) longest = size[1];
        if (longest < size[2]) longest = size[2];
        h = longest / (double)p.target_resolution;
    }
    sdfo_grid_info info{};
    for (int a = 0; a < 3; ++a)
    {
        const double raw = std::ceil(size[a] / h);
        SDFO_REQUIRE(std::isfinite(raw) && raw < 1e9, SDFO_ERR_INVALID_ARGUMENT,
                     "grid resolution out of range");
        const int rawN = std::max(1, (int)raw);
        info.shape[a] = snap_resolution(rawN, p.max_resolution);
        info.bmin[a] = bmin[a];
        info.voxel[a] = h;
    }
    for (int a = 0; a < 3; ++a) info.bmax[a] = bmin[a] + (double)info.shape[a] * h;
    info.layout = SDFO_LAYOUT_DENSE;
    info.storage = SDFO_STORAGE_FP32;
    info.has_hessian = 1;
    return info;
}

namespace {
std::atomic<int> g_bvh_mode{SDFO_BVH_REFERENCE};
std::atomic<int> g_fill_tile{(3 << 8) | 3}; // log2 x << 8 | log2 y: 8 x 8 x 4
FillTile fill_tile()
{
    const int v = g_fill_tile.load();
    return FillTile{v >> 8, v & 255};
}
} // namespace

int bvh_mode() { return g_bvh_mode.load(); }
void set_bvh_mode(int m) { g_bvh_mode.store(m); }
namespace {
std::atomic<int> g_sign_mode{SDFO_SIGN_RAY_PARITY};
} // namespace
int sign_mode() { return g_sign_mode.load(); }
void set_sign_mode(int m) { g_sign_mode.store(m); }
namespace {
// stackless by default: the same results; 1.31M-triangle icosphere sparse
// fill 70.6 ms against 89.0 with the per-thread stack, hollow cylinder even
std::atomic<int> g_lbvh_stackless{1};
} // namespace
int lbvh_stackless() { return g_lbvh_stackless.load(); }
namespace {
std::atomic<int> g_triangle_cull{1};
} // namespace
int triangle_cull() { return g_triangle_cull.load(); }
void set_triangle_cull(int on) { g_triangle_cull.store(on ? 1 : 0); }
void set_lbvh_stackless(int on) { g_lbvh_stackless.store(on ? 1 : 0); }
void set_fill_tile(int lx, int ly) { g_fill_tile.store(((lx > 0 ? lx : 3) << 8) | (ly > 0 ? ly : 3)); }
void get_fill_tile(int* lx, int* ly)
{
    const FillTile t = fill_tile();
    *lx = t.lx;
    *ly = t.ly;
}


namespace {
// The warp-wide fill's data over `tree`, where the fills use it: the
// reference-order tree with the triangle cull on (it needs the FP32 boxes), from
// kWarpFillTris triangles and, where the number of voxels is known, a quarter as
// many pairs of patches (64 voxels) as SMs.  Below that the per-thread traversal
// has little to diverge over and its one launch is the cheaper.  Whole builds by
// it and warp-wide: 128 triangles into 64 x 64 x 32 voxels 0.24 and 0.28 ms, 256
// triangles 0.33 and 0.30; 3,072 triangles into 8 x 8 x 24 0.63 and 0.78, 4,608
// into 24 x 24 x 8 1.31 and 0.80.
constexpr int kWarpFillTris = 256;
bool build_warp_tree(DeviceWarpTree& w, const AnyTree& tree, const sdfo_grid_info& grid, int64_t voxels, cudaStream_t s)
{
    if (tree.mode == SDFO_BVH_LBVH || !triangle_cull() || tree.ref.n < kWarpFillTris ||
        tree.ref.n > INT_MAX / kMaxCellsPerTri || !std::isfinite(tree.ref.extent) ||
        voxels < 16 * (int64_t)current_sm_count())
        return false;
    w.build(tree.ref.view(), tree.ref.lo, tree.ref.hi, grid, tree.ref.extent, s);
    return true;
}
} // namespace

sdfo_grid* build_dense(const double* verts, int64_t nv, const int32_t* tris, int64_t nt,
                       const sdfo_build_params& p, cudaStream_t s)
{
    const auto t0 = std::chrono::steady_clock::now();
    std::unique_ptr<sdfo_grid> g(new sdfo_grid());
    g->info = setup_grid(verts, nv, p);
    SDFO_CUDA(cudaGetDevice(&g->device));
    const int64_t N = (int64_t)g->info.shape[0] * g->info.shape[1] * g->info.shape[2];
    g->stored_voxels = N;
    g->stats.triangles = (int32_t)nt;
    // the grid's storage (setup_ms counts these allocations)
    g->d.phin = dalloc<float4>((size_t)N);
    g->d.phi64 = dalloc<double>((size_t)N);
    g->d.n64 = dalloc<double>((size_t)N * 3);
    g->d.w64 = dalloc<double>((size_t)N * 3);
    g->d.h64 = dalloc<double>((size_t)N * 6);
    g->d.hess6 = dalloc<float>((size_t)N * 6);
    DeviceBuffer<int> status(1);
    SDFO_CUDA(cudaMemsetAsync(status.get(), 0, sizeof(int), s));
    g->stats.setup_ms =
        std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    Timer tm(s);
    AnyTree tree{bvh_mode()};
    tree.build(verts, nv, tris, nt, scene_extent(verts, nv, g->info), s);
    DeviceWarpTree warp;
    const bool warp_fill = build_warp_tree(warp, tree, g->info, N, s);
    g->stats.bvh_nodes = tree.node_count(nt);
    g->stats.bvh_ms = tm.lap();
    const SpecD sp = spec_of(g->info);
    const FillTile tile = fill_tile();
    if (warp_fill)
    {
        DenseJob job{};
        job.s = sp;
        job.shape(tile);
        job.phi64 = g->d.phi64;
        job.n64 = g->d.n64;
        job.w64 = g->d.w64;
        job.phin = g->d.phin;
        warp.fill(job, status.get(), s);
    }
    else
        tree.visit([&](auto view) {
            k_dense_fill<<<tile.grid(sp), 256, 0, s>>>(view, sp, tile, g->d.phi64, g->d.n64, g->d.w64, g->d.phin,
                                                       status.get());
        });
    SDFO_CHECK_LAUNCH();
    g->stats.fill_ms = tm.lap();
    k_dense_hessian<<<(unsigned)((N + 255) / 256), 256, 0, s>>>(sp, g->d.n64, g->d.h64, g->d.hess6);
    SDFO_CHECK_LAUNCH();
    build_stencil_layouts(g.get(), s);
    g->stats.hessian_ms = tm.lap();
    check_status(status, s);
    g->stats.voxels_filled = N;
    g->stats.total_ms =
        std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    return g.release();
}

void count_dense_traversal(const double* verts, int64_t nv, const int32_t* tris, int64_t nt,
                           const sdfo_build_params& p, cudaStream_t s, sdfo_traversal_stats* out)
{
    const sdfo_grid_info info = setup_grid(verts, nv, p);
    AnyTree tree{bvh_mode()};
    tree.build(verts, nv, tris, nt, scene_extent(verts, nv, info), s);
    DeviceBuffer<int> status(1);
    DeviceBuffer<unsigned long long> sums(5);
    SDFO_CUDA(cudaMemsetAsync(status.get(), 0, sizeof(int), s));
    SDFO_CUDA(cudaMemsetAsync(sums.get(), 0, 5 * sizeof(unsigned long long), s));
    const SpecD sp = spec_of(info);
    const FillTile tile = fill_tile();
    tree.visit([&](auto view) {
        k_dense_count<<<tile.grid(sp), 256, 0, s>>>(view, sp, tile, sums.get(), status.get());
    });
    SDFO_CHECK_LAUNCH();
    unsigned long long h[5] = {0, 0, 0, 0, 0};
    SDFO_CUDA(cudaMemcpyAsync(h, sums.get(), sizeof(h), cudaMemcpyDeviceToHost, s));
    check_status(status, s); // synchronises s
    out->voxels = (int64_t)info.shape[0] * info.shape[1] * info.shape[2];
    out->nearest_nodes = (int64_t)h[0];
    out->nearest_triangles = (int64_t)h[1];
    out->ray_nodes = (int64_t)h[2];
    out->ray_triangles = (int64_t)h[3];
    out->nearest_triangles_exact = (int64_t)h[4];
}

sdfo_grid* build_sparse(const double* verts, int64_t nv, const int32_t* tris, int64_t nt,
                        const sdfo_sparse_build_params& p, cudaStream_t s)
{
    const auto t0 = std::chrono::steady_clock::now();
    std::unique_ptr<sdfo_grid> g(new sdfo_grid());
    g->info = setup_grid(verts, nv, p.base);
    SDFO_CUDA(cudaGetDevice(&g->device));
    const int bd = p.block_dim;
    // SdfBuilder.cpp:835-842
    const double h = std::max({g->info.voxel[0], g->info.voxel[1], g->info.voxel[2]});
    const double band = p.band_distance > 0.0 ? p.band_distance : (double)p.band_voxels * h;
    const double blockRadius = 0.5 * std::sqrt(3.0) * (double)bd * h;
    volatile double act = band + (double)p.halo_voxels * h;
    act = act + blockRadius;
    const double activation = act;
    g->info.layout = SDFO_LAYOUT_SPARSE;
    g->info.block_dim = bd;
    g->info.halo_voxels = p.halo_voxels;
    g->info.band_distance = band;
    g->info.has_hessian = p.store_hessian ? 1 : 0;
    for (int a = 0; a < 3; ++a) g->nb[a] = (g->info.shape[a] + bd - 1) / bd;
    const int total = g->nb[0] * g->nb[1] * g->nb[2];
    g->stats.triangles = (int32_t)nt;
    g->stats.candidate_blocks = total;
    g->stats.setup_ms =
        std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    Timer tm(s);
    AnyTree tree{bvh_mode()};
    tree.build(verts, nv, tris, nt, scene_extent(verts, nv, g->info), s);
    DeviceWarpTree warp;
    const bool warp_fill = build_warp_tree(warp, tree, g->info, INT64_MAX, s);
    g->stats.bvh_nodes = tree.node_count(nt);
    g->stats.bvh_ms = tm.lap();
    DeviceBuffer<int> status(1);
    SDFO_CUDA(cudaMemsetAsync(status.get(), 0, sizeof(int), s));
    const SpecD sp = spec_of(g->info);
    DeviceBuffer<int32_t> flags(total), slots(total);
    const int T = spread_threads(total);
    tree.visit([&](auto view) {
        k_sparse_activate<<<(total + T - 1) / T, T, 0, s>>>(view, sp, bd, g->nb[0], g->nb[1], g->nb[2],
                                                             activation, flags.get(), status.get());
    });
    SDFO_CHECK_LAUNCH();
    size_t temp = 0;
    SDFO_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, temp, flags.get(), slots.get(), total, s));
    DeviceBuffer<unsigned char> tmp(temp);
    SDFO_CUDA(cub::DeviceScan::ExclusiveSum(tmp.get(), temp, flags.get(), slots.get(), total, s));
    int last_flag = 0, last_slot = 0;
    SDFO_CUDA(cudaMemcpyAsync(&last_flag, flags.get() + total - 1, sizeof(int), cudaMemcpyDeviceToHost, s));
    SDFO_CUDA(cudaMemcpyAsync(&last_slot, slots.get() + total - 1, sizeof(int), cudaMemcpyDeviceToHost, s));
    SDFO_CUDA(cudaStreamSynchronize(s));
    const int B = last_flag + last_slot;
    g->info.block_count = B;
    const int V = bd * bd * bd;
    g->stored_voxels = (int64_t)B * V;
    g->d.table = dalloc<int32_t>((size_t)total);
    g->d.ijk = dalloc<int32_t>((size_t)(B > 0 ? B : 1) * 3);
    k_sparse_table<<<(total + T - 1) / T, T, 0, s>>>(total, g->nb[0], g->nb[1], flags.get(), slots.get(),
                                                      g->d.table, g->d.ijk);
    SDFO_CHECK_LAUNCH();
    if (B > 0)
    {
        g->d.phin = dalloc<float4>((size_t)B * V);
        if (warp_fill)
        {
            BrickJob job{};
            job.s = sp;
            job.bd = bd;
            job.bricks = B;
            job.ijk = g->d.ijk;
            job.phin = g->d.phin;
            warp.fill(job, status.get(), s);
        }
        else
            tree.visit([&](auto view) {
                k_sparse_fill<<<B, 256, 0, s>>>(view, sp, bd, g->d.ijk, g->d.phin, status.get());
            });
        SDFO_CHECK_LAUNCH();
    }
    g->stats.fill_ms = tm.lap();
    if (B > 0 && p.store_hessian)
    {
        g->d.hess6 = dalloc<float>((size_t)B * V * 6);
        const int64_t stored = (int64_t)B * V;
        k_sparse_hessian<<<(unsigned)((stored + T - 1) / T), T, 0, s>>>(
            sp, bd, g->nb[0], g->nb[1], stored, g->d.ijk, g->d.table, g->d.phin, g->d.hess6);
        SDFO_CHECK_LAUNCH();
    }
    build_stencil_layouts(g.get(), s);
    g->stats.hessian_ms = tm.lap();
    check_status(status, s);
    g->stats.voxels_filled = (int64_t)B * V;
    g->stats.total_ms =
        std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    return g.release();
}

} // namespace sdfo
