// Ray marching (MapRenderingDelegate, src/ray_tracing.cu:255-401) for one map
// or a batch.
//
// Every ray follows the reference's sample sequence: start at z = 0.1 m (or,
// with z-range tiles, at the last 1-voxel step before the tile's nearest
// allocated block), SDF-proportional steps near surfaces, one-voxel steps
// where a sample is unobserved, trilinear interpolation within 0.5 of the
// surface, two refinement steps after the zero crossing. Work that cannot
// change the result is skipped:
//   * inside an unallocated block, where the reference reads "invalid, 1.0"
//     and steps one voxel at a time, the steps up to the block's exit are
//     taken as one integer jump; before the tile's nearest allocated block
//     these jumps need no lookup and are taken when the ray starts;
//   * whole empty cubes of blocks are recognised from the block grid's
//     occupancy words, so that the jumps inside one need no lookup either;
//   * the trilinear corners of all rays of a warp are read together, whether
//     they lie in one block or two.
// What bounds it: the instructions and branches (at 640x480 the kernel issues
// 70 % of the time while all its warps run) and, in scenes seen at grazing
// angles, the slowest tiles' latency. Against a lookup per block through a
// warp-shared cache and the hash table, event time of the launch, three rooms
// each: 48 -> 26 us at 160x120 / 16 mm, 63 -> 32 at 320x240 / 8 mm, 96 -> 58 at
// 640x480 / 5 mm, 293 -> 208 at 1280x720 / 4 mm, 97 -> 50 a view at 517x389,
// 320 -> 108 for an 800x600 full march (raycast_mode 1).
//
// Scheduling: the kernel is persistent. Each warp takes 8x4-pixel tiles from
// one device-side queue shared by every map of the batch until it runs dry.
// A map's tiles are handed out in a selectable order, alternating from both
// ends of the image by default (tile_at).
// (Refilling lanes from a larger group as their rays finish was measured
// 2.8x slower: lanes at different depths scatter their loads and lookups.)
#include "march.cuh"

namespace vmapb {

template <class V, int FMT, bool WIDE>
__device__ __forceinline__ void raycast_tiles(const V& views, int order, int tw)
{
    stage_entry();
    __shared__ int pre[kMaxBatch + 1];
    map_prefix(views, [tw](const MapView& v) { return ray_tiles(v, tw); }, pre);
    // the z-range pass before this launch linked every allocated block of the
    // maps it renders
    if (blockIdx.x == 0 && threadIdx.x == 0)
        for (int mi = 0; mi < views.count(); ++mi)
            if (views[mi].out.vmap) views[mi].m.ctr[C_LINKED] = (unsigned)allocated_blocks(views[mi].m);
    const int nmaps = views.count();
    const int total = pre[nmaps];
    const int lane = threadIdx.x & 31;
    // a warp's first tile is its own number (consecutive tiles on different
    // SMs), the others come from the queue
    const int warps = (int)(gridDim.x * (blockDim.x >> 5));
    int item = (int)((threadIdx.x >> 5) * gridDim.x + blockIdx.x);
    while (item < total) {
        const int mi = map_of(pre, nmaps, item);
        march_tile<FMT, true, WIDE>(views[mi], item - pre[mi], pre[mi + 1] - pre[mi], order, tw, lane);
        if (lane == 0) item = warps + (int)atomicAdd(views.queue, 1u);
        item = __shfl_sync(0xffffffffu, item, 0);
    }
}

// 4 CTAs per SM (at most 64 registers) measured faster than the 3 that 76
// registers allow: latency hiding outweighs a small register spill.
template <class V, int FMT>
__global__ void __launch_bounds__(256, 4) raycast_kernel(const __grid_constant__ V views, int order, int tw)
{
    raycast_tiles<V, FMT, false>(views, order, tw);
}

// The same for launches with a view whose rays leave the narrow range, at the 3
// CTAs per SM that its 70-77 registers allow. A room 3 km from the origin, 640x480
// / 5 mm: 73 us (55 at the origin, narrow; 83 with a lookup per block through a
// warp-shared cache and the hash table); 320x240 / 8 mm at 9 km 51 us (82), 58 a
// view at 517x389 (80), 232 for an 800x600 full march (373).
template <class V, int FMT>
__global__ void __launch_bounds__(256, 3) march_wide_kernel(const __grid_constant__ V views, int order, int tw)
{
    raycast_tiles<V, FMT, true>(views, order, tw);
}

template <class V, int FMT, bool WIDE>
static cudaError_t raycast_persistent(const V& views, const Launcher& l, cudaStream_t s)
{
    static void (*const kernel)(const V, int, int) = WIDE ? march_wide_kernel<V, FMT> : raycast_kernel<V, FMT>;
    // resident CTAs per SM of this instantiation at 128 and 256 threads (a
    // static initialiser runs once, thread-safely, on the first launch)
    auto fits = [](int threads) {
        int o = 0;
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, kernel, threads, 0) != cudaSuccess || o < 1 ? 1 : o;
    };
    static const int occ[2] = {fits(128), fits(256)};
    const int threads = l.rayThreads == 128 ? 128 : 256;
    const int fit = occ[threads == 256];
    // CTAs beyond those resident would only start once others finish: cap at occupancy
    const int per_sm = l.raycast > 0 && l.raycast < fit ? l.raycast : fit;
    return launch_stage<V>(kernel, stage_grid(l, per_sm), threads, s, views, l.tileOrder, l.tileW);
}

template <class V, int FMT>
static cudaError_t raycast_format(const V& views, bool wide, const Launcher& l, cudaStream_t s)
{
    return wide ? raycast_persistent<V, FMT, true>(views, l, s) : raycast_persistent<V, FMT, false>(views, l, s);
}

template <class V>
cudaError_t launch_raycast(const V& views, int fmt, bool wide, const Launcher& l, cudaStream_t s)
{
    switch (fmt) {
    case VMAP_VOXEL_REF: return raycast_format<V, VMAP_VOXEL_REF>(views, wide, l, s);
    case VMAP_VOXEL_F32: return raycast_format<V, VMAP_VOXEL_F32>(views, wide, l, s);
    case VMAP_VOXEL_F16: return raycast_format<V, VMAP_VOXEL_F16>(views, wide, l, s);
    case VMAP_VOXEL_I16: return raycast_format<V, VMAP_VOXEL_I16>(views, wide, l, s);
    default: return cudaErrorInvalidValue;
    }
}

template cudaError_t launch_raycast<OneView>(const OneView&, int, bool, const Launcher&, cudaStream_t);
template cudaError_t launch_raycast<ManyViews>(const ManyViews&, int, bool, const Launcher&, cudaStream_t);

}  // namespace vmapb
