// Fusion path: block allocation along depth rays, visible-block selection and
// the projective TSDF / weight / colour update, for one map or a batch.
//
// Reference: src/depth_fusion.cu (FuseImage :199-301, FuseDepthAndImage
// :383-488, CheckVisibleBlocks :494-539) and the device helpers of
// include/map_struct.h. The reference synchronises the device three times and
// copies the visible count to the host on every fuse; here the three kernels
// run back to back on one stream, over every map of a batch at once, and the
// counts stay in device memory.
#include "stages.cuh"

namespace vmapb {

// ---------------------------------------------------------------- allocation
// A 256-thread CTA per 32 x kStageTileH-pixel tile, kStageTileH / 8 depth
// pixels per thread. The samples of a pixel's band are walked without touching
// global memory: each block a pixel enters is staged in a CTA-wide
// shared-memory set, and once the whole tile has been walked its distinct
// blocks (a few dozen) are looked up in parallel, one thread per block, and the
// missing ones inserted. A warp so waits on one table round trip per tile
// instead of one per sample step, and the block set is the one a per-sample
// insertion gives. The CTA of item 0 also clears the visible counters the next
// kernel accumulates into.
// Bound by instructions (940 per 32 pixels; 1,110 with the walk on conversions,
// IEEE divisions and 64-bit keys): 19.8 -> 16.9 us at 640x480 / 5 mm, 43.6 ->
// 36.2 us at 1280x720 / 4 mm, launch included.
// 8 resident CTAs per SM (at most 32 registers) measured faster than the 6
// that 38 registers allow (20.9 against 22.1 us per 640x480 frame).
constexpr int kTileSet = 1024;  // open-addressed set of one tile's blocks (8 KB), any view
// The set of a near view's tile: 32-bit keys (band_keys) and a list of the
// entries in use, so that neither the insertion nor the clearing visits the
// empty ones. A key that finds no place in kNearProbes goes straight to the
// table.
constexpr int kNearSet = 512, kNearProbes = 16;

__device__ __forceinline__ void near_insert(const DevMap& m, const BandBase& b, unsigned key)
{
    const int x = (int)(key & 1023u) + b.x, y = (int)(key >> 10 & 1023u) + b.y, z = (int)(key >> 20) + b.z;
    // in steady state nearly every block is there already: one read tells
    if (m.grid && block_find<false>(m, x, y, z) >= 0) return;
    hash_insert(m, x, y, z);
}

// Tile `item` of the launch: its view, and this thread's column and first row.
template <class V>
__device__ __forceinline__ const MapView& alloc_tile(const V& views, const int* pre, int item, int& x, int& y0)
{
    const int mi = map_of(pre, views.count(), item);
    const MapView& v = views[mi];
    const int t = item - pre[mi], tx = (v.cam.W + 31) >> 5;
    x = (t % tx) * 32 + (threadIdx.x & 31);
    y0 = (t / tx) * kStageTileH + (threadIdx.x >> 5);
    return v;
}

// Item prefix of the launch; block 0 clears the visible counters.
template <class V>
__device__ __forceinline__ int alloc_prologue(const V& views, int* pre)
{
    map_prefix(views, [](const MapView& v) { return alloc_tiles<kStageTileH>(v); }, pre);  // ends with __syncthreads
    const int nmaps = views.count();
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < nmaps; i += blockDim.x)
            if (views[i].in.active) views[i].m.ctr[C_VISIBLE] = 0u;
    return pre[nmaps];
}

template <class V>
__global__ void __launch_bounds__(256, 8) alloc_kernel(V views)
{
    stage_entry();
    __shared__ int pre[kMaxBatch + 1];
    __shared__ unsigned set[kNearSet];
    __shared__ unsigned short used[kNearSet];
    __shared__ int nused;
    for (int i = threadIdx.x; i < kNearSet; i += blockDim.x) set[i] = ~0u;
    if (threadIdx.x == 0) nused = 0;
    const int total = alloc_prologue(views, pre);
    for (int item = blockIdx.x; item < total; item += gridDim.x) {
        int x, y0;
        const MapView& v = alloc_tile(views, pre, item, x, y0);
        const BandBase base = band_base(v);
#pragma unroll 1
        for (int y = y0; y < y0 + kStageTileH; y += 8) {
            const float d = x < v.cam.W && y < v.cam.H ? read_depth(v.in, x, y) : __int_as_float(0x7fffffff);
            band_keys(v, base, x, y, d, threadIdx.x & 31, [&](unsigned key) {
                unsigned h = (key * 0x9E3779B1u) >> (32 - ilog2(kNearSet));
#pragma unroll 1
                for (int p = 0; p < kNearProbes; ++p) {
                    unsigned cur = *(volatile unsigned*)(set + h);
                    if (cur == ~0u) {
                        cur = atomicCAS(set + h, ~0u, key);
                        if (cur == ~0u) {
                            used[atomicAdd(&nused, 1)] = (unsigned short)h;
                            return;
                        }
                    }
                    if (cur == key) return;
                    h = (h + 1) & (kNearSet - 1);
                }
                near_insert(v.m, base, key);
            });
        }
        __syncthreads();
        const int n = nused;
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const int h = used[i];
            near_insert(v.m, base, set[h]);
            set[h] = ~0u;
        }
        __syncthreads();
        if (threadIdx.x == 0) nused = 0;
        __syncthreads();
    }
}

// The same for launches with a view that is not near (CamParams::near: voxels
// finer than 1.2 to 1.5 mm by the camera's angle, or a camera 2^20 voxels from the
// origin): the general walk and 64-bit keys. 18.9 us for a 640x480 frame at 1.2
// mm, 12.2 at 320x240; the one kernel that there was for all views took 17.5 and
// 12.1 and entered no blocks into a grid, which the whole frames gain by (118 ->
// 92 us, 103 -> 71). 8 CTAs per SM (32 registers) take 18.0 us but 1.2 us more
// of the 320x240 frame.
template <class V>
__global__ void __launch_bounds__(256, 6) far_alloc(V views)
{
    stage_entry();
    __shared__ int pre[kMaxBatch + 1];
    __shared__ unsigned long long set[kTileSet];
    for (int i = threadIdx.x; i < kTileSet; i += blockDim.x) set[i] = kEmptyKey;
    const int total = alloc_prologue(views, pre);
    for (int item = blockIdx.x; item < total; item += gridDim.x) {
        int x, y0;
        const MapView& v = alloc_tile(views, pre, item, x, y0);
#pragma unroll 1
        for (int y = y0; y < y0 + kStageTileH; y += 8)
            if (x < v.cam.W && y < v.cam.H)
                band_blocks(v, x, y, [&](unsigned long long key, int bx, int by, int bz) {
                    stage_block<kTileSet>(set, v.m, key, bx, by, bz);
                });
        __syncthreads();
        insert_staged<kTileSet>(set, v.m, threadIdx.x, blockDim.x);
        __syncthreads();
    }
}

// ---------------------------------------------------------------- visibility
// CheckEntryVisibilityFunctor without the full hash-table scan: allocated
// blocks are dense in pool order, so only min(alloc, capacity) 8-byte keys
// are read. Work items are 32-block groups of one map, one per warp. The
// map's visible counter must be zero on entry (cleared by alloc_kernel or the
// host).
template <class V>
__global__ void __launch_bounds__(256) visibility_kernel(V views)
{
    stage_entry();
    __shared__ int pre[kMaxBatch + 1];
    map_prefix(views, [](const MapView& v) { return v.in.active ? (allocated_blocks(v.m) + 31) >> 5 : 0; }, pre);
    const int nmaps = views.count();
    const int total = pre[nmaps];
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int w = warp; w < total; w += nwarps) {
        const int mi = map_of(pre, nmaps, w);
        visibility_group(views[mi], w - pre[mi], threadIdx.x & 31);
    }
}

// ----------------------------------------------------------------- fusion
// Bound by instructions and, once these are done, by the bytes of the updated
// voxels (2.4 TB/s of DRAM traffic at 22k visible blocks). Projecting with one
// reciprocal per voxel, packed divisions and no conversion instructions took it
// from 199 to 123 instructions per voxel: 49 -> 42.5 us at 640x480 / 5 mm and
// 172 -> 137 us at 1280x720 / 4 mm (45k visible blocks), launch included; a
// pixel's range checked by one unsigned comparison and unsigned addresses to
// 41.4 and 130 us. Prefetching the voxel words, or the next block's, into L2
// changes nothing or costs up to 7 us: the loads' latency is not what bounds it.
// Several maps: the view's fields are loaded and take registers, and reading a
// pixel's colour in two loads instead of three spills less (4 to 28 B instead
// of 28 to 108) and is faster, 2699 -> 2668 us for a step of 32 maps at 640x480
// with their rendering; for one map it is slower (FP16 at 1280x720: 130 -> 140).
// A team of 512 / kFuseVoxels threads per visible block, kFuseVoxels voxels
// of an x-row per thread; 256 / team blocks per CTA, grid-stride over the
// visible blocks of all maps. 6 resident CTAs per SM (at most 40 registers)
// measured faster than the 5 that 48 registers allow (56.9 against 59.4 us
// at 22.7k visible blocks) and than 8 voxels per thread at 4 CTAs per SM.
constexpr int kFuseVoxels = 4;
constexpr int kFuseTeam = kBlockVoxels / kFuseVoxels;

template <class V, int FMT>
__global__ void __launch_bounds__(256, 6) fuse_kernel(V views)
{
    stage_entry();
    __shared__ int pre[kMaxBatch + 1];
    map_prefix(views, [](const MapView& v) { return v.in.active ? (int)v.m.ctr[C_VISIBLE] : 0; }, pre);
    const int nmaps = views.count();
    const int total = pre[nmaps];
    constexpr int teams = 256 / kFuseTeam;
    const int team = threadIdx.x / kFuseTeam;
    const int v0 = (threadIdx.x % kFuseTeam) * kFuseVoxels;  // first voxel index of this thread
    for (int i = blockIdx.x * teams + team; i < total; i += gridDim.x * teams) {
        const int mi = map_of(pre, nmaps, i);
        const MapView& v = views[mi];
        fuse_voxels<FMT, kFuseVoxels, V::kMany>(v, v.m.visList[i - pre[mi]], v0);
    }
}

// ------------------------------------------------------------------- reset
// MapStruct::reset (map_struct.cu:29-42): empty hash slots and grid, zeroed voxels. A
// pool block is written only after it has been handed out, so only the
// allocated blocks hold anything to clear (all of them after a snapshot load
// that stopped half-way). Bound by the bytes it writes: emptying a 2^20-block
// FP32 + colour map (5.9 GB pool, 62 MB hash table and grid) that holds 8k blocks,
// fusing a frame and rendering it went from 958 us, with the whole pool cleared
// each time, to 166 (153 with the later steps in the other kernels).
__global__ void __launch_bounds__(256) reset_kernel(DevMap m, bool whole)
{
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x, nt = (size_t)gridDim.x * blockDim.x;
    const bool unknown = whole || m.ctr[C_UNKNOWN];
    index_clear(m, unknown, unknown ? 0 : allocated_blocks(m), t, nt);
    if (whole) return;  // the host clears the pool
    // block bytes are a multiple of 16 in every format, and the pool is 256-byte aligned
    const size_t blocks = unknown ? (size_t)m.capacity : (size_t)allocated_blocks(m);
    const size_t words = blocks * (size_t)m.blockBytes / sizeof(uint4);
    uint4* w = reinterpret_cast<uint4*>(m.pool);
    // What L2 holds is written at a fixed stride, in even shares (8,192 blocks of
    // 5,632 B: 28.3 us against 30.5 by chunks). More goes in chunks of 32 KB handed
    // out in the order of their addresses: at a fixed stride the CTAs drift apart
    // and DRAM is slower (2^18 blocks, 1.48 GB: 222 us against 267; 2^15 blocks 46
    // against 49). Every chunk is followed by one take, so the queue's word wraps
    // to zero with the last one.
    if (words < (size_t)(120 << 20) / sizeof(uint4)) {
        for (size_t i = t; i < words; i += nt) w[i] = make_uint4(0u, 0u, 0u, 0u);
        return;
    }
    constexpr int kChunk = 8 * 256;
    const unsigned chunks = (unsigned)((words + kChunk - 1) / kChunk);
    __shared__ unsigned s_next;
    for (unsigned c = blockIdx.x; c < chunks;) {
        if (threadIdx.x == 0) s_next = gridDim.x + atomicInc(m.ctr + C_CLEARQ, chunks - 1);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const size_t i = (size_t)c * kChunk + k * 256 + threadIdx.x;
            if (i < words) w[i] = make_uint4(0u, 0u, 0u, 0u);
        }
        __syncthreads();
        c = s_next;
        __syncthreads();
    }
}

// ------------------------------------------------------------------ launchers
template <class V>
cudaError_t launch_alloc(const V& views, int totalTiles, bool near, const Launcher& l, cudaStream_t s)
{
    return launch_stage<V>(near ? alloc_kernel<V> : far_alloc<V>, stage_grid(l, l.alloc, totalTiles), 256, s, views);
}

template <class V>
cudaError_t launch_visibility(const V& views, const Launcher& l, cudaStream_t s)
{
    return launch_stage<V>(visibility_kernel<V>, stage_grid(l, l.visibility), 256, s, views);
}

template <class V>
cudaError_t launch_fuse(const V& views, int fmt, const Launcher& l, cudaStream_t s)
{
    const int grid = stage_grid(l, l.fuse);
    switch (fmt) {
    case VMAP_VOXEL_REF: return launch_stage<V>(fuse_kernel<V, VMAP_VOXEL_REF>, grid, 256, s, views);
    case VMAP_VOXEL_F32: return launch_stage<V>(fuse_kernel<V, VMAP_VOXEL_F32>, grid, 256, s, views);
    case VMAP_VOXEL_F16: return launch_stage<V>(fuse_kernel<V, VMAP_VOXEL_F16>, grid, 256, s, views);
    case VMAP_VOXEL_I16: return launch_stage<V>(fuse_kernel<V, VMAP_VOXEL_I16>, grid, 256, s, views);
    default: return cudaErrorInvalidValue;
    }
}

template cudaError_t launch_alloc<OneView>(const OneView&, int, bool, const Launcher&, cudaStream_t);
template cudaError_t launch_alloc<ManyViews>(const ManyViews&, int, bool, const Launcher&, cudaStream_t);
template cudaError_t launch_visibility<OneView>(const OneView&, const Launcher&, cudaStream_t);
template cudaError_t launch_visibility<ManyViews>(const ManyViews&, const Launcher&, cudaStream_t);
template cudaError_t launch_fuse<OneView>(const OneView&, int, const Launcher&, cudaStream_t);
template cudaError_t launch_fuse<ManyViews>(const ManyViews&, int, const Launcher&, cudaStream_t);

// `whole`: the map's memory may hold anything (a new map), so the counters do
// not tell what to clear.
cudaError_t launch_reset(const DevMap& m, bool whole, const Launcher& l, cudaStream_t s)
{
    reset_kernel<<<l.numSMs * 8, 256, 0, s>>>(m, whole);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess && whole) e = cudaMemsetAsync(m.pool, 0, (size_t)m.capacity * m.blockBytes, s);
    if (e != cudaSuccess) return e;
    return cudaMemsetAsync(m.ctr, 0, C_COUNT * sizeof(unsigned), s);
}

}  // namespace vmapb
