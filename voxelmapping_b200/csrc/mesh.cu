// Marching cubes over all allocated blocks, triangle centroids and the dense
// block export.
//
// Reference: src/marching_cubes.cu (select_blocks :25-50, read_sdf_list
// :68-104, interpolateLinear :106-115, make_vertex :117-207, emit loop
// :209-242, compute_surface_point_kernel :314-328). The reference runs 64
// threads per block, looks every cube corner up through the hash table (8
// chain walks per cube) and takes one global atomic per triangle. Here a warp
// turns a block plus its +x/+y/+z halo (9x9x9 voxels, 7 neighbour lookups) into
// bit rows, finds the cubes that cross the surface with bit operations, reserves
// the block's output range with one atomic and emits with one lane per triangle.
#include "vmap_launch.h"
#include "mc_table.inc"

namespace vmapb {

__device__ const unsigned long long kMcTri[256] = VMAP_MC_TRI_PACKED_INIT;

// interpolateLinear: |v| < 1e-6 (a double literal) is |v| <= 1e-6f for floats
__device__ __forceinline__ float mc_interp(float v1, float v2)
{
    if (fabsf(v1) <= 1e-6f) return 0.f;
    if (fabsf(v2) <= 1e-6f) return 1.f;
    if (fabsf(__fsub_rn(v1, v2)) <= 1e-6f) return 0.f;
    return __fdiv_rn(__fsub_rn(0.f, v1), __fsub_rn(v2, v1));
}

constexpr int kHalo = 9;       // 8 voxels + 1 halo layer per axis
constexpr int kMeshWarps = 4;  // warps of a CTA, one block each at a time
constexpr int kMeshList = 512; // triangles a warp emits at a time

// Edge e of a cube (make_vertex, marching_cubes.cu:145-204): places of its two
// corners in the halo cube relative to corner 0's, whether the fraction runs
// back along the axis, the axis, and the other coordinates' offsets. Looked up,
// since a switch over the 12 edges runs each case that a lane of the warp has.
constexpr unsigned mc_edge(int from, int to, bool back, int axis, int ox, int oy, int oz)
{
    constexpr unsigned place[8] = {0, 1, kHalo + 1, kHalo, 81, 82, 81 + kHalo + 1, 81 + kHalo};
    return place[from] | place[to] << 8 | (unsigned)back << 16 | 1u << (17 + axis) | (unsigned)(ox | oy << 1 | oz << 2) << 20;
}
__device__ const unsigned kMcEdge[12] = {
    mc_edge(0, 1, false, 0, 0, 0, 0), mc_edge(1, 2, false, 1, 1, 0, 0), mc_edge(2, 3, true, 0, 0, 1, 0),
    mc_edge(3, 0, true, 1, 0, 0, 0),  mc_edge(4, 5, false, 0, 0, 0, 1), mc_edge(5, 6, false, 1, 1, 0, 1),
    mc_edge(6, 7, true, 0, 0, 1, 1),  mc_edge(7, 4, true, 1, 0, 0, 1),  mc_edge(0, 4, false, 2, 0, 0, 0),
    mc_edge(1, 5, false, 2, 1, 0, 0), mc_edge(2, 6, false, 2, 1, 1, 0), mc_edge(3, 7, false, 2, 0, 1, 0)};

// The vertex on edge `e` (kMcEdge) of the cube at integer voxel coordinates
// (bx, by, bz) with corner 0's TSDF at sdf[0].
__device__ __forceinline__ float3 edge_vertex(unsigned e, const float* sdf, float bx, float by, float bz)
{
    float t = mc_interp(sdf[e & 255u], sdf[e >> 8 & 255u]);
    if (e >> 16 & 1u) t = __fsub_rn(1.f, t);
    return make_float3(__fadd_rn(bx, e >> 17 & 1u ? t : (float)(e >> 20 & 1u)),
                       __fadd_rn(by, e >> 18 & 1u ? t : (float)(e >> 21 & 1u)),
                       __fadd_rn(bz, e >> 19 & 1u ? t : (float)(e >> 22 & 1u)));
}

// One block's extraction by one warp. Its voxels and the halo layer (217 voxels
// of up to 7 neighbours) are read with 23 independent loads a lane; ballots turn
// them into two bits a voxel, observed and inside (TSDF < 0), kept as 9-bit rows
// along x. Whether the 8 cubes of a row are complete and cross the surface is
// then a handful of operations on four rows at once, and only the cubes that do
// (about a tenth) are looked at one by one.
//
// Counting is bound by the reads' latency (99 MB in 51 us), emission by its
// instructions (600 per 32 triangles) and the 180 MB it writes. Against a CTA per
// block that stages 9^3 floats and tests every cube from 8 of them, 23k FP32
// blocks with 2.5 M triangles: counting 155 -> 51 us, emission 369 -> 150 us.
template <int FMT, bool EMIT>
__global__ void __launch_bounds__(32 * kMeshWarps, EMIT ? 7 : 12) mesh_kernel(DevMap m, float* verts, float* norms, unsigned maxTris)
{
    typedef typename Fmt<FMT>::Word Word;
    constexpr unsigned full = 0xffffffffu;
    constexpr int kSdf = EMIT ? kHalo * kHalo * kHalo : 1, kList = EMIT ? kMeshList : 1, kOut = EMIT ? 32 : 1;
    __shared__ unsigned long long s_tab[256];
    __shared__ float s_sdf[kMeshWarps][kSdf];                       // x fastest
    __shared__ unsigned s_ob[kMeshWarps][20], s_in[kMeshWarps][20]; // ballots: rows of the block (16), +y (2), +z (2)
    __shared__ unsigned short s_rob[kMeshWarps][kHalo * kHalo], s_rin[kMeshWarps][kHalo * kHalo];  // rows, y fastest
    __shared__ unsigned short s_list[kMeshWarps][kList];            // cube | triangle << 9
    __shared__ float s_v[kMeshWarps][9 * kOut], s_n[kMeshWarps][3 * kOut];
    __shared__ unsigned s_edge[12];
    for (int i = threadIdx.x; i < 256; i += blockDim.x) s_tab[i] = kMcTri[i];
    if (threadIdx.x < 12) s_edge[threadIdx.x] = kMcEdge[threadIdx.x];
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float* sdf = s_sdf[wid];
    unsigned* obw = s_ob[wid];
    unsigned* inw = s_in[wid];
    unsigned short *rob = s_rob[wid], *rin = s_rin[wid];
    const int n = allocated_blocks(m);
    unsigned counted = 0;
    for (int blk = blockIdx.x * kMeshWarps + wid; blk < n; blk += gridDim.x * kMeshWarps) {
        const int3 bp = unpack_key(m.blockKeys[blk]);
        int nb = blk;  // lane k < 8: the neighbour at (k & 1, k >> 1 & 1, k >> 2 & 1)
        if (lane > 0 && lane < 8) nb = block_find(m, bp.x + (lane & 1), bp.y + (lane >> 1 & 1), bp.z + (lane >> 2));
        // voxel li of neighbour k, whose place in the halo cube is (x, y, z): its two bits
        auto read = [&](int slot, bool on, int li, int x, int y, int z, bool& ob, bool& in) {
            ob = in = false;
            float v = 1.f;
            if (on && slot >= 0) {
                const Word w = ld_map<true>(Layout<FMT>::words(m, slot) + li);
                if (Fmt<FMT>::observed(w)) {
                    ob = true;
                    v = Fmt<FMT>::tsdf(w);
                    in = v < 0.f;
                }
            }
            if constexpr (EMIT) {
                if (on) sdf[(z * kHalo + y) * kHalo + x] = v;
            }
        };
        __syncwarp();  // the last block's rows and values have been used
        bool ob, in;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int li = i * 32 + lane;
            read(blk, true, li, li & 7, li >> 3 & 7, li >> 6, ob, in);
            const unsigned a = __ballot_sync(full, ob), b = __ballot_sync(full, in);
            if (lane == 0) {
                obw[i] = a;
                inw[i] = b;
            }
        }
        const int nx = __shfl_sync(full, nb, 1), ny = __shfl_sync(full, nb, 2), nz = __shfl_sync(full, nb, 4);
        unsigned xob = 0, xin = 0;  // bit j: the +x voxel of row lane + 32 j
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int r = lane + 32 * j;  // row r: y = r & 7, z = r >> 3
            read(nx, true, 8 * r, 8, r & 7, r >> 3, ob, in);
            xob |= (unsigned)ob << j;
            xin |= (unsigned)in << j;
            read(ny, true, 64 * (r >> 3) + (r & 7), r & 7, 8, r >> 3, ob, in);
            const unsigned ya = __ballot_sync(full, ob), yb = __ballot_sync(full, in);
            read(nz, true, r, r & 7, r >> 3, 8, ob, in);
            const unsigned za = __ballot_sync(full, ob), zb = __ballot_sync(full, in);
            if (lane == 0) {
                obw[16 + j] = ya;
                inw[16 + j] = yb;
                obw[18 + j] = za;
                inw[18 + j] = zb;
            }
        }
        // the edges +x+y (lanes 0-7, along z), +x+z (8-15, along y), +y+z (16-23, along x) and the corner (24)
        const int e = lane & 7, kind = lane >> 3;
        const int en = __shfl_sync(full, nb, kind == 0 ? 3 : kind == 1 ? 5 : kind == 2 ? 6 : 7);
        read(en, lane < 25, kind == 0 ? 64 * e : kind == 1 ? 8 * e : e, kind == 2 ? e : 8, kind == 1 ? e : 8, kind == 0 ? e : 8,
             ob, in);
        const unsigned eob = __ballot_sync(full, ob), ein = __ballot_sync(full, in);
        __syncwarp();
        auto byte = [](const unsigned* w, int r) { return w[r >> 2] >> (8 * (r & 3)) & 255u; };
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int r = lane + 32 * j, at = (r >> 3) * kHalo + (r & 7);
            rob[at] = (unsigned short)(byte(obw, r) | (xob >> j & 1u) << 8);
            rin[at] = (unsigned short)(byte(inw, r) | (xin >> j & 1u) << 8);
        }
        if (lane < 16) {  // rows (8, z), then (y, 8)
            const int at = lane < 8 ? lane * kHalo + 8 : 8 * kHalo + lane - 8;
            rob[at] = (unsigned short)(byte(obw + 16, lane) | (eob >> lane & 1u) << 8);
            rin[at] = (unsigned short)(byte(inw + 16, lane) | (ein >> lane & 1u) << 8);
        } else if (lane == 16) {
            rob[8 * kHalo + 8] = (unsigned short)(eob >> 16 & 511u);
            rin[8 * kHalo + 8] = (unsigned short)(ein >> 16 & 511u);
        }
        __syncwarp();
        // cubes of rows lane and lane + 32 that are complete and cross the surface
        unsigned cross[2], rows[2][4];
        unsigned cnt = 0;
        auto cube_case = [](const unsigned* r, int x) {  // corner order (0,0,0),(1,0,0),(1,1,0),(0,1,0), then z + 1
            const unsigned a = r[0] >> x & 3u, b = r[1] >> x & 3u, c = r[2] >> x & 3u, d = r[3] >> x & 3u;
            return a | (b & 2u) << 1 | (b & 1u) << 3 | c << 4 | (d & 2u) << 5 | (d & 1u) << 7;
        };
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int r = lane + 32 * j, at = (r >> 3) * kHalo + (r & 7);
            const unsigned o = rob[at] & rob[at + 1] & rob[at + kHalo] & rob[at + kHalo + 1];
            rows[j][0] = rin[at];
            rows[j][1] = rin[at + 1];
            rows[j][2] = rin[at + kHalo];
            rows[j][3] = rin[at + kHalo + 1];
            const unsigned any = rows[j][0] | rows[j][1] | rows[j][2] | rows[j][3];
            const unsigned all = rows[j][0] & rows[j][1] & rows[j][2] & rows[j][3];
            cross[j] = o & o >> 1 & (any | any >> 1) & ~(all & all >> 1) & 255u;
            for (unsigned c = cross[j]; c; c &= c - 1) cnt += (unsigned)(s_tab[cube_case(rows[j], __ffs(c) - 1)] >> 60);
        }
        if constexpr (!EMIT) {
            counted += cnt;
        } else {
            unsigned first = cnt;  // exclusive scan of the lanes' triangles
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const unsigned v = __shfl_up_sync(full, first, d);
                if (lane >= d) first += v;
            }
            const unsigned total = __shfl_sync(full, first, 31);
            first -= cnt;
            if (total == 0) continue;
            unsigned base = 0;
            if (lane == 0) base = atomicAdd(m.ctr + C_TRI, total);
            base = __shfl_sync(full, base, 0);
            for (unsigned lo = 0; lo < total; lo += kMeshList) {  // the list's triangles [lo, lo + kMeshList)
                unsigned q = first;
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    for (unsigned c = cross[j]; c; c &= c - 1) {
                        const int x = __ffs(c) - 1;
                        const unsigned k = (unsigned)(s_tab[cube_case(rows[j], x)] >> 60);
                        for (unsigned t = 0; t < k; ++t, ++q)
                            if (q - lo < kMeshList) s_list[wid][q - lo] = (unsigned short)((lane + 32 * j) * 8 + x | t << 9);
                    }
                __syncwarp();
                const unsigned here = min(total - lo, (unsigned)kMeshList);
                for (unsigned g = 0; g < here; g += 32) {  // 32 triangles at a time, a lane each
                    const unsigned t0 = base + lo + g;
                    if (t0 >= maxTris) break;
                    const unsigned some = min(min(here - g, 32u), maxTris - t0);
                    if ((unsigned)lane < some) {
                        const unsigned entry = s_list[wid][g + lane];
                        const int cube = entry & 511, k = entry >> 9, x = cube & 7, y = cube >> 3 & 7, z = cube >> 6;
                        const int at = z * kHalo + y, e0 = at * kHalo + x;
                        const unsigned r[4] = {rin[at], rin[at + 1], rin[at + kHalo], rin[at + kHalo + 1]};
                        const unsigned long long code = s_tab[cube_case(r, x)];
                        const float fbx = __int2float_rn(bp.x * 8 + x), fby = __int2float_rn(bp.y * 8 + y),
                                    fbz = __int2float_rn(bp.z * 8 + z);
                        // reversed winding: tri[2] = v[a], tri[1] = v[b], tri[0] = v[c], all * voxel size
                        const unsigned edges = (unsigned)(code >> (12 * k));
                        const float3 va = edge_vertex(s_edge[edges & 15u], sdf + e0, fbx, fby, fbz);
                        const float3 vb = edge_vertex(s_edge[edges >> 4 & 15u], sdf + e0, fbx, fby, fbz);
                        const float3 vc = edge_vertex(s_edge[edges >> 8 & 15u], sdf + e0, fbx, fby, fbz);
                        const float3 t2 = make_float3(__fmul_rn(va.x, m.vs), __fmul_rn(va.y, m.vs), __fmul_rn(va.z, m.vs));
                        const float3 t1 = make_float3(__fmul_rn(vb.x, m.vs), __fmul_rn(vb.y, m.vs), __fmul_rn(vb.z, m.vs));
                        const float3 t0v = make_float3(__fmul_rn(vc.x, m.vs), __fmul_rn(vc.y, m.vs), __fmul_rn(vc.z, m.vs));
                        const float3 nrm = normalized(
                            cross3(make_float3(__fsub_rn(t1.x, t0v.x), __fsub_rn(t1.y, t0v.y), __fsub_rn(t1.z, t0v.z)),
                                   make_float3(__fsub_rn(t2.x, t0v.x), __fsub_rn(t2.y, t0v.y), __fsub_rn(t2.z, t0v.z))));
                        float* o = s_v[wid] + 9 * lane;
                        o[0] = t0v.x; o[1] = t0v.y; o[2] = t0v.z;
                        o[3] = t1.x; o[4] = t1.y; o[5] = t1.z;
                        o[6] = t2.x; o[7] = t2.y; o[8] = t2.z;
                        s_n[wid][3 * lane] = nrm.x;
                        s_n[wid][3 * lane + 1] = nrm.y;
                        s_n[wid][3 * lane + 2] = nrm.z;
                    }
                    __syncwarp();
                    // the 32 triangles leave as whole lines; 9 * 4 stores of single floats at a stride of 36 bytes
                    // wrote every sector 8 times over
                    float* vo = verts + 9 * (size_t)t0;
#pragma unroll
                    for (int i = 0; i < 9; ++i)
                        if (i * 32 + lane < 9 * (int)some) vo[i * 32 + lane] = s_v[wid][i * 32 + lane];
                    if (norms) {
                        float* no = norms + 9 * (size_t)t0;
#pragma unroll
                        for (int i = 0; i < 9; ++i) {
                            const int f = i * 32 + lane, t = f / 9;
                            if (t < (int)some) no[f] = s_n[wid][3 * t + (f - 9 * t) % 3];
                        }
                    }
                    __syncwarp();
                }
            }
        }
    }
    if constexpr (!EMIT) {
        counted = __reduce_add_sync(full, counted);
        if (lane == 0 && counted) atomicAdd(m.ctr + C_TRI, counted);
    }
}

// A pass without an output buffer only counts: it flags nothing.
__global__ void mesh_finish_kernel(DevMap m, unsigned maxTris, unsigned* ntrisOut, bool emitting)
{
    const unsigned n = m.ctr[C_TRI];
    if (emitting && n > maxTris) atomicOr(m.ctr + C_ERR, VMAP_FLAG_BUFFER_FULL);
    if (ntrisOut) *ntrisOut = n;
}

// compute_surface_point_kernel (marching_cubes.cu:314-328): (a + b + c) / 3
__global__ void surface_points_kernel(const float* v, unsigned n, float* pts)
{
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
#pragma unroll
    for (int i = 0; i < 3; ++i)
        pts[3 * (size_t)t + i] =
            __fdiv_rn(__fadd_rn(__fadd_rn(v[9 * (size_t)t + i], v[9 * (size_t)t + 3 + i]), v[9 * (size_t)t + 6 + i]), 3.f);
}

// Dense export of blocks [first, first + count) in pool order.
template <int FMT, bool COLOR>
__global__ void export_kernel(DevMap m, int first, int count, int* coords, float* tsdf, float* weight, uint8_t* rgb)
{
    typedef Layout<FMT> L;
    for (int b = blockIdx.x; b < count; b += gridDim.x) {
        const int slot = first + b;
        if (threadIdx.x == 0) {
            const int3 p = unpack_key(m.blockKeys[slot]);
            coords[3 * b] = p.x;
            coords[3 * b + 1] = p.y;
            coords[3 * b + 2] = p.z;
        }
        for (int i = threadIdx.x; i < kBlockVoxels; i += blockDim.x) {
            const size_t o = (size_t)b * kBlockVoxels + i;
            const typename Fmt<FMT>::Word w = L::words(m, slot)[i];
            tsdf[o] = Fmt<FMT>::tsdf(w);
            weight[o] = Fmt<FMT>::weight(w);
            if constexpr (COLOR) {
                if (rgb) {
                    const unsigned char* c = m.pool + (size_t)slot * m.blockBytes + L::kRgbOff;
                    rgb[3 * o] = c[i];
                    rgb[3 * o + 1] = c[kBlockVoxels + i];
                    rgb[3 * o + 2] = c[2 * kBlockVoxels + i];
                }
            }
        }
    }
}

// A pass with an output buffer emits, one without only counts. The grid is
// l.mesh times 256 threads per SM, at most what is resident: a CTA that waits for
// others to end would start its share of the blocks late.
template <int FMT, bool EMIT>
static void mesh_pass(const DevMap& m, float* verts, float* norms, unsigned maxTris, const Launcher& l, cudaStream_t s)
{
    constexpr int threads = 32 * kMeshWarps;
    static const int fit = [] {
        int o = 0;
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, mesh_kernel<FMT, EMIT>, threads, 0) != cudaSuccess || o < 1 ? 1 : o;
    }();
    const int per_sm = l.mesh * (256 / threads) < fit ? l.mesh * (256 / threads) : fit;
    mesh_kernel<FMT, EMIT><<<stage_grid(l, per_sm), threads, 0, s>>>(m, verts, norms, maxTris);
}

template <int FMT>
static void mesh_format(const DevMap& m, float* verts, float* norms, unsigned maxTris, const Launcher& l, cudaStream_t s)
{
    if (verts) mesh_pass<FMT, true>(m, verts, norms, maxTris, l, s);
    else mesh_pass<FMT, false>(m, verts, norms, maxTris, l, s);
}

cudaError_t launch_mesh(const DevMap& m, int fmt, float* verts, float* norms, unsigned maxTris, unsigned* ntrisOut,
                        const Launcher& l, cudaStream_t s)
{
    cudaError_t e = cudaMemsetAsync(m.ctr + C_TRI, 0, sizeof(unsigned), s);
    if (e != cudaSuccess) return e;
    switch (fmt) {
    case VMAP_VOXEL_REF: mesh_format<VMAP_VOXEL_REF>(m, verts, norms, maxTris, l, s); break;
    case VMAP_VOXEL_F32: mesh_format<VMAP_VOXEL_F32>(m, verts, norms, maxTris, l, s); break;
    case VMAP_VOXEL_F16: mesh_format<VMAP_VOXEL_F16>(m, verts, norms, maxTris, l, s); break;
    case VMAP_VOXEL_I16: mesh_format<VMAP_VOXEL_I16>(m, verts, norms, maxTris, l, s); break;
    default: return cudaErrorInvalidValue;
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    mesh_finish_kernel<<<1, 1, 0, s>>>(m, maxTris, ntrisOut, verts != nullptr);
    return cudaGetLastError();
}

cudaError_t launch_surface_points(const float* verts, unsigned n, float* pts, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    surface_points_kernel<<<(n + 255) / 256, 256, 0, s>>>(verts, n, pts);
    return cudaGetLastError();
}

template <int FMT>
static void export_dispatch(const DevMap& m, bool color, int first, int count, int* coords, float* tsdf,
                            float* weight, uint8_t* rgb, cudaStream_t s)
{
    const int grid = count < 4096 ? count : 4096;
    if (color) export_kernel<FMT, true><<<grid, 256, 0, s>>>(m, first, count, coords, tsdf, weight, rgb);
    else export_kernel<FMT, false><<<grid, 256, 0, s>>>(m, first, count, coords, tsdf, weight, rgb);
}

cudaError_t launch_export(const DevMap& m, int fmt, bool color, int first, int count, int* coords, float* tsdf,
                          float* weight, uint8_t* rgb, cudaStream_t s)
{
    if (count <= 0) return cudaSuccess;
    switch (fmt) {
    case VMAP_VOXEL_REF: export_dispatch<VMAP_VOXEL_REF>(m, color, first, count, coords, tsdf, weight, rgb, s); break;
    case VMAP_VOXEL_F32: export_dispatch<VMAP_VOXEL_F32>(m, color, first, count, coords, tsdf, weight, rgb, s); break;
    case VMAP_VOXEL_F16: export_dispatch<VMAP_VOXEL_F16>(m, color, first, count, coords, tsdf, weight, rgb, s); break;
    case VMAP_VOXEL_I16: export_dispatch<VMAP_VOXEL_I16>(m, color, first, count, coords, tsdf, weight, rgb, s); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace vmapb
