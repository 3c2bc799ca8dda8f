// Ray marcher device code (MapRenderingDelegate, src/ray_tracing.cu:255-401)
// shared by the ray-marching kernel and the persistent batch step: per-ray
// state, the sample loop and one warp's tile.
#pragma once

#include "vmap_launch.h"

namespace vmapb {

// A warp marches one tile of 32 neighbouring rays (tw x 32/tw pixels, 8 x 4
// by default): neighbouring rays sample neighbouring voxels at similar
// depths, so a warp's loads and hash lookups share sectors.
__device__ __forceinline__ int ray_tiles(const MapView& v, int tw)
{
    const int th = 32 / tw;
    return v.out.vmap ? ((v.cam.W + tw - 1) / tw) * ((v.cam.H + th - 1) / th) : 0;
}

__device__ __forceinline__ float3 fma3(float k, float3 d, float3 r)
{
    return make_float3(__fmaf_rn(k, d.x, r.x), __fmaf_rn(k, d.y, r.y), __fmaf_rn(k, d.z, r.z));
}

// Per-lane state of one ray. cx, cy, cz: floor codes (March::fl) of a voxel in
// the region that the last lookup settled: the aligned cube of side cmask + 1
// voxels, 8 (one block) with its slot in cblk, or 8, 32 or 128 that hold no
// allocated block (cblk -1).
struct Ray {
    int x, y;
    float3 res, dir, inv;
    float dist_s, dist_lim;
    float sdf;
    bool valid;
    int cx, cy, cz, cmask, cblk;
};

// WIDE: some ray of the view may leave the narrow range (narrow_limit, set per
// view by the host from the image corners). Otherwise a floor is one full-rate add,
// rounded down, of 1.5 * 2^23: the low 22 bits of the sum are floor(p), and
// subtracting the constant again gives it as a float, both exact below 2^22.
// The conversion instructions that do the same run at a quarter of the rate or
// less, and a trilinear sample needs a dozen of them.
template <int FMT, bool NC, bool WIDE>
struct March {
    typedef Fmt<FMT> F;
    typedef typename F::Word Word;
    static constexpr float kFloorAdd = 12582912.f;  // 1.5 * 2^23

    // floor(p) as an integer code: equal in the low 22 bits, differences exact
    static __device__ __forceinline__ int fl(float p)
    {
        if constexpr (WIDE) return __float2int_rd(p);
        else return __float_as_int(__fadd_rd(p, kFloorAdd));
    }
    // the code as a float
    static __device__ __forceinline__ float ff(int i)
    {
        if constexpr (WIDE) return __int2float_rn(i);
        else return __fsub_rn(__int_as_float(i), kFloorAdd);
    }
    // voxel index in its block
    static __device__ __forceinline__ int at(int ix, int iy, int iz) { return local_idx(ix, iy, iz); }

    // read_sdf (ray_tracing.cu:272-286) on a loaded word
    static __device__ __forceinline__ float value(Word w, bool& valid)
    {
        valid = F::observed(w);
        return valid ? F::tsdf(w) : 1.f;
    }

    static __device__ __forceinline__ float voxel(const DevMap& m, int slot, int ix, int iy, int iz, bool& valid)
    {
        if (slot >= 0) return value(ld_map<NC>(Layout<FMT>::words(m, slot) + at(ix, iy, iz)), valid);
        valid = false;
        return 1.f;
    }

    // Block coordinates of a floor code. Narrow codes themselves agree with
    // the coordinates in the bits that the grid's cells and tags use.
    static __device__ __forceinline__ int block(int i)
    {
        if constexpr (WIDE) return i >> 3;
        else return (i >> 3) - (__builtin_bit_cast(int, kFloorAdd) >> 3);
    }
    // Slot that grid entry e gives the block of floor codes (ix, iy, iz), -1: absent.
    static __device__ __forceinline__ int slot_of(const DevMap& m, unsigned long long e, int ix, int iy, int iz)
    {
        const int bx = ix >> 3, by = iy >> 3, bz = iz >> 3;
        const unsigned hi = (unsigned)(e >> 32), tag = WIDE ? grid_tag(m, bx, by, bz) : grid_tag_bits(m, bx, by, bz);
        if ((!WIDE || tag) && (hi & ~kGridShared) == tag) return (int)(unsigned)e;
        return hi & kGridShared ? hash_find<NC>(m, block(ix), block(iy), block(iz)) : -1;
    }
    // Slot of the block of floor codes (ix, iy, iz).
    static __device__ __forceinline__ int find(const DevMap& m, int ix, int iy, int iz)
    {
        if (WIDE && !m.grid) return hash_find<NC>(m, ix >> 3, iy >> 3, iz >> 3);
        return slot_of(m, ld_map<NC>(grid_cell(m, grid_brick8(m, ix, iy, iz), grid_bit8(ix, iy, iz))), ix, iy, iz);
    }

    // read_sdf_interped (ray_tracing.cu:288-321): corners floor(p + {0,1}^3),
    // x fastest; lerps contracted as fma((1 - a), s0, a * s1).
    static __device__ __forceinline__ float lerp8(const float* s, float ax, float ay, float az)
    {
        const float bx = __fsub_rn(1.f, ax), by = __fsub_rn(1.f, ay), bz = __fsub_rn(1.f, az);
        const float r0 = __fmaf_rn(bx, s[0], __fmul_rn(ax, s[1]));
        const float r1 = __fmaf_rn(bx, s[2], __fmul_rn(ax, s[3]));
        const float r2 = __fmaf_rn(by, r0, __fmul_rn(ay, r1));
        const float r4 = __fmaf_rn(bx, s[4], __fmul_rn(ax, s[5]));
        const float r5 = __fmaf_rn(bx, s[6], __fmul_rn(ax, s[7]));
        const float r3 = __fmaf_rn(by, r4, __fmul_rn(ay, r5));
        return __fmaf_rn(bz, r2, __fmul_rn(az, r3));
    }

    // Corners of a trilinear read: fractions and the floor codes of p and p + 1.
    struct Corners {
        float ax, ay, az;
        int x0, y0, z0, x1, y1, z1;
        // axes on which corner 1 lies in another block than corner 0 (bits
        // 0-2): the voxels are 1 or 2 apart, so bit 3 tells
        __device__ __forceinline__ int cross() const
        {
            return ((x0 ^ x1) >> 3 & 1) | ((y0 ^ y1) >> 2 & 2) | ((z0 ^ z1) >> 1 & 4);
        }
    };

    static __device__ __forceinline__ Corners corners(float3 p, int ix, int iy, int iz)
    {
        Corners c;
        c.x0 = ix;
        c.y0 = iy;
        c.z0 = iz;
        c.ax = __fsub_rn(p.x, ff(ix));
        c.ay = __fsub_rn(p.y, ff(iy));
        c.az = __fsub_rn(p.z, ff(iz));
        c.x1 = fl(__fadd_rn(p.x, 1.f));
        c.y1 = fl(__fadd_rn(p.y, 1.f));
        c.z1 = fl(__fadd_rn(p.z, 1.f));
        return c;
    }

    // Slot of the block of the farthest corner, past every axis on which the
    // corners leave corner 0's block `slot` (not for all three; `slot` itself
    // when they do not leave it): read together with the sample, so that the
    // corners' own reads need not wait for it and the other links of the block
    // are at hand.
    static __device__ __forceinline__ int far_slot(const DevMap& m, int slot, int cross)
    {
        return cross && cross < 7 ? ld_map<NC>(m.nbr + (6 * (size_t)slot + cross - 1)) : slot;
    }

    // Whether all 8 words are observed, by their smallest weight: the weight is
    // a word's float, or its high bits.
    static __device__ __forceinline__ bool all_observed(Word w0, Word w1, Word w2, Word w3, Word w4, Word w5, Word w6, Word w7)
    {
        if constexpr (sizeof(Word) == 8) {
            return fminf(fminf(fminf(w0.y, w1.y), fminf(w2.y, w3.y)), fminf(fminf(w4.y, w5.y), fminf(w6.y, w7.y))) > 0.f;
        } else {
            return min(min(min(w0, w1), min(w2, w3)), min(min(w4, w5), min(w6, w7))) >= 0x10000u;
        }
    }

    // Values of the 8 corners of c, all observed or not, from corner 0's block
    // `slot` (allocated), its far block and, for corners that leave it on
    // several axes, its forward neighbour links. w0: corner 0's word.
    //
    // Where at most one axis leaves the block, corner k's address is corner
    // 0's plus one byte offset per axis, whether that axis steps inside the
    // block or into the far one, so every lane of the warp issues the same 7
    // independent loads, where a branch per block layout took a round trip to
    // L2 each. floor(p + 1) is floor(p) + 1 or + 2, hence the general in-block
    // offsets. (All 8 corners read with every sample, to save the round trip
    // after it, measured 15-25 % slower: at full size instructions bound it.)
    static __device__ __forceinline__ bool corners8(const DevMap& m, int slot, int far, int cross, const Corners& c, Word w0,
                                                    float* s)
    {
        Word w[8];
        w[0] = w0;
        if (cross == 0 || cross == 1 || cross == 2 || cross == 4) {
            const bool gone = far < 0;  // the far corners' block is not allocated
            const long long hop = gone ? 0ll : (long long)(far - slot) * m.blockBytes;
            const char* a = reinterpret_cast<const char*>(Layout<FMT>::words(m, slot) + at(c.x0, c.y0, c.z0));
            const char* ax = a + ((c.x1 & 7) - (c.x0 & 7)) * (int)sizeof(Word) + (cross == 1 ? hop : 0ll);
            const long long dy = ((c.y1 & 7) - (c.y0 & 7)) * 8 * (int)sizeof(Word) + (cross == 2 ? hop : 0ll);
            const long long dz = ((c.z1 & 7) - (c.z0 & 7)) * 64 * (int)sizeof(Word) + (cross == 4 ? hop : 0ll);
            auto ld = [](const char* p) { return ld_map<NC>(reinterpret_cast<const Word*>(p)); };
            w[1] = ld(ax);
            w[2] = ld(a + dy);
            w[3] = ld(ax + dy);
            w[4] = ld(a + dz);
            w[5] = ld(ax + dz);
            w[6] = ld(a + dy + dz);
            w[7] = ld(ax + dy + dz);
            if (gone) {
#pragma unroll
                for (int k = 1; k < 8; ++k)
                    if (k & cross) w[k] = Word();
            }
        } else {
            // several axes: independent links, then independent corners, with
            // no branch a corner (each had two, run by some lane of half of
            // the warp's iterations); corners without a block read corner 0
            const int* L = m.nbr + 6 * (size_t)slot;
            int to[8];
#pragma unroll
            for (int k = 1; k < 8; ++k) {
                const int o = k & cross;  // corner k's block, as an offset from corner 0's
                const int link = ld_map<NC>(L + (o && o < 7 ? o - 1 : 0));
                to[k] = o == cross ? far : o ? link : slot;
            }
            if (cross == 7) to[7] = find(m, c.x1, c.y1, c.z1);  // no link to the far one on all axes
#pragma unroll
            for (int k = 1; k < 8; ++k) {
                const int vx = (k & 1) ? c.x1 : c.x0, vy = (k & 2) ? c.y1 : c.y0, vz = (k & 4) ? c.z1 : c.z0;
                w[k] = ld_map<NC>(Layout<FMT>::words(m, to[k] < 0 ? slot : to[k]) + at(vx, vy, vz));
                if (to[k] < 0) w[k] = Word();
            }
        }
        if (all_observed(w[0], w[1], w[2], w[3], w[4], w[5], w[6], w[7])) {  // most reads
#pragma unroll
            for (int k = 0; k < 8; ++k) s[k] = F::tsdf(w[k]);
            return true;
        }
        bool v;
#pragma unroll
        for (int k = 0; k < 8; ++k) s[k] = value(w[k], v);
        return false;
    }

    // Every 1-voxel step inside the unallocated block (bx, by, bz) reads
    // (1.0, invalid): jump to the first step past the block's exit (at least
    // one step). Exit faces: +8 where the ray runs up (and +0), +0 where it
    // runs down (and -0), so a zero component gives an infinite distance.
    // One multiply-add, rounded down, gives a coordinate's block in the narrow
    // form and a second one its exit face (both exact), so that a jump is some
    // 20 multiply-adds and 4 operations of the half-rate ALU, which bounds this
    // loop: with the faces from the integer codes it took 22 of them.
    static __device__ __forceinline__ void empty_jump(Ray& r)
    {
        auto face = [](float p, float d) {
            if constexpr (WIDE) return __int2float_rn((fl(p) & ~7) + (signbit(d) ? 0 : 8));
            else return __fmaf_rn(__fmaf_rd(p, 0.125f, kFloorAdd), 8.f, (signbit(d) ? 0.f : 8.f) - 8.f * kFloorAdd);
        };
        const float tx = __fmul_rn(__fsub_rn(face(r.res.x, r.dir.x), r.res.x), r.inv.x);
        const float ty = __fmul_rn(__fsub_rn(face(r.res.y, r.dir.y), r.res.y), r.inv.y);
        const float tz = __fmul_rn(__fsub_rn(face(r.res.z, r.dir.z), r.res.z), r.inv.z);
        const float t = fminf(fminf(tx, ty), tz);  // fminf drops the NaN of 0 * inf
        float up;
        if constexpr (WIDE) up = ceilf(t - 1e-3f);
        else up = __fsub_rn(__fadd_ru(__fsub_rn(t, 1e-3f), kFloorAdd), kFloorAdd);  // the same, t < 2^22
        const float k = fmaxf(1.f, up);
        r.res = fma3(k, r.dir, r.res);
        r.dist_s = __fadd_rn(r.dist_s, k);
    }

    // normalized(), with one reciprocal for its three divisions.
    static __device__ __forceinline__ float3 direction(float3 v)
    {
        const float s = __fmaf_rn(v.x, v.x, __fmaf_rn(v.z, v.z, __fmul_rn(v.y, v.y)));
        if (s > 0.f) {
            const float n = __fsqrt_rn(s), y = rcp_newton(n);
            v = make_float3(div_exact(v.x, n, y), div_exact(v.y, n, y), div_exact(v.z, n, y));
        }
        return v;
    }

    // Start a ray at pixel (x, y); false when it finishes at once (tile with
    // no allocated block: written as a miss).
    static __device__ __forceinline__ bool init(const MapView& v, Ray& r, int x, int y)
    {
        const RenderOut& o = v.out;
        const CamParams& c = v.cam;
        float zn = 0.f, zf = kMaxDepth;
        if (o.mode == 0) {
            const int t = (y >> 3) * o.tilesX + (x >> 3);
            const unsigned long long kn = ld_map<NC>(o.zmin + t), kf = ld_map<NC>(o.zmax + t);
            if ((unsigned)(kn >> 32) != ~o.epoch || (unsigned)(kf >> 32) != o.epoch) {
                const float qnan = __int_as_float(0x7fffffff);
                *(reinterpret_cast<float4*>(reinterpret_cast<char*>(o.vmap) + (size_t)y * o.vpitch) + x) =
                    make_float4(qnan, qnan, qnan, qnan);
                return false;
            }
            zn = __uint_as_float((unsigned)kn);
            zf = __uint_as_float((unsigned)kf);
        }
        const float3 p0 = unproject(x, y, kMinDepth, c.ifx, c.ify, c.cx, c.cy);
        const float dist0 = __fmul_rn(__fsqrt_rn(sqnorm(p0)), o.vsinv);
        float3 bs = xf_apply(v.T, p0.x, p0.y, p0.z);
        bs = make_float3(__fmul_rn(bs.x, o.vsinv), __fmul_rn(bs.y, o.vsinv), __fmul_rn(bs.z, o.vsinv));
        const float3 p1 = unproject(x, y, kMaxDepth, c.ifx, c.ify, c.cx, c.cy);
        const float dist_e = __fmul_rn(__fsqrt_rn(sqnorm(p1)), o.vsinv);
        float3 be = xf_apply(v.T, p1.x, p1.y, p1.z);
        be = make_float3(__fmul_rn(be.x, o.vsinv), __fmul_rn(be.y, o.vsinv), __fmul_rn(be.z, o.vsinv));
        r.dir = direction(make_float3(__fsub_rn(be.x, bs.x), __fsub_rn(be.y, bs.y), __fsub_rn(be.z, bs.z)));
        // reciprocals only bound the empty-block jump (taken with a 1e-3 margin):
        // approximate ones suffice; 1/(+-0) stays +-inf
        r.inv = make_float3(__fdividef(1.f, r.dir.x), __fdividef(1.f, r.dir.y), __fdividef(1.f, r.dir.z));
        r.res = bs;
        r.dist_s = dist0;
        r.dist_lim = dist_e;
        if (o.mode == 0) {
            // ray length (voxels) is proportional to camera depth along a ray
            const float g = div_exact(dist_e, kMaxDepth, 1.f / kMaxDepth);
            const float k0 = floorf(g * zn - dist0) - 2.f;
            if (k0 > 0.f) {
                r.res = fma3(k0, r.dir, r.res);
                r.dist_s = dist0 + k0;
            }
            r.dist_lim = fminf(dist_e, g * zf + 2.f);
            // A sample nearer than zn (the nearest depth of any allocated block
            // whose projection covers this tile, less a voxel) cannot lie in an
            // allocated block: the loop would look its block up, find it empty
            // and jump. Those jumps are taken here without lookups, with the
            // loop's jump arithmetic: the same blocks and sample lattice (an
            // instrumented run found every skipped block empty; positions agree
            // with the lookup path to float rounding).
            const float lim = g * zn - 1.f;
            while (r.dist_s < lim && r.dist_s < r.dist_lim) empty_jump(r);
        }
        r.x = x;
        r.y = y;
        r.sdf = 1.f;
        r.valid = false;
        // a region of its own: every code differs from it above the low 3 bits
        // (a wide one only from 2^31 voxels down does not, where no block can be)
        r.cx = r.cy = r.cz = INT_MIN;
        r.cmask = 7;
        r.cblk = -1;
        return true;
    }

    // Bits in which floor codes (ix, iy, iz) differ from the last looked-up
    // voxel's: none above r.cmask, and they lie in the same settled region.
    static __device__ __forceinline__ int moved(const Ray& r, int ix, int iy, int iz)
    {
        return (ix ^ r.cx) | (iy ^ r.cy) | (iz ^ r.cz);
    }

    // Looks the voxel up: the largest empty cube the occupancy words show
    // around it, or its block's slot. The three reads do not depend on one
    // another (the brick's word kept from the last lookup spared two of them at
    // the price of branches, and was slower).
    static __device__ __forceinline__ void settle(const DevMap& m, Ray& r, int ix, int iy, int iz)
    {
        if (WIDE && !m.grid) {
            r.cmask = 7;
            r.cblk = hash_find<NC>(m, ix >> 3, iy >> 3, iz >> 3);
            return;
        }
        const int brick8 = grid_brick8(m, ix, iy, iz), bit8 = grid_bit8(ix, iy, iz);
        const unsigned long long above = ld_map<NC>(m.occ2 + grid_region(m, ix, iy, iz));
        const unsigned long long here = ld_map<NC>(grid_occ(m, brick8));
        const unsigned long long e = ld_map<NC>(grid_cell(m, brick8, bit8));
        r.cmask = here ? 7 : above ? 31 : 127;
        r.cblk = slot_of(m, e, ix, iy, iz);
    }

    // Ray distance up to which a ray at res is certain to stay in its empty
    // cube: the exit distance from the cube with its exit faces drawn in by
    // `slack` voxels, the rounding of the positions on the way. (A margin on
    // the distance would not do: a ray of slope s to a face that is off by e
    // reaches it e / s early. The entry faces need none: a rounded step never
    // goes back.) A ray that starts within the slack looks its next position
    // up. (Wide views look at every position instead.)
    static __device__ __forceinline__ float run_limit(const Ray& r, float slack)
    {
        if constexpr (WIDE) return r.dist_s;
        const float far = (float)(r.cmask + 1) - slack;
        auto exit = [&](int i, float p, float d, float inv) {
            return (ff(i & ~r.cmask) + (signbit(d) ? slack : far) - p) * inv;
        };
        const float t = fminf(fminf(exit(r.cx, r.res.x, r.dir.x, r.inv.x), exit(r.cy, r.res.y, r.dir.y, r.inv.y)),
                              exit(r.cz, r.res.z, r.dir.z, r.inv.z));
        return fminf(r.dist_lim, r.dist_s + t);
    }

    // First half of a loop iteration: from the sample at res towards the first
    // one in an allocated block (slot r.cblk, its voxel in cx, cy, cz), over up
    // to kSeek empty cubes. Each unallocated block on the way reads (1.0,
    // invalid) and is jumped over, one jump a block as in the reference's
    // lattice, but looked up only once per empty cube. kSeek bounds how long
    // the rays of the warp that are in a block wait for those that cross empty
    // space, to about the time of a sample: at grazing views every iteration
    // has some ray with a long way to go, and a warp whose iterations all
    // waited for it took 438 turns of the jump loop where no ray of it made
    // more than 45 jumps.
    static constexpr int kSeek = 2;
    enum Seek { kOut, kBlock, kOnTheWay };  // the ray's range ended, in a block, neither yet

    static __device__ __forceinline__ Seek seek(const MapView& v, Ray& r)
    {
#pragma unroll 1
        for (int n = 0; n <= kSeek; ++n) {
            if (!(r.dist_s < r.dist_lim)) return kOut;
            if (n == kSeek) break;
            const int ix = fl(r.res.x), iy = fl(r.res.y), iz = fl(r.res.z);
            const int d = moved(r, ix, iy, iz);
            r.cx = ix;
            r.cy = iy;
            r.cz = iz;
            if (d & ~r.cmask) settle(v.m, r, ix, iy, iz);
            if (r.cblk >= 0) return kBlock;
            const float run = run_limit(r, v.out.slack);
            do empty_jump(r);
            while (r.dist_s < run);
            r.sdf = 1.f;
            r.valid = false;
        }
        return kOnTheWay;
    }

    // An unobserved voxel of an allocated block reads (1.0, invalid), and the
    // reference steps one voxel (ray_tracing.cu:372-378). Most rays meet none,
    // but runs of them make the slowest rays: at 640x480 / 5 mm the slowest
    // rays of the 200 slowest 8x4 tiles of a frame spend on average 13 of
    // their 19 iterations on them (an oracle count; 0.03 per ray over all
    // rays), and a tile lasts as long as its slowest ray.
    // So from an unobserved sample the next kRunAhead one-voxel samples inside
    // the same block are loaded together, and the unobserved ones that lead
    // are consumed in this iteration. The ray lands on the first sample that
    // is observed, lies outside the block or is past dist_lim, and the next
    // iteration takes it; positions and distances are the one-at-a-time
    // steps' own (the same fma and add chains).
    static constexpr int kRunAhead = 4;

    static __device__ __forceinline__ void unobserved_run(const MapView& v, Ray& r)
    {
        const Word* blk = Layout<FMT>::words(v.m, r.cblk);
        float3 q = r.res;
        float ds = r.dist_s;
        bool ok[kRunAhead];
        Word w[kRunAhead];
#pragma unroll
        for (int k = 0; k < kRunAhead; ++k) {
            q = fma3(1.f, r.dir, q);
            ds = __fadd_rn(ds, 1.f);
            const int ix = fl(q.x), iy = fl(q.y), iz = fl(q.z);
            ok[k] = ds < r.dist_lim && !(moved(r, ix, iy, iz) & ~7);
            w[k] = ld_map<NC>(blk + at(ix, iy, iz));  // (some voxel of the block where the sample is not in it)
        }
        int n = 1;  // samples consumed: this one, then the leading unobserved ones ahead
        bool run = true;
#pragma unroll
        for (int k = 0; k < kRunAhead; ++k) {
            run = run && ok[k] && !F::observed(w[k]);
            n += run ? 1 : 0;
        }
        for (int k = 0; k < n; ++k) {
            r.res = fma3(1.f, r.dir, r.res);
            r.dist_s = __fadd_rn(r.dist_s, 1.f);
        }
        r.sdf = 1.f;
        r.valid = false;
    }

    // Second half: one iteration of the reference loop at the sample at res,
    // voxel (cx, cy, cz) of block r.cblk; true when the ray leaves the loop.
    // The sample and the link its corners may need are read together, the
    // other corners after it.
    static __device__ __forceinline__ bool advance(const MapView& v, Ray& r)
    {
        const DevMap& m = v.m;
        const Corners c = corners(r.res, r.cx, r.cy, r.cz);
        const int cross = c.cross();
        const Word w0 = ld_map<NC>(Layout<FMT>::words(m, r.cblk) + at(c.x0, c.y0, c.z0));  // read_sdf at floor(res)
        const int far = far_slot(m, r.cblk, cross);
        bool valid;
        float sdf = value(w0, valid);
        if (!valid) {
            unobserved_run(v, r);
            return false;
        }
        if (sdf <= 0.5f && sdf >= -0.5f) {
            float s[8];
            valid = corners8(m, r.cblk, far, cross, c, w0, s);
            sdf = lerp8(s, c.ax, c.ay, c.az);
        }
        r.sdf = sdf;
        r.valid = valid;
        if (sdf <= 0.f) return true;
        const float st = valid ? fmaxf(__fmul_rn(sdf, v.out.rts), 1.f) : 1.f;
        r.res = fma3(st, r.dir, r.res);
        r.dist_s = __fadd_rn(r.dist_s, st);
        return false;
    }

    // After the loop: two refinement steps when the zero crossing was found
    // (ray_tracing.cu:381-393), then the camera-frame vertex or a miss. The
    // first step lands in the block the ray is in on 69 % of crossings and in
    // the one before on 27 % (640x480 / 5 mm, an oracle count).
    static __device__ __forceinline__ void finish(const MapView& v, Ray& r)
    {
        const RenderOut& o = v.out;
        bool found = false;
        if (r.sdf <= 0.f) {
            r.res = fma3(__fmul_rn(r.sdf, o.rts), r.dir, r.res);
            const int ix = fl(r.res.x), iy = fl(r.res.y), iz = fl(r.res.z);
            int slot = r.cblk;
            if (moved(r, ix, iy, iz) & ~7) slot = find(v.m, ix, iy, iz);
            bool valid = false;
            const Corners c = corners(r.res, ix, iy, iz);
            const int cross = c.cross();
            float e[8];
            if (slot >= 0) {
                const Word w0 = ld_map<NC>(Layout<FMT>::words(v.m, slot) + at(ix, iy, iz));
                valid = corners8(v.m, slot, far_slot(v.m, slot, cross), cross, c, w0, e);
            } else {
                // corner 0's block is not allocated: the read is invalid and the
                // pixel a miss, whatever the corners hold. (As a branch of its
                // own, without these lookups, the kernel was compiled to run
                // 0.5-1.4 % slower on the cases of several sizes, 4 % in one form.)
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int vx = (k & 1) ? c.x1 : c.x0, vy = (k & 2) ? c.y1 : c.y0, vz = (k & 4) ? c.z1 : c.z0;
                    bool ok;
                    e[k] = k & cross ? voxel(v.m, find(v.m, vx, vy, vz), vx, vy, vz, ok) : 1.f;
                }
            }
            const float s = lerp8(e, c.ax, c.ay, c.az);
            r.res = fma3(__fmul_rn(s, o.rts), r.dir, r.res);
            found = valid;
        }
        float4 out;
        if (found) {
            const float3 q = xf_apply(v.Ti, div_exact(r.res.x, o.vsinv, o.vsinvRcp), div_exact(r.res.y, o.vsinv, o.vsinvRcp),
                                      div_exact(r.res.z, o.vsinv, o.vsinvRcp));
            out = make_float4(q.x, q.y, q.z, 1.f);
        } else {
            const float qnan = __int_as_float(0x7fffffff);
            out = make_float4(qnan, qnan, qnan, qnan);
        }
        *(reinterpret_cast<float4*>(reinterpret_cast<char*>(o.vmap) + (size_t)r.y * o.vpitch) + r.x) = out;
    }
};

// The q-th of a map's nt tiles to be handed out, as a row-major index: order 0
// bottom rows first, 1 top rows first, 2 alternating from both ends (what a map
// starts with). The slow tiles are often those of the upper or the lower rows,
// seen at grazing angles, and started last they prolong the launch: alternating
// against bottom rows first 70 -> 64 us at 640x480, 131 -> 119 us for the 800x600
// full march, 67 -> 64 us a view at 517x389, no difference at 320x240 and on
// batches.
__host__ __device__ constexpr int tile_at(int order, int q, int nt)
{
    return order == 0 ? nt - 1 - q : order == 1 ? q : (q & 1) ? nt - 1 - (q >> 1) : (q >> 1);
}
static_assert(tile_at(0, 0, 5) == 4 && tile_at(0, 4, 5) == 0 && tile_at(1, 0, 5) == 0 && tile_at(1, 4, 5) == 4 &&
                  tile_at(2, 0, 5) == 0 && tile_at(2, 1, 5) == 4 && tile_at(2, 4, 5) == 2 && tile_at(2, 3, 4) == 2,
              "three different orders, each of all tiles");

// One warp marches tile q of the nt tiles of a map (q counts in the order the
// tiles are handed out).
template <int FMT, bool NC, bool WIDE>
__device__ __forceinline__ void march_tile(const MapView& v, int q, int nt, int order, int tw, int lane)
{
    typedef March<FMT, NC, WIDE> M;
    const int t = tile_at(order, q, nt);
    const int tx = (v.cam.W + tw - 1) / tw;
    const int x = (t % tx) * tw + (lane % tw), y = (t / tx) * (32 / tw) + (lane / tw);
    Ray r;
    const bool started = x < v.cam.W && y < v.cam.H && M::init(v, r, x, y);
    // warp-synchronous march: the lanes meet at both halves of an iteration,
    // so their sample and corner reads are issued together; finished lanes
    // idle until the tile is done, then all finish together
    bool live = started;
    while (__any_sync(0xffffffffu, live)) {
        int at = M::kOut;
        if (live) at = M::seek(v, r);
        __syncwarp();
        live = at == M::kOnTheWay || (at == M::kBlock && !M::advance(v, r));
    }
    if (started) M::finish(v, r);
}

}  // namespace vmapb
