/*
 * near.cuh -- neighbour search over the sorted particles themselves: an implicit 8-ary
 * tree of bounding boxes (8 consecutive particles of the Hilbert order make a block, 8
 * blocks a node of the next level, and so on up) and the warp search that walks it.
 *
 * Why beside the octree: a leaf's list is made for the widest particle of the leaf and
 * streamed by every group of it, so a group tests several times the pairs it accepts, and
 * where h varies (a scattered start, the edge of a concentrated set) one warp streams whole
 * lists for a few particles while the chip idles.  Here a group finds the 8-particle blocks
 * its members' spheres reach, and each member then takes only the blocks its OWN sphere
 * touches: on a lattice (58 neighbours) about 180 candidates per particle instead of 440,
 * and no list, no work items and no per-leaf bookkeeping between iterations.
 *
 * Boxes are FP32 relative to the root box's centre, in units of a power of two near its
 * largest side (so that squares stay in FP32's range whatever the caller's units), rounded
 * outward, and every radius
 * carries a slack above the rounding of the tests, so a block is never left out that
 * holds a pair the exact FP64 test accepts.  Blocks come out in ascending order and the
 * lanes of a step hold 32 consecutive candidates of one particle, so what is accepted is
 * in ascending j, the order of every sum.
 */
#pragma once

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "rows.cuh"
#include "state.hpp"
#include "tma.cuh"

namespace cosmo {

constexpr int kNearLevels = 9;     // level 0: blocks of 8 particles; 32 * 8^9 particles at most
constexpr int kNearBlocks = 128;   // blocks a warp holds at once
constexpr int kNearWarps  = 4;     // warps per block of the search kernels

// Up to this many particles a pass over rows gives each particle a warp: one lane each would
// leave most of the chip idle and last as long as the longest row.  Device us with a lane and
// with a warp a particle, lattice and periodic box of random particles:
//   particles       4,000              16,000             24,000             32,000
//   Newton loop     135  92, 372 224   162 145, 436 330   174 180, 486 410   176 204, 514 470
//   symmetric rows   34  25, 118  75    34  32, 136  98    38  36, 115  87    38  40, 130  99
//   gradient         58  30,  74  31    62  58,  84  62    66  83,  89  81    67 105,  87 103
//   force            60  30,  85  32    64  84,  91  94    69 126,  96 133    71 162, 101 175
// (48,000: the Newton loop 209 269, 597 623.)  The three passes of a solve together draw level
// between 24,000 (lattice) and above 32,000 (box, with more iterations); the force pass, whose
// energy sum is four dependent additions a pair, at 12,000 (65 70, 88 73).
constexpr int kWarpPerParticle = 32768;
constexpr int kWarpPerParticleForce = 12288;

// Extras: the pairs a row must gain from another particle's support, kExtra places a
// particle.  (Once appended to one list through one counter, then counted, scanned and placed:
// where h scatters there are ten a particle, and the counter's atomics took 5 ms of a
// 2-million-particle step.)
constexpr int kExtra = kQuintic ? 64 : 32;   // of 2 M quintic Plummer particles 1% gain more than 32

// Whether a solve over the block tree loses to one over lists: a large set of which every
// particle has more neighbours than a row holds -- 4/3 pi (R hfact)^3 of them at its converged
// h -- is all searches of single particles, where a leaf's groups share theirs.  Device times
// of the whole step, block tree and lists: box of 1,000,000 at hfact 1.5 (113 neighbours)
// 28.1 and 32.0 ms, 1.53 (120) 35.0 and 35.9, 1.55 (125) 41.2 and 37.9, 1.6 56.0 and 45.6,
// 2.2 102 and 83; at 1.6 450,000 25.4 and 24.8, 340,000 19.4 and 22.7, 150,000 8.9 and 9.3
// (a Plummer sphere 10.8 and 26.0).  Batches (whole solve): 10 boxes of 10,000 at 1.6 3.0
// and 3.5, 6 of 100,000 15.5 and 11.4, 24 of 100,000 60.0 and 40.4.
constexpr int kNearCrowded = 400000;

// The neighbours of a converged particle, over what a row holds.
inline double near_fill(double hfact)
{
    const double reach = kRadKernel * hfact;
    return 4.18879 * reach * reach * reach / kNbl;
}
inline bool near_crowded(int n, double hfact) { return n > kNearCrowded && near_fill(hfact) > 0.95; }

// Blocks a multiprocessor for the sweeps of the particles without a row, whose number is on
// the device: four where an average particle comes near not fitting one (150,000 in a box at
// hfact 1.6, nearly all of them: gradient 2.3 -> 1.3 ms with the packed pairs), else
// two: there are few or none.
inline int near_over_blocks(double hfact) { return near_fill(hfact) > 0.6 ? 4 : 2; }

// A node's box: centre, half extents (empty: negative infinity) and its largest h.
struct alignas(32) NearNode
{
    float cx, cy, cz, hmax, ex, ey, ez, pad;
};

// The block trees of one particle set, or of the sets of a batch one after the other in the
// sorted order (set s from its first particle p0 on).  Level l of set s starts at
// node[off[l] + (p0 >> (3 l + 3)) + s]: a set's nodes of a level never reach the next set's
// start, so no table is needed.  The live particle count (of the one set) is read on the
// device, so one set of arguments serves every solve.
struct NearTree
{
    const NearNode* __restrict__ node;
    const double4* __restrict__ xyzh;
    const DevBox* __restrict__ box;
    const int* nLive;
    int off[kNearLevels];
};

// One set of a batch, as the search kernels read it.  An open set's periods are infinite, so
// that one periodic instance of a kernel serves both (no separation is folded).
struct NearSet
{
    int p0, n;                 // first particle of the sorted order, live particles
    float lx, ly, lz, len;     // periods, largest side (scaled)
    double cx, cy, cz, scale;  // box centre, the search frame's scale
    double dlx, dly, dlz;      // periods
    double pmass;
};

// What a search knows of its set: the one set of a solve, or one of a batch.
struct NearView
{
    int p0, s, n;
    float lx, ly, lz;
};

__host__ __device__ inline int near_count(int n, int level) { return (n + (8 << (3 * level)) - 1) >> (3 * level + 3); }

// Per-warp shared scratch of a search.
struct NearScratch
{
    double4 P[32];                 // the members: position and one test value
    float4 Q[32];                  // position and squared reach in the search frame
    int front[kNearLevels][32];    // accepted nodes of each level, not yet expanded
    int blk[kNearBlocks];          // accepted blocks, ascending
    int sel[kNearBlocks + 8];      // those one member reaches, then kNearNone
};
constexpr int kNearNone = 0x0fffffff;   // a block whose particles lie beyond any set's

// The lane, kept in a register (read anew it costs an instruction at every use).
__device__ __forceinline__ int lane_id()
{
    int l;
    asm volatile("mov.u32 %0, %%laneid;" : "=r"(l));
    return l;
}

__device__ __forceinline__ NearNode ld_node(const NearNode* p)
{
    NearNode n;
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(n.cx), "=f"(n.cy), "=f"(n.cz), "=f"(n.hmax), "=f"(n.ex), "=f"(n.ey), "=f"(n.ez), "=f"(n.pad)
        : "l"(p));
    return n;
}

// Stores under a predicate, without a branch around them: a warp whose lanes differ in it
// would otherwise part and join again at every step of a search.
__device__ __forceinline__ void st_if(bool p, double* a, double v)
{
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %0, 0;\n\t@q st.global.f64 [%1], %2;\n\t}"
                 :: "r"(int(p)), "l"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void st_if(bool p, int* a, int v)
{
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %0, 0;\n\t@q st.global.s32 [%1], %2;\n\t}"
                 :: "r"(int(p)), "l"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void st_shared_if(bool p, int* a, int v)
{
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %0, 0;\n\t@q st.shared.s32 [%1], %2;\n\t}"
                 :: "r"(int(p)), "r"(smem_u32(a)), "r"(v) : "memory");
}

// The power of two that brings a length into [1, 2) (1 for one that is 0 or beyond any use).
__device__ __forceinline__ double near_scale(double len)
{
    const int e = int(__double_as_longlong(len) >> 52);   // the exponent's bits (len >= 0)
    return e > 0 && e <= 2045 ? __longlong_as_double((long long)(2046 - e) << 52) : 1.0;
}

// The search frame: box centre, scale and periods, and the slack of a radius.  Lengths in it
// are the caller's times the scale, which is exact: a reach of 2^64 or 2^-75 in the caller's
// units would have a square of infinity or 0 in FP32, and every block would pass its test or
// some of those it needs would not.  A relative coordinate a is rounded by at most 2^-24 |a|,
// and a gap's two subtractions (and the fold at the period) by as much again of terms no
// larger than the box, so the gap of a point errs by less than 2^-22 (len + |a|) per axis;
// 4e-7 (len + |a|_1) covers three axes.
struct NearFrame
{
    double cx, cy, cz, scale;
    float lx, ly, lz, len;

    __device__ __forceinline__ explicit NearFrame(const DevBox* b)
    {
        cx = b->lo[0] + 0.5 * b->len[0];
        cy = b->lo[1] + 0.5 * b->len[1];
        cz = b->lo[2] + 0.5 * b->len[2];
        scale = near_scale(fmax(b->len[0], fmax(b->len[1], b->len[2])));
        lx = float(b->len[0] * scale);
        ly = float(b->len[1] * scale);
        lz = float(b->len[2] * scale);
        len = fmaxf(lx, fmaxf(ly, lz));
    }
    __device__ __forceinline__ explicit NearFrame(const NearSet& s)
        : cx(s.cx), cy(s.cy), cz(s.cz), scale(s.scale), lx(s.lx), ly(s.ly), lz(s.lz), len(s.len)
    {
    }
    // a position, and a length rounded up, in the frame
    __device__ __forceinline__ float3 at(const double4& p) const
    {
        return make_float3(float((p.x - cx) * scale), float((p.y - cy) * scale), float((p.z - cz) * scale));
    }
    __device__ __forceinline__ float length(double r) const { return __double2float_ru(r * scale); }
    __device__ __forceinline__ float slack(float x, float y, float z) const
    {
        return 4e-7f * (len + fabsf(x) + fabsf(y) + fabsf(z));
    }
};

__device__ __forceinline__ NearView near_view(const NearTree& t, const NearFrame& f)
{
    return NearView{0, 0, *t.nLive, f.lx, f.ly, f.lz};
}

__device__ __forceinline__ const NearNode* near_node(const NearTree& t, const NearView& v, int level, int idx)
{
    return t.node + (t.off[level] + (v.p0 >> (3 * level + 3)) + v.s + idx);
}

// Squared gap between the box (c, e) and a node's box, at the nearest image.
template<bool Periodic>
__device__ __forceinline__ float near_gap2(float x, float y, float z, float ex, float ey, float ez, const NearNode& n,
                                           const NearView& f)
{
    float dx = fabsf(x - n.cx), dy = fabsf(y - n.cy), dz = fabsf(z - n.cz);
    if (Periodic)
    {
        dx = fminf(dx, f.lx - dx);
        dy = fminf(dy, f.ly - dy);
        dz = fminf(dz, f.lz - dz);
    }
    dx = fmaxf(dx - (ex + n.ex), 0.0f);
    dy = fmaxf(dy - (ey + n.ey), 0.0f);
    dz = fmaxf(dz - (ez + n.ez), 0.0f);
    return fmaf(dz, dz, fmaf(dy, dy, dx * dx));
}

// What a node's own h adds to a symmetric search's reach.
__device__ __forceinline__ float near_sym_reach(float hmax, float slack)
{
    return fmaf(hmax, float(kRadKernel) * 1.000001f, slack);
}

// The blocks within reach of the box (c, e) -- or, Sym, within a block's own support of it
// -- in ascending order, kNearBlocks at a time: flush(count) uses scr.blk and returns the
// reach to go on with (the members still searching may be narrower), negative to stop.
// The top level (at most 32 nodes) is tested first; then always the first four nodes of the
// deepest level that holds any are expanded, one child per lane, so each level holds at
// most 32 nodes and the blocks come out in order.  Stop = 1 hands out the nodes of level 1
// instead (of more than 256 particles).
template<int Stop, bool Periodic, bool Sym, class Flush>
__device__ __forceinline__ void near_blocks(const NearTree& t, const NearView& v, NearScratch& scr, float x, float y,
                                            float z, float ex, float ey, float ez, float reach, float slack,
                                            Flush&& flush)
{
    const int lane = lane_id();
    const uint32_t lt = (1u << lane) - 1u;
    // lane l: the nodes of level l and where they start
    const int myCount = lane < kNearLevels ? near_count(v.n, lane) : 0;
    const int myOff = lane < kNearLevels ? t.off[lane] + (v.p0 >> (3 * lane + 3)) + v.s : 0;
    const int top = __popc(__ballot_sync(0xffffffffu, myCount > 32));
    int nb = 0;
    int left = 0, pos = 0;   // lane l: nodes of level l not yet expanded, and the first of them
    auto test = [&](int level, int idx) {
        const NearNode n = ld_node(t.node + (__shfl_sync(0xffffffffu, myOff, level) + idx));
        const float r = Sym ? fmaxf(reach, near_sym_reach(n.hmax, slack)) : reach;
        return near_gap2<Periodic>(x, y, z, ex, ey, ez, n, v) <= r * r;
    };
    // children of up to four nodes, or the top level: accepted ones of level into the next list
    auto accept = [&](int level, int idx, bool valid) {
        const bool ok = test(level, valid ? idx : 0) && valid;
        const uint32_t m = __ballot_sync(0xffffffffu, ok);
        const int c = __popc(m);
        if (level == Stop)
        {
            st_shared_if(ok, scr.blk + nb + __popc(m & lt), idx);
            nb += c;
        }
        else
        {
            st_shared_if(ok, scr.front[level] + __popc(m & lt), idx);
            if (lane == level) { left = c; pos = 0; }
        }
        __syncwarp();
    };
    const int tops = __shfl_sync(0xffffffffu, myCount, top);
    accept(top, lane, lane < tops);
    int lev = top;
    for (;;)
    {
        int have = 0;
        while (lev > Stop && lev <= top && (have = __shfl_sync(0xffffffffu, left, lev)) == 0) ++lev;
        const bool end = lev <= Stop || lev > top;
        if (end || (lev == Stop + 1 && nb + 32 > kNearBlocks))
        {
            if (nb > 0) reach = flush(nb);
            if (end || reach < 0.0f) return;
            __syncwarp();
            nb = 0;
        }
        const int first = __shfl_sync(0xffffffffu, pos, lev);
        const int m = min(have, 4);
        const int node = scr.front[lev][first + min(lane >> 3, m - 1)];
        const int child = node * 8 + (lane & 7);
        const int below = __shfl_sync(0xffffffffu, myCount, lev - 1);
        if (lane == lev) { left -= m; pos += m; }
        accept(lev - 1, child, (lane >> 3) < m && child < below);
        if (lev > Stop + 1) --lev;
    }
}

__device__ __forceinline__ float warp_max_f(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Members of a warp's search in equal runs of consecutive lanes: as many lanes per run (a
// power of two) as keep every run's bounding box within kNearSpread of its largest reach,
// so that sparse members (an active list late in the loop, the edge of a set) do not share
// one search over everything between them, and all of a run in one set.  x, y, z, r, set:
// the lane's member (r < 0: none); on return the run's box (centre, half) and reach on every
// lane of it.
constexpr float kNearSpread = 1.5f;
struct NearRun
{
    int w;
    float cx, cy, cz, ex, ey, ez, reach;
};

template<bool Forest>
__device__ __forceinline__ NearRun near_runs(float x, float y, float z, float r, int set)
{
    const bool on = r >= 0.0f;
    float lx = on ? x : INFINITY, hx = on ? x : -INFINITY;
    float ly = on ? y : INFINITY, hy = on ? y : -INFINITY;
    float lz = on ? z : INFINITY, hz = on ? z : -INFINITY;
    int s0 = on ? set : 0x7fffffff, s1 = on ? set : -1;   // the run's sets
    NearRun u;
    u.w = 1;
    u.reach = r;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const float ax = fminf(lx, __shfl_xor_sync(0xffffffffu, lx, o)), bx = fmaxf(hx, __shfl_xor_sync(0xffffffffu, hx, o));
        const float ay = fminf(ly, __shfl_xor_sync(0xffffffffu, ly, o)), by = fmaxf(hy, __shfl_xor_sync(0xffffffffu, hy, o));
        const float az = fminf(lz, __shfl_xor_sync(0xffffffffu, lz, o)), bz = fmaxf(hz, __shfl_xor_sync(0xffffffffu, hz, o));
        const float rr = fmaxf(u.reach, __shfl_xor_sync(0xffffffffu, u.reach, o));
        const float ext = fmaxf(bx - ax, fmaxf(by - ay, bz - az));
        const int a0 = Forest ? min(s0, __shfl_xor_sync(0xffffffffu, s0, o)) : 0;
        const int a1 = Forest ? max(s1, __shfl_xor_sync(0xffffffffu, s1, o)) : 0;
        if (u.w != o || !__all_sync(0xffffffffu, !(ext > kNearSpread * rr) && (!Forest || a1 <= a0))) continue;
        if (Forest) { s0 = a0; s1 = a1; }
        lx = ax; hx = bx; ly = ay; hy = by; lz = az; hz = bz;
        u.reach = rr;
        u.w = 2 * o;
    }
    // box sides rounded by at most 2^-23 of the coordinates: inside the slack
    u.cx = 0.5f * (lx + hx); u.ex = fmaxf(hx - u.cx, u.cx - lx);
    u.cy = 0.5f * (ly + hy); u.ey = fmaxf(hy - u.cy, u.cy - ly);
    u.cz = 0.5f * (lz + hz); u.ez = fmaxf(hz - u.cz, u.cz - lz);
    return u;
}

NearTree near_tree(State& s);   // the arguments of a search of s's live particles

// One loop: its trees, the sets and the particles' set (a batch; null for one set), the
// particle arrays, the rows' j (or null), the particles its launches cover, and its scalars.
struct NearJob
{
    NearTree tree;
    const NearSet* sets;
    const int* setOf;
    double4* xyzh;
    double *rho, *gradh;
    int *converged, *rowsJ;
    int n, periodic;
    double pmass, tolh, hfact;
};

// A batch as its loop reads it: set s holds [offs[s], offs[s] + nAlive[s]) of the sorted order.
struct NearForest
{
    int n, nsets;
    const int *offs, *nAlive, *setOf;
    const DevBox* boxes;
    const double* pmass;
    double4* xyzh;
    double *rho, *gradh;
    int* converged;
};
void near_forest_newton(State& s, const NearForest& b, double tolh, double hfact, int maxIter, bool graph);
void near_forest_eval(State& s, const NearForest& b);

// Whether the block-tree loop L ended without a result, so that the passes after it have
// nothing to do: it was not run (a particle outside the box of its key), some h did not
// converge, or the largest support reaches half the box (halfBox; not a number for an open
// set).  L null: the list-based loop, which has told the host.
// (All loads before the first branch: the kernels that ask have a warp per particle, and each
// would wait for one load after the other -- 1.5 us of a 20,000-particle gradient sweep.)
__device__ __forceinline__ bool near_failed(const NearLoop* L, const DevScalars* ds, double halfBox)
{
    if (L == nullptr) return false;
    const int outside = ds->outside, active = L->active;
    const double hm = __longlong_as_double((long long)ds->hmaxConv);
    return (outside != 0) | (active > 0) | (kRadKernel * hm >= halfBox);
}

// As many blocks of a kernel as the device holds at once.
template<class K>
inline int persistent_blocks(const State& s, K kernel, int threads)
{
    int perSM = 0;
    COSMO_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, kernel, threads, 0));
    return std::max(1, perSM) * s.numSMs;
}

// Candidates of the blocks ids[0 .. ns) (ns >= 1): use(pj, j, valid) for 32 consecutive
// candidates per step (lane: its own), the next step's loads in flight meanwhile.  use
// returns false, on every lane, to stop.
template<class Use>
__device__ __forceinline__ void near_candidates(const int* ids, int ns, int nLive, const double4* __restrict__ xyzh,
                                                Use&& use)
{
    const int lane = threadIdx.x & 31;
    const int sub = lane >> 3, off = lane & 7;
    auto load = [&](int k, double4& p, int& j, bool& valid) {
        const int at = k + sub;
        j = ids[min(at, ns - 1)] * 8 + off;
        valid = at < ns && j < nLive;
        p = ldg4(xyzh + (valid ? j : 0));
    };
    // two sets of registers in turn: a step's loads are in flight while the one before it is
    // tested, and nothing is copied from one to the other
    double4 pa, pb;
    int ja, jb;
    bool va, vb;
    load(0, pa, ja, va);
    for (int k = 0;;)
    {
        load(k + 4, pb, jb, vb);
        if (!use(pa, ja, va)) return;
        if ((k += 4) >= ns) return;
        load(k + 4, pa, ja, va);
        if (!use(pb, jb, vb)) return;
        if ((k += 4) >= ns) return;
    }
}

// The same, the candidates that pass test(pj) packed: use(j, count) for up to 32 of them at a time,
// lane k < count the k-th, in ascending j (scr.sel holds those not handed out yet, held of
// them).  A search of one particle's support tests two to three candidates for each pair it
// accepts: evaluated where they were loaded, most lanes would wait for the others.  Call
// near_packed_end after the last blocks.
template<class Test, class Use>
__device__ __forceinline__ void near_packed(NearScratch& scr, int nb, int nLive, const double4* __restrict__ xyzh,
                                            int& held, Test&& test, Use&& use)
{
    const int lane = threadIdx.x & 31;
    near_candidates(scr.blk, nb, nLive, xyzh, [&](const double4& pj, int j, bool valid) {
        const bool ok = valid && test(pj);
        const uint32_t m = __ballot_sync(0xffffffffu, ok);
        if (ok) scr.sel[held + __popc(m & ((1u << lane) - 1u))] = j;
        held += __popc(m);
        __syncwarp();
        if (held < 32) return true;
        use(scr.sel[lane], 32);
        const int beyond = scr.sel[32 + lane];
        __syncwarp();
        held -= 32;
        if (lane < held) scr.sel[lane] = beyond;
        __syncwarp();
        return true;
    });
}

template<class Use>
__device__ __forceinline__ void near_packed_end(NearScratch& scr, int& held, Use&& use)
{
    const int lane = threadIdx.x & 31;
    if (held > 0) use(scr.sel[min(lane, held - 1)], held);
    held = 0;
    __syncwarp();
}

} // namespace cosmo
