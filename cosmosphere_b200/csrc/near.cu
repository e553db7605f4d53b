/*
 * near.cu -- the plain FP64 density solve over neighbour rows found by the block-tree search
 * (near.cuh): the reference's src/density_base.cu:237-334 and 804-886 for one particle set.
 *
 * Every active particle is in one of three lists.  Those without a row that is complete for
 * their h are searched (near_rows_kernel: r^2 and j of every neighbour within kNearMargin of
 * their support, at most kNbl); those with one take their Newton step from it, one lane
 * each; those with more neighbours than a row holds are summed straight from a search, one
 * warp each.  A step that leaves h inside the row's reach keeps the row, one that outgrows
 * it puts the particle back on the search list.  Lists, counts and decisions stay on the
 * device: the loop is one graph launch (a while node), or the same kernels from the host.
 *
 * The pairs a particle accepts, and their order, are those of any complete candidate
 * stream in ascending j, so h, rho and gradh agree with the oracle bit for bit.
 */
#include <algorithm>

#include "near.cuh"
#include "newton_step.cuh"
#include "state.hpp"

namespace cosmo {

namespace {

constexpr int kThreads = 32 * kNearWarps;

// Rows reach kNearMargin of the support at the h they are made for, so that they serve
// while h grows by up to that.  Measured on the lattice-100 loop (cold start / mid-run): 1.02
// 3.14 / 2.77 ms (particles outgrow their rows), 1.04 3.26 / 2.46, 1.10 3.68 / 2.55 (longer
// rows in every iteration).
constexpr double kNearMargin = 1.04;
constexpr float kNearWide = 1.5f;   // a member this much wider than its warp's mean searches alone
// Batches of blocks after which members that reach less than kNearShare of them search one by
// one: about what a search alone costs, so giving up late never costs more than twice the
// better choice (a 120,000-particle Plummer sphere's loop: 4.4 ms without, 3.05 at 6 batches,
// 3.25 at 4; lattices and boxes never get there).
constexpr int kNearPatience = 6;
constexpr float kNearShare = 0.1f;
constexpr double kCoverMargin = 1.0 + 1e-8;   // rows made for a converged h: just beyond the force test's slack
constexpr double kCoverSlack = 1.0 + 1e-9;    // a row serves the gradient and force passes at h kCoverSlack <= rowH

// ---------------------------------------------------------------- the block tree
__device__ __forceinline__ NearNode node_of(float lx, float ly, float lz, float hx, float hy, float hz, float hm)
{
    NearNode n;
    if (!(lx <= hx && ly <= hy && lz <= hz))
    {
        n.cx = n.cy = n.cz = 0.0f;
        n.ex = n.ey = n.ez = -INFINITY;
        n.hmax = 0.0f;
        n.pad = 0.0f;
        return n;
    }
    n.cx = 0.5f * lx + 0.5f * hx; n.ex = fmaxf(__fsub_ru(hx, n.cx), __fsub_ru(n.cx, lx));
    n.cy = 0.5f * ly + 0.5f * hy; n.ey = fmaxf(__fsub_ru(hy, n.cy), __fsub_ru(n.cy, ly));
    n.cz = 0.5f * lz + 0.5f * hz; n.ez = fmaxf(__fsub_ru(hz, n.cz), __fsub_ru(n.cz, lz));
    n.hmax = hm;
    n.pad = 0.0f;
    return n;
}

// A parent of up to eight nodes, combined from the given ones by a loop (count >= 1).
template<class Get>
__device__ __forceinline__ NearNode node_parent(int count, Get&& get)
{
    float lx = INFINITY, ly = INFINITY, lz = INFINITY, hx = -INFINITY, hy = -INFINITY, hz = -INFINITY, hm = 0.0f;
    for (int k = 0; k < count; ++k)
    {
        const NearNode c = get(k);
        lx = fminf(lx, __fsub_rd(c.cx, c.ex)); hx = fmaxf(hx, __fadd_ru(c.cx, c.ex));
        ly = fminf(ly, __fsub_rd(c.cy, c.ey)); hy = fmaxf(hy, __fadd_ru(c.cy, c.ey));
        lz = fminf(lz, __fsub_rd(c.cz, c.ez)); hz = fmaxf(hz, __fadd_ru(c.cz, c.ez));
        hm = fmaxf(hm, c.hmax);
    }
    return node_of(lx, ly, lz, hx, hy, hz, hm);
}

// Levels 0 to 2: 512 particles a block, one per thread; each level's boxes are reduced in
// shared memory and written once (one 32-byte read per particle: DRAM bound, 11 us at 1.4 M).
// A batch's blocks are its level-2 slots, each looked up to find its set.
template<bool Forest>
__global__ void __launch_bounds__(512)
near_leaf_levels_kernel(const __grid_constant__ NearTree t, NearNode* __restrict__ out,
                        const NearSet* __restrict__ sets, int nsets, int slots)
{
    __shared__ NearNode s0[64], s1[8];
    NearFrame f(t.box);
    NearView v = Forest ? NearView{0, 0, 0, 0.0f, 0.0f, 0.0f} : near_view(t, f);
    for (int q = blockIdx.x; q < slots; q += gridDim.x)
    {
        int b = q;
        if constexpr (Forest)
        {
            int lo = 0, hi = nsets;   // the last set whose slots start at or before q
            while (hi - lo > 1)
            {
                const int mid = (lo + hi) >> 1;
                if ((sets[mid].p0 >> 9) + mid <= q) lo = mid;
                else hi = mid;
            }
            f = NearFrame(sets[lo]);
            v = NearView{sets[lo].p0, lo, sets[lo].n, 0.0f, 0.0f, 0.0f};
            b = q - ((v.p0 >> 9) + lo);
        }
        if (b * 512 >= v.n) continue;
        const int i = b * 512 + int(threadIdx.x);
        float lx = INFINITY, ly = INFINITY, lz = INFINITY, hx = -INFINITY, hy = -INFINITY, hz = -INFINITY, hm = 0.0f;
        if (i < v.n)
        {
            const double4 p = t.xyzh[v.p0 + i];
            const double x = (p.x - f.cx) * f.scale, y = (p.y - f.cy) * f.scale, z = (p.z - f.cz) * f.scale;
            lx = __double2float_rd(x); hx = __double2float_ru(x);
            ly = __double2float_rd(y); hy = __double2float_ru(y);
            lz = __double2float_rd(z); hz = __double2float_ru(z);
            hm = f.length(p.w);
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1)
        {
            lx = fminf(lx, __shfl_xor_sync(0xffffffffu, lx, o)); hx = fmaxf(hx, __shfl_xor_sync(0xffffffffu, hx, o));
            ly = fminf(ly, __shfl_xor_sync(0xffffffffu, ly, o)); hy = fmaxf(hy, __shfl_xor_sync(0xffffffffu, hy, o));
            lz = fminf(lz, __shfl_xor_sync(0xffffffffu, lz, o)); hz = fmaxf(hz, __shfl_xor_sync(0xffffffffu, hz, o));
            hm = fmaxf(hm, __shfl_xor_sync(0xffffffffu, hm, o));
        }
        auto put = [&](int level, int idx, const NearNode& nd) { out[near_node(t, v, level, idx) - t.node] = nd; };
        if ((threadIdx.x & 7) == 0)
        {
            const NearNode nd = node_of(lx, ly, lz, hx, hy, hz, hm);
            s0[threadIdx.x >> 3] = nd;
            if (i < v.n) put(0, i >> 3, nd);
        }
        __syncthreads();
        if (threadIdx.x < 8)
        {
            const NearNode nd = node_parent(8, [&](int k) { return s0[threadIdx.x * 8 + k]; });
            s1[threadIdx.x] = nd;
            const int p = b * 8 + int(threadIdx.x);
            if (p * 64 < v.n) put(1, p, nd);
        }
        __syncthreads();
        if (threadIdx.x == 0) put(2, b, node_parent(8, [&](int k) { return s1[k]; }));
        __syncthreads();
    }
}

// The levels above, up to the first of at most 32 nodes: one block a set, level by level.
template<bool Forest>
__global__ void __launch_bounds__(1024)
near_upper_levels_kernel(const __grid_constant__ NearTree t, NearNode* out, const NearSet* __restrict__ sets)
{
    const NearFrame f(t.box);
    const NearView v = Forest ? NearView{sets[blockIdx.x].p0, int(blockIdx.x), sets[blockIdx.x].n, 0.0f, 0.0f, 0.0f}
                              : near_view(t, f);
    for (int l = 3; l < kNearLevels && near_count(v.n, l - 1) > 32; ++l)
    {
        const int below = near_count(v.n, l - 1), here = near_count(v.n, l);
        for (int q = threadIdx.x; q < here; q += blockDim.x)
            out[near_node(t, v, l, q) - t.node] =
                node_parent(min(8, below - 8 * q), [&](int k) { return out[near_node(t, v, l - 1, 8 * q + k) - t.node]; });
        __syncthreads();
    }
}

// The sets of a batch as the searches read them (boxes and live counts are those of the
// batch's key sort).
__global__ void near_sets_kernel(int nsets, const int* __restrict__ offs, const int* __restrict__ nAlive,
                                 const DevBox* __restrict__ boxes, const double* __restrict__ pmass,
                                 NearSet* __restrict__ sets)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nsets) return;
    const DevBox b = boxes[s];
    const NearFrame f(&b);
    const bool per = b.periodic != 0;
    const float inf = INFINITY;
    const double dinf = double(inf);
    sets[s] = NearSet{offs[s], nAlive[s],
                      per ? f.lx : inf, per ? f.ly : inf, per ? f.lz : inf, f.len,
                      f.cx, f.cy, f.cz, f.scale,
                      per ? b.len[0] : dinf, per ? b.len[1] : dinf, per ? b.len[2] : dinf, pmass[s]};
}

// ---------------------------------------------------------------- lists
// Append v to a list for the lanes that want to, one atomic per warp.
__device__ __forceinline__ void warp_append(bool want, int v, int* __restrict__ list, int* __restrict__ count)
{
    const uint32_t m = __ballot_sync(0xffffffffu, want);
    if (m == 0u) return;
    const int lane = threadIdx.x & 31;
    int base = 0;
    if (lane == 0) base = atomicAdd(count, __popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (want) list[base + __popc(m & ((1u << lane) - 1u))] = v;
}

// The same for a whole block of kThreads and three lists (to: 0, 1, 2, or -1 for none; every
// thread calls it): one atomic per block and list, so that particles next to each other in
// the sorted order stay together and the counters -- single addresses for the whole grid --
// take a quarter of the atomics.  sh: 3 (kNearWarps + 1) ints.
__device__ __forceinline__ void block_append(int to, int v, int* l0, int* c0, int* l1, int* c1, int* l2, int* c2,
                                             int* sh)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t m0 = __ballot_sync(0xffffffffu, to == 0), m1 = __ballot_sync(0xffffffffu, to == 1);
    const uint32_t m2 = __ballot_sync(0xffffffffu, to == 2);
    if (lane < 3) sh[lane * (kNearWarps + 1) + w] = __popc(lane == 0 ? m0 : (lane == 1 ? m1 : m2));
    __syncthreads();
    if (threadIdx.x < 3)
    {
        int* c = sh + threadIdx.x * (kNearWarps + 1);
        int* count = threadIdx.x == 0 ? c0 : (threadIdx.x == 1 ? c1 : c2);
        int run = 0;
        for (int k = 0; k < kNearWarps; ++k) { const int x = c[k]; c[k] = run; run += x; }
        c[kNearWarps] = run > 0 ? atomicAdd(count, run) : 0;
    }
    __syncthreads();
    if (to >= 0)
    {
        const int* c = sh + to * (kNearWarps + 1);
        const uint32_t m = to == 0 ? m0 : (to == 1 ? m1 : m2);
        int* list = to == 0 ? l0 : (to == 1 ? l1 : l2);
        list[c[kNearWarps] + c[w] + __popc(m & lt)] = v;
    }
    __syncthreads();
}

// Largest h used and largest converged h of a block's particles (as bit patterns, which
// order as the non-negative doubles they are), one atomic each per block.
__device__ __forceinline__ void note_h(unsigned long long seen, unsigned long long conv, DevScalars* ds,
                                       unsigned long long* sh)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
    {
        const unsigned long long a = __shfl_xor_sync(0xffffffffu, seen, o), b = __shfl_xor_sync(0xffffffffu, conv, o);
        seen = a > seen ? a : seen;
        conv = b > conv ? b : conv;
    }
    if (threadIdx.x == 0) sh[0] = sh[1] = 0;
    __syncthreads();
    if ((threadIdx.x & 31) == 0)
    {
        atomicMax(&sh[0], seen);
        atomicMax(&sh[1], conv);
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        if (sh[0]) atomicMax(&ds->hmaxSeen, sh[0]);
        if (sh[1]) atomicMax(&ds->hmaxConv, sh[1]);
    }
}

// All live particles are searched first (the identity list), or none where one lies outside
// the box of its key (the set is solved over lists instead); the counters of the row passes
// after the loop start from zero too.
__global__ void near_init_kernel(NearLoop* L, DevScalars* ds, int maxIter, int frozen)
{
    L->queue[threadIdx.x] = 0;
    if (threadIdx.x != 0) return;
    const int live = ds->nAlive, outside = ds->outside;
    const int n = outside ? 0 : live;
    L->iter = 0;
    L->maxIter = maxIter;
    L->active = n;
    L->all = frozen ? 0 : 1;
    L->cover = L->over = 0;
    L->cnt[0] = NearCounts{0, frozen ? 0 : n, 0, 0};
    L->cnt[1] = NearCounts{0, 0, 0, 0};
    L->ticket[0] = L->ticket[1] = 0;
    ds->extraCount = 0;
    ds->mergeOverflow = 0;
    ds->rowOverflow = 0;
    ds->coverNeed = 0;
    ds->rowsLive = n;
}

// The initial search list with fixed particles (the caller's mask through the sort order;
// they are neighbours only and count as converged): the others.
__global__ void __launch_bounds__(kThreads)
near_frozen_kernel(NearLoop* L, const int* __restrict__ order, const int* __restrict__ frozen,
                   const int* __restrict__ nLive, const double4* __restrict__ xyzh, int* __restrict__ converged,
                   double* __restrict__ hs, NearLists lists, DevScalars* __restrict__ ds)
{
    __shared__ int sh[3 * (kNearWarps + 1)];
    __shared__ unsigned long long shH[2];
    if (ds->outside) return;
    const int n = *nLive;
    unsigned long long hconv = 0;
    for (int b = blockIdx.x * kThreads; b < n; b += gridDim.x * kThreads)
    {
        const int k = b + int(threadIdx.x);
        const bool f = k < n && frozen[order[k]] != 0;
        if (k < n)
        {
            converged[k] = f ? 1 : 0;
            if (f)
            {
                const double h = xyzh[k].w;
                hs[k] = h;
                const unsigned long long b = (unsigned long long)__double_as_longlong(h);
                hconv = b > hconv ? b : hconv;
            }
        }
        // a fixed particle has no row yet: one is made at its h with the others' at the end
        block_append(k < n ? (f ? 2 : 1) : -1, k, nullptr, nullptr, lists.build[0], &L->cnt[0].build, lists.cover,
                     &L->cover, sh);
    }
    note_h(0, hconv, ds, shH);
}

__global__ void near_active_kernel(NearLoop* L) { L->active = L->cnt[0].build; }

// A batch starts with the live particles of all its sets (each set's come first in its part
// of the sorted order) on the search list.
__global__ void near_forest_zero_kernel(NearLoop* L, int maxIter)
{
    L->queue[threadIdx.x] = 0;
    if (threadIdx.x != 0) return;
    L->iter = 0;
    L->maxIter = maxIter;
    L->active = 0;
    L->all = 0;
    L->cover = L->over = 0;
    L->cnt[0] = L->cnt[1] = NearCounts{0, 0, 0, 0};
    L->ticket[0] = L->ticket[1] = 0;
}

__global__ void __launch_bounds__(kThreads)
near_forest_init_kernel(NearLoop* L, int n, const NearSet* __restrict__ sets, const int* __restrict__ setOf,
                        const __grid_constant__ NearLists lists)
{
    __shared__ int sh[3 * (kNearWarps + 1)];
    for (int b = blockIdx.x * kThreads; b < n; b += gridDim.x * kThreads)
    {
        const int k = b + int(threadIdx.x);
        bool live = false;
        if (k < n)
        {
            const NearSet& s = sets[setOf[k]];
            live = k - s.p0 < s.n;
        }
        block_append(live ? 0 : -1, k, lists.build[0], &L->cnt[0].build, nullptr, nullptr, nullptr, nullptr, sh);
    }
}

// Particles the loop left on its next search and sum lists (its iterations ran out): their rows,
// if they have one, do not reach their last h.  They join the cover list, so that an
// evaluation at that h finds them a row or puts them on the over list, as the others.  (Those
// on its row list keep a row that reaches it.)
__global__ void __launch_bounds__(kThreads)
near_pending_kernel(NearLoop* L, const __grid_constant__ NearLists lists)
{
    const int cur = L->iter & 1;
    const NearCounts c = L->cnt[cur];
    const int n = c.build + c.sum + c.huge;
    for (int b = blockIdx.x * kThreads; b < n; b += gridDim.x * kThreads)
    {
        const int k = b + int(threadIdx.x);
        const int s = k - c.build, u = s - c.sum;
        const int v = k >= n ? 0 : (s < 0 ? lists.build[cur][k] : (u < 0 ? lists.sum[cur][s] : lists.huge[cur][u]));
        warp_append(k < n, v, lists.cover, &L->cover);
    }
}

// Work in nq queues of consecutive items, one a multiprocessor: the warps of a multiprocessor
// take items from its own queue, so at any time they search next to one another and find
// each other's blocks in its L1 cache; one whose queue is empty goes on with the first that
// is not.  own: the warp's queue.  The item, or -1 when none is left.
__device__ __forceinline__ int queue_pop(int* queue, int nq, int items, int& own)
{
    const int lane = lane_id();
    for (;;)
    {
        const int a = int((long long)items * own / nq), b = int((long long)items * (own + 1) / nq);
        int k = 0;
        if (lane == 0) k = a < b ? atomicAdd(queue + own, 1) : 0;
        k = __shfl_sync(0xffffffffu, k, 0);
        if (a + k < b) return a + k;
        int next = -1;
        for (int q0 = 0; q0 < nq && next < 0; q0 += 32)
        {
            const int q = q0 + lane < nq ? (own + 1 + q0 + lane) % nq : own;
            const int left = int((long long)items * (q + 1) / nq) - int((long long)items * q / nq);
            const uint32_t m = __ballot_sync(0xffffffffu,
                                             q != own && *reinterpret_cast<volatile int*>(queue + q) < left);
            if (m) next = __shfl_sync(0xffffffffu, q, __ffs(m) - 1);
        }
        if (next < 0) return -1;
        own = next;
    }
}

__device__ __forceinline__ int sm_id()
{
    int s;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(s));
    return s;
}

// ---------------------------------------------------------------- rows
// Rows of the listed particles (all live ones when the list is the identity): the members of
// a warp are up to 32 consecutive entries -- fewer where the list is short, so that it still
// spreads over the chip -- in runs that search together (near_runs).  Each member takes the
// blocks its own sphere reaches and tests 32 candidates per step with the exact FP64 test;
// what passes is written at once, consecutive entries by consecutive lanes.  A row that
// would exceed kNbl is given up (its count is kNbl + 1) and stops its member's search.
// Bound by issue: on a lattice about 6 steps of 28 instructions and 80 for the blocks per
// particle.
//   cover = 0: rows for the next Newton iteration; complete rows go to the row list, the
//              others to the list of direct sums.
//   cover = 1: rows at the converged h of particles left without; the others are listed
//              (over) and marked as covering everything (rowH infinite: no pair of theirs
//              is looked for from the other side).
template<bool Forest, bool Periodic>
__global__ void __launch_bounds__(kThreads, 7)
near_rows_kernel(const __grid_constant__ NearTree t, const NearSet* __restrict__ sets, const int* __restrict__ setOf,
                 NearLoop* __restrict__ L, const __grid_constant__ NearLists lists, double* __restrict__ rowsR2,
                 int* __restrict__ rowsJ, int* __restrict__ nblCount, double* __restrict__ rowH, int cover, int nq)
{
    __shared__ NearScratch sScr[kNearWarps];
    const int lane = lane_id(), wib = threadIdx.x >> 5, sub = lane >> 3, off = lane & 7;
    const uint32_t lt = (1u << lane) - 1u;
    NearScratch& scr = sScr[wib];
    const int cur = L->iter & 1;
    const int n = cover ? L->cover : L->cnt[cur].build;
    if (n == 0) return;
    const int* list = cover ? lists.cover : (L->all ? nullptr : lists.build[cur]);
    const double margin = cover ? kCoverMargin : kNearMargin;
    const double wide2 = kRadK2 * (margin * margin);
    NearFrame f(t.box);
    NearView v = Forest ? NearView{0, 0, 0, 0.0f, 0.0f, 0.0f} : near_view(t, f);
    double lx = 0, ly = 0, lz = 0;
    if (Periodic && !Forest) { lx = t.box->len[0]; ly = t.box->len[1]; lz = t.box->len[2]; }
    int g = 32;
    while (g > 1 && n < g * int(gridDim.x) * kNearWarps) g >>= 1;
    int own = sm_id() % nq;
    for (;;)
    {
        const int w = queue_pop(L->queue, nq, (n + g - 1) / g, own);
        if (w < 0) break;
        const int at = w * g + lane;
        const bool mine = lane < g && at < n;
        const int i = mine ? (list ? list[at] : at) : 0;
        const int set = Forest ? setOf[i] : 0;
        const double4 pi = t.xyzh[i];
        if constexpr (Forest) f = NearFrame(sets[set]);
        const float3 rel = f.at(pi);
        const float x = rel.x, y = rel.y, z = rel.z;
        const float r = mine ? f.length(kRadKernel * margin * (1.0 + 1e-6) * pi.w) + f.slack(x, y, z) : -1.0f;
        scr.P[lane] = make_double4(pi.x, pi.y, pi.z, 1.0 / (pi.w * pi.w));
        scr.Q[lane] = make_float4(x, y, z, r * r * 1.000001f);
        // a member much wider than the others (a scattered h) searches by itself, after them
        const uint32_t all = __ballot_sync(0xffffffffu, mine);
        float mean = mine ? r : 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mean += __shfl_xor_sync(0xffffffffu, mean, o);
        uint32_t wide = __ballot_sync(0xffffffffu, mine && r * float(__popc(all)) > kNearWide * mean);
        const NearRun run = near_runs<Forest>(x, y, z, (wide >> lane) & 1u ? -1.0f : r, set);
        int rowLen = 0;
        uint32_t todo = all;
        __syncwarp();
        for (int a = 0; todo; a += run.w)
        {
            uint32_t members;
            float bx, by, bz, ex, ey, ez, reach;
            if (a < 32)
            {
                members = todo & ~wide & ((run.w == 32 ? 0xffffffffu : ((1u << run.w) - 1u)) << a);
                if (members == 0u) continue;
                bx = __shfl_sync(0xffffffffu, run.cx, a); ex = __shfl_sync(0xffffffffu, run.ex, a);
                by = __shfl_sync(0xffffffffu, run.cy, a); ey = __shfl_sync(0xffffffffu, run.ey, a);
                bz = __shfl_sync(0xffffffffu, run.cz, a); ez = __shfl_sync(0xffffffffu, run.ez, a);
                reach = __shfl_sync(0xffffffffu, run.reach, a);
            }
            else
            {
                const int p = __ffs(todo) - 1;
                members = 1u << p;
                bx = __shfl_sync(0xffffffffu, x, p);
                by = __shfl_sync(0xffffffffu, y, p);
                bz = __shfl_sync(0xffffffffu, z, p);
                reach = __shfl_sync(0xffffffffu, r, p);
                ex = ey = ez = 0.0f;
            }
            if constexpr (Forest)
            {
                const int sid = __shfl_sync(0xffffffffu, set, __ffs(members) - 1);
                const NearSet& st = sets[sid];
                v = NearView{st.p0, sid, st.n, st.lx, st.ly, st.lz};
                lx = st.dlx; ly = st.dly; lz = st.dlz;
            }
            const double4* at0 = t.xyzh + v.p0;
            bool apart = false;
            int batches = 0, hits = 0;
            float shared = 0.0f;
            near_blocks<0, Periodic, false>(t, v, scr, bx, by, bz, ex, ey, ez, reach, 0.0f, [&](int nb) -> float {
                // the blocks of this batch, kNearBlocks / 32 per lane
                constexpr int kU = kNearBlocks / 32;
                NearNode nd[kU];
                int id[kU];
#pragma unroll
                for (int u = 0; u < kU; ++u)
                {
                    const int k = 32 * u + lane;
                    id[u] = k < nb ? scr.blk[k] : -1;
                    if (32 * u < nb) nd[u] = ld_node(near_node(t, v, 0, max(id[u], 0)));
                }
                bool dropped = false;
                const int searching = __popc(todo & members);
                for (uint32_t rest = todo & members; rest; rest &= rest - 1)
                {
                    const int p = __ffs(rest) - 1;
                    const float4 q = scr.Q[p];
                    int ns = 0;
#pragma unroll
                    for (int u = 0; u < kU; ++u)
                    {
                        if (32 * u >= nb) break;
                        const bool hit = id[u] >= 0 &&
                                         near_gap2<Periodic>(q.x, q.y, q.z, 0.0f, 0.0f, 0.0f, nd[u], v) <= q.w;
                        const uint32_t m = __ballot_sync(0xffffffffu, hit);
                        st_shared_if(hit, scr.sel + ns + __popc(m & lt), id[u]);
                        ns += __popc(m);
                    }
                    if (ns == 0) continue;
                    hits += ns;
                    st_shared_if(lane < 8, scr.sel + ns + lane, kNearNone);
                    __syncwarp();
                    const double4 gp = scr.P[p];
                    const size_t row = size_t(__shfl_sync(0xffffffffu, i, p)) * kNbl;
                    double* outR = rowsR2 + row;
                    int* outJ = Forest ? nullptr : rowsJ + row;
                    int len = __shfl_sync(0xffffffffu, rowLen, p);
                    auto fetch = [&](int k, double4& pj, int& j) {
                        j = scr.sel[k + sub] * 8 + off;
                        pj = ldg4(at0 + min(j, v.n - 1));
                    };
                    // an entry beyond the row's room lands on its last one: the row is given up
                    auto take = [&](const double4& pj, int j) {
                        double dx = gp.x - pj.x, dy = gp.y - pj.y, dz = gp.z - pj.z;
                        nearest_image<Periodic>(dx, dy, dz, lx, ly, lz);
                        const double r2 = pair_r2(dx, dy, dz);
                        const bool acc = j < v.n && r2 * gp.w < wide2;
                        const uint32_t m = __ballot_sync(0xffffffffu, acc);
                        const int k = min(len + __popc(m & lt), kNbl - 1);
                        len += __popc(m);
                        st_if(acc, outR + k, r2);
                        if (!Forest) st_if(acc, outJ + k, j);
                    };
                    // two sets of registers in turn: a step's loads are in flight while the one
                    // before it is tested
                    double4 pa, pb;
                    int ja, jb;
                    fetch(0, pa, ja);
                    for (int k = 0; k < ns; k += 8)
                    {
                        fetch(k + 4, pb, jb);
                        take(pa, ja);
                        if (k + 4 >= ns) break;
                        fetch(k + 8, pa, ja);
                        take(pb, jb);
                    }
                    if (lane == p) rowLen = len;
                    if (len > kNbl)
                    {
                        todo &= ~(1u << p);
                        dropped = true;
                    }
                    __syncwarp();
                }
                // members that reach little of batch after batch: what lies between them (the flank
                // of a concentrated set) is tested by all of them, so they go on one by one,
                // from the start
                shared += float(searching) * float(nb);
                if (++batches == kNearPatience && searching > 1 && float(hits) < kNearShare * shared)
                {
                    if (((todo & members) >> lane) & 1u) rowLen = 0;
                    wide |= todo & members;
                    apart = true;
                    return -1.0f;
                }
                if (!dropped) return reach;
                // the members still searching may need less
                return warp_max_f(((todo & members) >> lane) & 1u ? r : -1.0f);
            });
            if (!apart) todo &= ~members;
            __syncwarp();
        }
        const bool full = mine && rowLen > kNbl;
        if (mine)
        {
            nblCount[i] = full ? kNbl + 1 : rowLen;
            rowH[i] = full ? (cover ? double(INFINITY) : 0.0) : margin * pi.w * (1.0 - 1e-12);
        }
        if (cover)
            warp_append(full, i, lists.over, &L->over);
        else
        {
            warp_append(mine && !full, i, lists.row[cur], &L->cnt[cur].row);
            warp_append(full, i, lists.sum[cur], &L->cnt[cur].sum);
        }
        __syncwarp();
    }
}

// Where a particle goes after its Newton step (the lists of block_append).  Converged: to the
// cover list when its row does not cover its h for the gradient and force passes, else
// nowhere.  Otherwise its next iteration is from its row while h stays inside the row's
// reach, from a new one beyond.
__device__ __forceinline__ int next_of(bool conv, double ho, double rowHi)
{
    if (conv) return ho * kCoverSlack <= rowHi ? -1 : 2;
    return ho <= rowHi ? 0 : 1;
}

// W and -q dW/dq - 3W of m records of q^2, one per lane.
__device__ __forceinline__ void eval_records(double2* rec, int m)
{
    for (int k = threadIdx.x & 31; k < m; k += 32)
    {
        const double q2 = rec[k].x;
        const double q = sqrt(q2);
        double wk, dwk;
        sph_kernel(q2, q, wk, dwk);
        rec[k] = make_double2(wk, -q * dwk - 3.0 * wk);
    }
}

// The records' two components added to the two sums one by one (even lanes one sum, odd lanes
// the other).
__device__ __forceinline__ double2 serial_add(const double2* rec, int m, double2 s)
{
    const bool odd = threadIdx.x & 1;
    const double* v = reinterpret_cast<const double*>(rec) + (odd ? 1 : 0);
    double t = odd ? s.y : s.x;
#pragma unroll 8
    for (int k = 0; k < m; ++k) t += v[2 * k];
    return make_double2(__shfl_sync(0xffffffffu, t, 0), __shfl_sync(0xffffffffu, t, 1));
}

// One Newton iteration from the rows.  Warp = false: one lane per particle streams its own row
// (8 bytes an entry), tests every entry with the exact test and adds in the row's order.
// Warp: one warp per particle (a small set), an entry per lane, the accepted values packed in
// order and then added one by one.
template<bool Forest, bool Warp>
__global__ void __launch_bounds__(kThreads)
near_step_kernel(const NearSet* __restrict__ sets, const int* __restrict__ setOf, NearLoop* __restrict__ L,
                 const __grid_constant__ NearLists lists, const double* __restrict__ rowsR2,
                 const int* __restrict__ nblCount, const double* __restrict__ rowH, double4* __restrict__ xyzh,
                 double* __restrict__ rho, double* __restrict__ gradh, int* __restrict__ converged,
                 double* __restrict__ hs, double pmass, double tolh, double hfact, DevScalars* __restrict__ ds)
{
    __shared__ int sh[3 * (kNearWarps + 1)];
    __shared__ unsigned long long shH[2];
    __shared__ double2 sRec[Warp ? kNearWarps : 1][Warp ? kNbl : 1];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int cur = L->iter & 1, nxt = cur ^ 1;
    const int n = L->cnt[cur].row;
    if (n == 0) return;
    const int* list = lists.row[cur];
    unsigned long long pairs = 0, seen = 0, hconv = 0;
    const int perBlock = Warp ? kNearWarps : kThreads;
    for (int b = blockIdx.x * perBlock; b < n; b += gridDim.x * perBlock)
    {
        const int at = b + (Warp ? wib : int(threadIdx.x));
        int to = -1;
        int i = 0;
        if (at < n)
        {
            i = list[at];
            const double hi = xyzh[i].w;
            const double hinv2 = 1.0 / (hi * hi);
            const double rh = rowH[i];
            double sr = 0.0, sg = 0.0;
            unsigned int gp = 0;
            const double* row = row_flat(rowsR2, uint32_t(i));
            const int cnt = nblCount[i];
            if constexpr (Warp)
            {
                double2* rec = sRec[wib];
                for (int k0 = 0; k0 < cnt; k0 += 32)
                {
                    const bool valid = k0 + lane < cnt;
                    const double q2 = (valid ? row[k0 + lane] : 0.0) * hinv2;
                    const bool acc = valid && q2 < kRadK2;
                    const uint32_t m = __ballot_sync(0xffffffffu, acc);
                    if (acc) rec[gp + __popc(m & ((1u << lane) - 1u))].x = q2;
                    gp += __popc(m);
                }
                __syncwarp();
                eval_records(rec, int(gp));
                __syncwarp();
                const double2 s = serial_add(rec, int(gp), make_double2(0.0, 0.0));
                sr = s.x;
                sg = s.y;
            }
            else
                for_flat_row(row, cnt, [&](double r2) {
                    const double q2 = r2 * hinv2;
                    if (!(q2 < kRadK2)) return;
                    ++gp;
                    const double q = sqrt(q2);
                    double wk, dwk;
                    sph_kernel(q2, q, wk, dwk);
                    sr += wk;
                    sg += -q * dwk - 3.0 * wk;
                });
            double ro, go, ho;
            int conv;
            newton_step(sr, sg, hi, Forest ? sets[setOf[i]].pmass : pmass, hfact, tolh, ro, go, ho, conv);
            if (!Warp || lane == 0)
            {
                pairs += gp;
                rho[i] = ro;
                gradh[i] = go;
                reinterpret_cast<double*>(xyzh + i)[3] = ho;
                const unsigned long long hb = (unsigned long long)__double_as_longlong(hi);
                const unsigned long long ob = (unsigned long long)__double_as_longlong(ho);
                seen = hb > seen ? hb : seen;
                if (conv)
                {
                    converged[i] = 1;
                    hs[i] = ho;
                    hconv = ob > hconv ? ob : hconv;
                }
                to = next_of(conv != 0, ho, rh);
            }
            if (Warp) __syncwarp();
        }
        block_append(to, i, lists.row[nxt], &L->cnt[nxt].row, lists.build[nxt], &L->cnt[nxt].build, lists.cover,
                     &L->cover, sh);
    }
    note_h(seen, hconv, ds, shH);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
    if (lane == 0 && pairs) atomicAdd(&ds->pairs[0], pairs);
}

// rho and d(rho)/dh at h from the un-normalised sums (src/density_base.cu:635-643).
__device__ __forceinline__ void eval_store(int i, double hi, double sr, double sg, double pmass,
                                           double* __restrict__ rho, double* __restrict__ gradh)
{
    const double hi1 = 1.0 / hi;
    const double hi31 = hi1 * hi1 * hi1;
    rho[i] = sr * kCnormk * pmass * hi31;
    gradh[i] = sg * kCnormk * pmass * (hi31 * hi1);
}

// The same for every live particle of a batch with a row, at its final h.
__global__ void __launch_bounds__(kThreads)
near_eval_kernel(int n, const NearSet* __restrict__ sets, const int* __restrict__ setOf,
                 const double* __restrict__ rowsR2, const int* __restrict__ nblCount, const double4* __restrict__ xyzh,
                 double* __restrict__ rho, double* __restrict__ gradh, DevScalars* __restrict__ ds)
{
    unsigned int gp = 0;
    const int i = blockIdx.x * kThreads + int(threadIdx.x);
    if (i < n)
    {
        const NearSet& s = sets[setOf[i]];
        if (i - s.p0 < s.n && unsigned(nblCount[i]) <= unsigned(kNbl))
        {
            const double hi = xyzh[i].w;
            const double hinv2 = 1.0 / (hi * hi);
            double sr = 0.0, sg = 0.0;
            for_flat_row(row_flat(rowsR2, uint32_t(i)), nblCount[i], [&](double r2) {
                const double q2 = r2 * hinv2;
                if (!(q2 < kRadK2)) return;
                ++gp;
                const double q = sqrt(q2);
                double wk, dwk;
                sph_kernel(q2, q, wk, dwk);
                sr += wk;
                sg += -q * dwk - 3.0 * wk;
            });
            eval_store(i, hi, sr, sg, s.pmass, rho, gradh);
        }
    }
    unsigned long long pairs = gp;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
    if ((threadIdx.x & 31) == 0 && pairs) atomicAdd(&ds->pairs[0], pairs);
}

// ---------------------------------------------------------------- direct sums
// A particle whose neighbours do not fit a row is summed straight from its search: accepted
// q^2 are packed into a record buffer in ascending j, evaluated one per lane, and W and
// -q dW/dq - 3W added in order.
constexpr int kNearRec = 256;        // records of one ordered sum
constexpr int kHugeWarps = 8;        // warps that share a particle of very many neighbours
constexpr unsigned int kHuge = 4096; // as many neighbours and more

// Successive rounded additions of v[0 .. m) to s, in parallel.  While the running sum stays
// in one binade, each addition rounds its term to a multiple u of that binade's last place
// and adds it exactly, so the rounded terms may be added in any order.  t = (w + C) - C with
// C = 1.5 * 2^e is that rounding (to nearest even).  A term exactly halfway (|w - t| = u/2)
// rounds by the parity of the running sum instead, and a sum that might leave the binade
// changes u: then ok is false and the terms must be added one by one.  up and down: the sums
// of the positive and the negative rounded terms (multiples of u, exact while below 2^e).
struct OrderedPart
{
    double up, down;
    bool ok;
};

struct Binade
{
    double a, lo, u, sign;   // |s|, 2^e <= |s| < 2^(e+1), 2^(e-52), the sign of s
    bool ok;
    __device__ __forceinline__ explicit Binade(double s)
    {
        a = fabs(s);
        sign = s < 0.0 ? -1.0 : 1.0;
        const int e = int(__double_as_longlong(a) >> 52);
        ok = e >= 64 && e <= 2000;   // not zero, tiny, huge, infinite or NaN
        lo = __longlong_as_double((long long)(ok ? e : 1023) << 52);
        u = lo * 2.220446049250313e-16;
    }
    // whether terms of these sums keep every partial sum inside the binade
    __device__ __forceinline__ bool holds(double up, double down) const
    {
        return up < lo && down < lo && a + up + 512.0 * u < 2.0 * lo && a - down - 512.0 * u >= lo;
    }
};

// Component c of the records, by one warp.
__device__ __forceinline__ OrderedPart ordered_part(const double2* rec, int c, int m, const Binade& b)
{
    const int lane = threadIdx.x & 31;
    const double C = 1.5 * b.lo, half = 0.5 * b.lo, tie = 0.5 * b.u;
    OrderedPart r{0.0, 0.0, b.ok};
#pragma unroll
    for (int k = 0; k < kNearRec / 32; ++k)
    {
        const int at = 32 * k + lane;
        const double w = at < m ? b.sign * (c ? rec[at].y : rec[at].x) : 0.0;
        const double t = (w + C) - C;
        r.ok = r.ok && fabs(w) < half && fabs(w - t) != tie;
        r.up += fmax(t, 0.0);
        r.down += fmax(-t, 0.0);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
    {
        r.up += __shfl_xor_sync(0xffffffffu, r.up, o);
        r.down += __shfl_xor_sync(0xffffffffu, r.down, o);
    }
    r.ok = __all_sync(0xffffffffu, r.ok);
    return r;
}

// The records' two components added to the two sums in order, by one warp: in parallel where
// a full buffer allows it, else one by one (even lanes one sum, odd lanes the other).
__device__ __forceinline__ double2 ordered_add(const double2* rec, int m, double2 s)
{
    bool doneW = false, doneG = false;
    if (m == kNearRec)
    {
        const Binade bw(s.x), bg(s.y);
        const OrderedPart w = ordered_part(rec, 0, m, bw), g = ordered_part(rec, 1, m, bg);
        if (w.ok && bw.holds(w.up, w.down)) { s.x = bw.sign * ((bw.a + w.up) - w.down); doneW = true; }
        if (g.ok && bg.holds(g.up, g.down)) { s.y = bg.sign * ((bg.a + g.up) - g.down); doneG = true; }
        if (doneW && doneG) return s;
    }
    const double2 one = serial_add(rec, m, s);
    return make_double2(doneW ? s.x : one.x, doneG ? s.y : one.y);
}

// m records of q^2 evaluated and added to the sums in order.
__device__ __noinline__ double2 near_add_records(double2* rec, int m, double2 s)
{
    __syncwarp();
    eval_records(rec, m);
    __syncwarp();
    s = ordered_add(rec, m, s);
    __syncwarp();
    return s;
}

// The Newton step of a directly summed particle, by one thread: stored, and the particle put
// on its next list by how many neighbours it had (got): enough room in a row once made,
// one warp's work, or a block's.
__device__ __forceinline__ void sum_finish(int i, double hi, double2 sums, unsigned int got, NearLoop* L,
                                           const NearLists& lists, int nxt, double4* xyzh, double* rho, double* gradh,
                                           int* converged, double* hs, double* rowH, double pmass, double tolh,
                                           double hfact, unsigned long long& seen, unsigned long long& hconv)
{
    double ro, go, ho;
    int conv;
    newton_step(sums.x, sums.y, hi, pmass, hfact, tolh, ro, go, ho, conv);
    rho[i] = ro;
    gradh[i] = go;
    reinterpret_cast<double*>(xyzh + i)[3] = ho;
    const unsigned long long hb = (unsigned long long)__double_as_longlong(hi);
    const unsigned long long ob = (unsigned long long)__double_as_longlong(ho);
    seen = hb > seen ? hb : seen;
    if (conv)
    {
        converged[i] = 1;
        hs[i] = ho;
        hconv = ob > hconv ? ob : hconv;
        if (got > kNbl)
        {
            // no row would hold them: it is among those without one at once (near_rows_kernel,
            // which counted kNbl + 1 for it, would find that out by another search)
            rowH[i] = double(INFINITY);
            lists.over[atomicAdd(&L->over, 1)] = i;
        }
        else
            lists.cover[atomicAdd(&L->cover, 1)] = i;
        return;
    }
    const double ratio = ho / hi, expect = double(got) * ratio * ratio * ratio;
    if (expect * (kNearMargin * kNearMargin * kNearMargin) < 0.95 * kNbl)
        lists.build[nxt][atomicAdd(&L->cnt[nxt].build, 1)] = i;
    else if (expect < double(kHuge))
        lists.sum[nxt][atomicAdd(&L->cnt[nxt].sum, 1)] = i;
    else
        lists.huge[nxt][atomicAdd(&L->cnt[nxt].huge, 1)] = i;
}

// One Newton iteration of the particles whose neighbours do not fit a row, one warp each.
// One that turns out to have kHuge of them is left to the block kernel.  Eval: rho and
// d(rho)/dh of the particles without a row (over list) at their h instead.
template<bool Forest, bool Periodic, bool Eval>
__global__ void __launch_bounds__(kThreads, 5)
near_sum_kernel(const __grid_constant__ NearTree t, const NearSet* __restrict__ sets,
                const int* __restrict__ setOf, NearLoop* __restrict__ L,
                const __grid_constant__ NearLists lists, double4* __restrict__ xyzh,
                double* __restrict__ rho, double* __restrict__ gradh, int* __restrict__ converged,
                double* __restrict__ hs, double* __restrict__ rowH, double pmass, double tolh, double hfact,
                DevScalars* __restrict__ ds)
{
    __shared__ NearScratch sScr[kNearWarps];
    __shared__ double2 sRec[kNearWarps][kNearRec];
    __shared__ unsigned long long shH[2];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    NearScratch& scr = sScr[wib];
    double2* rec = sRec[wib];
    const int cur = L->iter & 1, nxt = cur ^ 1;
    const int n = Eval ? L->over : L->cnt[cur].sum;
    if (n == 0) return;
    const int* list = Eval ? lists.over : lists.sum[cur];
    const unsigned int most = Eval ? 0xffffffffu : kHuge;
    NearFrame f(t.box);
    NearView v = Forest ? NearView{0, 0, 0, 0.0f, 0.0f, 0.0f} : near_view(t, f);
    double lx = 0, ly = 0, lz = 0;
    if (Periodic && !Forest) { lx = t.box->len[0]; ly = t.box->len[1]; lz = t.box->len[2]; }
    unsigned long long pairs = 0, seen = 0, hconv = 0;
    for (;;)
    {
        int w = 0;
        if (lane == 0) w = atomicAdd(&L->ticket[0], 1);
        w = __shfl_sync(0xffffffffu, w, 0);
        if (w >= n) break;
        const int i = list[w];
        const double4 pi = xyzh[i];
        if constexpr (Forest)
        {
            const int sid = setOf[i];
            const NearSet& st = sets[sid];
            f = NearFrame(st);
            v = NearView{st.p0, sid, st.n, st.lx, st.ly, st.lz};
            lx = st.dlx; ly = st.dly; lz = st.dlz;
            pmass = st.pmass;
        }
        const double4* at0 = t.xyzh + v.p0;
        const double hi = pi.w, hinv2 = 1.0 / (hi * hi);
        const float3 a = f.at(pi);
        const float x = a.x, y = a.y, z = a.z;
        const float r = f.length(kRadKernel * (1.0 + 1e-6) * hi) + f.slack(x, y, z);
        double2 sums = make_double2(0.0, 0.0);
        int nrec = 0;
        unsigned int got = 0;
        near_blocks<0, Periodic, false>(t, v, scr, x, y, z, 0.0f, 0.0f, 0.0f, r, 0.0f, [&](int nb) -> float {
            near_candidates(scr.blk, nb, v.n, at0, [&](const double4& pj, int, bool valid) {
                double dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
                nearest_image<Periodic>(dx, dy, dz, lx, ly, lz);
                const double q2 = pair_r2(dx, dy, dz) * hinv2;
                const bool acc = valid && q2 < kRadK2;
                const uint32_t m = __ballot_sync(0xffffffffu, acc);
                const int k = nrec + __popc(m & lt);
                if (acc && k < kNearRec) rec[k].x = q2;
                nrec += __popc(m);
                if (nrec >= kNearRec)
                {
                    sums = near_add_records(rec, kNearRec, sums);
                    got += kNearRec;
                    nrec -= kNearRec;   // those beyond the buffer start the next one
                    if (acc && k >= kNearRec) rec[k - kNearRec].x = q2;
                    __syncwarp();
                }
                return got < most;
            });
            return got < most ? r : -1.0f;
        });
        if (got >= most)
        {
            if (lane == 0) lists.huge[cur][atomicAdd(&L->cnt[cur].huge, 1)] = i;
            __syncwarp();
            continue;
        }
        sums = near_add_records(rec, nrec, sums);
        got += nrec;
        if (lane == 0)
        {
            pairs += got;
            if constexpr (Eval) eval_store(i, hi, sums.x, sums.y, pmass, rho, gradh);
            else
                sum_finish(i, hi, sums, got, L, lists, nxt, xyzh, rho, gradh, converged, hs, rowH, pmass, tolh, hfact,
                           seen, hconv);
        }
        __syncwarp();
    }
    if constexpr (!Eval) note_h(seen, hconv, ds, shH);
    if (lane == 0 && pairs) atomicAdd(&ds->pairs[0], pairs);
}

// The same for a particle of very many neighbours (the widest supports of a scattered start
// reach whole sets), one block each: the first warp walks the tree down to its 64-particle
// nodes, every warp takes four of them at a time, and the warps' record buffers are added in
// the warps' order -- together where all fit one binade without a tie, else one buffer after
// the other.  Alone on one warp such a particle took 17 ns a neighbour, 2 ms for the widest
// of 120,000 particles, which was the length of the iteration.
template<bool Forest, bool Periodic>
__global__ void __launch_bounds__(32 * kHugeWarps)
near_huge_kernel(const __grid_constant__ NearTree t, const NearSet* __restrict__ sets,
                const int* __restrict__ setOf, NearLoop* __restrict__ L,
                 const __grid_constant__ NearLists lists, double4* __restrict__ xyzh,
                 double* __restrict__ rho, double* __restrict__ gradh, int* __restrict__ converged,
                 double* __restrict__ hs, double* __restrict__ rowH, double pmass, double tolh, double hfact,
                 DevScalars* __restrict__ ds)
{
    __shared__ NearScratch scr;
    __shared__ double2 sRec[kHugeWarps][kNearRec];
    __shared__ int sSel[kHugeWarps][32];
    __shared__ OrderedPart sPart[kHugeWarps][2];
    __shared__ int sCount[kHugeWarps];
    __shared__ int sItem, sNodes;
    __shared__ double2 sSums;
    __shared__ unsigned long long shH[2];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    const int cur = L->iter & 1, nxt = cur ^ 1;
    const int n = L->cnt[cur].huge;
    if (n == 0) return;
    NearFrame f(t.box);
    NearView v = Forest ? NearView{0, 0, 0, 0.0f, 0.0f, 0.0f} : near_view(t, f);
    double lx = 0, ly = 0, lz = 0;
    if (Periodic && !Forest) { lx = t.box->len[0]; ly = t.box->len[1]; lz = t.box->len[2]; }
    double2* rec = sRec[wib];
    unsigned long long pairs = 0, seen = 0, hconv = 0;
    for (;;)
    {
        __syncthreads();
        if (threadIdx.x == 0)
        {
            sItem = atomicAdd(&L->ticket[1], 1);
            sSums = make_double2(0.0, 0.0);
        }
        __syncthreads();
        if (sItem >= n) break;
        const int i = lists.huge[cur][sItem];
        const double4 pi = xyzh[i];
        if constexpr (Forest)
        {
            const int sid = setOf[i];
            const NearSet& st = sets[sid];
            f = NearFrame(st);
            v = NearView{st.p0, sid, st.n, st.lx, st.ly, st.lz};
            lx = st.dlx; ly = st.dly; lz = st.dlz;
            pmass = st.pmass;
        }
        const double4* at0 = t.xyzh + v.p0;
        const double hi = pi.w, hinv2 = 1.0 / (hi * hi);
        const float3 a = f.at(pi);
        const float x = a.x, y = a.y, z = a.z;
        const float r = f.length(kRadKernel * (1.0 + 1e-6) * hi) + f.slack(x, y, z);
        const float r2max = r * r * 1.000001f;
        unsigned int got = 0;   // of this warp
        // the whole block over the 64-particle nodes scr.blk[0 .. cnt)
        auto work = [&](int cnt) {
            for (int c0 = 0; c0 < cnt; c0 += 4 * kHugeWarps)
            {
                const int at = c0 + 4 * wib + (lane >> 3);
                const int id = at < cnt ? scr.blk[at] * 8 + (lane & 7) : -1;
                bool hit = id >= 0 && id < near_count(v.n, 0);
                if (hit)
                    hit = near_gap2<Periodic>(x, y, z, 0.0f, 0.0f, 0.0f, ld_node(near_node(t, v, 0, id)), v) <= r2max;
                const uint32_t hm = __ballot_sync(0xffffffffu, hit);
                if (hit) sSel[wib][__popc(hm & lt)] = id;
                __syncwarp();
                int m = 0;
                if (hm)
                    near_candidates(sSel[wib], __popc(hm), v.n, at0, [&](const double4& pj, int, bool valid) {
                        double dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
                        nearest_image<Periodic>(dx, dy, dz, lx, ly, lz);
                        const double q2 = pair_r2(dx, dy, dz) * hinv2;
                        const bool acc = valid && q2 < kRadK2;
                        const uint32_t am = __ballot_sync(0xffffffffu, acc);
                        if (acc) rec[m + __popc(am & lt)].x = q2;   // at most 32 blocks of 8: kNearRec
                        m += __popc(am);
                        return true;
                    });
                got += m;
                __syncwarp();
                eval_records(rec, m);
                __syncwarp();
                const Binade bw(sSums.x), bg(sSums.y);
                const OrderedPart pw = ordered_part(rec, 0, m, bw), pg = ordered_part(rec, 1, m, bg);
                if (lane == 0) { sPart[wib][0] = pw; sPart[wib][1] = pg; sCount[wib] = m; }
                __syncthreads();
                if (wib == 0)
                {
                    double2 s = sSums;
                    bool okW = true, okG = true;
                    double uw = 0.0, dw = 0.0, ug = 0.0, dg = 0.0;
                    for (int k = 0; k < kHugeWarps; ++k)
                    {
                        okW = okW && sPart[k][0].ok; okG = okG && sPart[k][1].ok;
                        uw += sPart[k][0].up; dw += sPart[k][0].down;
                        ug += sPart[k][1].up; dg += sPart[k][1].down;
                    }
                    okW = okW && bw.holds(uw, dw);
                    okG = okG && bg.holds(ug, dg);
                    if (!okW || !okG)
                        for (int k = 0; k < kHugeWarps; ++k) s = ordered_add(sRec[k], sCount[k], s);
                    if (okW) s.x = bw.sign * ((bw.a + uw) - dw);
                    if (okG) s.y = bg.sign * ((bg.a + ug) - dg);
                    if (lane == 0) sSums = s;
                }
                __syncthreads();
            }
        };
        if (wib == 0)
        {
            near_blocks<1, Periodic, false>(t, v, scr, x, y, z, 0.0f, 0.0f, 0.0f, r, 0.0f, [&](int nb) -> float {
                if (lane == 0) sNodes = nb;
                __syncthreads();
                work(nb);
                return r;
            });
            if (lane == 0) sNodes = 0;
            __syncthreads();
        }
        else
            for (;;)
            {
                __syncthreads();
                const int cnt = sNodes;
                if (cnt == 0) break;
                work(cnt);
            }
        // the warps' counts (each lane holds its warp's)
        if (lane == 0) sCount[wib] = int(got);
        __syncthreads();
        if (threadIdx.x == 0)
        {
            unsigned int all = 0;
            for (int k = 0; k < kHugeWarps; ++k) all += unsigned(sCount[k]);
            pairs += all;
            sum_finish(i, hi, sSums, all, L, lists, nxt, xyzh, rho, gradh, converged, hs, rowH, pmass, tolh, hfact,
                       seen, hconv);
        }
    }
    note_h(seen, hconv, ds, shH);
    if (threadIdx.x == 0 && pairs) atomicAdd(&ds->pairs[0], pairs);
}

// End of an iteration: what it left active, the next one's lists in place, and whether it
// runs (the graph's while condition when run as a graph).
__global__ void near_epilogue_kernel(NearLoop* L, cudaGraphConditionalHandle more, int setCondition)
{
    L->queue[threadIdx.x] = 0;
    if (threadIdx.x != 0) return;
    const int it = L->iter, cur = it & 1, nxt = cur ^ 1;
    if (it < kLoopIters) L->activePerIter[it] = L->active;
    L->cnt[cur] = NearCounts{};
    L->ticket[0] = L->ticket[1] = 0;
    L->all = 0;
    L->active = L->cnt[nxt].row + L->cnt[nxt].build + L->cnt[nxt].sum + L->cnt[nxt].huge;
    L->iter = it + 1;
    if (setCondition) cudaGraphSetConditional(more, L->active > 0 && it + 1 < L->maxIter ? 1u : 0u);
}

} // namespace

// ---------------------------------------------------------------- host side
// The block trees of n particles in nsets sets: where each level starts, and the nodes in all.
static size_t near_layout(int n, int nsets, NearTree& t)
{
    size_t off = 0;
    for (int l = 0; l < kNearLevels; ++l)
    {
        t.off[l] = int(off);
        off += size_t(n >> (3 * l + 3)) + nsets + 1;
    }
    return off;
}

NearTree near_tree(State& s)
{
    NearTree t;
    near_layout(s.ngas, 1, t);
    t.node = reinterpret_cast<const NearNode*>(s.nearNode.get());
    t.xyzh = s.xyzh.get();
    t.box = s.box.get();
    t.nLive = &s.dscal.get()->nAlive;
    return t;
}

// The block tree of the sorted particles (their positions stay while a solve's h change;
// the boxes' h are those of the last call).
void near_build(State& s)
{
    const int n = std::max(s.ngas, 1);
    NearTree t;
    s.nearNode.resize(near_layout(n, 1, t) * (sizeof(NearNode) / sizeof(float4)), s.st);
    t = near_tree(s);
    NearNode* out = reinterpret_cast<NearNode*>(s.nearNode.get());
    const int slots = iceil(n, 512);
    near_leaf_levels_kernel<false><<<std::min(slots, 8 * s.numSMs), 512, 0, s.st>>>(t, out, nullptr, 1, slots);
    COSMO_LAUNCHED();
    if (n > 512 * 32)
    {
        near_upper_levels_kernel<false><<<1, 1024, 0, s.st>>>(t, out, nullptr);
        COSMO_LAUNCHED();
    }
}

static NearLists near_lists(State& s)
{
    NearLists l;
    for (int k = 0; k < 2; ++k)
    {
        l.row[k] = s.nearRow[k].get();
        l.build[k] = s.nearBuild[k].get();
        l.sum[k] = s.nearSum[k].get();
        l.huge[k] = s.nearHuge[k].get();
    }
    l.cover = s.nearCover.get();
    l.over = s.nearOver.get();
    return l;
}

// The buffers a loop over n particles needs beside the particles' own.
static void near_buffers(State& s, int n)
{
    for (auto* b : {&s.nearRow[0], &s.nearRow[1], &s.nearBuild[0], &s.nearBuild[1], &s.nearSum[0], &s.nearSum[1],
                    &s.nearHuge[0], &s.nearHuge[1], &s.nearCover, &s.nearOver})
        b->resize(n, s.st);
    s.hs.resize(n, s.st);
    s.nearLoop.resize(1, s.st);
}

// The instance of a kernel a job needs: one set, open or periodic, or the sets of a batch.
#define NEAR_PICK(kern, job, ...) \
    ((job).sets != nullptr ? kern<true, true __VA_ARGS__> \
                           : ((job).periodic ? kern<false, true __VA_ARGS__> : kern<false, false __VA_ARGS__>))
#define NEAR_COMMA ,

// One iteration's kernels, in the stream's order.
static void near_iteration(State& s, const NearJob& j, cudaGraphConditionalHandle more, int setCondition)
{
    const NearLists lists = near_lists(s);
    NearLoop* L = s.nearLoop.get();
    DevScalars* ds = s.dscal.get();
    auto rows = NEAR_PICK(near_rows_kernel, j);
    rows<<<persistent_blocks(s, rows, kThreads), kThreads, 0, s.st>>>(j.tree, j.sets, j.setOf, L, lists, s.nblR2.get(),
                                                                      j.rowsJ, s.nblCount.get(), s.nblH.get(), 0,
                                                                      std::min(s.numSMs, kNearQueues));
    COSMO_LAUNCHED();
    const bool warp = j.n <= kWarpPerParticle;
    auto step = j.sets ? (warp ? near_step_kernel<true, true> : near_step_kernel<true, false>)
                       : (warp ? near_step_kernel<false, true> : near_step_kernel<false, false>);
    step<<<iceil(j.n, warp ? kNearWarps : kThreads), kThreads, 0, s.st>>>(j.sets, j.setOf, L, lists, s.nblR2.get(), s.nblCount.get(),
                                                      s.nblH.get(), j.xyzh, j.rho, j.gradh, j.converged, s.hs.get(),
                                                      j.pmass, j.tolh, j.hfact, ds);
    COSMO_LAUNCHED();
    auto sum = NEAR_PICK(near_sum_kernel, j, NEAR_COMMA false);
    sum<<<persistent_blocks(s, sum, kThreads), kThreads, 0, s.st>>>(j.tree, j.sets, j.setOf, L, lists, j.xyzh, j.rho,
                                                                    j.gradh, j.converged, s.hs.get(), s.nblH.get(), j.pmass,
                                                                    j.tolh, j.hfact, ds);
    COSMO_LAUNCHED();
    // few particles have that many neighbours, if any: a block a multiprocessor
    auto huge = NEAR_PICK(near_huge_kernel, j);
    huge<<<s.numSMs, 32 * kHugeWarps, 0, s.st>>>(j.tree, j.sets, j.setOf, L, lists, j.xyzh, j.rho, j.gradh, j.converged,
                                                 s.hs.get(), s.nblH.get(), j.pmass, j.tolh, j.hfact, ds);
    COSMO_LAUNCHED();
    near_epilogue_kernel<<<1, kNearQueues, 0, s.st>>>(L, more, setCondition);
    COSMO_LAUNCHED();
}

// The loop as a graph: a while node over near_iteration.  It depends on the buffers, the
// solve's scalars and the particle count only.  defer: built for parameters met a second time
// in a row (a stepping caller's), as the list-based loop's is.  False: not run (the host loop
// is to be used).
static bool near_graph(State& s, const NearJob& j, int maxIter, bool defer)
{
    std::vector<unsigned char> key;
    auto add = [&](const auto& v) {
        const unsigned char* p = reinterpret_cast<const unsigned char*>(&v);
        key.insert(key.end(), p, p + sizeof(v));
    };
    for (const void* q : {(const void*)s.nearLoop.get(), (const void*)s.dscal.get(), (const void*)s.nearNode.get(),
                          (const void*)j.tree.xyzh, (const void*)j.tree.box, (const void*)j.sets, (const void*)j.setOf,
                          (const void*)s.nblR2.get(), (const void*)j.rowsJ, (const void*)s.nblCount.get(),
                          (const void*)s.nblH.get(), (const void*)j.rho, (const void*)j.gradh, (const void*)j.converged,
                          (const void*)s.hs.get(), (const void*)s.nearRow[0].get(), (const void*)s.nearRow[1].get(),
                          (const void*)s.nearBuild[0].get(), (const void*)s.nearBuild[1].get(),
                          (const void*)s.nearSum[0].get(), (const void*)s.nearSum[1].get(),
                          (const void*)s.nearHuge[0].get(), (const void*)s.nearHuge[1].get(),
                          (const void*)s.nearCover.get(), (const void*)s.nearOver.get()})
        add(q);
    for (int v : j.tree.off) add(v);
    for (int v : {j.n, j.periodic, s.numSMs, maxIter}) add(v);
    for (double v : {j.pmass, j.tolh, j.hfact}) add(v);
    s.loopKeyLast = key;
    if (!s.nearGraphExec || key != s.nearGraphKey)
    {
        if (defer && key != s.nearKeyPending)
        {
            s.nearKeyPending = key;
            return false;
        }
        if (s.nearGraphExec) COSMO_CUDA(cudaGraphExecDestroy(s.nearGraphExec));
        if (s.nearGraphDef) COSMO_CUDA(cudaGraphDestroy(s.nearGraphDef));
        s.nearGraphExec = nullptr;
        s.nearGraphDef = nullptr;
        s.nearGraphKey.clear();
        const unsigned long long launches0 = g_launches.load();
        cudaGraph_t g = nullptr;
        cudaGraphExec_t ex = nullptr;
        bool built = false;
        do
        {
            if (cudaGraphCreate(&g, 0) != cudaSuccess) break;
            cudaGraphConditionalHandle more;
            if (cudaGraphConditionalHandleCreate(&more, g, 1, cudaGraphCondAssignDefault) != cudaSuccess) break;
            cudaGraphNodeParams wp = {};
            wp.type = cudaGraphNodeTypeConditional;
            wp.conditional.handle = more;
            wp.conditional.type = cudaGraphCondTypeWhile;
            wp.conditional.size = 1;
            cudaGraphNode_t wnode;
            if (cudaGraphAddNode(&wnode, g, nullptr, 0, &wp) != cudaSuccess) break;
            cudaGraph_t body = wp.conditional.phGraph_out[0];
            if (cudaStreamBeginCaptureToGraph(s.st, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed) !=
                cudaSuccess)
                break;
            near_iteration(s, j, more, 1);
            if (cudaStreamEndCapture(s.st, &body) != cudaSuccess) break;
            if (cudaGraphInstantiate(&ex, g, 0) != cudaSuccess) break;
            built = true;
        } while (false);
        // what was captured did not run: the launches counted are those the graph executes
        s.nearKernels = g_launches.load() - launches0;
        g_launches -= s.nearKernels;
        if (!built)
        {
            cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
            if (cudaStreamIsCapturing(s.st, &cs) == cudaSuccess && cs != cudaStreamCaptureStatusNone)
            {
                cudaGraph_t junk = nullptr;
                cudaStreamEndCapture(s.st, &junk);
                if (junk) cudaGraphDestroy(junk);
            }
            if (ex) cudaGraphExecDestroy(ex);
            if (g) cudaGraphDestroy(g);
            (void)cudaGetLastError();
            return false;
        }
        s.nearGraphDef = g;
        s.nearGraphExec = ex;
        s.nearGraphKey = key;
        ++s.loopGraphBuilds;
    }
    COSMO_CUDA(cudaGraphLaunch(s.nearGraphExec, s.st));
    return true;
}

// The loop's iterations, as a graph or from the host.
static void near_run(State& s, const NearJob& j, int maxIter, bool graph, bool defer)
{
    s.lastLoopGraph = 0;
    s.nearLate.clear();
    if (graph && maxIter > 0 && maxIter <= kLoopIters && near_graph(s, j, maxIter, defer))
    {
        s.lastLoopGraph = 1;
        return;
    }
    for (int it = 0; it < maxIter; ++it)
    {
        near_iteration(s, j, cudaGraphConditionalHandle(0), 0);
        COSMO_CUDA(cudaMemcpyAsync(s.hsmall, s.nearLoop.get(), 4 * sizeof(int), cudaMemcpyDeviceToHost, s.st));
        COSMO_CUDA(cudaStreamSynchronize(s.st));
        if (s.hsmall[2] == 0) break;
        if (it + 1 >= kLoopIters && it + 1 < maxIter) s.nearLate.push_back(s.hsmall[2]);
    }
}

// The Newton loop of one plain solve over the block tree, every live (and not fixed)
// particle active.  Issued on the stream; near_results reads what it did.  rowsJ: the rows'
// j, for the gradient and force passes (may be null).
void near_newton(State& s, double pmass, double tolh, double hfact, int maxIter, bool allowGraph, int* rowsJ)
{
    const int n = std::max(s.nAlive, 1);
    DevScalars* ds = s.dscal.get();
    near_buffers(s, n);
    near_build(s);
    const bool frozen = s.frozenFor == s.ngas;
    near_init_kernel<<<1, kNearQueues, 0, s.st>>>(s.nearLoop.get(), ds, maxIter, frozen ? 1 : 0);
    COSMO_LAUNCHED();
    if (frozen)
    {
        near_frozen_kernel<<<std::min(iceil(n, kThreads), 8 * s.numSMs), kThreads, 0, s.st>>>(
            s.nearLoop.get(), s.orderA.get(), s.frozen.get(), &ds->nAlive, s.xyzh.get(), s.converged.get(), s.hs.get(),
            near_lists(s), ds);
        COSMO_LAUNCHED();
        near_active_kernel<<<1, 1, 0, s.st>>>(s.nearLoop.get());
        COSMO_LAUNCHED();
    }
    const NearJob j{near_tree(s), nullptr, nullptr, s.xyzh.get(), s.rho.get(), s.gradh.get(), s.converged.get(), rowsJ,
                    n, s.periodic, pmass, tolh, hfact};
    near_run(s, j, maxIter, allowGraph && s.newtonGraph, true);
}

// After the loop: rows at the converged h of the particles whose rows do not cover it.
void near_cover(State& s, int* rowsJ)
{
    auto rows = s.periodic ? near_rows_kernel<false, true> : near_rows_kernel<false, false>;
    rows<<<persistent_blocks(s, rows, kThreads), kThreads, 0, s.st>>>(near_tree(s), nullptr, nullptr, s.nearLoop.get(),
                                                                      near_lists(s), s.nblR2.get(), rowsJ,
                                                                      s.nblCount.get(), s.nblH.get(), 1, std::min(s.numSMs, kNearQueues));
    COSMO_LAUNCHED();
}

// What the loop did, once the stream has been read (h: its state on the host).
long long near_results(State& s, const NearLoop& h)
{
    if (s.lastLoopGraph) g_launches += (unsigned long long)h.iter * s.nearKernels;
    s.itersRun = h.iter;
    s.activePerIter.assign(h.activePerIter, h.activePerIter + std::min(h.iter, kLoopIters));
    s.activePerIter.insert(s.activePerIter.end(), s.nearLate.begin(), s.nearLate.end());
    return h.active;
}

// The Newton loop of a plain batch over its sets' block trees (the batch's arrays in b, its
// scratch in s), every live particle of every set active.  Issued on the stream.
void near_forest_newton(State& s, const NearForest& b, double tolh, double hfact, int maxIter, bool graph)
{
    NearTree t;
    const size_t nodes = near_layout(b.n, b.nsets, t);
    s.nearNode.resize(nodes * (sizeof(NearNode) / sizeof(float4)), s.st);
    s.nearSets.resize(b.nsets, s.st);
    near_buffers(s, b.n);
    s.nblR2.resize(size_t(b.n) * kNbl, s.st);
    s.nblCount.resize(b.n, s.st);
    s.nblH.resize(b.n, s.st);
    t.node = reinterpret_cast<const NearNode*>(s.nearNode.get());
    t.xyzh = b.xyzh;
    t.box = b.boxes;
    t.nLive = &s.dscal.get()->nAlive;
    NearNode* out = reinterpret_cast<NearNode*>(s.nearNode.get());
    near_sets_kernel<<<iceil(b.nsets, 256), 256, 0, s.st>>>(b.nsets, b.offs, b.nAlive, b.boxes, b.pmass,
                                                            s.nearSets.get());
    COSMO_LAUNCHED();
    const int slots = (b.n >> 9) + b.nsets + 1;
    near_leaf_levels_kernel<true><<<std::min(slots, 8 * s.numSMs), 512, 0, s.st>>>(t, out, s.nearSets.get(), b.nsets,
                                                                                  slots);
    COSMO_LAUNCHED();
    near_upper_levels_kernel<true><<<b.nsets, 1024, 0, s.st>>>(t, out, s.nearSets.get());
    COSMO_LAUNCHED();
    near_forest_zero_kernel<<<1, kNearQueues, 0, s.st>>>(s.nearLoop.get(), maxIter);
    COSMO_LAUNCHED();
    near_forest_init_kernel<<<std::min(iceil(b.n, kThreads), 16 * s.numSMs), kThreads, 0, s.st>>>(
        s.nearLoop.get(), b.n, s.nearSets.get(), b.setOf, near_lists(s));
    COSMO_LAUNCHED();
    near_active_kernel<<<1, 1, 0, s.st>>>(s.nearLoop.get());
    COSMO_LAUNCHED();
    const NearJob j{t, s.nearSets.get(), b.setOf, b.xyzh, b.rho, b.gradh, b.converged, nullptr, b.n, 1, 0.0, tolh,
                    hfact};
    near_run(s, j, maxIter, graph, false);
}

// rho and d(rho)/dh of every live particle of the batch at its final h, converged or not.
void near_forest_eval(State& s, const NearForest& b)
{
    NearTree t;
    near_layout(b.n, b.nsets, t);
    t.node = reinterpret_cast<const NearNode*>(s.nearNode.get());
    t.xyzh = b.xyzh;
    t.box = b.boxes;
    t.nLive = &s.dscal.get()->nAlive;
    const NearLists lists = near_lists(s);
    NearLoop* L = s.nearLoop.get();
    near_pending_kernel<<<std::min(iceil(b.n, kThreads), 2 * s.numSMs), kThreads, 0, s.st>>>(L, lists);
    COSMO_LAUNCHED();
    auto rows = near_rows_kernel<true, true>;
    rows<<<persistent_blocks(s, rows, kThreads), kThreads, 0, s.st>>>(t, s.nearSets.get(), b.setOf, L, lists,
                                                                      s.nblR2.get(), nullptr, s.nblCount.get(),
                                                                      s.nblH.get(), 1, std::min(s.numSMs, kNearQueues));
    COSMO_LAUNCHED();
    near_eval_kernel<<<iceil(b.n, kThreads), kThreads, 0, s.st>>>(b.n, s.nearSets.get(), b.setOf, s.nblR2.get(),
                                                                  s.nblCount.get(), b.xyzh, b.rho, b.gradh,
                                                                  s.dscal.get());
    COSMO_LAUNCHED();
    auto sum = near_sum_kernel<true, true, true>;
    sum<<<persistent_blocks(s, sum, kThreads), kThreads, 0, s.st>>>(t, s.nearSets.get(), b.setOf, L, lists, b.xyzh,
                                                                    b.rho, b.gradh, b.converged, s.hs.get(), nullptr, 0.0,
                                                                    0.0, 0.0, s.dscal.get());
    COSMO_LAUNCHED();
}

} // namespace cosmo
