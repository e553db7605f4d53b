/*
 * sort.cuh -- scans and the LSD radix sorts shared by the single-set and the
 * batched (forest) tree builds.  Internal-linkage kernels: each translation unit that
 * includes this gets its own copy.
 */
#pragma once

#include "common.cuh"
#include "tma.cuh"

namespace cosmo {
namespace {

constexpr int kBlk = 256;

__device__ __forceinline__ uint32_t ld_volatile_u32(const uint32_t* p)
{
    uint32_t v;
    asm volatile("ld.volatile.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// ------------------------------------------------------------------ scan (3 phase)
constexpr int kScanThreads = 1024;
constexpr int kScanItems   = 4;
constexpr int kScanTile    = kScanThreads * kScanItems;

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Block-wide exclusive scan of one value per thread; returns the exclusive prefix and
// the block total in *total.
__device__ uint32_t block_excl_scan(uint32_t v, uint32_t* total)
{
    __shared__ uint32_t sw[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nw = blockDim.x >> 5;
    const uint32_t inc = warp_incl_scan(v);
    if (lane == 31) sw[warp] = inc;
    __syncthreads();
    if (warp == 0)
    {
        uint32_t s = lane < nw ? sw[lane] : 0;
        s = warp_incl_scan(s);
        sw[lane] = s;
    }
    __syncthreads();
    const uint32_t before = warp ? sw[warp - 1] : 0;
    *total = sw[nw - 1];
    __syncthreads();
    return before + inc - v;
}

// nPtr (when given): the element count on the device, n then being a bound on it (a scan
// issued before its count is known, as a captured graph does).
__global__ void scan_reduce_kernel(const uint32_t* __restrict__ in, int n, uint32_t* __restrict__ bsum,
                                   const int* __restrict__ nPtr = nullptr)
{
    if (nPtr) n = *nPtr;
    const long base = long(blockIdx.x) * kScanTile + threadIdx.x * kScanItems;
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k)
        if (base + k < n) s += in[base + k];
    uint32_t tot;
    block_excl_scan(s, &tot);
    if (threadIdx.x == 0) bsum[blockIdx.x] = tot;
}

__global__ void scan_blocks_kernel(uint32_t* bsum, int nb, uint32_t* totalOut, uint32_t* out = nullptr,
                                   const int* __restrict__ nPtr = nullptr)
{
    if (nPtr) totalOut = out + *nPtr;   // the total goes after the last element
    // one block of kScanThreads; nb <= kScanTile
    const int base = threadIdx.x * kScanItems;
    uint32_t v[kScanItems], s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k)
    {
        v[k] = (base + k < nb) ? bsum[base + k] : 0;
        s += v[k];
    }
    uint32_t tot;
    uint32_t run = block_excl_scan(s, &tot);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k)
        if (base + k < nb)
        {
            bsum[base + k] = run;
            run += v[k];
        }
    if (threadIdx.x == 0) *totalOut = tot;
}

__global__ void scan_apply_kernel(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, int n,
                                  const uint32_t* __restrict__ boff, const int* __restrict__ nPtr = nullptr)
{
    if (nPtr) n = *nPtr;
    const long base = long(blockIdx.x) * kScanTile + threadIdx.x * kScanItems;
    uint32_t v[kScanItems], s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k)
    {
        v[k] = (base + k < n) ? in[base + k] : 0;
        s += v[k];
    }
    uint32_t tot;
    uint32_t run = block_excl_scan(s, &tot) + boff[blockIdx.x];
#pragma unroll
    for (int k = 0; k < kScanItems; ++k)
        if (base + k < n)
        {
            out[base + k] = run;
            run += v[k];
        }
}

// ------------------------------------------------------------------ onesweep radix sort
constexpr int kSortThreads = 256;
constexpr int kSortIpt     = 16;
constexpr int kSortTile    = kSortThreads * kSortIpt;
constexpr int kSortWarps   = kSortThreads / 32;
constexpr int kSortPasses  = 8;
constexpr uint32_t kLbAgg  = 1u << 30, kLbInc = 2u << 30, kLbMask = (1u << 30) - 1;

__global__ void digit_hist_kernel(const uint64_t* __restrict__ keys, int n, uint32_t* __restrict__ hist)
{
    __shared__ uint32_t s[kSortPasses][256];
    for (int i = threadIdx.x; i < kSortPasses * 256; i += blockDim.x) (&s[0][0])[i] = 0;
    __syncthreads();
    for (long i = long(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += long(gridDim.x) * blockDim.x)
    {
        const uint64_t k = keys[i];
#pragma unroll
        for (int p = 0; p < kSortPasses; ++p) atomicAdd(&s[p][(k >> (8 * p)) & 255u], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kSortPasses * 256; i += blockDim.x)
        if ((&s[0][0])[i]) atomicAdd(&hist[i], (&s[0][0])[i]);
}

__global__ void digit_base_kernel(const uint32_t* __restrict__ hist, uint32_t* __restrict__ base)
{
    // block p scans the 256 bins of pass p
    const uint32_t v = hist[blockIdx.x * 256 + threadIdx.x];
    uint32_t tot;
    base[blockIdx.x * 256 + threadIdx.x] = block_excl_scan(v, &tot);
}

// One stable counting pass of an LSD radix sort of (key, value) pairs, single pass per
// digit with decoupled look-back between tiles.  The digit is byte `shift/8` of the key,
// or -- when SetDigit -- of setOf[value] (the set id of the element's original index),
// which turns a finished key sort into a stable (set, key) segmented sort.
template<bool SetDigit>
__device__ __forceinline__ void
onesweep_body(const uint64_t* __restrict__ kin, const int* __restrict__ vin, uint64_t* __restrict__ kout,
                  int* __restrict__ vout, int n, int shift, const uint32_t* __restrict__ binBase,
                  uint32_t* lookback, unsigned int* tileTicket, int* err, const int* __restrict__ setOf,
                  long long waitNs)
{
    __shared__ uint32_t sHist[kSortWarps][256];
    __shared__ uint32_t sBase[256];
    __shared__ int sTile;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < kSortWarps * 256; i += kSortThreads) (&sHist[0][0])[i] = 0;
    if (tid == 0) sTile = int(atomicAdd(tileTicket, 1u));
    __syncthreads();
    const int tile = sTile;
    const long base = long(tile) * kSortTile + long(warp) * 32 * kSortIpt;

    uint64_t k[kSortIpt];
    int v[kSortIpt];
    uint32_t rank[kSortIpt];
#pragma unroll
    for (int it = 0; it < kSortIpt; ++it)
    {
        const long idx = base + it * 32 + lane;
        if (idx < n) { k[it] = kin[idx]; v[it] = vin ? vin[idx] : int(idx); }
        else { k[it] = 0; v[it] = 0; }
    }
    const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
    for (int it = 0; it < kSortIpt; ++it)
    {
        const bool valid = (base + it * 32 + lane) < n;
        const uint32_t d = valid ? (SetDigit ? (uint32_t(setOf[v[it]]) >> shift) & 255u
                                             : uint32_t(k[it] >> shift) & 255u)
                                 : 256u;
        const uint32_t peers = __match_any_sync(0xffffffffu, d);
        uint32_t c = 0;
        if (valid) c = sHist[warp][d];
        __syncwarp();
        rank[it] = c + __popc(peers & lt);
        if (valid && (peers & lt) == 0u) sHist[warp][d] = c + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    {
        const int d = tid;
        uint32_t total = 0;
#pragma unroll
        for (int w = 0; w < kSortWarps; ++w)
        {
            const uint32_t c = sHist[w][d];
            sHist[w][d] = total;
            total += c;
        }
        uint32_t* mine = lookback + size_t(tile) * 256 + d;
        if (tile == 0)
        {
            atomicExch(mine, kLbInc | total);
            sBase[d] = binBase[d];
        }
        else
        {
            atomicExch(mine, kLbAgg | total);
            uint32_t excl = 0;
            int p = tile - 1;
            WaitClock clk;
            while (p >= 0)
            {
                const uint32_t s = ld_volatile_u32(lookback + size_t(p) * 256 + d);
                if ((s & ~kLbMask) == 0u)
                {
                    if (clk.over(waitNs)) { atomicOr(err, int(kErrSortSpin)); break; }
                    continue;
                }
                excl += s & kLbMask;
                if (s & kLbInc) break;
                --p;
            }
            atomicExch(mine, kLbInc | (excl + total));
            sBase[d] = binBase[d] + excl;
        }
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < kSortIpt; ++it)
    {
        const long idx = base + it * 32 + lane;
        if (idx < n)
        {
            const uint32_t d = SetDigit ? (uint32_t(setOf[v[it]]) >> shift) & 255u : uint32_t(k[it] >> shift) & 255u;
            const uint32_t pos = sBase[d] + sHist[warp][d] + rank[it];
            kout[pos] = k[it];
            vout[pos] = v[it];
        }
    }
}


__global__ void __launch_bounds__(kSortThreads, 3)
onesweep_kernel(const uint64_t* __restrict__ kin, const int* __restrict__ vin, uint64_t* __restrict__ kout,
                int* __restrict__ vout, int n, int shift, const uint32_t* __restrict__ binBase,
                uint32_t* lookback, unsigned int* tileTicket, int* err, long long waitNs)
{
    onesweep_body<false>(kin, vin, kout, vout, n, shift, binBase, lookback, tileTicket, err, nullptr, waitNs);
}

__global__ void __launch_bounds__(kSortThreads)
onesweep_set_kernel(const uint64_t* __restrict__ kin, const int* __restrict__ vin, uint64_t* __restrict__ kout,
                    int* __restrict__ vout, int n, int shift, const uint32_t* __restrict__ binBase,
                    uint32_t* lookback, unsigned int* tileTicket, int* err, const int* __restrict__ setOf,
                    long long waitNs)
{
    onesweep_body<true>(kin, vin, kout, vout, n, shift, binBase, lookback, tileTicket, err, setOf, waitNs);
}

// ------------------------------------------------------------------ one-kernel radix sort
// All eight passes in one cooperative kernel, a block of 1024 threads on a multiprocessor,
// each with its share of the pairs (ipt a thread).  A pass: the block ranks its share by
// warps, puts it in digit order in shared memory, hands its 256 counts to the others, reads
// theirs, writes its share out in runs of one digit, and waits for all to have done so.
// The onesweep passes take a launch each and are bound by their chain of tiles (each waits
// for what the tiles before it hand on) and their stores to 32 sectors a warp: 512 pairs
// 100 -> 30 us, 20,000 136 -> 55, 500,000 183 -> 95, 1,000,000 270 -> 129, 2,000,000
// 470 -> 220 (random keys, clears and histogram included).  What is left is two exchanges
// over L2 a pass (about 5 us) and 32 warps a multiprocessor ranking, 1.2 us a pair a thread.
// The lanes of a digit from ballots, not match.any: 500,000 pairs 116 -> 101 us.  Counts
// read two blocks ahead, one where 16 pairs a thread leave no registers (deeper ones spill:
// 500,000 pairs 143 us).
constexpr int kBsThreads = 1024;
constexpr int kBsMaxIpt  = 16;
constexpr size_t kBsFixed = size_t(6 + 4) * 256 * 4 + 32 * 256 * 2 + 16;
inline size_t block_sort_smem(int ipt) { return kBsFixed + size_t(kBsThreads) * ipt * 12; }

__device__ __forceinline__ uint4 ld_volatile_u32x4(const uint32_t* p)
{
    uint4 v;
    asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}

// n pairs in (kA, vA), sorted there; (kB, vB) is scratch.  iota: the values are 0, 1, ...
// and vA holds nothing yet.  table: gridDim.x * 256 counts and the arrivals behind them,
// zeroed by the caller.  Every wait ends after waitNs (an error bit, and the block returns).
template<int Ipt>
__global__ void __launch_bounds__(kBsThreads, 1)
block_sort_kernel(uint64_t* kA, uint64_t* kB, int* vA, int* vB, int n, int ipt, int iota, uint32_t* table,
                  unsigned int* arrived, int* err, long long waitNs)
{
    extern __shared__ __align__(16) unsigned char smem[];
    uint64_t* sKey = reinterpret_cast<uint64_t*>(smem);
    int* sVal = reinterpret_cast<int*>(sKey + kBsThreads * ipt);
    uint32_t* sPart = reinterpret_cast<uint32_t*>(sVal + kBsThreads * ipt);   // [6][256]
    uint32_t* sLocal = sPart + 6 * 256;     // first slot of a digit in the block
    uint32_t* sGlobal = sLocal + 256;       // its first place in the output, less that slot
    uint32_t* sTot = sGlobal + 256;
    uint32_t* sWarp = sTot + 256;
    uint16_t* sHist = reinterpret_cast<uint16_t*>(sWarp + 256);   // [32][256]
    int* sStop = reinterpret_cast<int*>(sHist + 32 * 256);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int d = tid & 255, q = tid >> 8;
    const int G = gridDim.x, b = blockIdx.x;
    const int K = kBsThreads * ipt;
    const int first = b * K, mine = min(K, n - first);
    const uint32_t lt = (1u << lane) - 1u;
    uint16_t* hist = sHist + warp * 256;
    if (tid == 0) *sStop = 0;
    for (int p = 0; p < kSortPasses; ++p)
    {
        const uint64_t* ki = (p & 1) ? kB : kA;
        uint64_t* ko = (p & 1) ? kA : kB;
        const int* vi = (p & 1) ? vB : vA;
        int* vo = (p & 1) ? vA : vB;
        const int shift = 8 * p;
        for (int i = lane; i < 128; i += 32) reinterpret_cast<uint32_t*>(hist)[i] = 0;
        if (tid < 512) sPart[4 * 256 + tid] = 0;
        const int at = warp * 32 * ipt + lane;
        __syncwarp();
        uint64_t k[Ipt];
        uint32_t rank[(Ipt + 1) / 2];
#pragma unroll
        for (int it = 0; it < Ipt; ++it)
            if (it < ipt && at + it * 32 < mine) k[it] = __ldcg(ki + first + at + it * 32);
#pragma unroll
        for (int it = 0; it < Ipt; ++it)
        {
            if (it >= ipt) break;
            const bool valid = at + it * 32 < mine;
            const uint32_t dg = valid ? uint32_t(k[it] >> shift) & 255u : 256u;
            // the lanes of the same digit, from a ballot per bit
            uint32_t peers = __ballot_sync(0xffffffffu, valid);
            if (!valid) peers = ~peers;
#pragma unroll
            for (int bit = 0; bit < 8; ++bit)
            {
                const uint32_t m = __ballot_sync(0xffffffffu, (dg >> bit) & 1u);
                peers &= ((dg >> bit) & 1u) ? m : ~m;
            }
            uint32_t c = 0;
            if (valid) c = hist[dg];
            __syncwarp();
            const uint32_t r = c + __popc(peers & lt);
            rank[it / 2] = (it & 1) ? rank[it / 2] | r << 16 : r;
            if (valid && (peers & lt) == 0u) hist[dg] = uint16_t(c + __popc(peers));
            __syncwarp();
        }
        __syncthreads();
        // per digit: the warps' counts to their prefixes
        uint32_t c8[8], sum = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) { c8[w] = sHist[(q * 8 + w) * 256 + d]; sum += c8[w]; }
        sPart[q * 256 + d] = sum;
        __syncthreads();
        uint32_t run = 0, tot = 0;
#pragma unroll
        for (int o = 0; o < 4; ++o)
        {
            const uint32_t v = sPart[o * 256 + d];
            if (o < q) run += v;
            tot += v;
        }
#pragma unroll
        for (int w = 0; w < 8; ++w) { sHist[(q * 8 + w) * 256 + d] = uint16_t(run); run += c8[w]; }
        if (q == 0)
        {
            if (G > 1) __stcg(table + size_t(b) * 256 + d, uint32_t(p + 1) << 16 | tot);
            // the digit's first slot
            const uint32_t inc = warp_incl_scan(tot);
            if (lane == 31) sWarp[warp] = inc;
            sLocal[d] = inc - tot;
        }
        __syncthreads();
        if (tid < 256)
        {
            uint32_t before = 0;
            for (int w = 0; w < 8; ++w) before += w < warp ? sWarp[w] : 0;
            sLocal[d] += before;
        }
        __syncthreads();
        // the pairs to their slots
#pragma unroll
        for (int i0 = 0; i0 < Ipt; i0 += 4)
        {
            int v[4];
#pragma unroll
            for (int a = 0; a < 4; ++a)
            {
                const int it = i0 + a;
                if (it < ipt && at + it * 32 < mine)
                    v[a] = (p == 0 && iota) ? first + at + it * 32 : __ldcg(vi + first + at + it * 32);
            }
#pragma unroll
            for (int a = 0; a < 4; ++a)
            {
                const int it = i0 + a;
                if (it < ipt && at + it * 32 < mine)
                {
                    const uint32_t dg = uint32_t(k[it] >> shift) & 255u;
                    const uint32_t slot = sLocal[dg] + hist[dg] + ((rank[it / 2] >> (16 * (it & 1))) & 0xffffu);
                    sKey[slot] = k[it];
                    sVal[slot] = v[a];
                }
            }
        }
        // where each digit's pairs of this block go
        if (G > 1)
        {
            // 64 threads read a block's 256 counts, four each
            const int quad = tid & 63, g0 = tid >> 6;
            uint4 all = make_uint4(0, 0, 0, 0), before = all;
            WaitClock clk;
            bool gave = false;
            constexpr int kAhead = Ipt > 8 ? 1 : 2;
            for (int o0 = g0; o0 < G && !gave; o0 += 16 * kAhead)
            {
                uint4 w[kAhead];
                for (;;)
                {
                    bool ready = true;
#pragma unroll
                    for (int a = 0; a < kAhead; ++a)
                        if (o0 + 16 * a < G)
                            w[a] = ld_volatile_u32x4(table + size_t(o0 + 16 * a) * 256 + quad * 4);
#pragma unroll
                    for (int a = 0; a < kAhead; ++a)
                        if (o0 + 16 * a < G)
                            ready = ready && (w[a].x >> 16) == uint32_t(p + 1) && (w[a].y >> 16) == uint32_t(p + 1) &&
                                    (w[a].z >> 16) == uint32_t(p + 1) && (w[a].w >> 16) == uint32_t(p + 1);
                    if (ready) break;
                    if (clk.over(waitNs)) { gave = true; break; }
                }
#pragma unroll
                for (int a = 0; a < kAhead; ++a)
                    if (o0 + 16 * a < G)
                    {
                        const uint4 c = make_uint4(w[a].x & 0xffffu, w[a].y & 0xffffu, w[a].z & 0xffffu,
                                                   w[a].w & 0xffffu);
                        all.x += c.x; all.y += c.y; all.z += c.z; all.w += c.w;
                        if (o0 + 16 * a < b)
                        {
                            before.x += c.x; before.y += c.y; before.z += c.z; before.w += c.w;
                        }
                    }
            }
            if (gave) { atomicOr(err, int(kErrSortSpin)); *sStop = 1; }
            auto add = [&](uint32_t* to, const uint4& c) {
                atomicAdd(to, c.x);
                atomicAdd(to + 1, c.y);
                atomicAdd(to + 2, c.z);
                atomicAdd(to + 3, c.w);
            };
            if (g0 < G) add(sPart + 4 * 256 + quad * 4, all);
            if (g0 < b) add(sPart + 5 * 256 + quad * 4, before);
            __syncthreads();
            if (*sStop) return;
            if (q == 0)
            {
                const uint32_t tt = sPart[4 * 256 + d];
                const uint32_t inc = warp_incl_scan(tt);
                if (lane == 31) sWarp[warp] = inc;
                sTot[d] = inc - tt + sPart[5 * 256 + d];
            }
            __syncthreads();
            if (tid < 256)
            {
                uint32_t lower = 0;
                for (int w = 0; w < 8; ++w) lower += w < warp ? sWarp[w] : 0;
                sGlobal[d] = sTot[d] + lower - sLocal[d];
            }
        }
        __syncthreads();
        for (int i = tid; i < mine; i += kBsThreads)
        {
            const uint64_t key = sKey[i];
            const uint32_t dg = uint32_t(key >> shift) & 255u;
            const uint32_t pos = G > 1 ? sGlobal[dg] + i : i;
            __stcg(ko + pos, key);
            __stcg(vo + pos, sVal[i]);
        }
        if (p == kSortPasses - 1) break;
        // every block's pairs of this pass are written before any is read
        __threadfence();
        __syncthreads();
        if (G > 1)
        {
            if (tid == 0)
            {
                atomicAdd(arrived, 1u);
                WaitClock clk;
                while (ld_volatile_u32(arrived) < uint32_t(G) * uint32_t(p + 1))
                    if (clk.over(waitNs)) { atomicOr(err, int(kErrSortSpin)); *sStop = 1; break; }
                __threadfence();
            }
            __syncthreads();
            if (*sStop) return;
        }
    }
}

} // namespace
} // namespace cosmo
