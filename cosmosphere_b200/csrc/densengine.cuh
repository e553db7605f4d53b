/*
 * densengine.cuh -- the density sums of one warp group over its leaf's gather list, shared
 * by the single-set Newton kernel and the batched forest kernel, plain FP64 or mixed.
 *
 * The leaf's list is culled by the leaves' own boxes (near_ranges), and the candidates that
 * pass the group's region go into the warp's ring (GroupSource).
 *
 *   plain  each batch of up to 32 is tested with j on the lanes: for each group particle in
 *          turn, every lane tests its candidate, and the accepted pairs are appended,
 *          particle-major, to the warp's record buffer -- so each particle's records are
 *          contiguous and in ascending j.  The records are evaluated with one pair per lane
 *          (W and -q dW/dq - 3W), and each particle's owner lane adds its own records in
 *          order.  The exact FP64 test q^2 = r^2 / h_i^2 < R^2 (src/density_base.cu:270-283)
 *          and FP64 sums in ascending j: bit for bit the oracle's.
 * The periodic form with zero periods behaves, bit for bit, as the open form (the batched
 * kernel runs open and periodic sets through the one periodic instance).
 *
 *   mixed  coordinates relative to the group box centre (at the nearest periodic image
 *          of that centre when the box is small enough for it to be every pair's nearest
 *          image), the test and W, dW in FP32, sums in FP32 with Kahan compensation,
 *          combined in FP64.  Each particle's lane tests the candidates, two in a packed
 *          f32x2 instruction, and keeps the q^2 of those it accepts in a column of its own
 *          in shared memory; the columns are evaluated and added when one is nearly full.
 *          With the records of the plain form the owners' serial additions ran over a
 *          batch's longest list while most lanes had none: they were two fifths of the
 *          kernel's instructions, the FP64 filter over whole lists most of the rest
 *          (a solve of 40 sets of 10,000 to 300,000: 65.5 -> 46.4 ms; the Newton loop of a
 *          300,000-particle box 3.65 -> 3.15).  The batch code is the kernel's largest loop and stays there once:
 *          four copies of it stalled two issues in three on the instruction cache.
 */
#pragma once

#include "pairstream.cuh"

namespace cosmo {

constexpr int kRec = 256;   // pair records per warp

// Per-warp shared scratch of density_group: the ring, the group's particles and the pair
// records (mixed: the ring and the columns), and at kBoxAt the group's rounded box (read by the filter from shared memory
// rather than held in registers through the stream).
constexpr int kTest = 8;     // mixed: candidates a lane tests in one turn of its loop
// Mixed: a group of at most kFew particles (a leaf's last, or a cut group, which has
// thousands of candidates) is tested with a candidate a lane, and its kept pairs are evaluated
// by all lanes and only added by their owners: with a particle a lane most lanes had nothing
// to test or evaluate (the loop of a 30,000-particle Plummer sphere 16.9 -> 12.9 ms, 9 sets of
// 6,000 to 18,000 8.5 -> 7.1, 40 sets of 10,000 to 300,000 48.1 -> 46.4).  Lines at 8, 12 and
// 16: a quintic Plummer sphere of 14,000, whose cut groups hold nine, 13.0, 10.2 and 10.5 ms
// (with the plain form's records 12.3), of 8,000 (sixteen) 7.7, 7.7 and 7.0 (7.9), cubic ones
// 8.8, 8.2, 8.6 (10.3) and 5.6, 5.5, 5.8 (6.3).  Its columns
// lie one after the other, with as much room again for the second term: 118 pairs of two
// terms for each of eight particles, or 82 for each of twelve, fit in the columns' 2048 words
// beside the particles' own data; 236 words a particle keep the owners' accesses on
// different banks, 164 all but four of them.
constexpr int kFew = 12;
constexpr int kColumn = 64;   // mixed: accepted pairs a lane keeps before they are evaluated

template<bool Mixed>
struct DensScratch
{
    static constexpr int kBoxAt = Mixed ? (3 * kRing * 4 + kColumn * 32 * 4)
                                        : (kRing * 32 + 32 * 32 + 2 * kRec * 8);
    static constexpr int kBytes = kBoxAt + 64;
};

// q = sqrt(q2) in FP32 (q2 >= 0); exact 0 for the self pair.  A subnormal q2 counts as 0
// too (W and -q dW/dq - 3W round to the same for any q below 1e-18), which leaves out the
// scaling that rsqrtf does for such values.
__device__ __forceinline__ float sqrt_q(float q2)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(q2));
    return q2 >= 1.17549435e-38f ? q2 * r : 0.0f;
}

// Sums over the gather list of one group: the lanes [0, ng) own the group's particles
// (pi, with mine set); rhoi and gradhi receive the un-normalised sums (W and
// -q dW/dq - 3W over accepted j), gp the accepted pairs and gc the candidates offered.
template<bool Periodic, bool Mixed, bool Staged = false, bool Round = true, class Ranges>
__device__ __forceinline__ void density_group(unsigned char* scr, bool mine, int ng, const double4& pi, double lx,
                                              double ly, double lz, const GroupSource<Ranges>& list,
                                              const float4* __restrict__ leafBox, double& rhoi, double& gradhi,
                                              unsigned int& gp, unsigned int& gc)
{
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    const double hi = pi.w;
    const double hinv2 = 1.0 / (hi * hi);
    const double rs = kRadKernel * hi;
    const double rmax = warp_max(mine ? rs : 0.0);
    const GroupBox bx = group_box(mine, pi.x, pi.y, pi.z, rs, rmax);
    // Candidates, and the cells of a cut group's tree scan, are taken within the largest
    // support of the members' own bounding box (a rounded box: a single particle's is its
    // sphere), with the box's slack (1e-9 of the support, 1e-13 of |c|) on the radius, far
    // above the rounding of the exact test, so no accepted pair is lost.  Not Round: within
    // the box of the search spheres (the batched plain kernel: its sets' h do not scatter,
    // and its registers are tighter).  The mixed form of several particles filters by the
    // rounded box in FP32.  A single particle's partial sums, one a lane, depend on the
    // candidates' places in the ring: it keeps the FP64 filter.
    const GroupBox pb = group_box(mine, pi.x, pi.y, pi.z, 0.0, rmax);
    RoundBox* rbp = Round ? reinterpret_cast<RoundBox*>(scr + DensScratch<Mixed>::kBoxAt) : nullptr;
    const double rr = rmax + 1e-9 * rmax + 1e-13 * (fabs(pb.cx) + fabs(pb.cy) + fabs(pb.cz)) + 1e-300;
    if constexpr (Round)
    {
        if (lane == 0) *rbp = RoundBox{pb.cx, pb.cy, pb.cz, pb.ex, pb.ey, pb.ez, rr};
        __syncwarp();
    }
    const bool cube = !Round && (!Mixed || ng == 1);
    const GroupRegion region = group_region<Periodic>(cube ? bx : pb, cube ? 0.0 : rr, lx, ly, lz);
    GroupSource<NearRanges<Periodic, Ranges>> src{list.jlist, list.jb, list.nj,
                                                  near_ranges<Periodic>(list.ranges, leafBox, region), list.xyzh,
                                                  list.walk, list.tree, list.rc, list.re, list.stage};
    auto gather = [&](const double4& pj) {
        if (Mixed && ng > 1) return in_region<Periodic>(pj, region);
        if constexpr (Round) return in_round_box<Periodic>(pj, *rbp, lx, ly, lz);
        else return in_gather_box<Periodic>(pj, bx, lx, ly, lz);
    };
    gp = 0;
    gc = 0;
    if constexpr (!Mixed)
    {
        double4* ring = reinterpret_cast<double4*>(scr);
        double4* grp = ring + kRing;
        double* recA = reinterpret_cast<double*>(grp + 32);
        double* recB = recA + kRec;
        if (mine) grp[lane] = make_double4(pi.x, pi.y, pi.z, hinv2);
        __syncwarp();
        double sr = 0.0, sg = 0.0;
        src.template stream<true, false, false, Periodic, Staged>(
            ring, nullptr, nullptr, bx, 0.0, 0.0, 0.0, lx, ly, lz, gather,
            [&](const double4* rg, const float4*, const int*, int head, int count) {
                gc += count;
                const double4 pj = rg[(head + (lane < count ? lane : 0)) & (kRing - 1)];
                if (ng == 1)
                {
                    // a single particle (a cut group): every lane evaluates its own pair, the
                    // accepted values are packed into the record buffers in lane (= j) order,
                    // and the sums add them in that order from broadcast shared-memory loads
                    // -- one add per accepted pair, as in the oracle's loop, so the chain is
                    // bound by the add latency alone
                    const double4 g = grp[0];
                    double dx = g.x - pj.x, dy = g.y - pj.y, dz = g.z - pj.z;
                    nearest_image<Periodic>(dx, dy, dz, lx, ly, lz);
                    const double q2 = pair_r2(dx, dy, dz) * g.w;
                    const bool acc = lane < count && q2 < kRadK2;
                    double wv = 0.0, tv = 0.0;
                    if (acc)
                    {
                        const double q = sqrt(q2);
                        double wk, dwk;
                        sph_kernel(q2, q, wk, dwk);
                        wv = wk;
                        tv = -q * dwk - 3.0 * wk;
                    }
                    const uint32_t am = __ballot_sync(0xffffffffu, acc);
                    const int c = __popc(am);
                    gp += c;
                    if (acc)
                    {
                        recA[__popc(am & lt)] = wv;
                        recB[__popc(am & lt)] = tv;
                    }
                    __syncwarp();
                    for (int t = 0; t < c; ++t)
                    {
                        sr += recA[t];
                        sg += recB[t];
                    }
                    __syncwarp();
                    return;
                }
                int nrec = 0, segStart = 0, segCount = 0;
                auto flush = [&]() {
                    __syncwarp();
                    for (int r = lane; r < nrec; r += 32)
                    {
                        const double q2 = recA[r];
                        const double q = sqrt(q2);
                        double wk, dwk;
                        sph_kernel(q2, q, wk, dwk);
                        recA[r] = wk;
                        recB[r] = -q * dwk - 3.0 * wk;
                    }
                    __syncwarp();
                    for (int t = 0; t < segCount; ++t)
                    {
                        sr += recA[segStart + t];
                        sg += recB[segStart + t];
                    }
                    gp += segCount;
                    segCount = 0;
                    nrec = 0;
                    __syncwarp();
                };
                // four group particles per step: independent FP64 chains for the scheduler
                for (int i0 = 0; i0 < ng; i0 += 4)
                {
                    if (nrec + 4 * 32 > kRec) flush();
                    double q2u[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                    {
                        const double4 g = grp[min(i0 + u, 31)];
                        double dx = g.x - pj.x, dy = g.y - pj.y, dz = g.z - pj.z;
                        nearest_image<Periodic>(dx, dy, dz, lx, ly, lz);
                        q2u[u] = pair_r2(dx, dy, dz) * g.w;
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                    {
                        const bool acc = lane < count && i0 + u < ng && q2u[u] < kRadK2;
                        const uint32_t m = __ballot_sync(0xffffffffu, acc);
                        const int c = __popc(m);
                        if (acc) recA[nrec + __popc(m & lt)] = q2u[u];
                        if (lane == i0 + u) { segStart = nrec; segCount = c; }
                        nrec += c;
                    }
                }
                if (nrec > 0) flush();
            },
            rbp);
        rhoi = sr;
        gradhi = sg;
    }
    else
    {
        float* rx = reinterpret_cast<float*>(scr);   // the candidates' -x, -y, -z, kRing each
        // q^2 of accepted pair t at column[t * step]: interleaved by lanes, or, of a few
        // particles, one after the other with as much room again for the second term
        const bool few = ng <= kFew;
        float* columns = rx + 3 * kRing;
        const int room = few ? (ng <= 8 ? 118 : 82) : kColumn;
        float* column = columns + (few ? 2 * room * lane : lane);
        float* member = columns + kColumn * 32 - 4 * kFew;   // few: x, y, z, 1/h^2 of kFew each
        // relative coordinates at the centre's nearest image are every accepted pair's
        // nearest image when the box (search spheres included) spans under half a period
        const bool shifted = !Periodic || lx == 0.0 || (bx.ex < 0.5 * lx && bx.ey < 0.5 * ly && bx.ez < 0.5 * lz);
        const double sx = shifted && Periodic ? lx : 0.0, sy = shifted && Periodic ? ly : 0.0;
        const double sz = shifted && Periodic ? lz : 0.0;
        // a lane without a particle is infinitely far from everything
        const float inf = __int_as_float(0x7f800000);
        const float gx = mine ? float(pi.x - bx.cx) : inf, gy = mine ? float(pi.y - bx.cy) : inf;
        const float gz = mine ? float(pi.z - bx.cz) : inf, gh = mine ? float(hinv2) : 1.0f;
        const float2 gx2 = make_float2(gx, gx), gy2 = make_float2(gy, gy), gz2 = make_float2(gz, gz);
        const float2 gh2 = make_float2(gh, gh);
        const float Lx = float(lx), Ly = float(ly), Lz = float(lz);
        if (ng == 1)
        {
            // A single particle (mostly a cut group, of thousands of candidates, alone on its
            // multiprocessor at the end of an iteration): the p-th candidate that passes the
            // filter belongs to lane p mod 32, which keeps its own compensated partial sums,
            // combined in FP64 at the end.  A pair is evaluated where it was loaded and its
            // terms handed over, so four loads of 32 run side by side: one after the other
            // (through the ring) each waits out the last one's arithmetic (six mixed sets of
            // 6,000 to 114,000 particles: 12.9 -> 11.1 ms).
            const float x0 = __shfl_sync(0xffffffffu, gx, 0), y0 = __shfl_sync(0xffffffffu, gy, 0);
            const float z0 = __shfl_sync(0xffffffffu, gz, 0), h0 = __shfl_sync(0xffffffffu, gh, 0);
            const float none = __int_as_float(0x7fc00000);
            const uint32_t lt = (1u << lane) - 1u;
            float2* terms = reinterpret_cast<float2*>(scr);   // [4][32], by owner
            KahanF2 one;
            uint32_t passed = 0;
            src.template for_ranges<Periodic>(bx, lx, ly, lz, rbp, [&](uint32_t s0, uint32_t len, int nb, bool) {
                const uint32_t incl = warp_incl_scan_u32(len);
                const uint32_t excl = incl - len;
                const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
                for (uint32_t p0 = 0; p0 < total; p0 += 128)
                {
                    double4 pj[4];
                    bool pass[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                    {
                        const uint32_t p = p0 + 32 * u + lane;
                        int t = 0;
#pragma unroll
                        for (int step = 16; step > 0; step >>= 1)
                        {
                            const uint32_t e = __shfl_sync(0xffffffffu, excl, (t + step) & 31);
                            if (t + step < nb && e <= p) t += step;
                        }
                        const uint32_t j =
                            __shfl_sync(0xffffffffu, s0, t) + (p - __shfl_sync(0xffffffffu, excl, t));
                        pass[u] = p < total;
                        pj[u] = make_double4(0, 0, 0, 0);
                        if (pass[u]) pj[u] = ldg4(src.xyzh + j);
                    }
                    uint32_t m[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                    {
                        pass[u] = pass[u] && gather(pj[u]);
                        m[u] = __ballot_sync(0xffffffffu, pass[u]);
                    }
                    uint32_t at[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                    {
                        at[u] = passed;
                        passed += __popc(m[u]);
                        const float fx = float(image_offset(pj[u].x, bx.cx, sx));
                        const float fy = float(image_offset(pj[u].y, bx.cy, sy));
                        const float fz = float(image_offset(pj[u].z, bx.cz, sz));
                        float dx = x0 - fx, dy = y0 - fy, dz = z0 - fz;
                        if (Periodic && !shifted)
                        {
                            dx = axis_df<true>(x0, fx, Lx);
                            dy = axis_df<true>(y0, fy, Ly);
                            dz = axis_df<true>(z0, fz, Lz);
                        }
                        const float q2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx)) * h0;
                        const bool acc = pass[u] && q2 < float(kRadK2);
                        float2 v = make_float2(none, 0.0f);
                        if (acc)
                        {
                            const float q = sqrt_q(q2);
                            float wk, dwk;
                            sph_kernel_f(q2, q, wk, dwk);
                            v = make_float2(wk, fmaf(-q, dwk, -3.0f * wk));
                        }
                        if (pass[u]) terms[32 * u + ((at[u] + __popc(m[u] & lt)) & 31)] = v;
                        gp += __popc(__ballot_sync(0xffffffffu, acc));
                    }
                    __syncwarp();
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (((lane - at[u]) & 31u) < uint32_t(__popc(m[u])))
                        {
                            const float2 v = terms[32 * u + lane];
                            if (v.x == v.x) one.add(v.x, v.y);
                        }
                    __syncwarp();
                }
            });
            gc = passed;
            double a = one.first(), b = one.second();
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
            {
                a += __shfl_xor_sync(0xffffffffu, a, o);
                b += __shfl_xor_sync(0xffffffffu, b, o);
            }
            rhoi = a;
            gradhi = b;
            return;
        }
        if (few)
        {
            if (lane < kFew)
            {
                member[lane] = gx;
                member[kFew + lane] = gy;
                member[2 * kFew + lane] = gz;
                member[3 * kFew + lane] = gh;
            }
            __syncwarp();
        }
        KahanF2 sums;
        int kept = 0;
        auto evaluate = [&]() {
            if (few)
            {
                // every lane evaluates, the owners add
                __syncwarp();
                for (int i = 0; i < ng; ++i)
                {
                    const int c = __shfl_sync(0xffffffffu, kept, i);
                    float* w = columns + 2 * room * i;
                    for (int t = lane; t < c; t += 32)
                    {
                        const float q2 = w[t];
                        const float q = sqrt_q(q2);
                        float wk, dwk;
                        sph_kernel_f(q2, q, wk, dwk);
                        w[t] = wk;
                        w[room + t] = fmaf(-q, dwk, -3.0f * wk);
                    }
                }
                __syncwarp();
#pragma unroll 4
                for (int t = 0; t < kept; ++t) sums.add(column[t], column[room + t]);
            }
            else
#pragma unroll 2
                for (int t = 0; t < kept; ++t)
                {
                    const float q2 = column[32 * t];
                    const float q = sqrt_q(q2);
                    float wk, dwk;
                    sph_kernel_f(q2, q, wk, dwk);
                    sums.add(wk, fmaf(-q, dwk, -3.0f * wk));
                }
            gp += kept;
            kept = 0;
            __syncwarp();
        };
        src.template stream<false, true, false, Periodic, Staged>(
            nullptr, reinterpret_cast<float4*>(rx), nullptr, bx, sx, sy, sz, lx, ly, lz, gather,
            [&](const double4*, const float4*, const int*, int head, int count) {
                gc += count;
                // full batches start at a multiple of 32; a partial (last) one is filled up
                // with candidates infinitely far the other way
                if (lane >= count) rx[(head + lane) & (kRing - 1)] = inf;
                __syncwarp();
                if (__any_sync(0xffffffffu, kept > room - 32)) evaluate();
                if (few)
                {
                    // a candidate a lane (none beyond count: infinitely far), two particles
                    // a packed instruction
                    const int at = (head + lane) & (kRing - 1);
                    const float fx = rx[at], fy = rx[kRing + at], fz = rx[2 * kRing + at];
                    const uint32_t lt = (1u << lane) - 1u;
                    for (int i0 = 0; i0 < ng; i0 += 2)
                    {
                        const float2 mx = *reinterpret_cast<const float2*>(member + i0);
                        const float2 my = *reinterpret_cast<const float2*>(member + kFew + i0);
                        const float2 mz = *reinterpret_cast<const float2*>(member + 2 * kFew + i0);
                        const float2 mh = *reinterpret_cast<const float2*>(member + 3 * kFew + i0);
                        float2 q2;
                        if (!Periodic || shifted)
                        {
                            const float2 dx = __fadd2_rn(mx, make_float2(fx, fx));
                            const float2 dy = __fadd2_rn(my, make_float2(fy, fy));
                            const float2 dz = __fadd2_rn(mz, make_float2(fz, fz));
                            float2 r2 = __fmul2_rn(dx, dx);
                            r2 = __ffma2_rn(dy, dy, r2);
                            r2 = __ffma2_rn(dz, dz, r2);
                            q2 = __fmul2_rn(r2, mh);
                        }
                        else
                        {
                            const float ax = axis_df<true>(mx.x, -fx, Lx), bx = axis_df<true>(mx.y, -fx, Lx);
                            const float ay = axis_df<true>(my.x, -fy, Ly), by = axis_df<true>(my.y, -fy, Ly);
                            const float az = axis_df<true>(mz.x, -fz, Lz), bz = axis_df<true>(mz.y, -fz, Lz);
                            q2 = make_float2(fmaf(az, az, fmaf(ay, ay, ax * ax)) * mh.x,
                                             fmaf(bz, bz, fmaf(by, by, bx * bx)) * mh.y);
                        }
#pragma unroll
                        for (int u = 0; u < 2; ++u)
                        {
                            const float v = u ? q2.y : q2.x;
                            const bool acc = v < float(kRadK2);
                            const uint32_t m = __ballot_sync(0xffffffffu, acc);
                            const int base = __shfl_sync(0xffffffffu, kept, i0 + u);
                            if (acc) columns[2 * room * (i0 + u) + base + __popc(m & lt)] = v;
                            if (lane == i0 + u) kept += __popc(m);
                        }
                    }
                    return;
                }
                float* put = column + 32 * kept;
                const float* cand = rx + (head & (kRing - 1));
#pragma unroll 1
                for (int k0 = 0; k0 < count; k0 += kTest, cand += kTest)
                {
#pragma unroll
                    for (int k = 0; k < kTest; k += 4)
                    {
                        const float4 X = *reinterpret_cast<const float4*>(cand + k);
                        const float4 Y = *reinterpret_cast<const float4*>(cand + kRing + k);
                        const float4 Z = *reinterpret_cast<const float4*>(cand + 2 * kRing + k);
                        float q2u[4];
                        if (!Periodic || shifted)
                        {
#pragma unroll
                            for (int h = 0; h < 2; ++h)
                            {
                                const float2 dx = __fadd2_rn(gx2, h ? make_float2(X.z, X.w) : make_float2(X.x, X.y));
                                const float2 dy = __fadd2_rn(gy2, h ? make_float2(Y.z, Y.w) : make_float2(Y.x, Y.y));
                                const float2 dz = __fadd2_rn(gz2, h ? make_float2(Z.z, Z.w) : make_float2(Z.x, Z.y));
                                float2 r2 = __fmul2_rn(dx, dx);
                                r2 = __ffma2_rn(dy, dy, r2);
                                r2 = __ffma2_rn(dz, dz, r2);
                                const float2 q2 = __fmul2_rn(r2, gh2);
                                q2u[2 * h] = q2.x;
                                q2u[2 * h + 1] = q2.y;
                            }
                        }
                        else
                        {
                            const float xs[4] = {X.x, X.y, X.z, X.w}, ys[4] = {Y.x, Y.y, Y.z, Y.w};
                            const float zs[4] = {Z.x, Z.y, Z.z, Z.w};
#pragma unroll
                            for (int u = 0; u < 4; ++u)
                            {
                                const float dx = axis_df<true>(gx, -xs[u], Lx);
                                const float dy = axis_df<true>(gy, -ys[u], Ly);
                                const float dz = axis_df<true>(gz, -zs[u], Lz);
                                q2u[u] = fmaf(dz, dz, fmaf(dy, dy, dx * dx)) * gh;
                            }
                        }
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            if (q2u[u] < float(kRadK2))
                            {
                                *put = q2u[u];
                                put += 32;
                            }
                    }
                }
                kept = int(put - column) >> 5;
            },
            rbp);
        evaluate();
        rhoi = sums.first();
        gradhi = sums.second();
    }
}

} // namespace cosmo
