/*
 * force.cu -- the SPH force pass over the symmetric j-leaf lists: per-particle factors
 * (src/force.cu:92-137), pressure + artificial-viscosity accelerations, du/dt, vsigmax
 * and div v (src/force.cu:145-383), and the list rebuild with its hmax upsweep
 * (src/force.cu:19-88).  One warp per i-leaf; j runs in ascending Hilbert index, as the
 * oracle's, so the plain FP64 results agree with it bit for bit.
 */
#include <algorithm>

#include "near.cuh"
#include "pairstream.cuh"
#include "rows.cuh"
#include "state.hpp"
#include "workitems.cuh"

namespace cosmo {

namespace {

constexpr int kWarpsPerBlock = 4;
constexpr int kThreads = 32 * kWarpsPerBlock;

// The per-particle factors.  grkfac (prepB.x) is also written to the unused fourth
// component of vel4, so that a pair reads the j side's velocity and grkfac in one 32-byte
// record; the pair derives the j side's pr and auterm from prepA and thermo4 with the
// prep's own operations, so those are the same bits as prepB.y and prepB.z.
__global__ void force_prep_kernel(const double4* __restrict__ xyzh, const double* __restrict__ gradh,
                                  const double4* __restrict__ thermo4, int n, double pmass, double alphau,
                                  double hfact, double4* __restrict__ prepA, double4* __restrict__ prepB,
                                  double4* __restrict__ vel4, DevScalars* __restrict__ ds)
{
    const long i = long(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i == 0) ds->pairs[2] = 0;   // the force pass's pair counter
    if (i >= n) return;
    const double hi = xyzh[i].w;
    if (!(hi > 0.0))
    {
        prepA[i] = make_double4(0, 0, 0, 0);
        prepB[i] = make_double4(0, 0, 0, 0);
        vel4[i].w = 0.0;
        return;
    }
    const double hsq = 1.0 / (hi * hi);
    const double h4 = hsq * hsq;
    const double hfoh = hfact / hi;
    const double rho = pmass * hfoh * hfoh * hfoh;
    const double dhdrho = -hi / (3.0 * rho);
    const double omega = 1.0 - dhdrho * gradh[i];
    const double oinv = (omega > 0.0) ? (1 / omega) : 1.0;
    const double pro2 = thermo4[i].x;
    prepA[i] = make_double4(hsq, 1.0 / hi, rho, 1.0 / rho);
    const double grkfac = h4 * kCnormk * oinv;
    prepB[i] = make_double4(grkfac, pro2 * rho * rho, 0.5 * pmass * (1.0 / rho) * alphau,
                            kCnormk * oinv * h4 / rho);
    vel4[i].w = grkfac;
}

// The terms of one pair's force, put in the sums' own order: the i-side pressure (added), the
// j-side pressure (subtracted), the four energy terms (pdV, shock, the two conductions, added
// one after the other to one sum), div v, and the signal velocity (a maximum).
constexpr int kForceTerms = 12;
enum : int { kFix = 0, kFiy, kFiz, kFjx, kFjy, kFjz, kFpdv, kFdiss, kFcondi, kFcondj, kFdiv, kFvs };

// The i-side quantities of one particle and its force sums.
struct ForceAcc
{
    double4 p, v, t, a, b;      // xyzh, vel4, thermo4, prepA, prepB of i
    double itx = 0, ity = 0, itz = 0, jtx = 0, jty = 0, jtz = 0;
    double f4s = 0.0, vsm = 0.0, divs = 0.0;
    unsigned int gp = 0;

    __device__ __forceinline__ void load(uint32_t i, const double4* __restrict__ xyzh,
                                         const double4* __restrict__ vel4, const double4* __restrict__ thermo4,
                                         const double4* __restrict__ prepA, const double4* __restrict__ prepB)
    {
        p = xyzh[i]; v = vel4[i]; t = thermo4[i]; a = prepA[i]; b = prepB[i];
    }

    // One pair with j (src/force.cu:232-383): the exact tests dr^2 > 0 and
    // dr^2 < R^2 max(h_i^2, h_j^2)(1 + 1e-10), then the i-side and j-side terms, handed to
    // put(k, value) in the order of the sums (a side outside its support hands none).  The j
    // side is four 32-byte records (xyzh, prepA, vel4 with grkfac, thermo4).  Returns whether
    // either side took it.
    template<bool Periodic, bool Disc, class Put>
    __device__ __forceinline__ bool terms(const double4& pj, int j, const double4* __restrict__ vel4,
                                          const double4* __restrict__ thermo4, const double4* __restrict__ prepA,
                                          double lx, double ly, double lz, double pm, double alphau, double beta,
                                          int pdv, int shock, Put&& put) const
    {
        double dx = p.x - pj.x, dy = p.y - pj.y, dz = p.z - pj.z;
        nearest_image<Periodic>(dx, dy, dz, lx, ly, lz);
        const double dr2 = pair_r2(dx, dy, dz);
        if (!(dr2 > 0.0)) return false;
        const double hi = p.w, hj = pj.w;
        if (dr2 >= kRadK2 * fmax(hi * hi, hj * hj) * (1.0 + 1e-10)) return false;
        const double pro2i = t.x, vwavei = t.y, alphai = t.z, eni = t.w;
        const double hsqinvi = a.x, hinvi = a.y, rhoi = a.z, rho1i = a.w;
        const double grkfaci = b.x, pri = b.y, autermi = b.z;
        const double4 aj = ldg4(prepA + j);
        const double qi2 = dr2 * hsqinvi;
        const double qj2 = dr2 * aj.x;
        const double dr = sqrt(dr2);
        const double rij1 = 1.0 / dr;
        const double rx = dx * rij1, ry = dy * rij1, rz = dz * rij1;
        const double4 vj = ldg4(vel4 + j);
        const double dvx = v.x - vj.x, dvy = v.y - vj.y, dvz = v.z - vj.z;
        const double projv = dvx * rx + dvy * ry + dvz * rz;
        const double4 tj = ldg4(thermo4 + j);
        const double rhoj = aj.z, rho1j = aj.w, pro2j = tj.x;
        const double vwavej = tj.y, alphaj = tj.z, enj = tj.w;
        // the prep's pro2 * rho * rho and 0.5 * pmass * (1 / rho) * alphau, operation for
        // operation
        const double prj = pro2j * rhoj * rhoj, autermj = 0.5 * pm * rho1j * alphau;
        const double vsigi = fmax(vwavei - beta * projv, 0.0);
        const double vsigavi = fmax(alphai * vwavei - beta * projv, 0.0);
        const double vsigj = fmax(vwavej - beta * projv, 0.0);
        const double vsigavj = fmax(alphaj * vwavej - beta * projv, 0.0);
        const double pvs = fmax(vsigi, vsigj);
        double qr2i = 0.0, qr2j = 0.0;
        const double denij = eni - enj;
        const double vsigu = sqrt(fabs(pri - prj) * (2.0 / (rhoi + rhoj)));
        if (Disc)
        {
            const double hori = hi * rij1, horj = hj * rij1;
            if (projv < 0.0)
            {
                qr2i = -0.5 * rho1i * (alphai * vwavei - beta * projv) * hori * projv;
                qr2j = -0.5 * rho1j * (alphaj * vwavej - beta * projv) * horj * projv;
            }
            else
            {
                qr2i = -0.5 * rho1i * alphai * vwavei * hori * projv;
                qr2j = -0.5 * rho1j * alphaj * vwavej * horj * projv;
            }
        }
        else if (projv < 0.0)
        {
            qr2i = -0.5 * rho1i * vsigavi * projv;
            qr2j = -0.5 * rho1j * vsigavj * projv;
        }
        bool took = false;
        if (qi2 < kRadK2)
        {
            took = true;
            put(kFvs, pvs);
            double wk, dwk;
            const double q = dr * hinvi;
            sph_kernel(qi2, q, wk, dwk);
            put(kFdiv, pm * dwk * projv);
            const double gki = dwk * grkfaci;
            const double gpi = pm * (pro2i + qr2i) * gki;
            put(kFix, -gpi * rx); put(kFiy, -gpi * ry); put(kFiz, -gpi * rz);
            const double pdvi = pm * pro2i * projv * gki;
            const double dissi = Disc ? -0.5 * pm * rho1i * alphai * vwavei * (hi * rij1) * projv * projv * gki
                                      : pm * qr2i * projv * gki;
            const double condi = vsigu * denij * autermi * gki;
            if (pdv) put(kFpdv, pdvi);
            if (shock) put(kFdiss, dissi);
            put(kFcondi, condi);
        }
        if (qj2 < kRadK2)
        {
            took = true;
            put(kFvs, pvs);
            double wk, dwk;
            const double q = dr * aj.y;
            sph_kernel(qj2, q, wk, dwk);
            const double gkj = dwk * vj.w;
            const double gpj = pm * (pro2j + qr2j) * gkj;
            put(kFjx, gpj * rx); put(kFjy, gpj * ry); put(kFjz, gpj * rz);
            put(kFcondj, vsigu * denij * autermj * gkj);
        }
        return took;
    }

    // The pair's terms added to the sums.
    template<bool Periodic, bool Disc>
    __device__ __forceinline__ void add(const double4& pj, int j, const double4* __restrict__ vel4,
                                        const double4* __restrict__ thermo4, const double4* __restrict__ prepA,
                                        double lx, double ly, double lz, double pm, double alphau, double beta,
                                        int pdv, int shock)
    {
        const bool took = terms<Periodic, Disc>(pj, j, vel4, thermo4, prepA, lx, ly, lz, pm, alphau, beta, pdv, shock,
                                                [&](int k, double x) {
            switch (k)
            {
                case kFix: itx += x; break;
                case kFiy: ity += x; break;
                case kFiz: itz += x; break;
                case kFjx: jtx -= x; break;
                case kFjy: jty -= x; break;
                case kFjz: jtz -= x; break;
                case kFdiv: divs += x; break;
                case kFvs: vsm = fmax(vsm, x); break;
                default: f4s += x;
            }
        });
        if (took) ++gp;
    }

    __device__ __forceinline__ void store(uint32_t i, double* __restrict__ fx, double* __restrict__ fy,
                                          double* __restrict__ fz, double* __restrict__ f4,
                                          double* __restrict__ vsigmax, double* __restrict__ divvF) const
    {
        fx[i] = itx + jtx;
        fy[i] = ity + jty;
        fz[i] = itz + jtz;
        f4[i] = f4s;
        vsigmax[i] = vsm;
        divvF[i] = -divs * b.w;
    }
};

// Force pass over the group path (one warp per i-leaf, the symmetric list streamed in
// ascending j) for the particles whose rows overflowed (nblCount > kNbl), or for all when
// nblCount is null.
template<bool Periodic, bool Disc>
__global__ void __launch_bounds__(kThreads)
force_kernel(int nL, const uint32_t* __restrict__ layout, const uint32_t* __restrict__ jOffset,
             const uint32_t* __restrict__ jcount, const int* __restrict__ jlist, const double4* __restrict__ xyzh,
             const double4* __restrict__ vel4, const double4* __restrict__ thermo4,
             const double4* __restrict__ prepA, const double4* __restrict__ prepB, double* __restrict__ fx,
             double* __restrict__ fy, double* __restrict__ fz, double* __restrict__ f4,
             double* __restrict__ vsigmax, double* __restrict__ divvF, double pmass, double alphau, double beta,
             int pdv, int shock, const DevBox* __restrict__ box, const int* __restrict__ nblCount,
             DevScalars* __restrict__ ds)
{
    __shared__ double4 sRing[kWarpsPerBlock][kRing];
    __shared__ float4 sRingF[kWarpsPerBlock][kRing];
    __shared__ int sIdx[kWarpsPerBlock][kRing];
    const int wib = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int warpGlobal = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nWarps = (gridDim.x * blockDim.x) >> 5;
    double lx = 0, ly = 0, lz = 0;
    if (Periodic) { lx = box->len[0]; ly = box->len[1]; lz = box->len[2]; }
    unsigned long long pairs = 0;
    const double pm = pmass;
    if (nblCount != nullptr && ds->rowOverflow == 0) return;   // every row complete: nothing to do
    auto wanted = [&](uint32_t a) { return nblCount == nullptr || !row_ok(nblCount, a); };
    for (int leaf = warpGlobal; leaf < nL; leaf += nWarps)
    {
        const uint32_t p0 = layout[leaf], p1 = layout[leaf + 1];
        const uint32_t jb = jOffset[leaf], nj = jcount[leaf];
        for (uint32_t g = p0; g < p1; g += 64)
        {
          const uint32_t m0 = __ballot_sync(0xffffffffu, g + lane < p1 && wanted(g + lane));
          const uint32_t m1 = __ballot_sync(0xffffffffu, g + 32 + lane < p1 && wanted(g + 32 + lane));
          const int nAct = __popc(m0) + __popc(m1);
          const int G = (nAct + 31) >> 5;
          for (int grp = 0; grp < G; ++grp)
          {
            const int slot = group_slot(m0, m1, nAct, grp, G, lane);
            const bool mine = slot >= 0;
            const uint32_t i = g + uint32_t(mine ? slot : 0);
            ForceAcc A;
            A.load(i, xyzh, vel4, thermo4, prepA, prepB);
            const double hi = A.p.w;
            const double rg = kRadKernel * warp_max(mine ? hi : 0.0);
            const GroupBox bx = group_box(mine, A.p.x, A.p.y, A.p.z, 0.0, rg);
            // float prefilter: r_f^2 <= (R max(h_i, h_j) (1 + 1e-5) + margin)^2; the exact
            // tests run in the accept pass
            const float xf = float(A.p.x - bx.cx), yf = float(A.p.y - bx.cy), zf = float(A.p.z - bx.cz);
            const float mf = __double2float_ru(fp32_margin(bx, Periodic ? fmax(lx, fmax(ly, lz)) : 0.0) +
                                               1e-6 * rg);
            const float hif = float(hi);
            const float Lx = float(lx), Ly = float(ly), Lz = float(lz);
            stream_pairs(
                sRing[wib], sRingF[wib], sIdx[wib], bx.cx, bx.cy, bx.cz, jb, nj, jlist, layout, xyzh,
                [&](const double4& pj) { return in_sym_box<Periodic>(pj, bx, rg, lx, ly, lz); },
                [&](const double4* ring, const float4* ringf, const int* ringIdx, int head, int count) {
                  two_pass(ring, ringf, ringIdx, head, count, mine,
                  [&](const float4& pf) {
                    const float r = fmaf(float(kRadKernel) * 1.00001f, fmaxf(hif, pf.w), mf);
                    return r2_f32<Periodic>(xf, yf, zf, pf, Lx, Ly, Lz) <= r * r;
                  },
                  [&](const double4& pj, const float4&, int j) {
                    A.add<Periodic, Disc>(pj, j, vel4, thermo4, prepA, lx, ly, lz, pm, alphau, beta, pdv, shock);
                  });
                });
            if (!mine) continue;
            pairs += A.gp;
            A.store(i, fx, fy, fz, f4, vsigmax, divvF);
          }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
    if (lane == 0) atomicAdd(&ds->pairs[2], pairs);
}

// Symmetric rows: every live particle's j with dr^2 < R^2 max(h_i^2, h_j^2)(1 + 1e-10),
// ascending -- the force pass's pairs (which also need dr^2 > 0, tested where the row is
// used) and, at the converged h, every pair of the gather sweep (i itself included).
template<bool Periodic>
__global__ void __launch_bounds__(kThreads)
sym_rows_kernel(const int4* __restrict__ items, int cap, const uint32_t* __restrict__ layout,
                const uint32_t* __restrict__ jOffset, const uint32_t* __restrict__ jcount,
                const int* __restrict__ jlist, const double4* __restrict__ xyzh, const DevBox* __restrict__ box,
                const float4* __restrict__ leafBox, const double* __restrict__ hmaxLeaf, int* __restrict__ nbl,
                int* __restrict__ nblCount, DevScalars* __restrict__ ds, int prefilter)
{
    __shared__ __align__(16) unsigned char sScr[kWarpsPerBlock][kRowsScratch];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    double lx = 0, ly = 0, lz = 0;
    if (Periodic) { lx = box->len[0]; ly = box->len[1]; lz = box->len[2]; }
    const int nHeavy = ds->itemsHeavy, nItems = nHeavy + ds->itemsLight;
    for (;;)
    {
        const int w = next_item(ds, nHeavy, nItems, cap);
        if (w < 0) break;
        const Item d = decode_item(items[w], layout);
        const int slot = group_slot(d.m0, d.m1, d.nAct, d.grp, d.G, lane);
        const bool mine = slot >= 0;
        const uint32_t i = d.g0 + uint32_t(mine ? slot : 0);
        const double4 pi = xyzh[i];
        const double rg = kRadKernel * warp_max(mine ? pi.w : 0.0);
        const GroupBox bx = group_box(mine, pi.x, pi.y, pi.z, 0.0, rg);
        int rowLen = 0;
        // the force pass's test dr^2 < R^2 max(h_i^2, h_j^2)(1 + 1e-10), with each side's
        // bound formed once: rounding is monotone, so the bound of the larger h is the
        // larger bound and max(bound_i, bound_j) is the same double as the test's own
        auto bound = [](double h) { return kRadK2 * (h * h) * (1.0 + 1e-10); };
        // prefilter distances: R h (1 + 1e-10) bounds sqrt(bound(h)) for either side
        auto filt = [&](const double4& pj) { return in_sym_box<Periodic>(pj, bx, rg, lx, ly, lz); };
        // the listed leaves within the group's supports or their own
        auto ranges = near_ranges<Periodic>(LayoutRanges{layout}, leafBox,
                                            group_region<Periodic>(bx, rg * (1.0 + 1e-8), lx, ly, lz));
        ranges.hmaxLeaf = hmaxLeaf;
        auto candB = [](const double4& pj) { return kRadKernel * pj.w * (1.0 + 1e-10); };
        auto exact = [&](const double4& g, const double4& pj, int j) {
            double dx = g.x - pj.x, dy = g.y - pj.y, dz = g.z - pj.z;
            nearest_image<Periodic>(dx, dy, dz, lx, ly, lz);
            const double dr2 = pair_r2(dx, dy, dz);
            return RowEntry<int>{!(dr2 >= fmax(g.w, bound(pj.w))), j};
        };
        int* myRow = mine ? row_of(nbl, uint32_t(i)) : nullptr;
        const double4 gi = make_double4(pi.x, pi.y, pi.z, bound(pi.w));
        const double Bi = kRadKernel * pi.w * (1.0 + 1e-10);
        if (prefilter)
            rows_group<kRowStride, Periodic, true>(sScr[wib], mine, d.ng, gi, Bi, bx, lx, ly, lz, jOffset[d.leaf],
                                                   jcount[d.leaf], jlist, ranges, xyzh, filt, candB,
                                                   exact, myRow, rowLen);
        else
            rows_group<kRowStride, Periodic, false>(sScr[wib], mine, d.ng, gi, Bi, bx, lx, ly, lz, jOffset[d.leaf],
                                                    jcount[d.leaf], jlist, ranges, xyzh, filt, candB,
                                                    exact, myRow, rowLen);
        if (mine) nblCount[i] = rowLen;
        if (mine && rowLen > kNbl) ds->rowOverflow = 1;
    }
}

// Force pass over the rows: one lane per live particle, its row's pairs in ascending j --
// the group pass's pairs and order, so the results agree with it bit for bit.
template<bool Periodic, bool Disc>
__global__ void __launch_bounds__(kThreads)
force_row_kernel(int nAlive, const int* __restrict__ nbl, const int* __restrict__ nblCount,
                 const double4* __restrict__ xyzh, const double4* __restrict__ vel4,
                 const double4* __restrict__ thermo4, const double4* __restrict__ prepA,
                 const double4* __restrict__ prepB, double* __restrict__ fx, double* __restrict__ fy,
                 double* __restrict__ fz, double* __restrict__ f4, double* __restrict__ vsigmax,
                 double* __restrict__ divvF, double pmass, double alphau, double beta, int pdv, int shock,
                 const DevBox* __restrict__ box, DevScalars* __restrict__ ds)
{
    double lx = 0, ly = 0, lz = 0;
    if (Periodic) { lx = box->len[0]; ly = box->len[1]; lz = box->len[2]; }
    unsigned long long pairs = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nAlive; i += gridDim.x * blockDim.x)
    {
        if (!row_ok(nblCount, uint32_t(i))) continue;
        const int cnt = nblCount[i];
        ForceAcc A;
        A.load(uint32_t(i), xyzh, vel4, thermo4, prepA, prepB);
        const int* row = row_of(nbl, uint32_t(i));
        auto pair = [&](int j) {
            A.add<Periodic, Disc>(ldg4(xyzh + j), j, vel4, thermo4, prepA, lx, ly, lz, pmass, alphau, beta,
                                  pdv, shock);
        };
        for_row(row, cnt, pair);
        pairs += A.gp;
        A.store(uint32_t(i), fx, fy, fz, f4, vsigmax, divvF);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(&ds->pairs[2], pairs);
}

// Force pass with one warp per particle: 32 of its pairs at a time are evaluated, one per lane,
// and their terms added in ascending j with one sum per lane (a term a pair does not have is
// zero, which leaves its sum as it is).  Rows: all live particles of a small set over their
// rows.  Otherwise the particles without a row (the block-tree solve's over list), each over a
// search of its own support and every block's.
template<bool Periodic, bool Disc, bool Rows>
__global__ void __launch_bounds__(kThreads)
force_warp_kernel(const __grid_constant__ NearTree t, int n, const int* __restrict__ over, const int* __restrict__ nbl,
                  const int* __restrict__ nblCount, const double4* __restrict__ vel4,
                  const double4* __restrict__ thermo4, const double4* __restrict__ prepA,
                  const double4* __restrict__ prepB, double* __restrict__ fx, double* __restrict__ fy,
                  double* __restrict__ fz, double* __restrict__ f4, double* __restrict__ vsigmax,
                  double* __restrict__ divvF, double pmass, double alphau, double beta, int pdv, int shock,
                  DevScalars* __restrict__ ds)
{
    __shared__ NearScratch sScr[Rows ? 1 : kWarpsPerBlock];
    __shared__ double sTerm[kWarpsPerBlock][32 * (kForceTerms + 1)];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    constexpr int kStride = kForceTerms + 1;
    const NearFrame f(t.box);
    const NearView v = near_view(t, f);
    double lx = 0, ly = 0, lz = 0;
    if (Periodic) { lx = t.box->len[0]; ly = t.box->len[1]; lz = t.box->len[2]; }
    double* term = sTerm[wib];
    const bool energy = lane == 6, largest = lane == 8;
    const int first = lane < 6 ? kFix + lane : (lane == 6 ? kFpdv : (lane == 7 ? kFdiv : kFvs));
    unsigned long long pairs = 0;
    for (int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < n; w += (gridDim.x * blockDim.x) >> 5)
    {
        const int i = Rows ? w : over[w];
        const int cnt = Rows ? nblCount[i] : 0;
        if (Rows && unsigned(cnt) > unsigned(kNbl)) continue;
        ForceAcc A;
        A.load(uint32_t(i), t.xyzh, vel4, thermo4, prepA, prepB);
        // lanes 0-5: the pressure sums (the j side's terms stored negated), 6: the energy, 7:
        // div v, 8: vsig.  Every lane runs the energy's four additions, zeros for the others
        double sum = 0.0;
        auto pair = [&](const double4& pj, int j, bool valid) {
            double* mine = term + lane * kStride;
#pragma unroll
            for (int k = 0; k < kForceTerms; ++k) mine[k] = 0.0;
            const bool took = valid && A.terms<Periodic, Disc>(pj, j, vel4, thermo4, prepA, lx, ly, lz, pmass, alphau,
                                                               beta, pdv, shock,
                                                               [&](int k, double x) {
                                                                   mine[k] = k >= kFjx && k <= kFjz ? -x : x;
                                                               });
            A.gp += __popc(__ballot_sync(0xffffffffu, took));
            __syncwarp();
            const int c = 32 - __clz(__ballot_sync(0xffffffffu, valid));
#pragma unroll 4
            for (int k = 0; k < c; ++k)
            {
                const double* q = term + k * kStride;
                const double x0 = q[first], x1 = energy ? q[kFdiss] : 0.0;
                const double x2 = energy ? q[kFcondi] : 0.0, x3 = energy ? q[kFcondj] : 0.0;
                sum = largest ? fmax(sum, x0) : sum + x0;
                sum += x1;
                sum += x2;
                sum += x3;
            }
            __syncwarp();
            return true;
        };
        if constexpr (Rows)
        {
            const int* row = row_of(nbl, uint32_t(i));
            for (int k0 = 0; k0 < cnt; k0 += 32)
            {
                const bool valid = k0 + lane < cnt;
                const int j = valid ? row[size_t(k0 + lane) * kRowStride] : i;
                pair(ldg4(t.xyzh + j), j, valid);
            }
        }
        else
        {
            const float3 a = f.at(A.p);
            const float x = a.x, y = a.y, z = a.z;
            const float slack = f.slack(x, y, z);
            const float r = f.length(kRadKernel * (1.0 + 1e-6) * A.p.w) + slack;
            // the exact tests terms() starts with
            auto inside = [&](const double4& pj) {
                double dx = A.p.x - pj.x, dy = A.p.y - pj.y, dz = A.p.z - pj.z;
                nearest_image<Periodic>(dx, dy, dz, lx, ly, lz);
                const double dr2 = pair_r2(dx, dy, dz);
                return dr2 > 0.0 && !(dr2 >= kRadK2 * fmax(A.p.w * A.p.w, pj.w * pj.w) * (1.0 + 1e-10));
            };
            auto pairs32 = [&](int j, int count) { pair(ldg4(t.xyzh + j), j, lane < count); };
            int held = 0;
            near_blocks<0, Periodic, true>(t, v, sScr[wib], x, y, z, 0.0f, 0.0f, 0.0f, r, slack, [&](int nb) -> float {
                near_packed(sScr[wib], nb, v.n, t.xyzh, held, inside, pairs32);
                return r;
            });
            near_packed_end(sScr[wib], held, pairs32);
        }
        A.itx = __shfl_sync(0xffffffffu, sum, 0); A.ity = __shfl_sync(0xffffffffu, sum, 1);
        A.itz = __shfl_sync(0xffffffffu, sum, 2); A.jtx = __shfl_sync(0xffffffffu, sum, 3);
        A.jty = __shfl_sync(0xffffffffu, sum, 4); A.jtz = __shfl_sync(0xffffffffu, sum, 5);
        A.f4s = __shfl_sync(0xffffffffu, sum, 6);
        A.divs = __shfl_sync(0xffffffffu, sum, 7);
        A.vsm = __shfl_sync(0xffffffffu, sum, 8);
        if (lane == 0)
        {
            pairs += A.gp;
            A.store(uint32_t(i), fx, fy, fz, f4, vsigmax, divvF);
        }
    }
    if (lane == 0 && pairs) atomicAdd(&ds->pairs[2], pairs);
}

// Dead particles: no force (src/force.cu:191-200).
__global__ void force_dead_kernel(int nAlive, int n, double* fx, double* fy, double* fz, double* f4,
                                  double* vsigmax, double* divvF)
{
    const long i = nAlive + long(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    fx[i] = 0.0; fy[i] = 0.0; fz[i] = 0.0; f4[i] = 0.0; vsigmax[i] = 0.0; divvF[i] = 0.0;
}

} // namespace

void build_symmetric(State& s)
{
    DevScalars* ds = s.dscal.get();
    ensure_tree(s);
    const int nL = s.nLeaves;
    hmax_upsweep(s);
    build_lists(s, true);
    if (nL <= 0) return;
    const int grid = std::max(1, std::min(s.numSMs * 8, iceil(nL, kWarpsPerBlock)));
    const int nA = std::max(s.nAlive, 1);
    s.items.resize(nA, s.st);
    s.nbl.resize(row_buffer_entries(size_t(nA)), s.st);
    s.nblCount.resize(nA, s.st);
    begin_iteration_kernel<<<1, 32, 0, s.st>>>(ds, nullptr, 0);
    COSMO_LAUNCHED();
    COSMO_CUDA(cudaMemsetAsync(&ds->rowOverflow, 0, sizeof(int), s.st));
    plan_items_kernel<<<grid, kThreads, 0, s.st>>>(nullptr, nL, s.layout.get(), nullptr, s.jstream.get(),
                                                    s.xyzh.get(), s.items.get(), nA, ds);
    COSMO_LAUNCHED();
    auto rows = s.periodic ? sym_rows_kernel<true> : sym_rows_kernel<false>;
    rows<<<persistent_grid(s, rows, kThreads), kThreads, 0, s.st>>>(
        s.items.get(), nA, s.layout.get(), s.jOffset.get(), s.jcount.get(), s.jlist.get(), s.xyzh.get(),
        s.box.get(), s.leafBox.get(), s.hmaxLeaf.get(), s.nbl.get(), s.nblCount.get(), ds, s.symPrefilter);
    COSMO_LAUNCHED();
}

void compute_forces(State& s, double pmass, double beta, double alphau, bool disc, bool pdv, bool shock)
{
    const int n = s.ngas;
    DevScalars* ds = s.dscal.get();
    cudaEvent_t e0 = ev(s);
    s.forceSinceSolve = true;
    // The symmetric lists and rows are cached per tree (src/force.cu:19-24); the density
    // solve's gradient sweep has normally built the rows already (from the Newton rows, or
    // with the symmetric lists).
    // After a plain solve the mixed pass still goes over the leaves, and it has no walk for
    // particles without a row: they need the lists.
    if (s.precision == 1) ensure_tree(s);
    const bool noRow = s.precision == 1 && s.nearOverCount > 0;
    const bool rowsReady =
        s.rowsToken == s.token && ((s.rowsFromNewton && !noRow) || (s.jlistToken == s.token && s.listsSym));
    if (!rowsReady)
    {
        // positions may have been replaced in the sorted order since the tree was made
        ensure_tree(s);
        if (s.nLeaves > 0) leaf_boxes(s);
        build_symmetric(s);
        s.jlistToken = s.rowsToken = s.token;
        s.rowsFromNewton = false;
        s.hmaxNodeDone = true;
        cudaEvent_t e2 = ev(s);
        COSMO_CUDA(cudaStreamSynchronize(s.st));
        s.t.fjbuild += elapsed_s(e0, e2);
    }
    cudaEvent_t p0 = ev(s);
    force_prep_kernel<<<iceil(n, 256), 256, 0, s.st>>>(s.xyzh.get(), s.gradh.get(), s.thermo4.get(), n, pmass,
                                                       alphau, s.hfact, s.prepA.get(), s.prepB.get(),
                                                       s.vel4.get(), ds);
    COSMO_LAUNCHED();
    cudaEvent_t p1 = ev(s);
    const int nL = s.treeDone ? s.nLeaves : 0;   // the group pass's (no tree: no such pass)
    const int grid = std::max(1, std::min(s.numSMs * 8, iceil(nL, kWarpsPerBlock)));
    auto launch = [&](auto kern) {
        kern<<<grid, kThreads, 0, s.st>>>(nL, s.layout.get(), s.jOffset.get(), s.jcount.get(), s.jlist.get(),
                                          s.xyzh.get(), s.vel4.get(), s.thermo4.get(), s.prepA.get(),
                                          s.prepB.get(), s.fx.get(), s.fy.get(), s.fz.get(), s.f4.get(),
                                          s.vsigmax.get(), s.divvF.get(), pmass, alphau, beta, pdv ? 1 : 0,
                                          shock ? 1 : 0, s.box.get(), s.nblCount.get(), ds);
    };
    auto launchRows = [&](auto kern) {
        kern<<<std::max(1, iceil(s.nAlive, kThreads)), kThreads, 0, s.st>>>(
            s.nAlive, s.nbl.get(), s.nblCount.get(), s.xyzh.get(), s.vel4.get(), s.thermo4.get(), s.prepA.get(),
            s.prepB.get(), s.fx.get(), s.fy.get(), s.fz.get(), s.f4.get(), s.vsigmax.get(), s.divvF.get(), pmass,
            alphau, beta, pdv ? 1 : 0, shock ? 1 : 0, s.box.get(), ds);
    };
    // one lane per particle over its symmetric row; the group pass covers only the rows
    // that overflowed
    if (s.precision == 1)
        launch_force_mixed(s, pmass, beta, disc, pdv, shock);
    else if (s.nAlive > 0)
    {
        auto warps = [&](auto kern, int n, int blocks) {
            kern<<<blocks, kThreads, 0, s.st>>>(
                near_tree(s), n, s.nearOver.get(), s.nbl.get(), s.nblCount.get(), s.vel4.get(), s.thermo4.get(),
                s.prepA.get(), s.prepB.get(), s.fx.get(), s.fy.get(), s.fz.get(), s.f4.get(), s.vsigmax.get(),
                s.divvF.get(), pmass, alphau, beta, pdv ? 1 : 0, shock ? 1 : 0, ds);
            COSMO_LAUNCHED();
        };
        if (s.nAlive <= kWarpPerParticleForce)
        {
            const int blocks = std::max(1, iceil(s.nAlive, kWarpsPerBlock));
            if (s.periodic) { if (disc) warps(force_warp_kernel<true, true, true>, s.nAlive, blocks); else warps(force_warp_kernel<true, false, true>, s.nAlive, blocks); }
            else { if (disc) warps(force_warp_kernel<false, true, true>, s.nAlive, blocks); else warps(force_warp_kernel<false, false, true>, s.nAlive, blocks); }
        }
        else
        {
            if (s.periodic) { if (disc) launchRows(force_row_kernel<true, true>); else launchRows(force_row_kernel<true, false>); }
            else { if (disc) launchRows(force_row_kernel<false, true>); else launchRows(force_row_kernel<false, false>); }
            COSMO_LAUNCHED();
        }
        if (!s.rowsFromNewton)
        {
            // the group pass of the rows that overflowed (none: it returns at once)
            if (s.periodic) { if (disc) launch(force_kernel<true, true>); else launch(force_kernel<true, false>); }
            else { if (disc) launch(force_kernel<false, true>); else launch(force_kernel<false, false>); }
            COSMO_LAUNCHED();
        }
        else if (s.nearOverCount > 0)
        {
            // the particles whose rows would not hold their pairs.  A node's h are those its
            // boxes were made with, at the solve's start: remade at the converged h first
            near_build(s);
            const int m = s.nearOverCount, blocks = std::min(iceil(m, kWarpsPerBlock), 8 * s.numSMs);
            if (s.periodic) { if (disc) warps(force_warp_kernel<true, true, false>, m, blocks); else warps(force_warp_kernel<true, false, false>, m, blocks); }
            else { if (disc) warps(force_warp_kernel<false, true, false>, m, blocks); else warps(force_warp_kernel<false, false, false>, m, blocks); }
        }
    }
    if (n > s.nAlive)
    {
        force_dead_kernel<<<iceil(n - s.nAlive, 256), 256, 0, s.st>>>(s.nAlive, n, s.fx.get(), s.fy.get(),
                                                                      s.fz.get(), s.f4.get(), s.vsigmax.get(),
                                                                      s.divvF.get());
        COSMO_LAUNCHED();
    }
    cudaEvent_t p2 = ev(s);
    read_scalars(s);
    s.t.prep += elapsed_s(p0, p1);
    s.t.fkern += elapsed_s(p1, p2);
    check_dev_err(s, "force_gpu_c", false);
}

} // namespace cosmo
