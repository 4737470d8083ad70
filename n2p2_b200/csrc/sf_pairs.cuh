// Symmetry-function passes of the evaluation path (G values and the adjoint
// force pass), one block of four warps per centre atom; included by one
// translation unit per precision and pass.  They run the models whose angular
// functions have integer zeta and no shift (DevPairTable); the others run the
// kernels of sf_fast.cuh.
//
// Formulas: SymGrpExpRad::calculate (SymGrpExpRad.cpp:144-239),
// SymGrpExpAngn::calculate (SymGrpExpAngn.cpp:156-403),
// SymGrpExpAngw::calculate (SymGrpExpAngw.cpp:156-376).
//
//  * The atom's neighbours are staged once per block in shared memory, sorted
//    by element (stable; by distance within an element when a group's cutoff
//    is below the list's), as 16-byte records: a triplet reads each neighbour
//    with three (G) or four (forces) 16-byte loads.
//  * Candidate pairs (j, k) are tested in FP32 against the squared cutoff
//    plus the test's own rounding error; an accepted pair beyond the cutoff
//    gets f_c = 0, so the results do not depend on the test.  Accepted pairs
//    go to a ring per warp and are evaluated 32 at a time.
//  * Both passes walk rounds of matchings (pair_rounds.cuh); the force pass
//    adds a round's forces to distinct slots of the warp's own force arrays;
//    no atomics.
//  * All sums run in a fixed order: results are bitwise reproducible and do
//    not depend on the stage capacity.
//
// Bound: instruction issue (G 66 %, forces 58 % of the cycles; FP64 pipe 30 %
// and 35 %), then the latency of dependent FP64 and shared-memory
// instructions.  Per water atom (107 neighbours, 2548 narrow triplets, 8
// members) the G pass executes 28.5 k warp instructions: 5.7 k staging, radial
// functions and sums, 11 k candidates, 11.8 k triplets; the force pass 41 k.
// A warp per atom (the former specialised kernels) took 56 k and 73 k: its
// member grids had run-time exponents (selects and branches per factor) and
// every triplet read 14 separate values.  256 water boxes (133 k atoms), FP64:
// G 7.67 -> 4.9 ms, forces 11.1 -> 8.0 ms; mixed 5.10 -> 3.3 and 6.83 ->
// 5.1 ms; one 192-atom box, where the four warps per atom also fill the SMs:
// G 120 -> 26 us, forces 140 -> 33 us; 110,592 atoms with zeta up to 16 and
// wide groups: 15.0 -> 5.4 and 17.1 -> 9.5 ms.
// Not kept: testing rows (one j against 32 k) instead of rounds costs 33 %
// empty lanes; run-time branches over absent zeta slots cost more than summing
// them; the accepted pairs kept in global memory for the force pass save it
// 9 % and cost the G pass 10 %; warp shares that are not multiples of 64
// candidates, and the groups' short blocks started at different warps, change
// nothing (G 2.33 and 2.32 ms, forces 3.82 and 3.82 ms for 96 boxes).
#pragma once

#include <type_traits>

#include "kernels_common.cuh"
#include "kernels.hpp"
#include "pair_rounds.cuh"

namespace n2p2b200 {

namespace {

constexpr int kPairWarps = 4, kPairThreads = kPairWarps * 32;
constexpr int kRing = 128;           // accepted pairs of one warp waiting for a full step (< 32 + 64)
constexpr int kTestPad = 96;         // records past the stage that a warp's last candidates may read (and discard)
constexpr int kSumPitch = 36;        // doubles between the accumulators of warpSums: conflict-free both ways

template <typename T>
struct Pair2;
template <>
struct Pair2<double> { using V = double2; };
template <>
struct Pair2<float> { using V = float2; };

// Coefficients (ln 2 / 64)^n / n! of 2^(f/64), in the constant bank: the FP64
// instructions read them there, a literal costs two moves each.
constexpr double kLn64 = 0.69314718055994530942 / 64.0;
__constant__ double kExpCoef[5] = {kLn64, kLn64* kLn64 / 2.0, kLn64* kLn64* kLn64 / 6.0,
                                   kLn64* kLn64* kLn64* kLn64 / 24.0, kLn64* kLn64* kLn64* kLn64* kLn64 / 120.0};

// exp(-eta s) as 2^(c s / 64), c = -eta 64 / ln 2, -2^30 <= c s <= 0:
// table-driven exponential (P. T. P. Tang, ACM TOMS 15 (1989) 144): c s =
// k + f with |f| <= 1/2, 2^(k/64) from the 64-entry table and k's upper bits,
// 2^(f/64) - 1 by its series to order 5 (truncation 3.5e-17).  WIDE false:
// c s / 64 >= -1000; true: below 2^-1021 the result is 2^-1021 instead of the
// underflowing value (one instruction more: in every triplet it costs the
// passes 1 to 4 %, so only the radial functions and the instances for any
// zeta have it).
template <bool WIDE = false>
__device__ __forceinline__ double expScaled(double s, double c, const double* tab)
{
    constexpr double kShift = 6755399441055744.0;   // 1.5 2^52: adding it rounds to an integer
    double kd = fma(s, c, kShift);
    int k = __double2loint(kd);
    if (WIDE) k = max(k, -64 * 1021);
    kd -= kShift;
    const double f = fma(s, c, -kd);
    const double p = f * fma(f, fma(f, fma(f, fma(f, kExpCoef[4], kExpCoef[3]), kExpCoef[2]), kExpCoef[1]), kExpCoef[0]);
    const double t = tab[k & 63];
    const double w = __hiloint2double(__double2hiint(t) + (int)((unsigned)(k & ~63) << 14), __double2loint(t));
    return fma(w, p, w);
}

// FP32 form: c = -eta / ln 2.
template <bool WIDE = false>
__device__ __forceinline__ float expScaled(float s, float c, const double*)
{
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(s * c));
    return r;
}

// 1/sqrt(s): the hardware's approximation (relative error <= 2^-20) and one
// step of the third-order Householder iteration (residual e^3 5/16 < 1e-17).
__device__ __forceinline__ double invSqrt(double s)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(s));
    const double e = fma(-s * y, y, 1.0);
    return fma(fma(0.375, e, 0.5), y * e, y);
}

__device__ __forceinline__ float invSqrt(float s) { return rsqrtf(s); }

__device__ __forceinline__ double clampZero(double v)
{
    return __double2hiint(v) < 0 ? 0.0 : v;
}

__device__ __forceinline__ float clampZero(float v) { return fmaxf(v, 0.0f); }

// f_c(r) and df_c/dr of a pair.  CUT kCutPoly2: the poly2 function without an inner radius (r_ci = 0),
// f = u^3 (1 + 3x + 6x^2), df/dx = -30 x^2 u^2, x = r/r_c, u = 1 - x (no cancellation at r_c), 0 from r_c on.
constexpr int kCutAny = 0, kCutPoly2 = 6;

template <int CUT, typename T>
__device__ __forceinline__ void pairCutoff(DevCutoff const& c, T iw, T r, T& fc, T& dfc)
{
    if constexpr (CUT == kCutPoly2)
    {
        const T x = r * iw, u = clampZero(T(1) - x), xu = x * u;
        fc = u * u * u * ((T(6) * x + T(3)) * x + T(1));
        dfc = T(-30) * iw * (xu * xu);
    }
    else if constexpr (sizeof(T) == 8) cutoffFdf(c, r, fc, dfc);
    else cutoffFdfF32(c, r, fc, dfc);
}

// What a step needs of its group, in registers.
template <typename T>
struct GroupRegs
{
    T lam0, lam1, scale0, scale1, iw;
    __device__ __forceinline__ GroupRegs(DevPairGroup const& G, DevCutoff const& c)
    {
        if constexpr (sizeof(T) == 4)
        {
            lam0 = G.lambdaF[0];
            lam1 = G.lambdaF[1];
            scale0 = G.etaScaleF[0];
            scale1 = G.etaScaleF[1];
            iw = c.iwF;
        }
        else
        {
            lam0 = G.lambda[0];
            lam1 = G.lambda[1];
            scale0 = G.etaScale[0];
            scale1 = G.etaScale[1];
            iw = c.iw;
        }
    }
};

template <typename T>
__device__ __forceinline__ T groupStageScale(DevPairGroup const& G, int k)
{
    if constexpr (sizeof(T) == 4) return G.stageScaleF[k];
    else return G.stageScale[k];
}

template <typename T>
__device__ __forceinline__ T groupEta2(DevPairGroup const& G, int k)
{
    if constexpr (sizeof(T) == 4) return G.eta2F[k];
    else return G.eta2[k];
}

// x^n, n >= 0 warp-uniform.
template <typename T>
__device__ __forceinline__ T powAny(T x, int n)
{
    T r = T(1);
#pragma unroll 1
    while (n)
    {
        if (n & 1) r *= x;
        n >>= 1;
        if (n) x *= x;
    }
    return r;
}

template <typename T>
__device__ __forceinline__ T radialScale(DevRadial const& M)
{
    if constexpr (sizeof(T) == 4) return M.scaleF;
    else return M.scale;
}

template <typename T>
__device__ __forceinline__ T radialShift(DevRadial const& M)
{
    if constexpr (sizeof(T) == 4) return M.rsF;
    else return M.rs;
}

template <typename T>
__device__ __forceinline__ T radialEta2(DevRadial const& M)
{
    if constexpr (sizeof(T) == 4) return M.eta2F;
    else return M.eta2;
}

// ---------------------------------------------------------------------------
// Stage
// ---------------------------------------------------------------------------

// Per slot: position and 1/r, FP32 test position (the record itself in the
// FP32 form), r, and per pass the factors of the current angular group.
template <typename T, int CAP>
struct StageGeometry;

template <int CAP>
struct StageGeometry<double, CAP>
{
    double2 xy[CAP], zi[CAP];
    float4 test[CAP + kTestPad];
    double r[CAP];
    __device__ __forceinline__ void set(int s, double x, double y, double z, double d)
    {
        xy[s] = make_double2(x, y);
        zi[s] = make_double2(z, 1.0 / d);
        test[s] = make_float4((float)x, (float)y, (float)z, 0.0f);
        r[s] = d;
    }
    // record at byte offset o = 16 slot
    __device__ __forceinline__ void get(int o, double& x, double& y, double& z, double& ri) const
    {
        const double2 a = *reinterpret_cast<const double2*>(reinterpret_cast<const char*>(xy) + o);
        const double2 b = *reinterpret_cast<const double2*>(reinterpret_cast<const char*>(zi) + o);
        x = a.x;
        y = a.y;
        z = b.x;
        ri = b.y;
    }
    __device__ __forceinline__ const float4* records() const { return test; }
    __device__ __forceinline__ double* scratch() { return reinterpret_cast<double*>(xy); }
};

template <int CAP>
struct StageGeometry<float, CAP>
{
    float4 p[CAP + kTestPad];
    float r[CAP];
    __device__ __forceinline__ void set(int s, double x, double y, double z, double d)
    {
        p[s] = make_float4((float)x, (float)y, (float)z, (float)(1.0 / d));
        r[s] = (float)d;
    }
    __device__ __forceinline__ void get(int o, float& x, float& y, float& z, float& ri) const
    {
        const float4 a = *reinterpret_cast<const float4*>(reinterpret_cast<const char*>(p) + o);
        x = a.x;
        y = a.y;
        z = a.z;
        ri = a.w;
    }
    __device__ __forceinline__ const float4* records() const { return p; }
    __device__ __forceinline__ double* scratch() { return reinterpret_cast<double*>(p); }
};

// Enumeration of a group's candidates (pair_rounds.cuh) for this atom.
struct alignas(16) GroupShare
{
    int count, minor, nO, m1;   // candidates, per round, slots of the first block, modulus of the rounds
    int O0, P0, share;          // first slots of the blocks; candidates of one warp, a multiple of 64
    float inv;                  // 1 / minor
};

template <typename T, int CAP>
struct alignas(16) PairStage
{
    static constexpr int kChunks = (CAP + kPairThreads - 1) / kPairThreads * kPairWarps;   // 32-entry chunks
    StageGeometry<T, CAP> geo;
    double expTab[64];
    int queue[kPairWarps][kRing];
    int chunk[kDevMaxElements][kChunks];    // first slot of the element's entries of every chunk
    int begin[kDevMaxElements + 1];
    int nBelow[4][kDevMaxElements];         // per cutoff slot and element: block entries with r < r_c
    GroupShare share[kPairGroups];          // per angular group of the element (setGroupShares)
    short slotOf[CAP];                      // position in the atom's list -> slot
    short perm[CAP];                        // slot -> position
    unsigned todo[kPairWarps];
};

// Neighbours of one atom into the stage.  Ends without a barrier (begin and
// nBelow are complete): the caller adds what belongs to the slots (slotOf of
// the thread's own entries is set) and synchronises.
template <typename T, int CAP>
__device__ __forceinline__ void stageNeighbors(PairStage<T, CAP>& S, int64_t off, int n, DevModel const& model,
                                               BatchView const& b)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ne = model.numElements;
    constexpr int NC = (CAP + kPairThreads - 1) / kPairThreads;
    constexpr bool kEarly = NC <= 2;   // entries loaded before the barriers, hidden behind them
    double d[kEarly ? NC : 1], x[kEarly ? NC : 1], y[kEarly ? NC : 1], z[kEarly ? NC : 1];
    if constexpr (kEarly)
    {
#pragma unroll
        for (int c = 0; c < NC; ++c)
        {
            const int m = c * kPairThreads + tid;
            if (m < n)
            {
                d[c] = b.nbrD[off + m];
                x[c] = b.nbrDx[off + m];
                y[c] = b.nbrDy[off + m];
                z[c] = b.nbrDz[off + m];
            }
        }
    }
    if (tid < 64) S.expTab[tid] = model.expTable[tid];
    const int chunks = (n + 31) >> 5;
    for (int c = warp; c < chunks; c += kPairWarps)
    {
        const int m = c * 32 + lane;
        const int el = m < n ? (int)b.nbrElem[off + m] : -1;
        for (int e = 0; e < ne; ++e)
        {
            const unsigned bal = __ballot_sync(kFullMask, el == e);
            if (lane == 0) S.chunk[e][c] = __popc(bal);
        }
    }
    __syncthreads();
    if (tid == 0)
    {
        int at = 0;
        for (int e = 0; e < ne; ++e)
        {
            S.begin[e] = at;
            for (int c = 0; c < chunks; ++c)
            {
                const int t = S.chunk[e][c];
                S.chunk[e][c] = at;
                at += t;
            }
            if (!model.sortByDistance)
                for (int k = 0; k < 4; ++k) S.nBelow[k][e] = at - S.begin[e];
        }
        S.begin[ne] = at;
    }
    if (model.sortByDistance && tid >= 32 && tid < 64)
        for (int k = lane; k < 4 * kDevMaxElements; k += 32) S.nBelow[k / kDevMaxElements][k % kDevMaxElements] = 0;
    __syncthreads();
    if (model.sortByDistance)
    {
        double* rd = S.geo.scratch();
        for (int c = warp; c < chunks; c += kPairWarps)
        {
            const int m = c * 32 + lane;
            const int el = m < n ? (int)b.nbrElem[off + m] : -1;
            for (int e = 0; e < ne; ++e)
            {
                const unsigned bal = __ballot_sync(kFullMask, el == e);
                if (el == e)
                {
                    const int s = S.chunk[e][c] + __popc(bal & ((1u << lane) - 1u));
                    rd[s] = b.nbrD[off + m];
                    S.slotOf[m] = (short)s;
                }
            }
        }
        __syncthreads();
        for (int m = tid; m < n; m += kPairThreads)
        {
            const int el = (int)b.nbrElem[off + m], s = S.slotOf[m];
            const int b0 = S.begin[el], b1 = S.begin[el + 1];
            const double rs = rd[s];
            int rank = b0;
            for (int t = b0; t < b1; ++t)
            {
                const double rt = rd[t];
                rank += (rt < rs || (rt == rs && t < s)) ? 1 : 0;
            }
            for (int c = 0; c < model.numCutoffSlots; ++c)
                if (rs < model.cutoff[c].rc) atomicAdd(&S.nBelow[c][el], 1);
            S.slotOf[m] = (short)rank;   // this thread's own entry
        }
        __syncthreads();   // the scratch becomes the geometry
    }
#pragma unroll
    for (int c = 0; c < NC; ++c)
    {
        const int ch = c * kPairWarps + warp;
        if (ch >= chunks) break;
        const int m = ch * 32 + lane;
        const int el = m < n ? (int)b.nbrElem[off + m] : -1;
        int s = 0;
        if (model.sortByDistance) s = m < n ? S.slotOf[m] : 0;
        else
        {
            for (int e = 0; e < ne; ++e)
            {
                const unsigned bal = __ballot_sync(kFullMask, el == e);
                if (el == e) s = S.chunk[e][ch] + __popc(bal & ((1u << lane) - 1u));
            }
            if (m < n) S.slotOf[m] = (short)s;
        }
        if (m < n)
        {
            S.perm[s] = (short)m;
            if constexpr (kEarly) S.geo.set(s, x[c], y[c], z[c], d[c]);
            else S.geo.set(s, b.nbrDx[off + m], b.nbrDy[off + m], b.nbrDz[off + m], b.nbrD[off + m]);
        }
    }
}

// The staged positions of a candidate pair in FP32: inside the cutoff?
__device__ __forceinline__ bool nearPair(float4 a, float4 c, float rc2)
{
    const float dx = c.x - a.x, dy = c.y - a.y, dz = c.z - a.z;
    return fmaf(dx, dx, fmaf(dy, dy, dz * dz)) < rc2;
}

// Shared-memory accesses of the candidate loop at 32-bit addresses: the store
// happens where `on`, without a branch.
__device__ __forceinline__ void storeIf(unsigned addr, int v, bool on)
{
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q st.shared.u32 [%0], %1;\n\t}"
                 :
                 : "r"(addr), "r"(v), "r"((unsigned)on)
                 : "memory");
}

__device__ __forceinline__ float4 recordAt(unsigned addr)
{
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

__device__ __forceinline__ int wrapMin(int v, int w) { return (int)min((unsigned)v, (unsigned)w); }

// The shares of the element's angular groups, one thread each (after the
// barrier that completes the stage's begin and nBelow).
template <typename T, int CAP>
__device__ __forceinline__ void setGroupShares(PairStage<T, CAP>& S, DevPairTable const& gt, int first, int g1)
{
    for (int g = first + (int)threadIdx.x; g < g1; g += kPairThreads)
    {
        DevPairGroup const& G = gt.g[g];
        const bool same = G.e1 == G.e2;
        Phase ph[2];
        GroupShare h{};
        if (roundPhases(S.begin[G.e1], S.nBelow[G.cutoffSlot][G.e1], S.begin[G.e2], S.nBelow[G.cutoffSlot][G.e2], same, ph))
        {
            h.count = ph[0].count;
            h.minor = ph[0].minor;
            h.nO = ph[0].nO;
            h.m1 = same ? h.nO - 1 + (h.nO & 1) : ph[0].D;
            h.O0 = ph[0].O0;
            h.P0 = ph[0].P0;
            h.share = ((h.count + kPairWarps * 64 - 1) / (kPairWarps * 64)) * 64;
            h.inv = 1.0f / (float)h.minor;
        }
        S.share[g - first] = h;
    }
}

// The warp's share of a group's candidate pairs, in the rounds of
// pair_rounds.cuh; step(entry, ok) runs on 32 of them at a time.  Entry:
// round << 20 | slot j << 10 | slot k (slots < 1024); lanes with ok = false
// hold some pair of the group (or a slot twice).  Narrow groups: the
// candidates are tested and compacted into the warp's ring, two batches of 32
// per turn; no divergent branch: a lane past the share walks on over indices
// within kTestPad of the blocks and its pair is discarded.
template <bool NARROW, typename T, int CAP, typename Step>
__device__ __forceinline__ void groupPairs(PairStage<T, CAP>& S, GroupShare const& H, DevPairGroup const& G, int warp, int lane,
                                           Step step)
{
    const bool same = G.e1 == G.e2;
    const int count = H.count, minor = H.minor, nO = H.nO, m1 = H.m1;
    const int p1 = min((warp + 1) * H.share, count);
    int p = warp * H.share;
    if (p >= p1) return;
    const int first = (H.O0 << 10) + H.P0;
    // (x + 1/2) / minor truncates to the quotient: x < 2^20 and the FP32 error is below 1 / (2 minor)
    const int q32 = (int)(32.5f * H.inv), r32 = 32 - q32 * minor;
    int a = (int)(((float)(p + lane) + 0.5f) * H.inv), t = p + lane - a * minor;
    int left = p1 - p - lane;   // candidates of this lane while positive
    auto candidate = [&](int& entry, int& u, int& v) {
        bool in = left > 0;
        if (same)
        {
            u = a + t;
            u = wrapMin(u, u - m1);
            v = a - t;
            v = wrapMin(v, v + m1);
            if (t == 0) u = m1;
            in &= u < nO;
        }
        else
        {
            u = t;
            v = t + a;
            v = wrapMin(v, v - m1);
        }
        entry = (a << 20) + (u << 10) + v + first;
        t += r32;
        a += q32 + (t >= minor ? 1 : 0);
        t = wrapMin(t, t - minor);
        left -= 32;
        return in;
    };
    if constexpr (NARROW)
    {
        const unsigned below = (1u << lane) - 1u;
        const float rc2 = G.rc2Test;
        const unsigned at1 = (unsigned)__cvta_generic_to_shared(S.geo.records() + H.O0);
        const unsigned at2 = (unsigned)__cvta_generic_to_shared(S.geo.records() + H.P0);
        int* queue = S.queue[warp];
        const unsigned ring = (unsigned)__cvta_generic_to_shared(queue);
        int qh = 0, qn = 0;
        while (true)
        {
            while (qn < 32 && p < p1)
            {
                int e0, e1, u0, v0, u1, v1;
                bool in0 = candidate(e0, u0, v0);
                bool in1 = candidate(e1, u1, v1);
                in0 &= nearPair(recordAt(at1 + 16 * u0), recordAt(at2 + 16 * v0), rc2);
                in1 &= nearPair(recordAt(at1 + 16 * u1), recordAt(at2 + 16 * v1), rc2);
                const unsigned b0 = __ballot_sync(kFullMask, in0), b1 = __ballot_sync(kFullMask, in1);
                const int at = qh + qn, n0 = __popc(b0);
                storeIf(ring + 4 * ((at + __popc(b0 & below)) & (kRing - 1)), e0, in0);
                storeIf(ring + 4 * ((at + n0 + __popc(b1 & below)) & (kRing - 1)), e1, in1);
                qn += n0 + __popc(b1);
                p += 64;
            }
            if (qn <= 0) break;
            __syncwarp();
            step(queue[(qh + (lane < qn ? lane : 0)) & (kRing - 1)], lane < qn);
            qh = (qh + 32) & (kRing - 1);
            qn -= 32;
        }
        __syncwarp();
    }
    else
        for (; p < p1; p += 32)
        {
            int e, u, v;
            const bool in = candidate(e, u, v);
            step(in ? e : first, in);
        }
}

// Sums of eight per-lane values over the warp, in a fixed order: lane 4 c
// returns the sum of v[c].  `scratch`: 8 x kSumPitch doubles of the warp.
template <typename T>
__device__ __forceinline__ double warpSums(T const (&v)[8], double* scratch, int lane)
{
#pragma unroll
    for (int c = 0; c < 8; ++c) scratch[c * kSumPitch + lane] = (double)v[c];
    __syncwarp();
    const double* p = scratch + (lane >> 2) * kSumPitch + (lane & 3);
    double s = p[0];
#pragma unroll
    for (int k = 1; k < 8; ++k) s += p[4 * k];
    s += __shfl_xor_sync(kFullMask, s, 1);
    s += __shfl_xor_sync(kFullMask, s, 2);
    __syncwarp();
    return s;
}

// Atoms of the upper tiers, 128 tested at a time by the block: calls
// f(i) for every atom of the tier, the whole block together.
template <typename F>
__device__ __forceinline__ void forTierAtoms(unsigned* todo, BatchView const& b, int lower, int cap, bool flagOverflow, F f)
{
    const int tid = threadIdx.x;
    for (int base = blockIdx.x * kPairThreads; base < b.N; base += gridDim.x * kPairThreads)
    {
        const int i = base + tid;
        bool mine = false;
        if (i < b.N)
        {
            const int64_t off = b.nbrOffset[i], end = b.nbrOffset[i + 1];
            const int n = (int)(end - off);
            mine = end <= b.nbrCapacity && ((n <= cap && n > lower) || (flagOverflow && n > cap));
        }
        const unsigned bal = __ballot_sync(kFullMask, mine);
        if ((tid & 31) == 0) todo[tid >> 5] = bal;
        __syncthreads();
        for (int w = 0; w < kPairWarps; ++w)
        {
            unsigned m = todo[w];
            while (m)
            {
                f(base + w * 32 + __ffs(m) - 1);
                m &= m - 1;
            }
        }
        __syncthreads();
    }
}

// f(narrow, form) for a group of a model of form FORM: models with zeta up
// to 16 run the groups with zeta up to 4 in the shorter form, models with any
// integers those with zeta 1 to 4 in a form of their own (zeta {1, 3}, 33 k
// atoms: in the any-integer form G takes 2.48 and the forces 2.95 ms, in this
// one 1.61 and 2.53).
template <int FORM, typename F>
__device__ __forceinline__ void withForm(DevPairGroup const& G, F f)
{
    using True = std::integral_constant<bool, true>;
    using False = std::integral_constant<bool, false>;
    if (FORM == 0 && G.cubic)
    {
        if (G.type == 3) f(True{}, std::integral_constant<int, 4>{});
        else f(False{}, std::integral_constant<int, 4>{});
    }
    else if (FORM == 5 && !(G.levels >> 3))
    {
        if (G.type == 3) f(True{}, std::integral_constant<int, 3>{});
        else f(False{}, std::integral_constant<int, 3>{});
    }
    else if (G.type == 3) f(True{}, std::integral_constant<int, FORM>{});
    else f(False{}, std::integral_constant<int, FORM>{});
}

// ---------------------------------------------------------------------------
// G values
// ---------------------------------------------------------------------------

// w: per slot f_c times the Gaussians of the group's two etas.
template <typename T, int CAP>
struct alignas(16) ValuesStage
{
    PairStage<T, CAP> st;
    typename Pair2<T>::V w[CAP];
    T fc[CAP];
    double sums[kPairWarps][8 * kSumPitch];
    // followed by partial[kPairWarps][maxSF] doubles
};

template <typename T>
__device__ __forceinline__ typename Pair2<T>::V pairAt(typename Pair2<T>::V const* a, int o16)
{
    if constexpr (sizeof(T) == 8) return *reinterpret_cast<const double2*>(reinterpret_cast<const char*>(a) + o16);
    else return *reinterpret_cast<const float2*>(reinterpret_cast<const char*>(a) + (o16 >> 1));
}

// One step of a warp: 32 accepted pairs (lanes past `take` repeat the first
// one with weight 0).  acc[(eta * 2 + lambda) * Z + slot] += G terms.
// FORM 3, 5: zeta 2^slot (slots up to 4, 16), absent ones summed as well;
// 4: zeta 1 to 4; 0: any zeta, five slots.  TWO: the group has two etas.
template <typename T, int CAP, int CUT, bool NARROW, int FORM, bool TWO>
__device__ __forceinline__ void valuesStep(ValuesStage<T, CAP> const& S, DevPairGroup const& G, GroupRegs<T> const& R,
                                           DevCutoff const& cut, int e, bool ok, T* acc)
{
    constexpr int Z = FORM ? FORM : kPairLevels;
    const int oj = (e >> 6) & 0x3ff0, okk = (e << 4) & 0x3ff0;   // byte offsets of the slots' records
    T x1, y1, z1, i1, x2, y2, z2, i2;
    S.st.geo.get(oj, x1, y1, z1, i1);
    S.st.geo.get(okk, x2, y2, z2, i2);
    const auto wj = pairAt<T>(S.w, oj), wk = pairAt<T>(S.w, okk);
    const T cost = (x1 * x2 + y1 * y2 + z1 * z2) * (i1 * i2);
    T c0, c1 = T(0);
    if constexpr (TWO)
    {
        c0 = wj.x * wk.x;
        c1 = wj.y * wk.y;
    }
    else c0 = G.comp ? wj.y * wk.y : wj.x * wk.x;
    if constexpr (NARROW)
    {
        const T dx = x2 - x1, dy = y2 - y1, dz = z2 - z1;
        const T s = dx * dx + dy * dy + dz * dz;
        const T r = s * invSqrt(s);
        T f, df;
        pairCutoff<CUT>(cut, R.iw, r, f, df);
        if (!ok) f = T(0);
        c0 *= f * expScaled<FORM == 0>(s, R.scale0, S.st.expTab);
        if constexpr (TWO) c1 *= f * expScaled<FORM == 0>(s, R.scale1, S.st.expTab);
    }
    else if (!ok) c0 = c1 = T(0);
#pragma unroll
    for (int l = 0; l < 2; ++l)
    {
        T p = T(1) + (l ? R.lam1 : R.lam0) * cost;
        if constexpr (FORM == 0) p = clampZero(p);
        const T p1 = p;
#pragma unroll
        for (int z = 0; z < Z; ++z)
        {
            if (FORM && z > 0 && !(FORM == 4 && z == 2)) p = p * p;
            if (FORM == 0 && !(G.levels >> z & 1)) continue;
            const T q = FORM == 4 && z == 2 ? p1 * p : FORM ? p : powAny(p, G.zeta[z]);
            acc[l * Z + z] += c0 * q;
            if constexpr (TWO) acc[(2 + l) * Z + z] += c1 * q;
        }
    }
}

template <typename T, int CAP, int CUT, bool NARROW, int FORM, bool TWO>
__device__ __forceinline__ void valuesGroup(ValuesStage<T, CAP>& S, double* partial, DevModel const& model,
                                            DevPairGroup const& G, GroupShare const& H, int warp, int lane)
{
    constexpr int Z = FORM ? FORM : kPairLevels, ACC = (TWO ? 4 : 2) * Z;
    T acc[ACC];
#pragma unroll
    for (int q = 0; q < ACC; ++q) acc[q] = T(0);
    DevCutoff const& cut = model.cutoff[G.cutoffSlot];
    const GroupRegs<T> R(G, cut);
    groupPairs<NARROW>(S.st, H, G, warp, lane, [&](int e, bool ok) {
        valuesStep<T, CAP, CUT, NARROW, FORM, TWO>(S, G, R, cut, e, ok, acc);
    });
    // the grid's present members, eight sums at a time
    const DevMember* mem = model.members + G.memberBegin;
#pragma unroll
    for (int q0 = 0; q0 < ACC; q0 += 8)
    {
        T v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = q0 + q < ACC ? acc[q0 + q < ACC ? q0 + q : 0] : T(0);
        const double sum = warpSums(v, S.sums[warp], lane);
        const int q = q0 + (lane >> 2);
        if ((lane & 3) == 0 && q < ACC)
        {
            const int c = G.combo[q / Z * kPairLevels + q % Z];
            if (c >= 0) partial[mem[c].sf] = sum * mem[c].gNorm;
        }
    }
}

// Radial members of the slots of one element (r_s allowed).
template <typename T, int CAP>
__device__ __forceinline__ void valuesRadial(ValuesStage<T, CAP>& S, double* partial, DevModel const& model,
                                             DevPairTable const& gt, DevPairGroup const& G, const double* fcOwn, int warp,
                                             int lane)
{
    const DevMember* mem = model.members + G.memberBegin;
    const DevRadial* rad = gt.radial + G.radialBegin;
    const int b0 = S.st.begin[G.e1], b1 = S.st.begin[G.e1 + 1];
    const T rc = (T)G.rc;
    for (int m0 = 0; m0 < G.memberCount; m0 += 8)
    {
        T v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = T(0);
        for (int s = (b0 & ~31) + warp * 32 + lane; s - lane < b1; s += kPairThreads)
        {
            if (s < b0 || s >= b1) continue;
            const T r = S.st.geo.r[s];
            if (!(r < rc)) continue;
            const T fc = fcOwn ? (T)fcOwn[S.st.perm[s]] : S.fc[s];
#pragma unroll
            for (int q = 0; q < 8; ++q)
            {
                if (m0 + q < G.memberCount)
                {
                    DevRadial const& M = rad[m0 + q];
                    const T d = r - radialShift<T>(M);
                    v[q] += expScaled<true>(d * d, radialScale<T>(M), S.st.expTab) * fc;
                }
            }
        }
        double sum = 0.0;
        if ((b0 & ~31) + warp * 32 < b1) sum = warpSums(v, S.sums[warp], lane);
        const int q = m0 + (lane >> 2);
        if ((lane & 3) == 0 && q < G.memberCount) partial[mem[q].sf] = sum;
    }
}

template <typename T, int CAP, int CUT, int FORM>
__device__ __forceinline__ void atomValues(ValuesStage<T, CAP>& S, double* partialAll, DevModel const& model,
                                           BatchView const& b, DevPairTable const& gt, int i, int64_t off, int n)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ec = b.elem[i];
    DevElement const& E = model.el[ec];
    const int g0 = gt.begin[ec], g1 = gt.begin[ec + 1];
    if (g0 == g1) return;   // compact functions only
    // what the slots hold beside the geometry: the cutoff slot and etas of the group at hand
    int slot = -1;
    T eta0 = T(0), eta1 = T(0);
    bool factors = false;
    stageNeighbors<T, CAP>(S.st, off, n, model, b);
    auto stageFactors = [&](DevPairGroup const& G) {
        slot = G.cutoffSlot;
        factors = G.type != 2;
        eta0 = groupStageScale<T>(G, 0);
        eta1 = groupStageScale<T>(G, 1);
        const double* fc = b.nbrFc + (size_t)slot * b.nbrCapacity + off;
        for (int m = tid; m < n; m += kPairThreads)
        {
            const int s = S.st.slotOf[m];
            const T f = (T)fc[m];
            S.fc[s] = f;
            if (factors)
            {
                const T r = S.st.geo.r[s], r2 = r * r;
                typename Pair2<T>::V w;
                w.x = f * expScaled<FORM == 0>(r2, eta0, S.st.expTab);
                w.y = f * expScaled<FORM == 0>(r2, eta1, S.st.expTab);
                S.w[s] = w;
            }
        }
    };
    int first = g0;   // the first angular group's factors come with the stage
    while (first < g1 && gt.g[first].type == 2) ++first;
    setGroupShares(S.st, gt, first, g1);
    if (first < g1) stageFactors(gt.g[first]);
    else if (g0 < g1) stageFactors(gt.g[g0]);
    double* partial = partialAll + (size_t)warp * model.maxSF;
    __syncthreads();
    for (int g = g0; g < g1; ++g)
    {
        DevPairGroup const& G = gt.g[g];
        if (G.type == 2)
        {
            valuesRadial<T, CAP>(S, partial, model, gt, G,
                                 G.cutoffSlot == slot ? nullptr : b.nbrFc + (size_t)G.cutoffSlot * b.nbrCapacity + off,
                                 warp, lane);
            continue;
        }
        if (G.cutoffSlot != slot || !factors || groupStageScale<T>(G, 0) != eta0 || groupStageScale<T>(G, 1) != eta1)
        {
            __syncthreads();
            stageFactors(G);
            __syncthreads();
        }
        auto pairs = [&](auto narrow, auto form) {
            if (G.numEta == 2) valuesGroup<T, CAP, CUT, decltype(narrow)::value, decltype(form)::value, true>(S, partial, model, G, S.st.share[g - first], warp, lane);
            else valuesGroup<T, CAP, CUT, decltype(narrow)::value, decltype(form)::value, false>(S, partial, model, G, S.st.share[g - first], warp, lane);
        };
        withForm<FORM>(G, pairs);
    }
    __syncthreads();
    for (int k = gt.memberBegin[ec] + tid; k < gt.memberBegin[ec + 1]; k += kPairThreads)
    {
        const int q = model.members[k].sf;
        double sum = partialAll[q];
        for (int w = 1; w < kPairWarps; ++w) sum += partialAll[(size_t)w * model.maxSF + q];
        b.G[(size_t)i * b.gStride + q] = scaleG(model.scaling[E.sfBegin + q], sum);
    }
}

// TIER false: one block per atom (atoms with up to CAP neighbours); true:
// the atoms with lower < n <= CAP.
template <typename T, int CAP, int CUT, int FORM, bool TIER>
__global__ void __launch_bounds__(kPairThreads, TIER ? 1 : (sizeof(T) == 8 ? 6 : 8))
    kPairValues(const __grid_constant__ DevModel model, const __grid_constant__ BatchView b, int lower, int flagOverflow,
                const __grid_constant__ DevPairTable gt)
{
    extern __shared__ __align__(16) unsigned char smemRaw[];
    ValuesStage<T, CAP>& S = *reinterpret_cast<ValuesStage<T, CAP>*>(smemRaw);
    double* partial = reinterpret_cast<double*>(smemRaw + sizeof(ValuesStage<T, CAP>));
    if constexpr (!TIER)
    {
        const int i = blockIdx.x;
        const int64_t off = b.nbrOffset[i], end = b.nbrOffset[i + 1];
        const int n = (int)(end - off);
        if (end > b.nbrCapacity || n > CAP) return;
        atomValues<T, CAP, CUT, FORM>(S, partial, model, b, gt, i, off, n);
    }
    else
        forTierAtoms(S.st.todo, b, lower, CAP, flagOverflow != 0, [&](int i) {
            const int64_t off = b.nbrOffset[i];
            const int n = (int)(b.nbrOffset[i + 1] - off);
            if (n > CAP)
            {
                if (threadIdx.x == 0) atomicAdd(&b.status->badInput, 1);
                return;
            }
            atomValues<T, CAP, CUT, FORM>(S, partial, model, b, gt, i, off, n);
            __syncthreads();
        });
}

// ---------------------------------------------------------------------------
// Force pass
// ---------------------------------------------------------------------------
// With w_s = dE/dG_s * factorNorm_s, V = exp(-eta (rij^2 + rik^2 + rjk^2)),
// p = 1 + lambda cos and, per eta, Q = sum w p^zeta, R = dQ/dcos = sum w zeta lambda p^(zeta-1):
//   T1 = sum_eta V R,  T2 = sum_eta 2 eta V Q,  T3 = sum_eta V Q
// the derivative prefactors p1, p2, p3 (SymGrpExpAngn.cpp:305-337) contract to
//   P1 = pfc ((1/(rij rik) - cos/rij^2) T1 - T2) + fc(rik) fc(rjk) fc'(rij)/rij T3
//   P2 = the same with j and k exchanged
//   P3 = pfc (T1/(rij rik) + T2) - fc(rij) fc(rik) fc'(rjk)/rjk T3     (narrow)
//   P3 = pfc T1/(rij rik)                                              (wide)
// The force E_i puts on j gains P1 dr_ij + P3 dr_jk, on k P2 dr_ik - P3 dr_jk;
// the centre's own is minus the sum over its neighbours.

template <typename T, int CAP>
struct FactorStage;
template <int CAP>
struct FactorStage<double, CAP>
{
    double2 cut[CAP], gauss[CAP];   // (f_c, (df_c/dr)/r), Gaussians of the two etas
    __device__ __forceinline__ void set(int s, double fc, double dr, double e0, double e1)
    {
        cut[s] = make_double2(fc, dr);
        gauss[s] = make_double2(e0, e1);
    }
    __device__ __forceinline__ void get(int o, double& fc, double& dr, double& e0, double& e1) const
    {
        const double2 a = *reinterpret_cast<const double2*>(reinterpret_cast<const char*>(cut) + o);
        const double2 c = *reinterpret_cast<const double2*>(reinterpret_cast<const char*>(gauss) + o);
        fc = a.x;
        dr = a.y;
        e0 = c.x;
        e1 = c.y;
    }
};
template <int CAP>
struct FactorStage<float, CAP>
{
    float4 v[CAP];
    __device__ __forceinline__ void set(int s, float fc, float dr, float e0, float e1) { v[s] = make_float4(fc, dr, e0, e1); }
    __device__ __forceinline__ void get(int o, float& fc, float& dr, float& e0, float& e1) const
    {
        const float4 a = *reinterpret_cast<const float4*>(reinterpret_cast<const char*>(v) + o);
        fc = a.x;
        dr = a.y;
        e0 = a.z;
        e1 = a.w;
    }
};

// Coefficients of one angular group for the atom: per lambda and zeta slot
// (w of the two etas) and (w zeta lambda of the two etas).
template <typename T>
struct alignas(16) GroupCoef
{
    typename Pair2<T>::V w[2][kPairLevels], d[2][kPairLevels];
};

// Copies of a warp's force arrays: with two, two rounds of matchings are added
// at once.  FP32 2.48 -> 2.39 ms of a force pass; in FP64 the second copy costs
// the fifth block per SM (3.82 -> 4.02 ms).
template <typename T, int CAP>
constexpr int forceCopies()
{
    return sizeof(T) == 4 && CAP <= 384 ? 2 : 1;
}

template <typename T, int CAP>
struct alignas(16) ForcesStage
{
    static constexpr int kCopies = forceCopies<T, CAP>();
    PairStage<T, CAP> st;
    FactorStage<T, CAP> fac;
    typename Pair2<T>::V hxy[kPairWarps][kCopies][CAP];
    T hz[kPairWarps][kCopies][CAP];
    double self[kPairWarps][3];
    // followed by GroupCoef<T>[maxAngular], then cw[maxSF] doubles
};

template <typename T, int CAP, int CUT, bool NARROW, int FORM, bool TWO>
__device__ __forceinline__ void forcesStep(ForcesStage<T, CAP>& S, GroupCoef<T> const& C, DevPairGroup const& G,
                                           GroupRegs<T> const& R, T eta20, T eta21, DevCutoff const& cut, int e, bool ok,
                                           int warp, int lane)
{
    constexpr int Z = FORM ? FORM : kPairLevels;
    constexpr int COPIES = ForcesStage<T, CAP>::kCopies;
    using V = typename Pair2<T>::V;
    const int sj = (e >> 10) & 1023, sk = e & 1023;
    T x1, y1, z1, i1, x2, y2, z2, i2, f1, d1, f2, d2, v0, v1 = T(0);
    S.st.geo.get(sj << 4, x1, y1, z1, i1);
    S.st.geo.get(sk << 4, x2, y2, z2, i2);
    {
        T a0, a1, b0, b1;
        S.fac.get(sj << 4, f1, d1, a0, a1);
        S.fac.get(sk << 4, f2, d2, b0, b1);
        if constexpr (TWO)
        {
            v0 = a0 * b0;
            v1 = a1 * b1;
        }
        else v0 = G.comp ? a1 * b1 : a0 * b0;
    }
    const T ri = i1 * i2;
    const T cost = (x1 * x2 + y1 * y2 + z1 * z2) * ri;
    const T dx = x2 - x1, dy = y2 - y1, dz = z2 - z1;
    T f3 = T(1), d3 = T(0);
    if constexpr (NARROW)
    {
        const T s = dx * dx + dy * dy + dz * dz;
        const T i3 = invSqrt(s);
        pairCutoff<CUT>(cut, R.iw, s * i3, f3, d3);
        d3 *= i3;
        v0 *= expScaled<FORM == 0>(s, R.scale0, S.st.expTab);
        if constexpr (TWO) v1 *= expScaled<FORM == 0>(s, R.scale1, S.st.expTab);
    }
    T Q0 = T(0), R0 = T(0), Q1 = T(0), R1 = T(0);
#pragma unroll
    for (int l = 0; l < 2; ++l)
    {
        T p = T(1) + (l ? R.lam1 : R.lam0) * cost;
        if constexpr (FORM == 0) p = clampZero(p);
        T a = T(1), sq = p, u0 = T(0), u1 = T(0);
#pragma unroll
        for (int z = 0; z < Z; ++z)
        {
            if (FORM == 0 && !(G.levels >> z & 1)) continue;
            // a = p^(zeta - 1): 1, p, p^3, p^7, p^15 for the powers of two, 1, p, p^2, p^3 for 1 to 4
            if (FORM == 4 && z > 0) a = z == 1 ? p : a * p;
            else if (FORM && z > 0)
            {
                a = z == 1 ? p : a * sq;
                sq = sq * sq;
            }
            const T q = FORM ? a : p > T(0) ? powAny(p, G.zeta[z] - 1) : T(0);   // terms with p <= 0 vanish
            const V w = C.w[l][z], d = C.d[l][z];
            if (FORM && z == 0)
            {
                u0 = w.x;
                R0 += d.x;
                u1 = w.y;
                R1 += d.y;
            }
            else
            {
                u0 += w.x * q;
                R0 += d.x * q;
                if constexpr (TWO)
                {
                    u1 += w.y * q;
                    R1 += d.y * q;
                }
            }
        }
        Q0 += p * u0;
        if constexpr (TWO) Q1 += p * u1;
    }
    T T1 = v0 * R0, T3 = v0 * Q0, T2 = eta20 * T3;
    if constexpr (TWO)
    {
        T1 += v1 * R1;
        const T t = v1 * Q1;
        T3 += t;
        T2 += eta21 * t;
    }
    const T ff = f1 * f2, pfc = ff * f3, f3T = f3 * T3;
    const T P1 = pfc * ((ri - cost * (i1 * i1)) * T1 - T2) + d1 * (f2 * f3T);
    const T P2 = pfc * ((ri - cost * (i2 * i2)) * T1 - T2) + d2 * (f1 * f3T);
    const T P3 = NARROW ? pfc * (ri * T1 + T2) - ff * (d3 * T3) : pfc * (ri * T1);
    const T ox = P1 * x1 + P3 * dx, oy = P1 * y1 + P3 * dy, oz = P1 * z1 + P3 * dz;
    const T qx = P2 * x2 - P3 * dx, qy = P2 * y2 - P3 * dy, qz = P2 * z2 - P3 * dz;
    // inside a round no slot occurs twice: COPIES rounds at a time, each into its own copy
    const int rnd = ok ? (int)((unsigned)e >> 20) : -1;
    const int prev = __shfl_up_sync(kFullMask, rnd, 1);
    const unsigned heads = __ballot_sync(kFullMask, ok && (lane == 0 || prev != rnd));
    const int mine = __popc(heads & ((2u << lane) - 1u)) - 1;
    const int passes = (__popc(heads) + COPIES - 1) / COPIES;
    V* hxy = S.hxy[warp][mine & (COPIES - 1)];
    T* hz = S.hz[warp][mine & (COPIES - 1)];
    for (int r = 0; r < passes; ++r)
    {
        if (ok && mine / COPIES == r)
        {
            V a = hxy[sj], c = hxy[sk];
            T az = hz[sj], cz = hz[sk];
            a.x += ox;
            a.y += oy;
            az += oz;
            c.x += qx;
            c.y += qy;
            cz += qz;
            hxy[sj] = a;
            hz[sj] = az;
            hxy[sk] = c;
            hz[sk] = cz;
        }
        __syncwarp();
    }
}

template <typename T, int CAP, int CUT, bool NARROW, int FORM, bool TWO>
__device__ __forceinline__ void forcesGroup(ForcesStage<T, CAP>& S, GroupCoef<T> const& C, DevModel const& model,
                                            DevPairGroup const& G, GroupShare const& H, int warp, int lane)
{
    DevCutoff const& cut = model.cutoff[G.cutoffSlot];
    const GroupRegs<T> R(G, cut);
    const T eta20 = groupEta2<T>(G, 0), eta21 = groupEta2<T>(G, 1);
    groupPairs<NARROW>(S.st, H, G, warp, lane, [&](int e, bool ok) {
        forcesStep<T, CAP, CUT, NARROW, FORM, TWO>(S, C, G, R, eta20, eta21, cut, e, ok, warp, lane);
    });
}

template <typename T, int CAP, int CUT, int FORM>
__device__ __forceinline__ void atomForces(ForcesStage<T, CAP>& S, GroupCoef<T>* coef, double* cw, DevModel const& model,
                                           BatchView const& b, DevPairTable const& gt, int i, int64_t off, int n)
{
    constexpr int COPIES = ForcesStage<T, CAP>::kCopies;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ec = b.elem[i];
    const int g0 = gt.begin[ec], g1 = gt.begin[ec + 1];
    if (g0 == g1)   // compact functions only: their kernels add to these
    {
        for (int m = tid; m < n; m += kPairThreads) b.hx[off + m] = b.hy[off + m] = b.hz[off + m] = 0.0;
        if (tid < 3) b.fSelf[3 * (size_t)i + tid] = 0.0;
        return;
    }
    // dE/dG times the functions' normalisation, in member order
    const int m0 = gt.memberBegin[ec], mc = gt.memberBegin[ec + 1] - m0;
    const double* dEdG = b.dEdG + (size_t)i * b.gStride;
    for (int q = tid; q < mc; q += kPairThreads)
    {
        DevMember const& M = model.members[m0 + q];
        cw[q] = dEdG[M.sf] * M.factorNorm;
    }
    for (int s = lane; s < n; s += 32)
#pragma unroll
        for (int c = 0; c < COPIES; ++c)
        {
            typename Pair2<T>::V z;
            z.x = T(0);
            z.y = T(0);
            S.hxy[warp][c][s] = z;
            S.hz[warp][c][s] = T(0);
        }
    stageNeighbors<T, CAP>(S.st, off, n, model, b);
    int first = g0;
    while (first < g1 && gt.g[first].type == 2) ++first;
    setGroupShares(S.st, gt, first, g1);
    // cw is complete (barriers in stageNeighbors)
    for (int t = tid; t < (g1 - first) * 4 * kPairLevels; t += kPairThreads)
    {
        const int g = t / (4 * kPairLevels), c = t - g * 4 * kPairLevels;
        DevPairGroup const& G = gt.g[first + g];
        const int q = G.combo[c], z = c % kPairLevels, l = c / kPairLevels & 1, k = c / (2 * kPairLevels);
        const double w = q >= 0 ? cw[G.memberBegin - m0 + q] : 0.0;
        const double d = w * (double)G.zeta[z] * G.lambda[l];
        T* pw = &coef[g].w[l][z].x;
        T* pd = &coef[g].d[l][z].x;
        pw[k] = (T)w;
        pd[k] = (T)d;
    }
    int slot = -1;
    T eta0 = T(0), eta1 = T(0);
    auto stageFactors = [&](DevPairGroup const& G) {
        slot = G.cutoffSlot;
        eta0 = groupStageScale<T>(G, 0);
        eta1 = groupStageScale<T>(G, 1);
        const double* fc = b.nbrFc + (size_t)slot * b.nbrCapacity + off;
        const double* dfc = b.nbrDfc + (size_t)slot * b.nbrCapacity + off;
        for (int m = tid; m < n; m += kPairThreads)
        {
            const int s = S.st.slotOf[m];
            const T r = S.st.geo.r[s], r2 = r * r;
            S.fac.set(s, (T)fc[m], (T)(dfc[m] / b.nbrD[off + m]), expScaled<FORM == 0>(r2, eta0, S.st.expTab),
                      expScaled<FORM == 0>(r2, eta1, S.st.expTab));
        }
    };
    if (first < g1) stageFactors(gt.g[first]);
    __syncthreads();
    for (int g = first; g < g1; ++g)
    {
        DevPairGroup const& G = gt.g[g];
        if (G.cutoffSlot != slot || groupStageScale<T>(G, 0) != eta0 || groupStageScale<T>(G, 1) != eta1)
        {
            __syncthreads();
            stageFactors(G);
            __syncthreads();
        }
        GroupCoef<T> const& C = coef[g - first];
        auto pairs = [&](auto narrow, auto form) {
            if (G.numEta == 2) forcesGroup<T, CAP, CUT, decltype(narrow)::value, decltype(form)::value, true>(S, C, model, G, S.st.share[g - first], warp, lane);
            else forcesGroup<T, CAP, CUT, decltype(narrow)::value, decltype(form)::value, false>(S, C, model, G, S.st.share[g - first], warp, lane);
        };
        withForm<FORM>(G, pairs);
    }
    __syncthreads();
    // per slot: the warps' sums in order, then the radial members
    double fx = 0.0, fy = 0.0, fz = 0.0;
    for (int s = tid; s < n; s += kPairThreads)
    {
        T hx = T(0), hy = T(0), hz = T(0);
#pragma unroll
        for (int w = 0; w < kPairWarps; ++w)
#pragma unroll
            for (int c = 0; c < COPIES; ++c)
            {
                const auto v = S.hxy[w][c][s];
                hx += v.x;
                hy += v.y;
                hz += S.hz[w][c][s];
            }
        const int64_t e = off + S.st.perm[s];
        const T r = S.st.geo.r[s];
        T x, y, z, ri;
        S.st.geo.get(s << 4, x, y, z, ri);
        T P = T(0);
        for (int g = g0; g < first; ++g)
        {
            DevPairGroup const& G = gt.g[g];
            if (s < S.st.begin[G.e1] || s >= S.st.begin[G.e1 + 1] || !(r < (T)G.rc)) continue;
            T fc, dfc;
            if (G.cutoffSlot == slot)
            {
                T t0, t1;
                S.fac.get(s << 4, fc, dfc, t0, t1);
                dfc *= r;
            }
            else
            {
                fc = (T)b.nbrFc[(size_t)G.cutoffSlot * b.nbrCapacity + e];
                dfc = (T)b.nbrDfc[(size_t)G.cutoffSlot * b.nbrCapacity + e];
            }
            const DevRadial* rad = gt.radial + G.radialBegin;
            const double* c = cw + (G.memberBegin - m0);
            for (int q = 0; q < G.memberCount; ++q)
            {
                const T d = r - radialShift<T>(rad[q]);
                const T v = expScaled<true>(d * d, radialScale<T>(rad[q]), S.st.expTab);
                P += (T)c[q] * (dfc - radialEta2<T>(rad[q]) * d * fc) * v;
            }
        }
        P *= ri;
        hx += x * P;
        hy += y * P;
        hz += z * P;
        b.hx[e] = (double)hx;
        b.hy[e] = (double)hy;
        b.hz[e] = (double)hz;
        fx += (double)hx;
        fy += (double)hy;
        fz += (double)hz;
    }
    fx = warpSum(fx);
    fy = warpSum(fy);
    fz = warpSum(fz);
    if (lane == 0)
    {
        S.self[warp][0] = fx;
        S.self[warp][1] = fy;
        S.self[warp][2] = fz;
    }
    __syncthreads();
    if (tid < 3)
    {
        double t = 0.0;
        for (int w = 0; w < kPairWarps; ++w) t += S.self[w][tid];
        b.fSelf[3 * (size_t)i + tid] = -t;
    }
}

template <typename T, int CAP, int CUT, int FORM, bool TIER>
__global__ void __launch_bounds__(kPairThreads, TIER ? 1 : (sizeof(T) == 8 ? 5 : 6))
    kPairForces(const __grid_constant__ DevModel model, const __grid_constant__ BatchView b, int lower,
                const __grid_constant__ DevPairTable gt)
{
    extern __shared__ __align__(16) unsigned char smemRaw[];
    ForcesStage<T, CAP>& S = *reinterpret_cast<ForcesStage<T, CAP>*>(smemRaw);
    GroupCoef<T>* coef = reinterpret_cast<GroupCoef<T>*>(smemRaw + sizeof(ForcesStage<T, CAP>));
    double* cw = reinterpret_cast<double*>(coef + gt.maxAngular);
    if constexpr (!TIER)
    {
        const int i = blockIdx.x;
        const int64_t off = b.nbrOffset[i], end = b.nbrOffset[i + 1];
        const int n = (int)(end - off);
        if (end > b.nbrCapacity || n > CAP) return;
        atomForces<T, CAP, CUT, FORM>(S, coef, cw, model, b, gt, i, off, n);
    }
    else
        forTierAtoms(S.st.todo, b, lower, CAP, false, [&](int i) {
            const int64_t off = b.nbrOffset[i];
            atomForces<T, CAP, CUT, FORM>(S, coef, cw, model, b, gt, i, off, (int)(b.nbrOffset[i + 1] - off));
            __syncthreads();
        });
}

} // namespace

} // namespace n2p2b200
