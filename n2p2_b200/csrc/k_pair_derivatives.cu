// G and stored dG/dr (API form, FP64) of the models of the pair kernels
// (sf_pairs.cuh), one block of four warps per centre atom.
//
// A thread owns one neighbour j and walks the partners k of a group's other
// block; per member it sums p1, p3 and p3 dr_k, from which the owner's row is
// -(S1 - S3) dr_j - sum p3 dr_k and its share of the self derivative S1 dr_j
// (p1, p3: SymGrpExpAngn.cpp:305-337).  Every ordered pair is evaluated, so a
// row belongs to one thread and is written once; the G sums count each pair
// twice and are halved (exact).  A sweep over the partners takes up to
// kSweep members of one eta, so the pair's geometry, cutoff and exponential
// are shared by them.  Where a block has few owners the partners are cut into
// chunks, whose sums are added in order.  All sums run in a fixed order.
//
// Bound: FP64 instructions (about 50 per ordered pair and sweep, 14 per
// member).  The warp-per-atom kernel (k_symfunc.cu, now for the other models
// and atoms beyond kPairBigCap neighbours) evaluated its members with the
// general power, division and exponential functions and read and wrote the
// rows per neighbour and group: 32 boxes (10 k atoms, 14 functions) took it
// 7.76 ms, these kernels 0.88 ms.
#include "sf_pairs.cuh"

namespace n2p2b200 {

namespace {

constexpr int kSweep = 4;          // members of one sweep
constexpr int kSweepSums = 6;      // G, S1, S3, sum p3 dr_k
constexpr int kDerivCap = 192, kDerivBigCap = 1024;

template <int CAP>
struct alignas(16) DerivStage
{
    PairStage<double, CAP> st;
    FactorStage<double, CAP> fac;
    double part[3 * kSweep * kSweepSums * 32];     // sums of the chunks after the first: (chunks - 1) x owners <= 96
    double red[kPairWarps][kSweep][4];
};

// Sums over the block of v[0..3] of up to kSweep members; valid in `red`
// after the barrier that the caller places.
__device__ __forceinline__ void warpTotals(double (*red)[4], double const (&g)[kSweep], double const (&x)[kSweep],
                                           double const (&y)[kSweep], double const (&z)[kSweep], int count, int lane)
{
#pragma unroll
    for (int q = 0; q < kSweep; ++q)
    {
        if (q >= count) break;
        const double a = warpSum(g[q]), sx = warpSum(x[q]), sy = warpSum(y[q]), sz = warpSum(z[q]);
        if (lane == 0)
        {
            red[q][0] = a;
            red[q][1] = sx;
            red[q][2] = sy;
            red[q][3] = sz;
        }
    }
}

template <int CAP>
__device__ __forceinline__ void writeTotals(DerivStage<CAP>& S, DevModel const& model, BatchView const& b,
                                            DevElement const& E, const DevMember* mem, const short* index, int count, int i,
                                            double half)
{
    __syncthreads();
    const int tid = threadIdx.x;
    if (tid < count)
    {
        double t[4];
        for (int c = 0; c < 4; ++c)
        {
            t[c] = S.red[0][tid][c];
            for (int w = 1; w < kPairWarps; ++w) t[c] += S.red[w][tid][c];
        }
        DevMember const& M = mem[index[tid]];
        b.G[(size_t)i * b.gStride + M.sf] = scaleG(model.scaling[E.sfBegin + M.sf], t[0] * half * M.gNorm);
        double* p = b.dGdrSelf + ((size_t)i * b.gStride + M.sf) * 3;
        for (int c = 0; c < 3; ++c) p[c] = t[1 + c] * M.factorNorm;
    }
    __syncthreads();
}

template <int CAP, int CUT, bool NARROW>
__device__ __forceinline__ void angularSweep(DerivStage<CAP>& S, DevModel const& model, BatchView const& b, DevPairGroup const& G,
                                             int eta, const short* index, int count, int64_t off, int i)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    DevElement const& E = model.el[b.elem[i]];
    const DevMember* mem = model.members + G.memberBegin;
    DevCutoff const& cut = model.cutoff[G.cutoffSlot];
    const bool same = G.e1 == G.e2;
    const int A0 = S.st.begin[G.e1], nA = S.st.nBelow[G.cutoffSlot][G.e1];
    const int B0 = S.st.begin[G.e2], nB = S.st.nBelow[G.cutoffSlot][G.e2];
    const int owners = same ? nA : nA + nB;
    const int width = owners <= 32 ? 32 : owners <= 64 ? 64 : kPairThreads, chunks = kPairThreads / width;
    double lam[kSweep], zl[kSweep];
    int zm1[kSweep];
#pragma unroll
    for (int q = 0; q < kSweep; ++q)
    {
        DevMember const& M = mem[index[q < count ? q : 0]];
        lam[q] = M.lambda;
        zl[q] = M.zetaLambda;
        zm1[q] = M.zetaInt - 1;
    }
    double totG[kSweep], totX[kSweep], totY[kSweep], totZ[kSweep];
#pragma unroll
    for (int q = 0; q < kSweep; ++q) totG[q] = totX[q] = totY[q] = totZ[q] = 0.0;
    const double scale = G.etaScale[eta], eta2 = G.eta2[eta];
    const int staged = G.numEta == 2 ? eta : G.comp;   // the staged Gaussian of this width
    for (int base = 0; base < owners; base += width)
    {
        const int o = base + (tid & (width - 1)), chunk = tid / width;
        const bool mine = o < owners;
        const bool first = o < nA;   // the owner is of element e1
        const int j = mine ? (first ? A0 + o : B0 + o - nA) : A0;
        const int K0 = same || !first ? A0 : B0, nK = same || !first ? nA : nB;
        const int per = (nK + chunks - 1) / chunks, k0 = K0 + min(chunk * per, nK), k1 = K0 + min((chunk + 1) * per, nK);
        double sum[kSweep][kSweepSums];
#pragma unroll
        for (int q = 0; q < kSweep; ++q)
#pragma unroll
            for (int c = 0; c < kSweepSums; ++c) sum[q][c] = 0.0;
        double x1 = 0.0, y1 = 0.0, z1 = 0.0;
        if (mine)
        {
            double i1, f1, d1, e10, e11;
            S.st.geo.get(j << 4, x1, y1, z1, i1);
            S.fac.get(j << 4, f1, d1, e10, e11);
            const double e1 = staged ? e11 : e10, i11 = i1 * i1;
            for (int k = k0; k < k1; ++k)
            {
                if (k == j) continue;
                double x2, y2, z2, i2, f2, d2, e20, e21;
                S.st.geo.get(k << 4, x2, y2, z2, i2);
                S.fac.get(k << 4, f2, d2, e20, e21);
                const double ri = i1 * i2, cost = (x1 * x2 + y1 * y2 + z1 * z2) * ri;
                double V = e1 * (staged ? e21 : e20), f3 = 1.0, pr3 = 0.0;
                if constexpr (NARROW)
                {
                    const double dx = x2 - x1, dy = y2 - y1, dz = z2 - z1;
                    const double s = dx * dx + dy * dy + dz * dz;
                    const double i3 = invSqrt(s);
                    double d3;
                    pairCutoff<CUT>(cut, cut.iw, s * i3, f3, d3);
                    if (f3 == 0.0 && d3 == 0.0) continue;
                    V *= expScaled<CUT == kCutAny>(s, scale, S.st.expTab);
                    pr3 = f1 * f2 * d3 * i3;
                }
                const double pfc = f1 * f2 * f3, A3 = pfc * ri, A1 = pfc * (ri - cost * i11);
                const double B1 = f2 * f3 * d1 - pfc * eta2, B3 = NARROW ? pfc * eta2 - pr3 : 0.0;
#pragma unroll
                for (int q = 0; q < kSweep; ++q)
                {
                    if (q >= count) break;
                    const double p = 1.0 + lam[q] * cost;
                    if (!(p > 0.0)) continue;
                    const double X = V * powAny(p, zm1[q]);
                    const double p3 = X * (zl[q] * A3 + p * B3);
                    sum[q][0] += X * (p * pfc);
                    sum[q][1] += X * (zl[q] * A1 + p * B1);
                    sum[q][2] += p3;
                    sum[q][3] += p3 * x2;
                    sum[q][4] += p3 * y2;
                    sum[q][5] += p3 * z2;
                }
            }
        }
        if (chunks > 1)
        {
            __syncthreads();
            if (chunk > 0)
#pragma unroll
                for (int q = 0; q < kSweep; ++q)
                {
                    if (q >= count) break;
#pragma unroll
                    for (int c = 0; c < kSweepSums; ++c)
                        S.part[(q * kSweepSums + c) * 96 + (chunk - 1) * width + (tid & (width - 1))] = sum[q][c];
                }
            __syncthreads();
            if (chunk == 0)
#pragma unroll
                for (int q = 0; q < kSweep; ++q)
                {
                    if (q >= count) break;
#pragma unroll
                    for (int c = 0; c < kSweepSums; ++c)
                        for (int h = 0; h + 1 < chunks; ++h) sum[q][c] += S.part[(q * kSweepSums + c) * 96 + h * width + tid];
                }
        }
        if (mine && chunk == 0)
        {
            const size_t e = (size_t)off + S.st.perm[j];
#pragma unroll
            for (int q = 0; q < kSweep; ++q)
            {
                if (q >= count) break;
                DevMember const& M = mem[index[q]];
                totG[q] += sum[q][0];
                totX[q] += sum[q][1] * x1;
                totY[q] += sum[q][1] * y1;
                totZ[q] += sum[q][1] * z1;
                const double s = sum[q][1] - sum[q][2];
                double* p = b.dGdr + ((size_t)(first ? M.rowE1 : M.rowE2) * b.nbrCapacity + e) * 3;
                p[0] = -(s * x1 + sum[q][3]) * M.factorNorm;
                p[1] = -(s * y1 + sum[q][4]) * M.factorNorm;
                p[2] = -(s * z1 + sum[q][5]) * M.factorNorm;
            }
        }
    }
    warpTotals(S.red[warp], totG, totX, totY, totZ, count, lane);
    writeTotals<CAP>(S, model, b, E, mem, index, count, i, 0.5);
}

template <int CAP>
__device__ __forceinline__ void radialRows(DerivStage<CAP>& S, DevModel const& model, BatchView const& b, DevPairTable const& gt,
                                           DevPairGroup const& G, int64_t off, int i)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    DevElement const& E = model.el[b.elem[i]];
    const DevMember* mem = model.members + G.memberBegin;
    const DevRadial* rad = gt.radial + G.radialBegin;
    const double* fc = b.nbrFc + (size_t)G.cutoffSlot * b.nbrCapacity + off;
    const double* dfc = b.nbrDfc + (size_t)G.cutoffSlot * b.nbrCapacity + off;
    for (int m0 = 0; m0 < G.memberCount; m0 += kSweep)
    {
        const int count = min(kSweep, G.memberCount - m0);
        double totG[kSweep], totX[kSweep], totY[kSweep], totZ[kSweep];
#pragma unroll
        for (int q = 0; q < kSweep; ++q) totG[q] = totX[q] = totY[q] = totZ[q] = 0.0;
        for (int s = S.st.begin[G.e1] + tid; s < S.st.begin[G.e1 + 1]; s += kPairThreads)
        {
            const double r = S.st.geo.r[s];
            if (!(r < G.rc)) continue;
            const int m = S.st.perm[s];
            const double f = fc[m], df = dfc[m];
            double x, y, z, ri;
            S.st.geo.get(s << 4, x, y, z, ri);
#pragma unroll
            for (int q = 0; q < kSweep; ++q)
            {
                if (q >= count) break;
                DevRadial const& R = rad[m0 + q];
                DevMember const& M = mem[m0 + q];
                const double d = r - R.rs;
                const double v = expScaled<true>(d * d, R.scale, S.st.expTab);
                const double p1 = (df - R.eta2 * d * f) * v * ri;
                totG[q] += v * f;
                totX[q] += p1 * x;
                totY[q] += p1 * y;
                totZ[q] += p1 * z;
                double* p = b.dGdr + ((size_t)M.rowE1 * b.nbrCapacity + off + m) * 3;
                const double c = p1 * M.factorNorm;
                p[0] = -c * x;
                p[1] = -c * y;
                p[2] = -c * z;
            }
        }
        short index[kSweep];
#pragma unroll
        for (int q = 0; q < kSweep; ++q) index[q] = (short)(m0 + q);
        warpTotals(S.red[warp], totG, totX, totY, totZ, count, lane);
        writeTotals<CAP>(S, model, b, E, mem, index, count, i, 1.0);
    }
}

template <int CAP, int CUT>
__device__ __forceinline__ void atomDerivatives(DerivStage<CAP>& S, DevModel const& model, BatchView const& b,
                                                DevPairTable const& gt, int i, int64_t off, int n)
{
    const int tid = threadIdx.x;
    const int ec = b.elem[i];
    const int g0 = gt.begin[ec], g1 = gt.begin[ec + 1];
    // rows that no member fills (entries beyond a group's cutoff) are 0
    for (int r = 0; r < model.maxRows; ++r)
    {
        double* p = b.dGdr + ((size_t)r * b.nbrCapacity + off) * 3;
        for (int k = tid; k < 3 * n; k += kPairThreads) p[k] = 0.0;
    }
    stageNeighbors<double, CAP>(S.st, off, n, model, b);
    int slot = -1;
    double eta0 = 0.0, eta1 = 0.0;
    __syncthreads();
    for (int g = g0; g < g1; ++g)
    {
        DevPairGroup const& G = gt.g[g];
        if (G.type == 2)
        {
            radialRows<CAP>(S, model, b, gt, G, off, i);
            continue;
        }
        if (G.cutoffSlot != slot || G.stageScale[0] != eta0 || G.stageScale[1] != eta1)
        {
            __syncthreads();
            slot = G.cutoffSlot;
            eta0 = G.stageScale[0];
            eta1 = G.stageScale[1];
            const double* fc = b.nbrFc + (size_t)slot * b.nbrCapacity + off;
            const double* dfc = b.nbrDfc + (size_t)slot * b.nbrCapacity + off;
            for (int m = tid; m < n; m += kPairThreads)
            {
                const int s = S.st.slotOf[m];
                const double r = S.st.geo.r[s], r2 = r * r;
                S.fac.set(s, fc[m], dfc[m] / r, expScaled<CUT == kCutAny>(r2, eta0, S.st.expTab), expScaled<CUT == kCutAny>(r2, eta1, S.st.expTab));
            }
            __syncthreads();
        }
        for (int eta = 0; eta < G.numEta; ++eta)
        {
            short index[kSweep];
            int count = 0;
            for (int c = 0; c <= 2 * kPairLevels; ++c)
            {
                const int q = c < 2 * kPairLevels ? G.combo[eta * 2 * kPairLevels + c] : -1;
                if (q >= 0) index[count++] = (short)q;
                if (count == kSweep || (c == 2 * kPairLevels && count > 0))
                {
                    if (G.type == 3) angularSweep<CAP, CUT, true>(S, model, b, G, eta, index, count, off, i);
                    else angularSweep<CAP, CUT, false>(S, model, b, G, eta, index, count, off, i);
                    count = 0;
                }
            }
        }
    }
}

template <int CAP, int CUT, bool TIER>
__global__ void __launch_bounds__(kPairThreads, TIER ? 1 : 4)
    kPairDerivatives(const __grid_constant__ DevModel model, const __grid_constant__ BatchView b, int lower,
                     const __grid_constant__ DevPairTable gt)
{
    extern __shared__ __align__(16) unsigned char smemRaw[];
    DerivStage<CAP>& S = *reinterpret_cast<DerivStage<CAP>*>(smemRaw);
    if constexpr (!TIER)
    {
        const int i = blockIdx.x;
        const int64_t off = b.nbrOffset[i], end = b.nbrOffset[i + 1];
        const int n = (int)(end - off);
        if (end > b.nbrCapacity || n > CAP) return;
        atomDerivatives<CAP, CUT>(S, model, b, gt, i, off, n);
    }
    else
        forTierAtoms(S.st.todo, b, lower, CAP, false, [&](int i) {
            const int64_t off = b.nbrOffset[i];
            atomDerivatives<CAP, CUT>(S, model, b, gt, i, off, (int)(b.nbrOffset[i + 1] - off));
            __syncthreads();
        });
}

template <int CAP, int CUT, bool TIER>
void derivativesTier(DevModel const& m, DevPairTable const& gt, BatchView const& b, int blocks, int lower, cudaStream_t st)
{
    auto k = kPairDerivatives<CAP, CUT, TIER>;
    setDynamicSmemOnce(reinterpret_cast<const void*>(k), sizeof(DerivStage<CAP>));
    k<<<blocks, kPairThreads, sizeof(DerivStage<CAP>), st>>>(m, b, lower, gt);
}

} // namespace

void launchPairDerivatives(DevModel const& m, DevPairTable const& gt, BatchView const& b, int sms, cudaStream_t st)
{
    const int need = (b.N + kPairThreads - 1) / kPairThreads, tier = need < sms ? need : sms;
    if (m.pairForm <= 3 && m.cutoff[0].type == kCutPoly2 && m.cutoff[0].rci == 0.0)
    {
        derivativesTier<kDerivCap, kCutPoly2, false>(m, gt, b, b.N, -1, st);
        derivativesTier<kDerivBigCap, kCutPoly2, true>(m, gt, b, tier, kDerivCap, st);
    }
    else
    {
        derivativesTier<kDerivCap, kCutAny, false>(m, gt, b, b.N, -1, st);
        derivativesTier<kDerivBigCap, kCutAny, true>(m, gt, b, tier, kDerivCap, st);
    }
}

} // namespace n2p2b200
