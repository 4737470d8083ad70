// Launches of the pair kernels (sf_pairs.cuh) of one precision: the first
// tier's stage capacity (shape variant 0-2) with one block per atom, then the
// tiers of larger atoms, whose blocks look through the atoms 128 at a time.
#pragma once

#include "sf_pairs.cuh"

namespace n2p2b200 {

namespace {

constexpr int kPairMidCap = 384, kPairBigCap = 1024;

template <typename T, int CAP, int CUT, int FORM, bool TIER>
void pairValuesTier(DevModel const& m, DevPairTable const& gt, BatchView const& b, int blocks, int lower, int flag,
                    cudaStream_t st)
{
    const size_t smem = sizeof(ValuesStage<T, CAP>) + sizeof(double) * kPairWarps * (size_t)m.maxSF;
    auto k = kPairValues<T, CAP, CUT, FORM, TIER>;
    setDynamicSmemOnce(reinterpret_cast<const void*>(k), smem);
    k<<<blocks, kPairThreads, smem, st>>>(m, b, lower, flag, gt);
}

template <typename T, int CAP, int CUT, int FORM, bool TIER>
void pairForcesTier(DevModel const& m, DevPairTable const& gt, BatchView const& b, int blocks, int lower, cudaStream_t st)
{
    const size_t smem = sizeof(ForcesStage<T, CAP>) + sizeof(GroupCoef<T>) * (size_t)gt.maxAngular +
                        sizeof(double) * (size_t)m.maxSF;
    auto k = kPairForces<T, CAP, CUT, FORM, TIER>;
    setDynamicSmemOnce(reinterpret_cast<const void*>(k), smem);
    k<<<blocks, kPairThreads, smem, st>>>(m, b, lower, gt);
}

inline int tierBlocks(int N, int sms, int perSM)
{
    const int need = (N + kPairThreads - 1) / kPairThreads;
    return need < sms * perSM ? need : sms * perSM;
}

template <typename T, int CUT, int FORM>
void pairValues(DevModel const& m, DevPairTable const& gt, BatchView const& b, int sms, cudaStream_t st, int variant)
{
    const int cap0 = kSFShapeCapacity[variant];
    if (variant == 0) pairValuesTier<T, 128, CUT, FORM, false>(m, gt, b, b.N, -1, 0, st);
    else if (variant == 1) pairValuesTier<T, 160, CUT, FORM, false>(m, gt, b, b.N, -1, 0, st);
    else pairValuesTier<T, 192, CUT, FORM, false>(m, gt, b, b.N, -1, 0, st);
    pairValuesTier<T, kPairMidCap, CUT, FORM, true>(m, gt, b, tierBlocks(b.N, sms, 4), cap0, 0, st);
    pairValuesTier<T, kPairBigCap, CUT, FORM, true>(m, gt, b, tierBlocks(b.N, sms, 1), kPairMidCap, 1, st);
}

template <typename T, int CUT, int FORM>
void pairForces(DevModel const& m, DevPairTable const& gt, BatchView const& b, int sms, cudaStream_t st, int variant)
{
    const int cap0 = kSFShapeCapacity[variant];
    if (variant == 0) pairForcesTier<T, 128, CUT, FORM, false>(m, gt, b, b.N, -1, st);
    else if (variant == 1) pairForcesTier<T, 160, CUT, FORM, false>(m, gt, b, b.N, -1, st);
    else pairForcesTier<T, 192, CUT, FORM, false>(m, gt, b, b.N, -1, st);
    pairForcesTier<T, kPairMidCap, CUT, FORM, true>(m, gt, b, tierBlocks(b.N, sms, 2), cap0, st);
    pairForcesTier<T, kPairBigCap, CUT, FORM, true>(m, gt, b, tierBlocks(b.N, sms, 1), kPairMidCap, st);
}

// Instances: the poly2 cutoff with zeta powers of two up to 4 or 16, any
// cutoff with powers of two, and any integers (the only one for angular
// Gaussians that underflow inside the cutoff, pairForm 4).
template <typename T>
void pairValuesT(DevModel const& m, DevPairTable const& gt, BatchView const& b, int sms, cudaStream_t st, int variant)
{
    const bool poly2 = m.cutoff[0].type == kCutPoly2 && m.cutoff[0].rci == 0.0;
    if (m.pairForm == 1 && poly2) pairValues<T, kCutPoly2, 3>(m, gt, b, sms, st, variant);
    else if (m.pairForm == 2 && poly2) pairValues<T, kCutPoly2, 5>(m, gt, b, sms, st, variant);
    else if (m.pairForm <= 2) pairValues<T, kCutAny, 5>(m, gt, b, sms, st, variant);
    else pairValues<T, kCutAny, 0>(m, gt, b, sms, st, variant);
}

template <typename T>
void pairForcesT(DevModel const& m, DevPairTable const& gt, BatchView const& b, int sms, cudaStream_t st, int variant)
{
    const bool poly2 = m.cutoff[0].type == kCutPoly2 && m.cutoff[0].rci == 0.0;
    if (m.pairForm == 1 && poly2) pairForces<T, kCutPoly2, 3>(m, gt, b, sms, st, variant);
    else if (m.pairForm == 2 && poly2) pairForces<T, kCutPoly2, 5>(m, gt, b, sms, st, variant);
    else if (m.pairForm <= 2) pairForces<T, kCutAny, 5>(m, gt, b, sms, st, variant);
    else pairForces<T, kCutAny, 0>(m, gt, b, sms, st, variant);
}

} // namespace

} // namespace n2p2b200
