// Launch sequence of the general symmetry-function passes for one precision:
// the tiers of stage capacity.
#pragma once

#include "sf_fast.cuh"

namespace n2p2b200 {

namespace {

constexpr int kBigCap = 1024, kBigWarps = 1;    // last tier (flags larger atoms)
constexpr int kGenericCap = 160, kGenericWarps = 4;

int gridFor(int N, int warpsPerBlock, int sms, int perSM)
{
    int need = (N + warpsPerBlock - 1) / warpsPerBlock;
    int cap = sms * perSM;
    return need < cap ? (need > 0 ? need : 1) : cap;
}

template <typename T, int CAP, int WARPS>
void valuesTier(DevModel const& m, BatchView const& b, int sms, cudaStream_t st, int lower, int flag, int perSM)
{
    static_assert(sizeof(ValuesSmem<T, CAP>) % 16 == 0, "per-warp blocks must stay 16-byte aligned");
    const size_t smem = sizeof(ValuesSmem<T, CAP>) * WARPS;
    auto k = kSFValuesF<T, CAP, WARPS>;
    setDynamicSmemOnce(reinterpret_cast<const void*>(k), smem);
    k<<<gridFor(b.N, WARPS, sms, perSM), WARPS * 32, smem, st>>>(m, b, lower, flag);
}

template <typename T, int CAP, int WARPS>
void forcesTier(DevModel const& m, BatchView const& b, int sms, cudaStream_t st, int lower, int perSM)
{
    static_assert(sizeof(ForcesSmem<T, CAP>) % 16 == 0, "per-warp blocks must stay 16-byte aligned");
    const size_t smem = sizeof(ForcesSmem<T, CAP>) * WARPS;
    auto k = kSFForcesF<T, CAP, WARPS>;
    setDynamicSmemOnce(reinterpret_cast<const void*>(k), smem);
    k<<<gridFor(b.N, WARPS, sms, perSM), WARPS * 32, smem, st>>>(m, b, lower);
}

template <typename T>
void valuesT(DevModel const& m, BatchView const& b, int sms, cudaStream_t st)
{
    valuesTier<T, kGenericCap, kGenericWarps>(m, b, sms, st, -1, 0, 32);
    valuesTier<T, kBigCap, kBigWarps>(m, b, sms, st, kGenericCap, 1, 2);
}

template <typename T>
void forcesT(DevModel const& m, BatchView const& b, int sms, cudaStream_t st)
{
    forcesTier<T, kGenericCap, kGenericWarps>(m, b, sms, st, -1, 32);
    forcesTier<T, kBigCap, kBigWarps>(m, b, sms, st, kGenericCap, 2);
}

} // namespace

} // namespace n2p2b200
