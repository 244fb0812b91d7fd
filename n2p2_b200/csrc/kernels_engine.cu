// Neighbor lists supplied by an MD engine: the engine's entries (in its own
// order, with its force-array indices) regrouped on the device into the
// element-grouped structure of arrays that the symmetry-function kernels
// stage, and the reverse index from force targets to entries.
#include "device_common.cuh"
#include "kernels.h"

namespace n2p2b
{

namespace
{

// Thread per entry: elements and targets are in range.  It runs before
// anything of the list that is in place is overwritten, so that a refused
// list leaves the previous one (or the structure) as it was.
__global__ void engineCheckKernel(EngineListLaunch const L)
{
    long const e = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= L.entries) return;
    int const el = L.rawElem[e];
    int64_t const idx = L.rawIndex[e];
    if (el < 0 || el >= L.numElements || idx < 0 || idx >= L.numTargets)
        *L.bad = 1;
}

// Warp per atom: stable regrouping of its entries by neighbor element.  The
// distance is formed as InterfaceLammps::addNeighbor does (n.d = sqrt(d2),
// then scaled like the components), without contraction.  Entries are 36
// bytes in and 37 out: memory-bound, coalesced on the way in and in runs of
// one element on the way out.
__global__ void __launch_bounds__(128)
engineGroupKernel(EngineListLaunch const L)
{
    int const lane = threadIdx.x & 31;
    long const i = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i >= L.n) return;
    unsigned const below = (1u << lane) - 1u;
    long const b = L.off[i];
    int const cnt = L.off[i + 1] - (int)b;
    int at[kMaxElem];
#pragma unroll
    for (int e = 0; e < kMaxElem; ++e) at[e] = 0;
    for (int t = lane; t - lane < cnt; t += 32)
    {
        int const el = t < cnt ? L.rawElem[b + t] : -1;
#pragma unroll
        for (int e = 0; e < kMaxElem; ++e)
            if (e < L.numElements)
                at[e] += __popc(__ballot_sync(0xffffffffu, el == e));
    }
    int run = 0;
#pragma unroll
    for (int e = 0; e < kMaxElem; ++e)
        if (e < L.numElements)
        {
            int const c = at[e];
            if (lane == 0) L.nbrCountElem[i * L.numElements + e] = c;
            at[e] = run;
            run += c;
        }
    for (int t = lane; t - lane < cnt; t += 32)
    {
        bool const in = t < cnt;
        int const el = in ? L.rawElem[b + t] : -1;
        int pos = 0;
#pragma unroll
        for (int e = 0; e < kMaxElem; ++e)
            if (e < L.numElements)
            {
                unsigned const m = __ballot_sync(0xffffffffu, el == e);
                if (el == e) pos = at[e] + __popc(m & below);
                at[e] += __popc(m);
            }
        if (!in) continue;
        double const x = L.rawDr[3 * (b + t)], y = L.rawDr[3 * (b + t) + 1],
                     z = L.rawDr[3 * (b + t) + 2];
        double const d2 = __dadd_rn(__dadd_rn(__dmul_rn(x, x),
                                              __dmul_rn(y, y)),
                                    __dmul_rn(z, z));
        int const target = (int)L.rawIndex[b + t];
        long const o = b + pos;
        L.nbrIdx[o] = target;
        L.nbrEl[o] = (int8_t)el;
        L.dx[o] = __dmul_rn(x, L.scale);
        L.dy[o] = __dmul_rn(y, L.scale);
        L.dz[o] = __dmul_rn(z, L.scale);
        L.dd[o] = __dmul_rn(__dsqrt_rn(d2), L.scale);
        atomicAdd(&L.revCount[target], 1);
    }
}

// Thread per entry: a place in its target's segment.  The order inside a
// segment is that of the atomics; engineSortKernel makes it ascending.
__global__ void engineFillKernel(EngineListLaunch const L)
{
    long const e = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= L.entries) return;
    int const m = L.nbrIdx[e];
    int const k = atomicSub(&L.revCount[m], 1) - 1;
    L.revTmp[L.revOff[m] + k] = (int)e;
}

// Warp per target: its entries in ascending order (rank by counting; the
// segments of a condensed phase hold about a hundred).
__global__ void __launch_bounds__(128)
engineSortKernel(EngineListLaunch const L)
{
    int const lane = threadIdx.x & 31;
    long const m = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (m >= L.numTargets) return;
    int const b = L.revOff[m], c = L.revOff[m + 1] - b;
    int const* src = L.revTmp + b;
    for (int t = lane; t < c; t += 32)
    {
        int const v = src[t];
        int r = 0;
        for (int q = 0; q < c; ++q) r += src[q] < v ? 1 : 0;
        L.revEntry[b + r] = v;
    }
}

} // namespace

void launchEngineCheck(EngineListLaunch const& L, cudaStream_t s)
{
    cudaMemsetAsync(L.bad, 0, sizeof(int), s);
    if (L.entries == 0) return;
    noteLaunches(1);
    engineCheckKernel<<<(unsigned)((L.entries + 255) / 256), 256, 0, s>>>(L);
}

void launchEngineList(EngineListLaunch const& L, cudaStream_t s)
{
    int const tb = 128, warps = tb / 32;
    cudaMemsetAsync(L.revCount, 0, sizeof(int) * (std::size_t)L.numTargets, s);
    noteLaunches(L.entries > 0 ? 4 : 2);
    engineGroupKernel<<<(unsigned)((L.n + warps - 1) / warps), tb, 0, s>>>(L);
    launchOffsetScan(L.numTargets, L.revCount, L.revOff, s);
    if (L.entries == 0) return;
    engineFillKernel<<<(unsigned)((L.entries + 255) / 256), 256, 0, s>>>(L);
    engineSortKernel<<<(unsigned)((L.numTargets + warps - 1) / warps), tb, 0,
                       s>>>(L);
}

} // namespace n2p2b
