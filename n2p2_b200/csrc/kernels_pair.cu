// Host side of the two-pass symmetry-function path: shared-memory layout and
// dispatch to the kernels instantiated per cutoff type, precision and kind
// (kernels_pair_*.cu).
#include <algorithm>
#include <cstdlib>

#include "kernels.h"
#include "sf_impl.cuh"
#include "sf_pair.h"

namespace n2p2b
{

// One launcher per (cutoff type, kind, precision): pass 0 values, 1 forces.
#define N2P2B_PAIR_DECL(NAME)                                                 \
    void pairLaunch_##NAME(int, SFParams const&, PairParams const&,           \
                           PairLaunch const&, int, cudaStream_t);
N2P2B_PAIR_DECL(cos2)
N2P2B_PAIR_DECL(cos4)
N2P2B_PAIR_DECL(cosall)
N2P2B_PAIR_DECL(tanhu2)
N2P2B_PAIR_DECL(tanhu4)
N2P2B_PAIR_DECL(poly2)
N2P2B_PAIR_DECL(poly4)
N2P2B_PAIR_DECL(any2)
N2P2B_PAIR_DECL(any4)
N2P2B_PAIR_DECL(comp)
N2P2B_PAIR_DECL(anyall)
N2P2B_PAIR_DECL(cos2f)
N2P2B_PAIR_DECL(cos4f)
N2P2B_PAIR_DECL(cosallf)
N2P2B_PAIR_DECL(tanhu2f)
N2P2B_PAIR_DECL(tanhu4f)
N2P2B_PAIR_DECL(poly2f)
N2P2B_PAIR_DECL(poly4f)
N2P2B_PAIR_DECL(any2f)
N2P2B_PAIR_DECL(any4f)
N2P2B_PAIR_DECL(compf)
N2P2B_PAIR_DECL(anyallf)
#undef N2P2B_PAIR_DECL

namespace
{

constexpr int kWarpsPerCta = 4, kOwnersPerItem = 8;

constexpr std::size_t kSmemSM = 228 * 1024;

// Shared-memory layout of a pass (0 values, 1 forces) with L.wpa warps per
// atom; returns its bytes.
std::size_t layout(PairParams const& T, PairLaunch& L, int pass)
{
    std::size_t const r = L.precision != PREC_FP64 ? 4 : 8;
    std::size_t const cap = (std::size_t)L.cap, cs = cap + 1;
    std::size_t const words = (cap + 31) / 32;
    std::size_t at = 0;
    auto take = [&](int& off, std::size_t bytes) {
        off = (int)at;
        at += (bytes + 15) / 16 * 16;
    };
    int const ne = T.numElements;
    bool narrow = false;
    for (int e = 0; e < ne; ++e) narrow = narrow || T.narrow[e];
    take(L.oTab, r == 8 ? 8 * 256 : 0);    // kPairExp2
    // The tables of all elements, those of the inner loops first, while they
    // are small (the water potentials: 4 to 7 KB); else they are read
    // through L1.
    std::size_t const hot = sizeof(PairUnit) * T.unitBeg[ne]
                          + sizeof(PairRun) * T.runBeg[ne]
                          + sizeof(PairShape) * T.shapeBeg[ne];
    std::size_t const cold = sizeof(PairRadial) * T.radialBeg[ne]
                           + sizeof(PairCell) * T.cellBeg[ne];
    L.tables = (hot <= 24 * 1024 ? 1 : 0) | (cold <= 6 * 1024 ? 2 : 0);
    take(L.oTables, (L.tables & 1 ? hot : 0) + (L.tables & 2 ? cold : 0));
    std::size_t const team = at;
    at = 0;
    std::size_t const w = (std::size_t)L.wpa;
    take(L.oRec, 6 * r * cs);
    take(L.oFc, r * cs * std::max(T.maxFc - 1, 0));
    take(L.oRad, (pass == 0 ? 1 : 2) * r * cs * T.maxRad);
    if (narrow) take(L.oBits, 4 * cap * words);
    bool sorted = false;
    for (int e = 0; e < ne; ++e) sorted = sorted || T.sorted[e];
    if (sorted)
    {
        take(L.oSort, 4 * cap);
        if (pass == 1) take(L.oOrig, 2 * cap);
    }
    if (pass == 0)
    {
        take(L.oG, r * w * L.maxSF);
        // First positions and distances, then pair lists and lane sums.  A
        // warp's pair list holds the pairs of several rows, and at least one
        // row's.
        std::size_t const x = at;
        take(L.oPos, 16 * 32 * words);
        take(L.oDist, r * cap);
        std::size_t const y = at;
        at = x;
        L.pairCap = std::max(512, L.cap);
        take(L.oPairs, 4 * (std::size_t)L.pairCap * w);
        take(L.oRed, r * 8 * 33 * w);
        at = std::max(at, y);
    }
    else
    {
        take(L.oAr, r * cap);
        take(L.oDfc, r * cs * T.maxFc);
        take(L.oCoef, r * T.maxCells);
        take(L.oOrder, 2 * cap);
        if (w > 1) take(L.oF, 8 * 3 * cap);
        if (narrow)
        {
            take(L.oPre, 2 * cap * (ne + 1));
            take(L.oKey, 4 * cap);
        }
        // First positions, then partner lists.
        std::size_t const x = at;
        take(L.oPos, 16 * 32 * words);
        std::size_t const y = at;
        at = x;
        if (narrow) take(L.oList, 2 * kOwnersPerItem * cap * w);
        at = std::max(at, y);
    }
    L.teamBytes = (int)at;
    L.oTeam = (int)team;
    return team + at * (kWarpsPerCta / L.wpa);
}

void dispatch(int pass, SFParams const& P, PairParams const& dev,
              PairLaunch const& L, int shm, cudaStream_t s)
{
    bool const f = L.precision != PREC_FP64;
#define N2P2B_GO(NAME)                                                        \
    (f ? pairLaunch_##NAME##f(pass, P, dev, L, shm, s)                        \
       : pairLaunch_##NAME(pass, P, dev, L, shm, s))
    // Potentials of PK_POW2 units alone run on kernels without the other
    // kinds' code, as do those of compact units; the cosine kernels take the
    // cutoff as a series in r^2 (no inner radius).
    bool const z4 = dev.slots > 3;
    bool const cosine = P.cutoffType == 1
                     && (P.numGroups == 0 || P.groups[0].rci == 0.0);
    if (dev.kinds == 1 << PK_COMPACT) N2P2B_GO(comp);
    else if (dev.kinds & ~(1 << PK_POW2))
    {
        if (cosine) N2P2B_GO(cosall);
        else N2P2B_GO(anyall);
    }
    else if (cosine) z4 ? N2P2B_GO(cos4) : N2P2B_GO(cos2);
    else
        switch (P.cutoffType)
        {
        case 2: z4 ? N2P2B_GO(tanhu4) : N2P2B_GO(tanhu2); break;
        case 6: z4 ? N2P2B_GO(poly4) : N2P2B_GO(poly2); break;
        default: z4 ? N2P2B_GO(any4) : N2P2B_GO(any2); break;
        }
#undef N2P2B_GO
}

} // namespace

bool pairFits(PairParams const& T, int cap, int precision, int maxSF)
{
    PairLaunch L;
    L.cap = cap;
    L.precision = precision;
    L.maxSF = maxSF;
    L.wpa = kWarpsPerCta;
    return cap < 65536 && layout(T, L, 0) <= (std::size_t)kPairSmemBlock
        && layout(T, L, 1) <= (std::size_t)kPairSmemBlock;
}

void launchPair(int pass, SFParams const& P, PairParams const& host,
                PairParams const& dev, PairLaunch const& L0, cudaStream_t s)
{
    if (L0.n <= 0) return;
    PairLaunch L = L0;
    // One or four warps per atom.  One needs no barriers and adds no shares,
    // four keep the chip busy with fewer atoms and need a quarter of the
    // shared memory.  One if three blocks per multiprocessor fit (where they
    // do not, 2,048 atoms of anisole, one / four: values 4.1 / 1.6 ms, forces
    // 9.6 / 3.6) and:
    //  values  its warps fill two thirds of a wave, but do not just begin a
    //          second one (52 functions, FP64, one / four: 768 atoms 0.070 /
    //          0.062 ms, 1,200 0.080 / 0.086, 1,920 0.132 / 0.115, 3,072
    //          0.154 / 0.168, 24,576 0.97 / 1.16);
    //  forces  enough waves to even out the atoms' unequal work (FP64: 6,000
    //          atoms 0.68 / 0.64, 9,000 0.92 / 0.94, 24,576 2.41 / 2.52; FP32,
    //          92 functions: 4,200 0.370 / 0.365, 6,000 0.495 / 0.510);
    //          atoms of few neighbors have too few items of eight owners for
    //          four warps (1,728 atoms of Cu2S 0.267 / 0.308).
    L.wpa = 1;
    std::size_t shm = layout(host, L, pass);
    bool const f = L.precision != PREC_FP64;
    std::size_t const blocks = std::min<std::size_t>(
        f ? 4 : 3, kSmemSM / (shm + 1024));
    double const waves = (double)L.n
                       / ((double)(kWarpsPerCta * std::max<std::size_t>(blocks, 1))
                          * L.sms);
    bool one = waves >= 2.0 / 3.0 && (waves <= 1.0 || waves >= 1.3);
    if (pass == 1 && L.cap > 80) one = L.n >= (f ? 36 : 48) * L.sms;
    if (blocks < 3 || !one)
    {
        L.wpa = kWarpsPerCta;
        shm = layout(host, L, pass);
    }
    // N2P2B_PAIR_WPA=1 or 4 asks for one of the two (measurements, tests); one
    // warp per atom only where four atoms' shared memory fits a block.
    if (char const* e = std::getenv("N2P2B_PAIR_WPA"))
    {
        L.wpa = 1;
        if (std::atoi(e) != 1
            || layout(host, L, pass) > (std::size_t)kPairSmemBlock)
            L.wpa = kWarpsPerCta;
        shm = layout(host, L, pass);
    }
    noteLaunches(1);
    dispatch(pass, P, dev, L, (int)shm, s);
}

} // namespace n2p2b
