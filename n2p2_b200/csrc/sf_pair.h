// Tables and launch descriptors of the two-pass symmetry-function path
// (sf_pair.cuh): values in one pass, forces by the chain rule with dE/dG
// contracted before the triplet sums in a second one; dG/dr is not formed.
#pragma once

#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>
#include <string>
#include <vector>

#include "tables.h"

namespace n2p2b
{

// Angular functions are products of a radial part (a run: eta, rs and the
// cutoffs; compact: the radial window functions) and an angular part (a
// shape: zeta, lambda; compact: the window function of theta).  A group is
// cut into units of a few runs and shapes; the cells of a unit are the
// combinations of its runs and shapes, each the group's member with that run
// and shape or empty.  Kinds of units (the first two: rs = 0, lambda = +-1,
// integer zeta; shapes are the pairs (1 - cos)^zeta, (1 + cos)^zeta):
//   PK_POW2     zeta in 1, 2, 4 (, 8, 16): slot z is zeta = 2^z, slots that
//               the group has are set in PairUnit::mask.
//   PK_LADDER   other zeta, ascending, each reached from the one before by
//               squarings and multiplications (PairUnit::prog).
//               Both: cell (z, a, sign) at (z nr + a) 2 + sign.
//   PK_GENERAL  every other exponential function: cell (a, s) at a
//               kPairGenShapes + s.
//   PK_COMPACT  cell (a, s) at a kPairCompShapes + s.
enum PairKind { PK_POW2 = 0, PK_LADDER = 1, PK_GENERAL = 2, PK_COMPACT = 3 };
constexpr int kPairLadder = 4;        // values of zeta of a ladder unit
constexpr int kPairRuns = 4;          // PK_POW2 units
constexpr int kPairGenRuns = 4;       // the other exponential ones
constexpr int kPairGenShapes = 6;
constexpr int kPairCompRuns = 9;      // compact units
constexpr int kPairCompShapes = 6;
constexpr int kPairMaxRc = 4;         // (cutoff radius, weighted) per element
constexpr int kPairMaxRad = 16;       // radial window functions per element
// Dynamic shared memory of a block, at most: 227 KB less 1 KB for the
// kernels' static arrays.
constexpr int kPairSmemBlock = 226 * 1024;

struct PairUnit
{
    int      kind;
    int      narrow;      // 1: types 3, 13, 21, 24 (r_jk matters)
    int      weighted;    // 1: types 13, 24, 25 (every neighbor element)
    int      e1, e2;
    int      nr, ns;      // runs, shapes (ladder: values of zeta)
    int      fcSlot;      // exponential: staged cutoff values of (rc, Z)
    int      run, shape;  // first run / shape in the tables
    int      cell;        // first cell, relative to the element's cells
    int      group;       // DevGroup (cutoff of r_jk)
    int      hasRs;       // some run has rs != 0
    int      exactMask;   // rc is the element's largest narrow cutoff
    unsigned mask;        // PK_POW2
    int      core;        // PK_COMPACT: the shapes' common core function
                          // (CompactCore), 0 if they differ
    unsigned prog[4];     // ladder: steps to zeta z: count in bits 0-7, then
                          // one bit per step (0: P = P^2, 1: P = P p)
    double   rc2;         // squared cutoff radius (compact: largest rc)
    double   a2q;         // (pi / (2 rc))^2
    double   qf;          // -(pi / rc)^2 / 2
    double   zeta[4];     // ladder
};

// Cells of a unit of kind KIND.  PK_POW2 units have those of PairParams::slots values of
// zeta, which may be fewer than the slots a kernel is compiled for: kernels
// touch these cells and no others.
template <int KIND>
#ifdef __CUDACC__
__host__ __device__
#endif
inline int pairUnitCells(PairUnit const& u)
{
    if (KIND == PK_GENERAL) return u.nr * kPairGenShapes;
    if (KIND == PK_COMPACT) return u.nr * kPairCompShapes;
    return 2 * u.nr * u.ns;
}

struct PairRun
{
    double eta, rs;                       // exponential; compact: (rl, rc)
    double center, scale;                 // compact window function;
                                          // exponential: center = -eta / ln 2
    int    core, asym;
    int    slot;                          // compact: staged radial values
    int    pad;
};

struct PairShape
{
    double lambda, zl;                    // zl = zeta lambda
    double zeta;                          // compact: left, right in lambda,
    double center, scale;                 // zl; center and scale
    int    zi, useInt;                    // zi = zeta - 1; compact: zi = core
};

// Radial member (types 2, 12, 20, 23) with its parameters: eta and rs of an
// exponential one, the window function (rl, rc, center, scale, core, asym)
// of a compact one.
struct PairRadial
{
    int    compact, weighted;
    int    e1;            // neighbor element (weighted: every element)
    int    fcSlot;        // staged cutoff values, -1: form them (group)
    int    group;
    int    cell;          // relative to the element's cells
    int    core, asym;
    double eta, rs;       // compact: rl, rc
    double center, scale; // exponential: center = -eta / ln 2
};

struct PairCell
{
    int    sf;            // -1: empty
    double fn;            // factor of dG/d(sum): 2^(1-zeta) x scaling factor
};

struct PairFc { int group, weighted; };
struct PairRad
{
    double rl, rc, center, scale;
    int    core, asym, weighted, pad;
};

struct PairParams
{
    int unitBeg[kMaxElem + 1];
    int radialBeg[kMaxElem + 1];
    int cellBeg[kMaxElem + 1];
    int fcBeg[kMaxElem + 1];
    int radBeg[kMaxElem + 1];
    int runBeg[kMaxElem + 1];
    int shapeBeg[kMaxElem + 1];
    int narrow[kMaxElem];         // element has narrow units
    int sorted[kMaxElem];         // neighbors staged by distance (the element
                                  // has compact units)
    double narrowRc2[kMaxElem];   // largest squared cutoff of those
    int maxCells, maxFc, maxRad, numElements;
    int anyWeighted;              // some member weights by atomic number
    int slots;                    // PK_POW2: 3 (zeta <= 4) or 5 slots
    int kinds;                    // bit mask of the unit kinds
    double farAway;               // a distance beyond every cutoff
    PairUnit const*   units;
    PairRun const*    runs;
    PairShape const*  shapesTab;
    PairRadial const* radials;
    PairCell const*   cells;
    PairFc const*     fcs;
    PairRad const*    rads;
};

// Host tables.
struct PairTables
{
    bool        ok = false;
    std::string why;
    PairParams  p{};
    std::vector<PairUnit>   units;
    std::vector<PairRun>    runs;
    std::vector<PairShape>  shapes;
    std::vector<PairRadial> radials;
    std::vector<PairCell>   cells;
    std::vector<PairFc>     fcs;
    std::vector<PairRad>    rads;
};

// Builds the tables from the symmetry-function tables (host copies);
// ok = false with the reason for potentials that this path does not serve.
void buildPairTables(SFParams const& P, PairTables& t);

struct PairLaunch
{
    int            n = 0;
    int            cap = 0;           // neighbor staging capacity
    int            sms = 1;           // multiprocessors of the device
    int            precision = 0;
    int            maxSF = 0;
    // Byte offsets into dynamic shared memory (set by the launcher).
    int            oTab = 0, oTables = 0, oTeam = 0, teamBytes = 0;
    // ... and into a team's region.
    int            oPos = 0, oDist = 0, oRec = 0, oFc = 0, oDfc = 0, oRad = 0,
                   oCoef = 0, oBits = 0, oPre = 0, oOrder = 0, oKey = 0,
                   oList = 0, oOrig = 0, oSort = 0, oPairs = 0, oRed = 0, oG = 0, oAr = 0, oF = 0;
    int            tables = 0;        // bit 0: units, runs, shapes in smem,
                                      // bit 1: radial members, cells
    int            wpa = 1;           // warps per atom: 1 or 4
    int            pairCap = 0;       // entries of a warp's pair list
    int const*     elem = nullptr;
    int const*     nbrOff = nullptr;
    int const*     nbrCountElem = nullptr;
    double const*  dx = nullptr;
    double const*  dy = nullptr;
    double const*  dz = nullptr;
    double const*  dd = nullptr;
    SFScale const* scale = nullptr;
    void*          G = nullptr;       // values pass: [n][maxSF]
    void const*    dEdG = nullptr;    // forces pass: [n][maxSF]
    double*        pairF = nullptr;   // [entries][3]
    double*        selfF = nullptr;   // [n][3]
    int*           status = nullptr;
};

// Whether both passes' shared memory fits for `cap` neighbors.
bool pairFits(PairParams const& T, int cap, int precision, int maxSF);
// Pass 0 computes the values, pass 1 the pair and self forces; `host` and
// `dev` are the same tables with host and device pointers.
void launchPair(int pass, SFParams const& P, PairParams const& host,
                PairParams const& dev, PairLaunch const& L, cudaStream_t s);

} // namespace n2p2b
