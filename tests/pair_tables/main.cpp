// Reads exponential symmetry-function groups and prints the two-pass path's
// tables for them (test_pair_tables_cpu.py).
//   input:  elements, then per group: element type e1 e2 rc members, and per
//           member eta rs lambda zeta (groups in element order)
//   output: "ok slots kinds maxCells" or "no <reason>", then per unit
//           "unit element kind cell cells" and per radial member
//           "radial element cell"
#include <cmath>
#include <iostream>
#include <vector>

#include "sf_pair.h"

using namespace n2p2b;

static int cells(PairUnit const& u)
{
    switch (u.kind)
    {
    case PK_POW2: return pairUnitCells<PK_POW2>(u);
    case PK_LADDER: return pairUnitCells<PK_LADDER>(u);
    case PK_GENERAL: return pairUnitCells<PK_GENERAL>(u);
    default: return pairUnitCells<PK_COMPACT>(u);
    }
}

int main()
{
    SFParams P{};
    std::cin >> P.numElements;
    std::vector<DevGroup> groups;
    std::vector<DevMember> members;
    std::vector<int> owner;
    int e, count, next[kMaxElem] = {};
    DevGroup g{};
    while (std::cin >> e >> g.type >> g.e1 >> g.e2 >> g.rc >> count)
    {
        g.rc2 = g.rc * g.rc;
        g.mbeg = (int)members.size();
        g.mcnt = count;
        for (int m = 0; m < count; ++m)
        {
            DevMember d{};
            std::cin >> d.eta >> d.rs >> d.lambda >> d.zeta;
            d.zetaInt = (int16_t)std::lround(d.zeta);
            d.useIntPow = d.zetaInt == d.zeta;
            d.factorNorm = 1.0;
            d.sf = (int16_t)next[e]++;
            members.push_back(d);
        }
        groups.push_back(g);
        owner.push_back(e);
    }
    for (int k = 0; k <= P.numElements; ++k)
    {
        int at = 0;
        while (at < (int)owner.size() && owner[at] < k) ++at;
        P.groupBeg[k] = at;
    }
    P.numGroups = (int)groups.size();
    P.groups = groups.data();
    P.members = members.data();
    PairTables t;
    buildPairTables(P, t);
    if (!t.ok)
    {
        std::cout << "no " << t.why << "\n";
        return 0;
    }
    std::cout << "ok " << t.p.slots << " " << t.p.kinds << " "
              << t.p.maxCells << "\n";
    for (int k = 0; k < P.numElements; ++k)
    {
        for (int u = t.p.unitBeg[k]; u < t.p.unitBeg[k + 1]; ++u)
            std::cout << "unit " << k << " " << t.units[u].kind << " "
                      << t.units[u].cell << " " << cells(t.units[u]) << "\n";
        for (int r = t.p.radialBeg[k]; r < t.p.radialBeg[k + 1]; ++r)
            std::cout << "radial " << k << " " << t.radials[r].cell << "\n";
        std::cout << "cells " << k << " "
                  << t.p.cellBeg[k + 1] - t.p.cellBeg[k] << "\n";
    }
    return 0;
}
