// Host tables of the two-pass symmetry-function path (sf_pair.h), built from
// the group / member tables of the general kernels.
#include <algorithm>
#include <cmath>

#include "sf_pair.h"

namespace n2p2b
{

namespace
{

constexpr double kMinusLog2E = -0x1.71547652b82fep+0;   // -1 / ln 2

bool isRadial(int type)
{
    return type == 2 || type == 12 || type == 20 || type == 23;
}

// The exponentials take any exponent from 0 down whose size in their unit
// (ln 2 / 256) stays below 2^31; eta < 0 is left to the other kernels.  The
// largest sums of squares are those with the record of a partner far away:
// neighbors up to `rc` (the potential's largest cutoff) from the atom, the
// record at 2 rc, 3 rc between the two.
bool exponentFits(double eta, double rs, double rc, bool radial)
{
    auto square = [](double x) { return x * x; };
    double const a = std::fabs(rs);
    double const sum = radial ? square(rc + a)
        : square(std::max(rc, a)) + square(std::max(2.0 * rc, a))
          + square(std::max(3.0 * rc, a));
    return eta >= 0.0 && eta * sum < 5.8e6;
}

// Index of (group's rc, weighted) among the element's staged cutoff values,
// added if new; -1 if there are too many.
int fcSlotOf(SFParams const& P, PairTables& t, int beg, int group, int weighted)
{
    for (std::size_t k = beg; k < t.fcs.size(); ++k)
    {
        DevGroup const& o = P.groups[t.fcs[k].group];
        DevGroup const& g = P.groups[group];
        if (o.rc == g.rc && o.rci == g.rci && t.fcs[k].weighted == weighted)
            return (int)k - beg;
    }
    if ((int)t.fcs.size() - beg >= kPairMaxRc) return -1;
    t.fcs.push_back(PairFc{group, weighted});
    return (int)t.fcs.size() - 1 - beg;
}

int radSlotOf(PairTables& t, int beg, DevMember const& m, int weighted)
{
    for (std::size_t k = beg; k < t.rads.size(); ++k)
    {
        PairRad const& r = t.rads[k];
        if (r.rl == m.eta && r.rc == m.rs && r.core == m.zetaInt
            && r.asym == m.useIntPow && r.weighted == weighted)
            return (int)k - beg;
    }
    if ((int)t.rads.size() - beg >= kPairMaxRad) return -1;
    t.rads.push_back(PairRad{m.eta, m.rs, m.factorDeriv, m.zetaLambda,
                             m.zetaInt, m.useIntPow, weighted, 0});
    return (int)t.rads.size() - 1 - beg;
}

bool sameRun(DevMember const& a, DevMember const& b, bool compact)
{
    if (compact)
        return a.eta == b.eta && a.rs == b.rs && a.zetaInt == b.zetaInt
            && a.useIntPow == b.useIntPow;
    return a.eta == b.eta && a.rs == b.rs;
}

bool sameShape(DevMember const& a, DevMember const& b, bool compact)
{
    if (compact)
        return a.lambda == b.lambda && a.zeta == b.zeta
            && a.zetaInt == b.zetaInt;
    return a.lambda == b.lambda && a.zeta == b.zeta;
}

// The steps from zeta `from` to zeta `to` (1 <= from < to): binary digits of
// the quotient if it is whole, else of `to` from 1 (the ladder starts over:
// bit 31); false if they do not fit.
bool ladderSteps(int from, int to, unsigned& prog)
{
    bool const restart = to % from != 0;
    int const q = restart ? to : to / from;
    // Reaching q p from p by squarings needs q to be a power of two unless
    // p is the first power.
    if (!restart && from > 1 && (q & (q - 1)) != 0)
        return ladderSteps(1, to, prog) && ((prog |= 1u << 31), true);
    std::vector<int> ops;
    int top = 0;
    while ((q >> (top + 1)) != 0) ++top;
    for (int b = top - 1; b >= 0; --b)
    {
        ops.push_back(0);
        if ((q >> b) & 1) ops.push_back(1);
    }
    if (ops.size() > 20) return false;
    prog = (unsigned)ops.size() | (restart ? 1u << 31 : 0u);
    for (std::size_t k = 0; k < ops.size(); ++k)
        prog |= (unsigned)ops[k] << (8 + k);
    return true;
}

PairUnit unitOf(DevGroup const& g, PairTables const& t, int gi, int cells)
{
    PairUnit u{};
    u.narrow = g.type == 3 || g.type == 13 || g.type == 21 || g.type == 24;
    u.weighted = g.type == 13 || g.type == 24 || g.type == 25;
    u.e1 = g.e1;
    u.e2 = g.e2;
    u.run = (int)t.runs.size();
    u.shape = (int)t.shapes.size();
    u.cell = cells;
    u.group = gi;
    u.rc2 = g.rc2;
    u.a2q = 0.25 * g.a2;
    u.qf = -0.5 * g.a2;
    return u;
}

// Cuts angular group gi into units; false (with the reason) if the two-pass
// path does not serve it.
bool addGroup(SFParams const& P, PairTables& t, int fcBeg, int radBeg, int gi,
              int slots, int& cells)
{
    DevGroup const& g = P.groups[gi];
    DevMember const* M = P.members + g.mbeg;
    bool const compact = g.type >= 20;
    PairUnit const proto = unitOf(g, t, gi, cells);
    std::vector<int> runs, shapes;   // representatives (member indices)
    std::vector<std::pair<int, int>> at(g.mcnt);
    bool ladder = !compact;
    for (int m = 0; m < g.mcnt; ++m)
    {
        std::size_t a = 0, s = 0;
        while (a < runs.size() && !sameRun(M[runs[a]], M[m], compact)) ++a;
        if (a == runs.size()) runs.push_back(m);
        while (s < shapes.size() && !sameShape(M[shapes[s]], M[m], compact))
            ++s;
        if (s == shapes.size()) shapes.push_back(m);
        for (int o = 0; o < m; ++o)
            if (at[o] == std::make_pair((int)a, (int)s))
            {
                t.why = "a symmetry function is listed twice";
                return false;
            }
        at[m] = {(int)a, (int)s};
        if (compact) continue;
        if (M[m].lambda == 0.0 || M[m].zeta == 0.0)
        {
            t.why = "an angular function with lambda or zeta 0";
            return false;
        }
        if (!exponentFits(M[m].eta, M[m].rs, 0.5 * t.p.farAway, false))
        {
            t.why = "a negative or very large eta";
            return false;
        }
        if (M[m].rs < 0.0)
        {
            t.why = "a negative shift rs";
            return false;
        }
        ladder = ladder && M[m].rs == 0.0 && M[m].useIntPow
              && M[m].zetaInt >= 1 && std::fabs(M[m].lambda) == 1.0;
    }
    if (compact && proto.narrow)
        // The reference reuses f(r_jk) of a previous member with the same
        // radial range even if its core function differs; such groups stay
        // on the path that reproduces the reuse.
        for (std::size_t a = 0; a < runs.size(); ++a)
            for (std::size_t b = 0; b < a; ++b)
                if (M[runs[a]].eta == M[runs[b]].eta
                    && M[runs[a]].rs == M[runs[b]].rs)
                {
                    t.why = "narrow compact functions of one radial range "
                            "with different cores";
                    return false;
                }
    int fcSlot = 0;
    if (!compact)
    {
        fcSlot = fcSlotOf(P, t, fcBeg, gi, proto.weighted);
        if (fcSlot < 0)
        {
            t.why = "too many cutoff radii";
            return false;
        }
    }
    auto addRun = [&](PairUnit const& u, DevMember const& m) {
        PairRun r{};
        r.eta = m.eta;
        r.rs = m.rs;
        r.center = m.eta * kMinusLog2E;
        if (compact)
        {
            r.center = m.factorDeriv;
            r.scale = m.zetaLambda;
            r.core = m.zetaInt;
            r.asym = m.useIntPow;
            r.slot = radSlotOf(t, radBeg, m, u.weighted);
            if (r.slot < 0)
            {
                t.why = "too many radial window functions";
                return false;
            }
        }
        t.runs.push_back(r);
        return true;
    };
    if (ladder)
    {
        std::vector<int> zs;
        for (int s : shapes) zs.push_back(M[s].zetaInt);
        std::sort(zs.begin(), zs.end());
        zs.erase(std::unique(zs.begin(), zs.end()), zs.end());
        bool pow2 = true;
        for (int z : zs) pow2 = pow2 && (z & (z - 1)) == 0 && z <= 16;
        // As few units as possible: the geometry and the cutoff of a triplet
        // cost more than the empty cells of runs with other zeta.
        std::vector<std::vector<int>> parts;
        std::size_t const most = pow2 ? kPairRuns : kPairGenRuns;
        for (std::size_t a = 0; a < runs.size(); ++a)
        {
            if (a % most == 0) parts.emplace_back();
            parts.back().push_back((int)a);
        }
        std::size_t const step = pow2 ? zs.size() : (std::size_t)kPairLadder;
        for (auto const& part : parts)
            for (std::size_t z0 = 0; z0 < zs.size(); z0 += step)
            {
                PairUnit u = unitOf(g, t, gi, cells);
                u.kind = pow2 ? PK_POW2 : PK_LADDER;
                u.fcSlot = fcSlot;
                u.nr = (int)part.size();
                // PK_POW2 units hold every slot up to the potential's
                // largest.
                u.ns = pow2 ? slots
                            : (int)std::min(step, zs.size() - z0);
                bool any = false, fits = true;
                std::size_t const base = t.cells.size();
                t.cells.resize(base + 2 * u.nr * u.ns, PairCell{-1, 0.0});
                for (int z = 0; z < u.ns && !pow2; ++z)
                {
                    u.zeta[z] = zs[z0 + z];
                    fits = fits && ladderSteps(z ? zs[z0 + z - 1] : 1,
                                               zs[z0 + z], u.prog[z]);
                }
                if (!fits)
                {
                    t.why = "a large zeta";
                    return false;
                }
                for (int m = 0; m < g.mcnt; ++m)
                {
                    int a = 0;
                    while (a < u.nr && part[a] != at[m].first) ++a;
                    if (a == u.nr) continue;
                    for (int z = 0; z < u.ns; ++z)
                        if (M[m].zetaInt == (pow2 ? 1 << z : zs[z0 + z]))
                        {
                            t.cells[base + 2 * (z * u.nr + a)
                                    + (M[m].lambda > 0.0 ? 1 : 0)] =
                                PairCell{M[m].sf, M[m].factorNorm};
                            u.mask |= 1u << z;
                            any = true;
                        }
                }
                if (!any)
                {
                    t.cells.resize(base);
                    continue;
                }
                for (int a : part)
                    if (!addRun(u, M[runs[a]])) return false;
                cells += 2 * u.nr * u.ns;
                t.p.kinds |= 1 << u.kind;
                t.units.push_back(u);
            }
        return true;
    }
    int const maxR = compact ? kPairCompRuns : kPairGenRuns;
    int const maxS = compact ? kPairCompShapes : kPairGenShapes;
    for (std::size_t a0 = 0; a0 < runs.size(); a0 += maxR)
        for (std::size_t s0 = 0; s0 < shapes.size(); s0 += maxS)
        {
            PairUnit u = unitOf(g, t, gi, cells);
            u.kind = compact ? PK_COMPACT : PK_GENERAL;
            u.fcSlot = fcSlot;
            u.nr = (int)std::min<std::size_t>(maxR, runs.size() - a0);
            u.ns = (int)std::min<std::size_t>(maxS, shapes.size() - s0);
            std::size_t const base = t.cells.size();
            t.cells.resize(base + (std::size_t)u.nr * maxS, PairCell{-1, 0.0});
            bool any = false;
            for (int m = 0; m < g.mcnt; ++m)
            {
                int const a = at[m].first - (int)a0, s = at[m].second - (int)s0;
                if (a < 0 || a >= u.nr || s < 0 || s >= u.ns) continue;
                t.cells[base + (std::size_t)a * maxS + s] =
                    PairCell{M[m].sf, M[m].factorNorm};
                any = true;
            }
            if (!any)
            {
                t.cells.resize(base);
                continue;
            }
            for (int a = 0; a < u.nr; ++a)
            {
                DevMember const& m = M[runs[a0 + a]];
                if (!addRun(u, m)) return false;
                if (!compact && m.rs > 0.0) u.hasRs = 1;
            }
            for (int s = 0; s < u.ns; ++s)
            {
                DevMember const& m = M[shapes[s0 + s]];
                PairShape h{};
                h.lambda = m.lambda;
                if (compact)
                {
                    h.zl = m.zeta;
                    h.center = m.aCenter;
                    h.scale = m.aScale;
                    h.zi = m.zetaInt;
                }
                else
                {
                    h.zl = m.zetaLambda;
                    h.zeta = m.zeta;
                    h.zi = m.zetaInt - 1;
                    h.useInt = m.useIntPow;
                }
                t.shapes.push_back(h);
                if (compact)
                    u.core = s == 0 || u.core == h.zi ? h.zi : 0;
            }
            cells += u.nr * maxS;
            t.p.kinds |= 1 << u.kind;
            t.units.push_back(u);
        }
    return true;
}

} // namespace

void buildPairTables(SFParams const& P, PairTables& t)
{
    t = PairTables{};
    PairParams& p = t.p;
    p.numElements = P.numElements;
    p.slots = 3;
    double rcMax = 0.0;
    for (int g = 0; g < P.numGroups; ++g)
    {
        DevGroup const& d = P.groups[g];
        rcMax = std::max(rcMax, d.rc);
        if (d.type == 12 || d.type == 13 || d.type >= 23) p.anyWeighted = 1;
        if (isRadial(d.type) || d.type >= 20) continue;
        for (int m = 0; m < d.mcnt; ++m)
        {
            int const z = P.members[d.mbeg + m].zetaInt;
            if (z > 4 && (z & (z - 1)) == 0 && z <= 16) p.slots = 5;
        }
    }
    p.farAway = 2.0 * rcMax;
    for (int e = 0; e < P.numElements; ++e)
    {
        int const fcBeg = (int)t.fcs.size(), radBeg = (int)t.rads.size();
        int const cellBeg = (int)t.cells.size();
        p.unitBeg[e] = (int)t.units.size();
        p.radialBeg[e] = (int)t.radials.size();
        p.cellBeg[e] = cellBeg;
        p.fcBeg[e] = fcBeg;
        p.radBeg[e] = radBeg;
        p.runBeg[e] = (int)t.runs.size();
        p.shapeBeg[e] = (int)t.shapes.size();
        int cells = 0;
        for (int g = P.groupBeg[e]; g < P.groupBeg[e + 1]; ++g)
        {
            if (isRadial(P.groups[g].type)) continue;
            if (!addGroup(P, t, fcBeg, radBeg, g, p.slots, cells)) return;
            int const type = P.groups[g].type;
            if (type >= 20) p.sorted[e] = 1;
            if (type == 3 || type == 13 || type == 21 || type == 24)
            {
                p.narrow[e] = 1;
                p.narrowRc2[e] = std::max(p.narrowRc2[e], P.groups[g].rc2);
            }
        }
        for (int g = P.groupBeg[e]; g < P.groupBeg[e + 1]; ++g)
        {
            DevGroup const& d = P.groups[g];
            if (!isRadial(d.type)) continue;
            // Radial groups share the staged cutoff values where there is
            // room for their radius (-1: formed where they are needed).
            int const slot = d.type >= 20 ? -1
                : fcSlotOf(P, t, fcBeg, g, d.type == 12 ? 1 : 0);
            for (int m = 0; m < d.mcnt; ++m)
            {
                DevMember const& mm = P.members[d.mbeg + m];
                PairRadial r{};
                r.compact = d.type >= 20;
                r.weighted = d.type == 12 || d.type == 23;
                r.e1 = d.e1;
                r.fcSlot = slot;
                r.group = g;
                r.cell = cells++;
                r.eta = mm.eta;
                r.rs = mm.rs;
                r.center = mm.eta * kMinusLog2E;
                if (r.compact)
                {
                    r.core = mm.zetaInt;
                    r.asym = mm.useIntPow;
                    r.center = mm.factorDeriv;
                    r.scale = mm.zetaLambda;
                }
                else if (!exponentFits(mm.eta, mm.rs, rcMax, true))
                {
                    t.why = "a negative or very large eta";
                    return;
                }
                t.radials.push_back(r);
                t.cells.push_back(PairCell{mm.sf, mm.factorNorm});
            }
        }
        for (std::size_t k = p.unitBeg[e]; k < t.units.size(); ++k)
            t.units[k].exactMask = t.units[k].rc2 == p.narrowRc2[e] ? 1 : 0;
        p.maxCells = std::max(p.maxCells, cells);
        p.maxFc = std::max(p.maxFc, (int)t.fcs.size() - fcBeg);
        p.maxRad = std::max(p.maxRad, (int)t.rads.size() - radBeg);
    }
    for (int e = P.numElements; e <= kMaxElem; ++e)
    {
        p.unitBeg[e] = (int)t.units.size();
        p.radialBeg[e] = (int)t.radials.size();
        p.cellBeg[e] = (int)t.cells.size();
        p.fcBeg[e] = (int)t.fcs.size();
        p.radBeg[e] = (int)t.rads.size();
        p.runBeg[e] = (int)t.runs.size();
        p.shapeBeg[e] = (int)t.shapes.size();
    }
    t.ok = true;
}

} // namespace n2p2b
