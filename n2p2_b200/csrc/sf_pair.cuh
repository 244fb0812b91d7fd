// Symmetry functions in two passes without dG/dr (kernel templates).
//
// The force on a neighbor j of atom i is the chain rule
//   F_ij = sum_m dE/dG_m dG_m/d(r_i - r_j),
// a sum over members m and partners k.  Members outermost, as the reference
// does it, needs five sums per (j, m) and a stored vector per (j, m).  Here
// dE/dG is known first (values pass, then the networks) and the sum over the
// members is formed inside each triplet: with runs a (eta, rs) and shapes s
// (zeta, lambda) and c_as = dE/dG_as 2^(1-zeta) x scaling factor,
//   Phi = f_j f_k f_jk sum_a v_a sum_s c_as P_s(cos),  v_a = exp(-eta_a S),
// so that T = sum_a v_a B_a, D = sum_a eta_a v_a B_a, H = sum_a v_a B'_a with
// B_a = sum_s c_as P_s, B'_a = sum_s c_as P'_s give the triplet's force on j
// along dr_ij and dr_ik: four sums per owner j whatever the number of
// members.  Compact functions have the same form (run = radial window
// functions, shape = window function of theta).
//
// Values pass: CTA per atom; each unordered triplet once.  Warps walk the
// rows (j, k > j) of a unit, test r_jk with the lane on k and push the valid
// pairs into a 64-entry queue per warp, from which full warps of triplets
// are evaluated (97 % of the lanes busy); the unit's sums stay in registers
// (lane sums, then one fixed-order reduction per unit).
//
// Forces pass: CTA per atom; an item is eight owners j of one element on
// four lanes each, owners ordered by their partner counts so that the
// owners of an item have similar trip counts.  The item's lanes build the
// owners' partner lists from the validity mask, walk the units with the
// unit's parameters the same for the whole warp, and add the four slices
// at the end.  Each pair term has one writer: no atomics, fixed order.
#pragma once

#include "sf_impl.cuh"
#include "sf_pair.h"

namespace n2p2b
{
namespace sfp2
{

using namespace sfk;

constexpr int kT = 128;               // threads
constexpr int kW = kT / 32;           // warps
constexpr int kSl = 4;                // slices (lanes) per owner
constexpr int kOw = 32 / kSl;         // owners per item

constexpr double kLn64 = 0x1.62e42fefa39efp-7;     // ln2 / 64

template <typename R> struct V2;
template <> struct V2<double> { using T = double2; };
template <> struct V2<float>  { using T = float2; };

// Staged neighbor: position, 1/r, the first cutoff slot's f_c (x Z) and r^2
// in one record, so that a lane's loads of a partner share one address.  The
// record behind the last neighbor is a partner far away with f_c = 0, which
// idle lanes take.
template <typename R>
struct alignas(2 * sizeof(R)) Rec
{
    R x, y, z, ir, fc, r2;
};

template <typename R>
struct Staged
{
    Rec<R>*       rec;        // [cs]
    R*            fc;         // [fc slot - 1][cs]: f_c (x Z)
    R*            dfc;        // [fc slot][cs]: f_c'/r (x Z)
    R*            rad;        // [rad slot][2][cs]: window function, its
                              // derivative / r (x Z)
    double const* tab;        // exponential table
    int           cs;         // cap + 1
};

// Series coefficients of the FP64 kernels in the constant bank: an FMA takes
// one operand from there, while 64-bit literals cost two moves each in a loop
// that has no registers left to keep them.
struct PairConst
{
    double ex[5];      // 2^(f/64) - 1: coefficients of f^5 .. f
    double ch[10];     // cos(sqrt w): n = 9 .. 0 terms (start n = 10)
    double sh[10];     // sin(sqrt w) / sqrt w
    double ch10, sh10;
    double invL, shift;
};
__constant__ PairConst kPC = {
    {kLn64 * kLn64 * kLn64 * kLn64 * kLn64 / 120.0,
     kLn64 * kLn64 * kLn64 * kLn64 / 24.0, kLn64 * kLn64 * kLn64 / 6.0,
     kLn64 * kLn64 / 2.0, kLn64},
    {-InvFact<18>::value, InvFact<16>::value, -InvFact<14>::value,
     InvFact<12>::value, -InvFact<10>::value, InvFact<8>::value,
     -InvFact<6>::value, InvFact<4>::value, -InvFact<2>::value, 1.0},
    {-InvFact<19>::value, InvFact<17>::value, -InvFact<15>::value,
     InvFact<13>::value, -InvFact<11>::value, InvFact<9>::value,
     -InvFact<7>::value, InvFact<5>::value, -InvFact<3>::value, 1.0},
    InvFact<20>::value, InvFact<21>::value, -0x1.71547652b82fep+6, 0x1.8p52};

// Constants of one run: eta in the exponential's unit.
//   FP64: exp(-eta s) = 2^(k/64) 2^(f/64), k = rint(y), f = y - k with
//   y = -eta s 64/ln2; f is formed by one fma from s (no product rounding),
//   2^(f/64) - 1 by its Taylor polynomial of degree 5 in f (|f| <= 1/2:
//   truncation below 4e-17), 2^(j/64) from the table.  The error is that of
//   y's factor, |eta s| 2^-53, and 1 ulp, as for exp of the rounded
//   product.  Results below 2^-1020 stay near 2^-1020.
__device__ __forceinline__ double expScale(double eta)
{
    return eta * -0x1.71547652b82fep+6;
}
__device__ __forceinline__ double expScaled(double e2, double s,
                                            double const* tab)
{
    double const t = fma(s, e2, kPC.shift);
    int const k = max(__double2loint(t), -64 * 1020);
    double const f = fma(s, e2, kPC.shift - t);
    double p = fma(f, kPC.ex[0], kPC.ex[1]);
#pragma unroll
    for (int n = 2; n < 5; ++n) p = fma(p, f, kPC.ex[n]);
    double const q = p * f;
    double const tj = tab[k & (kExpTableSize - 1)];
    double const tm = __hiloint2double(
        __double2hiint(tj) + ((k >> 6) << 20), __double2loint(tj));
    return fma(tm, q, tm);
}
__device__ __forceinline__ float expScale(float eta)
{
    return eta * -1.44269504f;
}
__device__ __forceinline__ float expScaled(float e2, float s, double const*)
{
    float v;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(v) : "f"(s * e2));
    return v;
}
// eta from the scaled constant.
template <typename R>
__device__ __forceinline__ R expUnscale()
{
    return sizeof(R) == 8 ? R(-0x1.62e42fefa39efp-7) : R(-0.693147181f);
}

template <typename R, int N, int K>
struct SeriesR
{
    __device__ static __forceinline__ R run(R v, R acc)
    {
        constexpr double c = ((N & 1) ? -1.0 : 1.0) * InvFact<2 * N + K>::value;
        return SeriesR<R, N - 1, K>::run(v, fma(acc, v, R(c)));
    }
};
template <typename R, int K>
struct SeriesR<R, -1, K>
{
    __device__ static __forceinline__ R run(R, R acc) { return acc; }
};

// cos and sin(x)/x of the half angle from w = (a r / 2)^2 <= pi^2 / 4: FP64
// as halfAngleCosSinc; FP32 with the terms up to n = 6 (first omitted terms
// 6.5e-9 and 4.3e-10 relative to 1).
__device__ __forceinline__ double halfAngleCos(double w)
{
    double c = kPC.ch10;
#pragma unroll
    for (int n = 0; n < 10; ++n) c = fma(c, w, kPC.ch[n]);
    return c;
}
__device__ __forceinline__ void halfAngle(double w, double& ch, double& sh)
{
    ch = halfAngleCos(w);
    sh = kPC.sh10;
#pragma unroll
    for (int n = 0; n < 10; ++n) sh = fma(sh, w, kPC.sh[n]);
}
__device__ __forceinline__ void halfAngle(float w, float& ch, float& sh)
{
    ch = SeriesR<float, 5, 0>::run(w, (float)InvFact<12>::value);
    sh = SeriesR<float, 5, 1>::run(w, (float)InvFact<13>::value);
}
__device__ __forceinline__ float halfAngleCos(float w)
{
    return SeriesR<float, 5, 0>::run(w, (float)InvFact<12>::value);
}

// f_c(r_jk) and, with DERIV, q = f_c'(r_jk) / r_jk.  CT = 1 is the cosine
// cutoff without inner radius: power series in r_jk^2 (needs no r_jk unless
// `needR`), which go on beyond the cutoff: where the validity mask is not the
// unit's own, `weight` becomes 0 there.
template <typename R, int CT, bool DERIV>
__device__ __forceinline__ void cutoffJk(SFParams const& P, PairUnit const& u,
                                         R a2q, R qf, R rc2, bool exact,
                                         R r2, bool needR, R& fc, R& q, R& rjk,
                                         R& irjk, R& weight)
{
    rjk = irjk = R(0);
    if (CT != 1 || needR)
    {
        irjk = mrsqrt(r2);
        rjk = r2 * irjk;
    }
    if (CT == 1)
    {
        R const w = a2q * r2;
        if (DERIV)
        {
            R ch, sh;
            halfAngle(w, ch, sh);
            fc = ch * ch;
            q = qf * (sh * ch);
        }
        else
        {
            R const ch = halfAngleCos(w);
            fc = ch * ch;
            q = R(0);
        }
        if (sizeof(R) == 8 || !exact) weight = r2 < rc2 ? weight : R(0);
    }
    else
    {
        R d;
        cutoffFdf<R, CT>(P, P.dGroups[u.group], rjk, fc, d);
        q = d * irjk;
    }
}

// plambda^(zeta - 1) with the reference's zero for plambda <= 0; the
// exponent is the same for the whole warp.
template <typename R>
__device__ __forceinline__ R shapePower(R pl, PairShape const& h)
{
    R const v = h.useInt ? powInt(pl, h.zi)
                         : mpow(pl > R(0) ? pl : R(1), R(h.zeta) - R(1));
    return pl > R(0) ? v : R(0);
}

// The ladder of a unit: (1 -+ cos)^zeta and ^(zeta - 1) for its values of
// zeta one after another.
template <typename R>
struct Ladder
{
    R pm, pp;      // 1 - cos, 1 + cos
    R Pm, Pp;      // their zeta-th powers
    R mm, mp;      // and (zeta - 1)-th
    __device__ __forceinline__ explicit Ladder(R c)
    {
        Pm = pm = R(1) - c;
        Pp = pp = R(1) + c;
        mm = mp = R(1);
    }
    __device__ __forceinline__ void advance(unsigned prog)
    {
        int n = (int)(prog & 0xffu);
        if (n == 0) return;
        if (prog >> 31)
        {
            Pm = pm;
            Pp = pp;
            mm = mp = R(1);
        }
        unsigned ops = prog >> 8;
#pragma unroll 1
        do
        {
            if (ops & 1u)
            {
                mm = Pm;
                mp = Pp;
                Pm *= pm;
                Pp *= pp;
            }
            else
            {
                mm *= Pm;
                mp *= Pp;
                Pm *= Pm;
                Pp *= Pp;
            }
            ops >>= 1;
        }
        while (--n);
    }
};

// The warps that work on one atom together: all of the block (WPA = kW; few
// atoms, or many neighbors) or each on its own (WPA = 1: no block barriers,
// fewer half-empty batches, one final sum per unit).
template <int WPA>
struct Team
{
    static constexpr int kTeams = kW / WPA, kThreads = 32 * WPA;
    int team, tid, warp, lane;    // team of the block; place inside the team
    __device__ __forceinline__ Team()
    {
        lane = threadIdx.x & 31;
        team = (threadIdx.x >> 5) / WPA;
        warp = (threadIdx.x >> 5) % WPA;
        tid = threadIdx.x % kThreads;
    }
    __device__ __forceinline__ static void sync()
    {
        if (WPA == 1) __syncwarp();
        else __syncthreads();
    }
};

// Header of an atom.
struct Head
{
    int  ec, cnt;
    int  eb[kMaxElem + 1];
    long beg;
};

// Header of atom i, formed by one warp of the team.
__device__ __forceinline__ void readHead(PairParams const& T,
                                         PairLaunch const& L, int i, int lane,
                                         Head* h)
{
    int c = 0;
    if (lane < T.numElements)
        c = L.nbrCountElem[(long)i * T.numElements + lane];
    int const ec = L.elem[i], b0 = L.nbrOff[i], b1 = L.nbrOff[i + 1];
#pragma unroll
    for (int d = 1; d < 8; d <<= 1)
    {
        int const v = __shfl_up_sync(kFull, c, d);
        if (lane >= d) c += v;
    }
    if (lane < kMaxElem) h->eb[lane + 1] = c;
    if (lane == 0)
    {
        h->eb[0] = 0;
        h->ec = ec;
        h->beg = b0;
        h->cnt = b1 - b0;
    }
}

// Validity masks: partners whose distances from the atom and from t are
// inside the element's largest narrow cutoff.  FP64 kernels test 32-bit
// positions against a radius 2e-6 larger (their squared distances are off by
// at most 1e-6 rc^2), and the cutoff function decides; FP32 kernels test
// theirs.
__device__ __forceinline__ float maskRc2(PairParams const& T, int ec, bool fp64)
{
    return (float)(T.narrowRc2[ec] * (fp64 ? 1.0 + 4e-6 : 1.0));
}

// Word q of the row that the lane owns: the lane keeps its row's position and
// the partners' are broadcast, so a test costs one load, six operations, the
// comparison and a predicated OR, and no vote.  pos is readable up to the
// word's end.
__device__ __forceinline__ unsigned maskWord(float4 const* pos, int t, int q,
                                             int cnt, float rc2)
{
    float4 const a = pos[t];
    float4 const* p = pos + (q << 5);
    unsigned m = 0u;
#pragma unroll
    for (int k = 0; k < 32; ++k)
    {
        float4 const c = p[k];
        float const x = c.x - a.x, y = c.y - a.y, z = c.z - a.z;
        if (x * x + y * y + z * z < rc2) m |= 1u << k;
    }
    if (a.w != 0.0f) m = 0u;
    if (cnt - (q << 5) < 32) m &= (1u << (cnt & 31)) - 1u;
    return m;
}

template <typename R>
__device__ __forceinline__ R fcOf(Staged<R> const& S, int slot, int t)
{
    return slot == 0 ? S.rec[t].fc : S.fc[(slot - 1) * S.cs + t];
}

// Radial function of a member: value and derivative with respect to r,
// unscaled, from the cutoff's value and derivative.
template <typename R>
__device__ __forceinline__ void radialFdf(SFParams const& P,
                                          PairRadial const& m, R r, R fc,
                                          R dfc, double const* tab, R& v,
                                          R& dv)
{
    v = dv = R(0);
    if (m.compact)
    {
        if (r > R(m.eta) && r < R(m.rs))
            compactFdf<R>(m.core, m.asym != 0, R(m.center), R(m.scale), r,
                          R(P.E), v, dv);
        return;
    }
    R const d = r - R(m.rs), eta = R(m.eta);
    R const e = expScaled(expScale(eta), d * d, tab);
    v = e * fc;
    dv = e * (dfc - R(2) * eta * d * fc);
}

// Stages the neighbors of an atom; in the forces pass also the radial
// functions' part of dE_i/dr along dr_ij (arad), in the values pass the
// distances for them.
template <typename R, int CT, int WPA, bool DERIV>
__device__ __forceinline__ void stageAtom(SFParams const& P,
                                          PairParams const& T,
                                          PairLaunch const& L, Head const& h,
                                          Team<WPA> const& tm, float4* pos,
                                          R* dist, R* arad, R const* C,
                                          PairRadial const* radials,
                                          Staged<R> const& S)
{
    int const cs = S.cs, cnt = h.cnt, ec = h.ec;
    int const nf = T.fcBeg[ec + 1] - T.fcBeg[ec];
    int const nrad = T.radBeg[ec + 1] - T.radBeg[ec];
    for (int t = tm.tid; t <= cnt; t += Team<WPA>::kThreads)
    {
        if (t == cnt)
        {
            R const far = R(T.farAway);
            S.rec[t] = Rec<R>{far, R(0), R(0), R(1) / far, R(0), far * far};
            for (int f = 1; f < nf; ++f) S.fc[(f - 1) * cs + t] = R(0);
            for (int f = 0; f < 2 * nrad; ++f) S.rad[f * cs + t] = R(0);
            break;
        }
        double const d = L.dd[h.beg + t];
        R const r = R(d), ir = R(1.0 / d);
        R const x = R(L.dx[h.beg + t]), y = R(L.dy[h.beg + t]),
                z = R(L.dz[h.beg + t]);
        R const r2 = x * x + y * y + z * z;
        // Neighbors beyond the narrow cutoff are nobody's partners.
        pos[t] = (float)r2 < maskRc2(T, ec, sizeof(R) == 8)
            ? make_float4((float)x, (float)y, (float)z, 0.0f)
            : make_float4(1e18f, 0.0f, 0.0f, 1.0f);
        R Z = R(1), f0 = R(0);
        int el = 0;
        if (DERIV || T.anyWeighted)
        {
            while (t >= h.eb[el + 1]) ++el;
            Z = R(P.atomicNumber[el]);
        }
        R df0 = R(0);
        for (int f = 0; f < nf; ++f)
        {
            PairFc const pf = T.fcs[T.fcBeg[ec] + f];
            R v, dv;
            cutoffFdf<R, CT>(P, P.dGroups[pf.group], r, v, dv);
            if (pf.weighted) { v *= Z; dv *= Z; }
            if (f == 0) { f0 = v; df0 = dv; }
            else S.fc[(f - 1) * cs + t] = v;
            if (DERIV) S.dfc[f * cs + t] = dv * ir;
        }
        S.rec[t] = Rec<R>{x, y, z, ir, f0, r2};
        if (!DERIV) dist[t] = r;
        for (int f = 0; f < nrad; ++f)
        {
            PairRad const w = T.rads[T.radBeg[ec] + f];
            R v = R(0), dv = R(0);
            if (r > R(w.rl) && r < R(w.rc))
                compactFdf<R>(w.core, w.asym != 0, R(w.center), R(w.scale), r,
                              R(P.E), v, dv);
            if (w.weighted) { v *= Z; dv *= Z; }
            S.rad[(2 * f) * cs + t] = v;
            S.rad[(2 * f + 1) * cs + t] = dv * ir;
        }
        if (!DERIV) continue;
        R al = R(0), fc = R(0), dfc = R(0), ZZ = R(1);
        int last = -1;
        for (int q = T.radialBeg[ec]; q < T.radialBeg[ec + 1]; ++q)
        {
            PairRadial const& pr = radials[q];
            if (!pr.weighted && pr.e1 != el) continue;
            if (pr.group != last)
            {
                last = pr.group;
                ZZ = R(1);
                if (pr.fcSlot == 0)
                {
                    fc = f0;
                    dfc = df0;
                }
                else if (pr.fcSlot > 0)
                {
                    fc = S.fc[(pr.fcSlot - 1) * cs + t];
                    dfc = S.dfc[pr.fcSlot * cs + t] * r;
                }
                else
                {
                    if (!pr.compact)
                        cutoffFdf<R, CT>(P, P.dGroups[last], r, fc, dfc);
                    if (pr.weighted) ZZ = Z;
                }
            }
            R v, dv;
            radialFdf<R>(P, pr, r, fc, dfc, S.tab, v, dv);
            al += (C[pr.cell] * ZZ) * dv;
        }
        arad[t] = al * ir;
    }
}

// Angular parts phi_s of a general unit and, with DERIV, psi_s = d phi_s /
// d cos.
template <typename R, bool DERIV>
__device__ __forceinline__ void genShapes(int ns, PairShape const* sh, R c,
                                          R* phi, R* psi)
{
#pragma unroll
    for (int s = 0; s < kPairGenShapes; ++s)
    {
        phi[s] = R(0);
        if (DERIV) psi[s] = R(0);
        if (s < ns)
        {
            PairShape const& h = sh[s];
            R const pl = R(1) + R(h.lambda) * c;
            R const pm = shapePower(pl, h);
            phi[s] = pm * pl;
            if (DERIV) psi[s] = pm * R(h.zl);
        }
    }
}

// Window functions of theta of a compact unit, with DERIV their derivatives.
template <typename R, bool DERIV>
__device__ __forceinline__ void compShapes(SFParams const& P, int ns,
                                           PairShape const* sh, R theta,
                                           R* phi, R* psi)
{
#pragma unroll
    for (int s = 0; s < kPairCompShapes; ++s)
    {
        phi[s] = R(0);
        if (DERIV) psi[s] = R(0);
        if (s < ns)
        {
            PairShape const& h = sh[s];
            if (theta > R(h.lambda) && theta < R(h.zl))
            {
                R f, d;
                compactFdf<R>(h.zi, false, R(h.center), R(h.scale), theta,
                              R(P.E), f, d);
                phi[s] = f;
                if (DERIV) psi[s] = d;
            }
        }
    }
}

// Window functions of r_jk (narrow compact units).
template <typename R>
__device__ __forceinline__ void radJk(SFParams const& P, PairRun const& w,
                                      R rjk, R& f, R& d)
{
    f = d = R(0);
    if (rjk > R(w.eta) && rjk < R(w.rs))
        compactFdf<R>(w.core, w.asym != 0, R(w.center), R(w.scale), rjk,
                      R(P.E), f, d);
}

// Views of a team's region and of the block's exponential table.
template <typename R>
__device__ __forceinline__ Staged<R> views(unsigned char* sm,
                                           unsigned char* mine,
                                           PairLaunch const& L)
{
    Staged<R> S;
    S.rec = reinterpret_cast<Rec<R>*>(mine + L.oRec);
    S.fc = reinterpret_cast<R*>(mine + L.oFc);
    S.dfc = reinterpret_cast<R*>(mine + L.oDfc);
    S.rad = reinterpret_cast<R*>(mine + L.oRad);
    S.tab = reinterpret_cast<double const*>(sm + L.oTab);
    S.cs = 0;
    return S;
}

// Tables the inner loops read: in shared memory where they fit.
struct UnitTables
{
    PairUnit const*   u;
    PairRun const*    r;
    PairShape const*  s;
    PairRadial const* q;
    PairCell const*   c;
};

__device__ __forceinline__ UnitTables stageTables(PairParams const& T,
                                                  PairLaunch const& L,
                                                  unsigned char* sm)
{
    UnitTables t{T.units, T.runs, T.shapesTab, T.radials, T.cells};
    int const ne = T.numElements;
    unsigned char* at = sm + L.oTables;
    auto copy = [&](auto const*& p, int count) {
        int const bytes = (int)sizeof(*p) * count;
        for (int k = threadIdx.x; k < bytes / 8; k += kT)
            reinterpret_cast<double*>(at)[k] =
                reinterpret_cast<double const*>(p)[k];
        p = reinterpret_cast<decltype(p + 0)>(at);
        at += bytes;
    };
    if (L.tables & 1)
    {
        copy(t.u, T.unitBeg[ne]);
        copy(t.r, T.runBeg[ne]);
        copy(t.s, T.shapeBeg[ne]);
    }
    if (L.tables & 2)
    {
        copy(t.q, T.radialBeg[ne]);
        copy(t.c, T.cellBeg[ne]);
    }
    return t;
}

template <typename R>
__device__ __forceinline__ void stageExpTable(unsigned char* sm,
                                              PairLaunch const& L)
{
    if (sizeof(R) == 8)
    {
        double* tab = reinterpret_cast<double*>(sm + L.oTab);
        for (int j = threadIdx.x; j < kExpTableSize; j += kT)
            tab[j] = kExp2Table[j];
    }
}

// Which unit kinds a kernel holds.
constexpr int kHasPow2 = 1 << PK_POW2, kHasLadder = 1 << PK_LADDER,
              kHasGeneral = 1 << PK_GENERAL, kHasCompact = 1 << PK_COMPACT;

// ---------------------------------------------------------------------------
// Values pass.
// ---------------------------------------------------------------------------

// What a warp needs to walk a unit's pairs.
template <typename R>
struct Walk
{
    Staged<R> W;
    unsigned const* bits; // [t][words], k > t
    unsigned* pairs;      // the warp's pair list [pairCap]
    R*        red;        // 16 x 33 lane sums
    R*        Gp;         // the warp's sums [maxSF]
    PairCell const* cells;
    int       words, pairCap, b1, x1, b2, x2, same, lane, warp, warps;
};

// Word q of row t, restricted to partners in [lo, hi).
template <bool NARROW>
__device__ __forceinline__ unsigned rowWord(unsigned const* row, int q, int lo,
                                            int hi)
{
    unsigned m = NARROW ? row[q] : kFull;
    int const b = q << 5;
    if (b < lo) m &= kFull << (lo & 31);
    if (hi - b < 32) m &= (1u << (hi & 31)) - 1u;
    return m;
}

// The unit's pairs (t, k), k > t, to f(t, k) for 32 pairs at a time.  The
// team's warps take the rows in turn; a warp's lanes count the set bits of a
// row each, and write their pairs behind one another into the warp's list (rows that
// do not fit any more wait for the next round).  Idle lanes of a round's
// last batch get the far record.
template <typename R, bool NARROW, typename F>
__device__ __forceinline__ void walkPairs(Walk<R> const& w, F&& f)
{
    int const lane = w.lane, none = w.W.cs - 1;
#pragma unroll 1
    for (int t0 = w.b1 + w.warp; t0 < w.x1; t0 += 32 * w.warps)
    {
        int const t = t0 + lane * w.warps;
        int const lo = w.same ? t + 1 : w.b2;
        int const q0 = lo >> 5, q1 = t < w.x1 ? (w.x2 + 31) >> 5 : 0;
        unsigned const* row = w.bits + t * w.words;
        int n = 0;
        if (lo < w.x2)
            for (int q = q0; q < q1; ++q)
                n += __popc(rowWord<NARROW>(row, q, lo, w.x2));
        int s = n;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1)
        {
            int const v = __shfl_up_sync(kFull, s, d);
            if (lane >= d) s += v;
        }
        int const total = __shfl_sync(kFull, s, 31);
#pragma unroll 1
        for (int done = 0; done < total;)
        {
            bool const mine = n > 0 && s - n >= done
                           && s <= done + w.pairCap;
            if (mine)
            {
                unsigned* out = w.pairs + (s - n - done);
                for (int q = q0; q < q1; ++q)
                {
                    unsigned m = rowWord<NARROW>(row, q, lo, w.x2);
                    unsigned const base = ((unsigned)t << 16)
                                        + (unsigned)((q << 5) - 1);
                    while (m)
                    {
                        *out++ = base + (unsigned)__ffs(m);
                        m &= m - 1;
                    }
                }
            }
            int const end = __reduce_max_sync(kFull, mine ? s : 0);
            int const np = end - done;
            done = end;
            __syncwarp();
#pragma unroll 1
            for (int b = lane; b < np + lane; b += 32)
            {
                unsigned const code = b < np ? w.pairs[b] : (unsigned)none;
                f((int)(code >> 16), (int)(code & 0xffffu));
            }
            __syncwarp();
        }
    }
}

// Adds the lanes' sums of N cells to the warp's values: sixteen cells at a
// time, lane (row, half) adds sixteen lanes of its cell, then its neighbor.
template <typename R, int N>
__device__ __forceinline__ void flushCells(Walk<R> const& w, R const (&acc)[N],
                                           int cell0, int cells)
{
#pragma unroll
    for (int c0 = 0; c0 < N; c0 += 16)
    {
        if (c0 < cells)
        {
#pragma unroll
            for (int c = 0; c < 16; ++c)
                if (c0 + c < N) w.red[c * 33 + w.lane] = acc[c0 + c];
            __syncwarp();
            int const row = w.lane >> 1;
            R v = R(0);
#pragma unroll
            for (int q = 0; q < 16; ++q)
                v += w.red[row * 33 + (w.lane & 1) * 16 + q];
            v += __shfl_xor_sync(kFull, v, 1);
            if ((w.lane & 1) == 0 && c0 + row < cells)
            {
                int const sf = w.cells[cell0 + c0 + row].sf;
                if (sf >= 0) w.Gp[sf] += v;
            }
            __syncwarp();
        }
    }
}

// acc += v x ((1 - cos)^zeta, (1 + cos)^zeta) of the slots zeta = 2^z that
// the unit has.
template <typename R, int CT, int NZ, int NR, int MASK, bool NARROW>
__device__ __forceinline__ void pow2Values(SFParams const& P,
                                           UnitTables const& tb,
                                           PairUnit const& u,
                                           Walk<R> const& w)
{
    R acc[NZ * NR * 2];
#pragma unroll
    for (int c = 0; c < NZ * NR * 2; ++c) acc[c] = R(0);
    R e2[NR];
#pragma unroll
    for (int a = 0; a < NR; ++a) e2[a] = expScale(R(tb.r[u.run + a].eta));
    R const a2q = R(u.a2q), rc2 = R(u.rc2);
    bool const exact = u.exactMask != 0;
    int const slot = u.fcSlot;
    unsigned const mask = MASK ? (unsigned)MASK : u.mask;
    walkPairs<R, NARROW>(w, [&](int tt, int kk) {
        Rec<R> const A = w.W.rec[tt], B = w.W.rec[kk];
        R const f1 = slot == 0 ? A.fc : w.W.fc[(slot - 1) * w.W.cs + tt];
        R const f2 = slot == 0 ? B.fc : w.W.fc[(slot - 1) * w.W.cs + kk];
        R const c = (A.x * B.x + A.y * B.y + A.z * B.z) * (A.ir * B.ir);
        R m = f1 * f2;
        R s = A.r2 + B.r2;
        if (NARROW)
        {
            R const x = A.x - B.x, y = A.y - B.y, z = A.z - B.z;
            R const s3 = x * x + y * y + z * z;
            R f3, q, r3, ir3;
            cutoffJk<R, CT, false>(P, u, a2q, R(0), rc2, exact, s3, false, f3,
                                   q, r3, ir3, m);
            m *= f3;
            s += s3;
        }
        R v[NR];
#pragma unroll
        for (int a = 0; a < NR; ++a) v[a] = m * expScaled(e2[a], s, w.W.tab);
        R Pm = R(1) - c, Pp = R(1) + c;
#pragma unroll
        for (int z = 0; z < NZ; ++z)
        {
            if ((mask >> z) & 1u)
            {
#pragma unroll
                for (int a = 0; a < NR; ++a)
                {
                    acc[(z * NR + a) * 2] += v[a] * Pm;
                    acc[(z * NR + a) * 2 + 1] += v[a] * Pp;
                }
            }
            if (z + 1 < NZ)
            {
                Pm *= Pm;
                Pp *= Pp;
            }
        }
    });
    flushCells<R, NZ * NR * 2>(w, acc, u.cell, 2 * NZ * NR);
}

template <typename R, int CT, int NR, bool NARROW>
__device__ __forceinline__ void ladderValues(SFParams const& P,
                                             UnitTables const& tb,
                                             PairUnit const& u,
                                             Walk<R> const& w)
{
    R acc[kPairLadder * NR * 2];
#pragma unroll
    for (int c = 0; c < kPairLadder * NR * 2; ++c) acc[c] = R(0);
    int const nr = u.nr;
    R e2[NR];
#pragma unroll
    for (int a = 0; a < NR; ++a)
        e2[a] = expScale(R(tb.r[u.run + min(a, nr - 1)].eta));
    R const a2q = R(u.a2q), rc2 = R(u.rc2);
    bool const exact = u.exactMask != 0;
    int const slot = u.fcSlot, ns = u.ns;
    unsigned prog[kPairLadder];
#pragma unroll
    for (int z = 0; z < kPairLadder; ++z) prog[z] = u.prog[z];
    walkPairs<R, NARROW>(w, [&](int tt, int kk) {
        Rec<R> const A = w.W.rec[tt], B = w.W.rec[kk];
        R const f1 = slot == 0 ? A.fc : w.W.fc[(slot - 1) * w.W.cs + tt];
        R const f2 = slot == 0 ? B.fc : w.W.fc[(slot - 1) * w.W.cs + kk];
        R const c = (A.x * B.x + A.y * B.y + A.z * B.z) * (A.ir * B.ir);
        R m = f1 * f2;
        R s = A.r2 + B.r2;
        if (NARROW)
        {
            R const x = A.x - B.x, y = A.y - B.y, z = A.z - B.z;
            R const s3 = x * x + y * y + z * z;
            R f3, q, r3, ir3;
            cutoffJk<R, CT, false>(P, u, a2q, R(0), rc2, exact, s3, false, f3,
                                   q, r3, ir3, m);
            m *= f3;
            s += s3;
        }
        R v[NR];
#pragma unroll
        for (int a = 0; a < NR; ++a)
            v[a] = a < nr ? m * expScaled(e2[a], s, w.W.tab) : R(0);
        Ladder<R> l(c);
#pragma unroll
        for (int z = 0; z < kPairLadder; ++z)
            if (z < ns)
            {
                l.advance(prog[z]);
#pragma unroll
                for (int a = 0; a < NR; ++a)
                {
                    acc[(z * NR + a) * 2] += v[a] * l.Pm;
                    acc[(z * NR + a) * 2 + 1] += v[a] * l.Pp;
                }
            }
    });
    // Cells of the runs that exist, one zeta at a time.
#pragma unroll
    for (int z = 0; z < kPairLadder; ++z)
        if (z < ns)
        {
            R one[NR * 2];
#pragma unroll
            for (int c = 0; c < NR * 2; ++c) one[c] = acc[z * NR * 2 + c];
            flushCells<R, NR * 2>(w, one, u.cell + 2 * z * nr, 2 * nr);
        }
}

template <typename R, int CT, bool NARROW>
__device__ __forceinline__ void generalValues(SFParams const& P,
                                              UnitTables const& tb,
                                              PairUnit const& u,
                                              Walk<R> const& w)
{
    constexpr int S = kPairGenShapes;
    R acc[kPairGenRuns * S];
#pragma unroll
    for (int c = 0; c < kPairGenRuns * S; ++c) acc[c] = R(0);
    R const a2q = R(u.a2q), rc2 = R(u.rc2);
    bool const exact = u.exactMask != 0;
    int const slot = u.fcSlot, ns = u.ns, nr = u.nr;
    bool const hasRs = u.hasRs != 0;
    PairRun const* const runs = tb.r + u.run;
    PairShape const* const sh = tb.s + u.shape;
    walkPairs<R, NARROW>(w, [&](int tt, int kk) {
        Rec<R> const A = w.W.rec[tt], B = w.W.rec[kk];
        R const f1 = slot == 0 ? A.fc : w.W.fc[(slot - 1) * w.W.cs + tt];
        R const f2 = slot == 0 ? B.fc : w.W.fc[(slot - 1) * w.W.cs + kk];
        R const c = (A.x * B.x + A.y * B.y + A.z * B.z) * (A.ir * B.ir);
        R m = f1 * f2;
        R s = A.r2 + B.r2, r3 = R(0), ir3 = R(0);
        if (NARROW)
        {
            R const x = A.x - B.x, y = A.y - B.y, z = A.z - B.z;
            R const s3 = x * x + y * y + z * z;
            R f3, q;
            cutoffJk<R, CT, false>(P, u, a2q, R(0), rc2, exact, s3, hasRs, f3,
                                   q, r3, ir3, m);
            m *= f3;
            s += s3;
        }
        R phi[S];
        genShapes<R, false>(ns, sh, c, phi, (R*)nullptr);
        R const rA = A.r2 * A.ir, rB = B.r2 * B.ir;
#pragma unroll
        for (int a = 0; a < kPairGenRuns; ++a)
            if (a < nr)
            {
                R x = s;
                if (hasRs)
                {
                    R const rs = R(runs[a].rs);
                    x = (rA - rs) * (rA - rs) + (rB - rs) * (rB - rs);
                    if (NARROW) x += (r3 - rs) * (r3 - rs);
                }
                R const v = m * expScaled(expScale(R(runs[a].eta)), x,
                                          w.W.tab);
#pragma unroll
                for (int q = 0; q < S; ++q) acc[a * S + q] += v * phi[q];
            }
    });
    flushCells<R, kPairGenRuns * S>(w, acc, u.cell, nr * S);
}

template <typename R, bool NARROW>
__device__ __forceinline__ void compactValues(SFParams const& P,
                                              UnitTables const& tb,
                                              PairUnit const& u,
                                              Walk<R> const& w)
{
    constexpr int S = kPairCompShapes, N = kPairCompRuns * S;
    R acc[N];
#pragma unroll
    for (int c = 0; c < N; ++c) acc[c] = R(0);
    int const ns = u.ns, nr = u.nr, cs = w.W.cs;
    PairRun const* const runs = tb.r + u.run;
    PairShape const* const sh = tb.s + u.shape;
    walkPairs<R, NARROW>(w, [&](int tt, int kk) {
        Rec<R> const A = w.W.rec[tt], B = w.W.rec[kk];
        R const c = (A.x * B.x + A.y * B.y + A.z * B.z) * (A.ir * B.ir);
        bool const ok = c > R(-1) && c < R(1);
        R phi[S];
        compShapes<R, false>(P, ns, sh, acos(ok ? c : R(0)), phi,
                             (R*)nullptr);
        R rjk = R(0);
        if (NARROW)
        {
            R const x = A.x - B.x, y = A.y - B.y, z = A.z - B.z;
            rjk = sqrt(x * x + y * y + z * z);
        }
#pragma unroll
        for (int a = 0; a < kPairCompRuns; ++a)
            if (a < nr)
            {
                PairRun const& r = runs[a];
                R const* tab = w.W.rad + 2 * r.slot * cs;
                R v = tab[tt] * tab[kk];
                if (NARROW)
                {
                    R f, d;
                    radJk(P, r, rjk, f, d);
                    v *= f;
                }
                v = ok ? v : R(0);
#pragma unroll
                for (int s = 0; s < S; ++s) acc[a * S + s] += v * phi[s];
            }
    });
    flushCells<R, N>(w, acc, u.cell, nr * S);
}

template <typename R, int CT, int NZ, int MASK, bool NARROW>
__device__ __forceinline__ void pow2ValuesN(SFParams const& P, UnitTables const& tb,
    PairUnit const& u, Walk<R> const& w)
{
    switch (u.nr)
    {
    case 1: pow2Values<R, CT, NZ, 1, MASK, NARROW>(P, tb, u, w); break;
    case 2: pow2Values<R, CT, NZ, 2, MASK, NARROW>(P, tb, u, w); break;
    case 3: pow2Values<R, CT, NZ, 3, MASK, NARROW>(P, tb, u, w); break;
    default: pow2Values<R, CT, NZ, 4, MASK, NARROW>(P, tb, u, w); break;
    }
}
// The sets {1}, {1, 4}, {1, 2, 4} and {1, 2, 4, 16} of zeta are compiled without tests of the slots (a test is a branch, which keeps the
// compiler from overlapping the slots' work with the exponentials'); other sets test them.
template <typename R, int CT, int NZ, bool SETS>
__device__ __forceinline__ void pow2ValuesNarrow(SFParams const& P, UnitTables const& tb,
    PairUnit const& u, Walk<R> const& w)
{
    if (!SETS)
    {
        pow2ValuesN<R, CT, NZ, 0, true>(P, tb, u, w);
        return;
    }
    switch (u.mask)
    {
    case 1u: pow2ValuesN<R, CT, NZ, 1, true>(P, tb, u, w); break;
    case 5u: pow2ValuesN<R, CT, NZ, 5, true>(P, tb, u, w); break;
    case 7u: pow2ValuesN<R, CT, NZ, 7, true>(P, tb, u, w); break;
    case 23u: if (NZ > 3) { pow2ValuesN<R, CT, NZ, 23, true>(P, tb, u, w); break; }
    default: pow2ValuesN<R, CT, NZ, 0, true>(P, tb, u, w); break;
    }
}

template <typename R, int CT, int NZ, int KINDS, int WPA, int MINB>
__global__ void __launch_bounds__(kT, MINB)
pairValueKernel(__grid_constant__ SFParams const P,
                __grid_constant__ PairParams const T,
                __grid_constant__ PairLaunch const L)
{
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ Head heads[kW];
    if (L.status[ST_FLAGS] & FLAG_ABORT) return;
    using Tm = Team<WPA>;
    Tm const tm;
    int const lane = tm.lane, warp = tm.warp;
    int const cap = L.cap, maxSF = L.maxSF;
    unsigned char* const mine = sm + L.oTeam + tm.team * L.teamBytes;
    float4* const pos = reinterpret_cast<float4*>(mine + L.oPos);
    R* const dist = reinterpret_cast<R*>(mine + L.oDist);
    unsigned* const bits = reinterpret_cast<unsigned*>(mine + L.oBits);
    R* const Gp = reinterpret_cast<R*>(mine + L.oG);
    Walk<R> w;
    w.W = views<R>(sm, mine, L);
    w.bits = bits;
    w.pairs = reinterpret_cast<unsigned*>(mine + L.oPairs) + L.pairCap * warp;
    w.pairCap = L.pairCap;
    w.red = reinterpret_cast<R*>(mine + L.oRed) + warp * 16 * 33;
    w.Gp = Gp + warp * maxSF;
    w.lane = lane;
    w.warp = warp;
    w.warps = WPA;
    w.words = (cap + 31) >> 5;
    stageExpTable<R>(sm, L);
    UnitTables const tb = stageTables(T, L, sm);
    Head& h = heads[tm.team];
    __syncthreads();
    for (int i = blockIdx.x * Tm::kTeams + tm.team; i < L.n;
         i += gridDim.x * Tm::kTeams)
    {
        if (warp == 0) readHead(T, L, i, lane, &h);
        Tm::sync();
        int const ec = h.ec, cnt = h.cnt;
        if (cnt > cap)
        {
            if (tm.tid == 0)
            {
                atomicOr(&L.status[ST_FLAGS], FLAG_SF_CAPACITY);
                atomicCAS(&L.status[ST_BAD_ATOM], -1, i);
            }
            Tm::sync();
            continue;
        }
        w.W.cs = cnt + 1;
        w.cells = tb.c + T.cellBeg[ec];
        for (int k = tm.tid; k < WPA * maxSF; k += Tm::kThreads) Gp[k] = R(0);
        stageAtom<R, CT, WPA, false>(P, T, L, h, tm, pos, dist, (R*)nullptr,
                                     (R const*)nullptr, tb.q, w.W);
        Tm::sync();
        // Validity mask, upper triangle: (32 rows, word) per warp.
        if (T.narrow[ec])
        {
            float const rc2 = maskRc2(T, ec, sizeof(R) == 8);
            int const nb = (cnt + 31) >> 5;
            int task = 0;
            for (int rb = 0; rb < nb; ++rb)
                for (int q = rb; q < nb; ++q)
                    if ((task++ & (WPA - 1)) == warp)
                    {
                        int const t = (rb << 5) + lane;
                        unsigned const m = maskWord(pos, t, q, cnt, rc2);
                        if (t < cnt) bits[t * w.words + q] = m;
                    }
        }
        // Radial functions: up to four members of one neighbor element per
        // warp, lanes over the neighbors.
        {
            int item = 0;
            int const qe = T.radialBeg[ec + 1];
            for (int q = T.radialBeg[ec]; q < qe;)
            {
                int const grp = tb.q[q].group;
                int q1 = q + 1;
                while (q1 < qe && q1 - q < 4 && tb.q[q1].group == grp) ++q1;
                if ((item++ & (WPA - 1)) == warp)
                {
                    PairRadial const& pr = tb.q[q];
                    bool const all = pr.weighted != 0;
                    int const b = all ? 0 : h.eb[pr.e1];
                    int const e = all ? cnt : h.eb[pr.e1 + 1];
                    R a[4] = {R(0), R(0), R(0), R(0)};
                    for (int t = b + lane; t < e; t += 32)
                    {
                        R fc = R(0), dfc = R(0), Z = R(1);
                        R const r = dist[t];
                        if (pr.fcSlot >= 0) fc = fcOf(w.W, pr.fcSlot, t);
                        else
                        {
                            if (!pr.compact)
                                cutoffFdf<R, CT>(P, P.dGroups[grp], r, fc,
                                                 dfc);
                            if (all)
                            {
                                int el = 0;
                                while (t >= h.eb[el + 1]) ++el;
                                Z = R(P.atomicNumber[el]);
                            }
                        }
#pragma unroll
                        for (int c = 0; c < 4; ++c)
                            if (q + c < q1)
                            {
                                R v, dv;
                                radialFdf<R>(P, tb.q[q + c], r, fc, dfc,
                                             w.W.tab, v, dv);
                                a[c] += Z * v;
                            }
                    }
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        if (q + c < q1)
                        {
#pragma unroll
                            for (int o = 16; o > 0; o >>= 1)
                                a[c] += __shfl_xor_sync(kFull, a[c], o);
                            if (lane == 0)
                                w.Gp[w.cells[tb.q[q + c].cell].sf] += a[c];
                        }
                }
                q = q1;
            }
        }
        Tm::sync();
        for (int ui = T.unitBeg[ec]; ui < T.unitBeg[ec + 1]; ++ui)
        {
            PairUnit const& u = tb.u[ui];
            if (u.weighted)
            {
                w.b1 = 0;
                w.x1 = w.x2 = cnt;
                w.same = 1;
            }
            else
            {
                w.b1 = h.eb[u.e1]; w.x1 = h.eb[u.e1 + 1];
                w.b2 = h.eb[u.e2]; w.x2 = h.eb[u.e2 + 1];
                w.same = (u.e1 == u.e2) ? 1 : 0;
            }
            if ((KINDS & kHasPow2) && (KINDS == kHasPow2 || u.kind == PK_POW2))
            {
                if (u.narrow) pow2ValuesNarrow<R, CT, NZ, KINDS == kHasPow2>(P, tb, u, w);
                else pow2ValuesN<R, CT, NZ, 0, false>(P, tb, u, w);
            }
            else if ((KINDS & kHasLadder) && u.kind == PK_LADDER)
            {
                if (u.narrow) ladderValues<R, CT, kPairGenRuns, true>(P, tb, u, w);
                else ladderValues<R, CT, kPairGenRuns, false>(P, tb, u, w);
            }
            else if ((KINDS & kHasGeneral) && u.kind == PK_GENERAL)
            {
                if (u.narrow) generalValues<R, CT, true>(P, tb, u, w);
                else generalValues<R, CT, false>(P, tb, u, w);
            }
            else if (KINDS & kHasCompact)
            {
                if (u.narrow) compactValues<R, true>(P, tb, u, w);
                else compactValues<R, false>(P, tb, u, w);
            }
        }
        Tm::sync();
        SFScale const* sc = L.scale + (long)ec * maxSF;
        R* const G = static_cast<R*>(L.G) + (long)i * maxSF;
        for (int s = tm.tid; s < P.numSF[ec]; s += Tm::kThreads)
        {
            SFScale const q = sc[s];
            double v = 0.0;
#pragma unroll
            for (int k = 0; k < WPA; ++k) v += (double)Gp[k * maxSF + s];
            G[s] = R(q.smin + q.b * (q.q * v - q.shift));
        }
        Tm::sync();
    }
}

// ---------------------------------------------------------------------------
// Forces pass.
// ---------------------------------------------------------------------------

// Owner j's values and its sums: al along dr_ij and the vector (vx, vy, vz)
// of the coefficients along dr_ik times dr_ik.
template <typename R>
struct Owner
{
    R x, y, z, ir, r2;
    R al, vx, vy, vz;
};

// One lane's share of an owner's partners in a unit: entries at, at + kSl,
// ... of the partner list (narrow) or of the partner range (wide).
struct Partners
{
    unsigned short const* list;   // the lane's first entry
    int at;                       // first partner (wide)
    int n;                        // this lane's partners
    int steps;                    // the warp's
    int t;                        // owner
};

template <bool NARROW>
__device__ __forceinline__ int partner(Partners const& p, int st, int none)
{
    if (NARROW) return st < p.n ? (int)p.list[st * 32] : none;
    int const k = p.at + st * kSl;
    return (st < p.n && k != p.t) ? k : none;
}

template <typename R, int CT, int NZ, int NR, int MASK, bool NARROW>
__device__ __forceinline__ void pow2Forces(SFParams const& P,
                                             UnitTables const& tb,
                                             PairUnit const& u, R const* C,
                                             Staged<R> const& W,
                                             Partners const& p, Owner<R>& o)
{
    using P2 = typename V2<R>::T;
    R e2[NR];
#pragma unroll
    for (int a = 0; a < NR; ++a) e2[a] = expScale(R(tb.r[u.run + a].eta));
    R const a2q = R(u.a2q), qf = R(u.qf), rc2 = R(u.rc2);
    bool const exact = u.exactMask != 0;
    int const slot = u.fcSlot, none = W.cs - 1;
    R const of = fcOf(W, slot, p.t), odf = W.dfc[slot * W.cs + p.t];
    unsigned const mask = MASK ? (unsigned)MASK : u.mask;
    R al = R(0), vx = R(0), vy = R(0), vz = R(0);
    P2 const* const C2 = reinterpret_cast<P2 const*>(C);
#pragma unroll 1
    for (int st = 0; st < p.steps; ++st)
    {
        int const k = partner<NARROW>(p, st, none);
        Rec<R> const B = W.rec[k];
        R fk = slot == 0 ? B.fc : W.fc[(slot - 1) * W.cs + k];
        R const dot = o.x * B.x + o.y * B.y + o.z * B.z;
        R const ir = o.ir * B.ir;
        R s = o.r2 + B.r2;
        R f3 = R(1), q = R(0);
        if (NARROW)
        {
            R const x = o.x - B.x, y = o.y - B.y, z = o.z - B.z;
            R const s3 = x * x + y * y + z * z;
            R r3, ir3;
            cutoffJk<R, CT, true>(P, u, a2q, qf, rc2, exact, s3, false, f3, q,
                                  r3, ir3, fk);
            s += s3;
        }
        R const cosv = dot * ir;
        R b[NR], h[NR];
        R Pm = R(1) - cosv, Pp = R(1) + cosv, mm = R(1), mp = R(1);
        R const pm = Pm, pp = Pp;
#pragma unroll
        for (int z = 0; z < NZ; ++z)
        {
            if ((mask >> z) & 1u)
            {
                // zeta (1 -+ cos)^(zeta-1); zeta = 1: 1.
                R const hp = R(1 << z) * mp, hm = R(1 << z) * mm;
#pragma unroll
                for (int a = 0; a < NR; ++a)
                {
                    P2 const c = C2[z * NR + a];
                    b[a] = z == 0 ? c.x * Pm : b[a] + c.x * Pm;
                    b[a] += c.y * Pp;
                    h[a] = z == 0 ? c.y : h[a] + c.y * hp;
                    h[a] = z == 0 ? h[a] - c.x : h[a] - c.x * hm;
                }
            }
            else if (z == 0)
            {
#pragma unroll
                for (int a = 0; a < NR; ++a) b[a] = h[a] = R(0);
            }
            if (z == 0)
            {
                mm = pm;
                mp = pp;
            }
            else
            {
                mm *= Pm;
                mp *= Pp;
            }
            if (z + 1 < NZ)
            {
                Pm *= Pm;
                Pp *= Pp;
            }
        }
        // T, D (in the exponential's unit) and H.
        R tt = R(0), hh = R(0), dd = R(0);
#pragma unroll
        for (int a = 0; a < NR; ++a)
        {
            R const v = expScaled(e2[a], s, W.tab);
            R const vb = v * b[a];
            tt += vb;
            dd += e2[a] * vb;
            hh += v * h[a];
        }
        R const ff = fk * f3;
        R const m = of * ff;
        R const md = (m * (R(2) * expUnscale<R>())) * dd;   // 2 m D
        R const mh = (m * hh) * ir;
        R a1 = (odf * ff) * tt - (mh * dot) * (o.ir * o.ir) - md;
        R ga = mh;
        if (NARROW)
        {
            R const x3 = (of * fk * q) * tt - md;
            a1 += x3;
            ga -= x3;
        }
        al += a1;
        vx += ga * B.x;
        vy += ga * B.y;
        vz += ga * B.z;
    }
    o.al = al;
    o.vx = vx;
    o.vy = vy;
    o.vz = vz;
}

template <typename R, int CT, bool NARROW>
__device__ __forceinline__ void ladderForces(SFParams const& P,
                                             UnitTables const& tb,
                                             PairUnit const& u, R const* C,
                                             Staged<R> const& W,
                                             Partners const& p, Owner<R>& o)
{
    using P2 = typename V2<R>::T;
    constexpr int NR = kPairGenRuns;
    int const nr = u.nr;
    R e2[NR];
#pragma unroll
    for (int a = 0; a < NR; ++a)
        e2[a] = expScale(R(tb.r[u.run + min(a, nr - 1)].eta));
    R const a2q = R(u.a2q), qf = R(u.qf), rc2 = R(u.rc2);
    bool const exact = u.exactMask != 0;
    int const slot = u.fcSlot, ns = u.ns, none = W.cs - 1;
    R const of = fcOf(W, slot, p.t), odf = W.dfc[slot * W.cs + p.t];
    unsigned prog[kPairLadder];
    R zeta[kPairLadder];
#pragma unroll
    for (int z = 0; z < kPairLadder; ++z)
    {
        prog[z] = u.prog[z];
        zeta[z] = R(u.zeta[z]);
    }
    R al = R(0), vx = R(0), vy = R(0), vz = R(0);
    P2 const* const C2 = reinterpret_cast<P2 const*>(C);
#pragma unroll 1
    for (int st = 0; st < p.steps; ++st)
    {
        int const k = partner<NARROW>(p, st, none);
        Rec<R> const B = W.rec[k];
        R fk = slot == 0 ? B.fc : W.fc[(slot - 1) * W.cs + k];
        R const dot = o.x * B.x + o.y * B.y + o.z * B.z;
        R const ir = o.ir * B.ir;
        R s = o.r2 + B.r2;
        R f3 = R(1), q = R(0);
        if (NARROW)
        {
            R const x = o.x - B.x, y = o.y - B.y, z = o.z - B.z;
            R const s3 = x * x + y * y + z * z;
            R r3, ir3;
            cutoffJk<R, CT, true>(P, u, a2q, qf, rc2, exact, s3, false, f3, q,
                                  r3, ir3, fk);
            s += s3;
        }
        R b[NR], h[NR];
        Ladder<R> l(dot * ir);
#pragma unroll
        for (int z = 0; z < kPairLadder; ++z)
            if (z == 0 || z < ns)
            {
                l.advance(prog[z]);
                R const hp = zeta[z] * l.mp, hm = zeta[z] * l.mm;
#pragma unroll
                for (int a = 0; a < NR; ++a)
                {
                    if (a >= nr) break;
                    P2 const c = C2[z * nr + a];
                    b[a] = z == 0 ? c.x * l.Pm : b[a] + c.x * l.Pm;
                    b[a] += c.y * l.Pp;
                    h[a] = z == 0 ? c.y * hp : h[a] + c.y * hp;
                    h[a] -= c.x * hm;
                }
            }
        // T, D (in the exponential's unit) and H.
        R tt = R(0), hh = R(0), dd = R(0);
#pragma unroll
        for (int a = 0; a < NR; ++a)
        {
            if (a >= nr) break;
            R const v = expScaled(e2[a], s, W.tab);
            R const vb = v * b[a];
            tt += vb;
            dd += e2[a] * vb;
            hh += v * h[a];
        }
        R const ff = fk * f3;
        R const m = of * ff;
        R const md = (m * (R(2) * expUnscale<R>())) * dd;   // 2 m D
        R const mh = (m * hh) * ir;
        R a1 = (odf * ff) * tt - (mh * dot) * (o.ir * o.ir) - md;
        R ga = mh;
        if (NARROW)
        {
            R const x3 = (of * fk * q) * tt - md;
            a1 += x3;
            ga -= x3;
        }
        al += a1;
        vx += ga * B.x;
        vy += ga * B.y;
        vz += ga * B.z;
    }
    o.al = al;
    o.vx = vx;
    o.vy = vy;
    o.vz = vz;
}

template <typename R, int CT, bool NARROW>
__device__ __forceinline__ void generalForces(SFParams const& P,
                                              UnitTables const& tb,
                                              PairUnit const& u, R const* C,
                                              Staged<R> const& W,
                                              Partners const& p, Owner<R>& o)
{
    using P2 = typename V2<R>::T;
    constexpr int S = kPairGenShapes;
    R const a2q = R(u.a2q), qf = R(u.qf), rc2 = R(u.rc2);
    bool const exact = u.exactMask != 0, hasRs = u.hasRs != 0;
    int const slot = u.fcSlot, ns = u.ns, nr = u.nr, none = W.cs - 1;
    R const of = fcOf(W, slot, p.t), odf = W.dfc[slot * W.cs + p.t];
    PairRun const* const runs = tb.r + u.run;
    PairShape const* const sh = tb.s + u.shape;
    P2 const* const C2 = reinterpret_cast<P2 const*>(C);
    R al = R(0), vx = R(0), vy = R(0), vz = R(0);
#pragma unroll 1
    for (int st = 0; st < p.steps; ++st)
    {
        int const k = partner<NARROW>(p, st, none);
        Rec<R> const B = W.rec[k];
        R fk = slot == 0 ? B.fc : W.fc[(slot - 1) * W.cs + k];
        R const dot = o.x * B.x + o.y * B.y + o.z * B.z;
        R const ir = o.ir * B.ir;
        R s = o.r2 + B.r2;
        R f3 = R(1), q = R(0), r3 = R(0), ir3 = R(0);
        if (NARROW)
        {
            R const x = o.x - B.x, y = o.y - B.y, z = o.z - B.z;
            R const s3 = x * x + y * y + z * z;
            cutoffJk<R, CT, true>(P, u, a2q, qf, rc2, exact, s3, hasRs, f3, q,
                                  r3, ir3, fk);
            s += s3;
        }
        R phi[S], psi[S];
        genShapes<R, true>(ns, sh, dot * ir, phi, psi);
        R const rA = o.r2 * o.ir, rB = B.r2 * B.ir;
        R tt = R(0), hh = R(0), d1 = R(0), d3 = R(0);
#pragma unroll 1
        for (int a = 0; a < nr; ++a)
        {
            R const eta = R(runs[a].eta), rs = R(runs[a].rs);
            R x = s;
            if (hasRs)
            {
                x = (rA - rs) * (rA - rs) + (rB - rs) * (rB - rs);
                if (NARROW) x += (r3 - rs) * (r3 - rs);
            }
            R const v = expScaled(expScale(eta), x, W.tab);
            R b = R(0), h = R(0);
#pragma unroll
            for (int j = 0; j < S / 2; ++j)
            {
                P2 const c = C2[a * (S / 2) + j];
                b += c.x * phi[2 * j];
                b += c.y * phi[2 * j + 1];
                h += c.x * psi[2 * j];
                h += c.y * psi[2 * j + 1];
            }
            R const vb = v * b, ev = eta * vb;
            tt += vb;
            hh += v * h;
            d1 += hasRs ? ev * (R(1) - rs * o.ir) : ev;
            d3 += hasRs ? ev * (R(1) - rs * ir3) : ev;
        }
        R const ff = fk * f3;
        R const m = of * ff;
        R const m2 = R(2) * m;
        R const mh = (m * hh) * ir;
        R a1 = (odf * ff) * tt - (mh * dot) * (o.ir * o.ir) - m2 * d1;
        R ga = mh;
        if (NARROW)
        {
            R const x3 = (of * fk * q) * tt - m2 * d3;
            a1 += x3;
            ga -= x3;
        }
        al += a1;
        vx += ga * B.x;
        vy += ga * B.y;
        vz += ga * B.z;
    }
    o.al = al;
    o.vx = vx;
    o.vy = vy;
    o.vz = vz;
}

template <typename R, bool NARROW>
__device__ __forceinline__ void compactForces(SFParams const& P,
                                              UnitTables const& tb,
                                              PairUnit const& u, R const* C,
                                              Staged<R> const& W,
                                              Partners const& p, Owner<R>& o)
{
    using P2 = typename V2<R>::T;
    constexpr int S = kPairCompShapes;
    int const ns = u.ns, nr = u.nr, cs = W.cs, none = cs - 1;
    PairRun const* const runs = tb.r + u.run;
    PairShape const* const sh = tb.s + u.shape;
    P2 const* const C2 = reinterpret_cast<P2 const*>(C);
    R al = R(0), vx = R(0), vy = R(0), vz = R(0);
#pragma unroll 1
    for (int st = 0; st < p.steps; ++st)
    {
        int const k = partner<NARROW>(p, st, none);
        Rec<R> const B = W.rec[k];
        R const dot = o.x * B.x + o.y * B.y + o.z * B.z;
        R const ir = o.ir * B.ir;
        R c = dot * ir;
        bool const ok = c > R(-1) && c < R(1);
        c = ok ? c : R(0);
        R const dacos = -mrsqrt(R(1) - c * c);
        R phi[S], psi[S];
        compShapes<R, true>(P, ns, sh, acos(c), phi, psi);
        R rjk = R(0), ir3 = R(0);
        if (NARROW)
        {
            R const x = o.x - B.x, y = o.y - B.y, z = o.z - B.z;
            R const s3 = x * x + y * y + z * z;
            ir3 = mrsqrt(s3 > R(0) ? s3 : R(1));
            rjk = s3 * ir3;
        }
        R x1 = R(0), x2 = R(0), x3 = R(0);
#pragma unroll 1
        for (int a = 0; a < nr; ++a)
        {
            PairRun const& w = runs[a];
            R const* tab = W.rad + 2 * w.slot * cs;
            R const rk = tab[k];
            R b = R(0), h = R(0);
#pragma unroll
            for (int j = 0; j < S / 2; ++j)
            {
                P2 const cc = C2[a * (S / 2) + j];
                b += cc.x * phi[2 * j];
                b += cc.y * phi[2 * j + 1];
                h += cc.x * psi[2 * j];
                h += cc.y * psi[2 * j + 1];
            }
            R const rj = tab[p.t], drj = tab[cs + p.t];
            if (NARROW)
            {
                R f, d;
                radJk(P, w, rjk, f, d);
                x3 += (rj * rk) * (d * b);
                b *= f;
                h *= f;
            }
            x1 += (drj * rk) * b;
            x2 += (rj * rk) * h;
        }
        if (!ok) x1 = x2 = x3 = R(0);
        x3 *= ir3;
        R const mh = (x2 * dacos) * ir;
        R const ga = mh - x3;
        al += x1 - (mh * dot) * (o.ir * o.ir) + x3;
        vx += ga * B.x;
        vy += ga * B.y;
        vz += ga * B.z;
    }
    o.al = al;
    o.vx = vx;
    o.vy = vy;
    o.vz = vz;
}

template <typename R, int CT, int NZ, int MASK, bool NARROW>
__device__ __forceinline__ void pow2ForcesN(SFParams const& P, UnitTables const& tb,
    PairUnit const& u, R const* C, Staged<R> const& W, Partners const& p,
    Owner<R>& o)
{
    switch (u.nr)
    {
    case 1: pow2Forces<R, CT, NZ, 1, MASK, NARROW>(P, tb, u, C, W, p, o); break;
    case 2: pow2Forces<R, CT, NZ, 2, MASK, NARROW>(P, tb, u, C, W, p, o); break;
    case 3: pow2Forces<R, CT, NZ, 3, MASK, NARROW>(P, tb, u, C, W, p, o); break;
    default: pow2Forces<R, CT, NZ, 4, MASK, NARROW>(P, tb, u, C, W, p, o); break;
    }
}
// The sets {1}, {1, 4}, {1, 2, 4} and {1, 2, 4, 16} of zeta are compiled without tests of the slots (52 functions,
// 6,144 atoms, FP64: 0.90 -> 0.71 ms); other sets test them.
template <typename R, int CT, int NZ, bool SETS>
__device__ __forceinline__ void pow2ForcesNarrow(SFParams const& P, UnitTables const& tb,
    PairUnit const& u, R const* C, Staged<R> const& W, Partners const& p,
    Owner<R>& o)
{
    if (!SETS)
    {
        pow2ForcesN<R, CT, NZ, 0, true>(P, tb, u, C, W, p, o);
        return;
    }
    switch (u.mask)
    {
    case 1u: pow2ForcesN<R, CT, NZ, 1, true>(P, tb, u, C, W, p, o); break;
    case 5u: pow2ForcesN<R, CT, NZ, 5, true>(P, tb, u, C, W, p, o); break;
    case 7u: pow2ForcesN<R, CT, NZ, 7, true>(P, tb, u, C, W, p, o); break;
    case 23u: if (NZ > 3) { pow2ForcesN<R, CT, NZ, 23, true>(P, tb, u, C, W, p, o); break; }
    default: pow2ForcesN<R, CT, NZ, 0, true>(P, tb, u, C, W, p, o); break;
    }
}

template <typename R, int CT, int NZ, int KINDS, int WPA, int MINB>
__global__ void __launch_bounds__(kT, MINB)
pairTermKernel(__grid_constant__ SFParams const P,
               __grid_constant__ PairParams const T,
               __grid_constant__ PairLaunch const L)
{
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ Head heads[kW];
    __shared__ int nextItem;
    if (L.status[ST_FLAGS] & FLAG_ABORT) return;
    using Tm = Team<WPA>;
    Tm const tm;
    int const lane = tm.lane, warp = tm.warp;
    int const ow = lane / kSl, sl = lane % kSl;
    int const cap = L.cap, words = (cap + 31) >> 5, ne = T.numElements;
    unsigned char* const mine = sm + L.oTeam + tm.team * L.teamBytes;
    float4* const pos = reinterpret_cast<float4*>(mine + L.oPos);
    Staged<R> W = views<R>(sm, mine, L);
    R* const C = reinterpret_cast<R*>(mine + L.oCoef);
    R* const arad = reinterpret_cast<R*>(mine + L.oAr);
    unsigned* const bits = reinterpret_cast<unsigned*>(mine + L.oBits);
    unsigned* const key = reinterpret_cast<unsigned*>(mine + L.oKey);
    unsigned short* const pre =
        reinterpret_cast<unsigned short*>(mine + L.oPre);
    unsigned short* const order =
        reinterpret_cast<unsigned short*>(mine + L.oOrder);
    unsigned short* const list =
        reinterpret_cast<unsigned short*>(mine + L.oList) + warp * kOw * cap;
    stageExpTable<R>(sm, L);
    UnitTables const tb = stageTables(T, L, sm);
    double* const F = reinterpret_cast<double*>(mine + L.oF);
    Head& h = heads[tm.team];
    __syncthreads();
    for (int i = blockIdx.x * Tm::kTeams + tm.team; i < L.n;
         i += gridDim.x * Tm::kTeams)
    {
        if (warp == 0) readHead(T, L, i, lane, &h);
        if (WPA > 1 && tm.tid == 0) nextItem = 0;
        Tm::sync();
        int const ec = h.ec, cnt = h.cnt;
        long const beg = h.beg;
        if (cnt > cap)
        {
            if (tm.tid == 0)
            {
                atomicOr(&L.status[ST_FLAGS], FLAG_SF_CAPACITY);
                atomicCAS(&L.status[ST_BAD_ATOM], -1, i);
            }
            Tm::sync();
            continue;
        }
        W.cs = cnt + 1;
        bool const anyNarrow = T.narrow[ec] != 0;
        // Coefficients dE/dG x factor: the units' cells (empty cells 0), then
        // the radial members'.
        {
            int const c0 = T.cellBeg[ec], nc = T.cellBeg[ec + 1] - c0;
            R const* row = static_cast<R const*>(L.dEdG) + (long)i * L.maxSF;
            for (int k = tm.tid; k < nc; k += Tm::kThreads)
            {
                PairCell const ce = tb.c[c0 + k];
                C[k] = ce.sf >= 0 ? row[ce.sf] * R(ce.fn) : R(0);
            }
        }
        Tm::sync();
        stageAtom<R, CT, WPA, true>(P, T, L, h, tm, pos, (R*)nullptr, arad, C,
                                    tb.q, W);
        Tm::sync();
        // Validity masks (narrow units), lanes own rows; with them per row the
        // partners of the elements below each one and in all, and the key
        // that orders the owners.
        if (anyNarrow)
        {
            float const rc2 = maskRc2(T, ec, sizeof(R) == 8);
            int const nb = (cnt + 31) >> 5;
            for (int rb = warp; rb < nb; rb += WPA)
            {
                int const t = (rb << 5) + lane;
                bool const in = t < cnt;
                int total = 0, e = 0;
                for (int q = 0; q < nb; ++q)
                {
                    unsigned m = maskWord(pos, t, q, cnt, rc2);
                    if (q == rb) m &= ~(1u << lane);
                    if (in) bits[t * words + q] = m;
                    for (; e < ne && h.eb[e] < (q + 1) << 5; ++e)
                        if (in)
                            pre[t * (ne + 1) + e] = (unsigned short)(
                                total
                                + __popc(m & ((1u << (h.eb[e] & 31)) - 1u)));
                    total += __popc(m);
                }
                if (in)
                {
                    for (; e <= ne; ++e)
                        pre[t * (ne + 1) + e] = (unsigned short)total;
                    key[t] = ((unsigned)total << 16) | (0xffffu - (unsigned)t);
                }
            }
        }
        Tm::sync();
        // Owners of each element by descending partner count (ties by
        // position).
        for (int t = tm.tid; t < cnt; t += Tm::kThreads)
        {
            int rank = t;
            if (anyNarrow)
            {
                int e = 0;
                while (t >= h.eb[e + 1]) ++e;
                unsigned const mine = key[t];
                int const q1 = h.eb[e + 1];
                rank = h.eb[e];
#pragma unroll 4
                for (int q = rank; q < q1; ++q) rank += key[q] > mine ? 1 : 0;
            }
            order[rank] = (unsigned short)t;
        }
        Tm::sync();

        double sx = 0.0;      // lanes sl < 3: minus the self force's part
        for (int it = 0;; ++it)
        {
            // Items in order; a block's warps take the next one as they get
            // done (their sums go through F, so the order does not matter).
            int item = it;
            if (WPA > 1)
            {
                if (lane == 0) item = atomicAdd(&nextItem, 1);
                item = __shfl_sync(kFull, item, 0);
            }
            int oe = 0, first = 0;
            for (; oe < ne; ++oe)
            {
                int const m = (h.eb[oe + 1] - h.eb[oe] + kOw - 1) / kOw;
                if (item < m) break;
                item -= m;
            }
            if (oe == ne) break;
            first = h.eb[oe] + item * kOw;
            bool const has = first + ow < h.eb[oe + 1];
            int const t = has ? (int)order[first + ow] : (int)order[first];
            Owner<R> o;
            {
                Rec<R> const a = W.rec[t];
                o.x = a.x; o.y = a.y; o.z = a.z; o.ir = a.ir; o.r2 = a.r2;
            }
            // Partner lists: the owner's lanes take its mask words in turn.
            if (anyNarrow)
            {
                __syncwarp();
                int base = 0;
                for (int w0 = 0; w0 << 5 < cnt; w0 += kSl)
                {
                    int const w = w0 + sl;
                    unsigned m = (has && w << 5 < cnt) ? bits[t * words + w] : 0u;
                    int const n = __popc(m);
                    int p = n;
    #pragma unroll
                    for (int d = 1; d < kSl; d <<= 1)
                    {
                        int const v = __shfl_up_sync(kFull, p, d, kSl);
                        if (sl >= d) p += v;
                    }
                    int at = base + p - n;
                    base += __shfl_sync(kFull, p, kSl - 1, kSl);
                    while (m)
                    {
                        int const k = 32 * w + __ffs(m) - 1;
                        m &= m - 1;
                        list[(at / kSl) * 32 + ow * kSl + (at % kSl)] =
                            (unsigned short)k;
                        ++at;
                    }
                }
                __syncwarp();
            }
            // The radial functions' part is along dr_ij too.
            double Al = (has && sl == 0) ? (double)arad[t] : 0.0;
            double Vx = 0.0, Vy = 0.0, Vz = 0.0;
            for (int ui = T.unitBeg[ec]; ui < T.unitBeg[ec + 1]; ++ui)
            {
                PairUnit const& u = tb.u[ui];
                int pe = 0;
                if (!u.weighted)
                {
                    if (u.e1 == oe) pe = u.e2;
                    else if (u.e2 == oe) pe = u.e1;
                    else continue;
                }
                int lo, n;
                if (u.narrow)
                {
                    unsigned short const* pr = pre + t * (ne + 1);
                    lo = u.weighted ? 0 : pr[pe];
                    n = (u.weighted ? pr[ne] : pr[pe + 1]) - lo;
                }
                else
                {
                    lo = u.weighted ? 0 : h.eb[pe];
                    n = (u.weighted ? cnt : h.eb[pe + 1]) - lo;
                }
                // Owners outside the unit's cutoff have no triplets.
                if (!has || !(o.r2 < R(u.rc2))) n = 0;
                Partners p;
                p.steps = (__reduce_max_sync(kFull, n) + kSl - 1) / kSl;
                p.n = (n - sl + kSl - 1) / kSl;
                p.t = t;
                int const at = lo + sl;
                p.at = at;
                p.list = list + (at / kSl) * 32 + ow * kSl + (at % kSl);
                R const* Cu = C + u.cell;
                if ((KINDS & kHasPow2)
                    && (KINDS == kHasPow2 || u.kind == PK_POW2))
                {
                    if (u.narrow)
                        pow2ForcesNarrow<R, CT, NZ, KINDS == kHasPow2>(P, tb, u, Cu, W, p,
                                                    o);
                    else pow2ForcesN<R, CT, NZ, 0, false>(P, tb, u, Cu, W,
                                                          p, o);
                }
                else if ((KINDS & kHasLadder) && u.kind == PK_LADDER)
                {
                    if (u.narrow)
                        ladderForces<R, CT, true>(P, tb, u, Cu, W, p, o);
                    else ladderForces<R, CT, false>(P, tb, u, Cu, W, p, o);
                }
                else if ((KINDS & kHasGeneral) && u.kind == PK_GENERAL)
                {
                    if (u.narrow)
                        generalForces<R, CT, true>(P, tb, u, Cu, W, p, o);
                    else generalForces<R, CT, false>(P, tb, u, Cu, W, p, o);
                }
                else if (KINDS & kHasCompact)
                {
                    if (u.narrow) compactForces<R, true>(P, tb, u, Cu, W, p, o);
                    else compactForces<R, false>(P, tb, u, Cu, W, p, o);
                }
                Al += (double)o.al;
                Vx += (double)o.vx;
                Vy += (double)o.vy;
                Vz += (double)o.vz;
            }
    #pragma unroll
            for (int d = 1; d < kSl; d <<= 1)
            {
                Al += __shfl_xor_sync(kFull, Al, d);
                Vx += __shfl_xor_sync(kFull, Vx, d);
                Vy += __shfl_xor_sync(kFull, Vy, d);
                Vz += __shfl_xor_sync(kFull, Vz, d);
            }
            if (has && sl < 3)
            {
                double const v = sl == 0 ? Vx : (sl == 1 ? Vy : Vz);
                double const* const a = sl == 0 ? L.dx
                                      : (sl == 1 ? L.dy : L.dz);
                double const f = Al * a[beg + t] + v;
                L.pairF[(beg + t) * 3 + sl] = f;
                if (WPA == 1) sx += f;
                else F[3 * t + sl] = f;
            }
        }
        // The self force: minus the sum of the pair terms.
        if (WPA == 1)
        {
#pragma unroll
            for (int d = kSl; d < 32; d <<= 1)
                sx += __shfl_xor_sync(kFull, sx, d);
            if (lane < 3) L.selfF[(long)i * 3 + lane] = -sx;
        }
        else
        {
            Tm::sync();
            if (warp < 3)
            {
                double v = 0.0;
                for (int t = lane; t < cnt; t += 32) v -= F[3 * t + warp];
                v = warpSum(v);
                if (lane == 0) L.selfF[(long)i * 3 + warp] = v;
            }
        }
        Tm::sync();
    }
}

} // namespace sfp2
} // namespace n2p2b
