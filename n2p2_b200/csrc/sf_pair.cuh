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
// Both passes: a team of one or four warps per atom (launchPair says when).
//
// Values pass: each unordered triplet once.  Lanes own the rows of the
// validity mask (r_jk < rc) and list their rows' valid pairs; the team walks
// the list 32 pairs at a time; the unit's sums stay in registers (lane sums,
// then one fixed-order reduction per unit).
//
// Forces pass: an item is eight owners j of one element on four lanes each,
// owners ordered by their partner counts so that the owners of an item have
// similar trip counts.  The item's lanes build the owners' partner lists
// from the validity mask, walk the units with the unit's parameters the same
// for the whole warp, and add the four slices at the end.  Each pair term
// has one writer: no atomics, fixed order.
//
// Precision.  The FP32 kernels form a triplet's terms in FP32, the sums over
// its members among them, and add them up in FP64: over an owner's partners,
// the radial functions of a neighbor, the units, the lanes and the neighbors.
// The storing kernels add a member's partners in FP32 and the members in
// FP64.  Forces' rms error against FP64 with exact dE/dG, 12 water boxes of
// 192 to 720 atoms, two passes / storing kernels: 52 functions 1.50e-7 /
// 2.32e-7, 92 functions 2.79e-7 / 5.03e-7, tanh^3 cutoff (27 and 30
// functions) 2.51e-7 / 2.47e-7; with FP32 sums over partners and radial
// functions 1.52, 3.07 and 2.61e-7.  FP64 inside the triplet as well leaves
// the errors where they are (92 functions 2.94e-7 against 3.08e-7 with FP32
// sums, 256 molecules) and takes a third more time.
//
// Bounds.  Memory is small (the neighbor entries once per pass, 24 B written
// per entry); the FP64 instructions (about 80 a triplet for the values, 130
// per owner for the forces, 3 runs x 4 shapes) and their latency at 12 to 16
// warps per multiprocessor bound both passes.  24,576 water atoms, 52
// functions, FP64: 0.96 + 2.4 ms, where dG/dr took 6.1 to form and 0.4 to
// contract (2 GB each way); 98,304 atoms, 92 functions, FP32: 2.8 + 7.0 ms
// against 25.1 + 1.5.
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

constexpr double kLn256 = 0x1.62e42fefa39efp-9;    // ln2 / 256

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
    R*            rad;        // [rad slot][cs] window functions (x Z); forces:
                              // [rad slot][2][cs] with derivative / r
    double const* tab;        // exponential table
    int           cs;         // cap + 1
};

// Polynomial coefficients of the FP64 kernels in the constant bank: an FMA
// takes one operand from there, while 64-bit literals cost two moves each in
// a loop that has no registers left to keep them.
//   ex: 2^(f/256) - 1 = f (ex3 + f (ex2 + ...)), Taylor.
//   ch, sh: cos(sqrt w) and sin(sqrt w) / sqrt w on 0 <= w <= (pi/2)^2 (r up
//   to the cutoff), interpolated at the Chebyshev nodes; their errors there,
//   rounding of the coefficients included, are 6.4e-17 and 1.4e-17 (a Taylor
//   series of that error needs two terms more).
struct PairConst
{
    double ex[4];
    double ch[9], sh[9];
    double shift;
};
__constant__ PairConst kPC = {
    {kLn256 * kLn256 * kLn256 * kLn256 / 24.0, kLn256 * kLn256 * kLn256 / 6.0,
     kLn256 * kLn256 / 2.0, kLn256},
    {0x1.9f237664fdb61p-45, -0x1.9350a15519b35p-37, 0x1.1eecdf2eb6420p-29,
     -0x1.27e4f97908e2ep-22, 0x1.a01a01994b814p-16, -0x1.6c16c16c09b34p-10,
     0x1.55555555553c4p-5, -0x1.ffffffffffffbp-2, 1.0},
    {0x1.88382132048bcp-49, -0x1.ae439c8976ed0p-41, 0x1.6123ccd07d338p-33,
     -0x1.ae6454d052da4p-26, 0x1.71de3a528cce3p-19, -0x1.a01a01a0147e9p-13,
     0x1.11111111110bcp-7, -0x1.5555555555555p-3, 1.0},
    0x1.8p52};

// 2^(j / 256), rounded to nearest; staged into shared memory.
constexpr int kPairExpSize = 256;
static __device__ double const kPairExp2[kPairExpSize] = {
    0x1.0000000000000p+0, 0x1.00b1afa5abcbfp+0, 0x1.0163da9fb3335p+0,
    0x1.02168143b0281p+0, 0x1.02c9a3e778061p+0, 0x1.037d42e11bbccp+0,
    0x1.04315e86e7f85p+0, 0x1.04e5f72f654b1p+0, 0x1.059b0d3158574p+0,
    0x1.0650a0e3c1f89p+0, 0x1.0706b29ddf6dep+0, 0x1.07bd42b72a836p+0,
    0x1.0874518759bc8p+0, 0x1.092bdf66607e0p+0, 0x1.09e3ecac6f383p+0,
    0x1.0a9c79b1f3919p+0, 0x1.0b5586cf9890fp+0, 0x1.0c0f145e46c85p+0,
    0x1.0cc922b7247f7p+0, 0x1.0d83b23395decp+0, 0x1.0e3ec32d3d1a2p+0,
    0x1.0efa55fdfa9c5p+0, 0x1.0fb66affed31bp+0, 0x1.1073028d7233ep+0,
    0x1.11301d0125b51p+0, 0x1.11edbab5e2ab6p+0, 0x1.12abdc06c31ccp+0,
    0x1.136a814f204abp+0, 0x1.1429aaea92de0p+0, 0x1.14e95934f312ep+0,
    0x1.15a98c8a58e51p+0, 0x1.166a45471c3c2p+0, 0x1.172b83c7d517bp+0,
    0x1.17ed48695bbc0p+0, 0x1.18af9388c8deap+0, 0x1.1972658375d2fp+0,
    0x1.1a35beb6fcb75p+0, 0x1.1af99f8138a1cp+0, 0x1.1bbe084045cd4p+0,
    0x1.1c82f95281c6bp+0, 0x1.1d4873168b9aap+0, 0x1.1e0e75eb44027p+0,
    0x1.1ed5022fcd91dp+0, 0x1.1f9c18438ce4dp+0, 0x1.2063b88628cd6p+0,
    0x1.212be3578a819p+0, 0x1.21f49917ddc96p+0, 0x1.22bdda27912d1p+0,
    0x1.2387a6e756238p+0, 0x1.2451ffb82140ap+0, 0x1.251ce4fb2a63fp+0,
    0x1.25e85711ece75p+0, 0x1.26b4565e27cddp+0, 0x1.2780e341ddf29p+0,
    0x1.284dfe1f56381p+0, 0x1.291ba7591bb70p+0, 0x1.29e9df51fdee1p+0,
    0x1.2ab8a66d10f13p+0, 0x1.2b87fd0dad990p+0, 0x1.2c57e39771b2fp+0,
    0x1.2d285a6e4030bp+0, 0x1.2df961f641589p+0, 0x1.2ecafa93e2f56p+0,
    0x1.2f9d24abd886bp+0, 0x1.306fe0a31b715p+0, 0x1.31432edeeb2fdp+0,
    0x1.32170fc4cd831p+0, 0x1.32eb83ba8ea32p+0, 0x1.33c08b26416ffp+0,
    0x1.3496266e3fa2dp+0, 0x1.356c55f929ff1p+0, 0x1.36431a2de883bp+0,
    0x1.371a7373aa9cbp+0, 0x1.37f26231e754ap+0, 0x1.38cae6d05d866p+0,
    0x1.39a401b7140efp+0, 0x1.3a7db34e59ff7p+0, 0x1.3b57fbfec6cf4p+0,
    0x1.3c32dc313a8e5p+0, 0x1.3d0e544ede173p+0, 0x1.3dea64c123422p+0,
    0x1.3ec70df1c5175p+0, 0x1.3fa4504ac801cp+0, 0x1.40822c367a024p+0,
    0x1.4160a21f72e2ap+0, 0x1.423fb2709468ap+0, 0x1.431f5d950a897p+0,
    0x1.43ffa3f84b9d4p+0, 0x1.44e086061892dp+0, 0x1.45c2042a7d232p+0,
    0x1.46a41ed1d0057p+0, 0x1.4786d668b3237p+0, 0x1.486a2b5c13cd0p+0,
    0x1.494e1e192aed2p+0, 0x1.4a32af0d7d3dep+0, 0x1.4b17dea6db7d7p+0,
    0x1.4bfdad5362a27p+0, 0x1.4ce41b817c114p+0, 0x1.4dcb299fddd0dp+0,
    0x1.4eb2d81d8abffp+0, 0x1.4f9b2769d2ca7p+0, 0x1.508417f4531eep+0,
    0x1.516daa2cf6642p+0, 0x1.5257de83f4eefp+0, 0x1.5342b569d4f82p+0,
    0x1.542e2f4f6ad27p+0, 0x1.551a4ca5d920fp+0, 0x1.56070dde910d2p+0,
    0x1.56f4736b527dap+0, 0x1.57e27dbe2c4cfp+0, 0x1.58d12d497c7fdp+0,
    0x1.59c0827ff07ccp+0, 0x1.5ab07dd485429p+0, 0x1.5ba11fba87a03p+0,
    0x1.5c9268a5946b7p+0, 0x1.5d84590998b93p+0, 0x1.5e76f15ad2148p+0,
    0x1.5f6a320dceb71p+0, 0x1.605e1b976dc09p+0, 0x1.6152ae6cdf6f4p+0,
    0x1.6247eb03a5585p+0, 0x1.633dd1d1929fdp+0, 0x1.6434634ccc320p+0,
    0x1.652b9febc8fb7p+0, 0x1.6623882552225p+0, 0x1.671c1c70833f6p+0,
    0x1.68155d44ca973p+0, 0x1.690f4b19e9538p+0, 0x1.6a09e667f3bcdp+0,
    0x1.6b052fa75173ep+0, 0x1.6c012750bdabfp+0, 0x1.6cfdcddd47645p+0,
    0x1.6dfb23c651a2fp+0, 0x1.6ef9298593ae5p+0, 0x1.6ff7df9519484p+0,
    0x1.70f7466f42e87p+0, 0x1.71f75e8ec5f74p+0, 0x1.72f8286ead08ap+0,
    0x1.73f9a48a58174p+0, 0x1.74fbd35d7cbfdp+0, 0x1.75feb564267c9p+0,
    0x1.77024b1ab6e09p+0, 0x1.780694fde5d3fp+0, 0x1.790b938ac1cf6p+0,
    0x1.7a11473eb0187p+0, 0x1.7b17b0976cfdbp+0, 0x1.7c1ed0130c132p+0,
    0x1.7d26a62ff86f0p+0, 0x1.7e2f336cf4e62p+0, 0x1.7f3878491c491p+0,
    0x1.80427543e1a12p+0, 0x1.814d2add106d9p+0, 0x1.82589994cce13p+0,
    0x1.8364c1eb941f7p+0, 0x1.8471a4623c7adp+0, 0x1.857f4179f5b21p+0,
    0x1.868d99b4492edp+0, 0x1.879cad931a436p+0, 0x1.88ac7d98a6699p+0,
    0x1.89bd0a478580fp+0, 0x1.8ace5422aa0dbp+0, 0x1.8be05bad61778p+0,
    0x1.8cf3216b5448cp+0, 0x1.8e06a5e0866d9p+0, 0x1.8f1ae99157736p+0,
    0x1.902fed0282c8ap+0, 0x1.9145b0b91ffc6p+0, 0x1.925c353aa2fe2p+0,
    0x1.93737b0cdc5e5p+0, 0x1.948b82b5f98e5p+0, 0x1.95a44cbc8520fp+0,
    0x1.96bdd9a7670b3p+0, 0x1.97d829fde4e50p+0, 0x1.98f33e47a22a2p+0,
    0x1.9a0f170ca07bap+0, 0x1.9b2bb4d53fe0dp+0, 0x1.9c49182a3f090p+0,
    0x1.9d674194bb8d5p+0, 0x1.9e86319e32323p+0, 0x1.9fa5e8d07f29ep+0,
    0x1.a0c667b5de565p+0, 0x1.a1e7aed8eb8bbp+0, 0x1.a309bec4a2d33p+0,
    0x1.a42c980460ad8p+0, 0x1.a5503b23e255dp+0, 0x1.a674a8af46052p+0,
    0x1.a799e1330b358p+0, 0x1.a8bfe53c12e59p+0, 0x1.a9e6b5579fdbfp+0,
    0x1.ab0e521356ebap+0, 0x1.ac36bbfd3f37ap+0, 0x1.ad5ff3a3c2774p+0,
    0x1.ae89f995ad3adp+0, 0x1.afb4ce622f2ffp+0, 0x1.b0e07298db666p+0,
    0x1.b20ce6c9a8952p+0, 0x1.b33a2b84f15fbp+0, 0x1.b468415b749b1p+0,
    0x1.b59728de5593ap+0, 0x1.b6c6e29f1c52ap+0, 0x1.b7f76f2fb5e47p+0,
    0x1.b928cf22749e4p+0, 0x1.ba5b030a1064ap+0, 0x1.bb8e0b79a6f1fp+0,
    0x1.bcc1e904bc1d2p+0, 0x1.bdf69c3f3a207p+0, 0x1.bf2c25bd71e09p+0,
    0x1.c06286141b33dp+0, 0x1.c199bdd85529cp+0, 0x1.c2d1cd9fa652cp+0,
    0x1.c40ab5fffd07ap+0, 0x1.c544778fafb22p+0, 0x1.c67f12e57d14bp+0,
    0x1.c7ba88988c933p+0, 0x1.c8f6d9406e7b5p+0, 0x1.ca3405751c4dbp+0,
    0x1.cb720dcef9069p+0, 0x1.ccb0f2e6d1675p+0, 0x1.cdf0b555dc3fap+0,
    0x1.cf3155b5bab74p+0, 0x1.d072d4a07897cp+0, 0x1.d1b532b08c968p+0,
    0x1.d2f87080d89f2p+0, 0x1.d43c8eacaa1d6p+0, 0x1.d5818dcfba487p+0,
    0x1.d6c76e862e6d3p+0, 0x1.d80e316c98398p+0, 0x1.d955d71ff6075p+0,
    0x1.da9e603db3285p+0, 0x1.dbe7cd63a8315p+0, 0x1.dd321f301b460p+0,
    0x1.de7d5641c0658p+0, 0x1.dfc97337b9b5fp+0, 0x1.e11676b197d17p+0,
    0x1.e264614f5a129p+0, 0x1.e3b333b16ee12p+0, 0x1.e502ee78b3ff6p+0,
    0x1.e653924676d76p+0, 0x1.e7a51fbc74c83p+0, 0x1.e8f7977cdb740p+0,
    0x1.ea4afa2a490dap+0, 0x1.eb9f4867cca6ep+0, 0x1.ecf482d8e67f1p+0,
    0x1.ee4aaa2188510p+0, 0x1.efa1bee615a27p+0, 0x1.f0f9c1cb6412ap+0,
    0x1.f252b376bba97p+0, 0x1.f3ac948dd7274p+0, 0x1.f50765b6e4540p+0,
    0x1.f6632798844f8p+0, 0x1.f7bfdad9cbe14p+0, 0x1.f91d802243c89p+0,
    0x1.fa7c1819e90d8p+0, 0x1.fbdba3692d514p+0, 0x1.fd3c22b8f71f1p+0,
    0x1.fe9d96b2a23d9p+0,
};

// Constants of one run: -eta in the exponential's unit, from the tables'
// -eta / ln 2 and rounded once (in FP32 its error is the same for every
// triplet of the run and does not average out).
//   FP64: exp(-eta s) = 2^(k/256) 2^(f/256), k = rint(y), f = y - k with
//   y = -eta s 256/ln2; f is formed by one fma from s (no product rounding),
//   2^(f/256) - 1 by its Taylor polynomial of degree 4 in f (|f| <= 1/2:
//   truncation below 4e-17), 2^(j/256) from the table.  The error is that of
//   y's factor, |eta s| 2^-53, and 1 ulp, as for exp of the rounded
//   product.  Results below 2^-1020 stay near 2^-1020.
template <typename R>
__device__ __forceinline__ R expScale(double e2)
{
    return sizeof(R) == 8 ? R(e2 * 256.0) : R(e2);
}
__device__ __forceinline__ double expScaled(double e2, double s,
                                            double const* tab)
{
    double const t = fma(s, e2, kPC.shift);
    int const k = max(__double2loint(t), -256 * 1020);
    double const f = fma(s, e2, kPC.shift - t);
    double p = fma(f, kPC.ex[0], kPC.ex[1]);
    p = fma(p, f, kPC.ex[2]);
    p = fma(p, f, kPC.ex[3]);
    double const q = p * f;
    double const tj = tab[k & (kPairExpSize - 1)];
    double const tm = __hiloint2double(
        __double2hiint(tj) + ((k >> 8) << 20), __double2loint(tj));
    return fma(tm, q, tm);
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
    return sizeof(R) == 8 ? R(-0x1.62e42fefa39efp-9) : R(-0.693147181f);
}

// cos and sin(x)/x of the half angle from w = (a r / 2)^2.  FP32: degrees 5
// and 4, interpolated likewise (errors 2.8e-8 and 8.2e-9).
__device__ __forceinline__ double halfAngleCos(double w)
{
    double c = kPC.ch[0];
#pragma unroll
    for (int n = 1; n < 9; ++n) c = fma(c, w, kPC.ch[n]);
    return c;
}
__device__ __forceinline__ void halfAngle(double w, double& ch, double& sh)
{
    ch = halfAngleCos(w);
    sh = kPC.sh[0];
#pragma unroll
    for (int n = 1; n < 9; ++n) sh = fma(sh, w, kPC.sh[n]);
}
__device__ __forceinline__ float halfAngleCos(float w)
{
    float c = fmaf(w, -2.605053911e-07f, 2.476010310e-05f);
    c = fmaf(c, w, -1.388836016e-03f);
    c = fmaf(c, w, 4.166663615e-02f);
    c = fmaf(c, w, -4.999999936e-01f);
    return fmaf(c, w, 1.0f);
}
__device__ __forceinline__ void halfAngle(float w, float& ch, float& sh)
{
    ch = halfAngleCos(w);
    float s = fmaf(w, 2.605095804e-06f, -1.980901230e-04f);
    s = fmaf(s, w, 8.333050103e-03f);
    s = fmaf(s, w, -1.666665795e-01f);
    sh = fmaf(s, w, 9.999999957e-01f);
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

// Transpose of the 32 x 32 bit matrix whose row l is lane l's word.
__device__ __forceinline__ unsigned transpose32(unsigned m, int lane)
{
    unsigned keep = 0x0000ffffu;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1)
    {
        unsigned const v = __shfl_xor_sync(kFull, m, d);
        m = (lane & d) ? ((m & ~keep) | ((v & ~keep) >> d))
                       : ((m & keep) | ((v & keep) << d));
        keep ^= keep << (d >> 1);
    }
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
    R const e = expScaled(expScale<R>(m.center), d * d, tab);
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
                                          unsigned short* orig,
                                          unsigned* sort,
                                          Staged<R> const& S)
{
    bool const sorted = T.sorted[h.ec] != 0;
    if (sorted)
    {
        // Keys that order the neighbors of an element by distance.
        for (int t = tm.tid; t < h.cnt; t += Team<WPA>::kThreads)
            sort[t] = __float_as_uint((float)L.dd[h.beg + t]);
        Team<WPA>::sync();
    }
    int const cs = S.cs, cnt = h.cnt, ec = h.ec;
    int const nf = T.fcBeg[ec + 1] - T.fcBeg[ec];
    int const nrad = T.radBeg[ec + 1] - T.radBeg[ec];
    for (int e = tm.tid; e <= cnt; e += Team<WPA>::kThreads)
    {
        int t = e;                  // place of entry e
        if (t == cnt)
        {
            R const far = R(T.farAway);
            S.rec[t] = Rec<R>{far, R(0), R(0), R(1) / far, R(0), far * far};
            for (int f = 1; f < nf; ++f) S.fc[(f - 1) * cs + t] = R(0);
            for (int f = 0; f < (DERIV ? 2 : 1) * nrad; ++f)
                S.rad[f * cs + t] = R(0);
            break;
        }
        double const d = L.dd[h.beg + e];
        double const id = 1.0 / d;
        R const r = R(d), ir = R(id);
        R const x = R(L.dx[h.beg + e]), y = R(L.dy[h.beg + e]),
                z = R(L.dz[h.beg + e]);
        int el = 0;
        if (DERIV || T.anyWeighted || sorted)
            while (e >= h.eb[el + 1]) ++el;
        if (sorted)
        {
            unsigned const mine = sort[e];
            t = h.eb[el];
            int const q1 = h.eb[el + 1];
#pragma unroll 4
            for (int q = h.eb[el]; q < q1; ++q)
                t += (sort[q] < mine || (sort[q] == mine && q < e)) ? 1 : 0;
            if (DERIV) orig[t] = (unsigned short)e;
        }
        R const r2 = x * x + y * y + z * z;
        // Neighbors beyond the narrow cutoff are nobody's partners.
        pos[t] = (float)r2 < maskRc2(T, ec, sizeof(R) == 8)
            ? make_float4((float)x, (float)y, (float)z, 0.0f)
            : make_float4(1e18f, 0.0f, 0.0f, 1.0f);
        R f0 = R(0);
        R const Z = T.anyWeighted ? R(P.atomicNumber[el]) : R(1);
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
            S.rad[(DERIV ? 2 * f : f) * cs + t] = v;
            if (DERIV) S.rad[(2 * f + 1) * cs + t] = dv * ir;
        }
        if (!DERIV) continue;
        double al = 0.0;
        R fc = R(0), dfc = R(0), ZZ = R(1);
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
            al += (double)((C[pr.cell] * ZZ) * dv);
        }
        arad[t] = R(al * id);
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
// The usual case, all of one unit p2, runs without branches.
template <typename R, bool DERIV>
__device__ __forceinline__ void compShapes(SFParams const& P,
                                           PairUnit const& un,
                                           PairShape const* sh, R theta,
                                           R* phi, R* psi)
{
    int const ns = un.ns;
    if (un.core == CC_POLY2)
    {
#pragma unroll
        for (int s = 0; s < kPairCompShapes; ++s)
        {
            phi[s] = R(0);
            if (DERIV) psi[s] = R(0);
            if (s < ns)
            {
                R const sc = R(sh[s].scale);
                R const v = (theta - R(sh[s].center)) * sc;
                R const x = v < R(0) ? -v : v;
                R const f = ((R(15) - R(6) * x) * x - R(10)) * (x * x * x)
                          + R(1);
                phi[s] = x < R(1) ? f : R(0);
                if (DERIV)
                {
                    // d/dx = -30 x^2 (1 - x)^2, times the sign of v.
                    R const y = x - x * x;
                    R const d = (v * (R(1) - x)) * y;
                    psi[s] = x < R(1) ? (R(-30) * sc) * d : R(0);
                }
            }
        }
        return;
    }
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
        for (int j = threadIdx.x; j < kPairExpSize; j += kT)
            tab[j] = kPairExp2[j];
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
    R*        red;        // 8 x 33 lane sums
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

// Adds the lanes' sums of N cells to the warp's values: eight cells at a
// time through shared memory, lane (row, quarter) adds eight lanes of its
// cell, then the quarters are added.
template <typename R, int N>
__device__ __forceinline__ void flushCells(Walk<R> const& w, R const (&acc)[N],
                                           int cell0, int cells)
{
#pragma unroll
    for (int c0 = 0; c0 < N; c0 += 8)
    {
        if (c0 < cells)
        {
#pragma unroll
            for (int c = 0; c < 8; ++c)
                if (c0 + c < N) w.red[c * 33 + w.lane] = acc[c0 + c];
            __syncwarp();
            int const row = w.lane >> 2;
            R v = R(0);
#pragma unroll
            for (int q = 0; q < 8; ++q)
                v += w.red[row * 33 + (w.lane & 3) * 8 + q];
            v += __shfl_xor_sync(kFull, v, 1);
            v += __shfl_xor_sync(kFull, v, 2);
            if ((w.lane & 3) == 0 && c0 + row < cells)
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
    for (int a = 0; a < NR; ++a) e2[a] = expScale<R>(tb.r[u.run + a].center);
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
    // Slots the unit does not have hold zeros and have no cells.
    flushCells<R, NZ * NR * 2>(w, acc, u.cell, pairUnitCells<PK_POW2>(u));
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
        e2[a] = expScale<R>(tb.r[u.run + min(a, nr - 1)].center);
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
                R const v = m * expScaled(expScale<R>(runs[a].center), x,
                                          w.W.tab);
#pragma unroll
                for (int q = 0; q < S; ++q) acc[a * S + q] += v * phi[q];
            }
    });
    flushCells<R, kPairGenRuns * S>(w, acc, u.cell,
                                    pairUnitCells<PK_GENERAL>(u));
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
    int const nr = u.nr, cs = w.W.cs;
    PairRun const* const runs = tb.r + u.run;
    PairShape const* const sh = tb.s + u.shape;
    walkPairs<R, NARROW>(w, [&](int tt, int kk) {
        Rec<R> const A = w.W.rec[tt], B = w.W.rec[kk];
        R const c = (A.x * B.x + A.y * B.y + A.z * B.z) * (A.ir * B.ir);
        bool const ok = c > R(-1) && c < R(1);
        R phi[S];
        compShapes<R, false>(P, u, sh, acos(ok ? c : R(0)), phi,
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
                R const* tab = w.W.rad + r.slot * cs;
                R v = tab[tt] * tab[kk];
                // Neighbors come by distance: windows that end early are
                // zero for most whole batches.
                if (!__any_sync(kFull, v != R(0))) continue;
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
    flushCells<R, N>(w, acc, u.cell, pairUnitCells<PK_COMPACT>(u));
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
// The sets {1}, {1, 4}, {1, 2, 4} and {1, 2, 4, 16} of zeta are compiled
// without tests of the slots (a test is a branch, which keeps the compiler
// from overlapping the slots' work with the exponentials'); other sets test
// them.
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
    w.red = reinterpret_cast<R*>(mine + L.oRed) + warp * 8 * 33;
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
        stageAtom<R, CT, WPA, false>(
            P, T, L, h, tm, pos, dist, (R*)nullptr, (R const*)nullptr, tb.q,
            (unsigned short*)nullptr,
            reinterpret_cast<unsigned*>(mine + L.oSort), w.W);
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

// Owner j's values and its sums (FP64 in all forms): al along dr_ij and the vector (vx, vy, vz)
// of the coefficients along dr_ik times dr_ik.
template <typename R>
struct Owner
{
    R      x, y, z, ir, r2;
    double al, vx, vy, vz;
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
    for (int a = 0; a < NR; ++a) e2[a] = expScale<R>(tb.r[u.run + a].center);
    R const a2q = R(u.a2q), qf = R(u.qf), rc2 = R(u.rc2);
    bool const exact = u.exactMask != 0;
    int const slot = u.fcSlot, none = W.cs - 1;
    R const of = fcOf(W, slot, p.t), odf = W.dfc[slot * W.cs + p.t];
    unsigned const mask = MASK ? (unsigned)MASK : u.mask;
    double al = 0.0, vx = 0.0, vy = 0.0, vz = 0.0;
    P2 const* const C2 = reinterpret_cast<P2 const*>(C);
    R h1[NR];             // zeta = 1: d/dcos is a constant
#pragma unroll
    for (int a = 0; a < NR; ++a) h1[a] = C2[a].y - C2[a].x;
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
                    if (z == 0) h[a] = h1[a];
                    else h[a] = (h[a] + c.y * hp) - c.x * hm;
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
        al += (double)a1;
        vx += (double)(ga * B.x);
        vy += (double)(ga * B.y);
        vz += (double)(ga * B.z);
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
        e2[a] = expScale<R>(tb.r[u.run + min(a, nr - 1)].center);
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
    double al = 0.0, vx = 0.0, vy = 0.0, vz = 0.0;
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
        al += (double)a1;
        vx += (double)(ga * B.x);
        vy += (double)(ga * B.y);
        vz += (double)(ga * B.z);
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
    double al = 0.0, vx = 0.0, vy = 0.0, vz = 0.0;
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
            R const v = expScaled(expScale<R>(runs[a].center), x, W.tab);
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
        al += (double)a1;
        vx += (double)(ga * B.x);
        vy += (double)(ga * B.y);
        vz += (double)(ga * B.z);
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
    int const nr = u.nr, cs = W.cs, none = cs - 1;
    PairRun const* const runs = tb.r + u.run;
    PairShape const* const sh = tb.s + u.shape;
    P2 const* const C2 = reinterpret_cast<P2 const*>(C);
    double al = 0.0, vx = 0.0, vy = 0.0, vz = 0.0;
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
        compShapes<R, true>(P, u, sh, acos(c), phi, psi);
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
            R const rj = tab[p.t], drj = tab[cs + p.t];
            // Neighbors come by distance: windows that end early are zero
            // for most whole steps.
            if (!__any_sync(kFull, rk != R(0)
                                       && (rj != R(0) || drj != R(0))))
                continue;
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
        al += (double)(x1 - (mh * dot) * (o.ir * o.ir) + x3);
        vx += (double)(ga * B.x);
        vy += (double)(ga * B.y);
        vz += (double)(ga * B.z);
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
// The sets {1}, {1, 4}, {1, 2, 4} and {1, 2, 4, 16} of zeta are compiled
// without tests of the slots (52 functions, 6,144 atoms, FP64: 0.90 -> 0.71
// ms); other sets test them.
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
    unsigned short* const orig =
        reinterpret_cast<unsigned short*>(mine + L.oOrig);
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
                C[k] = ce.sf >= 0 ? R((double)row[ce.sf] * ce.fn) : R(0);
            }
        }
        Tm::sync();
        stageAtom<R, CT, WPA, true>(
            P, T, L, h, tm, pos, (R*)nullptr, arad, C, tb.q, orig,
            reinterpret_cast<unsigned*>(mine + L.oSort), W);
        Tm::sync();
        // Validity masks (narrow units): (32 rows, word) blocks on and above
        // the diagonal, those below are their transposes.
        if (anyNarrow)
        {
            float const rc2 = maskRc2(T, ec, sizeof(R) == 8);
            int const nb = (cnt + 31) >> 5;
            int task = 0;
            for (int rb = 0; rb < nb; ++rb)
                for (int q = rb; q < nb; ++q)
                {
                    if ((task++ & (WPA - 1)) != warp) continue;
                    int const t = (rb << 5) + lane;
                    unsigned m = maskWord(pos, t, q, cnt, rc2);
                    if (q == rb)
                    {
                        m &= ~(1u << lane);
                        if (t < cnt) bits[t * words + q] = m;
                        continue;
                    }
                    bits[t * words + q] = m;
                    m = transpose32(m, lane);
                    int const u = (q << 5) + lane;
                    if (u < cnt) bits[u * words + rb] = m;
                }
            Tm::sync();
            // Per row the partners of the elements below each one and in
            // all, and the key that orders the owners.
            for (int t = tm.tid; t < cnt; t += Tm::kThreads)
            {
                int total = 0, e = 0;
                for (int q = 0; q < nb; ++q)
                {
                    unsigned const m = bits[t * words + q];
                    for (; e < ne && h.eb[e] < (q + 1) << 5; ++e)
                        pre[t * (ne + 1) + e] = (unsigned short)(
                            total + __popc(m & ((1u << (h.eb[e] & 31)) - 1u)));
                    total += __popc(m);
                }
                for (; e <= ne; ++e)
                    pre[t * (ne + 1) + e] = (unsigned short)total;
                key[t] = ((unsigned)total << 16) | (0xffffu - (unsigned)t);
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
                Al += o.al;
                Vx += o.vx;
                Vy += o.vy;
                Vz += o.vz;
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
                long const e = beg + (T.sorted[ec] ? (int)orig[t] : t);
                double const f = Al * a[e] + v;
                L.pairF[e * 3 + sl] = f;
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
