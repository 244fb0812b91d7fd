// Neighbor list on the device: Structure::remap + Structure::calculateNeighborList
// (libnnp/Structure.cpp:287-399, 1214-1247) with identical neighbor sets.
//
// Bit-exactness.  The reference tests, for every atom pair (i, j) and image
// shift bc in [-pbc, pbc]^3 (pbc from Structure::calculatePbcCopies),
//     dr = r_i - r_j + bc0 * a + bc1 * b + bc2 * c        (Vec3D ops, ISO C++)
//     dr.norm2() <= rc^2,  norm2 = x*x + y*y + z*z
// All products and sums below use __dmul_rn / __dadd_rn / __dsub_rn in that
// association, so no FMA contraction can change a rounding; sqrt is IEEE.
//
// Order.  Each atom's list is stored sorted by the key
//     ((element(j) * N + j) * nimg + img),
//     img = ((bc0 + p0)(2 p1 + 1) + bc1 + p1)(2 p2 + 1) + bc2 + p2
// i.e. grouped by neighbor element and, inside an element, in the reference's
// own (j ascending; bc0, bc1, bc2 ascending) order.  Element grouping gives the
// symmetry-function kernel contiguous per-element neighbor ranges.
//
// Three enumeration paths produce the same set:
//  * cell path: cells at least rc wide along every box vector, 27-cell stencil
//    with periodic wrap.  Used when every box vector's perpendicular width
//    exceeds rc (then pbc = 1) and every atom lies inside the cell (fractional
//    coordinates in [0, 1], true after remap): all neighbors then have
//    |bc| <= 1 and sit in adjacent cells.  An FP32 distance decides away from
//    the cutoff.  Hits are ranked by key per atom.
//  * brute path: all (j, bc) candidates in key order, the reference's own
//    enumeration; used for atoms outside the cell, open structures above the
//    lane path's size and boxes with more than 128 images.
//  * lane path (nlbLaneKernel): batches, structures of up to 640 atoms and
//    boxes that cannot be cut into cells, with up to 128 images; only the
//    images in reach are walked.
#include "device_common.cuh"
#include "kernels.h"

namespace n2p2b
{

// Structure::remap (libnnp/Structure.cpp:1223-1247) for one atom.
__device__ __forceinline__ void remapAtom(double r[3], double const box[3][3],
                                          double const inv[3][3])
{
    double f[3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
        f[k] = __dadd_rn(__dadd_rn(__dmul_rn(r[0], inv[0][k]),
                                   __dmul_rn(r[1], inv[1][k])),
                         __dmul_rn(r[2], inv[2][k]));
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
        if (f[k] > 1.0) f[k] = __dsub_rn(f[k], (double)(int)f[k]);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
        if (f[k] < 0.0)
            f[k] = __dadd_rn(f[k], __dsub_rn(1.0, (double)(int)f[k]));
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
        if (f[k] == 1.0) f[k] = 0.0;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
        r[k] = __dadd_rn(__dadd_rn(__dmul_rn(f[0], box[0][k]),
                                   __dmul_rn(f[1], box[1][k])),
                         __dmul_rn(f[2], box[2][k]));
    }
}

// Input positions (physical units) -> positions in computing units
// (remap, then Atom::toNormalizedUnits: r *= convLength), plus cell binning.
__global__ void nlPrepareKernel(int n, double const* __restrict__ posIn,
                                int doRemap, int normalize, double convLength,
                                PhysBox pb, NLParams p,
                                double* __restrict__ pos,
                                int* __restrict__ cellOf,
                                int* __restrict__ cellCount,
                                int* __restrict__ status)
{
    int const i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double r[3] = {posIn[3 * i + 0], posIn[3 * i + 1], posIn[3 * i + 2]};
    if (doRemap) remapAtom(r, pb.box, pb.invbox);
    if (normalize)
    {
        r[0] = __dmul_rn(r[0], convLength);
        r[1] = __dmul_rn(r[1], convLength);
        r[2] = __dmul_rn(r[2], convLength);
    }
    pos[3 * i + 0] = r[0];
    pos[3 * i + 1] = r[1];
    pos[3 * i + 2] = r[2];
    if (p.ncell[0] > 0)
    {
        int c[3];
        bool inside = true;
#pragma unroll
        for (int k = 0; k < 3; ++k)
        {
            double const f = r[0] * p.invbox[0][k] + r[1] * p.invbox[1][k]
                           + r[2] * p.invbox[2][k];
            if (!(f >= -1e-12 && f <= 1.0 + 1e-12)) inside = false;
            int ck = (int)floor(f * p.ncell[k]);
            c[k] = min(max(ck, 0), p.ncell[k] - 1);
        }
        if (!inside) atomicOr(&status[ST_FLAGS], FLAG_OUTSIDE_CELL);
        int const cell = (c[0] * p.ncell[1] + c[1]) * p.ncell[2] + c[2];
        cellOf[i] = cell;
        atomicAdd(&cellCount[cell], 1);
    }
}

// Atoms by cell, with FP32 positions for the distance test (one 16-byte load
// per candidate).  Counts the cells down: cellCount is zero afterwards.
__global__ void nlBinKernel(int n, double const* __restrict__ pos,
                            int const* __restrict__ elem,
                            int const* __restrict__ cellOf,
                            int const* __restrict__ cellStart,
                            int* __restrict__ cellCount,
                            float4* __restrict__ cellPos,
                            int8_t* __restrict__ cellEl)
{
    int const i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int const c = cellOf[i];
    int const at = cellStart[c] + atomicSub(&cellCount[c], 1) - 1;
    cellPos[at] = make_float4((float)pos[3 * i], (float)pos[3 * i + 1],
                              (float)pos[3 * i + 2], __int_as_float(i));
    cellEl[at] = (int8_t)elem[i];
}

// Exact reference displacement and cutoff test for candidate (j, bc).
__device__ __forceinline__ bool nlTest(NLParams const& p, double const ri[3],
                                       double const* __restrict__ pos, int j,
                                       int b0, int b1, int b2, double dr[3])
{
    double const db0 = (double)b0, db1 = (double)b1, db2 = (double)b2;
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
        double v = __dsub_rn(ri[k], pos[3 * j + k]);
        if (p.periodic)
        {
            v = __dadd_rn(v, __dmul_rn(db0, p.box[0][k]));
            v = __dadd_rn(v, __dmul_rn(db1, p.box[1][k]));
            v = __dadd_rn(v, __dmul_rn(db2, p.box[2][k]));
        }
        dr[k] = v;
    }
    double const n2 = __dadd_rn(__dadd_rn(__dmul_rn(dr[0], dr[0]),
                                          __dmul_rn(dr[1], dr[1])),
                                __dmul_rn(dr[2], dr[2]));
    return n2 <= p.rc2;
}

__device__ __forceinline__ int imgIndex(NLParams const& p, int b0, int b1,
                                        int b2)
{
    return ((b0 + p.pbc[0]) * (2 * p.pbc[1] + 1) + (b1 + p.pbc[1]))
           * (2 * p.pbc[2] + 1) + (b2 + p.pbc[2]);
}

__device__ __forceinline__ void imgDecode(NLParams const& p, int img, int& b0,
                                          int& b1, int& b2)
{
    int const n2 = 2 * p.pbc[2] + 1;
    int const n1 = 2 * p.pbc[1] + 1;
    b2 = img % n2 - p.pbc[2];
    img /= n2;
    b1 = img % n1 - p.pbc[1];
    b0 = img / n1 - p.pbc[0];
}

__device__ __forceinline__ unsigned long long nlKey(int ej, int j, int img,
                                                    int n, int nimg)
{
    return ((unsigned long long)ej * (unsigned long long)n
            + (unsigned long long)j) * (unsigned long long)nimg
           + (unsigned long long)img;
}

// A list's entries: key order, displacements, owner.
struct ListOut
{
    unsigned long long* key;
    int*                nbrIdx;
    int8_t*             nbrEl;
    double*             dx;
    double*             dy;
    double*             dz;
    double*             dd;
    int*                entryAtom;
};

__device__ __forceinline__ void writeEntry(ListOut const& o, long at, int i,
                                           unsigned long long key, int j,
                                           int ej, double const dr[3])
{
    double const n2 = __dadd_rn(__dadd_rn(__dmul_rn(dr[0], dr[0]),
                                          __dmul_rn(dr[1], dr[1])),
                                __dmul_rn(dr[2], dr[2]));
    o.key[at] = key;
    o.nbrIdx[at] = j;
    o.nbrEl[at] = (int8_t)ej;
    o.dx[at] = dr[0];
    o.dy[at] = dr[1];
    o.dz[at] = dr[2];
    o.dd[at] = __dsqrt_rn(n2);
    o.entryAtom[at] = i;
}

// ---------------------------------------------------------------------------
// Cell path.  Warp per atom.  MODE 0 counts hits (total and per element);
// MODE 1 collects the hits' keys, ranks them and writes the entries.
//
// Bound by the distance tests (6 to 7 candidates per neighbor).  The cells of
// one (c0, c1) row lie one after another in memory, so the 27 cells are 9
// runs of three cells (and the wrapped ends): a lane holds a run, the warp
// walks it 32 candidates at a time.  An FP32 distance decides outside
// rc^2 -+ slack: coordinates inside the cell are at most B = sum_k |a_k|, an
// image shift as well, so a component of the difference errs by less than
// 32 B 2^-24 and r^2 near the cutoff by 6 rc err + 3 err^2 (slack: four
// times that, at least 1e-4 rc^2); between them nlTest does.  Up to
// kCellHits keys of 32 bits are ranked in shared memory (one pass of 16-byte
// reads for four keys a lane), others in keyTmp.  24,576 water atoms, both
// modes, ranks and entries: 0.37 ms with an FP64 test of every candidate and
// 64-bit keys ranked in global memory, 0.20 ms so.
// ---------------------------------------------------------------------------
constexpr int kCellHits = 256, kCellWarps = 4;

template <int MODE>
__global__ void __launch_bounds__(32 * kCellWarps)
nlCellKernel(int n, __grid_constant__ NLParams const p, int numElements,
             double const* __restrict__ pos, int const* __restrict__ elem,
             int const* __restrict__ cellOf,
             int const* __restrict__ cellStart,
             float4 const* __restrict__ cellPos,
             int8_t const* __restrict__ cellEl, int* __restrict__ nbrCount,
             int* __restrict__ nbrCountElem, int const* __restrict__ nbrOff,
             unsigned long long* __restrict__ keyTmp, ListOut const out,
             int const* __restrict__ status)
{
    __shared__ __align__(16) unsigned found[MODE == 1 ? kCellWarps : 1]
                                           [MODE == 1 ? kCellHits : 4];
    __shared__ unsigned order[MODE == 1 ? kCellWarps : 1]
                             [MODE == 1 ? kCellHits : 1];
    if (status[ST_FLAGS] & (FLAG_OUTSIDE_CELL | FLAG_ABORT)) return;
    int const lane = threadIdx.x & 31;
    int const warp = threadIdx.x >> 5;
    int const i = blockIdx.x * kCellWarps + warp;
    if (i >= n) return;
    double const ri[3] = {pos[3 * i], pos[3 * i + 1], pos[3 * i + 2]};
    long const base = MODE == 1 ? (long)nbrOff[i] : 0;
    int const cnt = MODE == 1 ? nbrOff[i + 1] - (int)base : 0;
    bool const small = cnt <= kCellHits
        && (unsigned long long)numElements * n * p.nimg < 0xffffffffull;
    // Lane 3 r + k < 27: row r of the stencil; k = 0 its cells inside the
    // box, k = 1 and 2 the ones wrapped below and above.
    int first = 0, len = 0, img = 0;
    float sx = 0.0f, sy = 0.0f, sz = 0.0f;
    if (lane < 27)
    {
        int const cell = cellOf[i];
        int const c2 = cell % p.ncell[2];
        int v[2] = {cell / (p.ncell[2] * p.ncell[1]) + lane / 9 - 1,
                    (cell / p.ncell[2]) % p.ncell[1] + (lane / 3) % 3 - 1};
        int bc[3] = {0, 0, 0};
#pragma unroll
        for (int k = 0; k < 2; ++k)
        {
            if (v[k] < 0) { v[k] += p.ncell[k]; bc[k] = 1; }
            else if (v[k] >= p.ncell[k]) { v[k] -= p.ncell[k]; bc[k] = -1; }
        }
        int const row = (v[0] * p.ncell[1] + v[1]) * p.ncell[2];
        int lo = max(c2 - 1, 0), hi = min(c2 + 1, p.ncell[2] - 1);
        if (lane % 3 == 1)
        {
            bc[2] = 1;
            lo = p.ncell[2] - 1;
            hi = c2 == 0 ? lo : lo - 1;
        }
        if (lane % 3 == 2)
        {
            bc[2] = -1;
            lo = 0;
            hi = c2 == p.ncell[2] - 1 ? 0 : -1;
        }
        if (lo <= hi)
        {
            first = cellStart[row + lo];
            len = cellStart[row + hi + 1] - first;
        }
        img = imgIndex(p, bc[0], bc[1], bc[2]);
        float const b0 = (float)bc[0], b1 = (float)bc[1], b2 = (float)bc[2];
        sx = b0 * (float)p.box[0][0] + b1 * (float)p.box[1][0]
           + b2 * (float)p.box[2][0];
        sy = b0 * (float)p.box[0][1] + b1 * (float)p.box[1][1]
           + b2 * (float)p.box[2][1];
        sz = b0 * (float)p.box[0][2] + b1 * (float)p.box[1][2]
           + b2 * (float)p.box[2][2];
    }
    float const x = (float)ri[0], y = (float)ri[1], z = (float)ri[2];
    float const rc2 = (float)p.rc2;
    float B = 0.0f;
#pragma unroll
    for (int c = 0; c < 3; ++c)
        B = fmaxf(B, fabsf((float)p.box[0][c]) + fabsf((float)p.box[1][c])
                     + fabsf((float)p.box[2][c]));
    float const err = 32.0f * B * 5.9604645e-8f;
    float const slack = fmaxf(1e-4f * rc2, 4.0f * (6.0f * sqrtf(rc2) * err
                                                   + 3.0f * err * err));
    float const above = rc2 + slack, below = rc2 - slack;
    int const home = imgIndex(p, 0, 0, 0);
    // Hits per element: 16 bits each.
    unsigned long long cntElem[(kMaxElem + 3) / 4] = {};
    int total = 0;
    unsigned runs = __ballot_sync(0xffffffffu, len > 0);
    while (runs)
    {
        int const src = __ffs(runs) - 1;
        runs &= runs - 1;
        int const f = __shfl_sync(0xffffffffu, first, src);
        int const m = __shfl_sync(0xffffffffu, len, src);
        int const im = __shfl_sync(0xffffffffu, img, src);
        float const x0 = x + __shfl_sync(0xffffffffu, sx, src);
        float const y0 = y + __shfl_sync(0xffffffffu, sy, src);
        float const z0 = z + __shfl_sync(0xffffffffu, sz, src);
#pragma unroll 4
        for (int q = lane; q < ((m + 31) & ~31); q += 32)
        {
            bool hit = false;
            int j = 0;
            if (q < m)
            {
                float4 const a = cellPos[f + q];
                j = __float_as_int(a.w);
                float const dx = x0 - a.x, dy = y0 - a.y, dz = z0 - a.z;
                float const r2 = dx * dx + dy * dy + dz * dz;
                hit = r2 <= above && !(j == i && im == home);
                if (hit && r2 >= below)
                {
                    int b0, b1, b2;
                    double dr[3];
                    imgDecode(p, im, b0, b1, b2);
                    hit = nlTest(p, ri, pos, j, b0, b1, b2, dr);
                }
            }
            unsigned const hits = __ballot_sync(0xffffffffu, hit);
            if (hit)
            {
                int const ej = cellEl[f + q];
                if (MODE == 0)
                {
#pragma unroll
                    for (int k = 0; k < (kMaxElem + 3) / 4; ++k)
                        if (ej >> 2 == k)
                            cntElem[k] += 1ull << (16 * (ej & 3));
                }
                else
                {
                    int const at = total
                                 + __popc(hits & ((1u << lane) - 1u));
                    unsigned long long const key =
                        nlKey(ej, j, im, n, p.nimg);
                    if (at < cnt)
                    {
                        if (small) found[warp][at] = (unsigned)key;
                        else keyTmp[base + at] = key;
                    }
                }
            }
            total += __popc(hits);
        }
    }
    if (MODE == 0)
    {
        for (int e = 0; e < numElements; ++e)
        {
            unsigned long long w = 0;
#pragma unroll
            for (int k = 0; k < (kMaxElem + 3) / 4; ++k)
                if (e >> 2 == k) w = cntElem[k];
            int const v = __reduce_add_sync(
                0xffffffffu, (int)(w >> (16 * (e & 3))) & 0xffff);
            if (lane == 0) nbrCountElem[(long)i * numElements + e] = v;
        }
        if (lane == 0) nbrCount[i] = total;
        return;
    }
    unsigned* const mine = found[warp];
    unsigned* const sorted = order[warp];
    if (small)
    {
        // Pad to a whole 16-byte word with a key above all.
        if (lane < 4 && cnt + lane < ((cnt + 3) & ~3))
            mine[cnt + lane] = 0xffffffffu;
        __syncwarp();
        for (int t0 = 0; t0 < cnt; t0 += 128)
        {
            unsigned k[4];
            int r[4] = {0, 0, 0, 0};
#pragma unroll
            for (int c = 0; c < 4; ++c)
            {
                int const t = t0 + 32 * c + lane;
                k[c] = t < cnt ? mine[t] : 0u;
            }
            for (int u = 0; u < cnt; u += 4)
            {
                uint4 const v = *reinterpret_cast<uint4 const*>(mine + u);
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    r[c] += (v.x < k[c]) + (v.y < k[c]) + (v.z < k[c])
                          + (v.w < k[c]);
            }
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (t0 + 32 * c + lane < cnt) sorted[r[c]] = k[c];
        }
    }
    else
    {
        __syncwarp();
        for (int t = lane; t < cnt; t += 32)
        {
            unsigned long long const k = keyTmp[base + t];
            int r = 0;
            for (int u = 0; u < cnt; ++u) r += (keyTmp[base + u] < k);
            out.key[base + r] = k;
        }
    }
    __syncwarp();
    for (int t = lane; t < cnt; t += 32)
    {
        unsigned long long key;
        int j, im;
        if (small)
        {
            unsigned const k = sorted[t];
            unsigned const q = k / (unsigned)p.nimg;
            im = (int)(k - q * (unsigned)p.nimg);
            j = (int)(q % (unsigned)n);
            key = k;
        }
        else
        {
            key = out.key[base + t];
            unsigned long long const q = key / (unsigned long long)p.nimg;
            im = (int)(key - q * (unsigned long long)p.nimg);
            j = (int)(q % (unsigned long long)n);
        }
        int b0, b1, b2;
        imgDecode(p, im, b0, b1, b2);
        double dr[3];
        nlTest(p, ri, pos, j, b0, b1, b2, dr);
        writeEntry(out, base + t, i, key, j, elem[j], dr);
    }
}

// ---------------------------------------------------------------------------
// Brute path.  Warp per atom, candidates enumerated in key order:
// element-major, then j ascending (atomsByElem is sorted per element), then
// image.  MODE 0 counts; MODE 1 writes the entries.
// `onlyIfOutside`: the cell path was eligible, so run only if some atom was
// found outside the cell.
// ---------------------------------------------------------------------------
template <int MODE>
__global__ void nlBruteKernel(int n, NLParams p, int numElements,
                              int onlyIfOutside,
                              double const* __restrict__ pos,
                              int const* __restrict__ atomsByElem,
                              ElemStarts es,
                              int* __restrict__ nbrCount,
                              int* __restrict__ nbrCountElem,
                              int const* __restrict__ nbrOff,
                              ListOut const out,
                              int const* __restrict__ status)
{
    int const flags = status[ST_FLAGS];
    if (flags & FLAG_ABORT) return;
    if (onlyIfOutside && !(flags & FLAG_OUTSIDE_CELL)) return;
    int const lane = threadIdx.x & 31;
    int const i = (int)((blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5);
    if (i >= n) return;
    double const ri[3] = {pos[3 * i], pos[3 * i + 1], pos[3 * i + 2]};
    int total = 0;
    long const base = (MODE == 1) ? (long)nbrOff[i] : 0;
    int const nimg = p.nimg;
    for (int e = 0; e < numElements; ++e)
    {
        int const eb = es.start[e];
        long const ncand = (long)(es.start[e + 1] - eb) * nimg;
        int cntE = 0;
        for (long c0 = 0; c0 < ncand; c0 += 32)
        {
            long const c = c0 + lane;
            bool hit = false;
            int j = 0, img = 0;
            double dr[3];
            if (c < ncand)
            {
                j = atomsByElem[eb + (int)(c / nimg)];
                img = (int)(c % nimg);
                int b0, b1, b2;
                imgDecode(p, img, b0, b1, b2);
                if (!(j == i && b0 == 0 && b1 == 0 && b2 == 0))
                    hit = nlTest(p, ri, pos, j, b0, b1, b2, dr);
            }
            unsigned const m = __ballot_sync(0xffffffffu, hit);
            if (MODE == 1 && hit)
            {
                int const off = total + __popc(m & ((1u << lane) - 1u));
                writeEntry(out, base + off, i, nlKey(e, j, img, n, nimg), j,
                           e, dr);
            }
            total += __popc(m);
            cntE += __popc(m);
        }
        if (MODE == 0 && lane == 0)
            nbrCountElem[(long)i * numElements + e] = cntE;
    }
    if (MODE == 0 && lane == 0) nbrCount[i] = total;
}

// Exclusive scan of per-atom counts into offsets (n + 1 entries), total and
// maximum into the status words; flags overflow against `capacity`.
// Single block: tiles of 8,192 counts, eight per thread, warp scans.  cnt and
// off are 16-byte aligned (cudaMalloc'ed arrays).
__global__ void __launch_bounds__(1024)
nlScanKernel(int n, int const* __restrict__ cnt, int* __restrict__ off,
             long capacity, int* __restrict__ status)
{
    __shared__ int sWarp[32];
    __shared__ int sMax[32];
    constexpr int kPer = 8;               // consecutive counts per thread
    int const t = threadIdx.x, lane = t & 31, warp = t >> 5;
    long base = 0;
    int mx = 0;
    // A tile's counts are fetched while the tile before it is scanned.
    int v[kPer], nx[kPer];
    auto fetch = [&](int (&x)[kPer], int b) {
        if (b + kPer <= n)
        {
            int4 const p = *reinterpret_cast<int4 const*>(cnt + b);
            int4 const q = *reinterpret_cast<int4 const*>(cnt + b + 4);
            x[0] = p.x; x[1] = p.y; x[2] = p.z; x[3] = p.w;
            x[4] = q.x; x[5] = q.y; x[6] = q.z; x[7] = q.w;
        }
        else
        {
#pragma unroll
            for (int k = 0; k < kPer; ++k) x[k] = b + k < n ? cnt[b + k] : 0;
        }
    };
    fetch(nx, t * kPer);
    for (int tile = 0; tile < n; tile += 1024 * kPer)
    {
        int const b = tile + t * kPer;
        int s = 0;
#pragma unroll
        for (int k = 0; k < kPer; ++k)
        {
            v[k] = nx[k];
            mx = max(mx, v[k]);
            s += v[k];
        }
        if (tile < n - 1024 * kPer) fetch(nx, b + 1024 * kPer);
        int incl = s;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1)
        {
            int const u = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += u;
        }
        if (lane == 31) sWarp[warp] = incl;
        __syncthreads();
        if (warp == 0)
        {
            int w = sWarp[lane];
#pragma unroll
            for (int d = 1; d < 32; d <<= 1)
            {
                int const u = __shfl_up_sync(0xffffffffu, w, d);
                if (lane >= d) w += u;
            }
            sWarp[lane] = w;
        }
        __syncthreads();
        long run = base + (warp > 0 ? sWarp[warp - 1] : 0) + incl - s;
        base += sWarp[31];
        int o[kPer];
#pragma unroll
        for (int k = 0; k < kPer; ++k)
        {
            o[k] = (int)run;
            run += v[k];
        }
        if (b + kPer <= n)
        {
            *reinterpret_cast<int4*>(off + b) = make_int4(o[0], o[1], o[2],
                                                          o[3]);
            *reinterpret_cast<int4*>(off + b + 4) = make_int4(o[4], o[5],
                                                              o[6], o[7]);
        }
        else
        {
#pragma unroll
            for (int k = 0; k < kPer; ++k)
                if (b + k < n) off[b + k] = o[k];
        }
        __syncthreads();
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) sMax[warp] = mx;
    __syncthreads();
    if (warp == 0)
    {
        int const m = __reduce_max_sync(0xffffffffu, sMax[lane]);
        if (lane == 0)
        {
            off[n] = (int)min(base, (long)0x7fffffff);
            if (status)
            {
                status[ST_TOTAL_NBR] = (int)min(base, (long)0x7fffffff);
                status[ST_MAX_NBR] = m;
                if (base > capacity)
                    status[ST_FLAGS] |= FLAG_NBR_OVERFLOW | FLAG_ABORT;
            }
        }
    }
}

// Thread per entry: position of the mirror entry (j -> i, -bc) in j's list,
// found by binary search over j's sorted keys.  Exists by symmetry: IEEE
// rounding is sign-symmetric, so the mirror displacement is exactly -dr.
__global__ void nlMirrorKernel(int n, int nimg,
                               int const* __restrict__ elem,
                               int const* __restrict__ nbrOff,
                               unsigned long long const* __restrict__ key,
                               int const* __restrict__ nbrIdx,
                               int const* __restrict__ entryAtom,
                               int* __restrict__ mirror,
                               int* __restrict__ status)
{
    if (status[ST_FLAGS] & FLAG_ABORT) return;
    long const e = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (e >= (long)nbrOff[n]) return;
    int const i = entryAtom[e];
    int const j = nbrIdx[e];
    unsigned long long const nimgU = (unsigned long long)nimg;
    int const img = (int)(key[e] % nimgU);
    unsigned long long const want = nlKey(elem[i], i, nimg - 1 - img, n, nimg);
    long lo = nbrOff[j], hi = nbrOff[j + 1];
    while (lo < hi)
    {
        long const mid = (lo + hi) >> 1;
        if (key[mid] < want) lo = mid + 1;
        else hi = mid;
    }
    if (lo < nbrOff[j + 1] && key[lo] == want)
    {
        mirror[e] = (int)lo;
    }
    else
    {
        mirror[e] = -1;
        atomicOr(&status[ST_FLAGS], FLAG_MIRROR_MISSING);
    }
}

// ---------------------------------------------------------------------------
// Host-side launchers
// ---------------------------------------------------------------------------

void launchOffsetScan(long n, int const* cnt, int* off, cudaStream_t s)
{
    nlScanKernel<<<1, 1024, 0, s>>>((int)n, cnt, off, 0x7fffffffffffffffL,
                                    nullptr);
}

void launchNeighborList(NLLaunch const& L, cudaStream_t s)
{
    int const n = L.n;
    int const tb = 256;
    int const gAtoms = (n + tb - 1) / tb;
    int const warpsPerBlock = 4;
    int const gWarp = (n + warpsPerBlock - 1) / warpsPerBlock;
    int const gCell = (n + kCellWarps - 1) / kCellWarps;
    bool const cellEligible = L.p.ncell[0] > 0;
    ListOut const out{L.key, L.nbrIdx, L.nbrEl, L.dx, L.dy, L.dz, L.dd,
                      L.entryAtom};
    if (cellEligible)
        cudaMemsetAsync(L.cellCount, 0, sizeof(int) * (size_t)L.numCells, s);
    nlPrepareKernel<<<gAtoms, tb, 0, s>>>(n, L.posIn, L.doRemap, L.normalize,
                                          L.convLength, L.pb, L.p, L.pos,
                                          L.cellOf, L.cellCount, L.status);
    if (cellEligible)
    {
        nlScanKernel<<<1, 1024, 0, s>>>(L.numCells, L.cellCount, L.cellStart,
                                        0x7fffffffL, L.cellScanStatus);
        nlBinKernel<<<gAtoms, tb, 0, s>>>(n, L.pos, L.elem, L.cellOf,
                                          L.cellStart, L.cellCount, L.cellPos,
                                          L.cellEl);
        nlCellKernel<0><<<gCell, 32 * kCellWarps, 0, s>>>(
            n, L.p, L.numElements, L.pos, L.elem, L.cellOf, L.cellStart,
            L.cellPos, L.cellEl, L.nbrCount, L.nbrCountElem, L.nbrOff,
            L.keyTmp, out, L.status);
    }
    nlBruteKernel<0><<<gWarp, 32 * warpsPerBlock, 0, s>>>(
        n, L.p, L.numElements, cellEligible ? 1 : 0, L.pos, L.atomsByElem,
        L.es, L.nbrCount, L.nbrCountElem, L.nbrOff, out, L.status);
    nlScanKernel<<<1, 1024, 0, s>>>(n, L.nbrCount, L.nbrOff, L.capacity,
                                    L.status);
    if (cellEligible)
        nlCellKernel<1><<<gCell, 32 * kCellWarps, 0, s>>>(
            n, L.p, L.numElements, L.pos, L.elem, L.cellOf, L.cellStart,
            L.cellPos, L.cellEl, L.nbrCount, L.nbrCountElem, L.nbrOff,
            L.keyTmp, out, L.status);
    nlBruteKernel<1><<<gWarp, 32 * warpsPerBlock, 0, s>>>(
        n, L.p, L.numElements, cellEligible ? 1 : 0, L.pos, L.atomsByElem,
        L.es, L.nbrCount, L.nbrCountElem, L.nbrOff, out, L.status);
    long const cap = L.capacity;
    int const gE = (int)((cap + tb - 1) / tb);
    noteLaunches(cellEligible ? 9 : 5);
    nlMirrorKernel<<<gE > 0 ? gE : 1, tb, 0, s>>>(
        n, L.p.nimg, L.elem, L.nbrOff, L.key, L.nbrIdx,
        L.entryAtom, L.mirror, L.status);
}

// ===========================================================================
// Batches of independent structures (one neighbor list per structure, all
// structures' atoms concatenated).  Every structure keeps its own box and
// image range; candidates are the atoms of the same structure only, in the
// brute path's key order, so each structure's list is exactly the one
// Structure::calculateNeighborList builds for it alone.  Keys use the
// batch-wide image stride NIMG (the largest structure's image count) so
// that they stay unique and sorted.
// ===========================================================================

__global__ void nlbPrepareKernel(int n, double const* __restrict__ posIn,
                                 int const* __restrict__ structOf,
                                 BatchStruct const* __restrict__ bs,
                                 __grid_constant__ BatchStruct const one,
                                 int normalize, double convLength,
                                 double* __restrict__ pos)
{
    int const i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    BatchStruct const& S = structOf ? bs[structOf[i]] : one;
    double r[3] = {posIn[3 * i + 0], posIn[3 * i + 1], posIn[3 * i + 2]};
    if (S.doRemap) remapAtom(r, S.pb.box, S.pb.invbox);
    if (normalize)
    {
        r[0] = __dmul_rn(r[0], convLength);
        r[1] = __dmul_rn(r[1], convLength);
        r[2] = __dmul_rn(r[2], convLength);
    }
    pos[3 * i + 0] = r[0];
    pos[3 * i + 1] = r[1];
    pos[3 * i + 2] = r[2];
}

// Warp per atom; MODE 0 counts, MODE 1 writes the entries (in key order).
template <int MODE>
__global__ void nlbBruteKernel(int n, int numElements, int NIMG,
                               double const* __restrict__ pos,
                               int const* __restrict__ structOf,
                               BatchStruct const* __restrict__ bs,
                               int const* __restrict__ structAtoms,
                               int* __restrict__ nbrCount,
                               int* __restrict__ nbrCountElem,
                               int const* __restrict__ nbrOff,
                               ListOut const out,
                               int const* __restrict__ status)
{
    if (status[ST_FLAGS] & FLAG_ABORT) return;
    int const lane = threadIdx.x & 31;
    int const i = (int)((blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5);
    if (i >= n) return;
    BatchStruct const& S = bs[structOf[i]];
    NLParams const& p = S.p;
    double const ri[3] = {pos[3 * i], pos[3 * i + 1], pos[3 * i + 2]};
    int total = 0;
    long const base = (MODE == 1) ? (long)nbrOff[i] : 0;
    int const nimg = p.nimg;
    for (int e = 0; e < numElements; ++e)
    {
        int const eb = S.es[e];
        long const ncand = (long)(S.es[e + 1] - eb) * nimg;
        int cntE = 0;
        for (long c0 = 0; c0 < ncand; c0 += 32)
        {
            long const c = c0 + lane;
            bool hit = false;
            int j = 0, img = 0;
            double dr[3];
            if (c < ncand)
            {
                j = structAtoms[eb + (int)(c / nimg)];
                img = (int)(c % nimg);
                int b0, b1, b2;
                imgDecode(p, img, b0, b1, b2);
                if (!(j == i && b0 == 0 && b1 == 0 && b2 == 0))
                    hit = nlTest(p, ri, pos, j, b0, b1, b2, dr);
            }
            unsigned const m = __ballot_sync(0xffffffffu, hit);
            if (MODE == 1 && hit)
            {
                int const off = total + __popc(m & ((1u << lane) - 1u));
                writeEntry(out, base + off, i, nlKey(e, j, img, n, NIMG), j,
                           e, dr);
            }
            total += __popc(m);
            cntE += __popc(m);
        }
        if (MODE == 0 && lane == 0)
            nbrCountElem[(long)i * numElements + e] = cntE;
    }
    if (MODE == 0 && lane == 0) nbrCount[i] = total;
}

__global__ void nlbMirrorKernel(int n, int NIMG,
                                int const* __restrict__ elem,
                                int const* __restrict__ structOf,
                                BatchStruct const* __restrict__ bs,
                                int const* __restrict__ nbrOff,
                                unsigned long long const* __restrict__ key,
                                int const* __restrict__ nbrIdx,
                                int const* __restrict__ entryAtom,
                                int* __restrict__ mirror,
                                int* __restrict__ status)
{
    if (status[ST_FLAGS] & FLAG_ABORT) return;
    long const e = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (e >= (long)nbrOff[n]) return;
    int const i = entryAtom[e];
    int const j = nbrIdx[e];
    int const nimg = bs[structOf[i]].p.nimg;
    int const img = (int)(key[e] % (unsigned long long)NIMG);
    unsigned long long const want = nlKey(elem[i], i, nimg - 1 - img, n, NIMG);
    long lo = nbrOff[j], hi = nbrOff[j + 1];
    while (lo < hi)
    {
        long const mid = (lo + hi) >> 1;
        if (key[mid] < want) lo = mid + 1;
        else hi = mid;
    }
    if (lo < nbrOff[j + 1] && key[lo] == want)
    {
        mirror[e] = (int)lo;
    }
    else
    {
        mirror[e] = -1;
        atomicOr(&status[ST_FLAGS], FLAG_MIRROR_MISSING);
    }
}

// Neighbor list of batches and of small single structures with at most 128
// images: warp per atom i, lanes over the candidates j of one element
// (positions loaded once).  A lane walks only the images that can be in
// reach: with s_k the fractional coordinate of r_i - r_j along box vector k
// and w_k the distance between the cell's faces, an image b is at least
// |s_k + b_k| w_k away, so b_k runs from ceil(-rc / w_k - s_k) to
// floor(rc / w_k - s_k) inside [-pbc_k, pbc_k] (in FP32, widened by far more
// than its error): 1 to 8 images instead of 27.  An FP32 distance decides
// outside rc^2 -+ m, where m covers the FP32 rounding of the displacement and
// image-shift sums (m from a bound on their magnitudes, at least 1e-4 rc^2);
// between them the exact FP64 test of nlTest does, so the neighbor sets are
// those of the brute path.  Hits are kept as per-lane image bit masks and
// placed in key order (lane = j ascending, bits = image ascending) through a
// warp prefix sum; MODE 0 counts, MODE 1 writes the entries.  384 water boxes
// (101,160 atoms), both passes and the entries: 3.7 ms with all 27 images,
// 1.1 ms so.
template <int MODE>
__global__ void __launch_bounds__(256, 4)
nlbLaneKernel(int n, int numElements, int NIMG,
              double const* __restrict__ pos,
              int const* __restrict__ structOf,
              BatchStruct const* __restrict__ bs,
              __grid_constant__ BatchStruct const one,
              int const* __restrict__ structAtoms,
              int* __restrict__ nbrCount,
              int* __restrict__ nbrCountElem,
              int const* __restrict__ nbrOff, ListOut const out,
              int const* __restrict__ status)
{
    if (status[ST_FLAGS] & FLAG_ABORT) return;
    int const lane = threadIdx.x & 31;
    int const i = (int)((blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5);
    if (i >= n) return;
    BatchStruct const& S = structOf ? bs[structOf[i]] : one;
    NLParams const& p = S.p;
    float q[3], m1, m2;
    float a[3][3], inv[3][3], reach[3];
    float const rcf = sqrtf((float)p.rc2);
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
        q[k] = p.periodic ? (float)p.pbc[k] : 0.0f;
        float w = 0.0f;
#pragma unroll
        for (int c = 0; c < 3; ++c)
        {
            a[k][c] = (float)p.box[k][c];
            inv[k][c] = (float)p.invbox[c][k];
            w += inv[k][c] * inv[k][c];
        }
        reach[k] = rcf * sqrtf(w);
    }
    m1 = 2.0f * q[1] + 1.0f;
    m2 = 2.0f * q[2] + 1.0f;
    double const ri[3] = {pos[3 * i], pos[3 * i + 1], pos[3 * i + 2]};
    // Largest image shift per component: sum_r |pbc_r a_r|.
    float shiftMax = 0.0f;
#pragma unroll
    for (int c = 0; c < 3; ++c)
        shiftMax = fmaxf(shiftMax, fabsf(a[0][c]) * q[0]
                                   + fabsf(a[1][c]) * q[1]
                                   + fabsf(a[2][c]) * q[2]);
    int total = 0;
    long const base = (MODE == 1) ? (long)nbrOff[i] : 0;
    for (int e = 0; e < numElements; ++e)
    {
        int const eb = S.es[e];
        int const ne = S.es[e + 1] - eb;
        int cntE = 0;
        for (int j0 = 0; j0 < ne; j0 += 32)
        {
            int const jj = j0 + lane;
            unsigned mask[4] = {0u, 0u, 0u, 0u};
            int j = 0;
            if (jj < ne)
            {
                j = structAtoms[eb + jj];
                float const d0 = (float)(ri[0] - pos[3 * j + 0]);
                float const d1 = (float)(ri[1] - pos[3 * j + 1]);
                float const d2 = (float)(ri[2] - pos[3 * j + 2]);
                // Per component the FP32 sum of up to four terms of size
                // <= M errs by < 8 M 2^-24 (rounded box included); r^2
                // near the cutoff then errs by < 2 rc 3 e + 3 e^2.
                float const M = fmaxf(fmaxf(fabsf(d0), fabsf(d1)), fabsf(d2))
                              + shiftMax;
                float const err = 8.0f * M * 5.9604645e-8f;
                float const slack = fmaxf(1e-4f * (float)p.rc2,
                                          4.0f * (6.0f * rcf * err
                                                  + 3.0f * err * err));
                float const above = (float)p.rc2 + slack;
                float const below = (float)p.rc2 - slack;
                // The images of the range one after another (one loop: its
                // trip count is the largest number of images of a lane, not
                // the product of the largest ranges), counters as floats.
                float lo[3], hi[3];
#pragma unroll
                for (int k = 0; k < 3; ++k)
                {
                    float const f = d0 * inv[k][0] + d1 * inv[k][1]
                                  + d2 * inv[k][2];
                    float const r = reach[k] + 1e-3f + 1e-4f * fabsf(f);
                    lo[k] = fmaxf(-q[k], ceilf(-r - f));
                    hi[k] = fminf(q[k], floorf(r - f));
                }
                bool more = lo[0] <= hi[0] && lo[1] <= hi[1] && lo[2] <= hi[2];
                float b0 = lo[0], b1 = lo[1], b2 = lo[2];
                while (more)
                {
                    float const x = d0 + b0 * a[0][0] + b1 * a[1][0]
                                  + b2 * a[2][0];
                    float const y = d1 + b0 * a[0][1] + b1 * a[1][1]
                                  + b2 * a[2][1];
                    float const z = d2 + b0 * a[0][2] + b1 * a[1][2]
                                  + b2 * a[2][2];
                    float const r2 = x * x + y * y + z * z;
                    if (r2 <= above
                        && !(j == i && b0 == 0.0f && b1 == 0.0f && b2 == 0.0f))
                    {
                        double dr[3];
                        if (r2 < below
                            || nlTest(p, ri, pos, j, (int)b0, (int)b1,
                                      (int)b2, dr))
                        {
                            int const img = (int)(((b0 + q[0]) * m1 + b1
                                                   + q[1]) * m2 + b2 + q[2]);
#pragma unroll
                            for (int w = 0; w < 4; ++w)
                                if (img >> 5 == w) mask[w] |= 1u << (img & 31);
                        }
                    }
                    b2 += 1.0f;
                    if (b2 > hi[2])
                    {
                        b2 = lo[2];
                        b1 += 1.0f;
                        if (b1 > hi[1])
                        {
                            b1 = lo[1];
                            b0 += 1.0f;
                            more = b0 <= hi[0];
                        }
                    }
                }
            }
            int const c = __popc(mask[0]) + __popc(mask[1]) + __popc(mask[2])
                        + __popc(mask[3]);
            int incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                int const v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            int const sum = __shfl_sync(0xffffffffu, incl, 31);
            if (MODE == 1 && c > 0)
            {
                long o = base + total + incl - c;
#pragma unroll
                for (int w = 0; w < 4; ++w)
                {
                    unsigned m = mask[w];
                    while (m)
                    {
                        int const img = (w << 5) + __ffs(m) - 1;
                        m &= m - 1;
                        int b0, b1, b2;
                        imgDecode(p, img, b0, b1, b2);
                        double dr[3];
                        nlTest(p, ri, pos, j, b0, b1, b2, dr);
                        writeEntry(out, o, i, nlKey(e, j, img, n, NIMG), j,
                                   e, dr);
                        ++o;
                    }
                }
            }
            total += sum;
            cntE += sum;
        }
        if (MODE == 0 && lane == 0)
            nbrCountElem[(long)i * numElements + e] = cntE;
    }
    if (MODE == 0 && lane == 0) nbrCount[i] = total;
}

void launchNeighborListBatch(NLBatchLaunch const& L, cudaStream_t s)
{
    int const n = L.n;
    int const tb = 256;
    int const gAtoms = (n + tb - 1) / tb;
    int const wpb = L.warpsPerBlock > 0 ? L.warpsPerBlock : 4;
    int const gWarp = (n + wpb - 1) / wpb;
    nlbPrepareKernel<<<gAtoms, tb, 0, s>>>(n, L.posIn, L.structOf, L.bs, L.one,
                                           L.normalize, L.convLength, L.pos);
    long const cap = L.capacity;
    int const gE = (int)((cap + tb - 1) / tb);
    ListOut const out{L.key, L.nbrIdx, L.nbrEl, L.dx, L.dy, L.dz, L.dd,
                      L.entryAtom};
    // Structures with more than 128 images (boxes below rc / 2) take the
    // plain brute path.
    if (L.NIMG <= 128)
    {
        nlbLaneKernel<0><<<gWarp, 32 * wpb, 0, s>>>(
            n, L.numElements, L.NIMG, L.pos, L.structOf, L.bs, L.one,
            L.structAtoms, L.nbrCount, L.nbrCountElem, L.nbrOff, out,
            L.status);
        nlScanKernel<<<1, 1024, 0, s>>>(n, L.nbrCount, L.nbrOff, L.capacity,
                                        L.status);
        nlbLaneKernel<1><<<gWarp, 32 * wpb, 0, s>>>(
            n, L.numElements, L.NIMG, L.pos, L.structOf, L.bs, L.one,
            L.structAtoms, L.nbrCount, L.nbrCountElem, L.nbrOff, out,
            L.status);
        noteLaunches(5);
        if (L.structOf)
            nlbMirrorKernel<<<gE > 0 ? gE : 1, tb, 0, s>>>(
                n, L.NIMG, L.elem, L.structOf, L.bs, L.nbrOff, L.key,
                L.nbrIdx, L.entryAtom, L.mirror, L.status);
        else
            nlMirrorKernel<<<gE > 0 ? gE : 1, tb, 0, s>>>(
                n, L.NIMG, L.elem, L.nbrOff, L.key, L.nbrIdx, L.entryAtom,
                L.mirror, L.status);
        return;
    }
    nlbBruteKernel<0><<<gWarp, 32 * wpb, 0, s>>>(
        n, L.numElements, L.NIMG, L.pos, L.structOf, L.bs, L.structAtoms,
        L.nbrCount, L.nbrCountElem, L.nbrOff, out, L.status);
    nlScanKernel<<<1, 1024, 0, s>>>(n, L.nbrCount, L.nbrOff, L.capacity,
                                    L.status);
    nlbBruteKernel<1><<<gWarp, 32 * wpb, 0, s>>>(
        n, L.numElements, L.NIMG, L.pos, L.structOf, L.bs, L.structAtoms,
        L.nbrCount, L.nbrCountElem, L.nbrOff, out, L.status);
    noteLaunches(5);
    nlbMirrorKernel<<<gE > 0 ? gE : 1, tb, 0, s>>>(
        n, L.NIMG, L.elem, L.structOf, L.bs, L.nbrOff, L.key, L.nbrIdx,
        L.entryAtom, L.mirror, L.status);
}

} // namespace n2p2b
