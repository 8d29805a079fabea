// update.cu -- the element-wise kernels of the spin-adapted solve: MP2 start, energy, the update
// of one iteration and the DIIS extrapolation, all over the amplitudes i <= j.
//
// The amplitudes of a block are rows (pairs) of columns (virtuals).  A tile is up to 128 columns
// c <= K - c of some rows; a thread owns such a column and its partner's, the amplitudes (i,j,a) and
// (i,j,b): v(i-b) = v(a-j), so both take the same two Coulomb factors, denominator and mosaic sums,
// and each of the two places in the ring results that hold theirs serves both (16 bytes; k_rx_pos).
// What a thread per amplitude fetched for each one -- the four orbitals, the mirror's index, two
// Coulomb factors (16 bytes), four orbital energies, four mosaic sums, two ring values, most of them
// scattered -- is index arithmetic, two table lookups and a few loads for two.  The sums of a tile,
// the energy and the DIIS dot products, are reduced together (warp_sums): one after the other they
// were nearly half of the instructions.
// Latency decides: all warps resident (32 registers, a few spilled) and the |q|^2 table read through
// L1 -- no barrier before the arithmetic -- beat fewer warps with more rows in flight, and a table
// in shared memory.  Per launch, 100 twists of N=54 (485 plane waves), a thread per amplitude, a
// column of two rows each, a row of two columns: the update with the DIIS push (0.2 ms of DRAM
// traffic) 0.381, 0.294, 0.239 ms; the MP2 start 0.227, 0.148, 0.133 ms; four N=114 systems: update
// 0.125, 0.098, 0.075 ms.  (All before the column ranges of update_tiles.)
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "kernels.h"
#include "uegccd_internal.h"
#include "warp.cuh"

namespace uegccd {

namespace {

constexpr int kThreads = 128;
constexpr int kRows = 1;      // rows a thread has in flight, two columns each

// Sum and maxima over the CTA in a fixed order (valid in thread 0).
__device__ __forceinline__ void reduce3(double &sum, double &mx1, double &mx2)
{
    __shared__ double s[3][kThreads / 32];
    for (int o = 16; o > 0; o >>= 1) {
        sum += __shfl_down_sync(0xffffffffu, sum, o);
        mx1 = fmax(mx1, __shfl_down_sync(0xffffffffu, mx1, o));
        mx2 = fmax(mx2, __shfl_down_sync(0xffffffffu, mx2, o));
    }
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        s[0][w] = sum;
        s[1][w] = mx1;
        s[2][w] = mx2;
    }
    __syncthreads();
    if (threadIdx.x == 0)
        for (int k = 1; k < kThreads / 32; k++) {
            sum += s[0][k];
            mx1 = fmax(mx1, s[1][k]);
            mx2 = fmax(mx2, s[2][k]);
        }
}

__device__ __forceinline__ UTileDev load_tile(const UTileDev *__restrict__ tiles)
{
    UTileDev T;
    const int4 *p = reinterpret_cast<const int4 *>(tiles + blockIdx.x);
    int4 *q = reinterpret_cast<int4 *>(&T);
#pragma unroll
    for (int k = 0; k < (int)(sizeof(UTileDev) / sizeof(int4)); k++) q[k] = __ldg(p + k);
    return T;
}

// A tile's threads: groups of `width` lanes (32, 64 or 128, the least that holds the columns), a
// group per row; thread (grp, lane) makes the rows r0 + grp + k * ngrp, in each the column c and,
// where `two`, its partner's column pc.
struct Place {
    int grp, ngrp, c, pc;     // row group, groups, column and its partner's column
    bool ok, two;
};
__device__ __forceinline__ Place place(const UTileDev &T)
{
    const int width = T.nc <= 32 ? 32 : T.nc <= 64 ? 64 : 128;
    Place P;
    P.grp = threadIdx.x / width;
    P.ngrp = kThreads / width;
    const int l = threadIdx.x - P.grp * width;
    P.ok = l < T.nc;
    P.c = T.c0 + min(l, T.nc - 1);
    P.two = P.c < T.nvd;
    P.pc = P.two ? P.c + T.nvd + T.sd : P.c;
    return P;
}

}  // namespace

// ----------------------------------------------------------------------------
// MP2 (MP2.f90:56-74): t = v(i-a)/D, D = e_i + e_j - e_a - e_b.
// E(2) = 1/2 sum [T2aaaa (V_ijab - V_ijba) + T2abab V_ijab - T2abba V_ijba]
//      = sum t(ij,a) (2 v(i-a) - v(i-b))   after the a <-> b re-indexing; v(i-b) = v(a-j).
// The mirror (j,i,b) has the same integrals; its denominator is summed in its own order.
// A core pair's integrals are zero (CoreERI), so is its amplitude.
// ----------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads, 12) k_mp2(const UTileDev *__restrict__ tiles,
                                                  const SolveDev *__restrict__ solves,
                                                  const int16_t *__restrict__ vir, const int *__restrict__ vpk,
                                                  const int4 *__restrict__ rowpk, const double *__restrict__ eigen,
                                                  const double *__restrict__ vtab, double *__restrict__ t,
                                                  double *__restrict__ part_e, double *__restrict__ part_a,
                                                  double *__restrict__ part_b)
{
    const UTileDev T = load_tile(tiles);
    const int core = solves[T.solve].core_n;
    const double *__restrict__ V = vtab + T.vtab0;
    double e = 0.0, mx = 0.0, none = 0.0;
    const Place P = place(T);
    const double *ev = eigen + T.orb0;
    const double ea = ev[vir[T.vir0 + P.c]], eb = ev[vir[T.vir0 + P.pc]];
    const int na = vpk[T.vir0 + P.c], m2 = neg2(na), na2 = __dp4a(na, na, 0);
#pragma unroll 2
    for (int r = P.ok ? P.grp : T.nr; r < T.nr; r += P.ngrp) {
        const int q = T.r0 + r;
        const int4 R = __ldg(&rowpk[T.pair0 + q]);
        const int i = R.z & 0xffff, j = R.z >> 16;
        const double via = V[__dp4a(m2, R.x, na2 + __dp4a(R.x, R.x, 0))];
        const double vaj = V[__dp4a(m2, R.y, na2 + __dp4a(R.y, R.y, 0))];
        const double eij = ev[i] + ev[j], dab = eij - ea - eb, dba = eij - eb - ea;
        const bool z = i < core || j < core, pair = q < T.nd;
        const int row = T.t0 + q * T.v, mir = row + (T.nd + T.dg) * T.v;
        const double x = z ? 0.0 : via / dab, y = z || !pair ? 0.0 : via / dba;
        t[row + P.c] = x;
        if (pair) t[mir + P.pc] = y;
        e += (x + y) * (2.0 * via - vaj);
        mx = fmax(mx, fmax(fabs(x), fabs(y)));
        if (P.two) {   // v(i - b) = v(a - j)
            const double u = z ? 0.0 : vaj / dba, w = z || !pair ? 0.0 : vaj / dab;
            t[row + P.pc] = u;
            if (pair) t[mir + P.c] = w;
            e += (u + w) * (2.0 * vaj - via);
            mx = fmax(mx, fmax(fabs(u), fabs(w)));
        }
    }
    reduce3(e, mx, none);
    if (threadIdx.x == 0) {
        part_e[blockIdx.x] = e;
        part_a[blockIdx.x] = mx;
        part_b[blockIdx.x] = 0.0;
    }
}

// Energy of the current amplitudes and max|t| (the dT before the first iteration).
// kind 0, CCEnergy (CCD.f90:225-227): E = sum t(ij,a) (2 v(i-a) - v(a-j)) after re-indexing;
// kind 1, dRPA CCEnergy (dRPA.f90:206-210): E = sum t (2 v(a-i) - csosex v(b-i)), v(b-i) = v(a-j).
// A mirror's integrals are those of its pair.
__global__ void __launch_bounds__(kThreads) k_energy(const UTileDev *__restrict__ tiles,
                                                     const int *__restrict__ vpk, const int4 *__restrict__ rowpk,
                                                     const double *__restrict__ vtab, const double *__restrict__ t, int kind, double csosex,
                                                     double *__restrict__ part_e, double *__restrict__ part_a,
                                                     double *__restrict__ part_b)
{
    const UTileDev T = load_tile(tiles);
    const double *__restrict__ V = vtab + T.vtab0;
    double e = 0.0, mx = 0.0, none = 0.0;
    const Place P = place(T);
    const int na = vpk[T.vir0 + P.c], m2 = neg2(na), na2 = __dp4a(na, na, 0);
#pragma unroll 2
    for (int r = P.ok ? P.grp : T.nr; r < T.nr; r += P.ngrp) {
        const int q = T.r0 + r;
        const int4 R = __ldg(&rowpk[T.pair0 + q]);
        const int row = T.t0 + q * T.v, mir = row + (T.nd + T.dg) * T.v;
        const bool pair = q < T.nd;
        const double x = t[row + P.c], y = pair ? t[mir + P.pc] : 0.0;
        const double u = P.two ? t[row + P.pc] : 0.0, w = P.two && pair ? t[mir + P.c] : 0.0;
        const double via = V[__dp4a(m2, R.x, na2 + __dp4a(R.x, R.x, 0))];
        const double vaj = V[__dp4a(m2, R.y, na2 + __dp4a(R.y, R.y, 0))];
        if (kind == 0) {
            e += (x + y) * (2.0 * via - vaj) + (u + w) * (2.0 * vaj - via);
        } else {
            e += via * (x + y) * 2.0 - vaj * (x + y) * csosex;
            e += vaj * (u + w) * 2.0 - via * (u + w) * csosex;
        }
        mx = fmax(fmax(mx, fmax(fabs(x), fabs(y))), fmax(fabs(u), fabs(w)));
    }
    reduce3(e, mx, none);
    if (threadIdx.x == 0) {
        part_e[blockIdx.x] = e;
        part_a[blockIdx.x] = mx;
        part_b[blockIdx.x] = 0.0;
    }
}

// ----------------------------------------------------------------------------
// Fused residual / update / convergence / energy.
//   G = ladders (from k_ladder) + drivers + mosaics + rings + crossed rings
//   R = -G + D t                          (GetRes, CCD.f90:417)
//   t' = (G/D - (1-f) t)/f                (SolveCC, CCD.f90:380)
//   dT = max |t' - t|                     (CnvrgCC, CCD.f90:452-454)
//   E  = sum t' (2 v(i-a) - v(a-j))       (CCEnergy, CCD.f90:225-227 re-indexed)
// By the pair symmetry t(ij,a) = t(ji,b) each amplitude with i < j also updates its mirror
// (j,i,b); every term of G shares the symmetry.
// NV: 0 updates in place, or forms the residual only (mode 1: max|R|, and G where g_out is given);
// else the Pulay DIIS push: the new (t', e) pair goes to the solve's history slot and the partials
// of e . e_j of every stored j < NV - 1 to dpart.  NV 8 holds up to 7 vectors in 32 registers; more of them
// take NV 32, at six CTAs an SM instead of sixteen: an iteration of 100 twists of N=54 1.22 ms with 7
// vectors, 1.43 with 8, 1.51 with 16.
// ----------------------------------------------------------------------------
struct UpdateArgs {
    const UTileDev *tiles;
    const SolveDev *solves;
    const int16_t *vir;
    const int *vpk;
    const int4 *rowpk;
    const double *eigen, *vtab;
    double *t;                    // each amplitude i <= j reads its own value only: updated in place
    const double *g_ladder;
    const double *jvv, *joo;
    const double *dru, *drs2;     // dRPA: U and S2 of k_drpa_sums
    double *part_e, *part_dt, *part_r;
    double *g_out;                // optional: full G per amplitude (term checks); may be g_ladder
    const double *rx;             // ring and crossed-ring G, particle-hole layout
    const int2 *rpos;             // where each amplitude's two values sit in it
    const uint8_t *active;
    int do_ladder, do_mosaic, do_ring, do_xring, do_driver, mode;
    const IterState *st;
    int ndiis;
    int64_t namp;
    double *hist_t, *dpart;
    float *hist_e;
};

template <int NV, bool DRPA>
__global__ void __launch_bounds__(kThreads, NV <= 8 ? 16 : 6) k_update(UpdateArgs A)
{
    const UTileDev T = load_tile(A.tiles);
    if (!A.active[T.solve]) {
        if (threadIdx.x == 0) A.part_e[blockIdx.x] = A.part_dt[blockIdx.x] = A.part_r[blockIdx.x] = 0.0;
        return;
    }
    const Place P = place(T);
    const bool rings = !DRPA && (A.do_ring || A.do_xring), mos = A.do_mosaic != 0;
    // index 0: the column c, 1: its partner's
    double told[kRows][2], g[kRows][2], s1[kRows][2], s2[kRows][2];
    int2 ro[kRows];
#pragma unroll
    for (int k = 0; k < kRows; k++) {
        const int r = P.grp + k * P.ngrp, row = T.t0 + (T.r0 + r) * T.v;
        const bool in = P.ok && r < T.nr, two = in && P.two;
        told[k][0] = in ? A.t[row + P.c] : 0.0;
        told[k][1] = two ? A.t[row + P.pc] : 0.0;
        g[k][0] = in && A.do_ladder ? A.g_ladder[row + P.c] : 0.0;
        g[k][1] = two && A.do_ladder ? A.g_ladder[row + P.pc] : 0.0;
        ro[k] = in && rings ? A.rpos[row + P.c] : make_int2(0, 0);
    }
    const double *ev = A.eigen + T.orb0;
    const int a = A.vir[T.vir0 + P.c], b = A.vir[T.vir0 + P.pc];
    const double ea = ev[a], eb = ev[b];
    const double jab = mos ? A.jvv[T.jvv0 + a - T.O] + A.jvv[T.jvv0 + b - T.O] : 0.0;
    const int na = A.vpk[T.vir0 + P.c], m2 = neg2(na), na2 = __dp4a(na, na, 0);
#pragma unroll
    for (int k = 0; k < kRows; k++) {
        // the place of (ia, jb) holds the ring G of (ij, a) and the crossed-ring G of (ij, b), that
        // of (ib, ja) the ring G of (ij, b) and the crossed-ring G of (ij, a)
        const bool in = P.ok && P.grp + k * P.ngrp < T.nr && rings;
        const double2 zero = make_double2(0.0, 0.0);
        const double2 u = in ? __ldg(reinterpret_cast<const double2 *>(A.rx + ro[k].x)) : zero;
        const double2 w = in ? P.two ? __ldg(reinterpret_cast<const double2 *>(A.rx + ro[k].y)) : u : zero;
        s1[k][0] = A.do_ring ? u.x : 0.0;
        s1[k][1] = A.do_ring ? w.x : 0.0;
        s2[k][0] = A.do_xring ? w.y : 0.0;
        s2[k][1] = A.do_xring ? u.y : 0.0;
    }
    const int core = A.solves[T.solve].core_n;
    const double f = A.solves[T.solve].denom_factor;
    const bool pow2 = (__double_as_longlong(f) & 0xfffffffffffffLL) == 0;   // then x / f = x * (1 / f) exactly
    // the push of iteration niter goes to slot (niter - 1) % ndiis, with min(niter, ndiis) stored
    const int nb = NV > 0 ? A.st[T.solve].niter : 1;
    const int slot = NV > 0 ? (nb - 1) % A.ndiis : 0, nvec = NV > 0 ? min(nb, A.ndiis) : 0;
    const double *__restrict__ V = A.vtab + T.vtab0;
    double esum = 0.0, mx = 0.0;   // mx: max|dT|, or max|R| in mode 1
    float err[kRows][2];
#pragma unroll
    for (int k = 0; k < kRows; k++) {
        err[k][0] = err[k][1] = 0.0f;
        const int r = P.grp + k * P.ngrp;
        if (!P.ok || r >= T.nr) continue;
        const int q = T.r0 + r, row = T.t0 + q * T.v;
        const int4 R = __ldg(&A.rowpk[T.pair0 + q]);
        const int i = R.z & 0xffff, j = R.z >> 16;
        const bool pair = q < T.nd;
        const int mir = row + (T.nd + T.dg) * T.v;
        const double via = V[__dp4a(m2, R.x, na2 + __dp4a(R.x, R.x, 0))];
        const double vaj = V[__dp4a(m2, R.y, na2 + __dp4a(R.y, R.y, 0))];   // = v(i - b)
        const double jj = mos ? 0.5 * (jab + A.joo[T.joo0 + i] + A.joo[T.joo0 + j]) : 0.0;
        const double denom = ev[i] + ev[j] - ea - eb;
#pragma unroll
        for (int m = 0; m < 2; m++) {
            if (m == 1 && !P.two) continue;
            const double v1 = m == 0 ? via : vaj, v2 = m == 0 ? vaj : via, t0 = told[k][m];
            const int p = row + (m == 0 ? P.c : P.pc), pm = mir + (m == 0 ? P.pc : P.c);
            double x = g[k][m];
            if (A.do_driver) x += v1;   // GetG2Drivers: G2abab = V(n_i - n_a)
            if (mos) x -= jj * t0;
            if (DRPA) {
                if (A.do_ring) {   // linear and quadratic rings (k_drpa_sums)
                    const int xa = (m == 0 ? a : b) - T.O, xb = (m == 0 ? b : a) - T.O;
                    const int ia = T.phr0 + i * T.V + xa, jb = T.phr0 + j * T.V + xb;
                    const double u = A.dru[ia];
                    x += u + A.dru[jb] + 2.0 * u * A.drs2[jb];
                }
            } else {   // the ring G and the crossed-ring G, where k_rings left them (k_rx_pos)
                if (A.do_ring) x += s1[k][m];
                if (A.do_xring) x += s2[k][m];
            }
            if (i < core || j < core) x = 0.0;   // core pair: every term has a zero factor
            if (NV == 0 && A.mode != 0) {
                if (A.g_out) {
                    A.g_out[p] = x;
                    if (pair) A.g_out[pm] = x;
                }
                mx = fmax(mx, fabs(-x + denom * t0));
                continue;
            }
            const double y = x / denom - (1.0 - f) * t0, tn = pow2 ? y * (1.0 / f) : y / f;
            double d = fabs(tn - t0);
            if (!(fabs(tn) < 1e300)) d = __longlong_as_double(0x7ff0000000000000LL);  // +Inf marks NaN/Inf
            mx = fmax(mx, d);
            // dRPA: the SOSEX part at the end
            const double es = DRPA ? v1 * tn * 2.0 : tn * (2.0 * v1 - v2);
            esum += pair ? 2.0 * es : es;
            if (NV == 0) {
                A.t[p] = tn;
                if (pair) A.t[pm] = tn;
            } else {   // the history slot holds t'; the mirrors' entries are never read
                err[k][m] = (float)(tn - t0);
                A.hist_t[(int64_t)slot * A.namp + p] = tn;
                A.hist_e[(int64_t)slot * A.namp + p] = err[k][m];
            }
        }
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    constexpr int NS = NV == 0 ? 1 : NV;   // sums: the dot products, and the energy in the last place
    __shared__ double sd[kThreads / 32][NS], sm[kThreads / 32];
    double v[NS];
#pragma unroll
    for (int j = 0; j < NS - 1; j++) {
        // e . e_j; an amplitude with a mirror counts twice
        v[j] = 0.0;
        if (j < nvec)
#pragma unroll
            for (int k = 0; k < kRows; k++) {
                const int r = P.grp + k * P.ngrp, q = T.r0 + r;
                if (!P.ok || r >= T.nr) continue;
                const float *h = A.hist_e + (int64_t)j * A.namp + T.t0 + q * T.v;
                const double h0 = j == slot ? err[k][0] : h[P.c], h1 = j == slot ? err[k][1] : P.two ? h[P.pc] : 0.0f;
                const double e0 = err[k][0], e1 = err[k][1];
                v[j] = fma(q < T.nd ? 2.0 * e0 : e0, h0, v[j]);
                v[j] = fma(q < T.nd ? 2.0 * e1 : e1, h1, v[j]);
            }
    }
    v[NS - 1] = esum;
    const int at = warp_sums<NS>(v);
    if (at >= 0) sd[w][at] = v[0];
    mx = warp_max(mx);
    if (l == 0) sm[w] = mx;
    __syncthreads();
    if (threadIdx.x < NS) {
        double d = 0.0;
        for (int k = 0; k < kThreads / 32; k++) d += sd[k][threadIdx.x];
        if (threadIdx.x == NS - 1) A.part_e[blockIdx.x] = d;
        else if (threadIdx.x < kDiisMax) A.dpart[(int64_t)blockIdx.x * kDiisMax + threadIdx.x] = d;
    }
    if (threadIdx.x == 32) {
        for (int k = 1; k < kThreads / 32; k++) sm[0] = fmax(sm[0], sm[k]);
        A.part_dt[blockIdx.x] = A.mode == 0 ? sm[0] : 0.0;
        A.part_r[blockIdx.x] = A.mode == 0 ? 0.0 : sm[0];
    }
}

// t = sum_j c_j t'_j over the amplitudes i <= j, each also written to its mirror (j,i,b)
__global__ void __launch_bounds__(kThreads) k_diis_extrap(const UTileDev *__restrict__ tiles, int64_t namp,
                                                          const double *__restrict__ hist_t,
                                                          const double *__restrict__ coef, int ndiis,
                                                          double *__restrict__ t, const uint8_t *__restrict__ applied)
{
    const UTileDev T = load_tile(tiles);
    if (!applied[T.solve]) return;
    const double *c = coef + T.solve * kDiisMax;
    const Place P = place(T);
    double x[kRows][2];
#pragma unroll
    for (int k = 0; k < kRows; k++) x[k][0] = x[k][1] = 0.0;
    for (int j = 0; j < ndiis; j++) {
        const double cj = c[j];
        if (cj == 0.0) continue;   // a slot not yet filled has coefficient 0 and is not read
        const double *h = hist_t + (int64_t)j * namp;
#pragma unroll
        for (int k = 0; k < kRows; k++) {
            const int r = P.grp + k * P.ngrp, row = T.t0 + (T.r0 + r) * T.v;
            if (P.ok && r < T.nr) {
                x[k][0] = fma(cj, h[row + P.c], x[k][0]);
                if (P.two) x[k][1] = fma(cj, h[row + P.pc], x[k][1]);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < kRows; k++) {
        const int r = P.grp + k * P.ngrp, q = T.r0 + r, row = T.t0 + q * T.v, mir = row + (T.nd + T.dg) * T.v;
        if (!P.ok || r >= T.nr) continue;
        t[row + P.c] = x[k][0];
        if (P.two) t[row + P.pc] = x[k][1];
        if (q < T.nd) {
            t[mir + P.pc] = x[k][0];
            if (P.two) t[mir + P.c] = x[k][1];
        }
    }
}

void launch_mp2(const DevBatch &d, cudaStream_t st)
{
    k_mp2<<<d.nutiles, kThreads, 0, st>>>(d.utiles, d.solves, d.vir, d.vpk, d.rowpk,
                                                                     d.eigen, d.vtab, d.t, d.part_e,
                                                                     d.part_dt, d.part_r);
}

void launch_energy(const DevBatch &d, int kind, double csosex, cudaStream_t st)
{
    k_energy<<<d.nutiles, kThreads, 0, st>>>(d.utiles, d.vpk, d.rowpk, d.vtab,
                                                                        d.t, kind, csosex, d.part_e,
                                                                        d.part_dt, d.part_r);
}

void launch_update(const DevBatch &d, const TermFlags &f, int mode, double *g_out, const CtlBuffers *diis, int ndiis,
                   cudaStream_t st)
{
    UpdateArgs A;
    A.tiles = d.utiles; A.solves = d.solves; A.vir = d.vir; A.vpk = d.vpk; A.rowpk = d.rowpk;
    A.eigen = d.eigen; A.vtab = d.vtab;
    A.t = d.t; A.g_ladder = d.g; A.jvv = d.jvv; A.joo = d.joo; A.dru = d.dru; A.drs2 = d.drs2;
    A.part_e = d.part_e; A.part_dt = d.part_dt; A.part_r = d.part_r; A.g_out = g_out; A.active = d.active;
    A.do_ladder = f.do_ladder; A.do_mosaic = f.do_mosaic; A.do_ring = f.do_ring; A.do_xring = f.do_xring;
    A.do_driver = f.do_driver; A.mode = mode;
    A.rx = d.rx; A.rpos = d.rpos;
    A.st = diis ? diis->state : nullptr; A.ndiis = (diis && mode == 0) ? ndiis : 0; A.namp = d.namp;
    A.hist_t = diis ? diis->hist_t : nullptr; A.hist_e = diis ? diis->hist_e : nullptr;
    A.dpart = diis ? diis->part : nullptr;
    auto *k = f.drpa ? A.ndiis == 0 ? k_update<0, true> : A.ndiis <= 7 ? k_update<8, true> : k_update<32, true>
                     : A.ndiis == 0 ? k_update<0, false> : A.ndiis <= 7 ? k_update<8, false> : k_update<32, false>;
    k<<<d.nutiles, kThreads, 0, st>>>(A);
}

void launch_extrap(const DevBatch &d, const CtlBuffers &c, int ndiis, cudaStream_t st)
{
    k_diis_extrap<<<d.nutiles, kThreads, 0, st>>>(d.utiles, d.namp, c.hist_t, c.coef, ndiis, d.t, c.applied);
}

// The tiles of a block of `rows` rows and v columns c <= K - c: column ranges of 128 and what is left,
// each in ranges that fill the threads' rows.  (Ranges of equal width leave more lanes idle: 100
// twists of N=54, update 0.224 against 0.194 ms, extrapolation 0.116 against 0.103; ranges of 64
// 0.212, of 32 0.254.)
void update_tiles(int rows, int v, void (*emit)(void *, int, int, int, int), void *to)
{
    constexpr int w = kThreads;
    for (int c0 = 0; c0 < v; c0 += w) {
        const int nc = std::min(w, v - c0), width = nc <= 32 ? 32 : nc <= 64 ? 64 : 128;
        const int step = kRows * (kThreads / width);
        for (int r0 = 0; r0 < rows; r0 += step) emit(to, c0, nc, r0, std::min(step, rows - r0));
    }
}

}  // namespace uegccd
