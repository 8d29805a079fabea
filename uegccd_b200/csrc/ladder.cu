// ladder.cu -- the FP64 ladders (GetG2Ladders, CCD.f90:588-686) of the spin-adapted residual.
//
// Per K block, written as G_K = t_K W_K + H_K t_K:
//   particle-particle (CCD.f90:660-681): W_K[c][a] = v(c-a) over the block's virtuals;
//   hole-hole (CCD.f90:611-657): H_K[p][q] = v(i_p - k_q) + sum_c t_K[p][c] v(c - k_q),
//   p = (i,j), q = (k,l), after the pair-swap re-indexing t(kl,b) = t(lk,a).
// Only the rows p = (i,j) with i <= j are formed: by the pair symmetry t(ij,a) = t(ji,b)
// (T2abab(ij,ab) = T2abab(ji,ba)) the mirror row (j,i) at column b = K - a has the value of
// (i,j) at a, and k_update reads G on the rows i <= j only.
//
// Even and odd halves.  The partner map a -> K - a of a block leaves its Coulomb kernel as it
// is, v(Ka - Kc) = v(a - c), so over the columns c <= pc (pc the partner of c, h of them)
//   s_c = (t_c + t_pc)/2,  d_c = (t_c - t_pc)/2     (self-partner: s = t/2, d = 0)
//   P_a = sum_c (v(a-c) + v(a-pc)) s_c,   M_a = sum_c (v(a-c) - v(a-pc)) d_c
//   G_a = P_a + M_a,   G_pa = P_a - M_a
// -- half the multiply-adds of the full product, and half the Coulomb elements for a block's
// rows.  The columns q <= q' of H (q' the mirror pair) split the same way, v(k_q' - c) =
// v(k_q - pc), and so does the product H t, t(q',a) = t(q,pa).  So one pass over the columns c
// forms the particle-particle sums of the columns a and the sums of H together; H stays in
// shared memory and its product with t follows in the same CTA.
//
// Coulomb elements.  v(a-c) is a table lookup by |n_a - n_c|^2 = |a|^2 + |c|^2 - 2 a.c: one byte
// dot product of packed vectors (a scaled by -2) on top of |c|^2, and one shift-add.  32 lanes
// look up 32 different entries, and on one copy of the table those reads met about 5-way bank
// conflicts, which bounded the kernel.  The table is therefore kept in 16 copies, one per pair
// of banks (entry q at 128 q + 8 (lane mod 16) bytes): every lookup is conflict-free, for 12 KB
// at N=54.  Tables beyond 256 entries (32 KB of copies) keep one copy, beyond 1,024 stay in
// global memory.
//
// Two forms, by the rows i <= j of a block, one launch each (a tile is one CTA of 128 threads, the
// longest tiles first):
//   1-4 rows    FP64 FMAs: a lane owns two columns a, all rows; the s and d of a column c are
//               broadcast reads (2 cycles a row).  Per 32 columns and c: two lookups (4 shared-memory cycles),
//               2 + 2 rows FMA-pipe instructions (1 + rows cycles).  A DMMA tile would spend 8
//               cycles however few rows fill its 8-wide fragment.
//   5 and more  DMMA (mma.sync m8n8k4 f64; tcgen05 has no f64 kind), up to 16 rows a tile: each
//               lane makes its own element of the two Coulomb fragments.  8 cycles per 8 rows.
// Measured per residual, ladders and hole-hole sums together, against DMMA tiles over the full
// products with a separate hole-hole launch: 100 twists of N=54 (485 plane waves) 0.79 -> 0.38 ms
// (FMA form 0.20, at the limit of no pipe: shared memory 57%, issue 55%, with 39% of the warps, its
// largest stalls the barriers and first loads of its short tiles; DMMA form 0.17, its pipe 46% busy), four N=114 systems 0.70 -> 0.25 ms, 100 twists of N=14 21 -> 10.5 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>

#include "kernels.h"
#include "uegccd_internal.h"
#include "warp.cuh"

namespace uegccd {

namespace {

constexpr int kThreads = 128;
constexpr int kKC = 32;            // columns c per staged chunk, DMMA form (double-buffered)
constexpr int kFC = 256;           // the same, FMA form
constexpr int kLd = kKC + 4;       // row stride of the DMMA operands: = 4 mod 16 doubles, conflict-free
constexpr int kHLd = 36;           // row stride of H (at most 32 pairs q <= q'): likewise

// Table forms: 16 copies or one in shared memory, or global memory.
enum { kTab16 = 0, kTab1 = 1, kTabGlobal = 2 };

// One orbital as the row side of a lookup: its packed vector times -2 and where |n|^2 puts it.
struct Col {
    int m2, base;
};

// With 16 copies every |n|^2 is at most 127 (table16): the column side carries it
// in its fourth byte, against a 1 on the row side.
template <int TAB>
__device__ __forceinline__ Col make_col(int packed)
{
    const int n2 = __dp4a(packed, packed, 0);
    Col c;
    c.m2 = neg2(packed);
    if (TAB == kTab16) c.m2 |= 1 << 24;
    c.base = TAB == kTab16 ? (n2 << 7) + ((threadIdx.x & 15) << 3) : TAB == kTab1 ? n2 << 3 : n2;
    return c;
}
template <int TAB>
__device__ __forceinline__ int col_side(int packed)
{
    return TAB == kTab16 ? packed | (__dp4a(packed, packed, 0) << 24) : packed;
}

// v(a - c), c a column side; c2 = |c|^2 where it is not in the fourth byte
template <int TAB>
__device__ __forceinline__ double lookup(const char *tab, const double *__restrict__ gtab, const Col &a, int c, int c2)
{
    const int d = __dp4a(a.m2, c, TAB == kTab16 ? 0 : c2);
    if (TAB == kTab16) return *reinterpret_cast<const double *>(tab + (a.base + (d << 7)));
    if (TAB == kTab1) return *reinterpret_cast<const double *>(tab + (a.base + (d << 3)));
    return __ldg(gtab + a.base + d);
}
template <int TAB>
__device__ __forceinline__ double lookup(const char *tab, const double *__restrict__ gtab, const Col &a, int packed)
{
    return lookup<TAB>(tab, gtab, a, col_side<TAB>(packed), __dp4a(packed, packed, 0));
}

struct Args {
    const LadderTile64 *tiles;
    const int *vpk;          // packed vectors beside vir
    const int2 *ppk;         // packed vectors of i and j beside the pairs
    const double *vtab, *t;
    double *g;
    const uint8_t *active;
    int do_pp, do_hh, tab_bytes;
};

// What both forms use of a tile's block.
struct Blk {
    LadderTile64 T;
    int h;                   // columns c <= pc
    int nh, ncol;            // the tile's columns: nh pairs q <= q' of H, then the virtuals a0 .. a1
    const double *t;         // the block's amplitudes
    const double *gtab;      // the solve's |q|^2 table
    const int *vpk;
    const int2 *ppk;
};

__device__ __forceinline__ int packed_col(const Blk &K, int e)
{
    e = min(e, K.ncol - 1);   // lanes past the tile repeat its last column
    return e < K.nh ? __ldg(&K.ppk[e].x) : __ldg(&K.vpk[K.T.a0 + e - K.nh]);
}

// One column c <= pc as both forms stage it: the column sides of c and pc.
template <int TAB>
__device__ __forceinline__ int2 chunk_col(const Blk &K, int c)
{
    c = min(c, K.h - 1);   // past the end the staged amplitudes are zero
    return make_int2(col_side<TAB>(__ldg(&K.vpk[c])), col_side<TAB>(__ldg(&K.vpk[c < K.T.nvd ? c + K.h : c])));
}

__device__ __forceinline__ void load_pair(const Blk &K, int row, int c, double &x, double &y)
{
    const double *r = K.t + row * K.T.v;
    x = c < K.h ? __ldg(r + c) : 0.0;
    y = c < K.T.nvd ? __ldg(r + c + K.h) : 0.0;
}

// The |c|^2 of two column sides that do not carry them
template <int TAB>
__device__ __forceinline__ int2 norms(int2 c)
{
    return TAB == kTab16 ? make_int2(0, 0) : make_int2(__dp4a(c.x, c.x, 0), __dp4a(c.y, c.y, 0));
}

// The tile's block; false when its solve is not active.
__device__ __forceinline__ bool open_tile(const Args &A, Blk &K)
{
    const int4 *p = reinterpret_cast<const int4 *>(A.tiles + blockIdx.x);
    int4 *q = reinterpret_cast<int4 *>(&K.T);
#pragma unroll
    for (int k = 0; k < (int)(sizeof(LadderTile64) / sizeof(int4)); k++) q[k] = __ldg(p + k);
    if (!A.active[K.T.solve]) return false;
    K.h = K.T.nvd + K.T.sd;
    K.nh = A.do_hh ? K.T.nd + K.T.dg : 0;
    K.ncol = K.nh + K.T.a1 - K.T.a0;
    K.t = A.t + K.T.t0;
    K.gtab = A.vtab + K.T.vtab0;
    K.vpk = A.vpk + K.T.vir0;
    K.ppk = A.ppk + K.T.pair0;
    return true;
}

template <int TAB>
__device__ __forceinline__ void fill_table(const Blk &K, char *smem)
{
    double *tab = reinterpret_cast<double *>(smem);
    if (TAB == kTab16)
        for (int e = threadIdx.x; e < (K.T.q2max + 1) * 16; e += kThreads) tab[e] = __ldg(K.gtab + (e >> 4));
    else if (TAB == kTab1)
        for (int e = threadIdx.x; e <= K.T.q2max; e += kThreads) tab[e] = __ldg(K.gtab + e);
}

// ---- 1 to 4 rows ------------------------------------------------------------------------
// Units of 32 columns, two a lane: the broadcast reads of s and d serve both.  (Four a lane, more
// registers and code, measured the same; so did 24 to 32 warps an SM.)
constexpr int kUnits = 2;

template <int TAB, int R, int U>
__device__ __forceinline__ void fma_cols(double (&P)[kUnits][R], double (&M)[kUnits][R], const Col (&a)[kUnits], const char *tab,
                                         const double *gtab, const int2 *cl, const double2 *sd, int k0, int step,
                                         int n)
{
#pragma unroll 1
    for (int k = k0; k < n; k += step) {
        const int2 c = cl[k], c2 = norms<TAB>(c);
        double2 x[R];
#pragma unroll
        for (int r = 0; r < R; r++) x[r] = sd[k * R + r];
#pragma unroll
        for (int m = 0; m < U; m++) {
            const double v = lookup<TAB>(tab, gtab, a[m], c.x, c2.x), w = lookup<TAB>(tab, gtab, a[m], c.y, c2.y);
            const double wp = v + w, wm = v - w;
#pragma unroll
            for (int r = 0; r < R; r++) {
                P[m][r] = fma(wp, x[r].x, P[m][r]);
                M[m][r] = fma(wm, x[r].y, M[m][r]);
            }
        }
    }
}

// smem: H, kFC int2 column records, then kFC x R double2 amplitudes (the reduction area once they
// are read)
template <int TAB, int R>
__device__ __forceinline__ void ladder_fma(const Args &A, const Blk &K, const char *tab, char *smem)
{
    constexpr int UM = kUnits;
    double2 *hs = reinterpret_cast<double2 *>(smem);
    int2 *cl = reinterpret_cast<int2 *>(hs + R * R);
    double2 *sd = reinterpret_cast<double2 *>(cl + kFC);
    double *red = reinterpret_cast<double *>(sd);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the units go to the warps in even groups; with one or two groups the warps split the columns c
    const int units = (K.ncol + 31) >> 5, groups = (units + UM - 1) / UM, upg = (units + groups - 1) / groups;
    const int ks = groups == 1 ? 4 : groups == 2 ? 2 : 1;
    const int grp = warp / ks, split = warp - grp * ks, u0 = grp * upg;
    const int nu = grp < groups ? min(upg, units - u0) : 0;
    const bool on = nu > 0 && (A.do_pp || grp == 0);
    // a chunk's amplitudes and column records, all threads; most blocks are one chunk
    auto stage = [&](int c0, int n) {
#pragma unroll
        for (int r = 0; r < R; r++)
            for (int k = threadIdx.x; k < n; k += kThreads) {
                double x, y;
                load_pair(K, r, c0 + k, x, y);
                sd[k * R + r] = make_double2(0.5 * (x + y), c0 + k < K.T.nvd ? 0.5 * (x - y) : 0.0);
            }
        for (int k = threadIdx.x; k < n; k += kThreads) cl[k] = chunk_col<TAB>(K, c0 + k);
    };
    fill_table<TAB>(K, const_cast<char *>(tab));
    Col a[UM];
#pragma unroll
    for (int m = 0; m < UM; m++) a[m] = make_col<TAB>(packed_col(K, (u0 + m) * 32 + lane));
    double P[UM][R], M[UM][R];
#pragma unroll
    for (int m = 0; m < UM; m++)
#pragma unroll
        for (int r = 0; r < R; r++) P[m][r] = M[m][r] = 0.0;
    for (int c0 = 0; c0 < K.h; c0 += kFC) {
        const int n = min(kFC, K.h - c0);
        if (c0 > 0) __syncthreads();
        stage(c0, n);
        __syncthreads();
        if (!on) continue;
        if (nu == 2) fma_cols<TAB, R, 2>(P, M, a, tab, K.gtab, cl, sd, split, ks, n);
        else fma_cols<TAB, R, 1>(P, M, a, tab, K.gtab, cl, sd, split, ks, n);
    }
    if (ks > 1) {
        // the splits' sums into the first one's, in order
        __syncthreads();
        auto at = [&](int sp, int m, int r, int q) -> double & {
            return red[((((sp - 1) * groups + grp) * UM + m) * R + r) * 64 + q * 32 + lane];
        };
        if (split > 0)
#pragma unroll
            for (int m = 0; m < UM; m++)
                if (m < nu)
#pragma unroll
                    for (int r = 0; r < R; r++) {
                        at(split, m, r, 0) = P[m][r];
                        at(split, m, r, 1) = M[m][r];
                    }
        __syncthreads();
        if (split == 0)
            for (int sp = 1; sp < ks; sp++)
#pragma unroll
                for (int m = 0; m < UM; m++)
                    if (m < nu)
#pragma unroll
                        for (int r = 0; r < R; r++) {
                            P[m][r] += at(sp, m, r, 0);
                            M[m][r] += at(sp, m, r, 1);
                        }
    }
    const bool lead = split == 0;
    if (K.nh > 0) {
        // halves of H: (H[p][q] +- H[p][q'])/2
        if (lead && grp == 0 && lane < K.nh) {
            const int2 pk = __ldg(&K.ppk[lane]);
            const Col kq = make_col<TAB>(pk.x), lq = make_col<TAB>(pk.y);
#pragma unroll
            for (int r = 0; r < R; r++) {
                const int n = __ldg(&K.ppk[r].x);
                const double v = lookup<TAB>(tab, K.gtab, kq, n), w = lookup<TAB>(tab, K.gtab, lq, n);
                hs[r * R + lane] = make_double2(P[0][r] + 0.5 * (v + w), M[0][r] + 0.5 * (v - w));
            }
        }
        __syncthreads();
    }
    if (!lead) return;
#pragma unroll
    for (int m = 0; m < UM; m++) {
        const int e = (u0 + m) * 32 + lane, c = K.T.a0 + e - K.nh;
        if (m >= nu || e < K.nh || e >= K.ncol) continue;
        const bool pair = c < K.T.nvd;
        double p[R], q[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            p[r] = A.do_pp ? P[m][r] : 0.0;
            q[r] = A.do_pp ? M[m][r] : 0.0;
        }
        if (K.nh > 0)
#pragma unroll
            for (int k = 0; k < R; k++) {
                const double *row = K.t + k * K.T.v;
                const double u = __ldg(row + c), w = pair ? __ldg(row + c + K.h) : u;
                const double f = k < K.T.nd ? 1.0 : 0.5;   // the pair and its mirror, or the diagonal pair
                const double s = f * (u + w), d = f * (u - w);
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const double2 H = hs[r * R + k];
                    p[r] = fma(H.x, s, p[r]);
                    q[r] = fma(H.y, d, q[r]);
                }
            }
        double *out = A.g + K.T.t0 + c;
#pragma unroll
        for (int r = 0; r < R; r++) {
            out[r * K.T.v] = p[r] + q[r];
            if (pair) out[r * K.T.v + K.h] = p[r] - q[r];
        }
    }
}

// ---- 5 rows and more --------------------------------------------------------------------
// NN fragments of 8 rows; a warp covers MF fragments of 8 columns, the CTA 4 warps of them a
// pass.  Fragment layouts (PTX ISA, m8n8k4 .f64): A row = lane/4, col = lane%4; B row (k) =
// lane%4, col = lane/4; C row = lane/4, cols 2*(lane%4) + {0,1}.
// smem: 2 x kKC int2 column records, s and d of 2 x 8 NN rows, the halves of H (8 NN rows each)
template <int TAB, int NN>
__device__ __forceinline__ void ladder_mma(const Args &A, const Blk &K, const char *tab, char *smem)
{
    constexpr int MF = NN == 1 ? 4 : 2, WC = 8 * MF, PC = 4 * WC, NR = 8 * NN;
    int2 *cl = reinterpret_cast<int2 *>(smem);
    double *S = reinterpret_cast<double *>(cl + 2 * kKC), *D = S + 2 * NR * kLd;
    double *hs = D + 2 * NR * kLd, *hd = hs + NR * kHLd;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
    const int nchunk = (K.h + kKC - 1) / kKC, np = K.T.np, p0 = K.T.p0, orow = K.T.nd + K.T.dg;
    fill_table<TAB>(K, const_cast<char *>(tab));
    __syncthreads();
    for (int e0 = 0; e0 < K.ncol; e0 += PC) {
        const int base = e0 + warp * WC;
        const bool loop = A.do_pp || (e0 == 0 && K.nh > 0);
        const bool on = base < K.ncol && (A.do_pp || base < K.nh);
        Col a[MF];
#pragma unroll
        for (int m = 0; m < MF; m++) a[m] = make_col<TAB>(packed_col(K, base + m * 8 + gid));
        double P[MF][NN][2], M[MF][NN][2];
#pragma unroll
        for (int m = 0; m < MF; m++)
#pragma unroll
            for (int n = 0; n < NN; n++) P[m][n][0] = P[m][n][1] = M[m][n][0] = M[m][n][1] = 0.0;
        if (loop) {
            double x[2 * NN], y[2 * NN];
            int2 rec = make_int2(0, 0);
            auto fetch = [&](int j) {
#pragma unroll
                for (int k = 0; k < 2 * NN; k++) {
                    const int r = warp + 4 * k;
                    x[k] = y[k] = 0.0;
                    if (r < np) load_pair(K, p0 + r, j * kKC + lane, x[k], y[k]);
                }
                if (warp == 0) rec = chunk_col<TAB>(K, j * kKC + lane);
            };
            fetch(0);
            for (int j = 0; j < nchunk; j++) {
                const int b = j & 1, c = j * kKC + lane;
#pragma unroll
                for (int k = 0; k < 2 * NN; k++) {
                    const int r = warp + 4 * k;
                    S[(b * NR + r) * kLd + lane] = 0.5 * (x[k] + y[k]);
                    D[(b * NR + r) * kLd + lane] = c < K.T.nvd ? 0.5 * (x[k] - y[k]) : 0.0;
                }
                if (warp == 0) cl[b * kKC + lane] = rec;
                __syncthreads();
                if (j + 1 < nchunk) fetch(j + 1);
                if (on) {
                    const double *sb = S + (b * NR + gid) * kLd + tig, *db = D + (b * NR + gid) * kLd + tig;
                    const int n4 = min(kKC, K.h - j * kKC);
#pragma unroll 2
                    for (int k = 0; k < n4; k += 4) {
                        const int2 cc = cl[b * kKC + k + tig], c2 = norms<TAB>(cc);
                        double bs[NN], bd[NN];
#pragma unroll
                        for (int n = 0; n < NN; n++) {
                            bs[n] = sb[n * 8 * kLd + k];
                            bd[n] = db[n * 8 * kLd + k];
                        }
#pragma unroll
                        for (int m = 0; m < MF; m++) {
                            const double v = lookup<TAB>(tab, K.gtab, a[m], cc.x, c2.x);
                            const double w = lookup<TAB>(tab, K.gtab, a[m], cc.y, c2.y);
                            const double wp = v + w, wm = v - w;
#pragma unroll
                            for (int n = 0; n < NN; n++) {
                                dmma_884(P[m][n][0], P[m][n][1], wp, bs[n]);
                                dmma_884(M[m][n][0], M[m][n][1], wm, bd[n]);
                            }
                        }
                    }
                }
            }
        }
        if (K.nh > 0 && e0 == 0) {
            // halves of H: (H[p][q] +- H[p][q'])/2; all of a block's q lie in the first pass
#pragma unroll
            for (int m = 0; m < MF; m++) {
                const int q = base + m * 8 + gid;
                if (q >= K.nh) continue;
                const int2 pk = __ldg(&K.ppk[q]);
                const Col kq = make_col<TAB>(pk.x), lq = make_col<TAB>(pk.y);
#pragma unroll
                for (int n = 0; n < NN; n++)
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        const int r = n * 8 + 2 * tig + u;
                        double hp = 0.0, hm = 0.0;
                        if (r < np) {
                            const int nn = __ldg(&K.ppk[p0 + r].x);
                            const double v = lookup<TAB>(tab, K.gtab, kq, nn);
                            const double w = lookup<TAB>(tab, K.gtab, lq, nn);
                            hp = P[m][n][u] + 0.5 * (v + w);
                            hm = M[m][n][u] + 0.5 * (v - w);
                        }
                        hs[r * kHLd + q] = hp;
                        hd[r * kHLd + q] = hm;
                    }
            }
            __syncthreads();
        }
        if (base < K.ncol) {
            if (!A.do_pp)
#pragma unroll
                for (int m = 0; m < MF; m++)
#pragma unroll
                    for (int n = 0; n < NN; n++) P[m][n][0] = P[m][n][1] = M[m][n][0] = M[m][n][1] = 0.0;
            if (K.nh > 0) {
                for (int q0 = 0; q0 < orow; q0 += 4) {
                    const int q = q0 + tig;
                    const bool qok = q < orow;
                    const double *row = K.t + (qok ? q : 0) * K.T.v;
                    const double f = q < K.T.nd ? 1.0 : 0.5;   // the pair and its mirror, or the diagonal pair
                    double bs[NN], bd[NN];
#pragma unroll
                    for (int n = 0; n < NN; n++) {
                        bs[n] = qok ? hs[(n * 8 + gid) * kHLd + q] : 0.0;
                        bd[n] = qok ? hd[(n * 8 + gid) * kHLd + q] : 0.0;
                    }
#pragma unroll
                    for (int m = 0; m < MF; m++) {
                        const int e = base + m * 8 + gid, c = K.T.a0 + e - K.nh;
                        double s = 0.0, d = 0.0;
                        if (qok && e >= K.nh && e < K.ncol) {
                            const double u = __ldg(row + c), w = c < K.T.nvd ? __ldg(row + c + K.h) : u;
                            s = f * (u + w);
                            d = f * (u - w);
                        }
#pragma unroll
                        for (int n = 0; n < NN; n++) {
                            dmma_884(P[m][n][0], P[m][n][1], s, bs[n]);
                            dmma_884(M[m][n][0], M[m][n][1], d, bd[n]);
                        }
                    }
                }
            }
#pragma unroll
            for (int m = 0; m < MF; m++) {
                const int e = base + m * 8 + gid, c = K.T.a0 + e - K.nh;
                if (e < K.nh || e >= K.ncol) continue;
                double *out = A.g + K.T.t0 + c;
#pragma unroll
                for (int n = 0; n < NN; n++)
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        const int r = n * 8 + 2 * tig + u;
                        if (r >= np) continue;
                        double *o = out + (p0 + r) * K.T.v;
                        o[0] = P[m][n][u] + M[m][n][u];
                        if (c < K.T.nvd) o[K.h] = P[m][n][u] - M[m][n][u];
                    }
            }
        }
        __syncthreads();   // the next pass stages its first chunk
    }
}

template <int TAB>
__global__ void __launch_bounds__(kThreads, 7) k_ladder_fma(Args A)
{
    Blk K;
    if (!open_tile(A, K)) return;
    extern __shared__ __align__(16) char lsm[];
    char *sm = lsm + A.tab_bytes;
    switch (K.T.nd + K.T.dg) {
    case 1: ladder_fma<TAB, 1>(A, K, lsm, sm); break;
    case 2: ladder_fma<TAB, 2>(A, K, lsm, sm); break;
    case 3: ladder_fma<TAB, 3>(A, K, lsm, sm); break;
    default: ladder_fma<TAB, 4>(A, K, lsm, sm); break;
    }
}

template <int TAB>
__global__ void __launch_bounds__(kThreads, 5) k_ladder_mma(Args A)
{
    Blk K;
    if (!open_tile(A, K)) return;
    extern __shared__ __align__(16) char lsm[];
    char *sm = lsm + A.tab_bytes;
    if (K.T.np <= 8) ladder_mma<TAB, 1>(A, K, lsm, sm);
    else ladder_mma<TAB, 2>(A, K, lsm, sm);
}

int tab_form(int q2max, int n2max)
{
    return table16(q2max, n2max) ? kTab16 : q2max < kVtabSmemEntries ? kTab1 : kTabGlobal;
}
int tab_bytes(int form, int q2max)
{
    return form == kTab16 ? (q2max + 1) * 128 : form == kTab1 ? ((q2max + 1) * 8 + 15) / 16 * 16 : 0;
}

size_t fma_bytes(int r)
{
    const int ks_units = 3 * kUnits;   // three splits of one group; two groups in two splits need less
    return sizeof(double2) * r * r + sizeof(int2) * kFC +
           std::max(sizeof(double2) * kFC * r, sizeof(double) * ks_units * r * 64);
}

}  // namespace

// A launch of fewer tiles than the GPU holds at a time asks for so much shared memory that no SM takes
// more of them than its share: with the rings and the mosaics running beside it, the ladder's CTAs are
// else packed on the SMs that come free first, up to seven on one.  Up to four tiles an SM;
// with more the packing costs nothing.  Times of one iteration in us, not spread (the range of six
// graphs of the same batch) and spread: N=2, 6,000 plane waves (12 tiles) 290 to 1,150, 293; N=14, 3,000 (131) 176
// to 520, 176, and 9,000 (385) 890 to 2,020, 893 to 978; N=30, 2,500 (281) 362 to 502, 246; N=54, 2,500
// (466, and 256 of the DMMA form) 562 to 591, 394; one N=54 system with 485 plane waves (114 and 52) 73, 71,
// three 96, 87, eight (908 and 442, five an SM) 156 and, spread over five, 163.
constexpr int kSms = 148, kSpread = 4;
constexpr size_t kSmShared = 228 * 1024;   // of an SM; each CTA takes 1 KB of it for itself
size_t spread_bytes(int tiles)
{
    const int per_sm = (tiles + kSms - 1) / kSms;
    return per_sm >= 1 && per_sm <= kSpread ? kSmShared / (per_sm + 1) : 0;
}

size_t ladder_smem_bytes(int q2max, int n2max, int max_rows, int form, int tiles)
{
    const size_t tab = tab_bytes(tab_form(q2max, n2max), q2max);
    if (form == 0) {
        size_t b = 0;
        for (int r = 1; r <= std::min(max_rows, kLadderFmaRows); r++) b = std::max(b, fma_bytes(r));
        return std::max(tab + b, spread_bytes(tiles));
    }
    const int nr = max_rows <= 8 ? 8 : 16;
    return std::max(tab + sizeof(int2) * 2 * kKC + sizeof(double) * (2 * 2 * (size_t)nr * kLd + 2 * (size_t)nr * kHLd),
                    spread_bytes(tiles));
}

int ladder_chunk() { return kKC; }

void set_ladder_smem_limit(size_t bytes)
{
    static std::mutex mu;
    static size_t current_by_dev[kMaxDevices] = {};   // attributes are per device
    std::lock_guard<std::mutex> lock(mu);
    size_t &current = current_by_dev[current_device() % kMaxDevices];
    if (bytes <= std::max(current, (size_t)48 * 1024)) return;
    for (auto f : {k_ladder_fma<kTab16>, k_ladder_fma<kTab1>, k_ladder_fma<kTabGlobal>, k_ladder_mma<kTab16>,
                   k_ladder_mma<kTab1>, k_ladder_mma<kTabGlobal>})
        cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    current = bytes;
}

int launch_ladder(const DevBatch &d, const double *t, int do_pp, int do_hh, double *g, cudaStream_t st,
                  cudaStream_t st_mma)
{
    const int form = tab_form(d.q2max, d.n2max);
    Args A{d.ltiles, d.vpk, d.ppk, d.vtab, t, g, d.active, do_pp, do_hh, tab_bytes(form, d.q2max)};
    int n = 0;
    if (d.nltiles[1] > 0) {   // the longer tiles first
        Args B = A;
        B.tiles += d.nltiles[0];
        const size_t sm = d.ladder_smem[1];
        if (form == kTab16) k_ladder_mma<kTab16><<<d.nltiles[1], kThreads, sm, st_mma>>>(B);
        else if (form == kTab1) k_ladder_mma<kTab1><<<d.nltiles[1], kThreads, sm, st_mma>>>(B);
        else k_ladder_mma<kTabGlobal><<<d.nltiles[1], kThreads, sm, st_mma>>>(B);
        n++;
    }
    if (d.nltiles[0] > 0) {
        const size_t sm = d.ladder_smem[0];
        if (form == kTab16) k_ladder_fma<kTab16><<<d.nltiles[0], kThreads, sm, st>>>(A);
        else if (form == kTab1) k_ladder_fma<kTab1><<<d.nltiles[0], kThreads, sm, st>>>(A);
        else k_ladder_fma<kTabGlobal><<<d.nltiles[0], kThreads, sm, st>>>(A);
        n++;
    }
    return n;
}

}  // namespace uegccd
