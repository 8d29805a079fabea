// two_channel_mm.cu -- the two-channel CCD residual as matrix products.
//
// two_channel.cu forms every term of an amplitude in the reference's loops: per amplitude it
// walks all virtuals for the particle-particle ladder and NOcc orbitals five times for the
// hole-hole ladder, the rings and the crossed rings, 0.84 ms a residual at N=54 (485 plane
// waves), bound by the latency of its scattered loads.  Where no integral of the tables is
// excluded (the reference's "Min(V1,V2) < -80 -> Cycle" never fires) and no orbital is core, the
// two integrals of a term do not depend on each other and the sums are products:
//   ladders   C = W T, W[m][c] = v(n_m - n_c) for m a virtual (particle-particle) or an occupied
//             orbital (hole-hole sums), T[c][(ij)] both channels side by side; one FP64 DMMA
//             product with the direct and, when its flags differ, the exchange integrals
//   rings     per {Q, -Q} pair of particle-hole groups, with A_Q[i][k] = t(i, k, i+Q): the
//             quadratic sums are A W_Q and their products with A_Q, the linear ones A times the
//             integrals between occupied orbitals (crossed rings: Y_Q[i][k] = t(k, i, i+Q))
// Measured on one N=54 system (485 plane waves), rings without crossed rings, per residual:
//   staging + mosaics 11 us, product + hole-hole 39 us, rings 40 us, assembly 27 us = 0.12 ms
//   against k2_mosaic 44, k2_hh 37, k2_ringq 55, k2_assemble 705 us = 0.84 ms.
#include <algorithm>

#include "two_channel_mm.h"
#include "warp.cuh"

namespace uegccd {

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ int pack(int4 n) { return (n.x & 0xff) | ((n.y & 0xff) << 8) | ((n.z & 0xff) << 16); }

// |n_a - n_c|^2 of packed vectors (components within +-63)
__device__ __forceinline__ int q2p(int a, int c)
{
    const int d = __vsub4(a, c);
    return __dp4a(d, d, 0);
}

__device__ __forceinline__ int q2v(int4 a, int4 b)
{
    const int x = a.x - b.x, y = a.y - b.y, z = a.z - b.z;
    return x * x + y * y + z * z;
}

// W by rows c: direct integrals of the V virtuals and the O occupied orbitals, then (sets = 2)
// the exchange ones.  The padding stays zero (preset).
__global__ void k2m_weights(TcMm D, TcFlags f)
{
    const int c = blockIdx.x;
    const int4 nc = D.nv[D.O + c];
    for (int m = threadIdx.x; m < D.sets * (D.V + D.O); m += blockDim.x) {
        const int x = m >= D.V + D.O, r = m - x * (D.V + D.O);
        const int4 nm = D.nv[r < D.V ? D.O + r : r - D.V];
        const int flag = r < D.V ? (x ? f.lad_lin_x : f.lad_lin_d) : (x ? f.lad_quad_x : f.lad_quad_d);
        D.w[(int64_t)c * D.ldw + m] = D.vt[flag * D.nq + q2v(nc, nm)];
    }
}

// One CTA per virtual c: the row T[c] of both channels with the disallowed entries zero, and the
// mosaic sums (CCD.f90:507-585) of that c: Jvv(c), and Joo's terms per k, which the last CTA
// adds up in c order.
__global__ void __launch_bounds__(kThreads) k2m_stage(TcMm D, int flag, const double *__restrict__ tab,
                                                      const double *__restrict__ tba, double *__restrict__ jvv,
                                                      double *__restrict__ joo)
{
    extern __shared__ double sm[];
    double *s = sm, *vk = sm + max(D.O * D.O, kThreads);   // O*O terms, then v(c - k)
    __shared__ double red[kThreads / 32];
    __shared__ bool last;
    const int O = D.O, O2 = O * O, c = blockIdx.x;
    const int4 nc = D.nv[O + c];
    for (int k = threadIdx.x; k < O; k += kThreads) vk[k] = D.vt[flag * D.nq + q2v(nc, D.nv[k])];
    __syncthreads();
    const int *F = D.F + (int64_t)O2 * (O + c);
    double *row = D.t + (int64_t)c * D.ldt;
    const int64_t t0 = (int64_t)O2 * c;
    double sum = 0.0;
    for (int p = threadIdx.x; p < O2; p += kThreads) {
        const bool ok = F[p] > O;
        const double a = ok ? tab[t0 + p] : 0.0, b = ok ? tba[t0 + p] : 0.0;
        row[p] = a;
        row[O2 + p] = b;
        const int k = p % O, l = p / O;
        const double x = vk[k] * (2.0 * a + b) - vk[l] * (a + 2.0 * b);
        s[p] = x;
        sum += x;
    }
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0;
        for (int w = 0; w < kThreads / 32; w++) a += red[w];
        jvv[c] = a;
    }
    for (int k = threadIdx.x; k < O; k += kThreads) {
        double a = 0.0;
        for (int l = 0; l < O; l++) a += s[k + O * l];
        D.jpart[(int64_t)c * O + k] = a;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(D.done, 1) == D.V - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    // thread (k, part): the terms of every parts-th c, then the parts in order
    double *jp = s;   // O * parts <= max(kThreads, O) entries
    const int parts = max(1, kThreads / O);
    for (int e = threadIdx.x; e < O * parts; e += kThreads) {
        const int k = e % O, q = e / O;
        double a = 0.0;
#pragma unroll 8
        for (int cc = q; cc < D.V; cc += parts) a += __ldcg(&D.jpart[(int64_t)cc * O + k]);
        jp[e] = a;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < O; k += kThreads) {
        double a = 0.0;
        for (int q = 0; q < parts; q++) a += jp[q * O + k];
        joo[k] = a;
    }
    if (threadIdx.x == 0) *D.done = 0;
}

// C = A^T B: A by rows c (lda), B by rows c (ldb); 64 x 64 tiles, 4 warps of 32 x 32, chunks of
// 16 rows c through three cp.async stages.  All dimensions are padded to the tile with zeros.
// Row stride 68 doubles (= 4 mod 16): conflict-free fragments.
// Bound by DMMA: 970 x 1,458 x 458 (N=54, both integral sets) is 1.3 GFLOP, 35 us at the
// measured 37 TFLOP/s.
constexpr int kTile = 64, kKC = 16, kStages = 3, kLd = kTile + 4;

__global__ void __launch_bounds__(128, 4) k2m_gemm(const double *__restrict__ A, int lda, const double *__restrict__ B,
                                                   int ldb, double *__restrict__ C, int ldc, int kdim)
{
    extern __shared__ __align__(16) double sm[];
    double *As = sm, *Bs = sm + kStages * kKC * kLd;
    const int m0 = blockIdx.y * kTile, n0 = blockIdx.x * kTile;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
    const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
    auto issue = [&](int j) {
        const int s = j % kStages;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int e = threadIdx.x + q * 128, r = e >> 5, x = (e & 31) * 2;
            cp_async16(As + (s * kKC + r) * kLd + x, A + (int64_t)(j * kKC + r) * lda + m0 + x);
            cp_async16(Bs + (s * kKC + r) * kLd + x, B + (int64_t)(j * kKC + r) * ldb + n0 + x);
        }
    };
    double acc[4][4][2];
#pragma unroll
    for (int m = 0; m < 4; m++)
#pragma unroll
        for (int n = 0; n < 4; n++) acc[m][n][0] = acc[m][n][1] = 0.0;
    const int nk = kdim / kKC;
    for (int j = 0; j < kStages - 1; j++) {
        if (j < nk) issue(j);
        cp_async_commit();
    }
    for (int j = 0; j < nk; j++) {
        cp_async_wait<kStages - 2>();
        __syncthreads();
        if (j + kStages - 1 < nk) issue(j + kStages - 1);   // the stage read in the last round
        cp_async_commit();
        const double *a = As + (j % kStages) * kKC * kLd + wm + gid, *b = Bs + (j % kStages) * kKC * kLd + wn + gid;
#pragma unroll
        for (int k = 0; k < kKC; k += 4) {
            double af[4], bf[4];
#pragma unroll
            for (int m = 0; m < 4; m++) af[m] = a[(k + tig) * kLd + m * 8];
#pragma unroll
            for (int n = 0; n < 4; n++) bf[n] = b[(k + tig) * kLd + n * 8];
#pragma unroll
            for (int m = 0; m < 4; m++)
#pragma unroll
                for (int n = 0; n < 4; n++) dmma_884(acc[m][n][0], acc[m][n][1], af[m], bf[n]);
        }
    }
#pragma unroll
    for (int m = 0; m < 4; m++)
#pragma unroll
        for (int n = 0; n < 4; n++)
            *reinterpret_cast<double2 *>(C + (int64_t)(m0 + wm + m * 8 + gid) * ldc + n0 + wn + n * 8 + 2 * tig) =
                make_double2(acc[m][n][0], acc[m][n][1]);
}

// The hole-hole sums of every pair (i,j) and each pair (k,l) of its momentum (CCD.f90:597-631):
// h2 = V_ijkl + 1/2 sum_c (V_cdkl Tabab - V_cdlk Tabba), h3 = -V_ijlk + the channels swapped.
__global__ void k2m_hh(TcMm D, TcFlags f)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= D.nkl) return;
    const int O = D.O, O2 = O * O, ij = D.kl_ij[e], k = D.kl[e] & 0xffff, l = D.kl[e] >> 16;
    const int i = ij % O;
    const int64_t xo = D.sets == 2 ? (int64_t)(D.V + O) * D.ldt : 0;
    const double *rk = D.c + (int64_t)(D.V + k) * D.ldt + ij, *rl = D.c + xo + (int64_t)(D.V + l) * D.ldt + ij;
    const double v2 = D.vt[f.lad_lin_d * D.nq + q2v(D.nv[i], D.nv[k])];
    const double v3 = D.vt[f.lad_lin_x * D.nq + q2v(D.nv[i], D.nv[l])];
    D.h2[e] = v2 + 0.5 * (rk[0] - rl[O2]);
    D.h3[e] = -v3 + 0.5 * (rk[O2] - rl[0]);
}

// Rings (XR = false, CCD.f90:689-814) or crossed rings (CCD.f90:817-940) of one pair of groups
// Q (rows (i, x), n_x - n_i = Q) and -Q (rows (j, y)).  With k over the other group's occupied
// orbitals (t vanishes elsewhere) and l over the row's own group's:
//   rings    A[i][k] = t(i,k,x): xw = A W, W[k][l] = v(k - l - Q); sums S = sum_k A
//            amplitude (i,j,x): linear(i,j) + linear(j,i)
//                               + sum_l (2 Dq - 2 xw_ab - xw_ba)[i][l] A_ab[l][j] + (Dq - xw_ab)[i][l] A_ba[l][j]
//            second channel:    linear' + linear' - sum_l xw_ba[i][l] A_ba[l][j]
//   crossed  Y[i][k] = t(k,i,x): amplitude (i,j,y), with Y' the other group's matrix:
//            linear + linear + sum_l xw_ab[i][l] Y'_ab[j][l]
//            second channel: linear' + linear' - sum_l (2 Bq - xw_ab - 2 xw_ba)[i][l] Y'_ba[j][l]
//                                              - sum_l (Bq - xw_ba)[i][l] Y'_ab[j][l]
// Each pair (i, j) gives an amplitude of the group Q and one of -Q (the two directions).  A
// thread makes four rows i of one column, so that each integral looked up serves eight FMAs.
template <bool XR>
__device__ void rings_pair(const TcMm &D, const TcFlags &f, const int4 P, const double *__restrict__ tab,
                           const double *__restrict__ tba, double *__restrict__ g1, double *__restrict__ g2,
                           double *sm)
{
    const int n[2] = {P.y, P.w}, r0[2] = {P.x, P.z};
    const int ld[2] = {P.w | 1, P.y | 1};   // group 0's rows hold group 1's columns, and the reverse
    const int nm = max(n[0], n[1]), lr = nm | 1;
    double *Aa[2], *Ab[2], *Sa[2], *Sb[2];
    double *p = sm;
#pragma unroll
    for (int g = 0; g < 2; g++) {
        Aa[g] = p;
        p += n[g] * ld[g];
        Ab[g] = p;
        p += n[g] * ld[g];
    }
    double *R1 = p, *R2 = R1 + nm * lr, *R3 = R2 + nm * lr;
    p = R3 + nm * lr;
#pragma unroll
    for (int g = 0; g < 2; g++) {
        Sa[g] = p;
        p += nm;
        Sb[g] = p;
        p += nm;
    }
    int *q = reinterpret_cast<int *>(p);
    int *occ[2] = {q, q + nm}, *vir[2] = {q + 2 * nm, q + 3 * nm}, *no[2] = {q + 4 * nm, q + 5 * nm};
    const int O = D.O, O2 = O * O;
#pragma unroll
    for (int g = 0; g < 2; g++)
        for (int e = threadIdx.x; e < n[g]; e += kThreads) {
            const int ix = D.ph[r0[g] + e];
            occ[g][e] = ix & 0xffff;
            vir[g][e] = ix >> 16;
            no[g][e] = pack(D.nv[ix & 0xffff]);
        }
    __syncthreads();
    for (int e = threadIdx.x; e < n[0] * n[1]; e += kThreads) {
        const int i = e / n[1], j = e - i * n[1];
        const int oi = occ[0][i], oj = occ[1][j];
        const int64_t x = (int64_t)O2 * (vir[0][i] - O), y = (int64_t)O2 * (vir[1][j] - O);
        const int64_t u = x + (XR ? oj + O * oi : oi + O * oj), w = y + (XR ? oi + O * oj : oj + O * oi);
        Aa[0][i * ld[0] + j] = tab[u];
        Ab[0][i * ld[0] + j] = tba[u];
        Aa[1][j * ld[1] + i] = tab[w];
        Ab[1][j * ld[1] + i] = tba[w];
    }
    __syncthreads();
#pragma unroll
    for (int g = 0; g < 2; g++)
        for (int i = threadIdx.x; i < n[g]; i += kThreads) {
            double a = 0.0, b = 0.0;
            for (int k = 0; k < n[1 - g]; k++) {
                a += Aa[g][i * ld[g] + k];
                b += Ab[g][i * ld[g] + k];
            }
            Sa[g][i] = a;
            Sb[g][i] = b;
        }
    __syncthreads();
    const double *lx = D.vt + (XR ? f.xr_lin_x : f.ring_lin_x) * D.nq;
    const double *qx = D.vt + (XR ? f.xr_quad_x : f.ring_quad_x) * D.nq;
    const int Q0 = __vsub4(pack(D.nv[vir[0][0]]), no[0][0]);
    const int qq = q2p(Q0, 0);
    const double vl = D.vt[(XR ? f.xr_lin_d : f.ring_lin_d) * D.nq + qq];
    const double vq = D.vt[(XR ? f.xr_quad_d : f.ring_quad_d) * D.nq + qq];
#pragma unroll
    for (int g = 0; g < 2; g++) {
        const int h = 1 - g, na = n[g], nb = n[h];
        const double *A = Aa[g], *B = Ab[g], *A2 = Aa[h], *B2 = Ab[h];
        const int Q = g == 0 ? Q0 : __vsub4(0, Q0), nblk = (na + 3) / 4;
        for (int e = threadIdx.x; e < nblk * na; e += kThreads) {
            const int ib = e / na, l = e - ib * na, cl = __vadd4(no[g][l], Q);
            const double *ra[4];
            double xa[4], xb[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                ra[u] = A + min(ib * 4 + u, na - 1) * ld[g];
                xa[u] = xb[u] = 0.0;
            }
            for (int k = 0; k < nb; k++) {
                const double w = __ldg(&qx[q2p(no[h][k], cl)]);
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    xa[u] = fma(ra[u][k], w, xa[u]);
                    xb[u] = fma(ra[u][k + (B - A)], w, xb[u]);
                }
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int i = ib * 4 + u;
                if (i >= na) break;
                const double d = XR ? vq * (Sa[g][i] + 2.0 * Sb[g][i]) : vq * (2.0 * Sa[g][i] + Sb[g][i]);
                R1[i * lr + l] = XR ? xa[u] : 2.0 * d - 2.0 * xa[u] - xb[u];
                R2[i * lr + l] = XR ? 2.0 * d - xa[u] - 2.0 * xb[u] : d - xa[u];
                R3[i * lr + l] = XR ? d - xb[u] : -xb[u];
            }
        }
        __syncthreads();
        for (int e = threadIdx.x; e < nblk * nb; e += kThreads) {
            const int ib = e / nb, j = e - ib * nb, nj = no[h][j];
            int ri[4], ni[4];
            double la[4], lb[4], ma[4], mb[4], q1[4], q2[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                ri[u] = min(ib * 4 + u, na - 1);
                ni[u] = no[g][ri[u]];
                la[u] = lb[u] = ma[u] = mb[u] = q1[u] = q2[u] = 0.0;
            }
            for (int k = 0; k < nb; k++) {   // linear, row i: sum_k v(k - j) A[i][k]
                const double w = __ldg(&lx[q2p(no[h][k], nj)]);
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    la[u] = fma(w, A[ri[u] * ld[g] + k], la[u]);
                    lb[u] = fma(w, B[ri[u] * ld[g] + k], lb[u]);
                }
            }
            for (int k = 0; k < na; k++) {   // linear, row j of the other group, and the quadratic sums
                const double x = A2[j * ld[h] + k], y = B2[j * ld[h] + k];
                const int nk = no[g][k];
                const double ak = XR ? x : A[k * ld[g] + j], bk = XR ? y : B[k * ld[g] + j];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const double w = __ldg(&lx[q2p(nk, ni[u])]);
                    ma[u] = fma(w, x, ma[u]);
                    mb[u] = fma(w, y, mb[u]);
                    const int r = ri[u] * lr + k;
                    if (XR) {
                        q1[u] = fma(R1[r], ak, q1[u]);
                        q2[u] = fma(-R2[r], bk, q2[u]);
                        q2[u] = fma(-R3[r], ak, q2[u]);
                    } else {
                        q1[u] = fma(R1[r], ak, q1[u]);
                        q1[u] = fma(R2[r], bk, q1[u]);
                        q2[u] = fma(R3[r], bk, q2[u]);
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int i = ib * 4 + u;
                if (i >= na) break;
                double di = 0.0, dj = 0.0;
                if (XR) {
                    di = vl * (Sa[g][i] + 2.0 * Sb[g][i]);
                    dj = vl * (Sa[h][j] + 2.0 * Sb[h][j]);
                } else {
                    di = vl * (2.0 * Sa[g][i] + Sb[g][i]);
                    dj = vl * (2.0 * Sa[h][j] + Sb[h][j]);
                }
                const int a = XR ? vir[h][j] : vir[g][i];
                const int64_t o = occ[g][i] + O * occ[h][j] + (int64_t)O2 * (a - O);
                g1[o] = (XR ? 0.0 : di + dj) - la[u] - ma[u] + q1[u];
                g2[o] = (XR ? di + dj : 0.0) - lb[u] - mb[u] + q2[u];
            }
        }
        __syncthreads();   // the other direction rewrites R1..R3
    }
}

// Three CTAs an SM (80 registers, some spilled) and the largest pairs first: 43 -> 40 us.
__global__ void __launch_bounds__(kThreads, 3) k2m_rings(TcMm D, TcFlags f, int rings,
                                                      const double *__restrict__ tab, const double *__restrict__ tba)
{
    extern __shared__ double sm[];
    const int4 P = D.pairs[blockIdx.x];
    if (blockIdx.y == 0 && rings) rings_pair<false>(D, f, P, tab, tba, D.gr[0], D.gr[1], sm);
    else rings_pair<true>(D, f, P, tab, tba, D.gx[0], D.gx[1], sm);
}

// Every term of one amplitude x = (i,j,a), b its momentum partner, from the products above.
__global__ void __launch_bounds__(kThreads) k2m_assemble(TcMm D, TcFlags f, int mask, const double *__restrict__ tab,
                                                         const double *__restrict__ tba,
                                                         const double *__restrict__ jvv,
                                                         const double *__restrict__ joo, double *__restrict__ gab,
                                                         double *__restrict__ gba)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= D.n) return;
    const int O = D.O, O2 = O * O;
    const int ij = x % O2, i = ij % O, j = ij / O, va = x / O2, a = O + va;
    const int b = D.F[ij + (int64_t)O2 * a] - 1;
    if (b < O) {
        gab[x] = 0.0;
        gba[x] = 0.0;
        return;
    }
    const int vb = b - O;
    const double t1 = tab[x], t2 = tba[x];
    double g1 = 0.0, g2 = 0.0;
    if (mask & 1) {
        g1 = D.vt[f.drv_d * D.nq + q2v(D.nv[i], D.nv[a])];
        g2 = -D.vt[f.drv_x * D.nq + q2v(D.nv[i], D.nv[b])];
    }
    if (mask & 2) {
        const double s = 0.5 * (jvv[va] + jvv[vb] + joo[i] + joo[j]);
        g1 -= s * t1;
        g2 -= s * t2;
    }
    if (mask & 4) {
        const int e1 = D.kl0[ij + 1];
        for (int e = D.kl0[ij]; e < e1; e++) {
            const int kl = D.kl[e], y = (kl & 0xffff) + O * (kl >> 16) + O2 * va;
            const double h2 = 0.5 * D.h2[e], h3 = 0.5 * D.h3[e], u = tab[y], w = tba[y];
            g1 += h2 * u + h3 * w;
            g2 += h2 * w + h3 * u;
        }
        const int64_t xo = D.sets == 2 ? (int64_t)(D.V + O) * D.ldt : 0;
        const double *d = D.c + (int64_t)va * D.ldt + ij, *xx = D.c + xo + (int64_t)vb * D.ldt + ij;
        g1 += 0.5 * (d[0] - xx[O2]);
        g2 += 0.5 * (d[O2] - xx[0]);
    }
    if (mask & 8) {
        g1 += D.gr[0][x];
        g2 += D.gr[1][x];
    }
    if (mask & 16) {
        g1 += D.gx[0][x];
        g2 += D.gx[1][x];
    }
    gab[x] = g1;
    gba[x] = g2;
}

}  // namespace

size_t tc_mm_ring_smem(int n1, int n2)
{
    const size_t nm = std::max(n1, n2), lr = nm | 1;
    return sizeof(double) * (2 * ((size_t)n1 * (n2 | 1) + (size_t)n2 * (n1 | 1)) + 3 * nm * lr + 4 * nm) +
           sizeof(int) * 6 * nm;
}

size_t tc_mm_stage_smem(int O) { return sizeof(double) * (std::max((size_t)O * O, (size_t)kThreads) + O); }

cudaError_t tc_mm_limits()
{
    cudaError_t e = cudaFuncSetAttribute(k2m_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(2 * kStages * kKC * kLd * sizeof(double)));
    // the limits only grow in steps a system needs; the largest a CTA may have covers them all
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k2m_rings, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcMmSmemMax);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k2m_stage, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcMmSmemMax);
    return e;
}

void tc_mm_weights(const TcMm &D, const TcFlags &f, cudaStream_t st) { k2m_weights<<<D.V, kThreads, 0, st>>>(D, f); }

int tc_mm_residual(const TcMm &D, const TcFlags &f, int mask, const double *tab, const double *tba, double *jvv,
                   double *joo, double *gab, double *gba, cudaStream_t st)
{
    int n = 1;
    if (mask & 6) {
        k2m_stage<<<D.V, kThreads, tc_mm_stage_smem(D.O), st>>>(D, f.mosaic, tab, tba, jvv, joo);
        n++;
    }
    if (mask & 4) {
        k2m_gemm<<<dim3(D.ldt / kTile, (D.sets * (D.V + D.O) + kTile - 1) / kTile), 128,
                   2 * kStages * kKC * kLd * sizeof(double), st>>>(D.w, D.ldw, D.t, D.ldt, D.c, D.ldt, D.kdim);
        if (D.nkl > 0) k2m_hh<<<(D.nkl + 255) / 256, 256, 0, st>>>(D, f);
        n += 2;
    }
    const int rings = (mask & 8) != 0, xrings = (mask & 16) != 0;
    if ((rings || xrings) && D.npairs > 0) {
        k2m_rings<<<dim3(D.npairs, rings + xrings), kThreads, D.ring_smem, st>>>(D, f, rings, tab, tba);
        n++;
    }
    k2m_assemble<<<(D.n + kThreads - 1) / kThreads, kThreads, 0, st>>>(D, f, mask, tab, tba, jvv, joo, gab, gba);
    return n;
}

}  // namespace uegccd
