// rings.cu -- rings and crossed rings of the spin-adapted CCD residual (GetG2Rings, GetG2XRings,
// CCD.f90:689-940), linear and quadratic, on the FP64 tensor cores (mma.sync m8n8k4 f64).
//
// For every ph row (i,x), x virtual, with c = partner of (i,k,x):
//   X[k] = t(ik,x),  Y[k] = t(ik,c)                 (= t(ki,x) by the pair swap)
//   Sx = sum_k X, Sy = sum_k Y, vd = v(i-x)
//   Ex[j] = sum_k v(k-j) X[k],  Ey[j] = sum_k v(k-j) Y[k]
//   XW[l] = sum_k X[k] v(i+k-x-l), YW[l] = sum_k Y[k] v(i+k-x-l)
// the quadratic-ring intermediates of CCD.f90:774-797 / 902-925 are
//   A1 = J1 + J2 = 2 vd (2Sx - Sy) - 2 XW + YW,  A2 = J2 = vd (2Sx - Sy) - XW,  A3 = J3 = YW,
// and the amplitude (i,j,a) with partner b (rows ia, jb, ib, ja) gets
//   linear rings   (CCD.f90:716-763): 2 v(i-a)(Sx_ia + Sx_jb) - v(i-a)(Sy_ia + Sy_jb) - Ex_ia[j] - Ex_jb[i]
//   linear xrings  (CCD.f90:845-892): -Ey_ib[j] - Ey_ja[i]
//   quadratic rings  (CCD.f90:801-808): A1_ia . X_jb - A2_ia . Y_jb
//   quadratic xrings (CCD.f90:927-934): A3_ib . Y_ja
//
// The rows of momentum Q meet those of -Q only.  Rows a of group 1 are (i_a, x_a) with
// n_x - n_i = Q, rows b of group 2 (i_b, x_b) with -Q; t(i_a k, x_a) exists exactly for k in
// {i_b} (its partner is x_b), so every matrix has the group sizes as sides:
//   X[a][b] = t(i_a i_b, x_a)   Y[a][b] = t(i_b i_a, x_a)   (n1 x n2)
// and by the pair symmetry t(ij,a) = t(ji,b) group 2's matrices are their transposes.  With
//   W[b][a]  = v(n_{i_b} - n_{x_a}),  Vs1[a][a'] = v(n_{i_a'} - n_{i_a}),  Vs2 likewise for group 2
//   XW = X W,  U = Y W - Vs1,  z_a, z_b the row and column sums of 2X - Y
// the values of the pair (a, b) are
//   ring (i_a, i_b, x_a) = vd (z_a + z_b + z_a z_b)
//                          + sum_a' [XW[a][a'] (Y - 2X)[a'][b] + U[a][a'] X[a'][b]] - sum_b' X[a][b'] Vs2[b'][b]
//   xring(i_a, i_b, x_b) = sum_a' U[a][a'] Y[a'][b] - sum_b' Y[a][b'] Vs2[b'][b]
// k_update reads the two values of a pair (a, b) together: they belong to an amplitude and its
// partner, whose other two sit at one more place (k_rx_pos).
// Group 1 is the smaller group: 5 n1^2 n2 + 2 n1 n2^2 multiply-adds.
//
// A warp owns eight rows a for the whole pair: its XW and U stay in registers, as the A operand
// of the second product -- a C fragment holds columns 2t and 2t+1 of its row where the A operand
// of the next step wants column t and t+4, so the columns of W are handed to the lanes in that
// order.  Shared memory holds X and Y alone, a pair needs one barrier between staging and
// arithmetic (of its own warps: a CTA of six to eight works on 8, 4, 2 or 1 pairs at a time), and the
// row and column sums come out of the operands as they pass.  The Coulomb elements are looked up
// as in ladder.cu, in 16 copies of the table.
//
// Bound by DMMA (its pipe about half busy: 0.15 ms of products at 100 twists of N=54) and the
// latency of each pair's first loads; per residual, against the form with every matrix in shared
// memory and barriers between its phases: 100 twists of N=54 (485 plane waves) 0.425 -> 0.298 ms,
// four N=114 systems 0.341 -> 0.239 ms, 100 twists of N=14 12.2 -> 9.5 us.  Registers: two or three
// CTAs an SM; four (64 to 80 registers, spills) took 0.369 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>

#include "kernels.h"
#include "uegccd_internal.h"
#include "warp.cuh"

namespace uegccd {

namespace {

// pairs a CTA works on at a time, and its threads: six to eight warps
constexpr int ring_groups(int nf) { return nf == 1 ? 8 : nf == 2 ? 4 : nf <= 4 ? 2 : 1; }
constexpr int ring_threads(int nf) { return 32 * nf * ring_groups(nf); }
constexpr int ring_buffers(int nf) { return nf <= 4 ? 2 : 1; }

// The barrier of one group of warps (0: the whole CTA's)
__device__ __forceinline__ void group_sync(int id, int threads)
{
    asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}

struct Col {
    int m2, base;
};

// Row sides and column sides of a ph row's orbitals (RingRowDev); TAB16: 16 copies of the table
// and |n|^2 in the fourth byte of a column side, else one copy (shared or global memory).
template <bool TAB16>
__device__ __forceinline__ Col row_side(int m2, int n2)
{
    return Col{m2, TAB16 ? (n2 << 7) + ((int)(threadIdx.x & 15) << 3) : n2 << 3};
}

template <bool TAB16>
__device__ __forceinline__ double lookup(const char *tab, const Col &a, int c)
{
    const int d = __dp4a(a.m2, c, TAB16 ? 0 : __dp4a(c, c, 0));
    return *reinterpret_cast<const double *>(tab + (a.base + (d << (TAB16 ? 7 : 3))));
}

struct Args {
    const RingItemDev *items;
    const RingPairDev *pairs;
    const SolveDev *solves;
    const RingRowDev *rows;
    const double *vtab, *xy;
    double *rx;
    const uint8_t *active;
    int tab_bytes, pair_doubles;
};

// Starts the copies of one pair into its buffer: X and Y (8 NF rows, stride N2 + 4; the rows
// n1.. are zeroed), the row records of group 1, then those of group 2.
template <int NF>
__device__ __forceinline__ void fetch_pair(const RingPairDev &P, const double *__restrict__ xy,
                                           const RingRowDev *__restrict__ rows, double *buf, int t, int nt)
{
    constexpr int NR = 8 * NF;
    const int N2 = (P.n2 + 7) & ~7, l2 = N2 + 4, half = N2 / 2, lane = t & 31;
    double *X = buf, *Y = X + NR * l2;
    RingRowDev *rec = reinterpret_cast<RingRowDev *>(Y + NR * l2);
    const double *src = xy + P.xy0;
    for (int r = t >> 5; r < NR; r += nt >> 5)
        for (int c = lane; c < N2; c += 32) {
            double *dst = c < half ? X + r * l2 + 2 * c : Y + r * l2 + 2 * (c - half);
            if (r < P.n1) cp_async16(dst, src + 2 * (r * N2 + c));
            else *reinterpret_cast<double2 *>(dst) = make_double2(0.0, 0.0);
        }
    for (int r = t; r < P.n1 + P.n2; r += nt)
        cp_async16(rec + r, rows + (r < P.n1 ? P.r1 + r : P.r2 + r - P.n1));
}

// FN fragments of columns b from n0 of a warp's rows.
template <bool TAB16, int NF, int FN>
__device__ __forceinline__ void do_cols(const Args &A, const double *X, const double *Y, const double *Xr,
                                        const double *Yr, const RingRowDev *r2, const char *tab, int n0, int n2,
                                        int l2, int k2, const double (&xw)[NF][2], const double (&u)[NF][2], double z,
                                        double vd, bool store, double *out)
{
    const int lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
    double rg[FN][2], xr[FN][2], zb[FN];
    Col bc[FN];
#pragma unroll
    for (int f = 0; f < FN; f++) {
        rg[f][0] = rg[f][1] = xr[f][0] = xr[f][1] = zb[f] = 0.0;
        const RingRowDev R = r2[min(n0 + f * 8 + gid, n2 - 1)];
        bc[f] = row_side<TAB16>(R.mi, R.ni2);
    }
#pragma unroll 2
    for (int k = 0; k < k2; k += 4) {   // X Vs2, Y Vs2
        const double x = Xr[k], y = Yr[k];
        const int c = r2[min(k + tig, n2 - 1)].ci;
#pragma unroll
        for (int f = 0; f < FN; f++) {
            const double v = lookup<TAB16>(tab, bc[f], c);
            dmma_884(rg[f][0], rg[f][1], x, v);
            dmma_884(xr[f][0], xr[f][1], y, v);
        }
    }
#pragma unroll
    for (int f = 0; f < FN; f++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            rg[f][h] = -rg[f][h];
            xr[f][h] = -xr[f][h];
        }
#pragma unroll
    for (int q = 0; q < NF; q++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int a = (q * 8 + tig + 4 * h) * l2 + gid + n0;
#pragma unroll
            for (int f = 0; f < FN; f++) {
                const double x = X[a + f * 8], y = Y[a + f * 8], d = y - 2.0 * x;
                zb[f] -= d;
                dmma_884(rg[f][0], rg[f][1], xw[q][h], d);
                dmma_884(rg[f][0], rg[f][1], u[q][h], x);
                dmma_884(xr[f][0], xr[f][1], u[q][h], y);
            }
        }
#pragma unroll
    for (int f = 0; f < FN; f++) {
        zb[f] += __shfl_xor_sync(0xffffffffu, zb[f], 1);
        zb[f] += __shfl_xor_sync(0xffffffffu, zb[f], 2);   // z_b of column n0 + 8 f + gid
        const double z0 = __shfl_sync(0xffffffffu, zb[f], tig * 8);
        const double z1 = __shfl_sync(0xffffffffu, zb[f], tig * 8 + 4);
        if (!store) continue;
        double2 *o = reinterpret_cast<double2 *>(out) + n0 + f * 8;
        o[0] = make_double2(vd * (z + z0 + z * z0) + rg[f][0], xr[f][0]);
        o[1] = make_double2(vd * (z + z1 + z * z1) + rg[f][1], xr[f][1]);
    }
}

// The arithmetic of one pair: rows [8 w, 8 w + 8) of group 1.
template <bool TAB16, int NF>
__device__ __forceinline__ void do_pair(const Args &A, const RingPairDev &P, const double *buf, const char *tab, int w)
{
    constexpr int NR = 8 * NF;
    const int lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
    const int n1 = P.n1, n2 = P.n2, N2 = (n2 + 7) & ~7, l2 = N2 + 4, k2 = (n2 + 3) & ~3;
    const double *X = buf, *Y = X + NR * l2;
    const RingRowDev *r1 = reinterpret_cast<const RingRowDev *>(Y + NR * l2), *r2 = r1 + n1;
    const int m0 = w * 8;
    const double *Xr = X + (m0 + gid) * l2 + tig, *Yr = Y + (m0 + gid) * l2 + tig;
    const int ci_row = r1[min(m0 + gid, n1 - 1)].ci;
    // W's column of each fragment's lane: a' = 8 f + t for the C columns 2t, 8 f + 4 + t for 2t + 1
    Col xc[NF];
#pragma unroll
    for (int f = 0; f < NF; f++) {
        const RingRowDev R = r1[min(f * 8 + (gid >> 1) + (gid & 1) * 4, n1 - 1)];
        xc[f] = row_side<TAB16>(R.mx, R.nx2);
    }
    double xw[NF][2], u[NF][2], z = 0.0;
#pragma unroll
    for (int f = 0; f < NF; f++) xw[f][0] = xw[f][1] = u[f][0] = u[f][1] = 0.0;
#pragma unroll 2
    for (int k = 0; k < k2; k += 4) {
        const double x = Xr[k], y = Yr[k];
        const int c = r2[min(k + tig, n2 - 1)].ci;
        z += 2.0 * x - y;
#pragma unroll
        for (int f = 0; f < NF; f++) {
            const double v = lookup<TAB16>(tab, xc[f], c);
            dmma_884(xw[f][0], xw[f][1], x, v);
            dmma_884(u[f][0], u[f][1], y, v);
        }
    }
    z += __shfl_xor_sync(0xffffffffu, z, 1);
    z += __shfl_xor_sync(0xffffffffu, z, 2);   // z_a of row m0 + gid
#pragma unroll
    for (int f = 0; f < NF; f++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const RingRowDev R = r1[min(f * 8 + tig + 4 * h, n1 - 1)];
            u[f][h] -= lookup<TAB16>(tab, row_side<TAB16>(R.mi, R.ni2), ci_row);
        }
    const double vd = lookup<TAB16>(tab, row_side<TAB16>(r1[0].mx, r1[0].nx2), r1[0].ci);
    double *out = A.rx + P.xy0 + (int64_t)(m0 + gid) * 2 * N2 + 4 * tig;
    int n0 = 0;
    for (; n0 + 8 < N2; n0 += 16) do_cols<TAB16, NF, 2>(A, X, Y, Xr, Yr, r2, tab, n0, n2, l2, k2, xw, u, z, vd, m0 + gid < n1, out);
    if (n0 < N2) do_cols<TAB16, NF, 1>(A, X, Y, Xr, Yr, r2, tab, n0, n2, l2, k2, xw, u, z, vd, m0 + gid < n1, out);
}

// NF fragments of eight rows a (n1 <= 8 NF), a warp each; a CTA works on ring_groups(NF) pairs at a
// time.  With two buffers a group of warps has the copies of its next pair in flight while it works
// on one; the large pairs have one, and two CTAs an SM instead.
template <bool TAB16, int NF>
__global__ void __launch_bounds__(ring_threads(NF), NF <= 3 ? 3 : 2) k_rings(Args A)
{
    constexpr int GW = NF, NG = ring_groups(NF), GT = GW * 32, NT = ring_threads(NF);
    const RingItemDev I = A.items[blockIdx.x];
    if (!A.active[I.solve]) return;
    const SolveDev &s = A.solves[I.solve];
    extern __shared__ __align__(16) char rsm[];
    const double *gtab = A.vtab + s.vtab0;
    const char *tab = A.tab_bytes > 0 ? rsm : reinterpret_cast<const char *>(gtab);
    double *tb = reinterpret_cast<double *>(rsm);
    const RingRowDev *rows = A.rows + s.phr0;
    const int warp = threadIdx.x >> 5, grp = warp / GW, w = warp - grp * GW, t = threadIdx.x - grp * GT;
    constexpr int NB = ring_buffers(NF);
    double *buf = reinterpret_cast<double *>(rsm + A.tab_bytes) + (int64_t)grp * NB * A.pair_doubles;
    auto sync = [&]() {
        if (GW == 1) __syncwarp();
        else if (NG == 1) __syncthreads();
        else group_sync(1 + grp, GT);
    };
    RingPairDev P{};
    if (grp < I.count) {
        P = A.pairs[I.first + grp];
        fetch_pair<NF>(P, A.xy, rows, buf, t, GT);
    }
    cp_async_commit();
    if (TAB16)
        for (int e = threadIdx.x; e < (s.q2max + 1) * 16; e += NT) tb[e] = __ldg(gtab + (e >> 4));
    else if (A.tab_bytes > 0)
        for (int e = threadIdx.x; e <= s.q2max; e += NT) tb[e] = __ldg(gtab + e);
    __syncthreads();   // the table
    int b = 0;
    for (int pi = grp; pi < I.count; pi += NG) {
        const bool more = pi + NG < I.count;
        RingPairDev N{};
        if (more) N = A.pairs[I.first + pi + NG];
        if (NB == 2) {
            if (more) fetch_pair<NF>(N, A.xy, rows, buf + (b ^ 1) * A.pair_doubles, t, GT);
            cp_async_commit();
            cp_async_wait<1>();   // this pair's copies
        } else {
            cp_async_wait<0>();
        }
        sync();
        if (w * 8 < P.n1) do_pair<TAB16, NF>(A, P, buf + b * A.pair_doubles, tab, w);
        if (more) sync();   // this buffer takes the pair after the next (or the next)
        if (NB == 2) {
            b ^= 1;
        } else if (more) {
            fetch_pair<NF>(N, A.xy, rows, buf, t, GT);
            cp_async_commit();
        }
        P = N;
    }
}

bool tab16(const DevBatch &d) { return table16(d.q2max, d.n2max); }
int tab_bytes(const DevBatch &d)
{
    return tab16(d) ? (d.q2max + 1) * 128 : d.q2max < kVtabSmemEntries ? ((d.q2max + 1) * 8 + 15) / 16 * 16 : 0;
}

// doubles of one pair's buffer: X and Y of 8 nf rows of at most n2 columns, 16 bytes a row record
int pair_doubles(int nf, int n2) { return 2 * 8 * nf * (((n2 + 7) & ~7) + 4) + 2 * (8 * nf + n2); }

template <int NF>
void launch(const DevBatch &d, int c, const Args &A, cudaStream_t st)
{
    if (tab16(d)) k_rings<true, NF><<<d.nritems[c], ring_threads(NF), d.ring_smem[c], st>>>(A);
    else k_rings<false, NF><<<d.nritems[c], ring_threads(NF), d.ring_smem[c], st>>>(A);
}

}  // namespace

int ring_class(int n1)
{
    const int nf = (n1 + 7) / 8;
    return nf <= 4 ? nf - 1 : nf <= 6 ? 4 : nf <= 8 ? 5 : -1;
}

int ring_pairs_per_pass(int c) { return ring_groups(kRingFrags[c]); }

int ring_cta_threads(int pairs)
{
    int t = 0;
    for (int nf : kRingFrags)
        if (ring_groups(nf) == pairs) t = std::max(t, ring_threads(nf));
    return t;
}

size_t ring_smem_bytes(const DevBatch &d, int c, int max_n2)
{
    return tab_bytes(d) + sizeof(double) * (size_t)ring_buffers(kRingFrags[c]) * ring_groups(kRingFrags[c]) * pair_doubles(kRingFrags[c], max_n2);
}

void set_rings_smem_limit(size_t bytes)
{
    // keep the largest limit ever requested: batches of different sizes coexist
    static std::mutex mu;
    static size_t current_by_dev[kMaxDevices] = {};   // attributes are per device
    std::lock_guard<std::mutex> lock(mu);
    size_t &current = current_by_dev[current_device() % kMaxDevices];
    if (bytes <= std::max(current, (size_t)48 * 1024)) return;
    for (auto f : {k_rings<true, 1>, k_rings<true, 2>, k_rings<true, 3>, k_rings<true, 4>, k_rings<true, 6>,
                   k_rings<true, 8>, k_rings<false, 1>, k_rings<false, 2>, k_rings<false, 3>, k_rings<false, 4>,
                   k_rings<false, 6>, k_rings<false, 8>})
        cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    current = bytes;
}

int launch_rings(const DevBatch &d, const cudaStream_t *streams, int ns)
{
    int n = 0, off = 0, offs[kRingClasses];
    for (int c = 0; c < kRingClasses; c++) {
        offs[c] = off;
        off += d.nritems[c];
    }
    for (int c = kRingClasses - 1; c >= 0; c--) {   // the largest pairs first
        if (d.nritems[c] <= 0) continue;
        const Args A{d.ritems + offs[c], d.rpairs, d.solves, d.rrows, d.vtab, d.xy, d.rx, d.active, tab_bytes(d), d.ring_doubles[c]};
        const cudaStream_t st = streams[n % ns];
        switch (kRingFrags[c]) {
        case 1: launch<1>(d, c, A, st); break;
        case 2: launch<2>(d, c, A, st); break;
        case 3: launch<3>(d, c, A, st); break;
        case 4: launch<4>(d, c, A, st); break;
        case 6: launch<6>(d, c, A, st); break;
        default: launch<8>(d, c, A, st); break;
        }
        n++;
    }
    return n;
}

int ring_doubles(int c, int max_n2) { return pair_doubles(kRingFrags[c], max_n2); }

}  // namespace uegccd
