// kernels_fp64.cu -- the spin-adapted CCD / MP2 / dRPA iteration: mosaics, dRPA sums, the staging of the
// rings, index tables, the iteration's tail and its launch order.  (The ladders are in ladder.cu, the rings
// in rings.cu, the element-wise kernels in update.cu.)
//
// Storage (uegccd_internal.h): t(ij,a) = T2abab(i,j,a), block-packed by
// K = n_i + n_j.  The reference's abba and aaaa channels are recovered from
// T2abba(i,j,a) = -t(ij,b) and T2aaaa(i,j,a) = t(ij,a) - t(ij,b), which the
// reference keeps exactly at the MP2 start (MP2.f90:68-70) and which its
// equations preserve when rings and crossed rings are both on.
//
// Notation below: v(x-y) = V(n_x - n_y) is the Coulomb kernel of the reference
// (BaseERI, HEG.f90:969-976), generated from an integer |q|^2 table;
// b = partner of (i,j,a), i.e. n_b = n_i + n_j - n_a.
//
// Every term is derived by substituting the two spin relations into the
// reference loops and re-indexing the sums over the partner bijection a <-> b
// of each K block; each formula cites the loop it replaces.
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>

#include "kernels.h"
#include "uegccd_internal.h"
#include "warp.cuh"

namespace uegccd {

__device__ __forceinline__ int q2_of(int4 x, int4 y)
{
    int d0 = x.x - y.x, d1 = x.y - y.y, d2 = x.z - y.z;
    return d0 * d0 + d1 * d1 + d2 * d2;
}

// v(p - q) for orbitals p, q of solve s
__device__ __forceinline__ double vpq(const SolveDev &s, const int4 *__restrict__ nv4,
                                      const double *__restrict__ vtab, int p, int q)
{
    return __ldg(&vtab[s.vtab0 + q2_of(__ldg(&nv4[s.orb0 + p]), __ldg(&nv4[s.orb0 + q]))]);
}

__device__ __forceinline__ int posmap(const SolveDev &s, const int32_t *__restrict__ pos, int i, int j, int a)
{
    return __ldg(&pos[s.pos0 + ((int64_t)i * s.O + j) * s.V + (a - s.O)]);
}

// ----------------------------------------------------------------------------
// Block reductions (fixed order: deterministic for a given launch shape)
// ----------------------------------------------------------------------------
template <int NT>
__device__ __forceinline__ void block_reduce3(double &sum, double &mx1, double &mx2)
{
    __shared__ double s_sum[NT / 32], s_m1[NT / 32], s_m2[NT / 32];
    for (int o = 16; o > 0; o >>= 1) {
        sum += __shfl_down_sync(0xffffffffu, sum, o);
        mx1 = fmax(mx1, __shfl_down_sync(0xffffffffu, mx1, o));
        mx2 = fmax(mx2, __shfl_down_sync(0xffffffffu, mx2, o));
    }
    int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) { s_sum[w] = sum; s_m1[w] = mx1; s_m2[w] = mx2; }
    __syncthreads();
    if (w == 0) {
        sum = (l < NT / 32) ? s_sum[l] : 0.0;
        mx1 = (l < NT / 32) ? s_m1[l] : 0.0;
        mx2 = (l < NT / 32) ? s_m2[l] : 0.0;
        for (int o = 16; o > 0; o >>= 1) {
            sum += __shfl_down_sync(0xffffffffu, sum, o);
            mx1 = fmax(mx1, __shfl_down_sync(0xffffffffu, mx1, o));
            mx2 = fmax(mx2, __shfl_down_sync(0xffffffffu, mx2, o));
        }
    }
}

template <int NT>
__device__ __forceinline__ double block_sum(double v)
{
    __shared__ double s[NT / 32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) s[w] = v;
    __syncthreads();
    double r = 0.0;
    if (w == 0) {
        r = (l < NT / 32) ? s[l] : 0.0;
        for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
    }
    return r;  // valid in thread 0
}

// t'(ij,a) = t(ij,a) - t(ij,b): T2aaaa of spin-adapted amplitudes (MP2.f90:70), the dRPA
// start, in place: the thread of the smaller index of a partner pair forms both values.
__global__ void k_to_aaaa(int64_t n, const int32_t *__restrict__ partner, double *__restrict__ t)
{
    int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const int32_t q = partner[p];
    if (q < p) return;
    const double x = t[p], y = t[q];
    t[p] = x + (-y);
    if (q != p) t[q] = y + (-x);
}

// Per-solve reduction of the chunk partials in chunk order.
// out[3*s+0] = sum(part_e), out[3*s+1] = max(part_a), out[3*s+2] = max(part_b)
__global__ void k_reduce_solves(const int *__restrict__ chunk_begin, const double *__restrict__ part_e,
                                const double *__restrict__ part_a, const double *__restrict__ part_b,
                                double *__restrict__ out)
{
    const int s = blockIdx.x;
    const int c0 = chunk_begin[s], c1 = chunk_begin[s + 1];
    double e = 0.0, ma = 0.0, mb = 0.0;
    for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
        e += part_e[c];
        ma = fmax(ma, part_a[c]);
        mb = fmax(mb, part_b[c]);
    }
    block_reduce3<256>(e, ma, mb);
    if (threadIdx.x == 0) { out[3 * s + 0] = e; out[3 * s + 1] = ma; out[3 * s + 2] = mb; }
}

// (The ladders, CCD.f90:588-686, are in ladder.cu; they write G first, before k_update adds
// the other terms.)

// ----------------------------------------------------------------------------
// Mosaics (GetG2Mosaics, CCD.f90:548-582):
//   s(k,l,c) = v(c-k) (T2aaaa + T2abab)(kl,c) - v(c-l) (T2aaaa + T2abba)(kl,c)
//            = v(c-k) (2t(kl,c) - t(kl,d)) - v(c-l) (t(kl,c) - 2t(kl,d))
//   Jvv(c) = sum_{k,l} s(k,l,c),  Joo(k) = sum_{l,c} s(k,l,c)
// (dRPA's own mosaics, dRPA.f90:415-431, come from k_drpa_sums.)
// v(d-k) = v(c-l) and v(d-l) = v(c-k) for the partner d = K - c of c in the row (k,l), so
// s(k,l,d) = s(k,l,c), and by the pair symmetry s(l,k,c) is the same again: s is formed on the
// rows i <= j and the columns c <= d only, an element standing for two or four.
// s lives only in registers: one CTA per K block writes the block's row sums (-> Joo of the row's
// k) and column sums (-> Jvv of the column's c); k_mosaic_sum adds the partials of each target in
// a fixed order.  The threads own the columns, so that all warps stay busy however few rows a
// block has: a column's sum stays with its thread, four rows are in flight and their sums are
// reduced together.  Bound by latency (a short chain per block) and, beyond that, by reading half
// the amplitudes once.  Per iteration, 100 twists of N=54 (485 plane
// waves): 100 -> 50 us against every column by itself, its partner found through the map and the
// |q|^2 table staged by each CTA; 100 twists of N=14: 8 -> 5 us.
// ----------------------------------------------------------------------------
constexpr int kMosThreads = 128;
constexpr int kMaxOcc = 64;             // NOcc limit of a batch
constexpr int kMosRows = kMaxOcc / 2 + 4;   // rows i <= j of a block, rounded up to fours

__global__ void __launch_bounds__(kMosThreads, 12) k_mosaic_blk(const BlockDev *__restrict__ blocks,
                                                           const SolveDev *__restrict__ solves,
                                                           const int *__restrict__ vpk,
                                                           const int4 *__restrict__ rowpk,
                                                           const double *__restrict__ vtab,
                                                           const double *__restrict__ t,
                                                           double *__restrict__ mpart,
                                                           const uint8_t *__restrict__ active)
{
    constexpr int kW = kMosThreads / 32, kR = 4;
    __shared__ double wrs[kW][kMosRows];   // per-warp row sums
    const BlockDev B = blocks[blockIdx.x];
    if (!active[B.solve]) return;
    const double *__restrict__ V = vtab + solves[B.solve].vtab0;
    const int oc = B.nd + B.dg, h = B.nvd + B.sd;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int r = lane; r < kMosRows; r += 32) wrs[warp][r] = 0.0;
    __syncwarp();
    for (int cw = warp * 32; cw < h; cw += kMosThreads) {
        const int c = min(cw + lane, h - 1);
        const bool ok = cw + lane < h, pair = c < B.nvd;
        const int na = vpk[B.vir0 + c], m2 = neg2(na), na2 = __dp4a(na, na, 0);
        const double *col = t + B.t0 + c;
        const int po = pair ? h : 0;
        double cs = 0.0;
        for (int r0 = 0; r0 < oc; r0 += kR) {
            double x[kR], y[kR], sr[kR];
#pragma unroll
            for (int q = 0; q < kR; q++) {
                const bool in = ok && r0 + q < oc;
                x[q] = in ? col[(int64_t)(r0 + q) * B.v] : 0.0;
                y[q] = in ? col[(int64_t)(r0 + q) * B.v + po] : 0.0;   // t(kl, d), same row
            }
#pragma unroll
            for (int q = 0; q < kR; q++) {
                const int4 R = __ldg(&rowpk[B.pair0 + min(r0 + q, oc - 1)]);
                const double vck = V[__dp4a(m2, R.x, na2 + __dp4a(R.x, R.x, 0))];
                const double vcl = V[__dp4a(m2, R.y, na2 + __dp4a(R.y, R.y, 0))];
                const double s = vck * (2.0 * x[q] - y[q]) - vcl * (x[q] - 2.0 * y[q]);
                cs += r0 + q < B.nd ? 2.0 * s : s;
                sr[q] = pair ? 2.0 * s : s;
            }
            const int at = warp_sums<kR>(sr);
            if (at >= 0) wrs[warp][r0 + at] += sr[0];
        }
        if (ok) {
            mpart[B.col0 + c] = cs;
            if (pair) mpart[B.col0 + c + h] = cs;
        }
    }
    __syncthreads();
    for (int r = tid; r < oc; r += kMosThreads) {
        double rs = 0.0;
        for (int w = 0; w < kW; w++) rs += wrs[w][r];
        mpart[B.row0 + r] = rs;
        if (r < B.nd) mpart[B.row0 + r + oc] = rs;   // the mirror row
    }
}

// One warp per target: targets (s, y < V) are Jvv(c = O + y), (s, y >= V) are Joo(k = y - V).
// The per-target lists k_mosaic_sum adds, built once per batch, one CTA per solve: target y
// < V (the virtual O + y) lists the column partials of every block holding that virtual,
// target V + k the row partials of the pair rows (k, l); both in block order, the order
// k_mosaic_sum then adds them in.  A virtual is one column of a block at most, and an
// occupied k the first index of one row at most (l = K - k), so within a block the targets
// are distinct and the block's entries go in at once.  mt_start[tbase[s] + y] is the first
// entry of target y of solve s (entries from lbase[s] on); the last solve also writes the
// end sentinel.  cnt: V + O ints of dynamic shared memory.  Bound by the latency of the chain block ->
// orbitals -> place, block after block: 30 twists of N=54, 197 -> 70 us with four blocks'
// orbitals in flight and the places in shared memory.
__global__ void k_mosaic_targets(const SolveDev *__restrict__ solves, const BlockDev *__restrict__ blocks,
                                 const int16_t *__restrict__ vir, const int16_t *__restrict__ pair_i,
                                 const int *__restrict__ tbase, const int64_t *__restrict__ lbase,
                                 int32_t *__restrict__ mt_start, int32_t *__restrict__ mt_list)
{
    extern __shared__ int cnt[];
    const int sv = blockIdx.x;
    const SolveDev S = solves[sv];
    const int nt = S.V + S.O, t0 = tbase[sv];
    for (int y = threadIdx.x; y < nt; y += blockDim.x) cnt[y] = 0;
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int bi = warp; bi < S.nblk; bi += nw) {
        const BlockDev &B = blocks[S.blk0 + bi];
#pragma unroll 4
        for (int c = lane; c < B.v; c += 32) atomicAdd(&cnt[vir[B.vir0 + c] - S.O], 1);
        for (int r = lane; r < B.o; r += 32) atomicAdd(&cnt[S.V + pair_i[B.pair0 + r]], 1);
    }
    __syncthreads();
    if (warp == 0) {   // cnt becomes the place of each target's next entry; a lane has a run of targets
        const int per = (nt + 31) / 32, y0 = min(lane * per, nt), y1 = min(y0 + per, nt);
        int sum = 0;
        for (int y = y0; y < y1; y++) sum += cnt[y];
        int run = sum;
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, run, o);
            if (lane >= o) run += x;
        }
        run += (int)lbase[sv] - sum;
        for (int y = y0; y < y1; y++) {
            const int k = cnt[y];
            mt_start[t0 + y] = run;
            cnt[y] = run;
            run += k;
        }
        if (lane == 31) mt_start[t0 + nt] = run;   // the next solve's first entry, or the end sentinel
    }
    __syncthreads();
    // four blocks' orbitals are fetched together, then entered block by block
    constexpr int kAhead = 4;
    for (int b0 = 0; b0 < S.nblk; b0 += kAhead) {
        int v[kAhead], o[kAhead], vir0[kAhead], col0[kAhead], row0[kAhead], y[kAhead], r[kAhead];
#pragma unroll
        for (int k = 0; k < kAhead; k++) {
            const bool in = b0 + k < S.nblk;
            const BlockDev &B = blocks[S.blk0 + min(b0 + k, S.nblk - 1)];
            v[k] = in ? B.v : 0;
            o[k] = in ? B.o : 0;
            vir0[k] = B.vir0;
            col0[k] = (int)B.col0;
            row0[k] = (int)B.row0;
            r[k] = B.pair0;
        }
#pragma unroll
        for (int k = 0; k < kAhead; k++) {
            y[k] = (int)threadIdx.x < v[k] ? vir[vir0[k] + threadIdx.x] - S.O : 0;
            r[k] = (int)threadIdx.x < o[k] ? S.V + pair_i[r[k] + threadIdx.x] : 0;   // o <= 64 threads
        }
#pragma unroll
        for (int k = 0; k < kAhead; k++) {
            for (int c = threadIdx.x; c < v[k]; c += blockDim.x) {
                const int z = c == (int)threadIdx.x ? y[k] : vir[vir0[k] + c] - S.O;
                mt_list[cnt[z]++] = col0[k] + c;
            }
            if ((int)threadIdx.x < o[k]) mt_list[cnt[r[k]]++] = row0[k] + (int)threadIdx.x;
            __syncthreads();
        }
    }
}

void launch_mosaic_targets(const DevBatch &d, const int *tbase, const int64_t *lbase, size_t smem, cudaStream_t st)
{
    if (smem > 48 * 1024) cudaFuncSetAttribute(k_mosaic_targets, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k_mosaic_targets<<<d.nsolves, 512, smem, st>>>(d.solves, d.blocks, d.vir, d.pair_i, tbase, lbase, d.mt_start,
                                                   d.mt_list);
}

__global__ void __launch_bounds__(256) k_mosaic_sum(const int2 *__restrict__ targets, int ntargets,
                                                   const SolveDev *__restrict__ solves,
                                                   const int32_t *__restrict__ mt_start,
                                                   const int32_t *__restrict__ mt_list,
                                                   const double *__restrict__ mpart, double *__restrict__ jvv,
                                                   double *__restrict__ joo, const uint8_t *__restrict__ active)
{
    const int lane = threadIdx.x & 31;
    const int tix = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (tix >= ntargets) return;
    const int2 tg = targets[tix];
    if (!active[tg.x]) return;
    double a = 0.0;
    for (int e = mt_start[tix] + lane; e < mt_start[tix + 1]; e += 32) a += mpart[mt_list[e]];
    for (int off = 16; off > 0; off >>= 1) a += __shfl_down_sync(0xffffffffu, a, off);
    if (lane == 0) {
        const SolveDev s = solves[tg.x];
        if (tg.y < s.V) jvv[s.jvv0 + tg.y] = a;
        else joo[s.joo0 + tg.y - s.V] = a;
    }
}

// ----------------------------------------------------------------------------
// dRPA rings and mosaics (dRPA.f90:377-551) from two sums per particle-hole pair (i, x):
//   S1(i,x) = sum_k t(ik,x),   S2(i,x) = sum_k t(ki,d), d = n_k + n_x' the column whose partner
//                              is x in row (k,i)
// The quadratic sum J(i,a,l) = sum_k 2 t(ik,a) v(i-a) (dRPA.f90:517-535) does not depend on l
// -- the reference's test that d is a virtual is the test that (l,j,b) is allowed, which the
// apply makes again -- so with U = 2 v(i-a) S1 and v(j-b) = v(i-a) every ring term of one
// amplitude is
//   U(i,a) + U(j,b) + 2 U(i,a) S2(j,b)                      (dRPA.f90:476-545)
// and the mosaics s(k,l,c) = 2 v(c-k) t(kl,c) (dRPA.f90:415-431) add up to
//   Joo(k) = sum_c U(k,c),   Jvv(c) = sum_k U(k,c).
// k_update then reads three values per amplitude where it walked 3 NOcc of them.
//
// One CTA per (solve, i) and range of at most kDrpaCols virtuals, a thread per virtual x: each k adds
// one value of row (i,k) and one of its mirror (k,i), at the column of x in that row's block (colpos),
// in ascending k.  The last CTA of a range to finish adds the columns of U up for Jvv, the last
// range's the terms of Joo.  (One CTA for all of a wide basis: N=14 with 9,000 plane waves 135 us.)
// Bound by memory latency: every amplitude read twice, near-coalesced (18 bytes with the column
// index).  30 twists of N=54, 485 plane waves, per iteration: 0.052 ms here and 0.072 ms in
// k_update, against 0.489 ms for the (i, x, l) intermediate, 0.048 ms of mosaic kernels and
// 0.645 ms in k_update.
// ----------------------------------------------------------------------------
constexpr int kDrpaThreads = 256;

// Row and column lookups, one CTA per K block: drows[(i,j)] = {first packed index of row
// (i,j), block, nvd, nvd + sd}; colpos[block][x] = column of virtual x (both pre-set to -1).
__global__ void k_drpa_tables(const BlockDev *__restrict__ blocks, const SolveDev *__restrict__ solves,
                              const DrpaSolveDev *__restrict__ ds, const int16_t *__restrict__ pair_i,
                              const int16_t *__restrict__ pair_j, const int16_t *__restrict__ vir,
                              int4 *__restrict__ drows, int16_t *__restrict__ colpos)
{
    const BlockDev B = blocks[blockIdx.x];
    const SolveDev s = solves[B.solve];
    const DrpaSolveDev D = ds[B.solve];
    const int bl = blockIdx.x - s.blk0;
    for (int r = threadIdx.x; r < B.o; r += blockDim.x)
        drows[D.rij0 + (int64_t)pair_i[B.pair0 + r] * s.O + pair_j[B.pair0 + r]] =
            make_int4((int)(B.t0 + (int64_t)r * B.v), bl, B.nvd, B.nvd + B.sd);
    for (int c = threadIdx.x; c < B.v; c += blockDim.x)
        colpos[D.cp0 + (int64_t)bl * s.V + (vir[B.vir0 + c] - s.O)] = (int16_t)c;
}

__global__ void __launch_bounds__(kDrpaThreads)
    k_drpa_sums(const int4 *__restrict__ list, const SolveDev *__restrict__ solves,
                const DrpaSolveDev *__restrict__ ds, const int4 *__restrict__ drows,
                const int16_t *__restrict__ colpos, const int4 *__restrict__ nv4, const double *__restrict__ vtab,
                const double *__restrict__ t, double *u, double *__restrict__ s2, double *jpart,
                double *__restrict__ jvv, double *__restrict__ joo, int *done, int nranges,
                const uint8_t *__restrict__ active)
{
    const int4 L = list[blockIdx.x];
    if (!active[L.x]) return;
    const SolveDev s = solves[L.x];
    const DrpaSolveDev D = ds[L.x];
    const int O = s.O, V = s.V, i = L.y;
    const int x0 = L.z * kDrpaCols, x1 = min(x0 + kDrpaCols, V), range = D.ch0 + L.z;
    __shared__ int4 row[kMaxOcc];
    __shared__ int mrow[kMaxOcc];
    __shared__ bool last, whole;
    for (int k = threadIdx.x; k < O; k += kDrpaThreads) {
        row[k] = drows[D.rij0 + (int64_t)i * O + k];
        mrow[k] = drows[D.rij0 + (int64_t)k * O + i].x;
    }
    __syncthreads();
    const int16_t *cp = colpos + D.cp0;
    double usum = 0.0;
    for (int x = x0 + threadIdx.x; x < x1; x += kDrpaThreads) {
        double a1 = 0.0, a2 = 0.0;
#pragma unroll 4
        for (int k = 0; k < O; k++) {
            const int4 r = row[k];
            const int c = r.x >= 0 ? __ldg(&cp[(int64_t)r.y * V + x]) : -1;
            if (c >= 0) {
                const int pc = c < r.z ? c + r.w : c < r.w ? c : c - r.w;
                a1 += __ldg(&t[r.x + c]);
                a2 += __ldg(&t[mrow[k] + pc]);
            }
        }
        const double y = 2.0 * vpq(s, nv4, vtab, i, s.O + x) * a1;
        u[s.phr0 + (int64_t)i * V + x] = y;
        s2[s.phr0 + (int64_t)i * V + x] = a2;
        usum += y;
    }
    usum = block_sum<kDrpaThreads>(usum);
    if (threadIdx.x == 0) {
        if (D.nc == 1) joo[s.joo0 + i] = usum;
        else jpart[D.jp0 + i * D.nc + L.z] = usum;
    }
    // Jvv by the range's last CTA: its reads of u follow every other CTA's fence and count
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&done[range], 1) == O - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int x = x0 + threadIdx.x; x < x1; x += kDrpaThreads) {
        double a = 0.0;
        for (int k = 0; k < O; k++) a += __ldcg(&u[s.phr0 + (int64_t)k * V + x]);
        jvv[s.jvv0 + x] = a;
    }
    if (threadIdx.x == 0) {
        done[range] = 0;
        whole = D.nc > 1 && atomicAdd(&done[nranges + L.x], 1) == D.nc - 1;
    }
    __syncthreads();
    if (!whole) return;
    __threadfence();
    for (int k = threadIdx.x; k < O; k += kDrpaThreads) {
        double a = 0.0;
        for (int c = 0; c < D.nc; c++) a += __ldcg(&jpart[D.jp0 + k * D.nc + c]);
        joo[s.joo0 + k] = a;
    }
    if (threadIdx.x == 0) done[nranges + L.x] = 0;
}

// (The rings and crossed rings, CCD.f90:689-940, are in rings.cu.)

// One CTA per momentum block: for every element (pair r = (i, j), column c = a) the
// amplitude record (i, j, a, b), the position map entry (i, j, a) -> packed index and the packed
// index of the partner (i, j, b), b in column pcol[c] of the same block.  Beside them the packed
// vectors of the block's virtuals and pairs.
__global__ void k_block_tables(const BlockDev *__restrict__ blocks, const SolveDev *__restrict__ solves,
                               const int16_t *__restrict__ pair_i, const int16_t *__restrict__ pair_j,
                               const int16_t *__restrict__ vir, const int16_t *__restrict__ pcol,
                               const int *__restrict__ nvp, AmpInfo *__restrict__ amps, int32_t *__restrict__ pos,
                               int32_t *__restrict__ partner, int *__restrict__ vpk, int2 *__restrict__ ppk,
                               int4 *__restrict__ rowpk)
{
    const BlockDev B = blocks[blockIdx.x];
    const SolveDev s = solves[B.solve];
    const int n = B.o * B.v;
    for (int c = threadIdx.x; c < B.v; c += blockDim.x) vpk[B.vir0 + c] = nvp[s.orb0 + vir[B.vir0 + c]];
    for (int r = threadIdx.x; r < B.o; r += blockDim.x) {
        const int i = pair_i[B.pair0 + r], j = pair_j[B.pair0 + r];
        const int2 n = make_int2(nvp[s.orb0 + i], nvp[s.orb0 + j]);
        ppk[B.pair0 + r] = n;
        rowpk[B.pair0 + r] = make_int4(n.x, n.y, i | j << 16, 0);
    }
    for (int e = threadIdx.x; e < n; e += blockDim.x) {
        const int r = e / B.v, c = e - r * B.v;
        const int i = pair_i[B.pair0 + r], j = pair_j[B.pair0 + r];
        const int a = vir[B.vir0 + c], pc = pcol[B.vir0 + c];
        const int64_t p = B.t0 + e;
        amps[p] = AmpInfo{(int16_t)i, (int16_t)j, (int16_t)a, vir[B.vir0 + pc]};
        pos[s.pos0 + ((int64_t)i * s.O + j) * s.V + (a - s.O)] = (int32_t)p;
        partner[p] = (int32_t)(B.t0 + (int64_t)r * B.v + pc);
    }
}

// Ring gather indices per ph row (i, x) and occupied k: t(ik, x) and t(ki, x).
__global__ void k_ring_index(const ChunkDev *__restrict__ rchunks, const SolveDev *__restrict__ solves,
                             const int16_t *__restrict__ ph_i, const int16_t *__restrict__ ph_x,
                             const int32_t *__restrict__ pos, int32_t *__restrict__ ridx_x,
                             int32_t *__restrict__ ridx_y)
{
    const ChunkDev ch = rchunks[blockIdx.x];
    const SolveDev s = solves[ch.solve];
    const int e = ch.start + threadIdx.x;
    if (e >= s.O * s.V * s.O) return;
    const int r = e / s.O, k = e - r * s.O;
    const int i = ph_i[s.phr0 + r], x = ph_x[s.phr0 + r];
    ridx_x[s.ph0 + e] = posmap(s, pos, i, k, x);
    ridx_y[s.ph0 + e] = posmap(s, pos, k, i, x);
}

// One CTA per ring pair: where each of its rows (i, x) sits in the particle-hole arrays.
// Group-1 row a: ph_a = xy0 + 2 a N2 (its row of two values a column), ph_b = -1.  Group-2
// row b: ph_a = -1, ph_b = b.  (Rows of groups without a -Q partner keep -1, -1.)
__global__ void k_ph_tables(const RingPairDev *__restrict__ pairs, const SolveDev *__restrict__ solves,
                            const int16_t *__restrict__ ph_i, const int16_t *__restrict__ ph_x,
                            int32_t *__restrict__ ph_a, int32_t *__restrict__ ph_b)
{
    const RingPairDev P = pairs[blockIdx.x];
    const SolveDev s = solves[P.solve];
    const int N2 = (P.n2 + 7) & ~7;
    for (int r = threadIdx.x; r < P.n1 + P.n2; r += blockDim.x) {
        const bool g1 = r < P.n1;
        const int row = g1 ? P.r1 + r : P.r2 + (r - P.n1);
        const int i = ph_i[s.phr0 + row], x = ph_x[s.phr0 + row];
        const int64_t k = s.phr0 + (int64_t)i * s.V + (x - s.O);
        ph_a[k] = g1 ? P.xy0 + 2 * r * N2 : -1;
        ph_b[k] = g1 ? -1 : r - P.n1;
    }
}

// The orbitals of every ph row as k_rings looks them up; carry: |n|^2 in the fourth byte of the
// column side (against a 1 in the row sides), where it fits.
__global__ void k_ring_rows(int n, const int *__restrict__ row0, int nsolves, const SolveDev *__restrict__ solves,
                            const int16_t *__restrict__ ph_i, const int16_t *__restrict__ ph_x,
                            const int *__restrict__ nvp, int carry, RingRowDev *__restrict__ rows)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    int lo = 0, hi = nsolves - 1;   // the solve whose rows hold r
    while (lo < hi) {
        const int m = (lo + hi + 1) >> 1;
        if (row0[m] <= r) lo = m;
        else hi = m - 1;
    }
    const SolveDev &s = solves[lo];
    auto m2 = [&](int p) { return neg2(p) | (carry ? 1 << 24 : 0); };
    const int pi = nvp[s.orb0 + ph_i[r]], px = nvp[s.orb0 + ph_x[r]];
    RingRowDev R;
    const int ni2 = __dp4a(pi, pi, 0);
    R.ci = carry ? pi | (ni2 << 24) : pi;
    R.mi = m2(pi);
    R.mx = m2(px);
    R.ni2 = (int16_t)ni2;
    R.nx2 = (int16_t)__dp4a(px, px, 0);
    rows[r] = R;
}

void launch_ring_rows(const DevBatch &d, int n, const int *row0, cudaStream_t st)
{
    const int carry = table16(d.q2max, d.n2max);
    if (n > 0)
        k_ring_rows<<<(n + 255) / 256, 256, 0, st>>>(n, row0, d.nsolves, d.solves, d.ph_i, d.ph_x, d.nvp, carry, d.rrows);
}

// The particle-hole copy of t that k_rings reads, one CTA per {Q, -Q} pair: row a of group
// 1 gets X1[a][c] = t(i_a i_c, x_a) and Y1[a][c] = t(i_c i_a, x_a) for the rows c of group 2,
// through the per-row gather indices (ridx_x, ridx_y).  Each CTA writes its pair's rows
// contiguously; the indexed reads are all this small kernel does, so many of them are in
// flight at once (in k_rings, behind its DMMA phases, they were what the kernel waited on).
__global__ void k_ring_stage(const RingPairDev *__restrict__ pairs, const SolveDev *__restrict__ solves,
                               const int16_t *__restrict__ ph_i, const int32_t *__restrict__ ridx_x,
                               const int32_t *__restrict__ ridx_y, const double *__restrict__ t,
                               double *__restrict__ xy, const uint8_t *__restrict__ active)
{
    const RingPairDev P = pairs[blockIdx.x];
    if (!active[P.solve]) return;
    const SolveDev s = solves[P.solve];
    const int N2 = (P.n2 + 7) & ~7, O = s.O;
    for (int e = threadIdx.x; e < P.n1 * P.n2; e += blockDim.x) {
        const int a = e / P.n2, c = e - a * P.n2;
        const int64_t w = s.ph0 + (int64_t)(P.r1 + a) * O + ph_i[s.phr0 + P.r2 + c];
        const int px = __ldg(&ridx_x[w]), py = __ldg(&ridx_y[w]);
        double *row = xy + P.xy0 + (int64_t)a * 2 * N2;
        row[c] = px >= 0 ? __ldg(&t[px]) : 0.0;
        row[N2 + c] = py >= 0 ? __ldg(&t[py]) : 0.0;
    }
}

// Where k_update finds the ring values of an amplitude (i,j,a), i <= j and a <= b, and of its partner
// (i,j,b) in rx, once per batch.  k_rings leaves at (a, b) of a {Q, -Q} pair the ring G of
// (i_a, i_b, x_a) beside the crossed-ring G of (i_a, i_b, x_b), a in group 1.  The place of (i,a),
// (j,b) -- row (i,a), column (j,b) when (i,a) is in group 1, else its mirror's, row (j,b), column
// (i,a) -- holds the ring G of (i,j,a) and the crossed-ring G of (i,j,b); that of (i,b), (j,a) the
// ring G of (i,j,b) and the crossed-ring G of (i,j,a).
__global__ void __launch_bounds__(128) k_rx_pos(const UTileDev *__restrict__ tiles, const SolveDev *__restrict__ solves,
                                               const AmpInfo *__restrict__ amps, const int32_t *__restrict__ ph_a,
                                               const int32_t *__restrict__ ph_b, int2 *__restrict__ rpos)
{
    const UTileDev T = tiles[blockIdx.x];
    const SolveDev s = solves[T.solve];
    for (int e = threadIdx.x; e < T.nr * T.nc; e += blockDim.x) {
        const int64_t p = T.t0 + (int64_t)(T.r0 + e / T.nc) * T.v + T.c0 + e % T.nc;   // column a <= b
        const AmpInfo q = amps[p];
        const int V = s.V, O = s.O;
        const int32_t *pa = ph_a + s.phr0, *pb = ph_b + s.phr0;
        const int ia = q.i * V + q.a - O, jb = q.j * V + q.b - O, ib = q.i * V + q.b - O, ja = q.j * V + q.a - O;
        const int r = pa[ia] >= 0 ? pa[ia] + 2 * pb[jb] : pa[jb] + 2 * pb[ia];
        const int x = pa[ib] >= 0 ? pa[ib] + 2 * pb[ja] : pa[ja] + 2 * pb[ib];
        rpos[p] = make_int2(r, x);
    }
}

void launch_block_tables(const DevBatch &d, cudaStream_t st)
{
    if (d.nblocks > 0)
        k_block_tables<<<d.nblocks, 256, 0, st>>>(d.blocks, d.solves, d.pair_i, d.pair_j, d.vir, d.pcol, d.nvp,
                                                  d.amps, d.pos, d.partner, d.vpk, d.ppk, d.rowpk);
    if (d.nrpairs > 0) k_ph_tables<<<d.nrpairs, 128, 0, st>>>(d.rpairs, d.solves, d.ph_i, d.ph_x, d.ph_a, d.ph_b);
    if (d.nrpairs > 0 && d.nutiles > 0)
        k_rx_pos<<<d.nutiles, 128, 0, st>>>(d.utiles, d.solves, d.amps, d.ph_a, d.ph_b, d.rpos);
    if (d.nrchunks > 0)
        k_ring_index<<<d.nrchunks, kChunk, 0, st>>>(d.rchunks, d.solves, d.ph_i, d.ph_x, d.pos, d.ridx_x,
                                                    d.ridx_y);
}

// ----------------------------------------------------------------------------
// Pulay DIIS (new in this library; the reference's GetTFromDIIS, DIISCC.f90:52-131,
// builds a singular matrix and never extrapolates).  Error vector e = t' - t of
// the (damped) Jacobi step; history of ndiis (t', e) pairs per solve.
// k_update stores the solve's current slot and forms the dot products e . e_j of
// every stored j (per-chunk partials); k_tail reduces them per solve in chunk order.
// ----------------------------------------------------------------------------
constexpr int kMaxDiis = 16;
// ----------------------------------------------------------------------------
// Device-side iteration control.  Every solve of a batch carries its own state;
// one iteration is a fixed sequence of launches (residual terms -> update -> k_tail ->
// [DIIS extrapolation]), so it can be captured once as a CUDA graph and replayed.
// Converged solves stop being updated (their CTAs return at once) while the others continue.
// ----------------------------------------------------------------------------
// Pulay system [B 1; 1 0][c; l] = [0; 1] over nvec vectors, B scaled by its max
// diagonal; Gaussian elimination with partial pivoting, one lane per row (nvec + 1 <= 17), the
// matrix in shared memory.  Returns false if singular (the same in every lane).
__device__ bool pulay_warp(const double *B, int nvec, double *c, double (*A)[kMaxDiis + 2])
{
    const int lane = threadIdx.x & 31, n = nvec + 1;
    double scale = lane < nvec ? B[lane * kMaxDiis + lane] : 0.0;
    scale = fmax(0.0, scale);
    for (int o = 16; o > 0; o >>= 1) scale = fmax(scale, __shfl_xor_sync(0xffffffffu, scale, o));
    if (!(scale > 0.0) || !isfinite(scale)) return false;
    if (lane < n)
        for (int k = 0; k <= n; k++) {
            double x = 0.0;
            if (lane < nvec) x = k < nvec ? B[lane * kMaxDiis + k] / scale : k == nvec ? 1.0 : 0.0;
            else x = k < nvec ? 1.0 : k == n ? 1.0 : 0.0;
            A[lane][k] = x;
        }
    __syncwarp();
    for (int k = 0; k < n; k++) {
        double best = lane >= k && lane < n ? fabs(A[lane][k]) : -1.0;
        int piv = lane;
        for (int o = 16; o > 0; o >>= 1) {   // the first row of the largest entry
            const double x = __shfl_xor_sync(0xffffffffu, best, o);
            const int r = __shfl_xor_sync(0xffffffffu, piv, o);
            if (x > best || (x == best && r < piv)) {
                best = x;
                piv = r;
            }
        }
        if (best < 1e-14) return false;
        if (piv != k && lane <= n) {
            const double x = A[k][lane];
            A[k][lane] = A[piv][lane];
            A[piv][lane] = x;
        }
        __syncwarp();
        if (lane > k && lane < n) {
            const double f = A[lane][k] / A[k][k];
            for (int j = k; j <= n; j++) A[lane][j] -= f * A[k][j];
        }
        __syncwarp();
    }
    bool ok = true;
    if (lane == 0) {
        for (int k = n - 1; k >= 0; k--) {
            double x = A[k][n];
            for (int j = k + 1; j < n; j++) x -= A[k][j] * A[j][n];
            A[k][n] = x / A[k][k];
        }
        for (int j = 0; j < nvec; j++) ok = ok && isfinite(A[j][n]);
        if (ok)
            for (int j = 0; j < nvec; j++) c[j] = A[j][n];
    }
    return __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
}

// The end of an iteration, one CTA per solve: the energy and max|dT| from the chunk partials in
// chunk order, the new row of the Pulay matrix from the dot-product partials, the convergence
// decision and the Pulay coefficients.  init = 1: the start amplitudes' energy, recorded, and
// whether to iterate.  applied = the solves this iteration updated (k_diis_extrap runs on
// those); active = the ones that go on.  *stopped counts the others; the last of them sets *done,
// in host memory, so that the host learns of it without a copy.
// One launch with the elimination spread over a warp in shared memory, where the reduction, the
// row reduction, a one-thread-per-solve control (its 17 x 18 matrix in local memory) and the
// swap of the active flags were four launches: 22 -> 10.5 us an iteration on one N=54 solve,
// 58 -> 26 us on four of N=114.
__global__ void __launch_bounds__(256)
    k_tail(const int *__restrict__ chunk_begin, const double *__restrict__ part_e, const double *__restrict__ part_dt,
           const double *__restrict__ part_r, const double *__restrict__ dpart, IterState *__restrict__ st,
           double *__restrict__ Bm, double *__restrict__ coef, double *__restrict__ rec_e,
           double *__restrict__ rec_dt, int max_rec, uint8_t *active, uint8_t *__restrict__ applied,
           int *__restrict__ stopped, int *done, double tol, int max_iter, int ndiis, int init)
{
    const int s = blockIdx.x;
    if (!init && !active[s]) {
        if (threadIdx.x == 0) applied[s] = 0;
        return;
    }
    __shared__ double sd[8][kMaxDiis], brow[kMaxDiis], A[kMaxDiis + 1][kMaxDiis + 2];
    IterState S = st[s];
    const int c0 = chunk_begin[s], c1 = chunk_begin[s + 1];
    // this iteration pushed slot (niter - 1) % ndiis and has nvec = min(niter, ndiis) vectors
    const int nvec = !init && ndiis > 0 ? min(S.niter, ndiis) : 0, slot = nvec > 0 ? (S.niter - 1) % ndiis : 0;
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (nvec > 0) {
        double acc[kMaxDiis];
#pragma unroll
        for (int j = 0; j < kMaxDiis; j++) acc[j] = 0.0;
        for (int c = c0 + threadIdx.x; c < c1; c += 256) {
#pragma unroll
            for (int j = 0; j < kMaxDiis; j++)
                if (j < nvec) acc[j] += dpart[(int64_t)c * kMaxDiis + j];
        }
#pragma unroll
        for (int j = 0; j < kMaxDiis; j++)
            if (j < nvec) {
                double v = acc[j];
                for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
                if (l == 0) sd[w][j] = v;
            }
        __syncthreads();
        for (int j = w; j < nvec; j += 8) {
            double v = l < 8 ? sd[l][j] : 0.0;
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            if (l == 0) brow[j] = v;
        }
    }
    double e = 0.0, dt = 0.0, mr = 0.0;
    for (int c = c0 + threadIdx.x; c < c1; c += 256) {
        e += part_e[c];
        dt = fmax(dt, part_dt[c]);
        mr = fmax(mr, part_r[c]);
    }
    block_reduce3<256>(e, dt, mr);
    __syncthreads();   // brow
    if (w != 0) return;
    e = __shfl_sync(0xffffffffu, e, 0);
    dt = __shfl_sync(0xffffffffu, dt, 0);
    if (!init) S.niter += 1;
    const int r = S.niter - 1;
    if (l == 0 && r >= 0 && r < max_rec) {
        rec_e[(int64_t)s * max_rec + r] = e;
        rec_dt[(int64_t)s * max_rec + r] = dt;
    }
    S.e = e;
    S.dt = dt;
    const bool finite = isfinite(e) && isfinite(dt);
    const bool go = finite && dt >= tol && S.niter < max_iter;
    if (!finite) S.status = 3;
    if (nvec > 0) {
        double *B = Bm + (int64_t)s * kMaxDiis * kMaxDiis;
        double *c = coef + s * kMaxDiis;
        if (l < nvec) B[slot * kMaxDiis + l] = B[l * kMaxDiis + slot] = brow[l];
        if (l < kMaxDiis) c[l] = 0.0;
        __syncwarp();
        const bool solved = go && nvec >= 2 && pulay_warp(B, nvec, c, A);
        if (!solved && l == 0) c[slot] = 1.0;
    }
    if (!go && S.status == 0) S.status = (finite && dt >= tol) ? 2 : 1;
    if (l == 0) {
        st[s] = S;
        applied[s] = init ? 0 : 1;
        active[s] = go ? 1 : 0;
        if (!go && atomicAdd(stopped, 1) + 1 == (int)gridDim.x) {
            *(volatile int *)done = 1;
            __threadfence_system();
        }
    }
}

__global__ void k_copy(int64_t n, const double *__restrict__ src, double *__restrict__ dst)
{
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < n) dst[p] = src[p];
}

int launch_refresh(const DevBatch &d, cudaStream_t st)
{
    k_copy<<<(unsigned)((d.namp + 255) / 256), 256, 0, st>>>(d.namp, d.t, d.t_ref);
    return 1 + launch_ladder(d, d.t_ref, 1, 0, d.g_ref, st, st);
}

void launch_tail(const DevBatch &d, const CtlBuffers &c, double tol, int max_iter, int ndiis, int init,
                 cudaStream_t st)
{
    if (init) cudaMemsetAsync(c.stopped, 0, sizeof(int), st);
    k_tail<<<d.nsolves, 256, 0, st>>>(d.utile_begin, d.part_e, d.part_dt, d.part_r, c.part,
                                      c.state, c.Bm, c.coef, c.rec_e, c.rec_dt, c.max_rec, d.active, c.applied,
                                      c.stopped, c.done, tol, max_iter, ndiis, init);
}

// One iteration: residual + update, control, [DIIS extrapolation].  Returns launches.
int launch_iteration(const DevBatch &d, const CtlBuffers &c, const TermFlags &f, double tol, int max_iter,
                     int ndiis, cudaStream_t st, KernelTimer *kt, const Fork *fork)
{
    // the DIIS push (history slot and e . e_j partials) happens inside k_update
    int n = launch_residual(d, f, 0, nullptr, st, kt, &c, ndiis, fork);
    if (kt) kt->begin(KID_TAIL, st);
    launch_tail(d, c, tol, max_iter, ndiis, 0, st);
    if (kt) kt->end(st);
    n++;
    if (ndiis > 0) {
        if (kt) kt->begin(KID_EXTRAP, st);
        launch_extrap(d, c, ndiis, st);
        if (kt) kt->end(st);
        n++;
    }
    return n;
}

// ----------------------------------------------------------------------------
// Layout conversion between the packed amplitudes and the reference's
// T(NOcc,NOcc,NOcc+1:NAO) column-major arrays (one solve).
// ----------------------------------------------------------------------------
__global__ void k_pack(const SolveDev *__restrict__ solves, int sidx, const AmpInfo *__restrict__ amps,
                       const double *__restrict__ dense, double *__restrict__ t)
{
    const SolveDev s = solves[sidx];
    int loc = blockIdx.x * blockDim.x + threadIdx.x;
    if (loc >= s.namp) return;
    int64_t p = s.amp0 + loc;
    AmpInfo q = amps[p];
    // core pairs are held at zero (their integrals are zero; see uegccd_internal.h)
    t[p] = (q.i < s.core_n || q.j < s.core_n) ? 0.0 : dense[q.i + (int64_t)s.O * q.j + (int64_t)s.O * s.O * (q.a - s.O)];
}

// writes T2abab, T2abba = -t(ij,b), T2aaaa = t(ij,a) - t(ij,b) (any may be null);
// the dense arrays must be zeroed before (entries of forbidden (i,j,a) stay 0).
__global__ void k_unpack(const SolveDev *__restrict__ solves, int sidx, const AmpInfo *__restrict__ amps,
                         const int32_t *__restrict__ partner, const double *__restrict__ t,
                         double *__restrict__ d_abab, double *__restrict__ d_abba, double *__restrict__ d_aaaa)
{
    const SolveDev s = solves[sidx];
    int loc = blockIdx.x * blockDim.x + threadIdx.x;
    if (loc >= s.namp) return;
    int64_t p = s.amp0 + loc;
    AmpInfo q = amps[p];
    int64_t x = q.i + (int64_t)s.O * q.j + (int64_t)s.O * s.O * (q.a - s.O);
    double ta = t[p], tb = t[partner[p]];
    if (d_abab) d_abab[x] = ta;
    if (d_abba) d_abba[x] = -tb;
    if (d_aaaa) d_aaaa[x] = ta + (-tb);
}

// T2abab of every solve in the reference layout, solve after solve (dense_off[s]).
__global__ void k_unpack_all(const ChunkDev *__restrict__ chunks, const SolveDev *__restrict__ solves,
                             const int64_t *__restrict__ dense_off, const AmpInfo *__restrict__ amps,
                             const double *__restrict__ t, double *__restrict__ out)
{
    const ChunkDev ch = chunks[blockIdx.x];
    const SolveDev s = solves[ch.solve];
    const int loc = ch.start + threadIdx.x;
    if (loc >= s.namp) return;
    const int64_t p = s.amp0 + loc;
    const AmpInfo q = amps[p];
    out[dense_off[ch.solve] + q.i + (int64_t)s.O * q.j + (int64_t)s.O * s.O * (q.a - s.O)] = t[p];
}

void launch_unpack_all(const DevBatch &d, const int64_t *dense_off, const double *t, double *out, cudaStream_t st)
{
    k_unpack_all<<<d.nchunks, kChunk, 0, st>>>(d.chunks, d.solves, dense_off, d.amps, t, out);
}

// ----------------------------------------------------------------------------
// Structure factors on the momentum-transfer grid (CCEnergyAndSF, CCD.f90:290-331;
// DrvMBPT, MP2.f90:86-95).  For every stored (i,j,a) the reference adds
//   at q = n_a - n_i:  SfSum += T2aaaa + T2abab,  SfDSum += 2 T2abab,  SfXSum += T2aaaa - T2abab
//   at q = n_a - n_j:  SfSum -= T2aaaa + T2abba,  SfDSum -= 2 T2abba,  SfXSum -= T2aaaa - T2abba
// with T2abba(i,j,a) = -t(ij,b) and T2aaaa = T2abab + T2abba (CCD.f90:90).
// Particle-hole row (i,x) of group Q = n_x - n_i, with occupied k, holds the direct
// transfer of t(ik,x) and the exchange transfer of t(ki,x): every contribution to grid
// point Q comes from the rows of group Q.  One CTA per group therefore owns its grid
// point and writes it without atomics, summing in a fixed order.
// ----------------------------------------------------------------------------
constexpr int kSfThreads = 128;

__global__ void __launch_bounds__(kSfThreads)
    k_sf(const int2 *__restrict__ groups, const SolveDev *__restrict__ solves, int solve,
         const int16_t *__restrict__ ph_i, const int16_t *__restrict__ ph_x, const int4 *__restrict__ nv4,
         const int32_t *__restrict__ ridx_x, const int32_t *__restrict__ ridx_y,
         const int32_t *__restrict__ partner, const double *__restrict__ t, int S, double *__restrict__ grid,
         int *__restrict__ err)
{
    const int2 G = groups[blockIdx.x];   // rows [G.x, G.x + G.y) of the solve
    const SolveDev s = solves[solve];
    const int O = s.O, V = s.V;
    double sum = 0.0, dsum = 0.0, xsum = 0.0, cnt = 0.0;
    // position of the last contribution in the reference's loop order (I, J, A, then
    // direct before exchange): its SfV assignment is the one that stays
    long long last = -1;
    const int n = G.y * O;
    for (int e = threadIdx.x; e < n; e += kSfThreads) {
        const int r = G.x + e / O, k = e - (e / O) * O;
        const int64_t ri = s.ph0 + (int64_t)r * O + k;
        const int ir = ph_i[s.phr0 + r], xr = ph_x[s.phr0 + r] - O;
        const int pd = __ldg(&ridx_x[ri]);
        if (pd >= 0) {  // direct: (I,J,A) = (i,k,x)
            const double tab = __ldg(&t[pd]), tba = -__ldg(&t[__ldg(&partner[pd])]);
            const double taa = tab + tba;
            sum += taa + tab;
            dsum += 2.0 * tab;
            xsum += taa - tab;
            cnt += 1.0;
            last = max(last, (((long long)ir * O + k) * V + xr) * 2);
        }
        const int px = __ldg(&ridx_y[ri]);
        if (px >= 0) {  // exchange: (I,J,A) = (k,i,x)
            const double tab = __ldg(&t[px]), tba = -__ldg(&t[__ldg(&partner[px])]);
            const double taa = tab + tba;
            sum -= taa + tba;
            dsum -= 2.0 * tba;
            xsum -= taa - tba;
            cnt += 1.0;
            last = max(last, (((long long)k * O + ir) * V + xr) * 2 + 1);
        }
    }
    __shared__ double red[4][kSfThreads / 32];
    __shared__ long long red_last[kSfThreads / 32];
    double v[4] = {sum, dsum, xsum, cnt};
#pragma unroll
    for (int q = 0; q < 4; q++)
        for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
    for (int o = 16; o > 0; o >>= 1) last = max(last, __shfl_down_sync(0xffffffffu, last, o));
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) {
#pragma unroll
        for (int q = 0; q < 4; q++) red[q][w] = v[q];
        red_last[w] = last;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    double tot[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        tot[q] = red[q][0];
        for (int k = 1; k < kSfThreads / 32; k++) tot[q] += red[q][k];
    }
    for (int k = 1; k < kSfThreads / 32; k++) last = max(last, red_last[k]);
    last = max(last, red_last[0]);
    if (tot[3] == 0.0) return;   // no stored amplitude reaches this transfer
    // the last tuple (I,J): a core pair leaves SfV = 0 (its integral is zero under CoreN)
    const long long ij = (last >> 1) / V;
    const bool last_core = (int)(ij / O) < s.core_n || (int)(ij % O) < s.core_n;
    const int i = ph_i[s.phr0 + G.x], x = ph_x[s.phr0 + G.x];
    const int4 a = nv4[s.orb0 + x], b = nv4[s.orb0 + i];
    const int q0 = a.x - b.x, q1 = a.y - b.y, q2 = a.z - b.z;
    if (q0 < -S || q0 > S || q1 < -S || q1 > S || q2 < -S || q2 > S) {
        atomicExch(err, 1);
        return;
    }
    const int64_t W = 2 * S + 1, W3 = W * W * W;
    const int64_t c = (q0 + S) + W * ((q1 + S) + W * (int64_t)(q2 + S));
    grid[c] = tot[0];
    grid[W3 + c] = tot[1];
    grid[2 * W3 + c] = tot[2];
    grid[3 * W3 + c] = tot[3];
    grid[4 * W3 + c] = last_core ? 1.0 : 0.0;
}

void launch_sf(const DevBatch &d, const int2 *groups, int ngroups, int solve, int S, double *grid, int *err,
               cudaStream_t st)
{
    if (ngroups > 0)
        k_sf<<<ngroups, kSfThreads, 0, st>>>(groups, d.solves, solve, d.ph_i, d.ph_x, d.nv4, d.ridx_x, d.ridx_y,
                                            d.partner, d.t, S, grid, err);
}

// ----------------------------------------------------------------------------
// Launch wrappers
// ----------------------------------------------------------------------------
void launch_reduce(const DevBatch &d, cudaStream_t st)
{
    k_reduce_solves<<<d.nsolves, 256, 0, st>>>(d.utile_begin, d.part_e, d.part_dt, d.part_r, d.red);
}

void launch_drpa_tables(const DevBatch &d, cudaStream_t st)
{
    if (d.nblocks > 0)
        k_drpa_tables<<<d.nblocks, 256, 0, st>>>(d.blocks, d.solves, d.drsolves, d.pair_i, d.pair_j, d.vir, d.drows,
                                                 d.colpos);
}

void launch_to_aaaa(const DevBatch &d, cudaStream_t st)
{
    k_to_aaaa<<<(unsigned)((d.namp + 255) / 256), 256, 0, st>>>(d.namp, d.partner, d.t);
}

const char *kKernelNames[KID_COUNT] = {"k_mp2",      "k_energy",   "k_ladder",
                                      "k_mosaic_blk", "k_mosaic_sum", "k_drpa_sums", "k_update",
                                      "k_reduce_solves", "k_rings",
                                      "k_ladder_tc", "k_ring_stage", "k_tail", "k_diis_extrap"};

int tune_stage(DevBatch &d, cudaStream_t st)
{
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaError_t err = cudaEventCreate(&e0);
    if (err == cudaSuccess) err = cudaEventCreate(&e1);
    // the staging kernel's CTA size
    if (err == cudaSuccess && d.nrpairs > 0) {
        float best = 1e30f;
        for (int th : {64, 128, 256}) {
            auto run = [&]() {
                k_ring_stage<<<d.nrpairs, th, 0, st>>>(d.spairs, d.solves, d.ph_i, d.ridx_x, d.ridx_y, d.t, d.xy,
                                                       d.active);
            };
            run();
            cudaEventRecord(e0, st);
            run();
            run();
            cudaEventRecord(e1, st);
            if ((err = cudaEventSynchronize(e1)) != cudaSuccess) break;
            float ms = 0.f;
            cudaEventElapsedTime(&ms, e0, e1);
            if (ms < best) {
                best = ms;
                d.stage_threads = th;
            }
        }
    }
    if (err == cudaSuccess) err = cudaGetLastError();
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    return (int)err;
}

int launch_residual(const DevBatch &d, const TermFlags &f, int mode, double *g_out, cudaStream_t st,
                    KernelTimer *kt, const CtlBuffers *diis, int ndiis, const Fork *fork)
{
    KernelTimer dummy;
    if (!kt) kt = &dummy;
    int n = 0, classes = 0;
    for (int k : d.nritems) classes += k > 0;
    const bool side = fork && !kt->on && !f.drpa, apart = side && fork->terms && f.do_ladder;
    const cudaStream_t rs = apart ? fork->s[0] : st, ms = apart ? fork->s[1] : st;
    const cudaStream_t ls = apart && !f.mixed ? fork->s[2] : st;   // (the mixed ladder adds to what both forms leave)
    if (apart) {
        cudaEventRecord(fork->start, st);
        for (int k = 0; k < 3; k++) cudaStreamWaitEvent(fork->s[k], fork->start, 0);
    }
    if (f.do_ladder && d.nblocks > 0) {
        kt->begin(KID_LADDER, st);
        n += launch_ladder(d, d.t, (f.do_pp && !f.mixed) ? 1 : 0, f.do_hh, d.g, st, ls);
        kt->end(st);
        if (f.do_pp && f.mixed) {
            kt->begin(KID_LADDER_TC, st);
            n += launch_ladder_tc(d, d.t_ref, d.g_ref, d.tc_err, st);
            kt->end(st);
        }
    }
    if (f.do_mosaic && !f.drpa) {
        kt->begin(KID_MOSAIC_S, ms);
        k_mosaic_blk<<<d.nblocks, kMosThreads, 0, ms>>>(d.blocks, d.solves, d.vpk, d.rowpk, d.vtab, d.t, d.mpart,
                                                        d.active);
        kt->end(ms);
        kt->begin(KID_MOSAIC_RED, ms);
        k_mosaic_sum<<<(d.ntargets + 7) / 8, 256, 0, ms>>>(d.targets, d.ntargets, d.solves, d.mt_start, d.mt_list,
                                                           d.mpart, d.jvv, d.joo, d.active);
        kt->end(ms);
        n += 2;
    }
    if ((f.do_ring || f.do_mosaic) && f.drpa) {
        kt->begin(KID_DRPA_SUMS, st);
        k_drpa_sums<<<d.ndrlist, kDrpaThreads, 0, st>>>(d.drlist, d.solves, d.drsolves, d.drows, d.colpos, d.nv4,
                                                        d.vtab, d.t, d.dru, d.drs2, d.drj, d.jvv, d.joo, d.drdone,
                                                        d.ndrranges, d.active);
        kt->end(st);
        n++;
    }
    if ((f.do_ring || f.do_xring) && !f.drpa) {
        kt->begin(KID_RING_STAGE, rs);
        k_ring_stage<<<d.nrpairs, d.stage_threads, 0, rs>>>(d.spairs, d.solves, d.ph_i, d.ridx_x, d.ridx_y, d.t, d.xy,
                                                            d.active);
        kt->end(rs);
        n++;
        kt->begin(KID_RINGS, rs);
        const cudaStream_t lanes[3] = {rs, side ? fork->s[3] : rs, side ? fork->s[4] : rs};
        const int nl = side ? std::min(classes, 3) : 1;
        if (nl > 1) cudaEventRecord(fork->staged, rs);
        for (int k = 1; k < nl; k++) cudaStreamWaitEvent(lanes[k], fork->staged, 0);
        n += launch_rings(d, lanes, nl);
        for (int k = 1; k < nl; k++) {
            cudaEventRecord(fork->done[k + 2], lanes[k]);
            cudaStreamWaitEvent(rs, fork->done[k + 2], 0);
        }
        kt->end(rs);
    }
    if (apart) {
        for (int k = 0; k < 3; k++) {
            cudaEventRecord(fork->done[k], fork->s[k]);
            cudaStreamWaitEvent(st, fork->done[k], 0);
        }
    }
    kt->begin(KID_UPDATE, st);
    launch_update(d, f, mode, g_out, diis, ndiis, st);
    kt->end(st);
    n++;
    if (mode != 0) {   // in an iteration k_tail reduces the partials
        kt->begin(KID_REDUCE, st);
        k_reduce_solves<<<d.nsolves, 256, 0, st>>>(d.utile_begin, d.part_e, d.part_dt, d.part_r, d.red);
        kt->end(st);
        n++;
    }
    return n;
}

void launch_pack(const DevBatch &d, int s, int namp, const double *dense, cudaStream_t st)
{
    k_pack<<<(namp + 255) / 256, 256, 0, st>>>(d.solves, s, d.amps, dense, d.t);
}

void launch_unpack(const DevBatch &d, int s, int namp, const double *t, double *ab, double *ba, double *aa,
                   cudaStream_t st)
{
    k_unpack<<<(namp + 255) / 256, 256, 0, st>>>(d.solves, s, d.amps, d.partner, t, ab, ba, aa);
}

}  // namespace uegccd
