// two_channel_mm.h -- the two-channel CCD residual as matrix products (two_channel_mm.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "two_channel.h"

namespace uegccd {

constexpr size_t kTcMmSmemMax = 220 * 1024;   // dynamic shared memory a CTA may ask for

// Device arrays of one system.
struct TcMm {
    int O, V, n, nq;
    const int *F;               // FindIndex table of the system (two_channel.cu)
    const int4 *nv;
    const double *vt;           // integral tables by flag (no core orbital)
    // ladders: W by rows c < kdim (ldw columns), T by rows c (ldt columns), C = W^T T
    int sets, ldw, ldt, kdim;   // sets = 2 when the exchange flags differ from the direct ones
    double *w, *t, *c;
    double *jpart;              // V x O mosaic terms
    int *done;
    // pairs (k,l) of each pair's momentum: [kl0[ij], kl0[ij+1]), k | l << 16, and the ij of each
    int nkl;
    const int *kl0, *kl, *kl_ij;
    double *h2, *h3;
    // rings: pairs {first row of Q, rows, first row of -Q, rows}; rows i | x << 16
    int npairs;
    const int4 *pairs;
    const int *ph;
    size_t ring_smem;
    double *gr[2], *gx[2];      // ring and crossed-ring G of both channels
};

size_t tc_mm_ring_smem(int n1, int n2);
size_t tc_mm_stage_smem(int O);
cudaError_t tc_mm_limits();
void tc_mm_weights(const TcMm &D, const TcFlags &f, cudaStream_t st);
// G of the terms in mask (two_channel.h); returns the launches.
int tc_mm_residual(const TcMm &D, const TcFlags &f, int mask, const double *tab, const double *tba, double *jvv,
                   double *joo, double *gab, double *gba, cudaStream_t st);

}  // namespace uegccd
