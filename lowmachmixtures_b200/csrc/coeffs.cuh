// coeffs.cuh - launchers of the coefficient hierarchy (coeffs.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "stencil.cuh"

namespace lmm {

// Finest level: the caller's coefficients in, the level's arrays out.  o_:
// FP64, f_: FP32 (null: no FP32 copy).  o_pa null: 1/alpha (o_ainv) serves as
// the pressure's face coefficient; else it differs from it at walls.  flag_* =
// 1 when the level's theta*alpha (a), 1/alpha (p) are not one value on every
// face, val_* that value; the flags are zero before.
struct CoefFine {
    Dims D;
    double theta;
    const double* alpha[3];
    const double* beta;
    const double* gamma;   // null: zero
    const double* bed[3];
    int64_t ne[3];         // entries of the edge arrays
    double *o_alpha[3], *o_ainv[3], *o_pa[3], *o_beta, *o_gamma, *o_bed[3];
    float *f_alpha[3], *f_ainv[3], *f_pa[3], *f_beta, *f_gamma, *f_bed[3];
    int *flag_a, *flag_p;
    double *val_a, *val_p;
};
void launch_coeffs_fine(const CoefFine& A, cudaStream_t s);

// A coarse level (C) from the level above it (F); alpha[0] null: no velocity
// level, pa[0] null: no pressure level.
struct CoefCoarse {
    Dims F, C;
    const double *alpha[3], *beta, *gamma, *bed[3], *pa[3];
    double *o_alpha[3], *o_beta, *o_gamma, *o_bed[3], *o_pa[3];
    float *f_alpha[3], *f_beta, *f_gamma, *f_bed[3], *f_pa[3];
    int *flag_a, *flag_p;
    double *val_a, *val_p;
};
void launch_coeffs_coarse(const CoefCoarse& A, cudaStream_t s);

// dst[q][0..n) = src[q][0..n), q < count <= 8, in one launch
struct CopyFields {
    const double* src[8];
    double* dst[8];
    int64_t n;
};
void launch_copy_fields(const CopyFields& A, int count, cudaStream_t s);

}  // namespace lmm
