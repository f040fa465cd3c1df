// llg_adjblock.h -- launchers of the block form of the adjoint sweep (llg_adjblock.cu): IEEE
// complex128 states of 12 and more qubits, `sets` of them side by side.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>

#include <cuda_runtime.h>

#include "llg_internal.h"
#include "llg_launch.h"

namespace llg {

// CTAs a state for `tiles` tiles of 128 groups on each of `sets` states
int block_ctas(uint64_t tiles, int sets, int sms);
int cross_ctas(int n, int sets, int sms);  // of launch_cross

// R = sum over the groups of psi lambda^+ on the block's qubits, 32 x 32 a set (high parts, then low
// parts).  log2_bound: an integer at least log2(|psi| |lambda|); exps: per set the largest biased exponents of psi, then of lambda; partial: sets x ctas x 16 KB
cudaError_t launch_cross(const void* psi, const void* lam, int n, int sets, int ctas, const BlockDesc& bd, int log2_bound,
                         const uint32_t* exps, void* partial, double2* R, int* err_flag, cudaStream_t s);
// raises exps (2 sets words, zeroed by the caller) to the largest biased exponents
cudaError_t launch_max_exponent(const void* psi, const void* lam, int n, int sets, uint32_t* exps, cudaStream_t s);
// (cos, sin) of half the angles; occ_code: 2 parameter + anything
cudaError_t launch_angles(const double* params, int nparams, const int* occ_code, int nocc, int sets, double2* out, cudaStream_t s);
// |0..0> in every set (zeroed before); NaN in one whose angles are not all finite
cudaError_t launch_block_init(double2* psi, int n, const double2* angles, int nocc, int sets, cudaStream_t s);
// dE/dtheta of every parametrised gate, grads[set][occurrence], from R[step][set]
cudaError_t launch_block_grads(const double2* R, const BlockStep* steps, int nsteps, const BlockGate* gates, const double2* angles,
                               int nocc, int sets, double* grads, cudaStream_t s);

}  // namespace llg
