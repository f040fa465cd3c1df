// llg_launch.h -- host-side launchers of the state-vector kernels (llg_kernels.cu).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/llgpu.h"
#include "llg_internal.h"

namespace llg {

// Observable sum_k coef[cls[k]] * Z_{a[k]} (Z_{b[k]} if b[k] >= 0), terms grouped into at most
// kMaxZClasses coefficient classes so the kernels count parities per class in integers.
constexpr int kMaxZTerms = 64;
constexpr int kMaxZClasses = 4;
struct ZTerms {
    int32_t nterms;
    int32_t nclass;
    int32_t a[kMaxZTerms];
    int32_t b[kMaxZTerms];
    int32_t cls[kMaxZTerms];
    double coef[kMaxZClasses];
};

// Per-block partial results of a reduction: up to kRedSlots doubles per block (kCmpSlots for the
// two-state comparison); the engine's partial buffer holds kRedBlocks x kPartialSlots doubles.
constexpr int kRedSlots = 1 + kMaxZClasses;
constexpr int kCmpSlots = 6;
constexpr int kPartialSlots = 8;
constexpr int kRedBlocks = 1024;

size_t elem_bytes(int precision);

cudaError_t launch_init_basis(int P, void* psi, uint64_t size, uint64_t index, cudaStream_t s);
cudaError_t launch_exec_op(int P, void* psi, int n, const ExecOp& op, cudaStream_t s);
// threads: CTA size of the tile kernel (0: 512 for tiles of 10+ qubits, else half the tile)
// mirror: nullptr, or the device address of a host buffer that also receives the pass's output as
// FP64 (2 doubles per amplitude, full-state indexing)
// d_tables: the plan's phase tables (Plan::tables on the device), or nullptr for a plan without
// EX_PTAB ops; err_flag: a device int of the caller's that a CTA sets to 1 when its bulk tile load
// does not complete within the wait limit (the CTA then stores nothing)
cudaError_t launch_tile_pass(int P, void* psi, int n, const PassDesc& pd, const ExecOp* d_ops, const uint64_t* d_tables,
                             int threads, int* err_flag, cudaStream_t s, double* mirror = nullptr);
cudaError_t launch_from_f64(int P, const double* src, void* dst, uint64_t count, cudaStream_t s);
cudaError_t launch_to_f64(int P, const void* src, double* dst, uint64_t count, cudaStream_t s);
cudaError_t launch_probabilities(int P, const void* psi, double* out, uint64_t count, cudaStream_t s);
cudaError_t launch_scale(int P, void* psi, uint64_t count, double factor, cudaStream_t s);
// What a readout kernel leaves in pinned host memory: [norm2, W_0 .. W_{nclass-1}] (W_c = sum_i |a_i|^2 * #odd-parity terms of
// class c in i) and the state's timeout flags.
struct Readout {
    double red[kRedSlots];
    int flags[2];
};
// d_partials: device, kRedBlocks * kRedSlots doubles; d_ticket: a device word that is zero between launches
cudaError_t launch_reduce_z(int P, const void* psi, int n, const ZTerms& terms, double* d_partials, unsigned* d_ticket,
                            const int* d_flags, Readout* host, cudaStream_t s);

// Two states of equal size, any precisions: per block (kCmpSlots doubles each) Re <a|b>, Im <a|b>,
// <a|a>, <b|b>, max |a_i - b_i| and max |b_i| (over re and im parts); *nblocks = blocks written
cudaError_t launch_compare(int PA, const void* a, int PB, const void* b, uint64_t size, double* partials, int* nblocks,
                           cudaStream_t s);

int tile_max_qubits(int P);

// register-tiled pass (llg_tile_reg.cu) over a register program (to_register_program): complex64
// states, pd.t in [9, 13]; 2^(t-4) threads per CTA
cudaError_t launch_tile_reg(int P, void* psi, int n, const PassDesc& pd, const ExecOp* d_ops, cudaStream_t s,
                            double* mirror = nullptr);

// FP64 FMA operations per second of the current device (one timed launch of `iters` iterations)
cudaError_t fp64_fma_rate(int iters, double* fma_per_s);

// dense k-qubit block (llg_block.cu): bit j of a row/column index is qubit q[j]; the matrix is
// 2 * 4^k coefficient slots, row-major (re, im), packed for the state's precision
constexpr int kMaxBlockQubits = 5;
constexpr int kMaxBlockDim = 1 << kMaxBlockQubits;
struct BlockDesc {
    int32_t k;
    int32_t q[kMaxBlockQubits];
    uint64_t tmask;
};
cudaError_t launch_block(int P, void* psi, int n, const BlockDesc& bd, const uint64_t* d_mat, cudaStream_t s);
// Which entries of a block of k <= 4 qubits are nonzero (bit c of rows[r]) and real (bit c of
// real[r]); the block kernel then sums row r over those columns only.
struct BlockSparsity {
    uint32_t rows[16];
    uint32_t real[16];
};
cudaError_t launch_block_sparse(int P, void* psi, int n, const BlockDesc& bd, const uint64_t* d_mat,
                                const BlockSparsity& nz, cudaStream_t s);

// 4-qubit blocks on double-float and 3- and 4-qubit blocks on FP64 states of k + 7 or more qubits on the tensor cores
// (llg_block_tc.cu): the host slices the matrix (2 * 4^k doubles, row-major re/im) into
// block_tc_weight_bytes(k) of device input; a kernel whose products do not arrive within its
// wait limit sets *err_flag (a device int of the caller's) to 1
bool block_tc_eligible(int P, int n, int k);
size_t block_tc_weight_bytes(int P, int k);
void block_tc_prepare(int P, int k, const double* m, void* weights);
cudaError_t launch_block_tc(int P, void* psi, int n, const BlockDesc& bd, const void* d_weights, int* err_flag,
                            cudaStream_t s);

// dense 5-qubit blocks of 16-byte states on the tensor cores (llg_gateblock.cu): n >= kBlockMinQubits, bd.q
// in increasing order.  d_weights: gate_block_weight_bytes of device memory, filled by
// launch_gate_block_matrix (d_matrix: 32 x 32 row-major (re, im) doubles on the device, bit b of an
// index is bd.q[b]).  rows: the weights have row exponents of their own (launch_gate_block_matrix).  ready:
// the weights were complete before the stream's previous kernel began.  mirror: nullptr, or the device address of a mapped host buffer that also
// receives the output as FP64.  A kernel whose waits run out sets *err_flag to 1.
bool gate_block_eligible(int P, int n);
int64_t gate_block_launches();  // of this process, all forms
size_t gate_block_weight_bytes(int P);
cudaError_t launch_gate_block_matrix(int P, const double* d_matrix, void* d_weights, cudaStream_t s);
// the weights of `nblocks` blocks of a plan (d_steps: their steps, in order; d_matrices: of the kind-4
// gates), one after the other; with
// parametrised gates (kind 3) `sets` of them per block, d_angles holding (cos, sin) of the half angles,
// nocc a set; inverse: of the blocks' inverses
cudaError_t launch_gate_block_weights(int P, const BlockGate* d_gates, const BlockStep* d_steps, int nblocks, void* d_weights,
                                      cudaStream_t s, const double2* d_matrices = nullptr, const double2* d_angles = nullptr,
                                      int nocc = 0, int sets = 1, bool inverse = false);
// a block on `sets` FP64 states side by side from psi and (unless nullptr) as many from `second`, each
// set with its own weights, `ctas` CTAs a state.  max_exp: nullptr, or per state (2 sets) a word that is
// raised to the largest biased exponent stored
cudaError_t launch_gate_block_batch(void* psi, void* second, int sets, int ctas, int n, const BlockDesc& bd,
                                    const void* d_weights, bool ready, uint32_t* max_exp, int* err_flag, cudaStream_t s);
// One FP64 launch of blocks of different states: CTA i takes d_ctas[i] (device memory that was complete before the stream's
// previous kernel began, as the weights).
struct MixedCta {
    uint64_t offset;       // the state's first element
    uint64_t tmask;        // its five targets q, increasing
    uint32_t weights;      // index of the block's weights
    uint32_t first, step;  // tiles of 4096 amplitudes: first, first + step, ..
    int32_t n;
    int32_t q[5];
    int32_t pad;
};
cudaError_t launch_gate_block_mixed(void* arena, int ctas, const MixedCta* d_ctas, const void* d_weights, int* err_flag,
                                    cudaStream_t s);
cudaError_t launch_gate_block(int P, void* psi, int n, const BlockDesc& bd, const void* d_weights, bool rows, bool ready,
                              int* err_flag, cudaStream_t s, double* mirror = nullptr);

// process-wide tuning cache (llg_tune.cu), keyed by an FNV-1a hash of the workload's shape
uint64_t tune_hash(uint64_t h, uint64_t v);
uint64_t tune_hash_ops(uint64_t h, const llg_op* ops, int nops);
bool tune_cache_get(uint64_t key, llg_tune_result* out);
void tune_cache_put(uint64_t key, const llg_tune_result& r);

}  // namespace llg
