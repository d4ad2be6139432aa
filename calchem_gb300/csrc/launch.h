// launch.h -- host-side launchers of the device kernels, shared by the C ABI translation units.
#pragma once

#include <cuda_runtime.h>

#include "common.cuh"

namespace cxc {
// FP64 form (vxc_fp64.cu)
cudaError_t launch_fp64(const DevGrid& G, const EvalArgs& A, int n_ctas, cudaStream_t st);
size_t fp64_smem_bytes();
// The end of an evaluation in one kernel: the per-molecule deterministic (Exc, N_a, N_b) sums (batches
// [batch_off[i], batch_off[i + 1]) to out[i * n_out ...]; part = nullptr: none) and the completion of each
// molecule's V blocks (V[0] = nullptr: none).  mol_n, mol_off, batch_off = nullptr for one molecule.
enum FinishKind : int {
  kFinishFromLower = 0,  // the lower triangle copied into the upper one (FP64 SIMT form)
  kFinishFromUpper = 1,  // the upper into the lower (tensor-core form)
  kFinishSum = 2,        // V + V^T (FP64 form on the tensor cores)
  kFinishSumLower = 3    // the same in the lower triangle, zeros above it (the drop-in accumulation)
};
struct FinishArgs {
  const double* part;
  int n_batches;
  const int* batch_off;
  int n_mols;
  double* out;
  int n_out;
  double* V[2];  // per spin (V[1] = nullptr: one)
  int n;         // AOs (of the largest molecule)
  const int* mol_n;
  const long long* mol_off;
  int kind;
};
cudaError_t launch_finish(const FinishArgs& F, cudaStream_t st);
// Per-atom (Exc, tr(D Vxc)) shares: out[2 a ..] = sums of point_out over atom a's points.
cudaError_t launch_atom_shares(const double* point_out, const int* atom_pts, const int* atom_off, int n_atoms,
                               double* out, cudaStream_t st);
// FP64 form with its contractions on the tensor cores (vxc_f64tc.cu): A.Pa points at the fixed-point
// densities of launch_f64tc_prepare (alpha, then beta, then the rows' exponents); V is accumulated as the
// full square and completed by launch_finish (kFinishSum).
int f64tc_max_m();
size_t f64tc_slab_bytes(int max_m);
size_t f64tc_cache_block_bytes(int m);
cudaError_t f64tc_set_attributes();
cudaError_t launch_f64tc(const DevGrid& G, const EvalArgs& A, int n_ctas, cudaStream_t st);
cudaError_t launch_f64tc_prepare(const PrepareArgs& A, cudaStream_t st);
// Tensor-core form (vxc_mixed.cu)
int mixed_supported(int mode);
size_t mixed_slab_doubles(int max_m);
int mixed_ctas_per_sm(int tile_n);
int mixed_max_m();
cudaError_t launch_closed_shell_points(int xc, int precision, int n, const double* rho, const double* gam,
                                       double* out, cudaStream_t st);
cudaError_t launch_mixed(const DevGrid& G, const EvalArgs& A, int n_ctas, cudaStream_t st);
cudaError_t launch_mixed_prepare(const PrepareArgs& A, cudaStream_t st);
// TD-DFT kernel coefficients per point (fxc.cu): rho_grad [n][4] of the total density -> out [n][11].
cudaError_t launch_fxc_coef(const double* rho_grad, const double* w, int n_pts, int code, double* out,
                            cudaStream_t st);
// XC nuclear gradient (xc_grad.cu): per-CTA scratch, shared memory, the persistent kernel and the
// batch-ordered sum of its [batch][atom][3] partials into grad.
size_t grad_slab_doubles(int max_m);
size_t grad_smem_bytes(int n_atoms);
int grad_max_atoms();
cudaError_t launch_xc_grad(const DevGrid& G, const GradArgs& A, int n_ctas, cudaStream_t st);
cudaError_t launch_grad_reduce(const double* part, int n_batches, int n_atoms, double* grad, cudaStream_t st);
// The FP64 gradient's quadrature with its contractions on the tensor cores (xc_grad_f64tc.cu): A.Pa points at
// the fixed-point densities of launch_f64tc_prepare; the weight derivative is left to A.fx_out's reader;
// *status is set on a wait expiry.
bool grad_f64tc_fits(int max_m, int n_atoms);
size_t grad_f64tc_slab_doubles(int max_m);
cudaError_t launch_xc_grad_f64tc(const DevGrid& G, const GradArgs& A, int n_ctas, int* status, cudaStream_t st);
// Tensor-core form of the gradient (xc_grad_mixed.cu): GradArgs.Pa points at the split densities of
// launch_mixed_prepare (alpha, then beta); part must be zeroed; *status is set on a wait expiry.
size_t grad_mixed_slab_doubles(int max_m);
int grad_mixed_max_m();
cudaError_t launch_xc_grad_mixed(const DevGrid& G, const GradArgs& A, int n_ctas, int* status, cudaStream_t st);
// The weight derivative from the quadrature's GradArgs.fx_out (becke_mixed.cu, becke.cu): per-CTA rows of per-atom
// sums in part [n_ctas][3 n_atoms], n_ctas = becke_*_ctas; for larger molecules becke_*_table_doubles of scratch,
// which n_ctas keeps within budget bytes (one CTA at the least).
int becke_mixed_ctas(int n_pts, int n_atoms, size_t budget);
size_t becke_mixed_table_doubles(int n_ctas, int n_atoms);
cudaError_t launch_becke_mixed(const DevGrid& G, const GradArgs& A, const double* fx, double* part, double* tables,
                               int n_ctas, cudaStream_t st);
int becke_fp64_ctas(int n_pts, int n_atoms, size_t budget);
size_t becke_fp64_table_doubles(int n_ctas, int n_atoms);
cudaError_t launch_becke_fp64(const DevGrid& G, const GradArgs& A, const double* fx, double* part, double* tables,
                              int n_ctas, cudaStream_t st);
// raw[k] = raw_in[orig[k]], host[k] = host_in[orig[k]]: the caller's per-point arrays in planned order
cudaError_t launch_grad_gather(const double* raw_in, const int* host_in, const int* orig, int n, double* raw, int* host,
                               cudaStream_t st);
// grad[k] += sum over rows r (in order) of part[r][k]
cudaError_t launch_grad_accumulate(const double* part, int n_rows, int n_atoms, double* grad, cudaStream_t st);
// Dynamic shared-memory limits of the persistent kernels, set once per process (the launchers call
// these; a graph capture calls them first so that no attribute is set while capturing).
cudaError_t fp64_set_attributes();
cudaError_t mixed_set_attributes();
}  // namespace cxc
