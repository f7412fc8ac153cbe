// Host interface of the cluster-resident step (vv_cluster.cuh), compiled in
// its own translation unit.
#pragma once
#include <cuda_runtime.h>
#include <cstddef>

namespace vv {

struct ClInst;

// Shape of an instance on a cluster of `ctas` CTAs (ctas = 0: does not fit).
struct ClShape {
    int ctas, fam, rows, nch, slots;
    int kv, dsm;   // basis vectors and LU reciprocals kept in shared memory
    size_t smem;
};
ClShape cl_shape(int nx, int nv, bool pow2, int ctas, int tsz, size_t smem_limit);
// row kind of a grid (the kernel that runs it)
int cl_family(int nx, bool pow2);
// most clusters of that many CTAs resident on the current device, each CTA with
// the largest shared memory (0: none): a lower bound for every shape
int cl_resident(bool fp32, int fam, int ctas);
// largest dynamic shared memory of the kernel on the current device (0: it does not load)
size_t cl_smem_limit(bool fp32, int fam);
// carry levels of the v solves: the number of chunks over which every product
// of the LU multipliers falls below tol.  lf, lb: per v row, the largest
// squared forward and backward multiplier over the modes (their products
// bound the modes' own).
int cl_levels(const ClShape& s, int nv, const double* lf, const double* lb, double tol);
// slot-ordered tables from the mode-major LU reciprocals and the eigenvalues, on
// stream st (not waited for)
cudaError_t cl_tables(bool fp32, const ClShape& s, int nv, const void* dinv, const void* lambda, void* dinv_s,
                      void* lam_s, double ht, cudaStream_t st);
// one cluster per instance of tab, all of row kind fam (in the order `order`, or 0..n-1)
cudaError_t cl_launch(bool fp32, int fam, const ClInst* tab, const int* order, int n, int ctas, size_t smem, int mode,
                      cudaStream_t st);

}  // namespace vv
