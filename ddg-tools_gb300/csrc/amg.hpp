// Smoothed-aggregation algebraic multigrid for the preconditioner's Laplacian block
// K = W + eps M (RS/src/solve/precond.rs:157-460 factors L' by a sparse LDL^T on the CPU; this
// library solves it with multigrid V-cycles on the device instead, see saddle.cu).
#pragma once
#include <cstdint>
#include <vector>

#include "common.hpp"

namespace rsg {

// Storage and arithmetic type of the device hierarchy and its conjugate-gradient vectors: FP32.
// The multigrid solve is a preconditioner inside flexible FP64 GMRES, so its rounding only
// perturbs the preconditioner; GB300 runs FP32 at many times its FP64 rate. Dot products
// are added up in FP64 across blocks.
using mgreal = float;

struct Csr {
  int n = 0, m = 0;  // rows, columns
  std::vector<int> ptr, col;
  std::vector<double> val;
};

// Host setup: strength (|a_ij| >= 0.08 sqrt(a_ii a_jj)), greedy aggregation, the tentative
// prolongator of the constant near-null space, one damped-Jacobi smoothing step
// (omega = 4 / (3 rho(D^-1 A))), Galerkin coarse operators, down to at most `coarse_max` rows;
// the coarsest operator is inverted densely after adding z z^T (z its null vector).
struct AmgHost {
  std::vector<Csr> A, P, R;  // A[l] n_l x n_l, P[l] n_l x n_{l+1}, R[l] = P[l]^T
  std::vector<std::vector<double>> dinv;  // damped inverse diagonals of A[l]
  std::vector<double> coarse_inv;         // dense n_L x n_L
};
// groups (optional, one label per row): rows that form separate near-null blocks (the
// components of a surface whose barycenters are held one by one); the coarsest level is then
// regularised along the constant of every group instead of the global constant only.
AmgHost amg_setup(const Csr &A, int coarse_max = 300, int max_levels = 12,
                  const std::vector<uint32_t> *groups = nullptr);

// The hierarchy on the device: conjugate gradients preconditioned by V-cycles of two damped Jacobi
// sweeps before and after each coarser solve and a dense coarse solve, in one persistent kernel
// (amg.cu). Each sparse product gives a row to a group of 1-32 lanes sized to the matrix's mean row
// length (the coarse operators of smoothed aggregation have 40-70 nonzeros per row on a few
// hundred rows, where one thread per row would leave the GPU idle behind long serial loops).
struct AmgDevice {
  struct Mat {  // CSR with the column and the value of a nonzero side by side
    DevBuf<int> ptr;
    DevBuf<int2> cv;
    size_t nnz = 0;
    int tpr = 1;  // lanes per row
    void upload(const Csr &A, cudaStream_t s);
  };
  struct Level {
    int n = 0;
    Mat a, p, r;  // A_l, P_l (rows of level l), R_l (rows of level l + 1)
    DevBuf<mgreal> dinv;
    DevBuf<mgreal> x, b, res, t;  // up to 12 columns each
  };
  std::vector<Level> L;
  DevBuf<mgreal> cinv;
  void upload(const AmgHost &h, cudaStream_t s);
  // x ~ A_0^-1 b by `iters` steps of conjugate gradients per column, preconditioned by one
  // V-cycle each (x_0 = 0; iters = 1 is the V-cycle with the optimal step length), for n_0 x C
  // device arrays, C = 3, 6, 9 or 12 interleaved columns per row (x[row * C + c]). The
  // scalars stay on the device (no host synchronization); a fixed number of steps makes it a
  // nonlinear map of b, which flexible GMRES (the stored preconditioned vectors) allows.
  void pcg(rs_ctx *ctx, const mgreal *b, mgreal *x, int C, int iters);
  // Fails when an earlier solve gave up at a barrier, once for every such report (to be called when the stream
  // has been waited for; pcg calls it too, for the solves that nothing waited for).
  void check();
  unsigned wait_polls = 1u << 22;  // a wait across the grid gives up after that many polls (about two seconds)
  AmgDevice() = default;
  AmgDevice(const AmgDevice &) = delete;
  AmgDevice &operator=(const AmgDevice &) = delete;
  ~AmgDevice();

 private:
  template <int C>
  void launch(rs_ctx *ctx, const mgreal *b, mgreal *x, int iters);
  DevBuf<mgreal> cg_p, cg_q;  // with level 0's b and x as the residual and its preconditioned form
  DevBuf<double> cg_part;     // per-chunk partial sums of the dot products
  DevBuf<unsigned long long> counter;  // arrivals at the grid barrier
  int *error = nullptr, *error_dev = nullptr;  // mapped host memory: set by a solve that gave up
  int grid = 1, threads = 256, smem_bytes = 0;
  // one cluster of blocks where its shared memory holds three columns: the bytes (0: it does not)
  int cluster_threads = 256, cluster_smem = 0;
  cudaLaunchConfig_t cluster_config(cudaStream_t s, cudaLaunchAttribute &at) const;
};

}  // namespace rsg
