// The lexicographic SOR of FieldSolve::gssolver (src/field.cpp:70-139) on
// lattices that wrap (EPIC_POISSON_PERIODIC, EPIC_POISSON_DIRICHLET_X), iterate
// for iterate, with unit cells.
//
// A sweep updates node (i, j) from the new (i-1, j), (i, j-1) and the old
// (i+1, j), (i, j+1).  Where a row of nyi nodes wraps, its first node needs the
// last node of the sweep before, so a row holds one sweep at a time and the
// solve is a serial chain of nyi updates per sweep: row i does node j of sweep s
// at step i + j + P s, P = nyi (max(nxi, nyi) where columns wrap too), all rows
// side by side.  What counts is the length of one step.  An FP64 instruction of
// a warp holds its quarter of the SM for 64 cycles, and an update is seven
// (the product by 1/4 is exact, so its difference with the old value is one
// multiply-add): ty, tx, source + tx, + ty, the difference, omega's product, the
// new value, six of them a chain from the row above's last value.  So one CTA
// does it all, a thread per row: a value goes to the row below by a shuffle, the
// nodes lie in shared memory, and the row warps meet at a named barrier per
// step.  A cluster of CTAs (k_sor_cluster) spent 1.6 us on a step, most of it in
// its barrier and distributed loads; this one 0.25 us (measured, 64 x 64).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "epic_internal.cuh"
#include "epic_xsum.cuh"

namespace epic {

constexpr int SRW_T = 512;                  // threads: the row warps, and all of them for a residual
constexpr int SRW_ROWS = 256;               // rows: two warps per quarter of the SM
constexpr size_t SRW_SMEM = 200 * 1024;

// PER: columns wrap too (EPIC_POISSON_PERIODIC).  phi: rows of ld >= nyi + 2
// nodes, ld - 1 odd, so that the lanes' nodes of a step (one row and one column
// apart) lie in different banks.
template <bool PER>
__global__ void __launch_bounds__(SRW_T) k_sor_rows(SolverArgs a, int ld) {
  extern __shared__ double phi[];
  __shared__ double red[40];
  __shared__ double s_edge[2 * (1 + SRW_ROWS / 32)];  // by step parity: the last value of the last row above warp w
  const int nx = a.g.nx, ny = a.g.ny;
  const int i0 = PER ? 0 : 1, nxi = nx - 1 - i0, nyi = ny - 1, ni = nxi * nyi;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row_warps = (nxi + 31) >> 5;
  const int P = PER ? max(nxi + row_warps, nyi) : nyi, D = nxi + row_warps - 1 + nyi - 1;
  double* const src = a.work[1];   // rho K, minus its mean when periodic
  double* const snap = a.work[0];  // the checked sweep
  auto node = [&](int q) { return (i0 + q / nyi) * ny + q % nyi; };
  double smean = 0.0;
  if (PER) smean = block_exact_sum(ni, [&](int q) { return a.rho[node(q)] * a.K; }, red) / (double)ni;
  for (int q = threadIdx.x; q < nx * ny; q += SRW_T) {
    src[q] = a.rho[q] * a.K - smean;
    snap[q] = 0;
  }
  const int rows = row_warps * 32;
  for (int q = threadIdx.x; q < (rows + 1) * ld; q += SRW_T) phi[q] = 0;  // cold start (src/field.cpp:78-98)
  if (threadIdx.x < 2 * (1 + SRW_ROWS / 32)) s_edge[threadIdx.x] = 0;
  __syncthreads();
  // L2 residual (src/field.cpp:121-134) of the snapshot
  auto residual = [&]() {
    const double sum = block_exact_sum(
        ni,
        [&](int q) {
          const int r = q / nyi, j = q - r * nyi, k = (i0 + r) * ny + j;
          const int kE = PER && r == nxi - 1 ? j : k + ny, kW = PER && r == 0 ? (nxi - 1) * ny + j : k - ny;
          const int kN = j == nyi - 1 ? k - j : k + 1, kS = j ? k - 1 : k + nyi - 1;
          const double p = snap[k];
          const double tx = snap[kE] - 2 * p + snap[kW], ty = snap[kN] - 2 * p + snap[kS];
          const double R = (tx + ty) + src[k];
          return R * R;
        },
        red);
    return sqrt(sum / (nx * ny));
  };
  // The row of this thread (those beyond the lattice run along in rows of
  // their own that nobody reads).  A warp runs one step later than the rows
  // above it would have it, so that its first row's W is a step old and its
  // load is off the chain.  Own node nyi is a copy of node 0, so that the last
  // node finds its N beside it.
  const int row = threadIdx.x;
  const bool real = row < nxi;
  double* const own = phi + min(row, rows) * ld;
  const double* const below = row + 1 < nxi ? own + ld : PER ? phi : phi + rows * ld;  // walls: a row of zeros
  const double* const last = phi + (nxi - 1) * ld;
  // where lane 0 finds its next W: the edge values of the step before, the old
  // last row, or the row of zeros (no branch: every lane loads)
  const bool tight = PER && P == nxi + row_warps;  // the last row's node is then one step old as well
  const double* const first = wid || tight ? s_edge + wid : PER ? last : phi + rows * ld;
  const size_t at = (size_t)(i0 + (real ? row : 0)) * ny;
  const double* const srow = src + at;
  double* const prow = snap + at;
  double v = 0, old = 0;                              // the row's last value; the next node's old one
  double nN = 0, nE = 0, nk = 0, nk2 = srow[0];       // the next node's inputs
  double edge = 0;                                    // and, in lane 0, its W
  int j = -1 - row - wid;       // node of this step (j < 0: not yet, j >= nyi: between sweeps)
  int left = a.max_iter;        // sweeps to do
  constexpr int CHECK = 25;     // residual after sweeps 0, 25, 50, ... (src/field.cpp:118)
  int to_check = real ? 0 : -1; // sweeps to the next checked one
  int iter = 0, converged = 0;
  double L2 = 0;
  const long long t_end = (long long)D + (long long)P * (a.max_iter - 1);  // steps of all sweeps
  long long t = -1;
  for (int chk = 0; a.max_iter > 0; chk += CHECK) {
    const bool check = chk < a.max_iter;
    const long long stop = check ? (long long)D + (long long)P * chk : t_end;
    if (wid < row_warps) {
      for (int n = (int)(stop - t), par = (int)t & 1; n > 0; n--, par ^= 1) {
        const double ty = nN + v;
        const double up = __shfl_up_sync(0xffffffffu, v, 1);
        const double tx = nE + (lane == 0 ? edge : up);
        const double N = nN, sk = nk;
        // the next step's inputs: old values, at rest since the last sweep
        // (node 0 of this row and, where columns wrap, the first row's: since
        // this one)
        const bool wrap = j + 1 == P;
        const int j1 = wrap ? 0 : j + 1, jc = min(max(j1, 0), nyi);
        const int j2 = j1 + 1 == P ? 0 : min(max(j1 + 1, 0), nyi);
        nN = own[jc + 1];
        nE = below[jc];
        nk = nk2;
        nk2 = srow[j2];
        edge = first[wid || tight ? par * (1 + SRW_ROWS / 32) : PER ? jc : 0];
        const double b = (sk + tx) + ty;
        const double d = fma(0.25, b, -old);
        const double vn = old + a.omega * d;
        if ((unsigned)j < (unsigned)nyi) {
          own[j] = vn;
          if (j == 0) own[nyi] = vn;
          if (to_check == 0) prow[j] = vn;
          v = vn;
          old = N;  // also across sweeps: the N of the last node is this sweep's node 0
        }
        if (lane == 31) s_edge[(par ^ 1) * (1 + SRW_ROWS / 32) + wid + 1] = v;
        if (PER && row == nxi - 1) s_edge[(par ^ 1) * (1 + SRW_ROWS / 32)] = v;
        j = j1;
        if (wrap) {
          if (--left == 0) j = -1 << 30;
          to_check = to_check == 0 ? CHECK - 1 : to_check - 1;
        }
        if (row_warps > 1) asm volatile("bar.sync 1, %0;" ::"r"(row_warps * 32) : "memory");
        else __syncwarp();
      }
    }
    t = stop;
    __syncthreads();
    if (!check) break;
    L2 = residual();
    iter = chk + 1;
    if (L2 < a.tol) {
      converged = 1;
      break;
    }
    if (chk + CHECK >= a.max_iter) {  // no further check: the remaining sweeps
      iter = a.max_iter;
    }
  }
  // phi (the duplicated nodes and walls: launch_fill_poisson_nodes), of zero
  // mean when periodic
  if (a.max_iter <= 0) iter = 0;
  auto value = [&](int q) { return converged ? snap[node(q)] : phi[(q / nyi) * ld + q % nyi]; };
  double m = 0;
  if (PER) m = block_exact_sum(ni, value, red) / (double)ni;
  for (int q = threadIdx.x; q < ni; q += SRW_T) a.phi[node(q)] = PER ? value(q) - m : value(q);
  if (threadIdx.x == 0) {
    a.info->iterations = iter;
    a.info->converged = converged;
    a.info->error = L2;
    atomicAdd(a.iter_total, (unsigned long long)iter);
  }
}

// The wrapping lattices that one CTA holds, with unit cells; false otherwise.
// (The extensions have at least 5 x 5 nodes, epic_create.)
bool launch_sor_rows(cudaStream_t st, const SolverArgs& a) {
  if (a.poisson_bc == EPIC_POISSON_DIRICHLET || a.g.dx != 1.0 || a.g.dy != 1.0) return false;
  const bool per = a.poisson_bc == EPIC_POISSON_PERIODIC;
  const int nxi = a.g.nx - (per ? 1 : 2), nyi = a.g.ny - 1;
  const int ld = (nyi + 3) & ~1;
  const size_t smem = (size_t)((nxi + 31) / 32 * 32 + 1) * ld * sizeof(double);
  if (nxi < 3 || nyi < 4 || nxi > SRW_ROWS || smem > SRW_SMEM) return false;
  static std::atomic<bool> ready{false};
  if (!ready.load()) {
    cudaFuncSetAttribute(k_sor_rows<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SRW_SMEM);
    cudaFuncSetAttribute(k_sor_rows<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SRW_SMEM);
    ready.store(true);
  }
  if (per) k_sor_rows<true><<<1, SRW_T, smem, st>>>(a, ld);
  else k_sor_rows<false><<<1, SRW_T, smem, st>>>(a, ld);
  return true;
}

}  // namespace epic
