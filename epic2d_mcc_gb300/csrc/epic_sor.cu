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
// its barrier and distributed loads; this one 0.33 to 0.36 us (measured, 64 x 64).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "epic_internal.cuh"
#include "epic_xsum.cuh"

namespace epic {

constexpr int SRW_T = 512;                  // threads: the row warps, and all of them for a residual
constexpr int SRW_ROWS = 256;               // rows: two warps per quarter of the SM
constexpr int SRW_CHECK = 25;               // residual after sweeps 0, 25, 50, ... (src/field.cpp:118)
constexpr size_t SRW_SMEM = 200 * 1024;

// Steps between the starts of two sweeps, and of one sweep from its first row's
// first node to past its last row's last.
struct SorRowsPeriod {
  int P, D;
};
__host__ __device__ inline SorRowsPeriod sor_rows_period(bool per, int nxi, int nyi) {
  const int row_warps = (nxi + 31) >> 5, chain = nxi + row_warps;
  return {per && chain > nyi ? chain : nyi, chain - 1 + nyi - 1};
}

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
  const SorRowsPeriod pd = sor_rows_period(PER, nxi, nyi);
  const int P = pd.P, D = pd.D;
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
  constexpr int CHECK = SRW_CHECK;
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
// (The extensions have at least 5 x 5 nodes, epic_create.)  There is one
// snapshot: a checked sweep must end, D steps after its start, before the first
// row is at the next one, CHECK sweeps or CHECK P steps after it.  Lattices with
// walls and about 25 times as many rows as nodes a row are beyond that.
bool launch_sor_rows(cudaStream_t st, const SolverArgs& a) {
  if (a.poisson_bc == EPIC_POISSON_DIRICHLET || a.g.dx != 1.0 || a.g.dy != 1.0) return false;
  const bool per = a.poisson_bc == EPIC_POISSON_PERIODIC;
  const int nxi = a.g.nx - (per ? 1 : 2), nyi = a.g.ny - 1;
  const int ld = (nyi + 3) & ~1;
  const size_t smem = (size_t)((nxi + 31) / 32 * 32 + 1) * ld * sizeof(double);
  if (nxi < 3 || nyi < 4 || nxi > SRW_ROWS || smem > SRW_SMEM) return false;
  const SorRowsPeriod pd = sor_rows_period(per, nxi, nyi);
  if (pd.D - 1 >= SRW_CHECK * pd.P) return false;
  const void* kern = per ? (const void*)k_sor_rows<true> : (const void*)k_sor_rows<false>;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SRW_SMEM);  // of this device
  if (per) k_sor_rows<true><<<1, SRW_T, smem, st>>>(a, ld);
  else k_sor_rows<false><<<1, SRW_T, smem, st>>>(a, ld);
  return true;
}

// ---------------------------------------------------- walls, unit cells ---
// gssolver (src/field.cpp:70-139) and gsfluidsolver (:7-68), iterate for iterate.
//
// Without wrapping, sweep s may follow sweep s-1 at a distance of two steps, so
// ~nyi/2 sweeps are in flight and a step has work for many SMs.  The sweeps are
// split over a cluster: a slot is one sweep in flight, a thread of it one row,
// which does node j of its sweep at step i + j + (the sweep's start).  A slot
// needs, at each step, the vector of values that the slot of the sweep before
// produced a fixed number of steps ago (a row's new N, and the row below's E; the
// old value is the N of the step before), its own row above's last value (W) and
// its own last value (S): so the slots form a ring through which vectors flow in
// one direction only.  Within a CTA a vector is two steps old (shared memory,
// one barrier per step); to the next CTA it goes by remote stores into that CTA's
// ring of messages and is three steps old, which hides the way (~300 cycles)
// behind a step.  A word of a message that has not come yet holds a NaN that no
// operation gives (SST_NONE), so the readers poll the words that they need, and
// set them back after the step; the sender may use them again once the reader
// has counted the step as done (credit, every SST_LOOK steps; released by the
// reader and acquired by the sender, with fences on shared memory alone: whole
// ones would wait for the snapshots' stores too and took 4 % of a conductor
// deck's solve).  No phi lies in memory at all while the sweeps
// run.  (Splitting rows
// over the cluster, k_sor_cluster, needs values from both neighbours every step,
// and spent 2 us on it, most of it in the cluster barrier.)
//
// The sweeps that the reference checks (0, CHECK, 2 CHECK, ...) also store their
// values into one of SST_SNAPS snapshots; the last CTA of the cluster does nothing
// but take their residuals, while the sweeps go on, and stops them once one
// converged: its snapshot is the result.  A checked sweep starts only when the
// residual of the one that used its snapshot before is taken.
constexpr int SST_T = 512;       // threads: the slots' warps, at least SST_CHECK_T of them for the residuals
constexpr int SST_CHECK_T = 256;
constexpr int SST_CTAS = 16;
constexpr int SST_LOOK = 8;      // steps between looks at the stop word and at the next CTA's progress
constexpr int SST_SLACK = 3 * SST_LOOK;  // messages a CTA may be ahead of the next one's reads
constexpr int SST_SNAPS = 7;     // snapshots: work[1..7]
constexpr size_t SST_SMEM = 200 * 1024;
constexpr long long SST_NONE = (long long)0xFFF8A5C31E7D2B49ull;

struct SorStream {
  int C;            // CTAs with slots; one more takes the residuals
  int slots;        // per CTA
  int Wr;           // warps per slot
  int T;            // steps between the starts of a slot's sweeps
  int ring, extra;  // steps between the last slot of a CTA and the first of the next: ring, + 1 for the first `extra` CTAs
  int depth;        // messages in a CTA's ring
  int ld;           // doubles per vector: a wall, the rows, a wall
  int lds;          // doubles per row of the sources in shared memory (even: no bank conflicts)
  int terms;        // residual terms kept in shared memory
  int smem;
};
__host__ __device__ inline int sst_cross(const SorStream& t, int c) { return t.ring + (c < t.extra ? 1 : 0); }

__device__ __forceinline__ unsigned sst_smem(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned sst_map(const void* p, int rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(sst_smem(p)), "r"(rank));
  return r;
}
__device__ __forceinline__ void sst_put(unsigned addr, int v) {
  asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ int sst_get(const int* p) {
  int v;
  asm volatile("ld.volatile.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(sst_smem(p)) : "memory");
  return v;
}
// Of the word that lets the sweeps write a snapshot that has been read.
__device__ __forceinline__ void sst_put_release(unsigned addr, int v) {
  asm volatile("st.release.cluster.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ int sst_get_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.cluster.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(sst_smem(p)) : "memory");
  return v;
}
__device__ __forceinline__ double sst_ld(unsigned addr) {
  double v;
  asm volatile("ld.volatile.shared::cta.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void sst_st(unsigned addr, double v) {
  asm volatile("st.volatile.shared::cta.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}

template <bool FLUID>
__global__ void __launch_bounds__(SST_T) k_sor_stream(SolverArgs a, SorStream t) {
  extern __shared__ double sm[];
  __shared__ double red[40];
  __shared__ int s_cmd;      // 0 run, 1 stop, 2 gave up (written by the checking CTA or a wait that gave up)
  __shared__ int s_checked;  // residuals taken
  __shared__ int s_credit;   // steps that the next CTA has completed
  __shared__ int s_stop[2];  // what thread 0 saw of s_cmd, by looks
  __shared__ int s_ready[SST_SNAPS];  // checking CTA: 1 + the check whose snapshot is complete
  __shared__ int s_out[2];            // every CTA, at the end: converged, the check
  const int me = (int)blockIdx.x, C = t.C;
  const int nx = a.g.nx, ny = a.g.ny, nxi = nx - 2, nyi = ny - 2, nn = nx * ny;
  constexpr int CHECK = FLUID ? 50 : 25;  // src/field.cpp:118 and :52
  const long long spin = spin_or_default(a.spin);
  double* const msg = sm;                                               // [depth][ld]
  double* const vec = msg + t.depth * t.ld;                             // [slots][2][ld]
  double* const rK = a.work[0];
  const int nt = blockDim.x;
  for (int q = me * nt + threadIdx.x; q < nn; q += (C + 1) * nt) {
    if (!FLUID) rK[q] = a.rho[q] * a.K;
    a.phi[q] = 0;  // cold start, zero edges (src/field.cpp:78-98)
    for (int k = 1; k <= SST_SNAPS; k++) a.work[k][q] = 0;
  }
  if (me < C) {
    double* const k = vec + 2 * t.slots * t.ld;
    for (int q = threadIdx.x; q < nxi * nyi; q += nt) {
      const int i = q / nyi, j = q - i * nyi;
      const double r = a.rho[(i + 1) * ny + j + 1];
      k[i * t.lds + j] = FLUID ? r : r * a.K;
    }
    for (int q = threadIdx.x; q < (t.depth + 2 * t.slots) * t.ld; q += nt) {
      const int m = q % t.ld;  // the rows' words of the messages are not there yet
      sm[q] = q < t.depth * t.ld && m >= 1 && m <= nxi ? __longlong_as_double(SST_NONE) : 0.0;
    }
  }
  if (threadIdx.x == 0) s_cmd = s_checked = s_credit = s_stop[0] = s_stop[1] = s_out[0] = s_out[1] = 0;
  if (threadIdx.x < SST_SNAPS) s_ready[threadIdx.x] = 0;
  cooperative_groups::this_cluster().sync();

  int iter = 0;
  double L2 = 0;
  if (me == C) {
    // ---- residuals ----
    bool conv = false;
    for (int k = 0; (long long)k * CHECK < a.max_iter; k++) {
      if (threadIdx.x == 0) {
        long long n = 0;
        while (sst_get(&s_ready[k % SST_SNAPS]) != k + 1 && sst_get(&s_cmd) == 0)
          if (++n >= spin) s_cmd = 2;
        asm volatile("fence.acq_rel.cluster;" ::: "memory");
      }
      __syncthreads();
      if (sst_get(&s_cmd)) break;
      const double* const p = a.work[1 + k % SST_SNAPS];
      auto term = [&](int q) {
        const int i = 1 + q / nyi, m = i * ny + 1 + (q - (i - 1) * nyi);
        const double c = __ldcg(p + m);
        const double tx = __ldcg(p + m + ny) - 2 * c + __ldcg(p + m - ny);
        const double ty = __ldcg(p + m + 1) - 2 * c + __ldcg(p + m - 1);
        const double R = (tx + ty) + (FLUID ? (a.rho[m] - exp(c)) * a.K : __ldcg(rK + m));
        return R * R;
      };
      double sum;
      if (t.terms) {
        for (int q = threadIdx.x; q < nxi * nyi; q += nt) sm[q] = term(q);
        __syncthreads();
        sum = block_exact_sum(nxi * nyi, [&](int q) { return sm[q]; }, red);
      } else {
        sum = block_exact_sum(nxi * nyi, term, red);
      }
      L2 = sqrt(sum / (nx * ny));
      iter = k * CHECK + 1;
      conv = L2 < a.tol;
      if ((int)threadIdx.x < C) {
        if (conv) {
          sst_put(sst_map(&s_out[1], threadIdx.x), k);
          sst_put(sst_map(&s_out[0], threadIdx.x), 1);
          sst_put(sst_map(&s_cmd, threadIdx.x), 1);
        } else {
          sst_put_release(sst_map(&s_checked, threadIdx.x), k + 1);
        }
      }
      if (threadIdx.x == 0 && conv) {
        s_out[0] = 1;
        s_out[1] = k;
      }
      if (conv) break;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      if (sst_get(&s_cmd) == 2) atomicOr(a.flags, FLAG_TIMEOUT);
      if (!conv) iter = a.max_iter;
      a.info->iterations = iter;
      a.info->converged = conv;
      a.info->error = L2;
      atomicAdd(a.iter_total, (unsigned long long)iter);
    }
  } else if ((int)threadIdx.x < 32 * t.Wr * t.slots && a.max_iter > 0) {
    // ---- sweeps ----
    const int wid = threadIdx.x >> 5, slot = wid / t.Wr, i = (wid - slot * t.Wr) * 32 + (threadIdx.x & 31);
    const int team = 32 * t.Wr * t.slots, G = C * t.slots;
    const bool real = i < nxi, feeds = slot == t.slots - 1, fed = slot == 0;
    const int P = sst_cross(t, me), Pn = sst_cross(t, (me + 1) % C);
    int off = 2 * slot;
    for (int c = 1; c <= me; c++) off += 2 * (t.slots - 1) + sst_cross(t, c);
    // steps to the last sweep's last row and past it to its next start
    const int steps = t.T * ((a.max_iter - 1) / G + 2) + nxi;
    const size_t at = (size_t)(1 + (real ? i : 0)) * ny + 1;
    const unsigned ld_bytes = t.ld * 8, msg_bytes = t.depth * ld_bytes;
    unsigned next_msg = sst_map(msg, (me + 1) % C) + (i + 1) * 8;  // where the next value goes in the next CTA's messages
    const unsigned next_end = sst_map(msg, (me + 1) % C) + msg_bytes;
    const unsigned prev_credit = sst_map(&s_credit, (me + C - 1) % C);
    // shared addresses: this row's place in its slot's vector of this step (its
    // W lies before it in the last step's); its N (and E) in the last step's
    // vector of the slot before, or in the message; its source of node 0
    unsigned out = sst_smem(vec + slot * 2 * t.ld + i + 1);
    unsigned in = fed ? sst_smem(msg) + (i + 1) * 8 : sst_smem(vec + (slot - 1) * 2 * t.ld + i + 1) + ld_bytes;
    const unsigned msg_end = sst_smem(msg) + msg_bytes;
    int flip = (int)ld_bytes;  // to the other of the two vectors
    const int shift = real ? i : 0;
    const unsigned source = sst_smem(vec + 2 * t.slots * t.ld) + shift * t.lds * 8;
    // All rows of a slot share its place tau in [0, T): row i <= tau is at node
    // tau - i of sweep s, row i > tau (i < T) still at node tau - i + T of the
    // slot's sweep before; nodes from nyi on are the pause between sweeps.  What
    // depends on the sweep (whether there is one, where its values go) is the
    // same for all rows; a row takes it over at its node 0.
    int tau = t.T - 1 - off, s = me * t.slots + slot - G;
    int pos = tau - shift < 0 ? tau - shift + t.T : tau - shift;
    bool on_cur = false, on = false;
    double *dst_cur = nullptr, *dst_prev = nullptr, *dst = nullptr;
    // where a sweep's last row is stored and a barrier passed
    const int tau_done = (nxi - 1 + nyi) % t.T;
    const bool done_prev = nxi - 1 + nyi >= t.T;
    // A row's value is 0 while it pauses, which gives the nodes at the ends
    // their walls (S of node 0, and N of the last node from the slot before,
    // which is one node past it there).
    double v = 0, old = 0, sk = 0, k1 = sst_ld(source + min(pos + 1 == t.T ? 0 : pos + 1, nyi - 1) * 8);
    const int sends = feeds && real, clears = fed && real;
    // m steps without an event.  A step's length is what counts (7 FP64
    // instructions, six of them dependent, take 450 cycles of it), and a taken
    // branch costs as much as several instructions: everything rare happens
    // between these runs, and what only some warps do is predicated.
    auto run = [&](auto store, int m, bool take) {
#pragma unroll 1
      for (; m > 0; m--) {
        double N = sst_ld(in), E = sst_ld(in + 8);
        const double W = sst_ld(out + flip - 8);
        if (fed) {
          const bool none = __double_as_longlong(N) == SST_NONE || __double_as_longlong(E) == SST_NONE;
          if (take) {
            if (__builtin_expect(__any_sync(0xffffffffu, real && none), 0)) {  // not there yet
              long long tries = 0;
              do {
                if (sst_get(&s_cmd)) break;
                if (++tries >= spin) s_cmd = 2;
                N = sst_ld(in);
                E = sst_ld(in + 8);
              } while (__any_sync(0xffffffffu, real && (__double_as_longlong(N) == SST_NONE ||
                                                         __double_as_longlong(E) == SST_NONE)));
            }
          } else {
            N = E = 0;
          }
        }
        const double ty = N + v;
        const double tx = E + W;
        const double b = (sk + tx) + ty;
        on = real && (pos == 0 ? on_cur : on);
        if (store()) dst = pos == 0 ? dst_cur : dst;
        const double d = fma(0.25, b, -old);
        const double vn = old + a.omega * d;
        const bool active = on && pos < nyi;
        v = active ? vn : 0.0;
        sst_st(out, v);
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %2, 0;\n\t"
                     "@p st.relaxed.cluster.shared::cluster.f64 [%0], %1;\n\t}" ::"r"(next_msg),
                     "d"(v), "r"(sends)
                     : "memory");
        next_msg = next_msg + ld_bytes >= next_end ? next_msg + ld_bytes - msg_bytes : next_msg + ld_bytes;
        if (store() && active && dst) dst[at + pos] = v;
        old = N;
        if (FLUID) sk = (k1 - exp(N)) * a.K;
        else sk = k1;
        pos = pos + 1 == t.T ? 0 : pos + 1;
        k1 = sst_ld(source + min(pos + 1 == t.T ? 0 : pos + 1, nyi - 1) * 8);
        asm volatile("bar.sync 1, %0;" ::"r"(team) : "memory");
        if (fed) {
          if (take) {
            asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %2, 0;\n\t"
                         "@p st.volatile.shared::cta.f64 [%0], %1;\n\t}" ::"r"(in),
                         "d"(__longlong_as_double(SST_NONE)), "r"(clears)
                         : "memory");  // read by both its rows
            in = in + ld_bytes >= msg_end ? in + ld_bytes - msg_bytes : in + ld_bytes;
          }
        } else {
          in -= flip;
        }
        out += flip;
        flip = -flip;
      }
    };
    for (int n = 0, look = 0; n < steps; look ^= 1) {
      if (feeds) {  // room for the messages of these steps
        long long tries = 0;
        while (sst_get(&s_credit) < n + SST_LOOK - 1 - t.depth + Pn && sst_get(&s_cmd) == 0)
          if (++tries >= spin) s_cmd = 2;
        asm volatile("fence.acquire.sync_restrict::shared::cluster.cluster;" ::: "memory");
      }
      if (threadIdx.x == 0) s_stop[look] = sst_get(&s_cmd);
      for (int left = SST_LOOK; left > 0;) {
        if (tau == t.T) {  // the slot's next sweep
          tau = 0;
          s += G;
          dst_prev = dst_cur;
          on_cur = s < a.max_iter;
          dst_cur = nullptr;
          if (on_cur && s % CHECK == 0) {
            const int k = s / CHECK;
            if (k >= SST_SNAPS) {  // its snapshot must be free; once the sweeps are stopped it is not touched
              long long tries = 0;
              while (sst_get(&s_checked) <= k - SST_SNAPS && sst_get(&s_cmd) == 0)
                if (++tries >= spin) s_cmd = 2;
              __syncwarp();
              on_cur = sst_get_acquire(&s_checked) > k - SST_SNAPS;
            }
            dst_cur = a.work[1 + k % SST_SNAPS];
          } else if (s == a.max_iter - 1) {
            dst_cur = a.phi;
          }
        }
        if (tau == tau_done) {
          const int sd = done_prev ? s - G : s;
          if (i == 0 && (done_prev ? dst_prev : dst_cur) && sd % CHECK == 0) {
            asm volatile("fence.acq_rel.cluster;" ::: "memory");
            sst_put(sst_map(&s_ready[(sd / CHECK) % SST_SNAPS], C), sd / CHECK + 1);
          }
        }
        const bool take = !fed || n + 1 >= P;
        int m = min(left, (tau < tau_done ? tau_done : t.T) - tau);
        if (!take) m = min(m, P - 1 - n);
        if (dst_cur || dst_prev) run([] { return true; }, m, take);
        else run([] { return false; }, m, take);
        tau += m;
        left -= m;
        n += m;
      }
      if (s_stop[look]) break;
      // all but the last step's words are set back, and before a barrier
      if (threadIdx.x == 0) {
        asm volatile("fence.release.sync_restrict::shared::cta.cluster;" ::: "memory");
        sst_put(prev_credit, n - 1);
      }
    }
    if (sst_get(&s_cmd) == 2 && threadIdx.x == 0) atomicOr(a.flags, FLAG_TIMEOUT);
  }
  cooperative_groups::this_cluster().sync();
  // the converged sweep, or the last one where it was a checked one
  if (s_out[0] || (a.max_iter > 0 && (a.max_iter - 1) % CHECK == 0)) {
    const double* const p = a.work[1 + (s_out[0] ? s_out[1] : (a.max_iter - 1) / CHECK) % SST_SNAPS];
    for (int q = me * nt + threadIdx.x; q < nn; q += (C + 1) * nt) a.phi[q] = __ldcg(p + q);
  }
}

static bool sst_plan(const SolverArgs& a, SorStream* out) {
  SorStream t;
  const int nxi = a.g.nx - 2, nyi = a.g.ny - 2;
  if (nxi < 1 || nyi < 1) return false;
  t.Wr = (nxi + 31) / 32;
  if (32 * t.Wr > SST_T) return false;
  // one warp per quarter of the SM: more would only lengthen the steps
  t.slots = std::max(1, 4 / t.Wr);
  const int adv = 2 * (t.slots - 1) + 3;  // steps from a CTA's first slot to the next one's
  t.C = std::min(SST_CTAS - 1, std::max(1, (std::max(nyi + 1, nxi) + adv - 1) / adv));
  t.T = std::max(t.C * adv, std::max(nyi + 1, nxi));
  const int spare = t.T - t.C * adv;
  t.ring = 3 + spare / t.C;
  t.extra = spare % t.C;
  t.depth = t.ring + 1 + SST_SLACK;
  t.ld = 32 * t.Wr + 2;
  const size_t work = (size_t)(t.depth + 2 * t.slots) * t.ld * 8;
  const size_t terms = (size_t)nxi * nyi * 8;
  t.terms = terms <= SST_SMEM;
  t.lds = (nyi + 1) & ~1;
  const size_t sources = (size_t)nxi * t.lds * 8;
  t.smem = (int)std::max(work + sources, t.terms ? terms : 0);
  if (work + sources > SST_SMEM) return false;
  // steps are counted in 32 bits
  if ((long long)t.T * ((long long)a.max_iter / (t.C * t.slots) + 3) + nxi > (1ll << 29)) return false;
  *out = t;
  return true;
}

// gssolver's (fluid: gsfluidsolver's) lattice with walls and unit cells; false
// where it does not suit (then k_sor_cluster or k_sor_lex).
bool launch_sor_stream(cudaStream_t st, const SolverArgs& a_in, bool fluid) {
  SorStream t;
  if (a_in.poisson_bc != EPIC_POISSON_DIRICHLET || a_in.g.dx != 1.0 || a_in.g.dy != 1.0 || !sst_plan(a_in, &t))
    return false;
  SolverArgs a = a_in;
  a.spin = spin_limit();
  const void* kern = fluid ? (const void*)k_sor_stream<true> : (const void*)k_sor_stream<false>;
  if (!cluster_fits(kern, t.C + 1, SST_T, SST_SMEM, SST_SMEM)) return false;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = t.C + 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(t.C + 1);
  cfg.blockDim = dim3(std::max(SST_CHECK_T, 32 * t.Wr * t.slots));
  cfg.dynamicSmemBytes = t.smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return launched(fluid ? cudaLaunchKernelEx(&cfg, k_sor_stream<true>, a, t)
                        : cudaLaunchKernelEx(&cfg, k_sor_stream<false>, a, t));
}

}  // namespace epic
