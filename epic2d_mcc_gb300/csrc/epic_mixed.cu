// Particle kernels of the mixed-precision form.
//
// Record: cell (int32 node index i*ny + j of the cell's lower-left node),
// ox, oy (FP32 offsets inside the cell, [0, 1)), vx, vy, vz (FP32) — 24 bytes.
// The push reads and writes 20 of them (40 B per particle-step); the deposit
// reads 12; everything runs on the FP32 and integer pipes.  Offsets keep a
// uniform 2^-24-cell resolution over the whole domain, where FP32 absolute
// positions would lose precision with distance from the origin.
//
// Compiled with contraction (FMA) enabled: this form is checked against the
// FP64 oracle within stated tolerances, not bit for bit.
#include <cuda_runtime.h>

#include <algorithm>

#include "epic_device.cuh"
#include "epic_internal.cuh"
#include "epic_mixed.cuh"
#include "epic_xsum.cuh"

namespace epic {

// ------------------------------------------------------------ layout ---
// Upload: FP64 records {x, y, vx, vy, vz} -> mixed.  Species::AddParticle's
// positions become (cell, offset); a particle outside the grid raises
// FLAG_OUT_OF_GRID (the reference would throw at its first deposit).
__global__ void k_aos_to_mixed(Geom g, const double* __restrict__ aos, MixedSoA p, long long n, int* flags) {
  bool bad = false;
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
    const double* r = aos + 5 * q;
    int i, j;
    float ox, oy;
    const bool in_x = cell_offset((r[0] - g.x0) / g.dx, g.nx - 1, i, ox);
    const bool in_y = cell_offset((r[1] - g.y0) / g.dy, g.ny - 1, j, oy);
    bad |= !(in_x && in_y);
    p.cell[q] = i * g.ny + j;
    p.ox[q] = ox;
    p.oy[q] = oy;
    p.vx[q] = (float)r[2];
    p.vy[q] = (float)r[3];
    p.vz[q] = (float)r[4];
  }
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) set_flag(flags, FLAG_OUT_OF_GRID);
}

__global__ void k_mixed_to_aos(Geom g, double* __restrict__ aos, MixedSoA p, const long long* __restrict__ d_n) {
  const long long n = *d_n;
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
    const int c = p.cell[q];
    const int i = c / g.ny, j = c - i * g.ny;
    double* r = aos + 5 * q;
    // explicit roundings (no contraction): the batch's extraction computes the same
    r[0] = __dadd_rn(g.x0, __dmul_rn(__dadd_rn((double)i, (double)p.ox[q]), g.dx));
    r[1] = __dadd_rn(g.y0, __dmul_rn(__dadd_rn((double)j, (double)p.oy[q]), g.dy));
    r[2] = p.vx[q];
    r[3] = p.vy[q];
    r[4] = p.vz[q];
  }
}

void launch_aos_to_mixed(cudaStream_t st, const Geom& g, const double* aos, const MixedSoA& p, long long n,
                         int* flags, int grid) {
  k_aos_to_mixed<<<grid, PART_THREADS, 0, st>>>(g, aos, p, n, flags);
}

void launch_mixed_to_aos(cudaStream_t st, const Geom& g, double* aos, const MixedSoA& p, const long long* d_n,
                         int grid) {
  k_mixed_to_aos<<<grid, PART_THREADS, 0, st>>>(g, aos, p, d_n);
}

// ----------------------------------------------------------- deposit ---
// CIC / NGP deposit with integer weights (Domain::Scatter, src/domain.cpp:
// 205-228): the offsets are quantised to 2^-20 of a cell and the four CIC
// weights are exact integer products summing to 2^40, accumulated in int64
// (deterministic: integer addition is associative).  No node can overflow
// unless more than 2^23 particles share its four cells.  The finalisation
// multiplies by spwt * 2^-40.
template <int SHAPE>
__global__ void __launch_bounds__(PART_THREADS) k_deposit_mixed(Geom g, MixedSoA p, const long long* __restrict__ d_n,
                                                                unsigned long long* __restrict__ acc) {
  const long long n = *d_n;
  const long long S = 1ll << MIXED_OFFSET_BITS;
  const float fS = (float)S;
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
    const int c = __ldg(&p.cell[q]);
    const float ox = __ldg(&p.ox[q]), oy = __ldg(&p.oy[q]);
    if (SHAPE == EPIC_NGP) {
      // round(lx) with lx = i + ox >= 0: i + (ox >= 0.5)
      const int k = c + (ox >= 0.5f ? g.ny : 0) + (oy >= 0.5f ? 1 : 0);
      atomicAdd(&acc[k], (unsigned long long)(S * S));
    } else {
      const long long a = (long long)(ox * fS), b = (long long)(oy * fS);  // truncation, in [0, 2^20)
      atomicAdd(&acc[c], (unsigned long long)((S - a) * (S - b)));
      atomicAdd(&acc[c + g.ny], (unsigned long long)(a * (S - b)));
      atomicAdd(&acc[c + 1], (unsigned long long)((S - a) * b));
      atomicAdd(&acc[c + g.ny + 1], (unsigned long long)(a * b));
    }
  }
}

void launch_deposit_mixed(cudaStream_t st, const Geom& g, int shape, const MixedSoA& p, const long long* d_n,
                          unsigned long long* acc, int* flags, int grid) {
  (void)flags;
  if (shape == EPIC_NGP) k_deposit_mixed<EPIC_NGP><<<grid, PART_THREADS, 0, st>>>(g, p, d_n, acc);
  else k_deposit_mixed<EPIC_CIC><<<grid, PART_THREADS, 0, st>>>(g, p, d_n, acc);
}

// CIC deposit of the particles [*d_from, *d_n) (the MCC's ionisation
// products, appended after the push deposited the rest).
__global__ void __launch_bounds__(PART_THREADS) k_deposit_mixed_range(Geom g, MixedSoA p,
                                                                      const long long* __restrict__ d_from,
                                                                      const long long* __restrict__ d_n,
                                                                      unsigned long long* __restrict__ acc) {
  const long long from = *d_from, n = *d_n;
  const long long S = 1ll << MIXED_OFFSET_BITS;
  const float fS = (float)S;
  for (long long q = from + (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n;
       q += (long long)gridDim.x * blockDim.x) {
    const int c = p.cell[q];
    const long long a = (long long)(p.ox[q] * fS), b = (long long)(p.oy[q] * fS);
    atomicAdd(&acc[c], (unsigned long long)((S - a) * (S - b)));
    atomicAdd(&acc[c + g.ny], (unsigned long long)(a * (S - b)));
    atomicAdd(&acc[c + 1], (unsigned long long)((S - a) * b));
    atomicAdd(&acc[c + g.ny + 1], (unsigned long long)(a * b));
  }
}

void launch_deposit_mixed_range(cudaStream_t st, const Geom& g, const MixedSoA& p, const long long* d_from,
                                const long long* d_n, unsigned long long* acc, int grid) {
  k_deposit_mixed_range<<<grid, PART_THREADS, 0, st>>>(g, p, d_from, d_n, acc);
}

// CIC deposit of particles in no particular order (a state that never sorts).
//
// Sent straight to the grid, such particles are four 64-bit atomics each at
// random addresses, and the L2's atomic units bound the pass; on small grids
// equal addresses queue up as well.  Here a CTA owns a band of rows, holds its
// node words in shared memory, goes through its slice of all particles, keeps
// those of its band, and adds the words to the grid once at the end.  Bands
// are as few as 204 KB a CTA allow: each particle is looked at once per band,
// and only reading it (12 bytes, from L2 after the first band) is repeated;
// those of the band are queued so that whole warps deposit (without, the
// atomics of three bands ran a third full: push and deposit of the 256 x 256
// beam 275 us a step, 260 with).
//
// A word is two 32-bit halves, the low one added with the old value returned,
// which tells the carry: shared memory has no 64-bit add, and its emulation as
// a compare-and-swap loop took 2 to 3.5 times as long (8M particles on 64 x 64
// cells, push and deposit: 205 us with it, 142 so, 582 by atomics on the grid;
// 8 x 8: 436, 123, 1370; 256 x 256, three bands: 279, 222, 311).  What bounds
// it are the eight shared-memory atomics of a particle.  Integer sums: the
// order does not matter, and the result equals the other deposits'.
constexpr int DT_THREADS = 1024;
constexpr int DT_PER_THREAD = 8;  // consecutive particles a thread, loaded as vectors
constexpr int DT_CHUNK = DT_THREADS * DT_PER_THREAD;
constexpr int DT_QUEUE = 64;  // records a warp
constexpr int DT_QUEUES = DT_THREADS / 32 * DT_QUEUE * 8;  // 16 KB
constexpr int DT_MAX_SMEM = 204 * 1024;  // of words

__device__ __forceinline__ void dt_add(unsigned* lo, unsigned* hi, int k, unsigned long long w) {
  const unsigned l = (unsigned)w, old = atomicAdd(lo + k, l);
  atomicAdd(hi + k, (unsigned)(w >> 32) + (old + l < l));
}

// Band b: cell rows [b rows, (b + 1) rows), node rows one more.
// QUEUE (several bands): a warp's particles of its band wait in a queue of its
// own until 32 are there, as one 64-bit record each.
template <bool QUEUE>
__global__ void __launch_bounds__(DT_THREADS, 1) k_deposit_mixed_bands(Geom g, MixedSoA p,
                                                                       const long long* __restrict__ d_n,
                                                                       unsigned long long* __restrict__ acc, int bands,
                                                                       int rows) {
  extern __shared__ unsigned dt_words[];
  constexpr int P = DT_PER_THREAD;
  constexpr unsigned S = 1u << MIXED_OFFSET_BITS;
  const float fS = (float)S;
  const long long n = *d_n;
  const int band = blockIdx.x % bands, slice = blockIdx.x / bands, slices = gridDim.x / bands;
  const int r0 = band * rows, nr = min(rows, g.nx - 1 - r0);
  const int c0 = r0 * g.ny, span = nr * g.ny, words = span + g.ny;
  if ((long long)slice * DT_CHUNK >= n) return;
  unsigned* const lo = dt_words;
  unsigned* const hi = dt_words + words;
  for (int k = threadIdx.x; k < 2 * words; k += DT_THREADS) dt_words[k] = 0;
  const int lane = threadIdx.x & 31;
  // past the words of a whole band, 8-byte aligned
  unsigned long long* const queue =
      reinterpret_cast<unsigned long long*>(dt_words + 2 * (rows + 1) * g.ny) + (threadIdx.x >> 5) * DT_QUEUE;
  int waiting = 0;
  auto deposit = [&](int m, unsigned a, unsigned b) {
    dt_add(lo, hi, m, (unsigned long long)(S - a) * (S - b));
    dt_add(lo, hi, m + g.ny, (unsigned long long)a * (S - b));
    dt_add(lo, hi, m + 1, (unsigned long long)(S - a) * b);
    dt_add(lo, hi, m + g.ny + 1, (unsigned long long)a * b);
  };
  __syncthreads();
  for (long long chunk = (long long)slice * DT_CHUNK; chunk < n; chunk += (long long)slices * DT_CHUNK) {
    const long long q0 = chunk + (long long)threadIdx.x * P;
    int c[P];
    float ox[P], oy[P];
    if (q0 + P <= n) {
#pragma unroll
      for (int h = 0; h < P / 4; h++) {
        const int4 cc = __ldg(reinterpret_cast<const int4*>(p.cell + q0) + h);
        const float4 xx = __ldg(reinterpret_cast<const float4*>(p.ox + q0) + h);
        const float4 yy = __ldg(reinterpret_cast<const float4*>(p.oy + q0) + h);
        c[4 * h] = cc.x; c[4 * h + 1] = cc.y; c[4 * h + 2] = cc.z; c[4 * h + 3] = cc.w;
        ox[4 * h] = xx.x; ox[4 * h + 1] = xx.y; ox[4 * h + 2] = xx.z; ox[4 * h + 3] = xx.w;
        oy[4 * h] = yy.x; oy[4 * h + 1] = yy.y; oy[4 * h + 2] = yy.z; oy[4 * h + 3] = yy.w;
      }
    } else {
#pragma unroll
      for (int k = 0; k < P; k++) {
        const long long q = q0 + k;
        c[k] = q < n ? __ldg(&p.cell[q]) : -1;
        ox[k] = q < n ? __ldg(&p.ox[q]) : 0.f;
        oy[k] = q < n ? __ldg(&p.oy[q]) : 0.f;
      }
    }
#pragma unroll
    for (int k = 0; k < P; k++) {
      const int m = c[k] - c0;
      const bool in = (unsigned)m < (unsigned)span;
      const unsigned a = (unsigned)(int)(ox[k] * fS), b = (unsigned)(int)(oy[k] * fS);
      if (!QUEUE) {
        if (in) deposit(m, a, b);
        continue;
      }
      const unsigned mask = __ballot_sync(0xffffffffu, in);
      if (in)
        queue[waiting + __popc(mask & ((1u << lane) - 1))] =
            (unsigned long long)m << 40 | (unsigned long long)a << 20 | b;
      waiting += __popc(mask);
      if (waiting >= 32) {
        __syncwarp();
        waiting -= 32;
        const unsigned long long v = queue[waiting + lane];
        __syncwarp();
        deposit((int)(v >> 40), (unsigned)(v >> 20) & (S - 1), (unsigned)v & (S - 1));
      }
    }
  }
  if (QUEUE) {
    __syncwarp();
    if (lane < waiting) {
      const unsigned long long v = queue[lane];
      deposit((int)(v >> 40), (unsigned)(v >> 20) & (S - 1), (unsigned)v & (S - 1));
    }
  }
  __syncthreads();
  for (int k = threadIdx.x; k < words; k += DT_THREADS) {
    const unsigned long long w = (unsigned long long)hi[k] << 32 | lo[k];
    if (w) atomicAdd(acc + c0 + k, w);
  }
}

// Bands of so many cell rows each that their words, with one row of nodes more,
// fit a CTA; none is empty.
struct DepositBands {
  int rows, bands;
};
static DepositBands deposit_bands(const Geom& g) {
  const int most = DT_MAX_SMEM / 8 / g.ny - 1;  // cell rows that fit
  const int want = (g.nx - 1 + most - 1) / most, rows = (g.nx - 1 + want - 1) / want;
  return {rows, (g.nx - 1 + rows - 1) / rows};
}

// Grids of up to eight bands (450 x 450 nodes) whose rows are short enough that a
// band has several.  Measured over whole steps: 400 x 400 cells (seven bands) 1.06
// to 1.1 times as fast as the fused push and deposit, 256 x 256 1.2, 128 x 128 2;
// with few particles (4 a cell) level.
bool deposit_bands_fit(const Geom& g) { return g.ny <= DT_MAX_SMEM / 8 / 8 && deposit_bands(g).bands <= 8; }

void launch_deposit_mixed_bands(cudaStream_t st, const Geom& g, const MixedSoA& p, const long long* d_n,
                                unsigned long long* acc) {
  const DepositBands b = deposit_bands(g);
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int smem = (b.rows + 1) * g.ny * 8 + (b.bands > 1 ? DT_QUEUES : 0);
  const auto kern = b.bands > 1 ? k_deposit_mixed_bands<true> : k_deposit_mixed_bands<false>;
  // the same value whatever the grid: other threads may be launching it too
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, DT_MAX_SMEM + DT_QUEUES);
  kern<<<b.bands * std::max(1, sms / b.bands), DT_THREADS, smem, st>>>(g, p, d_n, acc, b.bands, b.rows);
}

// -------------------------------------------------------------- push ---
// gather32 / advance / push_mixed_one: epic_mixed.cuh (shared with the batch).
template <int SHAPE, int BC>
__global__ void __launch_bounds__(PART_THREADS) k_push_mixed(Geom g, MixedSoA p, const long long* __restrict__ d_n,
                                                             const FieldCell* __restrict__ ef, float qmK_dt, float cx,
                                                             float cy) {
  const long long n = *d_n;
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
    int c = p.cell[q];
    float ox = p.ox[q], oy = p.oy[q], vx = p.vx[q], vy = p.vy[q];
    push_mixed_one<SHAPE, BC>(g, ef, qmK_dt, cx, cy, c, ox, oy, vx, vy);
    p.cell[q] = c;
    p.ox[q] = ox;
    p.oy[q] = oy;
    p.vx[q] = vx;
    p.vy[q] = vy;
  }
}

// Periodic or reflective walls, CIC: the push, the deposit of the new
// positions into acc (deposit_warp_sorted) and, with SEL, the MCC's first
// pass over the pushed electrons (mcc_candidate on the new velocities,
// warp-aggregated appends to sel.cand) in one pass over the particles.  Each
// thread takes DEP_PER_THREAD particles with vector loads and stores, in groups
// of four consecutive ones 128 apart, so that a warp's accesses cover whole lines
// (eight consecutive ones left half of every sector to a second access: 1.95 ms
// for 2.1e8 sorted particles, 1.73 so; 1.26 ms is the memory's rate).  What
// bounds it is latency at 24 warps an SM: more warps spill, and fetching the next
// chunk early gained nothing.  Without DEP the deposit is left out (k_deposit_mixed_bands follows).
// The particles, the integer sums and the candidate set (in another
// order, which the MCC does not depend on) equal those of k_push_mixed +
// k_deposit_mixed_sorted + k_mcc_select.
template <int BC, bool SEL, bool DEP>
__global__ void __launch_bounds__(PART_THREADS, 3) k_push_mixed_dep(Geom g, MixedSoA p, const long long* __restrict__ d_n,
                                                                 const FieldCell* __restrict__ ef, float qmK_dt,
                                                                 float cx, float cy, unsigned long long* __restrict__ acc,
                                                                 SelectArgs sel) {
  constexpr int P = DEP_PER_THREAD;
  __shared__ DepWarp tables[DEP ? PART_THREADS / 32 : 1];
  DepWarp& w = tables[DEP ? threadIdx.x >> 5 : 0];
  const long long n = *d_n;
  const unsigned long long step = SEL ? *sel.d_step : 0ull;
  const int lane = threadIdx.x & 31;
  if (DEP) dep_init(w);
  for (long long chunk = (long long)blockIdx.x * DEP_CHUNK; chunk < n; chunk += (long long)gridDim.x * DEP_CHUNK) {
    const long long q0 = chunk + (threadIdx.x >> 5) * DEP_WARP_CHUNK + 4 * lane;  // and 128 further, ...
    int c[P];
    float ox[P], oy[P], vx[P], vy[P], vz[P];
#pragma unroll
    for (int h = 0; h < P; h += 4) {
      const long long q = q0 + 32 * h;
      if (q + 4 <= n) {
        const int4 cc = *reinterpret_cast<const int4*>(p.cell + q);
        const float4 a = *reinterpret_cast<const float4*>(p.ox + q);
        const float4 b = *reinterpret_cast<const float4*>(p.oy + q);
        const float4 u = *reinterpret_cast<const float4*>(p.vx + q);
        const float4 v = *reinterpret_cast<const float4*>(p.vy + q);
        c[h] = cc.x; c[h + 1] = cc.y; c[h + 2] = cc.z; c[h + 3] = cc.w;
        ox[h] = a.x; ox[h + 1] = a.y; ox[h + 2] = a.z; ox[h + 3] = a.w;
        oy[h] = b.x; oy[h + 1] = b.y; oy[h + 2] = b.z; oy[h + 3] = b.w;
        vx[h] = u.x; vx[h + 1] = u.y; vx[h + 2] = u.z; vx[h + 3] = u.w;
        vy[h] = v.x; vy[h + 1] = v.y; vy[h + 2] = v.z; vy[h + 3] = v.w;
        if (SEL) {
          const float4 w = *reinterpret_cast<const float4*>(p.vz + q);
          vz[h] = w.x; vz[h + 1] = w.y; vz[h + 2] = w.z; vz[h + 3] = w.w;
        }
      } else {
#pragma unroll
        for (int k = h; k < h + 4; k++) {
          const long long m = q + k - h;
          const bool in = m < n;
          c[k] = in ? p.cell[m] : -1;
          ox[k] = in ? p.ox[m] : 0.f;
          oy[k] = in ? p.oy[m] : 0.f;
          vx[k] = in ? p.vx[m] : 0.f;
          vy[k] = in ? p.vy[m] : 0.f;
          vz[k] = (SEL && in) ? p.vz[m] : 0.f;
        }
      }
    }
    unsigned int cand = 0;
#pragma unroll
    for (int k = 0; k < P; k++)
      if (c[k] >= 0) {
        push_mixed_one<EPIC_CIC, BC>(g, ef, qmK_dt, cx, cy, c[k], ox[k], oy[k], vx[k], vy[k]);
        if (SEL && mcc_candidate(sel, q0 + 31 * (k & ~3) + k, step, vx[k], vy[k], vz[k])) cand |= 1u << k;
      }
#pragma unroll
    for (int h = 0; h < P; h += 4) {
      const long long q = q0 + 32 * h;
      if (q + 4 <= n) {
        *reinterpret_cast<int4*>(p.cell + q) = make_int4(c[h], c[h + 1], c[h + 2], c[h + 3]);
        *reinterpret_cast<float4*>(p.ox + q) = make_float4(ox[h], ox[h + 1], ox[h + 2], ox[h + 3]);
        *reinterpret_cast<float4*>(p.oy + q) = make_float4(oy[h], oy[h + 1], oy[h + 2], oy[h + 3]);
        *reinterpret_cast<float4*>(p.vx + q) = make_float4(vx[h], vx[h + 1], vx[h + 2], vx[h + 3]);
        *reinterpret_cast<float4*>(p.vy + q) = make_float4(vy[h], vy[h + 1], vy[h + 2], vy[h + 3]);
      } else {
#pragma unroll
        for (int k = h; k < h + 4; k++)
          if (c[k] >= 0) {
            const long long m = q + k - h;
            p.cell[m] = c[k];
            p.ox[m] = ox[k];
            p.oy[m] = oy[k];
            p.vx[m] = vx[k];
            p.vy[m] = vy[k];
          }
      }
    }
    if (SEL && __any_sync(0xffffffffu, cand != 0)) {  // one atomic per warp with candidates
      const unsigned int mine = __popc(cand);
      unsigned int incl = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      unsigned int base = 0;
      if (lane == 31) base = atomicAdd(sel.cand_count, incl);
      unsigned int o = __shfl_sync(0xffffffffu, base, 31) + incl - mine;
#pragma unroll
      for (int k = 0; k < P; k++)
        if (cand & (1u << k)) sel.cand[o++] = (unsigned int)(q0 + 31 * (k & ~3) + k);
    }
    if (DEP) deposit_warp_sorted(acc, w, ConstNy{g.ny}, c, ox, oy);
  }
}

// Open boundaries or conductors: push + stable in-place compaction with
// ordered tiles (the FP64 form's scheme; see k_push_compact in
// epic_particles.cu).  COND: a particle that ends inside a conductor, its
// position taken as x0 + (i + ox) dx in FP64, is erased too
// (src/species.cpp:80-165).
template <int SHAPE, int BC, bool COND>
__global__ void __launch_bounds__(PART_THREADS) k_push_mixed_compact(Geom g, MixedSoA p, long long* d_n,
                                                                     const FieldCell* __restrict__ ef, float qmK_dt,
                                                                     float cx, float cy, unsigned long long* status,
                                                                     unsigned int* tile_ctr, int* flags,
                                                                     long long spin, CondSet cs) {
  constexpr int ITEMS = SCAN_TILE / PART_THREADS;
  __shared__ int sm[40];
  __shared__ unsigned long long s_prefix;
  __shared__ int s_tile;
  const long long n = *d_n;
  const int num_tiles = (int)((n + SCAN_TILE - 1) / SCAN_TILE);
  for (;;) {
    if (threadIdx.x == 0) s_tile = (int)atomicAdd(tile_ctr, 1u);
    __syncthreads();
    const int tile = s_tile;
    if (tile >= num_tiles) break;
    const long long base = (long long)tile * SCAN_TILE;
    int c[ITEMS], keep[ITEMS];
    float ox[ITEMS], oy[ITEMS], vx[ITEMS], vy[ITEMS], vz[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; k++) {
      const long long q = base + (long long)k * PART_THREADS + threadIdx.x;
      keep[k] = 0;
      if (q < n) {
        c[k] = p.cell[q]; ox[k] = p.ox[q]; oy[k] = p.oy[q]; vx[k] = p.vx[q]; vy[k] = p.vy[q]; vz[k] = p.vz[q];
        keep[k] = push_mixed_one<SHAPE, BC>(g, ef, qmK_dt, cx, cy, c[k], ox[k], oy[k], vx[k], vy[k]);
        if (COND && keep[k]) {
          int i, j;
          split_cell(c[k], g.ny, i, j);
          const double x = __dadd_rn(g.x0, __dmul_rn(__dadd_rn((double)i, (double)ox[k]), g.dx));
          const double y = __dadd_rn(g.y0, __dmul_rn(__dadd_rn((double)j, (double)oy[k]), g.dy));
          keep[k] = !in_conductor(cs, x, y);
        }
      }
    }
    int rank[ITEMS];
    const int tile_total = tile_ranks(keep, rank, sm);
    if (threadIdx.x < 32) {
      const unsigned long long before = tile_lookback(status, tile, (unsigned long long)tile_total, flags, spin);
      if (threadIdx.x == 0) s_prefix = before;
    }
    __syncthreads();
    const unsigned long long prefix = s_prefix;
    if (prefix != ~0ull) {
#pragma unroll
      for (int k = 0; k < ITEMS; k++) {
        if (keep[k]) {
          const long long o = (long long)prefix + rank[k];
          p.cell[o] = c[k]; p.ox[o] = ox[k]; p.oy[o] = oy[k]; p.vx[o] = vx[k]; p.vy[o] = vy[k]; p.vz[o] = vz[k];
        }
      }
      if (tile == num_tiles - 1 && threadIdx.x == 0) *d_n = (long long)prefix + tile_total;
    }
    __syncthreads();
  }
}

void launch_push_mixed(cudaStream_t st, const Geom& g, int shape, int bc, const MixedSoA& p, long long* d_n,
                       const FieldCell* ef, float qmK_dt, float cx, float cy, int* flags,
                       unsigned long long* tile_status, unsigned int* tile_ctr, int grid,
                       unsigned long long* dep_acc, const SelectArgs* sel, const CondSet* cond, bool bands) {
  if (cond) {  // the compacting push with the conductor test, for any wall rule
#define PC(SH, B) \
  k_push_mixed_compact<SH, B, true><<<grid, PART_THREADS, 0, st>>>(g, p, d_n, ef, qmK_dt, cx, cy, tile_status, tile_ctr, \
                                                                   flags, spin_limit(), *cond)
#define PCB(SH)                          \
  do {                                   \
    if (bc == EPIC_OPEN) PC(SH, EPIC_OPEN); \
    else if (bc == EPIC_PBC) PC(SH, EPIC_PBC); \
    else PC(SH, EPIC_REFLECTIVE);        \
  } while (0)
    if (shape == EPIC_NGP) PCB(EPIC_NGP);
    else PCB(EPIC_CIC);
#undef PCB
#undef PC
    return;
  }
#define PM(SH, B) k_push_mixed<SH, B><<<grid, PART_THREADS, 0, st>>>(g, p, d_n, ef, qmK_dt, cx, cy)
  if (dep_acc && shape == EPIC_CIC && (bc == EPIC_PBC || bc == EPIC_REFLECTIVE)) {
    const SelectArgs a = sel ? *sel : SelectArgs{};
    // one wave of resident CTAs (the kernel strides over the chunks)
#define PD(B, S)                                                                                                   \
  do {                                                                                                             \
    if (bands)                                                                                                     \
      k_push_mixed_dep<B, S, false><<<resident_grid(k_push_mixed_dep<B, S, false>, PART_THREADS), PART_THREADS, 0, \
                                      st>>>(g, p, d_n, ef, qmK_dt, cx, cy, dep_acc, a);                            \
    else                                                                                                           \
      k_push_mixed_dep<B, S, true><<<resident_grid(k_push_mixed_dep<B, S, true>, PART_THREADS), PART_THREADS, 0,   \
                                     st>>>(g, p, d_n, ef, qmK_dt, cx, cy, dep_acc, a);                             \
  } while (0)
    if (bc == EPIC_PBC) { if (sel) PD(EPIC_PBC, true); else PD(EPIC_PBC, false); }
    else { if (sel) PD(EPIC_REFLECTIVE, true); else PD(EPIC_REFLECTIVE, false); }
    if (bands) launch_deposit_mixed_bands(st, g, p, d_n, dep_acc);
#undef PD
    return;
  }
  if (bc == EPIC_OPEN) {
    if (shape == EPIC_NGP)
      k_push_mixed_compact<EPIC_NGP, EPIC_OPEN, false><<<grid, PART_THREADS, 0, st>>>(
          g, p, d_n, ef, qmK_dt, cx, cy, tile_status, tile_ctr, flags, spin_limit(), CondSet{});
    else
      k_push_mixed_compact<EPIC_CIC, EPIC_OPEN, false><<<grid, PART_THREADS, 0, st>>>(
          g, p, d_n, ef, qmK_dt, cx, cy, tile_status, tile_ctr, flags, spin_limit(), CondSet{});
  } else if (bc == EPIC_PBC) {
    if (shape == EPIC_NGP) PM(EPIC_NGP, EPIC_PBC);
    else PM(EPIC_CIC, EPIC_PBC);
  } else {
    if (shape == EPIC_NGP) PM(EPIC_NGP, EPIC_REFLECTIVE);
    else PM(EPIC_CIC, EPIC_REFLECTIVE);
  }
#undef PM
}

// Species::Rewind_species (src/species.cpp:229-246): v -= (0.5*qm*K*DT) E.
template <int SHAPE>
__global__ void __launch_bounds__(PART_THREADS) k_rewind_mixed(Geom g, MixedSoA p, const long long* __restrict__ d_n,
                                                               const FieldCell* __restrict__ ef, float hqmK_dt) {
  const long long n = *d_n;
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
    float ex, ey;
    gather32<SHAPE>(g, ef, p.cell[q], p.ox[q], p.oy[q], ex, ey);
    p.vx[q] = fmaf(-hqmK_dt, ex, p.vx[q]);
    p.vy[q] = fmaf(-hqmK_dt, ey, p.vy[q]);
  }
}

void launch_rewind_mixed(cudaStream_t st, const Geom& g, int shape, const MixedSoA& p, const long long* d_n,
                         const FieldCell* ef, float hqmK_dt, int* flags, int grid) {
  (void)flags;
  if (shape == EPIC_NGP) k_rewind_mixed<EPIC_NGP><<<grid, PART_THREADS, 0, st>>>(g, p, d_n, ef, hqmK_dt);
  else k_rewind_mixed<EPIC_CIC><<<grid, PART_THREADS, 0, st>>>(g, p, d_n, ef, hqmK_dt);
}

// ------------------------------------------------------- reductions ---
// Energy / momentum sums of the FP32 velocities (Species::Compute_KE /
// Compute_Momentum, src/species.cpp:248-297): momenta accumulated in FP64,
// squares as fixed-point integers.
//
// In FP64 a particle's energy is 15 instructions of a pipe that takes two lanes
// a clock: 1.05e8 particles took 2.4 ms, a sixth of the memory's rate; so 0.43,
// call and copy of the result included.  The square of a 24-bit significand is 48 bits exactly, one integer multiply; a
// thread adds the squares to a 64-bit sum whose unit it doubles as larger terms
// or a large sum arrive (rare after the first particles), at 2^-52 of the
// largest term or finer (the largest itself is exact), and converts once at the
// end.
struct SquareSum {
  unsigned long long v = 0;  // v 2^unit
  int unit = -400;
  double odd = 0;            // infinities and NaN
  __device__ __forceinline__ void add(float x) {
    const unsigned b = __float_as_uint(x) & 0x7FFFFFFFu;
    const int e = (int)(b >> 23);
    const int t = e == 255 ? 1 << 20 : 2 * max(e, 1) - 310;  // the square is m 2^t
    const unsigned s = (b & 0x7FFFFFu) | (e ? 0x800000u : 0u);
    const unsigned long long m = (unsigned long long)s * s << 10;
    if (t > unit || v >> 62) {
      if (e == 255) {
        odd += (double)x * x;
        return;
      }
      const int to = max(t + 6, v >> 62 ? unit + 8 : unit);
      v = to - unit < 64 ? ((v >> (to - unit - 1)) + 1) >> 1 : 0;
      unit = to;
    }
    v += (xs_shr(m << 1, (unsigned)(unit - t)) + 1) >> 1;
  }
  // Exact up to one rounding to 53 bits.
  __device__ __forceinline__ double value() const {
    return __dadd_rn(__dmul_rn(__ull2double_rn(v), xs_double((uint64_t)(1023 + max(unit, -1000)) << 52)), odd);
  }
};

__device__ __forceinline__ double warp_sum_m(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

template <int WHAT>
__global__ void __launch_bounds__(PART_THREADS) k_particle_sums_mixed(MixedSoA p, const long long* __restrict__ d_n,
                                                                      double vn, double* partials) {
  const long long n = *d_n, first = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long stride = (long long)gridDim.x * blockDim.x;
  double s0 = 0, s1 = 0, s2 = 0;
  if (WHAT == 0) {
    SquareSum a, b, c;
    for (long long q = first; q < n / 4; q += stride) {
      const float4 x = reinterpret_cast<const float4*>(p.vx)[q], y = reinterpret_cast<const float4*>(p.vy)[q],
                   z = reinterpret_cast<const float4*>(p.vz)[q];
      a.add(x.x); a.add(x.y); a.add(x.z); a.add(x.w);
      b.add(y.x); b.add(y.y); b.add(y.z); b.add(y.w);
      c.add(z.x); c.add(z.y); c.add(z.z); c.add(z.w);
    }
    const long long q = (n & ~3ll) + first;
    if (q < n) {
      a.add(p.vx[q]);
      b.add(p.vy[q]);
      c.add(p.vz[q]);
    }
    s0 = a.value() * vn * vn;
    s1 = b.value() * vn * vn;
    s2 = c.value() * vn * vn;
  } else {
    for (long long q = first; q < n; q += stride) {
      const double a = p.vx[q], b = p.vy[q], c = p.vz[q];
      s0 += a * vn;
      s1 += b * vn;
      s2 += c * vn;
    }
  }
  __shared__ double sm[3][PART_THREADS / 32];
  s0 = warp_sum_m(s0);
  s1 = warp_sum_m(s1);
  s2 = warp_sum_m(s2);
  if ((threadIdx.x & 31) == 0) {
    sm[0][threadIdx.x >> 5] = s0;
    sm[1][threadIdx.x >> 5] = s1;
    sm[2][threadIdx.x >> 5] = s2;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double t = 0;
    for (int w = 0; w < PART_THREADS / 32; w++) t += sm[threadIdx.x][w];
    partials[blockIdx.x * 3 + threadIdx.x] = t;
  }
}

__global__ void k_sum_partials3_m(const double* partials, int nblocks, double* out) {
  const int c = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (c >= 3) return;
  double t = 0;
  for (int b = lane; b < nblocks; b += 32) t += partials[b * 3 + c];
  t = warp_sum_m(t);
  if (lane == 0) out[c] = t;
}

void launch_particle_sums_mixed(cudaStream_t st, int what, const MixedSoA& p, const long long* d_n, double vel_norm,
                                double* partials, double* out3, int grid) {
  if (what == 0) k_particle_sums_mixed<0><<<grid, PART_THREADS, 0, st>>>(p, d_n, vel_norm, partials);
  else k_particle_sums_mixed<1><<<grid, PART_THREADS, 0, st>>>(p, d_n, vel_norm, partials);
  k_sum_partials3_m<<<1, 96, 0, st>>>(partials, grid, out3);
}

}  // namespace epic
