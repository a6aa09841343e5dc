// FieldSolve::pcgsolver (src/field.cpp:212-264) with pcg()
// (linearalgebra/solvers.h:73-100) in the eigenbasis of its operator.
//
// The operator on the lattice of unknowns (Lattice: R rows of C columns) is
// -L, L = T_R (x) I + I (x) T_C with T the negative second difference, and
// the Jacobi preconditioner is the constant -1/4, which scales every iterate
// of CG alike and drops out.  The orthonormal, symmetric sine (walls) and
// Hartley (periodic) transforms Q diagonalise T, and CG commutes with an
// orthogonal change of basis: its iterates on (L, b) are Q times its iterates
// on (Q L Q, Q b).  In that basis a vector component only ever meets its own
// eigenvalue, so an iteration has no neighbours, no halo and no exchange but
// the two dot products.  And every residual is a polynomial in L applied to
// b, so the components of one eigenvalue stay in fixed proportion: the set of
// components with equal eigenvalue by symmetry (k and n - k of a periodic
// direction, (j, k) and (k, j) of a square lattice) is carried as one
// component of its norm.  A solve keeps 1/2 of the lattice's components with
// walls on a square, 1/8 on a periodic square, 1/4, 1/2 or all elsewhere.
// The iterates are the reference's up to rounding (checked against the
// oracle: equal iteration counts, phi within 1e-12).
//
// One cooperative launch runs the whole solve: b transformed line by line,
// the iterations with each component in a thread's registers, and the
// solution transformed back.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "epic_internal.cuh"
#include "epic_xsum.cuh"

namespace epic {

constexpr int PM_T = 256;           // threads that hold components
constexpr int PM_ALL = PM_T + 32;   // and the scalar warp
constexpr int PM_W = PM_T / 32;
constexpr int PM_CLUSTER = 16;      // CTAs of the one-cluster form
constexpr int PM_MAX_BLOCKS = 160;  // CTAs of the whole-GPU form: five words of each sum per polling lane
constexpr int PM_MAX_SIDE = 2048;   // lattice side whose transform tables fit shared memory
constexpr int PM_MAX_NPT = 16;      // components per thread

// ---- barrier of the set-up and final phases ----
// One cluster: its hardware barrier.  Whole GPU: each CTA counts its own
// episodes, so an arrival is a fire-and-forget red.release by thread 0 after a
// __syncthreads that orders the block's writes before it.  Bounded:
// FLAG_TIMEOUT and false on giving up.
template <bool CLUSTER>
__device__ __forceinline__ bool pm_barrier(unsigned int* bar, int* flags, unsigned int& target, int* s_ok,
                                           long long limit) {
  if (CLUSTER) {
    cooperative_groups::this_cluster().sync();
    return true;
  }
  __syncthreads();
  target += gridDim.x;
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(bar), "r"(1u) : "memory");
    int ok = 1;
    long long spins = 0;
    for (;;) {
      unsigned int v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
      if ((int)(v - target) >= 0) break;
      if (++spins >= limit) {
        atomicOr(flags, FLAG_TIMEOUT);
        ok = 0;
        break;
      }
    }
    *s_ok = ok;
  }
  __syncthreads();
  return *s_ok;
}

// ---- scalars ----
// The few scalars of an iteration are a serial chain between the words'
// arrival and the next update, and the totals are integers already.  An FP64
// instruction of a warp holds its quarter of the SM for 64 cycles, converting
// a 64-bit integer to FP64 takes ~215 and a library division ~590 (measured),
// a 64 x 64-bit high product ~40: so the scalars are 64-bit significands with
// an exponent, value = m 2^e, the top bit of m set (m = 0: zero), truncated;
// 11 bits more than FP64 carries.  alpha and beta are rounded once.
struct PmF {
  unsigned long long m;
  int e;
};

// V 2^E
__device__ __forceinline__ PmF pmf_from(unsigned long long V, int E) {
  const int z = V ? __clzll((long long)V) : 0;
  return PmF{V << z, E - z};
}
__device__ __forceinline__ PmF pmf_mul(PmF a, PmF b) {
  const unsigned long long hi = __umul64hi(a.m, b.m);
  const int up = hi >> 63 ? 0 : 1;
  PmF r;
  r.m = hi << up;
  r.e = a.e + b.e + 64 - up;
  return r;
}
// a - b; neg: the sign
__device__ __forceinline__ PmF pmf_sub(PmF a, PmF b, bool& neg) {
  const int E = a.m == 0 ? b.e : b.m == 0 ? a.e : max(a.e, b.e);
  const unsigned long long am = xs_shr(a.m, (unsigned)min(E - a.e, 64)), bm = xs_shr(b.m, (unsigned)min(E - b.e, 64));
  neg = bm > am;
  const unsigned long long d = neg ? bm - am : am - bm;
  const int z = d ? __clzll((long long)d) : 0;
  PmF r;
  r.m = d << z;
  r.e = E - z;
  return r;
}
// 1/a (a not 0): with x = m/2^63 in [1, 2) and y0 the approximate reciprocal
// of its leading 21 bits, err = 1 - x y0 (exact, y0 has 21 bits), 1/x =
// y0 (1 + err + err^2 + err^3 + ...).  rcp.approx.ftz.f64 reads and gives 20
// fraction bits: |err| < 2^-18, err^4 < 2^-72.
__device__ __forceinline__ PmF pmf_recip(PmF a) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;"
      : "=d"(y)
      : "d"(__hiloint2double(0x3FF00000 | (int)((a.m >> 43) & 0xFFFFF), 0)));
  const unsigned h = (unsigned)__double2hiint(y);  // (0.5, 1]: exponent 1022, or 1023 for 1.0
  const unsigned Y = h >= 0x3FF00000u ? 1u << 21 : (h & 0xFFFFFu) | 0x100000u;            // y0 2^21
  const xs_uint prod = (xs_uint)a.m * Y;                                        // x y0 2^84
  const long long er = (long long)((((xs_int)1 << 84) - (xs_int)prod) >> 4);    // err 2^80, |err| < 2^-18
  const int eh = (int)(er >> 31);                                               // err 2^49
  const long long e2 = (long long)eh * eh;                                      // err^2 2^98
  const long long f = er + (e2 >> 18) + (((long long)(int)(e2 >> 49) * eh) >> 18);
  const unsigned long long q = ((unsigned long long)Y << 42) + (unsigned long long)(long long)(((xs_int)f * Y) >> 38);
  PmF r;
  r.m = q >> 63 ? ~0ull : q << 1;  // q = 2^63 / x <= 2^63
  r.e = -127 - a.e;
  return r;
}
// The nearest double (results outside the normal range: 0 or infinity).
__device__ __forceinline__ double pmf_double(PmF a, bool neg) {
  const unsigned long long q = (a.m >> 11) + ((a.m >> 10) & 1);  // [2^52, 2^53]; the carry moves into the exponent
  const int E = a.e + 63 + 1023;
  unsigned long long b = ((unsigned long long)(unsigned)(E - 1) << 52) + q;
  if (a.m == 0 || E <= 0) b = 0;
  if (a.m && E >= 2046) b = 0x7FFull << 52;
  return xs_double(b | (neg ? 1ull << 63 : 0));
}

// ---- the two dot products ----
// Sums of squares as 64-bit fixed-point integers on the integer pipe, summed
// as three limbs with redux.sync over a warp and carried across CTAs in words
// that are at once the barrier: a 64-bit word holds its sum (62 bits) and the
// round's tag (2 bits).  Nothing but the words crosses CTAs in an iteration, so
// relaxed accesses suffice.  Words alternate by round parity: a CTA writes
// those of round k + 2 only after it has seen every word of k + 1, whose
// writers had read all words of k; tags of the same parity differ between
// rounds that follow each other.
//
// Over the whole GPU every CTA writes its two words to global memory and one
// of its warps polls all of them (nothing queues on one address, and no second
// trip fetches totals); in one cluster every warp writes its two words into
// the shared memory of every CTA, and the poll is local: ~380 cycles against
// ~1,500 (measured, 16 and 152 CTAs).  Global words are first polled PM_DELAY
// cycles after the own ones are written: polls in flight while the others'
// words arrive hold them up (152 CTAs: 3,700 cycles polled at once, 1,500 after
// 200 to 400).  Whole iterations, first poll after 350, 400, 475, 525 cycles:
// 129 x 129 2.08, 1.87, 1.82, 1.85 us; 98 x 145 1.98, 1.86, 1.83, 1.85; 257 x 256
// 1.80, 1.83, 1.85, 1.88; 1024 x 1024 periodic 2.50, 2.53, 2.55, 2.59.
//
// Anchors: against the biased exponent E of the last total, a term with biased
// exponent e is its significand times 2^(6 + e - E), so the last total stands at
// 2^58.  Terms are rounded PM_FRAC bits below that unit (622,592 of them: half a
// unit off) and only the words to the unit itself: at most 160 words, evenly
// spread, are 2^-56 of the last total off (worst case 2^-52), whatever the number
// of terms.  (Each term rounded to the unit: 2^-54 with 4,000 terms, 2^-50 with
// 600,000; alpha of 65,000 terms up to 7e-16 off, 6e-17 so.)  A total below a
// quarter of its anchor has lost two of those bits, and its round is repeated with
// the anchors it has found.  Each sum has its own anchor.  A sum beyond 2^61 (a
// total that grew eightfold in one step) or a term beyond 2^61 marks the word; the
// round is then repeated with anchors PM_WIDEN higher.  A sum that stays beyond
// every anchor is not finite: phi is NaN then, as the reference's would be.
constexpr int PM_TOP = 6;
constexpr int PM_SCALE = -1075 - PM_TOP;  // a sum V against anchor E is V 2^(E + PM_SCALE)
constexpr int PM_WIDEN = 24;
constexpr int PM_NARROW = 52;  // lower, where nothing of a total shows
constexpr int PM_FRAC = 9;
constexpr int PM_DELAY = 400;
constexpr unsigned long long PM_OUT = (1ull << 62) - 1;

// A thread's sum against an anchor.
struct PmSum {
  unsigned long long v = 0;  // units
  unsigned f = 0;            // 2^-PM_FRAC of one
  bool out = false;          // a term or the sum is out of range
  // m 2^-n units
  __device__ __forceinline__ void add(unsigned long long m, int n) {
    const unsigned long long below = xs_shl(m, (unsigned)(64 - n)) | xs_shr(m, (unsigned)(n - 64));
    v += xs_shr(m, (unsigned)n);
    f += ((unsigned)(below >> (63 - PM_FRAC)) + 1) >> 1;
    out |= (m && n < 3) || (v >> 61) != 0;
  }
};

// r^2 and L r^2 of a component, added to the sums.  From the significands: a
// 64 x 64-bit high product takes ~40 cycles of the integer pipe, an FP64 product
// holds the warp's quarter of the SM for 64 and its result would have to be
// taken apart again (an iteration at 257 x 257: 1.89 us with FP64 products,
// 1.82 us so; with 16 components a thread, 1024 x 1024: 6.8 against 6.0 us).
// Cut at 2^-62 of the term, where an FP64 product is rounded at 2^-53.
__device__ __forceinline__ void pm_terms(PmSum& s0, PmSum& s1, double r, double L, int E0, int E1) {
  const unsigned long long b = xs_bits(r), l = xs_bits(L);  // L >= 0
  const int eb = (int)((b >> 52) & 0x7FF), el = (int)(l >> 52);
  const unsigned long long m = eb ? (b << 11) | (1ull << 63) : 0ull;  // |r| = m 2^(eb - 1086); below the normal range: 0
  const unsigned long long lm = el ? (l << 11) | (1ull << 63) : 0ull;
  const unsigned long long p = __umul64hi(m, m), q = __umul64hi(p, lm);  // r^2 = p 2^(2 eb - 2108), L r^2 = q 2^(2 eb + el - 3130)
  s0.add(p, E0 + 1027 - 2 * eb);  // shifts to the anchors
  s1.add(q, E1 + 2049 - 2 * eb - el);
  s0.out |= eb >= 2047;
}

// A warp's total in every lane, as three limbs whose sums over the eight warps of
// a CTA still fit 32 bits: 14 bits of units with the bits below, 24, and the rest
// (2^23 and more: out of range).
constexpr int PM_L1 = 14, PM_L2 = PM_L1 + 24;
template <int NPT>
__device__ __forceinline__ uint3 pm_warp_sum(const PmSum& s) {
  unsigned long long v = s.v;
  unsigned f = s.f;
  if (NPT > 1) {
    v += f >> PM_FRAC;
    f &= (1u << PM_FRAC) - 1;
  }
  uint3 l;
  l.x = __reduce_add_sync(0xffffffffu, (((unsigned)v & ((1u << PM_L1) - 1)) << PM_FRAC) + f);
  l.y = __reduce_add_sync(0xffffffffu, (unsigned)(v >> PM_L1) & ((1u << 24) - 1));
  l.z = __reduce_add_sync(0xffffffffu, s.out ? 1u << (61 - PM_L2) : (unsigned)(v >> PM_L2));
  return l;
}
// Limbs as units, rounded; saturated to PM_OUT from 2^61 on.
__device__ __forceinline__ unsigned long long pm_units(uint3 l) {
  const unsigned long long t = ((l.x + (1u << (PM_FRAC - 1))) >> PM_FRAC) + ((unsigned long long)l.y << PM_L1) +
                               ((unsigned long long)l.z << PM_L2);
  return l.z >> (61 - PM_L2) || t >> 61 ? PM_OUT : t;
}

__device__ __forceinline__ void pm_store(ulonglong2* p, int half, unsigned long long w) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(reinterpret_cast<unsigned long long*>(p) + half), "l"(w)
               : "memory");
}
__device__ __forceinline__ ulonglong2 pm_load(const ulonglong2* p) {
  ulonglong2 v;
  asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
               : "=l"(v.x), "=l"(v.y)
               : "l"(p)
               : "memory");
  return v;
}
__device__ __forceinline__ void pm_store_cluster(unsigned addr, unsigned long long w) {
  asm volatile("st.relaxed.cluster.shared::cluster.u64 [%0], %1;" ::"r"(addr), "l"(w) : "memory");
}
__device__ __forceinline__ unsigned long long pm_load_cta(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.volatile.shared::cta.u64 %0, [%1];"
               : "=l"(v)
               : "r"((unsigned)__cvta_generic_to_shared(p))
               : "memory");
  return v;
}

// Named barriers between the component warps and the scalar warp.
__device__ __forceinline__ void pm_bar_sync(int id) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(PM_ALL) : "memory");
}
__device__ __forceinline__ void pm_bar_arrive(int id) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(PM_ALL) : "memory");
}

// One CTA's exact partial of a sum of non-negative FP64 values: V * 2^(a - 1129).
struct PmPartial {
  unsigned long long lo;
  long long hi;
  long long a;
  long long pad;
};

// ---- transforms ----
// One direction of n unknowns: sine, Q_jk = sqrt(2/(n+1)) sin(pi j k/(n+1)),
// j, k in [1, n]; or Hartley, Q_jk = cas(2 pi j k/n)/sqrt(n), j, k in [0, n).
// Tables (tab): sin(pi m/(n+1)), m < 2(n+1); or cos and then sin(2 pi m/n),
// m < n.  eig: the n eigenvalues of the negative second difference.
struct PmDir {
  int n, sine, M;  // M: period of the angle index
  int tab, ntab, eig;  // offsets into the tables
  int np;          // pairs of outputs of a line
  double scale;
};

struct PcgModes {
  PmDir r, c;       // along a column (R unknowns), along a row (C unknowns)
  int nA, nC;       // distinct row and column indices
  int swap;         // (a, c) and (c, a) are one component
  int N, per;       // components, and per CTA
  int B;            // CTAs
  int cluster;      // one cluster of B CTAs, else the whole-GPU form
  int ntab;         // doubles of all tables
  int tab_in_work;  // tables in work[2] (else in the partials buffer)
  int smem;         // bytes of dynamic shared memory
};

// Byte offsets in the partials buffer: words [2][B], the error's partials,
// the tables of small lattices.
constexpr size_t PM_PART_OFF = 2 * PM_MAX_BLOCKS * sizeof(ulonglong2);
constexpr size_t PM_TAB_OFF = PM_PART_OFF + PM_MAX_BLOCKS * sizeof(PmPartial);
constexpr int PM_TAB_MAX = (int)((16 * 320 * sizeof(double) - PM_TAB_OFF) / sizeof(double));
static_assert(PM_TAB_OFF < 16 * 320 * sizeof(double), "words and partials must fit the solver partials buffer");

__device__ void pm_table_entry(const PmDir& d, int q, double* tab) {
  if (q < d.ntab) {
    double v;
    if (d.sine) v = sinpi((double)q / (double)(d.n + 1));
    else v = q < d.n ? cospi(2.0 * q / (double)d.n) : sinpi(2.0 * (q - d.n) / (double)d.n);
    tab[d.tab + q] = v;
  } else {
    const int k = q - d.ntab;
    const double s = d.sine ? sinpi((k + 1) / (2.0 * (d.n + 1))) : sinpi(k / (double)d.n);
    tab[d.eig + k] = 4.0 * s * s;
  }
}

// nlines transforms along direction d, line `l` read by load(l, j) and written
// by store(l, k, value), j, k in [0, n).  FP64-pipe bound (an FP64 instruction
// of a warp holds its quarter of the SM for 64 cycles), so what counts is
// their number: the lines are folded about their middle (the bases are even
// or odd about it), which halves them to n^2 / 2 per line.  Where the halves
// fold again (Hartley of even n: about the quarter, by the parity of k; sine of
// odd n: the even outputs, by the parity of k / 2), n^2 / 4 or 3 n^2 / 8 are
// left (1024 x 1024 periodic, set-up and four passes: 3.77 ms with one fold,
// 2.03 with two).  An item is a line
// and a pair of its outputs, one thread's work; the CTAs take equal runs of
// items (whole lines would leave a third of the SMs idle with 255 lines on
// 152).
template <class Load, class Store>
__device__ void pm_lines(const PmDir& d, int nlines, const double* gtab, double* sm, const Load& load,
                         const Store& store) {
  const int n = d.n, M = d.M, np = d.np, ld = 2 * (n / 2 + 2);
  double* const tab = sm;
  double* const lines = sm + d.ntab;
  for (int q = threadIdx.x; q < d.ntab; q += PM_ALL) tab[q] = __ldcg(gtab + d.tab + q);
  const double* const tab1 = d.sine ? tab : tab + n;
  const bool quarter = !d.sine && n % 2 == 0, half = d.sine && n % 2 == 1;  // second folds
  const int j0 = d.sine ? 1 : 0, J = d.sine ? (n + 1) / 2 : quarter ? n / 4 : n / 2;  // folded indices j0..J
  const int nj = J - j0 + 1, J2 = (n + 1) / 4;
  const int items = nlines * np, share = (items + gridDim.x - 1) / gridDim.x;
  const int lo = blockIdx.x * share, hi = min(items, lo + share);
  for (int base = lo; base < hi; base += PM_T) {
    const int end = min(hi, base + PM_T), l0 = base / np, nl = (end - 1) / np - l0 + 1;
    __syncthreads();
    for (int q = threadIdx.x; q < nl * nj; q += PM_ALL) {
      const int l = q / nj, j = j0 + q - l * nj;
      double* const to = lines + l * ld;
      const int a = d.sine ? j - 1 : j, b = d.sine ? n - j : (j ? n - j : 0);
      const double xa = load(l0 + l, a), xb = a != b ? load(l0 + l, b) : 0.0;
      const double e = xa + xb, o = a != b ? xa - xb : 0.0;
      if (!quarter && !half) {
        to[j] = e;
        to[ld / 2 + j] = o;
        continue;
      }
      if (half) to[j] = e;
      const int h = (half ? (n + 1) / 2 : n / 2) - j;  // the partner
      if (half && (h < 1 || j > J2)) continue;         // the middle's odd part is 0; partners are taken with j
      const int a2 = half ? h - 1 : h, b2 = half ? n - h : n - h;
      const bool self = h == j;
      const double ya = self ? 0.0 : load(l0 + l, a2), yb = self || a2 == b2 ? 0.0 : load(l0 + l, b2);
      const double e2 = ya + yb, o2 = a2 != b2 ? ya - yb : 0.0;
      if (half) {
        to[ld / 2 + j - 1] = o + o2;
        to[ld / 2 + J2 + j - 1] = self ? 0.0 : o - o2;
      } else {
        to[j] = e + e2;
        to[ld / 4 + j] = self ? 0.0 : e - e2;
        to[2 * (ld / 4) + j] = self ? 0.0 : o - o2;
        to[3 * (ld / 4) + j] = o + o2;
      }
    }
    __syncthreads();
    const int it = base + threadIdx.x;
    if (threadIdx.x >= PM_T || it >= end) continue;
    const int line = it / np, m = it - line * np;
    const int k0 = d.sine ? 2 * m + 1 : m, k1 = d.sine ? 2 * m + 2 : m;
    const double* const at = lines + (line - l0) * ld;
    const double* const e = at + (quarter && (m & 1) ? ld / 4 : 0);
    const double* const o = half ? at + ld / 2 - 1 + (m & 1 ? J2 : 0)
                            : quarter ? at + (2 + (m & 1)) * (ld / 4) : at + ld / 2;
    const int Jo = half ? J2 : J;
    const int d0 = k0 % M, d1 = k1 % M;
    double s0 = 0, s1 = 0;
    int i0 = d.sine ? d0 : 0, i1 = d.sine ? d1 : 0;
#pragma unroll 4
    for (int j = j0; j <= Jo; j++) {
      s0 = fma(e[j], tab[i0], s0);
      s1 = fma(o[j], tab1[i1], s1);
      i0 += d0;
      i0 -= i0 >= M ? M : 0;
      i1 += d1;
      i1 -= i1 >= M ? M : 0;
    }
#pragma unroll 4
    for (int j = Jo + 1; j <= J; j++) {
      s0 = fma(e[j], tab[i0], s0);
      i0 += d0;
      i0 -= i0 >= M ? M : 0;
    }
    if (d.sine) {
      store(line, k0 - 1, d.scale * s0);
      if (k1 <= n) store(line, k1 - 1, d.scale * s1);
    } else {
      store(line, m, d.scale * (s0 + s1));
      if (m && 2 * m != n) store(line, n - m, d.scale * (s0 - s1));
    }
  }
}

// Component u as its row and column indices (a, c).
__device__ __forceinline__ void pm_component(const PcgModes& t, int u, int& a, int& c) {
  if (!t.swap) {
    a = u / t.nC;
    c = u - a * t.nC;
    return;
  }
  // a <= c: rows a and nA - 1 - a of the triangle side by side
  const int p = u / (t.nA + 1), q = u - p * (t.nA + 1);
  if (q < t.nA - p) {
    a = p;
    c = p + q;
  } else {
    a = t.nA - 1 - p;
    c = a + q - (t.nA - p);
  }
}

// f(index) for every lattice component of the distinct component (a, c);
// component (row m, column k) of the transformed lattice is at k * R + m.
template <class F>
__device__ __forceinline__ void pm_orbit(const PcgModes& t, int a, int c, const F& f) {
  const int R = t.r.n, C = t.c.n;
  const bool ra = !t.r.sine && a && 2 * a != R, rc = !t.c.sine && c && 2 * c != C;
  auto four = [&](int m, bool m2, int k, bool k2) {
    f(k * R + m);
    if (m2) f(k * R + R - m);
    if (k2) {
      f((C - k) * R + m);
      if (m2) f((C - k) * R + R - m);
    }
  };
  four(a, ra, c, rc);
  if (t.swap && a != c) four(c, rc, a, ra);  // R = C there
}

template <int NPT, bool CLUSTER>
__global__ void __launch_bounds__(PM_ALL) k_pcg_modes(SolverArgs a, PcgModes t) {
  extern __shared__ double sm[];
  __shared__ uint4 s_sum[2][PM_W];  // the warps' (r, r) and (r, L r) as limbs
  // one cluster: the words [parity][(r, r), (r, L r)][CTA][warp]
  __shared__ unsigned long long s_word[CLUSTER ? 2 * 2 * PM_CLUSTER * PM_W : 1];
  __shared__ int s_ok, s_it, s_nan, s_e[PM_W + 1];
  // by round parity: a warp without components may still read those of a
  // round when the scalar warp writes the next one's
  __shared__ int s_done[2], s_E[2][2], s_again[2];
  __shared__ double s_alpha[2], s_beta[2];
  __shared__ unsigned long long s_v[PM_W + 1][2];
  const Lattice lat = make_lattice(a.g.nx, a.g.ny, a.poisson_bc);
  const int R = lat.R, C = lat.C, nb = gridDim.x, me = blockIdx.x;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const double dx2 = a.g.dx * a.g.dx;
  const long long spin = spin_or_default(a.spin);
  ulonglong2* const words = reinterpret_cast<ulonglong2*>(a.partials);
  PmPartial* const parts = reinterpret_cast<PmPartial*>(reinterpret_cast<char*>(a.partials) + PM_PART_OFF);
  double* const gtab =
      t.tab_in_work ? a.work[2] : reinterpret_cast<double*>(reinterpret_cast<char*>(a.partials) + PM_TAB_OFF);
  double* const T1 = a.work[0];  // [row][column mode]
  double* const Bh = a.work[1];  // [column mode][row mode]
  unsigned int target = 0;
  // src/field.cpp:234-252: -rho dx^2 (L/LDe)^2, zero on the reference's grid
  // edges; every unknown of an extension lattice.
  auto rhs = [&](int r, int c) -> double {
    const int k = lattice_node(lat, r, c);
    if (lat.mode == EPIC_POISSON_DIRICHLET) {
      const int i = k / a.g.ny, j = k - i * a.g.ny;
      if (i == 0 || i == a.g.nx - 1 || j == 0 || j == a.g.ny - 1) return 0.0;
    }
    return -a.rho[k] * dx2 * a.K;
  };
  auto barrier = [&]() { return pm_barrier<CLUSTER>(a.bar, a.flags, target, &s_ok, spin); };

  // tables (shared when both directions are alike) and this CTA's words
  {
    const int nr = t.r.ntab + R, nall = t.c.tab == t.r.tab ? nr : nr + t.c.ntab + C;
    for (int q = me * PM_ALL + threadIdx.x; q < nall; q += nb * PM_ALL)
      if (q < nr) pm_table_entry(t.r, q, gtab);
      else pm_table_entry(t.c, q - nr, gtab);
    if (CLUSTER) {
      for (int q = threadIdx.x; q < 4 * PM_CLUSTER * PM_W; q += PM_ALL) s_word[q] = 0;
    } else if (threadIdx.x < 4) {
      pm_store(words + (threadIdx.x >> 1) * nb + me, threadIdx.x & 1, 0);
    }
  }
  if (!barrier()) return;
  pm_lines(t.c, R, gtab, sm, rhs, [&](int l, int k, double v) { T1[l * C + k] = v; });
  if (!barrier()) return;
  pm_lines(
      t.r, C, gtab, sm, [&](int l, int j) { return __ldcg(&T1[j * C + l]); },
      [&](int l, int k, double v) { Bh[l * R + k] = v; });
  if (!barrier()) return;

  // this thread's components: r = |b| of the component, L its eigenvalue
  const bool periodic = lat.mode == EPIC_POISSON_PERIODIC;
  const bool scalar = wid == PM_W;
  double r[NPT], L[NPT], q[NPT], w[NPT];
  auto component = [&](int j, int& ca, int& cc) -> bool {
    const int k = threadIdx.x + PM_T * j, u = me * t.per + k;
    if (scalar || k >= t.per || u >= t.N) return false;
    pm_component(t, u, ca, cc);
    return !(periodic && ca == 0 && cc == 0);  // the constant mode: b projected onto zero mean, phi of zero mean
  };
  auto norm_of = [&](int ca, int cc) {
    double s = 0;
    pm_orbit(t, ca, cc, [&](int k) {
      const double v = __ldcg(&Bh[k]);
      s = fma(v, v, s);
    });
    return sqrt(s);
  };
  int emax = 0;
#pragma unroll
  for (int j = 0; j < NPT; j++) {
    int ca, cc;
    r[j] = L[j] = q[j] = 0.0;
    if (component(j, ca, cc)) {
      r[j] = norm_of(ca, cc);
      L[j] = __ldcg(gtab + t.r.eig + ca) + __ldcg(gtab + t.c.eig + cc);
    }
    w[j] = L[j] * r[j];
    emax = max(emax, (int)(xs_bits(r[j] * r[j]) >> 52));
  }
  const double bmean = periodic ? __ldcg(&Bh[0]) / sqrt((double)R * (double)C) : 0.0;
  emax = (int)__reduce_max_sync(0xffffffffu, (unsigned)emax);
  if (lane == 0 && emax) atomicMax(a.bar + 1, (unsigned)emax);
  if (!barrier()) return;
  // anchors of the first round: far above the largest term (which may be
  // infinite or NaN)
  const int E0 = min((int)__ldcg(a.bar + 1), 2046) + PM_WIDEN;

  // min(n*n, max_iteration) as pcg() caps it: n*n in 32-bit int arithmetic for
  // the reference's lattice (it wraps, as there), in 64 bits for the extensions.
  const int n = R * C;
  const unsigned int cap32 = (unsigned int)n * (unsigned int)n;
  const long long cap = lat.mode == EPIC_POISSON_DIRICHLET ? (long long)(int)cap32 : (long long)n * n;
  const int maxit = cap < a.max_iter ? (int)cap : a.max_iter;

  // The Chronopoulos-Gear form: with gamma = (r, r), delta = (r, L r) of the
  // current r, beta = gamma/gamma_prev, eta = delta - beta^2 eta_prev, alpha =
  // gamma/eta, q = L r + beta q (= L p), r -= alpha q: one reduction per
  // iteration.  Neither p nor the solution is carried: at the end it is
  // (b - r) / L, component by component, whose residual is r exactly.
  //
  // What bounds an iteration: 4 dependent FP64 instructions per 128 components
  // of a CTA (64 cycles each), the words' trip, and the integer chains before
  // and after it.  The scalar warp turns the words into alpha and beta while
  // the others form L r, and hands them beta (for q) before alpha.
  const int nw = min(PM_W, (t.per + 31) >> 5);  // warps with components
  int it = 0, rd = 0;  // iterations, rounds
  int E[2] = {E0, E0 + 3};
  if (scalar) {
    // Even lanes work on (r, r) and what follows from it, odd lanes on
    // (r, L r), in the same instructions.
    const bool odd = lane & 1;
    PmF rrinv{0, 0}, g{0, 0};  // 1/gamma and eta/gamma^2 of the last iteration
    for (;;) {
      const int par = rd & 1;
      const unsigned tag = ((rd >> 1) + 1) & 3u;
      // this lane's share of the words, and whether one is out of range
      unsigned long long sg = 0, sd = 0;
      bool out = false, late = false;
      constexpr int Q = CLUSTER ? PM_CLUSTER * PM_W / 32 : PM_MAX_BLOCKS / 32;
      const int words_here = CLUSTER ? nb * nw : nb;
      ulonglong2 w[Q];
      bool have[Q];
      ulonglong2* const slot = words + par * nb;
#pragma unroll
      for (int k = 0; k < Q; k++) {
        have[k] = lane + 32 * k >= words_here;
        w[k] = make_ulonglong2(0, 0);
      }
      if (!CLUSTER) {
        // the sum of the warps' values: (r, r) in even lanes, (r, L r) in odd
        pm_bar_sync(1);
        uint3 l = make_uint3(0, 0, 0);
#pragma unroll
        for (int k = 0; k < PM_W; k++) {
          const uint4 v = s_sum[odd][k];
          l.x += v.x;
          l.y += v.y;
          l.z += v.z;
        }
        const unsigned long long S = pm_units(l);
        if (lane < 2) pm_store(slot + me, lane, (S << 2) | tag);
        const long long c0 = clock64();
        while (clock64() - c0 < PM_DELAY) {
        }
      }
      for (long long spins = 0;;) {
        bool all = true;
#pragma unroll
        for (int k = 0; k < Q; k++) {
          if (!have[k]) {
            if (CLUSTER) {
              const int i = lane + 32 * k, c = i / nw;
              const unsigned long long* const p = s_word + (par * 2 * PM_CLUSTER + c) * PM_W + i - c * nw;
              w[k] = make_ulonglong2(pm_load_cta(p), pm_load_cta(p + PM_CLUSTER * PM_W));
            } else {
              w[k] = pm_load(slot + lane + 32 * k);
            }
          }
        }
#pragma unroll
        for (int k = 0; k < Q; k++) {
          have[k] = have[k] || (((unsigned)w[k].x & 3u) == tag && ((unsigned)w[k].y & 3u) == tag);
          all &= have[k];
        }
        if (__all_sync(0xffffffffu, all)) break;
        if (++spins >= spin) {
          late = true;
          break;
        }
      }
#pragma unroll
      for (int k = 0; k < Q; k++) {
        sg += w[k].x >> 2;
        sd += w[k].y >> 2;
        out |= (w[k].x | w[k].y) >> 63;
      }
      unsigned lg[3], ld[3];
#pragma unroll
      for (int k = 0; k < 3; k++) {
        lg[k] = __reduce_add_sync(0xffffffffu, (unsigned)(sg >> (22 * k)) & (k < 2 ? (1u << 22) - 1 : ~0u));
        ld[k] = __reduce_add_sync(0xffffffffu, (unsigned)(sd >> (22 * k)) & (k < 2 ? (1u << 22) - 1 : ~0u));
      }
      out = __any_sync(0xffffffffu, out) || lg[2] >> 17 || ld[2] >> 17;
      const PmF gam = pmf_from(lg[0] + ((unsigned long long)lg[1] << 22) + ((unsigned long long)lg[2] << 44), E[0] + PM_SCALE);
      const PmF del = pmf_from(ld[0] + ((unsigned long long)ld[1] << 22) + ((unsigned long long)ld[2] << 44), E[1] + PM_SCALE);
      // their exponents; where nothing of them shows, lower ones to look at
      const int eg = gam.m ? gam.e + 63 + 1023 : E[0] - PM_NARROW, ed = del.m ? del.e + 63 + 1023 : E[1] - PM_NARROW;
      // below 2^56 units, a quarter of the anchor (from the limb, beside the chain to beta)
      const bool faint = (lg[2] < 1u << 12 && E[0] > 0) || (ld[2] < 1u << 12 && E[1] > 0);
      const bool again = !late && (out ? E[0] < 4096 : faint);
      const bool nan = out && !again;
      // beta = gamma/gamma_prev (even lanes), gamma^2 (odd lanes)
      const PmF p1 = pmf_mul(gam, odd ? gam : rrinv);
      if (lane == 0) {
        s_beta[par] = it == 0 ? 0.0 : pmf_double(p1, false);
        s_again[par] = again;
        if (again) {
          s_E[par][0] = out ? E[0] + PM_WIDEN : eg;
          s_E[par][1] = out ? E[1] + PM_WIDEN : ed;
        }
      }
      __syncwarp();
      pm_bar_arrive(2);
      if (again) {
        E[0] = out ? E[0] + PM_WIDEN : eg;
        E[1] = out ? E[1] + PM_WIDEN : ed;
        rd++;
        continue;
      }
      // odd lanes: eta = delta - gamma^2 g, 1/eta, alpha = gamma/eta; even
      // lanes: 1/gamma, 1/gamma^2
      bool neg = false;
      PmF eta = del;
      if (it > 0) eta = pmf_sub(del, pmf_mul(p1, g), neg);
      const PmF inv = pmf_recip(odd ? eta : gam);
      const PmF p2 = pmf_mul(odd ? gam : inv, inv);
      const bool done =
          late || nan || it >= maxit || xs_bits(pmf_double(gam, false)) < a.tol_bits;  // sqrt(r.r) < tol
      if (lane == 1) {
        s_alpha[par] = eta.m ? pmf_double(p2, neg) : xs_double(0x7FF8000000000000ull);
        s_E[par][0] = eg;
        s_E[par][1] = ed;
        s_done[par] = done;
        if (done) {
          s_ok = !late;
          s_nan = nan;
          s_it = nan ? maxit : it;
          if (late) atomicOr(a.flags, FLAG_TIMEOUT);
        }
      }
      __syncwarp();
      pm_bar_arrive(3);
      if (done) break;
      // for the next iteration, in every lane
      rrinv.m = __shfl_sync(0xffffffffu, inv.m, 0);
      rrinv.e = __shfl_sync(0xffffffffu, inv.e, 0);
      eta.m = __shfl_sync(0xffffffffu, eta.m, 1);
      eta.e = __shfl_sync(0xffffffffu, eta.e, 1);
      PmF i2;
      i2.m = __shfl_sync(0xffffffffu, p2.m, 0);
      i2.e = __shfl_sync(0xffffffffu, p2.e, 0);
      g = pmf_mul(eta, i2);
      E[0] = eg;
      E[1] = ed;
      it++;
      rd++;
    }
  } else {
    unsigned remote = 0;
    if (CLUSTER) {
      const unsigned own = (unsigned)__cvta_generic_to_shared(
          s_word + ((lane & 1) * PM_CLUSTER + me) * PM_W + wid);
      asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(own), "r"(min(lane >> 1, nb - 1)));
    }
    bool again = true;
    for (;;) {
      const int par = rd & 1;
      PmSum s0, s1;
      const double al = again ? 0.0 : s_alpha[par ^ 1];
#pragma unroll
      for (int j = 0; j < NPT; j++) {
        if (wid * 32 + PM_T * j < t.per) {
          if (!again) r[j] = fma(-al, q[j], r[j]);
          pm_terms(s0, s1, r[j], L[j], E[0], E[1]);
        }
      }
      const uint3 l0 = pm_warp_sum<NPT>(s0), l1 = pm_warp_sum<NPT>(s1);
      const uint3 l = lane & 1 ? l1 : l0;
      if (CLUSTER) {
        if (wid < nw && lane < 2 * nb)
          pm_store_cluster(remote + par * 2 * PM_CLUSTER * PM_W * 8, (pm_units(l) << 2) | (((rd >> 1) + 1) & 3u));
      } else {
        if (lane < 2) s_sum[lane][wid] = make_uint4(l.x, l.y, l.z, 0);
        __syncwarp();
        pm_bar_arrive(1);
      }
#pragma unroll
      for (int j = 0; j < NPT; j++)
        if (wid * 32 + PM_T * j < t.per) w[j] = L[j] * r[j];
      pm_bar_sync(2);
      again = s_again[par];
      if (!again) {
        const double be = s_beta[par];
#pragma unroll
        for (int j = 0; j < NPT; j++)
          if (wid * 32 + PM_T * j < t.per) q[j] = fma(be, q[j], w[j]);
        pm_bar_sync(3);
        if (s_done[par]) break;
      }
      E[0] = s_E[par][0];
      E[1] = s_E[par][1];
      rd++;
    }
  }
  __syncthreads();
  it = s_it;
  if (CLUSTER) {
    // all CTAs of the cluster leave together (words may still be arriving)
    if (!s_ok) atomicOr(a.flags, FLAG_TIMEOUT);
  } else if (!s_ok) {
    return;
  }

  // the solution of (-L) phi = b, each lattice component in its proportion of b
#pragma unroll
  for (int j = 0; j < NPT; j++) {
    int ca, cc;
    const bool own = component(j, ca, cc);
    if (own) {
      const double bt = norm_of(ca, cc);
      const double f = s_nan ? xs_double(0x7FF8000000000000ull) : bt != 0 ? -((bt - r[j]) / L[j]) / bt : 0.0;
      pm_orbit(t, ca, cc, [&](int k) { Bh[k] = f * __ldcg(&Bh[k]); });
    } else if (periodic && me == 0 && threadIdx.x == 0 && j == 0) {
      Bh[0] = 0.0;  // component (0, 0) is the first
    }
  }
  if (!barrier()) return;
  pm_lines(
      t.r, C, gtab, sm, [&](int l, int j) { return __ldcg(&Bh[l * R + j]); },
      [&](int l, int k, double v) { T1[k * C + l] = v; });
  if (!barrier()) return;
  // phi, with the extensions' duplicated nodes and zero walls
  const int nx = a.g.nx, ny = a.g.ny;
  pm_lines(
      t.c, R, gtab, sm, [&](int l, int j) { return __ldcg(&T1[l * C + j]); },
      [&](int l, int k, double v) {
        const int at = lattice_node(lat, l, k);
        a.phi[at] = v;
        if (lat.mode == EPIC_POISSON_DIRICHLET) return;
        if (k == 0) a.phi[at + C] = v;
        if (periodic && l == 0) {
          a.phi[at + (nx - 1) * ny] = v;
          if (k == 0) a.phi[at + (nx - 1) * ny + C] = v;
        }
      });
  if (lat.mode == EPIC_POISSON_DIRICHLET_X)
    for (int j = me * PM_ALL + threadIdx.x; j < ny; j += nb * PM_ALL) a.phi[j] = a.phi[(nx - 1) * ny + j] = 0.0;
  if (!barrier()) return;

  // domain.error = |A x - b| / n (src/field.cpp:258-259), n = nx ny: each
  // thread's sum in FP64 with what its additions round off beside it, the
  // threads' sums added exactly
  double e2 = 0, rest = 0;
  for (int m = me * PM_ALL + threadIdx.x; m < n; m += nb * PM_ALL) {
    const int row = m / C, col = m - row * C;
    const int up = lattice_wrap(row - 1, R, lat.wrap_r), dn = lattice_wrap(row + 1, R, lat.wrap_r);
    const int lf = lattice_wrap(col - 1, C, lat.wrap_c), rt = lattice_wrap(col + 1, C, lat.wrap_c);
    double sum = 0;
    if (up >= 0) sum += __ldcg(&a.phi[lattice_node(lat, up, col)]);
    if (lf >= 0) sum += __ldcg(&a.phi[lattice_node(lat, row, lf)]);
    sum = fma(-4.0, __ldcg(&a.phi[lattice_node(lat, row, col)]), sum);
    if (rt >= 0) sum += __ldcg(&a.phi[lattice_node(lat, row, rt)]);
    if (dn >= 0) sum += __ldcg(&a.phi[lattice_node(lat, dn, col)]);
    const double e = sum - (rhs(row, col) - bmean);
    const double sq = e * e, t = e2 + sq, z = t - e2;
    rest += (e2 - (t - z)) + (sq - z);
    e2 = t;
  }
  emax = xs_exponent(e2);
  if (emax == 2047) rest = 0;  // infinite or NaN already
  emax = (int)__reduce_max_sync(0xffffffffu, (unsigned)emax);
  if (lane == 0) s_e[wid] = emax;
  __syncthreads();
  emax = 0;
  for (int k = 0; k <= PM_W; k++) emax = max(emax, s_e[k]);
  const xs_int ev = xs_warp_sum(xs_from_double(e2, emax) + xs_from_double(rest, emax));
  if (lane == 0) {
    s_v[wid][0] = (unsigned long long)(xs_uint)ev;
    s_v[wid][1] = (unsigned long long)((xs_uint)ev >> 64);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    xs_uint tot = 0;
    for (int k = 0; k <= PM_W; k++) tot += ((xs_uint)s_v[k][1] << 64) | s_v[k][0];
    PmPartial o;
    o.lo = (unsigned long long)tot;
    o.hi = (long long)(tot >> 64);
    o.a = emax;
    o.pad = 0;
    parts[me] = o;
  }
  if (!barrier()) return;
  if (me == 0 && wid == 0) {
    int am = 0;
    for (int k = lane; k < nb; k += 32) am = max(am, (int)__ldcg(&parts[k].a));
    am = (int)__reduce_max_sync(0xffffffffu, (unsigned)am);
    xs_int tot = 0;
    for (int k = lane; k < nb; k += 32)
      tot += xs_realign((xs_int)(((xs_uint)(unsigned long long)__ldcg(&parts[k].hi) << 64) | __ldcg(&parts[k].lo)),
                        (int)__ldcg(&parts[k].a), am);
    tot = xs_warp_sum(tot);
    if (lane == 0) {
      const double err = xs_to_double(tot, am);
      a.info->iterations = it;
      a.info->converged = it < maxit;
      a.info->error = sqrt(err) / (nx * ny);
      atomicAdd(a.iter_total, (unsigned long long)it);
    }
  }
}

constexpr int PM_SMEM_MAX = 72 * 1024;  // of a side of PM_MAX_SIDE

static PmDir pm_dir(int n, int wrap) {
  PmDir d;
  d.n = n;
  d.sine = !wrap;
  d.M = wrap ? n : 2 * (n + 1);
  d.ntab = 2 * (wrap ? n : n + 1);
  d.tab = d.eig = 0;
  d.np = wrap ? n / 2 + 1 : (n + 1) / 2;
  d.scale = wrap ? 1.0 / std::sqrt((double)n) : std::sqrt(2.0 / (n + 1));
  return d;
}

// The plan for at most max_blocks CTAs; false when the lattice is too large
// (the global-memory k_pcg then runs).
static bool pm_plan(const Lattice& l, int max_blocks, PcgModes* out) {
  PcgModes t;
  const int R = l.R, C = l.C;
  if (R < 1 || C < 1 || R > PM_MAX_SIDE || C > PM_MAX_SIDE) return false;
  t.nA = l.wrap_r ? R / 2 + 1 : R;
  t.nC = l.wrap_c ? C / 2 + 1 : C;
  t.swap = R == C && l.wrap_r == l.wrap_c;
  t.N = t.swap ? t.nA * (t.nA + 1) / 2 : t.nA * t.nC;
  // One cluster while 16 CTAs hold the components in two rounds of their FP64
  // pipes (128 components a round): its words travel in a quarter of the
  // time.  Beyond, the rounds cost more than that, and the transforms want
  // every SM.  A cluster takes as many CTAs as give one round each.
  t.cluster = t.N <= 2 * 128 * PM_CLUSTER;
  if (t.cluster) t.B = t.N <= 256 ? 1 : std::min(PM_CLUSTER, (t.N + 127) / 128);
  else t.B = std::min(std::min(max_blocks, PM_MAX_BLOCKS), (t.N + 63) / 64);
  if (t.B < 1 || (t.cluster && t.B > max_blocks)) t.B = std::max(1, max_blocks);
  t.per = (t.N + t.B - 1) / t.B;
  if (t.cluster && t.per > PM_T) t.cluster = 0;
  if (t.per > PM_T * PM_MAX_NPT) return false;
  t.r = pm_dir(R, l.wrap_r);
  t.c = pm_dir(C, l.wrap_c);
  t.r.tab = 0;
  t.r.eig = t.r.ntab;
  if (t.swap) {
    t.c.tab = t.r.tab;
    t.c.eig = t.r.eig;
    t.ntab = t.r.ntab + R;
  } else {
    t.c.tab = t.r.ntab + R;
    t.c.eig = t.c.tab + t.c.ntab;
    t.ntab = t.c.eig + C;
  }
  t.tab_in_work = t.ntab > PM_TAB_MAX;
  if (t.tab_in_work && t.ntab > R * C) return false;
  auto smem = [](const PmDir& d) { return d.ntab + (PM_T / d.np + 2) * 2 * (d.n / 2 + 2); };
  t.smem = (int)sizeof(double) * std::max(smem(t.r), smem(t.c));
  if (t.smem > PM_SMEM_MAX) return false;
  *out = t;
  return true;
}

// (the attribute is set for every launch: cluster_fits)
template <int NPT>
static bool pm_launch(cudaStream_t st, const SolverArgs& a, const PcgModes& t) {
  const void* kern = (const void*)k_pcg_modes<NPT, false>;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, PM_SMEM_MAX);
  SolverArgs args = a;
  PcgModes plan = t;
  void* params[] = {&args, &plan};
  return launched(cudaLaunchCooperativeKernel(kern, dim3(t.B), dim3(PM_ALL), params, t.smem, st));
}

// False if the device cannot co-schedule the cluster.
static bool pm_launch_cluster(cudaStream_t st, const SolverArgs& a, const PcgModes& t) {
  if (!cluster_fits((const void*)k_pcg_modes<1, true>, t.B, PM_ALL, PM_SMEM_MAX, PM_SMEM_MAX)) return false;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = t.B;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(t.B);
  cfg.blockDim = dim3(PM_ALL);
  cfg.dynamicSmemBytes = t.smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return launched(cudaLaunchKernelEx(&cfg, k_pcg_modes<1, true>, a, t));
}

// Launches the solve (bar[0..1] zeroed on the stream before it); false where
// the lattice is too large for it.
bool launch_pcg_modes(cudaStream_t st, const SolverArgs& a, int max_blocks) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  max_blocks = std::min(max_blocks, sms);  // one CTA per SM: all resident
  PcgModes t;
  if (!pm_plan(make_lattice(a.g.nx, a.g.ny, a.poisson_bc), max_blocks, &t)) return false;
  SolverArgs m = a;
  m.tol_bits = xs_bits(xs_sqrt_threshold(a.tol));
  if (t.cluster && pm_launch_cluster(st, m, t)) return true;
  const int npt = (t.per + PM_T - 1) / PM_T;
  if (npt <= 1) return pm_launch<1>(st, m, t);
  if (npt <= 2) return pm_launch<2>(st, m, t);
  if (npt <= 4) return pm_launch<4>(st, m, t);
  if (npt <= 8) return pm_launch<8>(st, m, t);
  return pm_launch<16>(st, m, t);
}

}  // namespace epic
