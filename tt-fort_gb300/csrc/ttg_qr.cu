// Householder QR of tall blocks over many SMs, LAPACK reflector convention
// (dgeqrf + dorgqr: dqr, matrix_util.f90:37-61; zgeqrf + zungqr: zqr, :64-90;
// beta = -sign(re alpha) ||x||, a column that is already zero below its
// diagonal keeps it: tau = 0).
//
// GB300 has two FP64 FMAs per clock on each SM, so a factorisation in one CTA
// is bound by one SM's FP64 pipe.  Here the rows are dealt out cyclically over
// G CTAs and stay in their shared memory for the whole call.  Per column there
// is one reduction: every CTA applies the reflector to its rows and, in the
// same pass, forms its part of the next column's products with all later
// columns (the reflector needs only these and one row: v^H a = a_c +
// conj(scale) x^H a), so the G parts are exchanged once per column.  Q is then
// formed in place from the last reflector to the first, NB of them per exchange:
// the products of a panel's reflectors with each other and with Q's columns
// are enough to apply them one after the other (w_k = tau_k (v_k^H q - sum_{l>k}
// v_k^H v_l w_l), q -= sum_k v_k w_k).  One reflector per exchange took as
// long as the factorisation: 1240 us in all for 5248 x 86, 407 for 844 x 41,
// 329 for 128 x 64; now 835, 246, 272, three quarters of it the factorisation.
//
//   cluster form  G <= 8 CTAs of one cluster exchange through distributed
//                 shared memory, one cluster barrier per column (2.2k clocks,
//                 and 1.9k for the reflector's root and quotients);
//   grid form     clusters of 8 over the whole GPU (cooperative launch): parts
//                 are added within a cluster, and the clusters' sums, a share
//                 of the columns per CTA, go through global memory as tagged
//                 words (ttg_words.cuh); where few columns are left every CTA's
//                 part does.  One trip through L2 per column; handing all parts
//                 to one CTA and its sum back took two (10.2k clocks of a step
//                 of 5248 x 86, so 8.8k).  A cluster whose wait ran out fills
//                 its rows of Q and R with NaN, and tau.
// Both add the parts in a fixed order, so results are bit-reproducible.
#include "ttg_common.cuh"
#include "ttg_words.cuh"
#include <algorithm>
#include <array>
#include <cstdint>

namespace ttg {
namespace qr {

template <class T> struct C;
template <> struct C<double> {
  static __device__ __forceinline__ double zero() { return 0.0; }
  static __device__ __forceinline__ double one() { return 1.0; }
  static __device__ __forceinline__ double nan() { return __longlong_as_double(0x7ff8000000000000ll); }
  static __device__ __forceinline__ double conj(double a) { return a; }
  static __device__ __forceinline__ double neg(double a) { return -a; }
  static __device__ __forceinline__ double mul(double a, double b) { return a * b; }
  static __device__ __forceinline__ double add(double a, double b) { return a + b; }
  static __device__ __forceinline__ double fma(double a, double b, double c) { return ::fma(a, b, c); }
  static __device__ __forceinline__ bool is_zero(double a) { return a == 0.0; }
  static __device__ __forceinline__ double shfl(double v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
  // reflector of (alpha, ||x||^2): beta, tau, scale of x (0 0 for none)
  static __device__ __forceinline__ void reflect(double alpha, double x2, double& beta, double& tau,
                                                 double& sc) {
    if (x2 == 0.0) {
      beta = alpha; tau = 0.0; sc = 0.0;
      return;
    }
    const double t = ::fma(alpha, alpha, x2);
    const double nrm = sqrt(t);
    beta = alpha >= 0 ? -nrm : nrm;
    tau = (beta - alpha) / beta;
    sc = 1.0 / (alpha - beta);
  }
  static __device__ __forceinline__ double sq(double s) { return s; }
};
template <> struct C<double2> {
  static __device__ __forceinline__ double2 zero() { return make_double2(0.0, 0.0); }
  static __device__ __forceinline__ double2 one() { return make_double2(1.0, 0.0); }
  static __device__ __forceinline__ double2 nan() {
    const double q = __longlong_as_double(0x7ff8000000000000ll);
    return make_double2(q, q);
  }
  static __device__ __forceinline__ double2 conj(double2 a) { return make_double2(a.x, -a.y); }
  static __device__ __forceinline__ double2 neg(double2 a) { return make_double2(-a.x, -a.y); }
  static __device__ __forceinline__ double2 mul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
  }
  static __device__ __forceinline__ double2 add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
  static __device__ __forceinline__ double2 fma(double2 a, double2 b, double2 c) {
    c.x = ::fma(a.x, b.x, c.x);
    c.x = ::fma(-a.y, b.y, c.x);
    c.y = ::fma(a.x, b.y, c.y);
    c.y = ::fma(a.y, b.x, c.y);
    return c;
  }
  static __device__ __forceinline__ bool is_zero(double2 a) { return a.x == 0.0 && a.y == 0.0; }
  static __device__ __forceinline__ double2 shfl(double2 v, int o) {
    v.x = __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y = __shfl_xor_sync(0xffffffffu, v.y, o);
    return v;
  }
  static __device__ __forceinline__ void reflect(double2 alpha, double x2, double2& beta, double2& tau,
                                                 double2& sc) {
    if (x2 == 0.0 && alpha.y == 0.0) {
      beta = alpha; tau = zero(); sc = zero();
      return;
    }
    const double t = ::fma(alpha.x, alpha.x, ::fma(alpha.y, alpha.y, x2));
    const double nrm = sqrt(t);
    const double b = alpha.x >= 0 ? -nrm : nrm;
    beta = make_double2(b, 0.0);
    tau = make_double2((b - alpha.x) / b, -alpha.y / b);
    const double2 d = make_double2(alpha.x - b, alpha.y);
    const double q = d.x * d.x + d.y * d.y;
    sc = make_double2(d.x / q, -d.y / q);
  }
  static __device__ __forceinline__ double sq(double2 s) { return s.x; }
};

constexpr int NT = 256;
constexpr int NCMAX = 40;            // clusters of the grid form, at most
constexpr int GMAX = 152;            // its CTAs, at most
// the grid form sends every CTA's part where a CTA adds at most FLAT columns and
// columns times clusters stay within FLATW (844 x 41 on 8 clusters: 268 -> 248
// us; without the second limit 5248 x 86 on 14 clusters 834 -> 840, with it 830)
constexpr int FLAT = 16, FLATW = 512;

constexpr int NB = 8;                // reflectors per exchange in forming Q, at most
constexpr int FT = NB;               // threads per column in forming Q

// values of one exchange: a factorisation step's m columns; nb products of
// each of up to r columns of Q and of the panel's nb columns with themselves
__host__ __device__ inline size_t xchg_elems(int n, int m, int nb) {
  const size_t r = n < m ? n : m, q = nb > 1 ? (r + nb) * nb : r;
  return nb > 0 && q > (size_t)m ? q : (size_t)m;
}
// elements of T in shared memory: rows, reflectors (of a panel of nb; nb = 0:
// no Q to form), next ones, sums, row of the current column, tau, this CTA's
// parts (twice in the cluster form's factorisation, with its row)
__host__ __device__ inline size_t part_elems(int n, int m, bool grid, int nb) {
  const size_t E = xchg_elems(n, m, nb);
  return grid || E > 2 * (size_t)m ? E : 2 * (size_t)m;
}
// the sums (of the grid form's factorisation for two exchanges)
__host__ __device__ inline size_t sum_elems(int n, int m, bool grid, int nb) {
  const size_t E = xchg_elems(n, m, nb);
  return !grid || E > 2 * (size_t)m ? E : 2 * (size_t)m;
}
__host__ __device__ inline size_t smem_elems(int n, int m, int G, bool grid, int nb) {
  const size_t chunk = (size_t)(n + G - 1) / G, ld = chunk | 1;
  const int r = n < m ? n : m;
  return ld * m + 2 * chunk * (nb > 1 ? nb : 1) + sum_elems(n, m, grid, nb) + m + r +
         part_elems(n, m, grid, nb) + (grid ? 0 : 2 * (size_t)m);
}
// 64-bit words of the grid form in global memory: the clusters' parts, the
// current row and the CTAs' parts of the last columns, each for exchanges of
// even and of odd number
template <class T> inline size_t grid_words(int n, int m, int clusters, int nb) {
  return 2 * ((size_t)clusters * xchg_elems(n, m, nb) + (size_t)m + (size_t)GMAX * FLAT * kMaxCluster) *
         words::count<T>;
}

template <class T, bool GRID>
__global__ void __launch_bounds__(NT) qr_rows_kernel(int n, int m, T* __restrict__ Ag,
                                                     T* __restrict__ R, T* __restrict__ taug, int G,
                                                     int CL, int lgt, int nb, unsigned long long* part,
                                                     unsigned int* bar) {
  using O = C<T>;
  namespace cgr = cooperative_groups;
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ T s_beta, s_tau, s_sc;
  __shared__ int s_fail[2];                             // of odd and even exchanges
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int b = blockIdx.x, r = min(n, m);
  cgr::cluster_group cl = cgr::this_cluster();
  constexpr int W = words::count<T>;
  const int chunk = (n + G - 1) / G, ld = chunk | 1;
  const int nloc = b < n ? (n - b + G - 1) / G : 0;     // rows b, b + G, ...
  T* A = reinterpret_cast<T*>(dyn);
  const size_t E = xchg_elems(n, m, nb);
  T* vb = A + (size_t)ld * m;
  T* xb = vb + (size_t)chunk * (nb > 1 ? nb : 1);
  T* S = xb + (size_t)chunk * (nb > 1 ? nb : 1);
  T* row = S + sum_elems(n, m, GRID, nb);
  T* tau = row + m;
  T* mine = tau + r;                                    // this CTA's parts
  T* mine_row = mine + part_elems(n, m, GRID, nb);      // cluster form: [2][m]
  unsigned long long* rowg = part + 2 * (size_t)(G / CL) * E * W;   // grid form: [2][m]
  unsigned long long* flat = rowg + 2 * (size_t)m * W;              // [2][G][FLAT CL]
  const int tpc = 1 << lgt, sub = tid & (tpc - 1), grp = tid >> lgt, ngrp = NT >> lgt;
  int par = 0;
  unsigned int epoch = 1;
  bool fail = false;
  if (tid < 2) s_fail[tid] = 0;
  // A grid that did not come as clusters of CL (a profiler that starts a
  // cooperative launch by itself can lose them) must not go on: the layout of
  // the words and the shared-memory ranks follow CL
  if ((int)cl.num_blocks() != CL || (int)gridDim.x != G) {
    for (int c = warp; c < m; c += NT / 32)
      for (int i = lane; i < nloc; i += 32) {
        const int gi = b + G * i;
        Ag[(i64)n * c + gi] = O::nan();
        if (R && gi < r) R[gi + (i64)r * c] = O::nan();
      }
    if (b == 0)
      for (int c = tid; c < r; c += NT) taug[c] = O::nan();
    return;
  }

  for (int c = warp; c < m; c += NT / 32)
    for (int i = lane; i < nloc; i += 32) A[(size_t)ld * c + i] = Ag[(i64)n * c + b + (i64)G * i];
  cl.sync();                                             // every peer runs from here on

  auto got = [&](const unsigned long long* w, unsigned long long (&x)[W], T& v) {
    if (words::take<T>(w, x, v, epoch, bar)) return true;
    for (int q = 0; q < CL; ++q) *cl.map_shared_rank(&s_fail[epoch & 1], q) = 1;
    return false;
  };
  auto publish = [&](int j, T s) { mine[j] = s; };
  auto publish_row = [&](int j, T v) {
    if (GRID) words::put(rowg + ((size_t)par * m + j) * W, v, epoch);
    else mine_row[(size_t)par * m + j] = v;
  };
  // grid form, few columns left: the CTAs' parts go to global memory as they are
  auto is_flat = [&](int j0) { return GRID && (m - j0) * (G / CL) <= FLATW && m - j0 <= FLAT * CL; };
  auto publish_col = [&](int j0, int j, T s) {
    if (is_flat(j0))
      words::put(flat + (((size_t)(epoch & 1) * G + b) * (FLAT * CL) + (j - j0)) * W, s, epoch);
    else
      mine[GRID ? j : par * m + j] = s;
  };
  // sum of the cluster's parts of value j, requested together
  auto cluster_sum = [&](size_t j) {
    T x[kMaxCluster];
#pragma unroll
    for (int q = 0; q < kMaxCluster; ++q)
      if (q < CL) x[q] = cl.map_shared_rank(mine, q)[j];
    T t = x[0];
#pragma unroll
    for (int q = 1; q < kMaxCluster; ++q)
      if (q < CL) t = O::add(t, x[q]);
    return t;
  };
  // the parts published for values [j0, j1) and (with_row) the row beside them:
  // sums to S, row to row.
  // For the factorisation (with_row) warp 0 goes straight on to the reflector
  // of column j0, whose sum its first lane holds: a square root and two
  // quotients, 1.9k clocks of a small block's 4.7k per column
  auto exchange = [&](int j0, int j1, int owner, bool with_row) {
    T* Sx = S + (GRID && with_row && (epoch & 1) ? m : 0);
    if constexpr (GRID) {
      // each CTA of a cluster takes a share of the values: adds the cluster's
      // parts, hands the sum to the same share of every cluster, adds theirs
      // and leaves the result with its cluster
      constexpr int LV = 8, QL = (NCMAX + LV - 1) / LV;  // lanes per value, parts per lane
      const int rank = (int)cl.block_rank(), cid = b / CL, nc = G / CL;
      const int per = (j1 - j0 + CL - 1) / CL, s0 = j0 + rank * per, s1 = min(j1, s0 + per);
      unsigned long long* pb = part + (size_t)(epoch & 1) * nc * E * W;
      unsigned long long y[W];
      if (with_row && j0 + tid < j1) words::load<T>(rowg + ((size_t)par * m + j0 + tid) * W, y);
      if (with_row && is_flat(j0)) {
        // at most FLAT values per CTA: one hop, every part read directly (peers
        // may still read the sums of the exchange before: they alternate)
        constexpr int LF = NT / FLAT, QF = (GMAX + LF - 1) / LF;
        __syncthreads();
        const int j = s0 + tid / LF, l = tid % LF;
        const unsigned long long* pf =
            flat + ((size_t)(epoch & 1) * G * (FLAT * CL) + (j - j0)) * W;
        unsigned long long x[QF][W];
#pragma unroll
        for (int k = 0; k < QF; ++k)
          if (j < s1 && l + LF * k < G) words::load<T>(pf + (size_t)(l + LF * k) * (FLAT * CL) * W, x[k]);
        T t = O::zero();
#pragma unroll
        for (int k = 0; k < QF; ++k) {
          T v;
          if (j < s1 && l + LF * k < G && got(pf + (size_t)(l + LF * k) * (FLAT * CL) * W, x[k], v))
            t = O::add(t, v);
        }
        __syncwarp();
#pragma unroll
        for (int o = 1; o < LF; o <<= 1) t = O::add(t, O::shfl(t, o));
        if (j < s1 && l < CL) cl.map_shared_rank(Sx, l)[j] = t;
      } else {
        cl.sync();
        for (int j = s0 + tid; j < s1; j += NT) words::put(pb + ((size_t)cid * E + j) * W, cluster_sum(j), epoch);
        for (int jb = s0; jb < s1; jb += NT / LV) {
          const int j = jb + tid / LV, l = tid % LV;
          unsigned long long x[QL][W];
#pragma unroll
          for (int k = 0; k < QL; ++k)
            if (j < s1 && l + LV * k < nc) words::load<T>(pb + ((size_t)(l + LV * k) * E + j) * W, x[k]);
          T t = O::zero();
#pragma unroll
          for (int k = 0; k < QL; ++k) {
            T v;
            if (j < s1 && l + LV * k < nc && got(pb + ((size_t)(l + LV * k) * E + j) * W, x[k], v)) t = O::add(t, v);
          }
          __syncwarp();
#pragma unroll
          for (int o = 1; o < LV; o <<= 1) t = O::add(t, O::shfl(t, o));
          if (j < s1 && l < CL) cl.map_shared_rank(Sx, l)[j] = t;
        }
      }
      if (with_row)
        for (int j = j0 + tid; j < j1; j += NT) {
          T v;
          if (j != j0 + tid) words::load<T>(rowg + ((size_t)par * m + j) * W, y);
          if (got(rowg + ((size_t)par * m + j) * W, y, v)) row[j] = v;
        }
      cl.sync();
    } else {
      cl.sync();
      for (int j = j0 + tid; j < j1; j += NT) {
        S[j] = cluster_sum(j + (size_t)par * m);
        if (with_row) row[j] = cl.map_shared_rank(mine_row, owner)[(size_t)par * m + j];
      }
    }
    if (with_row && warp == NT / 32 - 1) {
      // the quotients on two partitions of the SM (in the cluster form this warp,
      // seldom with a column of its own, adds column j0 once more: 128 x 64 284 ->
      // 272 us)
      T be, ta, sc;
      if (GRID) O::reflect(row[j0], O::sq(Sx[j0]), be, ta, sc);
      else O::reflect(cl.map_shared_rank(mine_row, owner)[(size_t)par * m + j0],
                      O::sq(cluster_sum(j0 + (size_t)par * m)), be, ta, sc);
      if (lane == 0) s_sc = sc;
    }
    if (with_row && warp == 0) {
      __syncwarp();
      T be, ta, sc;
      O::reflect(row[j0], O::sq(Sx[j0]), be, ta, sc);
      if (lane == 0) {
        s_beta = be;
        s_tau = ta;
        tau[j0] = ta;
      }
    }
    fail = GRID && s_fail[epoch & 1] != 0;          // one answer in a cluster: set before its barrier
    par ^= 1;
    ++epoch;
    __syncthreads();
  };
  // the same for the nb products per column in forming Q: in the cluster form
  // each CTA adds a share of them and hands it to all
  auto exchange_q = [&](int cnt) {
    if constexpr (GRID) {
      exchange(0, cnt, 0, false);
    } else {
      cl.sync();
      const int per = (cnt + G - 1) / G;
      for (int j = b * per + tid; j < min(cnt, (b + 1) * per); j += NT) {
        const T t = cluster_sum(j);
#pragma unroll
        for (int q = 0; q < kMaxCluster; ++q)
          if (q < G) cl.map_shared_rank(S, q)[j] = t;
      }
      cl.sync();
    }
  };
  auto group_sum = [&](T s) {
    for (int o = 1; o < tpc; o <<= 1) s = O::add(s, O::shfl(s, o));
    return s;
  };

  // products of column 0 (below row 0) with all columns
  for (int i = tid; i < nloc; i += NT) xb[i] = b + G * i > 0 ? A[i] : O::zero();
  __syncthreads();
  for (int jb = 0; jb < m; jb += ngrp) {
    const int j = jb + grp;
    T s = O::zero();
    if (j < m) {
      const T* a = A + (size_t)ld * j;
      for (int i = sub; i < nloc; i += tpc) s = O::fma(O::conj(xb[i]), a[i], s);
    }
    s = group_sum(s);
    if (sub == 0 && j < m) {
      publish_col(0, j, s);
      if (b == 0) publish_row(j, A[(size_t)ld * j]);
    }
  }
  exchange(0, m, 0, true);

  for (int c = 0; c < r && !fail; ++c) {
    const T be = s_beta, ta = s_tau, sc = s_sc;
    const bool on = !O::is_zero(ta);
    const T ctau = O::conj(ta), csc = O::conj(sc);
    // f_j = conj(tau) v^H a_j
    const T* Sc = S + (GRID && !(epoch & 1) ? m : 0);    // of the exchange just done
    auto coef = [&](int j) { return O::mul(ctau, O::fma(csc, Sc[j], row[j])); };
    const bool next = c + 1 < m;
    const int i0 = c > b ? (c - b + G - 1) / G : 0;     // first own row >= c
    {
      T* ac = A + (size_t)ld * c;
      T* an = ac + ld;
      const T fn = (on && next) ? O::neg(coef(c + 1)) : O::zero();
      for (int i = i0 + tid; i < nloc; i += NT) {
        const int gi = b + G * i;
        T v = O::zero();
        if (gi == c) {
          v = on ? O::one() : O::zero();
          ac[i] = be;
        } else if (on) {
          v = O::mul(ac[i], sc);
          ac[i] = v;
        }
        vb[i] = v;
        if (next) {
          const T x = O::fma(v, fn, an[i]);
          an[i] = x;
          xb[i] = gi > c + 1 ? x : O::zero();
        }
      }
    }
    __syncthreads();
    if (!next) break;
    const bool more = c + 1 < r;                         // another reflector follows
    for (int jb = c + 1; jb < m; jb += ngrp) {
      const int j = jb + grp;
      T s = O::zero();
      if (j < m) {
        T* a = A + (size_t)ld * j;
        const T f = (on && j > c + 1) ? O::neg(coef(j)) : O::zero();
        for (int i = i0 + sub; i < nloc; i += tpc) {
          T x = a[i];
          if (j > c + 1) {
            x = O::fma(vb[i], f, x);
            a[i] = x;
          }
          if (more) {
            s = O::fma(O::conj(xb[i]), x, s);
            if (b + G * i == c + 1) publish_row(j, x);
          }
        }
      }
      s = group_sum(s);
      if (more && sub == 0 && j < m) publish_col(c + 1, j, s);
    }
    if (!more) break;
    exchange(c + 1, m, (c + 1) % G, true);
  }
  __syncthreads();

  // R: rows 0..r-1, zero below the diagonal (R null: factor only, A keeps the
  // reflectors below R)
  for (int c = R ? warp : m; c < m; c += NT / 32)
    for (int i = lane; i < nloc; i += 32) {
      const int gi = b + G * i;
      if (gi < r) R[gi + (i64)r * c] = fail ? O::nan() : (gi <= c ? A[(size_t)ld * c + i] : O::zero());
    }
  if (b == 0)
    for (int c = tid; c < r; c += NT) taug[c] = fail ? O::nan() : tau[c];
  __syncthreads();

  // Q in place, a panel of nb reflectors at a time from the last: column c of a
  // panel becomes the product of its reflectors 0..c with e_c, later columns
  // that of all.  Exchanged values: nb to each column from the panel's first
  // on (v_k^H q; v_k's row c in the panel itself), then v_k^H v_l to each l.
  auto panel = [&](T* d, int j0, int w) {                // v_0 .. v_{w-1}, zero beyond
    for (int e = tid; e < nb * nloc; e += NT) {
      const int k = e / nloc, i = e - k * nloc, gi = b + G * i;
      T v = O::zero();
      if (k < w) v = gi > j0 + k ? A[(size_t)ld * (j0 + k) + i] : (gi == j0 + k ? O::one() : O::zero());
      d[k * chunk + i] = v;
    }
  };
  // applies panel [j0, j0 + w) in vb to columns from j0 on and leaves the
  // products of panel [jn, jn + nb) in xb (jn < 0: none); w = 0: products only
  auto pass = [&](int j0, int w, int jn, int wn) {
    const int first = jn >= 0 ? jn : j0, gcol = jn >= 0 && nb > 1 ? wn : 0;
    const int cnt = r - first + gcol;
    const int i0 = j0 > b ? (j0 - b + G - 1) / G : 0;
    const int in = jn > b ? (jn - b + G - 1) / G : 0;
    for (int ub = 0; ub < cnt; ub += NT / FT) {
      const int u = ub + tid / FT, c = first + u, sub = tid & (FT - 1);
      T s[NB];
#pragma unroll
      for (int k = 0; k < NB; ++k) s[k] = O::zero();
      if (u < cnt && c < r && c >= j0) {
        T* a = A + (size_t)ld * c;
        const bool own = c < j0 + w;                     // a column of the panel: starts as e_c
        const int kc = min(c - j0, w - 1);
        T f[NB];
#pragma unroll
        for (int k = 0; k < NB; ++k) f[k] = k <= kc ? S[(size_t)(c - j0) * nb + k] : O::zero();
        for (int i = (own ? 0 : i0) + sub; i < nloc; i += FT) {
          T x = own ? (b + G * i == c ? O::one() : O::zero()) : a[i];
#pragma unroll
          for (int k = 0; k < NB; ++k)
            if (k <= kc) x = O::fma(vb[k * chunk + i], f[k], x);
          a[i] = x;
          if (jn >= 0) {
#pragma unroll
            for (int k = 0; k < NB; ++k)
              if (k < nb) s[k] = O::fma(O::conj(xb[k * chunk + i]), x, s[k]);
          }
        }
      } else if (u < cnt && c < r) {                     // the next panel's own columns
        const int i = (c - b) / G;
        if (sub == 0 && c >= b && b + G * i == c) {
#pragma unroll
          for (int k = 0; k < NB; ++k)
            if (k < nb) s[k] = O::conj(xb[k * chunk + i]);
        }
      } else if (u < cnt) {
        const T* a = xb + (size_t)(c - r) * chunk;
        for (int i = in + sub; i < nloc; i += FT) {
#pragma unroll
          for (int k = 0; k < NB; ++k)
            if (k < c - r) s[k] = O::fma(O::conj(xb[k * chunk + i]), a[i], s[k]);
        }
      }
      if (jn >= 0) {
        // sums over the FT lanes by halving: lane k is left with that of v_k
#pragma unroll
        for (int o = NB / 2; o > 0; o >>= 1) {
          const bool up = (sub & o) != 0;
#pragma unroll
          for (int k = 0; k < o; ++k) s[k] = O::add(up ? s[k + o] : s[k], O::shfl(up ? s[k] : s[k + o], o));
        }
        if (sub < nb && u < cnt) publish(u * nb + sub, s[0]);
      }
    }
    if (jn >= 0) exchange_q(cnt * nb);
  };
  if constexpr (!GRID) cl.sync();                        // peers may still read this CTA's parts
  if (R && !fail) {
    int j0 = (r - 1) / nb * nb, w = r - j0;
    panel(xb, j0, w);
    __syncthreads();
    pass(r, 0, j0, w);
    while (!fail) {
      T* t = vb;
      vb = xb;
      xb = t;
      // S of column c becomes -w
      const T* g = S + (size_t)(r - j0) * nb;
      for (int c = j0 + tid; c < r; c += NT) {
        T* sc = S + (size_t)(c - j0) * nb;
        const int kc = min(c - j0, w - 1);
        T x[NB];
#pragma unroll
        for (int k = 0; k < NB; ++k) x[k] = k <= kc ? sc[k] : O::zero();
#pragma unroll
        for (int l = NB - 1; l >= 0; --l)
          if (l <= kc) {
            const T v = O::neg(O::mul(tau[j0 + l], x[l]));
            sc[l] = v;
#pragma unroll
            for (int k = 0; k < l; ++k) x[k] = O::fma(g[l * nb + k], v, x[k]);
          }
      }
      if (j0 > 0) panel(xb, j0 - nb, nb);
      __syncthreads();
      pass(j0, w, j0 > 0 ? j0 - nb : -1, nb);
      if (j0 == 0) break;
      j0 -= nb;
      w = nb;
    }
  }
  __syncthreads();
  for (int c = warp; c < m; c += NT / 32)
    for (int i = lane; i < nloc; i += 32)
      Ag[(i64)n * c + b + (i64)G * i] = fail ? O::nan() : A[(size_t)ld * c + i];
  cl.sync();                                             // peers may still read this CTA's parts
}

}  // namespace qr

namespace {
constexpr size_t kSmemMax = 220 * 1024;

// The form with the least estimated time (us): the busiest CTA's two FMAs per
// element and reflector at 3.2 per ns, and the latency of a step, r of them in
// the factorisation and one per panel in forming Q (one CTA 2.8 us, a cluster
// 3.0, nc clusters 4.2 + 0.12 nc).  Measured on GB300 over G (us; one CTA of
// the former kernel, then G = 8, 32, 64, 112; clusters of 4 took 875 us at
// G = 128 for the 5248 x 86 block, 2280 for 512 x 256):
//    128 x  64     895 |  272   288   334     -
//    320 x 128    4400 |  890   671   746   824
//    512 x 256   22407 | 3392  1856  1732  1846
//   1968 x  82    8776 | 2011   753   620   619
//   5248 x  86   25150 |    -  1466   994   829
//   2048 x 512  284916 |    -     -  8128  6783
//    256 x   8 complex   190 |  77    77    82    94
//    512 x  32 complex  2620 | 420   293   291   329
struct Pick { int G, CL; bool grid; int nb; };
// clusters of CL CTAs that the GPU holds at once (0: none, or not known)
template <class T> int max_clusters(int CL) {
  static const std::array<int, 3> held = [] {
    std::array<int, 3> h{0, 0, 0};
    if (cudaFuncSetAttribute(qr::qr_rows_kernel<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kSmemMax) != cudaSuccess)
      return h;
    for (int k = 0; k < 3; ++k) {
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute at;
      at.id = cudaLaunchAttributeClusterDimension;
      at.val.clusterDim.x = 2u << k;
      at.val.clusterDim.y = at.val.clusterDim.z = 1;
      cfg.gridDim = dim3(2u << k);
      cfg.blockDim = dim3(qr::NT);
      cfg.dynamicSmemBytes = kSmemMax;
      cfg.attrs = &at;
      cfg.numAttrs = 1;
      int c = 0;
      if (cudaOccupancyMaxActiveClusters(&c, qr::qr_rows_kernel<T, true>, &cfg) == cudaSuccess)
        h[k] = std::min(c, qr::NCMAX);
      else (void)cudaGetLastError();
    }
    return h;
  }();
  return held[CL == 8 ? 2 : (CL == 4 ? 1 : 0)];
}

template <class T>
Pick pick(int n, int m, bool form_q, size_t work) {
  using qr::NT;
  const double cx = sizeof(T) == 16 ? 4.0 : 1.0;
  const int r = std::min(n, m);
  // later columns of all columns, in the factorisation and in forming Q
  const double cols = (double)r * m - 0.5 * (double)r * r + (form_q ? 0.5 * (double)r * r : 0.0);
  Pick best{0, 0, false, 0};
  double bt = 1e300;
  auto try_form = [&](int CL, int nc) {
    const int G = CL * nc;
    const bool grid = nc > 1;
    if (G > 1 && n < 2 * G) return;
    if (grid && (nc > max_clusters<T>(CL) || G > qr::GMAX)) return;
    // the widest panel that fits
    int nb = form_q ? qr::NB : 0;
    auto fits = [&] {
      return qr::smem_elems(n, m, G, grid, nb) * sizeof(T) <= kSmemMax &&
             (!grid || (size_t)r + 32 + qr::grid_words<double>(n, m, nc, nb) <= work);
    };
    while (nb > 1 && !fits()) nb /= 2;
    if (!fits()) return;
    const double rows = (n + G - 1) / G;
    const double step = grid ? 4.2 + 0.12 * nc : (G == 1 ? 2.8 : 3.0);
    double t = 2.0 * cx * rows * cols / 3.2e3 + step * r + (nb ? (1.0 + 1.0 / nb) * step * r / nb : 0.0);
    // fewer columns than warps: 32 threads a column in the factorisation, FT in
    // forming Q, each a chain of dependent FMAs over its rows (25600 x 1 in one cluster
    // 107 us, over the GPU 61; 12000 x 2 171 and 58)
    if (m < NT / 32) t += rows * (0.004 * r + (nb ? 0.022 : 0.0)) * (sizeof(T) == 16 ? 2.0 : 1.0);
    if (t < bt) { bt = t; best = {G, CL, grid, nb}; }
  };
  for (int CL : {1, 2, 4, 8}) try_form(CL, 1);
  for (int nc = 2; nc <= qr::NCMAX; nc += 2) try_form(kMaxCluster, nc);
  return best;
}

template <class T>
bool run(int n, int m, T* A, T* R, T* tau, size_t work, cudaStream_t s) {
  const Pick p = pick<T>(n, m, R != nullptr, work);
  if (p.G == 0) return false;
  const int r = std::min(n, m);
  const size_t smem = qr::smem_elems(n, m, p.G, p.grid, p.nb) * sizeof(T);
  int G = p.G, nb = p.nb;
  // threads per column: about one column per group, two rows or more per lane
  const int chunk = (n + p.G - 1) / p.G;
  int lgt = 0;
  while (lgt < 5 && (qr::NT >> (lgt + 1)) >= m && chunk >= (4 << lgt)) ++lgt;
  if (p.grid) {
    unsigned long long* part = (unsigned long long*)(((uintptr_t)(tau + r) + 63) & ~(uintptr_t)63);
    const size_t words = qr::grid_words<T>(n, m, G / p.CL, nb);
    unsigned int* bar = (unsigned int*)(part + words);
    TTG_CUDA(cudaMemsetAsync(part, 0, words * 8 + 8, s));
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = p.CL;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeCooperative;
    at[1].val.cooperative = 1;
    cfg.gridDim = dim3(G);
    cfg.blockDim = dim3(qr::NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    TTG_CUDA(cudaLaunchKernelEx(&cfg, qr::qr_rows_kernel<T, true>, n, m, A, R, tau, G, p.CL, lgt, nb, part, bar));
    ++g_launches;
    return true;
  }
  static const cudaError_t rc = cudaFuncSetAttribute(
      qr::qr_rows_kernel<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
  TTG_CUDA(rc);
  launch_ex(qr::qr_rows_kernel<T, false>, dim3(p.G), dim3(qr::NT), dim3(p.G, 1, 1), false, smem, s, n,
            m, A, R, tau, G, G, lgt, nb, (unsigned long long*)nullptr, (unsigned int*)nullptr);
  return true;
}
}  // namespace

// Work of the grid form, in elements: tau, then two words' worth per value of
// parts, sums and rows; the failure flag.  For blocks of up to m columns (the rows
// that a sweep's have are not known):
size_t qr_work_elems(i64 n, i64 m, bool form_q) {
  return (size_t)std::min(n, m) + 32 + qr::grid_words<double>((int)n, (int)m, qr::NCMAX, form_q ? qr::NB : 0);
}
// and for one block, with Q: of the form that it takes (8 rows of a million columns
// take none of the grid's, whose words would be 1.3 GB)
size_t qr_call_elems(i64 n, i64 m, bool cplx) {
  const Pick p = cplx ? pick<double2>((int)n, (int)m, true, SIZE_MAX) : pick<double>((int)n, (int)m, true, SIZE_MAX);
  return (size_t)std::min(n, m) + 32 + (p.grid ? qr::grid_words<double>((int)n, (int)m, p.G / p.CL, p.nb) : 0);
}

bool qr_rows(int n, int m, double* A, double* R, double* tau, size_t work, cudaStream_t s) {
  return run<double>(n, m, A, R, tau, work, s);
}
bool qr_rows_factor(int n, int m, double* A, double* tau, size_t work, cudaStream_t s) {
  return run<double>(n, m, A, (double*)nullptr, tau, work, s);
}
bool qr_rows(int n, int m, double2* A, double2* R, double2* tau, size_t work, cudaStream_t s) {
  return run<double2>(n, m, A, R, tau, work, s);
}

}  // namespace ttg
