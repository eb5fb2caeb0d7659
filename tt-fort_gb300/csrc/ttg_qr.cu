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
// formed in place from the last reflector to the first in the same way.
//
//   cluster form  G <= 8 CTAs of one cluster exchange through distributed
//                 shared memory, one cluster barrier per column;
//   grid form     up to one CTA per SM (cooperative launch): parts go to
//                 global memory as tagged words (ttg_words.cuh), CTA j % G adds
//                 those of column j in CTA order and hands the sum to all (a
//                 step of the 5248 x 86 block took 7.8 us with two grid
//                 barriers, 7.0 so).  A CTA whose wait ran out fills its rows
//                 with NaN.
// Both add the parts in a fixed order, so results are bit-reproducible.
#include "ttg_common.cuh"
#include "ttg_words.cuh"
#include <algorithm>

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
  static __device__ __forceinline__ double ldcg(const double* p) { return __ldcg(p); }
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
  static __device__ __forceinline__ double2 ldcg(const double2* p) { return __ldcg(p); }
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
constexpr int GMAX = 152;            // CTAs of the grid form

// elements of T in shared memory: rows, reflector, next column, sums and row of
// the current column, tau, and (cluster form) this CTA's parts and row, twice
__host__ __device__ inline size_t smem_elems(int n, int m, int G, bool grid) {
  const size_t chunk = (size_t)(n + G - 1) / G, ld = chunk | 1;
  const int r = n < m ? n : m;
  return ld * m + 2 * chunk + 2 * (size_t)m + r + (grid ? 0 : 4 * (size_t)m);
}

template <class T, bool GRID>
__global__ void __launch_bounds__(NT) qr_rows_kernel(int n, int m, T* __restrict__ Ag,
                                                     T* __restrict__ R, T* __restrict__ taug, int G,
                                                     int lgt, unsigned long long* part,
                                                     unsigned int* bar) {
  using O = C<T>;
  namespace cgr = cooperative_groups;
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ T s_beta, s_tau, s_sc;
  __shared__ int s_fail;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int b = blockIdx.x, r = min(n, m);
  constexpr int W = words::count<T>;
  const int chunk = (n + G - 1) / G, ld = chunk | 1;
  const int nloc = b < n ? (n - b + G - 1) / G : 0;     // rows b, b + G, ...
  T* A = reinterpret_cast<T*>(dyn);
  T* vb = A + (size_t)ld * m;
  T* xb = vb + chunk;
  T* S = xb + chunk;
  T* row = S + m;
  T* tau = row + m;
  T* mine = tau + r;                                    // cluster form: [2][m] parts, [2][m] row
  unsigned long long* tot = part + (size_t)G * m * W;   // grid form: [m], then [2][m] row
  unsigned long long* rowg = tot + (size_t)m * W;
  const int tpc = 1 << lgt, sub = tid & (tpc - 1), grp = tid >> lgt, ngrp = NT >> lgt;
  int par = 0;
  unsigned int epoch = 1;
  bool fail = false;
  if (tid == 0) s_fail = 0;

  for (int c = warp; c < m; c += NT / 32)
    for (int i = lane; i < nloc; i += 32) A[(size_t)ld * c + i] = Ag[(i64)n * c + b + (i64)G * i];
  __syncthreads();

  auto got = [&](const unsigned long long* w, unsigned long long (&x)[W], T& v) {
    if (words::take<T>(w, x, v, epoch, bar)) return true;
    s_fail = 1;
    return false;
  };
  // the parts that publish() left for columns [j0, j1) and (with_row) the row
  // beside them: sums to S, row to row
  auto publish = [&](int j, T s) {
    if (GRID) words::put(part + ((size_t)b * m + j) * W, s, epoch);
    else mine[(size_t)par * m + j] = s;
  };
  auto publish_row = [&](int j, T v) {
    if (GRID) words::put(rowg + ((size_t)par * m + j) * W, v, epoch);
    else mine[(size_t)(2 + par) * m + j] = v;
  };
  // for the factorisation (with_row) warp 0 goes straight on to the reflector
  // of column j0, whose sum its first lane holds: a square root and two
  // quotients, 1.9k clocks of a small block's 4.7k per column
  auto exchange = [&](int j0, int j1, int owner, bool with_row) {
    if constexpr (GRID) {
      // CTA j % G adds column j, one warp each
      for (int j = j0 + ((b - j0) % G + G) % G + warp * G; j < j1; j += G * (NT / 32)) {
        // the lane's parts are requested together: one trip to L2, not five
        constexpr int QL = (GMAX + 31) / 32;
        unsigned long long x[QL][W];
#pragma unroll
        for (int k = 0; k < QL; ++k)
          if (lane + 32 * k < G) words::load<T>(part + ((size_t)(lane + 32 * k) * m + j) * W, x[k]);
        T t = O::zero();
#pragma unroll
        for (int k = 0; k < QL; ++k) {
          T v;
          if (lane + 32 * k < G && got(part + ((size_t)(lane + 32 * k) * m + j) * W, x[k], v))
            t = O::add(t, v);
        }
        __syncwarp();
        for (int o = 16; o > 0; o >>= 1) t = O::add(t, O::shfl(t, o));
        if (lane == 0) words::put(tot + (size_t)j * W, t, epoch);
      }
      for (int j = j0 + tid; j < j1; j += NT) {
        T v;
        unsigned long long x[W], y[W];
        words::load<T>(tot + (size_t)j * W, x);
        if (with_row) words::load<T>(rowg + ((size_t)par * m + j) * W, y);
        if (got(tot + (size_t)j * W, x, v)) S[j] = v;
        if (with_row && got(rowg + ((size_t)par * m + j) * W, y, v)) row[j] = v;
      }
    } else {
      cgr::cluster_group cl = cgr::this_cluster();
      cl.sync();
      for (int j = j0 + tid; j < j1; j += NT) {
        T t = O::zero();
        for (int q = 0; q < G; ++q) t = O::add(t, cl.map_shared_rank(mine, q)[(size_t)par * m + j]);
        S[j] = t;
        if (with_row) row[j] = cl.map_shared_rank(mine, owner)[(size_t)(2 + par) * m + j];
      }
    }
    if (with_row && warp == 0) {
      __syncwarp();
      T be, ta, sc;
      O::reflect(row[j0], O::sq(S[j0]), be, ta, sc);
      if (lane == 0) { s_beta = be; s_tau = ta; s_sc = sc; tau[j0] = ta; }
    }
    par ^= 1;
    ++epoch;
    __syncthreads();
    fail = GRID && s_fail != 0;
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
      publish(j, s);
      if (b == 0) publish_row(j, A[(size_t)ld * j]);
    }
  }
  exchange(0, m, 0, true);

  for (int c = 0; c < r && !fail; ++c) {
    const T be = s_beta, ta = s_tau, sc = s_sc;
    const bool on = !O::is_zero(ta);
    const T ctau = O::conj(ta), csc = O::conj(sc);
    // f_j = conj(tau) v^H a_j
    auto coef = [&](int j) { return O::mul(ctau, O::fma(csc, S[j], row[j])); };
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
      if (more && sub == 0 && j < m) publish(j, s);
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
    for (int c = tid; c < r; c += NT) taug[c] = tau[c];
  __syncthreads();

  // Q in place: columns r-1..0; column j becomes H_j e_j, later columns H_j q_c
  for (int j = R ? r - 1 : -1; j >= 0 && !fail; --j) {
    const T ta = tau[j];
    const int i0 = j > b ? (j - b + G - 1) / G : 0;
    T* aj = A + (size_t)ld * j;
    const T* ap = aj - ld;                               // the next reflector, column j - 1
    const T nt = O::neg(ta);
    for (int i = tid; i < nloc; i += NT) {
      const int gi = b + G * i;
      T v = O::zero(), q = O::zero();
      if (gi == j) {
        v = O::one();
        q = O::add(O::one(), nt);
      } else if (gi > j) {
        v = aj[i];
        q = O::mul(nt, v);
      }
      vb[i] = v;
      aj[i] = q;
      if (j > 0) xb[i] = gi > j - 1 ? ap[i] : O::zero();
    }
    __syncthreads();
    for (int cb = j; cb < r; cb += ngrp) {
      const int c = cb + grp;
      T s = O::zero();
      if (c < r) {
        T* a = A + (size_t)ld * c;
        const T f = c > j ? O::neg(O::mul(ta, S[c])) : O::zero();
        for (int i = i0 + sub; i < nloc; i += tpc) {
          T x = a[i];
          if (c > j) {
            x = O::fma(vb[i], f, x);
            a[i] = x;
          }
          if (j > 0) s = O::fma(O::conj(xb[i]), x, s);
        }
      }
      s = group_sum(s);
      if (j > 0 && sub == 0 && c < r) publish(c, s);
    }
    if (j > 0) exchange(j, r, 0, false);
  }
  __syncthreads();
  for (int c = warp; c < m; c += NT / 32)
    for (int i = lane; i < nloc; i += 32)
      Ag[(i64)n * c + b + (i64)G * i] = fail ? O::nan() : A[(size_t)ld * c + i];
  if constexpr (!GRID) cgr::this_cluster().sync();       // peers may still read this CTA's parts
}

}  // namespace qr

// work of the grid form, in elements: tau, then two words' worth per value of
// parts [G][m], sums [m], rows [2][m]; the failure flag
size_t qr_work_elems(i64 n, i64 m) {
  return (size_t)std::min(n, m) + 2 * (size_t)(qr::GMAX + 3) * m + 32;
}

namespace {
constexpr size_t kSmemMax = 220 * 1024;

template <class T> bool grid_ok(int n, int m, int G) {
  return qr::smem_elems(n, m, G, true) * sizeof(T) <= kSmemMax;
}

// The form with the least estimated time (us): the busiest CTA's two FMAs per
// element and reflector, at half the FP64 pipe's rate, and 2 r steps of
// latency (one CTA 2.0 us, a cluster 2.2, a grid 2.6 + 0.02 G).  Measured on
// GB300 over G (us; one CTA of the former kernel, then G = 8, 32, 76, 152):
//    128 x  64     895 |  329   477   609   785
//    512 x 256   22407 | 3904  2727  2950  3487
//   1968 x  82    8776 | 2481  1139  1009  1031
//   5248 x  86   25150 |    -  2146  1451  1467
//   2048 x 512  284916 |    -     -  9914  9624
//    256 x   8 complex   190 | 75  120   123   144
struct Pick { int G; bool grid; };
template <class T>
Pick pick(int n, int m, bool form_q, bool have_work) {
  const double cx = sizeof(T) == 16 ? 4.0 : 1.0;
  const int r = std::min(n, m);
  // later columns of all columns, in the factorisation and in forming Q
  const double cols = (double)r * m - 0.5 * (double)r * r + (form_q ? 0.5 * (double)r * r : 0.0);
  const double steps = (form_q ? 2.0 : 1.0) * r;
  auto est = [&](int G, bool grid) {
    const double rows = (n + G - 1) / G;
    return 2.0 * cx * rows * cols / 1.9e3 + (grid ? 2.6 + 0.02 * G : (G == 1 ? 2.0 : 2.2)) * steps;
  };
  Pick best{0, false};
  double bt = 1e300;
  for (int G : {1, 2, 4, 8}) {
    if (G > 1 && n < 2 * G) continue;
    if (qr::smem_elems(n, m, G, false) * sizeof(T) > kSmemMax) continue;
    const double t = est(G, false);
    if (t < bt) { bt = t; best = {G, false}; }
  }
  if (have_work)
    for (int G : {16, 32, 48, 76, 114, qr::GMAX}) {
      if (n < 2 * G || !grid_ok<T>(n, m, G)) continue;
      const double t = est(G, true);
      if (t < bt) { bt = t; best = {G, true}; }
    }
  return best;
}

template <class T>
bool run(int n, int m, T* A, T* R, T* tau, size_t work, cudaStream_t s) {
  const bool have = work >= qr_work_elems(n, m);
  Pick p = pick<T>(n, m, R != nullptr, have);
  if (p.G == 0) return false;
  const int r = std::min(n, m);
  const size_t smem = qr::smem_elems(n, m, p.G, p.grid) * sizeof(T);
  // threads per column: about one column per group, two rows or more per lane
  const int chunk = (n + p.G - 1) / p.G;
  int lgt = 0;
  while (lgt < 5 && (qr::NT >> (lgt + 1)) >= m && chunk >= (4 << lgt)) ++lgt;
  if (p.grid) {
    static const int coop = [] {
      int dev = 0, nsm = 0, per = 0;
      if (cudaFuncSetAttribute(qr::qr_rows_kernel<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kSmemMax) != cudaSuccess ||
          cudaGetDevice(&dev) != cudaSuccess ||
          cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
          cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, qr::qr_rows_kernel<T, true>, qr::NT,
                                                        kSmemMax) != cudaSuccess)
        return 0;
      return nsm * per;
    }();
    if (coop < p.G) return false;
    unsigned long long* part = (unsigned long long*)(((uintptr_t)(tau + r) + 63) & ~(uintptr_t)63);
    const size_t words = (size_t)(p.G + 3) * m * (sizeof(T) / 4);
    unsigned int* bar = (unsigned int*)(part + words);
    TTG_CUDA(cudaMemsetAsync(part, 0, words * 8 + 8, s));
    void* args[] = {&n, &m, &A, &R, &tau, &p.G, &lgt, &part, &bar};
    TTG_CUDA(cudaLaunchCooperativeKernel((const void*)qr::qr_rows_kernel<T, true>, dim3(p.G),
                                         dim3(qr::NT), args, smem, s));
    ++g_launches;
    return true;
  }
  static const cudaError_t rc = cudaFuncSetAttribute(
      qr::qr_rows_kernel<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
  TTG_CUDA(rc);
  launch_ex(qr::qr_rows_kernel<T, false>, dim3(p.G), dim3(qr::NT), dim3(p.G, 1, 1), false, smem, s, n,
            m, A, R, tau, p.G, lgt, (unsigned long long*)nullptr, (unsigned int*)nullptr);
  return true;
}
}  // namespace

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
