// AMEn linear solver (dtt_amen_solve, ttamen.f90:29-252) on the GPU, behind
// the flat-array entry point of tt_amen_solve (tt_adapt_als.f90:513).
//
// Every core, interface (X'AX, X'Y, Z'AX, Z'Y) and Krylov basis stays in
// HBM.  The sweep follows the reference step by step:
//   right-to-left: (z update), QR of x (and z) pushing R left, Phi updates
//   left-to-right: local rhs = Phi_XY y Phi_XY, residual, local solve
//     (dense LU below max_full_size, GMRES(40) x 2 otherwise), residual-based
//     SVD truncation (dtt_trunc), enrichment with the projected residual,
//     z update, QR of x and z to the right, Phi updates
//   stop when the largest local residual is below tol.
// Two GPU-shaped restatements keep the arithmetic but change the order:
//   * GMRES uses Arnoldi with classical Gram-Schmidt applied twice (the
//     reference applies Householder reflectors, ttlocsolve.f90:509-682);
//     both minimise the same residual over the same Krylov space;
//   * the truncation scan evaluates the candidate ranks from the top in
//     batches of 8 local matvecs and keeps the reference's rule: the chosen
//     rank is one more than the largest rank whose residual exceeds tol.
// The enrichment TT z starts from the splitmix64/Box-Muller stream shared
// with the oracle.
#include "ttg_davidson.cuh"
#include "ttg_words.cuh"
#include <algorithm>
#include <cmath>
#include <cstring>

namespace ttg {

void gemm_tn_small(int M, int N, i64 K, const double* A, i64 lda, const double* B, i64 ldb,
                   double* C, int ldc, double alpha, double beta, cudaStream_t s);
void gemm_nn_small(i64 R, int N, int K, const double* A, i64 lda, const double* B, int ldb,
                   double* C, i64 ldc, double alpha, double beta, cudaStream_t s);

namespace {

inline int eb(i64 n) { return (int)std::max<i64>(1, std::min<i64>(4096, (n + 255) / 256)); }

__global__ void axpy_kernel(i64 n, double a, const double* x, double* y) {
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x)
    y[i] = fma(a, x[i], y[i]);
}
// y = x - z
__global__ void sub_kernel(i64 n, const double* x, const double* z, double* y) {
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x)
    y[i] = x[i] - z[i];
}
__global__ void scal_kernel(i64 n, const double* sdev, int invert, double* x) {
  const double s = invert ? 1.0 / sdev[0] : sdev[0];
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x)
    x[i] *= s;
}
// out[j] = sum_i x[i + ld*j]^2, grid (bx, ncols); the bx CTAs of a column are
// one cluster and add their partials in rank order (deterministic)
__global__ void sqnorm_cols_kernel(i64 n, const double* x, i64 ld, double* out) {
  const int j = blockIdx.y;
  double acc = 0.0;
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
    const double v = x[i + ld * j];
    acc = fma(v, v, acc);
  }
  const double t = cluster_sum(acc);
  if (blockIdx.x == 0 && threadIdx.x == 0) out[j] = t;
}
void sqnorm_cols(i64 n, const double* x, i64 ld, int ncols, double* out, cudaStream_t s) {
  const int bx = (int)std::max<i64>(1, std::min<i64>(kMaxCluster, (n + 2047) / 2048));
  launch_clustered(sqnorm_cols_kernel, dim3(bx, ncols), dim3(256), dim3(bx, 1, 1), 0, s, n, x,
                   ld, out);
}
__global__ void sqrt_kernel(int n, double* x) {
  if (threadIdx.x < n) x[threadIdx.x] = sqrt(x[threadIdx.x]);
}
// Y (n x c) = X[:, j] - rhs for every column j (residuals of candidates)
__global__ void sub_cols_kernel(i64 n, int c, const double* X, const double* rhs, double* Y) {
  for (i64 e = blockIdx.x * (i64)blockDim.x + threadIdx.x; e < n * c; e += (i64)gridDim.x * blockDim.x)
    Y[e] = X[e] - rhs[e % n];
}

// dense solve B x = b (N <= 64), partial pivoting (dgesv), one CTA
__global__ void lu_solve_kernel(int N, double* B, double* x, int* info) {
  __shared__ int piv;
  __shared__ double pv;
  for (int k = 0; k < N; ++k) {
    if (threadIdx.x == 0) {
      int p = k;
      double best = fabs(B[k + N * k]);
      for (int i = k + 1; i < N; ++i) {
        double v = fabs(B[i + N * k]);
        if (v > best) { best = v; p = i; }
      }
      piv = p;
      pv = best;
      if (best == 0.0) info[0] = k + 1;
    }
    __syncthreads();
    if (pv == 0.0) return;
    const int p = piv;
    if (p != k) {
      for (int j = threadIdx.x; j < N; j += blockDim.x) {
        double t = B[k + N * j]; B[k + N * j] = B[p + N * j]; B[p + N * j] = t;
      }
      if (threadIdx.x == 0) { double t = x[k]; x[k] = x[p]; x[p] = t; }
    }
    __syncthreads();
    const double d = B[k + N * k];
    for (int i = k + 1 + threadIdx.x; i < N; i += blockDim.x) B[i + N * k] /= d;
    __syncthreads();
    for (int e = threadIdx.x; e < (N - k - 1) * (N - k - 1); e += blockDim.x) {
      const int i = k + 1 + e % (N - k - 1), j = k + 1 + e / (N - k - 1);
      B[i + N * j] -= B[i + N * k] * B[k + N * j];
    }
    if (threadIdx.x == 0)
      for (int i = k + 1; i < N; ++i) x[i] -= B[i + N * k] * x[k];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    for (int i = N - 1; i >= 0; --i) {
      double v = x[i];
      for (int j = i + 1; j < N; ++j) v -= B[i + N * j] * x[j];
      x[i] = v / B[i + N * i];
    }
  }
}

// One Arnoldi step after the matvec, over a resident grid: w = V[:, j+1] is made
// orthogonal to V[:, 0..j] by classical Gram-Schmidt applied twice and scaled to
// norm 1; h[0..j] the coefficients, h[j+1] the norm.  CTA b holds its rows of w
// in shared memory; V is read four times from L2.  The parts of the products
// are exchanged as tagged words (CTA c % G adds those of column c in CTA order),
// with them |w|^2 in the second pass: |w - V h2|^2 = |w|^2 - |h2|^2 as long as
// the second pass takes off less than a tenth, else the norm is summed afresh.
// Bound by its two exchanges (about 9 us) and 4 N (j + 1) FMAs; the nine
// launches it replaces took about 65 us more a step (AMEn solve of the d = 4,
// n = 24 grid, 3400 steps of up to 24 * 82 * 28 unknowns: 412 -> 187 ms).
constexpr int AR_NT = 256, AR_G = 152, AR_SLOTS = 64, AR_CHUNK = 8192;
constexpr size_t AR_WORDS = 2 * (size_t)(AR_G + 1) * AR_SLOTS + 8;   // 64-bit words of an exchange area
__global__ void __launch_bounds__(AR_NT) arnoldi_kernel(i64 N, int j, int chunk, double* __restrict__ V,
                                                        double* __restrict__ h,
                                                        unsigned long long* part, unsigned int epoch) {
  extern __shared__ double w[];                          // [chunk]
  __shared__ double seg_s[8][AR_SLOTS];
  __shared__ double tot_s[AR_SLOTS], h_s[AR_SLOTS];
  __shared__ int fail;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, G = gridDim.x, b = blockIdx.x;
  const i64 lo = (i64)b * chunk;
  const int n = (int)max((i64)0, min((i64)chunk, N - lo));
  unsigned long long* tot = part + (size_t)G * AR_SLOTS * 2;
  unsigned int* flag = (unsigned int*)(part + 2 * (size_t)(AR_G + 1) * AR_SLOTS);
  const double* Vb = V + lo;
  double* wg = V + N * (j + 1) + lo;
  if (tid == 0) fail = 0;
  for (int i = tid; i < n; i += AR_NT) w[i] = wg[i];
  __syncthreads();
  // tot_s[c] = V_c . w for c < nc, then w . w when ww
  auto products = [&](int nc, bool ww) {
    const int C = nc + (ww ? 1 : 0), nseg = C >= 8 ? 1 : 8 / C;
    for (int t = warp; t < C * nseg; t += AR_NT / 32) {
      const int c = t % C, sg = t / C, i1 = (int)((i64)n * (sg + 1) / nseg);
      const double* v = Vb + N * c;
      double a0 = 0.0, a1 = 0.0;
      int i = (int)((i64)n * sg / nseg) + lane;
      if (c < nc) {
        for (; i + 96 < i1; i += 128) {
          const double x0 = v[i], x1 = v[i + 32], x2 = v[i + 64], x3 = v[i + 96];
          a0 = fma(x0, w[i], a0);
          a1 = fma(x1, w[i + 32], a1);
          a0 = fma(x2, w[i + 64], a0);
          a1 = fma(x3, w[i + 96], a1);
        }
        for (; i < i1; i += 32) a0 = fma(v[i], w[i], a0);
      } else {
        for (; i < i1; i += 32) a0 = fma(w[i], w[i], a0);
      }
      a0 += a1;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) a0 += __shfl_xor_sync(0xffffffffu, a0, o);
      if (lane == 0) seg_s[sg][c] = a0;
    }
    __syncthreads();
    if (tid < C) {
      double t = 0.0;
      for (int sg = 0; sg < nseg; ++sg) t += seg_s[sg][tid];
      if (G == 1) tot_s[tid] = t;
      else words::put(part + ((size_t)b * AR_SLOTS + tid) * 2, t, epoch);
    }
    if (G > 1) {
      for (int c = b + warp * G; c < C; c += G * (AR_NT / 32)) {
        constexpr int QL = (AR_G + 31) / 32;
        unsigned long long x[QL][2];
#pragma unroll
        for (int k = 0; k < QL; ++k)
          if (lane + 32 * k < G) words::load<double>(part + ((size_t)(lane + 32 * k) * AR_SLOTS + c) * 2, x[k]);
        double t = 0.0;
#pragma unroll
        for (int k = 0; k < QL; ++k) {
          double v;
          if (lane + 32 * k < G) {
            // (a part that did not come: NaN to every CTA, or the others would take the
            // sum of the rest)
            if (words::take<double>(part + ((size_t)(lane + 32 * k) * AR_SLOTS + c) * 2, x[k], v, epoch, flag)) t += v;
            else t = __longlong_as_double(0x7ff8000000000000ll);
          }
        }
        __syncwarp();
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) words::put(tot + (size_t)c * 2, t, epoch);
      }
      if (tid < C) {
        unsigned long long x[2];
        double v = 0.0;
        words::load<double>(tot + (size_t)tid * 2, x);
        if (!words::take<double>(tot + (size_t)tid * 2, x, v, epoch, flag)) fail = 1;
        tot_s[tid] = v;
      }
    }
    ++epoch;
    __syncthreads();
  };
  // w -= V[:, 0..j] tot_s
  auto subtract = [&]() {
    for (int i = tid; i < n; i += AR_NT) {
      double a0 = w[i], a1 = 0.0;
      int c = 0;
      for (; c + 8 <= j + 1; c += 8) {
        double x[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) x[u] = Vb[N * (c + u) + i];
#pragma unroll
        for (int u = 0; u < 8; u += 2) {
          a0 = fma(-x[u], tot_s[c + u], a0);
          a1 = fma(-x[u + 1], tot_s[c + u + 1], a1);
        }
      }
      for (; c <= j; ++c) a0 = fma(-Vb[N * c + i], tot_s[c], a0);
      w[i] = a0 + a1;
    }
    __syncthreads();
  };
  products(j + 1, false);
  if (tid <= j) h_s[tid] = tot_s[tid];
  subtract();
  products(j + 1, true);
  double h2 = 0.0;
  if (warp == 0) {
    for (int c = lane; c <= j; c += 32) h2 = fma(tot_s[c], tot_s[c], h2);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) h2 += __shfl_xor_sync(0xffffffffu, h2, o);
    if (lane == 0) {
      const double ww = tot_s[j + 1];
      h_s[AR_SLOTS - 1] = h2 <= 0.1 * ww ? ww - h2 : -1.0;   // NaN: summed afresh
    }
  }
  if (tid <= j) h_s[tid] += tot_s[tid];
  subtract();
  double n2 = h_s[AR_SLOTS - 1];                             // the same value in every CTA
  if (!(n2 >= 0.0)) {
    products(0, true);
    n2 = tot_s[0];
  }
  if (tid == 0) seg_s[0][0] = sqrt(n2);
  __syncthreads();
  const double nrm = fail ? __longlong_as_double(0x7ff8000000000000ll) : seg_s[0][0];
  const double sc = 1.0 / nrm;
  for (int i = tid; i < n; i += AR_NT) wg[i] = w[i] * sc;
  if (b == 0) {
    if (tid <= j) h[tid] = h_s[tid];
    if (tid == j + 1) h[tid] = nrm;
  }
}

// core_{k+1} with rho zero rows appended: out ((r+rho) x p) from in (r x p)
__global__ void pad_rows_kernel(i64 r, i64 rho, i64 p, const double* in, double* out) {
  const i64 R = r + rho;
  for (i64 e = blockIdx.x * (i64)blockDim.x + threadIdx.x; e < R * p; e += (i64)gridDim.x * blockDim.x) {
    const i64 i = e % R, c = e / R;
    out[e] = i < r ? in[i + r * c] : 0.0;
  }
}

// the identity block of ort0 for wide matrices: m x m identity
__global__ void eye_kernel(i64 m, double* out) {
  for (i64 e = blockIdx.x * (i64)blockDim.x + threadIdx.x; e < m * m; e += (i64)gridDim.x * blockDim.x)
    out[e] = (e % m == e / m) ? 1.0 : 0.0;
}

}  // namespace

// splitmix64 uniform in (0, 1] and standard normal (Box-Muller), the stream
// the oracle uses for the enrichment TT z
static inline double sm_uniform(unsigned long long k) {
  unsigned long long z = k * 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z = z ^ (z >> 31);
  return ((double)(z >> 11) + 1.0) * 0x1.0p-53;
}
void sm_normals(unsigned long long seed, i64 count, double* out) {
  for (i64 i = 0; i < count; ++i) {
    const double u1 = sm_uniform(seed * 1000003ull + 2 * (unsigned long long)i + 1);
    const double u2 = sm_uniform(seed * 1000003ull + 2 * (unsigned long long)i + 2);
    out[i] = std::sqrt(-2.0 * std::log(u1)) * std::cos(2.0 * 3.141592653589793 * u2);
  }
}


// ---------------------------------------------------------------------------
// the solver
// ---------------------------------------------------------------------------
namespace {

struct DevTT {
  std::vector<i64> n, r, cap;
  std::vector<double*> c;
  i64 size(int k) const { return r[k] * n[k] * r[k + 1]; }
};

struct Arena {
  char* base = nullptr;
  size_t top = 0, capb = 0;
  ~Arena() { if (base) cudaFree(base); }
  void alloc(size_t b) {
    if (cudaMalloc(&base, b) != cudaSuccess) {
      base = nullptr;
      throw Error{TTG_ERR_NOMEM, "amen: device allocation failed"};
    }
    capb = b;
  }
  double* take(size_t count) {
    size_t b = (count * sizeof(double) + 255) & ~size_t(255);
    if (top + b > capb) throw Error{TTG_ERR_NOMEM, "amen: device arena exhausted"};
    double* p = (double*)(base + top);
    top += b;
    return p;
  }
};

inline size_t al8(size_t count) { return (count * sizeof(double) + 255) & ~size_t(255); }

// device buffers of one GMRES: V (N x (nr+1)), w (N), gm (4096 doubles:
// Hessenberg columns, Ritz coefficients), red (64), h (pinned host, >= 1024
// doubles), words (AR_WORDS 64-bit words: the Arnoldi steps' exchanges)
struct GmresBufs {
  double *V, *w, *gm, *red, *h;
  unsigned long long* words;
};

// GMRES(nr) x iters for L x = b (x0 = 0) with Arnoldi by classical
// Gram-Schmidt applied twice; stops when |residual| / |b| < tol (the
// Householder GMRES of the reference minimises the same residual over the
// same Krylov space, ttlocsolve.f90:509-682, tt_linalg.f90:651-845).
// Returns whether the residual reached tol (false: stopped after iters
// restarts, which the reference tolerates).  The Hessenberg columns come to the
// host four steps at a time, which applies their Givens rotations and solves
// for the coefficients (serial work on at most 61 numbers: a CUDA thread took
// 10 us a column and 50 us a solve for it).
template <class MV>
bool gmres_cgs2(const MV& mv, i64 N, const double* b, double* x, double tol, int nr, int iters,
                const GmresBufs& G, cudaStream_t s) {
  double* H = G.gm;                    // four Hessenberg columns of AR_SLOTS
  double* y = G.gm + 4 * AR_SLOTS;
  double* V = G.V;
  double* red = G.red;
  double* h = G.h;                     // pinned: scalars, then Hessenberg columns, then y
  double* hH = h + 16;
  double* hy = hH + 4 * AR_SLOTS;
  std::vector<double> R((size_t)(nr + 1) * nr), cs(nr), sn(nr), g(nr + 1);
  auto sync = [&]() { TTG_CUDA(cudaStreamSynchronize(s)); };
  static const int coop = [] {
    int dev = 0, nsm = 0, per = 0;
    if (cudaFuncSetAttribute(arnoldi_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             AR_CHUNK * (int)sizeof(double)) != cudaSuccess ||
        cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, arnoldi_kernel, AR_NT,
                                                      AR_CHUNK * sizeof(double)) != cudaSuccess)
      return 0;
    return nsm * per;
  }();
  // CTAs: at least 128 rows each, at most one per SM and AR_CHUNK rows (larger
  // problems take the separate products)
  const int ctas = (int)std::max<i64>(1, std::min<i64>(std::min(AR_G, coop), (N + 127) / 128));
  int chunk = (int)std::min<i64>((N + ctas - 1) / ctas, AR_CHUNK + 1);
  const bool fused = coop > 0 && chunk <= AR_CHUNK;
  unsigned int epoch = 1;
  if (fused) TTG_CUDA(cudaMemsetAsync(G.words, 0, AR_WORDS * sizeof(unsigned long long), s));
  auto arnoldi = [&](int j, double* hcol) {
    double* wv = V + N * (j + 1);
    if (fused) {
      i64 NN = N;
      int jj = j;
      double *vv = V, *hh = hcol;
      unsigned long long* ww = G.words;
      void* args[] = {&NN, &jj, &chunk, &vv, &hh, &ww, &epoch};
      TTG_CUDA(cudaLaunchCooperativeKernel((const void*)arnoldi_kernel, dim3(ctas), dim3(AR_NT), args,
                                           (size_t)chunk * sizeof(double), s));
      ++g_launches;
      epoch += 3;
      return;
    }
    double* h2 = G.gm + 5 * AR_SLOTS;
    gemm_tn_small(j + 1, 1, N, V, N, wv, N, hcol, j + 2, 1.0, 0.0, s);
    gemm_nn_small(N, 1, j + 1, V, N, hcol, j + 2, wv, N, -1.0, 1.0, s);
    gemm_tn_small(j + 1, 1, N, V, N, wv, N, h2, j + 2, 1.0, 0.0, s);
    gemm_nn_small(N, 1, j + 1, V, N, h2, j + 2, wv, N, -1.0, 1.0, s);
    axpy_kernel<<<1, 64, 0, s>>>(j + 1, 1.0, h2, hcol);
    TTG_CHECK_LAUNCH();
    sqnorm_cols(N, wv, N, 1, red, s);
    sqrt_kernel<<<1, 32, 0, s>>>(1, red);
    TTG_CHECK_LAUNCH();
    TTG_CUDA(cudaMemcpyAsync(hcol + j + 1, red, sizeof(double), cudaMemcpyDeviceToDevice, s));
    scal_kernel<<<eb(N), 256, 0, s>>>(N, red, 1, wv);
    TTG_CHECK_LAUNCH();
  };
  TTG_CUDA(cudaMemsetAsync(x, 0, sizeof(double) * N, s));
  double nrmb = -1.0, curres = 1.0;
  for (int it = 0; it < iters; ++it) {
    // w = b - L x
    mv(x, G.w, 1);
    sub_kernel<<<eb(N), 256, 0, s>>>(N, b, G.w, G.w);
    TTG_CHECK_LAUNCH();
    sqnorm_cols(N, G.w, N, 1, red, s);
    TTG_CUDA(cudaMemcpyAsync(h, red, sizeof(double), cudaMemcpyDeviceToHost, s));
    sync();
    const double beta = std::sqrt(h[0]);
    if (it == 0) nrmb = beta;
    if (beta == 0.0) return true;
    TTG_CUDA(cudaMemcpyAsync(V, G.w, sizeof(double) * N, cudaMemcpyDeviceToDevice, s));
    h[1] = 1.0 / beta;
    TTG_CUDA(cudaMemcpyAsync(red + 8, h + 1, sizeof(double), cudaMemcpyHostToDevice, s));
    scal_kernel<<<eb(N), 256, 0, s>>>(N, red + 8, 0, V);
    TTG_CHECK_LAUNCH();
    std::fill(g.begin(), g.end(), 0.0);
    g[0] = beta;
    int jdone = 0;
    for (int j = 0; j < nr; ++j) {
      mv(V + N * j, V + N * (j + 1), 1);
      arnoldi(j, H + AR_SLOTS * (j & 3));
      jdone = j + 1;
      // the Hessenberg columns are read back every 4th step (and at the
      // last): a host synchronisation per step would bound the solve by
      // latency.  The first step below tol ends the cycle exactly as a
      // per-step test would: the Givens-reduced R and g of steps 0..j are
      // final after step j, so the extra steps only cost their matvecs.
      if (jdone % 4 == 0 || jdone == nr) {
        const int j0 = ((jdone - 1) / 4) * 4;
        TTG_CUDA(cudaMemcpyAsync(hH, H, sizeof(double) * AR_SLOTS * (jdone - j0),
                                 cudaMemcpyDeviceToHost, s));
        sync();
        bool conv = false;
        for (int q = j0; q < jdone && !conv; ++q) {
          // previous rotations, a new one, g
          double* c = hH + AR_SLOTS * (q - j0);
          for (int i = 0; i < q; ++i) {
            const double a = c[i], e = c[i + 1];
            c[i] = cs[i] * a + sn[i] * e;
            c[i + 1] = -sn[i] * a + cs[i] * e;
          }
          const double a = c[q], e = c[q + 1], den = std::hypot(a, e);
          cs[q] = den > 0 ? a / den : 1.0;
          sn[q] = den > 0 ? e / den : 0.0;
          c[q] = den;
          g[q + 1] = -sn[q] * g[q];
          g[q] = cs[q] * g[q];
          for (int i = 0; i <= q; ++i) R[i + (size_t)(nr + 1) * q] = c[i];
          curres = std::fabs(g[q + 1]) / nrmb;
          if (curres < tol) { jdone = q + 1; conv = true; }
        }
        if (conv) break;
      }
    }
    for (int i = jdone - 1; i >= 0; --i) {
      double v = g[i];
      for (int k = i + 1; k < jdone; ++k) v -= R[i + (size_t)(nr + 1) * k] * hy[k];
      hy[i] = v / R[i + (size_t)(nr + 1) * i];
    }
    // hy is rewritten only after a later synchronisation
    TTG_CUDA(cudaMemcpyAsync(y, hy, sizeof(double) * jdone, cudaMemcpyHostToDevice, s));
    gemm_nn_small(N, 1, jdone, V, N, y, jdone, x, N, 1.0, 1.0, s);
    if (curres < tol) return true;
  }
  return false;
}

// a local solve that stopped at its iteration cap: counted, or an error when
// the context asks for strict caps
void note_capped(ttg_ctx* ctx, const char* who) {
  ++ctx->stat_capped;
  if (ctx->strict)
    throw Error{TTG_ERR_NOCONV, std::string(who) +
                                    ": local GMRES reached its restart cap before its tolerance"};
}

}  // namespace


struct AmenParams {
  int d;
  std::vector<i64> n, ra, ry, rx;
  const double *crA, *crY, *crX0;
  double tol;
  i64 rmax;
  int kick, nswp, local_iters, local_restart, max_full_size, verb;
  unsigned long long seed;
  int method = TTG_METHOD_PLAIN;
};

struct AmenOut {
  std::vector<double> cores;
  std::vector<i64> rx;
  int sweeps = 0;
  double res_max = 0.0;
  long long matvecs = 0;
};

class AmenSolver {
 public:
  AmenSolver(ttg_ctx* ctx, const AmenParams& P) : P_(P), s_(ctx->stream), ctx_(ctx) {
    ctx->stat_capped = 0;
  }
  void run(AmenOut& out);

 private:
  AmenParams P_;
  cudaStream_t s_;
  ttg_ctx* ctx_;
  Arena mem_;
  DevTT x_, y_, z_;
  std::vector<double*> A_;
  std::vector<double*> pxax_, pxy_, pzax_, pzy_;
  size_t tau_n_ = 0;   // elements of tau_
  unsigned long long* words_ = nullptr;   // exchanges of the Arnoldi steps
  double *tmpA_, *tmpB_, *tmpC_, *R_, *tau_, *rhs_, *resid_, *sol_, *xnew_, *scr_, *svU_, *svS_,
      *svVt_, *svScr_, *cand_, *candY_, *red_, *V_, *w_, *gm_, *dense_;
  double* h_ = nullptr;   // pinned
  long long nmv_ = 0;
  double real_tol_ = 0.0;
  static constexpr int kBatch = 8;

  void sync() { TTG_CUDA(cudaStreamSynchronize(s_)); }
  LocalDims dims(const DevTT& xx, const DevTT& yy, int k) const {
    return LocalDims{xx.r[k], xx.n[k], xx.r[k + 1], yy.r[k], yy.n[k], yy.r[k + 1], P_.ra[k], P_.ra[k + 1]};
  }
  double norm2(const double* v, i64 n) {
    sqnorm_cols(n, v, n, 1, red_, s_);
    TTG_CUDA(cudaMemcpyAsync(h_, red_, sizeof(double), cudaMemcpyDeviceToHost, s_));
    sync();
    return std::sqrt(h_[0]);
  }
  void gemm(int M, int N, int K, const double* A, i64 sAm, i64 sAk, const double* B, i64 sBk,
            i64 sBn, double* C, i64 sCm, i64 sCn, double alpha = 1.0, double beta = 0.0) {
    GemmF64 g;
    g.M = M; g.N = N; g.K = K;
    g.A = A; g.sAm = sAm; g.sAk = sAk;
    g.B = B; g.sBk = sBk; g.sBn = sBn;
    g.C = C; g.sCm = sCm; g.sCn = sCn;
    g.alpha = alpha; g.beta = beta;
    gemm_f64(g, s_);
  }
  void qr(DevTT& t, int k, int dir);
  void yax(double* phi_new, const double* phi_old, const DevTT& yy, const DevTT& xx, int k, int dir,
           bool withA);
  // out (a.r[k] n x b.r[k+1]) = phi_l (a.r[k] x y.r[k]) y_k phi_r (y.r[k+1] x b.r[k+1])
  void project_y(const double* pl, const double* pr, i64 rl, i64 rr, int k, double* out);
  void local_mv(const LocalDims& L, const double* p1, const double* p2, int k, const double* x,
                double* yv, int nvec) {
    bfun3_f64(L, p1, A_[k], p2, x, yv, nvec, scr_, s_);
    nmv_ += nvec;
  }
  void gmres(const LocalDims& L, int k, const double* b, double* x, double tol);
  void gmres_split(const LocalDims& L, int k, const double* b, double* x, double tol);
  void* split_mem_ = nullptr;
  size_t split_bytes_ = 0;
  double *ir_r_ = nullptr, *ir_d_ = nullptr;
  long long split_mv_ = 0;
  void trunc(int k, double tol, const double* rhs, double rhs_norm);
};

void AmenSolver::qr(DevTT& t, int k, int dir) {
  auto& n = t.n;
  auto& r = t.r;
  if (dir > 0) {
    const i64 m = r[k] * n[k], rr = r[k + 1], p = n[k + 1] * r[k + 2];
    if (m >= rr) {
      TTG_CUDA(cudaMemcpyAsync(tmpA_, t.c[k], sizeof(double) * m * rr, cudaMemcpyDeviceToDevice, s_));
      qr_householder((int)m, (int)rr, tmpA_, R_, tau_, tau_n_, s_);
      TTG_CUDA(cudaMemcpyAsync(t.c[k], tmpA_, sizeof(double) * m * rr, cudaMemcpyDeviceToDevice, s_));
      gemm((int)rr, (int)p, (int)rr, R_, 1, rr, t.c[k + 1], 1, rr, tmpB_, 1, rr);
      TTG_CUDA(cudaMemcpyAsync(t.c[k + 1], tmpB_, sizeof(double) * rr * p, cudaMemcpyDeviceToDevice, s_));
    } else {
      // ort0 of a wide block: identity core, the block moves right
      gemm((int)m, (int)p, (int)rr, t.c[k], 1, m, t.c[k + 1], 1, rr, tmpB_, 1, m);
      TTG_CUDA(cudaMemcpyAsync(t.c[k + 1], tmpB_, sizeof(double) * m * p, cudaMemcpyDeviceToDevice, s_));
      eye_kernel<<<eb(m * m), 256, 0, s_>>>(m, t.c[k]);
      TTG_CHECK_LAUNCH();
      r[k + 1] = m;
    }
  } else {
    const i64 m = n[k] * r[k + 1], rr = r[k], p = r[k - 1] * n[k - 1];
    transpose_f64(rr, m, t.c[k], tmpA_, s_);    // m x rr
    if (m >= rr) {
      qr_householder((int)m, (int)rr, tmpA_, R_, tau_, tau_n_, s_);
      transpose_f64(m, rr, tmpA_, t.c[k], s_);   // rr x m
      // core_{k-1} (p x rr) R^T
      gemm((int)p, (int)rr, (int)rr, t.c[k - 1], 1, p, R_, rr, 1, tmpB_, 1, p);
      TTG_CUDA(cudaMemcpyAsync(t.c[k - 1], tmpB_, sizeof(double) * p * rr, cudaMemcpyDeviceToDevice, s_));
    } else {
      // core_{k-1} (p x rr) * core_k (rr x m), core_k = I_m
      gemm((int)p, (int)m, (int)rr, t.c[k - 1], 1, p, t.c[k], 1, rr, tmpB_, 1, p);
      TTG_CUDA(cudaMemcpyAsync(t.c[k - 1], tmpB_, sizeof(double) * p * m, cudaMemcpyDeviceToDevice, s_));
      eye_kernel<<<eb(m * m), 256, 0, s_>>>(m, t.c[k]);
      TTG_CHECK_LAUNCH();
      r[k] = m;
    }
  }
}

void AmenSolver::yax(double* phi_new, const double* phi_old, const DevTT& yy, const DevTT& xx, int k,
                     int dir, bool withA) {
  if (withA) {
    LocalDims L = dims(xx, yy, k);
    if (dir > 0) phi_left_f64(L, phi_old, A_[k], xx.c[k], yy.c[k], phi_new, scr_, s_);
    else phi_right_f64(L, phi_old, A_[k], xx.c[k], yy.c[k], phi_new, scr_, s_);
  } else {
    if (dir > 0) phi2_left_f64(xx.r[k], xx.r[k + 1], yy.r[k], xx.n[k], yy.r[k + 1], phi_old, xx.c[k], yy.c[k], phi_new, scr_, s_);
    else phi2_right_f64(xx.r[k], xx.r[k + 1], yy.r[k], xx.n[k], yy.r[k + 1], phi_old, xx.c[k], yy.c[k], phi_new, scr_, s_);
  }
}

void AmenSolver::project_y(const double* pl, const double* pr, i64 rl, i64 rr, int k, double* out) {
  const i64 n = y_.n[k], y1 = y_.r[k], y2 = y_.r[k + 1];
  gemm((int)rl, (int)(n * y2), (int)y1, pl, 1, rl, y_.c[k], 1, y1, tmpC_, 1, rl);
  gemm((int)(rl * n), (int)rr, (int)y2, tmpC_, 1, rl * n, pr, 1, y2, out, 1, rl * n);
}


// GMRES(local_restart) x local_iters for L x = b (x0 = 0), relative tolerance
// against ||b||.
void AmenSolver::gmres(const LocalDims& L, int k, const double* b, double* x, double tol) {
  if (P_.method == TTG_METHOD_SPLIT) { gmres_split(L, k, b, x, tol); return; }
  const i64 N = L.xsize();
  const int nr = (int)std::min<i64>(std::min<i64>(N, P_.local_restart), 60);
  const double* p1 = pxax_[k];
  const double* p2 = pxax_[k + 1];
  auto mv = [&](const double* in, double* out, int nv) { local_mv(L, p1, p2, k, in, out, nv); };
  if (!gmres_cgs2(mv, N, b, x, tol, nr, P_.local_iters, GmresBufs{V_, w_, gm_, red_, h_, words_}, s_))
    note_capped(ctx_, "dtt_amen_solve");
}


// Chosen form of the local solve: iterative refinement in FP64 around GMRES
// on the BF16x3 tensor-core operator.  Each pass solves A~ d = r (r the FP64
// residual) to the relative accuracy the split operator can carry (1e-4, or
// less when the target is closer), adds d, and recomputes the FP64
// residual; the target tol is the one the plain GMRES is given, measured in
// FP64.
void AmenSolver::gmres_split(const LocalDims& L, int k, const double* b, double* x, double tol) {
  const i64 N = L.xsize();
  const int nr = (int)std::min<i64>(std::min<i64>(N, P_.local_restart), 60);
  MatvecFn mvlow;
  split_matvec_factory(L, pxax_[k], A_[k], pxax_[k + 1], kBatch, split_mem_, split_bytes_, s_,
                       &mvlow);
  auto mvs = [&](const double* in, double* out, int nv) { mvlow(in, out, nv); split_mv_ += nv; };
  const GmresBufs G{V_, w_, gm_, red_, h_, words_};
  const double nb = norm2(b, N);
  TTG_CUDA(cudaMemsetAsync(x, 0, sizeof(double) * N, s_));
  TTG_CUDA(cudaMemcpyAsync(ir_r_, b, sizeof(double) * N, cudaMemcpyDeviceToDevice, s_));
  double nrr = nb;
  for (int it = 0; it < 8 && nrr > tol * nb; ++it) {
    const double inner = std::max(tol * nb / nrr, 1e-4);
    gmres_cgs2(mvs, N, ir_r_, ir_d_, inner, nr, P_.local_iters, G, s_);
    axpy_kernel<<<eb(N), 256, 0, s_>>>(N, 1.0, ir_d_, x);
    TTG_CHECK_LAUNCH();
    local_mv(L, pxax_[k], pxax_[k + 1], k, x, ir_r_, 1);        // FP64 residual b - A x
    sub_kernel<<<eb(N), 256, 0, s_>>>(N, b, ir_r_, ir_r_);
    TTG_CHECK_LAUNCH();
    nrr = norm2(ir_r_, N);
  }
  split_matvec_check(s_);
  if (nrr > tol * nb) note_capped(ctx_, "dtt_amen_solve");
}

// dtt_trunc dir=+1 with the residual criterion (ttnodeop.f90:227-302)
void AmenSolver::trunc(int k, double tol, const double* rhs, double rhs_norm) {
  auto& r = x_.r;
  const i64 n = x_.n[k];
  const i64 m = r[k] * n, rr = r[k + 1], p = x_.n[k + 1] * r[k + 2];
  const int rmin = (int)std::min(m, rr);
  // SVD of core k (m x rr): U (m x rmin), s, Vt (rmin x rr)
  svd_jacobi((int)m, (int)rr, x_.c[k], svU_, svS_, svVt_, svScr_, (int*)(red_ + 16), s_);
  // Vt rows scaled by s: W = diag(s) Vt
  scale_rows_f64(rmin, rr, svVt_, rmin, svS_, s_);
  LocalDims L = dims(x_, x_, k);
  const i64 N = L.xsize();
  int rnew = rmin - 1;
  int fail = 0;   // largest candidate rank whose residual exceeds tol (0: none)
  MatvecFn mvlow;
  if (P_.method == TTG_METHOD_SPLIT)
    split_matvec_factory(L, pxax_[k], A_[k], pxax_[k + 1], kBatch, split_mem_, split_bytes_, s_,
                       &mvlow);
  while (rnew >= 1 && !fail) {
    const int cnt = std::min(kBatch, rnew);
    if (P_.method == TTG_METHOD_SPLIT) {
      // A x_c - rhs = (A x - rhs) - A (x - x_c): the first term is the FP64
      // residual of the full core (resid_), the second the discarded part
      // U[:, rc:] W[rc:, :] through the split operator, whose relative error
      // is then relative to the candidate's own residual
      for (int c = 0; c < cnt; ++c) {
        const int rc = rnew - c;
        gemm((int)m, (int)rr, rmin - rc, svU_ + m * rc, 1, m, svVt_ + rc, 1, rmin, cand_ + N * c, 1, m);
      }
      mvlow(cand_, candY_, cnt);
      split_mv_ += cnt;
      sub_cols_kernel<<<eb(N * cnt), 256, 0, s_>>>(N, cnt, candY_, resid_, candY_);
      TTG_CHECK_LAUNCH();
    } else {
      // candidates rank rnew, rnew-1, ..., rnew-cnt+1: core_c = U[:, :rc] W[:rc, :]
      for (int c = 0; c < cnt; ++c) {
        const int rc = rnew - c;
        gemm((int)m, (int)rr, rc, svU_, 1, m, svVt_, 1, rmin, cand_ + N * c, 1, m);
      }
      local_mv(L, pxax_[k], pxax_[k + 1], k, cand_, candY_, cnt);
      sub_cols_kernel<<<eb(N * cnt), 256, 0, s_>>>(N, cnt, candY_, rhs, candY_);
      TTG_CHECK_LAUNCH();
    }
    sqnorm_cols(N, candY_, N, cnt, red_, s_);
    TTG_CUDA(cudaMemcpyAsync(h_, red_, sizeof(double) * cnt, cudaMemcpyDeviceToHost, s_));
    sync();
    for (int c = 0; c < cnt; ++c) {
      if (std::sqrt(h_[c]) / rhs_norm > tol) {
        fail = rnew - c;
        break;
      }
    }
    rnew -= cnt;
  }
  if (P_.method == TTG_METHOD_SPLIT) split_matvec_check(s_);
  int rk = fail + 1;
  if (rk > rmin) rk = rmin;
  rk = (int)std::min<i64>(rk, P_.rmax);
  // xnew = U[:, :rk] W[:rk, :] (m x rr), core k = U[:, :rk], core k+1 = W[:rk,:] core_{k+1}
  gemm((int)m, (int)rr, rk, svU_, 1, m, svVt_, 1, rmin, xnew_, 1, m);
  TTG_CUDA(cudaMemcpyAsync(x_.c[k], svU_, sizeof(double) * m * rk, cudaMemcpyDeviceToDevice, s_));
  gemm(rk, (int)p, (int)rr, svVt_, 1, rmin, x_.c[k + 1], 1, rr, tmpB_, 1, rk);
  TTG_CUDA(cudaMemcpyAsync(x_.c[k + 1], tmpB_, sizeof(double) * rk * p, cudaMemcpyDeviceToDevice, s_));
  r[k + 1] = rk;
}


void AmenSolver::run(AmenOut& out) {
  const int d = P_.d;
  auto& n = P_.n;
  const int kick = P_.kick;
  TTG_REQUIRE(d >= 2, "amen: d must be >= 2");
  TTG_REQUIRE(P_.rx[0] == 1 && P_.rx[d] == 1 && P_.ry[0] == 1 && P_.ry[d] == 1 &&
              P_.ra[0] == 1 && P_.ra[d] == 1, "boundary ranks must be 1");
  real_tol_ = P_.tol / std::sqrt((double)(d - 1)) / 2.0;   // resid_damp = 2
  // capacities: x ranks never exceed max(initial, rmax + kickrank) nor the
  // size of either side of the bond
  std::vector<i64> left(d + 1, 1), right(d + 1, 1);
  for (int k = 1; k <= d; ++k) left[k] = std::min<i64>(left[k - 1] * n[k - 1], 1ll << 40);
  for (int k = d - 1; k >= 0; --k) right[k] = std::min<i64>(right[k + 1] * n[k], 1ll << 40);
  x_.n = n; y_.n = n; z_.n = n;
  x_.r = P_.rx; y_.r = P_.ry;
  x_.cap.assign(d + 1, 1);
  for (int k = 1; k < d; ++k)
    x_.cap[k] = std::min(std::max(P_.rx[k], P_.rmax + kick), std::min(left[k], right[k]) + kick);
  z_.r.assign(d + 1, 1);
  for (int k = 1; k < d; ++k) z_.r[k] = kick > 0 ? kick : 1;
  i64 Nmax = 1, cmax = 1, pmax = 1, ramax = 1, ymax = 1;
  for (int k = 0; k < d; ++k) {
    Nmax = std::max(Nmax, x_.cap[k] * n[k] * x_.cap[k + 1]);
    ramax = std::max(ramax, P_.ra[k + 1]);
    ymax = std::max(ymax, P_.ry[k + 1]);
  }
  cmax = Nmax;
  for (int k = 0; k <= d; ++k) pmax = std::max(pmax, x_.cap[k] * x_.cap[k] * P_.ra[k]);
  size_t scr = 0;
  for (int k = 0; k < d; ++k) {
    LocalDims L{x_.cap[k], n[k], x_.cap[k + 1], x_.cap[k], n[k], x_.cap[k + 1], P_.ra[k], P_.ra[k + 1]};
    scr = std::max(scr, bfun3_f64_scratch(L, kBatch));
    scr = std::max(scr, phi_f64_scratch(L));
  }
  size_t svds = 0;
  for (int k = 0; k < d; ++k) svds = std::max(svds, svd_scratch((int)(x_.cap[k] * n[k]), (int)x_.cap[k + 1]));
  const int nr = (int)std::min<i64>(std::min<i64>(Nmax, P_.local_restart), 60);
  i64 yt = 0;
  for (int k = 0; k < d; ++k) yt += P_.ry[k] * n[k] * P_.ry[k + 1];
  i64 at = 0;
  for (int k = 0; k < d; ++k) at += P_.ra[k] * n[k] * n[k] * P_.ra[k + 1];
  i64 tcap = cmax;
  for (int k = 0; k < d; ++k)
    tcap = std::max(tcap, std::max(x_.cap[k], z_.r[k]) * n[k] * std::max(ymax, P_.ry[k]));
  size_t total = al8(at);
  for (int k = 0; k < d; ++k) total += al8(x_.cap[k] * n[k] * x_.cap[k + 1]) + al8(P_.ry[k] * n[k] * P_.ry[k + 1]) +
                                       al8(z_.r[k] * n[k] * z_.r[k + 1]);
  for (int k = 0; k <= d; ++k)
    total += al8(x_.cap[k] * x_.cap[k] * P_.ra[k]) + al8(x_.cap[k] * P_.ry[k]) +
             al8(z_.r[k] * x_.cap[k] * P_.ra[k]) + al8(z_.r[k] * P_.ry[k]);
  {
    const i64 rcap = *std::max_element(x_.cap.begin(), x_.cap.end());   // widest QR
    tau_n_ = std::max<size_t>(8192, qr_work_elems(rcap, rcap));
  }
  total += 2 * al8(cmax) + al8(tcap) + al8(Nmax) * 5 + al8(cmax) + al8(tau_n_) + scr + 256;
  total += svds + 256 + 3 * al8(cmax) + al8(8192);
  total += 2 * al8(Nmax * kBatch) + al8(Nmax * (nr + 1)) + al8(Nmax) + al8(4096) + al8(AR_WORDS) +
           al8((size_t)std::min<i64>(P_.max_full_size, 64) * 64) + (1 << 16);
  size_t splitb = 0;
  if (P_.method == TTG_METHOD_SPLIT) {
    for (int k = 0; k < d; ++k) {
      LocalDims L{x_.cap[k], n[k], x_.cap[k + 1], x_.cap[k], n[k], x_.cap[k + 1], P_.ra[k], P_.ra[k + 1]};
      TTG_REQUIRE(split_op_supported(L), "amen: local problem too large for the split operator");
      splitb = std::max(splitb, split_matvec_bytes(L, kBatch));
    }
    total += splitb + 1024 + 2 * al8(Nmax);
  }
  mem_.alloc(total);
  double* dA = mem_.take(at);
  A_.resize(d);
  {
    i64 off = 0;
    for (int k = 0; k < d; ++k) { A_[k] = dA + off; off += P_.ra[k] * n[k] * n[k] * P_.ra[k + 1]; }
  }
  x_.c.resize(d); y_.c.resize(d); z_.c.resize(d);
  for (int k = 0; k < d; ++k) {
    x_.c[k] = mem_.take(x_.cap[k] * n[k] * x_.cap[k + 1]);
    y_.c[k] = mem_.take(P_.ry[k] * n[k] * P_.ry[k + 1]);
    z_.c[k] = mem_.take(z_.r[k] * n[k] * z_.r[k + 1]);
  }
  pxax_.resize(d + 1); pxy_.resize(d + 1); pzax_.resize(d + 1); pzy_.resize(d + 1);
  for (int k = 0; k <= d; ++k) {
    pxax_[k] = mem_.take(x_.cap[k] * x_.cap[k] * P_.ra[k]);
    pxy_[k] = mem_.take(x_.cap[k] * P_.ry[k]);
    pzax_[k] = mem_.take(z_.r[k] * x_.cap[k] * P_.ra[k]);
    pzy_[k] = mem_.take(z_.r[k] * P_.ry[k]);
  }
  tmpA_ = mem_.take(cmax); tmpB_ = mem_.take(cmax); tmpC_ = mem_.take(tcap);
  rhs_ = mem_.take(Nmax); resid_ = mem_.take(Nmax); sol_ = mem_.take(Nmax); xnew_ = mem_.take(Nmax);
  w_ = mem_.take(Nmax);
  R_ = mem_.take(cmax);
  tau_ = mem_.take(tau_n_);
  scr_ = (double*)mem_.take(scr / sizeof(double) + 1);
  svScr_ = (double*)mem_.take(svds / sizeof(double) + 1);
  svU_ = mem_.take(cmax); svS_ = mem_.take(8192); svVt_ = mem_.take(cmax);
  cand_ = mem_.take(Nmax * kBatch); candY_ = mem_.take(Nmax * kBatch);
  V_ = mem_.take(Nmax * (nr + 1));
  red_ = mem_.take(64);
  gm_ = mem_.take(4096);
  words_ = (unsigned long long*)mem_.take(AR_WORDS);
  dense_ = mem_.take(64 * 64);
  if (P_.method == TTG_METHOD_SPLIT) {
    split_mem_ = (void*)mem_.take(splitb / sizeof(double) + 128);
    split_bytes_ = splitb;
    ir_r_ = mem_.take(Nmax);
    ir_d_ = mem_.take(Nmax);
  }
  TTG_CUDA(cudaMallocHost(&h_, 4096 * sizeof(double)));
  struct HG { double* p; ~HG() { if (p) cudaFreeHost(p); } } hg{h_};

  // upload
  TTG_CUDA(cudaMemcpyAsync(dA, P_.crA, sizeof(double) * at, cudaMemcpyHostToDevice, s_));
  {
    i64 ox = 0, oy = 0;
    for (int k = 0; k < d; ++k) {
      TTG_CUDA(cudaMemcpyAsync(x_.c[k], P_.crX0 + ox, sizeof(double) * x_.size(k), cudaMemcpyHostToDevice, s_));
      TTG_CUDA(cudaMemcpyAsync(y_.c[k], P_.crY + oy, sizeof(double) * y_.size(k), cudaMemcpyHostToDevice, s_));
      ox += x_.size(k);
      oy += y_.size(k);
    }
  }
  if (kick > 0) {
    i64 zt = 0;
    for (int k = 0; k < d; ++k) zt += z_.size(k);
    std::vector<double> zh(zt);
    sm_normals(P_.seed, zt, zh.data());
    i64 oz = 0;
    for (int k = 0; k < d; ++k) {
      TTG_CUDA(cudaMemcpyAsync(z_.c[k], zh.data() + oz, sizeof(double) * z_.size(k), cudaMemcpyHostToDevice, s_));
      oz += z_.size(k);
    }
    sync();
  }
  for (double* ph : {pxax_[0], pxax_[d], pxy_[0], pxy_[d], pzax_[0], pzax_[d], pzy_[0], pzy_[d]})
    fill_f64(ph, 1, 1.0, s_);

  int swp_done = 0;
  double res_max = 0.0;
  for (int swp = 1; swp <= P_.nswp; ++swp) {
    swp_done = swp;
    for (int k = d - 1; k >= 1; --k) {
      if (kick > 0 && swp > 1) {
        LocalDims Lz = dims(x_, z_, k);
        local_mv(Lz, pzax_[k], pzax_[k + 1], k, x_.c[k], z_.c[k], 1);
        project_y(pzy_[k], pzy_[k + 1], z_.r[k], z_.r[k + 1], k, rhs_);
        sub_kernel<<<eb(z_.size(k)), 256, 0, s_>>>(z_.size(k), z_.c[k], rhs_, z_.c[k]);
        TTG_CHECK_LAUNCH();
      }
      qr(x_, k, -1);
      yax(pxax_[k], pxax_[k + 1], x_, x_, k, -1, true);
      yax(pxy_[k], pxy_[k + 1], x_, y_, k, -1, false);
      if (kick > 0) {
        qr(z_, k, -1);
        yax(pzax_[k], pzax_[k + 1], z_, x_, k, -1, true);
        yax(pzy_[k], pzy_[k + 1], z_, y_, k, -1, false);
      }
    }
    res_max = 0.0;
    double err_max = 0.0;
    for (int k = 0; k < d; ++k) {
      const i64 rx1 = x_.r[k], rx2 = x_.r[k + 1];
      LocalDims L = dims(x_, x_, k);
      const i64 N = L.xsize();
      project_y(pxy_[k], pxy_[k + 1], rx1, rx2, k, rhs_);
      local_mv(L, pxax_[k], pxax_[k + 1], k, x_.c[k], resid_, 1);
      sub_kernel<<<eb(N), 256, 0, s_>>>(N, resid_, rhs_, resid_);
      TTG_CHECK_LAUNCH();
      const double nr_rhs = norm2(rhs_, N);
      double err = norm2(resid_, N) / nr_rhs;
      res_max = std::max(res_max, err);
      if (err > real_tol_) {
        if (N < P_.max_full_size && N <= 64) {
          fullmat_f64(rx1, n[k], rx2, P_.ra[k], P_.ra[k + 1], pxax_[k], A_[k], pxax_[k + 1], dense_, s_);
          TTG_CUDA(cudaMemcpyAsync(sol_, resid_, sizeof(double) * N, cudaMemcpyDeviceToDevice, s_));
          TTG_CUDA(cudaMemsetAsync(red_ + 32, 0, sizeof(int), s_));
          lu_solve_kernel<<<1, 256, 0, s_>>>((int)N, dense_, sol_, (int*)(red_ + 32));
          TTG_CHECK_LAUNCH();
        } else {
          gmres(L, k, resid_, sol_, real_tol_ / err);
        }
        sub_kernel<<<eb(N), 256, 0, s_>>>(N, x_.c[k], sol_, x_.c[k]);
        TTG_CHECK_LAUNCH();
        err_max = std::max(err_max, norm2(sol_, N) / norm2(x_.c[k], N));
        local_mv(L, pxax_[k], pxax_[k + 1], k, x_.c[k], resid_, 1);
        sub_kernel<<<eb(N), 256, 0, s_>>>(N, resid_, rhs_, resid_);
        TTG_CHECK_LAUNCH();
        err = norm2(resid_, N) / nr_rhs;
      }
      if (k < d - 1) {
        if (kick > 0) {
          err = std::max(err, real_tol_ * 2.0);
          trunc(k, err, rhs_, nr_rhs);
          // sol = A xnew projected on (x-left, z-right) - Phi_XY y Phi_ZY
          LocalDims Lxz{rx1, n[k], rx2, rx1, n[k], z_.r[k + 1], P_.ra[k], P_.ra[k + 1]};
          local_mv(Lxz, pxax_[k], pzax_[k + 1], k, xnew_, sol_, 1);
          LocalDims Lzz{rx1, n[k], rx2, z_.r[k], n[k], z_.r[k + 1], P_.ra[k], P_.ra[k + 1]};
          local_mv(Lzz, pzax_[k], pzax_[k + 1], k, xnew_, z_.c[k], 1);
          project_y(pxy_[k], pzy_[k + 1], rx1, z_.r[k + 1], k, rhs_);
          sub_kernel<<<eb(rx1 * n[k] * z_.r[k + 1]), 256, 0, s_>>>(rx1 * n[k] * z_.r[k + 1], sol_, rhs_, sol_);
          TTG_CHECK_LAUNCH();
          project_y(pzy_[k], pzy_[k + 1], z_.r[k], z_.r[k + 1], k, rhs_);
          sub_kernel<<<eb(z_.size(k)), 256, 0, s_>>>(z_.size(k), z_.c[k], rhs_, z_.c[k]);
          TTG_CHECK_LAUNCH();
          // enrich: core k = [core k | sol], core k+1 gets zero rows
          const i64 rho = z_.r[k + 1];
          const i64 m = x_.r[k] * n[k], rk = x_.r[k + 1], p = n[k + 1] * x_.r[k + 2];
          TTG_REQUIRE(rk + rho <= x_.cap[k + 1], "amen: rank capacity exceeded");
          TTG_CUDA(cudaMemcpyAsync(x_.c[k] + m * rk, sol_, sizeof(double) * m * rho,
                                   cudaMemcpyDeviceToDevice, s_));
          pad_rows_kernel<<<eb((rk + rho) * p), 256, 0, s_>>>(rk, rho, p, x_.c[k + 1], tmpB_);
          TTG_CHECK_LAUNCH();
          TTG_CUDA(cudaMemcpyAsync(x_.c[k + 1], tmpB_, sizeof(double) * (rk + rho) * p,
                                   cudaMemcpyDeviceToDevice, s_));
          x_.r[k + 1] = rk + rho;
          qr(x_, k, +1);
          qr(z_, k, +1);
          yax(pzax_[k + 1], pzax_[k], z_, x_, k, +1, true);
          yax(pzy_[k + 1], pzy_[k], z_, y_, k, +1, false);
        } else {
          qr(x_, k, +1);
        }
        yax(pxax_[k + 1], pxax_[k], x_, x_, k, +1, true);
        yax(pxy_[k + 1], pxy_[k], x_, y_, k, +1, false);
      }
    }
    if (P_.verb > 0) {
      i64 mr = *std::max_element(x_.r.begin(), x_.r.end());
      fprintf(stderr, "amen_solve: swp=%d, max_dx=%.3e, max_res=%.3e, max_rank=%lld\n", swp,
              err_max, res_max, (long long)mr);
    }
    if (res_max < P_.tol) break;
  }
  sync();
  i64 tot = 0;
  for (int k = 0; k < d; ++k) tot += x_.size(k);
  out.cores.resize(tot);
  i64 off = 0;
  for (int k = 0; k < d; ++k) {
    TTG_CUDA(cudaMemcpyAsync(out.cores.data() + off, x_.c[k], sizeof(double) * x_.size(k),
                             cudaMemcpyDeviceToHost, s_));
    off += x_.size(k);
  }
  sync();
  out.rx = x_.r;
  out.sweeps = swp_done;
  out.res_max = res_max;
  out.matvecs = nmv_ + split_mv_;
}


// ---------------------------------------------------------------------------
// tt_amen_solve of tt_adapt_als.f90 (alternating half sweeps, Householder
// GMRES correction, residual-based truncation from the top, kick by an
// incremental Cholesky of [Y-projection, A-projection])
// ---------------------------------------------------------------------------
namespace {

// B(n1, n3, n2, n4) = A(n1, n2, n3, n4)   (dperm1324, tt_linalg.f90:101-120)
__global__ void perm1324_kernel(i64 n1, i64 n2, i64 n3, i64 n4, const double* __restrict__ A,
                                double* __restrict__ B) {
  const i64 tot = n1 * n2 * n3 * n4;
  for (i64 e = blockIdx.x * (i64)blockDim.x + threadIdx.x; e < tot; e += (i64)gridDim.x * blockDim.x) {
    const i64 i1 = e % n1, i2 = (e / n1) % n2, i3 = (e / (n1 * n2)) % n3, i4 = e / (n1 * n2 * n3);
    B[i1 + n1 * (i3 + n3 * (i2 + n2 * i4))] = A[e];
  }
}
// out ((m1 + m2) x nc) = [A (m1 x nc); B (m2 x nc)]   (drow_add, tt_linalg.f90:54-69)
__global__ void concat_rows_kernel(i64 m1, i64 m2, i64 nc, const double* __restrict__ A,
                                   const double* __restrict__ B, double* __restrict__ out) {
  const i64 M = m1 + m2;
  for (i64 e = blockIdx.x * (i64)blockDim.x + threadIdx.x; e < M * nc; e += (i64)gridDim.x * blockDim.x) {
    const i64 r = e % M, c = e / M;
    out[e] = r < m1 ? A[r + m1 * c] : B[(r - m1) + m2 * c];
  }
}
// incremental Cholesky (duchol_fort) pieces; A(i, k) = dA[i * si + k * sk],
// i < n rows, k < m columns
__global__ void uchol_diag_kernel(i64 n, i64 m, const double* __restrict__ dA, i64 si, i64 sk,
                                  double* __restrict__ dd) {
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
    double acc = 0.0;
    for (i64 k = 0; k < m; ++k) { const double v = dA[i * si + k * sk]; acc = fma(v, v, acc); }
    dd[i] = acc;
  }
}
// first index of the largest |dd| (idamax), one block
__global__ void argmax_abs_kernel(i64 n, const double* __restrict__ dd, int* __restrict__ out) {
  __shared__ double sv[32];
  __shared__ int si[32];
  double v = -1.0;
  int idx = 0x7fffffff;
  for (i64 i = threadIdx.x; i < n; i += blockDim.x) {
    const double a = fabs(dd[i]);
    if (a > v || (a == v && (int)i < idx)) { v = a; idx = (int)i; }
  }
  for (int o = 16; o > 0; o >>= 1) {
    const double v2 = __shfl_xor_sync(0xffffffffu, v, o);
    const int i2 = __shfl_xor_sync(0xffffffffu, idx, o);
    if (v2 > v || (v2 == v && i2 < idx)) { v = v2; idx = i2; }
  }
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) { sv[w] = v; si[w] = idx; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double bv = -1.0;
    int bi = 0x7fffffff;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q)
      if (sv[q] > bv || (sv[q] == bv && si[q] < bi)) { bv = sv[q]; bi = si[q]; }
    *out = bi;
  }
}
// du[:, c] = A A(maxi, :)^T - sum_{j < c} lam_j du(maxi, j) du[:, j]
__global__ void uchol_col_kernel(i64 n, i64 m, const double* __restrict__ dA, i64 si, i64 sk,
                                 const int* __restrict__ maxi_p, int c, const double* __restrict__ lam,
                                 double* __restrict__ du) {
  const i64 mi = *maxi_p;
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
    double acc = 0.0;
    for (i64 k = 0; k < m; ++k) acc = fma(dA[i * si + k * sk], dA[mi * si + k * sk], acc);
    for (int j = 0; j < c; ++j) acc -= lam[j] * du[mi + n * j] * du[i + n * j];
    du[i + n * c] = acc;
  }
}
__global__ void uchol_pick_kernel(i64 n, const int* __restrict__ maxi_p, int c,
                                  const double* __restrict__ du, double* __restrict__ out) {
  *out = du[*maxi_p + n * c];
}
// du[:, c] /= sqrt(|piv|); dd -= du[:, c]^2
__global__ void uchol_scale_kernel(i64 n, int c, const double* __restrict__ piv, double* __restrict__ du,
                                   double* __restrict__ dd) {
  const double inv = 1.0 / sqrt(fabs(*piv));
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
    const double v = du[i + n * c] * inv;
    du[i + n * c] = v;
    dd[i] -= v * v;
  }
}
// dv (k x k) = dx dx^T + diag(lam), dx = R(:, k-1) (R k x k)
__global__ void uchol_dv_kernel(int k, const double* __restrict__ R, const double* __restrict__ lam,
                                double* __restrict__ dv) {
  for (int e = threadIdx.x; e < k * k; e += blockDim.x) {
    const int i = e % k, j = e / k;
    dv[e] = R[i + k * (k - 1)] * R[j + k * (k - 1)] + (i == j ? lam[i] : 0.0);
  }
}

}  // namespace

// buffers of uchol_run: small >= 1024 doubles, dd and tmp >= n (and n * k),
// tau >= 16, h pinned host, ired >= 16 ints
struct UcholWork {
  double *small, *dd, *tmp, *tau, *h;
  int* ired;
};

// duchol_fort (tt_linalg.f90:540-642).  trans: dA is n x m, else m x n.
// Writes du (n x real) and returns real (the Fortran loop index: numvec, or
// the failing step when the pivot vanishes).
static int uchol_run(bool trans, i64 m, i64 n, const double* dA, int numvec, double* du,
                     const UcholWork& W, cudaStream_t s) {
  TTG_REQUIRE(numvec <= 16, "uchol: at most 16 vectors");
  const i64 si = trans ? 1 : m, sk = trans ? n : 1;
  double* lam = W.small;          // numvec <= 16
  double* Rk = W.small + 16;      // k x k
  double* dv = W.small + 272;     // k x k
  double* V = W.small + 528;      // k x k
  double* piv = W.small + 784;
  TTG_CUDA(cudaMemsetAsync(lam, 0, sizeof(double) * 16, s));
  TTG_CUDA(cudaMemsetAsync(du, 0, sizeof(double) * n * numvec, s));
  uchol_diag_kernel<<<eb(n), 256, 0, s>>>(n, m, dA, si, sk, W.dd);
  TTG_CHECK_LAUNCH();
  int cnt = 0;
  bool broke = false;
  while (cnt < numvec) {
    argmax_abs_kernel<<<1, 256, 0, s>>>(n, W.dd, W.ired);
    TTG_CHECK_LAUNCH();
    uchol_col_kernel<<<eb(n), 256, 0, s>>>(n, m, dA, si, sk, W.ired, cnt, lam, du);
    TTG_CHECK_LAUNCH();
    uchol_pick_kernel<<<1, 1, 0, s>>>(n, W.ired, cnt, du, piv);
    TTG_CHECK_LAUNCH();
    TTG_CUDA(cudaMemcpyAsync(W.h, piv, sizeof(double), cudaMemcpyDeviceToHost, s));
    TTG_CUDA(cudaStreamSynchronize(s));
    if (std::sqrt(std::fabs(W.h[0])) < 1e-300) { broke = true; break; }
    uchol_scale_kernel<<<eb(n), 256, 0, s>>>(n, cnt, piv, du, W.dd);
    TTG_CHECK_LAUNCH();
    const int k = cnt + 1;
    qr_householder((int)n, k, du, Rk, W.tau, 16, s);          // du[:, :k] = Q, Rk = R
    uchol_dv_kernel<<<1, 256, 0, s>>>(k, Rk, lam, dv);
    TTG_CHECK_LAUNCH();
    syev_jacobi(k, dv, k, lam, V, k, W.ired + 8, s);      // ascending, as dsyev
    GemmF64 g;
    g.M = (int)n; g.N = k; g.K = k;
    g.A = du; g.sAm = 1; g.sAk = n;
    g.B = V; g.sBk = 1; g.sBn = k;
    g.C = W.tmp; g.sCm = 1; g.sCn = n;
    gemm_f64(g, s);
    TTG_CUDA(cudaMemcpyAsync(du, W.tmp, sizeof(double) * n * k, cudaMemcpyDeviceToDevice, s));
    ++cnt;
  }
  return broke ? cnt + 1 : numvec;
}

// dbfun3_right (tt_linalg.f90:210-240): y (rx1 ra1) x (n ry2) from x
// (rx1, m, rx2) and Phi2 (rx2, ra2, ry2); tA, tB hold
// max(rx1 m ra2 ry2, ra1 n ry2 rx1) doubles each.
static void bfun3_right_run(i64 rx1, i64 m, i64 rx2, i64 n, i64 ry2, i64 ra1, i64 ra2,
                            const double* A, const double* phi2, const double* x, double* y,
                            double* tA, double* tB, cudaStream_t s) {
  auto gemm = [&](int M, int N, int K, const double* Am, i64 sAm, i64 sAk, const double* Bm,
                  i64 sBk, i64 sBn, double* C, i64 sCm, i64 sCn) {
    GemmF64 g;
    g.M = M; g.N = N; g.K = K;
    g.A = Am; g.sAm = sAm; g.sAk = sAk;
    g.B = Bm; g.sBk = sBk; g.sBn = sBn;
    g.C = C; g.sCm = sCm; g.sCn = sCn;
    gemm_f64(g, s);
  };
  gemm((int)(rx1 * m), (int)(ra2 * ry2), (int)rx2, x, 1, rx1 * m, phi2, 1, rx2, tA, 1, rx1 * m);
  transpose_f64(rx1, m * ra2 * ry2, tA, tB, s);                             // j,a2,c2,b1
  gemm((int)(ra1 * n), (int)(ry2 * rx1), (int)(m * ra2), A, 1, ra1 * n, tB, 1, m * ra2, tA, 1,
       ra1 * n);                                                           // a1,i,c2,b1
  transpose_f64(ra1 * n * ry2, rx1, tA, y, s);                              // b1,a1,i,c2
}

struct AlsParams {
  int d;
  std::vector<i64> n, ra, ry, rx;
  const double *crA, *crY, *crX0;
  double eps;
  i64 rmax;
  int kick, nswp, nrestart, niters, verb;
  char prec = 0;   // 0 (none) or the block-Jacobi type 'c', 'l', 'r'
};

// device array that grows on demand (block-Jacobi blocks: their size follows
// the current ranks, which the rank capacities bound only loosely)
struct GrowBuf {
  double* p = nullptr;
  size_t cap = 0;
  ~GrowBuf() { if (p) cudaFree(p); }
  double* ensure(size_t count, cudaStream_t s) {
    if (count <= cap) return p;
    TTG_CUDA(cudaStreamSynchronize(s));
    if (p) cudaFree(p);
    p = nullptr;
    cap = 0;
    if (cudaMalloc(&p, count * sizeof(double)) != cudaSuccess) {
      p = nullptr;
      throw Error{TTG_ERR_NOMEM, "amen: preconditioner allocation failed"};
    }
    cap = count;
    return p;
  }
};

class AlsSolver {
 public:
  AlsSolver(ttg_ctx* ctx, const AlsParams& P) : P_(P), s_(ctx->stream), ctx_(ctx) {
    ctx->stat_capped = 0;
  }
  void run(AmenOut& out);

 private:
  AlsParams P_;
  cudaStream_t s_;
  ttg_ctx* ctx_;
  Arena mem_;
  std::vector<i64> n_, rx_, cap_;
  size_t tau_n_ = 0;   // elements of tau_
  unsigned long long* words_ = nullptr;   // exchanges of the Arnoldi steps
  std::vector<double*> x_, A_, Y_, phiA_, phiy_;
  double *rhs_, *r0_, *sol_, *w_, *V_, *gm_, *red_, *kickY_, *kickB_, *tA_, *tB_, *tC_, *U_, *S_,
      *Vt_, *svScr_, *cand_, *candY_, *Um_, *Rm_, *Rq_, *tau_, *tmp_, *scr_, *du_, *dd_, *small_;
  int* ired_;
  double* h_ = nullptr;
  long long nmv_ = 0;
  GrowBuf jacs_, jscr_;
  static constexpr int kBatch = 8;

  void sync() { TTG_CUDA(cudaStreamSynchronize(s_)); }
  LocalDims dims(int k) const {
    return LocalDims{rx_[k], n_[k], rx_[k + 1], rx_[k], n_[k], rx_[k + 1], P_.ra[k], P_.ra[k + 1]};
  }
  void gemm(int M, int N, int K, const double* A, i64 sAm, i64 sAk, const double* B, i64 sBk,
            i64 sBn, double* C, i64 sCm, i64 sCn, double alpha = 1.0, double beta = 0.0) {
    GemmF64 g;
    g.M = M; g.N = N; g.K = K;
    g.A = A; g.sAm = sAm; g.sAk = sAk;
    g.B = B; g.sBk = sBk; g.sBn = sBn;
    g.C = C; g.sCm = sCm; g.sCn = sCn;
    g.alpha = alpha; g.beta = beta;
    gemm_f64(g, s_);
  }
  double norm2(const double* v, i64 n) {
    sqnorm_cols(n, v, n, 1, red_, s_);
    TTG_CUDA(cudaMemcpyAsync(h_, red_, sizeof(double), cudaMemcpyDeviceToHost, s_));
    sync();
    return std::sqrt(h_[0]);
  }
  void mv(int k, const double* x, double* y, int nv) {
    bfun3_f64(dims(k), phiA_[k], A_[k], phiA_[k + 1], x, y, nv, scr_, s_);
    nmv_ += nv;
  }
  void qr(i64 m, i64 c, double* A, double* R) { qr_householder((int)m, (int)c, A, R, tau_, tau_n_, s_); }
  void upd_left(int i);
  void upd_right(int i);
  int scan(int i, int rmin, const double* L, i64 ldl, const double* Rr, i64 ldr, i64 rows, i64 cols,
           const double* rhs, double nrhs, double res_new, double eps2);
  int uchol(bool trans, i64 m, i64 n, const double* dA, int numvec, double* du);
  void bfun3_left(int i, const double* x, double* y);
  void bfun3_right(int i, const double* x, double* y);
};

void AlsSolver::upd_left(int i) {
  phi_left_f64(dims(i), phiA_[i], A_[i], x_[i], x_[i], phiA_[i + 1], scr_, s_);
  phi2_left_f64(P_.ry[i], P_.ry[i + 1], rx_[i], n_[i], rx_[i + 1], phiy_[i], Y_[i], x_[i],
                phiy_[i + 1], scr_, s_);
}

void AlsSolver::upd_right(int i) {
  phi_right_f64(dims(i), phiA_[i + 1], A_[i], x_[i], x_[i], phiA_[i], scr_, s_);
  phi2_right_f64(P_.ry[i], P_.ry[i + 1], rx_[i], n_[i], rx_[i + 1], phiy_[i + 1], Y_[i], x_[i],
                 phiy_[i], scr_, s_);
}

// Residual-based rank scan from the top (tt_adapt_als.f90:812-829, 917-934):
// candidate rank c gives the core L[:, :c] R[:c, :] (rows x cols); the kept
// rank is one more than the first c (counting down from rmin-1) whose
// residual exceeds both 2 res_new and eps2, or 1 when none does.  Candidates
// are evaluated kBatch at a time with one block matvec.
int AlsSolver::scan(int i, int rmin, const double* L, i64 ldl, const double* Rr, i64 ldr, i64 rows,
                    i64 cols, const double* rhs, double nrhs, double res_new, double eps2) {
  const i64 N = rows * cols;
  int c0 = rmin - 1;
  while (c0 >= 1) {
    const int cnt = std::min(kBatch, c0);
    for (int q = 0; q < cnt; ++q)
      gemm((int)rows, (int)cols, c0 - q, L, 1, ldl, Rr, 1, ldr, cand_ + N * q, 1, rows);
    mv(i, cand_, candY_, cnt);
    sub_cols_kernel<<<eb(N * cnt), 256, 0, s_>>>(N, cnt, candY_, rhs, candY_);
    TTG_CHECK_LAUNCH();
    sqnorm_cols(N, candY_, N, cnt, red_, s_);
    TTG_CUDA(cudaMemcpyAsync(h_, red_, sizeof(double) * cnt, cudaMemcpyDeviceToHost, s_));
    sync();
    for (int q = 0; q < cnt; ++q) {
      const double e = std::sqrt(h_[q]) / nrhs;
      if (e > res_new * 2.0 && e > eps2) return c0 - q + 1;
    }
    c0 -= cnt;
  }
  return 1;
}

int AlsSolver::uchol(bool trans, i64 m, i64 n, const double* dA, int numvec, double* du) {
  return uchol_run(trans, m, n, dA, numvec, du, UcholWork{small_, dd_, tmp_, tau_, h_, ired_}, s_);
}

// dbfun3_left as the reference writes it (tt_linalg.f90:242-253): Phi1's
// (ry1, rx1, ra1) memory is multiplied as an (ra1*ry1) x rx1 matrix.
// y: (ry1 n) x (rx2 ra2), ry1 = rx1 = rx_[i].
void AlsSolver::bfun3_left(int i, const double* x, double* y) {
  const i64 rx1 = rx_[i], m = n_[i], rx2 = rx_[i + 1], ry1 = rx1, n = m;
  const i64 ra1 = P_.ra[i], ra2 = P_.ra[i + 1];
  gemm((int)(ra1 * ry1), (int)(m * rx2), (int)rx1, phiA_[i], 1, ra1 * ry1, x, 1, rx1, tA_, 1,
       ra1 * ry1);                                                         // (a1,c1),(j,b2)
  perm1324_kernel<<<eb(ra1 * ry1 * m * rx2), 256, 0, s_>>>(ra1, ry1, m, rx2, tA_, tB_);  // a1,j,c1,b2
  TTG_CHECK_LAUNCH();
  perm1324_kernel<<<eb(ra1 * n * m * ra2), 256, 0, s_>>>(ra1, n, m, ra2, A_[i], tC_);   // a1,j,i,a2
  TTG_CHECK_LAUNCH();
  gemm((int)(ry1 * rx2), (int)(n * ra2), (int)(ra1 * m), tB_, ra1 * m, 1, tC_, 1, ra1 * m, tA_, 1,
       ry1 * rx2);                                                         // (c1,b2),(i,a2)
  perm1324_kernel<<<eb(ry1 * rx2 * n * ra2), 256, 0, s_>>>(ry1, rx2, n, ra2, tA_, y);   // c1,i,b2,a2
  TTG_CHECK_LAUNCH();
}

// dbfun3_right (tt_linalg.f90:210-240): y (rx1 ra1) x (n ry2), ry2 = rx2
void AlsSolver::bfun3_right(int i, const double* x, double* y) {
  bfun3_right_run(rx_[i], n_[i], rx_[i + 1], n_[i], rx_[i + 1], P_.ra[i], P_.ra[i + 1], A_[i],
                  phiA_[i + 1], x, y, tA_, tB_, s_);
}

void AlsSolver::run(AmenOut& out) {
  const int d = P_.d;
  n_ = P_.n;
  rx_ = P_.rx;
  const auto& ry = P_.ry;
  const auto& ra = P_.ra;
  TTG_REQUIRE(d >= 2, "amen: d must be >= 2");
  TTG_REQUIRE(rx_[0] == 1 && rx_[d] == 1 && ry[0] == 1 && ry[d] == 1 && ra[0] == 1 && ra[d] == 1,
              "boundary ranks must be 1");
  const double eps2 = P_.eps / std::sqrt((double)d);
  const int kick0 = P_.kick;
  const int kpad = std::max(kick0, 0);
  // rank capacities: the kept rank is at most min(rmax, both sides of the
  // bond), and the kick adds at most kickrank
  std::vector<i64> left(d + 1, 1), right(d + 1, 1);
  for (int k = 1; k <= d; ++k) left[k] = std::min<i64>(left[k - 1] * n_[k - 1], 1ll << 40);
  for (int k = d - 1; k >= 0; --k) right[k] = std::min<i64>(right[k + 1] * n_[k], 1ll << 40);
  cap_.assign(d + 1, 1);
  for (int k = 1; k < d; ++k)
    cap_[k] = std::max(rx_[k], std::min(P_.rmax, std::min(left[k], right[k])) + kpad);
  i64 Nmax = 1, ramax = 1, rymax = 1, T = 1, KB = 1, Mmax = 1, SVD = 1, PHS = 1, Cmax = 1;
  size_t scr = 0, svs = 0;
  for (int k = 0; k <= d; ++k) { ramax = std::max(ramax, ra[k]); rymax = std::max(rymax, ry[k]); }
  for (int k = 0; k < d; ++k) {
    const i64 c1 = cap_[k], c2 = cap_[k + 1], nk = n_[k];
    Nmax = std::max(Nmax, c1 * nk * c2);
    Mmax = std::max(Mmax, std::max(c1 * nk, nk * c2));
    T = std::max(T, std::max(ra[k], ra[k + 1]) * std::max(c1, c2) * std::max(c1, c2) * nk *
                        std::max(ra[k], ra[k + 1]) + ra[k] * nk * nk * ra[k + 1]);
    KB = std::max(KB, c1 * nk * (ry[k + 1] + c2 * ra[k + 1]));
    KB = std::max(KB, (ry[k] + c1 * ra[k]) * nk * c2);
    Cmax = std::max(Cmax, std::max(c1 * nk * c2, std::max(ry[k], c1) * nk * std::max(ry[k + 1], c2)));
    LocalDims L{c1, nk, c2, c1, nk, c2, ra[k], ra[k + 1]};
    scr = std::max(scr, bfun3_f64_scratch(L, kBatch));
    scr = std::max(scr, phi_f64_scratch(L));
    scr = std::max(scr, (size_t)(4 * std::max(ry[k], c1) * nk * std::max(ry[k + 1], c2) * 8));
    svs = std::max(svs, svd_scratch((int)(c1 * nk), (int)c2));
    svs = std::max(svs, svd_scratch((int)c1, (int)(nk * c2)));
    SVD = std::max(SVD, c1 * nk * c2 + std::max(c1 * nk, nk * c2) * std::min(std::max(c1 * nk, nk * c2), std::max(c1, c2)));
    PHS = std::max(PHS, c1 * c1 * ra[k]);
  }
  const int nr = (int)std::min<i64>(std::min<i64>(Nmax, P_.nrestart), 60);
  i64 at = 0, yt = 0;
  for (int k = 0; k < d; ++k) {
    at += ra[k] * n_[k] * n_[k] * ra[k + 1];
    yt += ry[k] * n_[k] * ry[k + 1];
  }
  const i64 M2 = Mmax * std::max<i64>(Mmax, 1);
  {
    const i64 rcap = *std::max_element(cap_.begin(), cap_.end()) + 16;
    tau_n_ = std::max<size_t>(8192, qr_work_elems(rcap, rcap));
  }
  size_t total = al8(at) + al8(yt);
  for (int k = 0; k < d; ++k) total += al8(cap_[k] * n_[k] * cap_[k + 1]);
  for (int k = 0; k <= d; ++k) total += al8(cap_[k] * cap_[k] * ra[k]) + al8(cap_[k] * ry[k]);
  total += 4 * al8(Nmax) + al8(Nmax * (nr + 1)) + al8(4096) + al8(AR_WORDS) + al8(64) + al8(Cmax) +
           al8(KB) +
           3 * al8(T) + al8(SVD) + al8(1024) + al8(SVD) + svs + 256 + 2 * al8(Nmax * kBatch) +
           al8(M2) + 2 * al8(M2) + al8(tau_n_) + al8(M2) + scr + 256 + al8(Mmax * 16) +
           al8(Mmax) + al8(1024) + al8(64) + (1 << 16);
  mem_.alloc(total);
  double* dA = mem_.take(at);
  double* dY = mem_.take(yt);
  A_.resize(d); Y_.resize(d); x_.resize(d);
  {
    i64 oa = 0, oy = 0;
    for (int k = 0; k < d; ++k) {
      A_[k] = dA + oa; oa += ra[k] * n_[k] * n_[k] * ra[k + 1];
      Y_[k] = dY + oy; oy += ry[k] * n_[k] * ry[k + 1];
    }
  }
  for (int k = 0; k < d; ++k) x_[k] = mem_.take(cap_[k] * n_[k] * cap_[k + 1]);
  phiA_.resize(d + 1); phiy_.resize(d + 1);
  for (int k = 0; k <= d; ++k) {
    phiA_[k] = mem_.take(cap_[k] * cap_[k] * ra[k]);
    phiy_[k] = mem_.take(cap_[k] * ry[k]);
  }
  rhs_ = mem_.take(Nmax); r0_ = mem_.take(Nmax); sol_ = mem_.take(Nmax); w_ = mem_.take(Nmax);
  V_ = mem_.take(Nmax * (nr + 1));
  gm_ = mem_.take(4096);
  words_ = (unsigned long long*)mem_.take(AR_WORDS);
  red_ = mem_.take(64);
  kickY_ = mem_.take(Cmax);
  kickB_ = mem_.take(KB);
  tA_ = mem_.take(T); tB_ = mem_.take(T); tC_ = mem_.take(T);
  U_ = mem_.take(SVD); S_ = mem_.take(1024); Vt_ = mem_.take(SVD);
  svScr_ = (double*)mem_.take(svs / sizeof(double) + 1);
  cand_ = mem_.take(Nmax * kBatch); candY_ = mem_.take(Nmax * kBatch);
  Um_ = mem_.take(M2); Rm_ = mem_.take(M2); Rq_ = mem_.take(M2);
  tau_ = mem_.take(tau_n_);
  tmp_ = mem_.take(M2);
  scr_ = (double*)mem_.take(scr / sizeof(double) + 1);
  du_ = mem_.take(Mmax * 16);
  dd_ = mem_.take(Mmax);
  small_ = mem_.take(1024);
  ired_ = (int*)mem_.take(64);
  TTG_CUDA(cudaMallocHost(&h_, 4096 * sizeof(double)));
  struct HG { double* p; ~HG() { if (p) cudaFreeHost(p); } } hg{h_};

  TTG_CUDA(cudaMemcpyAsync(dA, P_.crA, sizeof(double) * at, cudaMemcpyHostToDevice, s_));
  TTG_CUDA(cudaMemcpyAsync(dY, P_.crY, sizeof(double) * yt, cudaMemcpyHostToDevice, s_));
  {
    i64 ox = 0;
    for (int k = 0; k < d; ++k) {
      const i64 sz = rx_[k] * n_[k] * rx_[k + 1];
      TTG_CUDA(cudaMemcpyAsync(x_[k], P_.crX0 + ox, sizeof(double) * sz, cudaMemcpyHostToDevice, s_));
      ox += sz;
    }
  }
  for (double* ph : {phiA_[0], phiA_[d], phiy_[0], phiy_[d]}) fill_f64(ph, 1, 1.0, s_);

  // initial QR, left to right (tt_adapt_als.f90:618-644)
  for (int i = 0; i + 1 < d; ++i) {
    const i64 m_ = rx_[i] * n_[i], rr = rx_[i + 1], p = n_[i + 1] * rx_[i + 2];
    const i64 rnew = std::min(m_, rr);
    TTG_CUDA(cudaMemcpyAsync(Um_, x_[i], sizeof(double) * m_ * rr, cudaMemcpyDeviceToDevice, s_));
    qr(m_, rr, Um_, Rq_);
    TTG_CUDA(cudaMemcpyAsync(x_[i], Um_, sizeof(double) * m_ * rnew, cudaMemcpyDeviceToDevice, s_));
    gemm((int)rnew, (int)p, (int)rr, Rq_, 1, rnew, x_[i + 1], 1, rr, tmp_, 1, rnew);
    TTG_CUDA(cudaMemcpyAsync(x_[i + 1], tmp_, sizeof(double) * rnew * p, cudaMemcpyDeviceToDevice, s_));
    rx_[i + 1] = rnew;
    upd_left(i);
  }

  const GmresBufs G{V_, w_, gm_, red_, h_, words_};
  double res_max = 0.0, last_res = 0.0, err_max = 0.0;
  int i = d - 1, dir = -1, swp = 1, kick = kick0;
  while (swp <= P_.nswp) {
    const i64 r1 = rx_[i], r2 = rx_[i + 1], nk = n_[i];
    const i64 N = r1 * nk * r2;
    // local right-hand side (tt_adapt_als.f90:657-687)
    if (dir < 0) {
      gemm((int)(ry[i] * nk), (int)r2, (int)ry[i + 1], Y_[i], 1, ry[i] * nk, phiy_[i + 1], 1,
           ry[i + 1], kickY_, 1, ry[i] * nk);
      gemm((int)r1, (int)(nk * r2), (int)ry[i], phiy_[i], 1, r1, kickY_, 1, ry[i], rhs_, 1, r1);
    } else {
      gemm((int)r1, (int)(nk * ry[i + 1]), (int)ry[i], phiy_[i], 1, r1, Y_[i], 1, ry[i], kickY_, 1, r1);
      gemm((int)(r1 * nk), (int)r2, (int)ry[i + 1], kickY_, 1, r1 * nk, phiy_[i + 1], 1, ry[i + 1],
           rhs_, 1, r1 * nk);
    }
    // residual and the GMRES correction (:725-797)
    mv(i, x_[i], r0_, 1);
    sub_kernel<<<eb(N), 256, 0, s_>>>(N, r0_, rhs_, r0_);
    TTG_CHECK_LAUNCH();
    const double nrhs = norm2(rhs_, N);
    double err = norm2(r0_, N) / nrhs;
    res_max = std::max(res_max, err);
    double res_new = err;
    const double tau = eps2 / (err * 2.0);
    if (tau < 1.0) {
      const int nrs = (int)std::min<i64>(std::min<i64>(P_.nrestart, N), 60);
      if (P_.prec) {
        // right preconditioning (tt_linalg.f90:689-690,733-735): GMRES on A P,
        // correction P z (tt_adapt_als.f90:746-781); cand_ holds P v
        const char pt = P_.prec;
        const i64 nk_ = nk;
        double* jacs = jacs_.ensure((size_t)jac_size(pt, r1, nk_, r2), s_);
        double* jscr = jscr_.ensure((size_t)jac_gen_scratch(pt, r1, nk_, r2, ra[i], ra[i + 1]), s_);
        jac_gen_f64(pt, r1, nk_, r2, ra[i], ra[i + 1], phiA_[i], A_[i], phiA_[i + 1], jacs, jscr, s_);
        auto mvf = [&](const double* in, double* o, int nv) {
          jac_apply_f64(pt, r1, nk_, r2, jacs, in, cand_, nv, s_);
          mv(i, cand_, o, nv);
        };
        if (!gmres_cgs2(mvf, N, r0_, sol_, tau, nrs, P_.niters, G, s_))
          note_capped(ctx_, "tt_amen_solve");
        jac_apply_f64(pt, r1, nk_, r2, jacs, sol_, candY_, 1, s_);
        TTG_CUDA(cudaMemcpyAsync(sol_, candY_, sizeof(double) * N, cudaMemcpyDeviceToDevice, s_));
      } else {
        auto mvf = [&](const double* in, double* o, int nv) { mv(i, in, o, nv); };
        if (!gmres_cgs2(mvf, N, r0_, sol_, tau, nrs, P_.niters, G, s_))
          note_capped(ctx_, "tt_amen_solve");
      }
      sub_kernel<<<eb(N), 256, 0, s_>>>(N, x_[i], sol_, x_[i]);
      TTG_CHECK_LAUNCH();
      mv(i, x_[i], r0_, 1);
      sub_kernel<<<eb(N), 256, 0, s_>>>(N, r0_, rhs_, r0_);
      TTG_CHECK_LAUNCH();
      res_new = norm2(r0_, N) / nrhs;
      err_max = std::max(err_max, norm2(sol_, N) / norm2(x_[i], N));
    }
    if (dir > 0 && i < d - 1) {
      // truncation and kick to the right (:807-897)
      const i64 m_ = r1 * nk, rr = r2, p = n_[i + 1] * rx_[i + 2];
      i64 rnew = std::min(rr, m_);
      if (kick > 0 || kick == -1) {
        const int rmin = (int)std::min(m_, rr);
        svd_jacobi((int)m_, (int)rr, x_[i], U_, S_, Vt_, svScr_, ired_ + 16, s_);
        scale_rows_f64(rmin, rr, Vt_, rmin, S_, s_);                     // W = diag(s) Vt
        int nn = scan(i, rmin, U_, m_, Vt_, rmin, m_, rr, rhs_, nrhs, res_new, eps2);
        nn = (int)std::min<i64>(nn, P_.rmax);
        // Um = U[:, :nn], Rm = W[:nn, :]
        TTG_CUDA(cudaMemcpyAsync(Um_, U_, sizeof(double) * m_ * nn, cudaMemcpyDeviceToDevice, s_));
        copy_rows_f64(rmin, nn, rr, Vt_, Rm_, s_);
        rnew = nn;
        if (kick > 0) {
          // kick_block (m_ x (ry2 + rr ra2)) = [Y-projection | dbfun3_left]
          TTG_CUDA(cudaMemcpyAsync(kickB_, kickY_, sizeof(double) * m_ * ry[i + 1],
                                   cudaMemcpyDeviceToDevice, s_));
          bfun3_left(i, x_[i], kickB_ + m_ * ry[i + 1]);
          const int mm = uchol(true, rr * ra[i + 1] + ry[i + 1], m_, kickB_,
                               (int)std::min<i64>(kick, m_), du_);
          TTG_CUDA(cudaMemcpyAsync(Um_ + m_ * nn, du_, sizeof(double) * m_ * mm,
                                   cudaMemcpyDeviceToDevice, s_));
          pad_rows_kernel<<<eb((nn + mm) * rr), 256, 0, s_>>>(nn, mm, rr, Rm_, tmp_);
          TTG_CHECK_LAUNCH();
          rnew = std::min<i64>(m_, nn + mm);
          qr(m_, nn + mm, Um_, Rq_);                                      // Rq (rnew x nn+mm)
          gemm((int)rnew, (int)rr, nn + mm, Rq_, 1, rnew, tmp_, 1, nn + mm, Rm_, 1, rnew);
        }
      } else {
        TTG_CUDA(cudaMemcpyAsync(Um_, x_[i], sizeof(double) * m_ * rr, cudaMemcpyDeviceToDevice, s_));
        qr(m_, rr, Um_, Rm_);
      }
      TTG_REQUIRE(rnew <= cap_[i + 1], "amen: rank capacity exceeded");
      TTG_CUDA(cudaMemcpyAsync(x_[i], Um_, sizeof(double) * m_ * rnew, cudaMemcpyDeviceToDevice, s_));
      gemm((int)rnew, (int)p, (int)rr, Rm_, 1, rnew, x_[i + 1], 1, rr, tmp_, 1, rnew);
      TTG_CUDA(cudaMemcpyAsync(x_[i + 1], tmp_, sizeof(double) * rnew * p, cudaMemcpyDeviceToDevice, s_));
      rx_[i + 1] = rnew;
      upd_left(i);
    }
    if (dir < 0 && i > 0) {
      // truncation and kick to the left (:900-1040)
      const i64 m_ = nk * r2, rl = r1, p = rx_[i - 1] * n_[i - 1];
      i64 rnew = std::min(m_, rl);
      if (kick > 0 || kick == -1) {
        const int rmin = (int)std::min(m_, rl);
        svd_jacobi((int)rl, (int)m_, x_[i], U_, S_, Vt_, svScr_, ired_ + 16, s_);
        scale_cols_f64(rl, rmin, U_, rl, S_, s_);                        // L = U diag(s)
        int nn = scan(i, rmin, U_, rl, Vt_, rmin, rl, m_, rhs_, nrhs, res_new, eps2);
        nn = (int)std::min<i64>(nn, P_.rmax);
        // Cm = Vt[:nn, :]^T (m_ x nn), Rm = L[:, :nn]^T (nn x rl)
        copy_rows_f64(rmin, nn, m_, Vt_, tmp_, s_);
        transpose_f64(nn, m_, tmp_, Um_, s_);
        transpose_f64(rl, nn, U_, Rm_, s_);
        rnew = nn;
        if (kick > 0) {
          // kick_block ((ry1 + rl ra1) x m_) = [Y-projection; dbfun3_right]
          bfun3_right(i, x_[i], tC_);
          concat_rows_kernel<<<eb((ry[i] + rl * ra[i]) * m_), 256, 0, s_>>>(ry[i], rl * ra[i], m_,
                                                                          kickY_, tC_, kickB_);
          TTG_CHECK_LAUNCH();
          const int mm = uchol(false, rl * ra[i] + ry[i], m_, kickB_, (int)std::min<i64>(kick, m_), du_);
          TTG_CUDA(cudaMemcpyAsync(Um_ + m_ * nn, du_, sizeof(double) * m_ * mm,
                                   cudaMemcpyDeviceToDevice, s_));
          pad_rows_kernel<<<eb((nn + mm) * rl), 256, 0, s_>>>(nn, mm, rl, Rm_, tmp_);
          TTG_CHECK_LAUNCH();
          rnew = std::min<i64>(m_, nn + mm);
          qr(m_, nn + mm, Um_, Rq_);
          gemm((int)rnew, (int)rl, nn + mm, Rq_, 1, rnew, tmp_, 1, nn + mm, Rm_, 1, rnew);
        }
      } else {
        transpose_f64(rl, m_, x_[i], Um_, s_);                          // m_ x rl
        qr(m_, rl, Um_, Rm_);
      }
      TTG_REQUIRE(rnew <= cap_[i], "amen: rank capacity exceeded");
      transpose_f64(m_, rnew, Um_, x_[i], s_);                          // rnew x m_
      // core i-1 (p x rl) * Rm^T (rl x rnew)
      gemm((int)p, (int)rnew, (int)rl, x_[i - 1], 1, p, Rm_, rnew, 1, tmp_, 1, p);
      TTG_CUDA(cudaMemcpyAsync(x_[i - 1], tmp_, sizeof(double) * p * rnew, cudaMemcpyDeviceToDevice, s_));
      rx_[i] = rnew;
      upd_right(i);
    }
    if ((dir > 0 && i == d - 1) || (dir < 0 && i == 0)) {
      last_res = res_max;
      if (P_.verb > 0) {
        i64 mr = *std::max_element(rx_.begin(), rx_.end());
        fprintf(stderr, "als_fort: iteration:%d(%d) max(ry):%lld err_max:%.3e res_max:%.3e\n", swp,
                dir, (long long)mr, err_max, res_max);
      }
    }
    if (dir > 0 && i == d - 1) {
      dir = -1;
      i += 1;
      if (kick < 0) break;
      if (res_max < P_.eps) kick = -1;
      ++swp;
      err_max = 0.0;
      res_max = 0.0;
    }
    if (dir < 0 && i == 0) {
      if (kick < 0) break;
      if (res_max < P_.eps) kick = -1;
      dir = 1;
      i -= 1;
      err_max = 0.0;
      res_max = 0.0;
    }
    i += dir;
  }
  sync();
  i64 tot = 0;
  for (int k = 0; k < d; ++k) tot += rx_[k] * n_[k] * rx_[k + 1];
  out.cores.resize(tot);
  i64 off = 0;
  for (int k = 0; k < d; ++k) {
    const i64 sz = rx_[k] * n_[k] * rx_[k + 1];
    TTG_CUDA(cudaMemcpyAsync(out.cores.data() + off, x_[k], sizeof(double) * sz,
                             cudaMemcpyDeviceToHost, s_));
    off += sz;
  }
  sync();
  out.rx = rx_;
  out.sweeps = std::min(swp, P_.nswp);
  out.res_max = last_res;
  out.matvecs = nmv_;
}

// ---------------------------------------------------------------------------
// tt_mvk4 (tt_adapt_als.f90:67-500): y ~ A x by alternating projections.
// The interfaces phi = Y'AX (ry, rx, ra) come from dphi_left/right with x and
// y different tensors; the projected core is dbfun3 of x's core; going left
// the kept rank is my_chop3 of the SVD plus a kick of min(kickrank, n ry2)
// incremental-Cholesky vectors of dbfun3_right (the right-going kick is off
// in the reference, so none is added going right).
// ---------------------------------------------------------------------------
struct MvkParams {
  int d;
  std::vector<i64> n, m, rx, ra, ry;
  const double *crA, *crX, *crY0;
  double eps;
  i64 rmax;
  int kick, nswp, verb;
};

class MvkSolver {
 public:
  MvkSolver(ttg_ctx* ctx, const MvkParams& P) : P_(P), s_(ctx->stream) {}
  void run(AmenOut& out);

 private:
  MvkParams P_;
  cudaStream_t s_;
  Arena mem_;
  std::vector<i64> ry_, cap_;
  std::vector<double*> y_, A_, X_, phi_;
  size_t tau_n_ = 0;   // elements of tau_
  double *cur_, *diff_, *red_, *U_, *S_, *Vt_, *svScr_, *Um_, *Rm_, *Rq_, *tmp_, *full_, *tA_,
      *tB_, *scr_, *du_, *dd_, *small_, *tau_;
  int* ired_;
  double* h_ = nullptr;

  LocalDims dims(int i) const {
    return LocalDims{P_.rx[i], P_.m[i], P_.rx[i + 1], ry_[i], P_.n[i], ry_[i + 1], P_.ra[i], P_.ra[i + 1]};
  }
  void sync() { TTG_CUDA(cudaStreamSynchronize(s_)); }
  void gemm(int M, int N, int K, const double* A, i64 sAm, i64 sAk, const double* B, i64 sBk,
            i64 sBn, double* C, i64 sCm, i64 sCn) {
    GemmF64 g;
    g.M = M; g.N = N; g.K = K;
    g.A = A; g.sAm = sAm; g.sAk = sAk;
    g.B = B; g.sBk = sBk; g.sBn = sBn;
    g.C = C; g.sCm = sCm; g.sCn = sCn;
    gemm_f64(g, s_);
  }
  double norm2(const double* v, i64 n) {
    sqnorm_cols(n, v, n, 1, red_, s_);
    TTG_CUDA(cudaMemcpyAsync(h_, red_, sizeof(double), cudaMemcpyDeviceToHost, s_));
    sync();
    return std::sqrt(h_[0]);
  }
  // my_chop3 of the rmin singular values in S_, capped at rmax
  int chop(int rmin, double eps2) {
    TTG_REQUIRE(rmin <= 4096, "tt_mvk4: rank above 4096");
    TTG_CUDA(cudaMemcpyAsync(h_, S_, sizeof(double) * rmin, cudaMemcpyDeviceToHost, s_));
    sync();
    return (int)std::min<i64>(ttg_my_chop3(rmin, h_, eps2), P_.rmax);
  }
};

void MvkSolver::run(AmenOut& out) {
  const int d = P_.d;
  const auto& n = P_.n;
  const auto& m = P_.m;
  const auto& rx = P_.rx;
  const auto& ra = P_.ra;
  ry_ = P_.ry;
  TTG_REQUIRE(d >= 2, "tt_mvk4: d must be >= 2");
  TTG_REQUIRE(rx[0] == 1 && rx[d] == 1 && ry_[0] == 1 && ry_[d] == 1 && ra[0] == 1 && ra[d] == 1,
              "boundary ranks must be 1");
  const double eps2 = P_.eps / std::sqrt((double)d);
  const int kick = P_.kick;
  const int kpad = std::max(kick, 0);
  std::vector<i64> left(d + 1, 1), right(d + 1, 1);
  for (int k = 1; k <= d; ++k) left[k] = std::min<i64>(left[k - 1] * n[k - 1], 1ll << 40);
  for (int k = d - 1; k >= 0; --k) right[k] = std::min<i64>(right[k + 1] * n[k], 1ll << 40);
  cap_.assign(d + 1, 1);
  for (int k = 1; k < d; ++k)
    cap_[k] = std::max(ry_[k], std::min(P_.rmax, std::min(left[k], right[k])) + kpad);
  i64 Nmax = 1, Mmax = 1, cmax = 1, T = 1, FB = 1, PH = 1, SVDU = 1;
  size_t scr = 0, svs = 0;
  for (int k = 0; k <= d; ++k) cmax = std::max(cmax, cap_[k]);
  for (int k = 0; k < d; ++k) {
    const i64 c1 = cap_[k], c2 = cap_[k + 1], nk = n[k];
    Nmax = std::max(Nmax, c1 * nk * c2);
    Mmax = std::max(Mmax, std::max(c1 * nk, nk * c2));
    LocalDims L{rx[k], m[k], rx[k + 1], c1, nk, c2, ra[k], ra[k + 1]};
    scr = std::max(scr, bfun3_f64_scratch(L, 1));
    scr = std::max(scr, phi_f64_scratch(L));
    T = std::max(T, std::max(rx[k] * m[k] * ra[k + 1] * c2, ra[k] * nk * c2 * rx[k]));
    FB = std::max(FB, rx[k] * ra[k] * nk * c2);
    svs = std::max(svs, svd_scratch((int)(c1 * nk), (int)c2));
    svs = std::max(svs, svd_scratch((int)c1, (int)(nk * c2)));
    SVDU = std::max(SVDU, std::max(c1 * nk, nk * c2) * std::min(std::max(c1 * nk, nk * c2), std::max(c1, c2)));
  }
  for (int k = 0; k <= d; ++k) PH = std::max(PH, cap_[k] * rx[k] * ra[k]);
  const i64 M2 = std::max(Nmax, Mmax * (cmax + kpad));
  const i64 R2 = (cmax + kpad) * (cmax + kpad);
  tau_n_ = std::max<size_t>(8192, qr_work_elems(cmax + kpad, cmax + kpad));
  i64 at = 0, xt = 0;
  for (int k = 0; k < d; ++k) {
    at += ra[k] * n[k] * m[k] * ra[k + 1];
    xt += rx[k] * m[k] * rx[k + 1];
  }
  size_t total = al8(at) + al8(xt);
  for (int k = 0; k < d; ++k) total += al8(cap_[k] * n[k] * cap_[k + 1]);
  for (int k = 0; k <= d; ++k) total += al8(std::max<i64>(1, cap_[k] * rx[k] * ra[k]));
  total += 2 * al8(Nmax) + al8(64) + 2 * al8(SVDU) + al8(4096) + svs + 256 + al8(M2) +
           2 * al8(R2) + al8(M2) + al8(FB) + 2 * al8(T) + scr + 256 + al8(Mmax * 16) +
           al8(Mmax) + al8(1024) + al8(tau_n_) + al8(64) + (1 << 16);
  mem_.alloc(total);
  double* dA = mem_.take(at);
  double* dX = mem_.take(xt);
  A_.resize(d); X_.resize(d); y_.resize(d); phi_.resize(d + 1);
  {
    i64 oa = 0, ox = 0;
    for (int k = 0; k < d; ++k) {
      A_[k] = dA + oa; oa += ra[k] * n[k] * m[k] * ra[k + 1];
      X_[k] = dX + ox; ox += rx[k] * m[k] * rx[k + 1];
    }
  }
  for (int k = 0; k < d; ++k) y_[k] = mem_.take(cap_[k] * n[k] * cap_[k + 1]);
  for (int k = 0; k <= d; ++k) phi_[k] = mem_.take(std::max<i64>(1, cap_[k] * rx[k] * ra[k]));
  cur_ = mem_.take(Nmax); diff_ = mem_.take(Nmax);
  red_ = mem_.take(64);
  U_ = mem_.take(SVDU); Vt_ = mem_.take(SVDU); S_ = mem_.take(4096);
  svScr_ = (double*)mem_.take(svs / sizeof(double) + 1);
  Um_ = mem_.take(M2); Rm_ = mem_.take(R2); Rq_ = mem_.take(R2); tmp_ = mem_.take(M2);
  full_ = mem_.take(FB); tA_ = mem_.take(T); tB_ = mem_.take(T);
  scr_ = (double*)mem_.take(scr / sizeof(double) + 1);
  du_ = mem_.take(Mmax * 16); dd_ = mem_.take(Mmax); small_ = mem_.take(1024);
  tau_ = mem_.take(tau_n_);
  ired_ = (int*)mem_.take(64);
  TTG_CUDA(cudaMallocHost(&h_, 4096 * sizeof(double)));
  struct HG { double* p; ~HG() { if (p) cudaFreeHost(p); } } hg{h_};
  const UcholWork UW{small_, dd_, tmp_, tau_, h_, ired_};

  TTG_CUDA(cudaMemcpyAsync(dA, P_.crA, sizeof(double) * at, cudaMemcpyHostToDevice, s_));
  TTG_CUDA(cudaMemcpyAsync(dX, P_.crX, sizeof(double) * xt, cudaMemcpyHostToDevice, s_));
  {
    i64 oy = 0;
    for (int k = 0; k < d; ++k) {
      const i64 sz = ry_[k] * n[k] * ry_[k + 1];
      TTG_CUDA(cudaMemcpyAsync(y_[k], P_.crY0 + oy, sizeof(double) * sz, cudaMemcpyHostToDevice, s_));
      oy += sz;
    }
  }
  fill_f64(phi_[0], 1, 1.0, s_);
  fill_f64(phi_[d], 1, 1.0, s_);
  auto upd_left = [&](int i) { phi_left_f64(dims(i), phi_[i], A_[i], X_[i], y_[i], phi_[i + 1], scr_, s_); };
  auto upd_right = [&](int i) { phi_right_f64(dims(i), phi_[i + 1], A_[i], X_[i], y_[i], phi_[i], scr_, s_); };

  // QR left to right, interfaces (tt_adapt_als.f90:190-223)
  for (int i = 0; i + 1 < d; ++i) {
    const i64 m_ = ry_[i] * n[i], rr = ry_[i + 1], p = n[i + 1] * ry_[i + 2];
    const i64 rnew = std::min(m_, rr);
    TTG_CUDA(cudaMemcpyAsync(Um_, y_[i], sizeof(double) * m_ * rr, cudaMemcpyDeviceToDevice, s_));
    qr_householder((int)m_, (int)rr, Um_, Rq_, tau_, tau_n_, s_);
    TTG_CUDA(cudaMemcpyAsync(y_[i], Um_, sizeof(double) * m_ * rnew, cudaMemcpyDeviceToDevice, s_));
    gemm((int)rnew, (int)p, (int)rr, Rq_, 1, rnew, y_[i + 1], 1, rr, tmp_, 1, rnew);
    TTG_CUDA(cudaMemcpyAsync(y_[i + 1], tmp_, sizeof(double) * rnew * p, cudaMemcpyDeviceToDevice, s_));
    ry_[i + 1] = rnew;
    upd_left(i);
  }

  double err_max = 0.0;
  int i = d - 1, dir = -1, swp = 1;
  while (swp <= P_.nswp) {
    const LocalDims L = dims(i);
    const i64 N = L.ysize();
    bfun3_f64(L, phi_[i], A_[i], phi_[i + 1], X_[i], cur_, 1, scr_, s_);
    sub_kernel<<<eb(N), 256, 0, s_>>>(N, y_[i], cur_, diff_);
    TTG_CHECK_LAUNCH();
    const double err = norm2(diff_, N) / norm2(cur_, N);
    err_max = std::max(err_max, err);
    if (P_.verb > 1)
      fprintf(stderr, "tt_mvk4: iteration:[%d,%d] err:%.3e ry(i):%lld err_max:%.3e\n", swp, i + 1, err,
              (long long)ry_[i], err_max);
    if (dir > 0 && i < d - 1) {
      // truncation to the right (:269-345)
      const i64 m_ = ry_[i] * n[i], rr = ry_[i + 1], p = n[i + 1] * ry_[i + 2];
      i64 rnew = std::min(rr, m_);
      if (kick > 0) {
        const int rmin = (int)std::min(m_, rr);
        svd_jacobi((int)m_, (int)rr, cur_, U_, S_, Vt_, svScr_, ired_ + 16, s_);
        const int nn = chop(rmin, eps2);
        scale_rows_f64(rmin, rr, Vt_, rmin, S_, s_);                     // diag(s) Vt
        TTG_CUDA(cudaMemcpyAsync(Um_, U_, sizeof(double) * m_ * nn, cudaMemcpyDeviceToDevice, s_));
        copy_rows_f64(rmin, nn, rr, Vt_, Rm_, s_);
        rnew = nn;
      } else {
        TTG_CUDA(cudaMemcpyAsync(Um_, cur_, sizeof(double) * m_ * rr, cudaMemcpyDeviceToDevice, s_));
        qr_householder((int)m_, (int)rr, Um_, Rm_, tau_, tau_n_, s_);
      }
      TTG_REQUIRE(rnew <= cap_[i + 1], "tt_mvk4: rank capacity exceeded");
      TTG_CUDA(cudaMemcpyAsync(y_[i], Um_, sizeof(double) * m_ * rnew, cudaMemcpyDeviceToDevice, s_));
      gemm((int)rnew, (int)p, (int)rr, Rm_, 1, rnew, y_[i + 1], 1, rr, tmp_, 1, rnew);
      TTG_CUDA(cudaMemcpyAsync(y_[i + 1], tmp_, sizeof(double) * rnew * p, cudaMemcpyDeviceToDevice, s_));
      ry_[i + 1] = rnew;
      upd_left(i);
    }
    if (dir < 0 && i > 0) {
      // truncation and kick to the left (:351-434)
      const i64 m_ = n[i] * ry_[i + 1], rl = ry_[i], p = ry_[i - 1] * n[i - 1];
      i64 rnew = std::min(m_, rl);
      if (kick > 0) {
        const int rmin = (int)std::min(m_, rl);
        svd_jacobi((int)rl, (int)m_, cur_, U_, S_, Vt_, svScr_, ired_ + 16, s_);
        const int nn = chop(rmin, eps2);
        scale_cols_f64(rl, rmin, U_, rl, S_, s_);                        // U diag(s)
        // Cm = Vt[:nn, :]^T (m_ x nn), Rm = (U diag(s))[:, :nn]^T (nn x rl)
        copy_rows_f64(rmin, nn, m_, Vt_, tmp_, s_);
        transpose_f64(nn, m_, tmp_, Um_, s_);
        transpose_f64(rl, nn, U_, Rm_, s_);
        // kick: dbfun3_right (rx1 ra1) x m_, incremental Cholesky 'N'
        bfun3_right_run(P_.rx[i], m[i], P_.rx[i + 1], n[i], ry_[i + 1], ra[i], ra[i + 1], A_[i],
                        phi_[i + 1], X_[i], full_, tA_, tB_, s_);
        const int mm = uchol_run(false, P_.rx[i] * ra[i], m_, full_, (int)std::min<i64>(kick, m_),
                                 du_, UW, s_);
        TTG_CUDA(cudaMemcpyAsync(Um_ + m_ * nn, du_, sizeof(double) * m_ * mm,
                                 cudaMemcpyDeviceToDevice, s_));
        pad_rows_kernel<<<eb((nn + mm) * rl), 256, 0, s_>>>(nn, mm, rl, Rm_, tmp_);
        TTG_CHECK_LAUNCH();
        rnew = std::min<i64>(m_, nn + mm);
        qr_householder((int)m_, nn + mm, Um_, Rq_, tau_, tau_n_, s_);
        gemm((int)rnew, (int)rl, nn + mm, Rq_, 1, rnew, tmp_, 1, nn + mm, Rm_, 1, rnew);
      } else {
        transpose_f64(rl, m_, cur_, Um_, s_);                            // m_ x rl
        qr_householder((int)m_, (int)rl, Um_, Rm_, tau_, tau_n_, s_);
      }
      TTG_REQUIRE(rnew <= cap_[i], "tt_mvk4: rank capacity exceeded");
      transpose_f64(m_, rnew, Um_, y_[i], s_);                           // rnew x m_
      gemm((int)p, (int)rnew, (int)rl, y_[i - 1], 1, p, Rm_, rnew, 1, tmp_, 1, p);
      TTG_CUDA(cudaMemcpyAsync(y_[i - 1], tmp_, sizeof(double) * p * rnew, cudaMemcpyDeviceToDevice, s_));
      ry_[i] = rnew;
      upd_right(i);
    }
    if (dir > 0 && i == d - 1) {
      TTG_CUDA(cudaMemcpyAsync(y_[i], cur_, sizeof(double) * N, cudaMemcpyDeviceToDevice, s_));
      if (P_.verb > 0)
        fprintf(stderr, "tt_mvk4: iteration:%d(%d) max(ry):%lld err_max:%.3e\n", swp, dir,
                (long long)*std::max_element(ry_.begin(), ry_.end()), err_max);
      dir = -1;
      i += 1;
      ++swp;
      if (err_max < P_.eps) break;
      err_max = 0.0;
    }
    if (dir < 0 && i == 0) {
      TTG_CUDA(cudaMemcpyAsync(y_[i], cur_, sizeof(double) * N, cudaMemcpyDeviceToDevice, s_));
      dir = 1;
      i -= 1;
    }
    i += dir;
  }
  sync();
  i64 tot = 0;
  for (int k = 0; k < d; ++k) tot += ry_[k] * n[k] * ry_[k + 1];
  out.cores.resize(tot);
  i64 off = 0;
  for (int k = 0; k < d; ++k) {
    const i64 sz = ry_[k] * n[k] * ry_[k + 1];
    TTG_CUDA(cudaMemcpyAsync(out.cores.data() + off, y_[k], sizeof(double) * sz,
                             cudaMemcpyDeviceToHost, s_));
    off += sz;
  }
  sync();
  out.rx = ry_;
  out.sweeps = std::min(swp, P_.nswp);
  out.res_max = err_max;
  out.matvecs = 0;
}

}  // namespace ttg

using namespace ttg;

// dtt_amen_solve (ttamen.f90:29-252) with flat arrays: the dtt type of the
// reference is not C-interoperable, so this entry point takes the packed cores
extern "C" int ttg_dtt_amen_solve(ttg_ctx* ctx, ttg_int d, const ttg_int* n, const ttg_int* m,
                                  const ttg_int* ry, const ttg_int* ra, const double* crA,
                                  const double* crY, const double* crX0, ttg_int* rx, double eps,
                                  ttg_int rmax, ttg_int kickrank, ttg_int nswp, int verb,
                                  int method) {
  if (!ctx) return TTG_ERR_ARG;
  try {
    TTG_CUDA(cudaSetDevice(ctx->device));
    TTG_REQUIRE(d > 1 && n && m && ry && ra && crA && crY && crX0 && rx, "null argument");
    TTG_REQUIRE(method == TTG_METHOD_PLAIN || method == TTG_METHOD_SPLIT, "unknown method");
    for (int k = 0; k < d; ++k) TTG_REQUIRE(n[k] == m[k], "amen needs square cores (n == m)");
    AmenParams P;
    P.method = method;
    P.d = (int)d;
    P.n.assign(n, n + d);
    P.ry.assign(ry, ry + d + 1);
    P.ra.assign(ra, ra + d + 1);
    P.rx.assign(rx, rx + d + 1);
    P.crA = crA; P.crY = crY; P.crX0 = crX0;
    P.tol = eps;
    P.rmax = rmax > 0 ? rmax : (1ll << 30);
    P.kick = kickrank >= 0 ? (int)kickrank : 4;
    P.nswp = nswp > 0 ? (int)nswp : 20;
    P.local_iters = 2;
    P.local_restart = 40;
    P.max_full_size = 50;
    P.verb = verb;
    P.seed = 0;
    long long l0 = g_launches;
    AmenOut out;
    AmenSolver solver(ctx, P);
    solver.run(out);
    for (int k = 0; k <= d; ++k) rx[k] = out.rx[k];
    ctx->result_core = std::move(out.cores);
    ctx->zresult_core.clear();
    ctx->stat_matvecs = out.matvecs;
    ctx->stat_sweeps = out.sweeps;
    ctx->stat_res = out.res_max;
    ctx->stat_launches = g_launches - l0;
  } catch (const ttg::Error& e) {
    ctx->last_error = e.msg;
    return e.code;
  }
  return TTG_OK;
}

// tt_amen_solve (tt_adapt_als.f90:513-1132)
extern "C" int ttg_amen_solve(ttg_ctx* ctx, ttg_int d, const ttg_int* n, const ttg_int* m,
                              const ttg_int* ry, const ttg_int* ra, const double* crA,
                              const double* crY, const double* crX0, ttg_int* rx, double eps,
                              ttg_int kickrank, ttg_int nswp, int verb, char prec,
                              ttg_int nrestart, ttg_int niters, ttg_int rmax, int method) {
  if (!ctx) return TTG_ERR_ARG;
  try {
    TTG_CUDA(cudaSetDevice(ctx->device));
    TTG_REQUIRE(d > 1 && n && m && ry && ra && crA && crY && crX0 && rx, "null argument");
    TTG_REQUIRE(method == TTG_METHOD_PLAIN, "amen: only the FP64 method is built");
    TTG_REQUIRE(prec == 'n' || prec == 'N' || prec == 0 || jac_type(prec),
                "amen: prec must be 'n', 'c', 'l' or 'r'");
    for (int k = 0; k < d; ++k) TTG_REQUIRE(n[k] == m[k], "amen needs square cores (n == m)");
    TTG_REQUIRE(kickrank <= 16, "amen: kickrank > 16");
    AlsParams P;
    P.d = (int)d;
    P.n.assign(n, n + d);
    P.ry.assign(ry, ry + d + 1);
    P.ra.assign(ra, ra + d + 1);
    P.rx.assign(rx, rx + d + 1);
    P.crA = crA; P.crY = crY; P.crX0 = crX0;
    P.eps = eps;
    P.rmax = rmax > 0 ? rmax : (1ll << 40);
    P.kick = (int)kickrank;
    P.nswp = nswp > 0 ? (int)nswp : 20;
    P.nrestart = nrestart > 0 ? (int)nrestart : 40;
    P.niters = niters > 0 ? (int)niters : 2;
    P.verb = verb;
    P.prec = jac_type(prec);
    long long l0 = g_launches;
    AmenOut out;
    AlsSolver solver(ctx, P);
    solver.run(out);
    for (int k = 0; k <= d; ++k) rx[k] = out.rx[k];
    ctx->result_core = std::move(out.cores);
    ctx->zresult_core.clear();
    ctx->stat_matvecs = out.matvecs;
    ctx->stat_sweeps = out.sweeps;
    ctx->stat_res = out.res_max;
    ctx->stat_launches = g_launches - l0;
  } catch (const ttg::Error& e) {
    ctx->last_error = e.msg;
    return e.code;
  }
  return TTG_OK;
}

// tt_mvk4 (tt_adapt_als.f90:67-500)
extern "C" int ttg_mvk4(ttg_ctx* ctx, ttg_int d, const ttg_int* n, const ttg_int* m,
                        const ttg_int* rx, const ttg_int* ra, const double* crA, const double* crX,
                        const double* crY0, ttg_int* ry, double eps, ttg_int rmax, ttg_int kickrank,
                        ttg_int nswp, int verb) {
  if (!ctx) return TTG_ERR_ARG;
  try {
    TTG_CUDA(cudaSetDevice(ctx->device));
    TTG_REQUIRE(d > 1 && n && m && rx && ra && crA && crX && crY0 && ry, "null argument");
    TTG_REQUIRE(rmax > 0, "tt_mvk4: rmax must be positive");
    TTG_REQUIRE(kickrank <= 16, "tt_mvk4: kickrank > 16");
    MvkParams P;
    P.d = (int)d;
    P.n.assign(n, n + d);
    P.m.assign(m, m + d);
    P.rx.assign(rx, rx + d + 1);
    P.ra.assign(ra, ra + d + 1);
    P.ry.assign(ry, ry + d + 1);
    P.crA = crA; P.crX = crX; P.crY0 = crY0;
    P.eps = eps;
    P.rmax = rmax;
    P.kick = (int)kickrank;
    P.nswp = nswp > 0 ? (int)nswp : 20;
    P.verb = verb;
    long long l0 = g_launches;
    AmenOut out;
    MvkSolver solver(ctx, P);
    solver.run(out);
    for (int k = 0; k <= d; ++k) ry[k] = out.rx[k];
    ctx->result_core = std::move(out.cores);
    ctx->zresult_core.clear();
    ctx->stat_matvecs = 0;
    ctx->stat_sweeps = out.sweeps;
    ctx->stat_res = out.res_max;
    ctx->stat_launches = g_launches - l0;
  } catch (const ttg::Error& e) {
    ctx->last_error = e.msg;
    return e.code;
  }
  return TTG_OK;
}
