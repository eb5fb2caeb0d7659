// Plain (FP64 / complex128) local operator and interface updates.
//
//   bfun3      y = Phi1 * A * Phi2 * x            ttals.f90:9-32   (dbfun3)
//   phi_left   Phi1' = sum Phi1 y A x             ttals.f90:203-227 (dphi_left)
//   phi_right  Phi2' = sum x Phi2 A y             ttals.f90:150-173 (dphi_right)
//   phi2_*     Y'X projections without A          ttals.f90:260-314
//   fullmat    dense local matrix                 tt_eigb.f90:88-105 (d2d_fullmat)
//   z*         complex versions, y conjugated     ttals.f90:34-57,85-108,176-256
//
// Each product is three GEMMs.  The reference transposes its intermediates
// between the GEMMs (dtransp, ttals.f90:22,26); here the intermediates are
// laid out so that every GEMM reads and writes them with unit stride:
//   T1[b1, j, a2, c2]   = x * Phi2              (rx1*m  x ra2*ry2)
//   T2[b1, a1, i, c2]   = A (x) T1, one GEMM per c2
//   y [c1, i, c2]       = Phi1 * T2             (ry1 x n*ry2)
// so the transposes cost nothing.  Large products run on the tensor cores
// (ttg_oz.cu: FP64 by error-free splitting), the others through gemm_f64 / gemm_z.
#include "ttg_common.cuh"
#include <algorithm>

namespace ttg {

// Scratch layout: two FP64 (or complex) intermediates, then the workspace of
// the split products (ttg_oz.cu) that the sizes can reach.
static size_t al256(size_t b) { return (b + 255) & ~size_t(255); }
// rows of Q = A Phi2 (see bfun3_f64): only for small modes, and only where a
// split product can follow
static i64 q_size(const LocalDims& L, int nvec) {
  if (L.n * L.m > 4 || oz_bytes(L.rx1 * nvec, L.n * L.ry2 * L.ra1, L.m * L.rx2, false) == 0) return 0;
  return L.n * L.ry2 * L.ra1 * L.m * L.rx2;
}
// group maxima and tables of a call's split products, whichever they are
static size_t stat_bytes(const LocalDims& L, int nvec) {
  const i64 K = std::max({L.rx2, L.m * L.ra2, L.rx1 * L.ra1, L.m * L.rx2, L.ry1, L.ra1 * L.n,
                          L.ra2 * L.ry2, L.n * L.ry2, L.rx1 * L.m});
  const i64 r = std::max(L.ra1, L.ra2);
  const i64 rows = std::max({L.rx1 * L.m * nvec + L.ra2 * L.ry2, L.rx1 * L.ry2 * nvec + L.ra1 * L.n,
                             L.rx1 * L.ry2 * nvec + L.ra2 * L.m, L.ry1 + L.n * L.ry2 * nvec,
                             L.rx1 * nvec + L.n * L.ry2 * L.ra1, L.rx1 * L.ra1 + L.n * L.ry2 * nvec,
                             L.rx1 * L.m * nvec + L.rx2, L.ry2 * L.ra2 + L.rx2, L.rx1 * L.ra1 + L.ry1});
  return kOzProducts * oz_stat_bytes(rows, K, r + std::min(nvec, kOzMaxVec), r);
}
static size_t bfun3_oz_bytes(const LocalDims& L, int nvec, bool cplx) {
  size_t b = std::max({oz_bytes(L.rx1 * L.m * nvec, L.ra2 * L.ry2, L.rx2, cplx),
                       oz_bytes(L.rx1 * L.ry2 * nvec, L.ra1 * L.n, L.m * L.ra2, cplx),
                       oz_bytes(L.ry1, L.n * L.ry2 * nvec, L.rx1 * L.ra1, cplx)});
  if (!cplx && L.n * L.m <= 4)
    b = std::max(b, oz_bytes(L.rx1 * nvec, L.n * L.ry2 * L.ra1, L.m * L.rx2, false));
  if (cplx)   // the adjoint's products
    b = std::max({b, oz_bytes(L.rx1 * L.ra1, L.n * L.ry2 * nvec, L.ry1, true),
                  oz_bytes(L.rx1 * L.ry2 * nvec, L.m * L.ra2, L.ra1 * L.n, true),
                  oz_bytes(L.rx1 * L.m * nvec, L.rx2, L.ra2 * L.ry2, true)});
  return b > 0 ? b + stat_bytes(L, nvec) : 0;
}
static size_t bfun3_t_bytes(const LocalDims& L, int nvec) {
  return al256((size_t)(std::max(L.t1size() * nvec, q_size(L, nvec)) + L.t2size() * nvec) * sizeof(double));
}
size_t bfun3_f64_scratch(const LocalDims& L, int nvec) {
  return bfun3_t_bytes(L, nvec) + bfun3_oz_bytes(L, nvec, false);
}
static size_t bfun3_z_t_bytes(const LocalDims& L, int nvec) {
  return al256((size_t)(L.t1size() + L.t2size()) * nvec * sizeof(double2));
}
size_t bfun3_z_scratch(const LocalDims& L, int nvec) {
  return bfun3_z_t_bytes(L, nvec) + bfun3_oz_bytes(L, nvec, true);
}

static size_t phi_t_bytes(const LocalDims& L, size_t elem) {
  i64 a = std::max(L.t1size(), L.rx1 * L.ra1 * L.n * L.ry2);
  i64 b = std::max(L.t2size(), L.rx1 * L.m * L.ra2 * L.ry2);
  return al256((size_t)(a + b) * elem);
}
static size_t phi_oz_bytes(const LocalDims& L, bool cplx) {
  const size_t b = std::max({oz_bytes(L.rx1 * L.ra1, L.n * L.ry2, L.ry1, cplx),
                             oz_bytes(L.rx1 * L.ry2, L.m * L.ra2, L.ra1 * L.n, cplx),
                             oz_bytes(L.ry2 * L.ra2, L.rx2, L.rx1 * L.m, cplx),
                             oz_bytes(L.rx1 * L.ra1, L.ry1, L.n * L.ry2, cplx)});
  return std::max(bfun3_oz_bytes(L, 1, cplx), b > 0 ? b + stat_bytes(L, 1) : 0);
}
size_t phi_f64_scratch(const LocalDims& L) {
  return phi_t_bytes(L, sizeof(double)) + phi_oz_bytes(L, false);
}
size_t phi_z_scratch(const LocalDims& L) {
  return phi_t_bytes(L, sizeof(double2)) + phi_oz_bytes(L, true);
}

static void fp64_product(const GemmF64& g, cudaStream_t s) { gemm_f64(g, s); }
static void fp64_product(const GemmZ& g, cudaStream_t s) { gemm_z(g, s); }

// The products g[0..n) of a call, each on the tensor cores where that is faster
// (ws: their workspace, null for the FP64 kernels only).  Interfaces mix blocks of
// different scale along an operator rank (1 and 1/h^2 for a Laplacian), and the
// two factors of a product whose K runs over it mix them the opposite way, so the
// hints name that rank where it is in K (the split products divide it out of both
// factors) and where it is in the rows (each block's outputs have an accuracy of
// their own).
static size_t stat_of(const OzGemm& o) {
  return oz_stat_bytes((i64)o.M + o.N, o.K, o.gnA + o.gnB, o.kr);
}
template <class G>
static size_t products_bytes(const G* g, const OzHint* h, int n) {   // the workspace of just these
  size_t stat = 0, planes = 0;
  for (int i = 0; i < n; ++i) {
    OzGemm o;
    if (!oz_plan(g[i], h[i], &o)) continue;
    stat += stat_of(o);
    planes = std::max(planes, oz_bytes(o.M, o.N, o.K, o.cplx));
  }
  return stat + planes;
}
template <class G>
static void run_products(const G* g, const OzHint* h, int n, void* ws, cudaStream_t s) {
  OzGemm o[kOzProducts];
  const OzGemm* split[kOzProducts];
  bool on[kOzProducts];
  int ns = 0;
  char* p = (char*)ws;
  for (int i = 0; i < n; ++i) {
    on[i] = ws && oz_plan(g[i], h[i], &o[i]);
    if (!on[i]) continue;
    o[i].stat = p;
    p += stat_of(o[i]);
    split[ns++] = &o[i];
  }
  // the first split product forms the others' scales
  if (ns > 0 && split[0]->kr > 0) oz_prepare(split, 1, s);
  for (int i = 0; i < n; ++i) {
    const bool first = on[i] && &o[i] == split[0];
    if (on[i]) oz_gemm(o[i], p, split + 1, first ? ns - 1 : 0, s);
    else fp64_product(g[i], s);
  }
}
// K of a product over (inner part, operator rank) or (operator rank, inner part):
// scales by Phi1's blocks (Phi1[c1, b1, a1]) or Phi2's (Phi2[b2, a2, c2])
template <class T>
static void scale_by_phi1(OzHint& h, const LocalDims& L, const T* phi1, int norm, i64 kd) {
  h.phi = (const double*)phi1; h.inner = L.ry1 * L.rx1; h.outer = 1;
  h.kr = (int)L.ra1; h.kd = (int)kd; h.norm = norm;
}
template <class T>
static void scale_by_phi2(OzHint& h, const LocalDims& L, const T* phi2, int norm, i64 kd) {
  h.phi = (const double*)phi2; h.inner = L.rx2; h.outer = L.ry2;
  h.kr = (int)L.ra2; h.kd = (int)kd; h.norm = norm;
}
static void rows_of(OzHint& h, int side, i64 groups, i64 run) {
  h.side = side; h.groups = (int)groups; h.run = (int)run;
}

template <class G, class T>
static void stage1(G& g, OzHint& h, const LocalDims& L, const T* x, const T* phi2, T* T1, int nvec) {
  // T1 (rx1*m x ra2*ry2) = x (rx1*m x rx2) * phi2 (rx2 x ra2*ry2)
  g.M = (int)(L.rx1 * L.m); g.N = (int)(L.ra2 * L.ry2); g.K = (int)L.rx2;
  g.A = x;    g.sAm = 1; g.sAk = L.rx1 * L.m;
  g.B = phi2; g.sBk = 1; g.sBn = L.rx2;
  g.C = T1;   g.sCm = 1; g.sCn = L.rx1 * L.m;
  g.nb1 = 1; g.nb2 = nvec;
  g.bA2 = L.xsize(); g.bB2 = 0; g.bC2 = L.t1size();
  h.nvec = nvec;
  rows_of(h, 2, L.ra2, 0);
}

template <class G, class T>
static void stage2(G& g, OzHint& h, const LocalDims& L, const T* A, const T* T1, const T* phi2, T* T2, int nvec) {
  // per (c2, vec): T2[b1,(a1,i)] = sum_(j,a2) A[(a1,i),(j,a2)] T1[b1,(j,a2)]
  g.M = (int)(L.ra1 * L.n); g.N = (int)L.rx1; g.K = (int)(L.m * L.ra2);
  g.A = A;  g.sAm = 1; g.sAk = L.ra1 * L.n;
  g.B = T1; g.sBk = L.rx1; g.sBn = 1;
  g.C = T2; g.sCm = L.rx1; g.sCn = 1;
  g.nb1 = (int)L.ry2; g.nb2 = nvec;
  g.bA1 = 0; g.bA2 = 0;
  g.bB1 = L.rx1 * L.m * L.ra2; g.bB2 = L.t1size();
  g.bC1 = L.rx1 * L.ra1 * L.n; g.bC2 = L.t2size();
  h.nvec = nvec;
  rows_of(h, 1, L.ra1, 0);
  scale_by_phi2(h, L, phi2, -1, L.m);
}

template <class G, class T>
static void stage3(G& g, OzHint& h, const LocalDims& L, const T* phi1, const T* T2, T* y, int nvec) {
  // y (ry1 x n*ry2) = phi1 (ry1 x rx1*ra1) * T2 (rx1*ra1 x n*ry2)
  g.M = (int)L.ry1; g.N = (int)(L.n * L.ry2); g.K = (int)(L.rx1 * L.ra1);
  g.A = phi1; g.sAm = 1; g.sAk = L.ry1;
  g.B = T2;   g.sBk = 1; g.sBn = L.rx1 * L.ra1;
  g.C = y;    g.sCm = 1; g.sCn = L.ry1;
  g.nb1 = 1; g.nb2 = nvec;
  g.bA2 = 0; g.bB2 = L.t2size(); g.bC2 = L.ysize();
  h.nvec = nvec;
  scale_by_phi1(h, L, phi1, 1, L.rx1);
}

// Q[kq + KQ (i + n (c2 + ry2 a1))] = sum_a2 A(a1,i,j,a2) Phi2(b2,a2,c2), kq = j + m b2.
// One block per (c2, a1): its n m ra2 core entries in shared memory, then a
// thread per b2 forms the n m outputs of that b2 from one read of Phi2.  Bound
// by its FP64 FMAs (m n <= 4).
__global__ void __launch_bounds__(128) q_kernel(int m, int rx2, int n, int ry2, int ra1, int ra2,
                                                const double* __restrict__ A,
                                                const double* __restrict__ phi2,
                                                double* __restrict__ Q) {
  extern __shared__ double core[];                // [a2][i + n j]
  pdl_wait();
  const int c2 = blockIdx.x, a1 = blockIdx.y, nm = n * m;
  for (int e = threadIdx.x; e < nm * ra2; e += blockDim.x)
    core[e] = A[a1 + (i64)ra1 * e];
  __syncthreads();
  const double* p2 = phi2 + (i64)rx2 * ra2 * c2;
  double* q = Q + (i64)m * rx2 * n * (c2 + (i64)ry2 * a1);
  for (int b2 = threadIdx.x; b2 < rx2; b2 += blockDim.x) {
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    for (int a2 = 0; a2 < ra2; ++a2) {
      const double p = p2[b2 + (i64)rx2 * a2];
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (e < nm) v[e] = fma(core[a2 * nm + e], p, v[e]);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (e < nm) q[(i64)m * rx2 * (e % n) + e / n + (i64)m * b2] = v[e];
  }
  pdl_trigger();
}

// Small modes (spin chains) at sizes where the products run on the tensor
// cores: the middle contraction would then be most of the time (its K = m ra2
// is too small to split: 105 MFLOP of FP64, 91 us, at r = 256, block of 8,
// beside 46 us for each of the two large products).  Contracting the core into
// Phi2 first costs K_Q times ra2 FMAs per row instead (11 us there) and makes
// the first product n times larger.
struct QRoute {
  OzGemm g, o3;     // T2 = X Q, then the third product (on: as a split product)
  GemmF64 g3;
  bool on = false;
  size_t stat() const { return stat_of(g) + (on ? stat_of(o3) : 0); }
};
static bool bfun3_q_plan(const LocalDims& L, const double* phi1, const double* x, double* Q,
                         double* T2, double* y, int nvec, QRoute* q) {
  const i64 M = L.rx1 * nvec, N = L.n * L.ry2 * L.ra1, K = L.m * L.rx2;
  if (q_size(L, nvec) == 0 || !oz_fits(M, N, K, false)) return false;
  const double core = 2.0 * (double)(L.ra1 * L.n) * (double)(L.m * L.ra2) * (double)(L.ry2 * L.rx1) * nvec / 1.0e6;
  const double first = 2.0 * (double)(L.rx1 * L.m * nvec) * (double)(L.ra2 * L.ry2) * (double)L.rx2 / 1.0e6;
  const double general = 8.0 + core +
                         std::min(first, oz_us(L.rx1 * L.m * nvec, L.ra2 * L.ry2, L.rx2, false));
  const double build = 2.0 * (double)N * (double)K * (double)L.ra2 / 1.0e6 + 4.0;
  if (build + oz_us(M, N, K, false) >= general) return false;
  if (L.ra1 >= 65536 || L.n * L.m * L.ra2 > 4096) return false;   // grid and shared memory
  OzGemm& g = q->g;   // T2[b1,a1,i,c2,v] = sum_kq X_v[b1,kq] Q[(i,c2,a1),kq]
  g.M = (int)M; g.N = (int)N; g.K = (int)K;
  g.A = x; g.am = {(int)L.rx1, 1, L.xsize()}; g.ak = L.rx1;
  g.B = Q; g.bn = {(int)N, K, 0}; g.bk = 1;
  g.C = T2; g.cm = {(int)L.rx1, 1, L.t2size()}; g.cn = {(int)(L.n * L.ry2), L.rx1 * L.ra1, L.rx1};
  g.gdB = (int)(L.n * L.ry2); g.gnB = (int)L.ra1;
  if (nvec > 1 && nvec <= kOzMaxVec && L.rx1 >= 8) { g.gdA = (int)L.rx1; g.gnA = nvec; }
  else g.gdA = g.M;
  if ((L.ra1 > 1 && g.gdB < 8) || L.ra1 > kOzMaxGroups) return false;
  OzHint h3;
  stage3(q->g3, h3, L, phi1, T2, y, nvec);
  q->on = oz_plan(q->g3, h3, &q->o3);
  return true;
}
static bool bfun3_q(const LocalDims& L, const double* phi1, const double* A, const double* phi2,
                    const double* x, double* Q, double* T2, double* y, int nvec, void* ws,
                    cudaStream_t s) {
  QRoute q;
  if (!bfun3_q_plan(L, phi1, x, Q, T2, y, nvec, &q)) return false;
  const OzGemm* later = &q.o3;
  char* p = (char*)ws + q.stat();
  q.g.stat = ws;
  q.o3.stat = (char*)ws + stat_of(q.g);
  launch_pdl(q_kernel, dim3((unsigned)L.ry2, (unsigned)L.ra1), dim3(128),
             sizeof(double) * L.n * L.m * L.ra2, s, (int)L.m, (int)L.rx2, (int)L.n, (int)L.ry2,
             (int)L.ra1, (int)L.ra2, A, phi2, Q);
  oz_gemm(q.g, p, &later, q.on ? 1 : 0, s);
  if (q.on) oz_gemm(q.o3, p, nullptr, 0, s);
  else gemm_f64(q.g3, s);
  return true;
}

template <class G, class T>
static void bfun3_products(G* g, OzHint* h, const LocalDims& L, const T* phi1, const T* A, const T* phi2,
                           const T* x, T* T1, T* T2, T* y, int nvec) {
  stage1(g[0], h[0], L, x, phi2, T1, nvec);
  stage2(g[1], h[1], L, A, T1, phi2, T2, nvec);
  stage3(g[2], h[2], L, phi1, T2, y, nvec);
}

void bfun3_f64(const LocalDims& L, const double* phi1, const double* A, const double* phi2,
               const double* x, double* y, int nvec, double* scratch, cudaStream_t s, bool split) {
  const i64 t1 = split ? std::max(L.t1size() * nvec, q_size(L, nvec)) : L.t1size() * nvec;
  double* T1 = scratch;
  double* T2 = scratch + t1;
  void* ws = split ? (char*)scratch + bfun3_t_bytes(L, nvec) : nullptr;
  if (ws && bfun3_q(L, phi1, A, phi2, x, T1, T2, y, nvec, ws, s)) return;
  GemmF64 g[3];
  OzHint h[3];
  bfun3_products(g, h, L, phi1, A, phi2, x, T1, T2, y, nvec);
  run_products(g, h, 3, ws, s);
}

void bfun3_z(const LocalDims& L, const double2* phi1, const double2* A, const double2* phi2,
             const double2* x, double2* y, int nvec, double2* scratch, cudaStream_t s) {
  double2* T1 = scratch;
  double2* T2 = scratch + L.t1size() * nvec;
  GemmZ g[3];
  OzHint h[3];
  bfun3_products(g, h, L, phi1, A, phi2, x, T1, T2, y, nvec);
  run_products(g, h, 3, (char*)scratch + bfun3_z_t_bytes(L, nvec), s);
}

// Adjoint product (zbfun3_transp, ttals.f90:85-108): x has the y layout
// (ry1, n, ry2), output y has the x layout (rx1, m, rx2); y = B^H x.
static void transp_products(GemmZ* gs, OzHint* h, const LocalDims& L, const double2* phi1,
                            const double2* A, const double2* phi2, const double2* x, double2* R1,
                            double2* R2, double2* y, int nvec) {
  const i64 p1 = L.rx1 * L.ra1 * L.n * L.ry2;     // R1[b1,a1,i,c2]
  const i64 p2 = L.rx1 * L.m * L.ra2 * L.ry2;     // R2[b1,j,a2,c2]
  {
    GemmZ& g = gs[0];   // R1[(b1,a1),(i,c2)] = sum_c1 conj(phi1[c1,(b1,a1)]) x[c1,(i,c2)]
    g.M = (int)(L.rx1 * L.ra1); g.N = (int)(L.n * L.ry2); g.K = (int)L.ry1;
    g.A = phi1; g.sAm = L.ry1; g.sAk = 1; g.conjA = true;
    g.B = x; g.sBk = 1; g.sBn = L.ry1;
    g.C = R1; g.sCm = 1; g.sCn = L.rx1 * L.ra1;
    g.nb2 = nvec; g.bB2 = L.ysize(); g.bC2 = p1;
    rows_of(h[0], 1, L.ra1, L.rx1);
  }
  {
    GemmZ& g = gs[1];   // per (c2, vec): R2[b1,(j,a2)] = sum_p conj(A[p,(j,a2)]) R1[b1,p]
    g.M = (int)(L.m * L.ra2); g.N = (int)L.rx1; g.K = (int)(L.ra1 * L.n);
    g.A = A; g.sAm = L.ra1 * L.n; g.sAk = 1; g.conjA = true;
    g.B = R1; g.sBk = L.rx1; g.sBn = 1;
    g.C = R2; g.sCm = L.rx1; g.sCn = 1;
    g.nb1 = (int)L.ry2; g.nb2 = nvec;
    g.bB1 = L.rx1 * L.ra1 * L.n; g.bB2 = p1;
    g.bC1 = L.rx1 * L.m * L.ra2; g.bC2 = p2;
    rows_of(h[1], 1, L.ra2, L.m);
    scale_by_phi1(h[1], L, phi1, -1, 1);
  }
  {
    GemmZ& g = gs[2];   // y[(b1,j), b2] = sum_(a2,c2) R2[(b1,j),(a2,c2)] conj(phi2[b2,(a2,c2)])
    g.M = (int)(L.rx1 * L.m); g.N = (int)L.rx2; g.K = (int)(L.ra2 * L.ry2);
    g.A = R2; g.sAm = 1; g.sAk = L.rx1 * L.m;
    g.B = phi2; g.sBk = L.rx2; g.sBn = 1; g.conjB = true;
    g.C = y; g.sCm = 1; g.sCn = L.rx1 * L.m;
    g.nb2 = nvec; g.bA2 = p2; g.bC2 = L.xsize();
    scale_by_phi2(h[2], L, phi2, -1, 1);
  }
  for (int i = 0; i < 3; ++i) h[i].nvec = nvec;
}
void bfun3_transp_z(const LocalDims& L, const double2* phi1, const double2* A,
                    const double2* phi2, const double2* x, double2* y, int nvec,
                    double2* scratch, cudaStream_t s) {
  GemmZ g[3];
  OzHint h[3];
  transp_products(g, h, L, phi1, A, phi2, x, scratch, scratch + L.rx1 * L.ra1 * L.n * L.ry2 * nvec, y, nvec);
  run_products(g, h, 3, (char*)scratch + bfun3_z_t_bytes(L, nvec), s);
}

template <class G, class T>
static void phi_right_products(G* gs, OzHint* h, const LocalDims& L, const T* phi2_old, const T* A, const T* x,
                               const T* y, T* phi2_new, T* scratch) {
  T* T1 = scratch;
  T* T2 = scratch + L.t1size();
  stage1(gs[0], h[0], L, x, phi2_old, T1, 1);
  stage2(gs[1], h[1], L, A, T1, phi2_old, T2, 1);
  {
    // phi2_new (rx1*ra1 x ry1) = T2 (rx1*ra1 x n*ry2) * y^T (n*ry2 x ry1)
    G& g = gs[2];
    g.M = (int)(L.rx1 * L.ra1); g.N = (int)L.ry1; g.K = (int)(L.n * L.ry2);
    g.A = T2; g.sAm = 1; g.sAk = L.rx1 * L.ra1;
    g.B = y; g.sBk = L.ry1; g.sBn = 1;
    g.C = phi2_new; g.sCm = 1; g.sCn = L.rx1 * L.ra1;
    if constexpr (sizeof(T) == 16) g.conjB = true;
    rows_of(h[2], 1, L.ra1, L.rx1);
  }
}

template <class G, class T>
static void phi_left_products(G* gs, OzHint* h, const LocalDims& L, const T* phi1_old, const T* A, const T* x,
                              const T* y, T* phi1_new, T* scratch) {
  const i64 psz = L.rx1 * L.ra1 * L.n * L.ry2;   // P[b1,a1,i,c2]
  T* P = scratch;
  T* Q = scratch + psz;                           // Q[b1,j,a2,c2]
  {
    G& g = gs[0];   // P[(b1,a1),(i,c2)] = sum_c1 phi1_old[c1,(b1,a1)] y[c1,(i,c2)]
    g.M = (int)(L.rx1 * L.ra1); g.N = (int)(L.n * L.ry2); g.K = (int)L.ry1;
    g.A = phi1_old; g.sAm = L.ry1; g.sAk = 1;
    g.B = y; g.sBk = 1; g.sBn = L.ry1;
    g.C = P; g.sCm = 1; g.sCn = L.rx1 * L.ra1;
    if constexpr (sizeof(T) == 16) g.conjB = true;
    rows_of(h[0], 1, L.ra1, L.rx1);
  }
  {
    G& g = gs[1];   // per c2: Q[b1,(j,a2)] = sum_(a1,i) A[(a1,i),(j,a2)] P[b1,(a1,i)]
    g.M = (int)(L.m * L.ra2); g.N = (int)L.rx1; g.K = (int)(L.ra1 * L.n);
    g.A = A; g.sAm = L.ra1 * L.n; g.sAk = 1;
    g.B = P; g.sBk = L.rx1; g.sBn = 1;
    g.C = Q; g.sCm = L.rx1; g.sCn = 1;
    g.nb1 = (int)L.ry2; g.bB1 = L.rx1 * L.ra1 * L.n; g.bC1 = L.rx1 * L.m * L.ra2;
    rows_of(h[1], 1, L.ra2, L.m);
    scale_by_phi1(h[1], L, phi1_old, -1, 1);
  }
  {
    G& g = gs[2];   // per a2: phi1_new[c2, b2] = sum_(b1,j) Q[(b1,j), a2, c2] x[(b1,j), b2]
    g.M = (int)L.ry2; g.N = (int)L.rx2; g.K = (int)(L.rx1 * L.m);
    g.A = Q; g.sAm = L.rx1 * L.m * L.ra2; g.sAk = 1;
    g.B = x; g.sBk = 1; g.sBn = L.rx1 * L.m;
    g.C = phi1_new; g.sCm = 1; g.sCn = L.ry2;
    g.nb1 = (int)L.ra2; g.bA1 = L.rx1 * L.m; g.bC1 = L.ry2 * L.rx2;
    rows_of(h[2], 1, L.ra2, L.ry2);
  }
}

// an interface update (the complex ones conjugate y)
template <class G, class T, class F>
static void phi_update(F products, const LocalDims& L, const T* phi, const T* A, const T* x, const T* y,
                       T* phi_new, T* scratch, cudaStream_t s) {
  G g[3];
  OzHint h[3];
  products(g, h, L, phi, A, x, y, phi_new, scratch);
  run_products(g, h, 3, (char*)scratch + phi_t_bytes(L, sizeof(T)), s);
}

// Scratch of one call of known sizes, in bytes: the split products that it takes
// and no others (the functions above bound every call of a sweep, and so hold room
// for products that are too large to be split, up to kOzMaxBytes).
template <class T> static T* any_pointer() { return (T*)256; }   // the plans look at none
size_t bfun3_f64_call(const LocalDims& L, int nvec_min, int nvec) {
  size_t most = 0;
  for (int nv = nvec_min; nv <= nvec; ++nv) {
    double* p = any_pointer<double>();
    QRoute q;
    GemmF64 g[3];
    OzHint h[3];
    bfun3_products(g, h, L, p, p, p, p, p, p, p, nv);
    size_t b = products_bytes(g, h, 3);
    if (bfun3_q_plan(L, p, p, p, p, p, nv, &q))
      b = q.stat() + std::max(oz_bytes(q.g.M, q.g.N, q.g.K, false), q.on ? oz_bytes(q.o3.M, q.o3.N, q.o3.K, false) : 0);
    most = std::max(most, bfun3_t_bytes(L, nv) + b);
  }
  return most;
}
size_t bfun3_z_call(const LocalDims& L, int nvec, bool transp) {
  double2* p = any_pointer<double2>();
  GemmZ g[3];
  OzHint h[3];
  if (transp) transp_products(g, h, L, p, p, p, p, p, p, p, nvec);
  else bfun3_products(g, h, L, p, p, p, p, p, p, p, nvec);
  return bfun3_z_t_bytes(L, nvec) + products_bytes(g, h, 3);
}
template <class G, class T> static size_t phi_call(const LocalDims& L, bool left) {
  T* p = any_pointer<T>();
  G g[3];
  OzHint h[3];
  if (left) phi_left_products(g, h, L, p, p, p, p, p, p);
  else phi_right_products(g, h, L, p, p, p, p, p, p);
  return phi_t_bytes(L, sizeof(T)) + products_bytes(g, h, 3);
}
size_t phi_f64_call(const LocalDims& L, bool left) { return phi_call<GemmF64, double>(L, left); }
size_t phi_z_call(const LocalDims& L, bool left) { return phi_call<GemmZ, double2>(L, left); }

void phi_right_f64(const LocalDims& L, const double* phi2_old, const double* A,
                   const double* x, const double* y, double* phi2_new, double* scratch,
                   cudaStream_t s) {
  phi_update<GemmF64>(phi_right_products<GemmF64, double>, L, phi2_old, A, x, y, phi2_new, scratch, s);
}
void phi_left_f64(const LocalDims& L, const double* phi1_old, const double* A,
                  const double* x, const double* y, double* phi1_new, double* scratch,
                  cudaStream_t s) {
  phi_update<GemmF64>(phi_left_products<GemmF64, double>, L, phi1_old, A, x, y, phi1_new, scratch, s);
}
void phi_right_z(const LocalDims& L, const double2* phi2_old, const double2* A,
                 const double2* x, const double2* y, double2* phi2_new, double2* scratch,
                 cudaStream_t s) {
  phi_update<GemmZ>(phi_right_products<GemmZ, double2>, L, phi2_old, A, x, y, phi2_new, scratch, s);
}
void phi_left_z(const LocalDims& L, const double2* phi1_old, const double2* A,
                const double2* x, const double2* y, double2* phi1_new, double2* scratch,
                cudaStream_t s) {
  phi_update<GemmZ>(phi_left_products<GemmZ, double2>, L, phi1_old, A, x, y, phi1_new, scratch, s);
}

void phi2_left_f64(i64 rx1, i64 rx2, i64 ry1, i64 n, i64 ry2, const double* phi1_old,
                   const double* x, const double* y, double* phi1_new, double* scratch,
                   cudaStream_t s) {
  // res1 (rx1 x n*ry2) = phi1_old^T (rx1 x ry1) * y (ry1 x n*ry2)    ttals.f90:309
  {
    GemmF64 g;
    g.M = (int)rx1; g.N = (int)(n * ry2); g.K = (int)ry1;
    g.A = phi1_old; g.sAm = ry1; g.sAk = 1;
    g.B = y; g.sBk = 1; g.sBn = ry1;
    g.C = scratch; g.sCm = 1; g.sCn = rx1;
    gemm_f64(g, s);
  }
  // phi1 (ry2 x rx2) = res1^T ((rx1 n) x ry2)^T * x (rx1 n x rx2)    ttals.f90:311
  {
    GemmF64 g;
    g.M = (int)ry2; g.N = (int)rx2; g.K = (int)(rx1 * n);
    g.A = scratch; g.sAm = rx1 * n; g.sAk = 1;
    g.B = x; g.sBk = 1; g.sBn = rx1 * n;
    g.C = phi1_new; g.sCm = 1; g.sCn = ry2;
    gemm_f64(g, s);
  }
}

void phi2_right_f64(i64 rx1, i64 rx2, i64 ry1, i64 n, i64 ry2, const double* phi2_old,
                    const double* x, const double* y, double* phi2_new, double* scratch,
                    cudaStream_t s) {
  // res1 (rx1 n x ry2) = x (rx1 n x rx2) * phi2_old (rx2 x ry2)       ttals.f90:273
  {
    GemmF64 g;
    g.M = (int)(rx1 * n); g.N = (int)ry2; g.K = (int)rx2;
    g.A = x; g.sAm = 1; g.sAk = rx1 * n;
    g.B = phi2_old; g.sBk = 1; g.sBn = rx2;
    g.C = scratch; g.sCm = 1; g.sCn = rx1 * n;
    gemm_f64(g, s);
  }
  // phi2 (rx1 x ry1) = res1 (rx1 x n ry2) * y^T (n ry2 x ry1)          ttals.f90:275
  {
    GemmF64 g;
    g.M = (int)rx1; g.N = (int)ry1; g.K = (int)(n * ry2);
    g.A = scratch; g.sAm = 1; g.sAk = rx1;
    g.B = y; g.sBk = ry1; g.sBn = 1;
    g.C = phi2_new; g.sCm = 1; g.sCn = rx1;
    gemm_f64(g, s);
  }
}

// B[(c1,i,c2),(b1,j,b2)] = sum_{a1,a2} phi1[c1,b1,a1] A[a1,i,j,a2] phi2[b2,a2,c2]
__global__ void fullmat_kernel(i64 rx1, i64 m, i64 rx2, i64 ra1, i64 ra2,
                               const double* __restrict__ phi1, const double* __restrict__ A,
                               const double* __restrict__ phi2, double* __restrict__ Bm) {
  const i64 N = rx1 * m * rx2;
  for (i64 e = blockIdx.x * (i64)blockDim.x + threadIdx.x; e < N * N;
       e += (i64)gridDim.x * blockDim.x) {
    i64 row = e % N, col = e / N;
    i64 c1 = row % rx1, i = (row / rx1) % m, c2 = row / (rx1 * m);
    i64 b1 = col % rx1, j = (col / rx1) % m, b2 = col / (rx1 * m);
    double acc = 0.0;
    for (i64 a2 = 0; a2 < ra2; ++a2) {
      double p2 = phi2[b2 + rx2 * (a2 + ra2 * c2)];
      if (p2 == 0.0) continue;
      double t = 0.0;
      for (i64 a1 = 0; a1 < ra1; ++a1)
        t += phi1[c1 + rx1 * (b1 + rx1 * a1)] * A[a1 + ra1 * (i + m * (j + m * a2))];
      acc += t * p2;
    }
    Bm[e] = acc;
  }
}

void fullmat_f64(i64 rx1, i64 m, i64 rx2, i64 ra1, i64 ra2, const double* phi1,
                 const double* A, const double* phi2, double* Bmat, cudaStream_t s) {
  i64 N = rx1 * m * rx2;
  int blocks = (int)std::min<i64>(4096, (N * N + 255) / 256);
  fullmat_kernel<<<blocks, 256, 0, s>>>(rx1, m, rx2, ra1, ra2, phi1, A, phi2, Bmat);
  TTG_CHECK_LAUNCH();
}

}  // namespace ttg
