// FP64 products on the tensor cores by error-free splitting.
//
// GB300 issues two FP64 FMAs per clock per SM (1.2 TFLOP/s) but 1.9 PFLOP/s of
// BF16 products with FP32 accumulation, so a large FP64 product is computed as
// a sum of exact BF16 products (the scheme of Ozaki, Ogita, Oishi and Rump,
// "Error-free transformations of matrix multiplication by using fast routines
// of matrix multiplication and its applications", Numer. Algorithms 59, 2012):
//
//   a_mk = 2^(ea_m - 55) I_mk,  |a_mk| < 2^ea_m for every k, I rounded to an
//   integer; I = sum_p d_p 256^(6-p) with balanced digits d_0..d_6 in
//   [-128, 128], each exact in BF16; likewise b_kn with eb_n.
//   sum_k a_mk b_kn = 2^(ea_m + eb_n - 14) sum_g 2^(-8 g) G_g,
//   G_g = sum_k sum_(p+q=g) d_p d'_q,  g = 0..6 (28 of the 49 digit products;
//   the others lie below 2^-56 of the row and column maxima).
//
// Every G_g is an integer that FP32 accumulation in tensor memory keeps
// exactly: |d d'| <= 2^14, so K = 256 terms of at most 4 digit products stay
// within 2^24; the groups g >= 4 could pass 2^24 only for constant digits of
// -128, and a rounding there lies at 2^-24 2^-32.  After 256 K the groups are
// drained into two 64-bit integers per element (no FP64 arithmetic), which
// sum exactly in any order, and the end result is rounded once.  The error
// left is that of I and of the dropped products: below 2^-51 K max_k |a_mk| max_k
// |b_kn|, while the FP64 FMA chain's bound is 2^-53 K sum_k |a_mk| |b_kn|.  With
// elements of one size the first is the smaller in practice (normal data, relative
// error in the norm 2.0 to 3.6e-16 against 2.8 to 9.2e-16).  A row that spans
// scales would lose its small elements' bits, and the operators' parts do differ in
// scale along the operator rank (1 and 1/h^2 in a Laplacian), the opposite way in
// the two factors of a product whose K runs over it: with elements 1 and nu, error
// nu 2e-17.  So
//   - the elements of A and B are scaled along K by powers of two (exact) from the
//     largest element of each operator rank block of an interface (OzGemm::phi),
//   - it is checked that for every group of rows of A and of columns of B (an
//     operator rank block of the result, a vector of a block) some k holds elements
//     of both whose product is within 2^5 of the groups' largest: then the error in
//     that part of the result is below 2^-46 K times the largest sum_k |a| |b| in it
//     (measured 2 to 3e-16 in the norm at nu = 1 to 1e12), and
//   - products that fail it (3% of a time stepper's, 2 to 9% of a linear solver's;
//     none with Gaussian interfaces) are formed by FP64 FMA chains.
//
// A row whose elements are not all finite, or whose largest element lies
// outside 2^(+-400), is flagged, and its product is formed by plain FP64 FMA
// chains, so infinities, NaN and extreme ranges give what they give there.
//
// Measured on GB300, FP64 kernels -> split products: chain product r=256, block
// of 8: 4560 -> 251 us (22 TFLOP/s of FP64 accuracy; its two products run at
// 46 and 44 TFLOP/s, i.e. 1.3 PFLOP/s of BF16); r=64, block of 5: 76.6 -> 36.0
// us; grid interface updates r = 82, 77, n = 64: 1908 -> 179 us; complex
// operator and adjoint r=48, n=32, block of 4: 6968 -> 384 us (without scales and
// check 241, 32.8, 160 and 351).  What bounds the product kernel is the operand traffic (43 KB a K step per SM, 1.4k clocks
// measured against 900 of MMA), for small ones its fixed ~10 us (pipeline
// fill, one drain, rounding); oz_us below holds both.
//
// Tensor memory: a 128 x 64 tile (128 x 32 for small products) with its seven
// groups side by side (448 of the 512 columns).  The digit planes of B sit
// stacked along N, so the MMA of A's plane p with B's planes 0..6-p writes groups
// p..6 in one instruction (two where N > 256): ten instructions per 16-wide K
// step, and A's planes are read from shared memory once per step.
#include "ttg_common.cuh"
#include "ttg_tcgen05.cuh"
#include <algorithm>
#include <climits>
#include <type_traits>

namespace ttg {
namespace oz {

using namespace tc;

constexpr int P = 7;            // digit planes
constexpr int BM = 128;         // rows of A's tiles; B's: 64, or 32 for small products
constexpr int KCHUNK = 16;      // 16-wide K steps between drains (256 K)
constexpr int STAGES = 5;
constexpr uint32_t A_PLANE = BM * 32;                      // bytes of a plane in one K step
constexpr uint32_t A_BYTES = P * A_PLANE;
__host__ __device__ constexpr uint32_t b_bytes(int bn) { return P * bn * 32; }
__host__ __device__ constexpr uint32_t stage_bytes(int bn) { return A_BYTES + b_bytes(bn); }   // 43,008 for 64
constexpr size_t smem_bytes(int bn) { return (size_t)STAGES * stage_bytes(bn) + 1024; }
constexpr int EPI_WARPS = 16;
constexpr int THREADS = 64 + 32 * EPI_WARPS;
constexpr int EMAX = 400;       // largest |exponent| of the fast path

// Largest elements of an operand's row groups (group r / gd of row r, gn gd = rows)
// as scaled exponents + EBIAS, 0 for zeros only, and where they are: per block of
// eight rows, its first group's rows and the next one's, over all of K; and along K
// for up to SLOTS blocks of a group, spread over it (rows of the first group).
constexpr int SROWS = 8, SLOTS = 16, EBIAS = 8192, FLAGGED = 1 << 30;
struct Groups {
  int rows, gd, gn;
  int stride;                   // every how manyth block that starts in a group has a slot
  int4* bm;                     // [block]: largest, its k, of the next group; FLAGGED
  short* part;                  // [group][slot][K]
  __host__ __device__ int first_block(int group) const { return (group * gd + SROWS - 1) / SROWS; }
  __device__ int slots(int group) const {
    return (first_block(group + 1) - first_block(group) + stride - 1) / stride;
  }
};
enum { UNKNOWN = 0, FINE = 1, CHAINS = 2 };
struct Side {                   // one operand, element (r, k) = src[map(r) + k * sk]
  const double* src;
  OzMap map;
  i64 sk;
  int rows, R;                  // logical rows; rows of a tile (BM or BN)
  unsigned char* planes;        // [rtile][K step][plane][R x 16 bf16, core matrices]
  int* expo;                    // per split row
  int vec;                      // real with sk == 1 and 16-byte aligned rows
  int cplx;                     // 0 real, 1: rows (re, im) x K (re, im), 2: K (re, im) only
  int conj;
  const short* tab;             // scales along K (null: none) by block k / kd % kr
  int kd, kr, sgn;
  Groups gr;
};

struct Args {
  const unsigned char *Ad, *Bd;
  const int *ea, *eb;
  int M, N, K;                  // product rows and columns; logical K (for the FP64 chain)
  int kt, kper, mtiles, ntiles, btile;
  int nz, cs;                   // K splits of a tile; cs > 1: added over clusters of cs CTAs
  double* C;
  OzMap cm, cn;
  longlong2* part;              // nz > cs: the clusters' sums [z / cs][n][row]
  const double *A, *B;          // original operands (FP64 chains)
  OzMap am, bn;
  i64 ak, bk;
  Groups ga, gb;
  int* state;                   // of the check: UNKNOWN, FINE, CHAINS
  int rows, cols;               // logical rows and columns
  int look;                     // CTA 0 of the product kernel makes it
  int cplx, conjA, conjB;       // complex: product rows (PAIR: columns) are (re, im)
};

// 32-bit division: a 64-bit one per stored element took a third of the product
__device__ __forceinline__ i64 at(const OzMap& m, int i) {
  const uint32_t q = (uint32_t)i / (uint32_t)m.d, r = (uint32_t)i - q * (uint32_t)m.d;
  return (i64)q * m.s2 + (i64)r * m.s1;
}

// bf16 pair from two digit bytes u (digit = u - 128): float 2^23 + u is exact,
// and so is the difference; its upper half is the bf16
__device__ __forceinline__ uint32_t digit_pair(uint32_t ja, uint32_t jb, uint32_t sel) {
  const float a = __uint_as_float(__byte_perm(ja, 0x4B000000u, sel)) - 8388736.f;
  const float b = __uint_as_float(__byte_perm(jb, 0x4B000000u, sel)) - 8388736.f;
  return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
}
__device__ __forceinline__ uint32_t top_pair(int ta, int tb) {
  const float a = __uint_as_float(0x4B400000u + (uint32_t)ta) - 12582912.f;
  const float b = __uint_as_float(0x4B400000u + (uint32_t)tb) - 12582912.f;
  return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
}

// The largest exponents of an interface's operator rank blocks, in TPARTS parts
// each: element i of block a, outer index o, lies at (o kr + a) inner + i.
constexpr int TPARTS = 8, TNONE = -32768, TSPAN = 300, NTABLES = kOzProducts - 1;
struct Table { const double* phi; short* tab; i64 inner, outer; int kr; };
struct Tables { Table t[NTABLES]; };
// block b of 256 threads, kr TPARTS of them per table
__device__ __forceinline__ void table_block(const Tables& ts, int b) {
  __shared__ int best_s;
  static_assert(NTABLES == 2, "two tables");
  const bool second = b >= ts.t[0].kr * TPARTS;
  if (second) b -= ts.t[0].kr * TPARTS;
  const Table t = second ? ts.t[1] : ts.t[0];
  const int a = b / TPARTS, part = b % TPARTS, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) best_s = TNONE;
  __syncthreads();
  // 8 warps per part: over the outer index, or over the elements of the only one
  const i64 w = part * 8 + warp, nw = TPARTS * 8;
  int best = TNONE;
  auto see = [&](double v) {
    const int e = (__double2hiint(v) >> 20) & 0x7ff;
    if (((__double2hiint(v) << 1) | __double2loint(v)) != 0 && e != 0x7ff) best = max(best, max(e, 1) - 1022);
  };
  if (t.outer == 1) {
    const double* x = t.phi + t.inner * a;
#pragma unroll 4
    for (i64 i = w * 32 + lane; i < t.inner; i += nw * 32) see(x[i]);
  } else {
    for (i64 o = w; o < t.outer; o += nw) {
      const double* x = t.phi + t.inner * (o * t.kr + a);
#pragma unroll 4
      for (i64 i = lane; i < t.inner; i += 32) see(x[i]);
    }
  }
  best = __reduce_max_sync(0xffffffffu, best);
  if (lane == 0) atomicMax(&best_s, best);
  __syncthreads();
  if (threadIdx.x == 0) t.tab[a * TPARTS + part] = (short)best_s;
}
__global__ void __launch_bounds__(256) tables_kernel(Tables t) {
  pdl_wait();
  pdl_trigger();
  table_block(t, blockIdx.x);
}

// Splits two operands in one launch (blocks [0, nblkA) take A).  A cluster of
// gridDim.y blocks takes 8 rows and all of K, its blocks every gridDim.y-th
// run of 256: a first pass finds the rows' largest exponents (joined over the
// cluster), a second writes the digits, each thread one 16-byte core-matrix
// row (8 K) per plane, and notes the largest exponents of the row groups.  Blocks
// past B's form the tables that the call's later products need.  Bound by its 8
// bytes read and 14 written per element (integer digits, no FP64 arithmetic).
// One copy of the code for both operands, and one of the stores: at these sizes its
// fetching counts (with a copy for each operand the kernel took 4 us more).
__global__ void __launch_bounds__(256, 3) split_kernel(const __grid_constant__ Side a, const __grid_constant__ Side b,
                                                       int nblkA, int nblk, const __grid_constant__ Tables tabs,
                                                       int K, int kt, int* state) {
  namespace cgr = cooperative_groups;
  cgr::cluster_group cl = cgr::this_cluster();
  __shared__ int key_s[SROWS], scaled_s;
  extern __shared__ __align__(16) short tab_s[];
  pdl_wait();
  if ((int)blockIdx.x >= nblk) {
    if (blockIdx.y == 0) table_block(tabs, blockIdx.x - nblk);
    return;
  }
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *state = UNKNOWN;
  const bool isA = (int)blockIdx.x < nblkA;
  const Side& S = isA ? a : b;
  const int blk = isA ? blockIdx.x : blockIdx.x - nblkA;
  const int row = threadIdx.x & 7, kg0 = (threadIdx.x >> 3) + 32 * blockIdx.y;
  const int kgs = 32 * gridDim.y;
  const int r = blk * SROWS + row;                   // row of src
  const bool real = r < S.rows;
  const double* p = S.src + (real ? at(S.map, r) * (S.cplx ? 2 : 1) : 0);
  const int groups = 2 * kt;
  double v[8];
  auto load = [&](int g) {
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = 0.0;
    if (!real) return;
    if (S.cplx) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int k = g * 4 + q;
        if (k < K) {
          const double2 z = *reinterpret_cast<const double2*>(p + 2 * (i64)k * S.sk);
          v[2 * q] = z.x;
          v[2 * q + 1] = S.conj ? -z.y : z.y;
        }
      }
    } else if (S.vec && g * 8 + 8 <= K) {
#pragma unroll
      for (int q = 0; q < 8; q += 2) {
        const double2 z = *reinterpret_cast<const double2*>(p + g * 8 + q);
        v[q] = z.x;
        v[q + 1] = z.y;
      }
    } else {
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int k = g * 8 + q;
        if (k < K) v[q] = p[(i64)k * S.sk];
      }
    }
  };
  // exponents of the scales of group g's eight + EBIAS, two to a word
  constexpr int NONFINITE = 1 << 20;
  uint32_t sc[4] = {EBIAS * 0x10001u, EBIAS * 0x10001u, EBIAS * 0x10001u, EBIAS * 0x10001u};
  auto scales = [&](int g) {
    if (S.cplx) {
      const uint2 t = *reinterpret_cast<const uint2*>(tab_s + 4 * g);
      sc[0] = __byte_perm(t.x, 0u, 0x1010);
      sc[1] = __byte_perm(t.x, 0u, 0x3232);
      sc[2] = __byte_perm(t.y, 0u, 0x1010);
      sc[3] = __byte_perm(t.y, 0u, 0x3232);
    } else {
      const uint4 t = *reinterpret_cast<const uint4*>(tab_s + 8 * g);
      sc[0] = t.x;
      sc[1] = t.y;
      sc[2] = t.z;
      sc[3] = t.w;
    }
  };
  auto scale = [&](int q) { return (int)(q & 1 ? sc[q >> 1] >> 16 : sc[q >> 1] & 0xffffu); };
  // (zeros count as 2^-1022 and less here, which no unflagged row's largest is near:
  // scales stay within 2^(+-300).  Integers only: an FP64 comparison holds the pipe
  // for 64 clocks)
  auto expo_of = [&](int q) { return (__double2hiint(v[q]) >> 20) & 0x7ff; };
  load(kg0);                                         // (beyond K: zeros)
  // while these are on their way: the block's place among the row groups, the scales
  const int group = blk * SROWS / S.gr.gd, in_group = blk - S.gr.first_block(group);
  const bool first = r / S.gr.gd == group, has_slot = blk * SROWS < S.rows && in_group % S.gr.stride == 0;
  short* part = has_slot ? S.gr.part + (size_t)(group * SLOTS + in_group / S.gr.stride) * ((K + 7) & ~7) : nullptr;
  if (threadIdx.x < SROWS) key_s[threadIdx.x] = 0;
  // the operator rank blocks' scales, behind the places of each k's
  const int per = S.cplx ? 4 : 8;
  short* of_block = tab_s + groups * per;
  if (S.tab && threadIdx.x < 32) {
    int ref = TNONE, most = 0;
    for (int c = threadIdx.x; c < S.kr; c += 32) {
      const uint4 t = *reinterpret_cast<const uint4*>(S.tab + c * TPARTS);
      const uint32_t m = __vmaxs2(__vmaxs2(t.x, t.y), __vmaxs2(t.z, t.w));
      of_block[c] = (short)max((int)(short)(m & 0xffffu), (int)m >> 16);
      ref = max(ref, (int)of_block[c]);
    }
    ref = __reduce_max_sync(0xffffffffu, ref);
    // blocks within a factor of two of the largest stay as they are
    for (int c = threadIdx.x; c < S.kr; c += 32) {
      const int d = of_block[c] == TNONE ? 0 : max(of_block[c] - ref, -TSPAN);
      of_block[c] = (short)(EBIAS + (d >= -1 ? 0 : S.sgn * d));
      most = max(most, -d);
    }
    if (threadIdx.x == 0) scaled_s = 0;
    __syncwarp();
    if (most > 1) scaled_s = 1;
  }
  __syncthreads();
  const bool scaled = S.tab && scaled_s != 0;
  if (scaled) {
    for (int k = threadIdx.x; k < groups * per; k += blockDim.x) tab_s[k] = of_block[k / S.kd % S.kr];
    __syncthreads();
  }
  int key = 0, key_g = kg0, top_e = 0;               // the row's largest here, in which group
  unsigned int nonzero = 0u;
  for (int g = kg0; g < groups; g += kgs) {
    if (g != kg0) load(g);
    if (scaled) scales(g);
    int here = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int x = expo_of(q);
      here = max(here, x + scale(q));
      top_e = max(top_e, x);
      nonzero |= ((unsigned)__double2hiint(v[q]) & 0x7fffffffu) | (unsigned)__double2loint(v[q]);
    }
    if (here > key) {
      key = here;
      key_g = g;
    }
  }
  key = nonzero == 0u ? 0 : (top_e == 0x7ff ? NONFINITE : key);
  const int own = key;
  atomicMax(&key_s[row], key);
  if (gridDim.y > 1) {
    cl.sync();
    for (unsigned q = 0; q < cl.num_blocks(); ++q) key = max(key, *cl.map_shared_rank(&key_s[row], q));
    cl.sync();   // no block leaves, or goes on, while another reads its maxima
  } else {
    __syncthreads();
    key = key_s[row];
  }
  const int e = key - EBIAS - 1022;
  const bool flag = key == NONFINITE || (key != 0 && (e > EMAX || e < -EMAX));
  const bool zero = key == 0 || flag;
  if (kg0 == 0) {
    const int ex = zero ? 0 : e;
    if (S.cplx == 1) {
      S.expo[2 * r] = ex;
      S.expo[2 * r + 1] = ex;
    } else {
      S.expo[r] = ex;
    }
  }
  // the row groups' largest of this block (of one of them that has it, its k)
  const int mine = real && !zero ? key : 0;
  int* at = nullptr;
  if (blk * SROWS < S.rows) {
    const unsigned rows8 = 0xffu << (threadIdx.x & 24);
    const int m0 = __reduce_max_sync(rows8, first ? mine : 0), m1 = __reduce_max_sync(rows8, first ? 0 : mine);
    const bool bad = __any_sync(rows8, flag);
    int* bm = reinterpret_cast<int*>(S.gr.bm + blk);
    if (kg0 == 0 && row < 2) bm[2 * row] = row ? m1 : (bad ? FLAGGED : m0);
    at = mine && own == key && key == (first ? m0 : m1) ? bm + (first ? 1 : 3) : nullptr;
  }
  for (int g = kg0; (g & ~3) < groups; g += kgs) {
    if (groups > kgs) {                              // one group per thread: still in registers
      load(g);
      if (scaled) scales(g);
    }
    if (at && g == key_g) {
      int k = 0;
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (expo_of(q) + scale(q) == key) k = q;
      *at = S.cplx ? g * 4 + k / 2 : g * 8 + k;
    }
    if (part) {
      // largest scaled exponents of these k over the rows, 16 bits each, by
      // halving: lane `row` is left with k = row of the eight
      uint32_t x[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t h = __byte_perm((unsigned)__double2hiint(v[2 * q]), (unsigned)__double2hiint(v[2 * q + 1]), 0x7632);
        x[q] = mine && first ? (h >> 4 & 0x07ff07ffu) + sc[q] : 0u;
        if (S.cplx) x[q] = __vmaxu2(x[q], __byte_perm(x[q], x[q], 0x1032));
      }
      uint32_t a0 = row & 4 ? x[2] : x[0], a1 = row & 4 ? x[3] : x[1];
      a0 = __vmaxu2(a0, __shfl_xor_sync(0xffffffffu, row & 4 ? x[0] : x[2], 4));
      a1 = __vmaxu2(a1, __shfl_xor_sync(0xffffffffu, row & 4 ? x[1] : x[3], 4));
      uint32_t b0 = __vmaxu2(row & 2 ? a1 : a0, __shfl_xor_sync(0xffffffffu, row & 2 ? a0 : a1, 2));
      b0 = __vmaxu2(b0, __shfl_xor_sync(0xffffffffu, b0, 1));
      const int k = S.cplx ? g * 4 + row / 2 : g * 8 + row;
      if (k < K && !(S.cplx && (row & 1))) part[k] = (short)(row & 1 ? b0 >> 16 : b0 & 0xffffu);
    }
    if (g >= groups) continue;
    int top[8];
    uint32_t jl[8], jh[8];                           // bytes of I + sum 128 256^i
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const unsigned hi = (unsigned)__double2hiint(v[q]), lo = (unsigned)__double2loint(v[q]);
      const int eq = (int)((hi >> 20) & 0x7ff);
      long long m = (long long)(((unsigned long long)(hi & 0xfffffu) << 32) | lo);
      if (eq) m |= 1ll << 52;
      const int sh = key - (max(eq, 1) + scale(q)) - 2;   // I = m 2^-sh
      long long I = 0;
      if (!zero) I = sh <= 0 ? m << -sh : (sh < 55 ? (m + (1ll << (sh - 1))) >> sh : 0);
      if (hi >> 31) I = -I;
      const long long J = I + 0x0000808080808080ll;
      jl[q] = (uint32_t)J;
      jh[q] = (uint32_t)((unsigned long long)J >> 32);
      top[q] = (int)(J >> 48);
    }
    // pairs (0,1) (2,3) (4,5) (6,7).  A doubled complex operand: the real part's row
    // (re, -im), then the imaginary part's (im, re); the second of a pair negated (I
    // -> -I digit by digit is again balanced: digits in [-128, 128])
    auto word = [&](int pl, int h) {
      if (pl == 0) return top_pair(top[2 * h], top[2 * h + 1]);
      if (pl < 3) return digit_pair(jh[2 * h], jh[2 * h + 1], pl == 1 ? 0x7651u : 0x7650u);
      return digit_pair(jl[2 * h], jl[2 * h + 1], 0x7650u + (6 - pl));
    };
    auto place = [&](int rr) {
      const int rt = rr / S.R, ri = rr % S.R;
      return S.planes + ((size_t)rt * kt + (g >> 1)) * ((size_t)P * S.R * 32) +
             (size_t)((ri >> 3) * 256 + (g & 1) * 128 + (ri & 7) * 16);
    };
    if (S.cplx != 1) {
      unsigned char* o = place(r);
#pragma unroll
      for (int pl = 0; pl < P; ++pl)
        *reinterpret_cast<uint4*>(o + (size_t)pl * S.R * 32) = make_uint4(word(pl, 0), word(pl, 1), word(pl, 2), word(pl, 3));
    } else {
      unsigned char* o = place(2 * r);               // 2 r + 1 lies 16 bytes on
      auto minus = [](uint32_t x) { return (x & 0x7fff0000u) ? x ^ 0x80000000u : x; };
      auto swap = [](uint32_t x) { return __byte_perm(x, x, 0x1032); };
#pragma unroll
      for (int pl = 0; pl < P; ++pl) {
        const uint32_t w0 = word(pl, 0), w1 = word(pl, 1), w2 = word(pl, 2), w3 = word(pl, 3);
        uint4* d = reinterpret_cast<uint4*>(o + (size_t)pl * S.R * 32);
        d[0] = make_uint4(minus(w0), minus(w1), minus(w2), minus(w3));
        d[1] = make_uint4(swap(w0), swap(w1), swap(w2), swap(w3));
      }
    }
  }
  pdl_trigger();
}

// hi 2^32 + lo as a double, times 2^sc, rounded once to nearest even; integer
// arithmetic only (the exponent stays in the normal range by the row limits)
__device__ __forceinline__ double to_double(long long hi, long long lo, int sc) {
  hi += lo >> 32;
  uint32_t l = (uint32_t)lo;
  const bool neg = hi < 0;
  if (neg) {
    l = 0u - l;
    hi = ~hi + (l == 0u ? 1 : 0);
  }
  const unsigned long long h = (unsigned long long)hi;
  if ((h | l) == 0ull) return 0.0;
  unsigned long long x;
  int off = 0;
  if (h < (1ull << 31)) {
    x = (h << 32) | l;
  } else {
    const int lz = __clzll((long long)h);            // 0 < lz <= 32
    x = (h << lz) | (lz == 32 ? (unsigned long long)l : (unsigned long long)(l >> (32 - lz)));
    if (lz < 32 && (l << lz) != 0u) x |= 1ull;       // sticky
    off = 32 - lz;
  }
  const int z = __clzll((long long)x);
  x <<= z;
  unsigned long long m = x >> 11;
  const unsigned int r = (unsigned int)(x & 0x7ffull);
  m += (r > 0x400u || (r == 0x400u && (m & 1ull))) ? 1ull : 0ull;
  const long long ex = (long long)(63 - z + off + sc + 1023);
  const unsigned long long bits = ((unsigned long long)ex << 52) + (m - (1ull << 52));
  return __longlong_as_double((long long)(bits | (neg ? 0x8000000000000000ull : 0ull)));
}

template <bool PAIR>
__device__ __forceinline__ i64 c_row(const Args& g, int row) {
  if (PAIR) return 2 * at(g.cm, row);
  return g.cplx ? 2 * at(g.cm, row >> 1) + (row & 1) : at(g.cm, row);
}

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}

template <bool PAIR>
__device__ __forceinline__ i64 c_col(const Args& g, int n) {
  if (PAIR) return 2 * at(g.cn, n >> 1) + (n & 1);
  return at(g.cn, n) * (g.cplx ? 2 : 1);
}

// whether any of 512 threads (the draining ones, or all of check_kernel) says so; all
// of them call it
__device__ __forceinline__ bool any_of_512(bool v) {
  uint32_t r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.u32 q, %1, 0;\n barrier.cta.red.or.pred p, 1, %2, q;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(r)
      : "r"((uint32_t)v), "n"(32 * EPI_WARPS)
      : "memory");
  return r != 0;
}

// Whether a product is one for the FP64 chains: a row is flagged, or the large
// elements of the operands do not meet.  For every group of A's rows and of B's
// columns, 2^APART times some k's product of largest elements must reach the product
// of the groups' largest (either 0: nothing to reach).  Looked for where one of
// them has its largest, then everywhere.  Thread e of 512; global memory is read past
// L1 (check_kernel looks before it waits for the kernels in front of it).
constexpr int APART = 3;
constexpr int PAIRS = 128;                        // pairs of groups looked at together
constexpr int WHERE = 18;                         // bits of a largest element's k (beyond: not looked for there)
struct Check {                                    // shared memory, zero at first
  unsigned int mx[2 * kOzMaxGroups];              // A's groups, then B's: largest, its k
  int seen[2][PAIRS];                             // the other side's largest there
};
__device__ __noinline__ bool needs_chains(const Args& g, Check& sh, int e) {
  constexpr int NE = 32 * EPI_WARPS, KMASK = (1 << WHERE) - 1;
  const int na = g.ga.gn, np = na * g.gb.gn, Kp = (g.K + 7) & ~7;
  bool bad = false;
#pragma unroll 1
  for (int side = 0; side < 2; ++side) {
    const Groups& s = side ? g.gb : g.ga;
    unsigned int* m = sh.mx + (side ? na : 0);
    const int n = (s.rows + SROWS - 1) / SROWS;
    for (int b = e; b - (e & 31) < n; b += NE) {
      const int4 v = b < n ? __ldcg(s.bm + b) : make_int4(0, 0, 0, 0);
      bad = bad || v.x == FLAGGED;
      const int group = s.gn == 1 ? 0 : min(b, n - 1) * SROWS / s.gd;
      const unsigned x = v.x > 0 ? (unsigned)(v.x & 0x3fff) << WHERE | min(v.y, KMASK) : 0u;
      int same;
      __match_all_sync(0xffffffffu, group, &same);
      if (same) {                                    // 32 atomics on one word are as many turns
        const unsigned y = __reduce_max_sync(0xffffffffu, x);
        if ((e & 31) == 0) atomicMax(&m[group], y);
      } else {
        atomicMax(&m[group], x);
      }
      if (v.z > 0) atomicMax(&m[group + 1], (unsigned)v.z << WHERE | min(v.w, KMASK));
    }
  }
  if (any_of_512(bad)) return true;
  bool open = false;
  for (int p0 = 0; p0 < np; p0 += PAIRS) {
    const int n = min(PAIRS, np - p0);
    // B's largest at A's k, and A's at B's: a load per pair, side and slot
#pragma unroll 1
    for (int t = e; t < n * 2 * SLOTS; t += NE) {
      const int q = t % SLOTS, side = t / SLOTS & 1, p = p0 + t / (2 * SLOTS), pb = p / na, pa = p - pb * na;
      const Groups& s = side ? g.ga : g.gb;
      const int gi = side ? pa : pb, k = min((int)sh.mx[side ? na + pb : pa] & KMASK, g.K - 1);
      int v = 0;
      if (q * s.stride < s.first_block(gi + 1) - s.first_block(gi)) v = __ldcg(s.part + (size_t)(gi * SLOTS + q) * Kp + k);
      v = __reduce_max_sync(0xffffu << (e & 16), v);
      if (q == 0) sh.seen[side][p - p0] = v;
    }
    any_of_512(false);
    if (e < n) {
      const unsigned a = sh.mx[(p0 + e) % na], b = sh.mx[na + (p0 + e) / na];
      const int ma = a >> WHERE, mb = b >> WHERE;
      const bool at_a = (int)(a & KMASK) < KMASK && sh.seen[0][e] >= mb - APART;
      const bool at_b = (int)(b & KMASK) < KMASK && sh.seen[1][e] >= ma - APART;
      open = open || (ma > 0 && mb > 0 && !at_a && !at_b);
    }
    open = any_of_512(open);
  }
  if (!open) return false;
#pragma unroll 1
  for (int p = 0; p < np; ++p) {
    const int a = sh.mx[p % na] >> WHERE, b = sh.mx[na + p / na] >> WHERE, need = a + b - APART;
    if (a == 0 || b == 0) continue;
    const int sa = g.ga.slots(p % na), sb = g.gb.slots(p / na);
    const short* pa = g.ga.part + (size_t)(p % na) * SLOTS * Kp;
    const short* pb = g.gb.part + (size_t)(p / na) * SLOTS * Kp;
    bool meet = false;
    for (int k0 = 0; k0 < g.K && !meet; k0 += NE) {
      const int k = k0 + e;
      int x = 0, y = 0;
#pragma unroll 4
      for (int q = 0; q < SLOTS; ++q) {
        if (k < g.K && q < sa) x = max(x, (int)__ldcg(pa + (size_t)q * Kp + k));
        if (k < g.K && q < sb) y = max(y, (int)__ldcg(pb + (size_t)q * Kp + k));
      }
      meet = any_of_512(x != 0 && y != 0 && x + y >= need);
    }
    if (!meet) return true;
  }
  return false;
}

constexpr int kMaxSplit = kMaxCluster;            // CTAs of a cluster that share a tile
constexpr float kCarry = 3221225472.f;   // 1.5 2^31: FP32 spacing 256
// an integer |x| < 2^22 held in FP32, without the conversion unit
__device__ __forceinline__ int small_int(float x) {
  return (int)(__float_as_uint(__fadd_rn(x, 12582912.f)) - 0x4B400000u);
}

// Persistent and warp-specialised: one CTA per SM walks the tiles (mt fastest,
// then nt, then the K split z).  Warp 0 issues the bulk copies into the ring
// (one for A's seven planes of a K step, one for B's), warp 1 the MMAs, warps
// 2-17 drain: warp w holds TMEM lanes 32 (w % 4).. and 16 of the 64 columns,
// and keeps their two 64-bit sums in registers over the tile's drains.  Every
// wait is bounded; a CTA whose wait ran out fills the outputs it has not
// finished with NaN.  The outputs are scaled by 2^(ea + eb - 14): hi 2^-16 + lo 2^-48.
// In CTA 0 they look first, while the first K steps run, whether the product is one
// for the FP64 chains (g.look; check_kernel does otherwise).
template <int BN, bool PAIR>
__global__ void __launch_bounds__(THREADS, 1) gemm_kernel(const __grid_constant__ Args g) {
  constexpr uint32_t B_BYTES = b_bytes(BN), STAGE = stage_bytes(BN);
  constexpr uint32_t TMEM = BN == 64 ? 512 : 256;   // columns: 7 BN, a power of two
  constexpr int CB = BN / 4;                        // columns of a draining warp
  static_assert(P * BN <= (int)TMEM && CB % 4 == 0, "tile width");
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES];
  __shared__ __align__(8) uint64_t acc_full, acc_empty, done_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int fail_s;
  __shared__ Check check_s;
  volatile int* fail = &fail_s;
  unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int total = g.mtiles * g.ntiles * g.nz;
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    mbar_init(smem_u32(&acc_full), 1);
    mbar_init(smem_u32(&acc_empty), EPI_WARPS);
    mbar_init(smem_u32(&done_bar), 1);
    fail_s = 0;
    fence_mbar_init();
  }
  if (g.look && blockIdx.x == 0)
    for (int i = tid; i < (int)(sizeof(Check) / sizeof(int)); i += THREADS) reinterpret_cast<int*>(&check_s)[i] = 0;
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_slot), TMEM);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t taddr = tmem_slot;
  pdl_wait();
  pdl_trigger();                                     // check_kernel may look beside this

  if (warp == 0) {
    if (lane == 0) {
      int it = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
        const int z = t % g.nz, rz = t / g.nz, mt = rz % g.mtiles, nt = rz / g.mtiles;
        const int k0 = z * g.kper, k1 = min(g.kt, k0 + g.kper);
        for (int k = k0; k < k1; ++k, ++it) {
          const int s = it % STAGES;
          if (it >= STAGES &&
              !mbar_wait_f(smem_u32(&empty_bar[s]), (uint32_t)((it / STAGES - 1) & 1), fail)) {
            ok = false;
            break;
          }
          unsigned char* st = base + (size_t)s * STAGE;
          const uint32_t bar = smem_u32(&full_bar[s]);
          mbar_expect_tx(bar, STAGE);
          bulk_g2s(smem_u32(st), g.Ad + ((size_t)mt * g.kt + k) * A_BYTES, A_BYTES, bar);
          bulk_g2s(smem_u32(st + A_BYTES), g.Bd + ((size_t)nt * g.kt + k) * B_BYTES, B_BYTES, bar);
        }
      }
      if (!ok) *fail = 1;
      if (!ok || *fail) {
        // the last fill of each stage may not have been consumed: let it land
        for (int s = 0; s < STAGES; ++s) {
          const int last = it - 1 - ((it - 1 - s) % STAGES + STAGES) % STAGES;
          if (last >= 0 && last < it) mbar_wait(smem_u32(&full_bar[s]), (uint32_t)((last / STAGES) & 1));
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      int it = 0, use = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
        const int z = t % g.nz, k0 = z * g.kper, k1 = min(g.kt, k0 + g.kper);
        for (int kc = k0; kc < k1 && ok; kc += KCHUNK, ++use) {
          if (use > 0 && !mbar_wait_f(smem_u32(&acc_empty), (uint32_t)((use - 1) & 1), fail)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const int ke = min(k1, kc + KCHUNK);
          for (int k = kc; k < ke; ++k, ++it) {
            const int s = it % STAGES;
            if (!mbar_wait_f(smem_u32(&full_bar[s]), (uint32_t)((it / STAGES) & 1), fail)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t sa = smem_u32(base + (size_t)s * STAGE), sb = sa + A_BYTES;
            const uint32_t acc0 = k > kc ? 1u : 0u;
#pragma unroll
            for (int p = 0; p < P; ++p) {
              // planes 0..6-p of B against plane p of A: groups p..6
              const int n = BN * (P - p), parts = n > 256 ? 2 : 1, w = n / parts;
              const uint64_t da = make_desc(sa + p * A_PLANE, LBO, SBO);
#pragma unroll
              for (int h = 0; h < parts; ++h)
                mma_bf16(taddr + (uint32_t)(p * BN + h * w), da,
                         make_desc(sb + (uint32_t)(h * w * 32), LBO, SBO), make_idesc(BM, w),
                         p > 0 ? 1u : acc0);
            }
            mma_commit(smem_u32(&empty_bar[s]));
          }
          if (ok) mma_commit(smem_u32(&acc_full));
        }
      }
      if (!ok) *fail = 1;
      mma_commit(smem_u32(&done_bar));
      mbar_wait(smem_u32(&done_bar), 0);   // every MMA issued here has completed
    }
    __syncwarp();
  } else {
    const int q = warp & 3, cb = ((warp - 2) >> 2) * CB;
    const uint32_t tb = taddr + ((uint32_t)(q * 32) << 16) + (uint32_t)cb;
    int use = 0;
    bool ok = true;
    if (g.look && blockIdx.x == 0) {
      const bool chains = needs_chains(g, check_s, tid - 64);
      if (tid == 64) *g.state = chains ? CHAINS : FINE;
    }
    for (int t = blockIdx.x; t < total; t += gridDim.x) {
      const int z = t % g.nz, rz = t / g.nz, mt = rz % g.mtiles, nt = rz / g.mtiles;
      const int k0 = z * g.kper, k1 = min(g.kt, k0 + g.kper);
      long long hi[CB];                              // sum = hi 2^32 + lo, in 2^-48
      uint32_t lo[CB];
#pragma unroll
      for (int c = 0; c < CB; ++c) { hi[c] = 0; lo[c] = 0u; }
      for (int kc = k0; kc < k1 && ok; kc += KCHUNK, ++use) {
        ok = __all_sync(0xffffffffu, mbar_wait_f(smem_u32(&acc_full), (uint32_t)(use & 1), fail));
        if (!ok) {
          if (lane == 0) *fail = 1;
          break;
        }
        tc_fence_after();
#pragma unroll
        for (int c0 = 0; c0 < CB; c0 += 4) {
          uint32_t v[P][4];
#pragma unroll
          for (int p = 0; p < P; ++p) tmem_ld4(tb + (uint32_t)(p * BN + c0), v[p]);
          tmem_ld_wait();
          if (c0 == CB - 4) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&acc_empty));
          }
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            // carry the groups down to bytes in FP32 (every step exact): l is
            // G less its nearest multiple of 256, which joins the group above
            float G[P];
#pragma unroll
            for (int p = 0; p < P; ++p) G[p] = __uint_as_float(v[p][c]);
#pragma unroll
            for (int p = P - 1; p > 0; --p) {
              const float h = __fsub_rn(__fadd_rn(G[p], kCarry), kCarry);
              G[p] = __fsub_rn(G[p], h);
              G[p - 1] = __fmaf_rn(h, 1.f / 256.f, G[p - 1]);
            }
            const int g12 = small_int(__fmaf_rn(G[1], 256.f, G[2]));
            const int g34 = small_int(__fmaf_rn(G[3], 256.f, G[4]));
            const int g56 = small_int(__fmaf_rn(G[5], 256.f, G[6]));
            const long long l = (long long)lo[c0 + c] + (long long)g34 * 65536 + g56;
            hi[c0 + c] += (long long)__float2int_rn(G[0]) * 65536 + g12 + (l >> 32);
            lo[c0 + c] = (uint32_t)l;
          }
        }
      }
      const int row = mt * BM + q * 32 + lane, n0 = nt * BN + cb;
      if (g.cs > 1) {
        // the CTA's only tile: every copy has landed and every MMA has read it,
        // so the ring holds the sums for the cluster (after a failure fail_s counts)
        longlong2* o = reinterpret_cast<longlong2*>(base) + cb * BM + q * 32 + lane;
#pragma unroll
        for (int c = 0; c < CB; ++c) o[c * BM] = make_longlong2(hi[c], (long long)lo[c]);
      } else {
        // lane c holds column c's exponent and offset
        const int nl = n0 + (lane & (CB - 1));
        const int my_eb = nl < g.N ? g.eb[nl] : 0;
        const i64 my_col = nl < g.N ? c_col<PAIR>(g, nl) : 0;
        const int ea = row < g.M ? g.ea[row] : 0;
        const i64 cr = row < g.M ? c_row<PAIR>(g, row) : 0;
        if constexpr (PAIR) {
          // columns (re, im) of one output: stored as a pair (N is even)
#pragma unroll
          for (int c = 0; c < CB; c += 2) {
            const int eb = __shfl_sync(0xffffffffu, my_eb, c);
            const i64 col = __shfl_sync(0xffffffffu, my_col, c);
            if (row < g.M && n0 + c < g.N)
              *reinterpret_cast<double2*>(g.C + cr + col) =
                  make_double2(to_double(hi[c], (long long)lo[c], ea + eb - 62),
                               to_double(hi[c + 1], (long long)lo[c + 1], ea + eb - 62));
          }
        } else {
#pragma unroll
          for (int c = 0; c < CB; ++c) {
            const int eb = __shfl_sync(0xffffffffu, my_eb, c);
            const i64 col = __shfl_sync(0xffffffffu, my_col, c);
            if (row < g.M && n0 + c < g.N)
              g.C[cr + col] = to_double(hi[c], (long long)lo[c], ea + eb - 62);
          }
        }
        if (!ok && row < g.M) {
#pragma unroll 1
          for (int n = n0; n < min(n0 + CB, g.N); ++n)
            g.C[cr + c_col<PAIR>(g, n)] = __longlong_as_double(0x7ff8000000000000ll);
        }
      }
    }
  }
  if (g.cs > 1) {
    // one tile per CTA; CTA `rank` adds its share of the columns over the
    // cluster (exact integers) and rounds, or leaves the cluster's sum
    namespace cgr = cooperative_groups;
    cgr::cluster_group cl = cgr::this_cluster();
    cl.sync();
    const int z = (int)blockIdx.x % g.nz, rz = (int)blockIdx.x / g.nz;
    const int mt = rz % g.mtiles, nt = rz / g.mtiles, rank = (int)cl.block_rank();
    const int share = (BN + g.cs - 1) / g.cs;
    bool bad = false;
    for (int p = 0; p < g.cs; ++p) bad = bad || *cl.map_shared_rank(&fail_s, p) != 0;
    const int row = mt * BM + (tid & (BM - 1));
    const longlong2* mine = reinterpret_cast<const longlong2*>(base) + (tid & (BM - 1));
    const bool live = tid < 4 * BM && row < g.M;
    const int ea = live ? g.ea[row] : 0;
    const i64 cr = live ? c_row<PAIR>(g, row) : 0;
    for (int c = rank * share + (tid >> 7); c < min(BN, (rank + 1) * share); c += 4) {
      const int n = nt * BN + c;
      if (!live || n >= g.N) break;
      longlong2 v[kMaxSplit];
#pragma unroll
      for (int p = 0; p < kMaxSplit; ++p)
        v[p] = p < g.cs ? *cl.map_shared_rank(mine + c * BM, p) : make_longlong2(0, 0);
      long long hi = v[0].x, lo = v[0].y;
#pragma unroll
      for (int p = 1; p < kMaxSplit; ++p) {
        hi += v[p].x;
        lo += v[p].y;
      }
      if (bad) hi = LLONG_MIN;                       // marks NaN
      if (g.nz > g.cs)
        g.part[((size_t)(z / g.cs) * g.ntiles * BN + n) * ((size_t)g.mtiles * BM) + row] =
            make_longlong2(hi, lo);
      else
        g.C[cr + c_col<PAIR>(g, n)] =
            hi == LLONG_MIN ? __longlong_as_double(0x7ff8000000000000ll) : to_double(hi, lo, ea + g.eb[n] - 62);
    }
    cl.sync();   // no CTA leaves while another reads its sums
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(taddr, TMEM);
}

// adds the clusters' sums (exact integers) and rounds
template <bool PAIR>
__global__ void __launch_bounds__(256) finish_kernel(const Args g) {
  pdl_wait();
  pdl_trigger();
  const size_t Mp = (size_t)g.mtiles * BM, Np = (size_t)g.ntiles * g.btile;
  const i64 total = (i64)Mp * g.N;
  for (i64 e = blockIdx.x * (i64)blockDim.x + threadIdx.x; e < total; e += (i64)gridDim.x * blockDim.x) {
    const int row = (int)(e % (i64)Mp), n = (int)(e / (i64)Mp);
    if (row >= g.M) continue;
    long long hi = 0, lo = 0;
    bool bad = false;
    for (int z = 0; z < g.nz / g.cs; ++z) {
      const longlong2 v = g.part[((size_t)z * Np + n) * Mp + row];
      bad = bad || v.x == LLONG_MIN;
      hi += v.x;
      lo += v.y;
    }
    g.C[c_row<PAIR>(g, row) + c_col<PAIR>(g, n)] =
        bad ? __longlong_as_double(0x7ff8000000000000ll) : to_double(hi, lo, g.ea[row] + g.eb[n] - 62);
  }
}

// FP64 FMA chains of a unit, 4 NI rows x 8 NJ columns: ks warps take every ks-th k, a
// lane rows ly + 4 i and columns lx + 8 j, and the warps' sums are added in order
// from red (16 / ks units at once; `here`: this one exists).  Bound by the FP64 pipe,
// as gemm_kernel of ttg_gemm.cu is: a load serves several FMAs of 64 clocks each.
// Units this small, and K over the warps, so that a product of few rows and columns
// keeps all SMs busy: 32 x 16 (complex 32 x 8), or 8 x 8 where those are fewer than
// SMs (phi_left with an infinity in Phi, r = 64, n = 40, whose last product has 192 x
// 64 results: 614 -> 395 us; FP64 kernels 311); four warps a unit where K is
// short.
template <class T, int NI, int NJ>
__device__ __forceinline__ void fp64_unit(const Args& g, bool here, int r0, int c0, int ks, T* red) {
  constexpr bool CPLX = sizeof(T) == 16;
  constexpr int E = 32 * NI * NJ;
  const int w16 = threadIdx.x >> 5, warp = w16 % ks, lane = threadIdx.x & 31, ly = lane >> 3, lx = lane & 7;
  const int K = here ? g.K : 0;
  const T *a[NI], *b[NJ];
#pragma unroll
  for (int i = 0; i < NI; ++i)
    a[i] = reinterpret_cast<const T*>(g.A) + at(g.am, min(r0 + ly + 4 * i, g.rows - 1)) + (i64)warp * g.ak;
#pragma unroll
  for (int j = 0; j < NJ; ++j)
    b[j] = reinterpret_cast<const T*>(g.B) + at(g.bn, min(c0 + lx + 8 * j, g.cols - 1)) + (i64)warp * g.bk;
  T acc[NI][NJ], x[NI], y[NJ];
#pragma unroll
  for (int i = 0; i < NI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j) acc[i][j] = T{};
  auto load = [&] {
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      x[i] = *a[i];
      a[i] += ks * g.ak;
    }
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      y[j] = *b[j];
      b[j] += ks * g.bk;
    }
  };
  constexpr bool AHEAD = !CPLX;                      // (complex: four times the FMAs per load)
  if (AHEAD && warp < K) load();
  for (int k = warp; k < K; k += ks) {
    if (!AHEAD) load();
    T u[NI], v[NJ];
#pragma unroll
    for (int i = 0; i < NI; ++i) u[i] = x[i];
#pragma unroll
    for (int j = 0; j < NJ; ++j) v[j] = y[j];
    if (AHEAD && k + ks < K) load();
#pragma unroll
    for (int i = 0; i < NI; ++i)
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        if constexpr (CPLX) {
          const double ui = g.conjA ? -u[i].y : u[i].y, vi = g.conjB ? -v[j].y : v[j].y;
          acc[i][j].x = fma(u[i].x, v[j].x, acc[i][j].x);
          acc[i][j].x = fma(-ui, vi, acc[i][j].x);
          acc[i][j].y = fma(u[i].x, vi, acc[i][j].y);
          acc[i][j].y = fma(ui, v[j].x, acc[i][j].y);
        } else {
          acc[i][j] = fma(u[i], v[j], acc[i][j]);
        }
      }
  }
  __syncthreads();                                   // the unit before is read
#pragma unroll
  for (int i = 0; i < NI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j) red[w16 * E + (i * NJ + j) * 32 + lane] = acc[i][j];
  __syncthreads();
  red += (w16 - warp) * E;
  for (int q = warp; here && q < NI * NJ; q += ks) {
    const int r = r0 + ly + 4 * (q / NJ), n = c0 + lx + 8 * (q % NJ);
    if (r >= g.rows || n >= g.cols) continue;
    T v = red[q * 32 + lane];
    for (int w = 1; w < ks; ++w) {
      const T t = red[w * E + q * 32 + lane];
      if constexpr (CPLX) {
        v.x += t.x;
        v.y += t.y;
      } else {
        v += t;
      }
    }
    reinterpret_cast<T*>(g.C)[at(g.cm, r) + at(g.cn, n)] = v;
  }
}

// After the product: whether it is one for the FP64 chains, and then the chains over
// the whole GPU.  The look is made, where the product kernel left SMs free, beside
// that kernel; what remains when it is done is one launch (1 to 2 us).  The look and
// the chains in the product kernel itself took 5 us more a product (time stepper d =
// 16, n = 32: 98.5 -> 95 ms), and the chains of a K split had its few SMs alone (such
// a product of the time stepper 180 us).  The chains take the time of the FP64
// kernels: phi_left with an infinity in Phi, r = 82, n = 64 942 us (FP64 kernels
// 1426), r = 256, n = 2 753 (777).
constexpr size_t kCheckSmem = sizeof(double) * EPI_WARPS * 512;
__global__ void __launch_bounds__(32 * EPI_WARPS, 1) check_kernel(const __grid_constant__ Args g) {
  extern __shared__ __align__(16) unsigned char check_dyn[];
  __shared__ Check sh;
  __shared__ int state_s;
  const int tid = threadIdx.x;
  for (int i = tid; i < (int)(sizeof(Check) / sizeof(int)); i += blockDim.x) reinterpret_cast<int*>(&sh)[i] = 0;
  // (what the split kernel wrote is there: every kernel in between has waited for it
  // before it let this one start)
  if (tid == 0) state_s = __ldcg(g.state);
  __syncthreads();
  int state = state_s;
  if (state == UNKNOWN) {
    state = needs_chains(g, sh, tid) ? CHAINS : FINE;
    if (tid == 0) *(volatile int*)g.state = state;
  }
  pdl_wait();
  if (state == FINE) return;
  const int ks = g.K >= 256 ? 16 : 4, at_once = EPI_WARPS / ks, mine = (tid >> 5) / ks;
  auto run = [&](auto t, auto ni, auto nj) {
    using T = decltype(t);
    constexpr int NI = decltype(ni)::value, NJ = decltype(nj)::value;
    const int mr = (g.rows + 4 * NI - 1) / (4 * NI), nc = (g.cols + 8 * NJ - 1) / (8 * NJ);
    const i64 units = (i64)mr * nc, steps = (units + at_once - 1) / at_once;
    for (i64 q = steps * blockIdx.x / gridDim.x; q < steps * (blockIdx.x + 1) / gridDim.x; ++q) {
      const i64 u = q * at_once + mine, v = u < units ? u : 0;
      fp64_unit<T, NI, NJ>(g, u < units, (int)(v % mr) * 4 * NI, (int)(v / mr) * 8 * NJ, ks,
                           reinterpret_cast<T*>(check_dyn));
    }
  };
  using One = std::integral_constant<int, 1>;
  using Two = std::integral_constant<int, 2>;
  using Eight = std::integral_constant<int, 8>;
  const bool few = (i64)((g.rows + 31) / 32) * ((g.cols + 15) / 16) < (i64)gridDim.x * at_once;
  if (g.cplx) few ? run(double2{}, Two{}, One{}) : run(double2{}, Eight{}, One{});
  else few ? run(double{}, Two{}, One{}) : run(double{}, Eight{}, Two{});
  pdl_trigger();
}

constexpr int SMS = 152;

struct Shape {
  i64 M, N, K;                  // split rows, columns, K
  i64 mt, nt, kt;
  int bn;
  bool dup_b;                   // complex: B's columns doubled, not A's rows
};
// 64 columns of B a tile, or 32 where those leave more than half of the SMs
// idle: half the drain and the rounding per CTA (r=64 chain product 38.5 -> 32.8
// us, grid interface updates 166 -> 160, time stepper 87.0 -> 85.1 ms, AMEn solve
// 170 -> 167 ms)
static Shape shape_of(i64 M, i64 N, i64 K, bool cplx, bool dup_b) {
  Shape s{cplx && !dup_b ? 2 * M : M, cplx && dup_b ? 2 * N : N, cplx ? 2 * K : K, 0, 0, 0, 64, dup_b};
  s.mt = (s.M + BM - 1) / BM;
  s.nt = (s.N + 63) / 64;
  if (s.mt * s.nt * 2 <= SMS) {
    s.bn = 32;
    s.nt = (s.N + 31) / 32;
  }
  s.kt = (s.K + 15) / 16;
  return s;
}
// A complex product is a real one with the rows of one operand doubled to (re,
// -im) and (im, re): the smaller operand, whose digits are then written twice,
// unless the tiles get more padding by it (complex
// operator and adjoint r=48, n=32, block of 4: 403 -> 351 us, the digits of its
// intermediates 38 -> 20 us)
static Shape shape(i64 M, i64 N, i64 K, bool cplx) {
  const Shape a = shape_of(M, N, K, cplx, false);
  if (!cplx || N >= M) return a;
  const Shape b = shape_of(M, N, K, true, true);
  const double area_a = (double)a.mt * a.nt * a.bn, area_b = (double)b.mt * b.nt * b.bn;
  return area_b <= 1.05 * area_a ? b : a;
}
// K split: only where the tiles leave SMs idle; at least KMIN K steps per chunk
// (a last chunk may be empty).  Up to eight chunks are one cluster where the
// GPU holds all of them (it holds 14 clusters of eight of these CTAs, 36 of
// four), more are clusters of four whose sums a second kernel adds.  Measured,
// at least 8 steps and a second kernel for every split -> this: r=64 chain
// product 40.1 -> 38.3 us, time stepper (d=16, n=32, r=8) 92.1 -> 88.4 ms,
// operator and adjoint r=48 407 -> 403 us (351 since), K = 5248 in 36 chunks unchanged
// (clusters of eight there: 167 -> 171 us; at least 2 steps: 88.4 -> 92 ms).
constexpr int KMIN = 4;
struct Split { int nz, cs, kper; };
static Split z_split(const Shape& s) {
  const i64 tiles = s.mt * s.nt;
  i64 nz = tiles * 2 > SMS ? 1 : std::max<i64>(1, std::min<i64>(144 / tiles, s.kt / KMIN)), cs = nz;
  if (nz > 4 && (s.kt / KMIN > kMaxSplit || tiles * nz > 112)) {
    nz -= nz % 4;
    cs = 4;
  }
  const i64 kper = (s.kt + nz - 1) / nz;
  if (cs == nz) cs = nz = (s.kt + kper - 1) / kper;
  return {(int)nz, (int)cs, (int)kper};
}
static inline size_t al(size_t b) { return (b + 255) & ~size_t(255); }

}  // namespace oz

double oz_us(i64 M, i64 N, i64 K, bool cplx) {
  const oz::Shape s = oz::shape(M, N, K, cplx);
  const oz::Split z = oz::z_split(s);
  const int nz = z.nz;
  const double waves = (double)((s.mt * s.nt * nz + oz::SMS - 1) / oz::SMS);
  const double ks = (double)((s.kt + nz - 1) / nz);
  const bool wide = s.bn == 64;
  const double mma = waves * (ks * (wide ? 950.0 : 800.0) + (ks / oz::KCHUNK + 1) * (wide ? 2500.0 : 1300.0) +
                              (wide ? 3000.0 : 2000.0)) / 1900.0;
  const double split = ((double)s.M + s.N) * s.K * 22.0 / 4.0e6;
  return mma + split + 12.0 + (nz > z.cs ? 5.0 : (nz > 1 ? 1.5 : 0.0));
}

size_t oz_bytes(i64 M, i64 N, i64 K, bool cplx) {
  if ((cplx ? 4.0 : 1.0) * (double)M * (double)N * (double)K < kOzMinMNK) return 0;
  // rows of both operands padded to the larger tile, doubled if complex: either
  // may become A and either may be the doubled one
  const i64 f = cplx ? 2 : 1, kt = (f * K + 15) / 16;
  const double rows = 128.0 * (double)((f * M + 127) / 128 + (f * N + 127) / 128);
  const double need = 14.0 * 16.0 * (double)kt * rows + 4.0 * rows +
                      (double)oz::SMS * oz::BM * 64 * 16.0 + 4096.0;
  return need > (double)kOzMaxBytes ? kOzMaxBytes : (size_t)need;
}

bool oz_fits(i64 M, i64 N, i64 K, bool cplx) {
  const size_t b = oz_bytes(M, N, K, cplx);
  return b > 0 && b < kOzMaxBytes;
}

size_t oz_stat_bytes(i64 rows, i64 K, i64 groups, i64 kr) {
  using namespace oz;
  return al(sizeof(int4) * (size_t)(rows / SROWS + 3)) + al(sizeof(short) * SLOTS * (size_t)(K + 7) * groups) +
         al(sizeof(short) * TPARTS * (size_t)kr);
}
static short* oz_tab(const OzGemm& g) {          // at the end of stat
  const size_t b = oz_stat_bytes((i64)g.M + g.N, g.K, g.gnA + g.gnB, g.kr);
  return (short*)((char*)g.stat + b - oz::al(sizeof(short) * oz::TPARTS * (size_t)g.kr));
}
static oz::Tables oz_tables(const OzGemm* const* later, int n, int* blocks) {
  oz::Tables t{};
  int m = 0;
  *blocks = 0;
  for (int i = 0; i < n; ++i)
    if (later[i]->kr > 0) {
      const OzGemm& g = *later[i];
      t.t[m++] = {g.phi, oz_tab(g), (g.cplx ? 2 : 1) * g.inner, g.outer, g.kr};
      *blocks += g.kr * oz::TPARTS;
    }
  return t;
}

// shared memory of the scales: of every k, then of the operator rank blocks
constexpr size_t kScaleSmem = 200 * 1024;
static size_t split_smem(const OzGemm& g) {
  return sizeof(short) * ((size_t)(((g.cplx ? 2 * (i64)g.K : g.K) + 15) / 16 * (g.cplx ? 8 : 16)) + g.kr);
}

void oz_gemm(const OzGemm& g, void* ws, const OzGemm* const* later, int nlater, cudaStream_t st) {
  using namespace oz;
  const Shape s = shape(g.M, g.N, g.K, g.cplx);
  TTG_REQUIRE(s.M < (1ll << 31) - BM && s.N < (1ll << 31) - 64 && s.K < (1ll << 30), "oz: size");
  char* p = (char*)ws;
  auto take = [&](size_t b) { char* r = p; p += al(b); return r; };
  const size_t ra = (size_t)s.mt * BM, rb = (size_t)s.nt * s.bn;
  unsigned char* Ad = (unsigned char*)take(14 * 16 * (size_t)s.kt * ra);
  unsigned char* Bd = (unsigned char*)take(14 * 16 * (size_t)s.kt * rb);
  int* ea = (int*)take(4 * ra);
  int* eb = (int*)take(4 * rb);
  const Split z = z_split(s);
  const int nz = z.nz, groups = nz / z.cs;
  longlong2* part = groups > 1 ? (longlong2*)take(sizeof(longlong2) * groups * ra * rb) : nullptr;
  auto vec = [&](const double* src, const OzMap& m, i64 sk) {
    return !g.cplx && sk == 1 && ((uintptr_t)src & 15) == 0 && (m.s1 & 1) == 0 && (m.s2 & 1) == 0;
  };
  const short* tab = g.kr > 0 ? oz_tab(g) : nullptr;
  int4* bm = (int4*)g.stat;
  short* gpart = (short*)((char*)g.stat + al(sizeof(int4) * (size_t)(((i64)g.M + g.N) / SROWS + 3)));
  int* state = (int*)(bm + ((i64)g.M + g.N) / SROWS + 2);
  auto stride = [](int gd) { return ((gd + SROWS - 1) / SROWS + 1 + SLOTS - 1) / SLOTS; };
  const Groups gra{g.M, g.gdA, g.gnA, stride(g.gdA), bm, gpart};
  const Groups grb{g.N, g.gdB, g.gnB, stride(g.gdB), bm + (g.M + SROWS - 1) / SROWS, gpart + (size_t)SLOTS * ((g.K + 7) & ~7) * g.gnA};
  int tblocks = 0;
  const Tables tables = oz_tables(later, nlater, &tblocks);
  const Side a{g.A, g.am, g.ak, g.M, BM, Ad, ea, vec(g.A, g.am, g.ak), g.cplx ? (s.dup_b ? 2 : 1) : 0, g.conjA,
               tab, g.kd, g.kr, -g.norm, gra};
  const Side b{g.B, g.bn, g.bk, g.N, s.bn, Bd, eb, vec(g.B, g.bn, g.bk), g.cplx ? (s.dup_b ? 1 : 2) : 0, g.conjB,
               tab, g.kd, g.kr, g.norm, grb};
  const int nA = (int)(ra / (a.cplx == 1 ? 2 : 1) / SROWS), nB = (int)(rb / (b.cplx == 1 ? 2 : 1) / SROWS);
  static const cudaError_t attr_rc = [] {
    cudaError_t r = cudaSuccess;
    auto set = [&](auto* k, int bn) {
      if (r == cudaSuccess)
        r = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(bn));
    };
    set(gemm_kernel<64, false>, 64);
    set(gemm_kernel<64, true>, 64);
    set(gemm_kernel<32, false>, 32);
    set(gemm_kernel<32, true>, 32);
    if (r == cudaSuccess)
      r = cudaFuncSetAttribute(split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kScaleSmem);
    if (r == cudaSuccess)
      r = cudaFuncSetAttribute(check_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCheckSmem);
    return r;
  }();
  TTG_CUDA(attr_rc);
  // few rows and a long K: K over a cluster (246 + 82 rows, K = 4928: 50 -> 17 us)
  int ky = 1;
  while (ky < kMaxCluster && (nA + nB) * ky < 2 * SMS && 2 * s.kt > 32 * ky) ky *= 2;
  launch_ex(split_kernel, dim3(nA + nB + tblocks, ky), dim3(256), dim3(ky > 1 ? 1 : 0, ky, 1), true,
            g.kr > 0 ? split_smem(g) : 0, st, a, b, nA, nA + nB, tables, g.K, (int)s.kt, state);
  Args x{};
  x.Ad = Ad; x.Bd = Bd; x.ea = ea; x.eb = eb;
  x.M = (int)s.M; x.N = (int)s.N; x.K = g.K;
  x.kt = (int)s.kt; x.kper = z.kper; x.mtiles = (int)s.mt; x.ntiles = (int)s.nt; x.btile = s.bn; x.nz = nz; x.cs = z.cs;
  x.C = g.C; x.cm = g.cm; x.cn = g.cn; x.part = part;
  x.A = g.A; x.B = g.B; x.am = g.am; x.bn = g.bn; x.ak = g.ak; x.bk = g.bk;
  x.cplx = g.cplx; x.conjA = g.conjA; x.conjB = g.conjB;
  x.ga = gra; x.gb = grb;
  x.state = state; x.rows = g.M; x.cols = g.N;
  const int grid = (int)std::min<i64>(SMS, s.mt * s.nt * nz);
  // where the product kernel, or finish_kernel, leaves check_kernel no SM to look on
  x.look = grid > SMS * 3 / 4 || groups > 1;
  auto kern = s.bn == 64 ? (s.dup_b ? gemm_kernel<64, true> : gemm_kernel<64, false>)
                         : (s.dup_b ? gemm_kernel<32, true> : gemm_kernel<32, false>);
  launch_ex(kern, dim3(grid), dim3(THREADS),
            dim3(z.cs > 1 ? z.cs : 0, 1, 1), true, smem_bytes(s.bn), st, x);
  if (groups > 1) {
    const int fb = (int)std::min<i64>(1024, ((i64)ra * s.N + 255) / 256);
    launch_pdl(s.dup_b ? finish_kernel<true> : finish_kernel<false>, dim3(fb), dim3(256), 0, st, x);
  }
  launch_pdl(check_kernel, dim3(SMS), dim3(32 * EPI_WARPS), kCheckSmem, st, x);
}

// A strided batched product as one split product: a batch over which one
// operand does not move joins the rows (or columns) of the other.  The side
// that C stores contiguously becomes the MMA's M (a warp's TMEM lanes).
// Returns false when the product does not have that form, does not fit the
// workspace rule, or the FP64 kernel is the faster.
template <class G>
static bool oz_plan_impl(const G& g, const OzHint& h, bool cplx, bool conjA, bool conjB, bool plain, OzGemm* out) {
  if (!plain || g.M <= 0 || g.N <= 0 || g.K <= 0) return false;
  i64 nb = (i64)g.nb1 * g.nb2, bA = g.bA1, bB = g.bB1, bC = g.bC1;
  if (g.nb1 == 1) {
    bA = g.bA2; bB = g.bB2; bC = g.bC2;
  } else if (g.nb2 > 1 && (g.bA2 != g.nb1 * g.bA1 || g.bB2 != g.nb1 * g.bB1 || g.bC2 != g.nb1 * g.bC1)) {
    return false;
  }
  i64 M = g.M, N = g.N;
  OzMap am{g.M, g.sAm, 0}, cm{g.M, g.sCm, 0}, bn{g.N, g.sBn, 0}, cn{g.N, g.sCn, 0};
  bool joinA = false, joinB = false;
  if (nb > 1) {
    if (bB == 0) { am.s2 = bA; cm.s2 = bC; M *= nb; joinA = true; }
    else if (bA == 0) { bn.s2 = bB; cn.s2 = bC; N *= nb; joinB = true; }
    else return false;
  }
  const bool swap = g.sCm != 1;
  if (swap && g.sCn != 1) return false;
  if (M >= (1ll << 29) || N >= (1ll << 29)) return false;
  const i64 Mo = swap ? N : M, No = swap ? M : N;
  if (!oz_fits(Mo, No, g.K, cplx)) return false;
  if (oz_us(Mo, No, g.K, cplx) >= gemm_fp64_us(g.M, g.N, g.K, (int)nb, cplx)) return false;
  // groups: the operator rank blocks of one side, the vectors of the other
  int gd[2] = {(int)M, (int)N}, gn[2] = {1, 1};
  if (h.side != 0) {
    const int t = h.side - 1;
    const i64 rows = t == 0 ? M : N;
    gn[t] = h.groups;
    if (h.run > 0) {
      TTG_REQUIRE(rows == (i64)h.run * h.groups, "oz: groups");
      gd[t] = h.run;
    } else {
      // interleaved: rows taken block by block instead (not the side C stores
      // contiguously, not a joined one)
      TTG_REQUIRE(!(t == 0 ? joinA : joinB) && rows % h.groups == 0, "oz: groups");
      OzMap& mo = t == 0 ? am : bn;
      OzMap& mc = t == 0 ? cm : cn;
      gd[t] = (int)(rows / h.groups);
      mo = {gd[t], mo.s1 * h.groups, mo.s1};
      mc = {gd[t], mc.s1 * h.groups, mc.s1};
    }
  }
  const int vt = joinA ? 0 : 1;
  const i64 per_vec = (vt == 0 ? M : N) / std::max(h.nvec, 1);
  if (h.nvec > 1 && h.nvec <= kOzMaxVec && (joinA || joinB) && gn[vt] == 1 && per_vec >= 8) {
    gn[vt] = h.nvec;
    gd[vt] = (int)per_vec;
  }
  // a group's runs hold the start of a block of eight rows
  if ((gn[0] > 1 && gd[0] < 8) || (gn[1] > 1 && gd[1] < 8) || gn[0] + gn[1] > 2 * kOzMaxGroups) return false;
  const int a = swap ? 1 : 0, b = 1 - a;
  OzGemm o;
  o.M = (int)Mo; o.N = (int)No; o.K = g.K; o.cplx = cplx;
  o.A = (const double*)(swap ? g.B : g.A); o.am = swap ? bn : am; o.ak = swap ? g.sBk : g.sAk;
  o.B = (const double*)(swap ? g.A : g.B); o.bn = swap ? am : bn; o.bk = swap ? g.sAk : g.sBk;
  o.C = (double*)g.C; o.cm = swap ? cn : cm; o.cn = swap ? cm : cn;
  o.conjA = swap ? conjB : conjA; o.conjB = swap ? conjA : conjB;
  o.gdA = gd[a]; o.gnA = gn[a]; o.gdB = gd[b]; o.gnB = gn[b];
  if (h.phi && h.kr <= kOzMaxTable) {
    o.phi = h.phi; o.inner = h.inner; o.outer = h.outer; o.kr = h.kr; o.kd = h.kd;
    o.norm = swap ? -h.norm : h.norm;
    if (split_smem(o) > kScaleSmem) o.kr = 0;          // (K beyond 100 thousand)
  }
  *out = o;
  return true;
}
// tables that g itself needs (no earlier split product to form them)
void oz_prepare(const OzGemm* const* g, int n, cudaStream_t s) {
  int blocks = 0;
  const oz::Tables t = oz_tables(g, n, &blocks);
  if (blocks > 0) launch_pdl(oz::tables_kernel, dim3(blocks), dim3(256), 0, s, t);
}
bool oz_plan(const GemmF64& g, const OzHint& h, OzGemm* out) {
  return oz_plan_impl(g, h, false, false, false, g.alpha == 1.0 && g.beta == 0.0, out);
}
bool oz_plan(const GemmZ& g, const OzHint& h, OzGemm* out) {
  const bool plain = g.alpha.x == 1.0 && g.alpha.y == 0.0 && g.beta.x == 0.0 && g.beta.y == 0.0;
  return oz_plan_impl(g, h, true, g.conjA, g.conjB, plain, out);
}

}  // namespace ttg
