// FP64 channel products on the Blackwell tensor cores.
//
// The products of the FP64 form, for every job (a channel block),
//     Out (+)= P + s phi_i phi_j P^T,   P = A B^T,   A, B: m x K FP64
// (or Out (+)= A B^T, A: m x K, B: n x K, for a plain job), to FP64 accuracy
// but not on the FP64 pipe, which runs at 1.2 TFLOP/s on this part: each row
// of A and of B is taken as 62-bit fixed point below its own exponent, cut
// into S = 9 balanced base-2^7 digits, exact in BF16, and the digit products
// of weight s + t < S are summed by tcgen05.mma into one FP32 tensor-memory
// accumulator per weight.
//
//  * Exactness.  The reduction is cut into chunks of at most CH x 32 elements,
//    so the sums of the six leading weights stay below 2^24 and are exact
//    integers; what the others round is below 2^-66 of the row maxima's
//    product.  Each chunk's sums are added as 64-bit integers (two words: the
//    leading five weights, the trailing four) and converted to FP64 once per
//    half of the product.
//  * The two halves, A B^T and s phi B A^T, have their own row exponents (a_i
//    + b_j and b_i + a_j), so they are separate chunks of one tile: only the
//    tiles of the upper triangle are computed, each written with its mirror.
//  * Error.  Fixed point is exact to 2^-63 of each row's largest element, FP64
//    to 2^-53 of each element, so the two differ where a sum is small against
//    its rows' maxima.  A tenth plane holds |a| and |b| as BF16 magnitudes
//    (exponents clamped at 2^-60), and one more MMA a step gives sum |a||b| of
//    every output and chunk.  A product with a zero factor has zero digits and
//    no error, so the digit error of a sum with n nonzero products is about
//    sqrt(n) 2^-63 (unit: the rows' exponents), that of an FP64 sum about
//    2^-54 sum |a||b|.  An element whose sum |a||b| is not zero, but below
//    2^-9 sqrt(n) in every chunk (n: the smaller of the two rows' counts of
//    nonzero elements), is not written but listed, and evaluated with FP64
//    FMAs; so is one of a row that holds an infinity, a NaN or magnitudes
//    outside 2^-423 .. 2^477, and what a timed-out wait left undone.  (An
//    estimate of the two errors, not a bound for the worst signs; but then too
//    a sum above that line stays within the classical bound of an FP64 sum,
//    (n + 5) 2^-53 sum |a||b| against n 2^-60.)
//  * Listed elements (exact_work): blocks of 8 x 8 with a mask, shared out over
//    all CTAs at the end, since one 128 x 32 tile of K = 1000 keeps an SM's FP64
//    pipe busy for 2 ms.  So the time depends on the operands.  FP64 commutator,
//    emax 6 / 8 / 10, in ms (on the FP64 pipe alone: 1.25 / 11.1 / 87.2):
//      random operators, none to a few elements listed    0.24 / 1.20 / 6.5
//      one a generator, 0.1 to 1% of the FP64 work        0.31 / 1.39 / 6.9
//      both falling off as e^(-1.0 |de|)                  0.54 / 3.4  / 30
//      a dominating diagonal                              0.61 / 4.1  / 39
//      both falling off as 2^(-4 |de|), 70 to 90% of it   0.96 / 7.2  / 61
//    (With the chunk's length as n and whole tiles of 128 x 32 listed, evaluated
//    by the CTA that found them: generator 0.95 / 4.7 / 20.8, falling off
//    1.25 / 11.6 / 97 and 1.62 / 14.6 / 112, diagonal 1.54 / 12.8 / 99.)  Tensor
//    commutators likewise: rank (2, 0, +), emax 6 / 8, 1.70 / 9.9 ms random, 4.7 /
//    43 falling off as 2^(-4 |de|), 4.9 / 51 on the FP64 pipe; smaller ones of such
//    operands are slower than there (emax 4 0.81 against 0.57), since an 8 x 8
//    block of a small matrix is half padding.
//
// What bounds it: for the long products the MMAs, 46 of 128 x 32 x 16 a K16
// step (merged to 11 instructions), next to the TMA stream of the ten planes
// (the emax=10 ladder: 2.6 ms, tensor pipe 58%, 13.4 TB/s from L2); for the
// short ones (Zbar, K <= 132) the epilogue.  With the FP64-pipe kernel the
// commutator takes 142 us at emax 2, 1.26 ms at emax 6, 87.2 ms at emax 10;
// with this one, and nothing else changed, it took 116 us, 0.38 ms and 7.7 ms
// (47 us, 0.24 ms and 6.5 ms by now): scalar products use it at every size,
// tensor ones from the sizes that capi_tensor.cu gives, and the FP64-pipe
// kernels run below those, where the planes do not fit (40 bytes an element
// pair of the operands) and inside a capture that comes before them.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <stdexcept>
#include <vector>

#include "kernels.cuh"
#include "prof.hpp"
#include "tcgen05.cuh"

namespace imsrg {

namespace {

constexpr int KB = 32;       // K elements per pipeline stage: one 64-byte swizzle row
constexpr int TM = 128;      // tile rows (UMMA M)
constexpr int TN = 32;       // tile columns (UMMA N per digit)
constexpr int S = 9;         // digits per element
constexpr int BETA = 7;      // bits between digits
constexpr int P = 62;        // bits of the fixed point: 6 in the top digit, 7 in each other
constexpr int NP = S + 1;    // planes: digits, then magnitudes
constexpr int NHI = 5;       // weights summed in the leading integer word
constexpr int CH = 20;       // K blocks per chunk: 6 x 65^2 x 32 CH < 2^24
constexpr int NSTAGE = 2;    // 2 x 100 KB of 227 KB
constexpr int SHORT_KB = 4;  // K blocks a job in plans that are sliced in one pass
constexpr int NINFO = 3;     // tiles whose job, exponents and phases wait in shared memory
constexpr int EPIW = 8;      // epilogue warps: two per TMEM lane quarter, 16 columns each
constexpr int COLS_W = TN / 2;
constexpr int BLK = 8;                // rows and columns of a listed block
constexpr int TILE_BLKS = (TM / BLK) * (TN / BLK);
constexpr int SHARE = 1 << 15;        // FP64 FMAs of a tile (8 us of an SM) from which listed blocks are shared out
constexpr int NB = 512 / TN;         // tensor-memory blocks
constexpr int OV = 2 * NP - NB;      // blocks that consecutive chunks share (see k_dgemm)
constexpr unsigned A_SLICE = TM * KB * 2, B_SLICE = TN * KB * 2;
constexpr unsigned STAGE = NP * (A_SLICE + B_SLICE);
constexpr int RAW_MIN = 600, RAW_MAX = 1500;  // biased exponents of rows whose products stay normal

static_assert(OV >= 0 && OV < NP, "a chunk's blocks exceed tensor memory");

struct DJob {
  long long a_off, b_off, out_off;
  double bscale;
  int m, n, K, lda, ldb, ldo;
  int kidx_off, w_off, phase_off;
  int bsel, sign, accumulate, nosym;
  int m_pad, nkb, nchunk;
  int exp_base;       // first row in the exponent arrays
  int row_base;       // first row in the planes: K block kb, row i is row_base + kb m_pad + i
};

struct DTile {
  int job, I, J;
};

// listed elements of a job's block: bit 8 r + c of mask is (i + r, j + c)
struct __align__(16) DBlock {
  unsigned long long mask;
  int job;
  int i, j;
  int pad[3];
};

__host__ __device__ __forceinline__ int chunk_begin(int nkb, int nchunk, int c) { return (int)((long long)nkb * c / nchunk); }

}  // namespace

struct DgemmPlan {
  int family = 0;
  int njobs = 0, ntiles = 0, grid = 0;
  long long rows = 0, exp_rows = 0;
  void* mem = nullptr;  // everything below
  DJob* d_jobs = nullptr;
  DTile* d_tiles = nullptr;
  int* d_cta = nullptr;
  __nv_bfloat16* arr[2] = {nullptr, nullptr};  // planes of A and of B
  // [2 exp_rows] raw row exponents of A, of B, [2 exp_rows] the rows' counts of
  // nonzero elements, [2 grid] listed blocks of each CTA: published, taken
  int* d_exp = nullptr;
  DBlock* d_list = nullptr;
  int4 *d_rblk = nullptr, *d_dblk = nullptr;
  int n_rblk = 0, n_dblk = 0;
  CUtensorMap maps[4];  // A rows of A, of B (128-row boxes); B rows of A, of B (32-row boxes)
  size_t smem = 0;
  bool share = false;  // listed blocks among all CTAs
  unsigned wait = WAIT_LIMIT;
};

// ----------------------------------------------------------------- device
namespace {

// biased exponent; 1 for a subnormal, so that only a zero gives 0
__device__ __forceinline__ int dexp1(double v)
{
  const unsigned long long b = (unsigned long long)__double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFull;
  const int E = (int)(b >> 52);
  return E == 0 && b != 0 ? 1 : E;
}

// B's column scale (job scale x launch scale x ladder weight): every weight of
// a closed shell is +-1, a sign flip; any other is an FP64 multiply, rounded
// as the FP64 kernel rounds it.  (The slicing passes spend one FP64
// instruction an element otherwise: 250 us instead of 55 for the emax=10
// ladder's exponents.)
enum { SC_PLUS = 0, SC_MINUS = 1, SC_OTHER = 2 };
__device__ __forceinline__ int scale_kind(double sc)
{
  const unsigned long long b = (unsigned long long)__double_as_longlong(sc);  // (not on the FP64 pipe)
  return (b & 0x7FFFFFFFFFFFFFFFull) == 0x3FF0000000000000ull ? (b >> 63 ? SC_MINUS : SC_PLUS) : SC_OTHER;
}
__device__ __forceinline__ double scaled(double v, int kind, double sc)
{
  if (kind == SC_OTHER) return v * sc;
  return __longlong_as_double(__double_as_longlong(v) ^ ((long long)kind << 63));
}

__device__ __forceinline__ bool row_bad(int raw) { return raw != 0 && (raw < RAW_MIN || raw > RAW_MAX); }
__device__ __forceinline__ int row_e(int raw) { return raw - 1022; }

// Raw row exponents of A and B (largest biased exponent of the row): a block
// per listed (job, 32-row group, 256-column chunk), partial maxima combined
// by atomicMax.  Bound by its operand loads: four columns in flight a thread.
__global__ void __launch_bounds__(256) k_dgemm_rowexp(const DJob* __restrict__ jobs, const int4* __restrict__ blocks,
                                                      const double* __restrict__ Abase, const double* __restrict__ B0,
                                                      const double* __restrict__ B1, const int* __restrict__ kidx,
                                                      const double* __restrict__ kw, double gbscale,
                                                      int* __restrict__ rexpA, int* __restrict__ rexpB,
                                                      int* __restrict__ cntA, int* __restrict__ cntB)
{
  __shared__ int sa[8][33], sb[8][33];  // largest exponent | count of nonzeros << 11
  __shared__ int s_col[256], s_kind[256];
  __shared__ double s_sc[256];
  const int4 bk = blocks[blockIdx.x];
  const DJob jb = jobs[bk.x];
  const int r = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int i = bk.y * 32 + r;
  const int t0 = bk.z * 256, tend = min(jb.K, t0 + 256);
  {
    const int t = t0 + threadIdx.x;
    if (t < tend) {
      s_col[threadIdx.x] = jb.kidx_off >= 0 ? kidx[jb.kidx_off + t] : t;
      s_sc[threadIdx.x] = jb.bscale * gbscale * (jb.w_off >= 0 ? kw[jb.w_off + t] : 1.0);
      s_kind[threadIdx.x] = scale_kind(s_sc[threadIdx.x]);
    }
  }
  __syncthreads();
  const double* A = Abase + jb.a_off;
  const double* B = (jb.bsel ? B1 : B0) + jb.b_off;
  const bool oka = i < jb.m, okb = i < jb.n;
  int ea = 0, eb = 0, na = 0, nb = 0;
  auto see = [](double v, int& e, int& n) {
    const int x = dexp1(v);
    e = max(e, x);
    n += x != 0;
  };
  int t = t0 + ty;
  for (; t + 24 < tend; t += 32) {
    double a[4], b[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long col = s_col[t + 8 * u - t0];
      a[u] = oka ? A[col * jb.lda + i] : 0.0;
      b[u] = okb ? B[col * jb.ldb + i] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      see(a[u], ea, na);
      see(scaled(b[u], s_kind[t + 8 * u - t0], s_sc[t + 8 * u - t0]), eb, nb);
    }
  }
  for (; t < tend; t += 8) {
    const long long col = s_col[t - t0];
    if (oka) see(A[col * jb.lda + i], ea, na);
    if (okb) see(scaled(B[col * jb.ldb + i], s_kind[t - t0], s_sc[t - t0]), eb, nb);
  }
  sa[ty][r] = ea | na << 11;
  sb[ty][r] = eb | nb << 11;
  __syncthreads();
  if (ty == 0) {
    for (int y = 1; y < 8; ++y) {
      ea = max(ea, sa[y][r] & 0x7FF);
      eb = max(eb, sb[y][r] & 0x7FF);
      na += sa[y][r] >> 11;
      nb += sb[y][r] >> 11;
    }
    if (ea) atomicMax(rexpA + jb.exp_base + i, ea);
    if (eb) atomicMax(rexpB + jb.exp_base + i, eb);
    if (na) atomicAdd(cntA + jb.exp_base + i, na);
    if (nb) atomicAdd(cntB + jb.exp_base + i, nb);
  }
}

// v 2^(P - e), rounded to an integer, for |v| < 2^e (v of a row in range)
__device__ __forceinline__ long long fixed_of(double v, int e)
{
  const long long bits = __double_as_longlong(v);
  const int E = (int)((bits >> 52) & 0x7FF);
  if (E == 0) return 0;
  const long long M = (bits & 0xFFFFFFFFFFFFFll) | 0x10000000000000ll;
  const int r = 1075 - E - P + e;  // right shift, >= 53 - P
  if (r > 54) return 0;
  const long long q = r <= 0 ? M << min(-r, P - 53) : (M + (1ll << (r - 1))) >> r;
  return bits < 0 ? -q : q;
}

// |v| 2^-e as BF16 (truncated), exponents clamped at 2^-60; 0 only for v = 0
__device__ __forceinline__ unsigned magnitude_of(double v, int e)
{
  const unsigned long long b = (unsigned long long)__double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFull;
  if (b == 0) return 0;
  const int x = (int)(b >> 52) - 1023 - e;  // <= -1
  if (x < -60) return (unsigned)(127 - 60) << 7;
  return ((unsigned)(127 + min(x, 0)) << 7) | (unsigned)((b >> 45) & 0x7F);
}

// The ten planes of A and of B for 32 rows from r0 and KB columns from t0 of
// a job, by a block of 256 threads: through shared memory to 16-byte stores
// (a plane's 32 x KB values are 2 KB in a row).  Bound by HBM: 16 bytes read
// and 40 written per element pair; every operand load of a thread is issued
// before its first conversion.  s_e: the rows' exponents in A and B.
constexpr int RW = (KB + 2) / 2;  // 17 words a row: a warp's 32 rows in 32 banks
struct SliceShared {
  unsigned dg[NP][32][RW];
  int e[2][32], col[KB], kind[KB];
  double sc[KB];
};

__device__ __forceinline__ void slice_block(SliceShared& sh, const DJob& jb, const double* __restrict__ A,
                                            const double* __restrict__ B, int r0, int kb, const int* __restrict__ kidx,
                                            const double* __restrict__ kw, double gbscale, long long plane_rows,
                                            __nv_bfloat16* __restrict__ pA, __nv_bfloat16* __restrict__ pB)
{
  const int t0 = kb * KB;
  if (threadIdx.x >= 32 && threadIdx.x < 32 + KB) {
    const int tt = threadIdx.x - 32, t = t0 + tt;
    sh.col[tt] = t < jb.K ? (jb.kidx_off >= 0 ? kidx[jb.kidx_off + t] : t) : 0;
    sh.sc[tt] = t < jb.K ? jb.bscale * gbscale * (jb.w_off >= 0 ? kw[jb.w_off + t] : 1.0) : 1.0;
    sh.kind[tt] = scale_kind(sh.sc[tt]);
  }
  __syncthreads();
  constexpr int NIT = 32 * (KB / 2) / 256;
  double v[2][NIT][2];
#pragma unroll
  for (int u = 0; u < NIT; ++u) {
    const int e = threadIdx.x + u * 256, i = r0 + (e & 31);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int tt = 2 * (e >> 5) + h;
      const bool ok = t0 + tt < jb.K;
      v[0][u][h] = ok && i < jb.m ? A[(long long)sh.col[tt] * jb.lda + i] : 0.0;
      v[1][u][h] = ok && i < jb.n ? B[(long long)sh.col[tt] * jb.ldb + i] : 0.0;
    }
  }
  long long bias = 0;  // half a digit in every lower digit: the fields of q + bias minus half are balanced
#pragma unroll
  for (int s = 1; s < S; ++s) bias += 1ll << (BETA * (S - 1 - s) + BETA - 1);
#pragma unroll
  for (int op = 0; op < 2; ++op) {
#pragma unroll
    for (int u = 0; u < NIT; ++u) {
      const int e = threadIdx.x + u * 256, r = e & 31, tp = e >> 5;
      long long q[2];
      unsigned mag[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const double x = op ? scaled(v[1][u][h], sh.kind[2 * tp + h], sh.sc[2 * tp + h]) : v[0][u][h];
        q[h] = fixed_of(x, sh.e[op][r]) + bias;
        mag[h] = magnitude_of(x, sh.e[op][r]);
      }
#pragma unroll
      for (int s = 0; s < S; ++s) {
        const int shf = BETA * (S - 1 - s);
        // small integer -> BF16: 1.5 * 2^23 + x minus 1.5 * 2^23, upper half; "- half" rides in the constant
        const int mg = s == 0 ? 0x4B400000 : 0x4B400000 - (1 << (BETA - 1));
        float f[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int x = s == 0 ? (int)(q[h] >> shf) : (int)((unsigned)(q[h] >> shf) & ((1u << BETA) - 1));
          f[h] = __int_as_float(mg + x) - 12582912.0f;
        }
        sh.dg[s][r][tp] = __byte_perm(__float_as_uint(f[0]), __float_as_uint(f[1]), 0x7632);
      }
      sh.dg[S][r][tp] = mag[0] | (mag[1] << 16);
    }
    __syncthreads();
    __nv_bfloat16* out = op ? pB : pA;
    const long long row0 = jb.row_base + (long long)kb * jb.m_pad + r0;
    for (int e = threadIdx.x; e < NP * 32 * (KB / 8); e += 256) {
      const int x = e % (KB / 8), r = (e / (KB / 8)) & 31, s = e / (32 * (KB / 8));
      const unsigned* d = &sh.dg[s][r][x * 4];
      *(uint4*)(out + ((long long)s * plane_rows + row0 + r) * KB + x * 8) = make_uint4(d[0], d[1], d[2], d[3]);
    }
    __syncthreads();
  }
}

// long reductions: a block per listed (job, 32-row group, KB-column group),
// the row exponents from k_dgemm_rowexp
__global__ void __launch_bounds__(256) k_dgemm_digits(const DJob* __restrict__ jobs, const int4* __restrict__ blocks,
                                                      const double* __restrict__ Abase, const double* __restrict__ B0,
                                                      const double* __restrict__ B1, const int* __restrict__ kidx,
                                                      const double* __restrict__ kw, double gbscale,
                                                      const int* __restrict__ rexpA, const int* __restrict__ rexpB,
                                                      long long plane_rows, __nv_bfloat16* __restrict__ pA,
                                                      __nv_bfloat16* __restrict__ pB)
{
  __shared__ SliceShared sh;
  const int4 bk = blocks[blockIdx.x];
  const DJob jb = jobs[bk.x];
  const int r0 = bk.y * 32;
  if (threadIdx.x < 32) {
    sh.e[0][threadIdx.x] = row_e(rexpA[jb.exp_base + r0 + threadIdx.x]);
    sh.e[1][threadIdx.x] = row_e(rexpB[jb.exp_base + r0 + threadIdx.x]);
  }
  slice_block(sh, jb, Abase + jb.a_off, (jb.bsel ? B1 : B0) + jb.b_off, r0, bk.z, kidx, kw, gbscale, plane_rows, pA, pB);
}

// short reductions (at most SHORT_KB K blocks a job): exponents, counts and
// planes of a 32-row group in one block, one launch where the long form takes a
// clear and two (the lists' counters are cleared here too)
__global__ void __launch_bounds__(256) k_dgemm_slice(const DJob* __restrict__ jobs, const int4* __restrict__ blocks,
                                                     const double* __restrict__ Abase, const double* __restrict__ B0,
                                                     const double* __restrict__ B1, const int* __restrict__ kidx,
                                                     const double* __restrict__ kw, double gbscale, int* __restrict__ rexpA,
                                                     int* __restrict__ rexpB, int* __restrict__ cntA, int* __restrict__ cntB,
                                                     int* __restrict__ nlist, int nclear, long long plane_rows,
                                                     __nv_bfloat16* __restrict__ pA, __nv_bfloat16* __restrict__ pB)
{
  __shared__ SliceShared sh;
  __shared__ int s_max[2][8][33];
  const int4 bk = blocks[blockIdx.x];
  const DJob jb = jobs[bk.x];
  const int r0 = bk.y * 32, r = threadIdx.x & 31, ty = threadIdx.x >> 5, i = r0 + r;
  const double* A = Abase + jb.a_off;
  const double* B = (jb.bsel ? B1 : B0) + jb.b_off;
  for (int c = blockIdx.x * 256 + threadIdx.x; c < nclear; c += gridDim.x * 256) nlist[c] = 0;
  int ea = 0, eb = 0, na = 0, nb = 0;
#pragma unroll 4
  for (int t = ty; t < jb.K; t += 8) {
    const long long col = jb.kidx_off >= 0 ? kidx[jb.kidx_off + t] : t;
    const double sc = jb.bscale * gbscale * (jb.w_off >= 0 ? kw[jb.w_off + t] : 1.0);
    const int xa = i < jb.m ? dexp1(A[col * jb.lda + i]) : 0;
    const int xb = i < jb.n ? dexp1(scaled(B[col * jb.ldb + i], scale_kind(sc), sc)) : 0;
    ea = max(ea, xa);
    eb = max(eb, xb);
    na += xa != 0;
    nb += xb != 0;
  }
  s_max[0][ty][r] = ea | na << 11;
  s_max[1][ty][r] = eb | nb << 11;
  __syncthreads();
  if (ty < 2) {
    int e = 0, n = 0;
    for (int y = 0; y < 8; ++y) {
      e = max(e, s_max[ty][y][r] & 0x7FF);
      n += s_max[ty][y][r] >> 11;
    }
    sh.e[ty][r] = row_e(e);
    (ty ? rexpB : rexpA)[jb.exp_base + i] = e;
    (ty ? cntB : cntA)[jb.exp_base + i] = n;
  }
  for (int kb = 0; kb < jb.nkb; ++kb)  // (slice_block's first barrier covers sh.e)
    slice_block(sh, jb, A, B, r0, kb, kidx, kw, gbscale, plane_rows, pA, pB);
}

struct DArgs {
  const DJob* jobs;
  const DTile* tiles;
  const int* cta_first;
  const int *rexpA, *rexpB, *cntA, *cntB;
  const int* phase;
  double* out;
  // to evaluate exactly: each CTA lists from TILE_BLKS times its first tile's
  // place; published[cta] entries of it are complete, taken[cta] taken
  DBlock* list;
  int *published, *taken;
  // for that: the operands as they are
  const double *A, *B0, *B1;
  const int* kidx;
  const double* kw;
  double gbscale;
  int gsign, accum, nomirror, share;
  unsigned wait;  // bound of every barrier wait
};

// what the roles of a CTA need to know of a tile, gathered one or two tiles
// ahead by a warp of its own: a chain of three dependent loads (tile, job,
// exponents), and sixteen exponent and phase loads a thread, cost the
// epilogue 30k of its 45k cycles a tile of the emax=10 Zbar product
struct TileInfo {
  double* O;
  int job, m, n, ldo, nosym, nkb, nchunk, m_pad, row_base, accumulate, I, J;
  int rrow[2][TM], rcol[2][TN];  // raw exponents of the tile's rows and columns, in each half
  float nrow[2][TM], ncol[2][TN];  // their counts of nonzero elements, times 2^-18
  int prow[TM], pcol[TN];        // phases (rows carry the job's sign too)
};

// what the magnitudes of a half's chunks say of a thread's 16 columns: sum
// |a||b| is not zero, and at least 2^-9 sqrt(count) in one of them
struct Guard {
  unsigned nonzero, enough;
};

// adds 16 columns of block g (a weight) to the thread's sums, or (g = S) tests
// the magnitudes, eight columns at a time (registers); n and nc: the row's and
// the columns' counts times 2^-18
template <int G>
__device__ __forceinline__ void take(unsigned taddr, long long (&hi)[COLS_W], long long (&lo)[COLS_W], Guard& gd, float n,
                                     const float* nc)
{
  if constexpr (G == S) {
#pragma unroll
    for (int h = 0; h < COLS_W; h += 8) {
      unsigned r[8];
      tmem_ld8(taddr + h, r);
      tmem_wait_ld();
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float x = __uint_as_float(r[c]);
        gd.nonzero |= (x != 0.f ? 1u : 0u) << (h + c);
        gd.enough |= (x * x >= fminf(n, nc[h + c]) ? 1u : 0u) << (h + c);
      }
    }
  } else {
    unsigned r[2][8];
    tmem_ld8(taddr, r[0]);
    tmem_ld8(taddr + 8, r[1]);
    tmem_wait_ld();
#pragma unroll
    for (int c = 0; c < COLS_W; ++c) {
      const float x = __uint_as_float(r[c >> 3][c & 7]);
      if (G < NHI)
        hi[c] += (long long)__float2int_rn(x) * (1ll << (BETA * (NHI - 1 - (G < NHI ? G : 0))));
      else
        lo[c] += (long long)__float2int_rn(x) * (1ll << (BETA * (S - 1 - (G < S ? G : 0))));
    }
  }
}

template <int G, int N>
__device__ __forceinline__ void take_run(unsigned base, long long (&hi)[COLS_W], long long (&lo)[COLS_W], Guard& gd, float n,
                                         const float* nc, bool live)
{
  if constexpr (N > 0) {
    if (live) take<G>(base + G * TN, hi, lo, gd, n, nc);
    take_run<G + 1, N - 1>(base, hi, lo, gd, n, nc, live);
  }
}

// (hi + lo 2^-28) 2^X as FP64, rounded once to nearest even (rows in range
// keep it normal).  Three 32-bit words and no branch: conversions and an FMA
// would run on the FP64 pipe, and the same steps with 64-bit shifts and
// branches took the emax=10 commutator from 7.71 to 8.02 ms.
__device__ __forceinline__ double value_of(long long hi, long long lo, int X)
{
  constexpr int LB = BETA * (S - NHI);
  const long long h = hi + (lo >> LB);
  // h 2^LB + l as a signed 96-bit number, then its magnitude
  const unsigned h0 = (unsigned)h, h1 = (unsigned)((unsigned long long)h >> 32), sg = (unsigned)((int)h1 >> 31);
  unsigned w0 = (h0 << LB | ((unsigned)lo & ((1u << LB) - 1))) ^ sg;
  unsigned w1 = __funnelshift_l(h0, h1, LB) ^ sg;
  unsigned w2 = (unsigned)((int)h1 >> (32 - LB)) ^ sg;
  asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, 0;\n\taddc.u32 %2, %2, 0;" : "+r"(w0), "+r"(w1), "+r"(w2) : "r"(sg & 1u));
  // leading one to bit 31 of w2
  int e = X + 1022 + 95 - LB;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const bool z = w2 == 0;
    e = z ? e - 32 : e;
    w2 = z ? w1 : w2;
    w1 = z ? w0 : w1;
    w0 = z ? 0 : w0;
  }
  const int sh = __clz(w2) & 31;
  const bool zero = w2 == 0;
  w2 = __funnelshift_l(w1, w2, sh);
  w1 = __funnelshift_l(w0, w1, sh);
  w0 <<= sh;
  // 53 bits of w2:w1; the leading one carries into the exponent field (and so does a carry out of rounding)
  unsigned ml = __funnelshift_r(w1, w2, 11), mh = (w2 >> 11) + ((unsigned)(e - sh) << 20);
  const unsigned tail = (w1 << 21) | (w0 != 0 ? 1u : 0u) | (ml & 1u);  // (low bits of w1 << 21 are 0)
  asm("add.cc.u32 %0, %0, %2;\n\taddc.u32 %1, %1, 0;" : "+r"(ml), "+r"(mh) : "r"(tail > 0x80000000u ? 1u : 0u));
  return zero ? 0.0 : __hiloint2double((int)(mh | (sg & 0x80000000u)), (int)ml);
}

// out (+)= v at (i, j) and, for a symmetrised job, its mirror
// (f: the job's sign and the phases of i and j)
__device__ __forceinline__ void put_exact(const DJob& jb, double* O, double f, int i, int j, double p1, double p2, bool accumulate,
                                          int nomirror)
{
  double* d = O + (long long)j * jb.ldo + i;
  if (jb.nosym) {
    *d = accumulate ? *d + p1 : p1;
    return;
  }
  const double v = p1 + f * p2, w = p2 + f * p1;
  *d = accumulate ? *d + v : v;
  if (i != j && !nomirror) {
    double* t = O + (long long)i * jb.ldo + j;
    *t = accumulate ? *t + w : w;
  }
}

// a thread's columns that the tile's matrix has, on or above the diagonal of a
// symmetrised job (those below are another element's mirror)
__device__ __forceinline__ unsigned own_columns(int i, int j0, int m, int n, int nosym)
{
  unsigned b = i >= m || j0 >= n ? 0u : n - j0 < COLS_W ? (1u << (n - j0)) - 1 : (1u << COLS_W) - 1;
  if (!nosym && i > j0) b &= i - j0 < COLS_W ? ~0u << (i - j0) : 0u;
  return b;
}

// lists the bad columns of a warp's 32 rows x 16 columns, by blocks; i, j: the
// first element of the lane's block
__device__ __forceinline__ void list_blocks(DBlock* list, int* n, int job, int i, int j, unsigned bad)
{
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int c = 0; c < COLS_W / BLK; ++c) {
    const unsigned b = (bad >> (BLK * c)) & 0xFFu;
    unsigned lo = (lane & 4) ? 0u : b << (8 * (lane & 3)), hi = (lane & 4) ? b << (8 * (lane & 3)) : 0u;
#pragma unroll
    for (int o = 1; o < BLK; o <<= 1) {
      lo |= __shfl_xor_sync(0xffffffffu, lo, o);
      hi |= __shfl_xor_sync(0xffffffffu, hi, o);
    }
    if ((lane & 7) == 0 && (lo | hi))
      list[atomicAdd(n, 1)] = {(unsigned long long)hi << 32 | lo, job, i, j + BLK * c};
  }
}

// the entries before n, written before this thread's last barrier, for other CTAs
__device__ __forceinline__ void publish(int* at, int n)
{
  __threadfence();
  *(volatile int*)at = n;
}

// the rank-th set bit of a block's mask
__device__ __forceinline__ int nth_bit(unsigned long long mask, int rank)
{
  int bit = 0;
#pragma unroll
  for (int w = 32; w > 0; w >>= 1) {
    const int c = __popcll((mask >> bit) & ((1ull << w) - 1));
    if (rank >= c) {
      rank -= c;
      bit += w;
    }
  }
  return bit;
}

__device__ __forceinline__ int sign_of(const DArgs& g, const DJob& jb, int i, int j)
{
  return (jb.sign != 0 ? jb.sign : g.gsign) * (jb.phase_off >= 0 ? g.phase[jb.phase_off + i] * g.phase[jb.phase_off + j] : 1);
}

__device__ __forceinline__ void put_listed(const DArgs& g, const DJob& jb, int sign, int i, int j, double p1, double p2)
{
  put_exact(jb, g.out + jb.out_off, (double)sign, i, j, p1, p2, g.accum > 0 || (g.accum < 0 && jb.accumulate), g.nomirror);
}

// At most FEW elements of a block, by a warp: 32 / n lanes an element take K by
// turns and meet in a fixed tree; operands straight from L1 and L2, two columns
// a lane in flight (eight: 4.47 against 4.08 ms at emax 8 with a dominating
// diagonal, and the code of a launch's first block is read cold).
constexpr int FEW = 16;
__device__ __forceinline__ void exact_few(const DArgs& g, const DJob& jb, const DBlock& e, int n)
{
  const int lane = threadIdx.x & 31, nosym = jb.nosym;
  const double *A = g.A + jb.a_off, *B = (jb.bsel ? g.B1 : g.B0) + jb.b_off;
  const int* kidx = jb.kidx_off >= 0 ? g.kidx + jb.kidx_off : nullptr;
  const double* kw = jb.w_off >= 0 ? g.kw + jb.w_off : nullptr;
  const double sc0 = jb.bscale * g.gbscale;
  const int kind0 = scale_kind(sc0);
  int sh = 0;  // 2^sh slots for n elements (a slot too many repeats the last one)
  while ((1 << sh) < n) ++sh;
  const int slot = lane & ((1 << sh) - 1), part = lane >> sh, parts = 32 >> sh;
  const int bit = nth_bit(e.mask, min(slot, n - 1)), i = e.i + (bit >> 3), j = e.j + (bit & 7);
  const int sign = sign_of(g, jb, i, j);
  double p1 = 0.0, p2 = 0.0;
  constexpr int U = 2;
  for (int t0 = 0; t0 < jb.K; t0 += 32) {
    const int t = min(t0 + lane, jb.K - 1), nt = min(32, jb.K - t0);
    const int col = kidx ? kidx[t] : t;
    const double sc = kw ? scaled(kw[t], kind0, sc0) : sc0;
    const int kind = scale_kind(sc);
    const bool fractions = __any_sync(0xffffffffu, kind == SC_OTHER);
    for (int u0 = 0; u0 < nt; u0 += U * parts) {
      double x[U], y[U], x2[U], y2[U];
#pragma unroll
      for (int v = 0; v < U; ++v) {
        const int k = u0 + v * parts + part;
        const long long c = __shfl_sync(0xffffffffu, col, min(k, nt - 1));
        const double *a = A + c * jb.lda, *b = B + c * jb.ldb;
        x[v] = k < nt ? a[i] : 0.0;
        y[v] = k < nt ? b[j] : 0.0;
        x2[v] = k < nt && !nosym ? a[j] : 0.0;
        y2[v] = k < nt && !nosym ? b[i] : 0.0;
      }
#pragma unroll
      for (int v = 0; v < U; ++v) {
        if (u0 + v * parts >= nt) break;
        const int k = min(u0 + v * parts + part, nt - 1), kd = __shfl_sync(0xffffffffu, kind, k);
        if (fractions) {
          const double s = __shfl_sync(0xffffffffu, sc, k);
          y[v] = scaled(y[v], kd, s);
          y2[v] = scaled(y2[v], kd, s);
        } else {  // (a sign flip: no multiply on the FP64 pipe)
          y[v] = scaled(y[v], kd & 1, 1.0);
          y2[v] = scaled(y2[v], kd & 1, 1.0);
        }
        p1 = fma(x[v], y[v], p1);
        if (!nosym) p2 = fma(x2[v], y2[v], p2);
      }
    }
  }
  for (int o = 1 << sh; o < 32; o <<= 1) {
    p1 += __shfl_xor_sync(0xffffffffu, p1, o);
    p2 += __shfl_xor_sync(0xffffffffu, p2, o);
  }
  if (part == 0 && slot < n) put_listed(g, jb, sign, i, j, p1, p2);
}

// More elements, E a lane.  Columns of the operands at the block's eight rows i
// and eight rows j are asynchronous copies of 8 bytes a lane into the warp's
// part of the pipeline's shared memory (one column a copy, or two of a plain
// job's), two steps of XK columns ahead; the few columns with a weight that is
// not 1 are scaled there, a common sign is applied at the end.  Bound by the
// FP64 pipe, one FMA a warp every 16 cycles of an SM.  (With every column scaled
// and one column of a plain job a copy: 78 against 61 ms for the emax 10
// commutator of operands falling off as 2^(-4 |de|), 80 against 44 for the tensor
// one at emax 8; the few this way: 1.70 against 1.46 ms at emax 8 with a
// generator.)
constexpr int XK = 32;  // columns a step
constexpr int XSTAGES = 3;
constexpr int XWARP = XSTAGES * XK * 32;  // doubles a warp
static_assert(EPIW * XWARP * 8 <= NSTAGE * (int)STAGE, "exact_work's buffers exceed the pipeline's");

// ALL: all 64 elements (E = 2): a lane's two are in one column
template <int E, bool NOSYM, bool ALL>
__device__ __forceinline__ void exact_many(const DArgs& g, const DJob& jb, const DBlock& e, int n, double* buf)
{
  constexpr int W = NOSYM ? 16 : 32;          // words of a column: A(i ..), [B(i ..), A(j ..),] B(j ..)
  constexpr int AT_AJ = 16, AT_BI = 8, AT_BJ = NOSYM ? 8 : 24;
  constexpr int STEP = XK * 32;               // doubles from one step's buffer to the next
  const int lane = threadIdx.x & 31;
  // what this lane copies (rows past the end repeat the last one, and are not
  // used): column k + half of row, k + half even in a plain job's first half
  const int strip = NOSYM ? ((lane >> 3) & 1) * 3 : lane >> 3, half = NOSYM ? lane >> 4 : 0;
  const int row = min((strip < 2 ? e.i : e.j) + (lane & 7), (strip & 1 ? jb.n : jb.m) - 1);
  const double* src = (strip & 1 ? (jb.bsel ? g.B1 : g.B0) + jb.b_off : g.A + jb.a_off) + row;
  const int ld = strip & 1 ? jb.ldb : jb.lda;
  const unsigned dst = smem_u32(buf) + lane * 8;
  const int* kidx = jb.kidx_off >= 0 ? g.kidx + jb.kidx_off : nullptr;
  const double* kw = jb.w_off >= 0 ? g.kw + jb.w_off : nullptr;
  const double sc0 = jb.bscale * g.gbscale;
  const int kind0 = scale_kind(sc0);
  int er[E], ec[E];  // row and column within the block (a lane too many repeats the last element)
  double p1[E], p2[E];
#pragma unroll
  for (int h = 0; h < E; ++h) {
    const int bit = ALL ? lane + 32 * h : nth_bit(e.mask, min(lane + 32 * h, n - 1));
    er[h] = bit >> 3;
    ec[h] = ALL ? lane & 7 : bit & 7;
    p1[h] = p2[h] = 0.0;
  }
  const int steps = (jb.K + XK - 1) / XK;
  auto column = [&](int step) { return kidx ? kidx[min(step * XK + lane, jb.K - 1)] : min(step * XK + lane, jb.K - 1); };
  int col = column(0);
  auto copy = [&](int step) {  // always one group, an empty one past the end (columns past it repeat the last)
    if (step < steps) {
      const unsigned d = dst + (step % XSTAGES) * (STEP * 8);
#pragma unroll 8
      for (int k = 0; k < XK; k += 32 / W) {
        const double* a = src + (long long)__shfl_sync(0xffffffffu, col, k + half) * ld;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d + k * (W * 8)), "l"(__cvta_generic_to_global(a)) : "memory");
      }
      col = column(step + 1);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  copy(0);
  copy(1);
  for (int step = 0; step < steps; ++step) {
    copy(step + 2);
    double* x = buf + (step % XSTAGES) * STEP;
    const int t0 = step * XK, nk = min(XK, jb.K - t0);
    const double w = kw && lane < nk ? kw[t0 + lane] : 1.0;
    asm volatile("cp.async.wait_group 2;" ::: "memory");
    __syncwarp();
    const double sc = kind0 == SC_OTHER ? sc0 * w : w;
    const int kind = lane < nk ? scale_kind(sc) : SC_PLUS;
    const unsigned scales = __ballot_sync(0xffffffffu, kind != SC_PLUS);
    if (scales) {
      for (unsigned m = scales; m; m &= m - 1) {
        const int k = __ffs(m) - 1, kd = __shfl_sync(0xffffffffu, kind, k);
        const double s = __shfl_sync(0xffffffffu, sc, k);
        if (lane < W && (lane >> 3 & 1)) x[k * W + lane] = scaled(x[k * W + lane], kd, s);
      }
      __syncwarp();
    }
#pragma unroll 4
    for (int k = 0; k < nk; ++k) {
      const double* q = x + k * W;
#pragma unroll
      for (int h = 0; h < E; ++h) {
        p1[h] = fma(q[er[h]], q[AT_BJ + (ALL ? ec[0] : ec[h])], p1[h]);
        if (!NOSYM) p2[h] = fma(q[AT_AJ + (ALL ? ec[0] : ec[h])], q[AT_BI + er[h]], p2[h]);
      }
    }
    __syncwarp();
  }
#pragma unroll
  for (int h = 0; h < E; ++h)
    if (lane + 32 * h < n)
      put_listed(g, jb, sign_of(g, jb, e.i + er[h], e.j + ec[h]), e.i + er[h], e.j + ec[h], kind0 == SC_MINUS ? -p1[h] : p1[h],
                 kind0 == SC_MINUS ? -p2[h] : p2[h]);
}

template <bool NOSYM>
__device__ __forceinline__ void exact_many(const DArgs& g, const DJob& jb, const DBlock& e, int n, double* buf)
{
  if (n <= 32)
    exact_many<1, NOSYM, false>(g, jb, e, n, buf);
  else if (n < 64)
    exact_many<2, NOSYM, false>(g, jb, e, n, buf);
  else
    exact_many<2, NOSYM, true>(g, jb, e, n, buf);
}

// the k-th block of a list that another CTA may have written
__device__ __forceinline__ void exact_block(const DArgs& g, const DBlock* at, double* buf)
{
  DBlock e;
  e.mask = __ldcg(&at->mask);
  e.job = __ldcg(&at->job);
  e.i = __ldcg(&at->i);
  e.j = __ldcg(&at->j);
  const DJob jb = g.jobs[e.job];
  const int n = __popcll(e.mask);
  if (n <= FEW)
    exact_few(g, jb, e, n);
  else if (jb.nosym)
    exact_many<true>(g, jb, e, n, buf);
  else
    exact_many<false>(g, jb, e, n, buf);
}

// The listed blocks, a warp at a time: this CTA's own n (all complete), then
// those that other CTAs have published by now.  Nothing waits: every CTA ends
// with its own list taken, by itself or by others.  Plans whose whole tiles
// take a few microseconds share nothing: looking at the other lists and drawing
// tickets would be as long (replay of nine FP64 pairs at emax 2 138.7 us
// against 128).
__device__ __noinline__ void exact_work(const DArgs& g, int n, double* buf)
{
  const int lane = threadIdx.x & 31, grid = gridDim.x;
  {
    // the first blocks by warp, then tickets, each drawn while the block before
    // is worked on (n is final, so counting past it harms nobody)
    const DBlock* list = g.list + (long long)g.cta_first[blockIdx.x] * TILE_BLKS;
    for (int k = (threadIdx.x >> 5) - 2; k < n;) {
      int next = k + EPIW;
      if (g.share && lane == 0) next = EPIW + atomicAdd(g.taken + blockIdx.x, 1);
      exact_block(g, list + k, buf);
      k = __shfl_sync(0xffffffffu, next, 0);
    }
  }
  if (!g.share) return;
  auto cta = [&](int d) { return (int)blockIdx.x + d < grid ? blockIdx.x + d : blockIdx.x + d - grid; };
  auto listed = [&](int d) { return d > 0 && d < grid ? *(volatile int*)(g.published + cta(d)) : 0; };
  int any = 0;
  for (int d = lane; d < grid; d += 32) any |= listed(d) > EPIW;
  if (!__any_sync(0xffffffffu, any)) return;
  for (int d0 = 0; d0 < grid; d0 += 32) {
    const int have = listed(d0 + lane);
    __threadfence();  // the entries after their count
    for (unsigned m = __ballot_sync(0xffffffffu, have > EPIW); m; m &= m - 1) {
      const int c = cta(d0 + __ffs(m) - 1), cn = __shfl_sync(0xffffffffu, have, __ffs(m) - 1);
      const DBlock* list = g.list + (long long)g.cta_first[c] * TILE_BLKS;
      for (;;) {
        int k = 0;
        if (lane == 0) {
          k = *(volatile int*)(g.taken + c);
          while (EPIW + k < cn) {
            const int old = atomicCAS(g.taken + c, k, k + 1);
            if (old == k) break;
            k = old;
          }
        }
        k = EPIW + __shfl_sync(0xffffffffu, k, 0);
        if (k >= cn) break;
        exact_block(g, list + k, buf);
      }
    }
  }
}

// Persistent kernel, one CTA per SM, each with its own run of tiles:
//   warp 0: TMA producer; warp 1: tensor memory and MMA issue (one thread);
//   warps 2-9: epilogue; warp 10: tile information.
// A chunk's ten blocks (nine weights, magnitudes) are NP x 32 of the 512
// columns of tensor memory.  Even chunks of a CTA start at column 0, odd ones
// end at the last, so consecutive chunks share OV = 4 blocks; the epilogue
// takes those first and releases them, and the next chunk's MMAs run under
// the rest.  (168 registers a thread: eleven warps on four register files are three a file.)
__global__ void __launch_bounds__(96 + 32 * EPIW, 1) k_dgemm(const __grid_constant__ CUtensorMap mAA,
                                                             const __grid_constant__ CUtensorMap mAB,
                                                             const __grid_constant__ CUtensorMap mBA,
                                                             const __grid_constant__ CUtensorMap mBB, DArgs g)
{
  constexpr int EPI_T = 32 * EPIW;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  // barriers: full[NSTAGE], empty[NSTAGE], acc_full[2], early, info_full[NINFO], info_empty[NINFO], drain; then the tensor-memory slot
  unsigned long long* bars = (unsigned long long*)(smem + NSTAGE * STAGE);
  unsigned* tmem_slot = (unsigned*)(bars + 2 * NSTAGE + 4 + 2 * NINFO);
  __shared__ TileInfo s_info[NINFO];
  __shared__ int s_err_, s_issued, s_nlist, s_published;  // listed blocks, how many of them are published
  volatile int& s_err = s_err_;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned sbase = smem_u32(smem), bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (NSTAGE + s); };
  auto acc_full = [&](int b) { return bar0 + 8u * (2 * NSTAGE + b); };
  const unsigned acc_early = bar0 + 8u * (2 * NSTAGE + 2);
  auto info_full = [&](int k) { return bar0 + 8u * (2 * NSTAGE + 3 + k); };
  auto info_empty = [&](int k) { return bar0 + 8u * (2 * NSTAGE + 3 + NINFO + k); };
  const unsigned drain = bar0 + 8u * (2 * NSTAGE + 3 + 2 * NINFO);
  if (threadIdx.x == 0) {
    s_err = 0;
    s_nlist = s_published = 0;
    for (int s = 0; s < NSTAGE; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(acc_full(0), 1);
    mbar_init(acc_full(1), 1);
    mbar_init(acc_early, EPI_T);
    mbar_init(drain, 1);
    for (int k = 0; k < NINFO; ++k) {
      mbar_init(info_full(k), 1);
      mbar_init(info_empty(k), EPI_T + 2);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem = *tmem_slot;
  const int tbeg = g.cta_first[blockIdx.x], ntile = g.cta_first[blockIdx.x + 1] - tbeg;

  if (warp == 2 + EPIW) {
    // ------------------------------------------------ tile information
    for (int t = 0; t < ntile; ++t) {
      const int k = t % NINFO;
      // (the lanes decide together too)
      const bool ok = !s_err && mbar_wait(info_empty(k), (unsigned)((t / NINFO) & 1) ^ 1u, g.wait);
      if (!__all_sync(0xffffffffu, ok)) {
        s_err = 1;
        break;
      }
      const DTile tl = g.tiles[tbeg + t];
      const DJob jb = g.jobs[tl.job];
      TileInfo& f = s_info[k];
      const int* ph = jb.phase_off >= 0 ? g.phase + jb.phase_off : nullptr;
      const int sign = jb.sign != 0 ? jb.sign : g.gsign;
      const int* ra = g.rexpA + jb.exp_base;
      const int* rb = g.rexpB + jb.exp_base;
      const int *na = g.cntA + jb.exp_base, *nb = g.cntB + jb.exp_base;
      int x[2][TM / 32 + 1], y[2][TM / 32 + 1], p[TM / 32 + 1];
#pragma unroll
      for (int u = 0; u <= TM / 32; ++u) {
        const int r = u < TM / 32 ? tl.I * TM + u * 32 + lane : tl.J * TN + lane;  // the last: the tile's columns
        const int lim = u < TM / 32 ? jb.m : jb.n;
        x[0][u] = r < lim ? (u < TM / 32 ? ra[r] : rb[r]) : 0;
        x[1][u] = r < lim && !jb.nosym ? (u < TM / 32 ? rb[r] : ra[r]) : 0;
        y[0][u] = r < lim ? (u < TM / 32 ? na[r] : nb[r]) : 0;
        y[1][u] = r < lim && !jb.nosym ? (u < TM / 32 ? nb[r] : na[r]) : 0;
        p[u] = ph && r < lim ? ph[r] : 1;
      }
      constexpr float N2 = 1.0f / (1 << 18);
#pragma unroll
      for (int u = 0; u < TM / 32; ++u) {
        f.rrow[0][u * 32 + lane] = x[0][u];
        f.rrow[1][u * 32 + lane] = x[1][u];
        f.nrow[0][u * 32 + lane] = (float)y[0][u] * N2;
        f.nrow[1][u * 32 + lane] = (float)y[1][u] * N2;
        f.prow[u * 32 + lane] = sign * p[u];
      }
      f.rcol[0][lane] = x[0][TM / 32];
      f.rcol[1][lane] = x[1][TM / 32];
      f.ncol[0][lane] = (float)y[0][TM / 32] * N2;
      f.ncol[1][lane] = (float)y[1][TM / 32] * N2;
      f.pcol[lane] = p[TM / 32];
      if (lane == 0) {
        f.O = g.out + jb.out_off;
        f.m = jb.m;
        f.n = jb.n;
        f.job = tl.job;
        f.ldo = jb.ldo;
        f.nosym = jb.nosym;
        f.nkb = jb.nkb;
        f.nchunk = jb.nchunk;
        f.m_pad = jb.m_pad;
        f.row_base = jb.row_base;
        f.accumulate = g.accum > 0 || (g.accum < 0 && jb.accumulate);
        f.I = tl.I;
        f.J = tl.J;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(info_full(k));
    }
  } else if (warp == 0) {
    // ------------------------------------------------ TMA producer
    if (lane == 0) {
      int it = 0;
      for (int t = 0; t < ntile && !s_err; ++t) {
        if (!mbar_wait(info_full(t % NINFO), (unsigned)((t / NINFO) & 1), g.wait)) {
          s_err = 1;
          break;
        }
        const TileInfo& f = s_info[t % NINFO];
        const int nkb = f.nkb, m_pad = f.m_pad, nhalf = f.nosym ? 1 : 2;
        const int rA = f.row_base + f.I * TM, rB = f.row_base + f.J * TN;
        mbar_arrive(info_empty(t % NINFO));
        for (int k = 0; k < nhalf * nkb; ++k, ++it) {
          const int st = it % NSTAGE;
          if (!mbar_wait(empty_bar(st), (unsigned)((it / NSTAGE) & 1) ^ 1u, g.wait)) {
            s_err = 1;
            break;
          }
          mbar_expect_tx(full_bar(st), STAGE);
          const bool second = k >= nkb;
          const int row = (second ? k - nkb : k) * m_pad;
          const unsigned sA = sbase + st * STAGE;
          tma_load_3d(sA, second ? &mAB : &mAA, 0, rA + row, full_bar(st));
          tma_load_3d(sA + NP * A_SLICE, second ? &mBA : &mBB, 0, rB + row, full_bar(st));
        }
      }
      s_issued = it;
    }
  } else if (warp == 1) {
    // ------------------------------------------------ MMA issuer
    if (lane == 0) {
      constexpr int MAXT = 256 / TN;
      int it = 0, cc = 0;
      for (int t = 0; t < ntile && !s_err; ++t) {
        if (!mbar_wait(info_full(t % NINFO), (unsigned)((t / NINFO) & 1), g.wait)) {
          s_err = 1;
          break;
        }
        const TileInfo& f = s_info[t % NINFO];
        const int nkb = f.nkb, nchunk = f.nchunk, nhalf = f.nosym ? 1 : 2;
        mbar_arrive(info_empty(t % NINFO));
        for (int hc = 0; hc < nhalf * nchunk && !s_err; ++hc, ++cc) {
          const int c = hc >= nchunk ? hc - nchunk : hc;
          const int len = chunk_begin(nkb, nchunk, c + 1) - chunk_begin(nkb, nchunk, c);
          // the shared blocks of the chunk before have been taken (and so all of the one before that)
          if (!mbar_wait(acc_early, (unsigned)((cc & 1) ^ 1), g.wait)) {
            s_err = 1;
            break;
          }
          tc_fence_after();
          const unsigned d = tmem + ((cc & 1) ? (NB - NP) * TN : 0);
          for (int kb = 0; kb < len; ++kb, ++it) {
            const int st = it % NSTAGE;
            if (!mbar_wait(full_bar(st), (unsigned)((it / NSTAGE) & 1), g.wait)) {
              s_err = 1;
              break;
            }
            tc_fence_after();
            const unsigned sA = sbase + st * STAGE;
            const unsigned long long a0 = sdesc_sw64(sA), b0 = sdesc_sw64(sA + NP * A_SLICE);
            const unsigned first = kb == 0 ? 0u : 1u;
            // the products (s, t) of one s over a run of t are one MMA: their
            // weights s + t are consecutive blocks of tensor memory, their B
            // tiles consecutive in shared memory
#pragma unroll
            for (int sub = 0; sub < KB / 16; ++sub) {
#pragma unroll
              for (int s = 0; s < S; ++s) {
                const unsigned long long ad = a0 + (unsigned long long)((s * A_SLICE + sub * 32) >> 4);
#pragma unroll
                for (int t0 = 0; t0 < S - s; t0 += MAXT) {
                  const int nt = (S - s - t0) < MAXT ? (S - s - t0) : MAXT;
                  tc_mma(d + (s + t0) * TN, ad, b0 + (unsigned long long)((t0 * B_SLICE + sub * 32) >> 4),
                         idesc_bf16(TM, nt * TN), (sub == 0 && s == 0) ? first : 1u);
                }
              }
              tc_mma(d + S * TN, a0 + (unsigned long long)((S * A_SLICE + sub * 32) >> 4),
                     b0 + (unsigned long long)((S * B_SLICE + sub * 32) >> 4), idesc_bf16(TM, TN),
                     sub == 0 ? first : 1u);
            }
            tc_commit(empty_bar(st));
          }
          if (s_err) break;
          tc_commit(acc_full(cc & 1));
        }
      }
    }
  } else {
    // ------------------------------------------------ epilogue
    const int q = warp & 3, cbeg = ((warp - 2) >> 2) * COLS_W, row = q * 32 + lane;
    int cc = 0, t = 0;
    for (; t < ntile; ++t) {
      const TileInfo& f = s_info[t % NINFO];
      // the epilogue warps decide together, so none waits at a barrier alone
      bool expired = barrier_any(1, EPI_T, !mbar_wait(info_full(t % NINFO), (unsigned)((t / NINFO) & 1), g.wait));
      if (expired) {
        s_err = 1;
        break;
      }
      // (the listing of the tile before is complete, that of this one not begun)
      if (threadIdx.x == 64 && s_nlist > s_published) publish(g.published + blockIdx.x, s_published = s_nlist);
      const int nosym = f.nosym, nchunk = f.nchunk;
      const int i = f.I * TM + row, j0 = f.J * TN + cbeg;
      // whether this warp writes any of its 32 x 16 elements: not where they
      // lie outside the matrix or below the diagonal.  A small job's tile is
      // mostly padding, and the warps share the pipe of the conversions:
      // commutator at emax 2 65.6 -> 61.8 us, 6 289 -> 281, 7 (Ca40) 630 -> 622
      const int row0 = f.I * TM + q * 32;
      const bool live = row0 < f.m && j0 < f.n && (nosym || row0 < j0 + COLS_W);
      unsigned bad = 0;  // this thread's columns that the digits cannot vouch for
      double v1[COLS_W], v2[COLS_W];
      for (int half = 0; half < (nosym ? 1 : 2); ++half) {
        long long hi[COLS_W], lo[COLS_W];
#pragma unroll
        for (int c = 0; c < COLS_W; ++c) hi[c] = lo[c] = 0;
        Guard gd{0, 0};
        for (int c = 0; c < nchunk; ++c, ++cc) {
          expired = barrier_any(1, EPI_T, !mbar_wait(acc_full(cc & 1), (unsigned)((cc >> 1) & 1), g.wait));
          if (expired) break;
          tc_fence_after();
          const unsigned lane_base = tmem + ((unsigned)(q * 32) << 16) + cbeg;
          if (cc & 1) {
            const unsigned base = lane_base + (NB - NP) * TN;
            take_run<0, OV>(base, hi, lo, gd, f.nrow[half][row], f.ncol[half] + cbeg, live);
            tc_fence_before();
            mbar_arrive(acc_early);
            take_run<OV, NP - OV>(base, hi, lo, gd, f.nrow[half][row], f.ncol[half] + cbeg, live);
          } else {
            take_run<NP - OV, OV>(lane_base, hi, lo, gd, f.nrow[half][row], f.ncol[half] + cbeg, live);
            tc_fence_before();
            mbar_arrive(acc_early);
            take_run<0, NP - OV>(lane_base, hi, lo, gd, f.nrow[half][row], f.ncol[half] + cbeg, live);
          }
        }
        if (expired) break;
        if (!live) continue;
        const int raw_i = f.rrow[half][row];
        bad |= row_bad(raw_i) ? (1u << COLS_W) - 1 : gd.nonzero & ~gd.enough;
#pragma unroll
        for (int c = 0; c < COLS_W; ++c) {
          const int raw_j = f.rcol[half][cbeg + c];
          bad |= (row_bad(raw_j) ? 1u : 0u) << c;
          const double v = value_of(hi[c], lo[c], row_e(raw_i) + row_e(raw_j) - (2 * P - 2 * BETA * (S - 1) + BETA * (NHI - 1)));
          if (half)
            v2[c] = v;
          else
            v1[c] = v;
        }
      }
      if (expired) {
        s_err = 1;
        break;
      }
      const int m = f.m, n = f.n, ldo = f.ldo;
      const bool accumulate = f.accumulate;
      double* O = f.O;
      // columns this thread writes: in the matrix, on or above the diagonal, not listed
      unsigned wd = own_columns(i, j0, m, n, nosym);
      bad &= wd;
      wd &= ~bad;
      if (__any_sync(0xffffffffu, bad)) list_blocks(g.list + (long long)tbeg * TILE_BLKS, &s_nlist, f.job, i & ~7, j0, bad);
      if (!nosym && live) {
        const int sp = f.prow[row];
#pragma unroll
        for (int c = 0; c < COLS_W; ++c) {
          const bool neg = sp * f.pcol[cbeg + c] < 0;
          v1[c] += neg ? -v2[c] : v2[c];
          v2[c] = neg ? -v1[c] : v1[c];
        }
      }
      mbar_arrive(info_empty(t % NINFO));
      unsigned wm = nosym || g.nomirror ? 0u : wd;
      if (i >= j0 && i < j0 + COLS_W) wm &= ~(1u << (i - j0));
      double* od = O + (long long)j0 * ldo + i;
      double* om = O + (long long)i * ldo + j0;
      if (!accumulate) {
#pragma unroll
        for (int c = 0; c < COLS_W; ++c) {
          if ((wd >> c) & 1) od[(long long)c * ldo] = v1[c];
          if ((wm >> c) & 1) om[c] = v2[c];
        }
      } else {
#pragma unroll
        for (int h = 0; h < COLS_W; h += 8) {
          // all old values of eight columns before their first store
          double x[8], y[8];
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            x[c] = (wd >> (h + c)) & 1 ? __ldcg(od + (long long)(h + c) * ldo) : 0.0;
            y[c] = (wm >> (h + c)) & 1 ? __ldcg(om + h + c) : 0.0;
          }
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            if ((wd >> (h + c)) & 1) od[(long long)(h + c) * ldo] = x[c] + v1[h + c];
            if ((wm >> (h + c)) & 1) om[h + c] = y[c] + v2[h + c];
          }
        }
      }
    }
    // a wait that ran out: the tiles not written are listed
    for (; t < ntile; ++t) {
      const DTile tl = g.tiles[tbeg + t];
      const DJob& jb = g.jobs[tl.job];
      const int i = tl.I * TM + row, j0 = tl.J * TN + cbeg;
      list_blocks(g.list + (long long)tbeg * TILE_BLKS, &s_nlist, tl.job, i & ~7, j0, own_columns(i, j0, jb.m, jb.n, jb.nosym));
    }
  }
  // every role has left its loop, and so has every copy and MMA, unless a wait
  // ran out; the lists are complete
  __syncthreads();
  if (s_err) drain_products(s_issued, NSTAGE, full_bar, drain);
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  } else if (warp >= 2 && warp < 2 + EPIW) {
    const int n = s_nlist;
    if (threadIdx.x == 64 && n > s_published) publish(g.published + blockIdx.x, n);
    exact_work(g, n, (double*)smem + (warp - 2) * XWARP);  // (the pipeline's shared memory is free)
  }
}

// a plane array as (K element, row, plane); a box is one K block x rows x all planes
void plane_map(CUtensorMap* m, void* base, long long rows, int box_rows)
{
  cuuint64_t dims[3] = {(cuuint64_t)KB, (cuuint64_t)rows, (cuuint64_t)NP};
  cuuint64_t strides[2] = {(cuuint64_t)KB * 2, (cuuint64_t)KB * 2 * (cuuint64_t)rows};
  cuuint32_t box[3] = {(cuuint32_t)KB, (cuuint32_t)box_rows, (cuuint32_t)NP};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = get_encode()(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, base, dims, strides, box, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) throw std::runtime_error("cuTensorMapEncodeTiled failed");
}

}  // namespace

// ------------------------------------------------------------------ host
size_t dgemm_plan_bytes(const std::vector<GemmJobDev>& jobs)
{
  // (planes, and the exponents and lists of the tiles; the job tables are small)
  size_t bytes = 1 << 20;
  for (const GemmJobDev& j : jobs) {
    const size_t n = j.nosym ? j.n : j.m, m_pad = (std::max<size_t>(j.m, n) + TM - 1) / TM * TM;
    const size_t nkb = std::max(1, (j.K + KB - 1) / KB);
    bytes += m_pad * (nkb * KB * 2 * NP * 2 + 4 * sizeof(int));
    bytes += (m_pad / TM) * ((n + TN - 1) / TN) * (sizeof(DTile) + sizeof(DBlock) * TILE_BLKS);
  }
  return bytes;
}

DgemmPlan* dgemm_plan_create(const std::vector<GemmJobDev>& jobs_in, int family)
{
  DgemmPlan* p = new DgemmPlan();
  p->family = family;
  std::vector<DJob> jobs;
  std::vector<DTile> tiles;
  std::vector<long long> cost;
  long long erow = 0, prow = 0;
  for (const GemmJobDev& j : jobs_in) {
    DJob d{};
    d.a_off = j.a_off;
    d.b_off = j.b_off;
    d.out_off = j.out_off;
    d.bscale = j.bscale;
    d.m = j.m;
    d.n = j.nosym ? j.n : j.m;
    d.K = j.K;
    d.lda = j.lda;
    d.ldb = j.ldb;
    d.ldo = j.ldo;
    d.kidx_off = j.kidx_off;
    d.w_off = j.w_off;
    d.phase_off = j.phase_off;
    d.bsel = j.bsel;
    d.sign = j.sign;
    d.accumulate = j.accumulate;
    d.nosym = j.nosym ? 1 : 0;
    d.m_pad = (std::max(d.m, d.n) + TM - 1) / TM * TM;
    d.nkb = std::max(1, (j.K + KB - 1) / KB);
    d.nchunk = (d.nkb + CH - 1) / CH;
    d.exp_base = (int)erow;
    d.row_base = (int)prow;
    erow += d.m_pad;
    prow += (long long)d.m_pad * d.nkb;
    if (prow > (1ll << 31) - TM || erow > (1ll << 31) - TM) {
      delete p;
      throw std::runtime_error("digit planes exceed 2^31 rows");
    }
    const int jix = (int)jobs.size();
    jobs.push_back(d);
    if (d.m == 0 || d.n == 0 || d.K == 0) continue;
    p->share = p->share || (long long)std::min(d.m, TM) * std::min(d.n, TN) * d.K * (d.nosym ? 1 : 2) > SHARE;
    // a tile costs its K blocks and, per chunk, about three of them in the epilogue, plus its stores
    const long long c = (d.nosym ? 1 : 2) * (d.nkb + 3 * d.nchunk) + 4;
    for (int I = 0; I * TM < d.m; ++I)
      for (int J = d.nosym ? 0 : I * (TM / TN); J * TN < d.n; ++J) {
        tiles.push_back({jix, I, J});
        cost.push_back(c);
      }
  }
  p->njobs = (int)jobs.size();
  p->ntiles = (int)tiles.size();
  p->rows = std::max<long long>(prow, TM);
  p->exp_rows = std::max<long long>(erow, TM);
  if (tiles.empty()) return p;
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  p->grid = std::max(1, std::min(nsm, p->ntiles));
  // longest first, each to the least loaded CTA; a CTA's tiles in that order
  std::vector<int> ord(tiles.size());
  for (size_t t = 0; t < ord.size(); ++t) ord[t] = (int)t;
  std::stable_sort(ord.begin(), ord.end(), [&](int a, int b) { return cost[a] > cost[b]; });
  std::vector<std::pair<long long, int>> heap;
  for (int b = 0; b < p->grid; ++b) heap.push_back({0, b});
  auto gt = [](const std::pair<long long, int>& x, const std::pair<long long, int>& y) { return x > y; };
  std::make_heap(heap.begin(), heap.end(), gt);
  std::vector<std::vector<int>> lists(p->grid);
  for (int t : ord) {
    std::pop_heap(heap.begin(), heap.end(), gt);
    heap.back().first += cost[t];
    lists[heap.back().second].push_back(t);
    std::push_heap(heap.begin(), heap.end(), gt);
  }
  std::vector<DTile> sorted;
  std::vector<int> first(p->grid + 1, 0);
  for (int b = 0; b < p->grid; ++b) {
    for (int t : lists[b]) sorted.push_back(tiles[t]);
    first[b + 1] = (int)sorted.size();
  }
  std::vector<int4> rb, db;
  int nkb_max = 0;
  for (const DJob& d : jobs) nkb_max = std::max(nkb_max, d.nkb);
  const bool shorts = nkb_max <= SHORT_KB;  // one slicing pass (n_dblk stays 0)
  for (int j = 0; j < p->njobs; ++j) {
    const DJob& d = jobs[j];
    if (d.m == 0 || d.n == 0 || d.K == 0) continue;
    for (int y = 0; y < d.m_pad / 32; ++y)
      for (int x = 0; x < (shorts ? 1 : (d.K + 255) / 256); ++x) rb.push_back(make_int4(j, y, x, 0));
  }
  // the digit pass starts on the operands that the exponent pass read last
  for (int j = p->njobs - 1; j >= 0 && !shorts; --j) {
    const DJob& d = jobs[j];
    if (d.m == 0 || d.n == 0 || d.K == 0) continue;
    for (int x = 0; x < d.nkb; ++x)
      for (int y = 0; y < d.m_pad / 32; ++y) db.push_back(make_int4(j, y, x, 0));
  }
  p->n_rblk = (int)rb.size();
  p->n_dblk = (int)db.size();
  try {
    // one allocation and one copy a plan (a batch of new operators makes two
    // plans a group): the tables, then the exponents, lists and planes
    size_t size = 0;
    auto take = [&](size_t bytes) {
      const size_t at = size;
      size += (std::max<size_t>(bytes, 16) + 1023) / 1024 * 1024;
      return at;
    };
    const size_t o_jobs = take(sizeof(DJob) * jobs.size()), o_tiles = take(sizeof(DTile) * sorted.size());
    const size_t o_cta = take(sizeof(int) * first.size());
    const size_t o_rblk = take(sizeof(int4) * rb.size()), o_dblk = take(sizeof(int4) * db.size());
    std::vector<char> tables(size, 0);
    std::memcpy(tables.data() + o_jobs, jobs.data(), sizeof(DJob) * jobs.size());
    std::memcpy(tables.data() + o_tiles, sorted.data(), sizeof(DTile) * sorted.size());
    std::memcpy(tables.data() + o_cta, first.data(), sizeof(int) * first.size());
    if (!rb.empty()) std::memcpy(tables.data() + o_rblk, rb.data(), sizeof(int4) * rb.size());
    if (!db.empty()) std::memcpy(tables.data() + o_dblk, db.data(), sizeof(int4) * db.size());
    const size_t o_exp = take(sizeof(int) * (4 * p->exp_rows + 2 * p->grid));
    const size_t o_list = take(sizeof(DBlock) * TILE_BLKS * (size_t)p->ntiles);
    const size_t o_arr[2] = {take((size_t)NP * p->rows * KB * 2), take((size_t)NP * p->rows * KB * 2)};
    if (cudaMalloc(&p->mem, size) != cudaSuccess) {
      p->mem = nullptr;
      cudaGetLastError();
      throw std::runtime_error("cudaMalloc");
    }
    if (cudaMemcpy(p->mem, tables.data(), tables.size(), cudaMemcpyHostToDevice) != cudaSuccess) throw std::runtime_error("cudaMemcpy");
    char* base = (char*)p->mem;
    p->d_jobs = (DJob*)(base + o_jobs);
    p->d_tiles = (DTile*)(base + o_tiles);
    p->d_cta = (int*)(base + o_cta);
    p->d_rblk = (int4*)(base + o_rblk);
    p->d_dblk = (int4*)(base + o_dblk);
    p->d_exp = (int*)(base + o_exp);
    p->d_list = (DBlock*)(base + o_list);
    for (int a = 0; a < 2; ++a) p->arr[a] = (__nv_bfloat16*)(base + o_arr[a]);
    for (int a = 0; a < 2; ++a) {
      plane_map(&p->maps[a], p->arr[a], p->rows, TM);
      plane_map(&p->maps[2 + a], p->arr[a], p->rows, TN);
    }
    int maxsm = 0;
    cudaDeviceGetAttribute(&maxsm, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    p->smem = 1024 + NSTAGE * STAGE + (2 * NSTAGE + 4 + 2 * NINFO) * 8 + 16;
    if (p->smem + sizeof(TileInfo) * NINFO + 64 > (size_t)maxsm) throw std::runtime_error("not enough shared memory for the FP64 product's pipeline");
    // (the whole shared memory, so that a second stream's kernels find some beside the CTA)
    if (cudaFuncSetAttribute(k_dgemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p->smem) != cudaSuccess ||
        cudaFuncSetAttribute(k_dgemm, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) != cudaSuccess) {
      cudaGetLastError();
      throw std::runtime_error("cudaFuncSetAttribute");
    }
  } catch (...) {
    dgemm_plan_destroy(p);
    throw;
  }
  return p;
}

void dgemm_plan_destroy(DgemmPlan* p)
{
  if (!p) return;
  if (p->mem) cudaFree(p->mem);
  delete p;
}

void dgemm_plan_set_wait(DgemmPlan* p, unsigned limit) { p->wait = limit; }

cudaError_t launch_dgemm(const DgemmPlan* p, const double* A, const double* B0, const double* B1, double* O, const int* kidx,
                         const double* kw, const int* phase, int gsign, double gbscale, int accum, bool mirror,
                         cudaStream_t st)
{
  if (p->ntiles == 0) return cudaSuccess;
  int *rexpA = p->d_exp, *rexpB = p->d_exp + p->exp_rows, *cntA = p->d_exp + 2 * p->exp_rows, *cntB = cntA + p->exp_rows;
  int* nlist = cntB + p->exp_rows;
  cudaError_t e;
  {
    ProfScope ps(p->family == 0 ? "dgemm_slice_ladder" : "dgemm_slice_zbar", st);
    if (p->n_dblk == 0) {
      k_dgemm_slice<<<p->n_rblk, 256, 0, st>>>(p->d_jobs, p->d_rblk, A, B0, B1, kidx, kw, gbscale, rexpA, rexpB, cntA, cntB,
                                               nlist, 2 * p->grid, p->rows, p->arr[0], p->arr[1]);
      count_launch();
    } else {
      if ((e = cudaMemsetAsync(p->d_exp, 0, sizeof(int) * (4 * p->exp_rows + 2 * p->grid), st)) != cudaSuccess) return e;
      k_dgemm_rowexp<<<p->n_rblk, 256, 0, st>>>(p->d_jobs, p->d_rblk, A, B0, B1, kidx, kw, gbscale, rexpA, rexpB, cntA, cntB);
      k_dgemm_digits<<<p->n_dblk, 256, 0, st>>>(p->d_jobs, p->d_dblk, A, B0, B1, kidx, kw, gbscale, rexpA, rexpB, p->rows,
                                                p->arr[0], p->arr[1]);
      count_launch(2);
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  ProfScope ps(p->family == 0 ? "dgemm_ladder" : "dgemm_zbar", st);
  DArgs a{p->d_jobs, p->d_tiles, p->d_cta, rexpA, rexpB, cntA, cntB, phase, O, p->d_list, nlist, nlist + p->grid,
          A, B0, B1, kidx, kw, gbscale, gsign, accum, mirror ? 0 : 1, p->share ? 1 : 0, p->wait};
  k_dgemm<<<p->grid, 96 + 32 * EPIW, p->smem, st>>>(p->maps[0], p->maps[1], p->maps[2], p->maps[3], a);
  count_launch();
  return cudaGetLastError();
}

}  // namespace imsrg
