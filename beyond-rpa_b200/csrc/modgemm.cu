// FP64-accurate matrix products on the int8 tensor cores by residue arithmetic.
//
//   C(i, j) = sum_k a(i, k) b(j, k)
//
// The modular scheme of Ozaki, Uchino and Imamura ("Ozaki Scheme II: a GEMM-oriented emulation of
// floating-point matrix multiplication using an integer modular technique", 2025): every row of a
// and b is scaled by a power of two and rounded to integers a', b' whose 2-norms stay below
// 2^58; |sum_k a' b'| is then below P / 2 for P the product of 15 pairwise coprime moduli <= 256
// (Cauchy-Schwarz, so the bound holds for every input), and the exact integer product follows from
// its 15 residues (Chinese remainder theorem).  Each residue is one int8 x int8 -> int32 matrix
// product of tcgen05 (kind::i8), exact as long as K <= 65536 per accumulation.  The only errors
// are the rounding of the operands (0.5 units of 2^-58 of the row norm) and one rounding of C, less
// than a chain of K FP64 additions leaves (tests/test_gpu_modgemm.py compares both).  The rounding is
// relative to the row, not to the entry: operands that may be graded against each other along K are
// brought to the same sizes first (launch_mod_balance); in X X^T, (V - 1)^T (V - 1), M R and L L^T both
// carry the same grading.
//
// On B200 the int8 pipe sustains 3.9 POP/s (random operands from shared memory, M 128 x N 256), so
// 15 products cost what 260 TFLOP/s of FP64 would, against 37 TFLOP/s of the FP64 pipe.
//
//  * mod_cols_kernel: operands whose K index is contiguous (column-major K x rows)
//  * mod_pi_kernel:   X_k(Q, ai) = sqrt(alpha c_k(ai)) R(Q, ai), transposed to ai-contiguous rows
//  * modgemm_pair_kernel: residues of C, 15 int8 products per tile, tiles of 256 x 256 on CTA pairs
//  * modgemm_chol_kernel: the same for block columns of Cholesky factors
//  * mod_*crt*:       C from its residues
#include <algorithm>
#include <utility>

#include "modgemm.cuh"

namespace rpa {

namespace {
// ------------------------------------------------------------------ residues of the operands
// For an integer x in (-2^63, 2^63): x + 2^63 has eight unsigned bytes b_j, and
// x = sum_j b_j 256^j - 2^63 = sum_j b_j (256^j mod p) + (-2^63 mod p)   (mod p): two 4-way byte
// dot products give a value v < 2^20 congruent to x.  v is reduced in FP32 (exact: v < 2^23): the
// dot product starts from the bits of 1.5 * 2^23, so its result is the float 1.5 * 2^23 + v.
template <int I>
struct ModConst {
  static constexpr uint32_t p = kModuli[I];
  static constexpr uint32_t pw(int j) {
    uint32_t r = 1;
    for (int t = 0; t < j; ++t) r = (r * 256u) % p;
    return p == 256u && j > 0 ? 0u : r;
  }
  static constexpr uint32_t wlo = pw(0) | pw(1) << 8 | pw(2) << 16 | pw(3) << 24;
  static constexpr uint32_t whi = pw(4) | pw(5) << 8 | pw(6) << 16 | pw(7) << 24;
  static constexpr uint32_t off = (p - (128u * pw(7)) % p) % p;  // -2^63 mod p
  static constexpr uint32_t init = 0x4B400000u + off;
};

template <int I>
__device__ __forceinline__ uint32_t mod_residue_bits(uint32_t lo, uint32_t hi) {
  using M = ModConst<I>;
  const float big = 12582912.0f;  // 1.5 * 2^23
  const float f = __uint_as_float(__dp4a(lo, M::wlo, __dp4a(hi, M::whi, M::init)));
  const float q = __fsub_rn(__fmaf_rn(__fsub_rn(f, big), 1.0f / (float)M::p, big), big);
  // 1.5 * 2^23 + r, |r| <= p / 2 (+ 1): its low byte is r as a signed 8-bit integer
  return __float_as_uint(__fmaf_rn(-(float)M::p, q, f));
}

// Residues of N (a multiple of 4) integers for modulus I, packed four to a word.
template <int I, int N>
__device__ __forceinline__ void mod_pack(const uint32_t (&lo)[N], const uint32_t (&hi)[N], uint32_t (&w)[N / 4]) {
#pragma unroll
  for (int t = 0; t < N / 4; ++t) {
    const uint32_t a = mod_residue_bits<I>(lo[4 * t], hi[4 * t]), b = mod_residue_bits<I>(lo[4 * t + 1], hi[4 * t + 1]);
    const uint32_t c = mod_residue_bits<I>(lo[4 * t + 2], hi[4 * t + 2]),
                   d = mod_residue_bits<I>(lo[4 * t + 3], hi[4 * t + 3]);
    w[t] = __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
  }
}

template <int N, class Store, int... I>
__device__ __forceinline__ void mod_all(const uint32_t (&lo)[N], const uint32_t (&hi)[N], const Store& store,
                                        std::integer_sequence<int, I...>) {
  (
      [&] {
        uint32_t w[N / 4];
        mod_pack<I, N>(lo, hi, w);
        store(I, w);
      }(),
      ...);
}

__device__ __forceinline__ void to_words(double x, uint32_t& lo, uint32_t& hi) {
  const unsigned long long u = (unsigned long long)__double2ll_rn(x) ^ 0x8000000000000000ull;
  lo = (uint32_t)u;
  hi = (uint32_t)(u >> 32);
}

// Columns of a column-major (K x rows) matrix: one warp per column, 8 consecutive k per lane.
// S: column r starts at S + r * ld; expo[r]: its power of two.  shift is subtracted from the diagonal;
// ks (optional) multiplies entry k of every column.
__global__ void __launch_bounds__(256) mod_cols_kernel(const double* __restrict__ S, int64_t ld, int64_t strideS,
                                                       int K, int64_t rows, int8_t* __restrict__ planes,
                                                       int64_t pitch, int64_t plane_stride, int64_t strideP,
                                                       int* __restrict__ expo, double shift,
                                                       const double* __restrict__ ks) {
  const int64_t r = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (r >= rows) return;
  const int z = blockIdx.y;
  const double* col = S + (int64_t)z * strideS + r * ld;
  auto entry = [&](int k) {
    const double x = col[k] - (k == r ? shift : 0.0);
    return ks ? x * __ldg(ks + k) : x;
  };
  auto sum = [&](double f) {
    double s2 = 0.0;
    for (int k = lane; k < K; k += 32) {
      const double x = entry(k) * f;
      s2 = fma(x, x, s2);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    return s2;
  };
  double s2 = sum(1.0);
  const int sh = mod_needs_shift(s2);  // squares that overflow or vanish: sum them scaled (warp-uniform)
  if (sh) s2 = sum(mod_pow2(sh));
  const int e = mod_exponent(s2, sh);
  if (lane == 0) expo[(int64_t)z * rows + r] = e;
  const double sc = mod_pow2(e);
  int8_t* out = planes + (int64_t)z * strideP + r * pitch;
  for (int k0 = 8 * lane; k0 < pitch; k0 += 256) {
    uint32_t lo[8], hi[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      to_words(k0 + i < K ? entry(k0 + i) * sc : 0.0, lo[i], hi[i]);
    mod_all<8>(
        lo, hi,
        [&](int m, const uint32_t(&w)[2]) {
          *reinterpret_cast<uint2*>(out + m * plane_stride + k0) = make_uint2(w[0], w[1]);
        },
        std::make_integer_sequence<int, kModCount>());
  }
}

// ---- sizes of two operands along K
// A product whose operands are graded against each other along K (large entries of a where those of b
// are small) would lose what the rows' own powers of two round away: 2^-58 of a row norm is much for a
// small entry that meets a large one.  Column k of a is therefore multiplied by 2^h and column k of b by
// 2^-h, exactly, so that their largest entries agree; then a' = a S, b' = b S^-1 (S diagonal, powers of
// two) give the same integers as a and b.  Sizes are the upper words of the largest magnitudes.
// K contiguous, entry (r, k) at S[r * ld + k]: a thread per k, 64 rows per CTA.
constexpr int kSizeRows = 64;
__global__ void __launch_bounds__(256) mod_ksize_cols_kernel(const double* __restrict__ S, int64_t ld, int64_t rows,
                                                             int64_t K, int* __restrict__ size) {
  const int64_t k = (int64_t)blockIdx.y * 256 + threadIdx.x;
  if (k >= K) return;
  const int64_t r0 = (int64_t)blockIdx.x * kSizeRows, r1 = min(rows, r0 + kSizeRows);
  int m = 0;
#pragma unroll 8
  for (int64_t r = r0; r < r1; ++r) m = max(m, __double2hiint(__ldg(S + r * ld + k)) & 0x7fffffff);
  atomicMax(size + k, m);
}
// Rows contiguous, entry (r, k) at S[r + k * ld]: a warp per k.
__global__ void __launch_bounds__(256) mod_ksize_rows_kernel(const double* __restrict__ S, int64_t ld, int64_t rows,
                                                             int64_t K, int* __restrict__ size) {
  const int64_t k = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (k >= K) return;
  int m = 0;
#pragma unroll 8
  for (int64_t r = threadIdx.x & 31; r < rows; r += 32) m = max(m, __double2hiint(__ldg(S + r + k * ld)) & 0x7fffffff);
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) size[k] = m;
}
// The factors of column k: 2^h for a; 2^-h, and the product's own scale of k, for b.
__global__ void mod_kfactor_kernel(const int* __restrict__ size_a, const int* __restrict__ size_b,
                                   const int* __restrict__ size_b2, const double* __restrict__ kscale, int64_t K,
                                   double* __restrict__ fa, double* __restrict__ fb) {
  const int64_t k = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (k >= K) return;
  const double s = kscale ? kscale[k] : 1.0;
  const int s2 = size_b2 ? size_b2[k] : kscale ? __double2hiint(s) & 0x7fffffff : 1023 << 20;
  const int h = mod_balance(size_a[k], size_b[k], s2);
  fa[k] = mod_pow2(h);
  fb[k] = mod_pow2(-h) * s;
}

// fac[k * nov + ai] = sqrt(alpha D / (D^2 + u_k^2))
__global__ void mod_chi_kernel(const double* __restrict__ D, int64_t nov, FreqGroup fg, double alpha,
                               double* __restrict__ fac) {
  const int64_t a = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= nov) return;
  const double d = D[a];
#pragma unroll
  for (int k = 0; k < kMaxKgLaunch; ++k)
    if (k < fg.n) fac[k * nov + a] = sqrt(alpha * d / fma(d, d, fg.u2[k]));
}

// part[split][k][Q] = sum over the split's ai of (fac_k R)^2: lane = Q, each warp 16 of the 128 ai of a
// chunk; the squared factors wait in shared memory ([ai][k], broadcast reads).  Reading the factors
// from global memory inside the sum took 2.46 ms at NQ 2048, 16384 ai, 16 frequencies.
constexpr int kNormWarps = 8;
__global__ void __launch_bounds__(256) mod_pi_norm_kernel(const double* __restrict__ R, int64_t ldR, int NQ,
                                                          int64_t nov, const double* __restrict__ fac, int kg,
                                                          int64_t per_split, double* __restrict__ part) {
  __shared__ __align__(16) double sm[kNormWarps * kMaxKgLaunch * 32];  // factors, then the warps' sums
  static_assert(128 * kMaxKgLaunch <= kNormWarps * kMaxKgLaunch * 32, "the factors fit");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int q = blockIdx.x * 32 + lane;
  const int64_t a0 = (int64_t)blockIdx.y * per_split, a1 = min(nov, a0 + per_split);
  double s[kMaxKgLaunch];
#pragma unroll
  for (int k = 0; k < kMaxKgLaunch; ++k) s[k] = 0.0;
  for (int64_t c = a0; c < a1; c += 128) {
    double r[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int64_t a = c + warp * 16 + j;
      r[j] = (q < NQ && a < a1) ? __ldg(R + q + ldR * a) : 0.0;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 128 * kMaxKgLaunch; i += 256) {
      const int k = i >> 7, j = i & 127;
      const double f = (k < kg && c + j < a1) ? __ldg(fac + k * nov + c + j) : 0.0;
      sm[j * kMaxKgLaunch + k] = f * f;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const double r2 = r[j] * r[j];
      const double2* f2 = reinterpret_cast<const double2*>(sm + (warp * 16 + j) * kMaxKgLaunch);
#pragma unroll
      for (int k = 0; k < kMaxKgLaunch / 2; ++k) {
        const double2 f = f2[k];
        s[2 * k] = fma(r2, f.x, s[2 * k]);
        s[2 * k + 1] = fma(r2, f.y, s[2 * k + 1]);
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kMaxKgLaunch; ++k) sm[(warp * kMaxKgLaunch + k) * 32 + lane] = s[k];
  __syncthreads();
  for (int idx = threadIdx.x; idx < kg * 32; idx += 256) {
    const int k = idx >> 5, l = idx & 31;
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < kNormWarps; ++w) t += sm[(w * kMaxKgLaunch + k) * 32 + l];
    if (blockIdx.x * 32 + l < NQ) part[((int64_t)blockIdx.y * kg + k) * NQ + blockIdx.x * 32 + l] = t;
  }
}

__global__ void mod_pi_expo_kernel(const double* __restrict__ part, int nsplit, int64_t n, int* __restrict__ expo) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double s = 0.0;
  for (int t = 0; t < nsplit; ++t) s += part[t * n + i];
  expo[i] = mod_exponent(s, 0);
}

// expo[r] of the rows of a column-major (rows x K) matrix, column k times fac[k] when given: lane = row,
// eight warps stride over k
__global__ void __launch_bounds__(256) mod_row_norm_kernel(const double* __restrict__ S, int64_t ld, int rows,
                                                           int64_t K, const double* __restrict__ fac,
                                                           int* __restrict__ expo) {
  __shared__ double red[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = blockIdx.x * 32 + lane;
  auto entry = [&](int64_t k) {
    const double x = r < rows ? S[r + ld * k] : 0.0;
    return fac ? x * __ldg(fac + k) : x;
  };
  auto sum = [&](double f) {
    // eight entries and factors on their way at a time
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    int64_t k = warp;
    for (; k + 56 < K; k += 64) {
      double x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = entry(k + 8 * u) * f;
#pragma unroll
      for (int u = 0; u < 8; ++u) s[u & 3] = fma(x[u], x[u], s[u & 3]);
    }
    for (; k < K; k += 8) {
      const double x = entry(k) * f;
      s[0] = fma(x, x, s[0]);
    }
    __syncthreads();
    red[warp][lane] = (s[0] + s[1]) + (s[2] + s[3]);
    __syncthreads();
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += red[w][lane];
    return t;
  };
  double s2 = sum(1.0);
  int shift = 0;
  if (__syncthreads_or(mod_needs_shift(s2) != 0)) {  // squares that overflow or vanish: sum them scaled
    shift = mod_needs_shift(s2);
    s2 = sum(mod_pow2(shift));
  }
  if (warp == 0 && r < rows) expo[r] = mod_exponent(s2, shift);
}

// planes[(k, m)][Q][ai]: a CTA takes a 32 x 128 block of R (read with Q across the lanes, kept in
// shared memory) and writes whole 128-byte lines, four ai per lane and one row per warp.  The lines
// are what bounds the pass: with 16 ai of 32 different rows per warp the stores of 15 planes were
// half sectors, and more CTAs per SM only made them slower (7.3 ms with one, 13.1 ms with three at
// NQ 2048, 16384 ai, 16 frequencies).
constexpr int kPiPitch = 128 + 4;
constexpr size_t kModPiSmem = sizeof(double) * (32 * kPiPitch + kMaxKgLaunch * 128);
// kFac false: the rows of R itself (one set of planes, no factors); with kg = 1 fac is any factor per column.
template <bool kFac>
__global__ void __launch_bounds__(256, 4) mod_pi_kernel(const double* __restrict__ R, int64_t ldR, int NQ, int64_t nov,
                                                        const double* __restrict__ fac, int kg,
                                                        const int* __restrict__ expo, int8_t* __restrict__ planes,
                                                        int64_t pitch) {
  extern __shared__ __align__(16) double mod_smem[];
  double* rs = mod_smem;                  // [32 Q][kPiPitch]
  double* fs = mod_smem + 32 * kPiPitch;  // [kg][128 ai]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int q0 = blockIdx.x * 32;
  const int64_t b0 = (int64_t)blockIdx.y * 128;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const int64_t a = b0 + warp + 8 * j;
    rs[lane * kPiPitch + warp + 8 * j] = (q0 + lane < NQ && a < nov) ? __ldg(R + q0 + lane + ldR * a) : 0.0;
  }
  if (kFac) {
    for (int i = threadIdx.x; i < kg * 128; i += 256) {
      const int64_t a = b0 + (i & 127);
      fs[i] = a < nov ? __ldg(fac + (i >> 7) * nov + a) : 0.0;
    }
  }
  __syncthreads();
  const int64_t plane_stride = (int64_t)NQ * pitch;
  for (int i = warp; i < 32 * kg; i += 8) {
    const int k = i >> 5, q = i & 31;
    if (q0 + q >= NQ) continue;
    const double sc = mod_pow2(expo[(int64_t)k * NQ + q0 + q]);
    const double2* r2 = reinterpret_cast<const double2*>(rs + q * kPiPitch + 4 * lane);
    const double2* f2 = reinterpret_cast<const double2*>(fs + k * 128 + 4 * lane);
    const double2 one = make_double2(1.0, 1.0);
    const double2 ra = r2[0], rb = r2[1], fa = kFac ? f2[0] : one, fb = kFac ? f2[1] : one;
    uint32_t lo[4], hi[4];
    to_words((ra.x * fa.x) * sc, lo[0], hi[0]);
    to_words((ra.y * fa.y) * sc, lo[1], hi[1]);
    to_words((rb.x * fb.x) * sc, lo[2], hi[2]);
    to_words((rb.y * fb.y) * sc, lo[3], hi[3]);
    int8_t* out = planes + ((int64_t)k * kModCount * NQ + q0 + q) * pitch + b0 + 4 * lane;
    mod_all<4>(
        lo, hi, [&](int m, const uint32_t(&w)[1]) { *reinterpret_cast<uint32_t*>(out + m * plane_stride) = w[0]; },
        std::make_integer_sequence<int, kModCount>());
  }
}

// ------------------------------------------------------------------ the products
constexpr int MG_TM = 128;   // rows of the first operand per tile (TMEM lanes): index j of C
constexpr int MG_TN = 256;   // rows of the second operand per tile (TMEM columns): index i of C
constexpr int MG_TK = 128;   // k bytes per stage (one 128-byte swizzle row)
constexpr int MG_STAGES = 4;
constexpr int MG_ABYTES = MG_TM * MG_TK;
constexpr int MG_BBYTES = MG_TN * MG_TK;
constexpr int MG_STAGE = MG_ABYTES + MG_BBYTES;  // 48 KB
constexpr int MG_THREADS = 576;                  // producer, MMA issuer, 16 epilogue warps
constexpr int MG_SMEM = MG_STAGES * MG_STAGE + 1024 + 256;
constexpr int MG_SEG = 65536 / MG_TK;  // stages per exact int32 accumulation (|r| <= 128: 2^14 per term)

// Instruction descriptor: kind::i8, A = B = signed 8-bit, D = signed 32-bit, both K-major, M x N.
constexpr uint32_t idesc_s8_s32(int M, int N) {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma_s8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Shared-memory descriptor, K-major operand, 128-byte swizzle: 8-row groups 1024 B apart.
__device__ __forceinline__ uint64_t desc_k_sw128(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | (uint64_t)1u << 16 | (uint64_t)(1024u >> 4) << 32 | (uint64_t)1u << 46 |
         (uint64_t)2u << 61;
}

// One tile of one modulus: operand rows j0 .. (128 lanes) and i0 .. (ni columns) of planes pa and pb.
struct MgUnit {
  int m, j0, i0, ni, pa, pb;
  uint8_t* out;  // residues of (j0, i0)
  int nj;        // rows of the tile that are stored
};

// Block column of a batch of Cholesky factors: a CTA takes one tile of one matrix and a third of the
// moduli.  CTAs live for microseconds, so that the launches of the critical path, on a stream of
// higher priority, find SMs (a persistent launch would hold them all until its end).
constexpr int MG_GROUPS = 3;
struct MgChol {
  const ModMat* mat;
  const ModCholArgs& a;
  int t, g;  // tile, third of the moduli
  __device__ __forceinline__ int begin() const { return g * (kModCount / MG_GROUPS); }
  __device__ __forceinline__ int end() const { return (g + 1) * (kModCount / MG_GROUPS); }
  __device__ __forceinline__ int step() const { return 1; }
  __device__ __forceinline__ int nch() const { return a.K / MG_TK; }
  __device__ __forceinline__ int64_t ldo() const { return mat->ldo; }
  __device__ __forceinline__ bool any() const {
    const int tj = t % a.ntj, ti = t / a.ntj;
    return a.col0 + tj * MG_TM < mat->n && a.col0 + ti * MG_TN < mat->n && tj <= 2 * ti + 1 && (tj == 0 || a.col0 + ti * MG_TN + (tj == 2 * ti + 1 ? MG_TM : 0) < mat->n);
  }
  __device__ __forceinline__ MgUnit get(int m) const {
    MgUnit x;
    const int tj = t % a.ntj, ti = t / a.ntj;
    x.m = x.pa = x.pb = m;
    x.ni = MG_TN;
    int i0 = ti * MG_TN;
    if (tj == 2 * ti + 1) {
      i0 += MG_TM;
      x.ni = MG_TM;
    }
    x.j0 = a.col0 + tj * MG_TM;
    x.i0 = a.col0 + i0;
    x.nj = min(MG_TM, min(a.nb, mat->n - a.col0) - tj * MG_TM);
    x.out = mat->res + (int64_t)m * a.nb * mat->ldo + (int64_t)(tj * MG_TM) * mat->ldo + i0;
    return x;
  }
};

__device__ __forceinline__ bool mg_wait_count(const int* c, int target) {
  for (uint32_t it = 0; it < (1u << 20); ++it) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(c) : "memory");
    if (v >= target) return true;
    __nanosleep(64);
  }
  return false;
}

// Residues of 64 accumulator columns (one row per lane) added to those in w, four to a word:
// r = acc mod p in [0, p].
__device__ __forceinline__ void mod_drain(uint32_t taddr, int p, int mg, uint32_t (&w)[16]) {
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    float v[32];
    tmem_ld_32x32b_x32(taddr + (uint32_t)(half * 32), v);
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      uint32_t r[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int acc = __float_as_int(v[4 * t + e]) + (int)((w[half * 8 + t] >> (8 * e)) & 255u);
        r[e] = (uint32_t)(acc - (__mulhi(acc, mg) >> 6) * p);
      }
      w[half * 8 + t] = __byte_perm(__byte_perm(r[0], r[1], 0x0040), __byte_perm(r[2], r[3], 0x0040), 0x5410);
    }
  }
}

template <class Src>
__device__ __forceinline__ void modgemm_body(const Src& src, const CUtensorMap* tmA, const CUtensorMap* tmB,
                                             const CUtensorMap* tmBh, int* err, const ModReduce& red) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + MG_STAGES * MG_STAGE);
  uint64_t* empty = full + MG_STAGES;
  uint64_t* acc_full = empty + MG_STAGES;
  uint64_t* acc_empty = acc_full + 2;
  uint64_t* drain = acc_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < MG_STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 16);
    }
    mbar_init(drain, 1);
    fence_mbar_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      // ------------------------------------------------------------ producer
      tma_prefetch_desc(tmA);
      tma_prefetch_desc(tmB);
      int stage = 0;
      uint32_t phase = 0, issued = 0, issued_par = 0;
      bool ok = true;
      for (int u = src.begin(); u < src.end() && ok; u += src.step()) {
        const MgUnit x = src.get(u);
        const CUtensorMap* mb = x.ni == MG_TN ? tmB : tmBh;
        const uint32_t bytes = (uint32_t)(MG_TM + x.ni) * MG_TK;
        for (int ch = 0; ch < src.nch(); ++ch) {
          if (!mbar_wait(&empty[stage], phase ^ 1u, err, kDevTimeoutTmaEmpty)) {
            ok = false;
            break;
          }
          mbar_arrive_expect_tx(&full[stage], bytes);
          uint8_t* st = smem + stage * MG_STAGE;
          tma_load_3d(st, tmA, &full[stage], ch * MG_TK, x.j0, x.pa);
          tma_load_3d(st + MG_ABYTES, mb, &full[stage], ch * MG_TK, x.i0, x.pb);
          issued |= 1u << stage;
          issued_par = (issued_par & ~(1u << stage)) | (phase << stage);
          if (++stage == MG_STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      // no bulk copy may still be landing in shared memory at exit
      for (int s = 0; s < MG_STAGES; ++s)
        if (issued & (1u << s)) mbar_wait(&full[s], (issued_par >> s) & 1u, err, kDevTimeoutDrain);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // ------------------------------------------------------------ MMA issuer
      int stage = 0, it = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int u = src.begin(); u < src.end() && ok; u += src.step()) {
        const MgUnit x = src.get(u);
        const uint32_t idesc = x.ni == MG_TN ? idesc_s8_s32(MG_TM, MG_TN) : idesc_s8_s32(MG_TM, MG_TM);
        for (int c0 = 0; c0 < src.nch() && ok; c0 += MG_SEG, ++it) {
          const int b = it & 1;
          if (!mbar_wait(&acc_empty[b], (uint32_t)((it >> 1) & 1) ^ 1u, err, kDevTimeoutAccEmpty)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t d = tmem_base + (uint32_t)(b * MG_TN);
          const int c1 = min(src.nch(), c0 + MG_SEG);
          for (int ch = c0; ch < c1; ++ch) {
            if (!mbar_wait(&full[stage], phase, err, kDevTimeoutTmaFull)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t sa = smem_u32(smem + stage * MG_STAGE), sb = sa + MG_ABYTES;
#pragma unroll
            for (int kk = 0; kk < MG_TK / 32; ++kk)
              mma_s8(d, desc_k_sw128(sa + kk * 32), desc_k_sw128(sb + kk * 32), idesc,
                     (ch > c0 || kk > 0) ? 1u : 0u);
            tc_commit(&empty[stage]);
            if (++stage == MG_STAGES) {
              stage = 0;
              phase ^= 1u;
            }
          }
          if (!ok) break;
          tc_commit(&acc_full[b]);
        }
      }
      // every issued MMA must complete before TMEM is freed
      tc_commit(drain);
      mbar_wait(drain, 0, err, kDevTimeoutDrain);
    }
  } else {
    // -------------------------------------------------------------- epilogue
    // warp w: TMEM lanes 32 (w mod 4) .., accumulator columns 64 ((w - 2) / 4) .. + 63.  Residues
    // r = acc mod p in [0, p], four to a word; a segment adds the previous segments' residue.
    const int quarter = warp & 3;
    const int col0 = ((warp - 2) >> 2) * 64;
    int it = 0;
    bool ok = true;
    for (int u = src.begin(); u < src.end() && ok; u += src.step()) {
      const MgUnit x = src.get(u);
      const int p = red.p[x.m];
      const int mg = red.magic[x.m];
      uint32_t w[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) w[i] = 0;
      for (int c0 = 0; c0 < src.nch(); c0 += MG_SEG, ++it) {
        const int b = it & 1;
        if (!mbar_wait(&acc_full[b], (uint32_t)((it >> 1) & 1), err, kDevTimeoutAccFull)) {
          ok = false;
          break;
        }
        tc_fence_after();
        if (col0 < x.ni) {
          mod_drain(tmem_base + (uint32_t)(b * MG_TN + col0) + ((uint32_t)(quarter * 32) << 16), p, mg, w);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[b]);
      }
      if (!ok) break;
      const int j = quarter * 32 + lane;
      if (col0 < x.ni && j < x.nj) {
        uint4* dst = reinterpret_cast<uint4*>(x.out + (int64_t)j * src.ldo() + col0);
#pragma unroll
        for (int t = 0; t < 4; ++t) dst[t] = make_uint4(w[4 * t], w[4 * t + 1], w[4 * t + 2], w[4 * t + 3]);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

__global__ void __launch_bounds__(MG_THREADS, 1)
    modgemm_chol_kernel(const ModMat* __restrict__ mats, const ModCholArgs a, const ModReduce red) {
  const ModMat* mat = mats + blockIdx.y;
  MgChol src{mat, a, (int)blockIdx.x / MG_GROUPS, (int)blockIdx.x % MG_GROUPS};
  if (!src.any()) return;  // CTA-uniform
  if (threadIdx.x == 0) {  // the producer
    tensormap_acquire(&mat->mA);
    tensormap_acquire(&mat->mB);
  }
  modgemm_body(src, &mat->mA, &mat->mB, &mat->mA, a.err, red);
}

// ------------------------------------------------------------------ CTA pairs
// The full and triangular products as 256 x 256 tiles on pairs of SMs (cta_group::2): each CTA loads
// 128 rows of either operand and accumulates 128 of the tile's rows, so that a k step moves 32 KB per
// CTA for the work that takes 48 KB of one CTA.  One int8 tile of 128 x 256 asks L2 for 96 bytes per
// clock and SM, and the tensor pipe of the one-CTA kernel was 76 % busy waiting for them.
// The even CTA issues every MMA; its `full` barriers count the bytes of both CTAs, `empty` and
// `acc_full` are signalled in both by multicast commits, `acc_empty` collects both epilogues.
constexpr int M2_STAGES = 6;
constexpr int M2_STAGE = 2 * MG_ABYTES;
constexpr int M2_SMEM = M2_STAGES * M2_STAGE + 1024 + 256;

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The even CTA's copy of a shared-memory object of this CTA.
__device__ __forceinline__ uint32_t leader_addr(const void* p) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_u32(p)));
  return a;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(void* dst, const void* tmap, uint32_t bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
      "%3, %4}], [%5];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void mma_s8_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on the barrier at this offset in both CTAs once the MMAs issued so far have completed.
__device__ __forceinline__ void commit_pair(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"((uint16_t)3)
      : "memory");
}

struct PairUnit {
  int m, j0, i0, pa, pb, zm;
};
__device__ __forceinline__ PairUnit pair_unit(int u, const ModGemmArgs& a) {
  PairUnit x;
  int ti, tj, z;
  if (a.tri) {  // (batch, modulus, tile), ti-major, tj <= ti
    const int zm = u / a.ntiles, t = u - zm * a.ntiles;
    z = zm / kModCount;
    x.m = zm - z * kModCount;
    ti = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
    while ((ti + 1) * (ti + 2) / 2 <= t) ++ti;
    while (ti * (ti + 1) / 2 > t) --ti;
    tj = t - ti * (ti + 1) / 2;
  } else {  // (modulus, tj, batch, ti): the rows of a shared first operand stay in L2 for every batch
    ti = u % a.nti;
    int q = u / a.nti;
    z = q % a.nz;
    q /= a.nz;
    tj = q % a.ntj;
    x.m = q / a.ntj;
  }
  x.zm = z * kModCount + x.m;
  x.j0 = tj * 256;
  x.i0 = ti * 256;
  x.pa = z * a.zplanesA + x.m;
  x.pb = z * a.zplanesB + x.m;
  return x;
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(MG_THREADS, 1)
    modgemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                        const ModGemmArgs a, const ModReduce red) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + M2_STAGES * M2_STAGE);
  uint64_t* empty = full + M2_STAGES;
  uint64_t* acc_full = empty + M2_STAGES;
  uint64_t* acc_empty = acc_full + 2;
  uint64_t* drain = acc_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_rank();
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < M2_STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 32);
    }
    mbar_init(drain, 1);
    fence_mbar_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      // ------------------------------------------------------------ producer: this CTA's halves
      tma_prefetch_desc(&tmA);
      tma_prefetch_desc(&tmB);
      int stage = 0;
      uint32_t phase = 0, issued = 0, issued_par = 0;
      bool ok = true, sync_wait = rank == 0;
      const int nmile = a.sync && rank == 0 ? (a.nch + a.sync_every - 1) / a.sync_every : 0;
      for (int u = pair; u < a.nunits && ok; u += npairs) {
        const PairUnit x = pair_unit(u, a);
        const int wave = (u - pair) / npairs;
        const int members = min(npairs, a.nunits - wave * npairs);
        for (int ch = 0; ch < a.nch; ++ch) {
          if (nmile && ch % a.sync_every == 0) {
            const int mi = ch / a.sync_every;
            int* row = a.sync + (int64_t)wave * nmile;
            asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(row + mi) : "memory");
            if (sync_wait && mi >= 2) sync_wait = mg_wait_count(row + mi - 2, members);
          }
          if (!mbar_wait(&empty[stage], phase ^ 1u, a.err, kDevTimeoutTmaEmpty)) {
            ok = false;
            break;
          }
          if (rank == 0) mbar_arrive_expect_tx(&full[stage], 2 * M2_STAGE);
          uint8_t* st = smem + stage * M2_STAGE;
          const uint32_t bar = leader_addr(&full[stage]);
          tma_load_3d_pair(st, &tmA, bar, ch * MG_TK, x.j0 + rank * MG_TM, x.pa);
          tma_load_3d_pair(st + MG_ABYTES, &tmB, bar, ch * MG_TK, x.i0 + rank * MG_TM, x.pb);
          issued |= 1u << stage;
          issued_par = (issued_par & ~(1u << stage)) | (phase << stage);
          if (++stage == M2_STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      // every issued load has landed (the even CTA counts the bytes of both) before the shared memory goes:
      // both CTAs meet at the cluster barrier below
      if (rank == 0) {
        for (int s = 0; s < M2_STAGES; ++s)
          if (issued & (1u << s) && !mbar_wait(&full[s], (issued_par >> s) & 1u, a.err, kDevTimeoutDrain)) break;
      }
      for (int s = 0; s < M2_STAGES; ++s)
        if (issued & (1u << s)) mbar_wait(&empty[s], (issued_par >> s) & 1u, a.err, kDevTimeoutTmaEmpty);
      // the last commit arrives in both CTAs: the odd one's shared memory must outlive its arrival too
      if (rank != 0) mbar_wait(drain, 0, a.err, kDevTimeoutDrain);
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      // ------------------------------------------------------------ MMA issuer (even CTA)
      constexpr uint32_t idesc = idesc_s8_s32(256, 256);
      int stage = 0, it = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int u = pair; u < a.nunits && ok; u += npairs) {
        for (int c0 = 0; c0 < a.nch && ok; c0 += MG_SEG, ++it) {
          const int b = it & 1;
          if (!mbar_wait(&acc_empty[b], (uint32_t)((it >> 1) & 1) ^ 1u, a.err, kDevTimeoutAccEmpty)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t d = tmem_base + (uint32_t)(b * 256);
          const int c1 = min(a.nch, c0 + MG_SEG);
          for (int ch = c0; ch < c1; ++ch) {
            if (!mbar_wait(&full[stage], phase, a.err, kDevTimeoutTmaFull)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t sa = smem_u32(smem + stage * M2_STAGE), sb = sa + MG_ABYTES;
#pragma unroll
            for (int kk = 0; kk < MG_TK / 32; ++kk)
              mma_s8_pair(d, desc_k_sw128(sa + kk * 32), desc_k_sw128(sb + kk * 32), idesc,
                          (ch > c0 || kk > 0) ? 1u : 0u);
            commit_pair(&empty[stage]);
            if (++stage == M2_STAGES) {
              stage = 0;
              phase ^= 1u;
            }
          }
          if (!ok) break;
          commit_pair(&acc_full[b]);
        }
      }
      // every issued MMA must complete before TMEM is freed
      commit_pair(drain);
      mbar_wait(drain, 0, a.err, kDevTimeoutDrain);
    }
  } else {
    // -------------------------------------------------------------- epilogue (both CTAs: 128 rows each)
    const int quarter = warp & 3;
    const int col0 = ((warp - 2) >> 2) * 64;
    const uint32_t release[2] = {leader_addr(&acc_empty[0]), leader_addr(&acc_empty[1])};
    int it = 0;
    bool ok = true;
    for (int u = pair; u < a.nunits && ok; u += npairs) {
      const PairUnit x = pair_unit(u, a);
      const int p = red.p[x.m];
      const int mg = red.magic[x.m];
      uint32_t w[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) w[i] = 0;
      for (int c0 = 0; c0 < a.nch; c0 += MG_SEG, ++it) {
        const int b = it & 1;
        if (!mbar_wait(&acc_full[b], (uint32_t)((it >> 1) & 1), a.err, kDevTimeoutAccFull)) {
          ok = false;
          break;
        }
        tc_fence_after();
        mod_drain(tmem_base + (uint32_t)(b * 256 + col0) + ((uint32_t)(quarter * 32) << 16), p, mg, w);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(release[b]);
      }
      if (!ok) break;
      const int j = x.j0 + rank * MG_TM + quarter * 32 + lane;
      if (j < a.rowsA) {
        uint4* dst = reinterpret_cast<uint4*>(a.out + (int64_t)x.zm * a.out_plane + (int64_t)j * a.ldo + x.i0 + col0);
#pragma unroll
        for (int t = 0; t < 4; ++t) dst[t] = make_uint4(w[4 * t], w[4 * t + 1], w[4 * t + 2], w[4 * t + 3]);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // both CTAs are done with each other's barriers and with the accumulators
  tc_fence_after();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512));
}

// Power of two of every row of a Cholesky factor, known beforehand: ||L_i||^2 = A_ii.  The products take the
// entries left of the diagonal only; for A = 1 + P, P positive semidefinite, L_ii^2 >= 1 and their norm is
// at most A_ii - 1, which keeps the digits of rows with small P_ii (graded Cholesky vectors).  The
// factorization's own rounding, n 2^-53 A_ii, is added fourfold.
__global__ void mod_chol_expo_kernel(const ModMat* __restrict__ mats, int unit_shift) {
  const ModMat& m = mats[blockIdx.y];
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= m.n) return;
  double s2 = m.A[i + m.ld * (int64_t)i];
  if (unit_shift) s2 = fmax(s2 - 1.0, 0.0) + 4.0 * m.n * 1.1102230246251565e-16 * s2;
  m.expo[i] = mod_exponent(s2, 0);
}

// Planes of columns c0 .. c0 + nb - 1 (nb a multiple of 128), rows row0 .. n - 1, of the factors: the
// block transposition of mod_pi_kernel.
__global__ void __launch_bounds__(256, 4) mod_chol_planes_kernel(const ModMat* __restrict__ mats, int row0, int c0) {
  __shared__ __align__(16) double rs[32 * kPiPitch];
  const ModMat& m = mats[blockIdx.z];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int q0 = row0 + blockIdx.x * 32, b0 = c0 + blockIdx.y * 128;
  if (q0 >= m.n) return;
#pragma unroll
  for (int j = 0; j < 16; ++j)
    rs[lane * kPiPitch + warp + 8 * j] = q0 + lane < m.n ? m.A[q0 + lane + m.ld * (int64_t)(b0 + warp + 8 * j)] : 0.0;
  __syncthreads();
  const int64_t plane_stride = (int64_t)m.n * m.pitch;
  for (int q = warp; q < 32 && q0 + q < m.n; q += 8) {
    const double sc = mod_pow2(m.expo[q0 + q]);
    const double2* r2 = reinterpret_cast<const double2*>(rs + q * kPiPitch + 4 * lane);
    const double2 ra = r2[0], rb = r2[1];
    uint32_t lo[4], hi[4];
    to_words(ra.x * sc, lo[0], hi[0]);
    to_words(ra.y * sc, lo[1], hi[1]);
    to_words(rb.x * sc, lo[2], hi[2]);
    to_words(rb.y * sc, lo[3], hi[3]);
    int8_t* out = m.planes + (int64_t)(q0 + q) * m.pitch + b0 + 4 * lane;
    mod_all<4>(
        lo, hi, [&](int k, const uint32_t(&w)[1]) { *reinterpret_cast<uint32_t*>(out + k * plane_stride) = w[0]; },
        std::make_integer_sequence<int, kModCount>());
  }
}

// A(i, j) -= (sum_k L(i, k) L(j, k)) for the block column at col0, from its residues.
__global__ void __launch_bounds__(256) mod_chol_crt_kernel(const ModMat* __restrict__ mats, int col0, int nb,
                                                           const ModCrt crt) {
  const ModMat& m = mats[blockIdx.z];
  const int j = blockIdx.y, i0 = 4 * (int)(blockIdx.x * 256 + threadIdx.x);  // relative to col0
  if (col0 + j >= m.n || col0 + i0 >= m.n || i0 + 3 < j) return;
  double c[4];
  mod_crt4(m.res + (int64_t)j * m.ldo + i0, (int64_t)nb * m.ldo, crt, c);
  const double sj = mod_pow2(-m.expo[col0 + j]);
  double* dst = m.A + col0 + m.ld * (int64_t)(col0 + j);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int i = i0 + e;
    if (i >= j && col0 + i < m.n) dst[i] -= c[e] * mod_pow2(-m.expo[col0 + i]) * sj;
  }
}

// ------------------------------------------------------------------ C from its residues
// Lower triangles Pi_z(i, j), i >= j (column-major, ld NQ): four consecutive i per thread.  With V (lower
// triangles, as C): the residues are those of (V - 1)^T (V - 1), and C = V^T V - 1 is put together without the
// cancellation: V + V^T - 2 + (V - 1)^T (V - 1).
__global__ void __launch_bounds__(256) mod_crt_lower_kernel(const uint8_t* __restrict__ res, int64_t plane,
                                                            int64_t ldo, const ModCrt crt,
                                                            const int* __restrict__ expo, int n,
                                                            double* __restrict__ C, int64_t ldc, int64_t strideC,
                                                            const double* __restrict__ V) {
  const int z = blockIdx.z, j = blockIdx.y;
  const int i0 = 4 * (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (i0 + 3 < j || i0 >= n) return;
  const uint8_t* src = res + (int64_t)z * kModCount * plane + (int64_t)j * ldo + i0;
  double c[4];
  mod_crt4(src, plane, crt, c);
  const double sj = mod_pow2(-expo[(int64_t)z * n + j]);
  const int64_t off = (int64_t)z * strideC + (int64_t)j * ldc;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int i = i0 + e;
    if (i < j || i >= n) continue;
    double x = c[e] * mod_pow2(-expo[(int64_t)z * n + i]) * sj;
    if (V) x += i == j ? 2.0 * (V[off + i] - 1.0) : V[off + i];
    C[off + i] = x;
  }
}

// C(i, j) = alpha * (...) + beta C(i, j), column-major: four consecutive i per thread
__global__ void __launch_bounds__(256) mod_crt_full_kernel(const uint8_t* __restrict__ res, int64_t plane, int64_t ldo,
                                                           const ModCrt crt, const int* __restrict__ expo_i,
                                                           const int* __restrict__ expo_j, int ni, int64_t nj,
                                                           double* __restrict__ C, int64_t ldc, double alpha,
                                                           double beta) {
  const int i0 = 4 * (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int64_t j = (int64_t)blockIdx.y + (int64_t)blockIdx.z * gridDim.y;
  if (i0 >= ni || j >= nj) return;
  double c[4];
  mod_crt4(res + j * ldo + i0, plane, crt, c);
  const double sj = alpha * mod_pow2(-expo_j[j]);
  double* dst = C + j * ldc;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int i = i0 + e;
    if (i < ni) {
      const double v = c[e] * mod_pow2(-expo_i[i]) * sj;
      dst[i] = beta == 0.0 ? v : fma(beta, dst[i], v);
    }
  }
}

// Adjoint accumulation from the residues of M_k R, M_k = (1 + Pi_k)^-1 - 1 (grad_accum_kernel without
// its Y_k): one warp per column ai, four consecutive q per lane.
__global__ void __launch_bounds__(256) mod_grad_kernel(const double* __restrict__ R, int64_t ldR,
                                                       const uint8_t* __restrict__ res, int64_t plane, int64_t ldo,
                                                       const ModCrt crt, const int* __restrict__ expo_m,
                                                       const int* __restrict__ expo_r, int NQ, int64_t nov,
                                                       const double* __restrict__ D, const GradGroup gg,
                                                       double* __restrict__ dR, int64_t lddR, double* __restrict__ dD,
                                                       int first) {
  const int64_t a = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (a >= nov) return;
  const double d = D[a];
  const double sr = mod_pow2(-expo_r[a]);
  // lane k holds the two factors of frequency k
  double cf = 0.0, df = 0.0;
  if (lane < gg.n) {
    const double den = fma(d, d, gg.u2[lane]);
    cf = 2.0 * gg.alpha * gg.f[lane] * d / den * sr;
    df = gg.alpha * gg.f[lane] * (gg.u2[lane] - d * d) / (den * den) * sr;
  }
  double dot = 0.0;
  for (int qb = 0; qb < NQ; qb += 128) {  // every lane takes every step: the shuffles need the whole warp
    const int q0 = qb + 4 * lane;
    double r[4], g[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      r[e] = q0 + e < NQ ? R[q0 + e + ldR * a] : 0.0;
      g[e] = first || q0 + e >= NQ ? 0.0 : dR[q0 + e + lddR * a];
    }
    for (int k = 0; k < gg.n; ++k) {
      const double cfac = __shfl_sync(0xffffffffu, cf, k), dfac = __shfl_sync(0xffffffffu, df, k);
      if (q0 >= NQ) continue;
      double c[4];
      mod_crt4(res + (int64_t)k * kModCount * plane + a * ldo + q0, plane, crt, c);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (q0 + e >= NQ) continue;
        const double m = c[e] * mod_pow2(-expo_m[(int64_t)k * NQ + q0 + e]);
        g[e] = fma(cfac, m, g[e]);
        dot = fma(dfac * r[e], m, dot);
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (q0 + e < NQ) dR[q0 + e + lddR * a] = g[e];
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) dot += __shfl_down_sync(0xffffffffu, dot, off);
  if (lane == 0) dD[a] = (first ? 0.0 : dD[a]) + dot;
}
}  // namespace

// ------------------------------------------------------------------ host side
namespace {
typedef unsigned __int128 u128;

struct ModTables {
  ModReduce red;
  ModCrt crt;
  ModTables() {
    u128 P = 1;
    for (int i = 0; i < kModCount; ++i) P *= kModuli[i];
    int bits = 0;
    for (u128 t = P; t; t >>= 1) ++bits;
    const int L = bits - 41;  // high parts hold 41 bits, so that sum_i 255 hi_i stays below 2^53
    const u128 low = ((u128)1 << L) - 1;
    auto dbl = [](u128 x) { return (double)(uint64_t)(x >> 64) * 18446744073709551616.0 + (double)(uint64_t)x; };
    for (int i = 0; i < kModCount; ++i) {
      const uint32_t p = kModuli[i];
      red.p[i] = (int)p;
      red.magic[i] = (int)((1ull << 38) / p + (p == 256 ? 0 : 1));
      const u128 Pi = P / p;
      const uint32_t r = (uint32_t)(Pi % p);
      uint32_t inv = 1;
      while ((r * inv) % p != 1) ++inv;
      const u128 W = Pi * inv;  // < P, = 1 mod p, = 0 mod the others
      crt.whi[i] = dbl(W >> L << L);
      crt.wlo[i] = dbl(W & low);
    }
    crt.phi = dbl(P >> L << L);
    crt.plo = dbl(P & low);
    crt.rp = 1.0 / dbl(P);
  }
};
const ModTables& tables() {
  static const ModTables t;
  return t;
}
}  // namespace

const ModCrt& mod_crt_tables() { return tables().crt; }

cudaError_t mod_map(PFN_cuTensorMapEncodeTiled_v12000 encode, CUtensorMap* m, void* planes, int64_t K, int64_t rows,
                    int64_t nplanes, int64_t pitch, int box_rows) {
  cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)rows, (cuuint64_t)nplanes};
  cuuint64_t strides[2] = {(cuuint64_t)pitch, (cuuint64_t)(pitch * rows)};
  cuuint32_t box[3] = {MG_TK, (cuuint32_t)box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return encode(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, planes, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
             ? cudaSuccess
             : cudaErrorInvalidValue;
}

cudaError_t launch_mod_cols(const double* S, int64_t ld, int64_t strideS, int K, int64_t rows, int batch,
                            int8_t* planes, int* expo, cudaStream_t stream, double shift, const double* ks) {
  if (rows <= 0 || batch <= 0) return cudaSuccess;
  const int64_t pitch = mod_pitch(K), plane = pitch * rows;
  mod_cols_kernel<<<dim3((unsigned)((rows + 7) / 8), (unsigned)batch), 256, 0, stream>>>(
      S, ld, strideS, K, rows, planes, pitch, plane, plane * kModCount, expo, shift, ks);
  ++g_launches;
  return cudaGetLastError();
}

cudaError_t launch_mod_pi(const double* R, int64_t ldR, int NQ, int64_t nov, const double* D, const FreqGroup& fg,
                          double alpha, double* fac, double* part, int nsplit, int* expo, int8_t* planes,
                          cudaStream_t stream) {
  const int64_t pitch = mod_pitch(nov);
  mod_chi_kernel<<<(unsigned)((nov + 255) / 256), 256, 0, stream>>>(D, nov, fg, alpha, fac);
  const int64_t per = (nov + nsplit - 1) / nsplit;
  mod_pi_norm_kernel<<<dim3((unsigned)((NQ + 31) / 32), (unsigned)nsplit), 256, 0, stream>>>(R, ldR, NQ, nov, fac,
                                                                                           fg.n, per, part);
  const int64_t n = (int64_t)fg.n * NQ;
  mod_pi_expo_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(part, nsplit, n, expo);
  const cudaError_t e =
      cudaFuncSetAttribute(mod_pi_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kModPiSmem);
  if (e != cudaSuccess) return e;
  mod_pi_kernel<true><<<dim3((unsigned)((NQ + 31) / 32), (unsigned)((pitch + 127) / 128)), 256, kModPiSmem, stream>>>(
      R, ldR, NQ, nov, fac, fg.n, expo, planes, pitch);
  g_launches += 4;
  return cudaGetLastError();
}

cudaError_t launch_mod_rows(const double* S, int64_t ld, int rows, int64_t K, const double* fac, int8_t* planes,
                            int* expo, cudaStream_t stream) {
  if (rows <= 0) return cudaSuccess;
  const int64_t pitch = mod_pitch(K);
  mod_row_norm_kernel<<<(unsigned)((rows + 31) / 32), 256, 0, stream>>>(S, ld, rows, K, fac, expo);
  const dim3 grid((unsigned)((rows + 31) / 32), (unsigned)((pitch + 127) / 128));
  constexpr size_t smem = sizeof(double) * (32 * kPiPitch + 128);
  static_assert(smem <= 48 * 1024, "no opt-in needed");
  if (fac) mod_pi_kernel<true><<<grid, 256, smem, stream>>>(S, ld, rows, K, fac, 1, expo, planes, pitch);
  else mod_pi_kernel<false><<<grid, 256, smem, stream>>>(S, ld, rows, K, nullptr, 1, expo, planes, pitch);
  g_launches += 2;
  return cudaGetLastError();
}

cudaError_t launch_mod_balance(const ModOperand& a, const ModOperand& b, const ModOperand* b2, int64_t K,
                               const double* kscale, int* sizes, double* fa, double* fb, cudaStream_t stream) {
  if (K <= 0 || a.rows <= 0 || b.rows <= 0) return cudaSuccess;
  const cudaError_t e = cudaMemsetAsync(sizes, 0, 3 * (size_t)K * sizeof(int), stream);
  if (e != cudaSuccess) return e;
  auto size = [&](const ModOperand& x, int* out) {
    if (x.s_k == 1)
      mod_ksize_cols_kernel<<<dim3((unsigned)((x.rows + kSizeRows - 1) / kSizeRows), (unsigned)((K + 255) / 256)), 256,
                              0, stream>>>(x.S, x.s_r, x.rows, K, out);
    else mod_ksize_rows_kernel<<<(unsigned)((K + 7) / 8), 256, 0, stream>>>(x.S, x.s_k, x.rows, K, out);
    ++g_launches;
  };
  size(a, sizes);
  size(b, sizes + K);
  if (b2) size(*b2, sizes + 2 * K);
  mod_kfactor_kernel<<<(unsigned)((K + 255) / 256), 256, 0, stream>>>(sizes, sizes + K, b2 ? sizes + 2 * K : nullptr,
                                                                     kscale, K, fa, fb);
  ++g_launches;
  return cudaGetLastError();
}

int64_t mod_sync_words(const ModGemmArgs& a, int num_sms) {
  if (a.sync_every <= 0) return 0;
  const int pairs = std::min(a.nunits, num_sms / 2);
  return pairs <= 0 ? 0 : (int64_t)((a.nunits + pairs - 1) / pairs) * ((a.nch + a.sync_every - 1) / a.sync_every);
}

cudaError_t mod_plan(ModGemmArgs& a, int rowsA, int rowsB, int64_t K, int nz, bool tri) {
  a.rowsA = rowsA;
  a.nch = (int)((K + MG_TK - 1) / MG_TK);
  a.tri = tri ? 1 : 0;
  a.nti = (rowsB + 255) / 256;
  a.ntj = (rowsA + 255) / 256;
  a.nz = nz;
  const int64_t tiles = tri ? (int64_t)a.nti * (a.nti + 1) / 2 : (int64_t)a.nti * a.ntj;
  const int64_t units = tiles * kModCount * nz;
  if (units > INT32_MAX) return cudaErrorInvalidValue;
  a.ntiles = (int)tiles;
  a.nunits = (int)units;
  return cudaSuccess;
}

cudaError_t launch_modgemm(const CUtensorMap& tmA, const CUtensorMap& tmB, const ModGemmArgs& a, int num_sms,
                           cudaStream_t stream) {
  if (a.nunits <= 0) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(modgemm_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, M2_SMEM);
  if (e != cudaSuccess) return e;
  modgemm_pair_kernel<<<2 * std::min(a.nunits, num_sms / 2), MG_THREADS, M2_SMEM, stream>>>(tmA, tmB, a, tables().red);
  ++g_launches;
  return cudaGetLastError();
}

cudaError_t launch_mod_crt_lower(const uint8_t* res, int64_t plane, int64_t ldo, const int* expo, int n, int batch,
                                 double* C, int64_t ldc, int64_t strideC, cudaStream_t stream, const double* V) {
  mod_crt_lower_kernel<<<dim3((unsigned)((n + 1023) / 1024), (unsigned)n, (unsigned)batch), 256, 0, stream>>>(
      res, plane, ldo, tables().crt, expo, n, C, ldc, strideC, V);
  ++g_launches;
  return cudaGetLastError();
}

cudaError_t launch_mod_crt_full(const uint8_t* res, int64_t plane, int64_t ldo, const int* expo_i, const int* expo_j,
                                int ni, int64_t nj, double* C, int64_t ldc, double alpha, double beta,
                                cudaStream_t stream) {
  if (ni <= 0 || nj <= 0) return cudaSuccess;
  const int64_t gy = std::min<int64_t>(nj, 32768);
  mod_crt_full_kernel<<<dim3((unsigned)((ni + 1023) / 1024), (unsigned)gy, (unsigned)((nj + gy - 1) / gy)), 256, 0,
                        stream>>>(res, plane, ldo, tables().crt, expo_i, expo_j, ni, nj, C, ldc, alpha, beta);
  ++g_launches;
  return cudaGetLastError();
}

cudaError_t launch_mod_grad(const double* R, int64_t ldR, const uint8_t* res, int64_t plane, int64_t ldo,
                            const int* expo_m, const int* expo_r, int NQ, int64_t nov, const double* D,
                            const GradGroup& gg, double* dR, int64_t lddR, double* dD, bool first,
                            cudaStream_t stream) {
  mod_grad_kernel<<<(unsigned)((nov + 7) / 8), 256, 0, stream>>>(R, ldR, res, plane, ldo, tables().crt, expo_m, expo_r,
                                                                 NQ, nov, D, gg, dR, lddR, dD, first ? 1 : 0);
  ++g_launches;
  return cudaGetLastError();
}

size_t mod_chol_bytes(int n, int nb, size_t* planes, size_t* res) {
  *planes = (size_t)kModCount * n * (size_t)mod_pitch(n);
  *res = (size_t)kModCount * nb * (size_t)((n + 255) / 256 * 256);
  return *planes + *res + ((size_t)n * sizeof(int) + 255) / 256 * 256;
}

cudaError_t mod_chol_fill(PFN_cuTensorMapEncodeTiled_v12000 encode, ModMat& m, double* A, int64_t ld, int n, int nb,
                          uint8_t* base) {
  size_t pb, rb;
  mod_chol_bytes(n, nb, &pb, &rb);
  m.A = A;
  m.ld = ld;
  m.n = n;
  m.pitch = (int)mod_pitch(n);
  m.ldo = (n + 255) / 256 * 256;
  m.planes = reinterpret_cast<int8_t*>(base);
  m.res = base + pb;
  m.expo = reinterpret_cast<int*>(base + pb + rb);
  cudaError_t e = mod_map(encode, &m.mA, m.planes, n, n, kModCount, m.pitch, MG_TM);
  return e == cudaSuccess ? mod_map(encode, &m.mB, m.planes, n, n, kModCount, m.pitch, MG_TN) : e;
}

cudaError_t launch_mod_chol_expo(const ModMat* mats, int nmat, int nmax, bool unit_shift, cudaStream_t stream) {
  mod_chol_expo_kernel<<<dim3((unsigned)((nmax + 255) / 256), (unsigned)nmat), 256, 0, stream>>>(mats,
                                                                                                unit_shift ? 1 : 0);
  ++g_launches;
  return cudaGetLastError();
}

cudaError_t launch_mod_chol_planes(const ModMat* mats, int nmat, int nmax, int row0, int c0, int nb,
                                   cudaStream_t stream) {
  if (row0 >= nmax) return cudaSuccess;
  mod_chol_planes_kernel<<<dim3((unsigned)((nmax - row0 + 31) / 32), (unsigned)(nb / 128), (unsigned)nmat), 256, 0,
                           stream>>>(mats, row0, c0);
  ++g_launches;
  return cudaGetLastError();
}

cudaError_t launch_mod_chol_update(const ModMat* mats, int nmat, int nmax, int col0, int nb, int K, int* err,
                                   cudaStream_t stream) {
  if (col0 >= nmax || K <= 0) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(modgemm_chol_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MG_SMEM);
  if (e != cudaSuccess) return e;
  ModCholArgs a;
  a.col0 = col0;
  a.nb = nb;
  a.K = K;
  a.ntj = nb / MG_TM;
  a.err = err;
  const int rows = nmax - col0, nti = (rows + MG_TN - 1) / MG_TN;
  modgemm_chol_kernel<<<dim3((unsigned)(nti * a.ntj * MG_GROUPS), (unsigned)nmat), MG_THREADS, MG_SMEM, stream>>>(
      mats, a, tables().red);
  mod_chol_crt_kernel<<<dim3((unsigned)((rows + 1023) / 1024), (unsigned)std::min(nb, rows), (unsigned)nmat), 256, 0,
                        stream>>>(mats, col0, nb, tables().crt);
  g_launches += 2;
  return cudaGetLastError();
}

}  // namespace rpa
