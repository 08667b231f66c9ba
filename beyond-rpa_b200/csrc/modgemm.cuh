// Residue-arithmetic products on the int8 tensor cores (modgemm.cu): moduli, scaling and the
// Chinese-remainder step shared by the kernels that read residues.
#pragma once
#include "kernels.h"

namespace rpa {

// Fifteen pairwise coprime moduli (256 = 2^8, 255 = 3 5 17, 253 = 11 23, 247 = 13 19, 217 = 7 31,
// the others prime): P = 2^117.8.
constexpr int kModCount = 15;
constexpr uint32_t kModuli[kModCount] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197};

// Rows are scaled to 2-norms in [2^57, 2^58): the product of two, < 2^116, stays well below P / 2
// (the rounding of at most 2^20 entries adds less than 2^10 to a norm).
constexpr int kModNormBits = 58;

// Chinese remainder weights split in two doubles: the high parts (41 bits) add up exactly.
struct ModCrt {
  double whi[kModCount], wlo[kModCount];
  double phi, plo, rp;  // P = phi + plo, 1 / P
};
struct ModReduce {
  int p[kModCount];
  int magic[kModCount];  // ceil(2^38 / p): (acc * magic) >> 38 = floor(acc / p) for |acc| <= 2^30 + 255
};

// Power of two (exponent) that brings a row of norm sqrt(s2) / 2^shift to a norm in [2^57, 2^58).  A zero
// row keeps 0.  A row with NaN or Inf returns a marker for which mod_pow2 is NaN, so its products are
// NaN (as the FP64 sums would be non-finite).
constexpr int kModNaNExpo = 1 << 20;
__host__ __device__ __forceinline__ int mod_exponent(double s2, int shift) {
  if (!(s2 > 0.0)) return s2 == 0.0 ? 0 : kModNaNExpo;
  if (s2 > 1.7e308) return kModNaNExpo;
  int e;
  frexp(sqrt(s2) * (1.0 + 1e-9), &e);  // norm < 2^e
  e = kModNormBits - e + shift;
  return e < -1000 ? -1000 : e > 1000 ? 1000 : e;
}
// Scaling (exponent) under which a sum of squares that overflowed or got lost in the denormals is
// taken again; 0: the sum is fine.  (A sum that is zero because the row is stays zero.)
__host__ __device__ __forceinline__ int mod_needs_shift(double s2) {
  return s2 > 1e300 ? -600 : (s2 < 1e-290 ? 400 : 0);
}
__device__ __forceinline__ double mod_pow2(int e) {
  if (e > 1000 || e < -1000) return __longlong_as_double(0x7FF8000000000000ll);
  return __longlong_as_double((long long)(1023 + e) << 52);
}

// h such that 2^h a and 2^-h b are of the same size, from the upper words of the magnitudes of a, b and a
// factor of b (zero or denormal ones count as 2^-1023).  No scaling where one is not finite.
__host__ __device__ __forceinline__ int mod_balance(int a, int b, int fb) {
  const int ea = a >> 20, eb = (b >> 20) + (fb >> 20) - 1023;
  if (ea >= 2047 || (b >> 20) >= 2047 || (fb >> 20) >= 2047) return 0;
  const int h = (eb - ea) >> 1;
  return h < -1000 ? -1000 : h > 1000 ? 1000 : h;
}

// Integers from four neighbouring columns of residues (one byte each, planes apart), as doubles
// rounded once: sum_i r_i W_i mod P in (-P/2, P/2).
__device__ __forceinline__ void mod_crt4(const uint8_t* src, int64_t plane, const ModCrt& crt, double (&c)[4]) {
  uint32_t w[kModCount];
#pragma unroll
  for (int m = 0; m < kModCount; ++m) w[m] = __ldg(reinterpret_cast<const uint32_t*>(src + m * plane));
  double hi[4] = {0.0, 0.0, 0.0, 0.0}, lo[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int m = 0; m < kModCount; ++m) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      // 2^52 + r - 2^52: a byte to a double without the slow integer conversion
      const double r = __hiloint2double(0x43300000, (int)((w[m] >> (8 * e)) & 255u)) - 4503599627370496.0;
      hi[e] = fma(r, crt.whi[m], hi[e]);
      lo[e] = fma(r, crt.wlo[m], lo[e]);
    }
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const double q = rint((hi[e] + lo[e]) * crt.rp);
    c[e] = fma(-q, crt.phi, hi[e]) + fma(-q, crt.plo, lo[e]);
  }
}

// Limits of the residue form, for the callers to keep to (beyond them the FP64 pipe takes over): summed
// lengths and orders that the conversions and the recombination put in a grid's second dimension, and tiles
// counted in 32 bits.
constexpr int64_t kModMaxK = (int64_t)65535 * 128;
constexpr int kModMaxOrder = 65535;
inline bool mod_units_fit(int64_t rowsA, int64_t rowsB, int64_t nz, bool tri) {
  const double ti = (double)((rowsB + 255) / 256), tj = (double)((rowsA + 255) / 256);
  return (tri ? ti * (ti + 1.0) / 2.0 : ti * tj) * kModCount * (double)nz < 2147483647.0;
}
inline int64_t mod_pitch(int64_t K) { return (K + 127) / 128 * 128; }

// One launch: residues of C(i, j) = sum_k a(j, k) b(i, k) for nz batches, j < rowsA (lanes),
// i < rowsB; tri: only the tiles that hold some i >= j.
struct ModGemmArgs {
  int rowsA;
  int nch;  // 128-wide k chunks
  int nti, ntj, nz, ntiles, nunits, tri;  // 256 x 256 tiles
  int zplanesA, zplanesB;  // planes between batches of each operand (0: shared)
  uint8_t* out;            // [z][modulus][j][i], i contiguous
  int64_t out_plane, ldo;  // bytes between planes; between j (a multiple of 256)
  int* sync;               // optional wave milestones (zeroed, mod_sync_words ints)
  int sync_every;
  int* err;
};

const ModCrt& mod_crt_tables();
cudaError_t mod_map(PFN_cuTensorMapEncodeTiled_v12000 encode, CUtensorMap* m, void* planes, int64_t K, int64_t rows,
                    int64_t nplanes, int64_t pitch, int box_rows);
// Residue planes [z][modulus][row][pitch] of the columns of S - shift * 1 (S: K x rows, column-major,
// strideS apart), entry k times ks[k] when ks is given.
cudaError_t launch_mod_cols(const double* S, int64_t ld, int64_t strideS, int K, int64_t rows, int batch,
                            int8_t* planes, int* expo, cudaStream_t stream, double shift = 0.0,
                            const double* ks = nullptr);
// Residue planes [modulus][row][pitch] of the rows of S (rows x K, column-major), column k times fac[k] when
// fac is given.
cudaError_t launch_mod_rows(const double* S, int64_t ld, int rows, int64_t K, const double* fac, int8_t* planes,
                            int* expo, cudaStream_t stream);
// fa[k], fb[k]: factors that bring column k of operands a and b to the same size (mod_balance), fb times
// kscale[k] when given.  With b2, column k of the second operand is made of products of entries of column k of b and of
// b2 (a Khatri-Rao product, of which only the factors are read).  sizes: 3 K ints.
struct ModOperand {
  const double* S;  // entry (r, k) at S[r * s_r + k * s_k], one stride 1
  int64_t s_r, s_k, rows;
};
cudaError_t launch_mod_balance(const ModOperand& a, const ModOperand& b, const ModOperand* b2, int64_t K,
                               const double* kscale, int* sizes, double* fa, double* fb, cudaStream_t stream);
// Residue planes [k][modulus][Q][pitch] of X_k; fac: fg.n * nov doubles, part: nsplit * fg.n * NQ.
cudaError_t launch_mod_pi(const double* R, int64_t ldR, int NQ, int64_t nov, const double* D, const FreqGroup& fg,
                          double alpha, double* fac, double* part, int nsplit, int* expo, int8_t* planes,
                          cudaStream_t stream);
cudaError_t mod_plan(ModGemmArgs& a, int rowsA, int rowsB, int64_t K, int nz, bool tri);
int64_t mod_sync_words(const ModGemmArgs& a, int num_sms);
// tmA, tmB: the operands' planes as boxes of 128 rows (mod_map).
cudaError_t launch_modgemm(const CUtensorMap& tmA, const CUtensorMap& tmB, const ModGemmArgs& a, int num_sms,
                           cudaStream_t stream);
// V (optional, leading dimension and stride of C): C = V^T V - 1 from the residues of (V - 1)^T (V - 1).
cudaError_t launch_mod_crt_lower(const uint8_t* res, int64_t plane, int64_t ldo, const int* expo, int n, int batch,
                                 double* C, int64_t ldc, int64_t strideC, cudaStream_t stream,
                                 const double* V = nullptr);
cudaError_t launch_mod_crt_full(const uint8_t* res, int64_t plane, int64_t ldo, const int* expo_i, const int* expo_j,
                                int ni, int64_t nj, double* C, int64_t ldc, double alpha, double beta,
                                cudaStream_t stream);
// Adjoint accumulation (launch_grad_accum) from the residues of M_k R: [k][modulus][ai][q].
cudaError_t launch_mod_grad(const double* R, int64_t ldR, const uint8_t* res, int64_t plane, int64_t ldo,
                            const int* expo_m, const int* expo_r, int NQ, int64_t nov, const double* D,
                            const GradGroup& gg, double* dR, int64_t lddR, double* dD, bool first,
                            cudaStream_t stream);
// ---- block columns of Cholesky factors (log-det trailing updates)
// One matrix: its factor's columns are converted panel by panel; a block column gets the products of
// all panels before it at once (K up to the order), so that it is read and written once.
struct ModMat {
  CUtensorMap mA, mB;  // planes as 128- and 256-row boxes
  double* A;
  int64_t ld;
  int8_t* planes;  // [modulus][row][pitch]
  uint8_t* res;    // [modulus][column of the block][ldo]
  int* expo;       // powers of two of the rows
  int n, pitch, ldo;
};
struct ModCholArgs {
  int col0, nb, K, ntj;
  int* err;
};
size_t mod_chol_bytes(int n, int nb, size_t* planes, size_t* res);  // of one matrix
cudaError_t mod_chol_fill(PFN_cuTensorMapEncodeTiled_v12000 encode, ModMat& m, double* A, int64_t ld, int n, int nb,
                          uint8_t* base);
cudaError_t launch_mod_chol_expo(const ModMat* mats, int nmat, int nmax, bool unit_shift, cudaStream_t stream);
// Planes of the factored columns c0 .. c0 + nb - 1, rows row0 and below.
cudaError_t launch_mod_chol_planes(const ModMat* mats, int nmat, int nmax, int row0, int c0, int nb,
                                   cudaStream_t stream);
// A(i, j) -= sum_{k < K} L(i, k) L(j, k) for i >= j, col0 <= j < col0 + nb.
cudaError_t launch_mod_chol_update(const ModMat* mats, int nmat, int nmax, int col0, int nb, int K, int* err,
                                   cudaStream_t stream);
}  // namespace rpa
