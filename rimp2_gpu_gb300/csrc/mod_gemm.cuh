// mod_gemm.cuh -- FP64 contractions on the FP16 tensor cores by residue
// arithmetic (mod_gemm.cu): operands, products and the general contraction.
#pragma once
#include "common.cuh"

namespace rimp2 {

constexpr int MG_P = 16;             // moduli
constexpr int MG_PLANES = MG_P + 1;  // and the plane of magnitudes
// least sum |a||b| of an element in the units of the magnitudes' plane, below
// which it is summed in FP64: 2^-8 of 2^24.  Rows are scaled by powers of two to norms
// between 2^11 and 2^12 of these units: 2^-8 to 2^-6 of ||a|| ||b||
constexpr float MG_TAU = 65536.0f;

constexpr int MG_K_MIN = 16, MG_K_MAX = 16384;  // lengths of a sum

// a row's (or column's) flags
constexpr unsigned MG_ROW_ZERO = 1;   // all zeros
constexpr unsigned MG_ROW_FP64 = 2;   // infinities, NaNs, extreme exponents: FP64 only
constexpr unsigned MG_ROW_EXACT = 4;  // no value was rounded
constexpr int MG_NO_LSB = 1 << 20;

// Rows of an operand: up to three dimensions, the first one fastest; element
// (row, k) at base + sum_d index_d st[d] + k sk.  cst: the strides in C; role:
// 0 the product's own index, 1 a batch index.
struct RowMap {
  const double *base;
  int ext[3];
  long long st[3], cst[3];
  int role[3];
  int rows, K;
  long long sk;
};

// The product of g as rows and columns: batch dimensions that move only one
// operand become more rows or columns of it.  False if one moves both.
bool fold_gemm(const GemmDesc &g, RowMap &A, RowMap &B);

#ifdef __CUDACC__
__device__ __forceinline__ long long row_off(const RowMap &M, int r) {
  const int d0 = r % M.ext[0], q = r / M.ext[0];
  const int d1 = q % M.ext[1], d2 = q / M.ext[1];
  return d0 * M.st[0] + d1 * M.st[1] + d2 * M.st[2];
}

__device__ __forceinline__ long long c_off(const RowMap &M, int r) {
  const int d0 = r % M.ext[0], q = r / M.ext[0];
  const int d1 = q % M.ext[1], d2 = q / M.ext[1];
  return d0 * M.cst[0] + d1 * M.cst[1] + d2 * M.cst[2];
}

// the index along the dimension with the given role (0: m or n, 1: batch)
__device__ __forceinline__ int role_index(const RowMap &M, int r, int role) {
  const int d0 = r % M.ext[0], q = r / M.ext[0];
  const int d1 = q % M.ext[1], d2 = q / M.ext[1];
  return (M.role[0] == role ? d0 : 0) + (M.role[1] == role ? d1 : 0) + (M.role[2] == role ? d2 : 0);
}

__device__ __forceinline__ void cp_async8(double *dst, const double *src, bool valid) {
  // 8-byte global -> shared copy; an invalid element is zero-filled (no read)
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src),
               "r"(valid ? 8 : 0)
               : "memory");
}

// The hardware's FP32 reciprocal of d (its bits moved into a float and back).
// False where d is outside the float range, zero or NaN.
__device__ __forceinline__ bool recip_f32(double d, double &r0) {
  const int hi = __double2hiint(d), ed = (hi >> 20) & 0x7FF;
  if (ed < 1023 - 120 || ed > 1023 + 120) return false;
  const float f = __int_as_float((hi & 0x80000000) | ((ed - 896) << 23) | ((hi & 0xFFFFF) << 3) |
                                 ((unsigned)__double2loint(d) >> 29));
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f));
  const int b = __float_as_int(r);
  r0 = __hiloint2double((b & 0x80000000) | ((((b >> 23) & 0xFF) + 896) << 20) | ((b >> 3) & 0xFFFFF),
                        b << 29);
  return true;
}

// 1/d: that reciprocal refined by a third-order step of Householder's method,
// r (1 + e + e^2) with e = 1 - d r: about an ulp.  FP64 operations run at 1/64 of
// the FP32 rate here: three of them.
__device__ __forceinline__ double recip_f64(double d) {
  double r0;
  if (!recip_f32(d, r0)) return 1.0 / d;
  const double e = fma(-d, r0, 1.0);
  return fma(r0, fma(e, e, e), r0);
}

// v / d: the quotient by that reciprocal corrected twice by its remainder
// v - d q (Markstein; 22, 44, 66 bits before the last rounding), five operations
__device__ __forceinline__ double div_f64(double v, double d) {
  const int ev = (__double2hiint(v) >> 20) & 0x7FF;
  double r;
  if (ev < 300 || ev > 1800 || !recip_f32(d, r)) return v / d;  // zeros, infinities, NaN, extremes
  double q = v * r;
  q = fma(fma(-d, q, v), r, q);
  return fma(fma(-d, q, v), r, q);
}

// 1/d for a positive normal d: the FP32 reciprocal of its significand, its
// exponent put back, refined by a third-order Newton step (Householder's method)
// to about an ulp.  No branch, so that the steps around it can overlap; odd: d is
// too near the ends of the range.
__device__ __forceinline__ double recip_pos(double d, bool &odd) {
  const int hi = __double2hiint(d), ed = (hi >> 20) & 0x7FF;
  odd |= ed < 2 || ed > 2040;
  const float f = __int_as_float(0x3F800000 | ((hi & 0xFFFFF) << 3) | ((unsigned)__double2loint(d) >> 29));
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f));
  const int b = __float_as_int(r);  // 0.5 .. 1
  const double r0 = __hiloint2double((((b >> 23) + 1919 - ed) << 20) | ((b >> 3) & 0xFFFFF), b << 29);
  const double e = fma(-d, r0, 1.0);
  return fma(r0, fma(e, e, e), r0);
}

// 1/sqrt(d) likewise: FP32 seed for the significand in [1, 4), third-order step.
__device__ __forceinline__ double rsqrt_pos(double d, bool &odd) {
  const int hi = __double2hiint(d), ed = (hi >> 20) & 0x7FF;
  odd |= ed < 2 || ed > 2040;
  const int up = (ed & 1) ^ 1;  // exponent ed - 1023 = 2 half + up
  const float f = __int_as_float(((127 + up) << 23) | ((hi & 0xFFFFF) << 3) | ((unsigned)__double2loint(d) >> 29));
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f));
  const int b = __float_as_int(r), half = (ed - 1023 - up) / 2;
  const double y = __hiloint2double((((b >> 23) + 896 - half) << 20) | ((b >> 3) & 0xFFFFF), b << 29);
  const double e = fma(-d * y, y, 1.0);
  return fma(y, e * fma(0.375, e, 0.5), y);
}

// C(m,n) = alpha v + beta C(m,n), v divided by the orbital-energy denominator
// if the product has one; P: RowMap A, B; C, alpha, beta, denom, eo, ev
template <class Params>
__device__ __forceinline__ void put_c(const Params &P, int m, int n, double v) {
  if (P.denom) {
    // RIMP2.F90:403-404: deltaEPS = EVocc(I)+EVocc(J)-EVvirt(B)-EVvirt(A)
    const double d = P.eo[role_index(P.A, m, 1)] + P.eo[role_index(P.B, n, 1)] -
                     P.ev[role_index(P.B, n, 0)] - P.ev[role_index(P.A, m, 0)];
    v = div_f64(v, d);
  }
  double *c = P.C + c_off(P.A, m) + c_off(P.B, n);
  v = P.alpha * v;
  if (P.beta != 0.0) v += P.beta * *c;
  *c = v;
}
#endif

// Residue planes of a set of rows: [plane][K chunk of 64][row][64] FP16.
struct ModOperand {
  DevBuf planes, e, flag;
  int rows = 0, nkc = 0;
};

size_t mod_operand_bytes(int rows, int K);
// out[plane][n][ldm] = residues of sum_k Q(m,k) L(n,k)
int mod_product(const ModOperand &L, const ModOperand &Q, signed char *out, long long ldm, bool lower,
                cudaStream_t s);
double mod_gemm_time(double m, double n, double k, bool lower);  // seconds, estimated
int mod_gemm_block(int K);
// The contraction of g, folded into rows A and columns B; *handled = false
// where it cannot be (length, capture, no room for the workspace): nothing was
// launched.
int mod_gemm(const GemmDesc &g, const RowMap &A, const RowMap &B, cudaStream_t s, bool *handled);

}  // namespace rimp2
