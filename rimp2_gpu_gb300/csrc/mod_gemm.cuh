// mod_gemm.cuh -- FP64 contractions on the FP16 tensor cores by residue
// arithmetic (mod_gemm.cu): operands, products and the general contraction.
#pragma once
#include "common.cuh"

namespace rimp2 {

constexpr int MG_P = 16;             // moduli
constexpr int MG_PLANES = MG_P + 1;  // and the plane of magnitudes
// least sum |a||b| of an element, as a part of ||a|| ||b|| = 2^24 in the units
// of the magnitudes' plane, below which it is summed in FP64
constexpr float MG_TAU = 65536.0f;
constexpr int MG_TILE_MAX = 512;     // of a 64 x 64 tile's elements; beyond it the whole tile is

constexpr int MG_K_MIN = 8, MG_K_MAX = 16384;  // lengths of a sum

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

// Residue planes of a set of rows: [plane][K chunk of 64][row][64] FP16.
struct ModOperand {
  DevBuf planes, e, flag;
  int rows = 0, nkc = 0;
};

size_t mod_operand_bytes(int rows, int K);
int mod_operand_alloc(ModOperand &op, int rows, int K, cudaStream_t s);
// rows [row0, row0 + op.rows) of M; col: as the columns' operand of a product
int mod_operand_fill(ModOperand &op, const RowMap &M, int row0, bool col, cudaStream_t s);
// out[plane][n][ldm] = residues of sum_k Q(m,k) L(n,k)
int mod_product(const ModOperand &L, const ModOperand &Q, signed char *out, long long ldm, bool lower,
                cudaStream_t s);
bool mod_gemm_pays(const GemmDesc &g, double m, double n);
double mod_gemm_time(double m, double n, double k, bool lower);  // seconds, estimated
int mod_gemm_block(int K);
// The contraction of g; *handled = false where FP64 tensor operations are the
// better way (or there is no room for the workspace): nothing was launched.
int mod_gemm(const GemmDesc &g, cudaStream_t s, bool *handled);

}  // namespace rimp2
