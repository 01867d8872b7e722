// mod_gemm.cu -- FP64 contractions on the FP16 tensor cores by residue
// arithmetic.
//
// GB300 runs FP64 tensor operations (DMMA) at 1.05 TFLOP/s and FP16 ones at
// 1900 TFLOP/s.  A contraction C(m,n) = sum_k A(m,k) B(k,n) of FP64 numbers is
// therefore evaluated with integers (the modular form of Ozaki's scheme:
// Ozaki, Uchino, Imamura, "Ozaki Scheme II", 2025):
//   1. every row of A and every column of B is scaled by a power of two and
//      rounded to integers a', b' with 2-norm at most 2^62 (62 bits where the
//      FP64 fraction has 53: an element keeps every bit it has down to 2^-9 of
//      its row's norm);
//   2. X = sum a' b' is an integer with |X| <= 2^124 (Cauchy-Schwarz), fixed
//      by its residues modulo 16 pairwise coprime numbers of at most 8 bits
//      whose product P is 2^125.1;
//   3. residues are at most 128 in magnitude, exact in FP16, and 1024 of their
//      products sum to at most 2^24: the FP32 accumulation of the tensor core
//      is exact, whatever its internal rounding;
//   4. the fraction X/P = sum_p r_p w_p / p mod 1, w_p = (P/p)^-1 mod p (Chinese
//      remainder theorem), is summed in 96-bit fixed point,
//      multiplied by P and rounded once to FP64 (a fraction below 2^-28 is
//      redone in exact integers): a sum that FP64 can hold comes out exact.
// Everything between the rounding to 62-bit integers and the final rounding
// is exact.  The rounding error of (1) in X is about 0.41 * 2^62, i.e.
// 0.41 * 2^-9 u * (2^124 / sum|a'||b'|) relative to u sum|a||b| (u = 2^-53),
// below what FP64 summation itself loses unless sum|a||b| is a tiny part of
// ||a|| ||b|| (rows whose large elements meet only small ones).  A 17th
// product of the magnitudes, in FP16, measures sum|a||b| for every element
// (from below, over all of K); an element whose measure is under 2^-8 of the largest
// norms' product (2^-8 to 2^-6 of ||a|| ||b||, as the scales are powers of two) is
// summed in FP64 instead (one warp per element, or a DMMA tile where an
// eighth of a tile needs it).  Rows with infinities, NaNs or extreme
// exponents take that way too, so every element is what FP64 arithmetic would
// make it, up to FP64's own rounding.
//
// Kernels: row_scale (norms -> exponents), residue (17 FP16 planes per
// operand), mod_gemm (persistent CTA pairs, 256 x 256 tiles, TMA + tcgen05,
// one product per plane; the epilogue reduces modulo p and stores bytes),
// crt_epilogue (fixed-point reconstruction, scaling, denominators; the
// elements and tiles to be summed in FP64).
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <vector>

#include "tc.cuh"
#include "mod_gemm.cuh"

namespace rimp2 {
void count_launch(int n);

namespace {

// --------------------------------------------------------------------------
// constants of the residue system
// --------------------------------------------------------------------------
typedef unsigned __int128 u128;

// Pairwise coprime, at most 251 but for 256: the FP32 reduction of a sum below
// 2^24 leaves |r| <= 0.507 p, which has to fit a signed byte (256 wraps onto
// itself).
struct ModTables {
  float p[MG_P], inv[MG_P];
  float limb[MG_P][5];    // 2^(13 l) mod p, symmetric
  int w[MG_P];            // (P/p)^-1 mod p, symmetric
  unsigned phi[4][12];    // byte b of round(2^96 (w / p mod 1)) for p = 4q .. 4q+3
  unsigned long long pm;  // P 2^-62
  unsigned long long plo, phi64;         // P
  unsigned long long wlo[MG_P], whi[MG_P];  // P / p
};

constexpr int sym(long long v, int p) {
  v %= p;
  if (v < 0) v += p;
  return (int)(2 * v > p ? v - p : v);
}

constexpr ModTables make_tables() {
  ModTables t{};
  const int ps[MG_P] = {256, 251, 249, 247, 245, 241, 239, 233, 229, 227, 223, 211, 199, 197, 193, 191};
  u128 P = 1;
  for (int i = 0; i < MG_P; ++i) P *= (u128)ps[i];
  for (int i = 0; i < MG_P; ++i) {
    const int p = ps[i];
    t.p[i] = (float)p;
    t.inv[i] = 1.0f / (float)p;
    const int q = (int)((P / (u128)p) % (u128)p);
    int inv = 0;
    for (int x = 1; x < p; ++x)
      if ((long long)x * q % p == 1) inv = x;
    long long w = 1;
    for (int l = 0; l < 5; ++l) {
      t.limb[i][l] = (float)sym(w, p);
      w = w * 8192 % p;
    }
    t.w[i] = sym(inv, p);
    const u128 phi = (((u128)inv << 96) + (u128)(p / 2)) / (u128)p;  // inv < p: below 2^96
    for (int b = 0; b < 12; ++b)
      t.phi[i >> 2][b] |= (unsigned)((phi >> (8 * b)) & 0xFF) << (8 * (i & 3));
    const u128 w128 = P / (u128)p;
    t.wlo[i] = (unsigned long long)w128;
    t.whi[i] = (unsigned long long)(w128 >> 64);
  }
  t.pm = (unsigned long long)(P >> 62);
  t.plo = (unsigned long long)P;
  t.phi64 = (unsigned long long)(P >> 64);
  return t;
}
constexpr ModTables HT = make_tables();
__constant__ ModTables DT = HT;

constexpr float MAGIC = 12582912.0f;  // 1.5 * 2^23: adds round to an integer

// --------------------------------------------------------------------------
// operands
// --------------------------------------------------------------------------
// Norm of a row in pieces: largest exponent, sum of squares relative to it
// (FP32: its rounding, below 2^-10, is inside the margin of the scale), the
// lowest set bit, and whether a value is infinite or NaN.
struct RowStat {
  int e;      // largest biased exponent so far (0: all zero)
  float ss;   // sum of (x 2^(1023-e))^2
  int lsb;    // exponent of the lowest set bit of any value
  int bad;
};

__device__ __forceinline__ float pow2f(int k) {  // 2^k, 0 below the normal range
  return k < -126 ? 0.0f : __uint_as_float((unsigned)(k + 127) << 23);
}

__device__ __forceinline__ void stat_add(RowStat &s, double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFull;
  if (b == 0) return;
  const int ed = (int)(b >> 52);
  if (ed == 0x7FF) {
    s.bad = 1;
    return;
  }
  const unsigned long long f = b & 0xFFFFFFFFFFFFFull;
  const int tz = f ? __ffsll((long long)f) - 1 : 52;
  s.lsb = min(s.lsb, (ed ? ed : 1) - 1075 + tz);
  if (ed > s.e) {
    s.ss *= pow2f(2 * (s.e - ed));
    s.e = ed;
  }
  const float m = __uint_as_float(0x3F800000u | (unsigned)(f >> 29)) * pow2f(ed - s.e);
  s.ss = fmaf(m, m, s.ss);
}

__device__ __forceinline__ void stat_merge(RowStat &s, int e, float ss, int lsb, int bad) {
  const int m = max(s.e, e);
  s.ss = s.ss * pow2f(2 * (s.e - m)) + ss * pow2f(2 * (e - m));
  s.e = m;
  s.lsb = min(s.lsb, lsb);
  s.bad |= bad;
}

// Scale exponent: ||x|| 2^e <= 2^62 / 1.002.  Rows with values beyond
// 2^+-400 are left to FP64: the reconstruction assembles exponents.
__device__ __forceinline__ void stat_store(const RowStat &s, int *e, unsigned char *flag) {
  if (s.bad || (s.e != 0 && (s.e < 1023 - 400 || s.e > 1023 + 400))) {
    *e = 0;
    *flag = MG_ROW_FP64;
    return;
  }
  if (s.e == 0) {  // zeros (a row of subnormal values has lsb < 0 and goes to FP64)
    *e = 0;
    *flag = s.lsb == MG_NO_LSB ? MG_ROW_ZERO : MG_ROW_FP64;
    return;
  }
  const float h = sqrtf(s.ss) * 1.002f;
  const int c = (int)((__float_as_uint(h) >> 23) & 0xFFu) - 127 + 1;
  const int ee = 62 - (s.e - 1023) - c;
  *e = ee;
  *flag = s.lsb + ee >= 0 ? MG_ROW_EXACT : 0;
}

// One operand's work of the two kernels below.
struct OpArgs {
  RowMap M;
  int row0, rows, nkc;
  int blocks;            // of the kernel's grid
  int *e;
  unsigned char *flag;
  __half *out;
  size_t plane;
};

// K-contiguous rows: one warp per row, four loads in flight per lane.  Rows
// along the fast direction: a block takes 32 rows, each warp a part of K.
// Both operands of a product in one launch (short ones are launch-bound).
__global__ void __launch_bounds__(256) row_scale_kernel(const __grid_constant__ OpArgs A,
                                                        const __grid_constant__ OpArgs B) {
  __shared__ RowStat sh[8][32];
  const bool second = (int)blockIdx.x >= A.blocks;
  const OpArgs &P = second ? B : A;
  const RowMap &M = P.M;
  const int blk = (int)blockIdx.x - (second ? A.blocks : 0);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  RowStat s{0, 0.0f, MG_NO_LSB, 0};
  if (M.sk == 1) {
    const int r = blk * 8 + w;
    if (r >= P.rows) return;
    const double *x = M.base + row_off(M, P.row0 + r);
    for (int k0 = lane; k0 < M.K; k0 += 128) {
      double v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = k0 + 32 * u < M.K ? x[k0 + 32 * u] : 0.0;
#pragma unroll
      for (int u = 0; u < 4; ++u) stat_add(s, v[u]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const int e2 = __shfl_xor_sync(0xffffffffu, s.e, o);
      const float s2 = __shfl_xor_sync(0xffffffffu, s.ss, o);
      const int l2 = __shfl_xor_sync(0xffffffffu, s.lsb, o);
      const int b2 = __shfl_xor_sync(0xffffffffu, s.bad, o);
      stat_merge(s, e2, s2, l2, b2);
    }
    if (lane == 0) stat_store(s, P.e + r, P.flag + r);
    grid_trigger();
    return;
  }
  const int r = blk * 32 + lane;
  if (r < P.rows) {
    const double *x = M.base + row_off(M, P.row0 + r);
    for (int k0 = w; k0 < M.K; k0 += 64) {
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = k0 + 8 * u < M.K ? x[(long long)(k0 + 8 * u) * M.sk] : 0.0;
#pragma unroll
      for (int u = 0; u < 8; ++u) stat_add(s, v[u]);
    }
  }
  sh[w][lane] = s;
  __syncthreads();
  if (w == 0 && r < P.rows) {
    for (int q = 1; q < 8; ++q) {
      const RowStat &t = sh[q][lane];
      stat_merge(s, t.e, t.ss, t.lsb, t.bad);
    }
    stat_store(s, P.e + r, P.flag + r);
  }
  grid_trigger();
}

// |x| 2^e rounded to an integer (< 2^63)
__device__ __forceinline__ unsigned long long to_int(double x, int e) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int ed = (int)((b >> 52) & 0x7FF);
  const unsigned long long m = (b & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
  const int sh = ed - 1075 + e;
  if (ed == 0 || sh < -54) return 0;
  return sh >= 0 ? m << sh : (m + (1ull << (-sh - 1))) >> (-sh);
}

// Residues of eight consecutive K values of one row: 16 bytes per plane.
// Five 13-bit limbs times the residues of 2^(13 l), summed in FP32 (exact:
// below 2^23), reduced once, packed to FP16 with the value's sign: 9 operations
// per value and modulus.  8 bytes read and 34 written a value bound it with them: 117
// us for 2048 x 8192, 6.0 TB/s at 82% of the issue slots.
__device__ __forceinline__ void residues8(const double (&v)[8], int e, bool live,
                                          __half *__restrict__ out, size_t plane) {
  float l[5][8];
  unsigned sg[4] = {0u, 0u, 0u, 0u};
  uint4 gq;
  __half2 *gh = reinterpret_cast<__half2 *>(&gq);
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const unsigned long long x = live ? to_int(v[u], e) : 0ull;
#pragma unroll
    for (int q = 0; q < 5; ++q)
      l[q][u] = __uint_as_float(0x4B000000u | (unsigned)((x >> (13 * q)) & 0x1FFFu)) - 8388608.0f;
    if (__double2hiint(v[u]) < 0) sg[u >> 1] |= (u & 1) ? 0x80000000u : 0x8000u;
  }
#pragma unroll
  for (int u = 0; u < 8; u += 2) {  // |x| 2^-50 (norm 2^12): the magnitudes' plane
    const float a = fmaf(l[4][u], 4.0f, fmaf(l[3][u], 4.8828125e-4f, l[2][u] * 5.9604645e-8f));
    const float b = fmaf(l[4][u + 1], 4.0f, fmaf(l[3][u + 1], 4.8828125e-4f, l[2][u + 1] * 5.9604645e-8f));
    gh[u >> 1] = __floats2half2_rn(a, b);
  }
  *reinterpret_cast<uint4 *>(out + (size_t)MG_P * plane) = gq;
#pragma unroll
  for (int p = 0; p < MG_P; ++p) {
    const float pf = DT.p[p], inv = DT.inv[p];
    uint4 o;
    unsigned *ow = reinterpret_cast<unsigned *>(&o);
#pragma unroll
    for (int u = 0; u < 8; u += 2) {
      float r[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float y = l[0][u + h] * DT.limb[p][0];
#pragma unroll
        for (int q = 1; q < 5; ++q)
          y = fmaf(l[q][u + h], DT.limb[p][q], y);
        const float q = fmaf(y, inv, MAGIC) - MAGIC;
        r[h] = fmaf(-q, pf, y);
      }
      const __half2 hh = __floats2half2_rn(r[0], r[1]);
      ow[u >> 1] = *reinterpret_cast<const unsigned *>(&hh) ^ sg[u >> 1];
    }
    *reinterpret_cast<uint4 *>(out + (size_t)p * plane) = o;
  }
}

// out[(p * nkc + kc) * rows + row][64]; a block takes 32 rows of one K chunk.
// A: the rows' operand, B: the columns'.  SCALE: the rows are one chunk long,
// the eight threads of a row find its scale themselves (no row_scale launch).
template <bool SCALE>
__global__ void __launch_bounds__(256) residue_kernel(const __grid_constant__ OpArgs A,
                                                      const __grid_constant__ OpArgs B) {
  __shared__ double sh[64][33];
  grid_wait();
  const bool second = (int)blockIdx.x >= A.blocks;
  const OpArgs &P = second ? B : A;
  const RowMap &M = P.M;
  const int blk = (int)blockIdx.x - (second ? A.blocks : 0);
  const int nrb = (P.rows + 31) / 32, kc = blk / nrb, rb = blk % nrb;
  const int rr = threadIdx.x >> 3, kq = threadIdx.x & 7, r = rb * 32 + rr, k0 = kc * 64 + kq * 8;
  double v[8];
  if (M.sk == 1) {
    if (r >= P.rows) return;
    const double *x = M.base + row_off(M, P.row0 + r);
    if ((((uintptr_t)x) & 15) == 0 && k0 + 8 <= M.K) {
#pragma unroll
      for (int u = 0; u < 8; u += 2) {
        const double2 d = *reinterpret_cast<const double2 *>(x + k0 + u);
        v[u] = d.x;
        v[u + 1] = d.y;
      }
    } else {
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = k0 + u < M.K ? x[k0 + u] : 0.0;
    }
  } else {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, rl = rb * 32 + lane;
    const double *x = M.base + (rl < P.rows ? row_off(M, P.row0 + rl) : 0);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = kc * 64 + w + 8 * u;
      sh[w + 8 * u][lane] = rl < P.rows && k < M.K ? x[(long long)k * M.sk] : 0.0;
    }
    __syncthreads();
    if (r >= P.rows) return;
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = sh[kq * 8 + u][rr];
  }
  int e;
  unsigned char flag;
  if (SCALE) {
    RowStat s{0, 0.0f, MG_NO_LSB, 0};
#pragma unroll
    for (int u = 0; u < 8; ++u) stat_add(s, v[u]);
    const unsigned group = 0xFFu << (threadIdx.x & 24);  // rows leave by groups of eight
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      const int e2 = __shfl_xor_sync(group, s.e, o);
      const float s2 = __shfl_xor_sync(group, s.ss, o);
      const int l2 = __shfl_xor_sync(group, s.lsb, o);
      const int b2 = __shfl_xor_sync(group, s.bad, o);
      stat_merge(s, e2, s2, l2, b2);
    }
    stat_store(s, &e, &flag);
    if (kq == 0) {
      P.e[r] = e;
      P.flag[r] = flag;
    }
  } else {
    e = P.e[r];
    flag = P.flag[r];
  }
  const bool live = !(flag & MG_ROW_FP64);
  __half *out = P.out + ((size_t)kc * P.rows + r) * 64 + kq * 8;
  residues8(v, e, live, out, P.plane);
  grid_trigger();
}

// --------------------------------------------------------------------------
// products: persistent CTA pairs
// --------------------------------------------------------------------------
// Work item = (plane, 256 columns n x TQ rows m of C): the columns' operand
// lies on the TMEM lanes (M = 256 over the pair), the rows' operand on the
// accumulator columns (N = TQ, half of it in each CTA), so that a thread
// stores runs of bytes along m.  Two (four) TQ-column accumulators per CTA: the
// MMAs of one item run while the epilogue reduces another.  Sums longer
// than 1024 are cut there (exactness) and joined modulo p in the epilogue's
// registers.  A 64-deep stage is 32 KB per CTA (TQ = 256), six stages.  Bound by the
// tensor cores: 1.77 PFLOP/s (1.36 ms for the triangle of 8192 columns, sums of
// 2048, 17 planes).
// TQ, the rows of C in a tile, is 128 or 64 where 256 would mostly be padding
// (a product with few rows; one with few columns is transposed): its MMAs and
// epilogue shrink with it, the lanes' operand is read as before (64 rows x 13148,
// sums of 64: 16 us; 24.5 while the arrival
// on an accumulator's barrier released the stores before it).
constexpr int MG_THREADS = 320;
constexpr int MG_SEG = 16;  // most K chunks of an exact sum
constexpr int mg_stage(int tq) { return PANEL_BYTES + tq / 2 * KSTEP * 2; }
constexpr int mg_nst(int tq) { return tq == 256 ? 6 : 8; }
constexpr int mg_nacc(int tq) { return tq == 256 ? 2 : 4; }  // accumulators: short sums need more in flight
constexpr int mg_smem(int tq) { return mg_nst(tq) * mg_stage(tq) + 1024 + 256; }
static_assert(tmem_alone(mg_smem(64)) && tmem_alone(mg_smem(128)) && tmem_alone(mg_smem(256)), "tensor memory");

struct MgParams {
  int rows_l, rows_q;        // rows per K chunk of the two operands
  int tiles_l, tiles_q;      // 256 columns, TQ rows
  int nkc, seg, nseg;        // K chunks, those of one exact sum, its number
  int lower;                 // square, only tiles with an element m >= n
  signed char *out;          // [plane][n][ldm]
  long long ldm;
  int *err;
};

// K chunks of one sum: the magnitudes need not be exact and are measured over all of K
__device__ __forceinline__ int mg_seg(const MgParams &P, int plane) { return plane == MG_P ? P.nkc : P.seg; }

// Items are numbered without gaps and dealt in turn: every pair of CTAs gets
// as many, also of a triangle's tiles.
__host__ __device__ inline int mg_tiles(const MgParams &P) {
  return P.lower ? P.tiles_q * (P.tiles_q + 1) / 2 : P.tiles_l * P.tiles_q;
}

__device__ __forceinline__ void mg_item(const MgParams &P, int item, int &plane, int &tl, int &tq) {
  const int tiles = mg_tiles(P);
  plane = item / tiles;
  const int t = item % tiles;
  if (P.lower) {
    int q = (int)((sqrtf(8.0f * t + 1.0f) - 1.0f) * 0.5f);
    while ((q + 1) * (q + 2) / 2 <= t) ++q;
    while (q * (q + 1) / 2 > t) --q;
    tq = q;
    tl = t - q * (q + 1) / 2;
    return;
  }
  // groups of eight column tiles: the tiles in flight share their operands in L2
  const int per = 8 * P.tiles_q, g = t / per, rem = t % per;
  const int gs = min(8, P.tiles_l - 8 * g);
  tl = 8 * g + rem % gs;
  tq = rem / gs;
}

template <int TQ>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(MG_THREADS, 1)
    mod_gemm_kernel(const __grid_constant__ CUtensorMap tmL, const __grid_constant__ CUtensorMap tmQ,
                    MgParams P) {
  constexpr int NST = mg_nst(TQ), STAGE = mg_stage(TQ);
  constexpr int NACC = mg_nacc(TQ);
  constexpr int NG = TQ / 32;  // groups of 16 accumulator columns per epilogue warp
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *base = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  // bars: full[NST], empty[NST], tfull[NACC], tempty[NACC], drain
  uint64_t *bars = (uint64_t *)(base + NST * STAGE);
  uint32_t *tmem_slot = (uint32_t *)(bars + 2 * NST + 2 * NACC + 1);
  volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const bool leader = rank == 0;
  const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[NST]);
  const uint32_t tfull0 = smem_u32(&bars[2 * NST]), tempty0 = smem_u32(&bars[2 * NST + NACC]);
  const uint32_t drain = smem_u32(&bars[2 * NST + 2 * NACC]);
  const uint32_t full0_L = map_shared(full0, 0), tempty0_L = map_shared(tempty0, 0);
  const uint32_t abort_peer = map_shared(smem_u32((const void *)abort_flag), rank ^ 1u);
  const int nitems = MG_PLANES * mg_tiles(P);
  const int pair = blockIdx.x >> 1, npair = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NST; ++s) {
      mbar_init(full0 + 8 * s, 1);   // rank 0: its producer's arrive + both CTAs' bytes
      mbar_init(empty0 + 8 * s, 1);  // multicast MMA commit
    }
    for (int u = 0; u < NACC; ++u) {
      mbar_init(tfull0 + 8 * u, 1);
      mbar_init(tempty0 + 8 * u, 16);  // the epilogue warps of both CTAs
    }
    mbar_init(drain, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&tmL) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&tmQ) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                     smem_u32(tmem_slot))
                 : "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers are initialised before any remote access
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  if (warp == 1)  // both CTAs hold their columns
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  grid_wait();

  if (warp == 0) {
    // --------------------- TMA producers (both CTAs) ---------------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0, armed = 0, armed_par = 0;
      bool ok = true;
      for (int item = pair; item < nitems && ok; item += npair) {
        int p, tl, tq;
        mg_item(P, item, p, tl, tq);
        const int rl = tl * 256 + 128 * (int)rank, rq = tq * TQ + TQ / 2 * (int)rank;
        for (int kc = 0; kc < P.nkc; ++kc) {
          if (!pair_wait(empty0 + 8 * stage, phase ^ 1, false, abort_flag, abort_peer, P.err, 21)) {
            ok = false;
            break;
          }
          if (leader) {
            mbar_expect_tx(full0 + 8 * stage, 2 * STAGE);
            armed |= 1u << stage;
            armed_par = (armed_par & ~(1u << stage)) | (phase << stage);
          }
          const uint32_t dst = smem_u32(base + stage * STAGE), fb = full0_L + 8 * stage;
          tma_load_3d_pair(dst, &tmL, fb, 0, kc * P.rows_l + rl, p);
          tma_load_3d_pair(dst + PANEL_BYTES, &tmQ, fb, 0, kc * P.rows_q + rq, p);
          if (++stage == NST) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      if (leader && (!ok || *abort_flag)) {  // copies in flight complete before the pair exits
        for (int s = 0; s < NST; ++s) {
          if (!((armed >> s) & 1u)) continue;
          const long long t0 = clock64();
          while (!mbar_test(full0 + 8 * s, (armed_par >> s) & 1u) && clock64() - t0 < WAIT_BUDGET) {
          }
        }
      }
    }
  } else if (warp == 1) {
    // --------------------- MMA issuer (rank 0 only) ----------------------
    if (lane == 0 && leader) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      unsigned t = 0;  // sums so far
      for (int item = pair; item < nitems && ok; item += npair) {
        int p, tl, tq;
        mg_item(P, item, p, tl, tq);
        const int seg = mg_seg(P, p);
        for (int s0 = 0; s0 < P.nkc && ok; s0 += seg, ++t) {
          const int u = (int)(t % NACC);
          if (t >= NACC && !pair_wait(tempty0 + 8 * u, (uint32_t)((t / NACC - 1) & 1), true, abort_flag,
                                   abort_peer, P.err, 22)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t d = tmem + (uint32_t)(u * TQ);
          const int s1 = min(P.nkc, s0 + seg);
          for (int kc = s0; kc < s1; ++kc) {
            if (!pair_wait(full0 + 8 * stage, phase, false, abort_flag, abort_peer, P.err, 23)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t sb = smem_u32(base + stage * STAGE);
#pragma unroll
            for (int k16 = 0; k16 < KSTEP / 16; ++k16)
              mma_f16_pair(d, smem_desc(sb + k16 * 32), smem_desc(sb + PANEL_BYTES + k16 * 32),
                           idesc_mn(256, TQ), (kc > s0 || k16 > 0) ? 1u : 0u);
            mma_commit_pair(empty0 + 8 * stage);  // frees the stage in both CTAs
            if (++stage == NST) {
              stage = 0;
              phase ^= 1;
            }
          }
          if (!ok) break;
          mma_commit_pair(tfull0 + 8 * u);
        }
      }
      mma_commit_pair(drain);  // both CTAs learn when the last MMA has completed
    }
  } else {
    // --------------------- epilogue (both CTAs) ---------------------------
    const int quad = warp & 3, half = (warp - 2) >> 2;
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
    const int nl = P.rows_l;
    unsigned t = 0;
    bool ok = true;
    for (int item = pair; item < nitems && ok; item += npair) {
      int p, tl, tq;
      mg_item(P, item, p, tl, tq);
      const int n = tl * 256 + 128 * (int)rank + quad * 32 + lane;
      const bool mag = p == MG_P;
      const float pf = mag ? 1.0f : DT.p[p], inv = mag ? 1.0f : DT.inv[p];
      uint32_t pk[NG][4];
      const int sums = mag ? 1 : P.nseg;  // counted: with the bound in K chunks 2% slower
      for (int s0 = 0; s0 < sums; ++s0, ++t) {
        const int u = (int)(t % NACC);
        ok = pair_wait(tfull0 + 8 * u, (uint32_t)((t / NACC) & 1), false, abort_flag, abort_peer, P.err, 24);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const uint32_t ta = tmem + lane_off + (uint32_t)(u * TQ + half * (TQ / 2));
#pragma unroll
        for (int g = 0; g < NG; ++g) {
          float v[16];
          tmem_ld16(ta + g * 16, v);
          tmem_wait_ld();
          if (mag) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint32_t w = 0u;
#pragma unroll
              for (int k = 0; k < 4; ++k) w |= v[4 * q + k] >= MG_TAU ? 1u << (8 * k) : 0u;
              pk[g][q] = w;
            }
          } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint32_t b[4];
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const float y = v[4 * q + k];
                float r = fmaf(-(fmaf(y, inv, MAGIC) - MAGIC), pf, y);
                if (s0) {  // join with the earlier sums' residue, modulo p
                  r += (float)(signed char)(pk[g][q] >> (8 * k));
                  r = fmaf(-(fmaf(r, inv, MAGIC) - MAGIC), pf, r);
                }
                b[k] = __float_as_uint(r + MAGIC);  // low byte: the residue
              }
              pk[g][q] = __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410);
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        // nothing to release: the accumulator's loads are complete (tcgen05.wait::ld), and
        // the arrival says no more than that; not for a barrier that stores rely on
        if (lane == 0) mbar_arrive_relaxed(tempty0_L + 8 * u);
      }
      if (ok && n < nl) {
        signed char *o = P.out + ((long long)p * nl + n) * P.ldm + tq * TQ + half * (TQ / 2);
#pragma unroll
        for (int g = 0; g < NG; ++g)
          *reinterpret_cast<uint4 *>(o + g * 16) = make_uint4(pk[g][0], pk[g][1], pk[g][2], pk[g][3]);
      }
    }
  }
  __syncthreads();
  if (warp == 1 && lane == 0) {
    // the last MMA of the pair has completed (it may write this CTA's TMEM)
    const long long t0 = clock64();
    while (!mbar_test(drain, 0) && clock64() - t0 < WAIT_BUDGET) {
    }
  }
  if (*abort_flag) {
    // after an abort the peer may still have copies in flight into its own
    // shared memory (their completion is counted in rank 0): give them time
    const long long t0 = clock64();
    while (clock64() - t0 < 4000000LL) {
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  }
}

// --------------------------------------------------------------------------
// reconstruction and epilogue
// --------------------------------------------------------------------------
__device__ __forceinline__ int dp4a_su(unsigned a, unsigned b, int c) {
  int d;
  asm("dp4a.s32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

// m 2^(x - 63) rounded to 53 bits, m's top bit set
__device__ __forceinline__ double assemble(unsigned long long m, int x, bool neg) {
  const unsigned long long f = (m >> 11) + ((m >> 10) & 1);  // 2^52 .. 2^53
  const unsigned long long bits = ((unsigned long long)(1022 + x) << 52) + f;
  return __longlong_as_double((long long)(bits | (neg ? 0x8000000000000000ull : 0ull)));
}

// X 2^-eab where |X / P| < 2^-28: X = sum_p v_p P/p - k P in 128-bit integers
// (wrapping), v_p = r_p w_p mod p, k the whole part of sum_p v_p / p.  Sums that cancel exactly,
// or nearly, come here: the fraction's 96 bits would leave them too few.
// src: the element's residues, one byte per plane.
__device__ __forceinline__ double crt_small(const signed char *src, long long plane, int eab) {
  unsigned long long lo = 0, hi = 0;
  float ks = 0.0f;
#pragma unroll 4
  for (int p = 0; p < MG_P; ++p) {
    const int rw = src[p * plane] * DT.w[p];
    const long long v = rw - (int)rintf((float)rw * DT.inv[p]) * (int)DT.p[p];
    ks = fmaf((float)v, DT.inv[p], ks);
    const unsigned long long w = DT.wlo[p], q = lo + w * (unsigned long long)v;
    hi += DT.whi[p] * (unsigned long long)v + (unsigned long long)__mul64hi((long long)w, v) +
          (w >> 63 ? (unsigned long long)v : 0ull) + (q < lo);
    lo = q;
  }
  const long long k = (long long)rintf(ks);
  const unsigned long long w = DT.plo, t = w * (unsigned long long)k;
  hi -= DT.phi64 * (unsigned long long)k + (unsigned long long)__mul64hi((long long)w, k) +
        (w >> 63 ? (unsigned long long)k : 0ull) + (lo < t);
  lo -= t;
  const bool neg = (long long)hi < 0;
  if (neg) {
    lo = ~lo + 1;
    hi = ~hi + (lo == 0);
  }
  if ((hi | lo) == 0) return 0.0;
  const int n = hi ? __clzll((long long)hi) : 64 + __clzll((long long)lo);
  unsigned long long m = n >= 64 ? lo << (n - 64) : n ? (hi << n) | (lo >> (64 - n)) : hi;
  if (n < 64 && (lo << n)) m |= 1;  // what lies below only matters beside a tie
  return assemble(m, 127 - n - eab, neg);
}

// X 2^-eab for the residues r[q] (four signed bytes each): the fraction X/P in
// 96-bit fixed point (wrapping: the whole part drops out) times P.  False where
// the fraction is too small for that (crt_small).
__device__ __forceinline__ bool crt_value(const unsigned (&r)[4], int eab, double &v) {
  int s[12];
#pragma unroll
  for (int b = 0; b < 12; ++b) {
    s[b] = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) s[b] = dp4a_su(r[q], DT.phi[q][b], s[b]);
  }
  const long long low = (long long)(s[0] + (s[1] << 8)) + ((long long)(s[2] + (s[3] << 8)) << 16);
  const unsigned lo = (unsigned)low;
  long long h = (long long)(s[4] + (s[5] << 8)) + (low >> 32);
  h += (long long)(s[6] + (s[7] << 8)) << 16;
  h += (long long)((unsigned long long)(long long)(s[8] + (s[9] << 8)) << 32);
  h += (long long)((unsigned long long)(long long)(s[10] + (s[11] << 8)) << 48);
  const bool neg = h < 0;
  const unsigned l2 = neg ? 0u - lo : lo;
  const unsigned long long H = neg ? ~(unsigned long long)h + (lo == 0) : (unsigned long long)h;
  if (H < (1ull << 36)) return false;
  const int n = __clzll((long long)H);  // 1 .. 27
  const unsigned long long m = (H << n) | ((unsigned long long)l2 >> (32 - n));
  // m 2^-(64 + n) is the fraction, pm 2^62 the modulus P
  const unsigned long long q = __umul64hi(m, DT.pm);
  const int z = q >> 63 ? 0 : 1;
  v = assemble(q << z, 125 - n - z - eab, neg);
  return true;
}

struct CrtParams {
  RowMap A, B;               // C's rows m (A) and columns n (B)
  int row0, col0;            // of this part
  int nm, nn;                // rows and columns of this part
  const signed char *res;    // [plane][n][ldm]
  long long ldm;
  const int *ea, *eb;
  const unsigned char *fa, *fb;
  double *C;
  double alpha, beta;
  const double *eo, *ev;
  int denom, lower;
  int nfast;                 // C's fast direction is n
  int sym;                   // rows and columns are the same vectors: C(n,m) comes with C(m,n)
};

// Whether an element is left to FP64: the flags of its row and column, and
// its bit of the magnitudes' plane.
__device__ __forceinline__ bool needs_fp64(unsigned f, unsigned fn, unsigned measured) {
  return ((f | fn) & MG_ROW_FP64) ||
         (!((f | fn) & MG_ROW_ZERO) && !(f & fn & MG_ROW_EXACT) && !measured);
}

// What becomes of the products: every FP64 operation, a comparison or one
// whose result is not used too, takes half a clock of the SM an element, so that
// the common forms are instances of their own.
enum : int { CRT_ANY, CRT_PLAIN /* C = v */, CRT_MINUS /* C -= v */, CRT_QUOTIENT /* C = v / d */ };

// What a row or column of C brings to its elements.
struct Side {
  long long off;   // in C
  double eo, ev;   // orbital energies of its indices
};
template <int MODE>
__device__ __forceinline__ Side side(const CrtParams &P, const RowMap &M, int r) {
  Side s;
  s.off = c_off(M, r);
  s.eo = s.ev = 0.0;
  if (MODE == CRT_QUOTIENT || (MODE == CRT_ANY && P.denom)) {
    s.eo = P.eo[role_index(M, r, 1)];
    s.ev = P.ev[role_index(M, r, 0)];
  }
  return s;
}

// A block takes 64 rows x CN columns of C; a thread four consecutive rows of
// two columns.  It reads 17 bytes and writes 8 per element; its instructions
// (some 170 an element) bound it, so what only depends on the row or the column
// (offsets with their divisions, orbital energies) is formed once a block.  A symmetric product (g
// of one set of vectors with itself) has only the tiles m >= n: C(n,m) is
// written along with C(m,n) through shared memory, with the same denominator
// (the reference subtracts the two virtual energies in the other order there).
// Values whose large elements meet only small ones leave whole tiles to FP64, where
// the FP64 unit bounds a block (19 us of an SM for 64 x 64 x 16).
constexpr int DK = 16, DP = 20;
constexpr int crt_tile_max(int cn) { return 64 * cn / 8; }  // of a tile's elements; beyond it the whole tile is summed in FP64
constexpr int crt_dmma_bytes(int cn) { return (2 * (64 + cn) * DP + 64 + cn) * (int)sizeof(double); }
constexpr int crt_mirror_bytes(int cn) { return 64 * (cn + 1) * (int)sizeof(double); }

template <int MODE, int CN>
__global__ void __launch_bounds__(8 * CN, 1024 / (8 * CN)) crt_epilogue_kernel(const __grid_constant__ CrtParams P) {
  constexpr int NT = 8 * CN, HALF = CN / 2, SP = CN + 1, LANES = HALF < 16 ? HALF : 16;
  __shared__ int count;
  __shared__ Side sr[64], sc[CN];           // the tile's rows and columns
  __shared__ long long rows[64], cols[CN];  // symmetric: offsets of the mirror's columns
  extern __shared__ double S[];             // symmetric: [64][SP]; a tile summed in FP64: its operands
  const int tm = blockIdx.x, tn = blockIdx.y, td = tn * CN / 64;  // td: the diagonal's row tile
  grid_wait();
  const bool sym = CN == 64 && P.sym;  // narrower blocks of a diagonal tile would choose each for itself
  if ((P.lower || sym) && tm < td) return;
  const int tid = threadIdx.x;
  const int mq = (P.nfast ? tid / LANES % 16 : tid % 16) * 4;
  const int nq = P.nfast ? tid % LANES + tid / (16 * LANES) * LANES : tid / 16;
  const int m0 = tm * 64 + mq, n0 = tn * CN + nq;
  const long long plane = (long long)P.nn * P.ldm;
  const bool mirror = sym && tm != td;
  if (tid == 0) count = 0;
  if (tid < 64 && tm * 64 + tid < P.nm)
    sr[tid] = side<MODE>(P, P.A, P.row0 + tm * 64 + tid);
  else if (tid >= 64 && tid < 64 + CN && tn * CN + tid - 64 < P.nn)
    sc[tid - 64] = side<MODE>(P, P.B, P.col0 + tn * CN + tid - 64);
  if (mirror) {
    if (tid < 64 && tm * 64 + tid < P.nm) rows[tid] = c_off(P.B, tm * 64 + tid);
    if (tid < CN && tn * CN + tid < P.nn) cols[tid] = c_off(P.A, tn * CN + tid);
  }
  __syncthreads();
  // which elements are summed in FP64
  unsigned todo = 0;
  unsigned fm = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) fm |= (unsigned)(m0 + k < P.nm ? P.fa[m0 + k] : (unsigned)MG_ROW_ZERO) << (8 * k);
#pragma unroll
  for (int y = 0; y < 2; ++y) {
    const int n = n0 + HALF * y;
    if (n >= P.nn) continue;
    const unsigned g = *reinterpret_cast<const unsigned *>(P.res + MG_P * plane + n * P.ldm + m0);
    const unsigned fn = P.fb[n];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (m0 + k < P.nm && needs_fp64((fm >> (8 * k)) & 0xFFu, fn, (g >> (8 * k)) & 1u)) todo |= 1u << (4 * y + k);
  }
  if (todo) atomicAdd(&count, __popc(todo));
  __syncthreads();
  const int lane = tid & 31;
  auto put = [&](int ml, int nl, double v) {
    const Side &a = sr[ml], &b = sc[nl];
    if (MODE == CRT_QUOTIENT || (MODE == CRT_ANY && P.denom))
      v = div_f64(v, a.eo + b.eo - b.ev - a.ev);  // RIMP2.F90:403-404
    if (MODE == CRT_ANY && P.alpha != 1.0) v *= P.alpha;
    if (mirror) S[ml * SP + nl] = v;
    double *c = P.C + a.off + b.off;
    if (MODE == CRT_MINUS) v = *c - v;
    if (MODE == CRT_ANY && P.beta != 0.0) v += P.beta * *c;
    *c = v;
  };
  if (count > crt_tile_max(CN)) {
    // the whole tile with FP64 tensor operations: 16 x 16 of it a warp, the next 16
    // terms on their way by cp.async.  Rows 0 .. 63 of a buffer are the tile's
    // rows, the others its columns.
    double(*buf)[64 + CN][DP] = reinterpret_cast<double(*)[64 + CN][DP]>(S);
    long long *off = reinterpret_cast<long long *>(S + 2 * (64 + CN) * DP);
    const int K = P.A.K;
    if (tid < 64)
      off[tid] = tm * 64 + tid < P.nm ? row_off(P.A, P.row0 + tm * 64 + tid) : -1;
    else if (tid < 64 + CN)
      off[tid] = tn * CN + tid - 64 < P.nn ? row_off(P.B, P.col0 + tn * CN + tid - 64) : -1;
    __syncthreads();
    auto load = [&](int b, int q0) {
#pragma unroll 2
      for (int t = tid; t < (64 + CN) * DK; t += NT) {
        const bool col = t >= 64 * DK;
        const RowMap &M = col ? P.B : P.A;
        const int u = col ? t - 64 * DK : t, ext = col ? CN : 64;
        const int i = M.sk == 1 ? u / DK : u % ext, q = M.sk == 1 ? u % DK : u / ext, r = col ? 64 + i : i;
        const bool live = off[r] >= 0 && q0 + q < K;
        cp_async8(&buf[b][r][q], live ? M.base + off[r] + (long long)(q0 + q) * M.sk : M.base, live);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // the warps of 16 rows on the four schedulers: rows that a narrow product does not
    // have leave none idle
    const int gid = lane >> 2, tig = lane & 3, warp = tid >> 5;
    const int wm = warp / (CN / 16) * 16, wn = warp % (CN / 16) * 16;
    const bool work = tm * 64 + wm < P.nm && tn * CN + wn < P.nn;
    double acc[2][2][2] = {};
    load(0, 0);
    int cur = 0;
#pragma unroll 1
    for (int q0 = 0; q0 < K; q0 += DK, cur ^= 1) {
      if (q0 + DK < K) {
        load(cur ^ 1, q0 + DK);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
      } else {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
      }
      __syncthreads();
#pragma unroll
      for (int ks = 0; ks < DK; ks += 4) {
        if (!work || q0 + ks >= K) break;  // zeros from here on
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
          for (int y = 0; y < 2; ++y)
            asm volatile(
                "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                : "+d"(acc[x][y][0]), "+d"(acc[x][y][1])
                : "d"(buf[cur][wm + 8 * x + gid][ks + tig]), "d"(buf[cur][64 + wn + 8 * y + gid][ks + tig]));
      }
      __syncthreads();  // the buffer is refilled two slabs later; after the last one: the operands give way to the mirror
    }
#pragma unroll 1
    for (int e = 0; e < 8; ++e) {
      const int ml = wm + 8 * (e >> 2) + gid, nl = wn + 8 * ((e >> 1) & 1) + 2 * tig + (e & 1);
      double v = 0.0;
#pragma unroll
      for (int x = 0; x < 8; ++x) v = e == x ? acc[x >> 2][(x >> 1) & 1][x & 1] : v;
      if (tm * 64 + ml < P.nm && tn * CN + nl < P.nn) put(ml, nl, v);
    }
  } else {
  int ea[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) ea[k] = m0 + k < P.nm ? P.ea[m0 + k] : 0;
  unsigned small = 0;
#pragma unroll 1
  for (int y = 0; y < 2; ++y) {
    const int n = n0 + HALF * y;
    if (n < P.nn) {
      unsigned w[MG_P];
      const signed char *src = P.res + n * P.ldm + m0;
#pragma unroll
      for (int p = 0; p < MG_P; ++p) w[p] = *reinterpret_cast<const unsigned *>(src + p * plane);
      const int eb = P.eb[n];
      // 4 x 4 byte transposes: r[k][q] holds planes 4q .. 4q+3 of row m0 + k
      unsigned r[4][4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const unsigned a = __byte_perm(w[4 * q], w[4 * q + 1], 0x5140), b = __byte_perm(w[4 * q + 2], w[4 * q + 3], 0x5140);
        const unsigned c = __byte_perm(w[4 * q], w[4 * q + 1], 0x7362), d = __byte_perm(w[4 * q + 2], w[4 * q + 3], 0x7362);
        r[0][q] = __byte_perm(a, b, 0x5410);
        r[1][q] = __byte_perm(a, b, 0x7632);
        r[2][q] = __byte_perm(c, d, 0x5410);
        r[3][q] = __byte_perm(c, d, 0x7632);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        double v;
        if (m0 + k >= P.nm || ((todo >> (4 * y + k)) & 1u)) continue;
        if (crt_value(r[k], ea[k] + eb, v))
          put(mq + k, nq + HALF * y, v);
        else
          small |= 1u << (4 * y + k);
      }
    }
  }
  // the few others: exact integers, or a sum in FP64 by one warp
  if (__any_sync(0xffffffffu, small | todo)) {
#pragma unroll 1
    for (int x = 0; x < 8; ++x) {
      const int k = x & 3, y = x >> 2, n = n0 + HALF * y;
      if ((small >> x) & 1u)
        put(mq + k, nq + HALF * y, crt_small(P.res + n * P.ldm + m0 + k, plane, P.ea[m0 + k] + P.eb[n]));
      unsigned mask = __ballot_sync(0xffffffffu, (todo >> x) & 1u);
      while (mask) {
        const int src = __ffs(mask) - 1;
        mask &= mask - 1;
        const int m = __shfl_sync(0xffffffffu, P.row0 + m0 + k, src);
        const int nn = __shfl_sync(0xffffffffu, P.col0 + n, src);
        const double *a = P.A.base + row_off(P.A, m), *b = P.B.base + row_off(P.B, nn);
        double s = 0.0;
        for (int q = lane; q < P.A.K; q += 32) s = fma(a[q * P.A.sk], b[q * P.B.sk], s);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == src) put(mq + k, nq + HALF * y, s);
      }
    }
  }
  }
  if (!mirror) return;
  __syncthreads();
  // C(n, m): rows along n are the fast direction here
  const int c = tid % CN;
  if (tn * CN + c < P.nn)
    for (int r = tid / CN; r < 64 && tm * 64 + r < P.nm; r += 8)
      P.C[cols[c] + rows[r]] = S[r * SP + c];
}

// --------------------------------------------------------------------------
// host side
// --------------------------------------------------------------------------
int encode_planes(CUtensorMap &tm, const ModOperand &op, int boxrows) {
  auto encode = get_encode();
  if (!encode) {
    set_error("cuTensorMapEncodeTiled entry point unavailable");
    return RIMP2_ERR_UNSUPPORTED;
  }
  const cuuint64_t rows = (cuuint64_t)op.rows * op.nkc;
  cuuint64_t dims[3] = {64, rows, MG_PLANES};
  cuuint64_t strides[2] = {128, rows * 128};
  cuuint32_t box[3] = {KSTEP, (cuuint32_t)boxrows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult cr = encode(&tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, op.planes.p, dims, strides, box, estr,
                       CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                       CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (cr != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed (%d)", (int)cr);
    return RIMP2_ERR_CUDA;
  }
  return RIMP2_OK;
}

}  // namespace

size_t mod_operand_bytes(int rows, int K) {
  const size_t nkc = (K + 63) / 64;
  return (size_t)MG_PLANES * nkc * rows * 128;
}

namespace {

OpArgs op_args(ModOperand &op, const RowMap &M, int row0, bool used) {
  OpArgs P;
  P.M = M;
  P.row0 = row0;
  P.rows = op.rows;
  P.nkc = op.nkc;
  P.blocks = used ? (M.sk == 1 ? (op.rows + 7) / 8 : (op.rows + 31) / 32) : 0;
  P.e = op.e.as<int>();
  P.flag = op.flag.as<unsigned char>();
  P.out = op.planes.as<__half>();
  P.plane = (size_t)op.nkc * op.rows * 64;
  return P;
}

// Residues of rows [r0, ..) of A into Q and of columns [c0, ..) of B into L;
// either may be in place already.
int fill_operands(ModOperand &Q, const RowMap &A, int r0, bool rows, ModOperand &L, const RowMap &B,
                  int c0, bool cols, cudaStream_t s) {
  OpArgs a = op_args(Q, A, r0, rows), b = op_args(L, B, c0, cols);
  const bool one = a.nkc == 1 && a.blocks + b.blocks > 0;
  if (!one) {
    row_scale_kernel<<<(unsigned)std::max(1, a.blocks + b.blocks), 256, 0, s>>>(a, b);
    count_launch(1);
  }
  a.blocks = rows ? a.nkc * ((a.rows + 31) / 32) : 0;
  b.blocks = cols ? b.nkc * ((b.rows + 31) / 32) : 0;
  if (a.blocks + b.blocks > 0) {
    if (one)
      residue_kernel<true><<<(unsigned)(a.blocks + b.blocks), 256, 0, s>>>(a, b);
    else
      RIMP2_CK(launch_ex(false, true, residue_kernel<false>, (unsigned)(a.blocks + b.blocks), 256, 0, s, a, b));
    count_launch(1);
  }
  RIMP2_CK(cudaGetLastError());
  return RIMP2_OK;
}

}  // namespace

// Rows of a tile: least work, smaller tiles paying for their operand reads.
static int tile_rows(double m) {
  auto cost = [&](int tq, double per_row) { return std::ceil(m / tq) * tq * per_row; };
  const double c256 = cost(256, 1.0), c128 = cost(128, 1.2), c64 = cost(64, 1.6);
  return c64 < c128 && c64 < c256 ? 64 : c128 < c256 ? 128 : 256;
}

template <int TQ>
static int launch_product(const CUtensorMap &tl, const CUtensorMap &tq, const MgParams &P, cudaStream_t s) {
  RIMP2_CK(cudaFuncSetAttribute(mod_gemm_kernel<TQ>, cudaFuncAttributeMaxDynamicSharedMemorySize, mg_smem(TQ)));
  int dev = 0, nsm = 0;
  RIMP2_CK(cudaGetDevice(&dev));
  RIMP2_CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  const long long nitems = (long long)MG_PLANES * mg_tiles(P);
  const int npair = (int)std::min<long long>(nitems, nsm / 2);
  // each kernel of a contraction is set up at the end of the one before
  RIMP2_CK(launch_ex(true, true, mod_gemm_kernel<TQ>, 2 * npair, MG_THREADS, mg_smem(TQ), s, tl, tq, P));
  count_launch(1);
  return RIMP2_OK;
}

int mod_product(const ModOperand &L, const ModOperand &Q, signed char *out, long long ldm, bool lower,
                cudaStream_t s) {
  const int TQ = lower ? 256 : tile_rows(Q.rows);
  CUtensorMap tl, tq;
  RIMP2_TRY(encode_planes(tl, L, TILE));
  RIMP2_TRY(encode_planes(tq, Q, TQ / 2));
  MgParams P;
  P.rows_l = L.rows;
  P.rows_q = Q.rows;
  P.tiles_l = (L.rows + 255) / 256;
  P.tiles_q = (Q.rows + TQ - 1) / TQ;
  P.nkc = L.nkc;
  const int nseg = (P.nkc + MG_SEG - 1) / MG_SEG;  // of about equal length
  P.seg = (P.nkc + nseg - 1) / nseg;
  P.nseg = (P.nkc + P.seg - 1) / P.seg;
  P.lower = lower;
  P.out = out;
  P.ldm = ldm;
  P.err = device_error_word();
  if (TQ == 64) return launch_product<64>(tl, tq, P, s);
  if (TQ == 128) return launch_product<128>(tl, tq, P, s);
  return launch_product<256>(tl, tq, P, s);
}

namespace {

struct Dim {
  int ext;
  long long st, cst;
  int role;
};

// Up to three dimensions into a row map, the fastest one first: by the
// operand's stride where rows lie along the fast direction of memory, else by
// C's (the operand is read along K either way).
bool make_map(RowMap &M, Dim *d, int nd, const double *base, long long sk, int K) {
  nd = (int)(std::remove_if(d, d + nd, [](const Dim &x) { return x.ext == 1; }) - d);
  std::stable_sort(d, d + nd, [&](const Dim &x, const Dim &y) {
    return sk == 1 ? x.cst < y.cst : x.st < y.st;
  });
  long long rows = 1;
  for (int k = 0; k < 3; ++k) {
    M.ext[k] = k < nd ? d[k].ext : 1;
    M.st[k] = k < nd ? d[k].st : 0;
    M.cst[k] = k < nd ? d[k].cst : 0;
    M.role[k] = k < nd ? d[k].role : -1;
    rows *= M.ext[k];
  }
  M.base = base;
  M.sk = sk;
  M.K = K;
  if (rows > 2147480000LL) return false;
  M.rows = (int)rows;
  return true;
}

template <int MODE, int CN>
int launch_crt_form(const CrtParams &P, cudaStream_t s) {
  const int bytes = std::max(crt_dmma_bytes(CN), P.sym ? crt_mirror_bytes(CN) : 0);
  const dim3 grid((unsigned)((P.nm + 63) / 64), (unsigned)((P.nn + CN - 1) / CN));
  RIMP2_CK(launch_ex(false, true, crt_epilogue_kernel<MODE, CN>, grid, 8 * CN, bytes, s, P));
  count_launch(1);
  return RIMP2_OK;
}

template <int CN>
int launch_crt_mode(const CrtParams &P, int mode, cudaStream_t s) {
  if (mode == CRT_PLAIN) return launch_crt_form<CRT_PLAIN, CN>(P, s);
  if (mode == CRT_MINUS) return launch_crt_form<CRT_MINUS, CN>(P, s);
  if (mode == CRT_QUOTIENT) return launch_crt_form<CRT_QUOTIENT, CN>(P, s);
  return launch_crt_form<CRT_ANY, CN>(P, s);
}

// Columns of a block.  64 cost least where the blocks are many (3000 x 3000, sums of 370:
// 212 us a product, 222 with 16); with up to six 64 x 64 tiles an SM sixteen are as
// fast (1600 x 1600: 93 and 91), and tiles left to FP64 spread over the SMs: 1600 x 1600
// with all of them 2189 and 1901 us, 300 x 300 with sums of 1000 1208 and 427.
// Up to 48 rows have 64 columns, whose warps share the rows that there are, and
// symmetric products have whole tiles, so that C(m,n) and C(n,m) are the same bits.
int launch_crt(const CrtParams &P, int mode, cudaStream_t s) {
  int dev = 0, nsm = 0;
  RIMP2_CK(cudaGetDevice(&dev));
  RIMP2_CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  const long long tiles = ((P.nm + 63) / 64) * (long long)((P.nn + 63) / 64) / (P.lower ? 2 : 1);
  if (!P.sym && P.nm > 48 && tiles <= 6LL * nsm) return launch_crt_mode<16>(P, mode, s);
  return launch_crt_mode<64>(P, mode, s);
}

// One contraction's kernels at a time on a device: a later one, on whatever
// stream and from whatever thread, starts when the earlier one's have ended.
// Contractions on three streams at once, without this order, stopped making
// progress on the GPU, when a CTA still gave up the allocation permit of its pair before
// the other had its columns.  Whether that was all is not known; what is left
// unbounded in the kernels, that allocation and the cluster barriers, cannot wait for
// another kernel (TMEM_SMEM_MIN, tc.cuh).  So they do not run at once.  The price: a
// contraction also waits for what stands before the last one on that one's stream,
// and small ones on several streams do not overlap (eight streams, nocc 6, nvirt 53,
// NBA 187: 69 us an energy, against 89 in the FP64 kernels that did overlap).
// Held while a contraction is queued; one that fails half way, or whose end could not
// be recorded, is waited for by the host before the next may be queued.
class ModOrder {
  static std::mutex mu;
  static std::vector<cudaEvent_t> last;  // by device
  std::unique_lock<std::mutex> lk;
  cudaStream_t s;
  cudaEvent_t *ev = nullptr;
  bool open = false;

 public:
  explicit ModOrder(cudaStream_t st) : lk(mu), s(st) {}
  int begin() {
    int dev = 0;
    RIMP2_CK(cudaGetDevice(&dev));
    if ((size_t)dev >= last.size()) last.resize(dev + 1, nullptr);
    ev = &last[dev];
    if (*ev)
      RIMP2_CK(cudaStreamWaitEvent(s, *ev, 0));
    else
      RIMP2_CK(cudaEventCreateWithFlags(ev, cudaEventDisableTiming));
    open = true;
    return RIMP2_OK;
  }
  int end() {
    if (inject_fault("record")) {
      set_error("injected event failure (RIMP2_FAULT_INJECT=record)");
      return RIMP2_ERR_CUDA;
    }
    RIMP2_CK(cudaEventRecord(*ev, s));
    open = false;
    return RIMP2_OK;
  }
  ~ModOrder() {
    if (open) cudaStreamSynchronize(s);
  }
};
std::mutex ModOrder::mu;
std::vector<cudaEvent_t> ModOrder::last;

constexpr size_t MG_PLANE_CAP = (size_t)6 << 30;  // bytes of one operand's planes per part
constexpr size_t MG_RES_CAP = (size_t)4 << 30;    // bytes of the residues of a part of C

// Most rows of an operand in a part, and most columns of a part whose rows take ldm
// bytes.  RIMP2_RESIDUE_PARTS=rows,columns: smaller ones, to reach parts in tests.
void part_caps(int K, long long *rows, long long ldm, long long *cols) {
  *rows = std::max<long long>(256, (long long)(MG_PLANE_CAP / mod_operand_bytes(1, K)) / 256 * 256);
  *cols = std::max<long long>(256, (long long)(MG_RES_CAP / (MG_PLANES * ldm)) / 256 * 256);
  *cols = std::min(*cols, *rows);
  const char *e = getenv("RIMP2_RESIDUE_PARTS");
  int r = 0, c = 0;
  if (e && sscanf(e, "%d,%d", &r, &c) == 2 && r >= 64 && c >= 64) {
    *rows = std::min<long long>(*rows, r);
    *cols = std::min<long long>(*cols, c);
  }
}

}  // namespace

bool fold_gemm(const GemmDesc &g, RowMap &A, RowMap &B) {
  Dim da[3] = {{g.M, g.sAm, g.sCm, 0}}, db[3] = {{g.N, g.sBn, g.sCn, 0}};
  int na = 1, nb = 1;
  const int ext[2] = {g.nb0, g.nb1};
  const long long sa[2] = {g.sAb0, g.sAb1}, sb[2] = {g.sBb0, g.sBb1}, sc[2] = {g.sCb0, g.sCb1};
  for (int k = 0; k < 2; ++k) {
    // with denominators the first batch index is the row's i, the second the column's j
    const bool row = g.denom ? k == 0 : sb[k] == 0;
    if (ext[k] > 1 && (row ? sb[k] : sa[k]) != 0) return false;
    if (row)
      da[na++] = {ext[k], sa[k], sc[k], 1};
    else
      db[nb++] = {ext[k], sb[k], sc[k], 1};
  }
  return make_map(A, da, na, g.A, g.sAk, g.K) && make_map(B, db, nb, g.B, g.sBk, g.K);
}

int mod_gemm(const GemmDesc &g, const RowMap &A0, const RowMap &B0, cudaStream_t s, bool *handled) {
  *handled = false;
  // few columns: transposed, so that they are the tile's narrow side
  const bool swap = !g.lower && !g.denom && B0.rows <= 128 && A0.rows > B0.rows;
  const RowMap &A = swap ? B0 : A0, &B = swap ? A0 : B0;
  if (g.K < MG_K_MIN || g.K > MG_K_MAX || g.alpha == 0.0) return RIMP2_OK;
  // a captured call keeps to the FP64 kernel: the order between contractions
  // (ModOrder) cannot reach into a graph
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
    (void)cudaGetLastError();
    return RIMP2_OK;
  }
  // parts: bounded workspaces, whatever the product's size
  long long cap_rows, cap_cols;
  part_caps(g.K, &cap_rows, 256, &cap_cols);
  const int ra = (int)std::min<long long>(A.rows, cap_rows);
  const long long ldm = ((long long)ra + 255) / 256 * 256;
  part_caps(g.K, &cap_rows, ldm, &cap_cols);
  const int rb = (int)std::min<long long>(B.rows, cap_cols);
  if (g.lower && (ra < A.rows || rb < B.rows)) return RIMP2_OK;
  if ((rb + 63) / 64 > 65535) return RIMP2_OK;
  ModOperand Q, L;
  Q.rows = ra;
  L.rows = rb;
  Q.nkc = L.nkc = (g.K + 63) / 64;
  // a product of one set of vectors with itself needs their residues once
  const bool same = ra == A.rows && rb == B.rows && A.rows == B.rows && A.base == B.base && A.sk == B.sk &&
                    memcmp(A.ext, B.ext, sizeof A.ext) == 0 && memcmp(A.st, B.st, sizeof A.st) == 0;
  DevBuf arena, res;
  {
    DevBuf *const buf[] = {&Q.planes, &L.planes, &res, &Q.e, &L.e, &Q.flag, &L.flag};
    const size_t bytes[] = {mod_operand_bytes(ra, g.K),
                            same ? 0 : mod_operand_bytes(rb, g.K),
                            (size_t)MG_PLANES * rb * ldm,
                            sizeof(int) * (size_t)ra,
                            sizeof(int) * (size_t)rb,
                            (size_t)ra,
                            (size_t)rb};
    if (alloc_parts(arena, buf, bytes, s) != RIMP2_OK) {
      (void)cudaGetLastError();  // no room: the FP64 kernel needs none
      clear_error();
      return RIMP2_OK;
    }
  }
  if (same) {
    L.planes.alias(Q.planes.p, Q.planes.n, s);
    L.e.alias(Q.e.p, Q.e.n, s);
    L.flag.alias(Q.flag.p, Q.flag.n, s);
  }
  ModOrder order(s);
  RIMP2_TRY(order.begin());
  CrtParams P;
  memset(&P, 0, sizeof P);
  P.A = A;
  P.B = B;
  P.res = res.as<signed char>();
  P.C = g.C;
  P.alpha = g.alpha;
  P.beta = g.beta;
  P.eo = g.eo;
  P.ev = g.ev;
  P.denom = g.denom;
  P.lower = g.lower;
  P.nfast = B.cst[0] < A.cst[0];
  P.sym = same && !g.lower && g.beta == 0.0 && A.rows > 256 && memcmp(A.role, B.role, sizeof A.role) == 0;
  const bool plain = g.alpha == 1.0 && g.beta == 0.0;
  const int mode = plain ? (g.denom ? CRT_QUOTIENT : CRT_PLAIN)
                   : !g.denom && g.alpha == -1.0 && g.beta == 1.0 ? CRT_MINUS : CRT_ANY;
  P.ea = Q.e.as<int>();
  P.fa = Q.flag.as<unsigned char>();
  P.eb = L.e.as<int>();
  P.fb = L.flag.as<unsigned char>();
  for (int r0 = 0; r0 < A.rows; r0 += ra) {
    Q.rows = std::min(ra, A.rows - r0);
    for (int c0 = 0; c0 < B.rows; c0 += rb) {
      const int nc = std::min(rb, B.rows - c0);
      const bool cols = !same && (r0 == 0 || rb < B.rows);
      if (cols || same) L.rows = nc;
      RIMP2_TRY(fill_operands(Q, A, r0, c0 == 0, L, B, c0, cols, s));
      P.row0 = r0;
      P.col0 = c0;
      P.nm = Q.rows;
      P.nn = nc;
      P.ldm = ((long long)Q.rows + 255) / 256 * 256;
      RIMP2_TRY(mod_product(L, Q, res.as<signed char>(), P.ldm, g.lower || P.sym, s));
      RIMP2_TRY(launch_crt(P, mode, s));
      RIMP2_CK(cudaGetLastError());
    }
  }
  RIMP2_TRY(order.end());
  if (inject_fault("wait")) report_device_error(24);
  *handled = true;
  return RIMP2_OK;
}

// Estimated time of the residue form: launches and latencies, the residues of
// both operands, the products, the reconstruction.
double mod_gemm_time(double m, double n, double k, bool lower) {
  auto up = [](double x, double t) { return std::ceil(x / t) * t; };
  if (!lower && n <= 128 && m > n) std::swap(m, n);
  const double kp = up(k, 64), part = lower ? 0.55 : 1.0, tq = lower ? 256 : tile_rows(m);
  const double rate = tq == 256 ? 1.3e15 : tq == 128 ? 1.3e15 / 1.2 : 1.3e15 / 1.6;
  return 20e-6 + (m + n) * kp * 10e-12 +
         part * (m * n * 14e-12 + 17.0 * 2.0 * up(m, tq) * up(n, 256) * (kp + 64) / rate);
}

// Rows and columns of a square product that runs as one part.
int mod_gemm_block(int K) {
  long long rows, cols;
  part_caps(K, &rows, (long long)std::sqrt((double)(MG_RES_CAP / MG_PLANES)) / 256 * 256, &cols);
  return (int)std::min(rows, cols);
}

}  // namespace rimp2
