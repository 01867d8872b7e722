// split_kernels.cu -- split-precision RI-MP2 energy on the tcgen05 tensor cores.
//
// Numerics (Ozaki-style integer slices carried in FP16):
//   For every column c=(a,i) of Calpha(:,a,i) a power-of-two scale s_c is
//   chosen so that |C*s_c| <= 2047.5 and ||round(C*s_c)||_2 <= 2^12.  Then
//     C*s_c = S0 + R1 (+ R2)
//   with S0 = round(C*s_c) an integer in [-2048,2048] (exact in FP16) and R1, R2
//   the FP16-rounded residuals.  The alpha contraction of two columns is
//     g*s_a*s_b = sum S0a S0b  +  sum (S0a R1b + R1a S0b + R1a R1b [+ S0a R2b + R2a S0b])
//   The first sum (accumulator L0) is a sum of integers whose every partial
//   sum is bounded by ||S0a|| ||S0b|| <= 2^24 (Cauchy-Schwarz), so the FP32
//   tensor-core accumulation is EXACT whatever its internal rounding mode.
//   The correction terms (accumulator L1) are ~2^-8 of g and uncorrelated
//   with it, so their FP32 rounding does not bias the energy.
//   The epilogue forms g in FP32, the denominator from hi/lo float pairs of
//   the FP64 orbital energies, and accumulates e_ij in FP32 per thread and
//   FP64 across threads; pair and total energies are reduced in FP64 with
//   compensation.
//
// Kernel layout (one persistent CTA per SM, 576 threads):
//   warp 0       TMA producer (128x64 FP16 boxes, 128B swizzle) and the
//                device-side work queue (atomic counter, 4-deep item ring)
//   warp 1       TMEM owner + single-thread tcgen05.mma issuer
//   warps 2..17  epilogue, four warps per TMEM lane quadrant (32 accumulator
//                columns each): tcgen05.ld, denominators, energy terms
//   Work item = (fragment, pair i<=j, tile pair A<=B): T1 = G_ij[A,B] =
//   C_iA^T C_jB and T2 = G_ji[A,B] = C_jA^T C_iB, each with L0/L1
//   accumulators in TMEM (4 x 128 columns = all 512).  The exchange integral
//   g_ij(b,a) = T2[a,b] therefore lives in the same TMEM lane/column as
//   g_ij(a,b) = T1[a,b], and no four-index quantity is ever written to
//   memory.  T1 is read out and released first, so the next item's T1 MMAs
//   overlap this item's T2 phase; diagonal tile pairs take T2 = T1^T through
//   shared memory.
// A one-residual-slice fragment with enough occupied orbitals and a long
// enough auxiliary space (the measured kernel table of capi.cu) runs instead
// on split_pair_kernel: clusters of two CTAs issuing cta_group::2 MMAs over
// two occupied pairs that share their B operand, with a third slice plane
// V = fp16(C*s) that folds R1a S0b + R1a R1b into R1a V (three products per
// element pair, a per-column correction removing the same-column bias).
// Every wait on an mbarrier is bounded by a clock budget; on expiry the
// kernel records an error code, drains its own copies and MMAs, frees TMEM
// and returns, and the host reports RIMP2_ERR_TIMEOUT.
#include <cuda_fp16.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <vector>

#include "tc.cuh"

namespace rimp2 {

void count_launch(int n);
void note_split_kernel(int k);  // 1 one-CTA, 2 paired-CTA
__global__ void pair_reduce_kernel(const double *__restrict__ part, int nper, const int *pairs,
                                   int npairs, int nocc, double *Epair);
__global__ void total_reduce_kernel(const double *Epair, int nocc, double *Etot);
__global__ void make_pairs_kernel(int nocc, int *pairs);

namespace {

constexpr int NTHREADS = 320;  // producer warp, MMA warp, 8 epilogue warps
// split_batch_kernel: producer warp, MMA warp and 16 epilogue warps (four per
// TMEM lane quadrant, 32 accumulator columns each; the launch bounds give
// them 96 registers).  On short auxiliary spaces a work item is bounded by
// its epilogue and hand-offs, not by its MMAs; 16 warps instead of 8 took
// 5-7% off such items (nocc=64 nvirt=512 NBA=256) and left long ones as
// they were.
constexpr int BATCH_EPI = 16;
constexpr int BATCH_THREADS = 64 + 32 * BATCH_EPI;

// OR of a predicate over the 256 epilogue threads (named barrier 1).  The
// epilogue warps leave their loop together on a failed bounded wait, so that
// none is left waiting at a later named barrier for a warp that has gone.
__device__ __forceinline__ bool epi_any(bool p) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred q, o;\n\t"
      "setp.ne.u32 q, %1, 0;\n\t"
      "bar.red.or.pred o, 1, 256, q;\n\t"
      "selp.u32 %0, 1, 0, o;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)p)
      : "memory");
  return r != 0;
}

// the same over the 512 epilogue threads of split_batch_kernel
__device__ __forceinline__ bool epi_any512(bool p) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred q, o;\n\t"
      "setp.ne.u32 q, %1, 0;\n\t"
      "bar.red.or.pred o, 1, 512, q;\n\t"
      "selp.u32 %0, 1, 0, o;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)p)
      : "memory");
  return r != 0;
}

// Reciprocal of an energy denominator (never zero or subnormal here): the
// hardware approximation (PTX rcp.approx.ftz.f32, about one ulp) refined by
// one Newton-Raphson step r' = r + r (1 - d r), whose residual 1 - d r is
// exact in one FMA; the result is within about half an ulp, so a fragment
// whose denominators are all equal does not accumulate a one-sided error.
__device__ __forceinline__ float rcp_denom(float d) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  const float e = fmaf(-d, r, 1.0f);
  return fmaf(r, e, r);
}

__device__ __forceinline__ void decode_tri(int q, int &A, int &B) {
  int b = (int)((sqrtf(8.0f * q + 1.0f) - 1.0f) * 0.5f);
  while ((b + 1) * (b + 2) / 2 <= q) ++b;
  while (b * (b + 1) / 2 > q) --b;
  B = b;
  A = q - b * (b + 1) / 2;
}

// --------------------------------------------------------------------------
// slicing kernel: Calpha (FP64) -> FP16 slices + per-column inverse scales
// --------------------------------------------------------------------------
// slices layout: [slice][col][Kpad] FP16, col = a + nvpad*i (padded columns
// and padded K are zero); inv_scale[col] = 2^-e.
//
// GB300 runs FP64 arithmetic at a small fraction of its FP32 rate, so the
// per-element work here avoids the FP64 pipe: the scaled value's integer
// part and remainder come from the mantissa bits by integer arithmetic
// (split_int below), the remainder is then rounded to FP16 slices in FP32.
// Only the per-column scale choice uses FP64, in one thread per column.
// One fragment of a batch: sizes, where its data lives, where its slices,
// scales, work items and pair energies go.
struct FragDesc {
  int nocc, nvirt, nvpad, NBA;
  int nks;              // K chunks of 64
  int ntp;              // tile pairs A<=B
  int ncol;             // nocc * nvpad
  int eo_off, ev_off;   // into eo2 / ev2
  int pair_base;        // first global pair index
  long long row_base;   // first 64-wide slice row (per slice plane)
  long long col_base;   // first inverse-scale index
  long long item_base;  // first work item
  long long pitem_base; // first pair item (paired-CTA kernel)
  const double *Ca, *eo, *ev;
  double *Epair, *Etot;
};

__device__ __forceinline__ int find_frag_item(const FragDesc *fr, int nfrag, long long x) {
  int lo = 0, hi = nfrag - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (fr[mid].item_base <= x)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ void decode_pair(int p, int &i, int &j) {
  int jj = (int)((sqrtf(8.0f * p + 1.0f) - 1.0f) * 0.5f);
  while ((jj + 1) * (jj + 2) / 2 <= p) ++jj;
  while (jj * (jj + 1) / 2 > p) --jj;
  j = jj;
  i = p - jj * (jj + 1) / 2;
}

// Per-element arithmetic of the slicing kernels in 32/64-bit integer
// operations on the FP64 bit pattern: GB300's FP64 pipe is far too slow for
// per-element work, and assembling floats with ldexpf costs several times
// more instructions (the slicing kernels are issue-bound, ncu).
//
// |v| truncated to float (mantissa cut to 24 bits), for a column's sum of
// squares: the exponent is rebiased in place; values below the float range
// count as 0, values above it as FLT_MAX.
__device__ __forceinline__ float abs_trunc_f32(unsigned long long mag) {
  const unsigned int ed = (unsigned int)(mag >> 52);
  if (ed < 897u) return 0.0f;
  if (ed > 1150u) return 3.4028234663852886e38f;
  return __uint_as_float((unsigned int)((mag >> 29) - (896ull << 23)));
}

// float -> double by moving bits (GB300 runs the F2F conversion on its slow
// FP64 pipe): normal floats and zero; a subnormal float becomes zero.
__device__ __forceinline__ double f2d_bits(float f) {
  const uint32_t u = __float_as_uint(f);
  const uint32_t ex = (u >> 23) & 0xFFu;
  const uint32_t hi = (u & 0x80000000u) | ((ex + 896u) << 20) | ((u >> 3) & 0xFFFFFu);
  const uint32_t lo = u << 29;
  return ex == 0 ? 0.0 : __hiloint2double((int)hi, (int)lo);
}

// v * p for p = 2^k (a normal float) by adding k to v's exponent field:
// exact; zero stays zero, a result below the normal range becomes zero.
__device__ __forceinline__ double scale_pow2(double v, float p) {
  const int k = (int)((__float_as_uint(p) >> 23) & 0xFFu) - 127;
  const long long bits = __double_as_longlong(v);
  const int ev = (int)((bits >> 52) & 0x7FF);
  if (ev == 0) return v;
  if (ev + k <= 0) return 0.0;
  return __longlong_as_double(bits + ((long long)k << 52));
}

// Split of a double x with |x 2^e| < 2^22 into q (an integer, rounded half to
// even; |q| <= 512 for the AO chunks, <= 2048 for Calpha columns) and r ~ x 2^e - q in FP32 arithmetic only (GB300's
// FP64 pipe is a small fraction of the FP32 one): v = |x| 2^e is the float
// f_hi holding the top 24 significant bits of x (exponent and fraction bits
// moved into place, no rounding) plus f_lo holding the next 23 bits (a 23-bit
// integer formed with the 2^23 magic constant, times a power of two);
// q = round(f_hi) with the 1.5 * 2^23 constant, r = (f_hi - q) + f_lo, where
// f_hi - q is exact and the sum rounds once (2^-25 of |r|).  Values below
// 2^-40 of the scaled unit, zeros and subnormals give q = r = 0.  The sign
// of x goes onto both.  Equal to split_int's results to within its rounding
// of r; tests/test_split_numerics_cpu.py restates these float operations and
// checks them against exact rational arithmetic.
__device__ __forceinline__ void split_f32(double x, int e, float &q, float &r) {
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
  const uint32_t sgn = hi & 0x80000000u;
  const int ed = (int)((hi >> 20) & 0x7FFu);
  const int E = ed - 1023 + e;  // |x| 2^e = 1.f 2^E
  const bool live = ed != 0 && E >= -40;
  const int Ec = live ? E : 0;
  const uint32_t frac23 = (__funnelshift_l(lo, hi, 3)) & 0x7FFFFFu;
  const float fhi = __uint_as_float(((uint32_t)(Ec + 127) << 23) | frac23);
  const float lo23 = __uint_as_float(0x4B000000u | ((lo >> 6) & 0x7FFFFFu)) - 8388608.0f;
  const float flo = lo23 * __uint_as_float((uint32_t)(Ec - 46 + 127) << 23);
  const float qm = (fhi + 12582912.0f) - 12582912.0f;
  const float rm = (fhi - qm) + flo;
  q = live ? __uint_as_float(__float_as_uint(qm) | sgn) : 0.0f;
  r = live ? __uint_as_float(__float_as_uint(rm) ^ sgn) : 0.0f;
}

// x = |v| 2^e split into q = rint(x) (round half to even; |q| <= 2048 by the
// choice of e) and the remainder r = x - q, from A = floor(x 2^32): the
// integer part and the 32 bits below it of the 53-bit mantissa.  r is exact
// to 2^-31 absolute, far below what the FP16 residual slices keep (R1 rounds
// r to 11 bits, R2 the rest to 11 more, ~2^-24 absolute).  The sign of v is
// applied to both.
__device__ __forceinline__ void split_int(unsigned long long b, int e, float &q, float &r) {
  const unsigned long long mag = b & 0x7FFFFFFFFFFFFFFFull;
  const int ed = (int)(mag >> 52);
  const int sh = 1075 - 32 - ed - e;  // A = M >> sh, M the mantissa with its leading 1
  unsigned long long A = 0;
  if (ed != 0 && sh < 64) {
    const unsigned long long M = (mag & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
    A = sh >= 0 ? (M >> sh) : (M << (-sh));
  }
  const unsigned long long qi = (A + 0x7FFFFFFFull + ((A >> 32) & 1ull)) >> 32;
  const long long fr = (long long)A - (long long)(qi << 32);  // in [-2^31, 2^31]
  float qf = (float)(unsigned int)qi;
  float rf = (float)(int)(fr >> 1) * 4.656612873077393e-10f;  // 2^-31
  if (b >> 63) {
    qf = -qf;
    rf = -rf;
  }
  q = qf;
  r = rf;
}

// Power-of-two scale exponent of a column from its largest magnitude (bits)
// and its FP32 sum of squares: |C 2^e| <= 2047.5 and ||C 2^e||_2 below 2^12
// with room for the rounding of NBA values.  Integer and FP32 arithmetic only
// (GB300's FP64 pipe is a small fraction of its FP32 rate, and the FP64
// sqrt/div/log2 of this choice, once per column, bounded the slicing
// kernels): with max |C| = m 2^E (m in [1, 2)), 2047.5 / m lies in
// (1023.75, 2047.5], so the magnitude bound allows e = 10 - E when m <=
// 2047.5 / 1024 = 2 - 2^-11 (fraction bits <= 0xFFE00 << 32) and 9 - E
// otherwise; the norm bound takes the binary exponent of the FP32 ratio,
// correctly rounded operations with a 2^-20 margin (float
// truncation of the squares underestimates ||C||^2 by < 2^-21 relative; the
// caller's exact integer check of ||S0||^2 keeps the exactness either way).
// Clamped to [-100, 100]; 0 for an all-zero column.
__device__ __forceinline__ int col_scale_exponent(unsigned long long mxb, float ss, int NBA) {
  if (mxb == 0) return 0;
  const int ed = (int)(mxb >> 52);
  if (ed == 0) return 100;  // largest value subnormal
  const int e1 = ((mxb & 0xFFFFFFFFFFFFFull) <= (0xFFE00ull << 32) ? 10 : 9) - (ed - 1023);
  int e2 = 127;
  if (ss > 0.0f) {
    const float r = (4096.0f - 0.5f * sqrtf((float)NBA)) / sqrtf(ss) * 0.99999905f;
    e2 = (int)((__float_as_uint(r) >> 23) & 0xFFu) - 127;  // floor(log2 r) for r normal
  }
  return max(-100, min(100, min(e1, e2)));
}

// Slices of every fragment: slice plane s, fragment f, K chunk kc, column c
// live at row (row_base_f + kc*ncol_f + c) of 64 FP16, i.e. one 2D-boxable
// K-chunk-major layout shared by all fragments (one tensor map per batch).
// grid.y = fragment, one warp per column.  At most 40 registers a thread, so
// that a 256-thread block fits in the registers a persistent energy kernel
// leaves free on its SM: in a batch graph the next group's slicing runs
// beside the current group's energy kernel.  (A single-pass form holding the
// column in registers was measured slower: a 12 KB column took ~40 KB of
// register file, leaving too few columns in flight per SM.)
__device__ __forceinline__ void slice_column(const FragDesc &F, int col, int nsl, long long plane,
                                             __half *__restrict__ slices,
                                             float *__restrict__ inv_scale, int vplane,
                                             float *__restrict__ dcorr) {
  const int lane = threadIdx.x & 31;
  const int a = col % F.nvpad, i = col / F.nvpad;
  const int Kpad = F.nks * 64;
  const __half hz = __float2half_rn(0.0f);
  __half *out = slices + (size_t)(F.row_base + col) * 64;
  const size_t kstride = (size_t)F.ncol * 64;  // next K chunk of the same column
  if (a >= F.nvirt) {
    for (int k0 = 4 * lane; k0 < Kpad; k0 += 128) {
      const size_t o = (size_t)(k0 >> 6) * kstride + (k0 & 63);
      for (int sl = 0; sl < nsl + vplane; ++sl)
        *reinterpret_cast<uint2 *>(out + sl * plane + o) = make_uint2(0u, 0u);
    }
    if (lane == 0) {
      inv_scale[F.col_base + col] = 1.0f;
      if (vplane) dcorr[F.col_base + col] = 0.0f;
    }
    return;
  }
  const int NBA = F.NBA;
  const double *c = F.Ca + ((size_t)i * F.nvirt + a) * NBA;
  unsigned long long mxb = 0;
  float ss = 0.0f;
  // four independent loads in flight per lane (the pass is latency-bound)
  for (int k0 = lane; k0 < NBA; k0 += 128) {
    double v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = (k0 + 32 * u < NBA) ? c[k0 + 32 * u] : 0.0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const unsigned long long mag =
          (unsigned long long)__double_as_longlong(v[u]) & 0x7FFFFFFFFFFFFFFFull;
      mxb = mag > mxb ? mag : mxb;
      const float f = abs_trunc_f32(mag);
      ss = fmaf(f, f, ss);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long other = __shfl_xor_sync(0xffffffffu, mxb, o);
    mxb = other > mxb ? other : mxb;
    ss += __shfl_xor_sync(0xffffffffu, ss, o);
  }
  int e = lane == 0 ? col_scale_exponent(mxb, ss, NBA) : 0;
  e = __shfl_sync(0xffffffffu, e, 0);
  if (vplane && lane == 0) dcorr[F.col_base + col] = 0.0f;
  for (int attempt = 0; attempt < 64; ++attempt) {
    long long n2 = 0;  // sum of S0^2 (integers; <= 2^24 is the test)
    float dsum = 0.0f;  // sum of R1 (V - S0 - R1) (V plane only)
    // four consecutive K values per lane (one 8-byte store per plane; a
    // 64-wide K chunk holds 16 lanes' groups); values beyond NBA are zeros
    for (int k0 = 4 * lane; k0 < Kpad; k0 += 128) {
      double v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = (k0 + u < NBA) ? c[k0 + u] : 0.0;
      __align__(8) __half h0[4], h1[4], h2[4], hv[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        float q, r;
        split_f32(v[u], e, q, r);  // zeros give q = r = 0
        h0[u] = __float2half_rn(q);  // integer |q| <= 2048: exact in FP16
        h1[u] = __float2half_rn(r);
        h2[u] = __float2half_rn(r - __half2float(h1[u]));
        // |q| < 2^23: its integer value from the 2^23 magic constant
        const int qi = __float_as_int(fabsf(q) + 8388608.0f) - 0x4B000000;
        n2 += qi * qi;  // |q| <= 2048: q^2 fits an int
        if (vplane) {
          // V = C*s in FP16; its rounding error against S0 + R1 is exact in FP32
          hv[u] = __float2half_rn(q + r);
          const float r1 = __half2float(h1[u]);
          dsum = fmaf(r1, (__half2float(hv[u]) - q) - r1, dsum);
        }
      }
      const size_t o = (size_t)(k0 >> 6) * kstride + (k0 & 63);
      *reinterpret_cast<uint2 *>(out + o) = *reinterpret_cast<const uint2 *>(h0);
      if (nsl > 1) *reinterpret_cast<uint2 *>(out + plane + o) = *reinterpret_cast<const uint2 *>(h1);
      if (nsl > 2)
        *reinterpret_cast<uint2 *>(out + 2 * plane + o) = *reinterpret_cast<const uint2 *>(h2);
      if (vplane)
        *reinterpret_cast<uint2 *>(out + nsl * plane + o) = *reinterpret_cast<const uint2 *>(hv);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n2 += __shfl_xor_sync(0xffffffffu, n2, o);
    if (n2 <= 16777216LL) {  // ||S0||^2 <= 2^24: L0 accumulation exact
      if (vplane) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) dsum += __shfl_xor_sync(0xffffffffu, dsum, o);
        if (lane == 0) dcorr[F.col_base + col] = dsum;
      }
      break;
    }
    --e;
  }
  if (lane == 0) inv_scale[F.col_base + col] = ldexpf(1.0f, -e);
}

__global__ void __launch_bounds__(256, 6)
    slice_batch_kernel(const FragDesc *__restrict__ fr, int nsl, long long plane,
                                   __half *__restrict__ slices, float *__restrict__ inv_scale,
                                   int col0, int col1, int vplane = 0,
                                   float *__restrict__ dcorr = nullptr) {
  // columns [col0, min(col1, ncol)) of each fragment
  const FragDesc &F = fr[blockIdx.y];
  const int col = col0 + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (col >= F.ncol || col >= col1) return;
  slice_column(F, col, nsl, plane, slices, inv_scale, vplane, dcorr);
}

// The columns of one set, its descriptor a kernel parameter (a captured call may be
// replayed when the host's copy is gone).
__global__ void __launch_bounds__(256, 6)
    slice_one_kernel(const __grid_constant__ FragDesc F, int nsl, long long plane,
                     __half *__restrict__ slices, float *__restrict__ inv_scale) {
  const int col = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (col < F.ncol) slice_column(F, col, nsl, plane, slices, inv_scale, 0, nullptr);
}

// orbital energies as hi/lo float pairs (padded virtuals get a large value so
// their denominators stay finite; their g is exactly zero). grid.y = fragment
__device__ __forceinline__ void eps_entry(const FragDesc &F, int t, float2 *eo2, float2 *ev2) {
  if (t < F.nocc) {
    const double v = F.eo[t];
    const float h = (float)v;
    eo2[F.eo_off + t] = make_float2(h, (float)(v - (double)h));
  }
  if (t < F.nvpad) {
    const double v = t < F.nvirt ? F.ev[t] : 1000.0;
    const float h = (float)v;
    ev2[F.ev_off + t] = make_float2(h, (float)(v - (double)h));
  }
}

__global__ void eps_batch_kernel(const FragDesc *__restrict__ fr, float2 *eo2, float2 *ev2) {
  eps_entry(fr[blockIdx.y], blockIdx.x * blockDim.x + threadIdx.x, eo2, ev2);
}

// Work items in queue order: fragments are enumerated heaviest first (the
// host orders the descriptors by K length), pairs j-major, tile pairs
// B-major.  item = {fragment, i | j<<16, tA | tB<<16, item id}.
// Work item t of fragment f.
__device__ __forceinline__ int4 work_item(const FragDesc &F, int f, long long t) {
  const long long loc = t - F.item_base;
  const int p = (int)(loc / F.ntp), q = (int)(loc % F.ntp);
  int i, j, tA, tB;
  decode_pair(p, i, j);
  decode_tri(q, tA, tB);
  return make_int4(f, i | (j << 16), tA | (tB << 16), (int)t);
}

__global__ void build_items_kernel(const FragDesc *__restrict__ fr, int nfrag, long long nitems,
                                   int4 *__restrict__ items) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= nitems) return;
  const int f = find_frag_item(fr, nfrag, t);
  items[t] = work_item(fr[f], f, t);
}

struct BatchParams {
  const FragDesc *frags;
  const int4 *items;
  long long nitems;       // this launch drains items [item_begin, nitems)
  long long item_begin;
  unsigned int *queue;     // next item counter (reset per launch)
  const float2 *eo2, *ev2;
  const float *inv_scale;
  double *part;            // [nitems]
  int *err;
};

constexpr int IQ = 4;  // item ring depth between the producer and the consumers
constexpr int TP = TILE + 1;  // padded row of the diagonal-tile transpose buffer (floats)

template <int NSL, int NSTAGE>
__global__ void __launch_bounds__(BATCH_THREADS, 1)
    split_batch_kernel(const __grid_constant__ CUtensorMap tmap, BatchParams P) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *base = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  constexpr int STAGE_BYTES = NSL * 2 * PANEL_BYTES;
  constexpr int NEPI = BATCH_EPI;  // epilogue warps: four per TMEM lane quadrant
  uint8_t *stages = base;
  uint64_t *bars = (uint64_t *)(base + NSTAGE * STAGE_BYTES);
  // bars: full[NSTAGE], empty[NSTAGE], t1full, t1empty, t2full, t2empty, drain,
  //       item_full[IQ], item_empty[IQ]
  constexpr int NB = 2 * NSTAGE + 5 + 2 * IQ;
  uint32_t *tmem_slot = (uint32_t *)(bars + NB);
  volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
  volatile int *item_q = (volatile int *)(tmem_slot + 2);  // [IQ]
  double *redd = (double *)(((uintptr_t)(tmem_slot + 2 + IQ) + 7) & ~(uintptr_t)7);  // [NEPI]
  // transpose buffer for diagonal tile pairs: 64 rows of T1, padded rows
  float *tbuf = (float *)(base + NSTAGE * STAGE_BYTES + 512);  // [64][TP]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t full0 = smem_u32(&bars[0]);
  const uint32_t empty0 = smem_u32(&bars[NSTAGE]);
  const uint32_t t1full = smem_u32(&bars[2 * NSTAGE]);
  const uint32_t t1empty = smem_u32(&bars[2 * NSTAGE + 1]);
  const uint32_t t2full = smem_u32(&bars[2 * NSTAGE + 2]);
  const uint32_t t2empty = smem_u32(&bars[2 * NSTAGE + 3]);
  const uint32_t drain = smem_u32(&bars[2 * NSTAGE + 4]);
  const uint32_t ifull0 = smem_u32(&bars[2 * NSTAGE + 5]);
  const uint32_t iempty0 = smem_u32(&bars[2 * NSTAGE + 5 + IQ]);

  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTAGE; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    mbar_init(t1full, 1);
    mbar_init(t1empty, NEPI);
    mbar_init(t2full, 1);
    mbar_init(t2empty, NEPI);
    mbar_init(drain, 1);
    for (int s = 0; s < IQ; ++s) {
      mbar_init(ifull0 + 8 * s, 1);
      mbar_init(iempty0 + 8 * s, 1 + NEPI);  // MMA issuer + epilogue warps
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&tmap) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                     smem_u32(tmem_slot))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  grid_wait();

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      int stage = 0, islot = 0;
      uint32_t phase = 0, iphase = 0;
      int armed[NSTAGE];
      for (int s = 0; s < NSTAGE; ++s) armed[s] = -1;
      bool ok = true;
      while (ok) {
        if (!mbar_wait(iempty0 + 8 * islot, iphase ^ 1, abort_flag, P.err, 5)) break;
        const long long id = P.item_begin + (long long)atomicAdd(P.queue, 1u);
        const int qidx = id < P.nitems ? (int)id : -1;
        item_q[islot] = qidx;
        mbar_arrive(ifull0 + 8 * islot);
        if (++islot == IQ) {
          islot = 0;
          iphase ^= 1;
        }
        if (qidx < 0) break;
        const int4 it = P.items[qidx];
        const FragDesc &F = P.frags[it.x];
        const int i = it.y & 0xFFFF, j = it.y >> 16, tA = it.z & 0xFFFF, tB = it.z >> 16;
        // T2 = T1 for i == j, and T2 = T1^T (shared-memory transpose) for A == B
        const int ntiles = (i == j || tA == tB) ? 1 : 2;
        for (int t = 0; t < ntiles && ok; ++t) {
          const int colA = (t == 0 ? i : j) * F.nvpad + tA * TILE;
          const int colB = (t == 0 ? j : i) * F.nvpad + tB * TILE;
          for (int kc = 0; kc < F.nks; ++kc) {
            if (!mbar_wait(empty0 + 8 * stage, phase ^ 1, abort_flag, P.err, 1)) {
              ok = false;
              break;
            }
            const uint32_t fb = full0 + 8 * stage;
            mbar_expect_tx(fb, STAGE_BYTES);
            armed[stage] = (int)phase;
            const uint32_t dst = smem_u32(stages + stage * STAGE_BYTES);
            const int rowk = (int)(F.row_base + (long long)kc * F.ncol);
#pragma unroll
            for (int sl = 0; sl < NSL; ++sl) {  // A panels, then the B panels back to back
              tma_load_3d(dst + sl * PANEL_BYTES, &tmap, fb, 0, rowk + colA, sl);
              tma_load_3d(dst + (NSL + sl) * PANEL_BYTES, &tmap, fb, 0, rowk + colB, sl);
            }
            if (++stage == NSTAGE) {
              stage = 0;
              phase ^= 1;
            }
          }
        }
      }
      if (!ok || *abort_flag) {  // drain copies in flight before the CTA can exit
        for (int s = 0; s < NSTAGE; ++s) {
          if (armed[s] < 0) continue;
          const long long t0 = clock64();
          while (!mbar_test(full0 + 8 * s, (uint32_t)armed[s]) && clock64() - t0 < WAIT_BUDGET) {
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer --------------------------------
    if (lane == 0) {
      int stage = 0, islot = 0;
      uint32_t phase = 0, iphase = 0;
      bool ok = true;
      long long nloc = 0;
      while (ok) {
        if (!mbar_wait(ifull0 + 8 * islot, iphase, abort_flag, P.err, 6)) break;
        const int qidx = item_q[islot];
        mbar_arrive(iempty0 + 8 * islot);
        if (++islot == IQ) {
          islot = 0;
          iphase ^= 1;
        }
        if (qidx < 0) break;
        const int4 it = P.items[qidx];
        const int nks = P.frags[it.x].nks;
        const int i = it.y & 0xFFFF, j = it.y >> 16, tA = it.z & 0xFFFF, tB = it.z >> 16;
        const int ntiles = (i == j || tA == tB) ? 1 : 2;
        for (int t = 0; t < 2 && ok; ++t) {
          // tile t's accumulators must have been read out for the previous item
          if (nloc > 0 &&
              !mbar_wait(t == 0 ? t1empty : t2empty, (uint32_t)((nloc - 1) & 1), abort_flag, P.err,
                         2)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t dL0 = tmem + (uint32_t)(t * 2 * TILE);
          const uint32_t dL1 = dL0 + TILE;
          for (int kc = 0; t < ntiles && kc < nks; ++kc) {
            if (!mbar_wait(full0 + 8 * stage, phase, abort_flag, P.err, 3)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t sb = smem_u32(stages + stage * STAGE_BYTES);
#pragma unroll
            for (int k16 = 0; k16 < KSTEP / 16; ++k16) {
              const uint32_t koff = k16 * 32;  // bytes inside the 128-byte swizzle row
              const uint64_t a0 = smem_desc(sb + 0 * PANEL_BYTES + koff);
              const uint64_t a1 = smem_desc(sb + 1 * PANEL_BYTES + koff);
              const uint64_t b0 = smem_desc(sb + NSL * PANEL_BYTES + koff);
              const uint64_t b1 = smem_desc(sb + (NSL + 1) * PANEL_BYTES + koff);
              const uint32_t acc = (kc > 0 || k16 > 0) ? 1u : 0u;
              // one N=256 MMA over the stacked B panels [S0b; R1b] fills
              // [L0 | L1]: L0 += S0a S0b (exact integer part), L1 += S0a R1b
              mma_f16_id(dL0, a0, b0, IDESC_N256, acc);
              mma_f16(dL1, a1, b0, 1u);  // R1a S0b
              mma_f16(dL1, a1, b1, 1u);  // R1a R1b
              if (NSL > 2) {
                const uint64_t a2 = smem_desc(sb + 2 * PANEL_BYTES + koff);
                const uint64_t b2 = smem_desc(sb + (NSL + 2) * PANEL_BYTES + koff);
                mma_f16(dL1, a0, b2, 1u);  // S0a R2b
                mma_f16(dL1, a2, b0, 1u);  // R2a S0b
              }
            }
            mma_commit(empty0 + 8 * stage);  // frees the stage when these MMAs finish
            if (++stage == NSTAGE) {
              stage = 0;
              phase ^= 1;
            }
          }
          if (!ok) break;
          mma_commit(t == 0 ? t1full : t2full);  // tile t of this item is complete
        }
        if (!ok) break;
        ++nloc;
      }
      // drain: all MMAs issued by this thread complete before TMEM is freed
      mma_commit(drain);
      const long long t0 = clock64();
      while (!mbar_test(drain, 0) && clock64() - t0 < WAIT_BUDGET) {
      }
    }
  } else {
    // ------------------------------ epilogue ----------------------------------
    const int ew = warp - 2;             // 0..15
    const int quad = warp & 3;           // TMEM lane quadrant this warp may access
    const int cbase = (ew >> 2) * 32;    // the 32 columns of the tile this warp reads
    const int row = quad * 32 + lane;    // tile row = a offset
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
    int islot = 0;
    uint32_t iphase = 0;
    long long nloc = 0;
    while (true) {
      const bool w0 = mbar_wait(ifull0 + 8 * islot, iphase, abort_flag, P.err, 7);
      if (epi_any512(!w0)) break;
      const int qidx = item_q[islot];
      __syncwarp();
      if (lane == 0) mbar_arrive(iempty0 + 8 * islot);
      if (++islot == IQ) {
        islot = 0;
        iphase ^= 1;
      }
      if (qidx < 0) break;
      const int4 it = P.items[qidx];
      const FragDesc &F = P.frags[it.x];
      const int i = it.y & 0xFFFF, j = it.y >> 16, tA = it.z & 0xFFFF, tB = it.z >> 16;
      const bool same = (i == j), diag = (tA == tB);
      const int nvpad = F.nvpad;
      const int a = tA * TILE + row;
      const float *scl = P.inv_scale + F.col_base;
      const float sa1 = scl[i * nvpad + a];  // scale of column (a,i)
      const float sa2 = scl[j * nvpad + a];  // scale of column (a,j)
      const float *sbj = scl + j * nvpad + tB * TILE + cbase;
      const float *sbi = scl + i * nvpad + tB * TILE + cbase;
      const float2 *evb = P.ev2 + F.ev_off + tB * TILE + cbase;
      // ---- T1 -> registers, then hand its TMEM back to the MMA issuer ----
      const bool w1 = mbar_wait(t1full, (uint32_t)(nloc & 1), abort_flag, P.err, 4);
      if (epi_any512(!w1)) break;
      tc_fence_after();
      const uint32_t t1 = tmem + lane_off + cbase;
      float g1[32];
#pragma unroll
      for (int c0 = 0; c0 < 32; c0 += 16) {
        float l0[16], l1[16];
        tmem_ld16(t1 + c0, l0);
        tmem_ld16(t1 + TILE + c0, l1);
        tmem_wait_ld();
#pragma unroll
        for (int k = 0; k < 16; ++k) g1[c0 + k] = (l0[k] + l1[k]) * (sa1 * sbj[c0 + k]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(t1empty);
      // ---- denominators ----
      const float2 ea = P.ev2[F.ev_off + a];
      const float2 ei = P.eo2[F.eo_off + i], ej = P.eo2[F.eo_off + j];
      // e_i + e_j in hi/lo form (two-sum of the hi parts, lo parts added)
      const float sh = ei.x + ej.x;
      const float bv = sh - ei.x;
      const float sl = (ei.x - (sh - bv)) + (ej.x - bv) + ei.y + ej.y;
      // per-row part of the denominator, again as an exact two-sum
      const float dh0 = sh - ea.x;
      const float bw = dh0 - sh;
      const float dl0 = ((sh - (dh0 - bw)) + (-ea.x - bw)) + (sl - ea.y);
      // ---- T2 and the energy terms ----
      const bool w2 = mbar_wait(t2full, (uint32_t)(nloc & 1), abort_flag, P.err, 8);
      if (epi_any512(!w2)) break;
      tc_fence_after();
      // items that do not read T2 (i = j, or A = B with T2 = T1^T) hand it
      // back to the MMA issuer at once
      bool t2_held = true;
      if (same || diag) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(t2empty);
        t2_held = false;
      }
      const uint32_t t2 = tmem + lane_off + 2 * TILE + cbase;
      // one 16-column chunk of energy terms, g2 supplied by `g2at(k)`
      auto terms = [&](int c0, const float *g2) -> float {
        float ef = 0.0f;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const float2 eb = evb[c0 + k];
          const float x1 = g1[c0 + k], x2 = g2[k];
          // d = (dh0 + dl0) - (eb.x + eb.y) with the leading subtraction exact
          const float dh = dh0 - eb.x;
          const float bz = dh - dh0;
          const float d = dh + (((dh0 - (dh - bz)) + (-eb.x - bz)) + (dl0 - eb.y));
          const float r = rcp_denom(d);
          const float num = diag ? x1 * fmaf(2.0f, x1, -x2) : 2.0f * fmaf(x1, x1 - x2, x2 * x2);
          ef = fmaf(num, r, ef);
        }
        return ef;
      };
      double eacc = 0.0;
      if (diag && !same) {
        // T2[a,b] = g_ij(b,a) = T1[b,a]: transpose T1 through shared memory in
        // two 64-row passes; pass h serves the warps that own columns [64h,64h+64)
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          asm volatile("bar.sync 1, 512;" ::: "memory");
          if ((row >> 6) == h) {
            float *dst = tbuf + (row - 64 * h) * TP + cbase;
#pragma unroll
            for (int k = 0; k < 32; ++k) dst[k] = g1[k];
          }
          asm volatile("bar.sync 1, 512;" ::: "memory");
          if ((cbase >> 6) == h) {
#pragma unroll
            for (int c0 = 0; c0 < 32; c0 += 16) {
              float g2[16];
#pragma unroll
              for (int k = 0; k < 16; ++k) g2[k] = tbuf[(cbase - 64 * h + c0 + k) * TP + row];
              eacc += (double)terms(c0, g2);
            }
          }
        }
      } else {
#pragma unroll
        for (int c0 = 0; c0 < 32; c0 += 16) {
          float g2[16];
          if (same) {
#pragma unroll
            for (int k = 0; k < 16; ++k) g2[k] = g1[c0 + k];
          } else {
            float l0[16], l1[16];
            tmem_ld16(t2 + c0, l0);
            tmem_ld16(t2 + TILE + c0, l1);
            tmem_wait_ld();
#pragma unroll
            for (int k = 0; k < 16; ++k) g2[k] = (l0[k] + l1[k]) * (sa2 * sbi[c0 + k]);
          }
          eacc += (double)terms(c0, g2);
        }
      }
      if (t2_held) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(t2empty);
      }
      // reduce the item's energy over the epilogue threads
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) eacc += __shfl_xor_sync(0xffffffffu, eacc, o);
      if (lane == 0) redd[ew] = eacc;
      asm volatile("bar.sync 1, 512;" ::: "memory");
      if (ew == 0 && lane == 0) {
        double tot = 0.0;
#pragma unroll
        for (int w = 0; w < NEPI; ++w) tot += redd[w];
        P.part[it.w] = tot;
      }
      asm volatile("bar.sync 1, 512;" ::: "memory");
      ++nloc;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  }
}

// ==========================================================================
// Paired-CTA form of the energy kernel (cta_group::2 on a cluster of two
// CTAs, M = 256).  The two CTAs of a pair evaluate the occupied pairs
// (i0, j) and (i0 + 1, j) for the same tile pair (A, B):
//   T1  = G_ij[A,B] = C_iA^T C_jB   (a on the TMEM lanes, b on the columns)
//   T2' = G_ij[B,A] = C_iB^T C_jA   (b on the lanes, a on the columns)
// Both products of an item have the same B operand in the two CTAs (C_jB,
// then C_jA), which the pair splits between its shared memories.  This
// kernel uses a third slice plane V = fp16(C*s) and folds the two R1a terms
// into one product, R1a S0b + R1a R1b = R1a V - R1a (V - S0 - R1), so a K16
// step is two MMAs (three products instead of four):
//   256x256: S0a x [S0b; R1b] -> [L0 | L1]   (B rows 0..127 = S0b from rank 0,
//                                             rows 128..255 = R1b from rank 1)
//   256x128: R1a x Vb -> L1                   (64 rows of V from each rank)
// The dropped term sum_k R1a (Vb - S0b - R1b) is a product of two
// independent rounding residues for distinct columns (a,i) != (b,j), an
// unbiased error of ~2^-21 of g that averages out of the pair energies; for
// the same column it is a sum of R1 times its own rounding error, a bias,
// which the slicing kernel computes per column (dcorr) and the epilogue
// subtracts from g_ii(a,a).  Each SM's tensor core reads 14 KB of operands
// per step (the one-CTA kernel: 28 KB for four products).
// T2' is transposed through shared memory in the epilogue, so that g_ij(a,b)
// and g_ij(b,a) meet in one thread.
// A pair item with i0 + 1 > j runs its second CTA as a dummy (results
// discarded); i0 == j (then the second CTA is a dummy) and A == B need only
// T1.  The even CTA of the pair (rank 0) owns the work queue, the TMA full
// barriers (both CTAs' copies complete on them), the MMA issue and the
// accumulator-empty barriers; its commits are multicast to both CTAs.  Every
// wait is bounded; a timeout in either CTA aborts both.
// --------------------------------------------------------------------------
constexpr int BHALF = TILE / 2;                  // B rows of an N=128 operand per CTA
constexpr int BPANEL_BYTES = BHALF * KSTEP * 2;  // 8 KB
// per-CTA stage: A panels S0a, R1a (16 KB each); Y = 128 rows of the N=256
// operand (rank 0: S0b, rank 1: R1b); W = 64 rows of Vb
constexpr int PAIR_STAGE_BYTES = 3 * PANEL_BYTES + BPANEL_BYTES;  // 56 KB
struct PairParams {
  const FragDesc *frags;
  const int4 *items;     // {fragment, i0 | j << 16, tA | tB << 16, tile pair index}
  long long nitems;      // this launch drains items [item_begin, nitems)
  long long item_begin;
  const float *dcorr;    // per column: sum over K of R1 (V - S0 - R1)
  unsigned int *queue;   // next item counter (reset per launch)
  const float2 *eo2, *ev2;
  const float *inv_scale;
  double *part;          // indexed like split_batch_kernel's work items
  float *xbuf;           // GX form: one 128x128 FP32 exchange tile per CTA of the grid
  int *err;
};

// Shared memory of split_pair_kernel<NSTAGE, GX>: the stage ring, barriers and
// item ring, and (GX = false) the 64-row transpose buffer.  With the exchange
// tile transposed through global scratch (GX = true) a fourth 56 KB stage
// fits in the 227 KB a CTA may hold.
constexpr int pair_smem_bytes(int nstage, bool gx) {
  return nstage * PAIR_STAGE_BYTES + 1024 + 512 + (gx ? 0 : 64 * TP * 4);
}
static_assert(tmem_alone(pair_smem_bytes(3, false)) && tmem_alone(pair_smem_bytes(4, true)), "tensor memory");

// Exchange-tile transpose through memory, for the GX form: each thread stores
// its 64 values of tile row `row` (columns [cbase, cbase+64)) as 16-byte
// vectors, and after a barrier reads column `row` back 16 values at a time,
// coalesced across the warp.  The .cg forms keep the round trip in L2, so no
// SM-local cache line of the previous item's tile is ever read.
__device__ __forceinline__ void st_cg4(float *p, float a, float b, float c, float d) {
  asm volatile("st.global.cg.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c),
               "f"(d)
               : "memory");
}
__device__ __forceinline__ float ld_cg(const float *p) {
  float v;
  asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
  return v;
}

template <int NSTAGE, bool GX>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NTHREADS, 1)
    split_pair_kernel(const __grid_constant__ CUtensorMap tmA,
                      const __grid_constant__ CUtensorMap tmB, PairParams P) {
  constexpr int STAGE_BYTES = PAIR_STAGE_BYTES;
  constexpr int NEPI = 8;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *base = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t *stages = base;
  uint64_t *bars = (uint64_t *)(base + NSTAGE * STAGE_BYTES);
  // bars: full[NSTAGE], empty[NSTAGE], t1full, t1empty, t2full, t2empty, drain,
  //       item_full[IQ], item_empty[IQ]
  constexpr int NB = 2 * NSTAGE + 5 + 2 * IQ;
  uint32_t *tmem_slot = (uint32_t *)(bars + NB);
  volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
  volatile int *item_q = (volatile int *)(tmem_slot + 2);  // [IQ]
  double *redd = (double *)(((uintptr_t)(tmem_slot + 2 + IQ) + 7) & ~(uintptr_t)7);  // [NEPI]
  float *tbuf = (float *)(base + NSTAGE * STAGE_BYTES + 512);  // [64][TP]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const bool leader = rank == 0;
  const uint32_t full0 = smem_u32(&bars[0]);
  const uint32_t empty0 = smem_u32(&bars[NSTAGE]);
  const uint32_t t1full = smem_u32(&bars[2 * NSTAGE]);
  const uint32_t t1empty = smem_u32(&bars[2 * NSTAGE + 1]);
  const uint32_t t2full = smem_u32(&bars[2 * NSTAGE + 2]);
  const uint32_t t2empty = smem_u32(&bars[2 * NSTAGE + 3]);
  const uint32_t drain = smem_u32(&bars[2 * NSTAGE + 4]);
  const uint32_t ifull0 = smem_u32(&bars[2 * NSTAGE + 5]);
  const uint32_t iempty0 = smem_u32(&bars[2 * NSTAGE + 5 + IQ]);
  // the pair's shared barriers live in rank 0
  const uint32_t full0_L = map_shared(full0, 0);
  const uint32_t t1empty_L = map_shared(t1empty, 0);
  const uint32_t t2empty_L = map_shared(t2empty, 0);
  const uint32_t iempty0_L = map_shared(iempty0, 0);
  const uint32_t abort_peer = map_shared(smem_u32((const void *)abort_flag), rank ^ 1u);

  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTAGE; ++s) {
      mbar_init(full0 + 8 * s, 1);   // rank 0: its producer's arrive + both CTAs' bytes
      mbar_init(empty0 + 8 * s, 1);  // multicast MMA commit
    }
    mbar_init(t1full, 1);
    mbar_init(t1empty, 2 * NEPI);  // epilogue warps of both CTAs
    mbar_init(t2full, 1);
    mbar_init(t2empty, 2 * NEPI);
    mbar_init(drain, 1);
    for (int s = 0; s < IQ; ++s) {
      mbar_init(ifull0 + 8 * s, 1);
      mbar_init(iempty0 + 8 * s, 2 + 2 * NEPI);  // MMA issuer, peer producer, all epilogue warps
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&tmA) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&tmB) : "memory");
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
      const uint32_t item_q_peer = map_shared(smem_u32((const void *)item_q), 1);
      const uint32_t ifull0_peer = map_shared(ifull0, 1);
      int stage = 0, islot = 0;
      uint32_t phase = 0, iphase = 0;
      uint32_t armed = 0, armed_par = 0;  // rank 0: stages with copies expected, and parity
      bool ok = true;
      while (ok) {
        int qidx;
        if (leader) {
          if (!pair_wait(iempty0 + 8 * islot, iphase ^ 1, true, abort_flag, abort_peer, P.err, 5))
            break;
          const long long id = P.item_begin + (long long)atomicAdd(P.queue, 1u);
          qidx = id < P.nitems ? (int)id : -1;
          item_q[islot] = qidx;
          st_remote_u32(item_q_peer + 4 * islot, (uint32_t)qidx);
          mbar_arrive(ifull0 + 8 * islot);
          mbar_arrive_remote(ifull0_peer + 8 * islot);
        } else {
          if (!pair_wait(ifull0 + 8 * islot, iphase, true, abort_flag, abort_peer, P.err, 5))
            break;
          qidx = item_q[islot];
          mbar_arrive_remote(iempty0_L + 8 * islot);
        }
        if (++islot == IQ) {
          islot = 0;
          iphase ^= 1;
        }
        if (qidx < 0) break;
        const int4 it = P.items[qidx];
        const FragDesc &F = P.frags[it.x];
        const int i0 = it.y & 0xFFFF, j = it.y >> 16, tA = it.z & 0xFFFF, tB = it.z >> 16;
        const int i = (i0 + (int)rank <= j) ? i0 + (int)rank : i0;  // a dummy loads i0's panels
        const int ntiles = (tA == tB || i0 == j) ? 1 : 2;
        for (int t = 0; t < ntiles && ok; ++t) {
          const int colA = i * F.nvpad + (t == 0 ? tA : tB) * TILE;
          const int colB = j * F.nvpad + (t == 0 ? tB : tA) * TILE;
          const int colH = colB + BHALF * (int)rank;  // this rank's half of the B rows
          for (int kc = 0; kc < F.nks; ++kc) {
            if (!pair_wait(empty0 + 8 * stage, phase ^ 1, false, abort_flag, abort_peer, P.err, 1)) {
              ok = false;
              break;
            }
            if (leader) {
              mbar_expect_tx(full0 + 8 * stage, 2 * STAGE_BYTES);
              armed |= 1u << stage;
              armed_par = (armed_par & ~(1u << stage)) | (phase << stage);
            }
            const uint32_t dst = smem_u32(stages + stage * STAGE_BYTES);
            const uint32_t fb = full0_L + 8 * stage;
            const int rowk = (int)(F.row_base + (long long)kc * F.ncol);
            tma_load_3d_pair(dst, &tmA, fb, 0, rowk + colA, 0);                // S0a
            tma_load_3d_pair(dst + PANEL_BYTES, &tmA, fb, 0, rowk + colA, 1);  // R1a
            tma_load_3d_pair(dst + 2 * PANEL_BYTES, &tmA, fb, 0, rowk + colB, (int)rank);  // Y
            tma_load_3d_pair(dst + 3 * PANEL_BYTES, &tmB, fb, 0, rowk + colH, 2);  // W: V half
            if (++stage == NSTAGE) {
              stage = 0;
              phase ^= 1;
            }
          }
        }
      }
      if (leader && (!ok || *abort_flag)) {  // copies in flight complete before the pair exits
        for (int s = 0; s < NSTAGE; ++s) {
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
      int stage = 0, islot = 0;
      uint32_t phase = 0, iphase = 0;
      bool ok = true;
      long long nloc = 0;
      while (ok) {
        if (!pair_wait(ifull0 + 8 * islot, iphase, false, abort_flag, abort_peer, P.err, 6)) break;
        const int qidx = item_q[islot];
        mbar_arrive_remote(iempty0_L + 8 * islot);
        if (++islot == IQ) {
          islot = 0;
          iphase ^= 1;
        }
        if (qidx < 0) break;
        const int4 it = P.items[qidx];
        const int nks = P.frags[it.x].nks;
        const int i0 = it.y & 0xFFFF, j = it.y >> 16, tA = it.z & 0xFFFF, tB = it.z >> 16;
        const int ntiles = (tA == tB || i0 == j) ? 1 : 2;
        for (int t = 0; t < 2 && ok; ++t) {
          // both CTAs' epilogues have read tile t of the previous item
          if (nloc > 0 && !pair_wait(t == 0 ? t1empty : t2empty, (uint32_t)((nloc - 1) & 1), true,
                                     abort_flag, abort_peer, P.err, 2)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t dL0 = tmem + (uint32_t)(t * 2 * TILE);
          const uint32_t dL1 = dL0 + TILE;
          for (int kc = 0; t < ntiles && kc < nks; ++kc) {
            if (!pair_wait(full0 + 8 * stage, phase, false, abort_flag, abort_peer, P.err, 3)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t sb = smem_u32(stages + stage * STAGE_BYTES);
#pragma unroll
            for (int k16 = 0; k16 < KSTEP / 16; ++k16) {
              const uint32_t koff = k16 * 32;  // bytes inside the 128-byte swizzle row
              const uint64_t a0 = smem_desc(sb + koff);
              const uint64_t a1 = smem_desc(sb + PANEL_BYTES + koff);
              const uint64_t by = smem_desc(sb + 2 * PANEL_BYTES + koff);
              const uint64_t bw = smem_desc(sb + 3 * PANEL_BYTES + koff);
              const uint32_t acc = (kc > 0 || k16 > 0) ? 1u : 0u;
              // [L0 | L1] += S0a x [S0b; R1b]: exact integer part and S0a R1b
              mma_f16_pair(dL0, a0, by, IDESC_PAIR_N256, acc);
              mma_f16_pair(dL1, a1, bw, IDESC_PAIR, 1u);  // R1a V (= R1a S0b + R1a R1b + R1a eps)
            }
            mma_commit_pair(empty0 + 8 * stage);  // frees the stage in both CTAs
            if (++stage == NSTAGE) {
              stage = 0;
              phase ^= 1;
            }
          }
          if (!ok) break;
          mma_commit_pair(t == 0 ? t1full : t2full);
        }
        if (!ok) break;
        ++nloc;
      }
      mma_commit_pair(drain);  // both CTAs learn when the last MMA has completed
    }
  } else {
    // --------------------- epilogue (both CTAs) ---------------------------
    const int ew = warp - 2;           // 0..7
    const int quad = warp & 3;         // TMEM lane quadrant this warp may access
    const int cbase = (ew >> 2) * 64;  // column half of the tile this warp reads
    const int row = quad * 32 + lane;  // TMEM lane = tile row
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
    int islot = 0;
    uint32_t iphase = 0;
    long long nloc = 0;
    while (true) {
      const bool w0 = pair_wait(ifull0 + 8 * islot, iphase, true, abort_flag, abort_peer, P.err, 7);
      if (epi_any(!w0)) break;
      const int qidx = item_q[islot];
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(iempty0_L + 8 * islot);
      if (++islot == IQ) {
        islot = 0;
        iphase ^= 1;
      }
      if (qidx < 0) break;
      const int4 it = P.items[qidx];
      const FragDesc &F = P.frags[it.x];
      const int i0 = it.y & 0xFFFF, j = it.y >> 16, tA = it.z & 0xFFFF, tB = it.z >> 16;
      const bool dummy = i0 + (int)rank > j;
      const int i = dummy ? i0 : i0 + (int)rank;
      const bool same = (i == j), diag = (tA == tB);
      const int nvpad = F.nvpad;
      const int a = tA * TILE + row;
      const float *scl = P.inv_scale + F.col_base;
      const float sa1 = scl[i * nvpad + a];                    // column (a,i)
      const float *sbj = scl + j * nvpad + tB * TILE + cbase;  // columns (b,j)
      const float2 *evb = P.ev2 + F.ev_off + tB * TILE + cbase;
      // ---- T1 -> registers, then release it ----
      const bool w1 = pair_wait(t1full, (uint32_t)(nloc & 1), false, abort_flag, abort_peer, P.err, 4);
      if (epi_any(!w1)) break;
      tc_fence_after();
      const uint32_t t1 = tmem + lane_off + cbase;
      float g1[64];
#pragma unroll
      for (int c0 = 0; c0 < 64; c0 += 16) {
        float l0[16], l1[16];
        tmem_ld16(t1 + c0, l0);
        tmem_ld16(t1 + TILE + c0, l1);
        tmem_wait_ld();
#pragma unroll
        for (int k = 0; k < 16; ++k) g1[c0 + k] = (l0[k] + l1[k]) * (sa1 * sbj[c0 + k]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(t1empty_L);
      if (same && diag && !dummy) {
        // g_ii(a,a): remove the same-column bias of the folded R1 V product
        const float corr = P.dcorr[F.col_base + i * nvpad + a] * (sa1 * sa1);
        const int kd = row - cbase;  // this row's diagonal element in the warp's column half
#pragma unroll
        for (int k = 0; k < 64; ++k)
          if (k == kd) g1[k] -= corr;
      }
      // ---- denominators (as split_batch_kernel) ----
      const float2 ea = P.ev2[F.ev_off + a];
      const float2 ei = P.eo2[F.eo_off + i], ej = P.eo2[F.eo_off + j];
      const float sh = ei.x + ej.x;
      const float bv = sh - ei.x;
      const float sl = (ei.x - (sh - bv)) + (ej.x - bv) + ei.y + ej.y;
      const float dh0 = sh - ea.x;
      const float bw = dh0 - sh;
      const float dl0 = ((sh - (dh0 - bw)) + (-ea.x - bw)) + (sl - ea.y);
      auto terms = [&](int c0, const float *g2) -> float {
        float ef = 0.0f;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const float2 eb = evb[c0 + k];
          const float x1 = g1[c0 + k], x2 = g2[k];
          const float dh = dh0 - eb.x;
          const float bz = dh - dh0;
          const float d = dh + (((dh0 - (dh - bz)) + (-eb.x - bz)) + (dl0 - eb.y));
          const float r = rcp_denom(d);
          const float num = diag ? x1 * fmaf(2.0f, x1, -x2) : 2.0f * fmaf(x1, x1 - x2, x2 * x2);
          ef = fmaf(num, r, ef);
        }
        return ef;
      };
      // ---- T2' and the energy terms ----
      const bool w2 = pair_wait(t2full, (uint32_t)(nloc & 1), false, abort_flag, abort_peer, P.err, 8);
      if (epi_any(!w2)) break;
      tc_fence_after();
      // each warp hands T2' back to the MMA issuer as soon as it has read its
      // rows (or at once when this item does not read T2'), so that the next
      // item's second chain can start while the energy terms are formed
      bool t2_held = true;
      auto release_t2 = [&]() {
        if (t2_held) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_remote(t2empty_L);
          t2_held = false;
        }
      };
      if (dummy || same || diag) release_t2();
      double eacc = 0.0;
      if (!dummy) {
        if (same) {  // g_ii is symmetric
#pragma unroll
          for (int c0 = 0; c0 < 64; c0 += 16) {
            float g2[16];
#pragma unroll
            for (int k = 0; k < 16; ++k) g2[k] = g1[c0 + k];
            eacc += (double)terms(c0, g2);
          }
        } else {
          // g2(a,b) = g_ij(b,a): T1 transposed (A == B) or T2' = G_ij[B,A]
          // transposed, through shared memory in two 64-row passes; pass h
          // serves the warps that own columns [64h, 64h+64)
          const uint32_t t2 = tmem + lane_off + 2 * TILE + cbase;
          const float sbi = scl[i * nvpad + tB * TILE + row];      // T2' row (b,i)
          const float *saj = scl + j * nvpad + tA * TILE + cbase;  // T2' columns (a,j)
          if constexpr (GX) {
            // every thread stores row `row` of the tile to transpose (T1 when
            // A == B, else T2'), then reads column `row` of it
            float *X = P.xbuf + (size_t)blockIdx.x * (TILE * TILE);
            float *dst = X + row * TILE + cbase;
            if (diag) {
#pragma unroll
              for (int k = 0; k < 64; k += 4) st_cg4(dst + k, g1[k], g1[k + 1], g1[k + 2], g1[k + 3]);
            } else {
#pragma unroll
              for (int c0 = 0; c0 < 64; c0 += 16) {
                float l0[16], l1[16];
                tmem_ld16(t2 + c0, l0);
                tmem_ld16(t2 + TILE + c0, l1);
                tmem_wait_ld();
                float v[16];
#pragma unroll
                for (int k = 0; k < 16; ++k) v[k] = (l0[k] + l1[k]) * (sbi * saj[c0 + k]);
#pragma unroll
                for (int k = 0; k < 16; k += 4) st_cg4(dst + c0 + k, v[k], v[k + 1], v[k + 2], v[k + 3]);
              }
              release_t2();
            }
            asm volatile("bar.sync 1, 256;" ::: "memory");
            const float *src = X + (size_t)cbase * TILE + row;
            float ga[16], gb[16];
#pragma unroll
            for (int k = 0; k < 16; ++k) ga[k] = ld_cg(src + k * TILE);
#pragma unroll
            for (int c0 = 0; c0 < 64; c0 += 32) {
#pragma unroll
              for (int k = 0; k < 16; ++k) gb[k] = ld_cg(src + (c0 + 16 + k) * TILE);
              eacc += (double)terms(c0, ga);
              if (c0 + 32 < 64) {
#pragma unroll
                for (int k = 0; k < 16; ++k) ga[k] = ld_cg(src + (c0 + 32 + k) * TILE);
              }
              eacc += (double)terms(c0 + 16, gb);
            }
          } else {
#pragma unroll 1
          for (int h = 0; h < 2; ++h) {
            asm volatile("bar.sync 1, 256;" ::: "memory");
            if ((row >> 6) == h) {
              float *dst = tbuf + (row - 64 * h) * TP + cbase;
              if (diag) {
#pragma unroll
                for (int k = 0; k < 64; ++k) dst[k] = g1[k];
              } else {
#pragma unroll
                for (int c0 = 0; c0 < 64; c0 += 16) {
                  float l0[16], l1[16];
                  tmem_ld16(t2 + c0, l0);
                  tmem_ld16(t2 + TILE + c0, l1);
                  tmem_wait_ld();
#pragma unroll
                  for (int k = 0; k < 16; ++k) dst[c0 + k] = (l0[k] + l1[k]) * (sbi * saj[c0 + k]);
                }
                release_t2();
              }
            }
            asm volatile("bar.sync 1, 256;" ::: "memory");
            if ((cbase >> 6) == h) {
#pragma unroll
              for (int c0 = 0; c0 < 64; c0 += 16) {
                float g2[16];
#pragma unroll
                for (int k = 0; k < 16; ++k) g2[k] = tbuf[(c0 + k) * TP + row];
                eacc += (double)terms(c0, g2);
              }
            }
          }
          }
        }
      }
      release_t2();
      // reduce the item's energy over the epilogue threads
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) eacc += __shfl_xor_sync(0xffffffffu, eacc, o);
      if (lane == 0) redd[ew] = eacc;
      asm volatile("bar.sync 1, 256;" ::: "memory");
      if (ew == 0 && lane == 0 && !dummy) {
        double tot = 0.0;
#pragma unroll
        for (int w = 0; w < NEPI; ++w) tot += redd[w];
        const long long p = (long long)j * (j + 1) / 2 + i;
        P.part[F.item_base + p * F.ntp + it.w] = tot;
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");
      ++nloc;
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
    // to land before either CTA exits
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

// Pair items of a group: per fragment, for each j the i0 = 0, 2, 4, ... <= j,
// times the tile pairs.  C(j) = number of pair items (without the tile-pair
// factor) before column j = floor(j/2) * floor(j/2 + 1) for even j and
// (floor(j/2) + 1)^2 for odd j.
__host__ __device__ inline long long pair_items_before(long long j) {
  const long long m = j / 2;
  return (j % 2 == 0) ? m * (m + 1) : (m + 1) * (m + 1);
}

// Pair item t of fragment f.
__device__ __forceinline__ int4 pair_item(const FragDesc &F, int f, long long t) {
  const long long loc = t - F.pitem_base;
  const long long p2 = loc / F.ntp;
  const int q = (int)(loc % F.ntp);
  int j = (int)(2.0 * sqrt((double)p2));
  if (j > F.nocc - 1) j = F.nocc - 1;
  while (j > 0 && pair_items_before(j) > p2) --j;
  while (j + 1 < F.nocc && pair_items_before(j + 1) <= p2) ++j;
  const int i0 = (int)(2 * (p2 - pair_items_before(j)));
  int tA, tB;
  decode_tri(q, tA, tB);
  return make_int4(f, i0 | (j << 16), tA | (tB << 16), q);
}

__global__ void build_pair_items_kernel(const FragDesc *__restrict__ fr, int nfrag,
                                        long long nitems, int4 *__restrict__ items) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= nitems) return;
  int lo = 0, hi = nfrag - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (fr[mid].pitem_base <= t)
      lo = mid;
    else
      hi = mid - 1;
  }
  items[t] = pair_item(fr[lo], lo, t);
}

// ==========================================================================
// Local-orbital fragment energy on the tensor cores (split form):
//   sum_ij,ab g_ij^ab / D (2 gt_ij^ab - gt_ij^ba),
// g from Calpha C, gt from its projected copy Ct (both sliced like Calpha).
// Two residual slices run here, one residual slice on split_eos_pair_kernel.
// Work item = (pair i<=j, tile pair A<=B, column half h): rows a in block A
// (128), columns b in the h-th 64-column half of block B.  Four 128x64 tiles
// per item: T1 = C_iA^T C_jB, T2 = C_jA^T C_iB, U1 = Ct_iA^T Ct_jB,
// U2 = Ct_jA^T Ct_iB, each with L0/L1 accumulators: 8 x 64 = 512 TMEM columns.
// Diagonal tile pairs compute T2/U2 too (no transpose), so each ordered (a,b)
// of A x A is met once over the two halves; i = j reuses T1/U1.
// Roles as in split_batch_kernel; a tile's accumulators are free for the next
// item once the epilogue has read them.
// --------------------------------------------------------------------------
constexpr int HALF = 64;
constexpr int HPANEL_BYTES = HALF * KSTEP * 2;  // 8 KB

struct EosParams {
  const float *inv;          // inverse scales: C columns [0, ncol), Ct columns [ncol, 2 ncol)
  const float2 *eo2, *ev2;   // hi/lo orbital energies (ev2 padded to nvpad)
  long long nitems;
  unsigned int *queue;
  double *part;              // [nitems]
  int *err;
  int nocc, nvirt, nvpad, nks, ntp, ncol;
  int rowC, rowCt;           // first slice row of C and of Ct (per plane)
};

// A stage holds S0a, R1a, R2a (128 rows) and S0b, R1b, R2b (64 rows).
constexpr int eos_stage_bytes(int nsl) { return nsl * (PANEL_BYTES + HPANEL_BYTES); }

__device__ __forceinline__ void eos_decode(const EosParams &P, long long id, int &i, int &j,
                                           int &tA, int &tB, int &h) {
  const int per = 2 * P.ntp;
  const int p = (int)(id / per), r = (int)(id % per);
  decode_pair(p, i, j);
  decode_tri(r >> 1, tA, tB);
  h = r & 1;
}

template <int NSL, int NSTAGE>
__global__ void __launch_bounds__(NTHREADS, 1)
    split_eos_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     EosParams P) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *base = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  constexpr int STAGE_BYTES = eos_stage_bytes(NSL);
  constexpr int NEPI = 8;
  uint8_t *stages = base;
  uint64_t *bars = (uint64_t *)(base + NSTAGE * STAGE_BYTES);
  // bars: full[NSTAGE], empty[NSTAGE], tfull[4], tempty[4], drain, item_full[IQ],
  //       item_empty[IQ]
  constexpr int NB = 2 * NSTAGE + 9 + 2 * IQ;
  uint32_t *tmem_slot = (uint32_t *)(bars + NB);
  volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
  volatile long long *item_q =
      (volatile long long *)(((uintptr_t)(tmem_slot + 2) + 7) & ~(uintptr_t)7);  // [IQ]
  double *redd = (double *)(item_q + IQ);                                       // [NEPI]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t full0 = smem_u32(&bars[0]);
  const uint32_t empty0 = smem_u32(&bars[NSTAGE]);
  const uint32_t tfull0 = smem_u32(&bars[2 * NSTAGE]);       // + 8 t
  const uint32_t tempty0 = smem_u32(&bars[2 * NSTAGE + 4]);  // + 8 t
  const uint32_t drain = smem_u32(&bars[2 * NSTAGE + 8]);
  const uint32_t ifull0 = smem_u32(&bars[2 * NSTAGE + 9]);
  const uint32_t iempty0 = smem_u32(&bars[2 * NSTAGE + 9 + IQ]);

  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTAGE; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int t = 0; t < 4; ++t) {
      mbar_init(tfull0 + 8 * t, 1);
      mbar_init(tempty0 + 8 * t, NEPI);
    }
    mbar_init(drain, 1);
    for (int s = 0; s < IQ; ++s) {
      mbar_init(ifull0 + 8 * s, 1);
      mbar_init(iempty0 + 8 * s, 1 + NEPI);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&tmA) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&tmB) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                     smem_u32(tmem_slot))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  // tiles in issue order o = 0..3: T1 (C), U1 (Ct), T2 (C), U2 (Ct), i.e. tile
  // t = 2 (o & 1) + (o >> 1); i = j items skip T2/U2

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      int stage = 0, islot = 0;
      uint32_t phase = 0, iphase = 0;
      int armed[NSTAGE];
      for (int s = 0; s < NSTAGE; ++s) armed[s] = -1;
      bool ok = true;
      while (ok) {
        if (!mbar_wait(iempty0 + 8 * islot, iphase ^ 1, abort_flag, P.err, 5)) break;
        const long long id = (long long)atomicAdd(P.queue, 1u);
        const long long qidx = id < P.nitems ? id : -1;
        item_q[islot] = qidx;
        mbar_arrive(ifull0 + 8 * islot);
        if (++islot == IQ) {
          islot = 0;
          iphase ^= 1;
        }
        if (qidx < 0) break;
        int i, j, tA, tB, h;
        eos_decode(P, qidx, i, j, tA, tB, h);
        const bool same = (i == j);
        for (int o = 0; o < 4 && ok; ++o) {
          const int t = ((o & 1) << 1) | (o >> 1);
          if (same && (t & 1)) continue;  // T2 = T1, U2 = U1
          const int rowbase = (t < 2) ? P.rowC : P.rowCt;
          const int ia = (t & 1) ? j : i, ib = (t & 1) ? i : j;
          const int colA = ia * P.nvpad + tA * TILE;
          const int colB = ib * P.nvpad + tB * TILE + h * HALF;
          for (int kc = 0; kc < P.nks; ++kc) {
            if (!mbar_wait(empty0 + 8 * stage, phase ^ 1, abort_flag, P.err, 1)) {
              ok = false;
              break;
            }
            const uint32_t fb = full0 + 8 * stage;
            mbar_expect_tx(fb, STAGE_BYTES);
            armed[stage] = (int)phase;
            const uint32_t dst = smem_u32(stages + stage * STAGE_BYTES);
            const int rowk = rowbase + kc * P.ncol;
#pragma unroll
            for (int sl = 0; sl < NSL; ++sl) {
              tma_load_3d(dst + sl * PANEL_BYTES, &tmA, fb, 0, rowk + colA, sl);
              tma_load_3d(dst + NSL * PANEL_BYTES + sl * HPANEL_BYTES, &tmB, fb, 0, rowk + colB,
                          sl);
            }
            if (++stage == NSTAGE) {
              stage = 0;
              phase ^= 1;
            }
          }
        }
      }
      if (!ok || *abort_flag) {  // drain copies in flight before the CTA can exit
        for (int s = 0; s < NSTAGE; ++s) {
          if (armed[s] < 0) continue;
          const long long t0 = clock64();
          while (!mbar_test(full0 + 8 * s, (uint32_t)armed[s]) && clock64() - t0 < WAIT_BUDGET) {
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer --------------------------------
    if (lane == 0) {
      constexpr uint32_t idesc = (IDESC & ~(0x3Fu << 17)) | ((uint32_t)(HALF >> 3) << 17);
      // N = 128: the two adjacent 64-row B panels [S0b; R1b] at once
      constexpr uint32_t idesc2 = IDESC;
      int stage = 0, islot = 0;
      uint32_t phase = 0, iphase = 0;
      bool ok = true;
      uint32_t used = 0, par = 0;  // per tile: committed before / commit count parity
      while (ok) {
        if (!mbar_wait(ifull0 + 8 * islot, iphase, abort_flag, P.err, 6)) break;
        const long long qidx = item_q[islot];
        mbar_arrive(iempty0 + 8 * islot);
        if (++islot == IQ) {
          islot = 0;
          iphase ^= 1;
        }
        if (qidx < 0) break;
        int i, j, tA, tB, h;
        eos_decode(P, qidx, i, j, tA, tB, h);
        const bool same = (i == j);
        for (int o = 0; o < 4 && ok; ++o) {
          const int t = ((o & 1) << 1) | (o >> 1);
          if (same && (t & 1)) continue;
          // the tile's previous accumulators must have been read out
          if (((used >> t) & 1) &&
              !mbar_wait(tempty0 + 8 * t, ((par >> t) & 1) ^ 1u, abort_flag, P.err, 2)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t dL0 = tmem + (uint32_t)(t * 2 * HALF);
          const uint32_t dL1 = dL0 + HALF;
          for (int kc = 0; kc < P.nks; ++kc) {
            if (!mbar_wait(full0 + 8 * stage, phase, abort_flag, P.err, 3)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t sb = smem_u32(stages + stage * STAGE_BYTES);
            const uint32_t sbB = sb + NSL * PANEL_BYTES;
#pragma unroll
            for (int k16 = 0; k16 < KSTEP / 16; ++k16) {
              const uint32_t koff = k16 * 32;
              const uint64_t a0 = smem_desc(sb + 0 * PANEL_BYTES + koff);
              const uint64_t a1 = smem_desc(sb + 1 * PANEL_BYTES + koff);
              const uint64_t b0 = smem_desc(sbB + 0 * HPANEL_BYTES + koff);
              const uint64_t b1 = smem_desc(sbB + 1 * HPANEL_BYTES + koff);
              const uint32_t acc = (kc > 0 || k16 > 0) ? 1u : 0u;
              // [L0 | L1] += S0a x [S0b; R1b]: exact integer part and S0a R1b
              mma_f16_id(dL0, a0, b0, idesc2, acc);
              mma_f16_id(dL1, a1, b0, idesc, 1u);   // R1a S0b
              mma_f16_id(dL1, a1, b1, idesc, 1u);   // R1a R1b
              if (NSL > 2) {
                const uint64_t a2 = smem_desc(sb + 2 * PANEL_BYTES + koff);
                const uint64_t b2 = smem_desc(sbB + 2 * HPANEL_BYTES + koff);
                mma_f16_id(dL1, a0, b2, idesc, 1u);  // S0a R2b
                mma_f16_id(dL1, a2, b0, idesc, 1u);  // R2a S0b
              }
            }
            mma_commit(empty0 + 8 * stage);
            if (++stage == NSTAGE) {
              stage = 0;
              phase ^= 1;
            }
          }
          if (!ok) break;
          mma_commit(tfull0 + 8 * t);  // tile t of this item is complete
          used |= 1u << t;
          par ^= 1u << t;
        }
      }
      // drain: all MMAs issued by this thread complete before TMEM is freed
      mma_commit(drain);
      const long long t0 = clock64();
      while (!mbar_test(drain, 0) && clock64() - t0 < WAIT_BUDGET) {
      }
    }
  } else {
    // ------------------------------ epilogue ----------------------------------
    // T1 and U1 are read into registers and released first, so the next
    // item's T1/U1 MMAs overlap this item's T2/U2 phase.
    const int ew = warp - 2;             // 0..7
    const int quad = warp & 3;
    const int cbase = (ew >> 2) * 32;    // 32 of the tile's 64 columns
    const int row = quad * 32 + lane;
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
    const uint32_t tbase = tmem + lane_off + cbase;
    int islot = 0;
    uint32_t iphase = 0;
    uint32_t par = 0;  // per tile: parity of the reads so far
    bool ok = true;
    while (ok) {
      const bool w0 = mbar_wait(ifull0 + 8 * islot, iphase, abort_flag, P.err, 7);
      if (epi_any(!w0)) break;
      const long long qidx = item_q[islot];
      __syncwarp();
      if (lane == 0) mbar_arrive(iempty0 + 8 * islot);
      if (++islot == IQ) {
        islot = 0;
        iphase ^= 1;
      }
      if (qidx < 0) break;
      int i, j, tA, tB, h;
      eos_decode(P, qidx, i, j, tA, tB, h);
      const bool same = (i == j), diag = (tA == tB);
      const int a = tA * TILE + row;
      const int b0 = tB * TILE + h * HALF + cbase;
      const float *sc = P.inv, *st = P.inv + P.ncol;
      const float sCi = sc[i * P.nvpad + a], sCj = sc[j * P.nvpad + a];
      const float sTi = st[i * P.nvpad + a], sTj = st[j * P.nvpad + a];
      const float2 ea = P.ev2[a];
      const float2 ei = P.eo2[i], ej = P.eo2[j];
      const float sh = ei.x + ej.x;
      const float bv = sh - ei.x;
      const float sl = (ei.x - (sh - bv)) + (ej.x - bv) + ei.y + ej.y;
      const float dh0 = sh - ea.x;
      const float bw = dh0 - sh;
      const float dl0 = ((sh - (dh0 - bw)) + (-ea.x - bw)) + (sl - ea.y);
      // one tile's 32 columns of this thread into registers, then release it
      auto take = [&](int t, const float *sr, float srow, float (&v)[32]) -> bool {
        const bool w = mbar_wait(tfull0 + 8 * t, (par >> t) & 1, abort_flag, P.err, 4);
        if (epi_any(!w)) return false;
        tc_fence_after();
#pragma unroll
        for (int c0 = 0; c0 < 32; c0 += 16) {
          float l0[16], l1[16];
          tmem_ld16(tbase + t * 2 * HALF + c0, l0);
          tmem_ld16(tbase + t * 2 * HALF + HALF + c0, l1);
          tmem_wait_ld();
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            v[c0 + k] = (l0[k] + l1[k]) * (srow * sr[b0 + c0 + k]);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(tempty0 + 8 * t);
        par ^= 1u << t;
        return true;
      };
      float g1[32], u1[32];
      if (!take(0, sc + j * P.nvpad, sCi, g1) || !take(2, st + j * P.nvpad, sTi, u1)) {
        ok = false;
        break;
      }

      double eacc = 0.0;
      if (same) {
        float ef = 0.0f;
#pragma unroll
        for (int k = 0; k < 32; ++k) {
          const float2 eb = P.ev2[b0 + k];
          const float dh = dh0 - eb.x;
          const float bz = dh - dh0;
          const float d = dh + (((dh0 - (dh - bz)) + (-eb.x - bz)) + (dl0 - eb.y));
          // g2 = g1, u2 = u1: diagonal g1 u1, otherwise 2 g1 u1
          ef = fmaf((diag ? 1.0f : 2.0f) * g1[k] * u1[k], rcp_denom(d), ef);
        }
        eacc = (double)ef;
      } else {
        float g2[32], u2[32];
        if (!take(1, sc + i * P.nvpad, sCj, g2) || !take(3, st + i * P.nvpad, sTj, u2)) {
          ok = false;
          break;
        }
#pragma unroll
        for (int c0 = 0; c0 < 32; c0 += 16) {
          float ef = 0.0f;
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            const float2 eb = P.ev2[b0 + c0 + k];
            const float dh = dh0 - eb.x;
            const float bz = dh - dh0;
            const float d = dh + (((dh0 - (dh - bz)) + (-eb.x - bz)) + (dl0 - eb.y));
            const int c = c0 + k;
            float num = g1[c] * fmaf(2.0f, u1[c], -u2[c]);
            if (!diag) num = fmaf(g2[c], fmaf(2.0f, u2[c], -u1[c]), num);
            ef = fmaf(num, rcp_denom(d), ef);
          }
          eacc += (double)ef;
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) eacc += __shfl_xor_sync(0xffffffffu, eacc, o);
      if (lane == 0) redd[ew] = eacc;
      asm volatile("bar.sync 1, 256;" ::: "memory");
      if (ew == 0 && lane == 0) {
        double tot = 0.0;
#pragma unroll
        for (int w = 0; w < NEPI; ++w) tot += redd[w];
        P.part[qidx] = tot;
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  }
}

// --------------------------------------------------------------------------
// One residual slice (three products): CTA pairs, both partitionings at once.
// The one-CTA form above moves 14 KB into shared memory and reads 14 KB of it
// per K16 step of 96 MMA cycles, more than the 128 bytes a clock that memory
// gives, so half the tensor time is lost; and it contracts Calpha with itself
// once per partitioning.  Here a pair of CTAs takes 256 rows (virtual blocks
// 2R and 2R+1 of one occupied pair) by a 128-column block, the columns'
// operand split between the two as in split_pair_kernel, and runs through the
// tiles T1, T2 of Calpha and U1, U2 of each projected copy in two alternating
// 256-column accumulators; g (T1, T2) waits in a thread-private stash (L2)
// for the tiles of both partitionings.  Products, their order and the energy
// terms are the one-CTA form's.  Row blocks beyond the column block (the pair
// (2R+1, 2R)) are a dummy's: 14% of the tiles at six blocks, 3% at 24.
// Measured (GB300, nvirt 741, nocc 59, NBA 2173, both partitionings): 33.8 ms,
// against 57.4 ms in two launches of the one-CTA form with the V plane.
// --------------------------------------------------------------------------
struct EosPairParams {
  const float *inv;      // inverse scales [set][ncol]: Calpha, then the projected copies
  const float *dcorr;    // [set][ncol]
  const float2 *eo2, *ev2;
  long long nitems, npart;
  unsigned int *queue;
  double *part;          // [copy][pair * ntp + tile pair], npart values each
  float *stash;          // per CTA [2][64][256]
  int *err;
  int nvpad, nks, nt, ntp, per, ncol, copies;
  int row0[3];           // first slice row of each set
};

// item -> occupied pair, row block, column block
__device__ __forceinline__ void eos_pair_decode(const EosPairParams &P, long long id, int &i, int &j,
                                                int &R, int &tB) {
  decode_pair((int)(id / P.per), i, j);
  int r = (int)(id % P.per);
  R = 0;
  while (r >= P.nt - 2 * R) {
    r -= P.nt - 2 * R;
    ++R;
  }
  tB = 2 * R + r;
}

constexpr int EP_NSTAGE = 3;
constexpr int EP_SMEM = EP_NSTAGE * PAIR_STAGE_BYTES + 1024 + 512;
static_assert(tmem_alone(EP_SMEM), "tensor memory");

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NTHREADS, 1)
    split_eos_pair_kernel(const __grid_constant__ CUtensorMap tmA,
                          const __grid_constant__ CUtensorMap tmB, EosPairParams P) {
  constexpr int NSTAGE = EP_NSTAGE, STAGE_BYTES = PAIR_STAGE_BYTES, NEPI = 8;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *base = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t *stages = base;
  uint64_t *bars = (uint64_t *)(base + NSTAGE * STAGE_BYTES);
  // bars: full[NSTAGE], empty[NSTAGE], tfull[2], tempty[2], drain, item_full[IQ], item_empty[IQ]
  constexpr int NB = 2 * NSTAGE + 5 + 2 * IQ;
  uint32_t *tmem_slot = (uint32_t *)(bars + NB);
  volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
  volatile int *item_q = (volatile int *)(tmem_slot + 2);  // [IQ]
  double *redd = (double *)(((uintptr_t)(tmem_slot + 2 + IQ) + 7) & ~(uintptr_t)7);  // [2][NEPI]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const bool leader = rank == 0;
  const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[NSTAGE]);
  const uint32_t tfull0 = smem_u32(&bars[2 * NSTAGE]), tempty0 = smem_u32(&bars[2 * NSTAGE + 2]);
  const uint32_t drain = smem_u32(&bars[2 * NSTAGE + 4]);
  const uint32_t ifull0 = smem_u32(&bars[2 * NSTAGE + 5]);
  const uint32_t iempty0 = smem_u32(&bars[2 * NSTAGE + 5 + IQ]);
  // the pair's shared barriers live in rank 0
  const uint32_t full0_L = map_shared(full0, 0), tempty0_L = map_shared(tempty0, 0);
  const uint32_t iempty0_L = map_shared(iempty0, 0);
  const uint32_t abort_peer = map_shared(smem_u32((const void *)abort_flag), rank ^ 1u);

  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTAGE; ++s) {
      mbar_init(full0 + 8 * s, 1);   // rank 0: its producer's arrive + both CTAs' bytes
      mbar_init(empty0 + 8 * s, 1);  // multicast MMA commit
    }
    for (int u = 0; u < 2; ++u) {
      mbar_init(tfull0 + 8 * u, 1);
      mbar_init(tempty0 + 8 * u, 2 * NEPI);  // epilogue warps of both CTAs
    }
    mbar_init(drain, 1);
    for (int s = 0; s < IQ; ++s) {
      mbar_init(ifull0 + 8 * s, 1);
      mbar_init(iempty0 + 8 * s, 2 + 2 * NEPI);  // MMA issuer, peer producer, all epilogue warps
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&tmA) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&tmB) : "memory");
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

  if (warp == 0) {
    // --------------------- TMA producers (both CTAs) ---------------------
    if (lane == 0) {
      const uint32_t item_q_peer = map_shared(smem_u32((const void *)item_q), 1);
      const uint32_t ifull0_peer = map_shared(ifull0, 1);
      int stage = 0, islot = 0;
      uint32_t phase = 0, iphase = 0, armed = 0, armed_par = 0;
      bool ok = true;
      while (ok) {
        int qidx;
        if (leader) {
          if (!pair_wait(iempty0 + 8 * islot, iphase ^ 1, true, abort_flag, abort_peer, P.err, 35))
            break;
          const long long id = (long long)atomicAdd(P.queue, 1u);
          qidx = id < P.nitems ? (int)id : -1;
          item_q[islot] = qidx;
          st_remote_u32(item_q_peer + 4 * islot, (uint32_t)qidx);
          mbar_arrive(ifull0 + 8 * islot);
          mbar_arrive_remote(ifull0_peer + 8 * islot);
        } else {
          if (!pair_wait(ifull0 + 8 * islot, iphase, true, abort_flag, abort_peer, P.err, 35)) break;
          qidx = item_q[islot];
          mbar_arrive_remote(iempty0_L + 8 * islot);
        }
        if (++islot == IQ) {
          islot = 0;
          iphase ^= 1;
        }
        if (qidx < 0) break;
        int i, j, R, tB;
        eos_pair_decode(P, qidx, i, j, R, tB);
        const int tA = min(2 * R + (int)rank, tB);  // a dummy loads block tB's rows
        for (int o = 0; o < 2 * (P.copies + 1) && ok; ++o) {
          const int set = o >> 1, t = o & 1;
          if (t && i == j) continue;  // T2 = T1, U2 = U1
          const int colA = (t ? j : i) * P.nvpad + tA * TILE;
          const int colB = (t ? i : j) * P.nvpad + tB * TILE;
          const int colH = colB + BHALF * (int)rank;  // this rank's half of the V rows
          for (int kc = 0; kc < P.nks; ++kc) {
            if (!pair_wait(empty0 + 8 * stage, phase ^ 1, false, abort_flag, abort_peer, P.err, 31)) {
              ok = false;
              break;
            }
            if (leader) {
              mbar_expect_tx(full0 + 8 * stage, 2 * STAGE_BYTES);
              armed |= 1u << stage;
              armed_par = (armed_par & ~(1u << stage)) | (phase << stage);
            }
            const uint32_t dst = smem_u32(stages + stage * STAGE_BYTES), fb = full0_L + 8 * stage;
            const int rowk = P.row0[set] + kc * P.ncol;
            tma_load_3d_pair(dst, &tmA, fb, 0, rowk + colA, 0);                            // S0a
            tma_load_3d_pair(dst + PANEL_BYTES, &tmA, fb, 0, rowk + colA, 1);              // R1a
            tma_load_3d_pair(dst + 2 * PANEL_BYTES, &tmA, fb, 0, rowk + colB, (int)rank);  // S0b / R1b
            tma_load_3d_pair(dst + 3 * PANEL_BYTES, &tmB, fb, 0, rowk + colH, 2);          // half of Vb
            if (++stage == NSTAGE) {
              stage = 0;
              phase ^= 1;
            }
          }
        }
      }
      if (leader && (!ok || *abort_flag)) {  // copies in flight complete before the pair exits
        for (int s = 0; s < NSTAGE; ++s) {
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
      int stage = 0, islot = 0;
      uint32_t phase = 0, iphase = 0;
      bool ok = true;
      long long n = 0;  // tiles so far
      while (ok) {
        if (!pair_wait(ifull0 + 8 * islot, iphase, false, abort_flag, abort_peer, P.err, 36)) break;
        const int qidx = item_q[islot];
        mbar_arrive_remote(iempty0_L + 8 * islot);
        if (++islot == IQ) {
          islot = 0;
          iphase ^= 1;
        }
        if (qidx < 0) break;
        int i, j, R, tB;
        eos_pair_decode(P, qidx, i, j, R, tB);
        for (int o = 0; o < 2 * (P.copies + 1) && ok; ++o) {
          if ((o & 1) && i == j) continue;
          const int u = (int)(n & 1);
          // both CTAs' epilogues have read this accumulator's previous tile
          if (n >= 2 && !pair_wait(tempty0 + 8 * u, (uint32_t)(((n >> 1) - 1) & 1), true, abort_flag,
                                   abort_peer, P.err, 32)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t dL0 = tmem + (uint32_t)(u * 2 * TILE), dL1 = dL0 + TILE;
          for (int kc = 0; kc < P.nks; ++kc) {
            if (!pair_wait(full0 + 8 * stage, phase, false, abort_flag, abort_peer, P.err, 33)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t sb = smem_u32(stages + stage * STAGE_BYTES);
#pragma unroll
            for (int k16 = 0; k16 < KSTEP / 16; ++k16) {
              const uint32_t koff = k16 * 32;
              const uint32_t acc = (kc > 0 || k16 > 0) ? 1u : 0u;
              // [L0 | L1] += S0a x [S0b; R1b], then L1 += R1a V
              mma_f16_pair(dL0, smem_desc(sb + koff), smem_desc(sb + 2 * PANEL_BYTES + koff),
                           IDESC_PAIR_N256, acc);
              mma_f16_pair(dL1, smem_desc(sb + PANEL_BYTES + koff),
                           smem_desc(sb + 3 * PANEL_BYTES + koff), IDESC_PAIR, 1u);
            }
            mma_commit_pair(empty0 + 8 * stage);  // frees the stage in both CTAs
            if (++stage == NSTAGE) {
              stage = 0;
              phase ^= 1;
            }
          }
          if (!ok) break;
          mma_commit_pair(tfull0 + 8 * u);
          ++n;
        }
      }
      mma_commit_pair(drain);  // both CTAs learn when the last MMA has completed
    }
  } else {
    // --------------------- epilogue (both CTAs) ---------------------------
    const int ew = warp - 2, quad = warp & 3;
    const int cbase = (ew >> 2) * 64;  // 64 of the tile's 128 columns
    const int row = quad * 32 + lane;
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
    float *st = P.stash + (size_t)blockIdx.x * (2 * 64 * 256) + (threadIdx.x - 64);
    int islot = 0;
    uint32_t iphase = 0;
    long long n = 0;
    bool ok = true;
    while (ok) {
      const bool w0 = pair_wait(ifull0 + 8 * islot, iphase, true, abort_flag, abort_peer, P.err, 37);
      if (epi_any(!w0)) break;
      const int qidx = item_q[islot];
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(iempty0_L + 8 * islot);
      if (++islot == IQ) {
        islot = 0;
        iphase ^= 1;
      }
      if (qidx < 0) break;
      int i, j, R, tB;
      eos_pair_decode(P, qidx, i, j, R, tB);
      const int tA = 2 * R + (int)rank;
      const bool dummy = tA > tB, same = i == j, diag = tA == tB;
      const int a = min(tA, tB) * TILE + row, b0 = tB * TILE + cbase;
      const float2 ea = P.ev2[a];
      const float2 ei = P.eo2[i], ej = P.eo2[j];
      const float sh = ei.x + ej.x;
      const float bv = sh - ei.x;
      const float sl = (ei.x - (sh - bv)) + (ej.x - bv) + ei.y + ej.y;
      const float dh0 = sh - ea.x;
      const float bw = dh0 - sh;
      const float dl0 = ((sh - (dh0 - bw)) + (-ea.x - bw)) + (sl - ea.y);
      auto rden = [&](int b) -> float {  // reciprocal denominator of (a, b)
        const float2 eb = P.ev2[b];
        const float dh = dh0 - eb.x;
        const float bz = dh - dh0;
        return rcp_denom(dh + (((dh0 - (dh - bz)) + (-eb.x - bz)) + (dl0 - eb.y)));
      };
      // g_ii(a,a) of each set carries the same-column bias sum_k R1 (V - S0 - R1)
      const int cd = (same && diag && a - b0 >= 0 && a - b0 < 64) ? a - b0 : -1;
      // this thread's 16 values of the current tile from column c0 on
      auto read = [&](int set, int t, uint32_t tb, float corr, int c0, float (&v)[16]) {
        const float *sc = P.inv + (size_t)set * P.ncol;
        const float srow = sc[(t ? j : i) * P.nvpad + a];
        const float *scol = sc + (t ? i : j) * P.nvpad + b0 + c0;
        float l0[16], l1[16];
        tmem_ld16(tb + c0, l0);
        tmem_ld16(tb + TILE + c0, l1);
        tmem_wait_ld();
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          float x = l0[k] + l1[k];
          if (c0 + k == cd && t == 0) x -= corr;
          v[k] = x * (srow * scol[k]);
        }
      };
      double eacc[2] = {0.0, 0.0};
      float u1[64];
      for (int o = 0; o < 2 * (P.copies + 1); ++o) {
        const int set = o >> 1, t = o & 1;
        if (t && same) continue;
        const int u = (int)(n & 1);
        const bool w = pair_wait(tfull0 + 8 * u, (uint32_t)((n >> 1) & 1), false, abort_flag,
                                 abort_peer, P.err, 34);
        if (epi_any(!w)) {
          ok = false;
          break;
        }
        ++n;
        tc_fence_after();
        const uint32_t tb = tmem + lane_off + (uint32_t)(u * 2 * TILE + cbase);
        const float corr = cd >= 0 ? P.dcorr[(size_t)set * P.ncol + i * P.nvpad + a] : 0.0f;
        double e = 0.0;
        if (dummy) {
        } else if (set == 0) {  // g: kept for the projected sets
#pragma unroll 1
          for (int c0 = 0; c0 < 64; c0 += 16) {
            float v[16];
            read(0, t, tb, corr, c0, v);
#pragma unroll
            for (int k = 0; k < 16; ++k) __stcg(st + (size_t)(t * 64 + c0 + k) * 256, v[k]);
          }
        } else if (t == 0) {
#pragma unroll
          for (int c0 = 0; c0 < 64; c0 += 16) {
            float v[16];
            read(set, 0, tb, corr, c0, v);
#pragma unroll
            for (int k = 0; k < 16; ++k) u1[c0 + k] = v[k];
          }
          if (same) {  // g2 = g1, u2 = u1: diagonal g1 u1, otherwise 2 g1 u1
#pragma unroll
            for (int c0 = 0; c0 < 64; c0 += 32) {
              float ef = 0.0f;
#pragma unroll
              for (int k = 0; k < 32; ++k)
                ef = fmaf((diag ? 1.0f : 2.0f) * __ldcg(st + (size_t)(c0 + k) * 256) * u1[c0 + k],
                          rden(b0 + c0 + k), ef);
              e += (double)ef;
            }
          }
        } else {
#pragma unroll
          for (int c0 = 0; c0 < 64; c0 += 16) {
            float u2[16];
            read(set, 1, tb, corr, c0, u2);
            float ef = 0.0f;
#pragma unroll
            for (int k = 0; k < 16; ++k) {
              const float g1 = __ldcg(st + (size_t)(c0 + k) * 256);
              const float g2 = __ldcg(st + (size_t)(64 + c0 + k) * 256);
              float num = g1 * fmaf(2.0f, u1[c0 + k], -u2[k]);
              if (!diag) num = fmaf(g2, fmaf(2.0f, u2[k], -u1[c0 + k]), num);
              ef = fmaf(num, rden(b0 + c0 + k), ef);
            }
            e += (double)ef;
          }
        }
        if (set == 1) eacc[0] += e;
        if (set == 2) eacc[1] += e;
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_remote(tempty0_L + 8 * u);
      }
      if (!ok) break;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        double e = eacc[c];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
        if (lane == 0) redd[c * NEPI + ew] = e;
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");
      if (ew == 0 && lane < P.copies && !dummy) {
        double tot = 0.0;
#pragma unroll
        for (int w = 0; w < NEPI; ++w) tot += redd[lane * NEPI + w];
        const long long p = (long long)j * (j + 1) / 2 + i;
        P.part[lane * P.npart + p * P.ntp + tB * (tB + 1) / 2 + tA] = tot;
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");
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

constexpr int eos_smem_bytes(int nsl, int nstage) {
  return nstage * eos_stage_bytes(nsl) + 1024 + 512;
}
static_assert(eos_smem_bytes(3, 3) >= TMEM_SMEM_MIN, "tensor memory");

// Self-test of the bounded-wait path: one thread waits on an mbarrier that
// nothing ever completes, with a short clock budget.  The wait must give up,
// raise the CTA abort flag and record `code` in the device error word, and
// the kernel must return normally.
__global__ void wait_selftest_kernel(long long budget, int *err) {
  __shared__ uint64_t bar;
  __shared__ int abort_flag;
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&bar), 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const bool ok = mbar_wait(smem_u32(&bar), 0, (volatile int *)&abort_flag, err, 99, budget);
    if (ok) atomicCAS(err, 0, 98);  // cannot happen: nothing arrives
  }
  __syncthreads();
}

// Self-test of the epilogue's reciprocal: rcp_denom(d) beside CUDA's
// correctly rounded single-precision reciprocal __frcp_rn(d).
__global__ void rcp_selftest_kernel(const float *__restrict__ d, float *__restrict__ r,
                                    float *__restrict__ ref, int n) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  r[t] = rcp_denom(d[t]);
  ref[t] = __frcp_rn(d[t]);
}

// --------------------------------------------------------------------------
// reductions of a batch (deterministic, compensated)
// --------------------------------------------------------------------------
__device__ __forceinline__ void two_sum_d(double a, double b, double &s, double &e) {
  s = a + b;
  const double bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}

// width: a power of two, the lanes from it on hold zeros
__device__ __forceinline__ void warp_sum_comp_d(double &s, double &c, int width = 32) {
  for (int o = width >> 1; o > 0; o >>= 1) {
    const double s2 = __shfl_xor_sync(0xffffffffu, s, o);
    const double c2 = __shfl_xor_sync(0xffffffffu, c, o);
    double t, e;
    if ((threadIdx.x & o) == 0)
      two_sum_d(s, s2, t, e);
    else
      two_sum_d(s2, s, t, e);
    s = t;
    c = ((threadIdx.x & o) == 0 ? c + c2 : c2 + c) + e;
  }
}

// one warp per (fragment, pair): Epair_f(i,j) = Epair_f(j,i) = sum of its items
__global__ void pair_reduce_batch_kernel(const FragDesc *__restrict__ fr, int nfrag,
                                         int npairs_total, const double *__restrict__ part) {
  const int gp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (gp >= npairs_total) return;
  int lo = 0, hi = nfrag - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (fr[mid].pair_base <= gp)
      lo = mid;
    else
      hi = mid - 1;
  }
  const FragDesc &F = fr[lo];
  const int p = gp - F.pair_base;
  const double *src = part + F.item_base + (long long)p * F.ntp;
  double s = 0.0, c = 0.0;
  for (int r = lane; r < F.ntp; r += 32) {
    double t, e;
    two_sum_d(s, src[r], t, e);
    s = t;
    c += e;
  }
  warp_sum_comp_d(s, c, tree_width(F.ntp));
  if (lane == 0) {
    int i, j;
    decode_pair(p, i, j);
    const double v = s + c;
    F.Epair[i + (size_t)F.nocc * j] = v;
    F.Epair[j + (size_t)F.nocc * i] = v;
  }
}

// one block per fragment: Etot_f = sum_ij Epair_f(i,j)
__global__ void total_reduce_batch_kernel(const FragDesc *__restrict__ fr) {
  const FragDesc &F = fr[blockIdx.x];
  __shared__ double ss[32], sc[32];
  double s = 0.0, c = 0.0;
  const size_t n = (size_t)F.nocc * F.nocc;
  for (size_t k = threadIdx.x; k < n; k += blockDim.x) {
    double t, e;
    two_sum_d(s, F.Epair[k], t, e);
    s = t;
    c += e;
  }
  warp_sum_comp_d(s, c);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) {
    ss[w] = s;
    sc[w] = c;
  }
  __syncthreads();
  if (w == 0) {
    const int nw = blockDim.x >> 5;
    s = lane < nw ? ss[lane] : 0.0;
    c = lane < nw ? sc[lane] : 0.0;
    warp_sum_comp_d(s, c);
    if (lane == 0) *F.Etot = s + c;
  }
}

// One fragment: everything before the energy kernel in one launch (slices, the
// descriptor, orbital energies, work items, counters), and both reductions in
// one.  A small call is bound by its launches: seven kernels, a memset and a
// copy took 50 us of GPU time at nocc = 8, nvirt = 96, NBA = 256.
struct SingleArgs {
  FragDesc F;
  FragDesc *frag;
  int slice_blocks, nsl, vplane, nitems, npitems, light_last;
  long long plane;
  __half *slices;
  float *inv, *dcorr;
  float2 *eo2, *ev2;
  int4 *items, *pitems;
  unsigned *queue;  // item counter, reduction blocks done
  double *part;
};

// The item that goes t-th into the queue: where the slices stay in L2, the tile pairs
// A < B (two products an item) before the pairs A = A (one), so that the last items,
// which leave SMs idle, are the short ones: 92.6 -> 78.9 us a call at nocc = 16, nvirt =
// 200, NBA = 1024 with the launches set up ahead (88), 267 -> 261 at 24/301/1203, 597 ->
// 590 at 40/300/1100 (106 MB of slices).  At 32/512/2048 (201 MB of 129 MB L2) the
// separated items read their panels from DRAM again: 1161 -> 1240 us.
__device__ __forceinline__ int queue_order(const SingleArgs &P, int t, int n) {
  const int ntp = P.F.ntp, nt = P.F.nvpad / TILE, noff = ntp - nt, pairs = n / ntp;
  if (!P.light_last || noff == 0) return t;
  const bool off = t < pairs * noff;
  const int u = off ? t : t - pairs * noff, per = off ? noff : nt, p = u / per;
  int A = u % per, B = A;
  if (off) {  // the k-th pair A < B
    int k = A;
    for (B = 1; k >= B; ++B) k -= B;
    A = k;
  }
  return p * ntp + B * (B + 1) / 2 + A;
}

__global__ void __launch_bounds__(256, 6) single_inputs_kernel(const __grid_constant__ SingleArgs P) {
  if ((int)blockIdx.x < P.slice_blocks) {
    const int col = (blockIdx.x * 256 + threadIdx.x) >> 5;
    if (col < P.F.ncol) slice_column(P.F, col, P.nsl, P.plane, P.slices, P.inv, P.vplane, P.dcorr);
    grid_trigger();
    return;
  }
  const int t = ((int)blockIdx.x - P.slice_blocks) * 256 + threadIdx.x;
  if (t == 0) {
    *P.frag = P.F;
    P.queue[0] = P.queue[1] = 0;
  }
  eps_entry(P.F, t, P.eo2, P.ev2);
  if (t < P.nitems) P.items[t] = work_item(P.F, 0, queue_order(P, t, P.nitems));
  if (t < P.npitems) P.pitems[t] = pair_item(P.F, 0, queue_order(P, t, P.npitems));
  grid_trigger();
}

// One warp per pair; the last block to finish sums the total.
__global__ void __launch_bounds__(256) single_reduce_kernel(const __grid_constant__ SingleArgs P) {
  __shared__ double ss[8], sc[8];
  __shared__ bool last;
  const FragDesc &F = P.F;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, p = blockIdx.x * 8 + w;
  grid_wait();
  if (p < F.nocc * (F.nocc + 1) / 2) {
    const double *src = P.part + (long long)p * F.ntp;
    double s = 0.0, c = 0.0;
    for (int r = lane; r < F.ntp; r += 32) {
      double t, e;
      two_sum_d(s, src[r], t, e);
      s = t;
      c += e;
    }
    warp_sum_comp_d(s, c, tree_width(F.ntp));
    if (lane == 0) {
      int i, j;
      decode_pair(p, i, j);
      const double v = s + c;
      F.Epair[i + (size_t)F.nocc * j] = v;
      F.Epair[j + (size_t)F.nocc * i] = v;
      __threadfence();
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(P.queue + 1, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  const int n = F.nocc * F.nocc, nw = min(8, (n + 255) / 256);  // warps of the total
  double s = 0.0, c = 0.0;
  if (w < nw) {
    for (int k = threadIdx.x; k < n; k += 32 * nw) {
      double t, e;
      two_sum_d(s, __ldcg(F.Epair + k), t, e);
      s = t;
      c += e;
    }
    warp_sum_comp_d(s, c);
    if (lane == 0) {
      ss[w] = s;
      sc[w] = c;
    }
  }
  __syncthreads();
  if (w == 0) {
    s = lane < nw ? ss[lane] : 0.0;
    c = lane < nw ? sc[lane] : 0.0;
    warp_sum_comp_d(s, c, tree_width(nw));
    if (lane == 0) *F.Etot = s + c;
  }
}

// --------------------------------------------------------------------------
// host side
// --------------------------------------------------------------------------
constexpr int smem_bytes(int nsl, int nstage) {
  return nstage * nsl * 2 * PANEL_BYTES + 1024 /*align*/ + 512 /*barriers, ring, etc*/ +
         64 * TP * 4 /*diagonal-tile transpose buffer*/;
}
static_assert(smem_bytes(2, 3) >= TMEM_SMEM_MIN && smem_bytes(3, 2) >= TMEM_SMEM_MIN, "tensor memory");

// One launch group of a batch: its fragments share a slice count and an
// energy kernel (one-CTA or paired), a slices buffer, the tensor maps and one
// persistent launch.
struct Group {
  int nsl = 2;
  int nfrag = 0;
  std::vector<FragDesc> fh;
  long long nitems = 0, R = 0, ncol_total = 0;
  int npairs_total = 0, max_ncol = 0, max_nv = 0, max_nocc = 0;
  DevBuf arena;  // the others are parts of it
  DevBuf frags, items, slices, inv, eo2, ev2, part, queue;
  CUtensorMap tm;
  // paired-CTA kernel (one residual slice): its pair items and B-half map
  bool pair = false;
  long long npitems = 0;
  DevBuf pitems, dcorr;  // dcorr: per-column diagonal correction of the V product
  CUtensorMap tmB;
  int pair_nstage = 3;  // 3: exchange transpose in shared memory; 4: through xbuf
  DevBuf xbuf;          // 4-stage form: one 64 KB exchange tile per CTA
};

// Stage count of the paired kernel for a group.  The fourth 56 KB stage
// (which needs the exchange tile transposed through global scratch instead
// of shared memory) covers the cross-CTA refill round trip on long product
// chains, but measured on GB300 it gains nothing where it matters: the
// nocc=128 nvirt=1024 NBA=4096 fragment takes 5% fewer cycles at the same
// time (the power cap lowers the clock), and the 256-fragment batch runs 6%
// slower (569-572 against 605-608 eff TFLOP/s, same box: the slower
// global-memory transpose is exposed on short items).  So three stages;
// RIMP2_PAIR_STAGES=4 in the environment selects the four-stage form.
int pair_stages_for(const std::vector<FragDesc> &fh) {
  (void)fh;
  const char *e = getenv("RIMP2_PAIR_STAGES");
  if (e && e[0] == '4') return 4;
  return 3;
}

int launch_pair(const Group &g, PairParams Q, int npair, cudaStream_t s, bool overlap = false) {
  Q.xbuf = g.xbuf.as<float>();
  cudaError_t e;
  if (g.pair_nstage == 4)
    e = launch_ex(true, overlap, split_pair_kernel<4, true>, 2 * npair, NTHREADS,
                  pair_smem_bytes(4, true), s, g.tm, g.tmB, Q);
  else
    e = launch_ex(true, overlap, split_pair_kernel<3, false>, 2 * npair, NTHREADS,
                  pair_smem_bytes(3, false), s, g.tm, g.tmB, Q);
  if (e != cudaSuccess) {
    set_error("paired energy kernel launch failed: %s", cudaGetErrorString(e));
    return RIMP2_ERR_CUDA;
  }
  return RIMP2_OK;
}

int build_group(Group &g, cudaStream_t s, bool single = false) {
  // heaviest fragments first: their items lead the queue
  std::stable_sort(g.fh.begin(), g.fh.end(),
                   [](const FragDesc &x, const FragDesc &y) { return x.nks > y.nks; });
  long long row = 0, col = 0, item = 0, pitem = 0;
  int eo = 0, ev = 0, pb = 0;
  for (auto &F : g.fh) {
    F.nvpad = (F.nvirt + TILE - 1) / TILE * TILE;
    F.nks = (F.NBA + KSTEP - 1) / KSTEP;
    const int nt = F.nvpad / TILE;
    F.ntp = nt * (nt + 1) / 2;
    F.ncol = F.nocc * F.nvpad;
    F.eo_off = eo;
    F.ev_off = ev;
    F.pair_base = pb;
    F.row_base = row;
    F.col_base = col;
    F.item_base = item;
    F.pitem_base = pitem;
    pitem += pair_items_before(F.nocc) * F.ntp;
    const int np = F.nocc * (F.nocc + 1) / 2;
    eo += F.nocc;
    ev += F.nvpad;
    pb += np;
    row += (long long)F.nks * F.ncol;
    col += F.ncol;
    item += (long long)np * F.ntp;
    g.max_ncol = std::max(g.max_ncol, F.ncol);
    g.max_nocc = std::max(g.max_nocc, F.nocc);
    g.max_nv = std::max(g.max_nv, std::max(F.nvpad, F.nocc));
  }
  g.nfrag = (int)g.fh.size();
  g.nitems = item;
  g.npitems = pitem;
  g.R = row;
  g.ncol_total = col;
  g.npairs_total = pb;
  if (g.R > 2147483647LL - TILE || g.nitems > 2147483647LL) {
    set_error("split batch too large for one launch (rows=%lld, items=%lld)", g.R, g.nitems);
    return RIMP2_ERR_ARG;
  }
  if (g.pair && g.npitems > 2147483647LL) {
    set_error("split batch too large for one launch (pair items=%lld)", g.npitems);
    return RIMP2_ERR_ARG;
  }
  const int planes = g.nsl + (g.pair ? 1 : 0);  // the paired kernel adds the V plane
  // one allocation, divided (ten of them were a third of a small call's host time)
  {
    DevBuf *buf[] = {&g.slices, &g.frags, &g.items, &g.pitems, &g.inv, &g.dcorr,
                     &g.eo2,    &g.ev2,   &g.part,  &g.queue};
    const size_t bytes[] = {sizeof(__half) * (size_t)planes * (size_t)g.R * 64,
                            sizeof(FragDesc) * g.nfrag,
                            single && g.pair ? 16 : sizeof(int4) * (size_t)g.nitems,
                            g.pair ? sizeof(int4) * (size_t)g.npitems : 16,
                            sizeof(float) * (size_t)g.ncol_total,
                            g.pair ? sizeof(float) * (size_t)g.ncol_total : 16,
                            sizeof(float2) * (size_t)eo,
                            sizeof(float2) * (size_t)ev,
                            sizeof(double) * (size_t)g.nitems,
                            2 * sizeof(unsigned int)};
    RIMP2_TRY(alloc_parts(g.arena, buf, bytes, s));
  }
  if (!single) {
    RIMP2_CK(cudaMemcpyAsync(g.frags.p, g.fh.data(), sizeof(FragDesc) * g.nfrag,
                             cudaMemcpyHostToDevice, s));
    build_items_kernel<<<(unsigned)((g.nitems + 255) / 256), 256, 0, s>>>(
        g.frags.as<FragDesc>(), g.nfrag, g.nitems, g.items.as<int4>());
    count_launch(1);
    RIMP2_CK(cudaGetLastError());
  }
  auto encode = get_encode();
  if (!encode) {
    set_error("cuTensorMapEncodeTiled entry point unavailable");
    return RIMP2_ERR_UNSUPPORTED;
  }
  cuuint64_t dims[3] = {64, (cuuint64_t)g.R, (cuuint64_t)planes};
  cuuint64_t strides[2] = {128, (cuuint64_t)g.R * 128};
  cuuint32_t box[3] = {KSTEP, TILE, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult cr = encode(&g.tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, g.slices.p, dims, strides, box,
                       estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                       CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (cr != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed (%d)", (int)cr);
    return RIMP2_ERR_CUDA;
  }
  if (!g.pair) {
    auto k = g.nsl == 2 ? split_batch_kernel<2, 3> : split_batch_kernel<3, 2>;
    RIMP2_CK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  smem_bytes(g.nsl, g.nsl == 2 ? 3 : 2)));
  }
  if (g.pair) {
    g.pair_nstage = pair_stages_for(g.fh);
    if (g.pair_nstage == 4) {
      int dev = 0, nsm = 0;
      RIMP2_CK(cudaGetDevice(&dev));
      RIMP2_CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
      RIMP2_TRY(g.xbuf.alloc(sizeof(float) * TILE * TILE * (size_t)nsm, s));
      RIMP2_CK(cudaFuncSetAttribute(split_pair_kernel<4, true>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    pair_smem_bytes(4, true)));
    } else {
      RIMP2_CK(cudaFuncSetAttribute(split_pair_kernel<3, false>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    pair_smem_bytes(3, false)));
    }
    cuuint32_t boxB[3] = {KSTEP, BHALF, 1};
    cr = encode(&g.tmB, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, g.slices.p, dims, strides, boxB, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS) {
      set_error("cuTensorMapEncodeTiled failed (%d)", (int)cr);
      return RIMP2_ERR_CUDA;
    }
    if (single) return RIMP2_OK;
    build_pair_items_kernel<<<(unsigned)((g.npitems + 255) / 256), 256, 0, s>>>(
        g.frags.as<FragDesc>(), g.nfrag, g.npitems, g.pitems.as<int4>());
    count_launch(1);
    RIMP2_CK(cudaGetLastError());
  }
  return RIMP2_OK;
}

// The group's inputs for its energy kernel: slices, scales, corrections and
// orbital-energy pairs (graph-capturable: no sync, no alloc).
int record_group_inputs(Group &g, cudaStream_t s) {
  if (g.nfrag == 0) return RIMP2_OK;
  const FragDesc *fr = g.frags.as<FragDesc>();
  dim3 grid((unsigned)((g.max_ncol * 32LL + 255) / 256), (unsigned)g.nfrag);
  slice_batch_kernel<<<grid, 256, 0, s>>>(fr, g.nsl, g.R * 64, g.slices.as<__half>(),
                                          g.inv.as<float>(), 0, 0x7fffffff, g.pair ? 1 : 0,
                                          g.dcorr.as<float>());
  dim3 g2((unsigned)((g.max_nv + 255) / 256), (unsigned)g.nfrag);
  eps_batch_kernel<<<g2, 256, 0, s>>>(fr, g.eo2.as<float2>(), g.ev2.as<float2>());
  count_launch(2);
  RIMP2_CK(cudaGetLastError());
  return RIMP2_OK;
}

// Enqueue one evaluation of the group on s (graph-capturable: no sync, no
// alloc); with_inputs = false when its inputs were enqueued elsewhere.
// single: a group of one fragment whose inputs and reductions take one launch each
int record_group(Group &g, cudaStream_t s, int nsm, cudaEvent_t *ev /* 3 or null */,
                 bool with_inputs = true, bool single = false) {
  if (g.nfrag == 0) return RIMP2_OK;
  const FragDesc *fr = g.frags.as<FragDesc>();
  if (ev) RIMP2_CK(cudaEventRecord(ev[0], s));
  SingleArgs A;
  // the kernels of one fragment are set up at the end of the one before (not in a
  // graph under capture, nor between timing events): 27 -> 23 us a call at nocc = 8,
  // nvirt = 96, NBA = 256, 271 -> 266 at 24/301/1203.  The inputs' blocks say so when
  // they are done; with the energy kernel saying so at its start, the waiting
  // reduction cost 6 to 16 us.
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  const bool overlap = single && !ev && cudaStreamIsCapturing(s, &cap) == cudaSuccess &&
                       cap == cudaStreamCaptureStatusNone;
  if (single) {
    A.F = g.fh[0];
    A.frag = g.frags.as<FragDesc>();
    A.slice_blocks = (int)((g.max_ncol * 32LL + 255) / 256);
    A.nsl = g.nsl;
    A.vplane = g.pair ? 1 : 0;
    A.nitems = g.pair ? 0 : (int)g.nitems;
    A.npitems = g.pair ? (int)g.npitems : 0;
    A.plane = g.R * 64;
    A.light_last = g.R * 128 * (g.nsl + A.vplane) <= 110000000LL;
    A.slices = g.slices.as<__half>();
    A.inv = g.inv.as<float>();
    A.dcorr = g.dcorr.as<float>();
    A.eo2 = g.eo2.as<float2>();
    A.ev2 = g.ev2.as<float2>();
    A.items = g.items.as<int4>();
    A.pitems = g.pitems.as<int4>();
    A.queue = g.queue.as<unsigned>();
    A.part = g.part.as<double>();
    const int rest = std::max(std::max(A.nitems, A.npitems), g.max_nv);
    single_inputs_kernel<<<(unsigned)(A.slice_blocks + (rest + 255) / 256), 256, 0, s>>>(A);
    count_launch(1);
    RIMP2_CK(cudaGetLastError());
  } else {
    if (with_inputs) RIMP2_TRY(record_group_inputs(g, s));
    RIMP2_CK(cudaMemsetAsync(g.queue.p, 0, sizeof(unsigned int), s));
  }
  BatchParams P;
  P.frags = fr;
  P.items = g.items.as<int4>();
  P.nitems = g.nitems;
  P.item_begin = 0;
  P.queue = g.queue.as<unsigned int>();
  P.eo2 = g.eo2.as<float2>();
  P.ev2 = g.ev2.as<float2>();
  P.inv_scale = g.inv.as<float>();
  P.part = g.part.as<double>();
  P.err = device_error_word();
  const int grid = (int)std::min<long long>(g.nitems, nsm);
  if (inject_fault("launch")) {
    set_error("injected launch failure (RIMP2_FAULT_INJECT=launch)");
    return RIMP2_ERR_CUDA;
  }
  if (ev) RIMP2_CK(cudaEventRecord(ev[1], s));
  if (g.pair) {
    PairParams Q;
    Q.frags = fr;
    Q.items = g.pitems.as<int4>();
    Q.nitems = g.npitems;
    Q.item_begin = 0;
    Q.dcorr = g.dcorr.as<float>();
    Q.queue = P.queue;
    Q.eo2 = P.eo2;
    Q.ev2 = P.ev2;
    Q.inv_scale = P.inv_scale;
    Q.part = P.part;
    Q.err = P.err;
    const int npair = (int)std::min<long long>(g.npitems, std::max(1, nsm / 2));
    RIMP2_TRY(launch_pair(g, Q, npair, s, overlap));
    note_split_kernel(2);
  } else if (g.nsl == 2) {
    note_split_kernel(1);
    RIMP2_CK(launch_ex(true, overlap, split_batch_kernel<2, 3>, grid, BATCH_THREADS, smem_bytes(2, 3), s,
                       g.tm, P));
  } else {
    note_split_kernel(1);
    RIMP2_CK(launch_ex(true, overlap, split_batch_kernel<3, 2>, grid, BATCH_THREADS, smem_bytes(3, 2), s,
                       g.tm, P));
  }
  count_launch(1);
  if (ev) RIMP2_CK(cudaEventRecord(ev[2], s));
  if (single) {
    RIMP2_CK(launch_ex(false, overlap, single_reduce_kernel, (unsigned)((g.npairs_total + 7) / 8), 256, 0, s, A));
    count_launch(1);
    return RIMP2_OK;
  }
  pair_reduce_batch_kernel<<<(unsigned)((g.npairs_total + 7) / 8), 256, 0, s>>>(
      fr, g.nfrag, g.npairs_total, g.part.as<double>());
  total_reduce_batch_kernel<<<g.nfrag, total_threads(g.max_nocc), 0, s>>>(fr);
  count_launch(2);
  RIMP2_CK(cudaGetLastError());
  return RIMP2_OK;
}

// ==========================================================================
// General split-precision GEMM on the same slices (used by the AO->MO
// transform): D[m][n] = sum_k A[m][k] B[n][k], A and B K-major FP16 slices
// with per-row power-of-two scales, exact integer L0 + residual L1 in TMEM,
// FP64 output (L0 and L1 combined in FP64) with arbitrary strides.
// Persistent: each CTA takes output tiles (128 x NT, NT <= 128) blockIdx.x,
// + gridDim.x, ... (all tiles have the same K), with two TMEM accumulator
// sets, so that the epilogue of one tile (TMEM -> FP64 stores) runs while
// the tensor core works on the next and the copy ring never drains between
// tiles.  Per K16 step one MMA over the stacked B planes [S0b; R1b] (N = 2 NT)
// gives L0 and S0a R1b, then R1a S0b, R1a R1b (and S0a R2b, R2a S0b with two
// residual slices) accumulate into L1.
// Roles: warp 0 TMA producer, warp 1 MMA issuer and TMEM owner, warps 2-9
// epilogue (two per TMEM lane quadrant, alternate 16-column chunks).  Every
// wait is bounded.
// ==========================================================================
struct GemmSP {
  int M, N, NT, nks, mtiles, ntiles, nbatch;
  long long a_ncol, b_ncol;        // rows per K chunk in each operand's slice layout
  long long a_row0, a_bstride;     // first row of batch 0 and row stride between batches
  long long b_row0, b_bstride;
  const float *a_inv, *b_inv;      // per-row inverse scales (indexed like the rows)
  double *out;
  long long sOm, sOn, sOb;
  uint32_t tmem_cols;              // TMEM columns allocated (a power of two >= 4 NT)
  int *err;
};

constexpr int GEMM_NST = 2;

constexpr int gemm_stage_bytes(int nsl, int NT) { return nsl * (PANEL_BYTES + NT * 128); }
constexpr int gemm_smem_bytes(int nsl, int NT) {
  return GEMM_NST * gemm_stage_bytes(nsl, NT) + 1024 + 256;
}
static_assert(gemm_smem_bytes(2, 16) >= TMEM_SMEM_MIN, "tensor memory");

constexpr int GEMM_EPI = 8;                       // epilogue warps: two per lane quadrant
constexpr int GEMM_THREADS = 64 + 32 * GEMM_EPI;

template <int NSL>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
    split_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                      GemmSP P) {
  constexpr int NST = GEMM_NST;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *base = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int NT = P.NT;
  const int BPL = NT * 128;  // bytes of one B plane (NT rows of 64 FP16)
  const int STAGE = NSL * (PANEL_BYTES + BPL);
  // bars: full[2], empty[2], tfull[2], tempty[2], drain
  uint64_t *bars = (uint64_t *)(base + NST * STAGE);
  uint32_t *tmem_slot = (uint32_t *)(bars + 2 * NST + 5);
  volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[NST]);
  const uint32_t tfull0 = smem_u32(&bars[2 * NST]), tempty0 = smem_u32(&bars[2 * NST + 2]);
  const uint32_t drain = smem_u32(&bars[2 * NST + 4]);
  const long long per_b = (long long)P.mtiles * P.ntiles;
  const long long nitems = per_b * P.nbatch;
  if (threadIdx.x == 0) {
    for (int st = 0; st < NST; ++st) {
      mbar_init(full0 + 8 * st, 1);
      mbar_init(empty0 + 8 * st, 1);
    }
    for (int u = 0; u < 2; ++u) {
      mbar_init(tfull0 + 8 * u, 1);
      mbar_init(tempty0 + 8 * u, GEMM_EPI);  // the epilogue warps
    }
    mbar_init(drain, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&tmA) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&tmB) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(P.tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  auto tile_rows = [&](long long item, long long &arow, long long &brow, int &b, int &mt, int &nt) {
    b = (int)(item / per_b);
    const long long rem = item % per_b;
    mt = (int)(rem / P.ntiles);
    nt = (int)(rem % P.ntiles);
    arow = P.a_row0 + (long long)b * P.a_bstride + (long long)mt * TILE;
    brow = P.b_row0 + (long long)b * P.b_bstride + (long long)nt * NT;
  };
  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      int armed[NST] = {-1, -1};
      bool ok = true;
      const uint32_t tx = (uint32_t)STAGE;
      for (long long item = blockIdx.x; item < nitems && ok; item += gridDim.x) {
        long long arow, brow;
        int b, mt, nt;
        tile_rows(item, arow, brow, b, mt, nt);
        for (int kc = 0; kc < P.nks; ++kc) {
          if (!mbar_wait(empty0 + 8 * stage, phase ^ 1, abort_flag, P.err, 11)) {
            ok = false;
            break;
          }
          const uint32_t fb = full0 + 8 * stage;
          mbar_expect_tx(fb, tx);
          armed[stage] = (int)phase;
          const uint32_t dst = smem_u32(base + stage * STAGE);
#pragma unroll
          for (int sl = 0; sl < NSL; ++sl) {  // A planes, then the B planes back to back
            tma_load_3d(dst + sl * PANEL_BYTES, &tmA, fb, 0, (int)(kc * P.a_ncol + arow), sl);
            tma_load_3d(dst + NSL * PANEL_BYTES + sl * BPL, &tmB, fb, 0,
                        (int)(kc * P.b_ncol + brow), sl);
          }
          if (++stage == NST) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      if (!ok || *abort_flag) {  // copies in flight land before the CTA can exit
        for (int st = 0; st < NST; ++st) {
          if (armed[st] < 0) continue;
          const long long t0 = clock64();
          while (!mbar_test(full0 + 8 * st, (uint32_t)armed[st]) && clock64() - t0 < WAIT_BUDGET) {
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer --------------------------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      const uint32_t id2 = idesc_mn(TILE, 2 * NT), id1 = idesc_mn(TILE, NT);
      long long t = 0;  // tiles of this CTA so far
      for (long long item = blockIdx.x; item < nitems && ok; item += gridDim.x, ++t) {
        const int u = (int)(t & 1);
        // the epilogue has read this accumulator set's previous tile
        if (t >= 2 &&
            !mbar_wait(tempty0 + 8 * u, (uint32_t)(((t >> 1) - 1) & 1), abort_flag, P.err, 14)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t dL0 = tmem + (uint32_t)(u * 2 * NT), dL1 = dL0 + (uint32_t)NT;
        for (int kc = 0; kc < P.nks; ++kc) {
          if (!mbar_wait(full0 + 8 * stage, phase, abort_flag, P.err, 12)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(base + stage * STAGE);
          const uint32_t sb = sa + NSL * PANEL_BYTES;
#pragma unroll
          for (int k16 = 0; k16 < KSTEP / 16; ++k16) {
            const uint32_t koff = k16 * 32;
            const uint64_t a0 = smem_desc(sa + koff), a1 = smem_desc(sa + PANEL_BYTES + koff);
            const uint64_t b0 = smem_desc(sb + koff), b1 = smem_desc(sb + BPL + koff);
            const uint32_t acc = (kc > 0 || k16 > 0) ? 1u : 0u;
            mma_f16_id(dL0, a0, b0, id2, acc);  // [L0 | L1] = S0a [S0b; R1b]
            mma_f16_id(dL1, a1, b0, id1, 1u);   // R1a S0b
            mma_f16_id(dL1, a1, b1, id1, 1u);   // R1a R1b
            if (NSL > 2) {
              const uint64_t a2 = smem_desc(sa + 2 * PANEL_BYTES + koff);
              const uint64_t b2 = smem_desc(sb + 2 * BPL + koff);
              mma_f16_id(dL1, a0, b2, id1, 1u);  // S0a R2b
              mma_f16_id(dL1, a2, b0, id1, 1u);  // R2a S0b
            }
          }
          mma_commit(empty0 + 8 * stage);
          if (++stage == NST) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        mma_commit(tfull0 + 8 * u);
      }
      mma_commit(drain);
      const long long t0 = clock64();
      while (!mbar_test(drain, 0) && clock64() - t0 < WAIT_BUDGET) {
      }
    }
  } else {
    // ------------------------------ epilogue ----------------------------------
    const int quad = warp & 3;
    const int half = (warp - 2) >> 2;  // 16-column chunks half, half + 2, ...
    const int row = quad * 32 + lane;
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
    long long t = 0;
    for (long long item = blockIdx.x; item < nitems; item += gridDim.x, ++t) {
      const int u = (int)(t & 1);
      if (!mbar_wait(tfull0 + 8 * u, (uint32_t)((t >> 1) & 1), abort_flag, P.err, 13)) break;
      tc_fence_after();
      long long arow, brow;
      int b, mt, nt;
      tile_rows(item, arow, brow, b, mt, nt);
      const long long m = (long long)mt * TILE + row;
      const float sa = P.a_inv[arow + row];  // 2^-e of this row
      const uint32_t taddr = tmem + lane_off + (uint32_t)(u * 2 * NT);
      double *orow = P.out + (long long)b * P.sOb + m * P.sOm;
      for (int c0 = 16 * half; c0 < NT; c0 += 32) {
        float l0[16], l1[16];
        tmem_ld16(taddr + c0, l0);
        tmem_ld16(taddr + NT + c0, l1);
        tmem_wait_ld();
        if (m < P.M) {
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            const int n = nt * NT + c0 + k;
            if (n < P.N) {
              // (L0 + L1) sa sb with one FP64 operation: L0 (an integer
              // below 2^24) and L1 times the row's power of two are exact
              // floats (|L1 sa| below 2^-126, far under the output's
              // resolution, flushes), their sum rounds once in FP64 as
              // (L0 + L1) does, and the column's power of two moves the
              // exponent.  The FP64 pipe, not the tensor core, bounded this
              // epilogue with FP64 conversions and products per element.
              const double v = f2d_bits(l0[k] * sa) + f2d_bits(l1[k] * sa);
              orow[(long long)n * P.sOn] = scale_pow2(v, P.b_inv[brow + c0 + k]);
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty0 + 8 * u);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(P.tmem_cols)
                 : "memory");
  }
}

// ==========================================================================
// Fused first half of the AO->MO transform on the tensor cores, one pass over
// the FP64 AO tensor:  H[i][alpha][mu] = sum_nu (alpha|mu nu) Cmo(nu, i),
// evaluated as sum_nu (alpha|nu mu) Cmo(nu, i): the three-centre integrals
// are symmetric in their two AO indices, and the middle one is the short
// stride (8 NBA bytes), so every 64-value chunk of a row lies in one memory
// page (the last index is 8 NBA nbas bytes apart: a chunk would touch 64).
// GEMM rows are (alpha, mu) -- 16 alpha x 8 mu per CTA tile, row r = a + 16 m
// -- K = nu in chunks of 64, N = the occupied orbitals (NT <= 80, padded to
// a multiple of 16).  The AO tensor is read once, in 64-nu chunks of the 32 rows
// (16 alpha x 2 mu) of a row group by TMA (rows that do not start on 16-byte
// boundaries in four boxes by parity: 1.35 ms at nbas = 509 of the transform,
// 1.35 at 510, where per-thread 8-byte copies took 1.94 against 1.65) and sliced
// by the converter warps (split_chunk) with a power-of-two scale per (row, K chunk):
// |x 2^e| <= 511.5, so S0 is a 10-bit integer, and with the occupied MO
// block sliced the same way (per column and chunk, precomputed) every
// partial sum of S0a S0b over a chunk is below 64 * 511^2 < 2^24: the integer
// part of each chunk's product is exact in FP32.  Products per element pair:
// S0 S0 (L0), S0 R1 + R1 S0 + R1 R1 + S0 R2 + R2 S0 (L1).  Each chunk's L0/L1
// go to one of two TMEM buffers; the fold scales them by the row and column
// scales of that chunk (powers of two: exact) and adds them into a double-float
// (FP32 hi + lo, two-sum) running total in registers, so the result carries
// ~2^-40 of the chunk products' magnitude.  A tile's last fold writes the totals
// as FP64 (bits moved, one FP64 add: the FP64 pipe is slow on GB300).
// Roles: warps 0-15 converters, warp 16 MMA issuer and TMEM owner.  As slicer a
// converter warp takes a K quarter of one row group, 16 values a thread; the
// four warps of a group, which exchange the chunk's maxima, sit on the four
// schedulers, so that each scheduler holds one warp of every group and a group's
// waits are filled by the others.  In the folds a warp is bound to the TMEM
// lanes of its quadrant and takes a quarter of the NT columns: in iteration n it
// slices chunk n and then folds chunk n - 1 while the tensor core runs chunk n.
// A CTA per SM walks over its tiles without a break between them (the first
// chunk of a tile is on its way while the last one of the tile before is
// folded).  Bound by the converter warps (issue 54% active; 52 instructions a
// value): 1.05 ms of the 1.32 at nbas = 509 (3.0 TB/s; the tensor's bytes alone
// take 0.48).  Steps at that size, transform: 1.91 ms; totals in registers, boxes
// by parity and groups across schedulers 1.53; fewer operations to split a value,
// one arrival a warp 1.46; one CTA per SM over its tiles 1.34; column scales
// loaded before the wait 1.32.  Prefetching the boxes of a further chunk into L2:
// 1.43.  Every wait is bounded; on expiry the CTA records an error code, drains
// its copies and MMAs and returns.
// --------------------------------------------------------------------------
constexpr int AH_TA = 16, AH_TM = 8;  // alpha x mu rows of a tile (16 x 8 = 128)
constexpr int AH_CONV = 16;
constexpr int AH_THREADS = 32 * (AH_CONV + 1);
constexpr int AH_NT_MAX = 80;

// How an AO chunk reaches shared memory.
enum : int {
  AH_COPY,  // per-thread 8-byte copies
  AH_BOX,   // a TMA box of 16 alpha x 64 k x 2 mu per row group
  AH_BOX4   // four boxes of 18 alpha x 32 k, one per parity of k and mu
};
struct AoMaps {
  CUtensorMap m[4];
};

struct AoHalfParams {
  const double *ao;   // (alpha|mu nu), alpha fastest: ao[alpha + NBA (mu + nbas nu)]
  int NBA, nbas, nocc, nks;
  int ta_tiles, tiles;  // alpha tiles (of 16), tiles
  unsigned shift;     // AH_BOX4: bit 2 (parity of k) + (parity of mu): its box starts 8 bytes early
  const float *sb;    // [chunk][NT] column scales of the sliced occupied MO block
  double *half;       // H[i][alpha][mu]
  uint32_t idesc;
  int *err;
};

constexpr int ah_b_plane(int NT) { return NT * 128; }  // bytes of one B plane (NT rows x 64 FP16)
constexpr int ah_stage_bytes(int NT) { return 3 * PANEL_BYTES + 3 * ah_b_plane(NT); }
// one FP64 chunk of the tile: 64 k of 128 rows, in runs of 16 alpha (18 in the
// form of four boxes)
constexpr int ah_slot_bytes(int form) { return KSTEP * AH_TM * (form == AH_BOX4 ? 18 : 16) * 8; }
constexpr int ah_smem_bytes(int form, int NT) {
  return 1024 + 2 * ah_stage_bytes(NT) + ah_slot_bytes(form) + 2 * 4 * 128 * 4 /*row max exchange*/ +
         4 * 128 /*row exponents*/ + 256 /*barriers, slot*/;
}
static_assert(ah_smem_bytes(AH_BOX, 16) >= TMEM_SMEM_MIN, "tensor memory");

// 8-byte asynchronous global -> shared copy; src_bytes = 0 fills zeros and
// reads nothing
__device__ __forceinline__ void cp_async8_zfill(uint32_t dst, const void *src, uint32_t src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(src_bytes)
               : "memory");
}

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, float *v) {
  uint32_t r[4];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
#pragma unroll
  for (int k = 0; k < 4; ++k) v[k] = __uint_as_float(r[k]);
}

// Fold of this thread's NC columns of one AO chunk's products into the running
// double-float totals: L0 and L1 scaled by the row and column powers of two
// (exact), added to hi/lo with a two-sum of the high parts (first chunk:
// assigned).
template <int NC>
__device__ __forceinline__ void ah_fold(uint32_t tL0, uint32_t tL1, float sa,
                                        const float4 (&sb)[NC / 4], bool first, float (&hi)[NC], float (&lo)[NC]) {
  constexpr int G = NC <= 16 ? NC : 8;  // columns read at a time (96 registers a thread)
#pragma unroll
  for (int g = 0; g < NC; g += G) {
    float l0[G], l1[G];
#pragma unroll
    for (int q = 0; q < G && g + q < NC; q += 4) {
      tmem_ld4(tL0 + g + q, l0 + q);
      tmem_ld4(tL1 + g + q, l1 + q);
    }
    tmem_wait_ld();
#pragma unroll
    for (int q = 0; q < G && g + q < NC; q += 4) {
      const float4 sb4 = sb[(g + q) / 4];
      const float sbk[4] = {sb4.x, sb4.y, sb4.z, sb4.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float sc = sa * sbk[k];  // power of two: the products below are exact
        const float xh = l0[q + k] * sc, xl = l1[q + k] * sc;
        float &h = hi[g + q + k], &l = lo[g + q + k];
        if (first) {
          h = xh;
          l = xl;
        } else {  // two-sum of the high parts, low parts added
          const float t = h + xh;
          const float bv = t - h;
          const float err = (h - (t - bv)) + (xh - bv);
          l = l + xl + err;
          h = t;
        }
      }
    }
  }
}

// Exponent e with |x| 2^e <= 511.5 (to within 2^-11) for the largest
// magnitude of a row or column chunk, from key = the top 32 bits of its FP64
// pattern (11 exponent, 20 fraction bits): mx = m 2^E with m in [1, 2), and
// m <= 1.998046875 (fraction key <= 0xFFE00) allows e = 8 - E.  A value that
// shares the key but has nonzero lower bits gives |x| 2^e < 511.5003, which
// rounds to |q| <= 512: still exact in FP16, and 64 products of two such
// integers stay <= 2^24, exact in FP32.  At most 126, so that 2^-e is a
// normal float; at least -126 (|x| < 2^134); 0 for a chunk of zeros and
// subnormals.
__device__ __forceinline__ int chunk_exponent_511(uint32_t key) {
  const int ed = (int)(key >> 20);
  if (ed == 0) return 0;
  const int E = ed - 1023;
  const int e = ((key & 0xFFFFFu) <= 0xFFE00u ? 8 : 7) - E;
  return max(-126, min(126, e));
}

// split_f32 for the values of a row chunk with exponent e, in fewer
// operations: shift = (e - 896) << 23 moves the exponent field along with the
// fraction bits (its value is at most 254: no carry into the sign), and least =
// (963 - e) << 20 holds |x| 2^e at 2^-60 or above, so that no case needs a
// select: below 2^-40, zeros and subnormals leave q = 0 and an r whose FP16
// parts are zero.  q and r are split_f32's otherwise.
__device__ __forceinline__ void split_chunk(double x, uint32_t least, uint32_t shift, float &q,
                                            float &r) {
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
  const uint32_t h = max(hi & 0x7FFFFFFFu, least);
  const uint32_t f = (__funnelshift_l(lo, h, 3) + shift) | (hi & 0x80000000u);
  const float v = __uint_as_float(f);                // x 2^e to 24 bits
  const float p = __uint_as_float(f & 0xFF800000u);  // its sign and power of two
  const float l = fmaf(__uint_as_float(0x4B000000u | ((lo >> 6) & 0x7FFFFFu)), 0x1p-46f, -0x1p-23f);
  q = (v + 12582912.0f) - 12582912.0f;
  r = fmaf(l, p, v - q);
}

// Bounded vote over the 128 converter threads of row group g (the four warps
// that hold the same tile rows; named barrier 3 + g).
__device__ __forceinline__ bool group_any(bool p, int g) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred q, o;\n\t"
      "setp.ne.u32 q, %1, 0;\n\t"
      "bar.red.or.pred o, %2, 128, q;\n\t"
      "selp.u32 %0, 1, 0, o;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)p), "r"(3 + g)
      : "memory");
  return r != 0;
}

// 17 warps: one scheduler holds five, whose registers allow 96 a thread.
template <int FORM, int NT>
__global__ void __maxnreg__(96)
    ao_half_kernel(const __grid_constant__ CUtensorMap tmB, const __grid_constant__ AoMaps tmAO,
                   AoHalfParams P) {
  constexpr int NC = NT / 4;  // columns of a converter thread's totals
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *base = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  constexpr int BPL = ah_b_plane(NT);
  constexpr int STAGE = 3 * PANEL_BYTES + 3 * BPL;
  uint8_t *stages = base;
  double *slot = (double *)(base + 2 * STAGE);  // the chunk's FP64 values
  uint32_t *smx = (uint32_t *)(base + 2 * STAGE + ah_slot_bytes(FORM));  // [2 parity][4 quarter][128]
  // [4][128]: a group may be two chunks ahead of another warp's fold, not four
  // (it waits for the MMAs of two chunks before, which waited for every warp)
  signed char *sexp = (signed char *)(smx + 2 * 4 * 128);
  uint64_t *bars = (uint64_t *)(sexp + 4 * 128);
  // bars: stage_full[2], stage_empty[2], acc_full[2], acc_empty[2], drain,
  //       ao_full[4] (the AO chunk of each row group, box forms)
  uint32_t *tmem_slot = (uint32_t *)(bars + 13);
  volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
  const uint32_t sfull0 = smem_u32(&bars[0]), sempty0 = smem_u32(&bars[2]);
  const uint32_t afull0 = smem_u32(&bars[4]), aempty0 = smem_u32(&bars[6]);
  const uint32_t drain = smem_u32(&bars[8]);
  const uint32_t aofull0 = smem_u32(&bars[9]);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // this CTA's tiles: blockIdx.x and every gridDim.x-th after it; its chunks in
  // one sequence n = 0 ... total - 1
  const int nks = P.nks;
  const int total = (P.tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x * nks;

  if (threadIdx.x == 0) {
    for (int b = 0; b < 2; ++b) {
      mbar_init(sfull0 + 8 * b, AH_CONV);       // converter warps (one with the B bytes)
      mbar_init(sempty0 + 8 * b, 1);            // MMA commit
      mbar_init(afull0 + 8 * b, 1);             // MMA commit
      mbar_init(aempty0 + 8 * b, AH_CONV);      // converter warps, after reading the chunk
    }
    mbar_init(drain, 1);
    for (int g = 0; g < 4; ++g) mbar_init(aofull0 + 8 * g, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&tmB) : "memory");
    if (FORM != AH_COPY)
      asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&tmAO.m[0]) : "memory");
  }
  if (warp == AH_CONV) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                     smem_u32(tmem_slot))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp < AH_CONV) {
    // --------------------------- slicers and folds ----------------------------
    // as a slicer: tile row r of row group rg, K quarter kq of each chunk
    const int rg = warp >> 2, kq = warp & 3;
    const int r = 32 * rg + lane;
    const int a_l = r % AH_TA, m_l = r / AH_TA;
    // in the folds: tile row (TMEM lane) re, columns col0 .. col0 + NC
    const int re = 32 * (warp & 3) + lane, col0 = (warp >> 2) * NC;
    const uint32_t te = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)col0;
    // row (alpha, mu) contracted over the middle index: (alpha|nu mu) =
    // (alpha|mu nu), and the middle index is 8 NBA bytes apart, so a chunk of
    // 64 values stays inside one memory page (the last index: 64 pages)
    const int within = r & 7;
    int armed = -1;  // thread 0: parity of the last stage it armed for the B copy
    int armed_b = 0;
    // this thread's 16 values of a chunk, k = 16 kq + j, in the FP64 slot: even j
    // at even + (j / 2) pitch, odd j at odd + (j / 2) pitch
    constexpr int pitch = FORM == AH_COPY ? 256 : FORM == AH_BOX ? 32 : 18;
    const double *even, *odd;
    if constexpr (FORM == AH_COPY) {  // [k][row]
      even = slot + (16 * kq) * 128 + r;
      odd = even + 128;
    } else if constexpr (FORM == AH_BOX) {  // [group][mu][k][alpha]
      even = slot + rg * 2048 + ((m_l & 1) * 64 + 16 * kq) * 16 + a_l;
      odd = even + 16;
    } else {  // [group][parity of k][parity of mu][k / 2][alpha + shift]
      const int mp = m_l & 1;
      even = slot + rg * 2304 + mp * 576 + 8 * kq * 18 + a_l + (P.shift >> mp & 1);
      odd = slot + rg * 2304 + (2 + mp) * 576 + 8 * kq * 18 + a_l + (P.shift >> (2 + mp) & 1);
    }
    const uint32_t aofull = aofull0 + 8 * rg;
    // box forms: lane 0 of the group's K-quarter-0 warp issues the group's boxes
    const bool ao_issuer = FORM != AH_COPY && kq == 0 && lane == 0;
    int ao_pending = -1;  // parity of a chunk in flight (issuer)
    auto issue_box = [&](int n, int tile, int c) {
      const int alpha0 = tile % P.ta_tiles * AH_TA, mu0 = tile / P.ta_tiles * AH_TM;
      if constexpr (FORM == AH_BOX) {
        mbar_expect_tx(aofull, AH_TA * KSTEP * 2 * 8);
        tma_load_3d(smem_u32(slot + rg * 2048), &tmAO.m[0], aofull, alpha0, c * KSTEP, mu0 + 2 * rg);
      } else {
        mbar_expect_tx(aofull, 4 * 576 * 8);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          tma_load_3d(smem_u32(slot + rg * 2304 + q * 576), &tmAO.m[q], aofull, alpha0,
                      c * (KSTEP / 2), mu0 / 2 + rg);
      }
      ao_pending = n & 1;
    };
    // L2 prefetch of a later chunk: thread t covers the 16-alpha run (128
    // bytes, at most two lines) of k = t / 8 and mu = mu0 + t % 8, so that
    // the chunk's cp.async copies find their data in L2; with one chunk in
    // flight per CTA the copies would otherwise wait out the slowest DRAM
    // access of each chunk
    auto prefetch_chunk = [&](int tile, int c) {
      const int alpha0 = tile % P.ta_tiles * AH_TA;
      const int k = c * KSTEP + (threadIdx.x >> 3);
      const int mu = tile / P.ta_tiles * AH_TM + (threadIdx.x & 7);
      if (k < P.nbas && mu < P.nbas) {
        const double *p = P.ao + alpha0 + (long long)P.NBA * k + (long long)P.NBA * P.nbas * mu;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(p + (min(AH_TA, P.NBA - alpha0) - 1)));
      }
    };
    const uint32_t myslot_s = smem_u32(even);
    auto issue_chunk = [&](int tile, int c) {
      const int alpha = tile % P.ta_tiles * AH_TA + a_l, mu = tile / P.ta_tiles * AH_TM + m_l;
      const bool live = alpha < P.NBA && mu < P.nbas;
      const int k0 = c * KSTEP + 16 * kq;
      const int lim = live ? min(16, P.nbas - k0) : 0;  // values that exist
      const double *p =
          P.ao + (live ? alpha + (long long)P.NBA * P.nbas * mu : 0) + (long long)P.NBA * k0;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        cp_async8_zfill(myslot_s + j * 128 * 8, j < lim ? (const void *)p : (const void *)P.ao,
                        j < lim ? 8u : 0u);
        p += P.NBA;
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // fold of the n-th chunk (chunk c of the tile) into this thread's totals; the
    // tile's last one writes them: 16-byte runs of two mu, which the four groups'
    // stores complete to 64 bytes in L2 (one FP64 add per output, bit-moved
    // conversions)
    float hi[NC], lo[NC];
    auto fold = [&](int n, int tile, int c) -> bool {
      const int b = n & 1;
      float4 sb[NC / 4];  // 16-byte loads, before the wait: offsets are multiples of 4
#pragma unroll
      for (int q = 0; q < NC / 4; ++q)
        sb[q] = __ldg(reinterpret_cast<const float4 *>(P.sb + (size_t)c * NT + col0) + q);
      if (!mbar_wait(afull0 + 8 * b, (uint32_t)((n >> 1) & 1), abort_flag, P.err, 25)) return false;
      tc_fence_after();
      const uint32_t tL0 = te + (uint32_t)(b * 2 * NT);
      const float sa = __int_as_float((127 - sexp[(n & 3) * 128 + re]) << 23);  // 2^-e
      ah_fold<NC>(tL0, tL0 + NT, sa, sb, c == 0, hi, lo);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(aempty0 + 8 * b);
      if (c + 1 == nks) {
        const int alpha = tile % P.ta_tiles * AH_TA + re % AH_TA;
        const int mu = tile / P.ta_tiles * AH_TM + re / AH_TA;
        if (alpha < P.NBA && mu < P.nbas) {
          double *o = P.half + ((long long)col0 * P.NBA + alpha) * P.nbas + mu;
#pragma unroll
          for (int k = 0; k < NC; ++k) {
            if (col0 + k < P.nocc) *o = f2d_bits(hi[k]) + f2d_bits(lo[k]);
            o += (long long)P.NBA * P.nbas;
          }
        }
      }
      return true;
    };
    bool ok_all = true, folded = true;
    int tile = blockIdx.x, c = 0;
    auto advance = [&](int &t, int &k) {
      if (++k == nks) {
        k = 0;
        t += gridDim.x;
      }
    };
    if (FORM != AH_COPY) {
      if (ao_issuer) issue_box(0, tile, 0);
    } else {
      issue_chunk(tile, 0);
    }
    int tp = tile, cp = 0;  // the chunk before
    for (int n = 0; n < total; ++n) {
      const int b = n & 1;
      int tn = tile, cn = c;  // the chunk after
      advance(tn, cn);
      bool landed = true;
      if (FORM != AH_COPY) {
        landed = mbar_wait(aofull, (uint32_t)(n & 1), abort_flag, P.err, 26);
        if (ao_issuer && landed) ao_pending = -1;
      } else {
        if (n + 1 < total) prefetch_chunk(tn, cn);
        // chunk n has landed (each thread reads only the values it copied)
        asm volatile("cp.async.wait_group 0;" ::: "memory");
      }
      double v[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = (j & 1 ? odd : even)[(j >> 1) * pitch];
      uint32_t key = 0;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const uint32_t kj = (uint32_t)(((unsigned long long)__double_as_longlong(v[j]) >> 32) &
                                       0x7FFFFFFFu);
        key = kj > key ? kj : key;
      }
      smx[(b * 4 + kq) * 128 + r] = key;
      bool ok = landed && folded;
      if (ok && n >= 2)
        ok = mbar_wait(sempty0 + 8 * b, (uint32_t)(((n - 2) >> 1) & 1), abort_flag, P.err, 21);
      // the four warps of a row group exchange their K quarters' maxima; the
      // groups do not wait for one another, and the four warps of a scheduler
      // belong to four groups, so that their latency-bound phases (loads,
      // slicing, TMEM round trips) interleave on it
      if (group_any(!ok, rg)) {
        ok_all = false;
        break;
      }
      // every warp of the group has its values: the group's box is free
      if (ao_issuer && n + 1 < total) issue_box(n + 1, tn, cn);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t o = smx[(b * 4 + q) * 128 + r];
        key = o > key ? o : key;
      }
      const int e = chunk_exponent_511(key);
      if (kq == 0) sexp[(n & 3) * 128 + r] = (signed char)e;
      const uint32_t least = (uint32_t)(963 - e) << 20, shift = (uint32_t)(e - 896) << 23;
      uint8_t *st = stages + b * STAGE;
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        __align__(16) __half2 h0[4], h1[4], h2[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {  // two values at a time, packed conversions
          float qa, ra, qb, rb;
          split_chunk(v[8 * g + 2 * q], least, shift, qa, ra);
          split_chunk(v[8 * g + 2 * q + 1], least, shift, qb, rb);
          h0[q] = __floats2half2_rn(qa, qb);  // |q| <= 512: exact in FP16
          h1[q] = __floats2half2_rn(ra, rb);
          const float2 f1 = __half22float2(h1[q]);
          h2[q] = __floats2half2_rn(ra - f1.x, rb - f1.y);
        }
        const int phys = (2 * kq + g) ^ within;  // 128-byte swizzle of 16-byte chunks
        const int off = (r >> 3) * 1024 + within * 128 + phys * 16;
        *reinterpret_cast<uint4 *>(st + 0 * PANEL_BYTES + off) = *reinterpret_cast<const uint4 *>(h0);
        *reinterpret_cast<uint4 *>(st + 1 * PANEL_BYTES + off) = *reinterpret_cast<const uint4 *>(h1);
        *reinterpret_cast<uint4 *>(st + 2 * PANEL_BYTES + off) = *reinterpret_cast<const uint4 *>(h2);
      }
      // generic-proxy writes of the A panels become visible to the tensor core
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (threadIdx.x == 0) {
        const uint32_t fb = sfull0 + 8 * b;
        mbar_expect_tx(fb, 3 * BPL);
        armed = (int)((n >> 1) & 1);
        armed_b = b;
        const uint32_t dst = smem_u32(st + 3 * PANEL_BYTES);
#pragma unroll
        for (int p = 0; p < 3; ++p) tma_load_3d(dst + p * BPL, &tmB, fb, 0, 0, 3 * c + p);
      } else if (lane == 0) {
        mbar_arrive(sfull0 + 8 * b);
      }
      // the next chunk's copies overlap the previous chunk's fold and the
      // next iteration's start (the L2 prefetch keeps their latency short)
      if (FORM == AH_COPY && n + 1 < total) issue_chunk(tn, cn);
      // the previous chunk is folded while this chunk's MMAs run; a failed
      // wait is told to the group at its next exchange
      if (n >= 1) folded = fold(n - 1, tp, cp);
      tp = tile;
      cp = c;
      tile = tn;
      c = cn;
    }
    // copies still in flight land before the CTA may exit
    if (FORM != AH_COPY) {
      if (ao_issuer && ao_pending >= 0) {
        const long long t0 = clock64();
        while (!mbar_test(aofull, (uint32_t)ao_pending) && clock64() - t0 < WAIT_BUDGET) {
        }
      }
    } else {
      asm volatile("cp.async.wait_all;" ::: "memory");
    }
    if (ok_all && folded) fold(total - 1, tp, cp);
    if (threadIdx.x == 0 && armed >= 0 && *abort_flag) {
      // the last B copy completes before the CTA may exit
      const long long t0 = clock64();
      while (!mbar_test(sfull0 + 8 * armed_b, (uint32_t)armed) && clock64() - t0 < WAIT_BUDGET) {
      }
    }
  } else if (warp == AH_CONV) {
    // ------------------------------ MMA issuer -------------------------------
    if (lane == 0) {
      for (int n = 0; n < total; ++n) {
        const int b = n & 1;
        if (!mbar_wait(sfull0 + 8 * b, (uint32_t)((n >> 1) & 1), abort_flag, P.err, 23)) break;
        if (n >= 2 &&
            !mbar_wait(aempty0 + 8 * b, (uint32_t)(((n - 2) >> 1) & 1), abort_flag, P.err, 24))
          break;
        tc_fence_after();
        const uint32_t sA = smem_u32(stages + b * STAGE);
        const uint32_t sB = sA + 3 * PANEL_BYTES;
        const uint32_t dL0 = tmem + (uint32_t)(b * 2 * NT);
        const uint32_t dL1 = dL0 + (uint32_t)NT;
#pragma unroll
        for (int k16 = 0; k16 < KSTEP / 16; ++k16) {
          const uint32_t koff = k16 * 32;
          const uint64_t a0 = smem_desc(sA + koff), a1 = smem_desc(sA + PANEL_BYTES + koff);
          const uint64_t a2 = smem_desc(sA + 2 * PANEL_BYTES + koff);
          const uint64_t b0 = smem_desc(sB + koff), b1 = smem_desc(sB + BPL + koff);
          const uint64_t b2 = smem_desc(sB + 2 * BPL + koff);
          const uint32_t acc = k16 > 0 ? 1u : 0u;  // each chunk starts its own sums
          mma_f16_id(dL0, a0, b0, P.idesc, acc);
          mma_f16_id(dL1, a0, b1, P.idesc, acc);
          mma_f16_id(dL1, a1, b0, P.idesc, 1u);
          mma_f16_id(dL1, a1, b1, P.idesc, 1u);
          mma_f16_id(dL1, a0, b2, P.idesc, 1u);
          mma_f16_id(dL1, a2, b0, P.idesc, 1u);
        }
        mma_commit(sempty0 + 8 * b);  // the stage may be refilled
        mma_commit(afull0 + 8 * b);   // the chunk's products are in TMEM
      }
      mma_commit(drain);
      const long long t0 = clock64();
      while (!mbar_test(drain, 0) && clock64() - t0 < WAIT_BUDGET) {
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == AH_CONV) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  }
}

// Occupied MO block sliced for ao_half_kernel: column n (orbital), chunk c of
// 64 nu values, scale per (column, chunk) with |x 2^e| <= 511.5; planes S0,
// R1, R2 at Bsl[(3 c + p) NT + n][64] (plain rows; the TMA copy swizzles
// them), scale 2^-e at sb[c NT + n].  One warp per (column, chunk); columns
// n >= nocc and nu >= nbas are zero.
__global__ void ao_occ_slice_kernel(const double *__restrict__ Cmo, int nbas, int nocc, int NT,
                                    int nks, __half *__restrict__ Bsl, float *__restrict__ sb) {
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= NT * nks) return;
  const int n = w % NT, c = w / NT;
  double v[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int nu = c * KSTEP + lane + 32 * q;
    v[q] = (n < nocc && nu < nbas) ? Cmo[(size_t)n * nbas + nu] : 0.0;
  }
  uint32_t key = 0;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const uint32_t kq =
        (uint32_t)(((unsigned long long)__double_as_longlong(v[q]) >> 32) & 0x7FFFFFFFu);
    key = kq > key ? kq : key;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const uint32_t other = __shfl_xor_sync(0xffffffffu, key, o);
    key = other > key ? other : key;
  }
  const int e = chunk_exponent_511(key);
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    float qv, rv;
    split_int((unsigned long long)__double_as_longlong(v[q]), e, qv, rv);
    const __half h1 = __float2half_rn(rv);
    const size_t k = lane + 32 * q;
    Bsl[((size_t)(3 * c + 0) * NT + n) * 64 + k] = __float2half_rn(qv);
    Bsl[((size_t)(3 * c + 1) * NT + n) * 64 + k] = h1;
    Bsl[((size_t)(3 * c + 2) * NT + n) * 64 + k] = __float2half_rn(rv - __half2float(h1));
  }
  if (lane == 0) sb[(size_t)c * NT + n] = ldexpf(1.0f, -e);
}

// AO tensor rows: row m' = mu + nbas*alpha of (alpha|mu nu) over K = nu.
// One CTA owns 32 alpha x 8 mu rows, one thread per row, warps alpha-fastest
// so every load of a nu-step is one 256-byte segment.  Same scale rule and
// slice layout as slice_batch_kernel.  The FP16 slices of each 64-wide nu
// chunk are staged in shared memory (16-byte chunks XOR-swizzled by alpha)
// and written out row-contiguous: the 8 mu rows of one alpha are 1 KB of
// consecutive memory.  The first CTA also sets the scale of the padding rows
// (their slices are zeroed by the host).
constexpr int AO_TA = 32, AO_TM = 8, AO_ROWS = AO_TA * AO_TM;

__global__ void __launch_bounds__(AO_ROWS) ao_slice_kernel(const double *__restrict__ ao, int NBA,
                                                          int nbas, long long nrows_pad, int nks,
                                                          int nsl, long long plane,
                                                          __half *__restrict__ slices,
                                                          float *__restrict__ inv_scale) {
  extern __shared__ uint4 stage[];  // [nsl][AO_ROWS rows][8 chunks of 8 halves]
  const int a_l = threadIdx.x & (AO_TA - 1), m_l = threadIdx.x / AO_TA;
  const int al = blockIdx.x * AO_TA + a_l, mu = blockIdx.y * AO_TM + m_l;
  const bool live = (al < NBA) && (mu < nbas);
  const long long MK = (long long)NBA * nbas;
  const size_t kstride = (size_t)nrows_pad * 64;
  if (blockIdx.x == 0 && blockIdx.y == 0)
    for (long long t = MK + threadIdx.x; t < nrows_pad; t += blockDim.x) inv_scale[t] = 1.0f;
  // row (alpha, mu) over K = nu read along the middle index: (alpha|mu nu) =
  // (alpha|nu mu), 8 NBA bytes apart, so a row's values stay within a few
  // memory pages (along the last index they are 8 NBA nbas bytes apart)
  const double *src = ao + (live ? al + (size_t)MK * mu : 0);  // element nu at src[NBA*nu]
  int e = 0;
  if (live) {
    unsigned long long mxb = 0;
    float ss = 0.0f;
    // sixteen independent loads in flight per thread (one 256-byte segment
    // per warp each): the loop is bound by memory latency, not arithmetic
    for (int nu0 = 0; nu0 < nbas; nu0 += 16) {
      double v[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) v[q] = (nu0 + q < nbas) ? src[(size_t)NBA * (nu0 + q)] : 0.0;
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const unsigned long long mag =
            (unsigned long long)__double_as_longlong(v[q]) & 0x7FFFFFFFFFFFFFFFull;
        mxb = mag > mxb ? mag : mxb;
        const float f = abs_trunc_f32(mag);
        ss = fmaf(f, f, ss);
      }
    }
    e = col_scale_exponent(mxb, ss, nbas);
  }
  const int rl = m_l + AO_TM * a_l;  // row within the CTA: the 8 mu of one alpha adjacent
  const int sw = a_l & 7;
  const __half hz = __float2half_rn(0.0f);
  for (int attempt = 0; attempt < 64; ++attempt) {
    long long n2 = 0;
    for (int kc = 0; kc < nks; ++kc) {
      for (int q00 = 0; q00 < 64; q00 += 16) {
        double v[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          const int nu = kc * 64 + q00 + q;
          v[q] = (live && nu < nbas) ? src[(size_t)NBA * nu] : 0.0;
        }
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          __align__(16) __half h0[8], h1[8], h2[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const int nu = kc * 64 + q00 + 8 * hh + q;
            h0[q] = h1[q] = h2[q] = hz;
            if (live && nu < nbas) {
              float qv, r;
              split_f32(v[8 * hh + q], e, qv, r);  // |x 2^e| <= 2047.5
              h0[q] = __float2half_rn(qv);
              h1[q] = __float2half_rn(r);
              h2[q] = __float2half_rn(r - __half2float(h1[q]));
              const int qi = __float_as_int(fabsf(qv) + 8388608.0f) - 0x4B000000;
              n2 += qi * qi;
            }
          }
          const int c = ((q00 >> 3) + hh) ^ sw;
          stage[(0 * AO_ROWS + rl) * 8 + c] = *reinterpret_cast<const uint4 *>(h0);
          if (nsl > 1) stage[(1 * AO_ROWS + rl) * 8 + c] = *reinterpret_cast<const uint4 *>(h1);
          if (nsl > 2) stage[(2 * AO_ROWS + rl) * 8 + c] = *reinterpret_cast<const uint4 *>(h2);
        }
      }
      __syncthreads();
      for (int j = threadIdx.x; j < AO_ROWS * 8; j += AO_ROWS) {
        const int r = j >> 3, c = j & 7;
        const int ra = r / AO_TM, rm = r % AO_TM;
        const int gal = blockIdx.x * AO_TA + ra, gmu = blockIdx.y * AO_TM + rm;
        if (gal < NBA && gmu < nbas) {
          const size_t row = (size_t)gmu + (size_t)nbas * gal;
          __half *dst = slices + (size_t)kc * kstride + row * 64 + c * 8;
          const int sc = c ^ (ra & 7);
          for (int sl = 0; sl < nsl; ++sl)
            *reinterpret_cast<uint4 *>(dst + sl * plane) = stage[(sl * AO_ROWS + r) * 8 + sc];
        }
      }
      __syncthreads();
    }
    // the norm bound makes a retry rare; the whole CTA repeats the pass with
    // a smaller scale on the rows that exceeded it
    const bool over = n2 > 16777216LL;
    if (!__syncthreads_or(over)) break;
    if (over) --e;
  }
  if (live) inv_scale[(size_t)mu + (size_t)nbas * al] = ldexpf(1.0f, -e);
}

}  // namespace

// A planned batch: up to three launch groups, workspace and (optionally)
// an instantiated CUDA graph of the whole evaluation.
struct SplitPlan {
  Group g[3];  // one residual slice (one-CTA), two residual slices, one residual slice (paired)
  PlainPlan *plain = nullptr;  // fragments planned in plain FP64 (slice count 0)
  int nsm = 0;
  cudaGraphExec_t gexec = nullptr;
  cudaGraph_t graph = nullptr;
  // graph form of a plan with several launch groups: inputs on a side branch
  cudaStream_t side = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_in[3] = {nullptr, nullptr, nullptr};
  ~SplitPlan() {
    if (gexec) cudaGraphExecDestroy(gexec);
    if (graph) cudaGraphDestroy(graph);
    for (auto &e : ev_in)
      if (e) cudaEventDestroy(e);
    if (ev_fork) cudaEventDestroy(ev_fork);
    if (side) cudaStreamDestroy(side);
    plain_plan_destroy(plain);
  }
  int launches() const {
    int n = plain_plan_launches(plain);
    for (auto &x : g)
      if (x.nfrag) n += 5;  // slicing, eps, kernel, two reductions
    return n;
  }
};

bool split_supported() { return get_encode() != nullptr; }

// Records the launch groups of a plan, one after the other (slicing, then
// the energy kernel and reductions of each group).  The overlapped form
// (RIMP2_BATCH_OVERLAP=1): with two or more groups, every group's inputs
// (slicing, orbital-energy pairs) go on a side branch, in the order the
// energy kernels run, and each energy kernel waits only for its own group's
// inputs, so the slicing of the next group runs while the current group's
// persistent kernel holds the SMs (a slicing block fits beside an energy
// CTA); the group with the least slicing work goes first, since nothing
// hides its inputs.
int record_plan_overlapped(SplitPlan *P, cudaStream_t s) {
  int order[3], n = 0;
  for (int k = 0; k < 3; ++k)
    if (P->g[k].nfrag) order[n++] = k;
  // measured on GB300 (256-fragment batch, same box, alternating runs):
  // 633.9 / 635.4 eff TFLOP/s with the groups one after the other against
  // 626.9 / 631.1 with the side branch -- under the power cap the slicing
  // beside an energy kernel costs that kernel more than it hides.  So the
  // groups run in sequence unless RIMP2_BATCH_OVERLAP=1.
  const char *ov = getenv("RIMP2_BATCH_OVERLAP");
  if (n < 2 || !(ov && ov[0] == '1')) {
    for (int k = 0; k < n; ++k) RIMP2_TRY(record_group(P->g[order[k]], s, P->nsm, nullptr));
    return RIMP2_OK;
  }
  int first = 0;
  for (int k = 1; k < n; ++k)
    if (P->g[order[k]].R < P->g[order[first]].R) first = k;  // R: 64-wide slice rows
  std::swap(order[0], order[first]);
  if (!P->side) {
    set_error("internal: side stream of the plan not created");
    return RIMP2_ERR_CUDA;
  }
  RIMP2_CK(cudaEventRecord(P->ev_fork, s));
  RIMP2_CK(cudaStreamWaitEvent(P->side, P->ev_fork, 0));
  for (int k = 0; k < n; ++k) {
    RIMP2_TRY(record_group_inputs(P->g[order[k]], P->side));
    RIMP2_CK(cudaEventRecord(P->ev_in[k], P->side));
  }
  for (int k = 0; k < n; ++k) {
    RIMP2_CK(cudaStreamWaitEvent(s, P->ev_in[k], 0));
    RIMP2_TRY(record_group(P->g[order[k]], s, P->nsm, nullptr, false));
  }
  return RIMP2_OK;
}

int split_plan_create(SplitPlan **out, int nfrag, const int *nocc, const int *nvirt, const int *NBA,
                      const double *const *Ca, const double *const *eo, const double *const *ev,
                      double *const *Epair, double *const *Etot, const int *nslices, bool graph,
                      cudaStream_t s) {
  *out = nullptr;
  // work items pack i | j << 16 and tA | tB << 16
  for (int f = 0; f < nfrag; ++f)
    if (nocc[f] > 65535 || (nvirt[f] + TILE - 1) / TILE > 65535) {
      set_error("split form: fragment %d too large for the work-item encoding (nocc=%d)", f,
                nocc[f]);
      return RIMP2_ERR_ARG;
    }
  SplitPlan *P = new SplitPlan();
  int dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&P->nsm, cudaDevAttrMultiProcessorCount, dev);
  P->g[0].nsl = 2;
  P->g[1].nsl = 3;
  P->g[2].nsl = 2;
  P->g[2].pair = true;
  std::vector<PlainFrag> plain;
  for (int f = 0; f < nfrag; ++f) {
    if (nslices && nslices[f] == 0) {
      PlainFrag F;
      memset(&F, 0, sizeof F);
      F.Ca = Ca[f];
      F.eo = eo[f];
      F.ev = ev[f];
      F.Epair = Epair[f];
      F.Etot = Etot[f];
      F.nocc = nocc[f];
      F.nvirt = nvirt[f];
      F.NBA = NBA[f];
      plain.push_back(F);
      continue;
    }
    FragDesc F;
    memset(&F, 0, sizeof F);
    F.nocc = nocc[f];
    F.nvirt = nvirt[f];
    F.NBA = NBA[f];
    F.Ca = Ca[f];
    F.eo = eo[f];
    F.ev = ev[f];
    F.Epair = Epair[f];
    F.Etot = Etot[f];
    const int ns = nslices ? nslices[f] : 1;
    P->g[ns >= 2 ? 1 : (pair_kernel_for(F.nocc, F.nvirt, F.NBA) ? 2 : 0)].fh.push_back(F);
  }
  for (auto &g : P->g) {
    if (g.fh.empty()) continue;
    int rc = build_group(g, s);
    if (rc != RIMP2_OK) {
      delete P;
      return rc;
    }
  }
  if (!plain.empty()) {
    int rc = plain_plan_create(&P->plain, (int)plain.size(), plain.data(), s);
    if (rc != RIMP2_OK) {
      delete P;
      return rc;
    }
  }
  if (graph) {
    int ngroups = 0;
    for (auto &g : P->g) ngroups += g.nfrag ? 1 : 0;
    if (ngroups >= 2) {  // the side branch of record_plan_overlapped
      if (cudaStreamCreateWithFlags(&P->side, cudaStreamNonBlocking) != cudaSuccess ||
          cudaEventCreateWithFlags(&P->ev_fork, cudaEventDisableTiming) != cudaSuccess ||
          cudaEventCreateWithFlags(&P->ev_in[0], cudaEventDisableTiming) != cudaSuccess ||
          cudaEventCreateWithFlags(&P->ev_in[1], cudaEventDisableTiming) != cudaSuccess ||
          cudaEventCreateWithFlags(&P->ev_in[2], cudaEventDisableTiming) != cudaSuccess) {
        set_error("stream/event creation for the batch graph failed");
        delete P;
        return RIMP2_ERR_CUDA;
      }
    }
    // the captured sequence needs the workspace already in place
    cudaError_t e = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) {
      set_error("graph capture start failed: %s", cudaGetErrorString(e));
      delete P;
      return RIMP2_ERR_CUDA;
    }
    const long long n0 = rimp2_kernel_launch_count();
    int rc = plain_plan_record(P->plain, s);
    if (rc == RIMP2_OK) rc = record_plan_overlapped(P, s);
    e = cudaStreamEndCapture(s, &P->graph);
    // captured launches run at each graph launch, not here
    count_launch(-(int)(rimp2_kernel_launch_count() - n0));
    if (rc != RIMP2_OK || e != cudaSuccess) {
      if (rc == RIMP2_OK) set_error("graph capture failed: %s", cudaGetErrorString(e));
      delete P;
      return rc != RIMP2_OK ? rc : RIMP2_ERR_CUDA;
    }
    e = cudaGraphInstantiate(&P->gexec, P->graph, 0);
    if (e != cudaSuccess) {
      set_error("graph instantiate failed: %s", cudaGetErrorString(e));
      delete P;
      return RIMP2_ERR_CUDA;
    }
  }
  *out = P;
  return RIMP2_OK;
}

int split_plan_execute(SplitPlan *P, cudaStream_t s) {
  if (P->gexec) {
    RIMP2_CK(cudaGraphLaunch(P->gexec, s));
    count_launch(P->launches());
    return RIMP2_OK;
  }
  const bool timed = timing_enabled();
  cudaEvent_t ev[4];
  if (timed)
    for (int k = 0; k < 4; ++k) RIMP2_CK(cudaEventCreate(&ev[k]));
  // a plan of plain fragments only is timed as one kernel interval
  const bool plain_only = !P->g[0].nfrag && !P->g[1].nfrag && !P->g[2].nfrag;
  if (timed && plain_only) {
    RIMP2_CK(cudaEventRecord(ev[0], s));
    RIMP2_CK(cudaEventRecord(ev[1], s));
  }
  RIMP2_TRY(plain_plan_record(P->plain, s));
  if (timed && plain_only) RIMP2_CK(cudaEventRecord(ev[2], s));
  for (auto &g : P->g) RIMP2_TRY(record_group(g, s, P->nsm, timed ? ev : nullptr));
  if (timed) {
    RIMP2_CK(cudaEventRecord(ev[3], s));
    RIMP2_CK(cudaEventSynchronize(ev[3]));
    float ms;
    for (int k = 0; k < 3; ++k) {
      RIMP2_CK(cudaEventElapsedTime(&ms, ev[k], ev[k + 1]));
      record_timing(k, ms);
    }
    for (int k = 0; k < 4; ++k) cudaEventDestroy(ev[k]);
  }
  return RIMP2_OK;
}

void split_plan_destroy(SplitPlan *P) { delete P; }

// Execution of a plan (no graph) whose inputs are still in host memory:
// copy c moves count[c] doubles from src[c] to dst[c].  The copies run on the
// copy streams cs[0..ncs) launch group by launch group, the group with the
// least Calpha first; copies that belong to no split group (orbital
// energies, the plain FP64 fragments) go before all of them.  Within a
// group each copy goes to the stream with the fewest bytes so far (the
// batched host call passes one stream: four were measured slower).  Each
// group's slicing waits only
// for its own fragments' copies, so the transfer of the later, larger
// groups overlaps the kernels of the earlier ones.  A copy belongs to the
// group whose fragment has dst as its Calpha address.  Several plans over
// one set of buffers run in turn: the first call waits for the allocation
// (wait_alloc), the later ones queue their copies behind its copies.
int split_plan_execute_host(SplitPlan *P, cudaStream_t s, const cudaStream_t *cs, int ncs,
                            int ncopy, double *const *dst, const double *const *src,
                            const size_t *count, bool wait_alloc) {
  struct Events {
    std::vector<cudaEvent_t> e;
    ~Events() {
      for (auto x : e) cudaEventDestroy(x);
    }
  } ev;
  auto event = [&](cudaEvent_t *out) -> int {
    RIMP2_CK(cudaEventCreateWithFlags(out, cudaEventDisableTiming));
    ev.e.push_back(*out);
    return RIMP2_OK;
  };
  std::vector<int> owner(ncopy, -1);  // launch group of each copy, -1: none
  size_t bytes[3] = {0, 0, 0};
  int order[3], n = 0;
  for (int k = 0; k < 3; ++k) {
    for (const auto &F : P->g[k].fh) {
      bytes[k] += (size_t)F.NBA * F.nvirt * F.nocc;
      for (int c = 0; c < ncopy; ++c)
        if (dst[c] == F.Ca) owner[c] = k;
    }
    if (P->g[k].nfrag) order[n++] = k;
  }
  std::sort(order, order + n, [&](int a, int b) { return bytes[a] < bytes[b]; });
  // the copy streams start after the destination buffers' allocation on s
  // (wait_alloc false: an earlier call on these streams already waited)
  if (wait_alloc) {
    cudaEvent_t e0;
    RIMP2_TRY(event(&e0));
    RIMP2_CK(cudaEventRecord(e0, s));
    for (int q = 0; q < ncs; ++q) RIMP2_CK(cudaStreamWaitEvent(cs[q], e0, 0));
  }
  // phase 0: copies outside the split groups; phase 1 + k: group order[k]
  std::vector<cudaEvent_t> done((size_t)(1 + n) * ncs);
  for (int ph = 0; ph <= n; ++ph) {
    const int want = ph == 0 ? -1 : order[ph - 1];
    std::vector<size_t> load(ncs, 0);
    for (int c = 0; c < ncopy; ++c) {
      if (owner[c] != want) continue;
      const int q = (int)(std::min_element(load.begin(), load.end()) - load.begin());
      load[q] += count[c];
      RIMP2_CK(cudaMemcpyAsync(dst[c], src[c], count[c] * sizeof(double), cudaMemcpyHostToDevice,
                               cs[q]));
    }
    for (int q = 0; q < ncs; ++q) {
      RIMP2_TRY(event(&done[(size_t)ph * ncs + q]));
      RIMP2_CK(cudaEventRecord(done[(size_t)ph * ncs + q], cs[q]));
    }
  }
  for (int q = 0; q < ncs; ++q) RIMP2_CK(cudaStreamWaitEvent(s, done[q], 0));
  RIMP2_TRY(plain_plan_record(P->plain, s));
  for (int k = 0; k < n; ++k) {
    for (int q = 0; q < ncs; ++q)
      RIMP2_CK(cudaStreamWaitEvent(s, done[(size_t)(1 + k) * ncs + q], 0));
    RIMP2_TRY(record_group(P->g[order[k]], s, P->nsm, nullptr));
  }
  return RIMP2_OK;
}

int bounded_wait_selftest(long long budget_cycles, cudaStream_t s) {
  wait_selftest_kernel<<<1, 32, 0, s>>>(budget_cycles, device_error_word());
  count_launch(1);
  RIMP2_CK(cudaGetLastError());
  return collect_device_error(s);
}

int rcp_denom_selftest(int n, const float *d, float *r, float *ref, cudaStream_t s) {
  DevBuf dd, dr, dref;
  const size_t b = sizeof(float) * (size_t)n;
  RIMP2_TRY(dd.alloc(b, s));
  RIMP2_TRY(dr.alloc(b, s));
  RIMP2_TRY(dref.alloc(b, s));
  RIMP2_CK(cudaMemcpyAsync(dd.p, d, b, cudaMemcpyHostToDevice, s));
  rcp_selftest_kernel<<<(n + 255) / 256, 256, 0, s>>>(dd.as<float>(), dr.as<float>(),
                                                      dref.as<float>(), n);
  count_launch(1);
  RIMP2_CK(cudaGetLastError());
  RIMP2_CK(cudaMemcpyAsync(r, dr.p, b, cudaMemcpyDeviceToHost, s));
  RIMP2_CK(cudaMemcpyAsync(ref, dref.p, b, cudaMemcpyDeviceToHost, s));
  RIMP2_CK(cudaStreamSynchronize(s));
  return RIMP2_OK;
}

// Host Calpha -> energies with the copy overlapped: occupied indices are
// copied in chunks on a second stream; once chunk c has landed, its columns
// are sliced and the work items of every pair (i <= j) with j in chunk c --
// whose inputs are then all on the device -- run as one persistent launch,
// while chunk c+1 is still in flight.  dCa must have room for the fragment.
int split_energy_streamed(const double *hCa, double *dCa, const SplitEnergyArgs &a,
                          cudaStream_t s, cudaStream_t copy_s, int chunk_occ) {
  // Occupied-index chunk boundaries: the first chunk small (its copy is the
  // only one nothing hides), later ones growing by half, since chunk c's
  // work grows with its column indices j while its copy does not; chunk_occ
  // caps the first chunk.  Chunk c is sliced on the slicing stream as soon
  // as its copy lands, beside chunk c-1's energy kernel, and its energy
  // kernel starts once it is sliced, so after the first few chunks the copy
  // engine and the slicer run ahead of the tensor cores.
  std::vector<int> bnd;
  for (int b = std::min(a.nocc, std::max(1, std::min(chunk_occ, 4))); ;) {
    bnd.push_back(b);
    if (b >= a.nocc) break;
    b = std::min(a.nocc, b + std::max(1, b / 2));
  }
  if (inject_fault("launch")) {  // before any copy is in flight
    set_error("injected launch failure (RIMP2_FAULT_INJECT=launch)");
    return RIMP2_ERR_CUDA;
  }
  SplitPlan *P = nullptr;
  const int ns = a.nslices;
  const double *dCaC = dCa;
  RIMP2_TRY(split_plan_create(&P, 1, &a.nocc, &a.nvirt, &a.NBA, &dCaC, &a.eo, &a.ev, &a.Epair,
                              &a.Etot, &ns, false, s));
  Group &g = P->g[0].nfrag ? P->g[0] : (P->g[1].nfrag ? P->g[1] : P->g[2]);
  const FragDesc &F = g.fh[0];
  const FragDesc *fr = g.frags.as<FragDesc>();
  int rc = RIMP2_OK;
  const int nchunk = (int)bnd.size();
  // ev[c]: chunk c copied (copy stream); ev[nchunk + c]: chunk c sliced
  // (slicing stream); ev[2 nchunk]: the plan's buffers exist (stream s)
  std::vector<cudaEvent_t> ev(2 * nchunk + 1, nullptr);
  for (auto &e : ev)
    if (rc == RIMP2_OK && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
      set_error("event creation failed");
      rc = RIMP2_ERR_CUDA;
    }
  // RIMP2_STREAM_SLICE=0: slice on s, between the energy launches
  const char *sv = getenv("RIMP2_STREAM_SLICE");
  cudaStream_t ss = (sv && sv[0] == '0') ? s : slice_stream();
  if (rc == RIMP2_OK && !ss) {
    set_error("slicing stream unavailable");
    rc = RIMP2_ERR_CUDA;
  }
  const size_t slab = (size_t)a.NBA * a.nvirt;  // doubles per occupied index
  // copies first, so the copy engine runs ahead of the compute stream
  for (int c = 0; c < nchunk && rc == RIMP2_OK; ++c) {
    const int i0 = c ? bnd[c - 1] : 0, i1 = bnd[c];
    cudaError_t e = cudaMemcpyAsync(dCa + slab * i0, hCa + slab * i0, sizeof(double) * slab * (i1 - i0),
                                    cudaMemcpyHostToDevice, copy_s);
    if (e == cudaSuccess) e = cudaEventRecord(ev[c], copy_s);
    if (e != cudaSuccess) {
      set_error("streamed copy failed: %s", cudaGetErrorString(e));
      rc = RIMP2_ERR_CUDA;
    }
  }
  if (rc == RIMP2_OK) {
    dim3 g2((unsigned)((g.max_nv + 255) / 256), 1);
    eps_batch_kernel<<<g2, 256, 0, s>>>(fr, g.eo2.as<float2>(), g.ev2.as<float2>());
    count_launch(1);
  }
  // slicing of every chunk on the slicing stream, each after its copy (and
  // after the plan's buffers, allocated on s); columns of different chunks
  // are disjoint in the slices, scales and corrections
  if (rc == RIMP2_OK) {
    cudaError_t e = cudaEventRecord(ev[2 * nchunk], s);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(ss, ev[2 * nchunk], 0);
    for (int c = 0; c < nchunk && e == cudaSuccess; ++c) {
      const int i0 = c ? bnd[c - 1] : 0, i1 = bnd[c];
      const int col0 = i0 * F.nvpad, col1 = i1 * F.nvpad;
      e = cudaStreamWaitEvent(ss, ev[c], 0);
      if (e != cudaSuccess) break;
      slice_batch_kernel<<<(unsigned)(((long long)(col1 - col0) * 32 + 255) / 256), 256, 0, ss>>>(
          fr, g.nsl, g.R * 64, g.slices.as<__half>(), g.inv.as<float>(), col0, col1,
          g.pair ? 1 : 0, g.dcorr.as<float>());
      count_launch(1);
      e = cudaGetLastError();
      if (e == cudaSuccess) e = cudaEventRecord(ev[nchunk + c], ss);
    }
    if (e != cudaSuccess) {
      set_error("streamed slicing failed: %s", cudaGetErrorString(e));
      rc = RIMP2_ERR_CUDA;
    }
  }
  BatchParams BP;
  BP.frags = fr;
  BP.items = g.items.as<int4>();
  BP.eo2 = g.eo2.as<float2>();
  BP.ev2 = g.ev2.as<float2>();
  BP.inv_scale = g.inv.as<float>();
  BP.part = g.part.as<double>();
  BP.err = device_error_word();
  for (int c = 0; c < nchunk && rc == RIMP2_OK; ++c) {
    const int i0 = c ? bnd[c - 1] : 0, i1 = bnd[c];
    cudaError_t e = cudaStreamWaitEvent(s, ev[nchunk + c], 0);
    if (e != cudaSuccess) {
      set_error("stream wait failed: %s", cudaGetErrorString(e));
      rc = RIMP2_ERR_CUDA;
      break;
    }
    e = cudaMemsetAsync(g.queue.p, 0, sizeof(unsigned int), s);
    if (e != cudaSuccess) {
      set_error("queue reset failed: %s", cudaGetErrorString(e));
      rc = RIMP2_ERR_CUDA;
      break;
    }
    if (g.pair) {
      // pair items with j in [i0, i1) (their i0' < i0'+1 <= j are already copied)
      PairParams Q;
      Q.frags = fr;
      Q.items = g.pitems.as<int4>();
      Q.item_begin = pair_items_before(i0) * F.ntp;
      Q.nitems = pair_items_before(i1) * F.ntp;
      Q.dcorr = g.dcorr.as<float>();
      Q.queue = g.queue.as<unsigned int>();
      Q.eo2 = BP.eo2;
      Q.ev2 = BP.ev2;
      Q.inv_scale = BP.inv_scale;
      Q.part = BP.part;
      Q.err = BP.err;
      const int npair = (int)std::min<long long>(Q.nitems - Q.item_begin, std::max(1, P->nsm / 2));
      note_split_kernel(2);
      rc = launch_pair(g, Q, npair, s);
      if (rc != RIMP2_OK) break;
    } else {
      // pairs (i<=j) with j in [i0, i1): pair indices [i0(i0+1)/2, i1(i1+1)/2)
      const long long pb = (long long)i0 * (i0 + 1) / 2, pe = (long long)i1 * (i1 + 1) / 2;
      BP.item_begin = pb * F.ntp;
      BP.nitems = pe * F.ntp;
      BP.queue = g.queue.as<unsigned int>();
      const int grid = (int)std::min<long long>(BP.nitems - BP.item_begin, P->nsm);
      note_split_kernel(1);
      // at the highest priority, like the paired kernel: the next chunk's
      // slicing blocks wait behind this kernel's CTAs, not ahead of them
      if (g.nsl == 2)
        e = launch_hi(split_batch_kernel<2, 3>, grid, BATCH_THREADS, smem_bytes(2, 3), s, g.tm, BP);
      else
        e = launch_hi(split_batch_kernel<3, 2>, grid, BATCH_THREADS, smem_bytes(3, 2), s, g.tm, BP);
      if (e != cudaSuccess) {
        set_error("split launch failed: %s", cudaGetErrorString(e));
        rc = RIMP2_ERR_CUDA;
        break;
      }
    }
    count_launch(1);
    e = cudaGetLastError();
    if (e != cudaSuccess) {
      set_error("split launch failed: %s", cudaGetErrorString(e));
      rc = RIMP2_ERR_CUDA;
    }
  }
  if (rc == RIMP2_OK) {
    pair_reduce_batch_kernel<<<(unsigned)((g.npairs_total + 7) / 8), 256, 0, s>>>(
        fr, g.nfrag, g.npairs_total, g.part.as<double>());
    total_reduce_batch_kernel<<<g.nfrag, total_threads(g.max_nocc), 0, s>>>(fr);
    count_launch(2);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
      set_error("reduction launch failed: %s", cudaGetErrorString(e));
      rc = RIMP2_ERR_CUDA;
    }
  }
  // on failure, copies may still be in flight into dCa: finish them before
  // the caller can release dCa
  if (rc != RIMP2_OK) {
    cudaStreamSynchronize(copy_s);
    if (ss && ss != s) cudaStreamSynchronize(ss);
    cudaStreamSynchronize(s);
  }
  for (auto &e : ev)
    if (e) cudaEventDestroy(e);
  split_plan_destroy(P);
  return rc;
}

// ---- general split GEMM: host side -------------------------------------------
int sliced_cols(SlicedOp &op, const double *src, int K, int nrows, int ngroups, int nsl,
                cudaStream_t s) {
  FragDesc F;
  memset(&F, 0, sizeof F);
  F.nocc = ngroups;
  F.nvirt = nrows;
  F.NBA = K;
  F.nvpad = (nrows + TILE - 1) / TILE * TILE;
  F.nks = (K + KSTEP - 1) / KSTEP;
  F.ncol = ngroups * F.nvpad;
  F.Ca = src;
  op.nsl = nsl;
  op.nks = F.nks;
  op.rows_per_group = F.nvpad;
  op.ncol = F.ncol;
  op.R = (long long)F.nks * F.ncol;
  if (op.R > 2147483647LL - TILE) {
    set_error("split GEMM operand too large (%lld rows)", op.R);
    return RIMP2_ERR_ARG;
  }
  RIMP2_TRY(op.slices.alloc(sizeof(__half) * (size_t)nsl * op.R * 64, s));
  RIMP2_TRY(op.inv.alloc(sizeof(float) * (size_t)op.ncol, s));
  slice_one_kernel<<<(unsigned)(((long long)F.ncol * 32 + 255) / 256), 256, 0, s>>>(
      F, nsl, op.R * 64, op.slices.as<__half>(), op.inv.as<float>());
  count_launch(1);
  RIMP2_CK(cudaGetLastError());
  return RIMP2_OK;
}

int sliced_ao(SlicedOp &op, const double *ao, int NBA, int nbas, int nsl, cudaStream_t s) {
  const long long rows = (long long)NBA * nbas;
  op.nsl = nsl;
  op.nks = (nbas + KSTEP - 1) / KSTEP;
  op.ncol = (rows + TILE - 1) / TILE * TILE;
  op.rows_per_group = op.ncol;
  op.R = (long long)op.nks * op.ncol;
  if (op.R > 2147483647LL - TILE) {
    set_error("AO operand too large (%lld rows)", op.R);
    return RIMP2_ERR_ARG;
  }
  RIMP2_TRY(op.slices.alloc(sizeof(__half) * (size_t)nsl * op.R * 64, s));
  RIMP2_TRY(op.inv.alloc(sizeof(float) * (size_t)op.ncol, s));
  // padding rows [rows, ncol) of every K chunk of every slice plane: the
  // chunks are equally spaced (ncol rows of 128 bytes) across the planes
  if (op.ncol > rows)
    RIMP2_CK(cudaMemset2DAsync(op.slices.as<__half>() + (size_t)rows * 64, (size_t)op.ncol * 128,
                               0, (size_t)(op.ncol - rows) * 128, (size_t)op.nks * nsl, s));
  const int smem = nsl * AO_ROWS * 128;
  RIMP2_CK(cudaFuncSetAttribute(ao_slice_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  dim3 grid((unsigned)((NBA + AO_TA - 1) / AO_TA), (unsigned)((nbas + AO_TM - 1) / AO_TM));
  ao_slice_kernel<<<grid, AO_ROWS, smem, s>>>(ao, NBA, nbas, op.ncol, op.nks, nsl, op.R * 64,
                                              op.slices.as<__half>(), op.inv.as<float>());
  count_launch(1);
  RIMP2_CK(cudaGetLastError());
  return RIMP2_OK;
}

static int encode_op(CUtensorMap &tm, const SlicedOp &op, int boxrows) {
  auto encode = get_encode();
  if (!encode) {
    set_error("cuTensorMapEncodeTiled entry point unavailable");
    return RIMP2_ERR_UNSUPPORTED;
  }
  cuuint64_t dims[3] = {64, (cuuint64_t)op.R, (cuuint64_t)op.nsl};
  cuuint64_t strides[2] = {128, (cuuint64_t)op.R * 128};
  cuuint32_t box[3] = {KSTEP, (cuuint32_t)boxrows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult cr = encode(&tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, op.slices.p, dims, strides, box,
                       estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                       CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (cr != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed (%d)", (int)cr);
    return RIMP2_ERR_CUDA;
  }
  return RIMP2_OK;
}

int split_gemm(const SlicedOp &A, long long a_row0, long long a_bstride, const SlicedOp &B,
               long long b_row0, long long b_bstride, int M, int N, int nbatch, double *out,
               long long sOm, long long sOn, long long sOb, cudaStream_t s) {
  if (A.nsl != B.nsl || A.nks != B.nks || M <= 0 || N <= 0 || nbatch <= 0) {
    set_error("split_gemm: operand mismatch or bad sizes");
    return RIMP2_ERR_ARG;
  }
  GemmSP P;
  memset(&P, 0, sizeof P);
  P.M = M;
  P.N = N;
  P.NT = N <= TILE ? (N + 15) / 16 * 16 : TILE;
  P.nks = A.nks;
  P.mtiles = (M + TILE - 1) / TILE;
  P.ntiles = (N + P.NT - 1) / P.NT;
  P.nbatch = nbatch;
  P.a_ncol = A.ncol;
  P.b_ncol = B.ncol;
  P.a_row0 = a_row0;
  P.a_bstride = a_bstride;
  P.b_row0 = b_row0;
  P.b_bstride = b_bstride;
  P.a_inv = A.inv.as<float>();
  P.b_inv = B.inv.as<float>();
  P.out = out;
  P.sOm = sOm;
  P.sOn = sOn;
  P.sOb = sOb;
  uint32_t cols = 32;
  while (cols < (uint32_t)(4 * P.NT)) cols <<= 1;
  P.tmem_cols = cols;
  P.err = device_error_word();
  const long long nitems = (long long)nbatch * P.mtiles * P.ntiles;
  if (nitems > 2147483647LL) {
    set_error("split_gemm: too many tiles");
    return RIMP2_ERR_ARG;
  }
  CUtensorMap tA, tB;
  RIMP2_TRY(encode_op(tA, A, TILE));
  RIMP2_TRY(encode_op(tB, B, P.NT));
  const int smem = gemm_smem_bytes(A.nsl, P.NT);
  auto kern = A.nsl == 3 ? split_gemm_kernel<3> : split_gemm_kernel<2>;
  RIMP2_CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  int dev = 0, nsm = 0, resident = 0;
  RIMP2_CK(cudaGetDevice(&dev));
  RIMP2_CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  RIMP2_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, kern, GEMM_THREADS, smem));
  // persistent CTAs whose TMEM allocations fit an SM together
  resident = std::max(1, std::min(resident, (int)(512 / cols)));
  const long long grid = std::min<long long>(nitems, (long long)nsm * resident);
  kern<<<(unsigned)grid, GEMM_THREADS, smem, s>>>(tA, tB, P);
  count_launch(1);
  RIMP2_CK(cudaGetLastError());
  return RIMP2_OK;
}

// First half of the AO->MO transform, fused (ao_half_kernel): the occupied MO
// block is sliced per (column, 64-wide nu chunk), then one pass over the AO
// tensor forms half[i][alpha][mu].  *handled = false (nothing launched) when
// nocc exceeds the kernel's 80 columns; the caller then takes the sliced path.
int ao_half_fused(const double *ao, int NBA, int nbas, const double *Cmo, int nocc, double *half,
                  cudaStream_t s, bool *handled) {
  *handled = false;
  const int NT = (nocc + 15) / 16 * 16;
  if (NT > AH_NT_MAX || nocc <= 0 || nbas < 2) return RIMP2_OK;  // callers: an occupied and a virtual orbital
  const char *env = getenv("RIMP2_AO_FUSED");  // =0: the sliced first half (for comparisons)
  if (env && env[0] == '0') return RIMP2_OK;
  auto encode = get_encode();
  if (!encode) {
    set_error("cuTensorMapEncodeTiled entry point unavailable");
    return RIMP2_ERR_UNSUPPORTED;
  }
  const int nks = (nbas + KSTEP - 1) / KSTEP;
  const long long ntiles = (long long)((NBA + AH_TA - 1) / AH_TA) * ((nbas + AH_TM - 1) / AH_TM);
  if (ntiles > 2147483647LL) {
    set_error("AO transform too large for one launch (%lld tiles)", ntiles);
    return RIMP2_ERR_ARG;
  }
  DevBuf Bsl, sb;
  RIMP2_TRY(Bsl.alloc(sizeof(__half) * (size_t)3 * nks * NT * 64, s));
  RIMP2_TRY(sb.alloc(sizeof(float) * (size_t)nks * NT, s));
  const long long nw = (long long)NT * nks;
  ao_occ_slice_kernel<<<(unsigned)((nw * 32 + 255) / 256), 256, 0, s>>>(
      Cmo, nbas, nocc, NT, nks, Bsl.as<__half>(), sb.as<float>());
  count_launch(1);
  RIMP2_CK(cudaGetLastError());
  CUtensorMap tm;
  cuuint64_t dims[3] = {64, (cuuint64_t)NT, (cuuint64_t)(3 * nks)};
  cuuint64_t strides[2] = {128, (cuuint64_t)NT * 128};
  cuuint32_t box[3] = {KSTEP, (cuuint32_t)NT, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult cr = encode(&tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, Bsl.p, dims, strides, box, estr,
                       CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                       CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (cr != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed (%d)", (int)cr);
    return RIMP2_ERR_CUDA;
  }
  AoHalfParams P;
  P.ao = ao;
  P.NBA = NBA;
  P.nbas = nbas;
  P.nocc = nocc;
  P.nks = nks;
  P.ta_tiles = (NBA + AH_TA - 1) / AH_TA;
  P.tiles = (int)ntiles;
  P.sb = sb.as<float>();
  P.half = half;
  P.idesc = (1u << 4) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(TILE >> 4) << 24);
  P.err = device_error_word();
  // The AO chunks arrive by TMA: in one box per row group where the rows of
  // the tensor start on 16-byte boundaries (even NBA, aligned base).
  // Elsewhere every second row along k and every second one along mu are 16-byte
  // multiples apart: four tensors, one per parity of k and of mu, each starting at
  // the boundary at or before its first element, in boxes two alpha wider.
  // Their chunk takes 72 KB instead of 64, which NT = 80 has no room for: it
  // keeps the copies (nbas = 677: 4.05 ms, against 3.27 at 680 in one box).
  int form = NBA % 2 == 0 && (uintptr_t)ao % 16 == 0 ? AH_BOX
             : NT < AH_NT_MAX                        ? AH_BOX4
                                                     : AH_COPY;
  AoMaps tmAO;
  memset(&tmAO, 0, sizeof tmAO);
  P.shift = 0;
  for (int q = 0; q < (form == AH_COPY ? 0 : form == AH_BOX ? 1 : 4); ++q) {
    const int kp = q >> 1, mp = q & 1, step = form == AH_BOX ? 1 : 2;
    const double *first = ao + (size_t)kp * NBA + (size_t)mp * NBA * nbas;
    const unsigned sh = (uintptr_t)first % 16 ? 1 : 0;
    P.shift |= sh << q;
    cuuint64_t adims[3] = {(cuuint64_t)NBA + sh, (cuuint64_t)((nbas - kp + step - 1) / step),
                           (cuuint64_t)((nbas - mp + step - 1) / step)};
    cuuint64_t astr[2] = {(cuuint64_t)step * NBA * 8, (cuuint64_t)step * NBA * nbas * 8};
    cuuint32_t abox[3] = {(cuuint32_t)(form == AH_BOX ? AH_TA : AH_TA + 2),
                          (cuuint32_t)(KSTEP / step), (cuuint32_t)(form == AH_BOX ? 2 : 1)};
    cr = encode(&tmAO.m[q], CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<double *>(first - sh), adims,
                astr, abox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS) {
      set_error("cuTensorMapEncodeTiled (AO tensor) failed (%d)", (int)cr);
      return RIMP2_ERR_CUDA;
    }
  }
  void (*kern)(CUtensorMap, AoMaps, AoHalfParams) = nullptr;
  switch (NT) {
    case 16: kern = form == AH_BOX ? ao_half_kernel<AH_BOX, 16> : ao_half_kernel<AH_BOX4, 16>; break;
    case 32: kern = form == AH_BOX ? ao_half_kernel<AH_BOX, 32> : ao_half_kernel<AH_BOX4, 32>; break;
    case 48: kern = form == AH_BOX ? ao_half_kernel<AH_BOX, 48> : ao_half_kernel<AH_BOX4, 48>; break;
    case 64: kern = form == AH_BOX ? ao_half_kernel<AH_BOX, 64> : ao_half_kernel<AH_BOX4, 64>; break;
    default: kern = form == AH_BOX ? ao_half_kernel<AH_BOX, 80> : ao_half_kernel<AH_COPY, 80>;
  }
  const int smem = ah_smem_bytes(form, NT);
  RIMP2_CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  int resident = 0;
  RIMP2_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, kern, AH_THREADS, smem));
  if (resident < 1) return RIMP2_OK;  // cannot be resident here: the sliced path runs
  int dev = 0, nsm = 0;
  RIMP2_CK(cudaGetDevice(&dev));
  RIMP2_CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  kern<<<(unsigned)std::min<long long>(ntiles, nsm), AH_THREADS, smem, s>>>(tm, tmAO, P);
  count_launch(1);
  RIMP2_CK(cudaGetLastError());
  *handled = true;
  return RIMP2_OK;
}

// Local-orbital fragment energy in the split form: slices of Calpha and of its
// projected copies Ct in one buffer, one persistent launch (split_eos_pair_kernel;
// split_eos_kernel with two residual slices),
// compensated FP64 pair and total reductions.
// Fragment energies of one or two projected copies of Calpha: Etot[c] from
// copy Ct[c].
int split_eos_energy(const double *Ca, const double *const *Ct, int copies, int NBA, int nvirt,
                     int nocc, const double *eo, const double *ev, double *Epair, double *Etot,
                     int nslices, cudaStream_t s) {
  const int nsl = nslices + 1;
  if (nsl > 2 && copies > 1) {  // the one-CTA kernel takes one copy
    for (int c = 0; c < copies; ++c)
      RIMP2_TRY(split_eos_energy(Ca, Ct + c, 1, NBA, nvirt, nocc, eo, ev, Epair, Etot + c, nslices, s));
    return RIMP2_OK;
  }
  auto encode = get_encode();
  if (!encode) {
    set_error("cuTensorMapEncodeTiled entry point unavailable");
    return RIMP2_ERR_UNSUPPORTED;
  }
  const int sets = copies + 1;
  FragDesc fh[3];
  memset(fh, 0, sizeof fh);
  const int nvpad = (nvirt + TILE - 1) / TILE * TILE;
  const int nks = (NBA + KSTEP - 1) / KSTEP;
  const int nt = nvpad / TILE;
  const int ntp = nt * (nt + 1) / 2;
  const long long ncol = (long long)nocc * nvpad;
  const long long R = (long long)sets * nks * ncol;
  const int npairs = nocc * (nocc + 1) / 2;
  const bool pair = nsl == 2;
  int per = 2 * ntp;  // items of an occupied pair
  if (pair) {
    per = 0;
    for (int r = 0; 2 * r < nt; ++r) per += nt - 2 * r;
  }
  const int nper = pair ? ntp : 2 * ntp;  // partial energies of an occupied pair
  const long long nitems = (long long)npairs * per, npart = (long long)npairs * nper;
  if (R > 2147483647LL - TILE && copies > 1) {  // too many rows for one tensor map: one copy at a time
    for (int c = 0; c < copies; ++c)
      RIMP2_TRY(split_eos_energy(Ca, Ct + c, 1, NBA, nvirt, nocc, eo, ev, Epair, Etot + c, nslices, s));
    return RIMP2_OK;
  }
  if (R > 2147483647LL - TILE || nitems > 2147483647LL || ncol > 2147483647LL) {
    set_error("split local-orbital energy: fragment too large (rows=%lld, items=%lld)", R, nitems);
    return RIMP2_ERR_ARG;
  }
  for (int f = 0; f < sets; ++f) {
    FragDesc &F = fh[f];
    F.nocc = nocc;
    F.nvirt = nvirt;
    F.nvpad = nvpad;
    F.NBA = NBA;
    F.nks = nks;
    F.ntp = ntp;
    F.ncol = (int)ncol;
    F.row_base = (long long)f * nks * ncol;
    F.col_base = (long long)f * ncol;
    F.Ca = f ? Ct[f - 1] : Ca;
    F.eo = eo;
    F.ev = ev;
  }
  int dev = 0, nsm = 0;
  RIMP2_CK(cudaGetDevice(&dev));
  RIMP2_CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  const int planes = nsl + (pair ? 1 : 0);  // one residual slice: V plane, three products
  DevBuf arena, frags, slices, inv, eo2, ev2, part, queue, pairs, dcorr, stash;
  {
    DevBuf *buf[] = {&slices, &frags, &inv, &dcorr, &eo2, &ev2, &part, &queue, &pairs, &stash};
    const size_t bytes[] = {sizeof(__half) * (size_t)planes * R * 64,
                            sizeof fh,
                            sizeof(float) * sets * (size_t)ncol,
                            pair ? sizeof(float) * sets * (size_t)ncol : 16,
                            sizeof(float2) * nocc,
                            sizeof(float2) * nvpad,
                            sizeof(double) * copies * (size_t)npart,
                            sizeof(unsigned int),
                            sizeof(int) * 2 * (size_t)npairs,
                            pair ? sizeof(float) * 2 * 64 * 256 * (size_t)nsm : 16};
    const int rc = alloc_parts(arena, buf, bytes, s);
    if (rc != RIMP2_OK && copies > 1) {  // no room for both copies at once
      (void)cudaGetLastError();
      clear_error();
      for (int c = 0; c < copies; ++c)
        RIMP2_TRY(split_eos_energy(Ca, Ct + c, 1, NBA, nvirt, nocc, eo, ev, Epair, Etot + c, nslices, s));
      return RIMP2_OK;
    }
    RIMP2_TRY(rc);
  }
  RIMP2_CK(cudaMemcpyAsync(frags.p, fh, sizeof fh, cudaMemcpyHostToDevice, s));
  const FragDesc *fr = frags.as<FragDesc>();
  slice_batch_kernel<<<dim3((unsigned)((ncol * 32 + 255) / 256), (unsigned)sets), 256, 0, s>>>(
      fr, nsl, R * 64, slices.as<__half>(), inv.as<float>(), 0, 0x7fffffff, pair ? 1 : 0,
      dcorr.as<float>());
  eps_batch_kernel<<<dim3((unsigned)((std::max(nvpad, nocc) + 255) / 256), 1), 256, 0, s>>>(
      fr, eo2.as<float2>(), ev2.as<float2>());
  count_launch(2);
  CUtensorMap tmA, tmB;
  cuuint64_t dims[3] = {64, (cuuint64_t)R, (cuuint64_t)planes};
  cuuint64_t strides[2] = {128, (cuuint64_t)R * 128};
  cuuint32_t boxA[3] = {KSTEP, TILE, 1}, boxB[3] = {KSTEP, HALF, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult cr = encode(&tmA, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, slices.p, dims, strides, boxA,
                       estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                       CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (cr == CUDA_SUCCESS)
    cr = encode(&tmB, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, slices.p, dims, strides, boxB, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (cr != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed (%d)", (int)cr);
    return RIMP2_ERR_CUDA;
  }
  RIMP2_CK(cudaMemsetAsync(queue.p, 0, sizeof(unsigned int), s));
  if (inject_fault("launch")) {
    set_error("injected launch failure (RIMP2_FAULT_INJECT=launch)");
    return RIMP2_ERR_CUDA;
  }
  if (pair) {
    EosPairParams P;
    P.inv = inv.as<float>();
    P.dcorr = dcorr.as<float>();
    P.eo2 = eo2.as<float2>();
    P.ev2 = ev2.as<float2>();
    P.nitems = nitems;
    P.npart = npart;
    P.queue = queue.as<unsigned int>();
    P.part = part.as<double>();
    P.stash = stash.as<float>();
    P.err = device_error_word();
    P.nvpad = nvpad;
    P.nks = nks;
    P.nt = nt;
    P.ntp = ntp;
    P.per = per;
    P.ncol = (int)ncol;
    P.copies = copies;
    for (int f = 0; f < 3; ++f) P.row0[f] = (int)((long long)f * nks * ncol);
    RIMP2_CK(cudaFuncSetAttribute(split_eos_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  EP_SMEM));
    const int npair = (int)std::min<long long>(nitems, std::max(1, nsm / 2));
    RIMP2_CK(launch_hi(split_eos_pair_kernel, 2 * npair, NTHREADS, EP_SMEM, s, tmA, tmB, P));
  } else {
    EosParams P;
    P.inv = inv.as<float>();
    P.eo2 = eo2.as<float2>();
    P.ev2 = ev2.as<float2>();
    P.nitems = nitems;
    P.queue = queue.as<unsigned int>();
    P.part = part.as<double>();
    P.err = device_error_word();
    P.nocc = nocc;
    P.nvirt = nvirt;
    P.nvpad = nvpad;
    P.nks = nks;
    P.ntp = ntp;
    P.ncol = (int)ncol;
    P.rowC = 0;
    P.rowCt = (int)((long long)nks * ncol);
    RIMP2_CK(cudaFuncSetAttribute(split_eos_kernel<3, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  eos_smem_bytes(3, 3)));
    const int grid = (int)std::min<long long>(nitems, nsm);
    split_eos_kernel<3, 3><<<grid, NTHREADS, eos_smem_bytes(3, 3), s>>>(tmA, tmB, P);
  }
  count_launch(1);
  RIMP2_CK(cudaGetLastError());
  make_pairs_kernel<<<(npairs + 255) / 256, 256, 0, s>>>(nocc, pairs.as<int>());
  count_launch(1);
  for (int c = 0; c < copies; ++c) {
    pair_reduce_kernel<<<(npairs + 7) / 8, 256, 0, s>>>(part.as<double>() + c * npart, nper,
                                                       pairs.as<int>(), npairs, nocc, Epair);
    total_reduce_kernel<<<1, total_threads(nocc), 0, s>>>(Epair, nocc, Etot + c);
    count_launch(2);
  }
  RIMP2_CK(cudaGetLastError());
  return RIMP2_OK;
}

int split_energy(const SplitEnergyArgs &a, cudaStream_t s, float *ms_kernel) {
  (void)ms_kernel;
  // work items pack i | j << 16 and tA | tB << 16
  if (a.nocc > 65535 || (a.nvirt + TILE - 1) / TILE > 65535) {
    set_error("split form: fragment 0 too large for the work-item encoding (nocc=%d)", a.nocc);
    return RIMP2_ERR_ARG;
  }
  int dev = 0, nsm = 0;
  RIMP2_CK(cudaGetDevice(&dev));
  RIMP2_CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  Group g;
  g.nsl = a.nslices >= 2 ? 3 : 2;
  g.pair = a.nslices < 2 && pair_kernel_for(a.nocc, a.nvirt, a.NBA);
  FragDesc F;
  memset(&F, 0, sizeof F);
  F.nocc = a.nocc;
  F.nvirt = a.nvirt;
  F.NBA = a.NBA;
  F.Ca = a.Ca;
  F.eo = a.eo;
  F.ev = a.ev;
  F.Epair = a.Epair;
  F.Etot = a.Etot;
  g.fh.push_back(F);
  RIMP2_TRY(build_group(g, s, true));  // its workspace is released stream-ordered
  const bool timed = timing_enabled();
  cudaEvent_t ev[4];
  if (timed)
    for (int k = 0; k < 4; ++k) RIMP2_CK(cudaEventCreate(&ev[k]));
  RIMP2_TRY(record_group(g, s, nsm, timed ? ev : nullptr, true, true));
  if (timed) {
    RIMP2_CK(cudaEventRecord(ev[3], s));
    RIMP2_CK(cudaEventSynchronize(ev[3]));
    float ms;
    for (int k = 0; k < 3; ++k) {
      RIMP2_CK(cudaEventElapsedTime(&ms, ev[k], ev[k + 1]));
      record_timing(k, ms);
    }
    for (int k = 0; k < 4; ++k) cudaEventDestroy(ev[k]);
  }
  return RIMP2_OK;
}

}  // namespace rimp2
