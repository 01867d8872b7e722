// front_end.cu -- Calpha from AO three-centre integrals on the GPU.
//
//   (alpha|a i) = sum_{mu,nu} Cmo(mu,nocc+a) Cmo(nu,i) (alpha|mu nu)
//   V = L L^T (Cholesky of the auxiliary metric)
//   Calpha(:,a,i) = L^{-1} (:|a i)
// so that sum_alpha Calpha(alpha,a,i) Calpha(alpha,b,j) = (ai|V^{-1}|bj).
// The reference starts from Calpha (RIMP2.F90:48-49); this front end has no
// counterpart there.  The AO->MO transform runs either on the FP64 contraction
// of fp64_kernels.cu or on the tcgen05 split GEMM (two residual FP16 slices,
// ~2^-33 relative per product); the Cholesky and the solve are FP64, blocked
// (64) so that all but O(n*64^2) of their work is GEMM:
//   Cholesky: panels of 256 columns, in them 64 at a time (diagonal block in
//             one CTA, rows below solved against it, update of the panel), the
//             rest updated once per panel;
//   solve:    all diagonal-block inverses in one launch, then by halves:
//             X_1, B_2 -= L_21 X_1, X_2 (GEMMs).
#include <cmath>
#include <cstring>
#include <vector>

#include "mod_gemm.cuh"
#include "tc.cuh"

namespace rimp2 {
void count_launch(int n);

namespace {

constexpr int NB = 64;

GemmDesc gdesc() {
  GemmDesc g;
  memset(&g, 0, sizeof g);
  g.alpha = 1.0;
  g.beta = 0.0;
  g.nb0 = g.nb1 = 1;
  return g;
}

// Diagonal 64x64 blocks: triangular inverse in shared memory, 256 threads.
// Blocks narrower than 64 (the last one) are padded with the identity, so the
// same code runs on every block.
constexpr int DP = NB + 1;                        // padded row (doubles)
constexpr int DIAG_SMEM = (2 * NB * DP + 5 * NB) * sizeof(double);

__device__ __forceinline__ void load_block(double (*A)[DP], const double *V, int n, int k0, int b) {
  for (int t = threadIdx.x; t < NB * NB; t += blockDim.x) {
    const int r = t & (NB - 1), c = t >> 6;
    A[r][c] = (r < b && c < b) ? V[(size_t)(k0 + r) + (size_t)n * (k0 + c)] : (r == c ? 1.0 : 0.0);
  }
  __syncthreads();
}

// X = A^{-1} for lower-triangular A (both NB x NB in shared memory): row by
// row forward substitution, four threads per column sharing each dot product.
// FP64 arithmetic is scarce on this part, so divisions become one
// reciprocal per row (rdiag, NB doubles of shared memory).
__device__ void tri_inverse(double (*A)[DP], double (*X)[DP], double *part, double *rdiag) {
  const int c = threadIdx.x & (NB - 1), q = threadIdx.x >> 6;  // q = 0..3
  if (threadIdx.x < NB) rdiag[threadIdx.x] = 1.0 / A[threadIdx.x][threadIdx.x];
  __syncthreads();
  for (int r = 0; r < NB; ++r) {
    double s = 0.0;
    for (int p = c + q; p < r; p += 4) s += A[r][p] * X[p][c];
    part[q * NB + c] = s;
    __syncthreads();
    if (q == 0) {
      const double d = (r == c ? 1.0 : 0.0) - (part[c] + part[NB + c] + part[2 * NB + c] +
                                               part[3 * NB + c]);
      X[r][c] = (c <= r) ? d * rdiag[r] : 0.0;
    }
    __syncthreads();
  }
}

constexpr int PS = NB + 4;  // padded row (doubles): DMMA operands from two rows of banks
__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// Sixteen columns of L D L^T in a warp: lane (r, h) holds row r's columns 2 j + h
// (the upper triangle comes along), left over their pivots.  first: the first
// pivot that is not positive (16: none); dmine: pivot r.  True if a reciprocal
// was out of range: then SLOW with the block's values again.
template <bool SLOW>
__device__ __forceinline__ bool factor16(double (&a)[8], int lane, double &dmine, int &first) {
  const int r = lane & 15, h = lane >> 4;
  bool odd = false;
  dmine = 1.0;
  first = 16;
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const double d = __shfl_sync(0xffffffffu, a[k >> 1], k + 16 * (k & 1));
    const double ark = __shfl_sync(0xffffffffu, a[k >> 1], r + 16 * (k & 1));
    const long long bits = __double_as_longlong(d);
    const bool ok = bits > 0 && bits <= 0x7FF0000000000000ll;  // d > 0
    first = !ok && first == 16 ? k : first;
    dmine = r == k && ok ? d : dmine;
    const double q = ok ? (SLOW ? 1.0 / d : recip_pos(d, odd)) : 1.0;
    const double f = -q * ark;
#pragma unroll
    for (int j = (k + 1) >> 1; j < 8; ++j) {  // columns past k: of j = k / 2 only the odd one
      double t = __shfl_sync(0xffffffffu, ark, 2 * j + h);
      if (2 * j == k) t = h ? t : 0.0;
      a[j] = fma(f, t, a[j]);
    }
  }
  return odd;
}

// In-place Cholesky of the b x b diagonal block at (k0,k0) of V (ld n); *bad =
// pivot+1 on a non-positive pivot; Dinv: the inverses of the first three of its
// four 16 x 16 diagonal blocks.  One CTA: the chain of 64 pivots bounds it, and in
// it the FP64 instructions of a warp, one in 64 clocks (each scheduler's unit does
// half an FMA a clock, idle lanes count): two lanes share a row.
// Sixteen columns at a time: their diagonal block in warp 0, columns over
// their pivot, the square roots at the end; the rows below by substitution
// (warps 1 to 3); then the next diagonal block with DMMA, the rest beside that
// block's factorisation on the other schedulers, as a warp of its own forms the
// block's inverse.  In us: 143 as a rank-one update per
// column with the inverse, 69 with the block in registers and a barrier per
// column, 71 as here with a lane per row (11 of them a block, 5.3 a
// substitution), 82 with the rows below in the lanes of the block's warp, 52 with
// the rest updated before the next block.
constexpr int PT = 384;
__global__ void __launch_bounds__(PT) potrf_block_kernel(double *V, int n, int k0, int b, int *bad,
                                                         double *Dinv) {
  __shared__ double A[NB][PS];
  __shared__ double rd[NB];  // 1 / L(k, k)
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, gid = lane >> 2, tig = lane & 3;
  const int r = lane & 15, h = lane >> 4;
  grid_wait();
#pragma unroll
  for (int t = threadIdx.x; t < NB * NB; t += PT) {
    const int i = t & (NB - 1), c = t >> 6;
    A[i][c] = i < b && c <= i ? V[(size_t)(k0 + i) + (size_t)n * (k0 + c)] : (i == c ? 1.0 : 0.0);
  }
  __syncthreads();
  if (w >= 8) {  // inverse of block w - 9: column `lane` by forward substitution
    if (w == 8) return;
    asm volatile("bar.sync %0, 288;" ::"r"(w - 7) : "memory");
    const int o = 16 * (w - 9);
    double x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = i == lane ? 1.0 : 0.0;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      x[i] *= rd[o + i];
#pragma unroll
      for (int p = i + 1; p < 16; ++p) x[p] = fma(-A[o + p][o + i], x[i], x[p]);
    }
    if (lane < 16)
#pragma unroll
      for (int i = 0; i < 16; ++i) Dinv[(w - 9) * 256 + i * 16 + lane] = x[i];
    return;
  }
  // 8 x 8 tile t of the lower triangle right of and below the 16 columns at o
  auto update = [&](int o, int t) {
    int ti = 0;
    while ((ti + 1) * (ti + 2) / 2 <= t) ++ti;
    const int r0 = o + 16 + 8 * ti, c0 = o + 16 + 8 * (t - ti * (ti + 1) / 2);
    double d0 = A[r0 + gid][c0 + 2 * tig], d1 = A[r0 + gid][c0 + 2 * tig + 1];
#pragma unroll
    for (int k = 0; k < 16; k += 4) dmma(d0, d1, -A[r0 + gid][o + k + tig], A[c0 + gid][o + k + tig]);
    A[r0 + gid][c0 + 2 * tig] = d0;
    A[r0 + gid][c0 + 2 * tig + 1] = d1;
  };
#pragma unroll 1
  for (int o = 0; o < NB; o += 16) {
    if (o > 0 && (w & 3) != 0) {  // the other tiles of the columns before
      const int n8 = (NB - o) / 8;
      for (int t = 3 + (w & 3) - 1 + 3 * (w >> 2); t < n8 * (n8 + 1) / 2; t += 6) update(o - 16, t);
    }
    if (w == 0) {
      double a[8], dmine;
      int first;
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] = r >= 2 * j + h ? A[o + r][o + 2 * j + h] : A[o + 2 * j + h][o + r];
      bool odd = factor16<false>(a, lane, dmine, first);
      double s = rsqrt_pos(dmine, odd);
      if (__any_sync(0xffffffffu, odd)) {
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] = r >= 2 * j + h ? A[o + r][o + 2 * j + h] : A[o + 2 * j + h][o + r];
        factor16<true>(a, lane, dmine, first);
        s = 1.0 / sqrt(dmine);
      }
      if (lane == 0 && first < 16) atomicCAS(bad, 0, k0 + o + first + 1);
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const double v = a[j] * __shfl_sync(0xffffffffu, s, 2 * j + h);
        if (r >= 2 * j + h) A[o + r][o + 2 * j + h] = v;
      }
      if (lane < 16) rd[o + r] = s;
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");
    if (o < 48) asm volatile("bar.arrive %0, 288;" ::"r"(2 + o / 16) : "memory");
    const int row = o + 16 * w + r;
    if (w >= 1 && w <= 3 && row < NB) {  // lane (r, h): its row's columns 2 j + h
      double x[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) x[j] = A[row][o + 2 * j + h];
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        const double xc = __shfl_sync(0xffffffffu, x[c >> 1] * rd[o + c], r + 16 * (c & 1));
        if (h == (c & 1)) x[c >> 1] = xc;
#pragma unroll
        for (int j = (c + 1) >> 1; j < 8; ++j) {
          double l = A[o + 2 * j + h][o + c];
          if (2 * j == c) l = h ? l : 0.0;
          x[j] = fma(-l, xc, x[j]);
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) A[row][o + 2 * j + h] = x[j];
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");
    // the next diagonal block's three tiles
    if (o < 48 && w >= 1 && w <= 3) update(o, w - 1);
    asm volatile("bar.sync 1, 256;" ::: "memory");
  }
#pragma unroll 8
  for (int x = 0; x < NB * NB / 256; ++x) {
    const int t = threadIdx.x + 256 * x, i = t & (NB - 1), c = t >> 6;
    if (i < b && c < b) V[(size_t)(k0 + i) + (size_t)n * (k0 + c)] = i >= c ? A[i][c] : 0.0;
  }
}

// X := X L^{-T} for the rows [k0+64, n) of the block column at k0, L its
// factored diagonal block: eight rows per CTA (136 CTAs at n = 1152).  Sixteen
// columns at a time: times the inverse of L_ll (Dinv; the last one is formed here by
// warp 4 meanwhile), then the later columns less X_l L_jl^T, with DMMA m8n8k4.
// A scheduler's unit takes 576 clocks for one of those, so that each product of
// 16 columns is dealt to the four warps: warp (y, z) takes its columns 8 y .. 8 y + 7
// and the terms 8 z .. 8 z + 7 of its sums; the two parts meet in shared memory.
// (In us: 34 column by column, with one chain of 64 dependent steps; 28 with a
// warp for each 16 columns and all inverses formed here first, 22 without those.)
__global__ void __launch_bounds__(160) panel_solve_kernel(double *V, int n, int k0, const double *Dinv) {
  __shared__ double Ls[NB][PS];     // L(j, c), with the inverses of its 16 x 16 diagonal blocks
  __shared__ double Ps[2][8][20];   // sixteen columns of the rows after the updates, in two parts
  __shared__ double Xs[2][8][PS];   // the solution, in two parts
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, gid = lane >> 2, tig = lane & 3;
  const int row0 = k0 + NB + blockIdx.x * 8;
  grid_wait();
  const int y = w & 1, z = w >> 1;
  double acc[4][2];  // rows gid, columns 16 j + 8 y + 2 tig + {0, 1}
  if (w < 4) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        acc[j][h] = z == 0 && row0 + gid < n
                        ? V[(size_t)(row0 + gid) + (size_t)n * (k0 + 16 * j + 8 * y + 2 * tig + h)]
                        : 0.0;
#pragma unroll 16
    for (int x = 0; x < NB * NB / 128; ++x) {
      const int t = threadIdx.x + 128 * x, j = t & (NB - 1), c = t >> 6;
      const bool inv = (j >> 4) == (c >> 4) && c < 48;
      Ls[j][c] = inv ? Dinv[(c >> 4) * 256 + (j & 15) * 16 + (c & 15)] : V[(size_t)(k0 + j) + (size_t)n * (k0 + c)];
    }
  }
  __syncthreads();
  if (w == 4) {  // inverse of L_33 by forward substitution: lane (c, h), column c's rows 2 j + h
    constexpr int o = 48;
    const int c = lane & 15, h = lane >> 4;
    const double mine = recip_f64(Ls[o + c][o + c]);
    double x[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = 2 * j + h == c ? 1.0 : 0.0;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const double q = __shfl_sync(0xffffffffu, mine, i);
      const double xi = __shfl_sync(0xffffffffu, x[i >> 1] * q, c + 16 * (i & 1));
      if (h == (i & 1)) x[i >> 1] = xi;
#pragma unroll
      for (int j = (i + 1) >> 1; j < 8; ++j) {
        double l = Ls[o + 2 * j + h][o + i];
        if (2 * j == i) l = h ? l : 0.0;
        x[j] = fma(-l, xi, x[j]);
      }
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 8; ++j) Ls[o + 2 * j + h][o + c] = x[j];
    asm volatile("bar.arrive 2, 160;" ::: "memory");
    return;
  }
#pragma unroll
  for (int l = 0; l < 4; ++l) {
#pragma unroll
    for (int h = 0; h < 2; ++h) Ps[z][gid][8 * y + 2 * tig + h] = acc[l][h];
    if (l < 3)
      asm volatile("bar.sync 1, 128;" ::: "memory");
    else
      asm volatile("bar.sync 2, 160;" ::: "memory");  // and the last inverse
    double x[2] = {0.0, 0.0};
#pragma unroll
    for (int k = 8 * z; k < 8 * z + 8; k += 4)  // X(r, c) = sum_k P(r, k) Inv(c, k)
      dmma(x[0], x[1], Ps[0][gid][k + tig] + Ps[1][gid][k + tig], Ls[16 * l + 8 * y + gid][16 * l + k + tig]);
#pragma unroll
    for (int h = 0; h < 2; ++h) Xs[z][gid][16 * l + 8 * y + 2 * tig + h] = x[h];
    asm volatile("bar.sync 1, 128;" ::: "memory");
#pragma unroll
    for (int k = 8 * z; k < 8 * z + 8; k += 4) {
      if (l == 3) break;
      const double v = -(Xs[0][gid][16 * l + k + tig] + Xs[1][gid][16 * l + k + tig]);
#pragma unroll
      for (int j = l + 1; j < 4; ++j) dmma(acc[j][0], acc[j][1], v, Ls[16 * j + 8 * y + gid][16 * l + k + tig]);
    }
  }
  for (int t = threadIdx.x; t < 8 * NB; t += 128) {
    const int r = t & 7, c = t >> 3;
    if (row0 + r < n) V[(size_t)(row0 + r) + (size_t)n * (k0 + c)] = Xs[0][r][c] + Xs[1][r][c];
  }
}

__global__ void zero_upper_kernel(double *V, int n) {
  const int c = blockIdx.y * blockDim.y + threadIdx.y;
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < n && r < c) V[(size_t)r + (size_t)n * c] = 0.0;
}

// Inverses of every diagonal block of the lower-triangular L (one CTA per
// block) into Linv (nblk x NB x NB).
__global__ void __launch_bounds__(256) tri_inverse_blocks_kernel(const double *L, int n,
                                                                double *Linv) {
  extern __shared__ double dsm[];
  double(*A)[DP] = reinterpret_cast<double(*)[DP]>(dsm);
  double(*X)[DP] = reinterpret_cast<double(*)[DP]>(dsm + NB * DP);
  double *part = dsm + 2 * NB * DP;
  double *rdiag = part + 4 * NB;
  const int k0 = blockIdx.x * NB;
  const int b = n - k0 < NB ? n - k0 : NB;
  load_block(A, L, n, k0, b);
  // only the lower triangle of L is meaningful
  for (int t = threadIdx.x; t < NB * NB; t += blockDim.x) {
    const int r = t & (NB - 1), c = t >> 6;
    if (r < c) A[r][c] = 0.0;
  }
  __syncthreads();
  tri_inverse(A, X, part, rdiag);
  double *out = Linv + (size_t)blockIdx.x * NB * NB;
  for (int t = threadIdx.x; t < NB * NB; t += blockDim.x) out[t] = X[t & (NB - 1)][t >> 6];
}

// The shared-memory opt-in is per device: set it on the current device.
int diag_kernels_init() {
  if (cudaFuncSetAttribute(tri_inverse_blocks_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           DIAG_SMEM) != cudaSuccess) {
    set_error("diagonal-block kernels: shared-memory attribute failed");
    return RIMP2_ERR_CUDA;
  }
  return RIMP2_OK;
}

}  // namespace

// V (n x n, ld n, device) -> lower Cholesky factor in place (strict upper
// zeroed).  Returns RIMP2_ERR_ARG if V is not positive definite.  Two levels:
// inside a panel of 256 columns, per 64 of them the diagonal block is factored
// (one CTA), the rows below solved against it and the panel's remaining
// columns updated; the columns right of the panel are updated once, over its
// whole width (a product of 256 terms a sum, which the residue form takes).
constexpr int CH_PANEL = 256;
int dev_cholesky(int n, double *V, cudaStream_t s) {
  DevBuf bad, dinv;  // dinv: inverses of a diagonal block's 16 x 16 blocks
  RIMP2_TRY(bad.alloc(sizeof(int), s));
  RIMP2_TRY(dinv.alloc(sizeof(double) * 3 * 256, s));
  RIMP2_CK(cudaMemsetAsync(bad.p, 0, sizeof(int), s));
  // C(r0.., c0 .. c0+nc) -= P(r0..) P(c0 .. c0+nc)^T, P the columns [k0, k0 + K)
  auto update = [&](int r0, int c0, int nc, int k0, int K, bool lower) -> int {
    GemmDesc g = gdesc();
    g.M = n - r0;
    g.N = nc;
    g.K = K;
    g.alpha = -1.0;
    g.beta = 1.0;
    g.lower = lower ? 1 : 0;
    g.A = V + (size_t)r0 + (size_t)n * k0;
    g.sAm = 1;
    g.sAk = n;
    g.B = V + (size_t)c0 + (size_t)n * k0;
    g.sBk = n;
    g.sBn = 1;
    g.C = V + (size_t)r0 + (size_t)n * c0;
    g.sCm = 1;
    g.sCn = n;
    return launch_gemm_f64(g, s);
  };
  for (int p0 = 0; p0 < n; p0 += CH_PANEL) {
    const int p1 = n - p0 < CH_PANEL ? n : p0 + CH_PANEL;
    for (int k0 = p0; k0 < p1; k0 += NB) {
      const int b = n - k0 < NB ? n - k0 : NB;
      RIMP2_CK(launch_ex(false, true, potrf_block_kernel, 1, PT, 0, s, V, n, k0, b, bad.as<int>(), dinv.as<double>()));
      count_launch(1);
      const int r0 = k0 + b;
      if (r0 >= n) break;
      RIMP2_CK(launch_ex(false, true, panel_solve_kernel, (n - r0 + 7) / 8, 160, 0, s, V, n, k0,
                         (const double *)dinv.as<double>()));
      count_launch(1);
      if (r0 < p1) RIMP2_TRY(update(r0, r0, p1 - r0, k0, NB, false));
    }
    if (p1 < n) RIMP2_TRY(update(p1, p1, n - p1, p0, p1 - p0, true));
  }
  zero_upper_kernel<<<dim3((n + 63) / 64, (n + 3) / 4), dim3(64, 4), 0, s>>>(V, n);
  count_launch(1);
  RIMP2_CK(cudaGetLastError());
  int h = 0;
  RIMP2_CK(cudaMemcpyAsync(&h, bad.p, sizeof(int), cudaMemcpyDeviceToHost, s));
  // an update that gave up leaves anything behind, also a pivot that is not positive
  RIMP2_TRY(collect_device_error(s));
  if (h) {
    set_error("auxiliary metric is not positive definite (pivot %d)", h - 1);
    return RIMP2_ERR_ARG;
  }
  return RIMP2_OK;
}

// Rows [k0, k0 + nn) of X = L^{-1} B: the first half, B -= L21 X of the second,
// the second half; 64 rows by the inverse of their diagonal block.  Halving
// keeps the products' sums long (n/2, n/4, ...): 2.1 n m updated elements at
// n = 1152 where 64 columns at a time update 9 n m.
static int trsm_rows(int n, int m, int k0, int nn, const double *L, const double *inv, double *B,
                     double *X, cudaStream_t s) {
  GemmDesc g = gdesc();
  g.N = m;
  g.sAm = 1;
  g.sBk = 1;
  g.sBn = n;
  g.sCm = 1;
  g.sCn = n;
  if (nn <= NB) {  // X_k = inv(L_kk) B_k
    g.M = nn;
    g.K = nn;
    g.A = inv + (size_t)(k0 / NB) * NB * NB;
    g.sAk = NB;
    g.B = B + k0;
    g.C = X + k0;
    return launch_gemm_f64(g, s);
  }
  const int n1 = (nn / 2 + NB - 1) / NB * NB;
  RIMP2_TRY(trsm_rows(n, m, k0, n1, L, inv, B, X, s));
  g.M = nn - n1;
  g.K = n1;
  g.alpha = -1.0;
  g.beta = 1.0;
  g.A = L + (size_t)(k0 + n1) + (size_t)n * k0;
  g.sAk = n;
  g.B = X + k0;
  g.C = B + k0 + n1;
  RIMP2_TRY(launch_gemm_f64(g, s));
  return trsm_rows(n, m, k0 + n1, nn - n1, L, inv, B, X, s);
}

// X = L^{-1} B for B (n x m, ld n).  B is overwritten (used as workspace).
// The inverses of all diagonal blocks come from one launch.
int dev_trsm_lower(int n, int m, const double *L, double *B, double *X, cudaStream_t s) {
  RIMP2_TRY(diag_kernels_init());
  const int nblk = (n + NB - 1) / NB;
  DevBuf inv;
  RIMP2_TRY(inv.alloc(sizeof(double) * NB * NB * (size_t)nblk, s));
  tri_inverse_blocks_kernel<<<nblk, 256, DIAG_SMEM, s>>>(L, n, inv.as<double>());
  count_launch(1);
  RIMP2_CK(cudaGetLastError());
  return trsm_rows(n, m, 0, n, L, inv.as<double>(), B, X, s);
}

// (alpha|a i) from (alpha|mu nu) and the MO coefficients
int dev_ao2mo(int NBA, int nbas, int nocc, int nvirt, const double *ao, const double *Cmo,
              double *out, cudaStream_t s) {
  const long long rows = (long long)NBA * nbas;
  if (rows > 2147483647LL) {
    set_error("ao2mo: NBA*nbas too large");
    return RIMP2_ERR_ARG;
  }
  DevBuf half;
  RIMP2_TRY(half.alloc(sizeof(double) * (size_t)rows * nocc, s));
  {  // half(alpha,mu,i) = sum_nu ao(alpha,mu,nu) Cmo(nu,i)
    GemmDesc g = gdesc();
    g.M = (int)rows;
    g.N = nocc;
    g.K = nbas;
    g.A = ao;
    g.sAm = 1;
    g.sAk = rows;
    g.B = Cmo;
    g.sBk = 1;
    g.sBn = nbas;
    g.C = half.as<double>();
    g.sCm = 1;
    g.sCn = rows;
    RIMP2_TRY(launch_gemm_f64(g, s));
  }
  {  // out(alpha,a,i) = sum_mu half(alpha,mu,i) Cmo(mu,nocc+a)
    GemmDesc g = gdesc();
    g.M = NBA;
    g.N = nvirt;
    g.K = nbas;
    g.A = half.as<double>();
    g.sAm = 1;
    g.sAk = NBA;
    g.sAb0 = rows;
    g.B = Cmo + (size_t)nbas * nocc;
    g.sBk = 1;
    g.sBn = nbas;
    g.C = out;
    g.sCm = 1;
    g.sCn = NBA;
    g.sCb0 = (long long)NBA * nvirt;
    g.nb0 = nocc;
    RIMP2_TRY(launch_gemm_f64(g, s));
  }
  return RIMP2_OK;
}

// (alpha|a i) on the tcgen05 tensor cores with exact-integer FP16 slices
// (S0 + two residual slices, ~2^-33 relative per product): the AO tensor is
// sliced with K = nu contiguous (rows mu + nbas*alpha), contracted with the
// occupied MO columns into half(i, alpha, mu), which is sliced again (rows
// (alpha, i), K = mu) and contracted with the virtual MO columns, written in
// the Calpha layout (alpha, a, i).
int dev_ao2mo_split(int NBA, int nbas, int nocc, int nvirt, const double *ao, const double *Cmo,
                    double *out, cudaStream_t s) {
  const int nsl = 3;
  const long long MK = (long long)NBA * nbas;
  DevBuf half;
  RIMP2_TRY(half.alloc(sizeof(double) * (size_t)MK * nocc, s));
  bool fused = false;
  RIMP2_TRY(ao_half_fused(ao, NBA, nbas, Cmo, nocc, half.as<double>(), s, &fused));
  if (!fused) {
    SlicedOp Aao, Bocc;
    RIMP2_TRY(sliced_ao(Aao, ao, NBA, nbas, nsl, s));
    RIMP2_TRY(sliced_cols(Bocc, Cmo, nbas, nocc, 1, nsl, s));
    // half[i][alpha][mu] = sum_nu ao(alpha,mu,nu) Cmo(nu,i); GEMM row m' = mu + nbas*alpha
    RIMP2_TRY(split_gemm(Aao, 0, 0, Bocc, 0, 0, (int)MK, nocc, 1, half.as<double>(), 1, MK, 0, s));
  }
  SlicedOp Ah, Bv;
  RIMP2_TRY(sliced_cols(Ah, half.as<double>(), nbas, NBA, nocc, nsl, s));
  RIMP2_TRY(sliced_cols(Bv, Cmo + (size_t)nbas * nocc, nbas, nvirt, 1, nsl, s));
  // out(alpha,a,i) = sum_mu half[i][alpha][mu] Cmo(mu,nocc+a)
  RIMP2_TRY(split_gemm(Ah, 0, Ah.rows_per_group, Bv, 0, 0, NBA, nvirt, nocc, out, 1, NBA,
                       (long long)NBA * nvirt, s));
  return RIMP2_OK;
}

int dev_calpha_from_ao(int NBA, int nbas, int nocc, int nvirt, const double *ao, const double *V,
                       const double *Cmo, double *Calpha, cudaStream_t s, bool split_transform) {
  DevBuf L, B;
  RIMP2_TRY(L.alloc(sizeof(double) * (size_t)NBA * NBA, s));
  RIMP2_CK(cudaMemcpyAsync(L.p, V, sizeof(double) * (size_t)NBA * NBA, cudaMemcpyDeviceToDevice, s));
  RIMP2_TRY(dev_cholesky(NBA, L.as<double>(), s));
  RIMP2_TRY(B.alloc(sizeof(double) * (size_t)NBA * nvirt * nocc, s));
  if (split_transform)
    RIMP2_TRY(dev_ao2mo_split(NBA, nbas, nocc, nvirt, ao, Cmo, B.as<double>(), s));
  else
    RIMP2_TRY(dev_ao2mo(NBA, nbas, nocc, nvirt, ao, Cmo, B.as<double>(), s));
  RIMP2_TRY(dev_trsm_lower(NBA, nvirt * nocc, L.as<double>(), B.as<double>(), Calpha, s));
  return RIMP2_OK;
}

}  // namespace rimp2

using namespace rimp2;

extern "C" int rimp2_calpha_from_ao_dev(int NBA, int nbas, int nocc, int nvirt, const double *dao,
                                        const double *dV, const double *dCmo, double *dCalpha,
                                        void *stream) {
  clear_error();
  RIMP2_REQ(NBA > 0 && nbas > 0 && nocc > 0 && nvirt > 0 && nocc + nvirt <= nbas,
            "rimp2_calpha_from_ao_dev: bad dims (need nocc+nvirt <= nbas)");
  RIMP2_REQ(dao && dV && dCmo && dCalpha, "rimp2_calpha_from_ao_dev: null array");
  RIMP2_TRY(ensure_device());
  cudaStream_t s = stream ? (cudaStream_t)stream : current_stream();
  return dev_calpha_from_ao(NBA, nbas, nocc, nvirt, dao, dV, dCmo, dCalpha, s, false);
}

extern "C" int rimp2_ao2mo_dev(int NBA, int nbas, int nocc, int nvirt, const double *dao,
                               const double *dCmo, double *dout, int split, void *stream) {
  clear_error();
  RIMP2_REQ(NBA > 0 && nbas > 0 && nocc > 0 && nvirt > 0 && nocc + nvirt <= nbas,
            "rimp2_ao2mo_dev: bad dims (need nocc+nvirt <= nbas)");
  RIMP2_REQ(dao && dCmo && dout, "rimp2_ao2mo_dev: null array");
  RIMP2_TRY(ensure_device());
  cudaStream_t s = stream ? (cudaStream_t)stream : current_stream();
  return split ? dev_ao2mo_split(NBA, nbas, nocc, nvirt, dao, dCmo, dout, s)
               : dev_ao2mo(NBA, nbas, nocc, nvirt, dao, dCmo, dout, s);
}

extern "C" int rimp2_calpha_from_ao_split_dev(int NBA, int nbas, int nocc, int nvirt,
                                              const double *dao, const double *dV,
                                              const double *dCmo, double *dCalpha, void *stream) {
  clear_error();
  RIMP2_REQ(NBA > 0 && nbas > 0 && nocc > 0 && nvirt > 0 && nocc + nvirt <= nbas,
            "rimp2_calpha_from_ao_split_dev: bad dims (need nocc+nvirt <= nbas)");
  RIMP2_REQ(dao && dV && dCmo && dCalpha, "rimp2_calpha_from_ao_split_dev: null array");
  RIMP2_TRY(ensure_device());
  cudaStream_t s = stream ? (cudaStream_t)stream : current_stream();
  return dev_calpha_from_ao(NBA, nbas, nocc, nvirt, dao, dV, dCmo, dCalpha, s, true);
}

extern "C" int rimp2_calpha_from_ao(const int *NBA, const int *nbas, const int *nocc,
                                    const int *nvirt, const double *ao, const double *V,
                                    const double *Cmo, double *Calpha) {
  clear_error();
  RIMP2_REQ(NBA && nbas && nocc && nvirt && *NBA > 0 && *nbas > 0 && *nocc > 0 && *nvirt > 0 &&
                *nocc + *nvirt <= *nbas,
            "rimp2_calpha_from_ao: bad dims (need nocc+nvirt <= nbas)");
  RIMP2_REQ(ao && V && Cmo && Calpha, "rimp2_calpha_from_ao: null array");
  RIMP2_TRY(ensure_device());
  cudaStream_t s = current_stream();
  const size_t nb = *NBA, n = *nbas;
  DevBuf dao, dV, dC, dOut;
  RIMP2_TRY(dao.alloc(sizeof(double) * nb * n * n, s));
  RIMP2_CK(cudaMemcpyAsync(dao.p, ao, sizeof(double) * nb * n * n, cudaMemcpyHostToDevice, s));
  RIMP2_TRY(dV.alloc(sizeof(double) * nb * nb, s));
  RIMP2_CK(cudaMemcpyAsync(dV.p, V, sizeof(double) * nb * nb, cudaMemcpyHostToDevice, s));
  RIMP2_TRY(dC.alloc(sizeof(double) * n * n, s));
  RIMP2_CK(cudaMemcpyAsync(dC.p, Cmo, sizeof(double) * n * n, cudaMemcpyHostToDevice, s));
  const size_t no = (size_t)nb * *nvirt * *nocc;
  RIMP2_TRY(dOut.alloc(sizeof(double) * no, s));
  RIMP2_TRY(dev_calpha_from_ao(*NBA, *nbas, *nocc, *nvirt, dao.as<double>(), dV.as<double>(),
                               dC.as<double>(), dOut.as<double>(), s, false));
  RIMP2_CK(cudaMemcpyAsync(Calpha, dOut.p, sizeof(double) * no, cudaMemcpyDeviceToHost, s));
  RIMP2_CK(cudaStreamSynchronize(s));
  RIMP2_CK(cudaGetLastError());
  return collect_device_error(s);
}

extern "C" int rimp2_cholesky_dev(int n, double *dV, void *stream) {
  clear_error();
  RIMP2_REQ(n > 0 && dV, "rimp2_cholesky_dev: bad arguments");
  RIMP2_TRY(ensure_device());
  cudaStream_t s = stream ? (cudaStream_t)stream : current_stream();
  return dev_cholesky(n, dV, s);
}

extern "C" int rimp2_trsm_lower_dev(int n, int m, const double *dL, double *dB, double *dX,
                                    void *stream) {
  clear_error();
  RIMP2_REQ(n > 0 && m > 0 && dL && dB && dX && dB != dX, "rimp2_trsm_lower_dev: bad arguments");
  RIMP2_TRY(ensure_device());
  cudaStream_t s = stream ? (cudaStream_t)stream : current_stream();
  return dev_trsm_lower(n, m, dL, dB, dX, s);
}
