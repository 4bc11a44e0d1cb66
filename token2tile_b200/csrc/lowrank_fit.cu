// Projection fit: matched rank-32 projections Uq, Uk of one attention call.
//
// Replaces `online_u` of the reference operator (token2tile/operator/deploy_step.py:122-149;
// batched variants integrations/sglang/backend/t2t_attn.py:181-239), which runs two [N,128]^T[N,128]
// products per head in fp64 cuBLAS and three cuSOLVER factorisations per head from a Python loop.
// Here the whole fit is three kernels, batched over heads, with no host round trip:
//
//   gram_kernel        G = X^T X on the tcgen05 tensor cores.  One CTA takes a slab of up to 8192 rows
//                      of one head: 128-row tiles arrive by TMA (rows past N read as zeros) and serve
//                      as BOTH operands of a 128 x 128 x 128 product (A = tile^T, B = tile, both
//                      MN-major views of the same shared-memory tile); fp32 accumulator in TMEM.
//                      HBM-bound: every input row is read once.
//   factor_kernel      sums the slabs in a fixed order in fp64 (M = G / N, deterministic) and writes F with
//                      F F^T = M: the symmetric root with the eigenvalues clamped at 1e-8, or, on the query side
//                      and where the clamp cannot matter, the Cholesky factor; for the query side F^-T too.
//   lowrank_kernel     C = Fq^T Fk, its singular triplets by one-sided Jacobi, the 32 largest:
//                      Uq = Fq^-T U_r S_r^(1/2),  Uk = Fk^-T V_r S_r^(1/2) = Fq U_r S_r^(-1/2)
//                      (V = C^T U S^-1 and Fk^-T Fk^T = I).
//
// One-sided (Hestenes) Jacobi orthogonalises the columns of W by plane rotations, W <- W J: for a
// symmetric positive semi-definite M the columns of the limit are e_i v_i, for a general C they are
// s_i u_i.  Eigenvectors of clamped eigenvalues are never normalised: because every clamped eigenvalue has
// the same value c, their joint contribution to f(M) is f(c) (I - sum of the other v v^T), whatever basis
// spans them.
//
// Whole fit: 2.2 ms at 2 heads x 4096 rows of clustered activations, 2.4 ms at 40 x 75,600, of which the last kernel's sweeps
// are 1.4 to 1.5 ms (1.84 ms with independent normal rows, 3.8 to 4.2 where a root needs its eigenvectors); 5.9 to 9.8 ms
// with both roots by Jacobi sweeps through shared memory.
#include <cuda.h>

#include "common.cuh"
#include "internal.h"
#include "t2t_b200.h"

namespace t2t {

// ---------------------------------------------------------------------------
// Gram matrices
// ---------------------------------------------------------------------------
constexpr int GR_ROWS = 128;                 // rows per tile
constexpr int GR_SLAB_TILES = 64;            // tiles per CTA: 8192 rows in one fp32 accumulation
constexpr int GR_TILE = GR_ROWS * kD * 2;    // 32 KB
constexpr int GR_STAGES = 3;
constexpr int GR_SMEM = GR_STAGES * GR_TILE + 128 + 1024;

__host__ __device__ inline int gram_slabs(int N) { return cdiv(cdiv(N, GR_ROWS), GR_SLAB_TILES); }

__global__ void __launch_bounds__(128) gram_kernel(const __grid_constant__ CUtensorMap mapQ,
                                                   const __grid_constant__ CUtensorMap mapK, float* __restrict__ partial,
                                                   int N, int* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (base - smem_u32(smem_raw));
  uint64_t* full = reinterpret_cast<uint64_t*>(sm + GR_STAGES * GR_TILE);      // [GR_STAGES] tile landed
  uint64_t* freeb = full + GR_STAGES;                                          // [GR_STAGES] products that read it finished
  uint64_t* done = freeb + GR_STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + GR_STAGES * GR_TILE + 64);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + GR_STAGES * GR_TILE + 72);

  const int tid = threadIdx.x, warp = tid >> 5;
  const int slab = blockIdx.x, h = blockIdx.y, slabs = gridDim.x;
  const int m = blockIdx.z * gridDim.y + h;      // matrix: the query side's first, then the key side's
  const CUtensorMap* map = blockIdx.z ? &mapK : &mapQ;
  const int tile0 = slab * GR_SLAB_TILES;
  const int ntiles = min(GR_SLAB_TILES, cdiv(N, GR_ROWS) - tile0);

  if (warp == 0) {
    tmem_alloc(tmem_slot, 128);
    tmem_relinquish();
  }
  if (tid == 0) {
    *abort_flag = 0;
    for (int i = 0; i < 2 * GR_STAGES + 1; ++i) mbar_init(full + i, 1);
    mbar_init_fence();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (tid == 0) {
    // ---- copies: two 64-column halves of a tile per stage ----
    for (int t = 0; t < ntiles; ++t) {
      const int st = t % GR_STAGES;
      if (t >= GR_STAGES && !mbar_wait(freeb + st, ((t / GR_STAGES) - 1) & 1, abort_flag)) break;
      mbar_arrive_expect_tx(full + st, GR_TILE);
      const uint32_t dst = base + st * GR_TILE;
      tma_load_tile3(dst, map, 0, (tile0 + t) * GR_ROWS, h, full + st);
      tma_load_tile3(dst + GR_ROWS * 128, map, 64, (tile0 + t) * GR_ROWS, h, full + st);
    }
  } else if (tid == 32) {
    // ---- products: G += tile^T tile, eight steps of 16 rows ----
    constexpr uint32_t idesc = make_idesc_bf16(128, 128, true, true);
    constexpr uint32_t dhi = sdesc_hi(1024);
    for (int t = 0; t < ntiles; ++t) {
      const int st = t % GR_STAGES;
      if (!mbar_wait(full + st, (t / GR_STAGES) & 1, abort_flag)) break;
      tc_fence_after();
      const uint32_t lo = sdesc_lo(base + st * GR_TILE, GR_ROWS * 128);
#pragma unroll
      for (int s = 0; s < 8; ++s)
        umma_ss_lo(tmem, lo + s * (2048 >> 4), lo + s * (2048 >> 4), dhi, idesc, (t > 0 || s > 0) ? 1u : 0u);
      umma_commit(freeb + st);
    }
    umma_commit(done);
  }
  __syncwarp();
  const bool ok = mbar_wait_warp(done, 0, abort_flag);
  tc_fence_after();
  if (ok) {
    float* dst = partial + ((size_t)m * slabs + slab) * (kD * kD) + (size_t)tid * kD;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint32_t v[32];
      tmem_ld32(tmem_addr(tmem, warp * 32, c * 32), v);
      tmem_wait_ld();
#pragma unroll
      for (int j = 0; j < 8; ++j)
        reinterpret_cast<uint4*>(dst + c * 32)[j] = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    }
  } else if (tid == 0 && status) {
    atomicCAS(status, ST_OK, ST_WAIT_TIMEOUT);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 128);
}

// ---------------------------------------------------------------------------
// one-sided Jacobi on a 128 x 128 fp64 matrix in shared memory
// ---------------------------------------------------------------------------
constexpr int JD = 128;                  // matrix order
constexpr int JLD = JD + 1;              // column stride in doubles: odd, so that rows can be walked as well as columns
constexpr int J_THREADS = 256;
constexpr int J_MAX_SWEEPS = 18;
constexpr double kJacobiDone2 = 9.0e-16;   // (3e-8)^2, and
constexpr float kJacobiDoneT = 1.0e-6f;    // the tangent of the angle: see jacobi_orthogonalise
constexpr int J_SMEM = JD * JLD * 8 + 2 * JD * 8 + 8 * 8 * 16 + 4 * JD * 8 + 64;
constexpr int F_SMEM = J_SMEM + JD * (JD + 1) / 2 * 8;      // factor_kernel: and a packed triangle
static_assert(J_SMEM % 16 == 0 && F_SMEM <= 227 * 1024, "shared memory of factor_kernel");

__device__ __forceinline__ double shfl_xor_d(double v, int m) {
  return __hiloint2double(__shfl_xor_sync(0xffffffffu, __double2hiint(v), m),
                          __shfl_xor_sync(0xffffffffu, __double2loint(v), m));
}

// Squared norms of the columns of W into nrm2[0..127] (every thread calls it).
__device__ void column_norms2(const double* W, double* nrm2) {
  const int tid = threadIdx.x, col = tid >> 1, sub = tid & 1;
  double acc = 0.0;
#pragma unroll 8
  for (int m = 0; m < 64; ++m) {
    const double x = W[col * JLD + sub + 2 * m];
    acc = fma(x, x, acc);
  }
  acc += shfl_xor_d(acc, 1);
  if (sub == 0) nrm2[col] = acc;
  __syncthreads();
}

// The two column segments a warp holds in registers: lane l has rows l, l + 32, l + 64, l + 96 of every column.  After R
// rounds the top column of pair i (0..7) is in t[(i + R) % 8], the bottom one in b[(i - R) % 8].
struct Columns {
  double t[8][4], b[8][4];
};

// The rotation that makes two columns with squared lengths alpha, beta and product gamma orthogonal.
//
// A round is a chain of dependent steps, and an fp64 step takes about sixteen times as long as an fp32 one, so what
// steers the rotation stays in fp32 where it can: t = tan of the angle is an fp32 value t0 plus an fp32 correction (one
// Newton step on gamma (t^2 - 1) + dx t = 0, its residual from exact fp32 products of the leading and trailing parts of
// gamma and dx; relative error of t 4.6e-14 at most over a million angles, t0 alone 3.2e-7).  The _rn forms are never
// contracted: a product whose rounding error is added back must not be fused with the sum behind it.
// (c, s) is normalised in fp64 to its last bits, so every rotation is orthogonal to fp64 precision.
struct Rotation {
  float t0;
  double t, c, s;
};
__device__ __forceinline__ Rotation rotation(double alpha, double beta, double gamma) {
  const double dx = beta - alpha;
  const float dh = (float)dx, dl = (float)(dx - (double)dh);
  const float gh = (float)gamma, gl = (float)(gamma - (double)gh);
  // the smaller root (in size) of t^2 + dx / gamma t - 1 = 0
  const float fx = fabsf(dh), fy = 2.0f * fabsf(gh);
  const float lo = __fdividef(fminf(fx, fy), fmaxf(fx, fy)), root = sqrtf(fmaf(lo, lo, 1.0f));
  float t0 = __fdividef(fy <= fx ? lo : 1.0f, fy <= fx ? 1.0f + root : lo + root);
  if (dh != 0.0f && (dh < 0.0f) != (gh < 0.0f)) t0 = -t0;
  const float q = __fmul_rn(t0, t0), p = __fsub_rn(q, 1.0f);
  const float pl = __fadd_rn(__fsub_rn(q, __fadd_rn(p, 1.0f)), fmaf(t0, t0, -q));      // t0^2 - 1 = p + pl
  const float a1 = __fmul_rn(gh, p), b1 = __fmul_rn(dh, t0);
  const float low = fmaf(gh, p, -a1) + fmaf(dh, t0, -b1) + fmaf(gh, pl, fmaf(gl, p, dl * t0));
  const float dt = -__fdividef(__fadd_rn(__fadd_rn(a1, b1), low), fmaf(2.0f * gh, t0, dh));
  Rotation r;
  r.t0 = t0;
  r.t = (double)t0 + (double)dt;
  const double y = (double)rsqrtf(fmaf(t0, t0, 1.0f)), y2 = y * y;
  const double ty = r.t * y, h = fma(-fma(r.t, r.t, 1.0), y2, 1.0);         // third-order step: error (1e-7)^3
  const double k = fma(h, 0.375, 0.5);
  r.c = fma(y * h, k, y);
  r.s = fma(ty * h, k, ty);
  return r;
}

// One round: the eight disjoint pairs (top, bottom) of a warp.  cx, cy: column numbers of pair lane & 7, whose angle
// this lane works out.
template <int R>
__device__ __forceinline__ void rotate8(Columns& w, int cx, int cy, double* nrm2, double2* cs, double tiny2, bool& again) {
  const int lane = threadIdx.x & 31;
  const double alpha = nrm2[cx], beta = nrm2[cy];
  double g[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const double(&x)[4] = w.t[(i + R) & 7];
    const double(&y)[4] = w.b[(i + 8 - R) & 7];
    g[i] = fma(x[1], y[1], x[0] * y[0]) + fma(x[3], y[3], x[2] * y[2]);
  }
  // eight sums over the warp: lane l ends up with that of pair l & 7
  const bool b0 = lane & 1, b1 = lane & 2, b2 = lane & 4;
  double u[4], v[2];
#pragma unroll
  for (int i = 0; i < 4; ++i) u[i] = (b0 ? g[2 * i + 1] : g[2 * i]) + shfl_xor_d(b0 ? g[2 * i] : g[2 * i + 1], 1);
#pragma unroll
  for (int i = 0; i < 2; ++i) v[i] = (b1 ? u[2 * i + 1] : u[2 * i]) + shfl_xor_d(b1 ? u[2 * i] : u[2 * i + 1], 2);
  double gamma = (b2 ? v[1] : v[0]) + shfl_xor_d(b2 ? v[0] : v[1], 4);
  gamma += shfl_xor_d(gamma, 8);
  gamma += shfl_xor_d(gamma, 16);
  const Rotation rot = rotation(alpha, beta, gamma);
  const double g2 = gamma * gamma, ab = alpha * beta;
  const bool live = alpha > tiny2 && beta > tiny2 && g2 > 1.0e-27 * ab;
  if (!__any_sync(0xffffffffu, live)) return;
  again = again || (live && (g2 > kJacobiDone2 * ab || fabsf(rot.t0) > kJacobiDoneT));
  if (lane < 8) {
    cs[lane] = live ? make_double2(rot.c, rot.s) : make_double2(1.0, 0.0);
    if (live) {
      nrm2[cx] = fmax(fma(-rot.t, gamma, alpha), 0.0);
      nrm2[cy] = fmax(fma(rot.t, gamma, beta), 0.0);
    }
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const double2 r = cs[i];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const double a = w.t[(i + R) & 7][m], b = w.b[(i + 8 - R) & 7][m];
      w.t[(i + R) & 7][m] = fma(r.x, a, -(r.y * b));
      w.b[(i + 8 - R) & 7][m] = fma(r.y, a, r.x * b);
    }
  }
  __syncwarp();      // cs and nrm2 may be written again
}

// Columns held at round r of the round-robin schedule (127 rounds): column 127 stays at the top of pair 0, the others
// move round a ring of 127.
__device__ __forceinline__ int top_column(int pair, int r) { return pair == 0 ? JD - 1 : (r + pair) % (JD - 1); }
__device__ __forceinline__ int bottom_column(int pair, int r) { return (r + (JD - 1) - pair) % (JD - 1); }

// Round R (mod 8) and the hand-over to the next one: one column enters and one leaves each segment of a warp.  The ring
// runs down the tops (towards pair 0) and up the bottoms: top 1 -> bottom 0, bottom 63 -> top 63.
template <int R>
__device__ __forceinline__ void jacobi_round(Columns& w, int& r, double* xch, double* nrm2, double2* cs, double tiny2, bool& again) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, pair = 8 * warp + (lane & 7);
  rotate8<R>(w, top_column(pair, r), bottom_column(pair, r), nrm2, cs, tiny2, again);
  r = r + 1 < JD - 1 ? r + 1 : 0;
  constexpr int TI = R & 7, TN = (R + 1) & 7, BI = (15 - R) & 7;      // registers of top 0, of top 1, of bottom 7
  double* tops = xch + (R & 1) * 16 * JD;                             // [8 warps][128] column leaving the tops
  double* bots = tops + 8 * JD;                                       // [8 warps][128] column leaving the bottoms
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    tops[warp * JD + lane + 32 * m] = warp == 0 ? w.t[TN][m] : w.t[TI][m];
    bots[warp * JD + lane + 32 * m] = w.b[BI][m];
  }
  if (warp == 0) {      // column 127 keeps its place while the registers' meaning moves on
#pragma unroll
    for (int m = 0; m < 4; ++m) w.t[TN][m] = w.t[TI][m];
  }
  __syncthreads();
  const double* from_top = warp < 7 ? tops + (warp + 1) * JD : bots + 7 * JD;
  const double* from_bot = warp > 0 ? bots + (warp - 1) * JD : tops;
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    w.t[TI][m] = from_top[lane + 32 * m];
    w.b[BI][m] = from_bot[lane + 32 * m];
  }
}

// Rotates column pairs of W (column j at W + j * JLD) until all columns are mutually orthogonal.  Every thread of
// the 256-thread CTA calls it.  W is overwritten meanwhile.
//
// The 64 pairs of a round are disjoint; a warp keeps the sixteen columns of eight neighbouring pairs in registers and
// passes one column of each segment on per round, so shared memory carries 32 KB a round instead of reading the matrix
// twice and writing it once (384 KB).  What bounds a round now is its chain of dependent steps: products, a reduction of
// five shuffles, the angle (worked out once per pair, not by every lane that holds a part of it), the rotation.  The
// order of the rotations fixes the signs of the result, so it is part of what callers see.
// A stretch of 128 rounds in which no pair turned by more than kJacobiDoneT and no cosine exceeded 3e-8 leaves angles of
// the order of its square, 128 x 1e-12, below the rounding of the fp32 factors: it is the last.  Small cosines alone do
// not tell: columns whose lengths agree to 1e-6 have them from the start and may still have to turn by 45 degrees.
__device__ void jacobi_orthogonalise(double* W, double* nrm2, double2* cs_all) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  double2* cs = cs_all + warp * 8;
  __syncthreads();      // W was just written by other threads
  column_norms2(W, nrm2);
  // a power of two brings the largest squared norm to 2^60 or so: the fp32 part of the angles stays in range
  double top = 0.0;
  for (int j = 0; j < JD; ++j) top = fmax(top, nrm2[j]);
  const int shift = top > 0.0 ? max(-500, min(500, (60 - ilogb(top)) / 2)) : 0;
  const double up = scalbn(1.0, shift), down = scalbn(1.0, -shift);
  __syncthreads();      // every thread has read the norms
  if (tid < JD) nrm2[tid] = nrm2[tid] * up * up;
  __syncthreads();
  // columns whose squared norm is below (1e-14 of the largest column)^2 are numerically zero: rotating
  // them against each other never settles and changes nothing that is used
  double big = 0.0;
  for (int j = 0; j < JD; ++j) big = fmax(big, nrm2[j]);
  const double tiny2 = 1.0e-28 * big;
  int r = 0;
  Columns w;
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      w.t[i][m] = W[top_column(8 * warp + i, 0) * JLD + lane + 32 * m] * up;
      w.b[i][m] = W[bottom_column(8 * warp + i, 0) * JLD + lane + 32 * m] * up;
    }
  __syncthreads();      // W now carries the columns that change warps
#pragma unroll 1
  for (int stretch = 0; stretch < J_MAX_SWEEPS; ++stretch) {
    bool again = false;
#pragma unroll 1
    for (int g = 0; g < 16; ++g) {
      jacobi_round<0>(w, r, W, nrm2, cs, tiny2, again);
      jacobi_round<1>(w, r, W, nrm2, cs, tiny2, again);
      jacobi_round<2>(w, r, W, nrm2, cs, tiny2, again);
      jacobi_round<3>(w, r, W, nrm2, cs, tiny2, again);
      jacobi_round<4>(w, r, W, nrm2, cs, tiny2, again);
      jacobi_round<5>(w, r, W, nrm2, cs, tiny2, again);
      jacobi_round<6>(w, r, W, nrm2, cs, tiny2, again);
      jacobi_round<7>(w, r, W, nrm2, cs, tiny2, again);
    }
    if (!__syncthreads_or(again ? 1 : 0)) break;
    // the running norms pick up rounding
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      double x = 0.0, y = 0.0;
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        x = fma(w.t[i][m], w.t[i][m], x);
        y = fma(w.b[i][m], w.b[i][m], y);
      }
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) {
        x += shfl_xor_d(x, d);
        y += shfl_xor_d(y, d);
      }
      if (lane == 0) {
        nrm2[top_column(8 * warp + i, r)] = x;
        nrm2[bottom_column(8 * warp + i, r)] = y;
      }
    }
    __syncwarp();      // the warp's next round reads its own columns' norms
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      W[top_column(8 * warp + i, r) * JLD + lane + 32 * m] = w.t[i][m] * down;
      W[bottom_column(8 * warp + i, r) * JLD + lane + 32 * m] = w.b[i][m] * down;
    }
  __syncthreads();
}

constexpr double kEigFloor = 1.0e-8;     // clamp of the reference (deploy_step.py:137-138)

// Steps 8 M .. 8 M + 7 of cholesky_inverse (which registers hold row and column k must be known when compiling).
template <int M>
__device__ __forceinline__ void cholesky_steps(double (&e)[16][4], double* Lc, double* pub, bool& ok) {
  const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
#pragma unroll 1
  for (int kk = 0; kk < 8 && ok; ++kk) {
    const int k = 8 * M + kk;
    double* col = pub + (k & 1) * 2 * JD;      // two sets in turn: one barrier a step
    double* row = col + JD;                    // multipliers of step k by column
    if (l == (k & 31)) {
#pragma unroll
      for (int m = 0; m < 16; ++m) {
        const int i = w + 8 * m;
        if (i >= k) {
          col[i] = e[m][M / 4];
          if (i > k) row[i] = e[m][M / 4];
        }
      }
    }
    if (w == kk) {
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const int j = l + 32 * n;
        if (j <= k) row[j] = j == k ? 1.0 : e[M][n];
      }
    }
    __syncthreads();
    const double piv = col[k];
    ok = piv > 0.0;                            // the same value in every thread
    if (ok) {
      const double isq = rsqrt(piv), inv = isq * isq;
      if (tid < JD) Lc[k * JLD + tid] = tid >= k ? col[tid] * isq : 0.0;
      double rr[4];
#pragma unroll
      for (int n = 0; n < 4; ++n) rr[n] = row[l + 32 * n] * inv;
#pragma unroll
      for (int m = 0; m < 16; ++m) {
        const int i = w + 8 * m;
        if (i > k) {
          const double c = col[i];
#pragma unroll
          for (int n = 0; n < 4; ++n) e[m][n] = fma(-c, rr[n], l + 32 * n == k ? 0.0 : e[m][n]);
        } else if (i == k) {
#pragma unroll
          for (int n = 0; n < 4; ++n) e[m][n] = l + 32 * n < k ? e[m][n] * isq : (l + 32 * n == k ? isq : 0.0);
        }
      }
    }
  }
}

// Cholesky factor and its inverse of the matrix whose lower triangle is in e: thread (warp w, lane l) holds the
// elements (w + 8 m, l + 32 n).  An element belongs to A until its column's step, to X = L^-1 afterwards: step k
// publishes column k of A and row k of X, and every later row i subtracts A_ik / A_kk times (A_kj for j > k, 1 for
// j = k, X_kj for j < k).  L goes to Lc (column k at Lc + k * JLD, zeros above the diagonal).  pub: 4 x 128 doubles.
// Returns false when a pivot is not positive; otherwise e holds X and the Frobenius norm^2 of X (the trace of the
// inverse matrix) is in *trace.
__device__ __forceinline__ bool cholesky_inverse(double (&e)[16][4], double* Lc, double* pub, double* red, double* trace) {
  const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
  bool ok = true;
  cholesky_steps<0>(e, Lc, pub, ok);
  cholesky_steps<1>(e, Lc, pub, ok);
  cholesky_steps<2>(e, Lc, pub, ok);
  cholesky_steps<3>(e, Lc, pub, ok);
  cholesky_steps<4>(e, Lc, pub, ok);
  cholesky_steps<5>(e, Lc, pub, ok);
  cholesky_steps<6>(e, Lc, pub, ok);
  cholesky_steps<7>(e, Lc, pub, ok);
  cholesky_steps<8>(e, Lc, pub, ok);
  cholesky_steps<9>(e, Lc, pub, ok);
  cholesky_steps<10>(e, Lc, pub, ok);
  cholesky_steps<11>(e, Lc, pub, ok);
  cholesky_steps<12>(e, Lc, pub, ok);
  cholesky_steps<13>(e, Lc, pub, ok);
  cholesky_steps<14>(e, Lc, pub, ok);
  cholesky_steps<15>(e, Lc, pub, ok);
  if (!ok) return false;
  double acc = 0.0;
#pragma unroll
  for (int m = 0; m < 16; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n)
      if (l + 32 * n <= w + 8 * m) acc = fma(e[m][n], e[m][n], acc);
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) acc += shfl_xor_d(acc, d);
  if (l == 0) red[w] = acc;
  __syncthreads();
  double sum = 0.0;
  for (int i = 0; i < 8; ++i) sum += red[i];
  *trace = sum;
  return true;
}

// Sum of v over the CTA (every thread calls it); red: 8 doubles.
__device__ __forceinline__ double block_sum(double v, double* red) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v += shfl_xor_d(v, d);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double sum = 0.0;
#pragma unroll
  for (int i = 0; i < 8; ++i) sum += red[i];
  return sum;
}

// The symmetric root of M = L L^T from its Cholesky factor: L^T = P H with P orthogonal and H = M^(1/2), and P is the
// limit of X <- (X + X^-T) / 2 as well as of X <- X (3 I - X^T X) / 2.  The first form is fast far from the limit and
// costs nothing for the first step, L^-1 being at hand; the second needs products only and doubles the correct digits
// once the singular values of X are near one (it converges below sqrt(3), which the first step ensures for condition
// numbers of M up to a thousand or so).  On entry e holds L^-1 (lower triangle), Lc column k of L at k * JLD; on
// success H is in out (row-major) and in e.  S: 128 * 129 / 2 doubles.  Returns false when the products do not converge.
// A singular value that starts above sqrt(3) may end at minus one and leave a symmetric H that is not positive: the
// caller checks that it is.
__device__ __forceinline__ bool polar_root(double (&e)[16][4], double inv_norm2, double* X, double* S, double* red,
                                           double* out) {
  const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
  for (int i = tid; i < JD * JD; i += J_THREADS) out[i] = X[(i & 127) * JLD + (i >> 7)];      // L, needed at the end
  double part = 0.0;
#pragma unroll
  for (int m = 0; m < 16; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const double lt = X[(w + 8 * m) * JLD + l + 32 * n];      // (L^T)_ij
      part = fma(lt, lt, part);
    }
  const double mu = sqrt(sqrt(inv_norm2 / block_sum(part, red)));
  part = 0.0;
#pragma unroll
  for (int m = 0; m < 16; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const int i = w + 8 * m, j = l + 32 * n;
      const double x = 0.5 * (mu * X[i * JLD + j] + (j <= i ? e[m][n] / mu : 0.0));
      e[m][n] = x;
      part = fma(x, x, part);
    }
  const double scale = sqrt((double)JD / block_sum(part, red));
#pragma unroll
  for (int m = 0; m < 16; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n) X[(w + 8 * m) * JLD + l + 32 * n] = e[m][n] * scale;
  __syncthreads();
  bool done = false;
#pragma unroll 1
  for (int step = 0; step < 9 && !done; ++step) {
#pragma unroll
    for (int m = 0; m < 16; ++m)
#pragma unroll
      for (int n = 0; n < 4; ++n) e[m][n] = 0.0;
#pragma unroll 2
    for (int k = 0; k < JD; ++k) {      // X^T X
      double xb[4];
#pragma unroll
      for (int n = 0; n < 4; ++n) xb[n] = X[k * JLD + l + 32 * n];
#pragma unroll
      for (int m = 0; m < 16; ++m) {
        const double xa = X[k * JLD + w + 8 * m];
#pragma unroll
        for (int n = 0; n < 4; ++n) e[m][n] = fma(xa, xb[n], e[m][n]);
      }
    }
    part = 0.0;
#pragma unroll
    for (int m = 0; m < 16; ++m)
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const int i = w + 8 * m, j = l + 32 * n;
        const double d = e[m][n] - (i == j ? 1.0 : 0.0);
        part = fma(d, d, part);
        if (j <= i) S[i * (i + 1) / 2 + j] = e[m][n];
        e[m][n] = 0.0;
      }
    const double off2 = block_sum(part, red);      // (its barriers publish S)
    if (!(off2 < 1.0e12)) return false;            // diverged, or not a number: the same in every thread
    done = off2 < 1.0e-14;                         // the step below squares 1e-7
#pragma unroll 2
    for (int k = 0; k < JD; ++k) {      // X S
      double sb[4];
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const int j = l + 32 * n;
        sb[n] = S[j <= k ? k * (k + 1) / 2 + j : j * (j + 1) / 2 + k];
      }
#pragma unroll
      for (int m = 0; m < 16; ++m) {
        const double xa = X[(w + 8 * m) * JLD + k];
#pragma unroll
        for (int n = 0; n < 4; ++n) e[m][n] = fma(xa, sb[n], e[m][n]);
      }
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < 16; ++m)
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        double& x = X[(w + 8 * m) * JLD + l + 32 * n];
        x = fma(-0.5, e[m][n], 1.5 * x);
      }
    __syncthreads();
  }
  if (!done) return false;
  // H = L P, symmetric up to rounding
  for (int i = tid; i < JD * JD; i += J_THREADS) {
    const int r = i >> 7, c = i & 127;
    if (c <= r) S[r * (r + 1) / 2 + c] = out[i];
  }
#pragma unroll
  for (int m = 0; m < 16; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n) e[m][n] = 0.0;
  __syncthreads();
#pragma unroll 1
  for (int k = 0; k < JD; ++k) {
    double xb[4];
#pragma unroll
    for (int n = 0; n < 4; ++n) xb[n] = X[k * JLD + l + 32 * n];
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      const int i = w + 8 * m;
      const double la = k <= i ? S[i * (i + 1) / 2 + k] : 0.0;
#pragma unroll
      for (int n = 0; n < 4; ++n) e[m][n] = fma(la, xb[n], e[m][n]);
    }
  }
  __syncthreads();
#pragma unroll
  for (int m = 0; m < 16; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n) X[(w + 8 * m) * JLD + l + 32 * n] = e[m][n];
  __syncthreads();
#pragma unroll
  for (int m = 0; m < 16; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const int i = w + 8 * m, j = l + 32 * n;
      e[m][n] = 0.5 * (X[i * JLD + j] + X[j * JLD + i]);
      out[i * JD + j] = e[m][n];
    }
  __syncthreads();
  return true;
}

// One CTA per second-moment matrix M (blockIdx.x < H: query side, else key side).
//   roots    [2 H][128][128] fp64: F with F F^T = M (eigenvalues clamped), row-major
//   invroots [H][128][128] fp64:   F^-T, query side only
//   bad      [2 H] int: 1 when the matrix holds a non-finite value (non-finite input)
//
// Query side: any factor serves.  With Fq = Mq^(1/2) O for an orthogonal O, the singular value decomposition of
// Fq^T Fk = O^T (Mq^(1/2) Fk) has the same S and V, its U is O^T times the other one, and Fq^-T U is the same matrix;
// one-sided Jacobi, which only sees products of columns, takes the same rotations too.  The Cholesky factor needs 128
// short steps and gives its inverse on the way; it is taken where the clamp cannot matter: where the trace of the
// inverse (an upper bound of 1 / smallest eigenvalue) is below 1 / kEigFloor.
// Key side: the symmetric root (another factor would turn the columns that the rotations work on, and with them the
// signs of the result), from the Cholesky factor where the clamp cannot matter and the products converge, else, and
// on the query side, from the eigenvectors.
__global__ void __launch_bounds__(J_THREADS, 1) factor_kernel(const float* __restrict__ partial, int slabs, int H,
                                                              double inv_n, double* __restrict__ roots,
                                                              double* __restrict__ invroots, int* __restrict__ bad) {
  extern __shared__ __align__(16) uint8_t jsm[];
  double* W = reinterpret_cast<double*>(jsm);
  double* nrm2 = W + JD * JLD;
  double* coef = nrm2 + JD;
  double2* cs = reinterpret_cast<double2*>(coef + JD);
  double* pub = reinterpret_cast<double*>(cs + 8 * 8);
  const int tid = threadIdx.x, m = blockIdx.x;
  const bool want_inv = m < H;

  // M = (sum of the slabs, in slab order) / N; symmetric, so rows can be read as columns
  const float* src = partial + (size_t)m * slabs * (JD * JD);
  auto moment = [&](int idx) {
    double acc = 0.0;
    for (int s = 0; s < slabs; ++s) acc += (double)src[(size_t)s * (JD * JD) + idx];
    return acc * inv_n;
  };
  double* Fo = roots + (size_t)m * JD * JD;
  double* Io = invroots + (size_t)m * JD * JD;
  {
    double e[16][4];
    bool finite = true;
#pragma unroll
    for (int a = 0; a < 16; ++a)
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        e[a][n] = moment(((tid >> 5) + 8 * a) * JD + (tid & 31) + 32 * n);
        finite = finite && isfinite(e[a][n]);
      }
    const int any_bad = __syncthreads_or(finite ? 0 : 1);
    if (tid == 0) bad[m] = any_bad;
    if (any_bad) return;      // the host raises; nothing below would converge on NaNs
    // key side: a second pass shows that the root is positive definite
    bool ok = true;
    int pass = 0;
#pragma unroll 1
    for (;; ++pass) {
      double trace = 0.0;
      ok = cholesky_inverse(e, W, pub, nrm2, &trace);
      __syncthreads();
      if (pass == 0) ok = ok && trace < 1.0 / kEigFloor;
      if (!ok || pass == 1 || want_inv) break;
      ok = polar_root(e, trace, W, reinterpret_cast<double*>(jsm + J_SMEM), nrm2, Fo);
      if (!ok) break;
    }
    if (ok) {
      if (!want_inv) return;
      for (int i = tid; i < JD * JD; i += J_THREADS) Fo[i] = W[(i & 127) * JLD + (i >> 7)];
      __syncthreads();
#pragma unroll
      for (int a = 0; a < 16; ++a)
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          const int i = (tid >> 5) + 8 * a, j = (tid & 31) + 32 * n;
          W[j * JLD + i] = j <= i ? e[a][n] : 0.0;
        }
      __syncthreads();
      for (int i = tid; i < JD * JD; i += J_THREADS) Io[i] = W[(i >> 7) * JLD + (i & 127)];
      return;
    }
  }
  __syncthreads();

  for (int i = tid; i < JD * JD; i += J_THREADS) W[(i >> 7) * JLD + (i & 127)] = moment(i);
  jacobi_orthogonalise(W, nrm2, cs);
  column_norms2(W, nrm2);
  // column i of W is e_i v_i: with l_i = max(e_i, floor),
  //   M^(1/2)  = sqrt(floor) I + sum_i (sqrt(l_i) - sqrt(floor)) v_i v_i^T
  //   M^(-1/2) = floor^(-1/2) I + sum_i (l_i^(-1/2) - floor^(-1/2)) v_i v_i^T
  // and v_i v_i^T = w_i w_i^T / e_i^2; the terms of clamped eigenvalues vanish.
  for (int pass = 0; pass < (want_inv ? 2 : 1); ++pass) {
    if (tid < JD) {
      const double e2 = nrm2[tid], e = sqrt(e2);
      double f = 0.0;
      if (e > kEigFloor) f = (pass == 0 ? sqrt(e) - sqrt(kEigFloor) : 1.0 / sqrt(e) - 1.0 / sqrt(kEigFloor)) / e2;
      coef[tid] = f;
    }
    __syncthreads();
    const int col = tid & 127, r0 = (tid >> 7) * 64;      // 64 rows x 1 column per thread
    double acc[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) acc[i] = 0.0;
    for (int k = 0; k < JD; ++k) {
      const double f = coef[k] * W[k * JLD + col];
#pragma unroll
      for (int i = 0; i < 64; ++i) acc[i] = fma(f, W[k * JLD + r0 + i], acc[i]);
    }
    const double diag = pass == 0 ? sqrt(kEigFloor) : 1.0 / sqrt(kEigFloor);
    double* dst = pass == 0 ? Fo : Io;
#pragma unroll
    for (int i = 0; i < 64; ++i) dst[(size_t)(r0 + i) * JD + col] = acc[i] + (r0 + i == col ? diag : 0.0);
    __syncthreads();
  }
}

// One CTA per head.  Uq, Uk fp32 [H][128][32].
__global__ void __launch_bounds__(J_THREADS, 1) lowrank_kernel(const double* __restrict__ roots,
                                                               const double* __restrict__ invroots, int H,
                                                               const int* __restrict__ bad, float* __restrict__ Uq,
                                                               float* __restrict__ Uk) {
  extern __shared__ __align__(16) uint8_t jsm[];
  double* W = reinterpret_cast<double*>(jsm);
  double* nrm2 = W + JD * JLD;
  double* coef = nrm2 + JD;                 // reused: the column chosen for each of the 32 ranks
  double2* cs = reinterpret_cast<double2*>(coef + JD);
  const int tid = threadIdx.x, h = blockIdx.x;
  if (bad[h] | bad[H + h]) return;
  const double* Fq = roots + (size_t)h * JD * JD;
  const double* Fk = roots + (size_t)(H + h) * JD * JD;
  const double* Iq = invroots + (size_t)h * JD * JD;

  // C = Fq^T Fk; column j of C goes to W + j * JLD
  {
    const int col = tid & 127, r0 = (tid >> 7) * 64;
    double acc[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) acc[i] = 0.0;
    for (int k = 0; k < JD; ++k) {
      const double b = Fk[(size_t)k * JD + col];
#pragma unroll
      for (int i = 0; i < 64; ++i) acc[i] = fma(Fq[(size_t)k * JD + r0 + i], b, acc[i]);
    }
#pragma unroll
    for (int i = 0; i < 64; ++i) W[col * JLD + r0 + i] = acc[i];
  }
  jacobi_orthogonalise(W, nrm2, cs);
  column_norms2(W, nrm2);      // column j is s_j u_j

  // rank of every column by decreasing singular value (ties: lower column first)
  int* pick = reinterpret_cast<int*>(coef);
  if (tid < JD) {
    const double mine = nrm2[tid];
    int rank = 0;
    for (int j = 0; j < JD; ++j) {
      const double o = nrm2[j];
      rank += (o > mine || (o == mine && j < tid)) ? 1 : 0;
    }
    if (rank < kR) pick[rank] = tid;
  }
  __syncthreads();
  // Uq[:, r] = Fq^-T w / sqrt(s),  Uk[:, r] = Fk^-T v sqrt(s) = Fq w / s^(3/2)     (w = s u, the chosen column;
  // v = C^T u / s and Fk^-T Fk^T = I)
  for (int e = tid; e < JD * kR; e += J_THREADS) {
    const int d = e >> 5, r = e & 31, j = pick[r];
    const double s2 = nrm2[j], s = sqrt(s2);
    double aq = 0.0, ak = 0.0;
    for (int k = 0; k < JD; ++k) {
      const double w = W[j * JLD + k];
      aq = fma(Iq[(size_t)d * JD + k], w, aq);
      ak = fma(Fq[(size_t)d * JD + k], w, ak);
    }
    const bool live = s > 0.0;
    Uq[((size_t)h * JD + d) * kR + r] = live ? (float)(aq / sqrt(s)) : 0.f;
    Uk[((size_t)h * JD + d) * kR + r] = live ? (float)(ak / (s * sqrt(s))) : 0.f;
  }
}

__global__ void __launch_bounds__(256) rotation_selftest_kernel(const double* __restrict__ pairs, double* __restrict__ out,
                                                                int n) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  const Rotation r = rotation(pairs[3 * i], pairs[3 * i + 1], pairs[3 * i + 2]);
  out[3 * i] = r.t;
  out[3 * i + 1] = r.c;
  out[3 * i + 2] = r.s;
}

}  // namespace t2t

using namespace t2t;

extern "C" int t2t_rotation_selftest(const double* pairs, double* out, int n, cudaStream_t st) {
  if (!pairs || !out || n <= 0) return T2T_ERR_ARG;
  rotation_selftest_kernel<<<cdiv(n, 256), 256, 0, st>>>(pairs, out, n);
  return cudaGetLastError() == cudaSuccess ? T2T_OK : T2T_ERR_CUDA;
}

static size_t fit_off_roots(int H, int N) { return (((size_t)2 * H * gram_slabs(N) * kD * kD * 4) + 255) & ~(size_t)255; }
static size_t fit_off_inv(int H, int N) { return fit_off_roots(H, N) + (size_t)2 * H * kD * kD * 8; }

extern "C" size_t t2t_lowrank_fit_ws_bytes(int H, int N) { return fit_off_inv(H, N) + (size_t)H * kD * kD * 8; }

extern "C" int t2t_lowrank_fit(const void* q, const void* k, float* Uq, float* Uk, int H, int N, void* ws,
                               size_t ws_bytes, int* d_bad, int* d_status, cudaStream_t st) {
  return t2t_lowrank_fit_strided(q, k, (long long)kD, (long long)N * kD, Uq, Uk, H, N, ws, ws_bytes, d_bad, d_status,
                                 st);
}

extern "C" int t2t_lowrank_fit_strided(const void* q, const void* k, long long row_stride, long long head_stride,
                                       float* Uq, float* Uk, int H, int N, void* ws, size_t ws_bytes, int* d_bad,
                                       int* d_status, cudaStream_t st) {
  if (!q || !k || !Uq || !Uk || !ws || !d_bad || H <= 0 || N <= 0) return T2T_ERR_ARG;
  if (row_stride < kD || head_stride <= 0) return T2T_ERR_ARG;
  if (ws_bytes < t2t_lowrank_fit_ws_bytes(H, N)) return T2T_ERR_WORKSPACE;
  char* w = static_cast<char*>(ws);
  float* partial = reinterpret_cast<float*>(w);
  double* roots = reinterpret_cast<double*>(w + fit_off_roots(H, N));
  double* invroots = reinterpret_cast<double*>(w + fit_off_inv(H, N));
  const int slabs = gram_slabs(N);
  if (cudaFuncSetAttribute(gram_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GR_SMEM) != cudaSuccess ||
      cudaFuncSetAttribute(factor_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, F_SMEM) != cudaSuccess ||
      cudaFuncSetAttribute(lowrank_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, J_SMEM) != cudaSuccess)
    return T2T_ERR_CUDA;
  CUtensorMap mq, mk;
  if (!make_head_tile_map(&mq, q, (uint64_t)N, (uint64_t)H, GR_ROWS, (uint64_t)row_stride, (uint64_t)head_stride) ||
      !make_head_tile_map(&mk, k, (uint64_t)N, (uint64_t)H, GR_ROWS, (uint64_t)row_stride, (uint64_t)head_stride))
    return T2T_ERR_CUDA;
  gram_kernel<<<dim3(slabs, H, 2), 128, GR_SMEM, st>>>(mq, mk, partial, N, d_status);
  factor_kernel<<<2 * H, J_THREADS, F_SMEM, st>>>(partial, slabs, H, 1.0 / (double)N, roots, invroots, d_bad);
  lowrank_kernel<<<H, J_THREADS, J_SMEM, st>>>(roots, invroots, H, d_bad, Uq, Uk);
  return cudaGetLastError() == cudaSuccess ? T2T_OK : T2T_ERR_CUDA;
}
