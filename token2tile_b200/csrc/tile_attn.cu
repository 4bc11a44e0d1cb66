// Task plan, packed exact tile attention and centroid residual + merge.
//
// Replaces the reference's tile_attn extension
// (token2tile/operator/kernels/tile_attn/src/kernel.cu: selected_kv_lengths,
// plan_kernel, attn_kernel, tail_wgmma_kernel), whose wgmma kernels do not
// exist on sm_100a.  Both hot kernels run their matrix products on the
// tcgen05 tensor cores with fp32 accumulators in tensor memory (TMEM):
//
//   attention:  S = Q K^T   (128 queries x 128 keys, K = 128)   operands in smem
//               O += P V    (P = exp2(S - m) as bf16 in TMEM, V in smem)
//   residual :  S = QU cks^T (128 queries x 128 centroids, K = 32)
//               T += P sumv (128 x 128, K = 128 centroids)
//
// One thread owns one query row (TMEM lane), so row maxima and sums need no
// shuffles.  K/V rows of a union are contiguous runs in the cluster-major
// copies kp/vp, fetched into 128-byte-swizzled tiles by TMA tile loads, TMA
// row gathers (four rows per instruction) and 16-byte cp.async.  Tasks of
// 129..256 query rows run in attn2_kernel on CTA pairs that share every
// product, tasks of up to 128 rows in attn_kernel, one CTA per SM; both are
// warp-specialised and persistent.  Every mbarrier wait is bounded; on a
// timeout the CTA raises a status word and leaves.
#include <cuda.h>

#include <mutex>

#include "common.cuh"
#include "internal.h"
#include "t2t_b200.h"

namespace t2t {

constexpr int QT = 128;          // query rows per tensor-core tile (one thread per row)
constexpr int TASK_ROWS = 256;   // query rows per task: tasks above QT rows run in attn2_kernel, the others in attn_kernel
constexpr int KT = 128;          // keys per tile
constexpr int MAX_RUNS = 1024;   // runs of selected clusters in one union
constexpr int PLAN_SORT_MAX = 2048;
constexpr int PLAN_THREADS = 1024;
constexpr int PLAN_HDR = 8;      // counters: [0] tasks, [1] cursor of attn_kernel, [2] cursor of attn2_kernel

// Layout of the plan (an int32 array owned by a structure snapshot): first row of every key cluster in kp / vp,
// one bit per key cluster saying whether it holds any token, the counters (on a 16-byte boundary, as the tasks behind
// them), the tasks, and the union length of every query cluster.
__host__ __device__ inline size_t plan_nonempty_offset(int H) { return (size_t)H * (kC + 1); }
__host__ __device__ inline size_t plan_counter_offset(int H) { return (plan_nonempty_offset(H) + (size_t)H * (kC / 32) + 3) & ~(size_t)3; }
__host__ __device__ inline size_t plan_task_offset(int H) { return plan_counter_offset(H) + PLAN_HDR; }
__host__ __device__ inline size_t plan_max_tasks(int H, int N, int CQ) { return (size_t)H * (CQ + cdiv(N, TASK_ROWS) + 1); }

struct PlanView {
  int* k_off;           // [H][C + 1]
  uint32_t* nonempty;   // [H][C / 32]
  int* counters;        // [PLAN_HDR]
  int4* tasks;          // (head, query cluster, first sorted row, rows)
  int* kv_lens;         // [H][CQ]
};
__host__ __device__ inline PlanView plan_view(int* plan, int H, int N, int CQ) {
  PlanView v;
  v.k_off = plan;
  v.nonempty = reinterpret_cast<uint32_t*>(plan + plan_nonempty_offset(H));
  v.counters = plan + plan_counter_offset(H);
  v.tasks = reinterpret_cast<int4*>(plan + plan_task_offset(H));
  v.kv_lens = plan + plan_task_offset(H) + 4 * plan_max_tasks(H, N, CQ);
  return v;
}

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// ---------------------------------------------------------------------------
// plan: key-cluster offsets, union lengths, tasks (most work first inside a head)
// ---------------------------------------------------------------------------
// Exclusive prefix of v over the PLAN_THREADS threads of the CTA (every thread calls it); scratch holds 32 ints.
__device__ __forceinline__ int block_prefix(int v, int* scratch, int& total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int inc = warp_incl_scan(v, lane);
  __syncthreads();
  if (lane == 31) scratch[w] = inc;
  __syncthreads();
  const int part = scratch[lane], parts = warp_incl_scan(part, lane);
  total = __shfl_sync(0xffffffffu, parts, 31);
  return __shfl_sync(0xffffffffu, parts - part, w) + inc - v;
}
static_assert(PLAN_THREADS == 32 * 32 && kC == 2 * PLAN_THREADS, "a warp scans the warps' sums; two key clusters a thread");

// One CTA per head.  A query cluster of n rows gives ceil(n / TASK_ROWS) tasks: full ones first, the remainder
// last (a remainder of at most QT rows costs one row tile instead of two).
// Bound by the latency of its steps (H CTAs in all): with 256 threads, which also went through the heads before theirs
// one after the other, 114 us at 40 heads of 720p and 20 at 2 x 4096.
__global__ void __launch_bounds__(PLAN_THREADS) plan_kernel(const int* __restrict__ qcount, const int* __restrict__ kcount,
                                                            const uint32_t* __restrict__ ubits, int H, int N, int CQ,
                                                            int* __restrict__ plan) {
  __shared__ int s_off[kC + 1];
  __shared__ unsigned long long s_key[PLAN_SORT_MAX];
  __shared__ int s_scan[32];
  const PlanView pv = plan_view(plan, H, N, CQ);
  const int h = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  // first kp / vp row of every key cluster (two consecutive clusters per thread) and the non-empty bits
  {
    const int2 c2 = make_int2(kcount[(size_t)h * kC + tid * 2], kcount[(size_t)h * kC + tid * 2 + 1]);
    int total;
    const int run = block_prefix(c2.x + c2.y, s_scan, total);
    s_off[tid * 2] = run;
    s_off[tid * 2 + 1] = run + c2.x;
    if (tid == PLAN_THREADS - 1) s_off[kC] = total;
    // sixteen neighbouring threads hold the bits of one 32-cluster word
    uint32_t word = ((c2.x > 0 ? 1u : 0u) | (c2.y > 0 ? 2u : 0u)) << (2 * (tid & 15));
#pragma unroll
    for (int d = 8; d > 0; d >>= 1) word |= __shfl_xor_sync(0xffffffffu, word, d);
    if ((tid & 15) == 0) pv.nonempty[(size_t)h * (kC / 32) + (tid >> 4)] = word;
  }
  __syncthreads();
  for (int i = tid; i <= kC; i += PLAN_THREADS) pv.k_off[(size_t)h * (kC + 1) + i] = s_off[i];

  // tokens in the union of every query cluster (a warp per cluster)
  for (int c = warp; c < CQ; c += PLAN_THREADS / 32) {
    const int n = qcount[(size_t)h * CQ + c];
    int len = 0;
    if (n > 0) {
      const uint32_t* words = ubits + ((size_t)h * CQ + c) * (kC / 32);
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int w = lane + 32 * half;
        for (uint32_t bits = words[w]; bits; bits &= bits - 1) {
          const int cl = w * 32 + __ffs(bits) - 1;
          len += s_off[cl + 1] - s_off[cl];
        }
      }
    }
    len = __reduce_add_sync(0xffffffffu, len);
    if (lane == 0) pv.kv_lens[(size_t)h * CQ + c] = len;
  }

  // the task array is head-major (the K / V rows of a head stay in L2 while its unions are read):
  // count the tasks of the heads before this one
  int first, mine;
  {
    int before = 0, own = 0;
    for (int i = tid; i < h * CQ; i += PLAN_THREADS) before += cdiv(qcount[i], TASK_ROWS);
    for (int i = tid; i < CQ; i += PLAN_THREADS) own += cdiv(qcount[(size_t)h * CQ + i], TASK_ROWS);
    block_prefix(before, s_scan, first);
    block_prefix(own, s_scan, mine);
  }
  if (h == H - 1 && tid == 0) pv.counters[0] = first + mine;

  int rows_before = 0, tasks_before = 0;
  for (int c0 = 0; c0 < CQ; c0 += PLAN_THREADS) {
    const int c = c0 + tid;
    const int n = c < CQ ? qcount[(size_t)h * CQ + c] : 0;
    const int nt = cdiv(n, TASK_ROWS);
    int tot_rows, tot_tasks;
    const int row0 = rows_before + block_prefix(n, s_scan, tot_rows);
    const int task0 = tasks_before + block_prefix(nt, s_scan, tot_tasks);
    for (int i = 0; i < nt; ++i)
      pv.tasks[first + task0 + i] = make_int4(h, c, row0 + i * TASK_ROWS, min(TASK_ROWS, n - i * TASK_ROWS));
    rows_before += tot_rows;
    tasks_before += tot_tasks;
  }
  __syncthreads();
  if (mine < 2 || mine > PLAN_SORT_MAX) return;

  // most work first (rows x union length); equal work keeps its order
  int pow2 = 2;
  while (pow2 < mine) pow2 <<= 1;
  for (int i = tid; i < pow2; i += PLAN_THREADS) {
    unsigned long long key = 0ull;
    if (i < mine) {
      const int4 t = pv.tasks[first + i];
      const unsigned long long work = min((unsigned long long)t.w * (unsigned long long)pv.kv_lens[(size_t)h * CQ + t.y], 0xFFFFFFFFull);
      key = (work << 32) | (unsigned long long)(0xFFFFFFFFu - (unsigned)i);
    }
    s_key[i] = key;
  }
  __syncthreads();
  for (int span = 2; span <= pow2; span <<= 1) {
    for (int step = span >> 1; step > 0; step >>= 1) {
      for (int i = tid; i < pow2; i += PLAN_THREADS) {
        const int j = i ^ step;
        if (j > i) {
          const unsigned long long x = s_key[i], y = s_key[j];
          const bool descending = (i & span) == 0;
          if (descending ? x < y : x > y) { s_key[i] = y; s_key[j] = x; }
        }
      }
      __syncthreads();
    }
  }
  int4 keep[PLAN_SORT_MAX / PLAN_THREADS];
  int k = 0;
  for (int i = tid; i < mine; i += PLAN_THREADS) keep[k++] = pv.tasks[first + (int)(0xFFFFFFFFu - (unsigned)(s_key[i] & 0xFFFFFFFFull))];
  __syncthreads();
  k = 0;
  for (int i = tid; i < mine; i += PLAN_THREADS) pv.tasks[first + i] = keep[k++];
}

// info: tasks, executed (query, key) pairs (low and high word), 0
__global__ void __launch_bounds__(1024) plan_info_kernel(PlanView pv, int CQ, int* __restrict__ info) {
  __shared__ unsigned long long s_pairs;
  if (threadIdx.x == 0) s_pairs = 0ull;
  __syncthreads();
  const int tasks = pv.counters[0];
  unsigned long long pairs = 0ull;
  for (int i = threadIdx.x; i < tasks; i += 1024) {
    const int4 t = pv.tasks[i];
    pairs += (unsigned long long)t.w * (unsigned long long)pv.kv_lens[(size_t)t.x * CQ + t.y];
  }
  atomicAdd(&s_pairs, pairs);
  __syncthreads();
  if (threadIdx.x == 0) {
    info[0] = tasks;
    info[1] = (int)(uint32_t)s_pairs;
    info[2] = (int)(uint32_t)(s_pairs >> 32);
    info[3] = 0;
  }
}

// ---------------------------------------------------------------------------
// shared pieces of the two tensor-core kernels
// ---------------------------------------------------------------------------
struct RowState {
  float m;      // reference maximum (log2 domain) the stored P and O are relative to
  float l;      // running denominator
};

constexpr float kLazy = 8.0f;   // rescale O only when the row maximum grows by more than 2^8

// Rescale the fp32 accumulator rows in TMEM by `alpha` (per thread = per row), few columns at a time: the attention's
// softmax threads hold a row of scores meanwhile.
__device__ __forceinline__ void rescale_rows(uint32_t tO_lane, float alpha) {
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    uint32_t v[16];
    tmem_ld16(tO_lane + c * 16, v);
    tmem_wait_ld();
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * alpha);
    tmem_st16(tO_lane + c * 16, v);
  }
}

// The union of one task as runs of consecutive kp / vp rows: maximal stretches of selected, non-empty key
// clusters that follow each other.  sRunStart[r] = first row of run r, sRunCum[r] = position of its first
// token in the union, sRunCum[runs] = union length, *runs_out = runs.  One warp does the work with the bitmap
// as 64-bit words (two bitmap words per lane): a run starts at a set bit whose lower neighbour is clear and
// ends at a set bit whose upper neighbour is clear, so the r-th start and the r-th end delimit run r.  A run
// list that would not fit raises the abort flag.
__device__ __forceinline__ void build_runs_warp(const int* __restrict__ koh, const uint32_t* __restrict__ ubr,
                                                const uint32_t* __restrict__ nonempty, int* sRunStart, int* sRunCum,
                                                int* runs_out, volatile int* abort_flag, int* status) {
  const int lane = threadIdx.x & 31;
  const unsigned long long sel = ((unsigned long long)(ubr[2 * lane + 1] & nonempty[2 * lane + 1]) << 32) |
                                 (unsigned long long)(ubr[2 * lane] & nonempty[2 * lane]);
  // neighbours across the lane boundary
  const unsigned long long below = __shfl_up_sync(0xffffffffu, sel, 1), above = __shfl_down_sync(0xffffffffu, sel, 1);
  const unsigned long long carry_in = lane > 0 ? below >> 63 : 0ull;
  const unsigned long long carry_out = lane < 31 ? (above & 1ull) << 63 : 0ull;
  unsigned long long starts = sel & ~((sel << 1) | carry_in);
  unsigned long long ends = sel & ~((sel >> 1) | carry_out);
  const int mine = __popcll(starts);
  const int before_s = warp_incl_scan(mine, lane) - mine;
  const int before_e = warp_incl_scan(__popcll(ends), lane) - __popcll(ends);
  const int runs = __shfl_sync(0xffffffffu, before_s + mine, 31);
  if (runs > MAX_RUNS) {      // cannot happen for C = 2048; guard the static arrays anyway
    if (lane == 0) { *abort_flag = 1; if (status) atomicExch(status, ST_BAD_PLAN); }
    return;
  }
  int r = before_s;
  for (; starts; starts &= starts - 1) sRunStart[r++] = koh[64 * lane + __ffsll((long long)starts) - 1];
  r = before_e;
  for (; ends; ends &= ends - 1) sRunCum[r++] = koh[64 * lane + __ffsll((long long)ends)];      // one past the run's last row
  __syncwarp();
  // lengths -> positions: every lane turns a block of consecutive runs into a running sum
  const int per = (runs + 31) >> 5, lo = min(lane * per, runs), hi = min(lo + per, runs);
  int sum = 0;
  for (int i = lo; i < hi; ++i) sum += sRunCum[i] - sRunStart[i];
  int pos = warp_incl_scan(sum, lane) - sum;
  const int total = __shfl_sync(0xffffffffu, pos + sum, 31);
  for (int i = lo; i < hi; ++i) {
    const int len = sRunCum[i] - sRunStart[i];
    sRunCum[i] = pos;
    pos += len;
  }
  if (lane == 0) { sRunCum[runs] = total; *runs_out = runs; }
}
constexpr int AT_TILE = KT * kD * 2;   // 32 KB: one 128-row tile of q, kp or vp

// kp / vp rows (all heads: `row0` is the head's first row) of union positions p0 .. p0 + 3, from the run list of
// build_runs.  `cursor` is the caller's run index from its previous, smaller p0 (0 at the start of a task): the
// run of p0 is found by stepping forward from it.  Positions past the union read the head's first row (their
// scores are masked).  Returns whether the four rows exist and are consecutive rows of kp / vp.
__device__ __forceinline__ bool union_rows(const int* sRunStart, const int* sRunCum, int nruns, int kvlen, int p0,
                                           int row0, int& cursor, int (&r)[4]) {
  int ru = cursor;
  while (ru + 1 < nruns && sRunCum[ru + 1] <= p0) ++ru;
  cursor = ru;
  int next = sRunCum[ru + 1];
  int row = sRunStart[ru] + p0 - sRunCum[ru];
  r[0] = p0 < kvlen ? row0 + row : row0;
#pragma unroll
  for (int j = 1; j < 4; ++j) {
    const int p = p0 + j;
    if (p >= next && ru + 1 < nruns) {
      ++ru;
      row = sRunStart[ru];
      next = sRunCum[ru + 1];
    } else {
      ++row;
    }
    r[j] = p < kvlen ? row0 + row : row0;
  }
  return p0 + 3 < kvlen && r[3] == r[0] + 3;
}

// Tensor maps over kp and vp as [H * N, 128] matrices with boxes of 1, 32 and 64 rows by 64 columns.
struct KVMaps {
  CUtensorMap k1, k32, k64, v1, v32, v64;
};

// How a warp fetches a 128-row K or V tile.  Lane g owns destination rows 4 g .. 4 g + 3, whose source rows are
// r[0..3]; `whole` says that they are four consecutive rows of kp / vp.  Groups that follow each other in the
// source as well form a stretch, and a stretch is fetched with 64-row tile loads, then 32-row tile loads, then
// four-row gathers for what is left (a tile load moves 2.6x / 1.8x the bytes per cycle of a gather; a swizzled
// tile may start at any multiple of four rows, the pattern being a function of the shared-memory address).
// Groups that straddle two runs of the union are gathered.  Returns what this lane issues for each 64-column
// block: FETCH_NONE (a tile load of a lower lane covers its rows), a gather, or a tile load starting at r[0].
enum { FETCH_NONE = 0, FETCH_GATHER = 1, FETCH_BOX32 = 2, FETCH_BOX64 = 3 };
__device__ __forceinline__ int fetch_plan(const int (&r)[4], bool whole, int lane, int seg) {
  const int prev = __shfl_up_sync(0xffffffffu, r[0], 1);
  const unsigned wmask = __ballot_sync(0xffffffffu, whole);
  const bool linked = whole && (lane & (seg - 1)) > 0 && ((wmask >> (lane - 1)) & 1u) && r[0] == prev + 4;
  const unsigned lmask = __ballot_sync(0xffffffffu, linked);      // bit g: group g continues the stretch of g - 1
  if (!whole) return FETCH_GATHER;
  const unsigned upto = 0xffffffffu >> (31 - lane);
  const int start = 31 - __clz((wmask & ~lmask) & upto);
  const unsigned above = ~lmask & ~upto;
  const int end = above ? __ffs(above) - 1 : 32;
  const int len = end - start, k = lane - start;
  const int k64 = len & ~15, k32 = k64 + ((len - k64) & ~7);
  if (k < k64) return (k & 15) == 0 ? FETCH_BOX64 : FETCH_NONE;
  if (k < k32) return ((k - k64) & 7) == 0 ? FETCH_BOX32 : FETCH_NONE;
  return FETCH_GATHER;
}
// ---------------------------------------------------------------------------
// softmax of a row of scores, shared by the two attention kernels
// ---------------------------------------------------------------------------
// Packed fp32 pairs (one instruction for two values) and the three-input maximum keep the instruction count of
// the softmax rows down: the MMA lane and the copy warps share their schedulers.
__device__ __forceinline__ unsigned long long pack_f2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack_f2(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long fma_f2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ unsigned long long add_f2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
// 2^y for two values y <= 8 without the special-function unit: round y to the nearest integer n (the
// magic-number add leaves n in the low mantissa bits), a cubic for 2^(y - n) on [-0.5, 0.5] (relative error
// 7.5e-5, well inside a bf16 rounding step), and n added to the exponent field.  Inputs below -125 count as
// -125 (2^-125 ~ 0).
__device__ __forceinline__ void exp2_fma2(float y0, float y1, float& p0, float& p1) {
  const unsigned long long y = pack_f2(fmaxf(y0, -125.0f), fmaxf(y1, -125.0f));
  const unsigned long long t = add_f2(y, pack_f2(12582912.0f, 12582912.0f));      // 1.5 * 2^23
  const unsigned long long n = add_f2(t, pack_f2(-12582912.0f, -12582912.0f));
  const unsigned long long f = fma_f2(n, pack_f2(-1.0f, -1.0f), y);
  unsigned long long p = fma_f2(pack_f2(0.055171408f, 0.055171408f), f, pack_f2(0.24261075f, 0.24261075f));
  p = fma_f2(p, f, pack_f2(0.69326097f, 0.69326097f));
  p = fma_f2(p, f, pack_f2(0.99992812f, 0.99992812f));
  float q0, q1, t0, t1;
  unpack_f2(p, q0, q1);
  unpack_f2(t, t0, t1);
  p0 = __int_as_float(__float_as_int(q0) + (__float_as_int(t0) << 23));
  p1 = __int_as_float(__float_as_int(q1) + (__float_as_int(t1) << 23));
}

// Softmax of one 128-column S row held in tensor memory: the row comes to registers once, its maximum is found there,
// then P = 2^(s * scale - m) goes back packed to bf16 (chunk c of S, columns 32 c .., becomes columns 16 c .. of P).
// All exponentials use the special-function unit (16 per cycle and SM, 1,024 cycles a tile).
// MASK: columns >= valid lie past the union and count as -inf, a weight of zero.
// The maximum comes before any weight of the tile: weights stay below 2^kLazy, so O and l keep the range of the values
// whatever the scores, and a key that dominates its row from beyond that weighs exactly one.  (One pass with the first
// tile's maximum as reference and corrections by the sums rounds the largest weight like any other, 2.326e-3 instead
// of 2.323e-3 against a float64 softmax, and sums reach 2^60.)
// The row to registers; returns its maximum (unscaled).
template <bool MASK>
__device__ __forceinline__ float row_scores(uint32_t tS_lane, int valid, uint32_t (&v)[4][32]) {
  float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
  tmem_ld32(tS_lane, v[0]);
  tmem_ld32(tS_lane + 32, v[1]);
  tmem_wait_ld();
  tmem_ld32(tS_lane + 64, v[2]);
  tmem_ld32(tS_lane + 96, v[3]);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    if (c == 2) tmem_wait_ld();
    if (MASK) {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (c * 32 + j >= valid) v[c][j] = 0xff800000u;      // -inf
    }
#pragma unroll
    for (int j = 0; j < 32; j += 8) {
      mx4[0] = max3(mx4[0], __uint_as_float(v[c][j]), __uint_as_float(v[c][j + 1]));
      mx4[1] = max3(mx4[1], __uint_as_float(v[c][j + 2]), __uint_as_float(v[c][j + 3]));
      mx4[2] = max3(mx4[2], __uint_as_float(v[c][j + 4]), __uint_as_float(v[c][j + 5]));
      mx4[3] = max3(mx4[3], __uint_as_float(v[c][j + 6]), __uint_as_float(v[c][j + 7]));
    }
  }
  return fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
}
// The row's weights relative to rs.m, written over S and added to rs.l.
__device__ __forceinline__ void row_weights(uint32_t tS_lane, const uint32_t (&v)[4][32], RowState& rs, float sc) {
  const unsigned long long sc2 = pack_f2(sc, sc), nm2 = pack_f2(-rs.m, -rs.m);
  unsigned long long ls2[2] = {0ull, 0ull};
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t pk[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      float y0, y1;
      unpack_f2(fma_f2(pack_f2(__uint_as_float(v[c][2 * j]), __uint_as_float(v[c][2 * j + 1])), sc2, nm2), y0, y1);
      const float p0 = ex2_approx(y0), p1 = ex2_approx(y1);
      ls2[j & 1] = add_f2(ls2[j & 1], pack_f2(p0, p1));
      pk[j] = pack_bf2(p0, p1);
    }
    tmem_st16(tS_lane + c * 16, pk);
  }
  float s0, s1, s2, s3;
  unpack_f2(ls2[0], s0, s1);
  unpack_f2(ls2[1], s2, s3);
  rs.l += (s0 + s1) + (s2 + s3);
}
// Registers move between the roles of a kernel: a softmax thread holds a whole row of S, the others need few.  Both
// kernels are launched with 128 registers a thread and every second warpgroup gives up what the softmax warpgroups take:
// 256 x (200 + 56) = 512 x 128.
constexpr int kLaunchRegs = 128, kSoftmaxRegs = 200, kRoleRegs = 56;
static_assert(kSoftmaxRegs + kRoleRegs == 2 * kLaunchRegs, "the split may not exceed what the launch holds");
// Whether a kernel that was built with `regs` registers a thread is launched with kLaunchRegs (registers come in eights).
// With fewer, which other compiler flags can bring about, take_registers would wait for what its CTA does not have.
inline bool split_fits(int regs) { return ((regs + 7) & ~7) == kLaunchRegs; }
__device__ __forceinline__ void take_registers() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(kSoftmaxRegs)); }
__device__ __forceinline__ void give_registers() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(kRoleRegs)); }

// One task as it travels through a CTA's two-slot ring.
struct TaskSlot {
  int end;      // nonzero: no task is left
  int head, first, rows, kvlen, runs;      // first: sorted row the task starts at
  int pad[2];
};

// Task `task` (none is left at numTasks) into `slot`, by one warp: record and union length, then the run list of its union.
__device__ __forceinline__ void prepare_task(const PlanView& pv, const uint32_t* __restrict__ ub, int CQ, int numTasks,
                                             int task, TaskSlot* slot, int* sRunStart, int* sRunCum,
                                             volatile int* abort_flag, int* status) {
  const int lane = threadIdx.x & 31;
  int4 tk = make_int4(0, 0, 0, 0);
  int len = 0;
  if (task < numTasks) {
    tk = pv.tasks[task];
    len = pv.kv_lens[(size_t)tk.x * CQ + tk.y];
  }
  if (len > 0)
    build_runs_warp(pv.k_off + (size_t)tk.x * (kC + 1), ub + ((size_t)tk.x * CQ + tk.y) * (kC / 32),
                    pv.nonempty + (size_t)tk.x * (kC / 32), sRunStart, sRunCum, &slot->runs, abort_flag, status);
  if (lane == 0) {
    slot->end = task >= numTasks || *abort_flag;
    slot->head = tk.x;
    slot->first = tk.z;
    slot->rows = tk.w;
    slot->kvlen = len;
  }
  __syncwarp();
}

// ---------------------------------------------------------------------------
// exact attention, tasks of QT + 1 .. TASK_ROWS rows
// ---------------------------------------------------------------------------
// The kernel runs on CTA pairs (clusters of two, one CTA per SM): group 0 of a task's rows on the even CTA, the leader,
// group 1 on the odd one, 128 rows each.  A product covers both groups (256 rows), and each CTA keeps only half of a K
// tile (64 keys) and half of a V tile (64 of the 128 columns), so that per SM a tile moves 96 KB through shared memory
// instead of 128 KB and tensor memory holds one group's O and three score buffers.  Roles of a CTA:
//   warps 0..3 / 4..7  softmax of the even / odd tiles, one thread per row of the group; the row's reference maximum
//                      travels from tile to tile through shared memory, each thread sums the weights of its own tiles
//   warp 8             leader: issues Q K^T (see elect_one)
//   warp 9             leader: issues P V, so that neither product waits in line behind the other's barriers (one warp for
//                      both left the tensor pipe idle for 500 of 1,750 cycles a tile); other CTA: takes the next task and
//                      builds the run list of its union, for both CTAs
//   warps 10..12       K tiles in turn (and Q tiles) by TMA, warps 13..15 V tiles: finding a tile's rows and issuing up to 32
//                      instructions, about 70 cycles each, takes a warp three times as long as the products
// S = Q K^T of tile g goes to score buffer g mod 3, two tiles ahead of P V, so that no softmax warp waits for the
// product behind its own weights: with two score buffers (one CTA, two groups that share a K / V stream) the chain
// softmax -> P V -> Q K^T took 3,770 cycles for two 128-row tiles.
// Barriers: QK and PV are the commits behind the products of a tile, on barrier tile mod 4, and reach both CTAs.  QK(g): S(g)
// is there, the K slot of tile g is free.  PV(g): O holds tile g, score buffer and V slot of tile g are free.  P[b],
// FULLK / FULLV / FULLQ and OFREE live in the leader and collect both CTAs' arrivals (and, for copies, both CTAs'
// bytes); TFREE lives in the other CTA, which overwrites both CTAs' copies of a task behind it, and collects everyone who reads
// one: releases at cluster scope, once per warp and task and where their fence is not waited for (a softmax warp's before its
// stores, those of QK and PV behind their products).  MEET[w]: the two softmax warps of rows 32 w .. have laid down their
// sums of a task.
constexpr int A2_THREADS = 16 * 32;
constexpr int A2_STAGES = 4;                              // K and V ring depth
constexpr int A2_HALF = AT_TILE / 2;                      // 16 KB: 64 keys of a K tile, 64 columns of a V tile
constexpr int A2_OFF_K = 2 * AT_TILE;                     // after two Q tiles (this task's, the next one's)
constexpr int A2_OFF_V = A2_OFF_K + A2_STAGES * A2_HALF;
constexpr int A2_OFF_MISC = A2_OFF_V + A2_STAGES * A2_HALF;
constexpr int RUN_INTS = 2 * MAX_RUNS + 8;                // one run list: [MAX_RUNS] starts, [MAX_RUNS + 1] positions
enum { B_QK = 0, B_PV = 4, B_P = 8, B_FULLK = 11, B_FULLV = B_FULLK + A2_STAGES, B_FULLQ = B_FULLV + A2_STAGES,
       B_FREEQ = B_FULLQ + 2, B_OFREE = B_FREEQ + 2, B_TFULL, B_TFREE = B_TFULL + 2, B_MEET = B_TFREE + 2,
       B_COUNT = B_MEET + 4 };
static_assert(A2_STAGES == 4, "ring slots and commits are counted alike");
constexpr int A2_CONSUMERS = (8 + 6) * 2 + 2;             // warps that read a task: softmax and copy, QK and PV
constexpr int A2_OFF_RING = A2_OFF_MISC + 512;            // two tasks
constexpr int A2_OFF_M = A2_OFF_RING + 2 * (int)sizeof(TaskSlot);      // [2][128] reference maxima of the even / odd tiles, with their tiles
constexpr int A2_OFF_FIN = A2_OFF_M + 2 * QT * 8;         // [2][2][128] (maximum, sum) of the two softmax warpgroups
constexpr int A2_OFF_RUNS = A2_OFF_FIN + 4 * QT * 8;
constexpr int A2_SMEM = A2_OFF_RUNS + 2 * RUN_INTS * 4 + 1024;
static_assert(B_COUNT * 8 + 16 <= 512, "the barriers fit their area");
static_assert(A2_SMEM <= 227 * 1024, "one CTA per SM");

// A row's reference maximum behind tile `tile`, from the thread that weighs that tile to the thread that weighs the next:
// value and tile number in one 64-bit word, so that neither needs a barrier (an mbarrier in between cost 440 cycles a tile).
__device__ __forceinline__ void put_tagged(unsigned long long* at, uint32_t tile, float m) {
  asm volatile("st.volatile.shared.b64 [%0], %1;\n" ::"r"(smem_u32(at)),
               "l"(((unsigned long long)tile << 32) | __float_as_uint(m)) : "memory");
}
__device__ __forceinline__ unsigned long long peek_tagged(const unsigned long long* at) {
  unsigned long long w;
  asm volatile("ld.volatile.shared.b64 %0, [%1];\n" : "=l"(w) : "r"(smem_u32(at)) : "memory");
  return w;
}
// Looks until `w` is tile `tile`'s in every lane: one answer for the warp, as in mbar_wait_warp.
__device__ __forceinline__ bool take_tagged(const unsigned long long* at, uint32_t tile, unsigned long long& w,
                                            volatile int* abort_flag, uint32_t limit) {
  for (uint32_t it = 0; it < limit; ++it) {
    if (__all_sync(0xffffffffu, (uint32_t)(w >> 32) == tile)) return true;
    if ((it & 255u) == 255u && __any_sync(0xffffffffu, *abort_flag != 0)) return false;
    w = peek_tagged(at);
  }
  *abort_flag = 1;
  return false;
}

// Rows of group 0 of a task of more than QT rows, whole warps of them; group 1 takes the rest.
__device__ __forceinline__ int group_rows(int rows) { return min((((rows + 1) >> 1) + 31) & ~31, rows); }

// The softmax warps of both kernels: warps 0..3 weigh a row's even tiles, warps 4..7 its odd ones (see attn2_kernel).
// `rank`, `lead` and `tfree` are the group of this CTA's rows and the cluster addresses of the pair's barriers; `LIMIT` bounds
// the waits.
template <bool PAIR, uint32_t LIMIT = kWaitSpinLimit>
__device__ __forceinline__ void softmax_role(uint64_t* bars, const TaskSlot* ring, unsigned long long* sM, float2* sFin,
                                             uint32_t tmem, uint32_t rank, uint32_t lead, uint32_t tfree,
                                             __nv_bfloat16* __restrict__ attn_out, float* __restrict__ attn_lse, int N,
                                             volatile int* abort_flag) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wg = warp >> 2, gw = warp & 3, row = gw * 32 + lane;
  const uint32_t tO_lane = tmem_addr(tmem + 3 * 128, gw * 32, 0);
  const float sc = 0.08838834764831845f * 1.4426950408889634f;   // 1/sqrt(128) * log2(e)
  // arrival on this CTA's barrier `own`, or on that of the pair at the cluster address `at`
  auto arrive = [&](int own, uint32_t at) {
    if (PAIR) mbar_arrive_peer(at); else mbar_arrive(bars + own);
  };
  // the task's slot and run list may be overwritten
  auto release_task = [&](uint32_t sl) {
    if (PAIR) mbar_release_peer(tfree + sl * 8); else mbar_arrive(bars + B_TFREE + sl);
  };
  uint32_t g = 0;      // tiles so far
  uint32_t q = 0;
  bool ok = true;
  for (uint32_t n = 0;; ++n) {
    const uint32_t sl = n & 1u;
    if (!(PAIR ? mbar_wait_warp_cluster(bars + B_TFULL + sl, (n >> 1) & 1u, abort_flag)
               : mbar_wait_warp(bars + B_TFULL + sl, (n >> 1) & 1u, abort_flag, LIMIT)))
      break;
    const int end = ring[sl].end, kvlen = ring[sl].kvlen, ntiles = cdiv(kvlen, KT);
    if (end) break;
    const int rows0 = PAIR ? group_rows(ring[sl].rows) : ring[sl].rows, myrows = rank ? ring[sl].rows - rows0 : rows0;
    const size_t at = (size_t)ring[sl].head * N + ring[sl].first + (row < myrows ? (rank ? rows0 : 0) + row : 0);
    const bool wr = row < myrows;
    if (ntiles == 0) {   // empty union: O = 0, lse = -inf
      if (wr) {
        uint4* dst = reinterpret_cast<uint4*>(attn_out + at * kD) + wg * 8;
#pragma unroll
        for (int i = 0; i < 8; ++i) dst[i] = make_uint4(0u, 0u, 0u, 0u);
        if (wg == 0) attn_lse[at] = -INFINITY;
      }
      __syncwarp();
      if (lane == 0) release_task(sl);
      continue;
    }
    // A warp whose rows all lie past the group's last row skips the arithmetic: its P rows stay
    // whatever S held, which only reaches O rows that are never stored.
    const bool active = gw * 32 < myrows;
    RowState rs;
    rs.m = -INFINITY;
    rs.l = 0.f;
    // this warpgroup's tiles: every other one
    const int t0 = (int)((wg ^ g) & 1u);
    uint32_t buf = (g + t0) % 3u;
    for (int t = t0; t < ntiles; t += 2) {
      const uint32_t gt = g + t, p = gt - 1u;
      const uint32_t tS_lane = tmem_addr(tmem + buf * 128, gw * 32, 0);
      ok = mbar_wait_warp(bars + B_QK + (gt & 3u), (gt >> 2) & 1u, abort_flag, LIMIT);
      if (!ok) break;
      tc_fence_after();
      if (active) {
        const int valid = kvlen - t * KT;
        uint32_t v[4][32];
        // the reference behind tile t - 1, from the thread that weighs it: looked at once before the row is here
        const unsigned long long* before = sM + (p & 1u) * QT + row;
        unsigned long long tagged = peek_tagged(before);
        const float mx = (valid >= KT ? row_scores<false>(tS_lane, KT, v) : row_scores<true>(tS_lane, valid, v)) * sc;
        if (t == 0) {
          rs.m = mx;
        } else {
          // one vote in the common case: the reference is there in every lane and stays
          const float seen = __uint_as_float((uint32_t)tagged);
          if (__any_sync(0xffffffffu, (uint32_t)(tagged >> 32) != p || seen != rs.m || mx > seen + kLazy)) {
            ok = take_tagged(before, p, tagged, abort_flag, LIMIT);
            if (!ok) break;
            const float m_in = __uint_as_float((uint32_t)tagged);
            if (m_in != rs.m) rs.l *= t > 1 ? ex2_approx(rs.m - m_in) : 0.f;
            rs.m = m_in;
            const bool grow = mx > rs.m + kLazy;
            if (__any_sync(0xffffffffu, grow)) {
              const float mnew = grow ? mx : rs.m;
              ok = mbar_wait_warp(bars + B_PV + (p & 3u), (p >> 2) & 1u, abort_flag, LIMIT);      // O holds the tiles up to t - 1
              if (!ok) break;
              const float alpha = ex2_approx(rs.m - mnew);
              tc_fence_after();
              rescale_rows(tO_lane, alpha);
              rs.l *= alpha;
              rs.m = mnew;
            }
          }
        }
        put_tagged(sM + (gt & 1u) * QT + row, gt, rs.m);
        row_weights(tS_lane, v, rs, sc);
        tmem_wait_st();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) arrive(B_P + buf, lead + (B_P + buf) * 8);
      buf = buf ? buf - 1 : 2;      // two on, of three
    }
    if (!ok) break;
    g += ntiles;
    // both warps of these rows meet, by a wait with a limit as everywhere (the other one may have left at a wait that gave
    // up): the sums of the two are relative to the maxima they saw last
    float2* fin = sFin + (q & 1u) * 2 * QT;
    fin[wg * QT + row] = make_float2(rs.m, rs.l);
    __syncwarp();
    if (lane == 0) mbar_arrive(bars + B_MEET + gw);
    ok = mbar_wait_warp(bars + B_MEET + gw, q & 1u, abort_flag, LIMIT);
    if (!ok) break;
    if (lane == 0) release_task(sl);      // the task is in registers; before the stores below, which a release would wait for
    const int lastwg = (g - 1u) & 1u;
    ok = mbar_wait_warp(bars + B_PV + ((g - 1u) & 3u), ((g - 1u) >> 2) & 1u, abort_flag, LIMIT);
    if (!ok) break;
    if (active) {
      tc_fence_after();
      const float2 a = fin[lastwg * QT + row], b = fin[(lastwg ^ 1) * QT + row];
      const float l = ntiles > 1 ? a.y + (b.x != a.x ? b.y * ex2_approx(b.x - a.x) : b.y) : a.y;
      const float inv = 1.0f / l;
      uint4* dst = reinterpret_cast<uint4*>(attn_out + at * kD) + wg * 8;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t v[32];
        tmem_ld32(tO_lane + wg * 64 + c * 32, v);
        tmem_wait_ld();
        if (wr) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            uint4 o;
            o.x = pack_bf2(__uint_as_float(v[8 * k + 0]) * inv, __uint_as_float(v[8 * k + 1]) * inv);
            o.y = pack_bf2(__uint_as_float(v[8 * k + 2]) * inv, __uint_as_float(v[8 * k + 3]) * inv);
            o.z = pack_bf2(__uint_as_float(v[8 * k + 4]) * inv, __uint_as_float(v[8 * k + 5]) * inv);
            o.w = pack_bf2(__uint_as_float(v[8 * k + 6]) * inv, __uint_as_float(v[8 * k + 7]) * inv);
            dst[c * 4 + k] = o;
          }
        }
      }
      if (wr && wg == 0) attn_lse[at] = (a.x + log2f(l)) * 0.6931471805599453f;
    }
    ++q;
    tc_fence_before();
    __syncwarp();
    if (lane == 0) arrive(B_OFREE, lead + B_OFREE * 8);
  }
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(A2_THREADS, 1) attn2_kernel(
    const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ KVMaps maps,
    const uint32_t* __restrict__ ub, const int* __restrict__ qperm,
    __nv_bfloat16* __restrict__ attn_out, float* __restrict__ attn_lse, int* __restrict__ plan, int H, int N, int CQ,
    int q_row_step, int q_head_step, int* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (base - smem_u32(smem_raw));
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + A2_OFF_MISC);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + A2_OFF_MISC + B_COUNT * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + A2_OFF_MISC + B_COUNT * 8 + 8);
  TaskSlot* ring = reinterpret_cast<TaskSlot*>(sm + A2_OFF_RING);
  unsigned long long* sM = reinterpret_cast<unsigned long long*>(sm + A2_OFF_M);
  float2* sFin = reinterpret_cast<float2*>(sm + A2_OFF_FIN);
  int* sRuns = reinterpret_cast<int*>(sm + A2_OFF_RUNS);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_rank();      // group of this CTA's rows; 0 leads

  // the kernel launched behind this one (tasks of at most QT rows) does not depend on it: let it be scheduled
  // as soon as SMs free up
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  if (warp == 0) {
    tmem_alloc_pair(tmem_slot, 512);
    tmem_relinquish_pair();
  }
  if (tid < 2 * QT) sM[tid] = ~0ull;      // no tile
  if (tid == 0) {
    *abort_flag = 0;
    for (int i = 0; i < B_COUNT; ++i) {
      int count = 1;
      if (i >= B_P && i < B_P + 3) count = 8;                                    // softmax warps of a tile, both CTAs
      else if (i >= B_MEET) count = 2;                                           // the softmax warps of the same rows
      else if (i >= B_FULLK && i < B_FULLK + A2_STAGES) count = 2;               // a copy warp of each CTA
      else if (i >= B_FULLV && i < B_FULLV + A2_STAGES) count = 2;
      else if (i == B_FULLQ || i == B_FULLQ + 1) count = 4;
      else if (i == B_OFREE) count = 16;
      else if (i == B_TFREE || i == B_TFREE + 1) count = A2_CONSUMERS;
      mbar_init(bars + i, count);
    }
    mbar_init_fence();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();      // both CTAs' barriers exist
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t lead = cluster_addr(base + A2_OFF_MISC, 0);      // the leader's barriers
  const uint32_t tfree = cluster_addr(base + A2_OFF_MISC, 1) + B_TFREE * 8;

  if (warp < 8) {
    // ================= softmax warps =================
    take_registers();
    softmax_role<true>(bars, ring, sM, sFin, tmem, rank, lead, tfree, attn_out, attn_lse, N, abort_flag);
  } else {
    give_registers();
    if (warp == 9 && rank == 1) {
      // ================= the next task and the run list of its union, one task ahead =================
      const PlanView pv = plan_view(plan, H, N, CQ);
      const int numTasks = pv.counters[0];
      for (uint32_t n = 0;; ++n) {
        const uint32_t sl = n & 1u;
        TaskSlot* slot = ring + sl;
        if (!mbar_wait_warp_cluster(bars + B_TFREE + sl, ((n >> 1) & 1u) ^ 1u, abort_flag)) break;
        int task = 0;
        if (lane == 0) {
          do { task = atomicAdd(&pv.counters[2], 1); } while (task < numTasks && pv.tasks[task].w <= QT);
          task = min(task, numTasks);
        }
        task = __shfl_sync(0xffffffffu, task, 0);
        int* runs = sRuns + sl * RUN_INTS;
        prepare_task(pv, ub, CQ, numTasks, task, slot, runs, runs + MAX_RUNS, abort_flag, status);
        // the same for the leader
        const bool end = slot->end;
        const uint32_t there = cluster_addr(smem_u32(runs), 0);
        if (!end && slot->kvlen > 0)
          for (int i = lane; i <= slot->runs; i += 32) {
            cluster_store(there + i * 4, runs[i]);
            cluster_store(there + (MAX_RUNS + i) * 4, runs[MAX_RUNS + i]);
          }
        if (lane < 6) cluster_store(cluster_addr(smem_u32(slot), 0) + lane * 4, reinterpret_cast<const int*>(slot)[lane]);
        __syncwarp();
        if (lane == 0) {
          mbar_release_peer(cluster_addr(smem_u32(bars + B_TFULL + sl), 0));
          mbar_arrive(bars + B_TFULL + sl);
        }
        if (end) break;
      }
    } else if (warp >= 10) {
      // ================= copy warps =================
      const int kind = warp >= 13, cw = warp - 10 - 3 * kind;      // 0: K and Q, 1: V; turn of the three
      // K: rows 64 rank .. of the tile, both 64-column blocks (half a warp each); V: all rows, block `rank`
      const int seg = kind ? 32 : 16, prow = kind ? lane * 4 : (int)rank * 64 + (lane & 15) * 4;
      const int col = kind ? (int)rank * 64 : (lane >> 4) * 64;
      const uint32_t off = base + (kind ? A2_OFF_V + lane * 512 : A2_OFF_K + (lane >> 4) * (A2_HALF / 2) + (lane & 15) * 512);
      const CUtensorMap* map1 = kind ? &maps.v1 : &maps.k1;
      const CUtensorMap* map32 = kind ? &maps.v32 : &maps.k32;
      const CUtensorMap* map64 = kind ? &maps.v64 : &maps.k64;
      const int bfull = kind ? B_FULLV : B_FULLK;
      uint32_t g = 0, q = 0;      // tiles, tasks with tiles so far
      int turn = 0;               // warp of tile g
      bool ok = true;
      for (uint32_t n = 0;; ++n) {
        const uint32_t sl = n & 1u;
        if (!mbar_wait_warp_cluster(bars + B_TFULL + sl, (n >> 1) & 1u, abort_flag)) break;
        const TaskSlot tk = ring[sl];
        if (tk.end) break;
        const int* sRunStart = sRuns + sl * RUN_INTS;
        const int* sRunCum = sRunStart + MAX_RUNS;
        const int ntiles = cdiv(tk.kvlen, KT);
        if (ntiles > 0 && kind == 0 && cw < 2) {
          // one 64-column block of the Q tile each; slots past the group repeat its first row
          const int rows0 = group_rows(tk.rows), nr = rank ? tk.rows - rows0 : rows0;
          const size_t rowbase = (size_t)tk.head * N + tk.first + (rank && nr > 0 ? rows0 : 0);
          int r[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            r[j] = tk.head * q_head_step + qperm[rowbase + (lane * 4 + j < nr ? lane * 4 + j : 0)] * q_row_step;
          ok = mbar_wait_warp(bars + B_FREEQ + (q & 1u), ((q >> 1) & 1u) ^ 1u, abort_flag);
          if (!ok) break;
          const uint32_t full = lead + (B_FULLQ + (q & 1u)) * 8;
          if (lane == 0) {
            if (rank == 0 && cw == 0) mbar_arrive_expect_tx(bars + B_FULLQ + (q & 1u), 2 * AT_TILE);
            else mbar_arrive_peer(full);
          }
          __syncwarp();
          tma_gather4_pair(base + (q & 1u) * AT_TILE + cw * (KT * 128) + lane * 512, &mapQ, cw * 64, r[0], r[1], r[2],
                           r[3], full);
        }
        int cursor = 0;
        for (int t = 0; t < ntiles; ++t, ++g) {
          if (turn != cw) { turn = turn == 2 ? 0 : turn + 1; continue; }
          turn = turn == 2 ? 0 : turn + 1;
          int r[4];
          const bool whole = union_rows(sRunStart, sRunCum, tk.runs, tk.kvlen, t * KT + prow, tk.head * N, cursor, r);
          const int what = fetch_plan(r, whole, lane, seg);
          const uint32_t slot = g & 3u;
          ok = g < 4u || mbar_wait_warp(bars + (kind ? B_PV : B_QK) + slot, ((g - 4u) >> 2) & 1u, abort_flag);
          if (!ok) break;
          const uint32_t full = lead + (bfull + slot) * 8;
          if (lane == 0) {
            if (rank == 0) mbar_arrive_expect_tx(bars + bfull + slot, 2 * A2_HALF);
            else mbar_arrive_peer(full);
          }
          const uint32_t dst = off + slot * A2_HALF;
          if (what == FETCH_GATHER) tma_gather4_pair(dst, map1, col, r[0], r[1], r[2], r[3], full);
          else if (what == FETCH_BOX32) tma_load_tile_pair(dst, map32, col, r[0], full);
          else if (what == FETCH_BOX64) tma_load_tile_pair(dst, map64, col, r[0], full);
        }
        if (!ok) break;
        if (ntiles > 0) ++q;
        __syncwarp();
        if (lane == 0) mbar_release_peer(tfree + sl * 8);
      }
    } else if (warp == 8 && rank == 0) {
      // ================= Q K^T: waits for the K tile and for P V to have read the score buffer =================
      constexpr uint32_t idescQK = make_idesc_bf16(256, KT, false, false);
      constexpr uint32_t dhi = sdesc_hi(1024);
      const uint32_t qlo = sdesc_lo(base, 16), klo = sdesc_lo(base + A2_OFF_K, 16);
      uint32_t g = 0, q = 0, tS = tmem;      // tiles, tasks with tiles, score buffer of the next tile
      bool ok = true;
      for (uint32_t n = 0; ok; ++n) {
        const uint32_t sl = n & 1u;
        if (!mbar_wait_warp_cluster(bars + B_TFULL + sl, (n >> 1) & 1u, abort_flag)) break;
        const int end = ring[sl].end, ntiles = cdiv(ring[sl].kvlen, KT);
        __syncwarp();
        if (end) break;
        if (ntiles == 0) {
          if (lane == 0) mbar_release_peer(tfree + sl * 8);
          continue;
        }
        if (!mbar_wait_warp(bars + B_FULLQ + (q & 1u), (q >> 1) & 1u, abort_flag)) break;
        const uint32_t a0 = qlo + (q & 1u) * (AT_TILE >> 4);
        for (int t = 0; t < ntiles; ++t, ++g) {
          const uint32_t slot = g & 3u, b0 = klo + slot * (A2_HALF >> 4);
          ok = mbar_wait_warp(bars + B_FULLK + slot, (g >> 2) & 1u, abort_flag) &&
               (g < 3u || mbar_wait_warp(bars + B_PV + ((g - 3u) & 3u), ((g - 3u) >> 2) & 1u, abort_flag));
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
#pragma unroll
            for (int s = 0; s < 8; ++s)
              umma_ss_pair(tS, a0 + (s >> 2) * ((QT * 128) >> 4) + (s & 3) * 2,
                           b0 + (s >> 2) * ((A2_HALF / 2) >> 4) + (s & 3) * 2, dhi, idescQK, s > 0 ? 1u : 0u);
            umma_commit_pair(bars + B_QK + slot);
            if (t + 1 == ntiles) umma_commit_pair(bars + B_FREEQ + (q & 1u));
          }
          __syncwarp();
          tS = tS == tmem + 256 ? tmem : tS + 128;
        }
        ++q;
        if (ok && lane == 0) mbar_release_peer(tfree + sl * 8);
      }
    } else if (warp == 9) {
      // ================= P V =================
      constexpr uint32_t idescPV = make_idesc_bf16(256, kD, false, true);
      constexpr uint32_t dhi = sdesc_hi(1024);
      const uint32_t vlo = sdesc_lo(base + A2_OFF_V, A2_HALF);
      const uint32_t tO = tmem + 3 * 128;
      uint32_t g = 0, q = 0, buf = 0, bph = 0;      // tiles, tasks with tiles, score buffer of the next tile and its phase
      bool ok = true;
      for (uint32_t n = 0; ok; ++n) {
        const uint32_t sl = n & 1u;
        if (!mbar_wait_warp_cluster(bars + B_TFULL + sl, (n >> 1) & 1u, abort_flag)) break;
        const int end = ring[sl].end, ntiles = cdiv(ring[sl].kvlen, KT);
        __syncwarp();
        if (end) break;
        if (ntiles == 0) {
          if (lane == 0) mbar_release_peer(tfree + sl * 8);
          continue;
        }
        // every softmax warp has read the O of the task before
        if (!mbar_wait_warp(bars + B_OFREE, (q & 1u) ^ 1u, abort_flag)) break;
        for (int t = 0; t < ntiles; ++t, ++g) {
          const uint32_t slot = g & 3u, v0 = vlo + slot * (A2_HALF >> 4), tS = tmem + buf * 128, add = t > 0 ? 1u : 0u;
          ok = mbar_wait_warp(bars + B_FULLV + slot, (g >> 2) & 1u, abort_flag) &&
               mbar_wait_warp(bars + B_P + buf, bph, abort_flag);
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
#pragma unroll
            for (int s8 = 0; s8 < 8; ++s8)
              umma_ts_pair(tO, tS + s8 * 8, v0 + s8 * (2048 >> 4), dhi, idescPV, s8 > 0 ? 1u : add);
            umma_commit_pair(bars + B_PV + slot);
          }
          __syncwarp();
          if (++buf == 3) { buf = 0; bph ^= 1u; }
        }
        ++q;
        if (ok && lane == 0) mbar_release_peer(tfree + sl * 8);
      }
    }
  }
  __syncwarp();
  if (*abort_flag) {
    if (tid == 0 && status) atomicCAS(status, ST_OK, ST_WAIT_TIMEOUT);
    // a wait gave up: let tile copies still in flight land before the shared memory is released
    for (int i = 0; i < 100; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();      // the other CTA no longer arrives here, and both are done with tensor memory
  if (warp == 0) tmem_dealloc_pair(tmem, 512);
}

// ---------------------------------------------------------------------------
// exact attention, tasks of at most QT rows
// ---------------------------------------------------------------------------
// attn2_kernel's pipeline on one CTA per SM: three score buffers and O fill tensor memory, the softmax of a tile belongs
// to one of two warpgroups, S = Q K^T runs two tiles ahead of P V.  A CTA keeps whole K and V tiles, 64 KB a tile for 128
// rows, so the loads bound it: tile loads (TMA) where 32 or more rows of the union are contiguous; of the groups of four
// rows between them a third comes by TMA gathers and the rest by 16-byte cp.async (26 and 28 B/clk alone).
// 404 k tiles at 720p x 40 heads take 3.4 ms, 2,300 cycles a tile and SM (3.70 with two CTAs per SM, single K / V buffers
// and the rows found by every copy warp), 321 k at 480p x 40 and 5 % 2.9 ms (3.28), 49 tasks at 2 x 4096 30 us less.
// With 64-row tile loads from any rows instead it would be 2.8 and 2.25 ms, with next to no loads 2.5 and 2.1.
//   warps 0..7   softmax (see softmax_role)
//   warp 8 / 9   issue Q K^T / P V
//   warp 10      the next task, the run list of its union, its Q tile
//   warp 11      the source rows of the next tiles and how they are fetched (see fetch_plan), a ring of A1_PLANS of them
//   warps 12, 13 the K tiles, warps 14, 15 the V tiles, half of a tile's copies each
// Barriers as in attn2_kernel; FULLK / FULLV take an arrival that announces the bytes of the TMA copies and one of every
// thread that copies, by the hardware once the thread's cp.async rows have landed.  PLAN / PFREE[g mod 8]: tile g's rows
// are there, its copy warps have read them.
constexpr int A1_THREADS = 16 * 32;
constexpr int A1_KST = 3, A1_VST = 2;                     // K and V ring depth; one Q tile
constexpr int A1_TEAM = 2;                                // warps that share a K tile, a V tile
constexpr int A1_PLANS = 8;
struct TilePlan {
  int rows[QT];                      // source row of every row of the tile
  unsigned gathers, box32, box64;    // four-row groups that are gathered, that start a 32- or 64-row tile load
  unsigned pad;
};
// Groups gathered by TMA rather than cp.async: 3.34 / 2.87 ms (720p / 480p) with a third of them, 3.44 / 2.91 with half,
// 3.36 / 3.01 with all, 3.4 / 3.2 with none.
constexpr unsigned kGatherByTma = 0x92492492u;
constexpr unsigned kSecondHalf = 0xccccccccu;             // groups whose copies the second warp of a team starts
enum { B_PLAN = B_COUNT, B_PFREE = B_PLAN + A1_PLANS, A1_BARS = B_PFREE + A1_PLANS };
constexpr int A1_OFF_K = AT_TILE;
constexpr int A1_OFF_V = A1_OFF_K + A1_KST * AT_TILE;
constexpr int A1_OFF_MISC = A1_OFF_V + A1_VST * AT_TILE;
constexpr int A1_OFF_RING = A1_OFF_MISC + 512;
constexpr int A1_OFF_M = A1_OFF_RING + 2 * (int)sizeof(TaskSlot);
constexpr int A1_OFF_FIN = A1_OFF_M + 2 * QT * 8;
constexpr int A1_OFF_ROWS = A1_OFF_FIN + 4 * QT * 8;      // [128] source rows of the Q tile
constexpr int A1_OFF_PLAN = A1_OFF_ROWS + QT * 4;
constexpr int A1_OFF_RUNS = A1_OFF_PLAN + A1_PLANS * (int)sizeof(TilePlan);
constexpr int A1_SMEM = A1_OFF_RUNS + 2 * RUN_INTS * 4 + 1024;
constexpr int A1_CONSUMERS = 8 + 2 + 1 + 2 * A1_TEAM;     // warps that read a task: softmax, QK and PV, rows, copy
static_assert(A1_SMEM <= 227 * 1024, "one CTA per SM");
static_assert(A1_KST <= 4 && A1_VST <= 4, "the commits of four tiles are told apart");
static_assert(A1_BARS * 8 + 16 <= 512 && A1_OFF_PLAN % 16 == 0, "the barriers fit their area");

// The four-row groups in `groups` of a 128-row tile, by one warp: cp.async of rows `rows[0..127]` (from `src`, whole rows of
// 128 columns) into the 128-byte-swizzled tile at `dst`.  A half-warp takes two of a group's rows, a lane 16 bytes of each.
__device__ __forceinline__ void copy_groups(uint32_t dst, const __nv_bfloat16* __restrict__ src, const int* rows,
                                            unsigned groups, int lane) {
  const int two = (lane >> 4) * 2, ch = lane & 15;
  const uint32_t at = dst + (ch >> 3) * (QT * 128) + two * 128, swz = ((ch & 7) ^ two) << 4;
  const __nv_bfloat16* from = src + ch * 8;
  while (groups) {
    int i[4];
    int2 two_rows[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      i[k] = __ffs(groups) - 1;
      groups &= groups - 1;
      two_rows[k] = *reinterpret_cast<const int2*>(rows + max(i[k], 0) * 4 + two);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (i[k] < 0) break;
      const uint32_t d = at + i[k] * 512, sw = swz ^ ((i[k] & 1) << 6);
      cp_async16(d + sw, from + (size_t)two_rows[k].x * kD);
      cp_async16(d + 128 + (sw ^ 16u), from + (size_t)two_rows[k].y * kD);
    }
  }
}

__global__ void __launch_bounds__(A1_THREADS, 1) attn_kernel(
    const __grid_constant__ KVMaps maps, const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ kp,
    const __nv_bfloat16* __restrict__ vp, const uint32_t* __restrict__ ub, const int* __restrict__ qperm,
    __nv_bfloat16* __restrict__ attn_out, float* __restrict__ attn_lse, int* __restrict__ plan, int H, int N, int CQ,
    int q_row_step, int q_head_step, int* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (base - smem_u32(smem_raw));
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + A1_OFF_MISC);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + A1_OFF_MISC + A1_BARS * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + A1_OFF_MISC + A1_BARS * 8 + 8);
  TaskSlot* ring = reinterpret_cast<TaskSlot*>(sm + A1_OFF_RING);
  unsigned long long* sM = reinterpret_cast<unsigned long long*>(sm + A1_OFF_M);
  float2* sFin = reinterpret_cast<float2*>(sm + A1_OFF_FIN);
  int* sRuns = reinterpret_cast<int*>(sm + A1_OFF_RUNS);
  TilePlan* plans = reinterpret_cast<TilePlan*>(sm + A1_OFF_PLAN);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (warp == 0) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  if (tid < 2 * QT) sM[tid] = ~0ull;      // no tile
  if (tid == 0) {
    *abort_flag = 0;
    for (int i = 0; i < A1_BARS; ++i) {
      int count = 1;
      if (i >= B_P && i < B_P + 3) count = 4;                                    // softmax warps of a tile
      else if (i >= B_MEET && i < B_MEET + 4) count = 2;                         // the softmax warps of the same rows
      else if (i >= B_FULLK && i < B_FULLK + A1_KST) count = 1 + 32 * A1_TEAM;
      else if (i >= B_FULLV && i < B_FULLV + A1_VST) count = 1 + 32 * A1_TEAM;
      else if (i == B_OFREE) count = 8;
      else if (i >= B_PFREE) count = 2 * A1_TEAM;
      else if (i == B_TFREE || i == B_TFREE + 1) count = A1_CONSUMERS;
      mbar_init(bars + i, count);
    }
    mbar_init_fence();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp < 8) {
    // ================= softmax warps =================
    take_registers();
    softmax_role<false>(bars, ring, sM, sFin, tmem, 0u, 0u, 0u, attn_out, attn_lse, N, abort_flag);
  } else {
    give_registers();
    if (warp == 10) {
      // ================= the next task, the run list of its union and its Q tile =================
      const PlanView pv = plan_view(plan, H, N, CQ);
      const int numTasks = pv.counters[0];
      int* sRows = reinterpret_cast<int*>(sm + A1_OFF_ROWS);
      const uint32_t q_last = (uint32_t)((H - 1) * q_head_step + (N - 1) * q_row_step);      // see kv_last
      uint32_t nq = 0;      // tasks with tiles so far
      for (uint32_t n = 0;; ++n) {
        const uint32_t sl = n & 1u;
        if (!mbar_wait_warp(bars + B_TFREE + sl, ((n >> 1) & 1u) ^ 1u, abort_flag)) break;
        int task = 0;
        if (lane == 0) {
          do { task = atomicAdd(&pv.counters[1], 1); } while (task < numTasks && pv.tasks[task].w > QT);
          task = min(task, numTasks);
        }
        task = __shfl_sync(0xffffffffu, task, 0);
        int* runs = sRuns + sl * RUN_INTS;
        prepare_task(pv, ub, CQ, numTasks, task, ring + sl, runs, runs + MAX_RUNS, abort_flag, status);
        const TaskSlot tk = ring[sl];
        if (lane == 0) mbar_arrive(bars + B_TFULL + sl);
        if (tk.end) break;
        if (tk.kvlen == 0) continue;
        // slots past the task repeat its first row; warps of slots past it compute nothing and need no rows
        const size_t rowbase = (size_t)tk.head * N + tk.first;
        int r[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int row = tk.head * q_head_step + qperm[rowbase + (lane * 4 + j < tk.rows ? lane * 4 + j : 0)] * q_row_step;
          r[j] = (int)min((uint32_t)row, q_last);
        }
        reinterpret_cast<int4*>(sRows)[lane] = make_int4(r[0], r[1], r[2], r[3]);
        __syncwarp();
        if (!mbar_wait_warp(bars + B_FREEQ, (nq & 1u) ^ 1u, abort_flag)) break;
        copy_groups(base, q, sRows, 0xffffffffu >> (32 - 8 * cdiv(tk.rows, 32)), lane);
        cp_async_commit();
        cp_async_wait<0>();
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(bars + B_FULLQ);
        ++nq;
      }
    } else if (warp == 11) {
      // ================= rows of the next tiles =================
      const uint32_t kv_last = (uint32_t)H * (uint32_t)N - 1u;
      uint32_t g = 0;             // tiles so far
      bool ok = true;
      for (uint32_t n = 0;; ++n) {
        const uint32_t sl = n & 1u;
        if (!mbar_wait_warp(bars + B_TFULL + sl, (n >> 1) & 1u, abort_flag)) break;
        const TaskSlot tk = ring[sl];
        if (tk.end) break;
        const int* sRunStart = sRuns + sl * RUN_INTS;
        const int* sRunCum = sRunStart + MAX_RUNS;
        const int ntiles = cdiv(tk.kvlen, KT);
        int first = 0;            // run of the tile's first row
        for (int t = 0; t < ntiles; ++t, ++g) {
          // lane j holds the position of run first + j: the run of this lane's first row is found among those, or
          // stepped to from the last one
          const int p0 = t * KT + lane * 4;
          const int cum = first + lane < tk.runs ? sRunCum[first + lane] : 0x7fffffff;
          int cursor = 0;
#pragma unroll
          for (int d = 16; d > 0; d >>= 1)
            if (__shfl_sync(0xffffffffu, cum, cursor + d) <= p0) cursor += d;
          cursor += first;
          int r[4];
          const bool whole = union_rows(sRunStart, sRunCum, tk.runs, tk.kvlen, p0, tk.head * N, cursor, r);
          const int what = fetch_plan(r, whole, lane, 32);
          first = __shfl_sync(0xffffffffu, cursor, 31);
          const unsigned gathers = __ballot_sync(0xffffffffu, what == FETCH_GATHER);
          const unsigned b32 = __ballot_sync(0xffffffffu, what == FETCH_BOX32), b64 = __ballot_sync(0xffffffffu, what == FETCH_BOX64);
          TilePlan* plan = plans + (g & (A1_PLANS - 1));
          ok = mbar_wait_warp(bars + B_PFREE + (g & (A1_PLANS - 1)), ((g / A1_PLANS) & 1u) ^ 1u, abort_flag);
          if (!ok) break;
          // cp.async has no bounds of its own: a plan that does not match kp / vp stays inside them
#pragma unroll
          for (int j = 0; j < 4; ++j) r[j] = (int)min((uint32_t)r[j], kv_last);
          reinterpret_cast<int4*>(plan->rows)[lane] = make_int4(r[0], r[1], r[2], r[3]);
          if (lane == 0) {
            plan->gathers = gathers;
            plan->box32 = b32;
            plan->box64 = b64;
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(bars + B_PLAN + (g & (A1_PLANS - 1)));
        }
        if (!ok) break;
        __syncwarp();
        if (lane == 0) mbar_arrive(bars + B_TFREE + sl);
      }
    } else if (warp >= 12) {
      // ================= copy warps =================
      const int kind = (warp - 12) / A1_TEAM, member = (warp - 12) % A1_TEAM;      // 0: K, 1: V
      const uint32_t depth = kind ? A1_VST : A1_KST;
      const __nv_bfloat16* src = kind ? vp : kp;
      const CUtensorMap* map1 = kind ? &maps.v1 : &maps.k1;
      const CUtensorMap* map32 = kind ? &maps.v32 : &maps.k32;
      const CUtensorMap* map64 = kind ? &maps.v64 : &maps.k64;
      uint32_t g = 0, slot = 0;                        // tiles so far, ring slot of the next one
      // the lanes whose copies this warp starts: half of the four-row groups (tile loads mostly start at multiples of four groups
      // and then are the first warp's)
      const unsigned mine_mask = member ? kSecondHalf : ~kSecondHalf;
      bool ok = true;
      for (uint32_t n = 0;; ++n) {
        const uint32_t sl = n & 1u;
        if (!mbar_wait_warp(bars + B_TFULL + sl, (n >> 1) & 1u, abort_flag)) break;
        const int end = ring[sl].end, ntiles = cdiv(ring[sl].kvlen, KT);
        __syncwarp();
        if (end) break;
        if (lane == 0) mbar_arrive(bars + B_TFREE + sl);
        for (int t = 0; t < ntiles; ++t, ++g, slot = slot + 1 == depth ? 0 : slot + 1) {
          const TilePlan* plan = plans + (g & (A1_PLANS - 1));
          ok = mbar_wait_warp(bars + B_PLAN + (g & (A1_PLANS - 1)), (g / A1_PLANS) & 1u, abort_flag);
          if (!ok) break;
          const int4 r = reinterpret_cast<const int4*>(plan->rows)[lane];
          const unsigned gathers = plan->gathers, b32 = plan->box32, b64 = plan->box64;
          ok = g < depth || mbar_wait_warp(bars + (kind ? B_PV : B_QK) + ((g - depth) & 3u), ((g - depth) >> 2) & 1u, abort_flag);
          if (!ok) break;
          uint64_t* full = bars + (kind ? B_FULLV : B_FULLK) + slot;
          const uint32_t dst = base + (kind ? A1_OFF_V : A1_OFF_K) + slot * AT_TILE, mine = dst + lane * 512;
          if (member == 0 && lane == 0) {
            const uint32_t bytes = (4u * __popc(gathers & kGatherByTma) + 32u * __popc(b32) + 64u * __popc(b64)) * kD * 2;
            if (bytes) mbar_arrive_expect_tx(full, bytes); else mbar_arrive(full);
          }
          __syncwarp();
          if (((b32 | b64) & mine_mask) >> lane & 1u) {
            const CUtensorMap* map = (b64 >> lane) & 1u ? map64 : map32;
            tma_load_tile(mine, map, 0, r.x, full);
            tma_load_tile(mine + KT * 128, map, 64, r.x, full);
          } else if ((gathers & kGatherByTma & mine_mask) >> lane & 1u) {
            tma_gather4(mine, map1, 0, r.x, r.y, r.z, r.w, full);
            tma_gather4(mine + KT * 128, map1, 64, r.x, r.y, r.z, r.w, full);
          }
          __syncwarp();
          copy_groups(dst, src, plan->rows, gathers & ~kGatherByTma & mine_mask, lane);
          cp_async_arrive(full);
          __syncwarp();
          if (lane == 0) mbar_arrive(bars + B_PFREE + (g & (A1_PLANS - 1)));
        }
        if (!ok) break;
      }
      cp_async_commit();
      cp_async_wait<0>();
    } else if (warp == 8) {
      // ================= Q K^T: waits for the K tile and for P V to have read the score buffer =================
      constexpr uint32_t idescQK = make_idesc_bf16(128, KT, false, false);
      constexpr uint32_t dhi = sdesc_hi(1024);
      const uint32_t qlo = sdesc_lo(base, 16), klo = sdesc_lo(base + A1_OFF_K, 16);
      uint32_t g = 0, nq = 0, tS = tmem;      // tiles, tasks with tiles, score buffer of the next tile
      uint32_t ks = 0, kph = 0;               // K slot and its phase
      bool ok = true;
      for (uint32_t n = 0; ok; ++n) {
        const uint32_t sl = n & 1u;
        if (!mbar_wait_warp(bars + B_TFULL + sl, (n >> 1) & 1u, abort_flag)) break;
        const int end = ring[sl].end, ntiles = cdiv(ring[sl].kvlen, KT);
        __syncwarp();
        if (end) break;
        if (lane == 0) mbar_arrive(bars + B_TFREE + sl);
        if (ntiles == 0) continue;
        if (!mbar_wait_warp(bars + B_FULLQ, nq & 1u, abort_flag)) break;
        for (int t = 0; t < ntiles; ++t, ++g) {
          const uint32_t b0 = klo + ks * (AT_TILE >> 4);
          ok = mbar_wait_warp(bars + B_FULLK + ks, kph, abort_flag) &&
               (g < 3u || mbar_wait_warp(bars + B_PV + ((g - 3u) & 3u), ((g - 3u) >> 2) & 1u, abort_flag));
          if (!ok) break;
          fence_proxy_async();      // rows that came by cp.async
          tc_fence_after();
          if (elect_one()) {
#pragma unroll
            for (int s = 0; s < 8; ++s) {
              const uint32_t off = (s >> 2) * ((QT * 128) >> 4) + (s & 3) * 2;      // 64-column block, 16 columns
              umma_ss_lo(tS, qlo + off, b0 + off, dhi, idescQK, s > 0 ? 1u : 0u);
            }
            umma_commit(bars + B_QK + (g & 3u));
            if (t + 1 == ntiles) umma_commit(bars + B_FREEQ);
          }
          __syncwarp();
          tS = tS == tmem + 256 ? tmem : tS + 128;
          if (++ks == A1_KST) { ks = 0; kph ^= 1u; }
        }
        ++nq;
      }
    } else {
      // ================= P V =================
      constexpr uint32_t idescPV = make_idesc_bf16(128, kD, false, true);
      constexpr uint32_t dhi = sdesc_hi(1024);
      const uint32_t vlo = sdesc_lo(base + A1_OFF_V, KT * 128);
      const uint32_t tO = tmem + 3 * 128;
      uint32_t g = 0, nq = 0, buf = 0, bph = 0;      // tiles, tasks with tiles, score buffer of the next tile and its phase
      uint32_t vs = 0, vph = 0;                      // V slot and its phase
      bool ok = true;
      for (uint32_t n = 0; ok; ++n) {
        const uint32_t sl = n & 1u;
        if (!mbar_wait_warp(bars + B_TFULL + sl, (n >> 1) & 1u, abort_flag)) break;
        const int end = ring[sl].end, ntiles = cdiv(ring[sl].kvlen, KT);
        __syncwarp();
        if (end) break;
        if (lane == 0) mbar_arrive(bars + B_TFREE + sl);
        if (ntiles == 0) continue;
        // every softmax warp has read the O of the task before
        if (!mbar_wait_warp(bars + B_OFREE, (nq & 1u) ^ 1u, abort_flag)) break;
        for (int t = 0; t < ntiles; ++t, ++g) {
          const uint32_t v0 = vlo + vs * (AT_TILE >> 4), tS = tmem + buf * 128, add = t > 0 ? 1u : 0u;
          ok = mbar_wait_warp(bars + B_FULLV + vs, vph, abort_flag) && mbar_wait_warp(bars + B_P + buf, bph, abort_flag);
          if (!ok) break;
          fence_proxy_async();      // rows that came by cp.async
          tc_fence_after();
          if (elect_one()) {
#pragma unroll
            for (int s8 = 0; s8 < 8; ++s8)
              umma_ts_lo(tO, tS + s8 * 8, v0 + s8 * (2048 >> 4), dhi, idescPV, s8 > 0 ? 1u : add);
            umma_commit(bars + B_PV + (g & 3u));
          }
          __syncwarp();
          if (++buf == 3) { buf = 0; bph ^= 1u; }
          if (++vs == A1_VST) { vs = 0; vph ^= 1u; }
        }
        ++nq;
      }
    }
  }
  __syncwarp();
  if (*abort_flag) {
    if (tid == 0 && status) atomicCAS(status, ST_OK, ST_WAIT_TIMEOUT);
    // a wait gave up: let copies still in flight land before the shared memory is released
    for (int i = 0; i < 100; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
  // This kernel may have started while the kernel launched before it (the tasks above QT rows) was still
  // running.  No CTA leaves before that grid has completed and its results are visible, so that this grid's
  // completion, which later work in the stream waits for, implies the other's.  (Without a programmatic
  // launch the instruction returns at once.)
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
}

// softmax_role on one task of two tiles where some of the commits it waits for never come (a bit of `commits` each: QK of
// tile 0 and 1, PV of tile 0 and 1) and only the lanes in `handed` find the maximum behind tile 0 in place: every warp has to
// leave within its limits.  All scores are 0 (bit 4 of `commits`: 1000 for the odd rows of tile 1), O holds 256.
__global__ void __launch_bounds__(256, 1) softmax_give_up_selftest_kernel(int commits, unsigned handed,
                                                                          __nv_bfloat16* __restrict__ attn_out,
                                                                          float* __restrict__ attn_lse,
                                                                          int* __restrict__ left, int* __restrict__ status) {
  __shared__ uint64_t bars[B_COUNT];
  __shared__ TaskSlot ring[2];
  __shared__ unsigned long long sM[2 * QT];
  __shared__ float2 sFin[4 * QT];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  volatile int* abort_flag = &abort_word;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == 0) {
    tmem_alloc(&tmem_slot, 512);
    tmem_relinquish();
  }
  sM[tid] = tid < QT && (handed >> lane & 1u) ? 0ull : ~0ull;      // tile 0, maximum 0
  if (tid == 0) {
    abort_word = 0;
    for (int i = 0; i < B_COUNT; ++i) {
      int count = 1;
      if (i >= B_P && i < B_P + 3) count = 4;
      else if (i >= B_MEET) count = 2;
      else if (i == B_OFREE) count = 8;
      else if (i == B_TFREE || i == B_TFREE + 1) count = A1_CONSUMERS;
      mbar_init(bars + i, count);
    }
    mbar_init_fence();
    ring[0] = TaskSlot{0, 0, 0, QT, 2 * KT, 1, {0, 0}};
    ring[1] = TaskSlot{1, 0, 0, 0, 0, 0, {0, 0}};
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  if (warp < 4) {
    for (int col = 0; col < 512; col += 16) {
      uint32_t v[16];
      const bool high = (commits & 16) && (lane & 1) && col >= 128 && col < 256;
      for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(col >= 384 ? 256.0f : high ? 1000.0f : 0.0f);
      tmem_st16(tmem_addr(tmem, warp * 32, col), v);
    }
    tmem_wait_st();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (tid == 0) {
    mbar_arrive(bars + B_TFULL);
    mbar_arrive(bars + B_TFULL + 1);
    for (int t = 0; t < 2; ++t) {
      if (commits >> t & 1) mbar_arrive(bars + B_QK + t);
      if (commits >> (2 + t) & 1) mbar_arrive(bars + B_PV + t);
    }
  }
  __syncwarp();
  softmax_role<false, 1u << 10>(bars, ring, sM, sFin, tmem, 0u, 0u, 0u, attn_out, attn_lse, QT, abort_flag);
  __syncwarp();
  if (lane == 0) left[warp] = 1;
  if (*abort_flag && tid == 0) atomicCAS(status, ST_OK, ST_WAIT_TIMEOUT);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

// ---------------------------------------------------------------------------
// centroid residual + merge, 128 sorted queries per CTA
// ---------------------------------------------------------------------------
constexpr int TL_Q = 128;                 // sorted queries per CTA (one softmax thread per row)
constexpr int TL_H = 64;                  // centroids per step
constexpr int TL_NH = kC / TL_H;          // steps per CTA
constexpr int TL_STAGES = 3;              // ring depth of the centroid and value-sum tiles
constexpr int TL_SQ = TL_Q * 128;         // 16 KB: QU rows padded to 128 B
constexpr int TL_SC = TL_H * kR * 2;      // 4 KB per stage: cks rows of 64 B
constexpr int TL_SV = TL_H * kD * 2;      // 16 KB per stage
constexpr int TL_OFF_C = TL_SQ;
constexpr int TL_OFF_V = TL_OFF_C + TL_STAGES * TL_SC;
constexpr int TL_OFF_CNT = TL_OFF_V + TL_STAGES * TL_SV;
constexpr int TL_OFF_BAR = TL_OFF_CNT + kC * 4;
// 85 KB: two CTAs share an SM, and no more than two (tensor memory holds two 256-column allocations)
constexpr int TL_SMEM = TL_OFF_BAR + 128 + 1024;
constexpr int TL_THREADS = 160;           // warps 0..3: one softmax thread per row; warp 4: the products
static_assert(TL_NH % 2 == 0 && TL_NH >= 4, "the two score regions alternate");
static_assert(3 * TL_SMEM > 228 * 1024, "at most two CTAs may share an SM");

// Work is pipelined over steps of 64 centroids.  Tensor memory holds two 64-column score regions and the
// 128-column accumulator T.  For step i (region b = i & 1):
//   MMA lane      S_b = QU cks_i^T  ->  commit on sReady[b]
//   softmax rows  wait sReady[b]; p = exp2(S_b - m) masked by the row's union, packed to bf16 into S_b;
//                 arrive on pReady[b]
//   MMA lane      wait pReady[b]; T += P_b sumv_i; S_b = QU cks_{i+2}^T; commit on sReady[b]
// so the tensor work of one region runs under the softmax of the other.  The MMA lane also feeds the products by TMA
// tile loads, on byte-counting barriers: once pReady[b] of step i shows that every row has seen the commit behind the
// products up to cks_i and sumv_{i-2}, it fetches cks_{i+3} and sumv_{i+1} into the stages those held.  (With the softmax
// threads copying cks by cp.async, each waited for its copy and fenced the proxies in every step: 3.10 ms at 720p x 40
// heads instead of 2.93.)
__global__ void __launch_bounds__(TL_THREADS, 2) tail_kernel(
    const __grid_constant__ CUtensorMap mapSumv, const __grid_constant__ CUtensorMap mapCks,
    const __nv_bfloat16* __restrict__ attn_out,
    const float* __restrict__ attn_lse,
    const __nv_bfloat16* __restrict__ QU, const int* __restrict__ ksz, const uint32_t* __restrict__ ub,
    const int* __restrict__ qlab, const int* __restrict__ qperm, const float* __restrict__ lam_s,
    const float* __restrict__ tailw_ptr, __nv_bfloat16* __restrict__ out, long long out_row_stride,
    long long out_head_stride, int N, int CQ,
    int* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t sQ = base, sC = base + TL_OFF_C, sV = base + TL_OFF_V;
  float* sCnt = reinterpret_cast<float*>(sm + TL_OFF_CNT);
  uint64_t* sReady = reinterpret_cast<uint64_t*>(sm + TL_OFF_BAR);        // [2], one arrival (tcgen05.commit)
  uint64_t* pReady = sReady + 2;                                          // [2], one arrival of every softmax warp
  uint64_t* vFull = sReady + 4;                                           // [TL_STAGES], bytes of one value-sum tile
  uint64_t* cFull = vFull + TL_STAGES;                                    // [TL_STAGES], bytes of one centroid tile
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + TL_OFF_BAR + 96);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + TL_OFF_BAR + 104);

  const int tid = threadIdx.x, warp = tid >> 5;
  const bool soft = warp < 4;
  const int h = blockIdx.y, qs = blockIdx.x * TL_Q;
  if (warp == 0) {
    tmem_alloc(tmem_slot, 256);
    tmem_relinquish();
  }
  if (tid == 0) {
    *abort_flag = 0;
    mbar_init(sReady + 0, 1);
    mbar_init(sReady + 1, 1);
    mbar_init(pReady + 0, TL_Q / 32);
    mbar_init(pReady + 1, TL_Q / 32);
    for (int st = 0; st < 2 * TL_STAGES; ++st) mbar_init(vFull + st, 1);
    mbar_init_fence();
  }
  const int j = qs + tid;
  const bool active = soft && j < N;
  const int orig = active ? qperm[(size_t)h * N + j] : 0;
  const int label = active ? qlab[(size_t)h * N + orig] : 0;
  const uint32_t* mrow = ub + ((size_t)h * CQ + label) * (kC / 32);

  if (soft) {
    // QU rows of the 128 sorted queries (64 B each, 4 chunks), behind the loads of their indices
    const int ch = tid & 3, r0 = tid >> 2;
    int o4[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) o4[u] = qs + r0 + 32 * u < N ? qperm[(size_t)h * N + qs + r0 + 32 * u] : -1;
    const int4* ksz4 = reinterpret_cast<const int4*>(ksz + (size_t)h * kC);
    int4 kz[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) kz[u] = ksz4[tid + TL_Q * u];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int r = r0 + 32 * u;
      cp_async16(sQ + sw128(r, ch), QU + ((size_t)h * N + max(o4[u], 0)) * kR + ch * 8, o4[u] >= 0 ? 16u : 0u);
    }
    cp_async_commit();
    // Four counts x y z w are kept as x z y w, every other two quads as z x w y: the weighted sum of a row runs over four
    // accumulators, two of them per packed multiply-add, and this is the order in which quad k meets them.
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float x = (float)kz[u].x, y = (float)kz[u].y, z = (float)kz[u].z, w = (float)kz[u].w;
      reinterpret_cast<float4*>(sCnt)[tid + TL_Q * u] = (tid & 2) ? make_float4(z, x, w, y) : make_float4(x, z, y, w);
    }
    cp_async_wait<0>();
    fence_proxy_async();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tS = tmem, tO = tmem + 2 * TL_H;
  constexpr uint32_t idescS = make_idesc_bf16(128, TL_H, false, false);
  constexpr uint32_t idescT = make_idesc_bf16(128, kD, false, true);
  constexpr float LOG2E = 1.4426950408889634f;

  if (warp == 4) {
    // ---- MMA warp: one elected lane issues (see elect_one) ----
    constexpr uint32_t dhi = sdesc_hi(1024);
    const uint32_t qlo = sdesc_lo(sQ, 16), clo = sdesc_lo(sC, 16), vlo = sdesc_lo(sV, TL_H * 128);
    // value sums of one step: 64 rows x 256 B as two 64-column blocks, one TMA tile load each
    auto load_v = [&](int step, int st) {
      uint64_t* bar = vFull + st;
      const uint32_t dst = sV + st * TL_SV;
      if (elect_one()) {
        mbar_arrive_expect_tx(bar, TL_SV);
        tma_load_tile(dst, &mapSumv, 0, h * kC + step * TL_H, bar);
        tma_load_tile(dst + TL_H * 128, &mapSumv, 64, h * kC + step * TL_H, bar);
      }
      __syncwarp();
    };
    auto load_c = [&](int step, int st) {
      if (elect_one()) {
        mbar_arrive_expect_tx(cFull + st, TL_SC);
        tma_load_tile(sC + st * TL_SC, &mapCks, 0, h * kC + step * TL_H, cFull + st);
      }
      __syncwarp();
    };
    // S_(step & 1) = QU cks_step^T, K = 32
    auto scores = [&](int b, int st) {
      const uint32_t c0 = clo + st * (TL_SC >> 4);
#pragma unroll
      for (int k = 0; k < 2; ++k)
        umma_ss_lo2(tS + b * TL_H, qlo + k * 2, dhi, c0 + k * 2, sdesc_hi_64b(), idescS, k > 0 ? 1u : 0u);
      umma_commit(sReady + b);
    };
    for (int step = 0; step < TL_STAGES; ++step) load_c(step, step);
    load_v(0, 0);
    const bool there = mbar_wait_warp(cFull + 0, 0, abort_flag) && mbar_wait_warp(cFull + 1, 0, abort_flag);
    tc_fence_after();
    __syncwarp();
    if (there && elect_one()) {
      scores(0, 0);
      scores(1, 1);
    }
    __syncwarp();
    int st = 0;      // stage of step i
    for (int i = 0; there && i < TL_NH; ++i) {
      const int b = i & 1, st1 = st == TL_STAGES - 1 ? 0 : st + 1, st2 = st1 == TL_STAGES - 1 ? 0 : st1 + 1;
      if (!mbar_wait_warp(pReady + b, (i >> 1) & 1, abort_flag)) break;
      // every softmax thread has seen the commit behind S_i and the product of step i - 2: their stages are free
      if (i + 1 < TL_NH) load_v(i + 1, st1);
      if (i + TL_STAGES < TL_NH) load_c(i + TL_STAGES, st);
      if (!mbar_wait_warp(vFull + st, (i / TL_STAGES) & 1, abort_flag)) break;
      if (i + 2 < TL_NH && !mbar_wait_warp(cFull + st2, ((i + 2) / TL_STAGES) & 1, abort_flag)) break;
      tc_fence_after();
      const uint32_t v0 = vlo + st * (TL_SV >> 4), first = i > 0 ? 1u : 0u;
      if (elect_one()) {
#pragma unroll
        for (int s8 = 0; s8 < TL_H / 16; ++s8)
          umma_ts_lo(tO, tS + b * TL_H + s8 * 8, v0 + s8 * (2048 >> 4), dhi, idescT, s8 > 0 ? 1u : first);
        if (i + 2 < TL_NH) scores(b, st2);
        else umma_commit(sReady + b);
      }
      __syncwarp();
      st = st1;
    }
  }
  bool dead = false;
  if (soft) {
    // ---- softmax rows ----
    const uint32_t tS_lane = tmem_addr(tS, warp * 32, 0), tO_lane = tmem_addr(tO, warp * 32, 0);
    float m = -INFINITY, phi = 0.f;     // m in log2 units
    uint2 mw_next = *reinterpret_cast<const uint2*>(mrow);   // union bits of the step's 64 centroids
    for (int i = 0; i < TL_NH; ++i) {
      const int b = i & 1;
      if (!mbar_wait_warp(sReady + b, (i >> 1) & 1, abort_flag)) { dead = true; break; }
      tc_fence_after();
      const uint2 mw2 = mw_next;
      if (i + 1 < TL_NH) mw_next = *reinterpret_cast<const uint2*>(mrow + (i + 1) * 2);
      float s[TL_H];
      {
        uint32_t v0[32], v1[32];
        tmem_ld32(tS_lane + b * TL_H, v0);
        tmem_ld32(tS_lane + b * TL_H + 32, v1);
        tmem_wait_ld();
#pragma unroll
        for (int k = 0; k < 32; ++k) {
          s[k] = __uint_as_float(v0[k]);
          s[32 + k] = __uint_as_float(v1[k]);
        }
      }
      // The scores are rounded to fp16 exactly as the selection saw them, and the members of the row's union
      // become -inf, both on packed pairs: shifting a word of union bits left by 7 - r puts the bits of the
      // centroids r, r + 8, r + 16, r + 24 on the sign bits of its four bytes, and a byte permute with sign
      // replication turns two such bytes into the select mask of a pair.  The scores stay in natural-log
      // units here; log2(e) is folded into the exponent's multiply-add below.
      const uint32_t mw[2] = {mw2.x, mw2.y};
      uint32_t sh[2][8];
#pragma unroll
      for (int w = 0; w < 2; ++w)
#pragma unroll
        for (int r = 0; r < 8; ++r) sh[w][r] = mw[w] << (7 - r);
      __half2 hm[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) hm[a] = __float2half2_rn(-INFINITY);
#pragma unroll
      for (int k = 0; k < TL_H; k += 2) {
        const int w = k >> 5, r = k & 7, jb = (k & 31) >> 3;
        const uint32_t sel = (8u | jb) * 0x11u | ((8u | (4u + jb)) * 0x11u) << 8;
        uint32_t msk;   // selector bit 3 of a nibble: replicate the chosen byte's sign over the result byte
        asm("prmt.b32 %0, %1, %2, %3;" : "=r"(msk) : "r"(sh[w][r]), "r"(sh[w][r + 1]), "r"(sel));
        const __half2 h2 = __floats2half2_rn(s[k], s[k + 1]);
        const uint32_t u = (*reinterpret_cast<const uint32_t*>(&h2) & ~msk) | (0xFC00FC00u & msk);
        const __half2 hq = *reinterpret_cast<const __half2*>(&u);
        hm[(k >> 1) & 3] = __hmax2(hm[(k >> 1) & 3], hq);
        const float2 g = __half22float2(hq);
        s[k] = g.x;
        s[k + 1] = g.y;
      }
      const float2 mxp = __half22float2(__hmax2(__hmax2(hm[0], hm[1]), __hmax2(hm[2], hm[3])));
      const float mx = fmaxf(mxp.x, mxp.y) * LOG2E;
      const bool grow = mx > m + kLazy || (m == -INFINITY && mx > -INFINITY);
      if (__any_sync(0xffffffffu, grow)) {
        const float mnew = grow ? mx : m;
        const float alpha = (m == -INFINITY) ? 0.f : ex2_approx(m - mnew);
        if (i > 0) {
          // T is rescaled in place: the product of step i - 1 may still be running, its commit is the
          // next completion of the other region's barrier (the same one step i + 1 waits for)
          if (!mbar_wait_warp(sReady + (b ^ 1), (((i - 1) >> 1) + 1) & 1, abort_flag)) { dead = true; break; }
          tc_fence_after();
          rescale_rows(tO_lane, alpha);
        }
        phi *= alpha;
        m = mnew;
      }
      const float nm = (m == -INFINITY) ? 0.f : -m;
      const unsigned long long l2e2 = pack_f2(LOG2E, LOG2E), nm2 = pack_f2(nm, nm);
      const float4* cnt4 = reinterpret_cast<const float4*>(sCnt + i * TL_H);
      unsigned long long even2 = 0ull, odd2 = 0ull;      // accumulators 0 and 2, 1 and 3
      uint32_t pk[TL_H / 2];
#pragma unroll
      for (int k = 0; k < TL_H / 4; ++k) {
        const float4 cn = cnt4[k];
        float y0, y1, y2, y3, p0, p1, p2, p3;
        unpack_f2(fma_f2(pack_f2(s[4 * k], s[4 * k + 1]), l2e2, nm2), y0, y1);
        unpack_f2(fma_f2(pack_f2(s[4 * k + 2], s[4 * k + 3]), l2e2, nm2), y2, y3);
        // every third group of four on the FMA pipe: the two CTAs of an SM share one special-function unit.
        // (A member of the row's union, -inf here, then weighs 2^-125 instead of an exact zero.)
        if (k % 3 == 2) {
          exp2_fma2(y0, y1, p0, p1);
          exp2_fma2(y2, y3, p2, p3);
        } else {
          p0 = ex2_approx(y0);
          p1 = ex2_approx(y1);
          p2 = ex2_approx(y2);
          p3 = ex2_approx(y3);
        }
        unsigned long long& acc = (k & 1) ? odd2 : even2;
        acc = fma_f2((k & 2) ? pack_f2(p2, p0) : pack_f2(p0, p2), pack_f2(cn.x, cn.y), acc);
        acc = fma_f2((k & 2) ? pack_f2(p3, p1) : pack_f2(p1, p3), pack_f2(cn.z, cn.w), acc);
        pk[2 * k] = pack_bf2(p0, p1);
        pk[2 * k + 1] = pack_bf2(p2, p3);
      }
      float ps4[4];
      unpack_f2(even2, ps4[0], ps4[2]);
      unpack_f2(odd2, ps4[1], ps4[3]);
      phi += (ps4[0] + ps4[1]) + (ps4[2] + ps4[3]);
      tmem_st32(tS_lane + b * TL_H, pk);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if ((tid & 31) == 0) mbar_arrive(pReady + b);
    }
    // the row of the exact part is fetched while the last products finish
    const uint4* src = reinterpret_cast<const uint4*>(attn_out + ((size_t)h * N + (active ? j : 0)) * kD);
    uint4 ex16[16];
#pragma unroll
    for (int g = 0; g < 16; ++g) ex16[g] = ldg_nc_v4(src + g);
    const float lam = lam_s[h], tw = *tailw_ptr;
    const float le = active ? attn_lse[(size_t)h * N + j] : 0.f;
    // the last commit on each region's barrier covers every product
    if (!dead) dead = !mbar_wait_warp(sReady + 0, (TL_NH >> 1) & 1, abort_flag);
    if (!dead) dead = !mbar_wait_warp(sReady + 1, (TL_NH >> 1) & 1, abort_flag);
    tc_fence_after();
    if (!dead) {
      // merge with the exact part (natural-log units from here on); rows past N
      // only take part in the warp-collective TMEM loads
      const float mt = (m == -INFINITY) ? 0.f : m * 0.6931471805599453f;
      float ex, st;
      if (le >= mt) { ex = 1.0f; st = __expf(mt - le); } else { ex = __expf(le - mt); st = 1.0f; }
      const float ph = st * phi;
      const bool bad = ph <= 1.0e-6f * ex;
      const float inv = 1.0f / fmaxf(ex + ph * tw, 1.0e-12f);
      const float we = bad ? 1.0f : ex * inv;
      const float wt = bad ? 0.0f : st * tw * lam * inv;
      uint4* dst = reinterpret_cast<uint4*>(out + (size_t)h * out_head_stride + (size_t)orig * out_row_stride);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t v[32];
        tmem_ld32(tO_lane + c * 32, v);
        tmem_wait_ld();
        if (active) {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            const uint4 e = ex16[c * 4 + g];
            uint4 o;
            if (bad) {
              o = e;
            } else {
              o.x = pack_bf2(fmaf(wt, __uint_as_float(v[8 * g + 0]), we * bf_lo(e.x)), fmaf(wt, __uint_as_float(v[8 * g + 1]), we * bf_hi(e.x)));
              o.y = pack_bf2(fmaf(wt, __uint_as_float(v[8 * g + 2]), we * bf_lo(e.y)), fmaf(wt, __uint_as_float(v[8 * g + 3]), we * bf_hi(e.y)));
              o.z = pack_bf2(fmaf(wt, __uint_as_float(v[8 * g + 4]), we * bf_lo(e.z)), fmaf(wt, __uint_as_float(v[8 * g + 5]), we * bf_hi(e.z)));
              o.w = pack_bf2(fmaf(wt, __uint_as_float(v[8 * g + 6]), we * bf_lo(e.w)), fmaf(wt, __uint_as_float(v[8 * g + 7]), we * bf_hi(e.w)));
            }
            dst[c * 4 + g] = o;
          }
        }
      }
    }
  }
  __syncwarp();
  if (*abort_flag) {
    if ((tid & 31) == 0 && status) atomicCAS(status, ST_OK, ST_WAIT_TIMEOUT);
    // a wait gave up: let tile copies still in flight land before the shared memory is released
    for (int i = 0; i < 100; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 256);
}

}  // namespace t2t

using namespace t2t;

namespace {
// Launch facts that do not change between calls: looked up (and the kernels' shared-memory limits raised)
// once per device and process, not on every call.
struct DeviceFacts {
  bool ready;
  int sms;
};
std::mutex g_facts_mutex;
const DeviceFacts* device_facts() {
  static DeviceFacts table[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  std::lock_guard<std::mutex> lock(g_facts_mutex);
  DeviceFacts* f = &table[dev];
  if (!f->ready) {
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) return nullptr;
    if (cudaFuncSetAttribute(attn_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, A1_SMEM) != cudaSuccess ||
        cudaFuncSetAttribute(attn2_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, A2_SMEM) != cudaSuccess ||
        cudaFuncSetAttribute(tail_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TL_SMEM) != cudaSuccess)
      return nullptr;
    cudaFuncAttributes small, large;
    if (cudaFuncGetAttributes(&small, attn_kernel) != cudaSuccess || cudaFuncGetAttributes(&large, attn2_kernel) != cudaSuccess ||
        !split_fits(small.numRegs) || !split_fits(large.numRegs))
      return nullptr;
    f->sms = sms;
    f->ready = true;
  }
  return f;
}

// Tensor maps are pure functions of (base address, rows, columns, box rows): the operator passes the same few buffers on
// every call, so the last encodings are kept.
struct MapSlot {
  const void* base;
  uint64_t rows;
  uint32_t box_rows;
  int cols;
  CUtensorMap map;
};
std::mutex g_map_mutex;
bool cached_row_map(CUtensorMap* out, const void* base, uint64_t rows, uint32_t box_rows, int cols = kD) {
  static MapSlot slots[32] = {};
  static unsigned next = 0;
  std::lock_guard<std::mutex> lock(g_map_mutex);
  for (const MapSlot& s : slots)
    if (s.base == base && s.rows == rows && s.box_rows == box_rows && s.cols == cols && s.base != nullptr) { *out = s.map; return true; }
  MapSlot fresh;
  fresh.base = base;
  fresh.rows = rows;
  fresh.box_rows = box_rows;
  fresh.cols = cols;
  if (!(cols == kD ? make_row_tile_map(&fresh.map, base, rows, box_rows) : make_rank_tile_map(&fresh.map, base, rows, box_rows)))
    return false;
  slots[next++ % 32] = fresh;
  *out = fresh.map;
  return true;
}
}  // namespace

extern "C" size_t t2t_tile_attn_plan_ints(int H, int N, int CQ) {
  return plan_task_offset(H) + 4 * plan_max_tasks(H, N, CQ) + (size_t)H * CQ;
}

extern "C" size_t t2t_tile_attn_ws_bytes(int H, int N) {
  return (((size_t)H * N * kD * 2 + 255) & ~(size_t)255) + (size_t)H * N * 4;
}

static void split_ws(void* ws, int H, int N, __nv_bfloat16** attn_out, float** attn_lse) {
  *attn_out = (__nv_bfloat16*)ws;
  *attn_lse = (float*)((char*)ws + (((size_t)H * N * kD * 2 + 255) & ~(size_t)255));
}

extern "C" int t2t_tile_attn_plan(const void* tile_sizes, const void* kcounts, const void* unip, int* plan, int H,
                                  int N, int CQ, cudaStream_t st) {
  if (!tile_sizes || !kcounts || !unip || !plan || H <= 0 || N <= 0 || CQ <= 0) return T2T_ERR_ARG;
  plan_kernel<<<H, PLAN_THREADS, 0, st>>>((const int*)tile_sizes, (const int*)kcounts, (const uint32_t*)unip, H, N, CQ, plan);
  return cudaGetLastError() == cudaSuccess ? T2T_OK : T2T_ERR_CUDA;
}

extern "C" int t2t_tile_attn_exact(const void* q, const void* kp, const void* vp, const void* unip,
                                   const void* qperm, int* plan, int H, int N, int CQ, void* ws, size_t ws_bytes,
                                   int* d_status, cudaStream_t st) {
  return t2t_tile_attn_exact_strided(q, (long long)kD, (long long)N * kD, kp, vp, unip, qperm, plan, H, N, CQ, ws,
                                     ws_bytes, d_status, st);
}

extern "C" int t2t_tile_attn_exact_strided(const void* q, long long q_row_stride, long long q_head_stride,
                                           const void* kp, const void* vp, const void* unip, const void* qperm,
                                           int* plan, int H, int N, int CQ, void* ws, size_t ws_bytes,
                                           int* d_status, cudaStream_t st) {
  if (!q || !kp || !vp || !unip || !qperm || !plan || !ws || H <= 0 || N <= 0 || CQ <= 0) return T2T_ERR_ARG;
  // q rows are fetched by TMA row gathers and 16-byte copies from a [rows, 128] view of the tensor: whole rows between rows
  if (q_row_stride < kD || q_head_stride <= 0 || (q_row_stride % kD) || (q_head_stride % kD)) return T2T_ERR_ARG;
  const int q_row_step = (int)(q_row_stride / kD), q_head_step = (int)(q_head_stride / kD);
  const uint64_t q_rows = (uint64_t)(H - 1) * q_head_step + (uint64_t)(N - 1) * q_row_step + 1;
  if (ws_bytes < t2t_tile_attn_ws_bytes(H, N)) return T2T_ERR_WORKSPACE;
  __nv_bfloat16* attn_out;
  float* attn_lse;
  split_ws(ws, H, N, &attn_out, &attn_lse);
  const PlanView pv = plan_view(plan, H, N, CQ);
  // the task cursors are the only per-dispatch state of a prepared plan
  if (cudaMemsetAsync(pv.counters + 1, 0, 2 * sizeof(int), st) != cudaSuccess) return T2T_ERR_CUDA;
  const DeviceFacts* facts = device_facts();
  if (!facts) return T2T_ERR_CUDA;
  const int sms = facts->sms;
  // tensor maps over q, kp, vp as matrices of whole rows: boxes of one row (four-row gathers), 32 and 64 rows
  CUtensorMap mq;
  KVMaps kv;
  const uint64_t rows = (uint64_t)H * (uint64_t)N;
  if (!cached_row_map(&mq, q, q_rows, 1) || !cached_row_map(&kv.k1, kp, rows, 1) ||
      !cached_row_map(&kv.k32, kp, rows, 32) || !cached_row_map(&kv.k64, kp, rows, 64) ||
      !cached_row_map(&kv.v1, vp, rows, 1) || !cached_row_map(&kv.v32, vp, rows, 32) ||
      !cached_row_map(&kv.v64, vp, rows, 64))
    return T2T_ERR_CUDA;
  // tasks above 128 rows first (CTA pairs, one CTA per SM with one of a task's two row tiles), then the others
  attn2_kernel<<<sms & ~1, A2_THREADS, A2_SMEM, st>>>(mq, kv, (const uint32_t*)unip, (const int*)qperm, attn_out,
                                                 attn_lse, plan, H, N, CQ, q_row_step, q_head_step, d_status);
  // The two kernels take disjoint tasks (own cursors, own output rows), so the second may start while the
  // first drains: it is launched with programmatic stream serialization and the first kernel releases its
  // dependents at once.  Their CTAs cannot share an SM (shared memory), so the second kernel's CTAs move in
  // as the first kernel's CTAs run out of tasks and exit.  Later work in the stream waits for both as usual.
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(sms);
  cfg.blockDim = dim3(A1_THREADS);
  cfg.dynamicSmemBytes = A1_SMEM;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, attn_kernel, kv, (const __nv_bfloat16*)q, (const __nv_bfloat16*)kp, (const __nv_bfloat16*)vp,
                         (const uint32_t*)unip, (const int*)qperm, attn_out, attn_lse, plan, H, N, CQ, q_row_step,
                         q_head_step, d_status) != cudaSuccess)
    return T2T_ERR_CUDA;
  return cudaGetLastError() == cudaSuccess ? T2T_OK : T2T_ERR_CUDA;
}

extern "C" int t2t_tile_attn_merge(const void* QU, const void* cks, const void* sumv, const void* kcounts,
                                   const void* unip, const void* qlab, const void* qperm, const void* lam,
                                   const float* tailw, void* out, int H, int N, int CQ, void* ws, size_t ws_bytes,
                                   int* d_status, cudaStream_t st) {
  return t2t_tile_attn_merge_strided(QU, cks, sumv, kcounts, unip, qlab, qperm, lam, tailw, out, (long long)kD,
                                     (long long)N * kD, H, N, CQ, ws, ws_bytes, d_status, st);
}

extern "C" int t2t_tile_attn_merge_strided(const void* QU, const void* cks, const void* sumv, const void* kcounts,
                                           const void* unip, const void* qlab, const void* qperm, const void* lam,
                                           const float* tailw, void* out, long long out_row_stride,
                                           long long out_head_stride, int H, int N, int CQ, void* ws,
                                           size_t ws_bytes, int* d_status, cudaStream_t st) {
  if (!QU || !cks || !sumv || !kcounts || !unip || !qlab || !qperm || !lam || !tailw || !out || !ws)
    return T2T_ERR_ARG;
  if (H <= 0 || N <= 0 || CQ <= 0) return T2T_ERR_ARG;
  if (out_row_stride < kD || out_head_stride <= 0 || (out_row_stride & 7) || (out_head_stride & 7)) return T2T_ERR_ARG;
  if (ws_bytes < t2t_tile_attn_ws_bytes(H, N)) return T2T_ERR_WORKSPACE;
  __nv_bfloat16* attn_out;
  float* attn_lse;
  split_ws(ws, H, N, &attn_out, &attn_lse);
  if (!device_facts()) return T2T_ERR_CUDA;
  // the value sums as an [H * 2048, 128] matrix, fetched 64 rows x 64 columns at a time
  CUtensorMap msv, mck;
  if (!cached_row_map(&msv, sumv, (uint64_t)H * kC, TL_H) || !cached_row_map(&mck, cks, (uint64_t)H * kC, TL_H, kR))
    return T2T_ERR_CUDA;
  tail_kernel<<<dim3(cdiv(N, TL_Q), H), TL_THREADS, TL_SMEM, st>>>(
      msv, mck, attn_out, attn_lse, (const __nv_bfloat16*)QU, (const int*)kcounts, (const uint32_t*)unip, (const int*)qlab, (const int*)qperm, (const float*)lam, tailw,
      (__nv_bfloat16*)out, out_row_stride, out_head_stride, N, CQ, d_status);
  return cudaGetLastError() == cudaSuccess ? T2T_OK : T2T_ERR_CUDA;
}

extern "C" int t2t_tile_attn(const void* q, const void* kp, const void* vp, const void* tile_sizes,
                             const void* kcounts, const void* unip, const void* QU, const void* cks,
                             const void* sumv, const void* lam, const void* qlab, const void* qperm,
                             const float* tailw, void* out, int* plan, int rebuild_plan, int H, int N, int CQ,
                             void* ws, size_t ws_bytes, int* d_status, cudaStream_t st) {
  int rc = T2T_OK;
  if (rebuild_plan) rc = t2t_tile_attn_plan(tile_sizes, kcounts, unip, plan, H, N, CQ, st);
  if (rc == T2T_OK) rc = t2t_tile_attn_exact(q, kp, vp, unip, qperm, plan, H, N, CQ, ws, ws_bytes, d_status, st);
  if (rc == T2T_OK)
    rc = t2t_tile_attn_merge(QU, cks, sumv, kcounts, unip, qlab, qperm, lam, tailw, out, H, N, CQ, ws, ws_bytes,
                             d_status, st);
  return rc;
}

extern "C" int t2t_tile_attn_plan_info(const int* plan, int H, int N, int CQ, int* d_info, cudaStream_t st) {
  if (!plan || !d_info) return T2T_ERR_ARG;
  const PlanView pv = plan_view(const_cast<int*>(plan), H, N, CQ);
  plan_info_kernel<<<1, 1024, 0, st>>>(pv, CQ, d_info);
  return cudaGetLastError() == cudaSuccess ? T2T_OK : T2T_ERR_CUDA;
}

extern "C" int t2t_register_split_selftest(int regs) { return split_fits(regs) ? T2T_OK : T2T_ERR_CUDA; }

extern "C" int t2t_softmax_give_up_selftest(int commits, unsigned handed, void* out, float* lse, int* d_left, int* d_status,
                                            cudaStream_t st) {
  if (!out || !lse || !d_left || !d_status) return T2T_ERR_ARG;
  softmax_give_up_selftest_kernel<<<1, 256, 0, st>>>(commits, handed, (__nv_bfloat16*)out, lse, d_left, d_status);
  return cudaGetLastError() == cudaSuccess ? T2T_OK : T2T_ERR_CUDA;
}
