// Nearest-centroid assignment on the tensor cores with exact verification.
//
// The label of a row is DEFINED by the fp32 fused-multiply-add chain of
// assign_exact_kernel (kmeans.cu): d(i,c) = fma chain over k from ||c||^2 with
// x_k * (-2 c_k), lowest index on ties.  Evaluating that chain for every
// (row, centroid) pair costs N * C * 32 FMAs on the CUDA cores.  Here tcgen05
// MMAs produce s(i,c) = x_i . c - ||c||^2 / 2 = -d / 2 directly: the centroid's
// row carries three more elements, -||c||^2 / 2 split into three bf16 pieces,
// which meet ones in the row of x (K = 48 instead of 32).  A thread per row then
// only has to find the largest value, and it does so by groups of 16 centroids:
// a maximum per group, the three best groups kept in order, and the 16 values of
// the best one.  A label is taken from these approximate values only when every
// other centroid is further away than twice a bound on |approximate - chain|;
// otherwise the exact chain decides, over the 32 centroids of the two best groups
// when the third is out of reach (nearly always), else over all centroids in reach.
// So the labels are bit-identical to the all-exact kernel.
//
// Error bound.  With s~ the tensor-core sum and s the real one,
// |s~ - s| <= kappa * (||x|| ||c|| + ||c||^2 / 2) with kappa = 2^-16 (the measured
// error of the fp32 accumulation is below 2^-20; tests/test_gpu_stages.py checks
// it); the three pieces hold ||c||^2 / 2 to 2^-25 of itself, and the 32-step chain
// is within 2^-19 (||c||^2 + 2 ||x|| ||c||) of the real value.  In units of d = -2 s
// all of it is covered by
//     eps_i = 2^-14 ||x_i|| max_c ||c|| + 2^-15 max_c ||c||^2 + 1e-36
// (the last term for pieces that underflow).
#include "common.cuh"
#include "internal.h"

namespace t2t {

constexpr int TA_ROWS = 128;                   // rows per tile: one thread each
constexpr int TA_CH = 128;                     // centroids per chunk
constexpr int TA_G = 16;                       // centroids per group
constexpr int TA_SA = TA_ROWS * 128;           // 16 KB: rows padded to 128 B
constexpr int TA_SB = TA_CH * 128;             // 16 KB per stage
constexpr int TA_SMEM = TA_SA + 2 * TA_SB + 128 + 1024;
constexpr int TA_THREADS = TA_ROWS;
constexpr int TA_FEW = 4;                      // this many rows with more than two groups in reach are settled one by one

__device__ __forceinline__ float ta_max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// Waits for the thread's outstanding TMEM loads and passes the loaded registers through, so that no use of them
// can be scheduled ahead of the wait.
__device__ __forceinline__ void tmem_wait_ld32(uint32_t (&v)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;\n"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                 "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]),
                 "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]), "+r"(v[21]), "+r"(v[22]), "+r"(v[23]),
                 "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]), "+r"(v[29])
               :
               : "memory");
  asm volatile("" : "+r"(v[30]), "+r"(v[31]) : : "memory");
}

// The three best groups of a row so far (m1 >= m2 >= m3, first centroid of the best two) and the values of the best.
struct Best {
  float m1, m2, m3;
  int i1, i2;
  float keep[TA_G];
};
__device__ __forceinline__ void best_push(Best& b, const uint32_t* v, int c0) {
  float x[TA_G];
#pragma unroll
  for (int e = 0; e < TA_G; ++e) x[e] = __uint_as_float(v[e]);
  const float gm = fmaxf(ta_max3(ta_max3(x[0], x[1], x[2]), ta_max3(x[3], x[4], x[5]), ta_max3(x[6], x[7], x[8])),
                         ta_max3(ta_max3(x[9], x[10], x[11]), ta_max3(x[12], x[13], x[14]), x[15]));
  b.m3 = fmaxf(b.m3, fminf(gm, b.m2));
  const bool up2 = gm > b.m2, up1 = gm > b.m1;
  if (__any_sync(0xffffffffu, up2)) {
    b.i2 = up1 ? b.i1 : (up2 ? c0 : b.i2);
    b.m2 = fmaxf(b.m2, fminf(gm, b.m1));
    if (__any_sync(0xffffffffu, up1)) {
      b.i1 = up1 ? c0 : b.i1;
      b.m1 = fmaxf(b.m1, gm);
#pragma unroll
      for (int e = 0; e < TA_G; ++e) b.keep[e] = up1 ? x[e] : b.keep[e];
    }
  }
}

// The defining chain d(x, c), c a row of 32 bf16 in global memory.
__device__ __forceinline__ float exact_distance(const float (&x)[kR], const __nv_bfloat16* __restrict__ c) {
  const uint4* cp = reinterpret_cast<const uint4*>(c);
  float cv[kR];
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    const uint4 w = cp[g];
    cv[8 * g + 0] = bf_lo(w.x); cv[8 * g + 1] = bf_hi(w.x);
    cv[8 * g + 2] = bf_lo(w.y); cv[8 * g + 3] = bf_hi(w.y);
    cv[8 * g + 4] = bf_lo(w.z); cv[8 * g + 5] = bf_hi(w.z);
    cv[8 * g + 6] = bf_lo(w.w); cv[8 * g + 7] = bf_hi(w.w);
  }
  float d = 0.f;
#pragma unroll
  for (int k = 0; k < kR; ++k) d = fmaf(cv[k], cv[k], d);
#pragma unroll
  for (int k = 0; k < kR; ++k) d = fmaf(x[k], -2.0f * cv[k], d);
  return d;
}
__device__ __forceinline__ void warp_argmin(float& best, int& bi) {
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) {
    const float ob = __shfl_xor_sync(0xffffffffu, best, m);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, m);
    if (ob < best || (ob == best && oi < bi)) { best = ob; bi = oi; }
  }
}

// One tile of 128 rows per CTA, four CTAs to an SM (128 TMEM columns each), each a chain of chunk -> norms -> product ->
// scan that the others fill.
//
// What bounds it: instruction issue and the chain.  The scan takes 13 instructions per 16 values plus the updates
// (three instructions a value in all); a CTA starts at the chunk its rows' own position points to, since warm-started
// centroids keep the order of the rows they came from, so updates get rare quickly.  The tensor pipe (three
// 128 x 128 x 16 steps a chunk, 192 cycles) is busy a sixth of the time.  Two tiles per CTA, sharing the centroids and
// their norms, waited longer at their barriers than they saved: 149 us for 5 x 75,600 rows and 2048 centroids against
// 141 (512 centroids: 58.5 against 56.8).
__global__ void __launch_bounds__(TA_THREADS, 4) assign_tc_kernel(const __nv_bfloat16* __restrict__ X,
                                                                  const __nv_bfloat16* __restrict__ cen,
                                                                  int* __restrict__ labels, int N, int Cn, int pin_begin,
                                                                  int pin_label, int* __restrict__ settled,
                                                                  int* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (base - smem_u32(smem_raw));
  constexpr int OFF_B = TA_SA;
  const uint32_t sA = base, sB = base + OFF_B;
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + OFF_B + 2 * TA_SB);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bar + 2);
  int* sCnMax = reinterpret_cast<int*>(bar + 3);
  int* sCount = reinterpret_cast<int*>(bar + 4);      // [2] rows to settle exactly: over two groups, over more

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h = blockIdx.y, row0 = blockIdx.x * TA_ROWS;
  const __nv_bfloat16* Xh = X + (size_t)h * N * kR;
  const __nv_bfloat16* ch = cen + (size_t)h * Cn * kR;

  if (warp == 0) {
    tmem_alloc(tmem_slot, 128);
    tmem_relinquish();
  }
  if (tid == 0) {
    *abort_flag = 0;
    *sCnMax = 0;
    sCount[0] = 0;
    sCount[1] = 0;
    mbar_init(bar, 1);
    mbar_init_fence();
  }
  const int lch = tid & 3, lr0 = tid >> 2;     // 4 chunks of 16 B per 64-byte row
  auto load_chunk = [&](int j, int st) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int r = lr0 + 32 * u;
      const bool valid = j * TA_CH + r < Cn;
      cp_async16(sB + st * TA_SB + sw128(r, lch), ch + (size_t)(valid ? j * TA_CH + r : 0) * kR + lch * 8, valid ? 16u : 0u);
    }
    cp_async_commit();
  };
  // the row tiles, with ones in elements 32..34 and zeros up to 47
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int r = lr0 + 32 * u;
    const bool valid = row0 + r < N;
    cp_async16(sA + sw128(r, lch), Xh + (size_t)(valid ? row0 + r : 0) * kR + lch * 8, valid ? 16u : 0u);
  }
  *reinterpret_cast<uint4*>(sm + sw128(tid, 4)) = make_uint4(0x3F803F80u, 0x00003F80u, 0u, 0u);
  *reinterpret_cast<uint4*>(sm + sw128(tid, 5)) = make_uint4(0u, 0u, 0u, 0u);
  for (int r = tid; r < 2 * TA_CH; r += TA_THREADS)
    *reinterpret_cast<uint4*>(sm + OFF_B + (r / TA_CH) * TA_SB + sw128(r % TA_CH, 5)) = make_uint4(0u, 0u, 0u, 0u);

  // -||c||^2 / 2 of the centroids of chunk j (stage st) as three bf16 pieces; -inf past the last centroid
  float cnmax = 0.f;
  auto augment = [&](int j, int st) {
    uint8_t* stage = sm + OFF_B + st * TA_SB;
    float s = 0.f;
#pragma unroll
    for (int q4 = 0; q4 < 4; ++q4) {
      const uint4 w = *reinterpret_cast<const uint4*>(stage + sw128(tid, q4));
      const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float lo = bf_lo(ws[e]), hi = bf_hi(ws[e]);
        s = fmaf(lo, lo, s);
        s = fmaf(hi, hi, s);
      }
    }
    const bool real = j * TA_CH + tid < Cn;
    // a NaN norm must reach the bound (every row is then settled exactly): compare bits, as atomicMax below does
    if (real && __float_as_int(s) > __float_as_int(cnmax)) cnmax = s;
    const float half = -0.5f * s;
    const uint32_t hi = real ? f_to_bf_bits(half) : 0xFF80u;
    const float r1 = half - __uint_as_float(hi << 16);
    const uint32_t mid = real ? f_to_bf_bits(r1) : 0u;
    const uint32_t lo = real ? f_to_bf_bits(r1 - __uint_as_float(mid << 16)) : 0u;
    *reinterpret_cast<uint4*>(stage + sw128(tid, 4)) = make_uint4(hi | (mid << 16), lo, 0u, 0u);
  };
  constexpr uint32_t idesc = make_idesc_bf16(128, TA_CH, false, false);
  auto issue = [&](int st, uint32_t tmem) {     // one warp (see elect_one)
    const uint32_t a0 = sdesc_lo(sA, 16), b0 = sdesc_lo(sB + st * TA_SB, 16);
    if (elect_one()) {
#pragma unroll
      for (int s2 = 0; s2 < 3; ++s2) umma_ss_lo(tmem, a0 + s2 * 2, b0 + s2 * 2, sdesc_hi(1024), idesc, s2 > 0 ? 1u : 0u);
      umma_commit(bar);
    }
    __syncwarp();
  };

  const int nch = cdiv(Cn, TA_CH);
  int j = (int)((long long)row0 * nch / N);      // first chunk; the others follow cyclically
  load_chunk(j, 0);
  cp_async_wait<0>();
  __syncthreads();
  augment(j, 0);
  int jn = j + 1 < nch ? j + 1 : 0;
  if (nch > 1) load_chunk(jn, 1);
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t t_lane = tmem_addr(tmem, warp * 32, 0);
  if (warp == 0) issue(0, tmem);

  Best b;
  b.m1 = b.m2 = b.m3 = -INFINITY;
  b.i1 = 0;
  b.i2 = -1;
#pragma unroll
  for (int e = 0; e < TA_G; ++e) b.keep[e] = -INFINITY;
  uint32_t ph = 0;
  bool dead = false;
  for (int i = 0; i < nch; ++i) {
    if (i + 1 < nch) {            // the next chunk is prepared while this one's product runs
      cp_async_wait<0>();
      __syncthreads();
      augment(jn, (i + 1) & 1);
      fence_proxy_async();
    }
    if (!mbar_wait_warp(bar, ph, abort_flag)) { dead = true; break; }
    ph ^= 1u;
    tc_fence_after();
    const int cbase = j * TA_CH;
    j = jn;
    jn = jn + 1 < nch ? jn + 1 : 0;
    if (i + 2 < nch) load_chunk(jn, i & 1);      // the product that read this stage has finished
    uint32_t va[32], vb[32];
    tmem_ld32(t_lane, va);
#pragma unroll
    for (int q = 0; q < 4; q += 2) {
      tmem_wait_ld32(va);
      tmem_ld32(t_lane + (q + 1) * 32, vb);
      best_push(b, va, cbase + q * 32);
      best_push(b, va + 16, cbase + q * 32 + 16);
      tmem_wait_ld32(vb);
      if (q == 0) tmem_ld32(t_lane + 64, va);
      best_push(b, vb, cbase + q * 32 + 32);
      best_push(b, vb + 16, cbase + q * 32 + 48);
    }
    tc_fence_before();
    __syncthreads();              // every row has read the scores, the next chunk's rows are complete
    if (warp == 0 && i + 1 < nch) {
      tc_fence_after();
      issue((i + 1) & 1, tmem);
    }
  }
  int* list = reinterpret_cast<int*>(sm + OFF_B);               // [2][TA_THREADS] rows to settle (the stages are free)
  int2* cand = reinterpret_cast<int2*>(sm + OFF_B + TA_SB);     // [TA_THREADS] first centroids of a row's two groups
  if (dead) {
    if (tid == 0 && status) atomicExch(status, ST_WAIT_TIMEOUT);
    cp_async_wait<0>();
  } else {
    if (cnmax != 0.f) atomicMax(sCnMax, __float_as_int(cnmax));
    __syncthreads();
    float xn = 0.f;               // ||x||^2 of this thread's row
#pragma unroll
    for (int q4 = 0; q4 < 4; ++q4) {
      const uint4 w = *reinterpret_cast<const uint4*>(sm + sw128(tid, q4));
      const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float lo = bf_lo(ws[e]), hi = bf_hi(ws[e]);
        xn = fmaf(lo, lo, xn);
        xn = fmaf(hi, hi, xn);
      }
    }
    const float cm = __int_as_float(*sCnMax);
    // 2 eps in units of d is eps in units of s = -d / 2
    const float eps = 6.103515625e-05f * sqrtf(xn) * sqrtf(cm) + 3.0517578125e-05f * cm + 1.0e-36f;
    float best = -INFINITY, second = b.m2;
    int bi = 0;
#pragma unroll
    for (int e = 0; e < TA_G; ++e) {
      second = fmaxf(second, fminf(best, b.keep[e]));
      if (b.keep[e] > best) { best = b.keep[e]; bi = e; }
    }
    const int row = row0 + tid;
    bool wide = false;            // more than two groups in reach
    if (row < N) {
      const bool pinned = pin_begin >= 0 && row >= pin_begin;
      labels[(size_t)h * N + row] = pinned ? pin_label : b.i1 + bi;
      if (!pinned && !(best - second > eps)) {             // true for NaN as well
        wide = !(b.m1 - b.m3 > eps);
        list[(wide ? TA_THREADS : 0) + atomicAdd(sCount + (wide ? 1 : 0), 1)] = tid;
        cand[tid] = make_int2(b.i1, b.i2);
      }
    }
    __syncthreads();
    if (settled && tid == 0 && sCount[0] + sCount[1] > 0) atomicAdd(settled, sCount[0] + sCount[1]);
    auto load_x = [&](int r, float (&x)[kR]) {
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const uint4 w = *reinterpret_cast<const uint4*>(sm + sw128(r, g));
        x[8 * g + 0] = bf_lo(w.x); x[8 * g + 1] = bf_hi(w.x);
        x[8 * g + 2] = bf_lo(w.y); x[8 * g + 3] = bf_hi(w.y);
        x[8 * g + 4] = bf_lo(w.z); x[8 * g + 5] = bf_hi(w.z);
        x[8 * g + 6] = bf_lo(w.w); x[8 * g + 7] = bf_hi(w.w);
      }
    };
    // a warp per row, a lane per centroid of its two best groups
    for (int e = warp; e < sCount[0]; e += TA_THREADS / 32) {
      const int r = list[e];
      const int2 two = cand[r];
      float x[kR];
      load_x(r, x);
      const int c = lane < TA_G ? two.x + lane : two.y + lane - TA_G;
      float d = INFINITY;
      int di = 0x7fffffff;
      if ((lane < TA_G || two.y >= 0) && c < Cn) {
        d = exact_distance(x, ch + (size_t)c * kR);
        di = c;
      }
      warp_argmin(d, di);
      if (lane == 0) labels[(size_t)h * N + row0 + r] = di;
    }
    // Rows with more than two groups in reach (many equal centroids, or values that are not finite): a few are settled one
    // after the other by the whole CTA, over all centroids (5.5 us each with 2048).
    float* wd = reinterpret_cast<float*>(sm + OFF_B + TA_SB + TA_THREADS * 8);      // [warps] distances, then indices
    int* wi = reinterpret_cast<int*>(wd + TA_THREADS / 32);
    for (int e = 0; sCount[1] <= TA_FEW && e < sCount[1]; ++e) {
      const int r = list[TA_THREADS + e];
      float x[kR];
      load_x(r, x);
      float d = INFINITY;
      int di = 0x7fffffff;
      for (int c = tid; c < Cn; c += TA_THREADS) {
        const float dc = exact_distance(x, ch + (size_t)c * kR);
        if (dc < d) { d = dc; di = c; }
      }
      warp_argmin(d, di);
      if (lane == 0) { wd[warp] = d; wi[warp] = di; }
      __syncthreads();
      if (tid == 0) {
        for (int w = 1; w < TA_THREADS / 32; ++w)
          if (wd[w] < d || (wd[w] == d && wi[w] < di)) { d = wd[w]; di = wi[w]; }
        labels[(size_t)h * N + row0 + r] = di == 0x7fffffff ? 0 : di;
      }
      __syncthreads();
    }
    // More of them - padding, constant frames: such rows sit together - go through the products once more, with the exact
    // chain for every centroid whose score is within eps of the row's best.  Of 32 centroids a warp first drops those
    // whose bits repeat a lower one's (that one ties and wins), then settles either one per step for each of its rows or
    // all of one row per step, whichever takes fewer steps.  Whole call, 1 head x 75,600 rows, 2048 centroids, a tenth of
    // the rows equal: 63 us (40 with none equal; 800 when every such row was settled by itself).
    if (sCount[1] > TA_FEW) {
      __syncthreads();                                      // the stages are free again
      const float cut = b.m1 - eps;
#pragma unroll
      for (int st = 0; st < 2; ++st)
        *reinterpret_cast<uint4*>(sm + OFF_B + st * TA_SB + sw128(tid, 5)) = make_uint4(0u, 0u, 0u, 0u);
      float d = INFINITY;
      int di = 0x7fffffff, seen = -1;      // seen: a centroid that was settled, copies of which come up most often
#pragma unroll 1
      for (int i = 0; i < nch; ++i) {
        const int st = i & 1;                               // a warp may still read the chunk before
        const uint8_t* stage = sm + OFF_B + st * TA_SB;
        load_chunk(i, st);
        cp_async_wait<0>();
        __syncthreads();
        augment(i, st);
        fence_proxy_async();
        tc_fence_before();
        __syncthreads();
        if (warp == 0) {
          tc_fence_after();
          issue(st, tmem);
        }
        if (!mbar_wait_warp(bar, ph, abort_flag)) {
          if (tid == 0 && status) atomicExch(status, ST_WAIT_TIMEOUT);
          break;
        }
        ph ^= 1u;
        tc_fence_after();
#pragma unroll 1
        for (int q = 0; q < 4; ++q) {
          uint32_t v[32], near = 0u;
          tmem_ld32(t_lane + q * 32, v);
          tmem_wait_ld32(v);
#pragma unroll
          for (int e = 0; e < 32; ++e)
            if (!(__uint_as_float(v[e]) < cut)) near |= 1u << e;      // NaN as well
          if (!wide) near = 0u;
          const int c0 = i * TA_CH + q * 32;
          if (c0 + 32 > Cn) near &= c0 < Cn ? (1u << (Cn - c0)) - 1u : 0u;
          if (!__any_sync(0xffffffffu, near != 0u)) continue;
          {
            uint32_t mine[16], hash = 0u;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              const uint4 w = *reinterpret_cast<const uint4*>(stage + sw128(q * 32 + lane, g));
              mine[4 * g] = w.x; mine[4 * g + 1] = w.y; mine[4 * g + 2] = w.z; mine[4 * g + 3] = w.w;
            }
#pragma unroll
            for (int k = 0; k < 16; ++k) hash = hash * 0x9E3779B1u + mine[k];
            const int first = __ffs(__match_any_sync(0xffffffffu, hash)) - 1;
            const uint4* old = reinterpret_cast<const uint4*>(ch + (size_t)max(seen, 0) * kR);
            bool copy = first < lane, again = seen >= 0;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              const uint4 w = *reinterpret_cast<const uint4*>(stage + sw128(q * 32 + first, g)), o = old[g];
              copy = copy && mine[4 * g] == w.x && mine[4 * g + 1] == w.y && mine[4 * g + 2] == w.z && mine[4 * g + 3] == w.w;
              again = again && mine[4 * g] == o.x && mine[4 * g + 1] == o.y && mine[4 * g + 2] == o.z && mine[4 * g + 3] == o.w;
            }
            near &= ~__ballot_sync(0xffffffffu, copy || again);
          }
          unsigned rows = __ballot_sync(0xffffffffu, near != 0u);
          if (rows) seen = c0 + __ffs(__reduce_or_sync(0xffffffffu, near)) - 1;
          float x[kR];
          if (__popc(rows) > (int)__reduce_max_sync(0xffffffffu, __popc(near))) {
            load_x(tid, x);
            for (; near; near &= near - 1u) {
              const int c = c0 + __ffs(near) - 1;
              const float dc = exact_distance(x, ch + (size_t)c * kR);
              if (dc < d) { d = dc; di = c; }
            }
            __syncwarp();
          } else {
            for (; rows; rows &= rows - 1u) {
              const int src = __ffs(rows) - 1;
              load_x(warp * 32 + src, x);
              const bool mine = (__shfl_sync(0xffffffffu, near, src) >> lane) & 1u;
              float dc = mine ? exact_distance(x, ch + (size_t)(c0 + lane) * kR) : INFINITY;
              int dj = c0 + lane;
              if (!(dc < INFINITY)) { dc = INFINITY; dj = 0x7fffffff; }      // NaN as well
              warp_argmin(dc, dj);
              if (lane == src && dc < d) { d = dc; di = dj; }
            }
          }
        }
      }
      if (wide) labels[(size_t)h * N + row] = di == 0x7fffffff ? 0 : di;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 128);
}

size_t assign_ws_bytes(int, int) { return sizeof(int); }      // the count of settled rows

int launch_assign(const __nv_bfloat16* X, const __nv_bfloat16* cen, int* labels, int H, int N, int Cn,
                  int pin_begin, int pin_label, int* settled, int* d_status, cudaStream_t st) {
  if (settled && cudaMemsetAsync(settled, 0, sizeof(int), st) != cudaSuccess) return T2T_ERR_CUDA;
  if (cudaFuncSetAttribute(assign_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TA_SMEM) != cudaSuccess)
    return T2T_ERR_CUDA;
  assign_tc_kernel<<<dim3(cdiv(N, TA_ROWS), H), TA_THREADS, TA_SMEM, st>>>(X, cen, labels, N, Cn, pin_begin, pin_label,
                                                                           settled, d_status);
  return cudaGetLastError() == cudaSuccess ? T2T_OK : T2T_ERR_CUDA;
}

}  // namespace t2t
