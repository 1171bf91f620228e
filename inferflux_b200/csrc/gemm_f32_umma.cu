// float32 matrix product C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]) on the tcgen05 tensor cores, for matrices that are not small.
//
// The tensor cores have no float32 operands.  A float32 number is the exact sum of three bfloat16 numbers, each the one nearest to
// what the ones before it leave (the exponent ranges are the same), and the product of two such numbers is exact in float32.  Of the
// nine products of parts the six largest are taken; the second part is at most 2^-8 of the number and the third 2^-17, so the three others together
// are at most 2^-24 of the product, of either sign.  (Parts cut off instead of rounded leave out up to 2^-21, always towards
// zero.)  The tensor core rounds its running sum towards zero at each step of 16 along K, which over a long K would cost
// more than plain float32 sums do.  So it sums 64 along K at a time, the small products first, and CUDA cores add these sums
// up in registers, in order and rounded to nearest.  Error against 64 bits (2-norm over 2-norm, normal operands; in brackets the
// fused multiply-adds in index order that gemm_f32.cu makes): K 256 0.9e-7 (2.9e-7), N 2,560 K 2,048 1.0e-7 (2.9e-7), N 22,016
// K 2,048 1.1e-7 (8.1e-7), N 2,048 K 11,008 1.3e-7 (6.7e-7), N 3,584 K 18,944 1.5e-7 (8.7e-7).
//
// How an output element is summed depends on N and K alone, as in gemm_f32.cu: K is cut into umma_slices(N, K) slices, a slice
// into steps of 64, and the slices' sums are added two by two, then the pairs in order, whatever M is, whichever tile width runs and
// whether a block makes one slice or two, so a row's result does not depend on what else is in
// the batch.  A slice's sum that is not finite (an operand was not, or a sum overflowed on the way), and one below 2^-64 that is not
// zero (operands so small that bfloat16 does not reach to their last bits), is made again by fused multiply-adds in index
// order.  So infinities and NaN are what these give (a sum that they would take beyond the range on the way and the tensor cores do
// not stays as it is), and for sums of 2^-64 and more what small operands lose, 2^-134 of the other operand a product, is below
// float32's rounding unless that other operand is beyond 2^32.
//
// A block takes 128 rows of W, the tile's M rows of the MMA, and tile_n tokens, its N columns.  W arrives as float32 by TMA
// (128-byte swizzle, K 64 a stage); a worker thread reads its part of a row's 64 values, cuts them up by conversions and
// subtractions (exact) and writes the three parts into tensor memory, where the MMA takes its A operand from: the parts never go
// back to shared memory, whose bandwidth the MMA's B operand (the tokens' three parts) needs.  Up to 64 tokens the same
// threads cut the tokens' values up as well (a warp of its own for them is ahead with one row and behind with eight); for more,
// split_kernel has done it once for all blocks and TMA brings the parts.
// Parts and sums are double-buffered: while the MMAs of one step run, the threads add the sums of the step before it and
// cut up the values of the step behind it.
//
// What bounds it: six MMAs a product, so 2,250 / 6 = 375 TFLOP/s at most; with few tokens the workers, of whose step (0.7 us alone on an
// SM, 1.2 beside another block) the MMAs fill a quarter, and reading W.  Us here (by multiply-adds), 301 rows: N 22,016 K 2,048 142
// (623), N 2,048 K 11,008 94 (373), N 2,560 K 2,048 40 (94); 64 rows 71 (251), 42 (182), 14 (50); 16 rows 41 (111), 28 (76), 8.6 (16.5); 8 rows 40
// (72), 27 (50), 8.4 (11.5); 4 rows 39 (46), 27 (33), 7.7 (9.7); 2 rows 39 (46), 27 (32), 7.5 (9.5); 1 row 39 (39), 26.5 (27), 7.2 (7.2), N 151,936
// K 2,048 205 (214).  Behind multiply-adds is one row of a square matrix of up to 2,048, whose blocks have few steps: 2,048 6.8 us (6.2), 1,024
// 5.7 (4.5), 512 5.3 (4.1), 256 4.2 (3.2); it stays here for the sake of its bits, which are those of every batch.  A decode step of one
// request (4 layers of the 3B sizes and the vocabulary) takes 827 us (876).
#include "gemm_f32_umma.h"
#include "umma.cuh"

namespace {

constexpr int FK64 = 64;                        // K per step
constexpr int W_STAGE = 128 * FK64 * 4;         // 32 KB: two boxes of 128 rows x 32 floats
constexpr int U_MAX_SLICES = 8;                  // of K: the largest portable cluster
constexpr int U_PARTS = 2;                       // into so many K and the columns are dealt out to the workers, four warps each
// the workers, and a warp each for W's copies, the MMAs and the tokens' copies
constexpr int U_THREADS = 128 * U_PARTS + 96;
constexpr unsigned U_IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 4) << 24);   // D float32, A and B bfloat16, K-major, M 128; N (in eighths) at bit 17

__host__ __device__ constexpr int u_w_stages(int tn) { return tn == 16 ? 3 : tn <= 64 ? 5 : tn <= 128 ? 4 : 3; }
__host__ __device__ constexpr int u_smem(int tn) { return u_w_stages(tn) * W_STAGE + 2 * 3 * tn * 128 + 1024; }
__host__ __device__ constexpr int u_columns(int tn) { return tn <= 32 ? 256 : 512; }     // of tensor memory: 2 x 3 x 32 for W's parts, 2 x tn for sums

__device__ __forceinline__ unsigned u_cluster_rank() { unsigned r; asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r)); return r; }
__device__ __forceinline__ void u_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ float4 u_read_peer4(unsigned saddr, int rank) {
  unsigned ra;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(saddr), "r"(rank));
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(ra) : "memory");
  return v;
}
// True for one lane of the warp, chosen in a way that the compiler knows to be one.  An MMA issued behind it takes the tensor core's time, 21
// cycles with 16 columns, 39 with 64, 80 with 160; behind lane == 0 it takes at least 61 (measured with one block).
__device__ __forceinline__ bool u_elect() {
  unsigned r;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(r));
  return r != 0;
}
// one arrival for the warp, once all its lanes have come here
__device__ __forceinline__ void u_arrive_warp(unsigned bar, int lane) {
  __syncwarp();
  if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}

// Takes two packed parts off two floats.
__device__ __forceinline__ void take_off(float& x0, float& x1, unsigned part) {
  asm("{\n .reg .b64 a, b;\n mov.b64 a, {%0, %1};\n mov.b64 b, {%2, %3};\n sub.rn.f32x2 a, a, b;\n mov.b64 {%0, %1}, a;\n}\n"
      : "+f"(x0), "+f"(x1) : "r"(part << 16), "r"(part & 0xFFFF0000u));
}
// Two floats into their three bfloat16 parts each, packed (the first in the low half): x = hi + mid + lo exactly, each part what
// the parts before it leave, rounded to nearest (hi to the largest finite one at most).  Below 2^-110 lo's last bits are below
// bfloat16's least number.  Infinities and NaN leave a NaN in lo.
__device__ __forceinline__ void cut(float x0, float x1, unsigned& hi, unsigned& mid, unsigned& lo) {
  asm("cvt.rn.satfinite.bf16x2.f32 %0, %1, %2;\n" : "=r"(hi) : "f"(x1), "f"(x0));
  take_off(x0, x1, hi);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(mid) : "f"(x1), "f"(x0));
  take_off(x0, x1, mid);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(lo) : "f"(x1), "f"(x0));
}

__device__ __forceinline__ void u_tmem_st8(unsigned taddr, const unsigned (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void u_tmem_ld8(unsigned taddr, unsigned (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}
__device__ __forceinline__ void u_mma(unsigned d, unsigned a_tmem, unsigned long long db, unsigned idesc, unsigned accumulate) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
               ::"r"(d), "r"(a_tmem), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void u_commit(unsigned bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}

constexpr unsigned U_SMALL = 0x1F800000u;        // 2^-64
// A sum that is to be made again: not finite, or below 2^-64 and not zero.
__device__ __forceinline__ bool odd_sum(float v) {
  const unsigned u = __float_as_uint(v) & 0x7FFFFFFFu;
  return u >= 0x7F800000u || (u < U_SMALL && u != 0);
}
// Makes the odd ones among sums [BOTH][TN][128] again, of slices slice_len long from k_begin on, called by all workers: the tokens that
// have any 16 a part at a time, W and the tokens through the shared memory behind the sums, the next 32 along K on their way
// meanwhile.  In a function of its own and with the sums in memory it leaves the kernel's registers alone (inlined it cost up to 7 %).
// (One NaN among 301 rows, N 22,016 K 2,048: 325 us where the product alone takes 142; in every row 1,750; 1 row 170 and 39.  A
// thread a sum by itself took 2,600, 55,800 and 1,780.)
template <int TN, int BOTH>
__device__ __noinline__ void sums_again(float* sums, unsigned* odd_tokens, const float* __restrict__ A, const float* __restrict__ W, long long lda,
                                        int M, int N, int K, int m0, int n0, int tile_n, int k_begin, int slice_len, int k_last) {
  constexpr int PARTS = U_PARTS, THREADS = 128 * PARTS, COLS = TN / PARTS, PITCH = 36;   // 36: 16-byte reads of eight rows meet no bank twice
  constexpr int W_EACH = 128 * 8 / THREADS, G = COLS < 16 ? COLS : 16;
  float *ws = sums + BOTH * TN * 128, *xs = ws + 128 * PITCH;          // [128][PITCH], [16 * PARTS][32]
  const int tid = threadIdx.x, row = tid & 127, part = tid >> 7, kc = (tid & 7) * 4;
#pragma unroll 1
  for (int h = 0; h < BOTH; ++h, sums += TN * 128) {
    const int k_first = min(k_last, k_begin + h * slice_len), k_end = min(k_last, k_first + slice_len);
    for (int i = 0; i < COLS; ++i) {
      const int t = part * COLS + i;
      if (odd_sum(sums[t * 128 + row]) && t < tile_n && m0 + t < M && n0 + row < N) atomicOr(&odd_tokens[t >> 5], 1u << (t & 31));
    }
    asm volatile("bar.sync 1, %0;\n" ::"n"(THREADS) : "memory");
#pragma unroll 1
    for (int g = 0; g < COLS / G; ++g) {
      auto flags = [&](int p) { const int t = p * COLS + g * G; return odd_tokens[t >> 5] >> (t & 31) & ((1u << G) - 1); };
      if (!(flags(0) | flags(PARTS - 1))) continue;                      // (the same for all workers)
      const unsigned mine = flags(part);
      const int at = tid >> 3, xt = (at / G) * COLS + g * G + (at % G);   // of the tokens' copies
      float4 wv[W_EACH], xv;
      auto load = [&](int k0) {
        const int k = k0 + kc;                                           // K is a multiple of 4
#pragma unroll
        for (int i = 0; i < W_EACH; ++i) {
          const int r = at + i * (THREADS / 8);
          wv[i] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (n0 + r < N && k < k_end) wv[i] = *reinterpret_cast<const float4*>(W + (size_t)(n0 + r) * K + k);
        }
        xv = make_float4(0.f, 0.f, 0.f, 0.f);
        if (at < G * PARTS && xt < tile_n && m0 + xt < M && k < k_end) {
          const float* p = A + (size_t)(m0 + xt) * lda + k;
          xv = make_float4(p[0], p[1], p[2], p[3]);
        }
      };
      float r[G];
#pragma unroll
      for (int i = 0; i < G; ++i) r[i] = 0.0f;
      load(k_first);
#pragma unroll 1
      for (int k0 = k_first; k0 < k_end; k0 += 32) {
        asm volatile("bar.sync 1, %0;\n" ::"n"(THREADS) : "memory");
#pragma unroll
        for (int i = 0; i < W_EACH; ++i) *reinterpret_cast<float4*>(ws + (at + i * (THREADS / 8)) * PITCH + kc) = wv[i];
        *reinterpret_cast<float4*>(xs + at * 32 + kc) = xv;
        asm volatile("bar.sync 1, %0;\n" ::"n"(THREADS) : "memory");
        load(k0 + 32);
#pragma unroll 2
        for (int c = 0; c < 32; c += 4) {
          const float4 w = *reinterpret_cast<const float4*>(ws + row * PITCH + c);
#pragma unroll
          for (int i = 0; i < G; ++i)
            if (mine >> i & 1) {
              const float4 x = *reinterpret_cast<const float4*>(xs + (part * G + i) * 32 + c);
              r[i] = fmaf(x.w, w.w, fmaf(x.z, w.z, fmaf(x.y, w.y, fmaf(x.x, w.x, r[i]))));
            }
        }
      }
#pragma unroll
      for (int i = 0; i < G; ++i) {
        float& v = sums[(part * COLS + g * G + i) * 128 + row];
        if (mine >> i & 1 && odd_sum(v)) v = r[i];
      }
    }
    asm volatile("bar.sync 1, %0;\n" ::"n"(THREADS) : "memory");      // all have read the flags before the next slice sets some
  }
}

// TN: token columns a block can hold.  BOTH: slices of K that it makes.  Grid: (tiles of tile_n tokens, tiles of 128 rows of W,
// slices of K / BOTH), the blocks of a tile a cluster.  Up to TN 64 A is read here; above, map_x describes split_kernel's parts [3][M][K].
template <int TN, int BOTH>
__global__ void __launch_bounds__(U_THREADS, TN == 16 ? 2 : 1)
gemm_f32_umma_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const float* __restrict__ A,
                     const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ C, int M, int N, int K, long long lda,
                     long long ldc, int tile_n, int slice_steps, int vec_a, int w_fixed, int* __restrict__ error_flag) {
  constexpr bool OWN_X = TN <= 64;
  constexpr int STAGES = u_w_stages(TN), PARTS = U_PARTS, WARPS = 4 * PARTS, COLS = TN / PARTS, UNITS = 16 / PARTS;   // a worker's columns, and float4 of W
  constexpr int X_ROWS = 2 * WARPS, X_PER = OWN_X && TN > X_ROWS ? TN / X_ROWS : 1;                                          // and float4 of the tokens
  extern __shared__ unsigned char u_smem_raw[];
  __shared__ __align__(8) unsigned long long bars[2 * STAGES + 6];   // w_full[s], w_empty[s], x_full[2], parts_full[2], mma_done[2]
  __shared__ unsigned tmem_slot;
  __shared__ int abort_s;
  __shared__ unsigned odd_tokens[(TN + 31) / 32];                      // tokens with sums that are to be made again
  const unsigned sbase = (g_smem_addr(u_smem_raw) + 1023u) & ~1023u, sx = sbase + STAGES * W_STAGE;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;   // (shuffled: known to be uniform)
  const unsigned w_full = g_smem_addr(&bars[0]), w_empty = g_smem_addr(&bars[STAGES]), x_full = g_smem_addr(&bars[2 * STAGES]);
  const unsigned parts_full = x_full + 16, mma_done = x_full + 32;
  volatile int* abort_flag = &abort_s;
  const int m0 = blockIdx.x * tile_n, n0 = blockIdx.y * 128;
  const int steps_all = (K + FK64 - 1) / FK64, step0 = min(steps_all, (int)blockIdx.z * BOTH * slice_steps);
  const int steps = min(steps_all, step0 + BOTH * slice_steps) - step0;
  auto copy_w = [&](int c) {
    const int st = c % STAGES;
    g_expect_tx(w_full + 8 * st, W_STAGE);
#pragma unroll
    for (int h = 0; h < 2; ++h)
      asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n"
                   ::"r"(sbase + st * W_STAGE + h * (W_STAGE / 2)), "l"(&map_w), "r"((step0 + c) * FK64 + 32 * h), "r"(n0), "r"(w_full + 8 * st) : "memory");
  };
  if (tid == 32 * WARPS) {
    abort_s = 0;
    for (int i = 0; i < (TN + 31) / 32; ++i) odd_tokens[i] = 0;
    for (int s = 0; s < STAGES; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(w_full + 8 * s));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(w_empty + 8 * s), "r"(WARPS));
    }
    for (int b = 0; b < 2; ++b) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(x_full + 8 * b));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(parts_full + 8 * b), "r"(WARPS));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(mma_done + 8 * b));
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    if (w_fixed)                                                       // the first tiles of W come while the others set up
      for (int c = 0; c < min(steps, STAGES); ++c) copy_w(c);
  }
  if (warp == WARPS + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(g_smem_addr(&tmem_slot)), "n"(u_columns(TN)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  pdl_launch_dependents();                       // behind the allocation: no block of the next kernel can be ahead of it at the tensor memory
  const unsigned tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);
  bool gave_up = false;
  float acc[COLS], first[BOTH == 2 ? COLS : 1];                        // first: of two slices
#pragma unroll
  for (int i = 0; i < COLS; ++i) acc[i] = 0.0f;
  if constexpr (BOTH == 2) {
#pragma unroll
    for (int i = 0; i < COLS; ++i) first[i] = 0.0f;
  }
  const int quarter = warp & 3, part = warp >> 2;                      // of a worker: its lanes of tensor memory, its part of K and of the columns

  if (warp == WARPS) {                                                    // W's copies
    if (lane == 0) {
      if (!w_fixed) pdl_wait();
      for (int c = w_fixed ? STAGES : 0; c < steps; ++c) {
        if (c == STAGES) pdl_wait();                                   // (bounded waits begin when the kernel ahead has finished)
        if (c >= STAGES && !g_wait(w_empty + 8 * (c % STAGES), (unsigned)((c / STAGES - 1) & 1), abort_flag)) { gave_up = true; break; }
        copy_w(c);
      }
    }
  } else if (warp == WARPS + 2) {                                             // the tokens' copies
    if (!OWN_X && lane == 0) {
      pdl_wait();
      for (int c = 0; c < steps; ++c) {
        const int b = c & 1;
        if (c >= 2 && !g_wait(mma_done + 8 * b, (unsigned)((c / 2 - 1) & 1), abort_flag)) { gave_up = true; break; }
        g_expect_tx(x_full + 8 * b, 3 * tile_n * 128);
        asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n"
                     ::"r"(sx + b * 3 * TN * 128), "l"(&map_x), "r"((step0 + c) * FK64), "r"(m0), "r"(0), "r"(x_full + 8 * b) : "memory");
      }
    }
  } else if (warp == WARPS + 1) {                                             // the MMAs
    if (u_elect()) {
      pdl_wait();
      const unsigned idesc = U_IDESC | ((unsigned)(tile_n >> 3) << 17);
      for (int c = 0; c < steps; ++c) {
        const int b = c & 1;
        const unsigned par = (unsigned)((c >> 1) & 1);
        if (!g_wait(parts_full + 8 * b, par, abort_flag)) { gave_up = true; break; }
        if (!OWN_X && !g_wait(x_full + 8 * b, par, abort_flag)) { gave_up = true; break; }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        const unsigned d = tmem + 192 + b * TN, wp = tmem + b * 96;
        const unsigned long long xd0 = g_desc(sx + b * 3 * TN * 128), xd[3] = {xd0, xd0 + (unsigned)(tile_n * 8), xd0 + (unsigned)(tile_n * 16)};
        // (W's part, the tokens' part), 0 the highest: the small products first
        constexpr int order[6][2] = {{2, 0}, {1, 1}, {0, 2}, {1, 0}, {0, 1}, {0, 0}};
#pragma unroll
        for (int p = 0; p < 6; ++p)
#pragma unroll
          for (int k = 0; k < 4; ++k)                                  // (a descriptor's address counts 16 bytes)
            u_mma(d, wp + order[p][0] * 32 + k * 8, xd[order[p][1]] + k * 2, idesc, (p | k) != 0);
        u_commit(mma_done + 8 * b);
      }
    }
  } else {
    const unsigned lanes = tmem + ((unsigned)(quarter * 32) << 16);
    const int row = quarter * 32 + lane;
    auto add_sums = [&](int c) {                                       // step c's sums into the registers
      if (!__all_sync(0xffffffffu, g_wait(mma_done + 8 * (c & 1), (unsigned)((c >> 1) & 1), abort_flag))) return false;
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
      for (int i = 0; i < COLS / 8; ++i) {
        if (part * COLS + i * 8 >= tile_n) break;                      // (the same for the warp)
        const unsigned at = lanes + 192 + (c & 1) * TN + part * COLS + i * 8;
        unsigned r[8];
        u_tmem_ld8(at, r);
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i * 8 + j] += __uint_as_float(r[j]);
      }
      if constexpr (BOTH == 2)
        if (c == slice_steps - 1) {
#pragma unroll
          for (int i = 0; i < COLS; ++i) { first[i] = acc[i]; acc[i] = 0.0f; }
        }
      return true;
    };
    float4 xr[X_PER];                                                  // the tokens' values of the step ahead: 16 threads a row, four values each
    auto load_x = [&](int c) {
      const int k = (step0 + c) * FK64 + (tid & 15) * 4;
#pragma unroll
      for (int i = 0; i < X_PER; ++i) {
        const int t = (tid >> 4) + X_ROWS * i, m = m0 + t;
        xr[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < tile_n && m < M && k < K && c < steps) {               // K is a multiple of 4
          const float* p = A + (size_t)m * lda + k;
          xr[i] = vec_a ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
        }
      }
    };
    if (OWN_X) { pdl_wait(); load_x(0); }
    else if (!w_fixed) pdl_wait();                                     // (W's copies wait, too)
    for (int c = 0; c < steps; ++c) {
      const int b = c & 1, st = c % STAGES;
      if (!OWN_X && c == 2) pdl_wait();
      bool ok = c < 2 || add_sums(c - 2);                              // (and its parts' places are free)
      ok = ok && g_wait(w_full + 8 * st, (unsigned)((c / STAGES) & 1), abort_flag);
      if (!__all_sync(0xffffffffu, ok)) { gave_up = true; break; }
      const unsigned wrow = sbase + st * W_STAGE + row * 128;
#pragma unroll
      for (int g = 0; g < UNITS / 4; ++g) {                            // 16 values at a time
        unsigned hi[8], mid[8], lo[8];
        const int u = part * UNITS + g * 4;                            // among the row's 16 units of 16 bytes, eight in each box
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float x, y, z, w;
          asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(x), "=f"(y), "=f"(z), "=f"(w)
                       : "r"(wrow + (u >> 3) * (W_STAGE / 2) + ((((u & 7) + j) ^ (row & 7)) << 4)) : "memory");
          cut(x, y, hi[2 * j], mid[2 * j], lo[2 * j]);
          cut(z, w, hi[2 * j + 1], mid[2 * j + 1], lo[2 * j + 1]);
        }
        const unsigned at = lanes + b * 96 + u * 2;
        u_tmem_st8(at, hi);
        u_tmem_st8(at + 32, mid);
        u_tmem_st8(at + 64, lo);
      }
      u_arrive_warp(w_empty + 8 * st, lane);
      if (OWN_X) {
#pragma unroll
        for (int i = 0; i < X_PER; ++i) {
          const int t = (tid >> 4) + X_ROWS * i, q = tid & 15;
          if (t >= tile_n) break;
          unsigned h0, m0_, l0, h1, m1, l1;
          cut(xr[i].x, xr[i].y, h0, m0_, l0);
          cut(xr[i].z, xr[i].w, h1, m1, l1);
          const unsigned to = sx + b * 3 * TN * 128 + t * 128 + (((q >> 1) ^ (t & 7)) << 4) + (q & 1) * 8;
          asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(to), "r"(h0), "r"(h1) : "memory");
          asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(to + tile_n * 128), "r"(m0_), "r"(m1) : "memory");
          asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(to + 2 * tile_n * 128), "r"(l0), "r"(l1) : "memory");
        }
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        load_x(c + 1);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      u_arrive_warp(parts_full + 8 * b, lane);
    }
    if (steps <= 2) pdl_wait();
    for (int c = steps < 2 ? 0 : steps - 2; c < steps && !gave_up; ++c) gave_up = !add_sums(c);
  }
  if (gave_up) {                                                       // a wait ran out: tell everyone, let copies in flight land
    atomicExch(error_flag, IFX_DEVICE_ERR_WAIT);
    abort_s = 1;
    __nanosleep(2000000);
  }
  // Every MMA has been waited for, every copy has landed: the ring's memory can take the slices' sums.
  // Whether there are sums to be made again, three instructions a sum: zero times it is not zero, or the least of the numbers that
  // are not zero (zeros come out largest) is below 2^-64.
  float zero = 0.0f;
  unsigned least = 0xFFFFFFFFu;
#pragma unroll
  for (int i = 0; i < COLS; ++i) {
    zero = fmaf(acc[i], 0.0f, zero);
    least = min(least, 2u * __float_as_uint(acc[i]) - 1u);
    if constexpr (BOTH == 2) {
      zero = fmaf(first[i], 0.0f, zero);
      least = min(least, 2u * __float_as_uint(first[i]) - 1u);
    }
  }
  if (__syncthreads_or(!(zero == 0.0f) || least < 2u * U_SMALL - 1u) && !*abort_flag && warp < WARPS) {
    float* sums = reinterpret_cast<float*>(u_smem_raw + (sbase - g_smem_addr(u_smem_raw)));
    float* own = sums + part * COLS * 128 + (tid & 127);
    // (where K ends in the first of two slices its sums are in acc)
    const int at = BOTH == 2 && steps >= slice_steps ? TN * 128 : 0;
#pragma unroll
    for (int i = 0; i < COLS; ++i) {
      if constexpr (BOTH == 2) own[TN * 128 - at + i * 128] = first[i];
      own[at + i * 128] = acc[i];
    }
    sums_again<TN, BOTH>(sums, odd_tokens, A, W, lda, M, N, K, m0, n0, tile_n, step0 * FK64, slice_steps * FK64, min(K, (step0 + steps) * FK64));
#pragma unroll
    for (int i = 0; i < COLS; ++i) {
      if constexpr (BOTH == 2) first[i] = own[TN * 128 - at + i * 128];
      acc[i] = own[at + i * 128];
    }
  }
  if constexpr (BOTH == 2) {
#pragma unroll
    for (int i = 0; i < COLS; ++i) acc[i] += first[i];
  }
  const int slices = gridDim.z;
  auto put = [&](int m, int n, float v) { C[(size_t)m * ldc + n] = v + (bias ? bias[n] : 0.0f); };
  if (slices == 1) {
    if (warp < WARPS) {
      const int n = n0 + quarter * 32 + lane;
      if (n < N)
#pragma unroll
        for (int i = 0; i < COLS; ++i) {
          const int t = part * COLS + i;
          if (t < tile_n && m0 + t < M) put(m0 + t, n, acc[i]);
        }
    }
  } else {
    __syncthreads();
    if (warp < WARPS) {
#pragma unroll
      for (int i = 0; i < COLS; ++i) {
        const int t = part * COLS + i;
        if (t < tile_n) asm volatile("st.shared.f32 [%0], %1;" ::"r"(sbase + (t * 128 + quarter * 32 + lane) * 4), "f"(acc[i]) : "memory");
      }
    }
    u_cluster_sync();
    const int rank = (int)u_cluster_rank();
    if (warp < WARPS) {                                                // a warp a token's 128 sums, all slices asked for together
      const int n = n0 + 4 * lane;
      for (int t = rank * WARPS + warp; t < tile_n && m0 + t < M; t += WARPS * slices) {
        float4 v[U_MAX_SLICES];
#pragma unroll
        for (int z = 0; z < U_MAX_SLICES; ++z)
          if (z < slices) v[z] = u_read_peer4(sbase + (t * 128 + 4 * lane) * 4, z);
        auto add = [](float4& a, const float4& b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; };
        float4 o = v[0];                                               // two by two, then the pairs in order
        if constexpr (BOTH == 2) {
#pragma unroll
          for (int z = 1; z < U_MAX_SLICES; ++z)
            if (z < slices) add(o, v[z]);
        } else {
          add(o, v[1]);
#pragma unroll
          for (int z = 2; z < U_MAX_SLICES; z += 2)
            if (z < slices) { add(v[z], v[z + 1]); add(o, v[z]); }
        }
        if (n < N) put(m0 + t, n, o.x);
        if (n + 1 < N) put(m0 + t, n + 1, o.y);
        if (n + 2 < N) put(m0 + t, n + 2, o.z);
        if (n + 3 < N) put(m0 + t, n + 3, o.w);
      }
    }
    u_cluster_sync();                                                  // no block leaves while another still reads its sums
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == WARPS + 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "n"(u_columns(TN)) : "memory");
}

// A's values cut into their parts [3][M][pitch] (zeros behind K), eight a thread.
__global__ void __launch_bounds__(256)
split_kernel(const float* __restrict__ A, uint4* __restrict__ parts, int M, int K, long long lda, int pitch, int vec_a) {
  pdl_enter();
  const int groups = pitch / 8;
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= (long long)M * groups) return;
  const int m = (int)(i / groups), k = (int)(i % groups) * 8;
  const float* p = A + (size_t)m * lda + k;
  float4 v[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    v[h] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (k + 4 * h < K) v[h] = vec_a ? *reinterpret_cast<const float4*>(p + 4 * h) : make_float4(p[4 * h], p[4 * h + 1], p[4 * h + 2], p[4 * h + 3]);
  }
  uint4 o[3];
  cut(v[0].x, v[0].y, o[0].x, o[1].x, o[2].x);
  cut(v[0].z, v[0].w, o[0].y, o[1].y, o[2].y);
  cut(v[1].x, v[1].y, o[0].z, o[1].z, o[2].z);
  cut(v[1].z, v[1].w, o[0].w, o[1].w, o[2].w);
#pragma unroll
  for (int q = 0; q < 3; ++q) parts[(long long)q * M * groups + i] = o[q];
}

// Slices of K, from N and K alone (1, 2, 4 or 8), each at least 256 long: blocks enough that their last round is a small part of all.
// (Shorter ones would be ahead for one row of a small matrix, 1,024 x 1,024 in 8 instead of 4 4.3 us instead of 5.6, and behind for
// many, 2,048 rows 74 instead of 50.)
int umma_slices(int N, int K) {
  const int rows = (N + 127) / 128;
  int s = 1;
  while (s < U_MAX_SLICES && rows * s < 256 && K / (2 * s) >= 256) s *= 2;
  return s;
}

constexpr int U_TWO_TOKENS = 96;                 // tokens up to which a block can take two slices: it needs registers for two sums of each
struct TokenTiles { int tn, count, both; };
// Tiles of tokens, and one slice or two a block, by the time that rounds of blocks over the SMs take.  Clusters of 4 and 8 blocks fit
// 132 and 120 of 148 SMs only (cudaOccupancyMaxActiveClusters), so two slices a block can save a round: us with two (with one), 1 row
// N 22,016 K 2,048 38.5 (44), 4,608 x 3,584 19.2 (20.3), 32 rows 2,048 x 2,048 10.6 (15.6), 700 rows 60 (72).  All of this is measured, in
// ns: a step takes 700 with 16 tokens (1,190 with two blocks an SM), 830, 1,000 and 1,090 with 32, 48 and 64, which the workers cut up
// as well, 800 with 80 to 1,110 with 160; a block has 2,000 and 19 a token of its own; two slices with 96 tokens, whose registers
// spill, take a twentieth more; split_kernel takes 2,500.  Over 16 shapes and numbers of rows from 100 to 2,048 the tiles chosen are
// within 8 % of the best ones, but for 100 rows x 2,048 K 320 (7.2 us, 6.4 with tiles of 32).
TokenTiles token_tiles(int M, int N, int slices, int steps, int sms) {
  TokenTiles best{16, 1, 1};
  long long best_cost = -1;
  for (int widest = 160; widest >= 16; widest -= 16) {                 // (of each width the fewest tiles)
    const int count = (M + widest - 1) / widest, tn = ((M + count - 1) / count + 15) / 16 * 16;
    for (int both = 1; both <= (slices > 1 && tn <= U_TWO_TOKENS ? 2 : 1); ++both) {
      const int cl = slices / both, fit = sms * (cl == 8 ? 120 : cl == 4 ? 132 : 148) / 148 / cl;   // clusters, at one block an SM
      const long long clusters = (long long)((N + 127) / 128) * count;
      const bool pairs = tn == 16 && clusters > fit;
      const long long rounds = (clusters + fit * (pairs ? 2 : 1) - 1) / (fit * (pairs ? 2 : 1));
      const int step = tn == 16 ? (pairs ? 1190 : 700) : tn <= 32 ? 830 : tn <= 48 ? 1000 : tn <= 64 ? 1090 : tn <= 96 ? 560 + 3 * tn : 310 + 5 * tn;
      const long long cost = rounds * ((long long)both * steps * step + 2000 + 19 * tn) * (both == 2 && tn > 64 ? 21 : 20) / 20 + (tn > 64 ? 2500 : 0);
      if (best_cost < 0 || cost < best_cost) { best = TokenTiles{tn, count, both}; best_cost = cost; }
    }
  }
  return best;
}

int u_sm_count(int* sms) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev);
  return (int)e;
}

template <int TN, int BOTH>
int launch_umma_f32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, long long lda, long long ldc,
                    int tn, int count, int slices, int steps, bool vec_a, void* scratch, int w_fixed, int* error_flag, cudaStream_t stream) {
  auto kern = gemm_f32_umma_kernel<TN, BOTH>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, u_smem(TN));
  if (e != cudaSuccess) return (int)e;
  PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (!enc) return IFX_ERR_UNSUPPORTED;
  CUtensorMap map_w, map_x = {};
  {
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)N};
    cuuint64_t strides[1] = {(cuuint64_t)K * 4};
    cuuint32_t box[2] = {32, 128}, estr[2] = {1, 1};
    if (enc(&map_w, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(W), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return IFX_ERR_UNSUPPORTED;
  }
  if (TN > 64) {
    const int pitch = (K + 7) / 8 * 8;
    cuuint64_t dims[3] = {(cuuint64_t)pitch, (cuuint64_t)M, 3};
    cuuint64_t strides[2] = {(cuuint64_t)pitch * 2, (cuuint64_t)M * pitch * 2};
    cuuint32_t box[3] = {FK64, (cuuint32_t)tn, 3}, estr[3] = {1, 1, 1};
    if (enc(&map_x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, scratch, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return IFX_ERR_UNSUPPORTED;
    const long long items = (long long)M * (pitch / 8);
    int rc = launch_pdl(split_kernel, dim3((unsigned)((items + 255) / 256)), dim3(256), 0, stream, A, (uint4*)scratch, M, K, lda, pitch, (int)vec_a);
    if (rc) return rc;
  }
  const int rc = launch_pdl_cluster(kern, dim3(count, (N + 127) / 128, slices / BOTH), dim3(U_THREADS), (size_t)u_smem(TN), stream, dim3(1, 1, slices / BOTH),
                                    map_w, map_x, A, W, bias, C, M, N, K, lda, ldc, tn, steps, (int)vec_a, w_fixed, error_flag);
  return rc ? rc : IFX_LAUNCH_CHECK();
}
}  // namespace

bool gemm_f32_umma_takes(const float* W, int N, int K) { return K % 4 == 0 && !((uintptr_t)W & 15) && N >= 256 && K >= 256; }

// More rows than this go piece by piece, so that their parts take 64 MB at most (but for K beyond 69,000, where 160 rows take more).  They
// then stay in the L2 besides: 8,192 rows x N 3,584 K 18,944 in pieces of 32 / 64 / 128 / 256 MB 5.56 / 5.44 / 5.75 / 5.83 ms, whole 5.81; N 2,048 K 11,008
// 2.34 / 2.17 / 2.18 / 2.23, 2.23; 2,048 rows of these 1.39 / 1.36 / 1.43 / 1.45, 1.45 and 0.60 / 0.56 / 0.56 / 0.55, 0.55.
constexpr long long U_SCRATCH = 64ll << 20;
static int piece_rows(int K) {
  const long long rows = U_SCRATCH / (6ll * ((K + 7) / 8 * 8)) / 160 * 160;
  return rows < 160 ? 160 : rows > (1 << 30) ? 1 << 30 : (int)rows;
}
long long gemm_f32_umma_scratch(int M, int K) {
  const int rows = M < piece_rows(K) ? M : piece_rows(K);
  return M > 64 ? 6ll * rows * ((K + 7) / 8 * 8) : 0;
}

int gemm_f32_umma(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, long long lda, long long ldc,
                  void* scratch, int w_fixed, int* error_flag, cudaStream_t stream) {
  if (!error_flag) return IFX_ERR_UNSUPPORTED;
  if (M > 64 && (!scratch || ((uintptr_t)scratch & 15))) return IFX_ERR_ALIGNMENT;
  int sms = 0;
  const int rc = u_sm_count(&sms);
  if (rc) return rc;
  const int most = piece_rows(K);
  if (M > most) {                                                      // (the parts of a piece are made when the piece before it is done)
    for (int m = 0; m < M; m += most) {
      const int r = gemm_f32_umma(A + m * lda, W, bias, C + m * ldc, M - m < most ? M - m : most, N, K, lda, ldc, scratch, w_fixed, error_flag, stream);
      if (r) return r;
    }
    return 0;
  }
  const int slices = umma_slices(N, K), steps_all = (K + FK64 - 1) / FK64, steps = (steps_all + slices - 1) / slices;
  const TokenTiles t = token_tiles(M, N, slices, steps, sms);
  const bool vec_a = lda % 4 == 0 && !((uintptr_t)A & 15);
#define IFX_TILE(TN, BOTH) launch_umma_f32<TN, BOTH>(A, W, bias, C, M, N, K, lda, ldc, t.tn, t.count, slices, steps, vec_a, scratch, w_fixed, error_flag, stream)
  if (t.both == 2) return t.tn <= 16 ? IFX_TILE(16, 2) : t.tn <= 32 ? IFX_TILE(32, 2) : t.tn <= 64 ? IFX_TILE(64, 2) : IFX_TILE(96, 2);
  return t.tn <= 16 ? IFX_TILE(16, 1) : t.tn <= 32 ? IFX_TILE(32, 1) : t.tn <= 64 ? IFX_TILE(64, 1)
         : t.tn <= 96 ? IFX_TILE(96, 1) : t.tn <= 128 ? IFX_TILE(128, 1) : IFX_TILE(160, 1);
#undef IFX_TILE
}
