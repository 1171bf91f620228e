// True float32 matrix product for the 32-bit path: C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]).
//
// The reference has no 32-bit model path (its traits cover half and bfloat16
// only, runtime/backends/cuda/native/common/dtype_traits.cuh:13-30) and calls
// cuBLAS with float32 accumulation for every projection
// (runtime/backends/cuda/native/cublas_gemm.cpp:84-102).  These kernels use
// plain float32 multiply-adds on CUDA cores, no reduced-precision mode; they take
// matrices with fewer than 256 rows, a K below 256 or rows off the 16-byte
// boundaries, the others go to gemm_f32_umma.cu.  How an output element is summed depends on N and K
// only: K is cut into k_slices(N, K) slices, the products of a slice are added
// in index order and the slices' sums in slice order, whatever M is and
// whichever kernel runs, so a row's result does not depend on what else is in
// the batch.
//
// Many rows (many_kernel): bound by the multiply-add pipe, with the 128 bytes a cycle that
// shared memory hands to registers close behind: the operands of an 8 x 8 tile a thread take
// as many cycles as its arithmetic (4 x 8 tiles were a tenth slower, A's values stored twice
// over to save their copies a fifth, 8 x 16 tiles no faster and too few blocks for a narrow
// product).  The paired multiply-add (two independent float32 operations an instruction, each
// rounded as fmaf is) leaves issue slots for the rest.  Tiles are stored K-major, columns
// permuted so that neither the transposing stores nor the 16-byte reads meet on a bank; the
// next tile is loaded into registers while the present one is multiplied.  301 rows: N 22,016
// K 2,048 623 us (44 TFLOP/s; 64 x 64 blocks of 4 x 4 a thread 1,167), N 2,048 K 11,008
// 373 us (2,116).  Where the blocks would not fill half the SMs they take 64 columns (8 x 4 a thread, twice
// the blocks; the same sums): 64 rows x N 300 x K 96 6.2 us against 9.9, 17 x 1,000 x 333 16.6 / 24.6, 64 x 512 x 512
// 14.4 / 24.6 (8.2, 20.1 and 34.4 by 64 x 64 blocks of 4 x 4 a thread).
//
// (These sizes go to the tensor cores now, but with rows of W off the 16-byte boundaries or K no multiple of 4.)
//
// Up to 16 rows (few_kernel; from 9 on only where ifx_gemm_f32 says so): bound by reading W.  A thread owns one output column and
// runs along its row of W, which arrives through a ring of cp.async copies.  One row
// against N 151,936 K 2,048: 205 us, 6.0 TB/s (1,406 us by 64 x 64 blocks).
#include "common.cuh"
#include "gemm_f32_umma.h"

namespace {
constexpr int BN = 128;

__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

__device__ __forceinline__ unsigned cluster_rank() { unsigned r; asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// the same place in the shared memory of the cluster's block `rank`
__device__ __forceinline__ float4 read_peer4(const float* p, int rank) {
  unsigned a = (unsigned)__cvta_generic_to_shared(p), ra;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(rank));
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(ra) : "memory");
  return v;
}

// Four values of a row at k .. k + 3, zeros beyond `end` (VEC: all rows 16-byte aligned and k, end multiples of 4).
template <bool VEC> __device__ __forceinline__ float4 load4(const float* row, int k, int end) {
  if (VEC) return k < end ? __ldg(reinterpret_cast<const float4*>(row + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
  return make_float4(k < end ? row[k] : 0.f, k + 1 < end ? row[k + 1] : 0.f, k + 2 < end ? row[k + 2] : 0.f, k + 3 < end ? row[k + 3] : 0.f);
}

constexpr int MK = 16;      // K per tile of many_kernel
constexpr int BM = 64;

// 128 threads, a warp as 8 x 4 lanes, the warps side by side along N: a lane has 2 groups of 4 rows, 32 apart, and CG
// groups of 4 columns, 16 apart.
template <bool VEC, bool SPLIT, int CG>
__global__ void __launch_bounds__(128, SPLIT ? 4 : 3)       // four blocks an SM hide the short slices' first loads (2,048 x 11,008: 373 us, 418 with three)
many_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ C,
            int M, int N, int K, long long lda, long long ldc, int slice_len, int) {
  constexpr int BN = 64 * CG, WR = BN / 32;                    // columns of a block, rows of W a thread loads
  pdl_enter();
  extern __shared__ __align__(16) float f32_smem[];
  float* As = f32_smem;                          // [2][MK][BM]
  float* Ws = f32_smem + 2 * MK * BM;            // [2][MK][BN]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;         // the blocks that share a tile of W run side by side
  const int k_begin = SPLIT ? min(K, (int)blockIdx.z * slice_len) : 0, k_end = SPLIT ? min(K, k_begin + slice_len) : K;
  const int mc = (lane >> 2) * 4, nc = warp * (16 * CG) + (lane & 3) * 4;

  const int lrow = tid >> 2, kq = tid & 3, lk = kq * 4;       // loads: rows lrow, + 32, ...; four values along K
  float4 ra[2], rw[WR];
  auto load = [&](int k0) {                                    // rows out of range read nothing
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int m = m0 + lrow + 32 * i;
      ra[i] = load4<VEC>(A + (size_t)(m < M ? m : 0) * lda, k0 + lk, m < M ? k_end : 0);
    }
#pragma unroll
    for (int i = 0; i < WR; ++i) {
      const int n = n0 + lrow + 32 * i;
      rw[i] = load4<VEC>(W + (size_t)(n < N ? n : 0) * K, k0 + lk, n < N ? k_end : 0);
    }
  };
  auto store = [&](int buf) {                                  // column c of row k stands at c ^ 8 (k / 4)
    float* a = As + buf * MK * BM + lk * BM + (lrow ^ (kq << 3));
    float* w = Ws + buf * MK * BN + lk * BN + (lrow ^ (kq << 3));
#pragma unroll
    for (int i = 0; i < 2; ++i) { a[32 * i] = ra[i].x; a[32 * i + BM] = ra[i].y; a[32 * i + 2 * BM] = ra[i].z; a[32 * i + 3 * BM] = ra[i].w; }
#pragma unroll
    for (int i = 0; i < WR; ++i) { w[32 * i] = rw[i].x; w[32 * i + BN] = rw[i].y; w[32 * i + 2 * BN] = rw[i].z; w[32 * i + 3 * BN] = rw[i].w; }
  };

  unsigned long long acc[8][2 * CG];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 2 * CG; ++j) acc[i][j] = 0ull;
  load(k_begin);
  store(0);
  __syncthreads();
  int buf = 0;
  for (int k0 = k_begin; k0 < k_end; k0 += MK) {
    const bool more = k0 + MK < k_end;
    if (more) load(k0 + MK);
    const float* a = As + buf * MK * BM;
    const float* w = Ws + buf * MK * BN;
#pragma unroll
    for (int kk = 0; kk < MK; ++kk) {
      const int x = (kk >> 2) << 3;
      float av[8];
      unsigned long long wv[2 * CG];
#pragma unroll
      for (int i = 0; i < 2; ++i) *reinterpret_cast<float4*>(av + 4 * i) = *reinterpret_cast<const float4*>(a + kk * BM + ((mc + 32 * i) ^ x));
#pragma unroll
      for (int i = 0; i < CG; ++i) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(w + kk * BN + ((nc + 16 * i) ^ x));
        wv[2 * i] = v.x;
        wv[2 * i + 1] = v.y;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const unsigned long long aa = pack2(av[i], av[i]);
#pragma unroll
        for (int j = 0; j < 2 * CG; ++j) fma2(acc[i][j], aa, wv[j]);
      }
    }
    if (more) store(buf ^ 1);
    __syncthreads();
    buf ^= 1;
  }
  if (!SPLIT) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int m = m0 + mc + (i >> 2) * 32 + (i & 3);
      if (m >= M) continue;
#pragma unroll
      for (int j = 0; j < 2 * CG; ++j) {
        const int n = n0 + nc + (j >> 1) * 16 + (j & 1) * 2;
        float lo, hi;
        unpack2(acc[i][j], lo, hi);
        if (n < N) C[(size_t)m * ldc + n] = lo + (bias ? bias[n] : 0.0f);
        if (n + 1 < N) C[(size_t)m * ldc + n + 1] = hi + (bias ? bias[n + 1] : 0.0f);
      }
    }
    return;
  }
  // the cluster's blocks hold the slices of one tile: each leaves its sums in shared memory and adds up its share of the rows
  const int slices = gridDim.z, rank = (int)cluster_rank();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float* row = f32_smem + (mc + (i >> 2) * 32 + (i & 3)) * BN + nc;
#pragma unroll
    for (int j = 0; j < 2 * CG; ++j) *reinterpret_cast<unsigned long long*>(row + (j >> 1) * 16 + (j & 1) * 2) = acc[i][j];
  }
  cluster_sync();
  const int rows = BM / slices;                                // 2, 4 or 8 slices
  for (int p = tid; p < rows * (BN / 4); p += 128) {
    const int r = rank * rows + p / (BN / 4), c = (p % (BN / 4)) * 4, m = m0 + r, n = n0 + c;
    if (m >= M || n >= N) continue;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int z = 0; z < slices; ++z) {
      const float4 v = read_peer4(f32_smem + r * BN + c, z);
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    const float o[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (n + i < N) C[(size_t)m * ldc + n + i] = o[i] + (bias ? bias[n + i] : 0.0f);
  }
  cluster_sync();                                              // no block leaves while another still reads its sums
}

constexpr int FK = 32, FSTAGES = 4, FPITCH = FK + 4;           // rows 36 floats apart: eight lanes' 16-byte reads meet no bank twice

__device__ __forceinline__ void cp16(float* dst, const float* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp4(float* dst, const float* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(valid ? 4 : 0) : "memory");
}

template <int R, bool VEC>
__global__ void __launch_bounds__(128)
few_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ C,
           int M, int N, int K, long long lda, long long ldc, int slice_len, int w_fixed) {
  pdl_launch_dependents();
  extern __shared__ __align__(16) float f32_smem[];
  float* Wr = f32_smem;                                        // [FSTAGES][BN][FPITCH]
  float* Ar = f32_smem + FSTAGES * BN * FPITCH;                // [FSTAGES][R][FK]
  const int tid = threadIdx.x, n0 = blockIdx.x * BN;
  const int k_begin = min(K, (int)blockIdx.z * slice_len), k_end = min(K, k_begin + slice_len);
  const int steps = (k_end - k_begin + FK - 1) / FK;
  auto copy_w = [&](int s) {
    if (s >= steps) return;
    float* dst = Wr + (s % FSTAGES) * BN * FPITCH;
    const int k0 = k_begin + s * FK;
    if (VEC) {
#pragma unroll
      for (int i = 0; i < BN * FK / 4 / 128; ++i) {
        const int p = tid + i * 128, r = p / (FK / 4), c = (p % (FK / 4)) * 4;
        const bool ok = n0 + r < N && k0 + c < k_end;
        cp16(dst + r * FPITCH + c, W + (ok ? (size_t)(n0 + r) * K + k0 + c : 0), ok);
      }
    } else {
      for (int p = tid; p < BN * FK; p += 128) {
        const int r = p / FK, c = p % FK;
        const bool ok = n0 + r < N && k0 + c < k_end;
        cp4(dst + r * FPITCH + c, W + (ok ? (size_t)(n0 + r) * K + k0 + c : 0), ok);
      }
    }
  };
  auto copy_a = [&](int s) {
    if (s >= steps) return;
    const int k0 = k_begin + s * FK;
    for (int p = tid; p < R * FK; p += 128) {
      const int r = p / FK, c = p % FK;
      const bool ok = r < M && k0 + c < k_end;
      cp4(Ar + (s % FSTAGES) * R * FK + p, A + (ok ? (size_t)r * lda + k0 + c : 0), ok);
    }
  };
  // a W that nothing pending writes: its first tiles are on their way before the kernel ahead has finished
  if (!w_fixed) pdl_wait();
#pragma unroll
  for (int s = 0; s < FSTAGES - 1; ++s) copy_w(s);
  pdl_wait();
#pragma unroll
  for (int s = 0; s < FSTAGES - 1; ++s) {
    copy_a(s);
    cp_async_commit();
  }
  float acc[R];
#pragma unroll
  for (int r = 0; r < R; ++r) acc[r] = 0.0f;
  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(FSTAGES - 2) : "memory");
    __syncthreads();                                           // tile s is there for all, tile s - 1 has been read by all
    copy_w(s + FSTAGES - 1);
    copy_a(s + FSTAGES - 1);
    cp_async_commit();
    const float* w = Wr + (s % FSTAGES) * BN * FPITCH + tid * FPITCH;
    const float* a = Ar + (s % FSTAGES) * R * FK;
#pragma unroll
    for (int c = 0; c < FK; c += 4) {
      const float4 wv = *reinterpret_cast<const float4*>(w + c);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float4 av = *reinterpret_cast<const float4*>(a + r * FK + c);
        acc[r] = fmaf(av.w, wv.w, fmaf(av.z, wv.z, fmaf(av.y, wv.y, fmaf(av.x, wv.x, acc[r]))));
      }
    }
  }
  cp_async_wait_all();
  const int n = n0 + tid, slices = gridDim.z;
  if (slices == 1) {
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (r < M && n < N) C[(size_t)r * ldc + n] = acc[r] + (bias ? bias[n] : 0.0f);
    return;
  }
  __syncthreads();                                             // the ring is free: the slices' sums go there
#pragma unroll
  for (int r = 0; r < R; ++r) f32_smem[r * BN + tid] = acc[r];
  cluster_sync();
  const int rank = (int)cluster_rank();
  for (int p = rank * 128 + tid; p < R * (BN / 4); p += slices * 128) {
    const int r = p / (BN / 4), c = (p % (BN / 4)) * 4;
    if (r >= M || n0 + c >= N) continue;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int z = 0; z < slices; ++z) {
      const float4 v = read_peer4(f32_smem + r * BN + c, z);
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    const float o[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (n0 + c + i < N) C[(size_t)r * ldc + n0 + c + i] = o[i] + (bias ? bias[n0 + c + i] : 0.0f);
  }
  cluster_sync();
}

// Slices of K, from N and K alone (1, 2, 4 or 8): enough that a few hundred rows of a narrow product fill the SMs, each
// at least 256 long.
int k_slices(int N, int K) {
  const int cols = (N + BN - 1) / BN;
  int s = 1;
  while (s < 8 && cols * s < 128 && K / (2 * s) >= 256) s *= 2;
  return s;
}
// whether tiles of 64 x 128 fill less than half the SMs
bool tiles_leave_idle(int M, int N, int slices, int sms) { return 2ll * ((M + BM - 1) / BM) * ((N + BN - 1) / BN) * slices <= sms; }
int sm_count(int* sms) {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return (int)e;
  }
  *sms = n;
  return 0;
}
int slice_length(int K, int slices) { return ((K + slices - 1) / slices + FK - 1) / FK * FK; }

template <typename Kern>
int launch_f32(Kern kern, dim3 grid, int threads, size_t smem, cudaStream_t stream, const float* A, const float* W, const float* bias,
               float* C, int M, int N, int K, long long lda, long long ldc, int slice_len, int w_fixed) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  const int rc = launch_pdl_cluster(kern, grid, dim3(threads), smem, stream, dim3(1, 1, grid.z), A, W, bias, C, M, N, K, lda, ldc, slice_len, w_fixed);
  return rc ? rc : IFX_LAUNCH_CHECK();
}

template <int R>
int few(bool vec, const float* A, const float* W, const float* bias, float* C, int M, int N, int K, long long lda, long long ldc,
        int w_fixed, cudaStream_t stream) {
  const int slices = k_slices(N, K);
  const dim3 grid((N + BN - 1) / BN, 1, slices);
  const size_t smem = (size_t)FSTAGES * (BN * FPITCH + R * FK) * sizeof(float);
  return vec ? launch_f32(few_kernel<R, true>, grid, 128, smem, stream, A, W, bias, C, M, N, K, lda, ldc, slice_length(K, slices), w_fixed)
             : launch_f32(few_kernel<R, false>, grid, 128, smem, stream, A, W, bias, C, M, N, K, lda, ldc, slice_length(K, slices), w_fixed);
}

template <bool SPLIT, int CG>
int many_wide(bool vec, const float* A, const float* W, const float* bias, float* C, int M, int N, int K, long long lda, long long ldc,
         int slices, cudaStream_t stream) {
  constexpr int BN = 64 * CG;
  const dim3 grid((M + BM - 1) / BM, (N + BN - 1) / BN, slices);
  size_t smem = (size_t)2 * MK * (BM + BN) * sizeof(float);
  if (SPLIT && smem < (size_t)BM * BN * sizeof(float)) smem = (size_t)BM * BN * sizeof(float);
  const int len = slice_length(K, slices);
  return vec ? launch_f32(many_kernel<true, SPLIT, CG>, grid, 128, smem, stream, A, W, bias, C, M, N, K, lda, ldc, len, 0)
             : launch_f32(many_kernel<false, SPLIT, CG>, grid, 128, smem, stream, A, W, bias, C, M, N, K, lda, ldc, len, 0);
}
template <bool SPLIT>
int many(bool vec, bool narrow, const float* A, const float* W, const float* bias, float* C, int M, int N, int K, long long lda,
         long long ldc, int slices, cudaStream_t stream) {
  return narrow ? many_wide<SPLIT, 1>(vec, A, W, bias, C, M, N, K, lda, ldc, slices, stream)
                : many_wide<SPLIT, 2>(vec, A, W, bias, C, M, N, K, lda, ldc, slices, stream);
}
}  // namespace

// A rows lda, C rows ldc elements apart, W contiguous, any K and alignment.  w_fixed: 1 = W is a parameter, which may be read
// before the kernel has waited for those ahead of it (see common.cuh on what that takes; here up to 16 rows, and the tensor
// cores, use it).  scratch: as many bytes as ifx_gemm_f32_scratch says for the same W, M, N and K, 16-byte aligned; null where that is 0.
// error_flag: a device word set if a bounded wait inside the kernel runs out.
IFX_API long long ifx_gemm_f32_scratch(const float* W, int M, int N, int K) {
  return M > 0 && K > 0 && gemm_f32_umma_takes(W, N, K) ? gemm_f32_umma_scratch(M, K) : 0;
}
IFX_API int ifx_gemm_f32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K,
                         long long lda, long long ldc, void* scratch, int w_fixed, int* error_flag, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return IFX_ERR_UNSUPPORTED;
  if (gemm_f32_umma_takes(W, N, K)) return gemm_f32_umma(A, W, bias, C, M, N, K, lda, ldc, scratch, w_fixed, error_flag, stream);
  const bool vec = (K % 4 == 0) && (((uintptr_t)W & 15) == 0);                       // of W's rows
  const bool vec_a = vec && (lda % 4 == 0) && (((uintptr_t)A & 15) == 0);
  if (M == 1) return few<1>(vec, A, W, bias, C, M, N, K, lda, ldc, w_fixed, stream);
  if (M <= 4) return few<4>(vec, A, W, bias, C, M, N, K, lda, ldc, w_fixed, stream);
  if (M <= 8) return few<8>(vec, A, W, bias, C, M, N, K, lda, ldc, w_fixed, stream);
  const int slices = k_slices(N, K);
  int sms = 0;
  const int rc = sm_count(&sms);
  if (rc) return rc;
  // (rows of W off the boundaries, K whole and few columns: 9 rows x 1,000 x 333 20.9 us streamed, 16.4 in tiles)
  if (M <= 16 && (vec || slices > 1 || !tiles_leave_idle(M, N, slices, sms))) return few<16>(vec, A, W, bias, C, M, N, K, lda, ldc, w_fixed, stream);
  const bool narrow = tiles_leave_idle(M, N, slices, sms);
  if (slices > 1) return many<true>(vec_a, narrow, A, W, bias, C, M, N, K, lda, ldc, slices, stream);
  return many<false>(vec_a, narrow, A, W, bias, C, M, N, K, lda, ldc, 1, stream);
}
