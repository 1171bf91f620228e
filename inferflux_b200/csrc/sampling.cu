// Token selection from float32 logits: argmax, repetition / frequency /
// presence penalties, and temperature sampling with top-k, top-p and min-p.
//
// Reference behaviour (runtime/backends/cuda/native/gpu_sampler.cu):
//   greedy      argmax over the row (:124-156, one block of 256, ties by thread order)
//   penalties   logit > 0 ? logit / rep : logit * rep;  -= freq * count;  -= pres if count > 0 (:22-48)
//   temperature softmax(logits / T) in three passes by one block (:216-267)
//   top-p       repeated arg-max until the cumulative probability reaches p (:273-330)
//   draw        one thread walks the cumulative sum against one uniform (:374-401)
// Here rows run in parallel, greedy returns the lowest index among equal
// maxima, top-k/top-p/min-p become a probability threshold on the float bit
// pattern, and the uniform comes from a counter-based generator keyed by
// (seed, counter) so a request's draws do not depend on the batch it is in.
// A row that fits the shared memory of a thread-block cluster (up to 406,912
// logits) is read once and held there by up to 8 blocks; the threshold is
// found by a radix search and all masses are added as integers (see
// sample_cluster_kernel).  Longer rows go to one block of 1024 threads per
// row that keeps exp(logit/T - max) in the caller's scratch `weights`
// [n_rows, vocab] float32 and bisects the threshold (sample_kernel).
#include "common.cuh"

namespace {
constexpr int ST = 1024;

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
// uniform in [0, 1) with 24 bits, from (seed, counter)
__device__ __forceinline__ float uniform01(unsigned long long seed, unsigned long long counter) {
  const unsigned long long x = mix64(mix64(seed) ^ (counter * 0xD1342543DE82EF95ull + 0x632BE59BD9B4E019ull));
  return (float)(x >> 40) * (1.0f / 16777216.0f);
}

struct ArgPair { float v; int i; };
__device__ __forceinline__ ArgPair better(ArgPair a, ArgPair b) {
  // larger value wins; equal values: lower index wins; NaN never wins
  if (b.i >= 0 && (a.i < 0 || b.v > a.v || (b.v == a.v && b.i < a.i))) return b;
  return a;
}
// The best pair of the warp / of the block, for every thread.  `scratch` holds 32 pairs.
__device__ __forceinline__ ArgPair warp_best(ArgPair best) {
  // values as integers of the same order (both zeros alike), 0 for none
  const unsigned bits = __float_as_uint(best.v + 0.0f), key = best.i < 0 ? 0u : bits ^ ((bits >> 31) ? 0xFFFFFFFFu : 0x80000000u);
  const unsigned top = __reduce_max_sync(0xffffffffu, key);
  const unsigned at = __reduce_min_sync(0xffffffffu, key == top ? (unsigned)best.i : 0xFFFFFFFFu);      // (an index of -1 is the largest)
  return ArgPair{__uint_as_float(top ^ ((top >> 31) ? 0x80000000u : 0xFFFFFFFFu)), (int)at};
}
__device__ ArgPair block_best(ArgPair best, ArgPair* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
  best = warp_best(best);
  __syncthreads();
  if (lane == 0) scratch[warp] = best;
  __syncthreads();
  return warp_best(lane < nwarps ? scratch[lane] : ArgPair{-INFINITY, -1});
}
__device__ ArgPair block_argmax(const float* row, int n, ArgPair* scratch) {
  ArgPair best{-INFINITY, -1};
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const float v = row[i];
    if (v == v) best = better(best, ArgPair{v, i});
  }
  return block_best(best, scratch);
}

__global__ void __launch_bounds__(ST) argmax_kernel(const float* __restrict__ logits, long long row_stride,
                                                    int* __restrict__ out, int vocab) {
  pdl_enter();
  __shared__ ArgPair scratch[32];
  const ArgPair b = block_argmax(logits + (size_t)blockIdx.x * row_stride, vocab, scratch);
  if (threadIdx.x == 0) out[blockIdx.x] = b.i < 0 ? 0 : b.i;
}

// A wide row in two steps: blocks (part, row) each find the best of a slice of the row, then one
// warp per row picks among the parts.  `slice` is a multiple of 4; with `vec` rows are 16-byte aligned.
constexpr int AP = 256;
__global__ void __launch_bounds__(AP) argmax_part_kernel(const float* __restrict__ logits, long long row_stride,
                                                         int2* __restrict__ part, int vocab, int slice, int vec) {
  pdl_enter();
  __shared__ ArgPair scratch[32];
  const float* row = logits + (size_t)blockIdx.y * row_stride;
  const int lo = blockIdx.x * slice, hi = min(vocab, lo + slice);
  ArgPair best{-INFINITY, -1};
  if (vec) {
    for (int i = lo + threadIdx.x * 4; i < hi; i += AP * 4) {
      if (i + 3 < hi) {
        const float4 v = *reinterpret_cast<const float4*>(row + i);
        if (v.x == v.x) best = better(best, ArgPair{v.x, i});
        if (v.y == v.y) best = better(best, ArgPair{v.y, i + 1});
        if (v.z == v.z) best = better(best, ArgPair{v.z, i + 2});
        if (v.w == v.w) best = better(best, ArgPair{v.w, i + 3});
      } else {
        for (int j = i; j < hi; ++j) {
          const float v = row[j];
          if (v == v) best = better(best, ArgPair{v, j});
        }
      }
    }
  } else {
    for (int i = lo + threadIdx.x; i < hi; i += AP) {
      const float v = row[i];
      if (v == v) best = better(best, ArgPair{v, i});
    }
  }
  best = block_best(best, scratch);
  if (threadIdx.x == 0) part[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = make_int2(__float_as_int(best.v), best.i);
}
__global__ void __launch_bounds__(32) argmax_final_kernel(const int2* __restrict__ part, int* __restrict__ out, int parts) {
  pdl_enter();
  ArgPair best{-INFINITY, -1};
  for (int p = threadIdx.x; p < parts; p += 32) {
    const int2 v = part[(size_t)blockIdx.x * parts + p];
    best = better(best, ArgPair{__int_as_float(v.x), v.y});
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgPair other{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
    best = better(best, other);
  }
  if (threadIdx.x == 0) out[blockIdx.x] = best.i < 0 ? 0 : best.i;
}

// recent_ids / recent_counts: [n_rows, max_recent]; n_recent[row] entries are valid, ids distinct.
__global__ void penalties_kernel(float* __restrict__ logits, long long row_stride, const int* __restrict__ recent_ids,
                                 const int* __restrict__ recent_counts, const int* __restrict__ n_recent,
                                 int max_recent, const float* __restrict__ rep, const float* __restrict__ freq,
                                 const float* __restrict__ pres, int vocab) {
  pdl_enter();
  const int row = blockIdx.x;
  float* lg = logits + (size_t)row * row_stride;
  const int n = min(n_recent[row], max_recent);
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    const int id = recent_ids[(size_t)row * max_recent + k];
    if (id < 0 || id >= vocab) continue;
    const int count = recent_counts[(size_t)row * max_recent + k];
    float v = lg[id];
    const float r = rep[row];
    v = v > 0.0f ? v / r : v * r;
    v -= freq[row] * (float)count;
    if (count > 0) v -= pres[row];
    lg[id] = v;
  }
}

// The same penalties from the tokens themselves, kept on the device: ring [n_slots, ring_size] holds each
// request's tokens in order of arrival, written round and round; totals[slot] = how many were written in
// all.  Row r belongs to the request in slots[r] (negative: no penalties for this row) and counts its
// latest min(last_n[r], total, ring_size) tokens.  A thread per token: the first occurrence of an id within
// the window applies the penalties for all of them.
__global__ void penalties_ring_kernel(float* __restrict__ logits, long long row_stride, const int* __restrict__ ring,
                                      int ring_size, const int* __restrict__ totals, const int* __restrict__ slots,
                                      const int* __restrict__ last_n, const float* __restrict__ rep,
                                      const float* __restrict__ freq, const float* __restrict__ pres, int vocab) {
  pdl_enter();
  extern __shared__ int window[];                       // [ring_size]
  const int row = blockIdx.x;
  const int slot = slots[row];
  if (slot < 0) return;
  const int total = totals[slot];
  const int n = min(min(last_n[row], total), ring_size);
  for (int t = threadIdx.x; t < n; t += blockDim.x) window[t] = ring[(size_t)slot * ring_size + (total - 1 - t) % ring_size];
  __syncthreads();
  float* lg = logits + (size_t)row * row_stride;
  for (int t = threadIdx.x; t < n; t += blockDim.x) {
    const int id = window[t];
    if (id < 0 || id >= vocab) continue;
    int count = 0;
    bool first = true;
    for (int u = 0; u < n; ++u)
      if (window[u] == id) { ++count; if (u < t) first = false; }
    if (!first) continue;
    float v = lg[id];
    const float r = rep[row];
    v = v > 0.0f ? v / r : v * r;
    v -= freq[row] * (float)count;
    v -= pres[row];
    lg[id] = v;
  }
}

// ring[slots[r]] gets ids[r] as its next token (rows with a negative slot are skipped)
__global__ void ring_append_kernel(int* __restrict__ ring, int ring_size, int* __restrict__ totals,
                                   const int* __restrict__ slots, const int* __restrict__ ids, int n_rows) {
  pdl_enter();
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= n_rows) return;
  const int slot = slots[row];
  if (slot < 0) return;
  const int t = totals[slot];
  ring[(size_t)slot * ring_size + t % ring_size] = ids[row];
  totals[slot] = t + 1;
}

// sum / count over the entries whose weight bits are >= bits
__device__ __forceinline__ void block_sum_count_ge(const float* w, int n, unsigned bits, float* red,
                                                   float* sum_out, int* count_out) {
  float s = 0.0f;
  int c = 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const float v = w[i];
    if (__float_as_uint(v) >= bits) { s += v; ++c; }
  }
  *sum_out = block_sum(s, red);
  *count_out = (int)(block_sum((float)c, red) + 0.5f);   // exact below 2^24 entries
}

__global__ void __launch_bounds__(ST)
sample_kernel(const float* __restrict__ logits, long long row_stride, float* __restrict__ weights,
              const float* __restrict__ temperature, const int* __restrict__ top_k, const float* __restrict__ top_p,
              const float* __restrict__ min_p, const unsigned long long* __restrict__ seeds,
              const unsigned long long* __restrict__ counters, int* __restrict__ out, int vocab) {
  pdl_enter();
  __shared__ ArgPair ascratch[32];
  __shared__ float red[32];
  __shared__ float seg_prefix[ST];
  __shared__ int chosen;
  const int row = blockIdx.x;
  const float* lg = logits + (size_t)row * row_stride;
  const float temp = temperature[row];
  const ArgPair top = block_argmax(lg, vocab, ascratch);
  if (temp <= 0.0f || top.i < 0) {
    if (threadIdx.x == 0) out[row] = top.i < 0 ? 0 : top.i;
    return;
  }
  float* w = weights + (size_t)row * vocab;
  const float inv_t = 1.0f / temp;
  const float mx = top.v * inv_t;
  for (int i = threadIdx.x; i < vocab; i += blockDim.x) {
    const float v = lg[i];
    w[i] = (v == v) ? expf(v * inv_t - mx) : 0.0f;     // in [0, 1], the maximum is exactly 1
  }
  __syncthreads();
  unsigned thr = 0u;                                    // keep entries with weight bits >= thr
  float kept_sum;
  int kept_count;
  const int k = top_k[row];
  if (k > 0 && k < vocab) {                             // largest threshold that keeps at least k entries
    unsigned lo = 0u, hi = 0x3F800000u;                 // bits of 0.0 .. 1.0
    while (lo < hi) {
      const unsigned mid = lo + (hi - lo + 1u) / 2u;
      block_sum_count_ge(w, vocab, mid, red, &kept_sum, &kept_count);
      if (kept_count >= k) lo = mid; else hi = mid - 1u;
    }
    thr = lo;
  }
  const float mp = min_p[row];
  if (mp > 0.0f) thr = max(thr, __float_as_uint(fminf(mp, 1.0f)));
  const float p = top_p[row];
  if (p > 0.0f && p < 1.0f) {                           // largest threshold whose kept mass is >= p of the mass kept so far
    float base_sum;
    block_sum_count_ge(w, vocab, thr, red, &base_sum, &kept_count);
    const float need = p * base_sum;
    unsigned lo = thr, hi = 0x3F800000u;
    while (lo < hi) {
      const unsigned mid = lo + (hi - lo + 1u) / 2u;
      block_sum_count_ge(w, vocab, mid, red, &kept_sum, &kept_count);
      if (kept_sum >= need) lo = mid; else hi = mid - 1u;
    }
    thr = lo;
  }
  // inverse CDF over the kept entries, in index order: thread t owns one contiguous segment
  const int seg = (vocab + ST - 1) / ST;
  const int begin = min(vocab, (int)threadIdx.x * seg), end = min(vocab, begin + seg);
  float mine = 0.0f;
  for (int i = begin; i < end; ++i) {
    const float v = w[i];
    if (__float_as_uint(v) >= thr) mine += v;
  }
  seg_prefix[threadIdx.x] = mine;
  if (threadIdx.x == 0) chosen = -1;
  __syncthreads();
  if (threadIdx.x == 0) {                                // 1024 additions: exclusive prefix, fixed order
    float run = 0.0f;
    for (int t = 0; t < ST; ++t) { const float s = seg_prefix[t]; seg_prefix[t] = run; run += s; }
    red[0] = run;
  }
  __syncthreads();
  const float total = red[0];
  const float target = uniform01(seeds[row], counters[row]) * total;
  const float before = seg_prefix[threadIdx.x];
  const bool last_seg = (threadIdx.x == ST - 1);
  const float after = last_seg ? INFINITY : seg_prefix[threadIdx.x + 1];
  if (mine > 0.0f && before <= target && target < after) {
    float run = before;
    int pick = -1, last_kept = -1;
    for (int i = begin; i < end; ++i) {
      const float v = w[i];
      if (__float_as_uint(v) >= thr && v > 0.0f) {
        run += v;
        last_kept = i;
        if (target < run) { pick = i; break; }
      }
    }
    if (pick < 0) pick = last_kept;
    if (pick >= 0) atomicMax(&chosen, pick);
  }
  __syncthreads();
  if (threadIdx.x == 0) out[row] = chosen >= 0 ? chosen : top.i;
}

// ------------------------------------------------------------------ a row on a cluster
// The same draw for rows that fit the shared memory of a thread-block cluster (8 blocks hold up to 406,912
// logits): every block keeps its slice of the row in shared memory, so the row is read from memory once and
// every later pass runs on chip.  The threshold for top-k / top-p is found by a radix search over the float
// bit pattern (three levels of 1,024 bins, histograms added across the cluster through distributed shared
// memory) instead of 30 bisection passes each, and all masses are summed as 64-bit fixed-point integers
// (weight * 2^39, the maximum weight is exactly 1), so the result does not depend on the order of any sum
// nor on how many blocks share the row.
constexpr int SC_THREADS = 1024, SC_BINS = 1024, SC_MAX_CL = 8;
constexpr int SC_LIST = 1024;                           // weights that a block can note down for the later levels, behind its slice
constexpr int SC_GATHER = 4096;                         // weights of all blocks that one can gather, in the histograms' place
constexpr int SC_MASS_KEY = (127 - 39) << 3;            // weights below this first-level key are below 2^-39: their mass is 0

struct SampleShared {
  unsigned limb[3][SC_BINS];                            // counts, or masses in three 16-bit limbs: 32-bit shared-memory adds
  unsigned long long hist[2][SC_BINS];                  // the limbs put together; two buffers: one is read by the cluster
                                                        // while the next fills
  union {
    unsigned long long warp_tot[32];
    ArgPair ascratch[32];                               // of the row's maximum, before the first scan
  };
  unsigned long long part_total, bcast;                 // what this block tells the others; what lies above the chosen bin
  int chosen;
  int listed;                                           // weights noted; more than there is room for: they did not fit
  float temp, top_p, min_p;                             // the row's numbers, asked for while the row is
  int top_k;
  float uniform;
  ArgPair best;
};
constexpr int SC_SHARED = 227 * 1024;                   // bytes a block can have
constexpr int SC_MAX_SLICE = (SC_SHARED - (int)sizeof(SampleShared)) / 16 * 4;      // floats of a row one block keeps
static_assert(SC_MAX_SLICE == 50864, "the row's limit above is eight of these");

__device__ __forceinline__ unsigned long long weight_fix(float w) { return __float2ull_rz(w * 549755813888.0f); }   // * 2^39

__device__ __forceinline__ unsigned cluster_rank() { unsigned r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// the address of the same shared-memory object in block `rank` of the cluster
template <typename T>
__device__ __forceinline__ const T* cluster_peer(const T* p, unsigned rank) {
  unsigned long long out;
  asm volatile("mapa.u64 %0, %1, %2;" : "=l"(out) : "l"((unsigned long long)p), "r"(rank));
  return reinterpret_cast<const T*>(out);
}

// inclusive sum over the block in thread order; every thread gets its own prefix
__device__ __forceinline__ unsigned long long block_scan_incl_u64(unsigned long long v, unsigned long long* warp_tot) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  __syncthreads();                                      // warp_tot may still be read from the call before
  if (lane == 31) warp_tot[warp] = v;
  __syncthreads();
  if (warp == 0) {                                      // the warps' totals -> what lies before each warp
    const unsigned long long own = warp_tot[lane];
    unsigned long long t = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long u = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += u;
    }
    warp_tot[lane] = t - own;
  }
  __syncthreads();
  return v + warp_tot[warp];
}
// One weight into this level's histogram.
template <bool COUNT>
__device__ __forceinline__ void radix_add(SampleShared& sh, unsigned key, float v) {
  if (COUNT) {
    atomicAdd(&sh.limb[0][key], 1u);
  } else {                                              // a slice has at most SC_MAX_SLICE entries, fewer than 2^16: no limb's sum passes 2^32
    const unsigned long long q = weight_fix(v);
    const unsigned l0 = (unsigned)(q & 0xFFFFu), l1 = (unsigned)(q >> 16) & 0xFFFFu, l2 = (unsigned)(q >> 32);
    if (l0) atomicAdd(&sh.limb[0][key], l0);
    if (l1) atomicAdd(&sh.limb[1][key], l1);            // none below 2^-23
    if (l2) atomicAdd(&sh.limb[2][key], l2);            // few weights are as large as 2^-7
  }
}
__device__ __forceinline__ void radix_clear(SampleShared& sh) {
#pragma unroll
  for (int i = 0; i < 3; ++i) sh.limb[i][threadIdx.x] = 0;
}

// f(w[i]) for this block's n weights, four neighbours a 16-byte read; a short slice one a thread, so that none waits for four
template <typename F> __device__ __forceinline__ void for_weights(const float* w, int n, F f) {
  if (n <= SC_THREADS) {
    if ((int)threadIdx.x < n) f(w[threadIdx.x]);
    return;
  }
  for (int i = 4 * threadIdx.x; i < (n & ~3); i += 4 * SC_THREADS) {
    const float4 v = *reinterpret_cast<const float4*>(w + i);
    f(v.x); f(v.y); f(v.z); f(v.w);
  }
  if ((int)threadIdx.x < (n & 3)) f(w[(n & ~3) + threadIdx.x]);
}

// The largest threshold T >= floor_bits such that the entries with bits >= T number (COUNT) or weigh (fixed point) at least
// a target; floor_bits if even that does not reach it.  w: this block's n weights.  The target is `count` or, of masses, the
// share p of all that the histogram's first level holds (the entries from floor_bits on).  The caller has cleared the limbs
// and filled the first level (bits 20 to 29 as the key).
//
// A level that the cluster's blocks make together costs a barrier of the cluster and eight reads of the others' shared memory a
// thread, some 4 us.  So the second level's walk over the weights notes down those that can still matter (of counts all from the
// first level's bin on, for the masses that may be asked for next; of masses those in the bin) in `list` (room for list_room);
// where they are few enough every block gathers those of all blocks and makes the rest of the search by itself.  gathered: how
// many a call has gathered (they stand in sh.hist), -1: none; with some from a call before, the whole search is local.
template <bool COUNT>
__device__ unsigned radix_threshold(SampleShared& sh, const float* w, int n, float* list, int list_room, unsigned floor_bits,
                                    unsigned long long count, float p, int& buffer, int cl, int& gathered) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, bin = SC_BINS - 1 - tid;    // thread order = bins from the top
  float* all = reinterpret_cast<float*>(sh.hist);
  unsigned prefix = 0;                                  // the bits above the level's ten, once decided
  unsigned long long above = 0, target = count;         // count / mass of the entries above the prefix's range
#pragma unroll 1
  for (int lev = 0; lev < 3; ++lev) {
    const int shift = 20 - 10 * lev;
    auto add = [&](float v) {
      const unsigned b = __float_as_uint(v);
      if ((b >> (shift + 10)) == prefix && b >= floor_bits) radix_add<COUNT>(sh, (b >> shift) & (SC_BINS - 1), v);
    };
    auto own = [&](int k) {
      return COUNT ? (unsigned long long)sh.limb[0][k]
                   : (unsigned long long)sh.limb[0][k] + ((unsigned long long)sh.limb[1][k] << 16) + ((unsigned long long)sh.limb[2][k] << 32);
    };
    auto clear = [&](int k) {                           // (a thread its own bins; counts leave the other two limbs alone)
      sh.limb[0][k] = 0;
      if (!COUNT) { sh.limb[1][k] = 0; sh.limb[2][k] = 0; }
    };
    unsigned long long tot = 0;
    if (gathered < 0) {
      unsigned long long* h = sh.hist[buffer & 1];
      ++buffer;
      if (lev == 1) {
        for_weights(w, n, [&](float v) {
          const unsigned b = __float_as_uint(v);
          if (COUNT ? (b >> 20) >= prefix : (b >> 20) == prefix && b >= floor_bits) {
            const int at = atomicAdd(&sh.listed, 1);
            if (at < list_room) list[at] = v;
          }
          add(v);
        });
      } else if (lev == 2) {
        for_weights(w, n, add);
      }
      __syncthreads();
      if (COUNT) reinterpret_cast<unsigned*>(h)[tid] = sh.limb[0][tid];
      else h[tid] = own(tid);
      clear(tid);
      if (tid == 0) {
        sh.chosen = 0;
        sh.bcast = above;
        if (lev == 0) sh.listed = 0;
      }
      cluster_sync_all();
      if (lev == 1) {                                   // how many the blocks have noted, the same in each of them
        const int theirs = lane < cl ? *cluster_peer(&sh.listed, lane) : 0;
        const bool fit = __all_sync(0xffffffffu, theirs <= list_room);
        int end = theirs;
#pragma unroll
        for (int o = 1; o < SC_MAX_CL; o <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, end, o);
          if (lane >= o) end += t;
        }
        const int total = __shfl_sync(0xffffffffu, end, SC_MAX_CL - 1);
        if (fit && total <= SC_GATHER) {
          gathered = total;
          int from = 0;
          for (int r = 0; r < cl; ++r) {
            const int to = __shfl_sync(0xffffffffu, end, r);
            for (int i = from + tid; i < to; i += SC_THREADS) all[i] = cluster_peer(list, r)[i - from];
            from = to;
          }
          __syncthreads();
          for (int i = tid; i < gathered; i += SC_THREADS) add(all[i]);
          __syncthreads();
          tot = own(bin);
          clear(bin);
        }
      }
      if (gathered < 0 && (COUNT || lev > 0 || bin >= SC_MASS_KEY)) {
        unsigned long long part[SC_MAX_CL];
#pragma unroll
        for (int r = 0; r < SC_MAX_CL; ++r)             // all loads in flight together
          part[r] = r >= cl ? 0ull : COUNT ? (unsigned long long)cluster_peer(reinterpret_cast<unsigned*>(h), r)[bin] : cluster_peer(h, r)[bin];
#pragma unroll
        for (int r = 0; r < SC_MAX_CL; ++r) tot += part[r];
      }
    } else {
      if (lev > 0)
        for (int i = tid; i < gathered; i += SC_THREADS) add(all[i]);
      __syncthreads();                                  // (and the level before has been read)
      if (tid == 0) { sh.chosen = 0; sh.bcast = above; }
      tot = own(bin);
      clear(bin);
    }
    unsigned long long reach = tot;                     // the entries in this bin and above it: within the warp, then what
#pragma unroll                                          // the warps before hold
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long t = __shfl_up_sync(0xffffffffu, reach, o);
      if (lane >= o) reach += t;
    }
    if (lane == 31) sh.warp_tot[warp] = reach;
    __syncthreads();
    const unsigned long long wt = sh.warp_tot[lane];
    unsigned long long before = lane < warp ? wt : 0ull;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    if (!COUNT && lev == 0) {
      unsigned long long base = wt;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) base += __shfl_xor_sync(0xffffffffu, base, o);
      target = (unsigned long long)((double)p * (double)base);
      if (target < 1) target = 1;
    }
    reach += before + above;
    if (reach >= target && reach - tot < target) {      // one bin at most; none: the lowest, and nothing above it is let go
      sh.chosen = bin;
      sh.bcast = reach - tot;
    }
    __syncthreads();
    above = sh.bcast;
    prefix = (prefix << 10) | (unsigned)sh.chosen;
  }
  return prefix > floor_bits ? prefix : floor_bits;
}

// Bound by latency: a row goes through its blocks' shared memory a few times, with a barrier of the cluster between (152,064 logits, 8 / 64
// rows: temperature alone 15.5 / 43 us, top-p 27 / 82, top-k and top-p 28 / 85, where each level was made by the whole cluster 31 / 105 and 44 / 144).  So the
// first level of the first histogram is made while the weights are, the mass that top-p refers to is the histogram's own sum,
// and the masses for the draw are added once, by the segments that the draw then looks into.
__global__ void __launch_bounds__(SC_THREADS, 2)        // two blocks per SM: 32 registers a thread
sample_cluster_kernel(const float* __restrict__ logits, long long row_stride, const float* __restrict__ temperature,
                      const int* __restrict__ top_k, const float* __restrict__ top_p, const float* __restrict__ min_p,
                      const unsigned long long* __restrict__ seeds, const unsigned long long* __restrict__ counters,
                      int* __restrict__ out, int vocab, int cl, int slice, int list_room) {
  pdl_enter();
  extern __shared__ __align__(16) float w_s[];          // this block's slice of the row: logits, then weights; then the list
  float* list = w_s + slice;
  __shared__ SampleShared sh;
  const int tid = threadIdx.x;
  const int row = blockIdx.x / cl;
  const int rank = (int)cluster_rank();
  const int begin = min(vocab, rank * slice), n = min(vocab, begin + slice) - begin;
  const float* lg = logits + (size_t)row * row_stride + begin;
  if (tid == 0) {
    sh.temp = temperature[row];
    sh.top_k = top_k[row];
    sh.top_p = top_p[row];
    sh.min_p = min_p[row];
    sh.uniform = uniform01(seeds[row], counters[row]);
  }
  // the slice into shared memory, and its best logit
  radix_clear(sh);
  ArgPair best{-INFINITY, -1};
  if ((((uintptr_t)lg) & 15) == 0) {
    for (int i = tid * 4; i < n; i += SC_THREADS * 4) {
      if (i + 4 <= n) {
        const float4 v = *reinterpret_cast<const float4*>(lg + i);
        *reinterpret_cast<float4*>(w_s + i) = v;
        if (v.x == v.x) best = better(best, ArgPair{v.x, begin + i});
        if (v.y == v.y) best = better(best, ArgPair{v.y, begin + i + 1});
        if (v.z == v.z) best = better(best, ArgPair{v.z, begin + i + 2});
        if (v.w == v.w) best = better(best, ArgPair{v.w, begin + i + 3});
      } else {
        for (int j = i; j < n; ++j) { const float v = lg[j]; w_s[j] = v; if (v == v) best = better(best, ArgPair{v, begin + j}); }
      }
    }
  } else {
    for (int i = tid; i < n; i += SC_THREADS) { const float v = lg[i]; w_s[i] = v; if (v == v) best = better(best, ArgPair{v, begin + i}); }
  }
  best = block_best(best, sh.ascratch);
  if (tid == 0) sh.best = best;
  cluster_sync_all();
  ArgPair top{-INFINITY, -1};
  {
    ArgPair peer[SC_MAX_CL];
#pragma unroll
    for (int r = 0; r < SC_MAX_CL; ++r) peer[r] = r < cl ? *cluster_peer(&sh.best, r) : ArgPair{-INFINITY, -1};
#pragma unroll
    for (int r = 0; r < SC_MAX_CL; ++r) top = better(top, peer[r]);                 // in rank order: the lowest index among equals
  }
  const float temp = sh.temp;
  if (temp <= 0.0f || top.i < 0) {
    if (rank == 0 && tid == 0) out[row] = top.i < 0 ? 0 : top.i;
    cluster_sync_all();                                 // no block leaves while another may still read its shared memory
    return;
  }
  const float inv_t = 1.0f / temp;
  const float mx = top.v * inv_t;
  const int k = sh.top_k;
  const float mp = sh.min_p, p = sh.top_p;
  const bool by_count = k > 0 && k < vocab, by_mass = p > 0.0f && p < 1.0f;
  const unsigned thr_min = mp > 0.0f ? __float_as_uint(fminf(mp, 1.0f)) : 0u;
  auto weight = [&](float v) { return (v == v) ? expf(v * inv_t - mx) : 0.0f; };      // in [0, 1], the maximum is exactly 1
  auto first_level = [&](float w) {
    const unsigned b = __float_as_uint(w);
    if (by_count) radix_add<true>(sh, (b >> 20) & (SC_BINS - 1), w);
    else if (by_mass && b >= thr_min) radix_add<false>(sh, (b >> 20) & (SC_BINS - 1), w);
  };
  const int n4 = n <= SC_THREADS ? 0 : n & ~3;          // (as for_weights)
  for (int i = 4 * tid; i < n4; i += 4 * SC_THREADS) {
    float4 v = *reinterpret_cast<float4*>(w_s + i);
    v = make_float4(weight(v.x), weight(v.y), weight(v.z), weight(v.w));
    *reinterpret_cast<float4*>(w_s + i) = v;
    if (by_count || by_mass) { first_level(v.x); first_level(v.y); first_level(v.z); first_level(v.w); }
  }
  if (tid < n - n4) {
    const float w = weight(w_s[n4 + tid]);
    w_s[n4 + tid] = w;
    first_level(w);
  }
  __syncthreads();
  int buffer = 0, gathered = -1;
  unsigned thr = 0u;                                    // keep entries with weight bits >= thr
  if (by_count) thr = radix_threshold<true>(sh, w_s, n, list, list_room, 0u, (unsigned long long)k, 0.0f, buffer, cl, gathered);
  thr = max(thr, thr_min);
  if (by_mass) {                                        // the largest threshold whose kept mass is >= p of the mass kept so far
    if (by_count) {
      auto add = [&](float v) {
        const unsigned b = __float_as_uint(v);
        if (b >= thr) radix_add<false>(sh, (b >> 20) & (SC_BINS - 1), v);
      };
      if (gathered < 0) {
        for_weights(w_s, n, add);
      } else {
        for (int i = tid; i < gathered; i += SC_THREADS) add(reinterpret_cast<float*>(sh.hist)[i]);
      }
    }
    thr = radix_threshold<false>(sh, w_s, n, list, list_room, thr, 0ull, p, buffer, cl, gathered);
  }
  // inverse CDF over the kept entries in index order: first the block that holds the target, then the thread, then the entry
  const int seg = ((n + SC_THREADS - 1) / SC_THREADS) | 1;      // odd: the threads' entries lie in different banks
  const int sb = min(n, tid * seg), se = min(n, sb + seg);
  unsigned long long s = 0;
  for (int i = sb; i < se; ++i) { const float v = w_s[i]; if (__float_as_uint(v) >= thr) s += weight_fix(v); }
  const unsigned long long incl = block_scan_incl_u64(s, sh.warp_tot), before = incl - s;
  if (tid == SC_THREADS - 1) sh.part_total = incl;
  cluster_sync_all();
  unsigned long long total = 0, offset = 0, block_total = 0;
#pragma unroll
  for (int r = 0; r < SC_MAX_CL; ++r) {
    const unsigned long long t = r < cl ? *cluster_peer(&sh.part_total, r) : 0ull;
    if (r < rank) offset += t;
    if (r == rank) block_total = t;
    total += t;
  }
  const unsigned long long target = (unsigned long long)((double)sh.uniform * (double)total);   // < total
  if (target >= offset && target - offset < block_total) {                    // block-uniform
    const unsigned long long local = target - offset;
    if (s > 0 && before <= local && local < incl) {     // exactly one thread
      unsigned long long run = before;
      int pick = se - 1;
      for (int i = sb; i < se; ++i) {
        const float v = w_s[i];
        if (__float_as_uint(v) >= thr) {
          run += weight_fix(v);
          if (local < run) { pick = i; break; }
        }
      }
      out[row] = begin + pick;
    }
  }
  cluster_sync_all();
}

inline int sample_slice(int vocab, int cl) { return ((vocab + cl - 1) / cl + 3) / 4 * 4; }
// Blocks per row for the cluster kernel (a power of two up to 8), or 0 if the row does not fit
inline int sample_cluster_blocks(int vocab) {
  int cl = 1;
  while (cl < SC_MAX_CL && (vocab + cl - 1) / cl > 8192) cl <<= 1;
  return sample_slice(vocab, cl) <= SC_MAX_SLICE ? cl : 0;
}

// Room for the list: what the slice leaves of a block's shared memory, or, where the blocks are more than the SMs and two fit one SM, of half
// of that (64 rows of 170,000 with top-p 90.5 us, 142.6 with the whole list and one block an SM).
inline int sample_list_room(int slice, long long blocks, int sms) {
  constexpr int PAIR = 228 * 1024 / 2 - 1024 - 64;      // of 228 KB an SM each block takes 1 KB besides its own
  const int used = (int)sizeof(SampleShared) + slice * (int)sizeof(float);
  const int left = ((blocks > sms && used <= PAIR ? PAIR : SC_SHARED - 64) - used) / (int)sizeof(float);
  return left < 0 ? 0 : left < SC_LIST ? left : SC_LIST;
}

int launch_sample_cluster(const float* logits, long long row_stride, const float* temperature, const int* top_k,
                          const float* top_p, const float* min_p, const unsigned long long* seeds,
                          const unsigned long long* counters, int* out, int n_rows, int vocab, int cl, cudaStream_t stream) {
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return (int)e;
  const int slice = sample_slice(vocab, cl), list_room = sample_list_room(slice, (long long)n_rows * cl, sms);
  const size_t smem = (size_t)(slice + list_room) * sizeof(float);
  e = cudaFuncSetAttribute(sample_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  const int rc = launch_pdl_cluster(sample_cluster_kernel, dim3(n_rows * cl), dim3(SC_THREADS), smem, stream, dim3(cl, 1, 1),
                                    logits, row_stride, temperature, top_k, top_p, min_p, seeds, counters, out, vocab, cl, slice, list_room);
  return rc ? rc : IFX_LAUNCH_CHECK();
}
}  // namespace

// out[row] = lowest index of the largest value of the row (0 for a row of NaNs).  `part` is scratch of
// n_rows * parts pairs of ints (8-byte aligned) for rows cut into `parts` slices, or null with parts <= 1.
IFX_API int ifx_argmax(const float* logits, long long row_stride, int* out, int n_rows, int vocab, void* part, int parts,
                       cudaStream_t stream) {
  if (n_rows <= 0) return 0;
  if (vocab <= 0) return IFX_ERR_UNSUPPORTED;
  int ifx_rc;
  if (parts <= 1 || !part) {
    ifx_rc = launch_pdl(argmax_kernel, dim3(n_rows), dim3(ST), 0, stream, logits, row_stride, out, vocab);
    return ifx_rc ? ifx_rc : IFX_LAUNCH_CHECK();
  }
  if (((uintptr_t)part & 7) || n_rows > 65535) return IFX_ERR_ALIGNMENT;
  const int slice = ((vocab + parts - 1) / parts + 3) / 4 * 4;
  const int vec = ((uintptr_t)logits & 15) == 0 && (row_stride & 3) == 0;
  ifx_rc = launch_pdl(argmax_part_kernel, dim3(parts, n_rows), dim3(AP), 0, stream, logits, row_stride, (int2*)part, vocab, slice, vec);
  if (!ifx_rc) ifx_rc = IFX_LAUNCH_CHECK();
  if (ifx_rc) return ifx_rc;
  ifx_rc = launch_pdl(argmax_final_kernel, dim3(n_rows), dim3(32), 0, stream, (const int2*)part, out, parts);
  return ifx_rc ? ifx_rc : IFX_LAUNCH_CHECK();
}

IFX_API int ifx_apply_penalties(float* logits, long long row_stride, const int* recent_ids, const int* recent_counts,
                                const int* n_recent, int max_recent, const float* rep, const float* freq,
                                const float* pres, int n_rows, int vocab, cudaStream_t stream) {
  if (n_rows <= 0 || max_recent <= 0) return 0;
  const int ifx_rc = launch_pdl(penalties_kernel, dim3(n_rows), dim3(128), 0, stream, logits, row_stride, recent_ids, recent_counts, n_recent, max_recent,
                                               rep, freq, pres, vocab);
  return ifx_rc ? ifx_rc : IFX_LAUNCH_CHECK();
}

// Penalties from the device-resident token rings (penalties_ring_kernel), and the rings' update with the
// tokens just sampled.  ring_size at most 4096.
IFX_API int ifx_apply_penalties_ring(float* logits, long long row_stride, const int* ring, int ring_size,
                                     const int* totals, const int* slots, const int* last_n, const float* rep,
                                     const float* freq, const float* pres, int n_rows, int vocab, cudaStream_t stream) {
  if (n_rows <= 0) return 0;
  if (ring_size < 1 || ring_size > 4096) return IFX_ERR_UNSUPPORTED;
  const int threads = ring_size < 256 ? (ring_size + 31) / 32 * 32 : 256;
  const int ifx_rc = launch_pdl(penalties_ring_kernel, dim3(n_rows), dim3(threads), (size_t)ring_size * sizeof(int), stream, logits,
                                row_stride, ring, ring_size, totals, slots, last_n, rep, freq, pres, vocab);
  return ifx_rc ? ifx_rc : IFX_LAUNCH_CHECK();
}

IFX_API int ifx_ring_append(int* ring, int ring_size, int* totals, const int* slots, const int* ids, int n_rows,
                            cudaStream_t stream) {
  if (n_rows <= 0) return 0;
  if (ring_size < 1) return IFX_ERR_UNSUPPORTED;
  const int ifx_rc = launch_pdl(ring_append_kernel, dim3((n_rows + 127) / 128), dim3(128), 0, stream, ring, ring_size, totals, slots, ids,
                                n_rows);
  return ifx_rc ? ifx_rc : IFX_LAUNCH_CHECK();
}

// The shared memory of ifx_sample's blocks: {blocks a row (0: not a cluster's row), bytes without the list, with it}.
IFX_API void ifx_sample_shared(int vocab, int n_rows, int sms, int* out) {
  const int cl = sample_cluster_blocks(vocab), slice = cl ? sample_slice(vocab, cl) : 0;
  out[0] = cl;
  out[1] = (int)sizeof(SampleShared) + slice * (int)sizeof(float);
  out[2] = out[1] + (cl ? sample_list_room(slice, (long long)n_rows * cl, sms) : 0) * (int)sizeof(float);
}

IFX_API int ifx_sample(const float* logits, long long row_stride, float* weights, const float* temperature,
                       const int* top_k, const float* top_p, const float* min_p, const unsigned long long* seeds,
                       const unsigned long long* counters, int* out, int n_rows, int vocab, cudaStream_t stream) {
  if (n_rows <= 0) return 0;
  if (vocab >= (1 << 24)) return IFX_ERR_UNSUPPORTED;
  if (const int cl = sample_cluster_blocks(vocab))     // rows that fit a cluster's shared memory; the scratch is not used
    return launch_sample_cluster(logits, row_stride, temperature, top_k, top_p, min_p, seeds, counters, out, n_rows, vocab, cl, stream);
  const int ifx_rc = launch_pdl(sample_kernel, dim3(n_rows), dim3(ST), 0, stream, logits, row_stride, weights, temperature, top_k, top_p, min_p, seeds,
                                           counters, out, vocab);
  return ifx_rc ? ifx_rc : IFX_LAUNCH_CHECK();
}

// ---------------------------------------------------------------- no allocation
// ifx_sample_static: ifx_sample for callers that cannot allocate (see sample_static.h).
// The scratch that ifx_sample takes from its caller lives here instead.
#include "sample_static.h"

namespace {
// exp(logit / T - max) of the rows of the call in progress; shared by all calls on the device
static __device__ __align__(256) float g_sample_static_weights[(size_t)IFX_SAMPLE_STATIC_MAX_ROWS *
                                                               IFX_SAMPLE_STATIC_MAX_VOCAB];
constexpr int kMaxDevices = 64;
float* g_sample_static_ptr[kMaxDevices] = {};   // device address of the array, per device, once looked up
}  // namespace

extern "C" const char* ifx_sample_static_message(int code) {
  switch (code) {
    case 0: return "success";
    case IFX_ERR_STATIC_TOO_LARGE:
      return "ifx_sample_static: n_rows or vocab is beyond the built-in scratch "
             "(at most 8 rows of at most 262144 logits); use ifx_sample with a buffer of your own";
    case IFX_ERR_UNSUPPORTED: return "ifx_sample_static: unsupported argument (vocab must be below 2^24, device index below 64)";
    default: return cudaGetErrorString((cudaError_t)code);
  }
}

extern "C" int ifx_sample_static(const float* logits, long long row_stride, const float* temperature,
                                 const int* top_k, const float* top_p, const float* min_p,
                                 const unsigned long long* seeds, const unsigned long long* counters, int* out,
                                 int n_rows, int vocab, cudaStream_t stream) {
  if (n_rows <= 0) return 0;
  if (n_rows > IFX_SAMPLE_STATIC_MAX_ROWS || vocab > IFX_SAMPLE_STATIC_MAX_VOCAB) return IFX_ERR_STATIC_TOO_LARGE;
  if (vocab < 1) return IFX_ERR_UNSUPPORTED;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= kMaxDevices) return IFX_ERR_UNSUPPORTED;
  float* scratch = g_sample_static_ptr[dev];
  if (!scratch) {
    // In host code the array's name is only a handle; the kernel needs its address on this device.
    e = cudaGetSymbolAddress((void**)&scratch, g_sample_static_weights);
    if (e != cudaSuccess) return (int)e;
    g_sample_static_ptr[dev] = scratch;
  }
  // rows are packed [n_rows, vocab]; every element a row reads is written first, so nothing is cleared
  const int ifx_rc = launch_pdl(sample_kernel, dim3(n_rows), dim3(ST), 0, stream, logits, row_stride, scratch, temperature, top_k, top_p, min_p, seeds,
                                           counters, out, vocab);
  return ifx_rc ? ifx_rc : IFX_LAUNCH_CHECK();
}

IFX_STAMP_READER(ifx_stamps_sampling)
