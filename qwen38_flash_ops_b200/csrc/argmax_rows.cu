// ArgmaxRows for B200: idx[r] = argmax_v x[r, v] with numpy semantics (lowest index on ties, the
// first NaN wins over everything, -0 == +0), optionally with the maximum as FP32.
//
// At decode row counts the op is latency, not bandwidth: a row of 151936 BF16 logits is 304 KB that is
// already in L2.  The kernel is built around that.
//   * One cluster of up to eight CTAs per row; a CTA issues all the 16-byte loads of its share of the row at
//     once (a scalar head and tail keep the vector body for odd vocabularies and unaligned rows), so a row
//     costs one round trip to L2.
//   * Long rows: the value first, the index after: a thread takes the maximum of its elements two at a time with the packed
//     NaN-propagating maximum (half an instruction an element; carrying an index along cost five, and a dependent
//     chain 48 elements long), warps meet in a redux and a shared-memory atomicMax, and only the threads that hold
//     the CTA's maximum look through their registers for its first position.  Short rows carry the index along (kFewLoads).
//   * Candidates travel as 64-bit keys whose unsigned maximum is the winner (argmax_key.cuh).
//   * The CTAs of a cluster do not meet at a barrier at the end.  CTA 0 owns one mbarrier and one key slot
//     per peer; a peer stores its key into CTA 0's shared memory, arrives on the barrier with release
//     semantics at cluster scope, and exits; CTA 0 alone waits (bounded), folds and writes.  The one cluster
//     barrier that must precede a remote arrival (the mbarrier has to exist) is split: every CTA arrives
//     right after it has issued its loads and waits only when its own result is ready, so the barrier's
//     latency lies under the memory latency.
// No workspace, no global atomics; the result does not depend on the launch geometry.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <climits>

#include "argmax_key.cuh"
#include "qfg_internal.h"
#include "stream_order.cuh"

namespace qfg {
namespace {

constexpr int kThreads = 512;   // 1024 threads per CTA measured slower at every row count
constexpr int kMaxCluster = 8;
// loads a thread has in flight: 8 CTAs x 512 threads x 6 (10) loads cover 151936 columns; ten for two-byte elements
// measured 0.5 us slower at one row
template <typename T>
constexpr int kInFlight = sizeof(T) == 4 ? 10 : 6;
// Rows of which a thread holds no more loads than this carry the index along with the value instead: the barrier and the
// second look that this saves cost more than the longer chain of compares (value first -> this: BF16 1 x 4099 3.17 -> 2.59
// us, 1024 x 500 10.3 -> 5.2, 4096 x 4099 36.6 -> 19.6, FP32 1 x 32000 3.74 -> 3.14, 1 x 77777 4.45 -> 4.03).  Above it the
// value first is the faster one (BF16 1 x 151936, five loads a thread: carried along 4.32, value first 3.78).
template <typename T>
constexpr int kFewLoads = sizeof(T) == 4 ? 5 : 2;
constexpr int kPeerSpin = 1 << 24;  // bound of CTA 0's wait for its peers (iterations of about 30 ns)

__device__ __forceinline__ float ToFloat(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float ToFloat(__half v) { return __half2float(v); }
__device__ __forceinline__ float ToFloat(float v) { return v; }

__device__ __forceinline__ uint32_t SharedAddr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

// The largest of the elements packed in 32-bit words, NaN if one is (no index yet): one instruction per word.
template <typename T>
struct WordMax;
template <>
struct WordMax<__nv_bfloat16> {
  static constexpr uint32_t kLowest = 0xFF80FF80u;  // -infinity
  __device__ __forceinline__ static uint32_t Max(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("max.NaN.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
  }
  __device__ __forceinline__ static float Value(uint32_t w) { return Fold(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u)); }
  __device__ __forceinline__ static float Fold(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
  }
};
template <>
struct WordMax<__half> {
  static constexpr uint32_t kLowest = 0xFC00FC00u;
  __device__ __forceinline__ static uint32_t Max(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("max.NaN.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
  }
  __device__ __forceinline__ static float Value(uint32_t w) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
    return WordMax<__nv_bfloat16>::Fold(f.x, f.y);
  }
};
template <>
struct WordMax<float> {
  static constexpr uint32_t kLowest = 0xFF800000u;
  __device__ __forceinline__ static uint32_t Max(uint32_t a, uint32_t b) {
    return __float_as_uint(WordMax<__nv_bfloat16>::Fold(__uint_as_float(a), __uint_as_float(b)));
  }
  __device__ __forceinline__ static float Value(uint32_t w) { return __uint_as_float(w); }
};

// A thread's running best, with its index.  Candidates come in order of their index, so that a strict comparison keeps the
// lowest index of equal values, and the first NaN stays.
struct Best {
  float v = 0.f;
  long long i = -1;
  __device__ __forceinline__ void Add(float c, long long idx) {
    if (i < 0 || c > v || (c != c && v == v)) {
      v = c;
      i = idx;
    }
  }
  __device__ __forceinline__ unsigned long long Key() const { return i < 0 ? 0ull : PackKey(v, i); }
};

// the value half of a key: equal for equal values, for -0 and +0 and for every NaN
__device__ __forceinline__ uint32_t ValueKey(float v) { return static_cast<uint32_t>(PackKey(v, 0) >> 32); }

template <typename T, bool FEW>
__global__ void __launch_bounds__(kThreads) ArgmaxRowsKernel(const T* __restrict__ x, long long V,
                                                             long long* __restrict__ idx_out,
                                                             float* __restrict__ val_out) {
  constexpr int kVecElems = 16 / sizeof(T), kLoads = FEW ? kFewLoads<T> : kInFlight<T>;
  __shared__ unsigned long long s_best;               // this CTA's best key
  __shared__ uint32_t s_value;                        // its value half, before the index is known
  __shared__ unsigned long long s_slot[kMaxCluster];  // CTA 0: the peers' keys
  __shared__ unsigned long long s_bar;                // CTA 0: mbarrier, one arrival per peer

  const int C = static_cast<int>(gridDim.x);  // the cluster spans the grid's x extent
  const int c = static_cast<int>(blockIdx.x);
  const long long row = blockIdx.y;
  GridDependencyWait();
  const T* xr = BehindWait(x) + row * V;
  const int tid = threadIdx.x, lane = tid & 31;

  // Row layout: `head` scalar elements up to the first 16-byte boundary, `nvec` vectors, a scalar tail;
  // the vectors are split evenly over the CTAs of the cluster.
  const uintptr_t addr = reinterpret_cast<uintptr_t>(xr);
  long long head = ((16 - (addr & 15)) & 15) / sizeof(T);
  if (head > V) head = V;
  const long long nvec = (V - head) / kVecElems;
  const long long per = (nvec + C - 1) / C;
  const long long vbeg = min(nvec, per * c), vend = min(nvec, vbeg + per);
  const uint4* xv = reinterpret_cast<const uint4*>(xr + head);

  // ---- the first batch of loads goes out before anything else
  constexpr uint32_t kLow = WordMax<T>::kLowest;
  const uint4 lowest = make_uint4(kLow, kLow, kLow, kLow);
  uint4 q[kLoads];
  long long v0 = vbeg + tid;
#pragma unroll
  for (int k = 0; k < kLoads; ++k) {
    const long long v = v0 + static_cast<long long>(k) * kThreads;
    q[k] = v < vend ? __ldg(xv + v) : lowest;
  }
  if (tid == 0) {
    s_best = 0ull;
    s_value = 0u;
    if (c == 0 && C > 1) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(SharedAddr(&s_bar)), "r"(C - 1) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
  }
  __syncthreads();
  if (C > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");

  // head goes to the first CTA, tail to the last: these few elements come with their index
  auto edge_key = [&] {
    unsigned long long edge = 0ull;
    if (c == 0) {
      for (long long i = tid; i < head; i += kThreads) edge = max(edge, PackKey(ToFloat(xr[i]), i));
    }
    if (c == C - 1) {
      for (long long i = head + nvec * kVecElems + tid; i < V; i += kThreads) edge = max(edge, PackKey(ToFloat(xr[i]), i));
    }
    return edge;
  };
  if constexpr (FEW) {
    Best best;
#pragma unroll
    for (int k = 0; k < kLoads; ++k) {
      const long long v = v0 + static_cast<long long>(k) * kThreads;
      if (v < vend) {
        const T* e = reinterpret_cast<const T*>(&q[k]);
#pragma unroll
        for (int j = 0; j < kVecElems; ++j) best.Add(ToFloat(e[j]), head + v * kVecElems + j);
      }
    }
    const unsigned long long wkey = WarpMaxKey(max(edge_key(), best.Key()));
    if (lane == 0 && wkey != 0ull) atomicMax(&s_best, wkey);
  } else {
    // the value first: the largest of every batch of this thread, and the first batch that holds the largest of all
    uint32_t top = 0u;  // ValueKey; 0 is below every value's
    long long top_v0 = v0;
    for (;;) {
      uint32_t m = kLow;
#pragma unroll
      for (int k = 0; k < kLoads; ++k) m = WordMax<T>::Max(m, WordMax<T>::Max(WordMax<T>::Max(q[k].x, q[k].y), WordMax<T>::Max(q[k].z, q[k].w)));
      const uint32_t key = v0 < vend ? ValueKey(WordMax<T>::Value(m)) : 0u;
      if (key > top) {
        top = key;
        top_v0 = v0;
      }
      const long long next = v0 + static_cast<long long>(kThreads) * kLoads;
      if (next >= vend) break;  // rows longer than one batch per thread take further round trips
      v0 = next;
#pragma unroll
      for (int k = 0; k < kLoads; ++k) {
        const long long v = v0 + static_cast<long long>(k) * kThreads;
        q[k] = v < vend ? __ldg(xv + v) : lowest;
      }
    }
    const unsigned long long edge = edge_key();
    const uint32_t mine = max(top, static_cast<uint32_t>(edge >> 32));
    const uint32_t wtop = __reduce_max_sync(0xffffffffu, mine);
    if (lane == 0 && wtop != 0u) atomicMax(&s_value, wtop);
    __syncthreads();

    // then the index, by the threads that hold the CTA's largest value (one, but for ties): their first such element
    const uint32_t cta_top = s_value;
    if (mine == cta_top && cta_top != 0u) {
      unsigned long long key = static_cast<uint32_t>(edge >> 32) == cta_top ? edge : 0ull;
      if (top == cta_top) {
        if (top_v0 != v0) {  // not the batch in hand
#pragma unroll
          for (int k = 0; k < kLoads; ++k) {
            const long long v = top_v0 + static_cast<long long>(k) * kThreads;
            q[k] = v < vend ? __ldg(xv + v) : lowest;
          }
        }
#pragma unroll
        for (int k = kLoads - 1; k >= 0; --k) {
          const long long v = top_v0 + static_cast<long long>(k) * kThreads;
          const uint32_t m = WordMax<T>::Max(WordMax<T>::Max(q[k].x, q[k].y), WordMax<T>::Max(q[k].z, q[k].w));
          if (v < vend && ValueKey(WordMax<T>::Value(m)) == cta_top) {
            const T* e = reinterpret_cast<const T*>(&q[k]);
#pragma unroll
            for (int j = 0; j < kVecElems; ++j) {
              const float f = ToFloat(e[j]);
              if (ValueKey(f) == cta_top) key = max(key, PackKey(f, head + v * kVecElems + j));  // the lower index is the larger key
            }
          }
        }
      }
      atomicMax(&s_best, key);
    }
  }
  __syncthreads();

  // the key of a NaN carries no payload: a NaN winner's value is read back from the row, bit for bit
  auto write_out = [&](unsigned long long key, bool ok) {
    const long long i = KeyIndex(key);
    idx_out[row] = ok ? i : -1;
    if (val_out != nullptr) val_out[row] = (ok && (key >> 32) == 0xFFFFFFFFull) ? ToFloat(xr[i]) : KeyValue(key);
  };
  if (C == 1) {
    if (tid == 0) write_out(s_best, true);
    return;
  }
  // every CTA of the cluster has started (so CTA 0's mbarrier exists) before anybody arrives on it
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (c != 0) {
    if (tid == 0) {
      uint32_t slot, bar;
      asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(slot) : "r"(SharedAddr(&s_slot[c])));
      asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(bar) : "r"(SharedAddr(&s_bar)));
      asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(slot), "l"(s_best) : "memory");
      asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
    }
    return;  // nobody reads this CTA's shared memory: it may leave
  }
  if (tid < 32) {
    uint32_t done = 0;
    for (int spin = 0; spin < kPeerSpin && !done; ++spin) {
      asm volatile("{ .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n selp.u32 %0, 1, 0, p;\n}"
                   : "=r"(done)
                   : "r"(SharedAddr(&s_bar))
                   : "memory");
    }
    unsigned long long key = 0ull;
    if (done) key = lane == 0 ? s_best : (lane < C ? s_slot[lane] : 0ull);
    key = WarpMaxKey(key);
    if (lane == 0) write_out(key, done != 0);  // a wait that ran out (a peer CTA never arrived) leaves an index no row can have
  }
}

template <typename T>
cudaError_t LaunchT(const T* x, int64_t rows, int64_t V, int64_t* idx, float* val, cudaStream_t s) {
  // enough CTAs per row that each thread sees a few vectors; at most the portable cluster size
  const long long vecs = V / (16 / static_cast<long long>(sizeof(T)));
  int cluster = 1;
  while (cluster < kMaxCluster && vecs > static_cast<long long>(cluster) * kThreads * 2) cluster *= 2;
  // Many rows fill the chip without that, and then a CTA's fixed cost (start, barriers, the exchange) is what counts:
  // at most two CTAs per SM, or one where half the CTAs still see a row in one batch of loads (BF16, before -> after:
  // 64 x 151936 8.7 -> 7.3 us, 128 x 151936 15.8 -> 10.7, 128 x 16384 4.25 -> 3.25).
  const long long sms = DeviceSmCount();
  while (cluster > 1 && (cluster * rows > 2 * sms ||
                         (cluster * rows > sms && vecs <= static_cast<long long>(cluster / 2) * kThreads * kInFlight<T>))) {
    cluster /= 2;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(cluster), static_cast<unsigned>(rows), 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(cluster);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1] = OverlapAttribute();
  cfg.attrs = attr;
  cfg.numAttrs = MayOverlapPredecessor(s) ? 2 : 1;
  const bool few = (vecs + cluster - 1) / cluster <= static_cast<long long>(kThreads) * kFewLoads<T>;
  return cudaLaunchKernelEx(&cfg, few ? ArgmaxRowsKernel<T, true> : ArgmaxRowsKernel<T, false>, x, static_cast<long long>(V),
                            reinterpret_cast<long long*>(idx), val);
}

// Folds gathered (value, index) keys: the unsigned maximum of the 64-bit words of a row.
__global__ void LmheadCombineKernel(const unsigned long long* __restrict__ keys, int ranks, int m,
                                    long long* __restrict__ idx, float* __restrict__ val) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= m) return;
  unsigned long long best = 0;
  for (int r = 0; r < ranks; ++r) {
    const unsigned long long k = keys[static_cast<size_t>(r) * m + row];
    best = k > best ? k : best;
  }
  if (idx != nullptr) idx[row] = KeyIndex(best);
  if (val != nullptr) val[row] = KeyValue(best);
}

}  // namespace

cudaError_t LaunchArgmaxRows(int dtype, const void* x, int64_t rows, int64_t vocab, int64_t* idx, float* val,
                             cudaStream_t stream) {
  if (rows < 1 || vocab < 1 || vocab >= INT_MAX || rows > 65535) return cudaErrorInvalidValue;
  switch (dtype) {
    case QFG_BFLOAT16: return LaunchT(static_cast<const __nv_bfloat16*>(x), rows, vocab, idx, val, stream);
    case QFG_FLOAT16: return LaunchT(static_cast<const __half*>(x), rows, vocab, idx, val, stream);
    case QFG_FLOAT: return LaunchT(static_cast<const float*>(x), rows, vocab, idx, val, stream);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t LaunchLmheadCombine(const uint64_t* keys, int ranks, int64_t m, int64_t* idx, float* val,
                                cudaStream_t stream) {
  if (ranks < 1 || m < 1) return cudaErrorInvalidValue;
  const int threads = 64;
  const int blocks = static_cast<int>((m + threads - 1) / threads);
  LmheadCombineKernel<<<blocks, threads, 0, stream>>>(reinterpret_cast<const unsigned long long*>(keys), ranks,
                                                      static_cast<int>(m), reinterpret_cast<long long*>(idx), val);
  return cudaGetLastError();
}

}  // namespace qfg
