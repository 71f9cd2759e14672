// Device code that the few-row kernels share (skinny_gemm.cu, skinny_stream.cu): loads and conversions, one k-step of MMAs,
// tile location, the staging of x, and the epilogue from the warps' partial sums to the stored outputs.
#pragma once

#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>


#include "argmax_key.cuh"
#include "qfg_internal.h"
#include "stream_order.cuh"

namespace qfg {
namespace {

namespace cg = cooperative_groups;

constexpr int kMaxThreads = 32 * kMaxWarps;  // warp-ring and tcgen05 kernels (20 warps: at most 102 registers per thread)

// ------------------------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t SmemAddr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void CpAsync16(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void CpAsync8(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void CpAsync4(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void CpAsyncCommit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void CpAsyncWait(int pending) {
  switch (pending) {
    case 0: asm volatile("cp.async.wait_group 0;" ::: "memory"); break;
    case 1: asm volatile("cp.async.wait_group 1;" ::: "memory"); break;
    case 2: asm volatile("cp.async.wait_group 2;" ::: "memory"); break;
    case 3: asm volatile("cp.async.wait_group 3;" ::: "memory"); break;
    case 4: asm volatile("cp.async.wait_group 4;" ::: "memory"); break;
    case 5: asm volatile("cp.async.wait_group 5;" ::: "memory"); break;
    case 6: asm volatile("cp.async.wait_group 6;" ::: "memory"); break;
    default: asm volatile("cp.async.wait_group 7;" ::: "memory"); break;
  }
}
__device__ __forceinline__ uint4 Lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint2 Lds64(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint32_t Lds8(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
// shared-memory loads at a register address plus a compile-time offset (folded into the instruction)
template <int OFF>
__device__ __forceinline__ uint4 Lds128At(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4+%5];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr), "n"(OFF));
  return v;
}
template <int OFF>
__device__ __forceinline__ uint2 Lds64At(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2+%3];" : "=r"(v.x), "=r"(v.y) : "r"(addr), "n"(OFF));
  return v;
}
template <int OFF>
__device__ __forceinline__ uint32_t Lds8At(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u8 %0, [%1+%2];" : "=r"(v) : "r"(addr), "n"(OFF));
  return v;
}
// 16 bytes from `base + off` to shared memory at `dst + OFF`; CACHED keeps the line in L1 (.ca) for neighbours
template <int OFF, bool CACHED>
__device__ __forceinline__ void CpAsync16At(uint32_t dst, const uint8_t* base, uint32_t off) {
  if constexpr (CACHED) {
    asm volatile("{ .reg .u64 a;\n mad.wide.u32 a, %2, 1, %1;\n cp.async.ca.shared.global [%0+%3], [a], 16;\n}" ::"r"(dst), "l"(base),
                 "r"(off), "n"(OFF)
                 : "memory");
  } else {
    asm volatile("{ .reg .u64 a;\n mad.wide.u32 a, %2, 1, %1;\n cp.async.cg.shared.global [%0+%3], [a], 16;\n}" ::"r"(dst), "l"(base),
                 "r"(off), "n"(OFF)
                 : "memory");
  }
}
__device__ __forceinline__ uint4 Ldg128(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}
__device__ __forceinline__ uint2 Ldg64(const void* p) {
  uint2 v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t Ldg8(const void* p) {
  uint32_t v;
  asm volatile("ld.global.nc.u8 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t Prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}
// Four E2M1 pairs (one per byte, low nibble -> low half) to four f16x2 registers.
__device__ __forceinline__ void CvtE2m1x8(uint32_t c, uint32_t (&r)[4]) {
  asm("{ .reg .b8 b0, b1, b2, b3;\n"
      " mov.b32 {b0, b1, b2, b3}, %4;\n"
      " cvt.rn.f16x2.e2m1x2 %0, b0;\n"
      " cvt.rn.f16x2.e2m1x2 %1, b1;\n"
      " cvt.rn.f16x2.e2m1x2 %2, b2;\n"
      " cvt.rn.f16x2.e2m1x2 %3, b3;\n}"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
      : "r"(c));
}
// Two E4M3 pairs (low 16 bits, high 16 bits) to two f16x2 registers.
__device__ __forceinline__ void CvtE4m3x4(uint32_t c, uint32_t& lo, uint32_t& hi) {
  asm("{ .reg .b16 h0, h1;\n"
      " mov.b32 {h0, h1}, %2;\n"
      " cvt.rn.f16x2.e4m3x2 %0, h0;\n"
      " cvt.rn.f16x2.e4m3x2 %1, h1;\n}"
      : "=r"(lo), "=r"(hi)
      : "r"(c));
}
__device__ __forceinline__ uint32_t CvtE4m3x2(uint32_t pair16) {
  uint32_t r;
  asm("{ .reg .b16 h0;\n cvt.u16.u32 h0, %1;\n cvt.rn.f16x2.e4m3x2 %0, h0;\n}" : "=r"(r) : "r"(pair16));
  return r;
}
// (a & mask) | (b & ~mask) in one instruction
__device__ __forceinline__ uint32_t BitSelect(uint32_t a, uint32_t b, uint32_t mask) {
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, 0xE4;" : "=r"(r) : "r"(a), "r"(b), "r"(mask));
  return r;
}
__device__ __forceinline__ uint32_t Hmul2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
// An exact f16x2 value as bf16x2 (the values here have at most 6 significant bits).
__device__ __forceinline__ uint32_t HalfPairToBf16Pair(uint32_t h) {
  const __half2 hv = *reinterpret_cast<const __half2*>(&h);
  const float2 f = __half22float2(hv);
  const __nv_bfloat162 b = __floats2bfloat162_rn(f.x, f.y);
  return *reinterpret_cast<const uint32_t*>(&b);
}
template <bool BF16>
__device__ __forceinline__ void Mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                    uint32_t b1) {
  if constexpr (BF16) {
    asm(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  } else {
    asm(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
}

__device__ __forceinline__ int CeilLog2(int v) { return v <= 1 ? 0 : 32 - __clz(v - 1); }

// (value, index) order of ArgmaxRows: NaN beats non-NaN, then larger value, then lower index.
__device__ __forceinline__ bool Better(float av, long long ai, float bv, long long bi) {
  if (av != av) return (bv == bv) || ai < bi;
  if (bv != bv) return false;
  return av > bv || (av == bv && ai < bi);
}
// W: 16-column groups a thread of the NVFP4 direct kernel owns.  With W = 2 a warp covers 256
// columns and thread group g owns groups g and g + 8 of them, i.e. two 8-byte runs 64 bytes
// apart in every row: fewer partly used sectors and less loop overhead per weight, and the
// 8-byte shared-memory reads stay aligned on rows that start 8 bytes off a 16-byte boundary.
template <int MODE, int W = 1>
struct Geom;
template <>
struct Geom<kBf16, 1> {
  static constexpr int kColsPerThread = 8, kBytesPerThread = 16, kMmas = 4;
};
template <>
struct Geom<kFp8, 1> {
  static constexpr int kColsPerThread = 16, kBytesPerThread = 16, kMmas = 8;
};
template <int W>
struct Geom<kNvfp4, W> {
  static constexpr int kColsPerThread = 16, kBytesPerThread = 8, kMmas = 8 * W;
};

// The raw bytes of one k-step of one thread: four consecutive weight rows (4t .. 4t+3 of the
// step) of its columns, plus the NVFP4 block-scale bytes of those rows (one byte per 16-column
// group).  The B fragment of the same thread is x[4t .. 4t+3] of the step: the k index of an MMA
// is a free permutation.
template <int MODE, int W = 1>
struct Raw {
  uint4 r[4];
};
template <int W>
struct Raw<kNvfp4, W> {
  uint2 r[W][4];
  uint32_t s[W][4];
};

// One k-step of one warp from registers: dequantise to k-paired operands and run the MMAs.
template <int MODE, bool SLOW, int W = 1>
__device__ __forceinline__ void ComputeStep(float (&acc)[Geom<MODE, W>::kMmas][4], const Raw<MODE, W>& w, uint32_t b0,
                                            uint32_t b1) {
  constexpr bool kBf16Mma = (MODE == kBf16) || SLOW;
  if constexpr (MODE == kBf16) {
    const uint32_t a[4] = {w.r[0].x, w.r[0].y, w.r[0].z, w.r[0].w}, b[4] = {w.r[1].x, w.r[1].y, w.r[1].z, w.r[1].w};
    const uint32_t c[4] = {w.r[2].x, w.r[2].y, w.r[2].z, w.r[2].w}, d[4] = {w.r[3].x, w.r[3].y, w.r[3].z, w.r[3].w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      Mma<true>(acc[i], Prmt(a[i], b[i], 0x5410u), Prmt(a[i], b[i], 0x7632u), Prmt(c[i], d[i], 0x5410u),
                Prmt(c[i], d[i], 0x7632u), b0, b1);
    }
  } else if constexpr (MODE == kFp8) {
    const uint32_t a[4] = {w.r[0].x, w.r[0].y, w.r[0].z, w.r[0].w}, b[4] = {w.r[1].x, w.r[1].y, w.r[1].z, w.r[1].w};
    const uint32_t c[4] = {w.r[2].x, w.r[2].y, w.r[2].z, w.r[2].w}, d[4] = {w.r[3].x, w.r[3].y, w.r[3].z, w.r[3].w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint32_t p[4], q[4];
      CvtE4m3x4(Prmt(a[i], b[i], 0x5140u), p[0], p[1]);
      CvtE4m3x4(Prmt(a[i], b[i], 0x7362u), p[2], p[3]);
      CvtE4m3x4(Prmt(c[i], d[i], 0x5140u), q[0], q[1]);
      CvtE4m3x4(Prmt(c[i], d[i], 0x7362u), q[2], q[3]);
      if constexpr (SLOW) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          p[e] = HalfPairToBf16Pair(p[e]);
          q[e] = HalfPairToBf16Pair(q[e]);
        }
      }
      Mma<kBf16Mma>(acc[2 * i], p[0], p[1], q[0], q[1], b0, b1);
      Mma<kBf16Mma>(acc[2 * i + 1], p[2], p[3], q[2], q[3], b0, b1);
    }
  } else {
#pragma unroll
    for (int h = 0; h < W; ++h) {
      const uint32_t s_ab = CvtE4m3x2(Prmt(w.s[h][0], w.s[h][1], 0x0040u));
      const uint32_t s_cd = CvtE4m3x2(Prmt(w.s[h][2], w.s[h][3], 0x0040u));
      const uint32_t a[2] = {w.r[h][0].x, w.r[h][0].y}, b[2] = {w.r[h][1].x, w.r[h][1].y};
      const uint32_t c[2] = {w.r[h][2].x, w.r[h][2].y}, d[2] = {w.r[h][3].x, w.r[h][3].y};
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        // byte q of `e_*`: (row A nibble, row B nibble) of column 8i + 2q; of `o_*`: column 8i + 2q + 1
        uint32_t e_ab[4], o_ab[4], e_cd[4], o_cd[4];
        CvtE2m1x8(BitSelect(a[i], b[i] << 4, 0x0F0F0F0Fu), e_ab);
        CvtE2m1x8(BitSelect(a[i] >> 4, b[i], 0x0F0F0F0Fu), o_ab);
        CvtE2m1x8(BitSelect(c[i], d[i] << 4, 0x0F0F0F0Fu), e_cd);
        CvtE2m1x8(BitSelect(c[i] >> 4, d[i], 0x0F0F0F0Fu), o_cd);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint32_t a0 = Hmul2(e_ab[q], s_ab), a1 = Hmul2(o_ab[q], s_ab);
          uint32_t a2 = Hmul2(e_cd[q], s_cd), a3 = Hmul2(o_cd[q], s_cd);
          if constexpr (SLOW) {
            a0 = HalfPairToBf16Pair(a0);
            a1 = HalfPairToBf16Pair(a1);
            a2 = HalfPairToBf16Pair(a2);
            a3 = HalfPairToBf16Pair(a3);
          }
          Mma<kBf16Mma>(acc[8 * h + 4 * i + q], a0, a1, a2, a3, b0, b1);
        }
      }
    }
  }
}

// What a CTA works on: a column tile of one weight and a slice of K.
struct Tile {
  int seg, n0, n1, kbeg, kend, kslice, crank, C;
};

__device__ __forceinline__ Tile LocateTile(const GemmParams& p) {
  Tile tl;
  int s = 0;
#pragma unroll
  for (int i = 1; i < kMaxSeg; ++i) s += (i < p.nseg && static_cast<int>(blockIdx.x) >= p.seg[i].tile_begin) ? 1 : 0;
  tl.seg = s;
  const Segment& sg = p.seg[s];
  // tile t covers granules [t G / T, (t + 1) G / T): in 32 bits, from G = quot T + rem (a 64-bit division is
  // a hundred instructions, and this is the first thing every CTA does)
  const unsigned t = blockIdx.x - static_cast<unsigned>(sg.tile_begin), T = static_cast<unsigned>(sg.tiles);
  const unsigned g0 = t * sg.gran_quot + t * sg.gran_rem / T, g1 = (t + 1) * sg.gran_quot + (t + 1) * sg.gran_rem / T;
  tl.n0 = static_cast<int>(g0) * p.gran;
  tl.n1 = min(sg.n - sg.tail_cols, static_cast<int>(g1) * p.gran);
  tl.C = static_cast<int>(gridDim.y);
  tl.crank = static_cast<int>(blockIdx.y);
  tl.kbeg = 0;
  tl.kend = p.K;
  if (tl.C > 1) {
    const unsigned ksteps_total = static_cast<unsigned>(p.K + 15) >> 4, C = gridDim.y, r = blockIdx.y;
    tl.kbeg = static_cast<int>(r * ksteps_total / C) * 16;
    tl.kend = min(p.K, static_cast<int>((r + 1) * ksteps_total / C) * 16);
  }
  tl.kslice = max(0, tl.kend - tl.kbeg);
  return tl;
}

struct SharedScratch {
  float inv_scale[kMaxRows];
  float scale[kMaxRows];
  uint32_t rmax[kMaxRows];  // largest BF16 magnitude bits of the row's K slice
  uint32_t rmin[kMaxRows];  // smallest non-zero BF16 magnitude bits (0x7FFF if the slice is all zero)
  float best_v[kMaxThreads / 32][kMaxRows];
  long long best_i[kMaxThreads / 32][kMaxRows];
  float gate[kMaxRows];  // SharedExpertDown: the BF16 sigmoid gate of every row (best_v holds its partial sums first)
  int last;
  int xfail;  // sharded LM head: a wait for a peer's keys ran out in this call
  unsigned long long rowkey[kMaxRows];  // fused LM head: the CTA's best key of every row (atomicMax of the warps' bests)
};

// The BF16 arithmetic of SharedExpertDown (src/common/sigmoid_acc.cuh:12-21, skinny_gemm.cuh:73-80): sigmoid
// in FP32 from exp(-|a|), rounded once to BF16; Swish = bf16(x * bf16(sigmoid(x))); swish_mul = bf16(Swish(g) * u).
__device__ __forceinline__ float RoundBf16(float v) { return __bfloat162float(__float2bfloat16(v)); }
__device__ __forceinline__ float SigmoidBf16(float a) {
  const float e = expf(-fabsf(a));
  return RoundBf16(a > 0.0f ? 1.0f / (1.0f + e) : e / (1.0f + e));
}
__device__ __forceinline__ uint32_t SwishMulBits(uint32_t g_bits, uint32_t u_bits) {  // one BF16 each, in the low 16 bits
  const float g = __uint_as_float(g_bits << 16), u = __uint_as_float(u_bits << 16);
  const float swish = RoundBf16(g * SigmoidBf16(g));
  return static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16(swish * u)));
}
__device__ __forceinline__ uint32_t SwishMulWord(uint32_t g2, uint32_t u2) {  // two BF16 per word
  return SwishMulBits(g2 & 0xFFFFu, u2 & 0xFFFFu) | (SwishMulBits(g2 >> 16, u2 >> 16) << 16);
}

// max / min-nonzero of the two BF16 magnitudes packed in a word
// Measurement aid, compiled in only with -DQFG_PHASE_TIMES: thread 0 of every CTA records the global timer
// at the phase boundaries into GemmParams::phase_times ([CTA][16]).
#ifdef QFG_PHASE_TIMES
__device__ __forceinline__ void Stamp(const GemmParams& p, int slot) {
  if (p.phase_times != nullptr && threadIdx.x == 0) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    p.phase_times[(static_cast<size_t>(blockIdx.y) * gridDim.x + blockIdx.x) * 16 + slot] = t;
  }
}
#else
__device__ __forceinline__ void Stamp(const GemmParams&, int) {}
#endif
__device__ __forceinline__ void TrackWord(uint32_t w, uint32_t& mx, uint32_t& mn) {
  const uint32_t lo = w & 0x7FFFu, hi = (w >> 16) & 0x7FFFu;
  mx = max(mx, max(lo, hi));
  mn = min(mn, min(lo != 0 ? lo : 0x7FFFu, hi != 0 ? hi : 0x7FFFu));
}

// two BF16 values times a power of two, as an FP16 pair (exact when the caller checked the range)
__device__ __forceinline__ uint32_t ScaleToHalf2(uint32_t w, float sc) {
  const float lo = __uint_as_float(w << 16) * sc, hi = __uint_as_float(w & 0xFFFF0000u) * sc;
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// Copies the CTA's K slice of x into shared memory and, for the quantised modes, rescales every
// row by a power of two and converts it to FP16.  WORDS = 4: 16-byte chunks (x 16-byte aligned,
// K % 8 == 0); WORDS = 1: 4-byte pairs (K is even and slices start on multiples of 16, so a pair
// never straddles a slice).  Returns true if the CTA must take the BF16 path.
// Position (in 16-bit elements) of element k of row m of the staged x.  TC = false: rows of `xpitch`
// elements.  TC = true: the K-major no-swizzle operand layout of tcgen05.mma - per k-step 256 bytes,
// two 8-row x 16-byte core matrices (k 0..7, then k 8..15), row m at 16 m bytes inside each.
template <bool TC>
__device__ __forceinline__ int XsIndex(int m, int k, int xpitch) {
  if constexpr (TC) {
    return (k >> 4) * 128 + ((k >> 3) & 1) * 64 + m * 8 + (k & 7);
  } else {
    return m * xpitch + k;
  }
}

// WALK = false keeps the per-item divisions: the register-streaming kernel holds its prefetched weights in
// registers across the staging, and with the walk's state added the compiler's schedule of its K loop lost
// 5 us on the 52 MB BF16 projection (measured), so that kernel stays on the form it was tuned with.
template <int MODE, int WORDS, bool TC = false, bool FUSE = false, bool WALK = true>
__device__ __forceinline__ bool StageXImpl(const GemmParams& p, const Tile& tl, uint16_t* xs, SharedScratch& sh) {
  constexpr int kElems = 2 * WORDS;
  constexpr int kBatch = 4;  // loads in flight per thread (eight measured slower: twice the cold code for one round trip less)
  // a CTA whose K slice is empty (more cluster ranks than k-steps) stages nothing and adds nothing
  if (tl.kslice <= 0) return false;
  const int tid = threadIdx.x, nthreads = blockDim.x, lane = tid & 31;
  const int M = p.M, xpitch = p.xpitch;
  const int kpad = (tl.kslice + 15) & ~15;
  const int chunks = kpad / kElems;
  const int total = M * chunks;
  uint32_t* xw = reinterpret_cast<uint32_t*>(xs);
  // Item idx is chunk (idx % chunks) of row (idx / chunks).  A thread's items are nthreads apart, so it walks
  // (row, k) by a fixed step instead of dividing per item: the staging is a few hundred dependent
  // instructions per warp, and the divisions were a third of them.
  const int step_m = nthreads / chunks, step_k = (nthreads - step_m * chunks) * kElems;
  const int first_m = tid / chunks, first_k = (tid - first_m * chunks) * kElems;
  auto advance = [&](int& m, int& kk) {
    m += step_m;
    kk += step_k;
    if (kk >= kpad) {
      kk -= kpad;
      ++m;
    }
  };

  // pass 1: global -> shared (raw BF16).  All loads of a batch are issued before the first is
  // consumed, so a batch costs one L2 round trip.
  int next_m = first_m, next_k = first_k;
  for (int base0 = 0; base0 < total; base0 += nthreads * kBatch) {  // warp-uniform trip count
    uint32_t v[kBatch][WORDS];
    int st_m = next_m, st_k = next_k;  // the store phase below walks the batch again (cheaper than keeping 2 x kBatch indices)
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      int m, kk;
      if constexpr (WALK) {
        m = next_m;
        kk = next_k;
        advance(next_m, next_k);
      } else {
        const int idx = base0 + tid + j * nthreads;
        m = idx < total ? idx / chunks : M;
        kk = (idx - m * chunks) * kElems;
      }
#pragma unroll
      for (int e = 0; e < WORDS; ++e) v[j][e] = 0;
      if (m < M) {
        if (kk < tl.kslice) {
          const uint16_t* src = p.x + static_cast<size_t>(m) * p.K + tl.kbeg + kk;
          if constexpr (WORDS == 4) {
            const uint4 q = __ldg(reinterpret_cast<const uint4*>(src));
            v[j][0] = q.x, v[j][1] = q.y, v[j][2] = q.z, v[j][3] = q.w;
          } else {
            v[j][0] = __ldg(reinterpret_cast<const uint32_t*>(src));
          }
          if constexpr (FUSE) {  // SharedExpertDown: the row of x is swish_mul(g, u)
            const uint16_t* src2 = p.x2 + static_cast<size_t>(m) * p.K + tl.kbeg + kk;
#pragma unroll
            for (int e = 0; e < WORDS; ++e) v[j][e] = SwishMulWord(v[j][e], __ldg(reinterpret_cast<const uint32_t*>(src2) + e));
          }
        }
      }
    }
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      bool live;
      int m, kk;
      if constexpr (WALK) {
        live = st_m < M;
        m = live ? st_m : 0;
        kk = st_k;
        advance(st_m, st_k);
      } else {
        const int idx = base0 + tid + j * nthreads;
        live = idx < total;
        m = live ? idx / chunks : 0;
        kk = (idx - m * chunks) * kElems;
      }
      if (live) {
        uint32_t* dst = xw + (XsIndex<TC>(m, kk, xpitch) >> 1);
        if constexpr (WORDS == 4) {
          *reinterpret_cast<uint4*>(dst) = make_uint4(v[j][0], v[j][1], v[j][2], v[j][3]);
        } else {
          *dst = v[j][0];
        }
      }
      if constexpr (MODE != kBf16) {
        uint32_t mx = 0, mn = 0x7FFFu;
#pragma unroll
        for (int e = 0; e < WORDS; ++e) TrackWord(v[j][e], mx, mn);
        // lanes of a warp almost always work on the same row: one pair of atomics per warp
        const int m0 = __shfl_sync(0xffffffffu, m, 0);
        if (__all_sync(0xffffffffu, m == m0)) {
          mx = __reduce_max_sync(0xffffffffu, mx);
          mn = __reduce_min_sync(0xffffffffu, mn);
          if (lane == 0) {
            atomicMax(&sh.rmax[m0], mx);
            atomicMin(&sh.rmin[m0], mn);
          }
        } else if (live) {
          atomicMax(&sh.rmax[m], mx);
          atomicMin(&sh.rmin[m], mn);
        }
      }
    }
  }
  if constexpr (MODE == kBf16) {
    __syncthreads();
    return false;
  } else {
    __syncthreads();
    // Power-of-two scale per row that puts the slice maximum in [2^14, 2^15).  Every non-zero
    // element must land in the normal FP16 range: exponent no more than 28 below the maximum's.
    bool ok = !p.force_slow;
#pragma unroll
    for (int m = 0; m < kMaxRows; ++m) {
      if (m < M) {
        const uint32_t a = sh.rmax[m];
        const int e = static_cast<int>(a >> 7);  // BF16 exponent field of the row maximum
        if (a != 0 && (e < 32 || e >= 255 || static_cast<int>(sh.rmin[m] >> 7) < e - 28)) ok = false;
      }
    }
    const bool slow = !ok;
    if (tid < kMaxRows) {
      float sc = 1.f;
      if (!slow && tid < M && sh.rmax[tid] != 0) sc = __uint_as_float((268u - (sh.rmax[tid] >> 7)) << 23);
      sh.scale[tid] = sc;
      sh.inv_scale[tid] = 1.f / sc;
    }
    __syncthreads();
    if (!slow) {
      // pass 2: in place, BF16 -> scaled FP16
      for (int m = first_m, kk = first_k; m < M; advance(m, kk)) {
        const float sc = sh.scale[m];
        uint32_t* px = xw + (XsIndex<TC>(m, kk, xpitch) >> 1);
        if constexpr (WORDS == 4) {
          uint4 q = *reinterpret_cast<uint4*>(px);
          q.x = ScaleToHalf2(q.x, sc);
          q.y = ScaleToHalf2(q.y, sc);
          q.z = ScaleToHalf2(q.z, sc);
          q.w = ScaleToHalf2(q.w, sc);
          *reinterpret_cast<uint4*>(px) = q;
        } else {
          *px = ScaleToHalf2(*px, sc);
        }
      }
      __syncthreads();
    }
    return slow;
  }
}

// Asynchronous staging of x for the warp-ring kernel.  The x loads of the staging above are issued after the
// ring prologue and queue behind its weight copies (50 - 130 KB per SM, one to three microseconds of the SM's
// share of the bandwidth) while every warp waits for them.  Here the CTA's K slice of x is copied raw into its
// place in shared memory with 16-byte cp.async BEFORE the weight copies are issued - the copy group is the
// oldest, so `cp.async.wait_group <weight groups>` completes it - and converted in place afterwards, while the
// weights are in flight.  Needs 16-byte rows of x (x 16-byte aligned, K % 8 == 0).
__device__ __forceinline__ bool XRowsAre16ByteAligned(const GemmParams& p) {
  return (reinterpret_cast<uintptr_t>(p.x) % 16 == 0) && (p.K % 8 == 0);
}
// Which 16-byte items of the staged x a thread handles.  A warp works on one row at a time (warp w on row
// w mod M, the warps of a row sharing its items; with fewer warps than rows, on rows w, w + warps, ...), so a
// row's maximum is reduced once per warp, and nothing here divides per item.  f(live, kk): elements kk .. kk + 7
// of the row, `live` false past the row's end (the trip count is warp-uniform); row_done(m) after each row.
template <class F, class G>
__device__ __forceinline__ void ForMyXItems(const GemmParams& p, const Tile& tl, F&& f, G&& row_done) {
  const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5, M = static_cast<unsigned>(p.M);
  const int chunks = ((tl.kslice + 15) & ~15) >> 3;
  const unsigned part = warp / M, row0 = warp - part * M;
  const unsigned cnt = nwarps > M ? (nwarps - row0 + M - 1) / M : 1u;  // warps that share row0
#pragma unroll 1
  for (unsigned m = row0; m < M; m += nwarps) {
#pragma unroll 1
    for (int c0 = static_cast<int>(32u * part); c0 < chunks; c0 += static_cast<int>(32u * cnt)) {
      const int c = c0 + static_cast<int>(lane);
      f(c < chunks, static_cast<int>(m), c * 8);
    }
    row_done(static_cast<int>(m));
  }
}
__device__ __forceinline__ void XCopyIssue(const GemmParams& p, const Tile& tl, uint16_t* xs) {
  if (tl.kslice <= 0) return;
  const uint32_t base = SmemAddr(xs);
  ForMyXItems(
      p, tl,
      [&](bool live, int m, int kk) {
        if (!live) return;
        const bool in = kk < tl.kslice;  // the slice is padded to whole k-steps with zeros
        const uint16_t* src = p.x + static_cast<size_t>(m) * p.K + tl.kbeg + kk;
        CpAsync16(base + static_cast<uint32_t>(m * p.xpitch + kk) * 2u, in ? src : p.x, in ? 16 : 0);
      },
      [](int) {});
}
// Second half: every thread's copies have completed (cp.async.wait_group).  Must be called by every thread of
// the CTA.  Returns true if the CTA must take the BF16 path.
template <int MODE>
__device__ __forceinline__ bool StageXConvert(const GemmParams& p, const Tile& tl, uint16_t* xs, SharedScratch& sh) {
  const int tid = threadIdx.x, lane = tid & 31, M = p.M;
  if (tid < kMaxRows) {
    sh.rmax[tid] = 0;
    sh.rmin[tid] = 0x7FFFu;
    sh.inv_scale[tid] = 1.f;
  }
  __syncthreads();  // the raw rows are visible to every thread
  if constexpr (MODE == kBf16) {
    return false;
  } else {
    if (tl.kslice <= 0) return false;
    uint32_t* xw = reinterpret_cast<uint32_t*>(xs);
    uint32_t mx = 0, mn = 0x7FFFu;
    ForMyXItems(
        p, tl,
        [&](bool live, int m, int kk) {
          if (live) {
            const uint4 q = *reinterpret_cast<const uint4*>(xw + ((m * p.xpitch + kk) >> 1));
            TrackWord(q.x, mx, mn);
            TrackWord(q.y, mx, mn);
            TrackWord(q.z, mx, mn);
            TrackWord(q.w, mx, mn);
          }
        },
        [&](int m) {
          mx = __reduce_max_sync(0xffffffffu, mx);
          mn = __reduce_min_sync(0xffffffffu, mn);
          if (lane == 0) {
            atomicMax(&sh.rmax[m], mx);
            atomicMin(&sh.rmin[m], mn);
          }
          mx = 0;
          mn = 0x7FFFu;
        });
    __syncthreads();
    // Power-of-two scale per row that puts the slice maximum in [2^14, 2^15).  Every non-zero element must
    // land in the normal FP16 range: exponent no more than 28 below the maximum's.
    bool ok = !p.force_slow;
#pragma unroll 1
    for (int m = 0; m < M; ++m) {
      const uint32_t a = sh.rmax[m];
      const int e = static_cast<int>(a >> 7);  // BF16 exponent field of the row maximum
      if (a != 0 && (e < 32 || e >= 255 || static_cast<int>(sh.rmin[m] >> 7) < e - 28)) ok = false;
    }
    const bool slow = !ok;
    auto scale_of = [&](int m) {
      const uint32_t a = sh.rmax[m];
      return (!slow && a != 0) ? __uint_as_float((268u - (a >> 7)) << 23) : 1.f;
    };
    if (tid < M) {  // for the epilogue, which runs behind further barriers
      const float sc = scale_of(tid);
      sh.scale[tid] = sc;
      sh.inv_scale[tid] = 1.f / sc;
    }
    if (!slow) {
      float sc = 1.f;
      int sc_row = -1;
      ForMyXItems(
          p, tl,
          [&](bool live, int m, int kk) {
            if (!live) return;
            if (m != sc_row) {
              sc = scale_of(m);
              sc_row = m;
            }
            uint4* px = reinterpret_cast<uint4*>(xw + ((m * p.xpitch + kk) >> 1));
            uint4 q = *px;
            q.x = ScaleToHalf2(q.x, sc);
            q.y = ScaleToHalf2(q.y, sc);
            q.z = ScaleToHalf2(q.z, sc);
            q.w = ScaleToHalf2(q.w, sc);
            *px = q;
          },
          [](int) {});
    }
    __syncthreads();
    return slow;
  }
}

// SharedExpertDown's staging: the gate of every row, then x = swish_mul(g, u) staged like a plain x.  Kept
// out of line: the streaming kernels were measured to slow down by several percent whenever code was added
// to their inlined body, executed or not, so everything this op adds to them is one call on a cold branch.
template <int MODE, bool TC>
__device__ __noinline__ bool StageXFused(const GemmParams& p, const Tile& tl, uint16_t* xs, SharedScratch& sh) {
  // gate logit of every row: thread-strided partial sums, warps in order, then bf16 -> sigmoid -> bf16.  All rows
  // at once - a thread reads a 16-byte chunk of gw and the same chunk of every row of gx before it adds anything -
  // so the gate costs one round trip to L2, not one per row (one row at a time took 1.7 us per row).
  const int tid = threadIdx.x, nthreads = blockDim.x, warp = tid >> 5, lane = tid & 31;
  const int M = p.M;
  float part[kMaxRows];
#pragma unroll
  for (int m = 0; m < kMaxRows; ++m) part[m] = 0.f;
  const bool gvec = (reinterpret_cast<uintptr_t>(p.gx) % 16 == 0) && (reinterpret_cast<uintptr_t>(p.gw) % 16 == 0) && (p.gk % 8 == 0);
  if (gvec) {
    const int chunks = p.gk >> 3;
    const uint4* gw4 = reinterpret_cast<const uint4*>(p.gw);
#pragma unroll 1
    for (int c = tid; c < chunks; c += nthreads) {
      const uint4 w = __ldg(gw4 + c);
      uint4 xv[kMaxRows];
#pragma unroll
      for (int m = 0; m < kMaxRows; ++m) {
        if (m < M) xv[m] = __ldg(reinterpret_cast<const uint4*>(p.gx + static_cast<size_t>(m) * p.gk) + c);
      }
      const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int m = 0; m < kMaxRows; ++m) {
        if (m < M) {
          const uint32_t xx[4] = {xv[m].x, xv[m].y, xv[m].z, xv[m].w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {  // elements in index order
            part[m] += __uint_as_float(xx[e] << 16) * __uint_as_float(ww[e] << 16);
            part[m] += __uint_as_float(xx[e] & 0xFFFF0000u) * __uint_as_float(ww[e] & 0xFFFF0000u);
          }
        }
      }
    }
  } else {
    for (int m = 0; m < M; ++m) {
      float acc = 0.f;
      const uint16_t* gxm = p.gx + static_cast<size_t>(m) * p.gk;
      for (int i = tid; i < p.gk; i += nthreads)
        acc += __uint_as_float(static_cast<uint32_t>(gxm[i]) << 16) * __uint_as_float(static_cast<uint32_t>(p.gw[i]) << 16);
      part[m] = acc;
    }
  }
#pragma unroll
  for (int m = 0; m < kMaxRows; ++m) {
    if (m < M) {  // warp-uniform
      float v = part[m];
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
      if (lane == 0) sh.best_v[warp][m] = v;
    }
  }
  __syncthreads();
  if (tid < kMaxRows) {
    float logit = 0.f;
    if (tid < p.M)
      for (int w = 0; w < (nthreads >> 5); ++w) logit += sh.best_v[w][tid];
    sh.gate[tid] = SigmoidBf16(RoundBf16(logit));
  }
  __syncthreads();
  // swish_mul reads x2 with the same vector width as x
  const bool vec8 = (reinterpret_cast<uintptr_t>(p.x) % 16 == 0) && (p.K % 8 == 0) && (reinterpret_cast<uintptr_t>(p.x2) % 16 == 0);
  if (vec8) return StageXImpl<MODE, 4, TC, true>(p, tl, xs, sh);
  return StageXImpl<MODE, 1, TC, true>(p, tl, xs, sh);
}

// Must be called by every thread of the CTA; sh.rmax / sh.rmin are initialised here.
template <int MODE, bool TC = false, bool WALK = true, bool FUSE = false>
__device__ __forceinline__ bool StageX(const GemmParams& p, const Tile& tl, uint16_t* xs, SharedScratch& sh) {
  if (threadIdx.x < kMaxRows) {
    sh.rmax[threadIdx.x] = 0;
    sh.rmin[threadIdx.x] = 0x7FFFu;
    sh.inv_scale[threadIdx.x] = 1.f;
  }
  __syncthreads();
  if constexpr (FUSE) return StageXFused<MODE, TC>(p, tl, xs, sh);
  const bool vec8 = (reinterpret_cast<uintptr_t>(p.x) % 16 == 0) && (p.K % 8 == 0);
  if (vec8) return StageXImpl<MODE, 4, TC, false, WALK>(p, tl, xs, sh);
  return StageXImpl<MODE, 1, TC, false, WALK>(p, tl, xs, sh);
}

// Position of column c of row m inside a row of the partial-sum array.  An MMA accumulator fragment puts the
// lanes of a warp 16 (or 8) columns apart in rows 2t and 2t + 1, and a row is a multiple of 32 floats long, so
// plain indexing made the 8-byte stores of a warp collide 8- to 16-way.  The exclusive-or moves column bits
// 5-6 and row bits 1-2 into the bank bits (1-4) and stays inside the aligned group of 32 columns.
__device__ __forceinline__ int RedCol(int c, int m) { return c ^ ((((c >> 5) & 3) << 1) ^ (((m >> 1) & 3) << 3)); }

// The part of the epilogue that starts from the partial sums in shared memory: `red` holds
// [nparts][M][TNc] floats (part w = the sum over the k-steps of K-group w), the cluster partials
// follow it.  Every thread of the CTA must call this after a __syncthreads() that follows the
// last write to `red`.
template <int MODE, bool FUSE = false>
__device__ __forceinline__ void EpilogueTail(const GemmParams& p, const Tile& tl, uint8_t* smem, SharedScratch& sh,
                                             int nparts, int TNc) {
  const int tid = threadIdx.x, nthreads = blockDim.x;
  const int warp = tid >> 5, lane = tid & 31;
  const int M = p.M, C = tl.C, n0 = tl.n0, n1 = tl.n1;
  const Segment& sg = p.seg[tl.seg];
  float* red = reinterpret_cast<float*>(smem);
  float* part = red + static_cast<size_t>(nparts) * M * TNc;
  const int ncols = n1 - n0;  // valid columns of the tile (<= TNc)
  // Fused argmax: rows are finished one at a time, so a thread carries the best (value, index) of the row in
  // hand only, and flush_row leaves the warp's best of that row in shared memory.  One copy of this code
  // serves every row: the epilogue runs once, from a cold instruction cache, and an eight-way unrolled form
  // of it was measured at 1.7 us per row.
  float cur_v = 0.f;
  long long cur_i = -1;
  // what every element needs from the parameter block, read once
  const float* const w_scale = sg.w_scale;
  const bool lm = p.lm != 0;
  const int out_begin = sg.out_begin, out_end = sg.out_end;
  const bool store = !lm || p.out[out_begin] != nullptr;
  const long long col_offset = p.lm_col_offset;
  auto finalize = [&](int m, int c, float v) {
    const int n = n0 + c;
    if (w_scale != nullptr) v *= w_scale[n];
    if constexpr (FUSE) {
      // SharedExpertDown: routed + bf16(bf16(sum) * gate), every step rounded to BF16 (skinny_gemm.cuh:226-240)
      const float shared = RoundBf16(RoundBf16(v) * sh.gate[m]);
      v = p.routed != nullptr ? __uint_as_float(static_cast<uint32_t>(p.routed[static_cast<size_t>(m) * sg.n + n]) << 16) + shared
                              : shared;
    }
    const __nv_bfloat16 b = __float2bfloat16(v);
    if (store) {
      int j = out_begin;
      for (int i = j + 1; i < out_end; ++i) {
        if (n >= p.col_begin[i]) j = i;
      }
      p.out[j][static_cast<size_t>(m) * p.width[j] + (n - p.col_begin[j])] = __bfloat16_as_ushort(b);
    }
    if (lm) {
      // a thread meets the columns of a row in increasing order: strict comparison, a NaN is never replaced
      const float f = __bfloat162float(b);
      if (cur_i < 0 || f > cur_v || (f != f && cur_v == cur_v)) {
        cur_v = f;
        cur_i = col_offset + n;
      }
    }
  };
  // The warp's best of row m joins the CTA's best of that row: keys (argmax_key.cuh), two redux per warp, one
  // shared-memory atomicMax.
  auto flush_row = [&](int m) {
    if (!lm) return;
    const unsigned long long key = WarpMaxKey(cur_i < 0 ? 0ull : PackKey(cur_v, cur_i));
    if (lane == 0 && key != 0ull) atomicMax(&sh.rowkey[m], key);
    cur_v = 0.f;
    cur_i = -1;
  };
  if (tid < kMaxRows) sh.rowkey[tid] = 0ull;
  __syncthreads();

  // All rows are finished side by side: a warp works on one row at a time - wpr warps per row, every lane on
  // columns 32 wpr apart in increasing order - so the rows' shared-memory (or cluster) round trips overlap
  // instead of following one another, and a warp reduces its candidates once per row it touches.
  const int nwarps = nthreads >> 5;
  const int wpr = max(1, nwarps / M), rows_per_pass = max(1, nwarps / wpr);
  const int my_row = warp / wpr, my_part = warp - my_row * wpr;
  auto for_my_columns = [&](int share, auto&& value) {  // value(m, j): column j of this CTA's share, 0 <= j < share
    for (int m0 = 0; m0 < M; m0 += rows_per_pass) {
      const int m = m0 + my_row;
      if (my_row < rows_per_pass && m < M) {
        for (int j = my_part * 32 + lane; j < share; j += wpr * 32) value(m, j);
        flush_row(m);
      }
    }
  };

  if (C == 1) {
    for_my_columns(ncols, [&](int m, int c) {
      float sum = 0.f;
      for (int w = 0; w < nparts; ++w) sum += red[(w * M + m) * TNc + RedCol(c, m)];
      finalize(m, c, sum * sh.inv_scale[m]);
    });
  } else {
    for (int m = 0; m < M; ++m) {
      const float inv = sh.inv_scale[m];
      for (int c = tid; c < TNc; c += nthreads) {
        float sum = 0.f;
        for (int w = 0; w < nparts; ++w) sum += red[(w * M + m) * TNc + RedCol(c, m)];
        part[m * TNc + c] = sum * inv;
      }
    }
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    const int cper = (TNc + C - 1) / C;  // the last rank's share may be short (any C <= 8)
    const int cb = tl.crank * cper;
    const int share = max(0, min(cper, ncols - cb));
    // The C partial sums of an output come from C CTAs' shared memory: all eight possible loads are issued
    // before the first is used (one round trip through the cluster network instead of C), then added in rank order.
    for_my_columns(share, [&](int m, int j) {
      const int idx = m * TNc + cb + j;
      float v[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) v[r] = r < C ? cluster.map_shared_rank(part, r)[idx] : 0.f;
      float sum = 0.f;
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        if (r < C) sum += v[r];
      }
      finalize(m, cb + j, sum);
    });
    cluster.sync();
  }

  if (p.lm) {
    // The warps' bests of every row (flush_row) folded into the workspace keys with a 64-bit atomic max.
    auto fold_into_keys = [&]() {
      __syncthreads();
      if (tid < M) {
        const unsigned long long best = sh.rowkey[tid];
        sh.rowkey[tid] = 0ull;
        if (best != 0ull) atomicMax(p.lm_keys + tid, best);
        __threadfence();
      }
      __syncthreads();
    };
    fold_into_keys();
    if (tid == 0) {
      const unsigned int total = gridDim.x * gridDim.y;
      const unsigned int prev = atomicAdd(p.lm_count, 1u);
      sh.last = (prev == total - 1) ? 1 : 0;
      __threadfence();
    }
    __syncthreads();
    if (sh.last) {
      unsigned long long tail_best = 0ull;  // thread m < M: best key of row m among the shared columns
      if (p.tail_groups > 0) {
        // the partial sums of the shared columns were stored before their CTAs counted themselves in:
        // add the K slices up in order, finish those columns and fold their best into the keys
        __threadfence();
        const int n_main = sg.n - p.tail_groups * 128;
        const int tcols = p.tail_groups * 128;
        // This runs after every other CTA has finished, so it is all on the critical path.  One output (row,
        // shared column) per thread and pass: all its slices are loaded before the first is added (one round
        // trip to L2), still in slice order.  A group is 128 columns wide, so the 32 outputs of a warp belong
        // to one row, which flush_row needs.
        const int outs = M * tcols;
        for (int o = tid; o < outs; o += nthreads) {
          const int m = o / tcols, j = o - m * tcols;
          const float* src = p.lm_tail + (static_cast<size_t>(j >> 7) * p.tail_split * kMaxRows + m) * 128 + (j & 127);
          float part[kMaxTailSplit];
#pragma unroll
          for (int c = 0; c < kMaxTailSplit; ++c) part[c] = c < p.tail_split ? __ldcg(src + static_cast<size_t>(c) * kMaxRows * 128) : 0.f;
          float sum = 0.f;
#pragma unroll
          for (int c = 0; c < kMaxTailSplit; ++c) sum += part[c];
          finalize(m, n_main + j - n0, sum * sh.inv_scale[m]);
          flush_row(m);
        }
        // no other CTA is left to see these keys: they join the global ones in registers below
        __syncthreads();
        if (tid < M) tail_best = sh.rowkey[tid];
      }
      unsigned long long key = 0ull;  // thread m < M: the winning key of row m
      if (p.xworld > 1) {
        // Sharded head: this rank's keys go straight into every rank's exchange buffer (peer memory) as
        // self-validating words - (upper or lower half of the key) << 32 | call count - so that one round of
        // 8-byte stores carries both the data and the signal that it has arrived: no fence, no separate flag.
        // Slots alternate with the parity of the call count: a rank that is one call ahead writes the other
        // slot.  Every rank then awaits - bounded - the words of all ranks in its own buffer and folds them;
        // the maximum of the order-preserving keys is the Better order, so every rank ends with the same
        // winner.  A wait that runs out sets the buffer's status and the row is folded without that peer.
        LmExchange* own = p.xpeer[p.xrank];
        const unsigned int epoch = own->epoch + 1;  // every thread reads it before thread 0 advances it below
        const int par = static_cast<int>(epoch & 1u);
        if (tid < M) {
          unsigned long long mine = atomicExch(p.lm_keys + tid, 0ull);
          sh.best_i[0][tid] = static_cast<long long>(tail_best > mine ? tail_best : mine);
        }
        if (tid == 0) sh.xfail = 0;
        __syncthreads();
        unsigned long long t_ready = 0, t_sent = 0;
        if (tid == 0) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_ready));
        const int nwords = 2 * M * p.xworld;
        for (int w = tid; w < nwords; w += nthreads) {
          const int r = w / (2 * M), rem = w - r * 2 * M, row = rem >> 1, half = rem & 1;
          const unsigned long long k = static_cast<unsigned long long>(sh.best_i[0][row]);
          const unsigned long long payload = half ? (k & 0xFFFFFFFFull) : (k >> 32);
          *reinterpret_cast<volatile unsigned long long*>(&p.xpeer[r]->words[par][p.xrank][row][half]) = (payload << 32) | epoch;
        }
        if (tid == 0) {
          own->epoch = epoch;
          asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_sent));
        }
        for (int w = tid; w < nwords; w += nthreads) {
          const int r = w / (2 * M), rem = w - r * 2 * M, row = rem >> 1, half = rem & 1;
          const volatile unsigned long long* word = &own->words[par][r][row][half];
          int spin = 0;
          while (static_cast<unsigned int>(*word) != epoch && spin < p.xspin) {
            ++spin;
            __nanosleep(32);
          }
          if (static_cast<unsigned int>(*word) != epoch) {
            own->status = 1;
            sh.xfail = 1;
          }
        }
        __syncthreads();
        if (tid < M) {
          for (int r = 0; r < p.xworld; ++r) {
            const unsigned long long w0 = *reinterpret_cast<const volatile unsigned long long*>(&own->words[par][r][tid][0]);
            const unsigned long long w1 = *reinterpret_cast<const volatile unsigned long long*>(&own->words[par][r][tid][1]);
            const bool arrived = static_cast<unsigned int>(w0) == epoch && static_cast<unsigned int>(w1) == epoch;
            const unsigned long long k = (w0 & 0xFFFFFFFF00000000ull) | (w1 >> 32);
            if (arrived && k > key) key = k;
          }
        }
        if (tid == 0) {
          // telemetry of the owner's last call: keys ready, stores issued, all words seen (or given up on)
          unsigned long long t_done;
          asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_done));
          own->t_ready = t_ready;
          own->t_sent = t_sent;
          own->t_done = t_done;
          if (p.lm_status_out != nullptr) *p.lm_status_out = static_cast<unsigned int>(sh.xfail);
        }
      } else if (tid < M) {
        key = atomicExch(p.lm_keys + tid, 0ull);
        key = tail_best > key ? tail_best : key;
      }
      if (tid < M) {
        if (p.lm_idx != nullptr) p.lm_idx[tid] = KeyIndex(key);
        if (p.lm_val != nullptr) p.lm_val[tid] = KeyValue(key);
        if (p.lm_key_out != nullptr) p.lm_key_out[tid] = key;
      }
      if (tid == 0) *p.lm_count = 0u;
    }
  }
}

// The accumulators of a consumer warp to its place among the partial sums in `smem`.
template <int MODE, int W = 1>
__device__ __forceinline__ void StorePartials(const GemmParams& p, const Tile& tl, float (&acc)[Geom<MODE, W>::kMmas][4], uint8_t* smem,
                                              bool warp_has_cols) {
  using G = Geom<MODE, W>;
  constexpr int NM = G::kMmas;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int wn = warp % p.wn, wk = warp / p.wn;
  const int M = p.M;
  const int cols_per_warp = 8 * G::kColsPerThread * W;
  const int TNc = p.wn * cols_per_warp;
  float* red = reinterpret_cast<float*>(smem);
  if (warp_has_cols) {
#pragma unroll
    for (int j = 0; j < NM; ++j) {
      // MMA j covers columns 2 (j % 8), +1 of the thread's (j / 8)-th column group (128 columns apart)
      const int per_group = G::kMmas / W;
      const int cl = wn * cols_per_warp + (j / per_group) * 8 * G::kColsPerThread + g * G::kColsPerThread + 2 * (j % per_group);
      const int m0 = 2 * t, m1 = 2 * t + 1;
      if (m0 < M) *reinterpret_cast<float2*>(&red[(wk * M + m0) * TNc + RedCol(cl, m0)]) = make_float2(acc[j][0], acc[j][2]);
      if (m1 < M) *reinterpret_cast<float2*>(&red[(wk * M + m1) * TNc + RedCol(cl, m1)]) = make_float2(acc[j][1], acc[j][3]);
    }
  } else {
    for (int m = 0; m < M; ++m)
      for (int c = lane; c < cols_per_warp; c += 32) red[(wk * M + m) * TNc + wn * cols_per_warp + c] = 0.f;
  }
}

// Reduction of the accumulators (wk warps, then the cluster), scaling, rounding, stores, and the
// fused argmax.  `smem` is reused for the partial sums; every thread of the CTA must call this
// after a __syncthreads() that ends all use of the shared memory by the main loop.
template <int MODE, int W = 1, bool FUSE = false>
__device__ __forceinline__ void Epilogue(const GemmParams& p, const Tile& tl, float (&acc)[Geom<MODE, W>::kMmas][4],
                                         uint8_t* smem, SharedScratch& sh, bool warp_has_cols) {
  StorePartials<MODE, W>(p, tl, acc, smem, warp_has_cols);
  __syncthreads();
  EpilogueTail<MODE, FUSE>(p, tl, smem, sh, p.wk, p.wn * 8 * Geom<MODE, W>::kColsPerThread * W);
}

}  // namespace
}  // namespace qfg
