// SkinnyGemm for up to eight rows, the weights streamed by tensor copies.
//
// One CTA per SM owns a column tile of one weight and one of `cluster` slices of K.  One lane of a producer warp copies
// boxes of R weight rows by the tile's width into a ring that fills the SM's shared memory; teams of wn x wk consumer
// warps take the stages in turn, warp (i, j) of a team the columns of its 128 bytes (64 for NVFP4) and k-steps j and j + wk
// of a stage, with the arithmetic of skinny_common.cuh.  The producer waits for nobody until the ring is full, so x is staged and converted
// while the first 200 KB per SM are on their way, and what is left of the call is the stream and the epilogue.
//
// Why tensor copies: one instruction fetches a whole box.  A copy-only kernel of this shape streams 52 MB in 10.4 us and
// the 437 MB LM head in 69 us, launch included, against 96 us for the rings of 16-byte cp.async copies that each warp
// issued for itself; they need 8 KB or more per copy instruction (boxes of 16 rows by 64 bytes reach 0.9 TB/s).
//
// Layout of a stage: R rows of `pitch` bytes, then (NVFP4) R rows of `spitch` bytes that hold the rows' block scales.
// A lane (g, t) reads rows 2t, 2t + 1, 2t + 8 and 2t + 9 of a k-step, 16 bytes (NVFP4: 8) at g: the rows of a quarter
// (half) warp have to lie 32 (64) bytes apart in the banks, which an odd number of 16-byte pieces per row gives, so boxes
// of an even number are copied one piece wider (swizzling would need boxes of exactly 128 bytes).
// NVFP4 weights whose N is an odd multiple of 128 have rows an odd multiple of eight bytes long: two rows are then one row
// of the tensor map, a stage holds R / 2 even rows and R / 2 odd rows, the latter copied from the 16-byte boundary before
// them, and `pitch` is 32 or 96 modulo 128.
//
// Every wait is bounded; a CTA that gives up on one writes NaN.
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <climits>
#include <cstdio>
#include <mutex>
#include <type_traits>

#include "skinny_common.cuh"
#include "swish.cuh"
#include "tensor_map.h"

namespace qfg {
namespace {

constexpr int kStreamWarps = 18;                             // consumers, at most
constexpr int kStreamThreads = 32 * (kStreamWarps + 2);      // and the producer, and the LM head's tail warp
constexpr int kStreamStages = 24;
constexpr int kStreamSpin = 1 << 20;  // tries of a wait, each suspended by the hardware for a while

struct StreamParams {
  GemmParams g;
  CUtensorMap wmap[kMaxSeg];  // stored rows (nibbles of NVFP4) in elements of eight bytes
  CUtensorMap smap[kMaxSeg];  // NVFP4 block scales
  CUtensorMap tail_wmap, tail_smap;
  int warps;                  // consumers: teams * wk * wn
  int teams, team_warps, team_wk, team_inv;  // team t takes stages t, t + teams, ...; 65536 / team_warps, rounded up
  int wn_inv;                 // 65536 / wn, rounded up
  int rows;                   // R = 32 team_wk
  int nstages;                // stages of the whole K range
  int odd;                    // rows in pairs (see above)
  int boxes, col_boxes;       // per stage (and half): boxes of box_rows rows, side by side the boxes of a swizzled tile
  int swizzle;                // 0, or the bytes of a swizzled box's rows
  uint32_t box_rows, pitch, spitch, half, shalf, scale_off, tx;
  int row_warps, row_pass, row_inv;  // how the consumer warps share the rows of x (ShareOf)
  int rank_cols;              // cluster: columns of the tile that a rank finishes
  uint32_t x_off;             // staged x in shared memory
  uint32_t tail_off, tail_pitch, tail_tx, tail_rows;
};

struct StreamCtl {
  unsigned long long full[kStreamStages], empty[kStreamStages], tail_full, x_full;
  volatile uint32_t fault;
};

__device__ __forceinline__ void BarInit(uint32_t a, int n) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(n) : "memory"); }
__device__ __forceinline__ void BarArrive(uint32_t a) {
  asm volatile("{ .reg .b64 st; mbarrier.arrive.shared::cta.b64 st, [%0]; }" ::"r"(a) : "memory");
}
__device__ __forceinline__ void BarExpect(uint32_t a, uint32_t bytes) {
  asm volatile("{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1; }" ::"r"(a), "r"(bytes) : "memory");
}
// False if the wait ran out, or spun while another wait of this CTA had.  True says nothing of the other waits: a copy that has
// landed is taken whatever became of the rest.
__device__ __forceinline__ bool BarWait(uint32_t a, uint32_t parity, StreamCtl& c) {
  for (int i = 0; i < kStreamSpin; ++i) {
    uint32_t ok;
    asm volatile("{ .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(a), "r"(parity) : "memory");
    if (ok) return true;
    if ((i & 255) == 255 && c.fault) return false;
  }
  c.fault = 1;
  return false;
}
// x in elements of eight bytes, an even number: a copy starts on 16 bytes
__device__ __forceinline__ void TmaLoad(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst), "l"(map),
               "r"(bar), "r"(x), "r"(y)
               : "memory");
}
// `bytes` contiguous bytes, a multiple of sixteen, from and to sixteen-byte boundaries
__device__ __forceinline__ void BulkLoad(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ bool ElectOne() {
  uint32_t yes;
  asm volatile("{ .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(yes)::"memory");
  return yes != 0;
}
// the B fragments of two k-steps: k-step a in v[0], v[1], k-step b in v[2], v[3]
__device__ __forceinline__ void LoadX2(uint32_t addr, uint32_t (&v)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(addr));
}

// Where a lane finds its rows: `w` the first of them in a k-step at the start of a region, d1 and d2 from row 2t to 2t + 1 and
// to 2t + 8, `step` from a k-step to the next; s, e1, e2, sstep the same of the scales.
struct LaneRows {
  uint32_t w, d1, d2, step, s, e1, e2, sstep;
};
template <int MODE>
__device__ __forceinline__ LaneRows RowsOf(const Segment& sg, int n0, int col_warp, int lane, int odd, uint32_t pitch, uint32_t spitch, uint32_t half,
                                           uint32_t shalf, int swizzle = 0, uint32_t rows = 0) {
  const int g = lane >> 2, t = lane & 3;
  LaneRows r;
  const uint32_t row = static_cast<uint32_t>(odd ? t : 2 * t), per = odd ? 4u : 8u;
  r.w = row * pitch + static_cast<uint32_t>(MODE == kNvfp4 ? col_warp * 64 + g * 8 : col_warp * 128 + g * 16);
  r.d1 = odd ? half + (static_cast<uint32_t>(sg.pitch) & 8u) : pitch;
  r.d2 = per * pitch;
  r.step = 2 * per * pitch;
  if (swizzle == 128) {  // pieces of 16 bytes exclusive-or the row, modulo eight
    const int piece = MODE == kNvfp4 ? (col_warp & 1) * 4 + (g >> 1) : g, at = piece ^ (2 * t);
    r.w = static_cast<uint32_t>(MODE == kNvfp4 ? col_warp >> 1 : col_warp) * rows * 128u + row * 128u + static_cast<uint32_t>(at * 16 + (MODE == kNvfp4 ? (g & 1) * 8 : 0));
    r.d1 = 128u + static_cast<uint32_t>(((at ^ 1) - at) * 16);
  } else if (swizzle == 64) {  // pieces exclusive-or half the row, modulo four (NVFP4, one group)
    r.w = row * 64u + static_cast<uint32_t>(((g >> 1) ^ t) * 16 + (g & 1) * 8);
  }
  const uint32_t scl = static_cast<uint32_t>(sg.n >> 1) + static_cast<uint32_t>(n0 >> 4), shift = scl & 8u;
  r.s = row * spitch + static_cast<uint32_t>(col_warp * 8 + g) + shift;
  r.e1 = odd ? shalf + ((scl + static_cast<uint32_t>(sg.pitch)) & 8u) - shift : spitch;
  r.e2 = per * spitch;
  r.sstep = 2 * per * spitch;
  return r;
}
template <int MODE>
__device__ __forceinline__ void LoadRows(Raw<MODE>& raw, const LaneRows& r, uint32_t w, uint32_t s) {
  if constexpr (MODE == kNvfp4) {
    raw.r[0][0] = Lds64(w);
    raw.r[0][1] = Lds64(w + r.d1);
    raw.r[0][2] = Lds64(w + r.d2);
    raw.r[0][3] = Lds64(w + r.d1 + r.d2);
    raw.s[0][0] = Lds8(s);
    raw.s[0][1] = Lds8(s + r.e1);
    raw.s[0][2] = Lds8(s + r.e2);
    raw.s[0][3] = Lds8(s + r.e1 + r.e2);
  } else {
    raw.r[0] = Lds128(w);
    raw.r[1] = Lds128(w + r.d1);
    raw.r[2] = Lds128(w + r.d2);
    raw.r[3] = Lds128(w + r.d1 + r.d2);
  }
}

// max and min of the non-zero of eight packed BF16 magnitudes, two at a time (min is kept less one, so that zero is never it)
__device__ __forceinline__ void TrackPair(uint32_t w, uint32_t& mx, uint32_t& mn) {
  w &= 0x7FFF7FFFu;
  mx = __vmaxu2(mx, w);
  mn = __vminu2(mn, __vsub2(w, 0x00010001u));
}
__device__ __forceinline__ uint4 ScaleToHalf8(uint4 v, float sc) {
  return make_uint4(ScaleToHalf2(v.x, sc), ScaleToHalf2(v.y, sc), ScaleToHalf2(v.z, sc), ScaleToHalf2(v.w, sc));
}

// the other way round: FP16 values times a power of two, exact where the products are normal FP16 numbers
__device__ __forceinline__ uint32_t RescaleHalf2(uint32_t w, float ratio) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
  const __half2 h = __floats2half2_rn(f.x * ratio, f.y * ratio);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ uint4 RescaleHalf8(uint4 v, float ratio) {
  return make_uint4(RescaleHalf2(v.x, ratio), RescaleHalf2(v.y, ratio), RescaleHalf2(v.z, ratio), RescaleHalf2(v.w, ratio));
}
// Whether one of eight FP16 magnitudes is below that of the bits `least`, or not finite.
__device__ __forceinline__ bool LostInHalf(uint4 v, uint32_t least) {
  v = make_uint4(v.x & 0x7FFF7FFFu, v.y & 0x7FFF7FFFu, v.z & 0x7FFF7FFFu, v.w & 0x7FFF7FFFu);
  const uint32_t mx = __vmaxu2(__vmaxu2(v.x, v.y), __vmaxu2(v.z, v.w)), mn = __vminu2(__vminu2(v.x, v.y), __vminu2(v.z, v.w));
  return max(mx & 0xFFFFu, mx >> 16) >= 0x7C00u || min(mn & 0xFFFFu, mn >> 16) < least;
}

struct StreamScratch {
  uint32_t xmax[kMaxRows][kStreamWarps], xmin[kMaxRows][kStreamWarps];
  float gate[kMaxRows][2];  // SharedExpertDown: the two halves of the gate's sum
};

// The consumer warps side by side on the rows of the call: `wpr` of them per row, `rpp` rows at a time.
struct RowShare {
  int row, part, wpr, rpp;
  bool any;
};
__device__ __forceinline__ RowShare ShareOf(const StreamParams& q, int warp) {
  RowShare r;
  r.wpr = q.row_warps;
  r.rpp = q.row_pass;
  r.row = (warp * q.row_inv) >> 16;  // warp / wpr
  r.part = warp - r.row * r.wpr;
  r.any = r.row < r.rpp && warp < q.warps;
  return r;
}

// x in FP16, the usual way: times 2^10, in one look at it.  Exact for zero and for magnitudes from 2^-27 (eight significant bits,
// the last of them FP16's smallest number after the scaling) to 2^6.
constexpr float kUsualScale = 1024.f;
constexpr uint32_t kUsualLeast = 127 - 27, kUsualMost = 127 + 5;  // exponent fields
__device__ __forceinline__ void Track(const uint4& v, uint32_t& mx, uint32_t& mn) {
  TrackPair(v.x, mx, mn);
  TrackPair(v.y, mx, mn);
  TrackPair(v.z, mx, mn);
  TrackPair(v.w, mx, mn);
}
__device__ __forceinline__ bool Unusual(uint32_t mx, uint32_t mn) {  // what Track saw
  const uint32_t most = max(mx & 0xFFFFu, mx >> 16), least = min(mn & 0xFFFFu, mn >> 16) + 1u;
  return most != 0 && ((most >> 7) > kUsualMost || (least >> 7) < kUsualLeast);
}
// What a warp's lanes saw of row m, for RowScale of all warps behind the next barrier; true: not all of it fits the usual scaling.
__device__ __forceinline__ bool Publish(StreamScratch& sx, int m, int part, int lane, uint32_t mx, uint32_t mn) {
  mx = __reduce_max_sync(0xffffffffu, max(mx & 0xFFFFu, mx >> 16));
  mn = __reduce_min_sync(0xffffffffu, min(mn & 0xFFFFu, mn >> 16));
  if (lane == 0) {
    sx.xmax[m][part] = mx;
    sx.xmin[m][part] = mn;
  }
  return mx != 0 && ((mx >> 7) > kUsualMost || ((mn + 1u) >> 7) < kUsualLeast);
}
// Pieces of eight elements that a lane has on their way at a time, and holds until the slice is known to fit.  Six: four, 0.8 us
// more for 17408 x 5120 and eight rows (18 us, slices of 5.7 pieces a lane); eight, 0.2 us more for four.
constexpr int kBatch = 6;
// The power of two that puts the maximum of row m of a slice in [2^14, 2^15), where every non-zero element then is a normal FP16
// number: an exponent no more than 28 below the maximum's.  `out`: some element is not.  `low`: one is below the usual window.
__device__ __forceinline__ float RowScale(const StreamScratch& sx, int m, int wpr, int lane, bool& out, bool& low) {
  const uint32_t mx = __reduce_max_sync(0xffffffffu, lane < wpr ? sx.xmax[m][lane] : 0u);
  const uint32_t mn = __reduce_min_sync(0xffffffffu, lane < wpr ? sx.xmin[m][lane] : 0xFFFFu);
  const int e = static_cast<int>(mx >> 7);  // BF16 exponent field of the row maximum
  low = ((mn + 1) >> 7) < kUsualLeast;
  out = mx != 0 && (e < 32 || e >= 255 || static_cast<int>((mn + 1) >> 7) < e - 28);
  return mx != 0 && !out ? __uint_as_float((268u - (mx >> 7)) << 23) : 1.f;
}

// Eight elements of x, or of swish_mul(g, u).
template <bool SWISH>
__device__ __forceinline__ uint4 LoadX8(const uint4* x, const uint4* u, int c) {
  const uint4 v = __ldg(x + c);
  if constexpr (SWISH) {
    const uint4 w = __ldg(u + c);
    return make_uint4(SwishMul2(v.x, w.x), SwishMul2(v.y, w.y), SwishMul2(v.z, w.z), SwishMul2(v.w, w.w));
  }
  return v;
}
// All rows as they are, for the BF16 path (rare).
template <bool SWISH>
__device__ __forceinline__ void StageXRaw(const StreamParams& q, int kbeg, int kslice, uint16_t* xs, SharedScratch& sh, int padded, const RowShare& rs, int lane) {
  const GemmParams& p = q.g;
  const uint16_t *const x = BehindWait(p.x), *const x2 = SWISH ? BehindWait(p.x2) : nullptr;
#pragma unroll 1
  for (int m = rs.row; rs.any && m < p.M; m += rs.rpp) {
    const uint4* src = reinterpret_cast<const uint4*>(x + static_cast<size_t>(m) * p.K + kbeg);
    const uint4* src2 = SWISH ? reinterpret_cast<const uint4*>(x2 + static_cast<size_t>(m) * p.K + kbeg) : nullptr;
    uint4* dst = reinterpret_cast<uint4*>(xs + m * p.xpitch);
#pragma unroll 4
    for (int c = rs.part * 32 + lane; c < padded >> 3; c += rs.wpr * 32) dst[c] = c < kslice >> 3 ? LoadX8<SWISH>(src, src2, c) : make_uint4(0, 0, 0, 0);
  }
  if (threadIdx.x < kMaxRows) sh.inv_scale[threadIdx.x] = 1.f;
  __syncthreads();
}

// A slice of x that the usual scaling did not fit, scaled by rows instead: from what the lanes hold of it where that is all, else from
// what lies in FP16 already.  That is exact wherever it is neither infinite nor, in a row with values below the window, 2^-17 or
// less (what they round to, or zero), and takes another power of two where it lies; only pieces of eight with something else among
// them are asked for again.  It costs such calls 0.1 (FP8 5120 x 10240, two rows: 11.6 us) to 2.9 us (NVFP4 5120 x 34816,
// eight rows: 24.1), or 4.6 where most pieces have values past 64 (FP8 5120 x 10240, eight rows: 16.5); staging all of it over again cost
// 0.8 to 5.5.  Returns true if a row's values are too far apart for FP16: all rows then are staged as they are.
__device__ __forceinline__ bool RestageX(const StreamParams& q, int kbeg, int kslice, uint16_t* xs, SharedScratch& sh, const StreamScratch& sx,
                                         const uint4 (&held)[kBatch], int padded, int warp, int lane) {
  const GemmParams& p = q.g;
  const RowShare rs = ShareOf(q, warp);
  const uint16_t* const x = BehindWait(p.x);
  const int valid = kslice >> 3, step = rs.wpr * 32, c_first = rs.part * 32 + lane;  // the zeros behind `valid` stay zeros
  bool bad = p.force_slow != 0;
#pragma unroll 1
  for (int m = rs.row; rs.any && m < p.M; m += rs.rpp) {
    bool out, low;
    const float sc = RowScale(sx, m, rs.wpr, lane, out, low), ratio = sc / kUsualScale;
    const uint32_t least = low ? 0x0081u : 0u;  // without such values a zero is a zero
    if (rs.part == 0 && lane == 0) sh.inv_scale[m] = 1.f / sc;
    bad = bad || out;
    if (out) continue;
    uint4* dst = reinterpret_cast<uint4*>(xs + m * p.xpitch);
    if (padded >> 3 <= kBatch * step && rs.rpp >= p.M) {  // one batch, of one row
#pragma unroll
      for (int i = 0; i < kBatch; ++i) {
        if (c_first + i * step < valid) dst[c_first + i * step] = ScaleToHalf8(held[i], sc);
      }
      continue;
    }
    const uint4* src = reinterpret_cast<const uint4*>(x + static_cast<size_t>(m) * p.K + kbeg);
#pragma unroll 1
    for (int c0 = c_first; c0 < valid; c0 += 32 * step) {
      uint32_t lost = 0;
      const int n = min(32, (valid - c0 + step - 1) / step);
#pragma unroll 2
      for (int i = 0; i < n; ++i) {
        const uint4 v = dst[c0 + i * step];
        lost |= LostInHalf(v, least) ? 1u << i : 0u;
        dst[c0 + i * step] = RescaleHalf8(v, ratio);
      }
#pragma unroll 1
      for (; lost != 0; lost &= lost - 1) {
        const int c = c0 + (__ffs(lost) - 1) * step;
        dst[c] = ScaleToHalf8(__ldg(src + c), sc);
      }
    }
  }
  if (!__any_sync(0xffffffffu, __syncthreads_or(bad))) return false;
  StageXRaw<false>(q, kbeg, kslice, xs, sh, padded, rs, lane);
  return true;
}

// The same for swish_mul, which is evaluated again, 1.2 us: what holding pieces or the extremes of the rows for it takes is 0.1 us of
// every call, of 6 us.
__device__ __forceinline__ bool RestageSwish(const StreamParams& q, int kbeg, int kslice, uint16_t* xs, SharedScratch& sh, StreamScratch& sx, int padded, int warp,
                                             int lane) {
  const GemmParams& p = q.g;
  const RowShare rs = ShareOf(q, warp);
  const uint16_t *const g = BehindWait(p.x), *const u = BehindWait(p.x2);
  const int valid = kslice >> 3, step = rs.wpr * 32, c_first = rs.part * 32 + lane;
#pragma unroll 1
  for (int m = rs.row; rs.any && m < p.M; m += rs.rpp) {
    const size_t at = static_cast<size_t>(m) * p.K + kbeg;
    uint4* dst = reinterpret_cast<uint4*>(xs + m * p.xpitch);
    uint32_t mx = 0, mn = 0xFFFFFFFFu;
#pragma unroll 1
    for (int c = c_first; c < valid; c += step) {
      const uint4 v = LoadX8<true>(reinterpret_cast<const uint4*>(g + at), reinterpret_cast<const uint4*>(u + at), c);
      dst[c] = v;
      Track(v, mx, mn);
    }
    Publish(sx, m, rs.part, lane, mx, mn);
  }
  __syncthreads();
  bool bad = p.force_slow != 0;
#pragma unroll 1
  for (int m = rs.row; rs.any && m < p.M; m += rs.rpp) {
    bool out, low;
    const float sc = RowScale(sx, m, rs.wpr, lane, out, low);
    if (rs.part == 0 && lane == 0) sh.inv_scale[m] = 1.f / sc;
    bad = bad || out;
    uint4* dst = reinterpret_cast<uint4*>(xs + m * p.xpitch);
#pragma unroll 1
    for (int c = c_first; c < valid; c += step) dst[c] = ScaleToHalf8(dst[c], sc);
  }
  if (!__any_sync(0xffffffffu, __syncthreads_or(bad))) return false;
  StageXRaw<true>(q, kbeg, kslice, xs, sh, padded, rs, lane);
  return true;
}

// x of the slice to shared memory, rows padded with zeros to whole stages (so that the K loop needs no end), for the
// quantised modes scaled by a power of two and converted to FP16 (skinny_common.cuh), all rows by the same one: one trip
// to L2 and one barrier.  (Looking for the rows' maxima first took a second pass and barrier: FP8 5120 x 10240, two rows,
// 12.6 -> 12.0 us; NVFP4 2560 x 2560, four rows, 6.4 -> 5.9, shared expert 640 x 2560 6.9 -> 6.2.)  Returns true if some value does not
// fit that scaling (RestageX).
template <int MODE>
__device__ __forceinline__ bool StageXStream(const StreamParams& q, const Tile& tl, uint16_t* xs, SharedScratch& sh, StreamScratch& sx, uint4 (&held)[kBatch],
                                             int padded, const RowShare& rs, int lane) {
  const GemmParams& p = q.g;
  const uint16_t* const x = BehindWait(p.x);
  const int chunks = padded >> 3, valid = tl.kslice >> 3, step = rs.wpr * 32, c_first = rs.part * 32 + lane;  // K is a multiple of eight
  bool bad = p.force_slow != 0;
#pragma unroll 1
  for (int m = rs.row; rs.any && m < p.M; m += rs.rpp) {
    uint32_t mx = 0, mn = 0xFFFFFFFFu;
    const uint4* src = reinterpret_cast<const uint4*>(x + static_cast<size_t>(m) * p.K + tl.kbeg);
    uint4* dst = reinterpret_cast<uint4*>(xs + m * p.xpitch);
#pragma unroll 1
    for (int c = c_first; c < chunks; c += kBatch * step) {
#pragma unroll
      for (int i = 0; i < kBatch; ++i) held[i] = c + i * step < valid ? __ldg(src + c + i * step) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int i = 0; i < kBatch; ++i) {
        if (c + i * step < chunks) {
          if constexpr (MODE != kBf16) Track(held[i], mx, mn);
          dst[c + i * step] = MODE == kBf16 ? held[i] : ScaleToHalf8(held[i], kUsualScale);
        }
      }
    }
    if constexpr (MODE != kBf16) bad = Publish(sx, m, rs.part, lane, mx, mn) || bad;
  }
  if (threadIdx.x < kMaxRows) sh.inv_scale[threadIdx.x] = MODE == kBf16 ? 1.f : 1.f / kUsualScale;  // for the epilogue, behind further barriers
  // every warp also sees the mbarriers
  if constexpr (MODE == kBf16) {
    __syncthreads();
    return false;
  } else {
    return __syncthreads_or(bad);
  }
}

// The head's: the producer has the rows copied, and they are only waited for; that gave it 3 us of 85 at four rows and cost calls of 5
// to 17 us 0.3 us, so the products load them.  Rows are scaled one by one: the usual scaling gained nothing in 90 us.  Where the copies
// did not come, the rows are scaled by NaN and so are the sums: the stages of the weights come all the same, and the loop would
// take them.  Returns true for the BF16 path.
template <int MODE>
__device__ __forceinline__ bool StageXHead(const StreamParams& q, const Tile& tl, uint16_t* xs, SharedScratch& sh, StreamScratch& sx, StreamCtl& ctl, int padded,
                                           const RowShare& rs, int lane) {
  const GemmParams& p = q.g;
  const int chunks = padded >> 3, valid = tl.kslice >> 3, step = rs.wpr * 32, c_first = rs.part * 32 + lane;
  const float kNaN = __uint_as_float(0x7FFFFFFFu);
  BarWait(SmemAddr(&ctl.x_full), 0, ctl);
#pragma unroll 1
  for (int m = rs.row; rs.any && m < p.M; m += rs.rpp) {
    uint4* dst = reinterpret_cast<uint4*>(xs + m * p.xpitch);
    uint32_t mx = 0, mn = 0xFFFFFFFFu;
#pragma unroll 4
    for (int c = c_first; c < chunks; c += step) {
      const uint4 v = c < valid ? dst[c] : make_uint4(0, 0, 0, 0);
      if (c >= valid) dst[c] = v;
      if constexpr (MODE != kBf16) Track(v, mx, mn);
    }
    if constexpr (MODE != kBf16) Publish(sx, m, rs.part, lane, mx, mn);
  }
  __syncthreads();
  if constexpr (MODE == kBf16) {
    if (threadIdx.x < kMaxRows) sh.inv_scale[threadIdx.x] = ctl.fault ? kNaN : 1.f;  // for the epilogue, behind further barriers
    return false;
  } else {
    bool bad = p.force_slow != 0;
#pragma unroll 1
    for (int m = rs.row; rs.any && m < p.M; m += rs.rpp) {
      bool out, low;
      const float row_scale = RowScale(sx, m, rs.wpr, lane, out, low), sc = ctl.fault ? kNaN : row_scale;
      bad = bad || out;
      if (rs.part == 0 && lane == 0) sh.inv_scale[m] = 1.f / sc;
      uint4* dst = reinterpret_cast<uint4*>(xs + m * p.xpitch);
#pragma unroll 2
      for (int c = c_first; c < chunks; c += step) dst[c] = ScaleToHalf8(dst[c], sc);
    }
    if (!__any_sync(0xffffffffu, __syncthreads_or(bad))) return false;
    StageXRaw<false>(q, tl.kbeg, tl.kslice, xs, sh, padded, rs, lane);
    return true;
  }
}

// SharedExpertDown's: x = swish_mul(g, u), and the gate of every row.  Everything a thread needs first is asked for before
// anything is computed, so that the phase is one trip to memory.  The gate's sum is made in an order of its own, whatever
// the number of rows: chunk c of eight elements to lane c mod 64, lanes by shuffles, the two halves in order.
template <int MODE>
__device__ __forceinline__ bool StageXShared(const StreamParams& q, const Tile& tl, uint16_t* xs, SharedScratch& sh, StreamScratch& sx, int padded,
                                             const RowShare& rs, int lane) {
  const GemmParams& p = q.g;
  const int chunks = padded >> 3, valid = tl.kslice >> 3, step = rs.wpr * 32, c_first = rs.part * 32 + lane, gate_chunks = p.gk >> 3;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  const uint16_t *const g_in = BehindWait(p.x), *const u_in = BehindWait(p.x2), *const gx_in = BehindWait(p.gx), *const gw_in = BehindWait(p.gw);
  bool bad = p.force_slow != 0;
  constexpr int kGate = 5;  // chunks of the gate a lane asks for at once: 2560 elements
#pragma unroll 1
  for (int m = rs.row; rs.any && m < p.M; m += rs.rpp) {
    const uint4* g = reinterpret_cast<const uint4*>(g_in + static_cast<size_t>(m) * p.K + tl.kbeg);
    const uint4* u = reinterpret_cast<const uint4*>(u_in + static_cast<size_t>(m) * p.K + tl.kbeg);
    const uint4* gx = reinterpret_cast<const uint4*>(gx_in + static_cast<size_t>(m) * p.gk);
    const uint4* gw = reinterpret_cast<const uint4*>(gw_in);
    uint4* dst = reinterpret_cast<uint4*>(xs + m * p.xpitch);
    uint4 gv = c_first < valid ? __ldg(g + c_first) : zero, uv = c_first < valid ? __ldg(u + c_first) : zero;
    for (int half = rs.part; half < 2; half += rs.wpr) {
      float sum = 0.f;
#pragma unroll 1
      for (int c = half * 32 + lane; c < gate_chunks; c += 64 * kGate) {
        uint4 a[kGate], b[kGate];
#pragma unroll
        for (int i = 0; i < kGate; ++i) {
          const bool in = c + 64 * i < gate_chunks;
          a[i] = in ? __ldg(gx + c + 64 * i) : zero;
          b[i] = in ? __ldg(gw + c + 64 * i) : zero;
        }
#pragma unroll
        for (int i = 0; i < kGate; ++i) {
          const uint32_t av[4] = {a[i].x, a[i].y, a[i].z, a[i].w}, bv[4] = {b[i].x, b[i].y, b[i].z, b[i].w};
          if (c + 64 * i < gate_chunks) {  // what lies past the end adds nothing, not even to an infinity
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              sum += __uint_as_float(av[e] << 16) * __uint_as_float(bv[e] << 16);
              sum += __uint_as_float(av[e] & 0xFFFF0000u) * __uint_as_float(bv[e] & 0xFFFF0000u);
            }
          }
        }
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
      if (lane == 0) sx.gate[m][half] = sum;
    }
    uint32_t mx = 0, mn = 0xFFFFFFFFu;
#pragma unroll 1
    for (int c = c_first; c < chunks;) {
      const int next = c + step;
      const uint4 gn = next < valid ? __ldg(g + next) : zero, un = next < valid ? __ldg(u + next) : zero;
      const uint4 v = make_uint4(SwishMul2(gv.x, uv.x), SwishMul2(gv.y, uv.y), SwishMul2(gv.z, uv.z), SwishMul2(gv.w, uv.w));
      dst[c] = MODE == kBf16 ? v : ScaleToHalf8(v, kUsualScale);
      if constexpr (MODE != kBf16) Track(v, mx, mn);
      gv = gn;
      uv = un;
      c = next;
    }
    if constexpr (MODE != kBf16) bad = bad || Unusual(mx, mn);
  }
  if (threadIdx.x < kMaxRows) sh.inv_scale[threadIdx.x] = MODE == kBf16 ? 1.f : 1.f / kUsualScale;  // for the epilogue, behind further barriers
  bool again = false;
  if constexpr (MODE == kBf16) {
    __syncthreads();
  } else {
    again = __syncthreads_or(bad);
  }
  if (threadIdx.x < p.M) sh.gate[threadIdx.x] = SigmoidBf16(RoundBf16(sx.gate[threadIdx.x][0] + sx.gate[threadIdx.x][1]));
  return again;
}

// The warps' partial sums in `smem` ([wk][M][TNc], see StorePartials) to the outputs, across the cluster where K is split:
// added in warp order, then in rank order.  `first_scale`, `first_routed`: what the thread's first column needs from global
// memory, read before the K loop.
template <int MODE, bool FUSE>
__device__ __forceinline__ void FinishStream(const StreamParams& q, const Tile& tl, uint8_t* smem, SharedScratch& sh, const RowShare& rs, int lane, int cb,
                                             int share, float first_scale, uint32_t first_routed) {
  const GemmParams& p = q.g;
  const Segment& sg = p.seg[tl.seg];
  const int M = p.M, C = tl.C, TNc = p.wn * 8 * Geom<MODE>::kColsPerThread;
  const float* red = reinterpret_cast<const float*>(smem);
  float* part = reinterpret_cast<float*>(smem) + p.wk * M * TNc;
  const int j_first = rs.part * 32 + lane, step = rs.wpr * 32;
  auto local = [&](int m, int c) {
    const float* at = red + m * TNc + RedCol(c, m);
    float sum = 0.f;
#pragma unroll 1
    for (int w = 0; w < p.wk; w += 8) {
      float v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = w + i < p.wk ? at[(w + i) * M * TNc] : 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (w + i < p.wk) sum += v[i];
      }
    }
    return sum * sh.inv_scale[m];
  };
  cg::cluster_group cluster = cg::this_cluster();
  if (C > 1) {
    for (int m = rs.row; rs.any && m < M; m += rs.rpp) {
      for (int c = j_first; c < TNc; c += step) part[m * TNc + c] = local(m, c);
    }
    cluster.sync();
  }
  for (int m = rs.row; rs.any && m < M; m += rs.rpp) {
    for (int j = j_first; j < share; j += step) {
      const int c = cb + j, n = tl.n0 + c;
      float v;
      if (C > 1) {
        // all ranks' sums are asked for before the first is added
        float r[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) r[i] = i < C ? cluster.map_shared_rank(part, i)[m * TNc + c] : 0.f;
        v = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (i < C) v += r[i];
        }
      } else {
        v = local(m, c);
      }
      const bool first = j == j_first && m == rs.row;
      if (MODE != kBf16 && sg.w_scale != nullptr) v *= j == j_first ? first_scale : sg.w_scale[n];
      if constexpr (FUSE) {
        // SharedExpertDown: routed + bf16(bf16(sum) * gate), every step rounded to BF16 (skinny_gemm.cuh:226-240)
        v = RoundBf16(RoundBf16(v) * sh.gate[m]);
        if (p.routed != nullptr) {
          const uint32_t r = first ? first_routed : p.routed[static_cast<size_t>(m) * sg.n + n];
          v = __uint_as_float(r << 16) + v;
        }
      }
      int o = sg.out_begin;
      for (int i = o + 1; i < sg.out_end; ++i) {
        if (n >= p.col_begin[i]) o = i;
      }
      p.out[o][static_cast<size_t>(m) * p.width[o] + (n - p.col_begin[o])] = __bfloat16_as_ushort(__float2bfloat16(v));
    }
  }
  if (C > 1) cluster.sync();  // no CTA leaves while a peer still reads its sums
}

enum StreamKind : int { kPlain = 0, kShared = 1, kHead = 2 };

#ifdef QFG_PHASE_TIMES
#define QFG_CLOCK(v) const long long v = clock64()
#else
#define QFG_CLOCK(v)
#endif

// Where a CTA's boxes begin, in elements of eight bytes: the stored values (nibbles), the block scales; and what a row takes.
struct BoxesAt {
  int x, scales, pitch;
};
template <int MODE>
__device__ __forceinline__ BoxesAt BoxesOf(const Segment& sg, int n0) {
  return {MODE == kBf16 ? n0 >> 2 : MODE == kFp8 ? n0 >> 3 : n0 >> 4, MODE == kNvfp4 ? ((sg.n >> 1) + (n0 >> 4)) >> 3 : 0, static_cast<int>(sg.pitch >> 3)};
}
// One lane has stage `s` of the slice copied to place `slot` of the ring.  The head makes `at` once: anew for every stage it took 81.5 us
// instead of 79.7 (5120 x 151936, four rows) and 43.5 instead of 42.6 (2560 x 151936, one).  The products, with few stages
// past the first round, make it anew: once they took 0.05 to 0.1 us more (NVFP4 17408 x 5120, four rows, 15.67 -> 15.80).
template <int MODE>
__device__ __forceinline__ void IssueStage(const StreamParams& q, int seg, const BoxesAt& at, int kbeg, uint32_t ring, StreamCtl& ctl, int s, int slot) {
  const uint32_t bar = SmemAddr(&ctl.full[0]) + static_cast<uint32_t>(slot) * 8u;
  uint32_t dst = ring + static_cast<uint32_t>(slot) * static_cast<uint32_t>(q.g.stage_bytes), sdst = dst + q.scale_off;
  int row = (kbeg + s * q.rows) >> q.odd;
  BarExpect(bar, q.tx);
#pragma unroll 1
  for (int b = 0; b < q.boxes; ++b) {
    TmaLoad(dst, &q.wmap[seg], at.x, row, bar);
#pragma unroll 1
    for (int c = 1; c < q.col_boxes; ++c) TmaLoad(dst + c * q.rows * 128, &q.wmap[seg], at.x + c * 16, row, bar);
    if constexpr (MODE == kNvfp4) {
      if (q.odd) TmaLoad(dst + q.half, &q.wmap[seg], (at.x + at.pitch) & ~1, row, bar);
      TmaLoad(sdst, &q.smap[seg], at.scales & ~1, row, bar);
      if (q.odd) TmaLoad(sdst + q.shalf, &q.smap[seg], (at.scales + at.pitch) & ~1, row, bar);
      sdst += q.box_rows * q.spitch;
    }
    dst += q.box_rows * q.pitch;
    row += static_cast<int>(q.box_rows);
  }
}

// One consumer warp's part of the K loop, added to `acc`: the stages of its team, two k-steps of each.  False: a wait ran out.
template <int MODE, bool SLOW>
__device__ __forceinline__ bool ConsumeStages(const StreamParams& q, int seg, int n0, int nst, uint32_t ring, StreamCtl& ctl, int warp, int lane,
                                              float (&acc)[Geom<MODE>::kMmas][4]) {
  const int team = (warp * q.team_inv) >> 16, part_k = (warp * q.wn_inv) >> 16, wn = warp - part_k * q.g.wn, wk = part_k - team * q.team_wk;
  const uint32_t full0 = SmemAddr(&ctl.full[0]), empty0 = SmemAddr(&ctl.empty[0]);
  // rows of x that do not exist read row 0; their sums are never stored
  const uint32_t x_row = ring + q.x_off + static_cast<uint32_t>(((lane & 7) < q.g.M ? (lane & 7) : 0) * q.g.xpitch * 2 + ((lane >> 3) & 1) * 16);
  // A warp without columns of its own (the last tile's) works on whatever its places hold; those sums are never stored.
  const LaneRows r = RowsOf<MODE>(q.g.seg[seg], n0, wn, lane, q.odd, q.pitch, q.spitch, q.half, q.shalf, q.swizzle, static_cast<uint32_t>(q.rows));
  // two k-steps of every stage, wk and wk + q.g.wk; ldmatrix takes x of the first for the lower half warp, of the second for the upper
  const uint32_t w0 = r.w + static_cast<uint32_t>(wk) * r.step, w1 = w0 + r.d1, w2 = w0 + r.d2, w3 = w1 + r.d2;
  const uint32_t s0 = q.scale_off + r.s + static_cast<uint32_t>(wk) * r.sstep, s1 = s0 + r.e1, s2 = s0 + r.e2, s3 = s1 + r.e2;
  const uint32_t wstep = static_cast<uint32_t>(q.team_wk) * r.step, sstep = static_cast<uint32_t>(q.team_wk) * r.sstep;
  const uint32_t first = static_cast<uint32_t>(team), teams = static_cast<uint32_t>(q.teams), stage_bytes = static_cast<uint32_t>(q.g.stage_bytes);
  const uint32_t at_step = teams * stage_bytes, bar_step = teams * 8u, xstep = teams * static_cast<uint32_t>(q.team_wk) * 64u;
  const uint32_t full_end = full0 + static_cast<uint32_t>(q.g.stages) * 8u;
  uint32_t x_at = x_row + static_cast<uint32_t>(wk + (lane >> 4) * q.team_wk + team * 2 * q.team_wk) * 32u;
  auto load = [&](Raw<MODE>& raw, uint32_t w, uint32_t s) {
    if constexpr (MODE == kNvfp4) {
      raw.r[0][0] = Lds64(w0 + w);
      raw.r[0][1] = Lds64(w1 + w);
      raw.r[0][2] = Lds64(w2 + w);
      raw.r[0][3] = Lds64(w3 + w);
      raw.s[0][0] = Lds8(s0 + s);
      raw.s[0][1] = Lds8(s1 + s);
      raw.s[0][2] = Lds8(s2 + s);
      raw.s[0][3] = Lds8(s3 + s);
    } else {
      raw.r[0] = Lds128(w0 + w);
      raw.r[1] = Lds128(w1 + w);
      raw.r[2] = Lds128(w2 + w);
      raw.r[3] = Lds128(w3 + w);
    }
  };
  uint32_t parity = 0, at = ring + first * stage_bytes, bar = full0 + first * 8u;
#pragma unroll 1
  for (int left = nst - team; left > 0; left -= static_cast<int>(teams)) {
    if (!BarWait(bar, parity, ctl)) return false;
    Raw<MODE> ra, rb;
    uint32_t xv[4];
    load(ra, at, at);
    LoadX2(x_at, xv);
    load(rb, at + wstep, at + sstep);
    __syncwarp();
    if (lane == 0) BarArrive(bar + (empty0 - full0));  // the stage is read
    ComputeStep<MODE, SLOW>(acc, ra, xv[0], xv[1]);
    ComputeStep<MODE, SLOW>(acc, rb, xv[2], xv[3]);
    x_at += xstep;
    at += at_step;
    bar += bar_step;
    if (bar >= full_end) {  // the stages are a multiple of the teams: a slot always serves the same one, which sees its every phase
      bar = full0 + first * 8u;
      at = ring + first * stage_bytes;
      parity ^= 1u;
    }
  }
  return true;
}

// The tail warp's k-steps of a left-over group of the LM head.
template <int MODE, bool SLOW>
__device__ __forceinline__ void ConsumeTail(const LaneRows& r, uint32_t w, uint32_t sc, uint32_t x_at, int count, float (&acc)[Geom<MODE>::kMmas][4]) {
#pragma unroll 1
  for (int i = 0; i < count; ++i) {
    Raw<MODE> ra;
    uint32_t xv[4];
    LoadRows<MODE>(ra, r, w, sc);
    LoadX2(x_at, xv);
    ComputeStep<MODE, SLOW>(acc, ra, xv[0], xv[1]);
    w += r.step;
    sc += r.sstep;
    x_at += 32;
  }
}

// What a CTA's threads know when x is staged.
struct StreamWork {
  Tile tl;
  int nst, warp, lane;
  uint32_t ring;
  uint8_t* smem;
  int cb, share;  // this thread's outputs, see FinishStream
  float first_scale;
  uint32_t first_routed;
  int tail_index, tail_first, tail_count, tail_col;  // shared tail of the fused LM head
};

// From staged x to the stored outputs.  `slow`: the BF16 path.
template <int MODE, int KIND>
__device__ __forceinline__ void StreamRest(bool slow, const StreamParams& q, const StreamWork& w, SharedScratch& sh, StreamCtl& ctl) {
  using G = Geom<MODE>;
  constexpr int NM = G::kMmas;
  constexpr bool kTail = MODE == kNvfp4 && KIND == kHead;
  const GemmParams& p = q.g;
  const Segment& sg = p.seg[w.tl.seg];
  const int warp = w.warp, lane = w.lane;
  const uint32_t ring = w.ring;
  uint8_t* const smem = w.smem;
  const uint32_t empty0 = SmemAddr(&ctl.empty[0]);
  float acc[NM][4];
#pragma unroll
  for (int j = 0; j < NM; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
  const int wn = warp - ((warp * q.wn_inv) >> 16) * p.wn;
  const bool consumer = warp < q.warps;
  constexpr int kWarpCols = 8 * G::kColsPerThread;
  // rows of x that do not exist read row 0; their sums are never stored
  const uint32_t x_row = ring + q.x_off + static_cast<uint32_t>(((lane & 7) < p.M ? (lane & 7) : 0) * p.xpitch * 2 + ((lane >> 3) & 1) * 16);
  QFG_CLOCK(loop_begin);

  if (warp == q.warps) {
    const BoxesAt boxes = BoxesOf<MODE>(sg, w.tl.n0);
    int slot = 0;
    uint32_t parity = 0;
    for (int s = p.stages; s < w.nst; ++s) {
      if (!BarWait(empty0 + slot * 8, parity, ctl)) break;
      if (ElectOne()) IssueStage<MODE>(q, w.tl.seg, KIND == kHead ? boxes : BoxesOf<MODE>(sg, w.tl.n0), w.tl.kbeg, ring, ctl, s, slot);
      __syncwarp();
      if (++slot == p.stages) {
        slot = 0;
        parity ^= 1u;
      }
    }
  } else if (consumer) {
    bool good;
    if (MODE != kBf16 && slow) {
      good = ConsumeStages<MODE, true>(q, w.tl.seg, w.tl.n0, w.nst, ring, ctl, warp, lane, acc);
    } else {
      good = ConsumeStages<MODE, false>(q, w.tl.seg, w.tl.n0, w.nst, ring, ctl, warp, lane, acc);
    }
    if (!good) {
#pragma unroll
      for (int j = 0; j < NM; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[j][e] = __uint_as_float(0x7FFFFFFFu);
    }
  } else if constexpr (kTail) {
    if (w.tail_index >= 0) {
      const uint32_t hw = q.odd ? q.tail_rows / 2 * q.tail_pitch : 0, hs = q.odd ? q.tail_rows / 2 * 16 : 0;
      const LaneRows r = RowsOf<MODE>(sg, w.tail_col, 0, lane, q.odd, q.tail_pitch, 16, hw, hs);
      const uint32_t rows = ring + q.tail_off + r.w, scales = ring + q.tail_off + q.tail_rows * q.tail_pitch + r.s;
      const uint32_t x_at = x_row + static_cast<uint32_t>(w.tail_first + (lane >> 4)) * 32u;
      const bool good = BarWait(SmemAddr(&ctl.tail_full), 0, ctl);
      if (good && slow) {
        ConsumeTail<MODE, true>(r, rows, scales, x_at, w.tail_count, acc);
      } else if (good) {
        ConsumeTail<MODE, false>(r, rows, scales, x_at, w.tail_count, acc);
      }
      float* const dst = p.lm_tail + static_cast<size_t>(w.tail_index) * kMaxRows * 128;
      const int g = lane >> 2, t = lane & 3;
#pragma unroll
      for (int j = 0; j < NM; ++j) {
        const int cl = g * 16 + 2 * j, m0 = 2 * t, m1 = 2 * t + 1;
        if (!good) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = __uint_as_float(0x7FFFFFFFu);
        if (m0 < p.M) *reinterpret_cast<float2*>(&dst[m0 * 128 + cl]) = make_float2(acc[j][0], acc[j][2]);
        if (m1 < p.M) *reinterpret_cast<float2*>(&dst[m1 * 128 + cl]) = make_float2(acc[j][1], acc[j][3]);
      }
      __threadfence();
    }
  }
#ifdef QFG_PHASE_TIMES
  if (p.phase_times != nullptr && threadIdx.x == 0) {
    unsigned long long* o = p.phase_times + (static_cast<size_t>(blockIdx.y) * gridDim.x + blockIdx.x) * 16;
    o[9] = clock64() - loop_begin;
  }
#endif
  Stamp(p, 3);
  if (p.trigger == 2) GridLaunchDependents();
  if (ctl.fault) __nanosleep(1000000);  // copies of a CTA that gave up may still be landing where the sums go now
  __syncthreads();
  if (consumer) StorePartials<MODE, 1>(p, w.tl, acc, smem, w.tl.n0 + wn * kWarpCols < w.tl.n1);
  __syncthreads();
  Stamp(p, 4);
  if constexpr (KIND == kHead) {
    EpilogueTail<MODE, false>(p, w.tl, smem, sh, p.wk, p.wn * kWarpCols);
  } else {
    FinishStream<MODE, KIND == kShared>(q, w.tl, smem, sh, ShareOf(q, warp), lane, w.cb, w.share, w.first_scale, w.first_routed);
  }
  Stamp(p, 5);
}

// KIND: plain, SharedExpertDown, fused LM head.
template <int MODE, int KIND>
__global__ void __launch_bounds__(kStreamThreads, 1) SkinnyGemmStreamKernel(const __grid_constant__ StreamParams q) {
  using G = Geom<MODE>;
  constexpr int NM = G::kMmas;
  constexpr bool kTail = MODE == kNvfp4 && KIND == kHead, kBulkX = KIND == kHead;
  extern __shared__ uint8_t smem_raw[];
  __shared__ SharedScratch sh;
  __shared__ StreamScratch sx;
  __shared__ StreamCtl ctl;
  const GemmParams& p = q.g;
  Stamp(p, 0);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  Tile tl = LocateTile(p);
  const Segment& sg = p.seg[tl.seg];
  // K in whole stages, so that no copy reaches into the next slice
  const int st0 = tl.crank * q.nstages / tl.C, nst = (tl.crank + 1) * q.nstages / tl.C - st0;
  tl.kbeg = st0 * q.rows;
  tl.kend = min(p.K, (st0 + nst) * q.rows);
  tl.kslice = max(0, tl.kend - tl.kbeg);
  const uint32_t ring = (SmemAddr(smem_raw) + 1023u) & ~1023u;  // swizzled boxes begin on 1024 bytes
  uint8_t* const smem = smem_raw + (ring - SmemAddr(smem_raw));
  const uint32_t full0 = SmemAddr(&ctl.full[0]), empty0 = SmemAddr(&ctl.empty[0]);

  // Shared tail of the fused LM head (see GemmParams::tail_groups): one K slice of a left-over column group per hosting CTA
  int tail_index = -1, tail_first = 0, tail_count = 0, tail_col = 0;
  if constexpr (kTail) {
    if (p.tail_groups > 0 && static_cast<int>(blockIdx.x) % p.tail_stride == 0) {
      const int i = static_cast<int>(blockIdx.x) / p.tail_stride;
      if (i < p.tail_groups * p.tail_split) {
        const int ksteps = (tl.kslice + 15) >> 4;
        tail_index = i;
        const int tg = i / p.tail_split, slice = i - tg * p.tail_split;
        tail_first = slice * ksteps / p.tail_split;
        tail_count = (slice + 1) * ksteps / p.tail_split - tail_first;
        tail_col = sg.n - p.tail_groups * 128 + tg * 128;
      }
    }
  }

  // ---- producer
  const uint32_t x_smem = ring + q.x_off, x_full = SmemAddr(&ctl.x_full);
  auto issue_x = [&]() {  // one lane
    const uint32_t bytes = static_cast<uint32_t>(tl.kslice) * 2u;
    BarExpect(x_full, bytes * static_cast<uint32_t>(p.M));
#pragma unroll 1
    for (int m = 0; m < p.M && bytes > 0; ++m)
      BulkLoad(x_smem + static_cast<uint32_t>(m * p.xpitch) * 2u, p.x + static_cast<size_t>(m) * p.K + tl.kbeg, bytes, x_full);
  };
  if (warp == q.warps) {
    if (ElectOne()) {
      if (kBulkX) BarInit(x_full, 1);
      for (int i = 0; i < p.stages; ++i) {
        BarInit(full0 + i * 8, 1);
        BarInit(empty0 + i * 8, q.team_warps);
      }
      BarInit(SmemAddr(&ctl.tail_full), 1);
      ctl.fault = kBulkX ? static_cast<uint32_t>(p.give_up) : 0u;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (!p.pdl_wait) GridDependencyWait();  // without the option the weights are the predecessor's to write too
    if (kBulkX) asm volatile("bar.arrive 1, %0;" ::"r"(static_cast<int>(blockDim.x)) : "memory");  // the others may wait on the barriers
    if (ElectOne()) {
      const BoxesAt boxes = BoxesOf<MODE>(sg, tl.n0);
      // x before the weights, so that it does not queue behind them - unless it may still be the predecessor kernel's to write
      if (kBulkX && !p.pdl_wait) issue_x();
      for (int s = 0; s < p.stages && s < nst; ++s) IssueStage<MODE>(q, tl.seg, KIND == kHead ? boxes : BoxesOf<MODE>(sg, tl.n0), tl.kbeg, ring, ctl, s, s);
      if constexpr (kTail) {
        if (tail_index >= 0) {
          const uint32_t bar = SmemAddr(&ctl.tail_full), dst = ring + q.tail_off, sdst = dst + q.tail_rows * q.tail_pitch;
          const uint32_t hw = q.tail_rows / 2 * q.tail_pitch, hs = q.tail_rows / 2 * 16;
          const int tx0 = tail_col >> 4, tsx = ((sg.n >> 1) + (tail_col >> 4)) >> 3, row = tail_first * 16;
          BarExpect(bar, q.tail_tx);
          if (q.odd) {  // even rows, odd rows
            TmaLoad(dst, &q.tail_wmap, tx0, row >> 1, bar);
            TmaLoad(dst + hw, &q.tail_wmap, (tx0 + boxes.pitch) & ~1, row >> 1, bar);
            TmaLoad(sdst, &q.tail_smap, tsx & ~1, row >> 1, bar);
            TmaLoad(sdst + hs, &q.tail_smap, (tsx + boxes.pitch) & ~1, row >> 1, bar);
          } else {      // upper half, lower half
            const int below = row + static_cast<int>(q.tail_rows / 2);
            TmaLoad(dst, &q.tail_wmap, tx0, row, bar);
            TmaLoad(dst + hw, &q.tail_wmap, tx0, below, bar);
            TmaLoad(sdst, &q.tail_smap, tsx & ~1, row, bar);
            TmaLoad(sdst + hs, &q.tail_smap, tsx & ~1, below, bar);
          }
        }
      }
    }
    __syncwarp();
  }
  const RowShare rs = ShareOf(q, warp);
  // this thread's outputs: columns cb + 32 part + lane, ... of the tile
  const int cper = tl.C > 1 ? q.rank_cols : p.wn * 8 * G::kColsPerThread, cb = tl.crank * cper;
  const int share = min(cper, tl.n1 - tl.n0 - cb), first_n = tl.n0 + cb + rs.part * 32 + lane;
  float first_scale = 1.f;
  uint32_t first_routed = 0;
  if constexpr (KIND != kHead) {
    if (MODE != kBf16 && sg.w_scale != nullptr && first_n < tl.n1) first_scale = __ldg(sg.w_scale + first_n);
  }
  // with pdl_wait the weights do not depend on the predecessor kernel, x may be its output
  GridDependencyWait();
  // Not at the start: a kernel that itself still waits would let the next ones in, and where several CTAs fit an SM a chain of
  // calls would pile up, CTAs of later calls in the places beside the running one's.  NVFP4 2560 x 2560 after itself, eight
  // rows, 12.2 -> 8.2 us a call (8.9 without programmatic launch); 1024 x 4096 and back, one row, 7.0 -> 6.3; 640 x 640 4.5 ->
  // 4.6; calls whose CTAs have their SMs to themselves the same.
  if (p.trigger == 1) GridLaunchDependents();
  if (kBulkX && p.pdl_wait && warp == q.warps) {
    if (ElectOne()) issue_x();
    __syncwarp();
  }
  if constexpr (KIND == kShared) {
    if (p.routed != nullptr && first_n < tl.n1 && rs.any && rs.row < p.M) first_routed = p.routed[static_cast<size_t>(rs.row) * sg.n + first_n];
  }
  uint16_t* const xs = reinterpret_cast<uint16_t*>(smem + q.x_off);
  const int padded = nst * q.rows;
  Stamp(p, 1);
  bool unusual = false, slow = false;
  uint4 held[kBatch];
  if constexpr (KIND == kShared) {
    unusual = StageXShared<MODE>(q, tl, xs, sh, sx, padded, rs, lane);
  } else if constexpr (KIND == kPlain) {
    unusual = StageXStream<MODE>(q, tl, xs, sh, sx, held, padded, rs, lane);
  } else {
    if (warp != q.warps) asm volatile("bar.sync 1, %0;" ::"r"(static_cast<int>(blockDim.x)) : "memory");
    slow = StageXHead<MODE>(q, tl, xs, sh, sx, ctl, padded, rs, lane);
  }
  Stamp(p, 2);

  const StreamWork w = {tl, nst, warp, lane, ring, smem, cb, share, first_scale, first_routed, tail_index, tail_first, tail_count, tail_col};
  // The votes are for the compiler: what a barrier returns is not known to be the same in every lane, and behind a branch on it the
  // loop's addresses and control leave the uniform registers, 15 instructions more per k-step and warp (NVFP4 5120 x 34816 22.3
  // -> 24.2 us, 17408 x 5120, four rows, 15.9 -> 17.2; `ncu` 12.9 -> 13.8 M warp instructions).
  if constexpr (KIND == kHead || MODE == kBf16) {
    StreamRest<MODE, KIND>(__any_sync(0xffffffffu, slow), q, w, sh, ctl);
  } else if (__all_sync(0xffffffffu, !unusual)) {
    StreamRest<MODE, KIND>(false, q, w, sh, ctl);
  } else {
    if constexpr (KIND == kShared) {
      slow = RestageSwish(q, tl.kbeg, tl.kslice, xs, sh, sx, padded, warp, lane);
    } else {
      slow = RestageX(q, tl.kbeg, tl.kslice, xs, sh, sx, held, padded, warp, lane);
    }
    StreamRest<MODE, KIND>(__any_sync(0xffffffffu, slow), q, w, sh, ctl);
  }
}

// ------------------------------------------------------------------------------ host
constexpr int kStreamSmem = 232448 - static_cast<int>(sizeof(SharedScratch) + sizeof(StreamScratch) + sizeof(StreamCtl)) - 256;
constexpr int kStreamPad = 1024;  // past the staged x: the tail warp's ldmatrix reads a k-step ahead

struct StreamSetup {
  cudaError_t status = cudaErrorNotReady;
  int slots[9] = {};  // clusters of so many CTAs, one per SM, that are resident at once
};
StreamSetup g_stream;

// Of a launch on the device that was set up; for a description without it, the loss in packing that planner.cc assumes.
int Resident(const PlanInput& in, int cluster) {
  if (g_stream.status == cudaSuccess && in.sm_count == DeviceSmCount()) return g_stream.slots[cluster];
  return cluster == 1 ? in.sm_count : std::max(1, in.sm_count * 8 / (10 * cluster));
}
bool Refused() { return g_stream.status != cudaSuccess && g_stream.status != cudaErrorNotReady; }

template <int MODE, int KIND>
cudaError_t SetUpStream() {
  return cudaFuncSetAttribute(SkinnyGemmStreamKernel<MODE, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, kStreamSmem);
}

template <int MODE>
cudaError_t SetUpMode() {
  cudaError_t err = SetUpStream<MODE, kPlain>();
  if (err == cudaSuccess) err = SetUpStream<MODE, kShared>();
  return err == cudaSuccess ? SetUpStream<MODE, kHead>() : err;
}

int StreamSlots(int cluster) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(1, static_cast<unsigned>(cluster));
  cfg.blockDim = dim3(static_cast<unsigned>(kStreamThreads));
  cfg.dynamicSmemBytes = kStreamSmem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = static_cast<unsigned>(cluster);
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, SkinnyGemmStreamKernel<kBf16, kPlain>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    n = std::max(1, DeviceSmCount() * 8 / (10 * cluster));
  }
  return n;
}

// rows x row_bytes, in elements of eight bytes
bool Encode8(CUtensorMap* map, const void* base, uint64_t rows, uint64_t row_bytes, uint32_t box_rows, uint32_t box_bytes, int swizzle = 0) {
  const cuuint64_t dims[2] = {row_bytes / 8, rows}, strides[1] = {row_bytes};
  const cuuint32_t box[2] = {box_bytes / 8, box_rows}, step[2] = {1, 1};
  const TensorMapEncodeFn fn = TensorMapEncoder();
  return fn != nullptr && fn(map, CU_TENSOR_MAP_DATA_TYPE_INT64, 2, const_cast<void*>(base), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
                             swizzle == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : swizzle == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int StreamGran(int mode) { return mode == kBf16 ? 8 : mode == kFp8 ? 16 : 128; }
int StreamGranBytes(int mode) { return mode == kNvfp4 ? 64 : 16; }

// The shared memory of a launch: a function of the plan and the rows of the call.
struct StreamLayout {
  int wn, pitch, spitch, swizzle, row_bytes, rows, boxes, box_rows, stage, nstages, xpitch, red, tail_rows, tail_bytes, stages, ring;
  size_t smem;
};
StreamLayout LayOut(int mode, bool odd, int K, const StreamPlan& plan, int m) {
  StreamLayout l = {};
  const int tile_bytes = plan.width * StreamGranBytes(mode);
  l.wn = mode == kNvfp4 ? plan.width : (tile_bytes + 127) / 128;
  l.swizzle = mode != kNvfp4 || odd ? 0 : tile_bytes % 128 == 0 ? 128 : tile_bytes == 64 ? 64 : 0;
  l.pitch = l.swizzle > 0 ? l.swizzle : odd ? tile_bytes + 32 : (tile_bytes / 16 | 1) * 16;
  l.row_bytes = l.swizzle > 0 ? tile_bytes : l.pitch;
  if (mode == kNvfp4) l.spitch = (plan.width * 8 + 8 + 15) / 16 * 16;
  l.rows = 32 * plan.wk;
  const int box_all = odd ? l.rows / 2 : l.rows;
  l.boxes = (box_all + 255) / 256;
  l.box_rows = box_all / l.boxes;
  l.stage = (l.rows * (l.row_bytes + l.spitch) + 1023) / 1024 * 1024;
  const int ksteps = (K + 15) / 16;
  l.nstages = (ksteps * 16 + l.rows - 1) / l.rows;
  const int slice = (l.nstages + plan.cluster - 1) / plan.cluster * l.rows;
  l.xpitch = (slice + 63) / 64 * 64 + 8;  // rows 16 bytes apart in the banks
  const int cols = l.wn * GeomOf(mode).cols_per_warp;
  l.red = (plan.wk * plan.teams + (plan.cluster > 1 ? 1 : 0)) * m * cols * 4;
  if (plan.tail > 0) {
    l.tail_rows = (ksteps + plan.tail_split - 1) / plan.tail_split * 16;
    l.tail_bytes = (l.tail_rows * ((odd ? 96 : 80) + 16) + 127) / 128 * 128;
  }
  const int fixed = m * l.xpitch * 2 + kStreamPad + l.tail_bytes;
  l.stages = std::min({kStreamStages, (kStreamSmem - 1024 - fixed) / l.stage, (l.nstages + plan.cluster - 1) / plan.cluster + plan.teams - 1});
  // whole rounds of the teams; where the slice has fewer stages than that, the last teams have none
  l.stages = std::max(l.stages / plan.teams, 1) * plan.teams;
  l.ring = (std::max(l.stages * l.stage, l.red) + 127) / 128 * 128;
  l.smem = static_cast<size_t>(l.ring) + fixed + 1024;
  return l;
}

template <int MODE, int KIND>
cudaError_t Launch(const StreamParams& q, int tiles, int threads, size_t smem, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(tiles), static_cast<unsigned>(q.g.cluster), 1);
  cfg.blockDim = dim3(static_cast<unsigned>(threads), 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n_attr = 0;
  if (q.g.cluster > 1) {
    attr[n_attr].id = cudaLaunchAttributeClusterDimension;
    attr[n_attr].val.clusterDim.x = 1;
    attr[n_attr].val.clusterDim.y = static_cast<unsigned>(q.g.cluster);
    attr[n_attr].val.clusterDim.z = 1;
    ++n_attr;
  }
  if (q.g.pdl_wait || MayOverlapPredecessor(stream)) attr[n_attr++] = OverlapAttribute();
  cfg.attrs = attr;
  cfg.numAttrs = n_attr;
  return cudaLaunchKernelEx(&cfg, SkinnyGemmStreamKernel<MODE, KIND>, q);
}

template <int MODE>
cudaError_t LaunchMode(const StreamParams& q, int tiles, int threads, size_t smem, cudaStream_t stream) {
  if (q.g.fuse) return Launch<MODE, kShared>(q, tiles, threads, smem, stream);
  return q.g.lm ? Launch<MODE, kHead>(q, tiles, threads, smem, stream) : Launch<MODE, kPlain>(q, tiles, threads, smem, stream);
}

bool OddRows(int mode, const PlanInput& in) {
  for (int s = 0; mode == kNvfp4 && s < in.nseg; ++s) {
    if (in.n[s] % 256 != 0) return true;
  }
  return false;
}

}  // namespace

cudaError_t ConfigureStreamKernels() {
  cudaError_t err = SetUpMode<kBf16>();
  if (err == cudaSuccess) err = SetUpMode<kFp8>();
  if (err == cudaSuccess) err = SetUpMode<kNvfp4>();
  for (int c = 1; err == cudaSuccess && c <= 8; ++c) g_stream.slots[c] = StreamSlots(c);
  g_stream.status = err;
  return err;
}

bool CompleteStreamPlan(const PlanInput& in, StreamPlan* plan) {
  if (Refused() || plan->width < 1 || plan->wk < 1 || plan->teams < 1 || plan->cluster < 1 || plan->cluster > 8) return false;
  if (in.K % 8 != 0 || in.K > (1 << 20) || in.row_align < (in.mode == kNvfp4 ? 8 : 16)) return false;
  const int gran = StreamGran(in.mode);
  const bool odd = OddRows(in.mode, in);
  int tiles = 0;
  if (plan->tail > 0) {
    // every left-over group's K range in up to sixteen slices, one per CTA
    if (!in.allow_tail || in.nseg != 1 || in.mode != kNvfp4 || plan->cluster != 1 || plan->tail > kMaxTailGroups || plan->tail >= in.n[0] / gran) return false;
  }
  for (int s = 0; s < in.nseg; ++s) {
    if (in.n[s] % gran != 0) return false;
    const int granules = in.n[s] / gran - plan->tail;
    plan->tiles[s] = (granules + plan->width - 1) / plan->width;
    tiles += plan->tiles[s];
  }
  if (plan->tail > 0) {
    if (tiles < 2 * plan->tail) return false;
    plan->tail_split = std::min(kMaxTailSplit, tiles / plan->tail);
  }
  const StreamLayout l = LayOut(in.mode, odd, in.K, *plan, kMaxRows);
  if (l.wn * plan->wk * plan->teams > kStreamWarps || l.pitch > 2048 || l.smem > kStreamSmem || l.tail_rows > 512) return false;
  // the boxes make up the stage (17 warps along K: 544 rows are not three boxes), each on the 128 bytes that a copy begins on
  if (l.boxes * l.box_rows != (odd ? l.rows / 2 : l.rows) || l.box_rows % 8 != 0) return false;
  // eight rows of x leave the ring room for the stages in use and as much on its way
  return l.stages >= std::min(plan->teams + (l.stage < 40960 ? 2 : 1), (l.nstages + plan->cluster - 1) / plan->cluster);
}

// The cheapest launch shape by a model (one B200, one to eight rows, microseconds).  Its terms were fitted to ordinary launches and to x staged
// in two passes, and so are the figures below; with launches that overlap and x staged in one look the choice is 3.6 % behind the best of
// some fifty launches tried on 146 such shapes (BF16 2.1, FP8 3.4, NVFP4 5.3; at worst 40: 2800 x 3712, seven rows, without a cluster):
//   the stream: all bytes at 6.0 TB/s, a ninth to a third more where tiles begin inside lines of 128 bytes; or a CTA's share
//   at 14 ns per KB, or slower where its ring (at four rows) is less than two microseconds of that; a row and 128 columns
//   of NVFP4 1.75 ns, its arithmetic (more where a tile is one group wide: two copied rows for 72 bytes, and few warps);
//   around it: 2.2 (BF16) or 3.4 for launch, first copies, x and the epilogue; 1.8 (a pair) to 2.5 (eight) more where ranks of a
//   cluster add up; 0.4 ns for each row of a slice past 5120, whose x is staged in further rounds; 2 for NVFP4 of several groups
//   per CTA over fewer than 1024 rows, whose few stages do not hide the first;
//   SharedExpertDown: swish_mul of the slice, which every CTA computes for itself.
// What a term decides, on 2000 random shapes (K 256 to 17408, N 256 to 23170, one to three weights, one to eight rows) with the
// model's choice 4.7 % behind the best launch tried.  Without it: lines of 128 bytes: 772 of 1339 BF16 / FP8 shapes get another
// launch, 1 % slower on average; least 1.5 ns a row: 361 of 1339, 20 % slower; ring of two microseconds: 8, 3 % slower; x past 5120
// rows: 71, 4 % slower; few stages of NVFP4: 347 of 661, 8 % slower; eight NVFP4 warps taken for sixteen (2.05): 46 of 661, 19 %
// slower; four taken for eight (2.3): 138, no difference on average; sixteen taken for eight (2.3): 26, 6 % faster, not
// followed up; swish_mul: 72 of 400 shared experts, 10 % (NVFP4 22 %) slower.
// Against other shapes: BF16 5120 x 5120 8 pieces wide, two teams of four warps, no cluster 11.1 (16 wide in clusters of three
// 12.7, 5 wide 12.8); FP8 6144 x 2560 in clusters of four to six 8.1 (of two 10.1); NVFP4 17408 x 5120 two groups wide in
// clusters of six 16.6 (one group, clusters of three 18.3); NVFP4 640 x 2560 in clusters of five 5.4 (none 6.4).
StreamPlan ChooseStreamPlan(const PlanInput& in) {
  StreamPlan best;
  if (Refused()) return best;
  const int gran = StreamGran(in.mode), ksteps = (in.K + 15) / 16;
  const bool odd = OddRows(in.mode, in), fp4 = in.mode == kNvfp4;
  // A vocabulary of at least four groups of 128 columns per SM and a few more: the head gives the few away in slices of K
  // (GemmParams::tail_groups), the plain product takes a group more per CTA and adds up K in the same order.
  if (in.nseg == 1 && fp4 && in.n[0] % gran == 0 && !in.fuse && Resident(in, 1) > 0) {
    const int slots = Resident(in, 1), groups = in.n[0] / gran, per = groups / slots, rest = groups % slots;
    if (per >= 4 && rest >= 1 && rest <= kMaxTailGroups && per < kStreamWarps) {
      PlanInput head = in;
      head.allow_tail = true;
      StreamPlan with, without;
      with.width = per;
      without.width = per + 1;
      with.wk = without.wk = 1;
      with.teams = without.teams = std::min(3, kStreamWarps / (per + 1));
      with.tail = rest;
      if (CompleteStreamPlan(head, &with) && CompleteStreamPlan(in, &without)) return in.allow_tail ? with : without;
    }
  }
  double best_cost = 1e30, total = 0;
  for (int s = 0; s < in.nseg; ++s) total += static_cast<double>(in.K) * in.n[s] * (in.mode == kBf16 ? 2.0 : in.mode == kFp8 ? 1.0 : 0.5625);
  for (int cluster = 1; cluster <= 8; ++cluster) {
    const int slots = Resident(in, cluster), slice = (ksteps + cluster - 1) / cluster * 16;
    const double around = (in.mode == kBf16 ? 2.2 : 3.4) + (cluster > 1 ? 1.7 + 0.1 * cluster : 0.0);
    if (cluster > 1 && (ksteps < 8 * cluster || total / 6.0e6 + around >= best_cost)) break;
    for (int width = fp4 ? 1 : 3; slots > 0 && width <= (fp4 ? kStreamWarps : 32); ++width) {
      const double extra = fp4 || width % 8 == 0 ? 1.0 : 1.0 + 1.0 / width, all = total * extra / 6.0e6;
      if (all + around >= best_cost) continue;
      int tiles = 0;
      for (int s = 0; s < in.nseg; ++s) tiles += (in.n[s] / gran + width - 1) / width;
      const int waves = (tiles + slots - 1) / slots;
      if (all + waves * around >= best_cost) continue;
      StreamPlan p;
      p.width = width;
      p.cluster = cluster;
      // Eight warps along K (as two teams where the arithmetic of a stage is short), fewer where columns take them or K is short.
      // The same 2000 shapes, time over that of the line taken: one column warp, BF16, slices below 512 rows 4 x 1, 4 x 2 1.03,
      // 8 x 1 1.04, from 1024 4 x 2, 8 x 1 1.00, 4 x 1 1.01 to 1.03; FP8 below 512 4 x 1, 8 x 1 and 4 x 2 1.00, to 1024 8 x 1 0.97,
      // beyond 8 x 1, 4 x 2 1.00 to 1.04, 4 x 1 1.10; NVFP4 below 1024 4 x 1, 8 x 1 0.93 to 0.96, to 2048 8 x 1, 8 x 2 1.05, 4 x 1
      // 1.11, beyond 8 x 2, 8 x 1 1.00, 4 x 2 1.06.  Two column warps: 4 x 2, BF16 / FP8 2 x 2 0.95 to 0.99, NVFP4 to 1024 4 x 1 0.98,
      // beyond 3 x 2 1.02 to 1.05.  Three and more: 4 x 1, 2 x 2 0.96 to 1.07.  One or two warps and one team: 1.1 to 3.
      const int wn = fp4 ? width : (width + 7) / 8;
      if (wn == 1) {
        p.wk = in.mode == kBf16 || in.fuse || slice < 1024 ? 4 : 8;
        p.teams = in.fuse || (in.mode == kBf16 && slice >= 1024) || (fp4 && slice >= 2048) ? 2 : 1;
      } else if (wn == 2) {
        p.wk = 4;
        p.teams = slice < 512 && !in.fuse ? 1 : 2;
      } else {
        p.wk = std::min(4, kStreamWarps / wn);
      }
      if (!CompleteStreamPlan(in, &p)) continue;
      const StreamLayout l = LayOut(in.mode, odd, in.K, p, 4);
      const double rows = static_cast<double>((l.nstages + cluster - 1) / cluster) * l.rows;
      const double ring_kb = l.stages * l.stage / 1024.0;
      double row_ns;
      if (fp4) {
        row_ns = wn > 1 ? 1.75 * wn : p.wk * p.teams >= 16 ? 2.05 : p.wk * p.teams >= 8 ? 2.3 : 4.5;
      } else {
        row_ns = std::max(1.5, width / 64.0 * (l.stages * cluster >= l.nstages ? 14.0 : std::max(14.0, 2000.0 / ring_kb)));
      }
      const double stream = std::max(all, waves * rows * row_ns * 1e-3);
      const double cost = stream + waves * around + std::max(0.0, rows - 5120) * 4e-4 + (fp4 && wn > 1 && slice < 1024 ? 2.0 : 0.0) +
                          (in.fuse ? rows * (in.mode == kBf16 ? 0.5e-3 : 3e-3) : 0);
      if (cost < best_cost) {
        best_cost = cost;
        best = p;
      }
    }
  }
  return best;
}

std::string DescribeStreamPlan(const StreamPlan& p) {
  char buf[96];
  std::snprintf(buf, sizeof(buf), "stream=%d/%d/%d/%d/%d", p.width, p.wk, p.teams, p.cluster, p.tail);
  return buf;
}

bool LaunchSkinnyStream(int mode, GemmParams& p, const StreamPlan& plan, cudaStream_t stream, cudaError_t* err) {
  *err = CheckConfiguredDevice();
  if (*err != cudaSuccess) return true;
  if (reinterpret_cast<uintptr_t>(p.x) % 16 != 0) return false;
  if (p.fuse && (p.gk % 8 != 0 || reinterpret_cast<uintptr_t>(p.x2) % 16 != 0 || reinterpret_cast<uintptr_t>(p.gx) % 16 != 0 || reinterpret_cast<uintptr_t>(p.gw) % 16 != 0))
    return false;
  StreamParams q;
  bool odd = false;
  for (int s = 0; s < p.nseg; ++s) odd = odd || (mode == kNvfp4 && p.seg[s].pitch % 16 != 0);
  const StreamLayout l = LayOut(mode, odd, p.K, plan, p.M);
  p.wn = l.wn;
  p.wk = plan.wk * plan.teams;
  p.cluster = plan.cluster;
  p.gran = StreamGran(mode);
  p.stages = l.stages;
  p.stage_bytes = l.stage;
  p.ring_bytes = l.ring;
  p.xpitch = l.xpitch;
  p.tail_groups = plan.tail;
  p.tail_split = plan.tail_split;
  int tiles = 0;
  for (int s = 0; s < p.nseg; ++s) {
    p.seg[s].tile_begin = tiles;
    p.seg[s].tiles = plan.tiles[s];
    p.seg[s].tail_cols = plan.tail * 128;
    p.seg[s].granules = (p.seg[s].n - p.seg[s].tail_cols) / p.gran;
    if (plan.tiles[s] < 1 || plan.tiles[s] > 65535) {
      *err = cudaErrorInvalidValue;
      return true;
    }
    p.seg[s].gran_quot = p.seg[s].granules / plan.tiles[s];
    p.seg[s].gran_rem = p.seg[s].granules % plan.tiles[s];
    tiles += plan.tiles[s];
  }
  p.tail_stride = plan.tail > 0 ? tiles / (plan.tail * plan.tail_split) : 0;
  if (plan.tail > 0 && (!p.lm || p.lm_tail == nullptr || p.tail_stride < 1)) {
    *err = cudaErrorInvalidValue;
    return true;
  }
  const uint32_t div = odd ? 2 : 1;
  q.boxes = l.boxes;
  q.box_rows = static_cast<uint32_t>(l.box_rows);
  for (int s = 0; s < p.nseg; ++s) {
    const Segment& sg = p.seg[s];
    const uint64_t rows = static_cast<uint64_t>(p.K) / div, row_bytes = static_cast<uint64_t>(sg.pitch) * div;
    if (!Encode8(&q.wmap[s], sg.w, rows, row_bytes, q.box_rows, static_cast<uint32_t>(l.pitch), l.swizzle)) return false;
    if (mode == kNvfp4 && !Encode8(&q.smap[s], sg.w, rows, row_bytes, q.box_rows, static_cast<uint32_t>(l.spitch))) return false;
    if (plan.tail > 0) {
      q.tail_pitch = odd ? 96 : 80;
      if (!Encode8(&q.tail_wmap, sg.w, rows, row_bytes, static_cast<uint32_t>(l.tail_rows) / 2, q.tail_pitch) ||
          !Encode8(&q.tail_smap, sg.w, rows, row_bytes, static_cast<uint32_t>(l.tail_rows) / 2, 16))
        return false;
      q.tail_rows = static_cast<uint32_t>(l.tail_rows);
      q.tail_tx = q.tail_rows * (q.tail_pitch + 16);
    }
  }
  q.g = p;
  q.teams = plan.teams;
  q.team_wk = plan.wk;
  q.team_warps = l.wn * plan.wk;
  q.team_inv = 65535 / q.team_warps + 1;
  q.warps = q.team_warps * plan.teams;
  q.rows = l.rows;
  q.nstages = l.nstages;
  q.odd = odd ? 1 : 0;
  q.pitch = static_cast<uint32_t>(l.pitch);
  q.spitch = static_cast<uint32_t>(l.spitch);
  q.half = static_cast<uint32_t>(l.rows / 2 * l.pitch);
  q.shalf = static_cast<uint32_t>(l.rows / 2 * l.spitch);
  q.swizzle = l.swizzle;
  q.col_boxes = l.swizzle > 0 ? l.row_bytes / l.swizzle : 1;
  q.scale_off = static_cast<uint32_t>(l.rows * l.row_bytes);
  q.tx = static_cast<uint32_t>(l.rows * (l.row_bytes + l.spitch));
  q.x_off = static_cast<uint32_t>(l.ring + l.tail_bytes);
  q.tail_off = static_cast<uint32_t>(l.ring);
  q.wn_inv = 65535 / l.wn + 1;
  q.row_warps = std::max(1, q.warps / p.M);
  q.row_pass = q.warps / q.row_warps;
  q.row_inv = 65535 / q.row_warps + 1;
  q.rank_cols = (l.wn * GeomOf(mode).cols_per_warp + plan.cluster - 1) / plan.cluster;
  const int threads = 32 * (q.warps + 1 + (plan.tail > 0 ? 1 : 0));
  *err = mode == kBf16 ? LaunchMode<kBf16>(q, tiles, threads, l.smem, stream)
         : mode == kFp8 ? LaunchMode<kFp8>(q, tiles, threads, l.smem, stream)
                        : LaunchMode<kNvfp4>(q, tiles, threads, l.smem, stream);
  return true;
}

}  // namespace qfg
