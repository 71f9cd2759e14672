// Calls with many rows on the tensor memory path: out[M, N] = x[M, K] @ W[K, N] with BF16, FP8 or NVFP4 weights,
// dequantised on the way into tensor memory or shared memory.
//
// A CTA computes tiles of 128 columns of W by `bm` rows of x (bm <= 256, a multiple of 16) with tcgen05.mma: the
// weights are the 128-row operand, read MN-major because a stored row of W is contiguous along N, and the rows of x
// are the bm-column operand, K-major as x is stored.  Both operands are BF16 in 128-byte-swizzled shared memory,
// 64 k per stage; the FP32 accumulators lie in tensor memory, two sets of them, so that the epilogue of a tile
// overlaps the products of the next.  Roles by warp:
//   0-3   epilogue: accumulators -> BF16 -> the output that owns the column
//   4     TMA producer: the x tile of every stage, and the weight tile where the weights are BF16
//   5     tensor memory allocation; one lane issues the MMAs
//   6     FP8 / NVFP4: copies the stored weights into a ring of their own (50-60 KB in flight per SM); 7 idles
//   8-23  FP8 / NVFP4: sixteen warps in two groups that take the stages in turn; a warp turns eight weight rows of a
//         stage into BF16, w_scale folded in before the one rounding
// Rows of x are what the dequantisation is shared by: at bm = 256 a stage takes the tensor core 512 cycles.
// TM, tiles of up to 128 rows of FP8 or NVFP4 (rows on 16 bytes): the weights are dequantised into tensor memory, by four groups of four
// warps, and the MMA reads its first operand there (DequantTmRole).
//
// K is split over the CTAs of a cluster where the tiles alone leave SMs idle; the ranks then add their accumulators
// through distributed shared memory in rank order.  PAIR: two CTAs of a cluster work on 256 columns with
// cta_group::2; each holds its own 128 columns of W and half of the rows of x, which halves what the SMs fetch of x
// from L2 (a 128 x 256 tile fetches 36 KB per 512 cycles, more than an SM's share of L2).
//
// What bounds it.  Few rows: MMAs of 64 cycles whatever their rows up to 64 (FP4 at 33 rows, 5120 x 17408: 18.3 us; through shared
// memory, whose bandwidth the operand written and read back took, 21.5, and the dequantisation pass and the library GEMM that this kernel
// took the place of, 86.6).  Many rows: the copies from L2 (20 KB a block and SM in pairs of 192 rows, 9.1 TB/s in all), the tensor core
// at its rate under the power cap, and the last wave (FP8, 509 rows, 5120 x 10240: 62 to 64 us against 92.5; FP4, 2048 rows, 5120 x
// 17408: 288 to 298 us against 333).  Through shared memory the weights are written MN-major because that is how a stored row
// lies: a nibble byte is two neighbouring columns.
//
// Every wait is bounded.  A CTA that gives up on one writes NaN to the rest of its tiles and leaves: the call then reports
// no error, but no output keeps what its memory held before.
#include <cooperative_groups.h>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <climits>
#include <cstdlib>
#include <map>
#include <mutex>
#include <stdexcept>
#include <string>
#include <type_traits>

#include "qfg_internal.h"
#include "stream_order.cuh"
#include "swish.cuh"
#include "tensor_map.h"

namespace qfg {
namespace {

namespace cg = cooperative_groups;

constexpr int kBn = 128;           // columns of W per CTA
constexpr int kBk = 64;            // k per block: one 128-byte swizzled row of x; a stage holds KS = 1 or 2 blocks
constexpr int kABytes = kBn * kBk * 2;
constexpr int kMaxStages = 8;
constexpr int kDqWarps = 8;        // warps that fill one stage, eight weight rows each
constexpr int kDqGroups = 2;       // groups of them, taking the stages in turn
constexpr int kLoadWarps = 2;     // the first copies the stored rows into the raw ring, the second keeps the others in groups of four
constexpr int kFirstDqWarp = 6 + kLoadWarps;
constexpr int kMaxRaw = 12;
constexpr int kSpin = 1 << 20;

// Inside this file NVFP4 has two modes.  Where N is an odd multiple of 128 the stored rows are an odd multiple of eight bytes
// long, and every second one starts off the 16 bytes that a tensor copy has to start on.  Two rows are then one row of the
// tensor map, and an odd row is copied from the 16-byte boundary before it.
constexpr int kNvfp4Odd = 3;
template <int MODE>
constexpr bool kFp4 = MODE == kNvfp4 || MODE == kNvfp4Odd;
constexpr int kOddPitch = 80;  // nibble bytes copied of an odd row: 8 before the 64 of the tile, and 16-byte steps

template <int MODE, int KS>
struct RawRing {  // ring of stored, undequantised stages
  static constexpr int kRows = kBk * KS;
  static constexpr int kScales = kRows * (MODE == kNvfp4Odd ? kOddPitch : 64);  // NVFP4: where a slot's scales begin
  static constexpr int kSlot = kFp4<MODE> ? kScales + kRows * 16 : kRows * 128;
  // even: a slot then always serves the same group of dequantising warps, which has seen its previous phase complete
  static constexpr int kDepth = MODE == kNvfp4 ? (KS == 1 ? 10 : 6) : MODE == kNvfp4Odd ? (KS == 1 ? 8 : 4) : (KS == 1 ? 6 : 4);
  static constexpr int kBytes = MODE == kBf16 ? 0 : kSlot * kDepth;
  static_assert(kDepth <= kMaxRaw && kDepth % kDqGroups == 0 && kSlot % 256 == 0, "raw ring");
};
// Kernels that hand the weights over in tensor memory (TM, see DequantTmRole): four stages of two blocks, behind the two sets of
// accumulators of at most 128 rows
constexpr int kTmKs = 2, kTmStages = 4, kTmGroups = 4, kTmWarps = 4, kTmColumns = 512, kTmFirst = kTmColumns - kTmStages * kTmKs * 32, kTmBm = kTmFirst / 2;
constexpr int kOutPitch = 80;                     // bytes of a row of 32 output columns in an epilogue warp's buffer: rows 16 bytes apart in the banks
constexpr int kOutBytes = 4 * 32 * kOutPitch;     // four warps, 32 rows of x each

struct DenseSeg {
  const uint8_t* w;
  const float* w_scale;
  long long pitch, total_bytes;
  int n, tile_begin, out_begin, out_end;
};

struct DenseParams {
  CUtensorMap xmap;
  CUtensorMap wmap[kMaxSeg];  // stored weights (nibbles of NVFP4), where their rows are 16-byte aligned
  CUtensorMap smap[kMaxSeg];  // NVFP4 block scales
  DenseSeg seg[kMaxSeg];
  uint16_t* out[kMaxOut];
  int col_begin[kMaxOut], width[kMaxOut];
  int nseg, M, K, ksteps, bm, m_tiles, tiles, stages;
  int raw_depth;  // TM: slots of the raw ring
  int give_up;    // testing: 1: x never comes and every wait is short
  uint32_t out_vec;  // outputs whose rows can be written 16 bytes at a time
};

struct Ctl {
  unsigned long long full[kMaxStages], empty[kMaxStages], acc_full[2], acc_empty[2], raw_full[kMaxRaw], raw_empty[kMaxRaw];
  uint32_t tmem;
  volatile uint32_t fault;
};

// ------------------------------------------------------------------------------ PTX
__device__ __forceinline__ uint32_t Smem(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void BarInit(uint32_t a, int n) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(n) : "memory"); }
__device__ __forceinline__ void BarArrive(uint32_t a) {
  asm volatile("{ .reg .b64 st; mbarrier.arrive.shared::cta.b64 st, [%0]; }" ::"r"(a) : "memory");
}
__device__ __forceinline__ uint32_t MapRank(uint32_t a, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void BarExpect(uint32_t a, uint32_t bytes) {
  asm volatile("{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1; }" ::"r"(a), "r"(bytes) : "memory");
}
// arrives on the barrier of this CTA, or of the leader of its pair
template <bool PAIR>
__device__ __forceinline__ void BarArriveLeader(uint32_t a) {
  if constexpr (PAIR) {
    asm volatile("{ .reg .b32 r;\n mapa.shared::cluster.u32 r, %0, 0;\n mbarrier.arrive.shared::cluster.b64 _, [r];\n}" ::"r"(a) : "memory");
  } else {
    BarArrive(a);
  }
}
__device__ __forceinline__ bool BarTry(uint32_t a, uint32_t parity) {
  uint32_t ok;
  asm volatile("{ .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(a), "r"(parity) : "memory");
  return ok != 0;
}
// the same without the pause of up to a microsecond that try_wait may take where the phase is still open
__device__ __forceinline__ bool BarTest(uint32_t a, uint32_t parity) {
  uint32_t ok;
  asm volatile("{ .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(a), "r"(parity) : "memory");
  return ok != 0;
}
// false once a wait of this CTA ran out
__device__ __forceinline__ bool BarWait(uint32_t a, uint32_t parity, Ctl& c) {
  for (int i = 0; i < kSpin; ++i) {
    if (BarTry(a, parity)) return true;
    if ((i & 255) == 255 && c.fault) return false;
  }
  c.fault = 1;
  return false;
}
// the same where what is waited for was written by another CTA of the cluster
__device__ __forceinline__ bool BarWaitCluster(uint32_t a, uint32_t parity, Ctl& c) {
  for (int i = 0; i < kSpin; ++i) {
    uint32_t ok;
    asm volatile("{ .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(a), "r"(parity) : "memory");
    if (ok) return true;
    if ((i & 255) == 255 && c.fault) return false;
  }
  c.fault = 1;
  return false;
}
template <bool PAIR>
__device__ __forceinline__ void TmaLoad(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  if constexpr (PAIR) {  // the barrier may be the leader's
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
                 "l"(map), "r"(bar), "r"(x), "r"(y)
                 : "memory");
  } else {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst), "l"(map),
                 "r"(bar), "r"(x), "r"(y)
                 : "memory");
  }
}
// one lane of a converged warp; unlike a test of the lane number it leaves the compiler's view of the operands uniform,
// which the MMA's descriptors need (a lane test cost 80 cycles per MMA and 350 per wait)
__device__ __forceinline__ bool ElectOne() {
  uint32_t yes;
  asm volatile("{ .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(yes)::"memory");
  return yes != 0;
}
template <bool PAIR>
__device__ __forceinline__ void MmaSs(uint32_t d, unsigned long long a, unsigned long long b, uint32_t idesc, bool add) {
  if constexpr (PAIR) {
    asm volatile("{ .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d), "l"(a), "l"(b),
                 "r"(idesc), "r"(add ? 1 : 0)
                 : "memory");
  } else {
    asm volatile("{ .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d), "l"(a), "l"(b),
                 "r"(idesc), "r"(add ? 1 : 0)
                 : "memory");
  }
}
template <bool PAIR>
__device__ __forceinline__ void MmaTs(uint32_t d, uint32_t a, unsigned long long b, uint32_t idesc, bool add) {
  if constexpr (PAIR) {
    asm volatile("{ .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n}" ::"r"(d), "r"(a), "l"(b),
                 "r"(idesc), "r"(add ? 1 : 0)
                 : "memory");
  } else {
    asm volatile("{ .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}" ::"r"(d), "r"(a), "l"(b),
                 "r"(idesc), "r"(add ? 1 : 0)
                 : "memory");
  }
}
// arrives on the barrier (of both CTAs of a pair) when the MMAs issued so far have completed
template <bool PAIR>
__device__ __forceinline__ void MmaCommit(uint32_t bar) {
  if constexpr (PAIR) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                 "h"(static_cast<uint16_t>(3))
                 : "memory");
  } else {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
  }
}
__device__ __forceinline__ void FenceBefore() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void FenceAfter() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// 128-byte swizzle; `lbo`: distance of the 64-element groups of an MN-major operand (unused K-major), `sbo`: of the
// groups of eight rows
__device__ __forceinline__ unsigned long long SmemDesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return static_cast<unsigned long long>((addr >> 4) & 0x3FFF) | (static_cast<unsigned long long>(lbo >> 4) << 16) |
         (static_cast<unsigned long long>(sbo >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void Lds128(uint32_t a, uint32_t (&v)[4]) {
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(a));
}
__device__ __forceinline__ void Lds64(uint32_t a, uint32_t (&v)[2]) {
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v[0]), "=r"(v[1]) : "r"(a));
}
__device__ __forceinline__ uint32_t Lds8(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void LdsmTrans(uint32_t a, uint32_t (&v)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(a));
}
// sixteen lanes of tensor memory by 32 columns: register 2 i + h of lane (g, t) is lane 8 h + g, column 4 i + t
__device__ __forceinline__ void StoreTmem(uint32_t a, const uint32_t (&v)[16]) {
  asm volatile("tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(a), "r"(v[0]),
               "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]),
               "r"(v[14]), "r"(v[15])
               : "memory");
}
__device__ __forceinline__ void Sts128(uint32_t a, const uint32_t* v) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
__device__ __forceinline__ void CvtE2m1x8(uint32_t c, uint32_t (&r)[4]) {
  asm("{ .reg .b8 b0, b1, b2, b3;\n mov.b32 {b0, b1, b2, b3}, %4;\n cvt.rn.f16x2.e2m1x2 %0, b0;\n cvt.rn.f16x2.e2m1x2 %1, b1;\n"
      " cvt.rn.f16x2.e2m1x2 %2, b2;\n cvt.rn.f16x2.e2m1x2 %3, b3;\n}"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(c));
}
__device__ __forceinline__ void CvtE4m3x4(uint32_t c, uint32_t& lo, uint32_t& hi) {
  asm("{ .reg .b16 h0, h1;\n mov.b32 {h0, h1}, %2;\n cvt.rn.f16x2.e4m3x2 %0, h0;\n cvt.rn.f16x2.e4m3x2 %1, h1;\n}" : "=r"(lo), "=r"(hi) : "r"(c));
}
__device__ __forceinline__ uint32_t Hmul2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
// An FP16 pair (exact products of the stored formats) as BF16, times the scales of its two columns.  The two products in
// one instruction help where the conversion is short (FP8, 40 rows of 5120 x 10240: 24.8 -> 23.4 us) and cost 1 us in the
// FP4 kernel (5120 x 17408: 24.5 -> 25.5), which is short of registers for the pairs.
template <int MODE, bool SCALED>
__device__ __forceinline__ uint32_t ToBf16(uint32_t h, float s0, float s1) {
  float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
  if constexpr (SCALED && MODE == kFp8) {
    asm("{ .reg .b64 a, b;\n mov.b64 a, {%0, %1};\n mov.b64 b, {%2, %3};\n mul.rn.f32x2 a, a, b;\n mov.b64 {%0, %1}, a;\n}"
        : "+f"(f.x), "+f"(f.y)
        : "f"(s0), "f"(s1));
  } else if constexpr (SCALED) {
    f.x *= s0;
    f.y *= s1;
  }
  const __nv_bfloat162 b = __floats2bfloat162_rn(f.x, f.y);
  return *reinterpret_cast<const uint32_t*>(&b);
}

// ------------------------------------------------------------------------------ the walk over tiles
struct TileAt {
  int seg, n0, m0;
};
// tiles of one column block follow one another (all row blocks of it, then the next), so the SMs share its weights in L2
template <bool PAIR>
__device__ __forceinline__ TileAt LocateDense(const DenseParams& p, int tile, int rank) {
  TileAt t;
  const int nt = tile / p.m_tiles;
  t.m0 = (tile - nt * p.m_tiles) * p.bm;
  t.seg = 0;
#pragma unroll
  for (int i = 1; i < kMaxSeg; ++i) t.seg += (i < p.nseg && nt >= p.seg[i].tile_begin) ? 1 : 0;
  t.n0 = (nt - p.seg[t.seg].tile_begin) * (PAIR ? 2 * kBn : kBn) + (PAIR ? rank * kBn : 0);
  return t;
}

// ------------------------------------------------------------------------------ loading warp
// Stored rows -> the raw ring, by one lane's tensor copies.  A slot holds one stage: FP8 [rows][128 bytes]; NVFP4 [rows][64
// nibble bytes], then [rows][the 16 bytes that hold the row's 8 block scales, at their offset in an aligned 16]; NVFP4 with
// odd rows [even rows][80], [odd rows][80], [even rows][16], [odd rows][16], the 80 of a row beginning up to 8 bytes before
// the tile.  (Such weights used to come in 8-byte cp.async pieces by two warps, 18 instructions a stage: 1024 rows of 5120 x
// 5248 81.2 us, now 48.7, and 54.8 by dequantisation and library GEMM; 33 rows 20.0, 13.2 and 24.5.)
template <int MODE, bool PAIR, int KS>
__device__ __forceinline__ void LoadTensor(const DenseParams& p, Ctl& ctl, int rank, int kbeg, int kcount, int first_tile, int tile_step, uint32_t ring,
                                           int depth = RawRing<MODE, KS>::kDepth) {
  using R = RawRing<MODE, KS>;
  const uint32_t full0 = Smem(&ctl.raw_full[0]), empty0 = Smem(&ctl.raw_empty[0]);
  int slot = 0;
  uint32_t parity = 1;
  bool first_round = true;
  for (int tile = first_tile; tile < p.tiles; tile += tile_step) {
    const TileAt t = LocateDense<PAIR>(p, tile, rank);
    const DenseSeg& sg = p.seg[t.seg];
    const int nib = t.n0 / 2, scl = sg.n / 2 + t.n0 / 16, odd = static_cast<int>(sg.pitch);
#pragma unroll 1
    for (int k = 0; k < kcount; ++k) {
      if (!first_round && !BarWait(empty0 + slot * 8, parity, ctl)) return;
      const uint32_t dst = ring + static_cast<uint32_t>(slot) * R::kSlot, bar = full0 + slot * 8;
      if (ElectOne()) {
        BarExpect(bar, R::kSlot);
        if constexpr (MODE == kNvfp4) {
          TmaLoad<false>(dst, &p.wmap[t.seg], nib, (kbeg + k) * R::kRows, bar);
          TmaLoad<false>(dst + R::kScales, &p.smap[t.seg], scl & ~15, (kbeg + k) * R::kRows, bar);
        } else if constexpr (MODE == kNvfp4Odd) {
          const int pair = (kbeg + k) * (R::kRows / 2);
          TmaLoad<false>(dst, &p.wmap[t.seg], nib, pair, bar);
          TmaLoad<false>(dst + R::kScales / 2, &p.wmap[t.seg], (nib + odd) & ~15, pair, bar);
          TmaLoad<false>(dst + R::kScales, &p.smap[t.seg], scl & ~15, pair, bar);
          TmaLoad<false>(dst + R::kScales + R::kRows * 8, &p.smap[t.seg], (scl + odd) & ~15, pair, bar);
        } else {
          TmaLoad<false>(dst, &p.wmap[t.seg], t.n0, (kbeg + k) * R::kRows, bar);
        }
      }
      __syncwarp();
      if (++slot == depth) {
        slot = 0;
        parity ^= 1u;
        first_round = false;
      }
    }
  }
}

// ------------------------------------------------------------------------------ dequantising warps
// A warp owns rows 8 w .. 8 w + 7 of its group's stages, all 128 columns.  A lane owns the 16 columns
// 16 (q + 4 a) of two of them (rows 2 (2 i + j) + par, i = 0, 1), with q = lane % 4, par = lane / 4 % 2, j = lane / 16
// and a = lane / 8 % 2 exclusive-or par.  That order keeps the 16-byte stores free of bank conflicts (the eight lanes of
// a store phase are four even chunks of an even and four of an odd row, which the swizzle moves apart) and the ring's
// loads too (the two rows' halves lie side by side in the banks).  These warps have no copies of their own in flight: the proxy fence that follows their stores waits for
// a thread's outstanding copies as well, so a warp that did both ran at one memory latency per stage (0.55 us, whatever
// the depth of its ring).
template <int MODE, bool SCALED, bool PAIR, int KS, int GROUPS>
__device__ __forceinline__ void DequantRole(const DenseParams& p, Ctl& ctl, int warp, int group, int lane, int rank, int kcount, int first_tile,
                                            int tile_step, uint32_t ring, uint32_t stage0, uint32_t block_bytes) {
  using R = RawRing<MODE, KS>;
  const uint32_t full0 = Smem(&ctl.full[0]), empty0 = Smem(&ctl.empty[0]), rfull0 = Smem(&ctl.raw_full[0]), rempty0 = Smem(&ctl.raw_empty[0]);
  const int q = lane & 3, par = (lane >> 2) & 1, a = ((lane >> 3) & 1) ^ par, jj = lane >> 4, g = q + 4 * a;
  // where the lane's chunks go: row r = 4 i + 2 jj + par of the warp's eight, chunks 2 q and 2 q + 1 exclusive-or r
  const int r0 = 2 * jj + par;
  const uint32_t st0 = stage0 + static_cast<uint32_t>(a * (kABytes / 2) + warp * 1024 + r0 * 128 + (((2 * q) ^ r0) * 16));
  const uint32_t row0 = static_cast<uint32_t>(warp * 8 + r0);
  // where they come from: bytes of a row, of its scales, and from the first of the lane's two rows (r0, r0 + 4) to the second;
  // the parity of its rows is par
  constexpr bool kOdd = MODE == kNvfp4Odd;
  constexpr uint32_t kRow = kOdd ? kOddPitch / 2 : kFp4<MODE> ? 64 : 128, kScaleRow = kOdd ? 8 : 16;
  const uint32_t first_row = kOdd ? row0 & ~1u : row0;
  const uint32_t rd_row = ring + first_row * kRow + static_cast<uint32_t>(g * (kFp4<MODE> ? 8 : 16)) + (kOdd ? static_cast<uint32_t>(par * (R::kScales / 2)) : 0u);
  const uint32_t rd_scale_row = ring + R::kScales + first_row * kScaleRow + static_cast<uint32_t>(g) + (kOdd ? static_cast<uint32_t>(par * R::kRows * 8) : 0u);
  int stage = group % p.stages, slot = group % R::kDepth, tile = first_tile, k = group;
  uint32_t parity = static_cast<uint32_t>(group / p.stages) & 1u, rparity = 0;
  bool first_round = group < p.stages;
  auto next_tile = [&]() {  // the stages alternate between the groups across tile boundaries too
    while (k >= kcount && tile < p.tiles) {
      k -= kcount;
      tile += tile_step;
    }
  };
  next_tile();
  while (tile < p.tiles) {
    const TileAt t = LocateDense<PAIR>(p, tile, rank);
    const DenseSeg& sg = p.seg[t.seg];
    float cs[SCALED ? 16 : 1];
    cs[0] = 1.f;
    if constexpr (SCALED) {
      const int n = t.n0 + 16 * g;
#pragma unroll
      for (int i = 0; i < 16; ++i) cs[i] = (sg.w_scale != nullptr && n + i < sg.n) ? __ldg(sg.w_scale + n + i) : 1.f;
    }
    // the offset in their 16 bytes: of the scales, n0 / 16 is a multiple of eight, N / 2 of sixteen; of an odd row, eight bytes
    const uint32_t shift = kOdd && par ? static_cast<uint32_t>(sg.pitch) & 8u : 0u;
    const uint32_t rd_w = rd_row + shift, rd_s = rd_scale_row + ((static_cast<uint32_t>(t.n0 >> 4) + shift) & 8u);
#pragma unroll 1
    for (; k < kcount; k += GROUPS) {
      // both asked at once, the answer of the second needed after the first conversions
      const bool room = first_round || BarTest(empty0 + stage * 8, parity ^ 1u);
      if (!BarWait(rfull0 + slot * 8, rparity, ctl)) return;
      const uint32_t at = static_cast<uint32_t>(slot) * R::kSlot;
      uint32_t raw[KS][2][4], sc[KS][2];
#pragma unroll
      for (int j = 0; j < KS; ++j) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if constexpr (kFp4<MODE>) {
            uint32_t v[2];
            Lds64(rd_w + at + j * (kBk * kRow) + i * (4 * kRow), v);
            raw[j][i][0] = v[0];
            raw[j][i][1] = v[1];
            sc[j][i] = Lds8(rd_s + at + j * (kBk * kScaleRow) + i * (4 * kScaleRow));
          } else {
            Lds128(rd_w + at + j * (kBk * kRow) + i * (4 * kRow), raw[j][i]);
          }
        }
      }
      uint32_t dst = st0 + static_cast<uint32_t>(stage * KS) * block_bytes;
#pragma unroll
      for (int j = 0; j < KS; ++j) {
        uint32_t o[2][8];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          uint32_t h[8];
          if constexpr (kFp4<MODE>) {
            uint32_t lo[4], hi[4], s, unused;
            CvtE4m3x4(sc[j][i] * 0x101u, s, unused);
            CvtE2m1x8(raw[j][i][0], lo);
            CvtE2m1x8(raw[j][i][1], hi);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              h[e] = Hmul2(lo[e], s);
              h[4 + e] = Hmul2(hi[e], s);
            }
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) CvtE4m3x4(raw[j][i][e], h[2 * e], h[2 * e + 1]);
          }
#pragma unroll
          for (int e = 0; e < 8; ++e) o[i][e] = ToBf16<MODE, SCALED>(h[e], cs[SCALED ? 2 * e : 0], cs[SCALED ? 2 * e + 1 : 0]);
        }
        if (j == 0 && !room && !BarWait(empty0 + stage * 8, parity ^ 1u, ctl)) return;
        // rows r0 and r0 + 4: the chunk index changes by bit 0 (second half of the columns) and bit 2 (row)
        Sts128(dst, o[0]);
        Sts128(dst ^ 16u, o[0] + 4);
        Sts128((dst + 512) ^ 64u, o[1]);
        Sts128((dst + 512) ^ 80u, o[1] + 4);
        dst += block_bytes;
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      // the raw slot is given back only here, behind stores that depend on its loads: the compiler is free to move a
      // plain shared-memory load past an arrival, and did so (stages overwritten before they were read)
      if (lane == 0) {
        BarArrive(rempty0 + slot * 8);
        BarArriveLeader<PAIR>(full0 + stage * 8);
      }
      slot += GROUPS;
      if (slot >= R::kDepth) {
        slot -= R::kDepth;
        rparity ^= 1u;
      }
      stage += GROUPS;
      if (stage >= p.stages) {
        stage -= p.stages;
        parity ^= 1u;
        first_round = false;
      }
    }
    next_tile();
  }
}

// Two values times the scales of their columns, in one instruction where the warps that do it set the pace (FP8, 33 rows of 5120 x 10240:
// 21.1 -> 20.2 us; in pairs, where they wait for room, 509 rows 59.5 -> 60.9).
template <bool PAIR>
__device__ __forceinline__ void ScalePair(float (&v)[2], const float (&s)[2]) {
  if constexpr (PAIR) {
    v[0] *= s[0];
    v[1] *= s[1];
  } else {
    asm("{ .reg .b64 a, b;\n mov.b64 a, {%0, %1};\n mov.b64 b, {%2, %3};\n mul.rn.f32x2 a, a, b;\n mov.b64 {%0, %1}, a;\n}"
        : "+f"(v[0]), "+f"(v[1])
        : "f"(s[0]), "f"(s[1]));
  }
}
// The same for tiles of up to 128 rows, with the weights in tensor memory instead of shared memory: there the tensor core's
// operand does not compete for the 128 bytes a cycle of shared memory, which a block of 64 k and few rows fills (16 KB
// written and 16 KB read of 54 KB at 33 rows: 400 cycles a block, an MMA every 85).  5120 x 17408, NVFP4, 17 / 33 / 64 rows 20.8 / 21.5 / 23.5
// -> 16.5 / 18.4 / 20.3 us, FP8 5120 x 10240 22.0 / 22.6 / 23.4 -> 17.1 / 17.9 / 18.6.  Four warps, one for each 32 lanes of tensor memory, take a stage; four such groups take the stages in
// turn.  Lane (g, t) loads two stored bytes of rows 2t and 2t + 1 of every eight by transposing loads (the ring is swizzled, so
// they are free of bank conflicts), turns them into FP32, by one mixed FMA each with the block scale of its row (NVFP4),
// and packs rows 2t and 2t + 1 of a column into the word that the operand wants: pairs along k, though the bytes hold pairs along N.
// Lane 16 s + 8 h + g of the 32 then is column 16 s + 2 g + h (FP8), or 4 g + 2 s + h (NVFP4) of the warp's, see TmColumn.
template <int MODE>
__device__ __forceinline__ int TmColumn(int s, int h, int g) {
  return MODE == kFp8 ? 16 * s + 2 * g + h : 4 * g + 2 * s + h;
}
template <int MODE, bool SCALED, bool PAIR>
__device__ __forceinline__ void DequantTmRole(const DenseParams& p, Ctl& ctl, int warp, int lane, int rank, int kcount, int first_tile, int tile_step, uint32_t ring,
                                              uint32_t tmem) {
  using R = RawRing<MODE, kTmKs>;
  constexpr bool kNib = kFp4<MODE>;
  const uint32_t full0 = Smem(&ctl.full[0]), empty0 = Smem(&ctl.empty[0]), rfull0 = Smem(&ctl.raw_full[0]), rempty0 = Smem(&ctl.raw_empty[0]);
  const int quad = warp & 3, group = warp >> 2, g = lane >> 2, t = lane & 3;
  // this lane's row address of a transposing load.  NVFP4: four times eight rows of the warp's 16 bytes; FP8: twice eight rows of
  // its two times 16 bytes.  Swizzled: 16-byte pieces exclusive-or bits 7 to 8 (9) of the address.
  const int row = kNib ? lane : (lane & 15), piece = kNib ? quad ^ ((lane >> 1) & 3) : (2 * quad + (lane >> 4)) ^ (lane & 7);
  const uint32_t rd = ring + static_cast<uint32_t>(row * (kNib ? 64 : 128) + piece * 16);
  const uint32_t rd_s = ring + R::kScales + static_cast<uint32_t>(2 * t * 16 + 2 * quad + (g >> 2));
  const uint32_t a0 = tmem + kTmFirst + (static_cast<uint32_t>(32 * quad) << 16);
  const float zero = -0.f;  // the addend that leaves the sign of a zero as it is
  int stage = group % kTmStages, slot = group % p.raw_depth, tile = first_tile, k = group;
  uint32_t parity = 0, rparity = 0;
  bool first_round = true;
  auto next_tile = [&]() {  // the stages go from group to group across tile boundaries too
    while (k >= kcount && tile < p.tiles) {
      k -= kcount;
      tile += tile_step;
    }
  };
  next_tile();
  while (tile < p.tiles) {
    const TileAt at_tile = LocateDense<PAIR>(p, tile, rank);
    const DenseSeg& sg = p.seg[at_tile.seg];
    float cs[2][2] = {{1.f, 1.f}, {1.f, 1.f}};
    if constexpr (SCALED) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int n = at_tile.n0 + 32 * quad + TmColumn<MODE>(i >> 1, i & 1, g);
        cs[i >> 1][i & 1] = (sg.w_scale != nullptr && n < sg.n) ? __ldg(sg.w_scale + n) : 1.f;
      }
    }
    const uint32_t shift = static_cast<uint32_t>(at_tile.n0 >> 4) & 8u;  // of the scales in their 16 bytes
#pragma unroll 1
    for (; k < kcount; k += kTmGroups) {
      const bool room = first_round || BarTest(empty0 + stage * 8, parity ^ 1u);
      if (!BarWait(rfull0 + slot * 8, rparity, ctl)) return;
      const uint32_t at = static_cast<uint32_t>(slot) * R::kSlot;
      bool free = room;
#pragma unroll
      for (int j = 0; j < kTmKs; ++j) {
        uint32_t v[2][16];
#pragma unroll
        for (int q = 0; q < (kNib ? 2 : 4); ++q) {
          uint32_t raw[4];
          LdsmTrans(rd + at + static_cast<uint32_t>((j * kBk + q * (kNib ? 32 : 16)) * (kNib ? 64 : 128)), raw);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float lo[2][2], hi[2][2];  // [set][half]: rows 2t and 2t + 1 of the lane's columns
            if constexpr (kNib) {
              const uint32_t rs = rd_s + at + shift + static_cast<uint32_t>((j * kBk + q * 32 + i * 8) * 16);
              uint32_t h[4], s, unused;
              CvtE4m3x4(Lds8(rs) | (Lds8(rs + 16) << 8), s, unused);
              CvtE2m1x8(raw[i], h);
#pragma unroll
              for (int u = 0; u < 2; ++u) {
                asm("{ .reg .f16 a, b, s, t;\n mov.b32 {a, b}, %2;\n mov.b32 {s, t}, %3;\n fma.rn.f32.f16 %0, a, s, %4;\n fma.rn.f32.f16 %1, b, s, %4;\n}"
                    : "=f"(lo[u][0]), "=f"(lo[u][1]) : "r"(h[u]), "r"(s), "f"(zero));
                asm("{ .reg .f16 a, b, s, t;\n mov.b32 {a, b}, %2;\n mov.b32 {s, t}, %3;\n fma.rn.f32.f16 %0, a, t, %4;\n fma.rn.f32.f16 %1, b, t, %4;\n}"
                    : "=f"(hi[u][0]), "=f"(hi[u][1]) : "r"(h[2 + u]), "r"(s), "f"(zero));
              }
#pragma unroll
              for (int u = 0; u < 2; ++u) {
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                  if (SCALED && e == 0) ScalePair<PAIR>(lo[u], cs[u]), ScalePair<PAIR>(hi[u], cs[u]);
                  v[u][2 * (4 * q + i) + e] = PackBf16(lo[u][e], hi[u][e]);
                }
              }
            } else {
              uint32_t ha, hb;
              CvtE4m3x4(raw[i], ha, hb);
              constexpr int u0 = 0;
              asm("{ .reg .f16 a, b;\n mov.b32 {a, b}, %2;\n add.f32.f16 %0, a, %3;\n add.f32.f16 %1, b, %3;\n}" : "=f"(lo[u0][0]), "=f"(lo[u0][1]) : "r"(ha), "f"(zero));
              asm("{ .reg .f16 a, b;\n mov.b32 {a, b}, %2;\n add.f32.f16 %0, a, %3;\n add.f32.f16 %1, b, %3;\n}" : "=f"(hi[u0][0]), "=f"(hi[u0][1]) : "r"(hb), "f"(zero));
              const int u = i >> 1, i8 = 2 * q + (i & 1);  // raw: rows 0 to 7, 8 to 15 of the first 16 bytes, then of the second
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                if (SCALED && e == 0) ScalePair<PAIR>(lo[u0], cs[u]), ScalePair<PAIR>(hi[u0], cs[u]);
                v[u][2 * i8 + e] = PackBf16(lo[u0][e], hi[u0][e]);
              }
            }
          }
        }
        if (!free && !BarWait(empty0 + stage * 8, parity ^ 1u, ctl)) return;
        if (j == 0) {
          free = true;
          __syncwarp();
          FenceAfter();
        }
        const uint32_t a = a0 + static_cast<uint32_t>((stage * kTmKs + j) * 32);
        StoreTmem(a, v[0]);
        StoreTmem(a + (16u << 16), v[1]);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      FenceBefore();
      __syncwarp();
      if (lane == 0) {  // behind stores that depend on the ring's loads, as in DequantRole
        BarArrive(rempty0 + slot * 8);
        BarArriveLeader<PAIR>(full0 + stage * 8);
      }
      slot += kTmGroups;
      if (slot >= p.raw_depth) {
        slot -= p.raw_depth;
        rparity ^= 1u;
      }
      // as many stages as groups: a group always fills the same one
      parity ^= 1u;
      first_round = false;
    }
    next_tile();
  }
}

template <int MODE>
constexpr int DenseThreads() {
  return 32 * (kFirstDqWarp + (MODE == kBf16 ? 0 : kDqWarps * kDqGroups));
}

// SPLIT: K is split over the CTAs of the cluster, one tile per cluster.  PAIR: see above.  Never both.  TM: the weights go through
// tensor memory.
template <int MODE, bool SCALED, bool PAIR, bool SPLIT, int KS, bool TM>
__global__ void __launch_bounds__(DenseThreads<MODE>(), 1) DenseTcKernel(const __grid_constant__ DenseParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ Ctl ctl;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const uint32_t smem = (Smem(smem_raw) + 1023u) & ~1023u;
  uint8_t* const smem_ptr = smem_raw + (smem - Smem(smem_raw));
  const int csize = (PAIR || SPLIT) ? static_cast<int>(cg::this_cluster().num_blocks()) : 1;
  const int rank = (PAIR || SPLIT) ? static_cast<int>(cg::this_cluster().block_rank()) : 0;
  const int first_tile = static_cast<int>(blockIdx.x) / csize, tile_step = static_cast<int>(gridDim.x) / csize;
  const int kbeg = SPLIT ? rank * p.ksteps / csize : 0;
  const int kcount = SPLIT ? (rank + 1) * p.ksteps / csize - kbeg : p.ksteps;
  const int xrows = PAIR ? p.bm / 2 : p.bm;
  static_assert(!TM || (KS == kTmKs && (MODE == kFp8 || MODE == kNvfp4)), "");
  constexpr int kX = TM ? 0 : kABytes;  // where x begins in a block
  const uint32_t block_bytes = static_cast<uint32_t>(kX + xrows * kBk * 2), stage_bytes = block_bytes * KS;
  const uint32_t full0 = Smem(&ctl.full[0]), empty0 = Smem(&ctl.empty[0]), accf0 = Smem(&ctl.acc_full[0]), acce0 = Smem(&ctl.acc_empty[0]);
  int acc_cols = TM ? kTmColumns : 32;
  while (acc_cols < 2 * p.bm) acc_cols *= 2;
  const int raw_depth = TM ? p.raw_depth : RawRing<MODE, KS>::kDepth;

  if (tid == 0) {
    for (int i = 0; i < p.stages; ++i) {
      BarInit(full0 + i * 8, 1 + (MODE == kBf16 ? 0 : (TM ? kTmWarps : kDqWarps) * (PAIR ? 2 : 1)));
      BarInit(empty0 + i * 8, 1);
    }
    for (int i = 0; i < 2; ++i) {
      BarInit(accf0 + i * 8, 1);
      BarInit(acce0 + i * 8, 4 * (PAIR ? 2 : 1));
    }
    for (int i = 0; MODE != kBf16 && i < raw_depth; ++i) {
      BarInit(Smem(&ctl.raw_full[i]), 1);
      BarInit(Smem(&ctl.raw_empty[i]), TM ? kTmWarps : kDqWarps);
    }
    ctl.fault = static_cast<uint32_t>(p.give_up);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 4 && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&p.xmap) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&p.wmap[0]) : "memory");
    if (kFp4<MODE>) asm volatile("prefetch.tensormap [%0];" ::"l"(&p.smap[0]) : "memory");
  }
  if (warp == 5) {
    if constexpr (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(Smem(&ctl.tmem)), "r"(acc_cols) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(Smem(&ctl.tmem)), "r"(acc_cols) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  FenceBefore();
  GridDependencyWait();
  __syncthreads();
  if constexpr (PAIR) cg::this_cluster().sync();  // the leader's barriers exist before the peer arrives on them
  FenceAfter();
  const uint32_t tmem = ctl.tmem;

  if (warp < 4) {
    // ---- epilogue
    const uint32_t raw_bytes = TM ? static_cast<uint32_t>(RawRing<MODE, KS>::kSlot * raw_depth) : static_cast<uint32_t>(RawRing<MODE, KS>::kBytes);
    const uint32_t buf = smem + static_cast<uint32_t>(p.stages) * stage_bytes + raw_bytes + static_cast<uint32_t>(warp * 32 * kOutPitch);
    int it = 0;
    bool good = true;  // false from the first wait that ran out: no sums come any more, and the tiles that are left become NaN
    for (int tile = first_tile; tile < p.tiles; tile += tile_step, ++it) {
      const int b = it & 1;
      good = good && BarWait(accf0 + b * 8, static_cast<uint32_t>((it >> 1) & 1), ctl);
      __syncwarp();
      FenceAfter();
      const TileAt t = LocateDense<PAIR>(p, tile, rank);
      const uint32_t src = tmem + (static_cast<uint32_t>(32 * warp) << 16) + static_cast<uint32_t>(b * p.bm);
      if constexpr (SPLIT) {  // lane = column 32 warp + lane of the tile
        // The sums go where the stages were.  After a wait that ran out, copies may still be landing there and other warps may
        // not have given up yet, and would write over the NaN that the peers are to see: leave them time (a flag for the peers,
        // read after they meet, made every call 3-5 % slower).
        for (int i = 0; i < 16 && !good; ++i) __nanosleep(1000000);
        for (int c = 0; c < p.bm; c += 16) {
          uint32_t v[16];
          asm volatile(
              "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
              : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
                "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
              : "r"(src + static_cast<uint32_t>(c)));
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          const int col = TM ? TmColumn<MODE>(lane >> 4, (lane >> 3) & 1, lane & 7) : lane;
          float* part = reinterpret_cast<float*>(smem_ptr) + c * kBn + 32 * warp + col;
#pragma unroll
          for (int i = 0; i < 16; ++i) part[i * kBn] = good ? __uint_as_float(v[i]) : __uint_as_float(0x7FFFFFFFu);
        }
      } else {
        // A lane stores eight columns of a row at a time: the accumulators come as 8 x 8 fragments, columns of W down
        // and rows of x across, and go through shared memory transposed.  One column per lane, two bytes a store, took
        // 50 cycles a row and warp (a tile of 176 rows: 8700 cycles, a sixth of a call).
        const DenseSeg& sg = p.seg[t.seg];
        const int chunk = lane & 3, row = lane >> 2, n = t.n0 + 32 * warp + 8 * chunk;  // widths are multiples of eight
        int j = sg.out_begin;
        for (int i = j + 1; i < sg.out_end; ++i) {
          if (n >= p.col_begin[i]) j = i;
        }
        const size_t width = static_cast<size_t>(p.width[j]);
        uint16_t* const out = p.out[j] + static_cast<size_t>(t.m0) * width + (n - p.col_begin[j]);
        const bool vec = (p.out_vec >> j) & 1u;
        const int rows = n < sg.n ? min(p.bm, p.M - t.m0) : 0;
        const uint32_t st = buf + static_cast<uint32_t>((((lane >> 4) & 1) * 8 + (lane & 7)) * kOutPitch + ((lane >> 3) & 1) * 16);
        const uint32_t ld = buf + static_cast<uint32_t>(row * kOutPitch + chunk * 16);
        for (int c = 0; c < p.bm; c += 32) {
          uint32_t v[2][2][8];  // [lower, upper 16 columns][16 rows][fragments]
#pragma unroll
          for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              if (k == 0 || c + 16 < p.bm) {
                uint32_t(&f)[8] = v[h][k];
                asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                             : "=r"(f[0]), "=r"(f[1]), "=r"(f[2]), "=r"(f[3]), "=r"(f[4]), "=r"(f[5]), "=r"(f[6]), "=r"(f[7])
                             : "r"(src + (static_cast<uint32_t>(16 * h) << 16) + static_cast<uint32_t>(c + 16 * k)));
              }
            }
          }
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          __syncwarp();  // the rows before have been read
#pragma unroll
          for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              if constexpr (TM) {
                if (k == 0 || c + 16 < p.bm) {
                  // lanes g and g + 8 are neighbouring columns: their words lie beside one another, rows 2t, 2t + 1 and eight on
                  const int lane_t = lane & 3, word = TmColumn<MODE>(h, 0, lane >> 2) / 2;
                  const uint32_t to = buf + static_cast<uint32_t>((16 * k + 2 * lane_t) * kOutPitch + word * 4);
                  const uint32_t(&f)[8] = v[h][k];
#pragma unroll
                  for (int i = 0; i < 4; ++i) {
                    const int lo = 4 * (i >> 1) + (i & 1);
                    const uint32_t w = good ? PackBf16(__uint_as_float(f[lo]), __uint_as_float(f[lo + 2])) : 0x7FFF7FFFu;
                    asm volatile("st.shared.b32 [%0], %1;" ::"r"(to + static_cast<uint32_t>((8 * (i >> 1) + (i & 1)) * kOutPitch)), "r"(w) : "memory");
                  }
                }
              } else if (k == 0 || c + 16 < p.bm) {
                uint32_t w[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  const __nv_bfloat162 two = __floats2bfloat162_rn(__uint_as_float(v[h][k][2 * i]), __uint_as_float(v[h][k][2 * i + 1]));
                  w[i] = good ? *reinterpret_cast<const uint32_t*>(&two) : 0x7FFF7FFFu;
                }
                asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(st + k * (16 * kOutPitch) + h * 32),
                             "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3])
                             : "memory");
              }
            }
          }
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int r = c + 8 * i + row;
            if (r < rows) {
              uint32_t o[4];
              Lds128(ld + i * (8 * kOutPitch), o);
              uint16_t* const dst = out + static_cast<size_t>(r) * width;
              if (vec) {
                *reinterpret_cast<uint4*>(dst) = make_uint4(o[0], o[1], o[2], o[3]);
              } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) dst[e] = static_cast<uint16_t>(o[e >> 1] >> (16 * (e & 1)));
              }
            }
          }
        }
      }
      FenceBefore();
      __syncwarp();
      if (lane == 0 && good) BarArriveLeader<PAIR>(acce0 + b * 8);
    }
  } else if (warp == 4) {
    // ---- x (and BF16 weights)
    int stage = 0, round = 0;
    bool good = p.give_up == 0;
    const uint32_t mine = static_cast<uint32_t>(KS * (xrows * kBk * 2 + (MODE == kBf16 ? kABytes : 0)));
    for (int tile = first_tile; tile < p.tiles && good; tile += tile_step) {
      const TileAt t = LocateDense<PAIR>(p, tile, rank);
      for (int k = 0; k < kcount; ++k) {
        if (round > 0 && !BarWait(empty0 + stage * 8, static_cast<uint32_t>((round - 1) & 1), ctl)) {
          good = false;
          break;
        }
        const uint32_t bar = PAIR ? MapRank(full0 + stage * 8, 0) : full0 + stage * 8;
        const uint32_t dst = smem + static_cast<uint32_t>(stage) * stage_bytes;
        if (ElectOne()) {
          if (rank == 0 || !PAIR) BarExpect(full0 + stage * 8, PAIR ? 2 * mine : mine);
#pragma unroll
          for (int j = 0; j < KS; ++j) {
            const int k0 = ((kbeg + k) * KS + j) * kBk;
            const uint32_t at = dst + static_cast<uint32_t>(j) * block_bytes;
            if constexpr (MODE == kBf16) {
              TmaLoad<PAIR>(at, &p.wmap[t.seg], t.n0, k0, bar);
              TmaLoad<PAIR>(at + kABytes / 2, &p.wmap[t.seg], t.n0 + 64, k0, bar);
            }
            TmaLoad<PAIR>(at + kX, &p.xmap, k0, t.m0 + (PAIR ? rank * xrows : 0), bar);
          }
        }
        __syncwarp();
        if (++stage == p.stages) {
          stage = 0;
          ++round;
        }
      }
    }
  } else if (warp == 5) {
    // ---- MMAs (the leader's, for both CTAs of a pair)
    if (!PAIR || rank == 0) {
      // FP32 accumulators, BF16 operands, A MN-major, N = bm, M = 128 (256 across a pair)
      const uint32_t idesc = 0x10u | (1u << 7) | (1u << 10) | (TM ? 0u : 1u << 15) | (static_cast<uint32_t>(p.bm >> 3) << 17) |
                             (static_cast<uint32_t>(PAIR ? 16 : 8) << 24);
      const unsigned long long a0 = SmemDesc(smem, kABytes / 2, 1024), b0 = SmemDesc(smem + kX, 16, 1024);
      int stage = 0, it = 0;
      uint32_t parity = 0;
      bool good = true, ready = false;
      for (int tile = first_tile; tile < p.tiles && good; tile += tile_step, ++it) {
        const int b = it & 1;
        if (it >= 2 && !BarWait(acce0 + b * 8, static_cast<uint32_t>(((it >> 1) - 1) & 1), ctl)) break;
        FenceAfter();
        const uint32_t d = tmem + static_cast<uint32_t>(b * p.bm);
        for (int k = 0; k < kcount; ++k) {
          if (!ready && !BarWait(full0 + stage * 8, parity, ctl)) {
            good = false;
            break;
          }
          FenceAfter();
          const uint32_t off = static_cast<uint32_t>(stage) * stage_bytes >> 4, done = empty0 + stage * 8, a_tm = tmem + kTmFirst + static_cast<uint32_t>(stage * KS * 32);
          if (++stage == p.stages) {
            stage = 0;
            parity ^= 1u;
          }
          ready = BarTest(full0 + stage * 8, parity);  // asked before the MMAs are issued, needed after
          if (ElectOne()) {
#pragma unroll
            for (int j = 0; j < KS; ++j) {
#pragma unroll
              for (int i = 0; i < kBk / 16; ++i) {
                const uint32_t at = off + j * (block_bytes >> 4);
                if constexpr (TM) {
                  MmaTs<PAIR>(d, a_tm + j * 32 + i * 8, b0 + at + i * (32 >> 4), idesc, k > 0 || i + j > 0);
                } else {
                  MmaSs<PAIR>(d, a0 + at + i * (2048 >> 4), b0 + at + i * (32 >> 4), idesc, k > 0 || i + j > 0);
                }
              }
            }
            MmaCommit<PAIR>(done);
            if (k == kcount - 1) MmaCommit<PAIR>(accf0 + b * 8);
          }
          __syncwarp();
        }
      }
    }
  } else if constexpr (MODE != kBf16) {
    const uint32_t ring = smem + static_cast<uint32_t>(p.stages) * stage_bytes;
    if (warp < kFirstDqWarp) {
      if (warp == 6) LoadTensor<MODE, PAIR, KS>(p, ctl, rank, kbeg, kcount, first_tile, tile_step, ring, raw_depth);
    } else {
      const int w = warp - kFirstDqWarp;
      if constexpr (TM) {
        DequantTmRole<MODE, SCALED, PAIR>(p, ctl, w, lane, rank, kcount, first_tile, tile_step, ring, tmem);
      } else {
        DequantRole<MODE, SCALED, PAIR, KS, kDqGroups>(p, ctl, w % kDqWarps, w / kDqWarps, lane, rank, kcount, first_tile, tile_step, ring, smem, block_bytes);
      }
    }
  }

  if constexpr (SPLIT) {
    // the ranks' sums meet: rank r finishes rows [r bm / C, (r + 1) bm / C) of the tile, adding in rank order
    cg::cluster_group cluster = cg::this_cluster();
    FenceBefore();
    cluster.sync();
    const TileAt t = LocateDense<PAIR>(p, first_tile, rank);
    const DenseSeg& sg = p.seg[t.seg];
    const float* part = reinterpret_cast<const float*>(smem_ptr);
    const int r0 = rank * p.bm / csize, r1 = (rank + 1) * p.bm / csize;
    const int c = (tid & 31) * 4, n = t.n0 + c;  // widths are multiples of eight: four columns belong to one output
    if (n < sg.n) {
      int j = sg.out_begin;
      for (int i = j + 1; i < sg.out_end; ++i) {
        if (n >= p.col_begin[i]) j = i;
      }
      uint16_t* const out = p.out[j] + (n - p.col_begin[j]);
      const size_t width = static_cast<size_t>(p.width[j]);
      const bool vec = (p.out_vec >> j) & 1u;
      const int rows = min(r1, p.M - t.m0), warps = static_cast<int>(blockDim.x) / 32;
      // ROWS rows a warp at a time, so that the loads of all of them and of all ranks are on their way together
      auto add_up = [&](auto rows_tag, auto ranks_tag) {
        constexpr int ROWS = decltype(rows_tag)::value, RANKS = decltype(ranks_tag)::value;
        for (int m0 = r0 + warp; m0 < rows; m0 += warps * ROWS) {
          float4 v[ROWS][RANKS];
#pragma unroll
          for (int i = 0; i < ROWS; ++i) {
#pragma unroll
            for (int r = 0; r < RANKS; ++r) {
              if (r < csize && m0 + i * warps < rows)
                v[i][r] = *reinterpret_cast<const float4*>(cluster.map_shared_rank(part, r) + (m0 + i * warps) * kBn + c);
            }
          }
#pragma unroll
          for (int i = 0; i < ROWS; ++i) {
            float4 s = v[i][0];
#pragma unroll
            for (int r = 1; r < RANKS; ++r) {
              if (r < csize) {
                s.x += v[i][r].x;
                s.y += v[i][r].y;
                s.z += v[i][r].z;
                s.w += v[i][r].w;
              }
            }
            if (m0 + i * warps < rows) {
              uint16_t* const dst = out + static_cast<size_t>(t.m0 + m0 + i * warps) * width;
              const __nv_bfloat162 lo = __floats2bfloat162_rn(s.x, s.y), hi = __floats2bfloat162_rn(s.z, s.w);
              const uint2 o = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
              if (vec) {
                *reinterpret_cast<uint2*>(dst) = o;
              } else {
                dst[0] = static_cast<uint16_t>(o.x);
                dst[1] = static_cast<uint16_t>(o.x >> 16);
                dst[2] = static_cast<uint16_t>(o.y);
                dst[3] = static_cast<uint16_t>(o.y >> 16);
              }
            }
          }
        }
      };
      if (csize <= 2) {
        add_up(std::integral_constant<int, 4>(), std::integral_constant<int, 2>());
      } else if (csize <= 4) {
        add_up(std::integral_constant<int, 3>(), std::integral_constant<int, 4>());
      } else {
        add_up(std::integral_constant<int, 1>(), std::integral_constant<int, 8>());
      }
    }
  }
  if (ctl.fault) __nanosleep(100000);  // copies of a CTA that gave up may still be landing
  FenceBefore();
  __syncthreads();
  if constexpr (PAIR || SPLIT) cg::this_cluster().sync();  // no CTA leaves while a peer still reads its shared memory
  if (warp == 5) {
    if constexpr (PAIR) {
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(acc_cols) : "memory");
    } else {
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(acc_cols) : "memory");
    }
  }
}

// ------------------------------------------------------------------------------ SharedExpertDown over many rows
// out = routed + bf16(bf16(swish_mul(g, u) @ W) * gate), gate = bf16(sigmoid(bf16(gx . gw))), in the same tiles and
// roles.  A tile of 128 columns is one of N / 128 that need the same rows of swish_mul, so the C CTAs of a cluster
// (neighbouring column tiles, the same rows) each evaluate a share of them: a warp or two per block of 64 k compute their
// CTA's rows, store them into this CTA's stage and send them to the others' with bulk copies between shared memories,
// which count themselves in on the receivers' barriers.  A stage is free when the MMAs of all C CTAs have read it
// (multicast commits).  The gates are shared the same way, by the warps that have nothing to do until the sums are complete,
// which all warps finish.
//
// The streaming kernels that served these calls eight rows at a time took 1403 us for 777 rows of FP8 640 x 2560; this
// one 16.8 in clusters of seven (25.5 with the dot products of the gates multiplied out ahead of the dequantisation and the outputs
// written a column per lane, 23.4 of them on the device).  What bounds it there is the exchange: 67 KB leave and reach an SM in
// 4500 cycles, 15 bytes a cycle, and a CTA needs 175 KB; `clock64` stamps, cycles: blocks evaluated 3500 to 7500 for the first,
// first MMA 12 000, last 24 000, written 28 000.  With few rows it is set-up (3500 cycles until the CTAs have met), the gates'
// trips to memory and 500 cycles a block of dequantisation (60 rows 9.8 us).
// Joining the gates' warps as theirs ends, items taken in turn: no faster at 777 rows, 4 % slower at 60.
struct DenseShared {
  DenseParams d;
  const uint16_t *g, *u, *gx, *gw, *routed;
  int gk, cluster;
  int trigger, pdl_wait;  // as in GemmParams
};

constexpr int kSwishWarps = 8;  // sixteen, at 64 registers a thread, measured no faster (27.0 us, and 5-10 % slower on small calls)
constexpr int kGateWarps = 4;   // the first four, which have nothing else to do until the sums are complete
template <int MODE>
constexpr int SharedThreads() {
  return 32 * (kFirstDqWarp + (MODE == kBf16 ? 0 : kDqWarps) + kSwishWarps);
}

__device__ __forceinline__ float RoundBf16(float v) { return __bfloat162float(__float2bfloat16(v)); }
__device__ __forceinline__ float SigmoidBf16(float a) {
  const float e = expf(-fabsf(a));
  return RoundBf16(a > 0.0f ? 1.0f / (1.0f + e) : e / (1.0f + e));
}
// Warps that share a block.  A barrier's parity tells a phase from the next only, so a warp must have seen a stage's
// previous block consumed (or a later one) before it waits for the stage again: no more blocks in hand than stages.
__device__ __forceinline__ int SwishWarpsPerBlock(int stages) { return kSwishWarps / (stages >= 8 ? 8 : stages >= 4 ? 4 : stages >= 2 ? 2 : 1); }
// The rows of a tile that a rank evaluates: its share of the groups of eight.
__device__ __forceinline__ int FirstRow(const DenseShared& q, int rank) { return rank * (q.d.bm >> 3) / q.cluster * 8; }

// swish_mul by one warp: eight rows by 64 k at a time, the next eight asked for before these are computed.
struct SwishRole {
  const DenseShared& q;
  const uint16_t *g, *u;
  int lane, rank, m0, blocks, sub, first, last, k, r0;
  uint4 gv[2], uv[2];

  __device__ __forceinline__ SwishRole(const DenseShared& call, int warp, int lane_, int rank_, int m0_) : q(call), lane(lane_), rank(rank_), m0(m0_) {
    if (warp < 0) return;  // another role's
    const int per_block = SwishWarpsPerBlock(q.d.stages), begin = FirstRow(q, rank), groups = (FirstRow(q, rank + 1) - begin) >> 3;
    blocks = kSwishWarps / per_block;
    sub = warp / blocks;
    first = begin + sub * groups / per_block * 8;
    last = begin + (sub + 1) * groups / per_block * 8;
    k = warp % blocks;
    r0 = first;
    g = BehindWait(q.g);
    u = BehindWait(q.u);
    Load(k, r0, gv, uv);
  }
  __device__ __forceinline__ void Load(int kk, int rr, uint4 (&a)[2], uint4 (&b)[2]) const {
    const int col = kk * kBk + (lane & 7) * 8;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int r = rr + 4 * j + (lane >> 3), m = m0 + r;
      a[j] = b[j] = make_uint4(0, 0, 0, 0);
      if (r < last && m < q.d.M && col < q.d.K) {  // K is a multiple of eight
        a[j] = __ldg(reinterpret_cast<const uint4*>(g + static_cast<size_t>(m) * q.d.K + col));
        b[j] = __ldg(reinterpret_cast<const uint4*>(u + static_cast<size_t>(m) * q.d.K + col));
      }
    }
  }
  __device__ __forceinline__ void Run(Ctl& ctl, uint32_t smem, uint32_t block_bytes) {
    const DenseParams& p = q.d;
    const uint32_t full0 = Smem(&ctl.full[0]), empty0 = Smem(&ctl.empty[0]);
    const int chunk = lane & 7;
    if (p.give_up) return;
    while (k < p.ksteps) {
      const int stage = k % p.stages, round = k / p.stages;
      const uint32_t dst = smem + static_cast<uint32_t>(stage) * block_bytes + kABytes;
      int kn = k, rn = r0 + 8;
      if (rn >= last) {
        rn = first;
        kn += blocks;
      }
      uint4 gn[2], un[2];
      if (kn < p.ksteps) Load(kn, rn, gn, un);
      // a warp without rows of its own still may not count itself in on a stage that is in use
      if (r0 == first && round > 0 && !BarWait(empty0 + stage * 8, static_cast<uint32_t>((round - 1) & 1), ctl)) return;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int r = r0 + 4 * j + (lane >> 3);
        if (r < last) {
          const uint32_t v[4] = {SwishMul2(gv[j].x, uv[j].x), SwishMul2(gv[j].y, uv[j].y), SwishMul2(gv[j].z, uv[j].z), SwishMul2(gv[j].w, uv[j].w)};
          Sts128(dst + static_cast<uint32_t>(r * 128 + ((chunk ^ (r & 7)) * 16)), v);
        }
      }
      if (kn != k) {  // the warp's rows of this block are complete
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (ElectOne()) {
          const uint32_t bytes = static_cast<uint32_t>((last - first) * 128), bar = full0 + stage * 8, src = dst + static_cast<uint32_t>(first * 128);
          // one warp of the block counts in what the other CTAs send
          const int mine = FirstRow(q, rank + 1) - FirstRow(q, rank);
          if (sub == 0) {
            BarExpect(bar, static_cast<uint32_t>((p.bm - mine) * 128));
          } else {
            BarArrive(bar);
          }
          int peer = rank;
          for (int i = 1; i < q.cluster && bytes > 0; ++i) {
            if (++peer == q.cluster) peer = 0;
            asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                             MapRank(src, static_cast<uint32_t>(peer))),
                         "r"(src), "r"(bytes), "r"(MapRank(bar, static_cast<uint32_t>(peer)))
                         : "memory");
          }
        }
        __syncwarp();
      }
      k = kn;
      r0 = rn;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        gv[j] = gn[j];
        uv[j] = un[j];
      }
    }
  }
};

// 32 products of a row of gx each for rows (g, g + 8) of a lane, added to nothing.
__device__ __forceinline__ float2 Dot32(const uint4& lo, const uint4& hi, const uint4& w) {
  float d[4];
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(lo.x), "r"(hi.x), "r"(lo.y), "r"(hi.y), "r"(w.x), "r"(w.y), "f"(0.f));
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(lo.z), "r"(hi.z), "r"(lo.w), "r"(hi.w), "r"(w.z), "r"(w.w));
  return make_float2(d[0], d[2]);
}

// This CTA's share of the gates, to every CTA of the cluster: asynchronous stores that count their bytes in on the
// receiver's barrier.  The dot products are MMAs of sixteen rows of gx with gw in every column: a lane reads 16 bytes of two
// rows, eight k of its own, and the same eight of gw, so that the order of k within an MMA is free (multiplied out they were
// 24 instructions per 16 bytes, a third of the call).  A warp takes a quarter of k; the quarters are added in order.
// An accumulator that runs through many MMAs is cut off at every one, not rounded: two add 32 products, and their sums go to FP32 sums by
// ordinary additions, eight of 2560 elements to each.  Gates that are not the 64-bit gate's BF16 number, of 2.5 million of twelve
// kinds (250 to 4096 elements, of both signs, of one, cancelling): 249 with running accumulators, 79 with FP32 multiply-adds, 54 so.
// The additions cost a call 0.03 to 0.25 us (BF16 1912 rows 608 x 1344 18.0 -> 18.3).
__device__ __forceinline__ void GateRole(const DenseShared& q, float* gate, float (*quarter)[256], uint32_t bar, int warp, int lane, int rank, int m0) {
  const uint16_t *const gx_in = BehindWait(q.gx), *const gw_in = BehindWait(q.gw);
  const int p0 = FirstRow(q, rank), part = FirstRow(q, rank + 1) - p0;
  const bool vec = reinterpret_cast<uintptr_t>(q.gx) % 16 == 0 && reinterpret_cast<uintptr_t>(q.gw) % 16 == 0 && q.gk % 8 == 0;
  if (vec) {
    const int g = lane >> 2, t = lane & 3, chunks = q.gk >> 3, steps = (chunks + 3) >> 2, s1 = (warp + 1) * steps / kGateWarps;
    constexpr int kAhead = 5;
    const uint4 zero = make_uint4(0, 0, 0, 0);
    for (int r0 = 0; r0 < part; r0 += 16) {
      const int m = m0 + p0 + r0 + g;
      const bool lo_in = m < q.d.M, hi_in = m + 8 < q.d.M && r0 + 8 < part;
      const uint4* lo_row = reinterpret_cast<const uint4*>(gx_in + static_cast<size_t>(m) * q.gk);
      const uint4* hi_row = reinterpret_cast<const uint4*>(gx_in + static_cast<size_t>(m + 8) * q.gk);
      const uint4* gw = reinterpret_cast<const uint4*>(gw_in);
      float2 c[3] = {};
#pragma unroll 1
      for (int s = warp * steps / kGateWarps; s < s1; s += kAhead) {
        uint4 lo[kAhead], hi[kAhead], w[kAhead];
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
          const int at = (s + i) * 4 + t;
          const bool in = s + i < s1 && at < chunks;  // nothing past the end is added, not even to an infinity
          lo[i] = in && lo_in ? __ldg(lo_row + at) : zero;
          hi[i] = in && hi_in ? __ldg(hi_row + at) : zero;
          w[i] = in ? __ldg(gw + at) : zero;
        }
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
          const float2 d = Dot32(lo[i], hi[i], w[i]);
          c[i % 3].x += d.x;
          c[i % 3].y += d.y;
        }
      }
      if (t == 0) {
        quarter[warp][r0 + g] = (c[0].x + c[1].x) + c[2].x;
        if (r0 + 8 < part) quarter[warp][r0 + 8 + g] = (c[0].y + c[1].y) + c[2].y;
      }
    }
  } else {
    // element by element, four rows at a time
    for (int r0 = warp * 4; r0 < part; r0 += kGateWarps * 4) {
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
      const int m = m0 + p0 + r0;
#pragma unroll 2
      for (int c = lane; c < q.gk; c += 32) {
        const float w = __uint_as_float(static_cast<uint32_t>(gw_in[c]) << 16);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (m + j < q.d.M) acc[j] += __uint_as_float(static_cast<uint32_t>(gx_in[static_cast<size_t>(m + j) * q.gk + c]) << 16) * w;
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], off);
        if (lane == 0) {
          quarter[0][r0 + j] = acc[j];
          quarter[1][r0 + j] = quarter[2][r0 + j] = quarter[3][r0 + j] = 0.f;
        }
      }
    }
  }
  asm volatile("bar.sync 1, %0;" ::"n"(32 * kGateWarps) : "memory");
  for (int r = warp * 32 + lane; r < part; r += 32 * kGateWarps) {
    const float logit = ((quarter[0][r] + quarter[1][r]) + quarter[2][r]) + quarter[3][r];
    const uint32_t value = __float_as_uint(SigmoidBf16(RoundBf16(logit))), at = Smem(gate + p0 + r);
    for (int peer = 0; peer < q.cluster; ++peer) {
      asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(MapRank(at, static_cast<uint32_t>(peer))), "r"(value),
                   "r"(MapRank(bar, static_cast<uint32_t>(peer)))
                   : "memory");
    }
  }
}

template <int MODE>
__global__ void __launch_bounds__(SharedThreads<MODE>(), 1) DenseSharedKernel(const __grid_constant__ DenseShared q) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ Ctl ctl;
  __shared__ float gate[256], quarter[kGateWarps][256];
  __shared__ unsigned long long gate_full;
  const DenseParams& p = q.d;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const uint32_t smem = (Smem(smem_raw) + 1023u) & ~1023u;
  const int C = q.cluster, rank = C > 1 ? static_cast<int>(cg::this_cluster().block_rank()) : 0, group = static_cast<int>(blockIdx.x) / C;
  const int tile = ((group / p.m_tiles) * C + rank) * p.m_tiles + group % p.m_tiles;  // the columns are padded to whole clusters
  const TileAt t = LocateDense<false>(p, tile, 0);
  const uint32_t block_bytes = static_cast<uint32_t>(kABytes + p.bm * kBk * 2);
  const uint32_t full0 = Smem(&ctl.full[0]), empty0 = Smem(&ctl.empty[0]), accf0 = Smem(&ctl.acc_full[0]);
  int acc_cols = 32;
  while (acc_cols < p.bm) acc_cols *= 2;

  if (tid == 0) {
    for (int i = 0; i < p.stages; ++i) {
      BarInit(full0 + i * 8, SwishWarpsPerBlock(p.stages) + (MODE == kBf16 ? 1 : kDqWarps));
      BarInit(empty0 + i * 8, C);
    }
    BarInit(accf0, 1);
    BarInit(Smem(&gate_full), 1);
    BarExpect(Smem(&gate_full), static_cast<uint32_t>(p.bm) * 4);
    for (int i = 0; MODE != kBf16 && i < RawRing<MODE, 1>::kDepth; ++i) {
      BarInit(Smem(&ctl.raw_full[i]), 1);
      BarInit(Smem(&ctl.raw_empty[i]), kDqWarps);
    }
    ctl.fault = static_cast<uint32_t>(p.give_up);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(Smem(&ctl.tmem)), "r"(acc_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // nothing of the call is read or written before this line: a predecessor may be writing any of it
  GridDependencyWait();
  if (q.trigger == 1) GridLaunchDependents();
  constexpr int kFirstSwish = kFirstDqWarp + (MODE == kBf16 ? 0 : kDqWarps), kSumGroups = (kFirstSwish + kSwishWarps) / 4;
  SwishRole swish(q, warp - kFirstSwish, lane, rank, t.m0);  // its first rows are on their way while the CTAs meet
  FenceBefore();
  __syncthreads();
  if (C > 1) cg::this_cluster().sync();  // every CTA's barriers exist
  FenceAfter();
  const uint32_t tmem = ctl.tmem;

  if (warp < kGateWarps) {
    GateRole(q, gate, quarter, Smem(&gate_full), warp, lane, rank, t.m0);
  } else if (warp == 4) {
    if constexpr (MODE == kBf16) {
      for (int k = 0; k < p.ksteps; ++k) {
        const int stage = k % p.stages, round = k / p.stages;
        if (round > 0 && !BarWait(empty0 + stage * 8, static_cast<uint32_t>((round - 1) & 1), ctl)) break;
        const uint32_t dst = smem + static_cast<uint32_t>(stage) * block_bytes;
        if (ElectOne()) {
          BarExpect(full0 + stage * 8, kABytes);
          TmaLoad<false>(dst, &p.wmap[0], t.n0, k * kBk, full0 + stage * 8);
          TmaLoad<false>(dst + kABytes / 2, &p.wmap[0], t.n0 + 64, k * kBk, full0 + stage * 8);
        }
        __syncwarp();
      }
    }
  } else if (warp == 5) {
    const uint32_t idesc = 0x10u | (1u << 7) | (1u << 10) | (1u << 15) | (static_cast<uint32_t>(p.bm >> 3) << 17) | (8u << 24);
    const unsigned long long a0 = SmemDesc(smem, kABytes / 2, 1024), b0 = SmemDesc(smem + kABytes, 16, 1024);
    for (int k = 0; k < p.ksteps; ++k) {
      const int stage = k % p.stages, round = k / p.stages;
      if (!BarWait(full0 + stage * 8, static_cast<uint32_t>(round & 1), ctl)) break;
      FenceAfter();
      const uint32_t off = static_cast<uint32_t>(stage) * block_bytes >> 4;
      if (ElectOne()) {
#pragma unroll
        for (int i = 0; i < kBk / 16; ++i) MmaSs<false>(tmem, a0 + off + i * (2048 >> 4), b0 + off + i * (32 >> 4), idesc, k > 0 || i > 0);
        if (C > 1) {
          asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(empty0 + stage * 8),
                       "h"(static_cast<uint16_t>((1 << C) - 1))
                       : "memory");
        } else {
          MmaCommit<false>(empty0 + stage * 8);
        }
        if (k == p.ksteps - 1) MmaCommit<false>(accf0);
      }
      __syncwarp();
    }
    if (q.trigger == 2) GridLaunchDependents();
  } else if (warp >= kFirstSwish) {
    swish.Run(ctl, smem, block_bytes);
  } else if (MODE != kBf16 && warp >= 6) {
    const uint32_t ring = smem + static_cast<uint32_t>(p.stages) * block_bytes;
    if constexpr (MODE != kBf16) {
      if (warp >= kFirstDqWarp) {
        // the products are exact in BF16 without w_scale, which the epilogue applies to the sums as the streaming kernels do
        DequantRole<MODE, false, false, 1, 1>(p, ctl, warp - kFirstDqWarp, 0, lane, 0, p.ksteps, tile, p.tiles, ring, smem, block_bytes);
      } else if (warp == 6) {
        LoadTensor<MODE, false, 1>(p, ctl, 0, 0, p.ksteps, tile, p.tiles, ring);
      }
    }
  }

  // The sums, by every warp: columns 32 (warp % 4) ... of the tile, sixteen rows at a time.  They come as fragments, columns
  // of W down and rows of x across, are scaled and rounded as such, and go through shared memory (where the stored
  // weights were, which nobody else writes or reads) transposed, so that routed is read and the output written
  // 16 bytes at a time.  A column per lane, two bytes an access, took a fifth of the call: 9500 of 42 100 cycles for 160 rows.
  __syncwarp();
  {
    const DenseSeg& sg = p.seg[0];
    const int quad = warp & 3, n0 = t.n0 + 32 * quad, chunk = lane & 3, row = lane >> 2, n = n0 + 8 * chunk;  // widths are multiples of eight
    float scale[2][2];
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const int at = n0 + 8 * h + row;
      scale[h >> 1][h & 1] = at < sg.n && sg.w_scale != nullptr ? __ldg(sg.w_scale + at) : 1.f;
    }
    const uint32_t src = tmem + (static_cast<uint32_t>(32 * quad) << 16), buf = smem + static_cast<uint32_t>(p.stages) * block_bytes + static_cast<uint32_t>(warp * 16 * kOutPitch);
    const uint32_t st = buf + static_cast<uint32_t>((((lane >> 4) & 1) * 8 + (lane & 7)) * kOutPitch + ((lane >> 3) & 1) * 16);
    const uint32_t ld = buf + static_cast<uint32_t>(row * kOutPitch + chunk * 16);
    const size_t at0 = static_cast<size_t>(t.m0) * sg.n + n;
    uint16_t* const out = p.out[0] + at0;
    const uint16_t* const routed = q.routed != nullptr ? q.routed + at0 : nullptr;
    const bool vec_out = reinterpret_cast<uintptr_t>(p.out[0]) % 16 == 0, vec_in = reinterpret_cast<uintptr_t>(q.routed) % 16 == 0;
    bool good = true, waited = false;
    for (int c = 16 * (warp >> 2); c < p.bm && t.m0 + c < p.M; c += 16 * kSumGroups) {
      uint32_t rt[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = c + 8 * i + row;
        rt[i][0] = rt[i][1] = rt[i][2] = rt[i][3] = 0;
        if (n < sg.n && routed != nullptr && t.m0 + r < p.M) {
          const uint16_t* const from = routed + static_cast<size_t>(r) * sg.n;
          if (vec_in) {
            const uint4 v = *reinterpret_cast<const uint4*>(from);
            rt[i][0] = v.x, rt[i][1] = v.y, rt[i][2] = v.z, rt[i][3] = v.w;
          } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) rt[i][e >> 1] |= static_cast<uint32_t>(from[e]) << (16 * (e & 1));
          }
        }
      }
      if (!waited) {
        good = BarWaitCluster(Smem(&gate_full), 0, ctl) && BarWait(accf0, 0, ctl);
        waited = true;
        __syncwarp();
        FenceAfter();
      }
      uint32_t v[2][8];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t(&f)[8] = v[h];
        asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(f[0]), "=r"(f[1]), "=r"(f[2]), "=r"(f[3]), "=r"(f[4]), "=r"(f[5]), "=r"(f[6]), "=r"(f[7])
                     : "r"(src + (static_cast<uint32_t>(16 * h) << 16) + static_cast<uint32_t>(c)));
      }
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      __syncwarp();  // the rows before have been read
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = PackBf16(__uint_as_float(v[h][2 * i]) * scale[h][i & 1], __uint_as_float(v[h][2 * i + 1]) * scale[h][i & 1]);
        asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(st + h * 32), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3])
                     : "memory");
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = c + 8 * i + row;
        if (n < sg.n && t.m0 + r < p.M) {
          const float gt = gate[r];
          uint32_t o[4];
          Lds128(ld + i * (8 * kOutPitch), o);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            // every step rounded to BF16 (the reference's skinny_gemm.cuh:226-240)
            float lo = RoundBf16(Lo(o[e]) * gt), hi = RoundBf16(Hi(o[e]) * gt);
            if (routed != nullptr) lo += Lo(rt[i][e]), hi += Hi(rt[i][e]);
            o[e] = good ? PackBf16(lo, hi) : 0x7FFF7FFFu;
          }
          uint16_t* const dst = out + static_cast<size_t>(r) * sg.n;
          if (vec_out) {
            *reinterpret_cast<uint4*>(dst) = make_uint4(o[0], o[1], o[2], o[3]);
          } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) dst[e] = static_cast<uint16_t>(o[e >> 1] >> (16 * (e & 1)));
          }
        }
      }
    }
    // a CTA leaves when its own sums are complete, and with them every copy into it: warps without rows wait too
    if (!waited) {
      BarWaitCluster(Smem(&gate_full), 0, ctl);
      BarWait(accf0, 0, ctl);
      __syncwarp();
    }
  }
  if (ctl.fault) __nanosleep(100000);
  FenceBefore();
  __syncthreads();
  if (C > 1) cg::this_cluster().sync();  // no CTA leaves while a peer may still write to it
  if (warp == 5) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(acc_cols) : "memory");
}

// ------------------------------------------------------------------------------ host
// rows x cols elements of `elem` bytes (2: BF16, boxes swizzled in 128 bytes; 1: bytes, plain or swizzled as given), row-major
bool Encode(CUtensorMap* map, const void* base, int elem, uint64_t rows, uint64_t cols, uint64_t pitch_bytes, uint32_t box_rows, uint32_t box_cols,
            int swizzle = 0) {
  const cuuint64_t dims[2] = {cols, rows}, strides[1] = {pitch_bytes};
  const cuuint32_t box[2] = {box_cols, box_rows}, step[2] = {1, 1};
  const TensorMapEncodeFn fn = TensorMapEncoder();
  return fn != nullptr &&
         fn(map, elem == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, step,
            CU_TENSOR_MAP_INTERLEAVE_NONE, elem == 2 || swizzle == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : swizzle == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_NONE,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

constexpr int kSmemLimit = 232448 - 1024 - static_cast<int>(sizeof(Ctl)) - 64;

// DenseSharedKernel has the gates and their quarters besides
constexpr int kSharedSmemLimit = kSmemLimit - 1024 * (1 + kGateWarps) - 64;

int RawBytes(int mode, int ks) {
  if (mode == kFp8) return ks == 2 ? RawRing<kFp8, 2>::kBytes : RawRing<kFp8, 1>::kBytes;
  if (mode == kNvfp4) return ks == 2 ? RawRing<kNvfp4, 2>::kBytes : RawRing<kNvfp4, 1>::kBytes;
  if (mode == kNvfp4Odd) return ks == 2 ? RawRing<kNvfp4Odd, 2>::kBytes : RawRing<kNvfp4Odd, 1>::kBytes;
  return 0;
}
int BlocksFor(int mode, int xrows, int ks) { return (kSmemLimit - kOutBytes - RawBytes(mode, ks)) / (kABytes + xrows * kBk * 2); }

template <int MODE, bool SCALED, bool PAIR, bool SPLIT, int KS, bool TM = false>
cudaError_t LaunchOne(const DenseParams& p, int ctas, int cluster, size_t smem, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(ctas));
  cfg.blockDim = dim3(static_cast<unsigned>(DenseThreads<MODE>()));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  if (cluster > 1) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(cluster);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.numAttrs = 1;
  }
  if (MayOverlapPredecessor(stream)) attr[cfg.numAttrs++] = OverlapAttribute();
  return cudaLaunchKernelEx(&cfg, DenseTcKernel<MODE, SCALED, PAIR, SPLIT, KS, TM>, p);
}

// Whether there are kernels of two blocks a stage.  The unpaired tiles of FP8 and NVFP4 that do not take tensor memory are too large for
// enough of those.
template <int MODE, bool PAIR>
constexpr bool kTwoBlocks = PAIR || MODE == kBf16 || MODE == kNvfp4Odd;

template <int MODE, bool SCALED>
cudaError_t LaunchMode(const DenseParams& p, bool pair, int ks, bool tm, int ctas, int cluster, size_t smem, cudaStream_t stream) {
  if constexpr (MODE == kFp8 || MODE == kNvfp4) {
    if (tm && pair) return LaunchOne<MODE, SCALED, true, false, kTmKs, true>(p, ctas, 2, smem, stream);
    if (tm && cluster > 1) return LaunchOne<MODE, SCALED, false, true, kTmKs, true>(p, ctas, cluster, smem, stream);
    if (tm) return LaunchOne<MODE, SCALED, false, false, kTmKs, true>(p, ctas, 1, smem, stream);
  }
  if (pair) return ks == 2 ? LaunchOne<MODE, SCALED, true, false, 2>(p, ctas, 2, smem, stream) : LaunchOne<MODE, SCALED, true, false, 1>(p, ctas, 2, smem, stream);
  if constexpr (kTwoBlocks<MODE, false>) {
    if (ks == 2) return cluster > 1 ? LaunchOne<MODE, SCALED, false, true, 2>(p, ctas, cluster, smem, stream) : LaunchOne<MODE, SCALED, false, false, 2>(p, ctas, 1, smem, stream);
  }
  return cluster > 1 ? LaunchOne<MODE, SCALED, false, true, 1>(p, ctas, cluster, smem, stream) : LaunchOne<MODE, SCALED, false, false, 1>(p, ctas, 1, smem, stream);
}

template <int MODE>
cudaError_t LaunchShared(const DenseShared& q, int ctas, size_t smem, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(ctas));
  cfg.blockDim = dim3(static_cast<unsigned>(SharedThreads<MODE>()));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(q.cluster);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1] = OverlapAttribute();
  cfg.attrs = attr;
  cfg.numAttrs = q.pdl_wait || MayOverlapPredecessor(stream) ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, DenseSharedKernel<MODE>, q);
}

// ------------------------------------------------------------------------------ set-up, once per device
// The shared-memory limit of a kernel belongs to a device, and so do the clusters it holds at once.
constexpr int kMaxCluster = 8;
struct DeviceSetup {
  int device;
  int slots[kMaxCluster + 1];  // clusters of so many CTAs, one per SM, that are resident at once
};
std::mutex g_setup_mu;
std::map<int, DeviceSetup> g_setup;  // devices that are done; an entry stays as it is
std::atomic<const DeviceSetup*> g_setup_last{nullptr};  // the last one asked for: a process mostly drives one

template <int MODE, bool SCALED, int KS>
cudaError_t SetUpShape() {
  cudaError_t err = cudaFuncSetAttribute(DenseTcKernel<MODE, SCALED, true, false, KS, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit + 1024);
  if constexpr (KS == 1 || kTwoBlocks<MODE, false>) {
    if (err == cudaSuccess)
      err = cudaFuncSetAttribute(DenseTcKernel<MODE, SCALED, false, false, KS, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit + 1024);
    if (err == cudaSuccess)
      err = cudaFuncSetAttribute(DenseTcKernel<MODE, SCALED, false, true, KS, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit + 1024);
  }
  if constexpr (KS == kTmKs && (MODE == kFp8 || MODE == kNvfp4)) {
    if (err == cudaSuccess)
      err = cudaFuncSetAttribute(DenseTcKernel<MODE, SCALED, true, false, KS, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit + 1024);
    if (err == cudaSuccess)
      err = cudaFuncSetAttribute(DenseTcKernel<MODE, SCALED, false, false, KS, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit + 1024);
    if (err == cudaSuccess)
      err = cudaFuncSetAttribute(DenseTcKernel<MODE, SCALED, false, true, KS, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit + 1024);
  }
  return err;
}
template <int MODE, bool SCALED>
cudaError_t SetUpMode() {
  const cudaError_t err = SetUpShape<MODE, SCALED, 1>();
  return err == cudaSuccess ? SetUpShape<MODE, SCALED, 2>() : err;
}
template <int MODE>
cudaError_t SetUpShared() {
  return cudaFuncSetAttribute(DenseSharedKernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSharedSmemLimit);
}

// A GPC's SMs rarely divide by the size (33 clusters of four, fewer than 16 of eight), and a cluster too many costs a
// second wave.
int QuerySlots(int cluster) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(cluster));
  cfg.blockDim = dim3(static_cast<unsigned>(DenseThreads<kBf16>()));
  cfg.dynamicSmemBytes = kSmemLimit;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(cluster);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, DenseTcKernel<kBf16, false, false, true, 1, false>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    n = std::max(1, DeviceSmCount() * 8 / (10 * cluster));
  }
  return n;
}

// The set-up of the current device, made on the first request.  Only a success is kept.
cudaError_t SetUpDevice(const DeviceSetup** out) {
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  *out = g_setup_last.load(std::memory_order_acquire);
  if (*out != nullptr && (*out)->device == dev) return cudaSuccess;
  std::lock_guard<std::mutex> lock(g_setup_mu);
  auto it = g_setup.find(dev);
  if (it == g_setup.end()) {
    err = SetUpMode<kBf16, false>();
    if (err == cudaSuccess) err = SetUpMode<kFp8, false>();
    if (err == cudaSuccess) err = SetUpMode<kFp8, true>();
    if (err == cudaSuccess) err = SetUpMode<kNvfp4, false>();
    if (err == cudaSuccess) err = SetUpMode<kNvfp4, true>();
    if (err == cudaSuccess) err = SetUpMode<kNvfp4Odd, false>();
    if (err == cudaSuccess) err = SetUpMode<kNvfp4Odd, true>();
    if (err == cudaSuccess) err = SetUpShared<kBf16>();
    if (err == cudaSuccess) err = SetUpShared<kFp8>();
    if (err == cudaSuccess) err = SetUpShared<kNvfp4>();
    if (err == cudaSuccess) err = SetUpShared<kNvfp4Odd>();
    if (err != cudaSuccess) return err;
    DeviceSetup d = {dev, {}};
    for (int c = 1; c <= kMaxCluster; ++c) d.slots[c] = QuerySlots(c);
    it = g_setup.emplace(dev, d).first;
  }
  *out = &it->second;
  g_setup_last.store(*out, std::memory_order_release);
  return cudaSuccess;
}

// describes a stored weight to the copy engine
bool EncodeWeight(DenseParams& p, int mode, int s, const Segment& sg, int K, int ks, bool tm = false) {
  const uint64_t rows = static_cast<uint64_t>(K), pitch = static_cast<uint64_t>(sg.pitch), n = static_cast<uint64_t>(sg.n);
  if (mode == kBf16) return Encode(&p.wmap[s], sg.w, 2, rows, n, pitch, kBk, 64);
  if (mode == kFp8) return Encode(&p.wmap[s], sg.w, 1, rows, n, pitch, kBk * ks, kBn, tm ? 128 : 0);
  const uint64_t rows_in_one = mode == kNvfp4Odd ? 2 : 1;  // K is a multiple of eight
  const uint32_t box = static_cast<uint32_t>(kBk * ks / rows_in_one);
  return Encode(&p.wmap[s], sg.w, 1, rows / rows_in_one, pitch * rows_in_one, pitch * rows_in_one, box, mode == kNvfp4Odd ? kOddPitch : kBn / 2, tm ? 64 : 0) &&
         Encode(&p.smap[s], sg.w, 1, rows / rows_in_one, pitch * rows_in_one, pitch * rows_in_one, box, 16);
}

// which of the file's modes a call is: one weight of odd rows makes all of them be read that way
int KernelMode(int mode, const GemmParams& p) {
  for (int s = 0; s < p.nseg && mode == kNvfp4; ++s) {
    if (p.seg[s].pitch % 16 != 0) return kNvfp4Odd;
  }
  return mode;
}

}  // namespace

// Called when a node is created, so that the first call finds nothing left to do and may be captured, and again by each
// call, which may have another device current.
cudaError_t ConfigureDenseKernels() {
  const DeviceSetup* setup = nullptr;
  return SetUpDevice(&setup);
}

// Launch shape: rows per tile, CTAs that split K, pairs.  The cheapest by a model fitted to measured launches (one B200; us).
// A block of 64 k costs a single CTA 0.17 + 0.0011 bm (bm = 48: 0.22, 128: 0.31, 256: 0.45), a pair 0.13 + 0.00098 bm
// (128: 0.25, 192: 0.32, 256: 0.38) and no less than its dequantisation (0.24); around the blocks 4 + 0.008 bm, 0.9 more for a pair, and 1.8 + 0.01 bm more where ranks add up: with
// less for those two, as K = 5120 alone had suggested, short K was split and paired where that loses (BF16 146 x 400 x
// 3728 6.3 us in pairs of 64, 5.5 in single tiles of 48; over 150 random calls the shape chosen took 3.7 % longer than the
// best one, and takes 1.8).  More row tiles than needed are tried because they can fill the last wave better (509 rows,
// N = 10240: 3 x 192 56 us, 2 x 256 61 us).
// Through tensor memory (up to 128 rows of FP8 or NVFP4) a block costs 0.167 + 0.00041 bm, a pair or a small tile 0.175 (scaled 0.2);
// a seventh more past 40 us, and 0.7 a wave.  Several row tiles of longer calls stay with larger tiles: those of 128
// rows dequantise the weights more often and run against the power cap (NVFP4 509 rows 5120 x 17408 74.4 us in pairs of 256 rows, 80.4 in
// tiles of 128).  On 57 calls (rows 9 to 2048, K 320 to 17408, N 512 to 17408) the shape chosen takes 0.1 % longer than the best one tried, 1.8 % at
// worst.  Tensor memory was tried up to 192 rows, a block a stage: 0.36 a block in pairs, whatever their rows (FP8 400 rows 5120 x
// 10240 52.8 -> 63.1 us).
DenseTcPlan ChooseDenseTcPlan(int mode, const GemmParams& p, int64_t m, int sm_count) {
  const DeviceSetup* setup = nullptr;
  if (SetUpDevice(&setup) != cudaSuccess) throw std::runtime_error("SkinnyGemm(dense): the kernels could not be set up on this device");
  DenseTcPlan best;
  double best_cost = 1e30, bytes = 0;
  for (int s = 0; s < p.nseg; ++s) {
    bytes += static_cast<double>(p.seg[s].total_bytes);
  }
  const int64_t blocks = (p.K + kBk - 1) / kBk, least = (m + 255) / 256;
  const int kernel_mode = KernelMode(mode, p);
  const bool tm_weights = kernel_mode == kFp8 || kernel_mode == kNvfp4;
  bool scaled = false;
  for (int s = 0; s < p.nseg; ++s) scaled = scaled || p.seg[s].w_scale != nullptr;
  for (int pair = 0; pair <= 1; ++pair) {
    int64_t n_tiles = 0;
    for (int s = 0; s < p.nseg; ++s) n_tiles += (p.seg[s].n + (pair ? 255 : 127)) / (pair ? 256 : 128);
    for (int64_t mt = least; mt <= 2 * least + 2 && mt <= m; ++mt) {
      const int bm = static_cast<int>(((m + mt - 1) / mt + 15) / 16 * 16);
      if (bm > 256 || (pair && bm < 64)) continue;
      const int64_t tiles = n_tiles * ((m + bm - 1) / bm);
      const bool tm = tm_weights && bm <= kTmBm;
      const double step = tm ? std::max(pair ? 0.0 : 0.167 + 0.00041 * bm, scaled ? 0.199 : 0.175)
                             : std::max(pair ? 0.13 + 0.00098 * bm : 0.17 + 0.0011 * bm, mode == kBf16 ? 0.0 : 0.24);
      for (int split = 1; split <= (pair ? 1 : 8) && 4 * split <= std::max<int64_t>(blocks, 4); ++split) {
        const int64_t slots = pair ? sm_count / 2 : split == 1 ? sm_count : setup->slots[split];
        if (slots < 1) break;  // the device holds no such cluster
        const int64_t waves = (tiles + slots - 1) / slots;
        if (split > 1 && waves > 1) break;
        double work = static_cast<double>(waves * ((blocks + split - 1) / split)) * step;
        if (tm && mt > 1 && work > 40.0) continue;
        if (tm) work += 0.146 * std::max(0.0, work - 40.0) + 0.7 * static_cast<double>(waves - 1);
        const double cost = std::max(work, bytes / 6.3e6) + 4 + 0.008 * bm + (split > 1 ? 1.8 + 0.01 * bm : pair ? 0.9 : 0);
        if (cost < best_cost) {
          best_cost = cost;
          best.bm = bm;
          best.split = split;
          best.pair = pair;
        }
      }
    }
  }
  return best;
}

// 16-byte rows of x; weights that a tensor map describes, or NVFP4 ones in whole 128-column groups; every output a
// multiple of eight columns; rows that fit the kernel's 32-bit counts with a tile to spare.
bool DenseTcEligible(int mode, const GemmParams& p, int64_t m) {
  if (m > INT_MAX / 2 || p.K % 8 != 0 || reinterpret_cast<uintptr_t>(p.x) % 16 != 0) return false;
  for (int s = 0; s < p.nseg; ++s) {
    const Segment& sg = p.seg[s];
    if (reinterpret_cast<uintptr_t>(sg.w) % 16 != 0) return false;
    if (sg.n % (mode == kNvfp4 ? 128 : mode == kFp8 ? 16 : 8) != 0) return false;
  }
  const int n_out = p.seg[p.nseg - 1].out_end;
  for (int o = 0; o < n_out; ++o) {
    if (p.out[o] == nullptr || p.width[o] % 8 != 0) return false;
  }
  return TensorMapEncoder() != nullptr;
}

// Whether a launch shape hands the weights over in tensor memory, two blocks a stage; one block goes through shared memory.
bool TakesTm(int mode, const DenseTcPlan& plan) { return (mode == kFp8 || mode == kNvfp4) && plan.bm <= kTmBm && plan.ks != 1; }

bool LaunchDenseTc(int weights, const GemmParams& g, int64_t m, const DenseTcPlan& plan, cudaStream_t stream) {
  const int mode = KernelMode(weights, g);
  if (plan.bm < 16 || plan.bm > 256 || plan.bm % 16 != 0 || plan.split < 1 || plan.split > 8 || (plan.pair && plan.split != 1) || plan.ks < 0 || plan.ks > 2)
    throw std::runtime_error("SkinnyGemm(dense): bad launch shape");
  DenseParams p = {};
  p.nseg = g.nseg;
  p.M = static_cast<int>(m);
  p.K = g.K;
  p.give_up = g.give_up;
  p.bm = plan.bm;
  const int xrows = plan.pair ? p.bm / 2 : p.bm;
  const bool tm = TakesTm(mode, plan);
  int ks = tm ? kTmKs : plan.ks > 0 ? plan.ks : BlocksFor(mode, xrows, 2) >= 6 ? 2 : 1;
  // the dequantising groups take the stages in turn: fewer stages than groups would run off the ring
  if (!tm && BlocksFor(mode, xrows, ks) < kDqGroups * ks) throw std::runtime_error("SkinnyGemm(dense): bad launch shape");
  if (!tm && !plan.pair && (mode == kFp8 || mode == kNvfp4)) ks = 1;  // kTwoBlocks
  const int blocks = BlocksFor(mode, xrows, ks);
  p.ksteps = (g.K + kBk * ks - 1) / (kBk * ks);
  if (!Encode(&p.xmap, g.x, 2, static_cast<uint64_t>(m), static_cast<uint64_t>(g.K), static_cast<uint64_t>(g.K) * 2, static_cast<uint32_t>(xrows), kBk))
    return false;
  bool scaled = false;
  int n_tiles = 0;
  for (int s = 0; s < g.nseg; ++s) {
    const Segment& sg = g.seg[s];
    p.seg[s] = {sg.w, sg.w_scale, sg.pitch, sg.total_bytes, sg.n, n_tiles, sg.out_begin, sg.out_end};
    n_tiles += (sg.n + (plan.pair ? 255 : 127)) / (plan.pair ? 256 : 128);
    scaled = scaled || sg.w_scale != nullptr;
  }
  for (int s = 0; s < g.nseg; ++s) {
    if (!EncodeWeight(p, mode, s, g.seg[s], g.K, ks, tm)) return false;
  }
  const int n_out = g.seg[g.nseg - 1].out_end;
  for (int o = 0; o < n_out; ++o) {
    p.out[o] = g.out[o];
    p.col_begin[o] = g.col_begin[o];
    p.width[o] = g.width[o];
    if (reinterpret_cast<uintptr_t>(g.out[o]) % 16 == 0) p.out_vec |= 1u << o;
  }
  p.m_tiles = static_cast<int>((m + p.bm - 1) / p.bm);
  if (static_cast<int64_t>(p.m_tiles) * n_tiles > INT_MAX / 16) return false;
  p.tiles = p.m_tiles * n_tiles;
  const int cluster = plan.pair ? 2 : std::min(plan.split, p.ksteps);
  p.stages = tm ? kTmStages : std::min(kMaxStages, blocks / ks);
  size_t smem = 1024 + static_cast<size_t>(p.stages) * ks * ((tm ? 0 : kABytes) + xrows * kBk * 2) + kOutBytes;
  if (tm) {
    const int slot = ks * (mode == kFp8 ? RawRing<kFp8, 1>::kSlot : RawRing<kNvfp4, 1>::kSlot);
    p.raw_depth = smem + 2 * kTmGroups * slot <= static_cast<size_t>(kSmemLimit) ? 2 * kTmGroups : kTmGroups;
    smem += static_cast<size_t>(p.raw_depth) * slot;
  } else {
    smem += static_cast<size_t>(RawBytes(mode, ks));
  }
  const int slots = std::max(1, DeviceSmCount() / cluster);
  const int ctas = cluster * (cluster > 1 && !plan.pair ? p.tiles : std::min(p.tiles, slots));
  cudaError_t err = ConfigureDenseKernels();
  if (err != cudaSuccess) throw std::runtime_error(std::string("SkinnyGemm(dense): ") + cudaGetErrorString(err));
  if (mode == kBf16) {
    err = LaunchMode<kBf16, false>(p, plan.pair != 0, ks, tm, ctas, cluster, smem, stream);
  } else if (mode == kFp8) {
    err = scaled ? LaunchMode<kFp8, true>(p, plan.pair != 0, ks, tm, ctas, cluster, smem, stream) : LaunchMode<kFp8, false>(p, plan.pair != 0, ks, tm, ctas, cluster, smem, stream);
  } else if (mode == kNvfp4) {
    err = scaled ? LaunchMode<kNvfp4, true>(p, plan.pair != 0, ks, tm, ctas, cluster, smem, stream)
                 : LaunchMode<kNvfp4, false>(p, plan.pair != 0, ks, tm, ctas, cluster, smem, stream);
  } else {
    err = scaled ? LaunchMode<kNvfp4Odd, true>(p, plan.pair != 0, ks, tm, ctas, cluster, smem, stream)
                 : LaunchMode<kNvfp4Odd, false>(p, plan.pair != 0, ks, tm, ctas, cluster, smem, stream);
  }
  if (err == cudaSuccess) err = cudaGetLastError();
  if (err != cudaSuccess) throw std::runtime_error(std::string("SkinnyGemm(dense): ") + cudaGetErrorString(err));
  return true;
}

// SharedExpertDown: 16-byte rows of g and u as well.
bool DenseSharedEligible(int mode, const GemmParams& p, int64_t m) {
  return p.fuse && p.nseg == 1 && DenseTcEligible(mode, p, m) && reinterpret_cast<uintptr_t>(p.x2) % 16 == 0;
}

// Rows per tile and CTAs per cluster, by a model fitted to measured launches (us).  `own`: the rows that a CTA evaluates.  A
// block of 64 k costs 0.027 for each of them, and no less than 0.4 (dequantisation, MMAs, the waits between the roles); around the
// blocks 1.6 + 0.0064 bm, 0.14 for each gate of 2560 elements, 1.4 + 0.19 c where CTAs share.  On 52 shapes (17 to 2048
// rows, K 256 to 2560, N 1024 to 5120, the three types) the shape chosen takes 0.4 % longer than the best of the 100 tried, 8 %
// at worst (BF16 2048 rows 2560 x 1024 43.5 us, 40.4 in tiles of 128 and clusters of four); the model before this
// one, made for clusters of up to four with even shares, 3 % and 22 % (FP8 621 rows 2256 x 2400 34.4, 28.3).
DenseTcPlan ChooseDenseSharedPlan(const GemmParams& p, int64_t m, int sm_count) {
  const DeviceSetup* setup = nullptr;
  if (SetUpDevice(&setup) != cudaSuccess) throw std::runtime_error("SharedExpertDown: the kernels could not be set up on this device");
  DenseTcPlan best;
  double best_cost = 1e30;
  const int64_t n_tiles = (p.seg[0].n + kBn - 1) / kBn;
  const double blocks = (p.K + kBk - 1) / kBk;
  for (int c = 1; c <= kMaxCluster; ++c) {
    const int64_t slots = c == 1 ? sm_count : setup->slots[c], groups = (n_tiles + c - 1) / c;
    if (slots < 1) break;
    for (int bm = (8 * c + 15) / 16 * 16; bm <= 256; bm += 16) {
      const int64_t waves = (groups * ((m + bm - 1) / bm) + slots - 1) / slots;
      const int own = (bm / 8 + c - 1) / c * 8;
      const double block = std::max(0.004 + 0.027 * own + 0.00024 * (bm - own), 0.40 + 0.00014 * bm);
      const double cost = waves * (blocks * block + 1.6 + 0.0064 * bm + 0.14 / 2560 * own * p.gk + (c > 1 ? 1.4 + 0.19 * c : 0.0));
      if (cost < best_cost) {
        best_cost = cost;
        best.bm = bm;
        best.split = c;
        best.ks = 1;
      }
    }
  }
  return best;
}

bool LaunchDenseShared(int weights, const GemmParams& g, int64_t m, const DenseTcPlan& plan, cudaStream_t stream) {
  const int mode = KernelMode(weights, g);
  const int C = plan.split;
  // Shares are even and clusters of 1, 2 or 4 where a pinned shape does not name the blocks per stage, of which there is one: "48,4" and "64,3"
  // have always been errors, and who pins one of them to be told so still is.
  const bool even = (C == 1 || C == 2 || C == 4) && plan.bm % (8 * C) == 0;
  if (C < 1 || C > kMaxCluster || plan.bm < 16 || plan.bm > 256 || plan.bm % 16 != 0 || plan.bm < 8 * C || (!even && plan.ks != 1))
    throw std::runtime_error("SharedExpertDown: bad launch shape");
  DenseShared q = {};
  DenseParams& p = q.d;
  const Segment& sg = g.seg[0];
  p.nseg = 1;
  p.M = static_cast<int>(m);
  p.K = g.K;
  p.give_up = g.give_up;
  p.bm = plan.bm;
  p.ksteps = (g.K + kBk - 1) / kBk;
  p.seg[0] = {sg.w, sg.w_scale, sg.pitch, sg.total_bytes, sg.n, 0, 0, 1};
  p.out[0] = g.out[0];
  p.width[0] = sg.n;
  if (!EncodeWeight(p, mode, 0, sg, g.K, 1)) return false;
  const int64_t n_tiles = ((sg.n + kBn - 1) / kBn + C - 1) / C * C, m_tiles = (m + p.bm - 1) / p.bm;
  if (n_tiles * m_tiles > INT_MAX / 16) return false;
  p.m_tiles = static_cast<int>(m_tiles);
  p.tiles = static_cast<int>(n_tiles * m_tiles);
  const int block = kABytes + p.bm * kBk * 2;
  // behind the stages the stored weights, and in their place each warp's buffer for the outputs
  const int behind = std::max(RawBytes(mode, 1), (mode == kBf16 ? SharedThreads<kBf16>() : SharedThreads<kFp8>()) / 32 * 16 * kOutPitch);
  p.stages = std::min(kMaxStages, (kSharedSmemLimit - 1024 - behind) / block);
  q.g = g.x;
  q.u = g.x2;
  q.gx = g.gx;
  q.gw = g.gw;
  q.routed = g.routed;
  q.gk = g.gk;
  q.cluster = C;
  q.trigger = g.trigger;
  q.pdl_wait = g.pdl_wait;
  const size_t smem = 1024 + static_cast<size_t>(p.stages) * block + behind;
  // like the streaming kernels that take the shorter calls of this op, it runs on the device they were set up for
  cudaError_t err = CheckConfiguredDevice();
  if (err == cudaSuccess) err = ConfigureDenseKernels();
  if (err == cudaSuccess) {
    err = mode == kBf16    ? LaunchShared<kBf16>(q, p.tiles, smem, stream)
          : mode == kFp8   ? LaunchShared<kFp8>(q, p.tiles, smem, stream)
          : mode == kNvfp4 ? LaunchShared<kNvfp4>(q, p.tiles, smem, stream)
                           : LaunchShared<kNvfp4Odd>(q, p.tiles, smem, stream);
  }
  if (err == cudaSuccess) err = cudaGetLastError();
  if (err != cudaSuccess) throw std::runtime_error(std::string("SharedExpertDown: ") + cudaGetErrorString(err));
  return true;
}

}  // namespace qfg
