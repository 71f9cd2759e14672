// SkinnyGemm for B200 (sm_100a): y[M, N] = x[M, K] @ W[K, N] for M <= 8 rows, streaming W once.
//
// A CTA of wn x wk warps owns one column tile of one weight and one 1/cluster slice of K.  A warp
// consumes 16 weight rows x (64 or 128) columns per k-step: a thread holds four rows of its 8/16
// columns, turns them into k-paired 16-bit operands (BF16: byte permute; FP8: byte permute +
// cvt.e4m3x2; NVFP4: nibble interleave + cvt.e2m1x2 + one packed multiply by the E4M3 block
// scales) and issues m16n8k16 MMAs with the weights as the 16-row operand and x (padded to 8 rows)
// as the 8-column operand.  Every weight and every product is exact; accumulation is FP32.
//
// Calls whose rows tensor copies can fetch go to skinny_stream.cu; these kernels take the rest (K not a multiple of eight, x
// off 16 bytes, rows off 16 bytes or NVFP4 widths off 128) and launch shapes pinned with the `plan` option.  Two of them share
// that arithmetic and differ in how the weight bytes reach the registers:
//   * SkinnyGemmDirectKernel (the fast path): every warp streams its own rows from HBM into a
//     warp-private shared-memory ring with lane-private cp.async copies, `depth` k-steps ahead of
//     the MMAs.  No CTA barrier in the K loop; the bytes in flight per SM are warps x depth x
//     1-2 KiB, bounded by shared memory rather than registers (a B200 needs well over 100 KiB in
//     flight per SM to stream at HBM speed).  Needs 16-byte aligned rows (8 for NVFP4) and whole
//     thread chunks.
//   * SkinnyGemmRingKernel (any 4-byte aligned layout, ragged column tails): all threads feed a
//     multi-stage shared-memory ring with cp.async pieces of 16, 8 or 4 bytes with zero fill.
//
// Partial sums are combined in a fixed order: across the wk warps through shared memory, then
// across the CTAs of the cluster through distributed shared memory, then scaled by the per-column
// w_scale, rounded once to BF16 and routed to the output that owns the column.  With `lm` set the
// epilogue also folds the BF16-rounded values into a per-row (max, index) key (fused LM head).
//
// The quantised modes run the MMA in FP16 (the only type cvt.e2m1x2 / cvt.e4m3x2 produce).  x is
// BF16, so each CTA rescales its K slice of every x row by a power of two that puts the row
// maximum in [2^14, 2^15) and converts it to FP16; if any element is not exactly representable
// (dynamic range above 2^28 inside one slice, infinities, NaNs) the CTA takes the BF16 path
// instead, which converts the dequantised weights to BF16 and multiplies by the unscaled x.
// Both paths feed the tensor core exact operands.
#include <algorithm>
#include <climits>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>
#include <utility>

#include "skinny_common.cuh"

namespace qfg {
namespace {

constexpr int kRingThreads = 256;  // ring kernel: up to 8 warps

// ------------------------------------------------------------------------------ direct kernel
// Every warp streams its own weight rows into a warp-private shared-memory ring with 16-byte
// cp.async.cg copies (L1 bypass), DEPTH k-steps ahead of the MMAs.  There is no CTA barrier in
// the K loop, and the bytes in flight per SM (warps x DEPTH x 2-3 KiB) are bounded by shared
// memory, not by registers.  Measured on B200: this copy pattern streams at over 6 TB/s with 16
// warps per SM, where 8-byte copies through L1 or register loads at the same occupancy stay
// below 4 TB/s.
//
// Ring slot of one warp.
//   BF16 / FP8: [4 rows][32 lanes][16 bytes]; every lane copies exactly the bytes it consumes.
//   NVFP4: the warp's 64 W nibble bytes of each of the 16 rows, copied as aligned 16-byte pieces
//     (a chunk that starts 8 bytes off a 16-byte boundary - odd rows of a weight whose packed
//     pitch is 8 mod 16, like the 151936-column LM head, or a tile whose first column is 16 mod
//     32 - takes one piece more and is read back at an offset of 8), then the one or two aligned
//     pieces around the warp's 8 W block-scale bytes of each row.  Rows 8..15 of the nibble area
//     and every fourth row of the scale area are displaced by 32 bytes, which puts the four row
//     groups a warp-wide shared-memory load touches into distinct banks.
// A lane owns up to kPieces pieces; their sources are one 64-bit base, advanced by a k-step
// stride per step, plus a 32-bit offset each.
template <typename T>
__device__ __forceinline__ void Pin(T& v) {
  asm volatile("" : "+r"(v));  // keeps a loop invariant in its register instead of being recomputed
}
__device__ __forceinline__ void CpAsync16If(uint32_t pred, uint32_t dst, const uint8_t* base, uint32_t off) {
  asm volatile(
      "{ .reg .pred p; .reg .u64 a;\n"
      " setp.ne.b32 p, %0, 0;\n"
      " mad.wide.u32 a, %3, 1, %2;\n"
      " @p cp.async.cg.shared.global [%1], [a], 16;\n}" ::"r"(pred), "r"(dst), "l"(base), "r"(off)
      : "memory");
}

template <int MODE, int W>
struct DirectSlot {
  using G = Geom<MODE, W>;
  static constexpr int kNibPitch = 64 * W + 16;                 // NVFP4: bytes per nibble row of a warp
  static constexpr int kNibBytes = MODE == kNvfp4 ? 16 * kNibPitch + 32 : 4 * 32 * G::kBytesPerThread;
  static constexpr int kSclPitch = 32;
  static constexpr int kSclBytes = MODE == kNvfp4 ? 16 * kSclPitch + 96 : 0;
  static constexpr int kBytes = kNibBytes + kSclBytes;
  static constexpr int kPiecesPerRow = 4 * W + 3;               // NVFP4: 4W+1 nibble pieces, 2 scale pieces
  static constexpr int kPieces = MODE == kNvfp4 ? (16 * kPiecesPerRow + 31) / 32 : 4;
  __device__ static constexpr int NibRow(int r) { return r * kNibPitch + ((r >> 3) & 1) * 32; }
  __device__ static constexpr int SclRow(int r) { return kNibBytes + r * kSclPitch + (r >> 2) * 32; }
};

// One warp's NVFP4 stream (128 columns): copy plan, ring and read offsets of the direct kernel, W = 1.
template <int DEPTH>
struct Nvfp4Stream {
  using S = DirectSlot<kNvfp4, 1>;
  static constexpr int NP = S::kPieces;
  const uint8_t* gbase;
  long long step_stride;
  uint32_t off[NP], dst[NP], pmask, rd_w[2], rd_s[2], ring;
  int nsteps, careful_step, row0, lane, kstride;

  // k-steps wk, wk + p.wk, ... of the CTA's K slice
  __device__ __forceinline__ void Setup(const GemmParams& p, const Tile& tl, const Segment& sg, int colwarp, int wk,
                                        uint32_t ring_addr, bool active) {
    const int ksteps = (tl.kslice + 15) >> 4;
    SetupRange(tl, sg, colwarp, wk, (active && ksteps > wk) ? (ksteps - wk + p.wk - 1) / p.wk : 0, p.wk, ring_addr);
  }

  // k-steps k_first, k_first + k_stride, ... (k_count of them) of the CTA's K slice; colwarp is a column of the weight
  __device__ __forceinline__ void SetupRange(const Tile& tl, const Segment& sg, int colwarp, int k_first, int k_count,
                                             int k_stride, uint32_t ring_addr) {
    lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const long long pitch = sg.pitch;
    const int ksteps = (tl.kslice + 15) >> 4;
    nsteps = k_count;
    kstride = k_stride;
    // the slice's last k-step is copied by the careful path
    careful_step = (k_count > 0 && ksteps - 1 >= k_first && (ksteps - 1 - k_first) % k_stride == 0 &&
                    (ksteps - 1 - k_first) / k_stride < k_count)
                       ? (ksteps - 1 - k_first) / k_stride
                       : -1;
    row0 = tl.kbeg + k_first * 16;
    step_stride = static_cast<long long>(k_stride) * 16 * pitch;
    ring = ring_addr;
    const long long warp_col_byte = colwarp / 2;
    gbase = sg.w + static_cast<long long>(row0) * pitch + warp_col_byte - 16;
    const int mis = static_cast<int>(pitch & 8);
    const int cshift = static_cast<int>(warp_col_byte & 8);
    const long long sabs = static_cast<long long>(sg.n >> 1) + (colwarp >> 4);
    const int so_even = static_cast<int>(sabs & 15), so_odd = static_cast<int>((sabs + mis) & 15);
    const int sh_even = cshift, sh_odd = (mis + cshift) & 15;
    pmask = 0;
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      const int slot = lane + 32 * j;
      const int r = slot / S::kPiecesPerRow, c = slot - r * S::kPiecesPerRow;
      off[j] = 0;
      dst[j] = 0;
      if (r < 16) {
        if (c < 5) {
          const int shift = (r & 1) ? sh_odd : sh_even;
          if (c < 4 || shift != 0) pmask |= 1u << j;
          off[j] = static_cast<uint32_t>(static_cast<long long>(r) * pitch + (c * 16 - shift) + 16);
          dst[j] = static_cast<uint32_t>(S::NibRow(r) + c * 16);
        } else {
          const int c2 = c - 5;
          const int o = (r & 1) ? so_odd : so_even;
          if (c2 == 0 || o + 8 > 16) pmask |= 1u << j;
          off[j] = static_cast<uint32_t>(static_cast<long long>(r) * pitch + (sabs - o + c2 * 16 - warp_col_byte) + 16);
          dst[j] = static_cast<uint32_t>(S::SclRow(r) + c2 * 16);
        }
      }
    }
    const int rbase = S::NibRow(4 * t) + g * 8, sbase = S::SclRow(4 * t) + g;
    rd_w[0] = static_cast<uint32_t>(rbase + sh_even);
    rd_w[1] = static_cast<uint32_t>(rbase + sh_odd);
    rd_s[0] = static_cast<uint32_t>(sbase + so_even);
    rd_s[1] = static_cast<uint32_t>(sbase + so_odd);
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      Pin(off[j]);
      Pin(dst[j]);
    }
    Pin(pmask);
    Pin(rd_w[0]);
    Pin(rd_w[1]);
    Pin(rd_s[0]);
    Pin(rd_s[1]);
  }

  __device__ __forceinline__ void Issue(const GemmParams& p, const Tile& tl, const Segment& sg, int s, uint32_t slot_addr) {
    if (s != careful_step) {
#pragma unroll
      for (int j = 0; j < NP; ++j) CpAsync16If(pmask & (1u << j), slot_addr + dst[j], gbase, off[j]);
    } else {
      const int r0 = row0 + s * kstride * 16;
#pragma unroll
      for (int j = 0; j < NP; ++j) {
        if (pmask & (1u << j)) {
          const int r = (lane + 32 * j) / S::kPiecesPerRow;
          const uint8_t* src = gbase + off[j];
          const long long room = sg.total_bytes - (src - sg.w);
          const int bytes = (r0 + r >= tl.kend) ? 0 : room >= 16 ? 16 : room > 0 ? static_cast<int>(room) : 0;
          CpAsync16(slot_addr + dst[j], bytes > 0 ? src : sg.w, bytes);
        }
      }
    }
    gbase += step_stride;
  }

  __device__ __forceinline__ void Prologue(const GemmParams& p, const Tile& tl, const Segment& sg) {
#pragma unroll
    for (int d = 0; d < DEPTH - 1; ++d) {
      if (d < nsteps) Issue(p, tl, sg, d, ring + d * S::kBytes);
      CpAsyncCommit();
    }
  }

  // consume(raw, s) for every local step s, DEPTH - 1 steps behind the copies
  template <class F>
  __device__ __forceinline__ void Run(const GemmParams& p, const Tile& tl, const Segment& sg, F&& consume) {
    const uint32_t ring_end = ring + DEPTH * S::kBytes;
    uint32_t rd_slot = ring, wr_slot = ring + (DEPTH - 1) * S::kBytes;
    for (int s = 0; s < nsteps; ++s) {
      __syncwarp();
      if (s + DEPTH - 1 < nsteps) Issue(p, tl, sg, s + DEPTH - 1, wr_slot);
      CpAsyncCommit();
      asm volatile("cp.async.wait_group %0;" ::"n"(DEPTH - 1) : "memory");
      __syncwarp();
      Raw<kNvfp4, 1> raw;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        raw.r[0][i] = Lds64(rd_slot + rd_w[i & 1] + i * S::kNibPitch);
        raw.s[0][i] = Lds8(rd_slot + rd_s[i & 1] + i * S::kSclPitch);
      }
      wr_slot = rd_slot;
      rd_slot += S::kBytes;
      if (rd_slot == ring_end) rd_slot = ring;
      consume(raw, s);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  }
};

// One warp's stream through its shared-memory ring: copy plan, read offsets and the K loop.
//
// A loop iteration handles a PAIR of the warp's k-steps (2 x 16 weight rows): one cp.async wait, one warp
// barrier, the copies of the pair DEPTH - 1 pairs ahead, then all shared-memory loads of both steps and
// their dequantisation and MMAs, which the compiler interleaves.  The body is not unrolled over the ring -
// the ring position is one register added to the few per-lane address registers - because the K loop runs
// out of the instruction cache of an SM sub-partition: a body over about 8 KB was measured 5-25 % slower.
//
// Slot of one k-step (RingSlot).  NVFP4 (column tiles start on multiples of 128 columns): 16 rows of
// 5 aligned 16-byte pieces around the row's 64 nibble bytes - the fifth is needed only where the chunk
// starts 8 bytes off a 16-byte boundary (odd rows of a weight whose packed pitch is 8 mod 16, like the
// 151936-column LM head) - then 16 rows of the one aligned piece that holds the row's 8 scale bytes.  The
// 160 nibble pieces of a pair are five copy instructions (piece index lane + 32 j), its 32 scale pieces a
// sixth, which keeps its lines in L1 (.ca): the four column warps whose scale bytes share a 32-byte sector
// then fetch it from L2 once, and the stream is bound by the sectors that cross from L2 to the SM (measured:
// 9.4 TB/s of sector traffic at 2.07 sector bytes per payload byte without this, 4.5 TB/s of weights).
// A lane whose index names an unneeded piece repeats piece 0 of that row (same source, same destination), so
// no copy is predicated.  Rows 8..15 of both areas are displaced (32 / 16 bytes), which puts the four rows a
// warp-wide load touches into distinct banks.  BF16 / FP8: [4 rows][32 lanes][16 bytes] per step, a lane
// copies exactly the bytes it consumes.  The last k-step of a K slice is copied by a careful path (rows past
// K read as zero, pieces clamped to the end of the tensor); a pair that contains it, or has no second step,
// takes that path for both steps.
template <int MODE>
struct RingSlot {
  static constexpr int kNibPitch = 80;
  static constexpr int kNibBytes = MODE == kNvfp4 ? 16 * kNibPitch + 32 : 4 * 32 * 16;
  static constexpr int kSclPitch = 16;
  static constexpr int kSclBytes = MODE == kNvfp4 ? 16 * kSclPitch + 16 : 0;
  static constexpr int kBytes = kNibBytes + kSclBytes;
  static constexpr int NP = MODE == kNvfp4 ? 6 : 8;  // copy instructions per pair of k-steps
  __device__ static constexpr int NibRow(int r) { return r * kNibPitch + ((r >> 3) & 1) * 32; }
  __device__ static constexpr int SclRow(int r) { return kNibBytes + r * kSclPitch + ((r >> 3) & 1) * 16; }
};
static_assert(RingSlot<kNvfp4>::kBytes == 1584 && RingSlot<kBf16>::kBytes == 2048, "keep RingSlotBytes() in step");

// The pieces of a lane within a pair of k-steps: source offset from the pair's base, destination offset in the
// ring, and (careful path) the row within the pair, 5 bits each.
template <int NP>
struct CopyPieces {
  uint32_t off[NP], dst[NP];
};
// Copies the pieces of a pair that belong to existing steps, with clamped sizes.
template <int NP>
__device__ __noinline__ void IssueCareful(const uint8_t* w, long long total_bytes, const uint8_t* gbase, int kend, int row0,
                                          int row_step, unsigned long long rows, CopyPieces<NP> pc, uint32_t slot_off, int steps) {
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    const int rr = static_cast<int>((rows >> (5 * j)) & 31u);  // step of the pair (bit 4) and row within it
    const int e = rr >> 4, r = rr & 15;
    if (e < steps) {
      const uint8_t* src = gbase + pc.off[j];
      const long long room = total_bytes - (src - w);
      const int bytes = (row0 + e * row_step + r >= kend) ? 0 : room >= 16 ? 16 : room > 0 ? static_cast<int>(room) : 0;
      CpAsync16(pc.dst[j] + slot_off, bytes > 0 ? src : w, bytes);
    }
  }
}

template <int MODE, int DEPTH>
struct WarpRing {
  using S = RingSlot<MODE>;
  static constexpr int NP = S::NP;
  static constexpr int kPairBytes = 2 * S::kBytes;
  static_assert(DEPTH >= 2 && DEPTH <= 4, "ring depth in pairs of k-steps");

  const uint8_t* gbase;  // next pair to copy, less 16 bytes (piece offsets are unsigned)
  long long step_stride;
  CopyPieces<NP> pc;     // dst includes the ring's address
  uint32_t rd_w[2], rd_s[2];
  unsigned long long rows;
  int nsteps, nfast, row_next, row_step;
  bool scales_l1;  // NVFP4: keep the scale pieces' lines in L1 (pays only while the CTA leaves L1 room beside its shared memory)

  // Local step s is k-step k_first + s * k_stride of the CTA's K slice, k_count steps in all.  `colwarp`:
  // first column of the warp; `lane_cols_ok`: the lane's own columns exist (BF16 / FP8 lanes past the
  // tile's last column copy the warp's first chunk instead; their sums are never stored).
  __device__ __forceinline__ void Setup(const Tile& tl, const Segment& sg, int colwarp, bool lane_cols_ok, int k_first,
                                        int k_count, int k_stride, uint32_t ring) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const long long pitch = sg.pitch;
    const int ksteps = (tl.kslice + 15) >> 4;
    nsteps = k_count;
    const int last = ksteps - 1 - k_first;
    const bool has_last = k_count > 0 && last >= 0 && last % k_stride == 0 && last / k_stride < k_count;
    nfast = has_last ? last / k_stride : nsteps;
    row_next = tl.kbeg + k_first * 16;
    row_step = k_stride * 16;
    step_stride = static_cast<long long>(k_stride) * 16 * pitch;
    rows = 0;
    scales_l1 = false;
    if constexpr (MODE == kNvfp4) {
      const long long warp_col_byte = colwarp / 2;  // a multiple of 64
      gbase = sg.w + static_cast<long long>(row_next) * pitch + warp_col_byte - 16;
      const int mis = static_cast<int>(pitch & 8);  // odd rows start 8 bytes off a 16-byte boundary
      const long long sabs = static_cast<long long>(sg.n >> 1) + (colwarp >> 4);  // scale bytes within the row: 0 or 8 mod 16
      const int so_even = static_cast<int>(sabs & 15), so_odd = static_cast<int>((sabs + mis) & 15);
#pragma unroll
      for (int j = 0; j < NP; ++j) {
        int e, r;
        long long src;
        uint32_t dst;
        if (j < 5) {  // nibble piece lane + 32 j of the pair's 2 x 16 x 5
          const int q = lane + 32 * j;
          e = q / 80;
          const int qq = q - e * 80;
          r = qq / 5;
          int c = qq - r * 5;
          const int shift = (r & 1) ? mis : 0;
          if (c == 4 && shift == 0) c = 0;
          src = c * 16 - shift;
          dst = static_cast<uint32_t>(S::NibRow(r) + c * 16);
        } else {      // scale piece of row lane % 16 of step lane / 16
          e = lane >> 4;
          r = lane & 15;
          const int o = (r & 1) ? so_odd : so_even;
          src = sabs - o - warp_col_byte;
          dst = static_cast<uint32_t>(S::SclRow(r));
        }
        pc.off[j] = static_cast<uint32_t>(static_cast<long long>(e) * step_stride + static_cast<long long>(r) * pitch + src + 16);
        pc.dst[j] = ring + dst + static_cast<uint32_t>(e * S::kBytes);
        rows |= static_cast<unsigned long long>(e * 16 + r) << (5 * j);
      }
      const int rbase = S::NibRow(4 * t) + g * 8, sbase = S::SclRow(4 * t) + g;
      rd_w[0] = ring + static_cast<uint32_t>(rbase);
      rd_w[1] = ring + static_cast<uint32_t>(rbase + mis);
      rd_s[0] = ring + static_cast<uint32_t>(sbase + so_even);
      rd_s[1] = ring + static_cast<uint32_t>(sbase + so_odd);
    } else {
      const long long warp_col_byte = MODE == kBf16 ? static_cast<long long>(colwarp) * 2 : colwarp;
      gbase = sg.w + static_cast<long long>(row_next) * pitch + warp_col_byte - 16;
      const int gsrc = lane_cols_ok ? g : 0;
#pragma unroll
      for (int j = 0; j < NP; ++j) {
        const int e = j >> 2, i = j & 3;
        pc.off[j] = static_cast<uint32_t>(static_cast<long long>(e) * step_stride + static_cast<long long>(4 * t + i) * pitch + gsrc * 16 + 16);
        pc.dst[j] = ring + static_cast<uint32_t>(e * S::kBytes + i * 512 + lane * 16);
        rows |= static_cast<unsigned long long>(e * 16 + 4 * t + i) << (5 * j);
      }
      rd_w[0] = rd_w[1] = ring + static_cast<uint32_t>(lane * 16);
      rd_s[0] = rd_s[1] = 0;
    }
  }

  // copies the pair of local steps (s0, s0 + 1) - the next ones in order - into the slots at `slot_off`
  __device__ __forceinline__ void IssuePair(const Tile& tl, const Segment& sg, int s0, uint32_t slot_off) {
    if (s0 + 1 < nfast) {
#pragma unroll
      for (int j = 0; j < NP; ++j) {
        if (MODE == kNvfp4 && j == NP - 1 && scales_l1) {
          CpAsync16At<0, true>(pc.dst[j] + slot_off, gbase, pc.off[j]);
        } else {
          CpAsync16At<0, false>(pc.dst[j] + slot_off, gbase, pc.off[j]);
        }
      }
    } else if (s0 < nsteps) {
      IssueCareful<NP>(sg.w, sg.total_bytes, gbase, tl.kend, row_next, row_step, rows, pc, slot_off, nsteps - s0);
    }
    gbase += 2 * step_stride;
    row_next += 2 * row_step;
  }

  // the first DEPTH - 1 pairs in flight
  __device__ __forceinline__ void Prologue(const Tile& tl, const Segment& sg) {
#pragma unroll
    for (int d = 0; d < DEPTH - 1; ++d) {
      IssuePair(tl, sg, 2 * d, static_cast<uint32_t>(d * kPairBytes));
      CpAsyncCommit();
    }
  }

  template <int OFF>
  __device__ __forceinline__ void LoadStep(Raw<MODE, 1>& raw, uint32_t w0, uint32_t w1, uint32_t s0, uint32_t s1) const {
    if constexpr (MODE == kNvfp4) {
      raw.r[0][0] = Lds64At<OFF>(w0);
      raw.r[0][1] = Lds64At<OFF + S::kNibPitch>(w1);
      raw.r[0][2] = Lds64At<OFF + 2 * S::kNibPitch>(w0);
      raw.r[0][3] = Lds64At<OFF + 3 * S::kNibPitch>(w1);
      raw.s[0][0] = Lds8At<OFF>(s0);
      raw.s[0][1] = Lds8At<OFF + S::kSclPitch>(s1);
      raw.s[0][2] = Lds8At<OFF + 2 * S::kSclPitch>(s0);
      raw.s[0][3] = Lds8At<OFF + 3 * S::kSclPitch>(s1);
    } else {
      raw.r[0] = Lds128At<OFF>(w0);
      raw.r[1] = Lds128At<OFF + 512>(w0);
      raw.r[2] = Lds128At<OFF + 1024>(w0);
      raw.r[3] = Lds128At<OFF + 1536>(w0);
    }
  }

  // consume(raw_a, raw_b, has_b) for every pair of local steps in order, DEPTH - 1 pairs behind the copies
  template <class F>
  __device__ __forceinline__ void Run(const Tile& tl, const Segment& sg, F&& consume) {
    const int npairs = (nsteps + 1) >> 1;
    uint32_t rd_off = 0, wr_off = static_cast<uint32_t>((DEPTH - 1) * kPairBytes);
    for (int i = 0; i < npairs; ++i) {
      asm volatile("cp.async.wait_group %0;" ::"n"(DEPTH - 2) : "memory");
      __syncwarp();  // every lane's copies of this pair are visible, and every lane is done reading the previous pair
      IssuePair(tl, sg, 2 * (i + DEPTH - 1), wr_off);
      CpAsyncCommit();
      Raw<MODE, 1> raw_a, raw_b;
      const uint32_t w0 = rd_w[0] + rd_off, w1 = rd_w[1] + rd_off, s0 = rd_s[0] + rd_off, s1 = rd_s[1] + rd_off;
      LoadStep<0>(raw_a, w0, w1, s0, s1);
      LoadStep<S::kBytes>(raw_b, w0, w1, s0, s1);
      consume(raw_a, raw_b, 2 * i + 1 < nsteps);
      wr_off = rd_off;
      rd_off += kPairBytes;
      if (rd_off == static_cast<uint32_t>(DEPTH * kPairBytes)) rd_off = 0;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  }
};

// DEPTH: pairs of k-steps in every warp's ring (2, 3 or 4)
// FUSE: the SharedExpertDown form (x = swish_mul(g, u) and the gate while x is staged, the gated rounding chain
// in the epilogue).  A kernel of its own, so that the plain kernels carry none of that code: they were measured
// to lose 2-3 % whenever it changed, run or not.
template <int MODE, int DEPTH, bool FUSE = false>
__global__ void __launch_bounds__(kMaxThreads, 1) SkinnyGemmDirectKernel(const __grid_constant__ GemmParams p) {
  using G = Geom<MODE, 1>;
  using S = RingSlot<MODE>;
  constexpr int NM = G::kMmas;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ SharedScratch sh;

  if (p.trigger == 1) GridLaunchDependents();
  Stamp(p, 0);
  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int wn = warp % p.wn, wk = warp / p.wn;
  const Tile tl = LocateTile(p);
  const Segment& sg = p.seg[tl.seg];

  // this thread's columns and this warp's k-steps (local step s is k-step wk + s * p.wk of the slice)
  constexpr int cols_per_warp = 8 * G::kColsPerThread;
  const int colwarp = tl.n0 + wn * cols_per_warp;
  const bool warp_has_cols = colwarp < tl.n1;
  const bool cvalid = colwarp + g * G::kColsPerThread < tl.n1;
  const int ksteps = (tl.kslice + 15) >> 4;
  const uint32_t ring_addr = SmemAddr(smem) + static_cast<uint32_t>(warp) * (DEPTH * 2 * S::kBytes);

  // Shared tail of the fused LM head: a warp without columns of the tile (the last warp column of the CTA)
  // streams one K slice of one left-over column group through the same loop and stores FP32 partial sums.
  bool tail_worker = false;
  int tail_index = 0, first_step = wk, step_stride = p.wk, step_count = (warp_has_cols && ksteps > wk) ? (ksteps - wk + p.wk - 1) / p.wk : 0;
  int stream_col = colwarp;
  if constexpr (MODE == kNvfp4) {
    if (p.tail_groups > 0 && !warp_has_cols && wn == p.wn - 1) {
      // one (group, K slice) per idle warp: spread over the CTAs, or in order where the CTAs are few
      bool mine = true;
      if (p.tail_stride > 0) {
        tail_index = static_cast<int>(blockIdx.x) / p.tail_stride;
        mine = tail_index * p.tail_stride == static_cast<int>(blockIdx.x) && wk == tail_index % p.wk;
      } else {
        tail_index = static_cast<int>(blockIdx.x) * p.wk + wk;
      }
      if (mine && tail_index < p.tail_groups * p.tail_split) {
        tail_worker = true;
        const int tg = tail_index / p.tail_split, slice = tail_index - tg * p.tail_split;
        const unsigned split = static_cast<unsigned>(p.tail_split);
        first_step = static_cast<int>(static_cast<unsigned>(slice) * ksteps / split);
        step_count = static_cast<int>(static_cast<unsigned>(slice + 1) * ksteps / split) - first_step;
        step_stride = 1;
        stream_col = sg.n - p.tail_groups * 128 + tg * 128;
      }
    }
  }

  // x first (unless it is still the predecessor kernel's to write): its copies then do not queue behind the weights
  uint16_t* xs = reinterpret_cast<uint16_t*>(smem + p.ring_bytes);
  const bool x_async = !FUSE && XRowsAre16ByteAligned(p);
  if (x_async && !p.pdl_wait) {
    XCopyIssue(p, tl, xs);
    CpAsyncCommit();
  }
  // weights do not depend on the predecessor kernel: get the first k-steps in flight, then wait
  WarpRing<MODE, DEPTH> ring;
  ring.Setup(tl, sg, stream_col, cvalid, first_step, step_count, step_stride, ring_addr);
  ring.scales_l1 = p.scales_l1 != 0;
  ring.Prologue(tl, sg);
  if (p.pdl_wait) GridDependencyWait();
  Stamp(p, 1);

  bool slow;
  if (x_async) {
    if (p.pdl_wait) {  // x belongs to the predecessor until now
      XCopyIssue(p, tl, xs);
      CpAsyncCommit();
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group %0;" ::"n"(DEPTH - 1) : "memory");
    }
    slow = StageXConvert<MODE>(p, tl, xs, sh);
  } else {
    slow = StageX<MODE, false, true, FUSE>(p, tl, xs, sh);
  }
  Stamp(p, 2);

  float acc[NM][4];
#pragma unroll
  for (int j = 0; j < NM; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;

  // lanes whose x row does not exist read row 0; their accumulators are never stored
  uint32_t x_rd = SmemAddr(xs) + static_cast<uint32_t>(((g < p.M ? g : 0) * p.xpitch + 4 * t + first_step * 16) * 2);
  const uint32_t x_step = static_cast<uint32_t>(step_stride) * 32u;
  // One copy of the loop per operand path: the loop body then holds a single dequantisation.
  auto k_loop = [&](auto slow_tag) {
    constexpr bool kSlow = decltype(slow_tag)::value;
    ring.Run(tl, sg, [&](const Raw<MODE, 1>& raw_a, const Raw<MODE, 1>& raw_b, bool has_b) {
      const uint2 xa = Lds64(x_rd);
      ComputeStep<MODE, kSlow, 1>(acc, raw_a, xa.x, xa.y);
      if (has_b) {  // warp-uniform
        const uint2 xb = Lds64(x_rd + x_step);
        ComputeStep<MODE, kSlow, 1>(acc, raw_b, xb.x, xb.y);
      }
      x_rd += 2 * x_step;
    });
  };
  if constexpr (MODE == kBf16) {
    k_loop(std::false_type{});
  } else {
    if (slow) {
      k_loop(std::true_type{});
    } else {
      k_loop(std::false_type{});
    }
  }
  if constexpr (MODE == kNvfp4) {
    if (tail_worker) {
      float* dstp = p.lm_tail + static_cast<size_t>(tail_index) * kMaxRows * 128;
#pragma unroll
      for (int j = 0; j < NM; ++j) {
        const int cl = g * 16 + 2 * j;
        const int m0 = 2 * t, m1 = 2 * t + 1;
        if (m0 < p.M) *reinterpret_cast<float2*>(&dstp[m0 * 128 + cl]) = make_float2(acc[j][0], acc[j][2]);
        if (m1 < p.M) *reinterpret_cast<float2*>(&dstp[m1 * 128 + cl]) = make_float2(acc[j][1], acc[j][3]);
      }
      __threadfence();
    }
  }
  Stamp(p, 3);
  if (p.trigger == 2) GridLaunchDependents();
  __syncthreads();
  Stamp(p, 4);
  Epilogue<MODE, 1, FUSE>(p, tl, acc, smem, sh, warp_has_cols);
  Stamp(p, 5);
}


// ------------------------------------------------------------------------------ register-streaming kernel
// BF16 / FP8 only.  Every warp loads its rows straight into registers with 128-bit non-allocating
// loads, D k-steps ahead of the MMAs: no shared-memory ring, no cp.async, nothing to fill before the
// first MMA.  On the 50 MB decode projections (a dozen k-steps per warp) that start-up matters more
// than the deeper prefetch of the warp rings; on long streams the rings win.
constexpr int kRegThreads = 512;

template <int MODE, bool FUSE = false>
__global__ void __launch_bounds__(kRegThreads, 1) SkinnyGemmRegKernel(const __grid_constant__ GemmParams p) {
  using G = Geom<MODE>;
  constexpr int NM = G::kMmas;
  constexpr int D = MODE == kBf16 ? 4 : 3;  // k-steps in flight per warp (16 registers each)
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ SharedScratch sh;

  if (p.trigger == 1) GridLaunchDependents();
  Stamp(p, 0);
  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int wn = warp % p.wn, wk = warp / p.wn;
  const Tile tl = LocateTile(p);
  const Segment& sg = p.seg[tl.seg];
  const long long pitch = sg.pitch;

  // this thread's columns and this warp's k-steps (local step s is k-step wk + s * p.wk of the slice)
  const int cols_per_warp = 8 * G::kColsPerThread;
  const int colbase = tl.n0 + wn * cols_per_warp + g * G::kColsPerThread;
  const bool warp_has_cols = tl.n0 + wn * cols_per_warp < tl.n1;
  // threads past the tile's last column load nothing; their pointer is parked on the tile's first chunk
  const bool cvalid = colbase < tl.n1;
  const int colload = cvalid ? colbase : tl.n0;
  const int ksteps = (tl.kslice + 15) >> 4;
  const int nsteps = ksteps > wk ? (ksteps - wk + p.wk - 1) / p.wk : 0;
  // only the last k-step of the slice can be partial (K not a multiple of 16)
  const bool tail_here = (tl.kslice & 15) != 0 && ((ksteps - 1) % p.wk) == wk;
  const long long col_byte = (MODE == kBf16) ? static_cast<long long>(colload) * 2 : (MODE == kFp8) ? colload : colload / 2;
  // a thread owns rows 4t .. 4t+3 of a k-step (the k index of an MMA is a free permutation)
  const uint8_t* wq = sg.w + static_cast<long long>(tl.kbeg + wk * 16 + 4 * t) * pitch + col_byte;  // next step to load
  const long long scale_delta = static_cast<long long>(sg.n >> 1) + (colload >> 4) - col_byte;
  const long long step_stride = static_cast<long long>(p.wk) * 16 * pitch;
  const long long pitch2 = 2 * pitch, pitch3 = 3 * pitch;

  // loads local step s (steps are loaded in increasing order, so a running pointer suffices)
  auto load_step = [&](Raw<MODE>& raw, int s) {
    const uint8_t* q0 = wq;
    wq += step_stride;
    if (tail_here && s == nsteps - 1) {
      const int r = tl.kbeg + (wk + s * p.wk) * 16 + 4 * t;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const bool ok = cvalid && r + i < tl.kend;
        if constexpr (MODE == kNvfp4) {
          raw.r[i] = ok ? Ldg64(q0 + i * pitch) : make_uint2(0, 0);
          raw.s[i] = ok ? Ldg8(q0 + i * pitch + scale_delta) : 0u;
        } else {
          raw.r[i] = ok ? Ldg128(q0 + i * pitch) : make_uint4(0, 0, 0, 0);
        }
      }
      return;
    }
    const uint8_t* q1 = q0 + pitch;
    const uint8_t* q2 = q0 + pitch2;
    const uint8_t* q3 = q0 + pitch3;
    if (!cvalid) {  // columns past the tile: nothing to stream, the sums are never stored
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if constexpr (MODE == kNvfp4) {
          raw.r[i] = make_uint2(0, 0);
          raw.s[i] = 0u;
        } else {
          raw.r[i] = make_uint4(0, 0, 0, 0);
        }
      }
      return;
    }
    if constexpr (MODE == kNvfp4) {
      raw.r[0] = Ldg64(q0);
      raw.r[1] = Ldg64(q1);
      raw.r[2] = Ldg64(q2);
      raw.r[3] = Ldg64(q3);
      raw.s[0] = Ldg8(q0 + scale_delta);
      raw.s[1] = Ldg8(q1 + scale_delta);
      raw.s[2] = Ldg8(q2 + scale_delta);
      raw.s[3] = Ldg8(q3 + scale_delta);
    } else {
      raw.r[0] = Ldg128(q0);
      raw.r[1] = Ldg128(q1);
      raw.r[2] = Ldg128(q2);
      raw.r[3] = Ldg128(q3);
    }
  };

  // x first (unless it is still the predecessor kernel's to write): its copies then do not queue behind the weights
  uint16_t* xs = reinterpret_cast<uint16_t*>(smem + p.ring_bytes);
  const bool x_async = !FUSE && XRowsAre16ByteAligned(p);
  if (x_async && !p.pdl_wait) {
    XCopyIssue(p, tl, xs);
    CpAsyncCommit();
  }
  // weights do not depend on the predecessor kernel: get the first k-steps in flight, then wait
  Raw<MODE> buf[D];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    if (warp_has_cols && d < nsteps) load_step(buf[d], d);
  }
  Stamp(p, 1);
  if (p.pdl_wait) GridDependencyWait();

  bool slow;
  if (x_async) {
    if (p.pdl_wait) {
      XCopyIssue(p, tl, xs);
      CpAsyncCommit();
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    slow = StageXConvert<MODE>(p, tl, xs, sh);
  } else {
    slow = StageX<MODE, false, false, FUSE>(p, tl, xs, sh);
  }
  Stamp(p, 2);

  float acc[NM][4];
#pragma unroll
  for (int j = 0; j < NM; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;

  const uint32_t xs_addr = SmemAddr(xs) + static_cast<uint32_t>((g * p.xpitch + 4 * t) * 2);
  const bool has_row = g < p.M;
  if (warp_has_cols) {
    for (int base = 0; base < nsteps; base += D) {
#pragma unroll
      for (int d = 0; d < D; ++d) {
        const int s = base + d;
        if (s < nsteps) {
          uint32_t b0 = 0, b1 = 0;
          if (has_row) {
            const uint2 xv = Lds64(xs_addr + static_cast<uint32_t>(wk + s * p.wk) * 32u);
            b0 = xv.x;
            b1 = xv.y;
          }
          if constexpr (MODE == kBf16) {
            ComputeStep<MODE, false>(acc, buf[d], b0, b1);
          } else {
            if (slow) {
              ComputeStep<MODE, true>(acc, buf[d], b0, b1);
            } else {
              ComputeStep<MODE, false>(acc, buf[d], b0, b1);
            }
          }
          if (s + D < nsteps) load_step(buf[d], s + D);
        }
      }
    }
  }
  Stamp(p, 3);
  if (p.trigger == 2) GridLaunchDependents();
  __syncthreads();
  Stamp(p, 4);
  Epilogue<MODE, 1, FUSE>(p, tl, acc, smem, sh, warp_has_cols);
  Stamp(p, 5);
}

// ------------------------------------------------------------------------------ tcgen05 kernel
// NVFP4 only.  The warp rings, the dequantisation and the epilogue are those of the direct kernel;
// the MMAs move from the legacy mma.sync pipe (measured: busy 62 % of all cycles and the first
// limiter of the direct kernel) to tcgen05.mma with the accumulators in tensor memory:
//   * warps come in groups of four side by side in N (a warpgroup, 512 columns); warp q of a group
//     can only touch TMEM lanes [32 q, 32 q + 32), so the four warps together fill the 128 lanes of
//     an A tile.  Per k-step a warp stores its eight 16-column x 16-row fragments with two
//     tcgen05.st.16x256b.x4 - that shape has exactly the register layout of the mma.sync A
//     fragment - into four A tiles (fragment j goes to tile j / 2, lanes 16 (j % 2) + ...).
//   * x is staged as the K-major no-swizzle B operand (8 rows x 16 k per step; rows 8..15 of the
//     N = 16 instruction alias the next step's bytes and land in accumulator columns nobody reads).
//   * one extra warp issues, in increasing k order, four M128 N16 K16 MMAs per warpgroup k-step and
//     commits them to the mbarrier that frees the A buffer (three buffers per warpgroup).  All K
//     groups of a column group accumulate into the same TMEM tile, so the sum over K runs in
//     k order whatever wk is.
//   * tile columns past wn x 128 (at most 128 more) are handled by wk extra warps on the mma.sync
//     path, so that a tile does not have to be a multiple of 512 columns.
// Every wait on an mbarrier is bounded.
constexpr int kTcBuffers = 3;
constexpr int kTcSpin = 1 << 22;
constexpr int kTcMaxGroups = 8;  // warpgroups per CTA (TMEM: groups x buffers x 32 + 64 per column group <= 512)

__device__ __forceinline__ void MbarInit(uint32_t addr, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(addr), "r"(count) : "memory");
}
__device__ __forceinline__ void MbarArrive(uint32_t addr) {
  asm volatile("{ .reg .b64 st; mbarrier.arrive.shared::cta.b64 st, [%0]; }" ::"r"(addr) : "memory");
}
// false if the phase did not complete within the spin limit (the caller carries on; results are then wrong
// but nothing hangs)
__device__ __forceinline__ bool MbarWait(uint32_t addr, uint32_t parity) {
  uint32_t done = 0;
  for (int spin = 0; spin < kTcSpin && !done; ++spin) {
    asm volatile("{ .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(done)
                 : "r"(addr), "r"(parity)
                 : "memory");
  }
  return done != 0;
}
__device__ __forceinline__ void TcFenceBefore() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void TcFenceAfter() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

struct TcShared {
  unsigned long long full[kTcMaxGroups][kTcBuffers];   // 4 arrivals: the warps of the group stored their fragments
  unsigned long long empty[kTcMaxGroups][kTcBuffers];  // 1 arrival: the MMAs that read the buffer completed
  unsigned long long done;                             // 1 arrival: every MMA of the CTA completed
  uint32_t tmem_base;
  uint32_t fault;
};

// The A operand registers of the eight 16-column MMAs of one k-step (fr[j] = {a0, a1, a2, a3} of MMA j as
// ComputeStep would pass them to mma.sync).
template <bool SLOW>
__device__ __forceinline__ void Nvfp4Fragments(const Raw<kNvfp4, 1>& w, uint32_t (&fr)[8][4]) {
  const uint32_t s_ab = CvtE4m3x2(Prmt(w.s[0][0], w.s[0][1], 0x0040u));
  const uint32_t s_cd = CvtE4m3x2(Prmt(w.s[0][2], w.s[0][3], 0x0040u));
  const uint32_t a[2] = {w.r[0][0].x, w.r[0][0].y}, b[2] = {w.r[0][1].x, w.r[0][1].y};
  const uint32_t c[2] = {w.r[0][2].x, w.r[0][2].y}, d[2] = {w.r[0][3].x, w.r[0][3].y};
#pragma unroll
  for (int i = 0; i < 2; ++i) {
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
      fr[4 * i + q][0] = a0;
      fr[4 * i + q][1] = a1;
      fr[4 * i + q][2] = a2;
      fr[4 * i + q][3] = a3;
    }
  }
}

// Fragments `half`, `half` + 2, `half` + 4, `half` + 6 of a k-step into lanes [lane_base, lane_base + 16) of the
// four A tiles of a buffer (32 TMEM columns from `taddr`).  A 16x256b store takes, per 8-column tile,
// (row g: k 4t..4t+1), (row g: k 4t+2..4t+3), (row g + 8: ...), (row g + 8: ...) = a0, a2, a1, a3.
__device__ __forceinline__ void TcStoreHalf(uint32_t taddr, const uint32_t (&fr)[8][4], int half) {
  const uint32_t(&f0)[4] = fr[half], (&f1)[4] = fr[half + 2], (&f2)[4] = fr[half + 4], (&f3)[4] = fr[half + 6];
  asm volatile(
      "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(
          taddr),
      "r"(f0[0]), "r"(f0[2]), "r"(f0[1]), "r"(f0[3]), "r"(f1[0]), "r"(f1[2]), "r"(f1[1]), "r"(f1[3]), "r"(f2[0]), "r"(f2[2]),
      "r"(f2[1]), "r"(f2[3]), "r"(f3[0]), "r"(f3[2]), "r"(f3[1]), "r"(f3[3])
      : "memory");
}

template <int DEPTH>
__global__ void __launch_bounds__(kMaxThreads, 1) SkinnyGemmTcKernel(const __grid_constant__ GemmParams p) {
  using S = DirectSlot<kNvfp4, 1>;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ SharedScratch sh;
  __shared__ __align__(8) TcShared tc;

  if (p.trigger == 1) GridLaunchDependents();
  Stamp(p, 0);
  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int nd = p.wn * p.wk;        // dequantising warps feeding tcgen05
  const int ngroups = p.wn >> 2;     // column groups of 512
  const bool is_tc = warp < nd, is_issuer = warp == nd, is_legacy = warp > nd;
  const int wn = is_tc ? warp % p.wn : p.wn;                       // legacy warps own the column warp after the last
  const int wk = is_tc ? warp / p.wn : (is_legacy ? warp - nd - 1 : 0);
  const int q = wn & 3, ng = wn >> 2;                              // quadrant and column group of a TC warp
  const int unit = wk * ngroups + ng;                              // warpgroup index
  const Tile tl = LocateTile(p);
  const Segment& sg = p.seg[tl.seg];
  const int colwarp = tl.n0 + wn * 128;
  const bool warp_has_cols = !is_issuer && colwarp < tl.n1;
  const int ksteps = (tl.kslice + 15) >> 4;
  const int TNc = (p.wn + 1) * 128;

  if (tid == 0) {
    for (int u = 0; u < p.wk * ngroups; ++u)
      for (int b = 0; b < kTcBuffers; ++b) {
        MbarInit(SmemAddr(&tc.full[u][b]), 4);
        MbarInit(SmemAddr(&tc.empty[u][b]), 1);
      }
    MbarInit(SmemAddr(&tc.done), 1);
    tc.fault = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  const int d_cols = ngroups * 64;
  const int need_cols = d_cols + p.wk * ngroups * kTcBuffers * 32;
  const int alloc_cols = need_cols <= 32 ? 32 : need_cols <= 64 ? 64 : need_cols <= 128 ? 128 : need_cols <= 256 ? 256 : 512;
  if (is_issuer) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(SmemAddr(&tc.tmem_base)), "r"(alloc_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }

  Nvfp4Stream<DEPTH> st;
  st.Setup(p, tl, sg, colwarp, wk, SmemAddr(smem) + static_cast<uint32_t>(is_legacy ? nd + wk : warp) * (DEPTH * S::kBytes),
           warp_has_cols);
  // a TC warp without columns still takes part in the barrier protocol of its group
  const int proto_steps = (is_tc && ksteps > wk) ? (ksteps - wk + p.wk - 1) / p.wk : 0;
  if (!is_issuer) st.Prologue(p, tl, sg);
  if (p.pdl_wait) GridDependencyWait();
  Stamp(p, 1);

  uint16_t* xs = reinterpret_cast<uint16_t*>(smem + p.ring_bytes);
  const bool slow = p.fuse ? StageX<kNvfp4, true, true, true>(p, tl, xs, sh) : StageX<kNvfp4, true>(p, tl, xs, sh);
  TcFenceBefore();
  __syncthreads();
  TcFenceAfter();
  Stamp(p, 2);
  const uint32_t tmem = tc.tmem_base;

  float acc[8][4];  // legacy warps only
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;

  if (is_tc) {
    const uint32_t a_base = tmem + static_cast<uint32_t>(d_cols + unit * kTcBuffers * 32) + (static_cast<uint32_t>(32 * q) << 16);
    const uint32_t full0 = SmemAddr(&tc.full[unit][0]), empty0 = SmemAddr(&tc.empty[unit][0]);
    int b = 0, round = 0;  // buffer of step s and how many times the buffers were cycled
    auto publish = [&](const Raw<kNvfp4, 1>* raw) {
      uint32_t fr[8][4];
      if (raw != nullptr) {
        if (slow) {
          Nvfp4Fragments<true>(*raw, fr);
        } else {
          Nvfp4Fragments<false>(*raw, fr);
        }
      }
      if (round > 0 && !MbarWait(empty0 + b * 8, static_cast<uint32_t>((round - 1) & 1))) tc.fault = 1;
      if (raw != nullptr) {
        TcFenceAfter();
        const uint32_t ta = a_base + static_cast<uint32_t>(b * 32);
        TcStoreHalf(ta, fr, 0);
        TcStoreHalf(ta + (16u << 16), fr, 1);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        TcFenceBefore();
      }
      __syncwarp();
      if (lane == 0) MbarArrive(full0 + b * 8);
      if (++b == kTcBuffers) {
        b = 0;
        ++round;
      }
    };
    if (warp_has_cols) {
      st.Run(p, tl, sg, [&](const Raw<kNvfp4, 1>& raw, int) { publish(&raw); });
    } else {
      for (int s = 0; s < proto_steps; ++s) publish(nullptr);
    }
  } else if (is_issuer) {
    if (lane == 0) {
      const uint32_t idesc = 0x10u | (2u << 17) | (8u << 24) | (slow ? ((1u << 7) | (1u << 10)) : 0u);
      const uint32_t xa = SmemAddr(xs);
      const int max_steps = (ksteps + p.wk - 1) / p.wk;
      int b = 0, round = 0;
      for (int s = 0; s < max_steps; ++s) {
        for (int wkI = 0; wkI < p.wk; ++wkI) {
          const int kk = wkI + s * p.wk;
          if (kk >= ksteps) break;
          // x tile of k-step kk: 256 bytes; K chunks 128 bytes apart; rows 8..15 alias the next 256 bytes
          const unsigned long long desc = static_cast<unsigned long long>(((xa + static_cast<uint32_t>(kk) * 256u) >> 4) & 0x3FFF) |
                                          (static_cast<unsigned long long>(128 >> 4) << 16) |
                                          (static_cast<unsigned long long>(256 >> 4) << 32) | (1ull << 46);
          for (int gi = 0; gi < ngroups; ++gi) {
            const int u = wkI * ngroups + gi;
            if (!MbarWait(SmemAddr(&tc.full[u][b]), static_cast<uint32_t>(round & 1))) tc.fault = 1;
            TcFenceAfter();
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint32_t d_t = tmem + static_cast<uint32_t>(gi * 64 + i * 16);
              const uint32_t a_t = tmem + static_cast<uint32_t>(d_cols + (u * kTcBuffers + b) * 32 + i * 8);
              asm volatile(
                  "{ .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                  " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n}" ::"r"(d_t),
                  "r"(a_t), "l"(desc), "r"(idesc), "r"(kk > 0 ? 1 : 0), "r"(0)
                  : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             SmemAddr(&tc.empty[u][b]))
                         : "memory");
          }
        }
        if (++b == kTcBuffers) {
          b = 0;
          ++round;
        }
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(SmemAddr(&tc.done))
                   : "memory");
    }
    __syncwarp();
  } else {
    // mma.sync path for the tile's columns past the warpgroups
    const int x_row = g < p.M ? g : 0;
    uint32_t x_rd = SmemAddr(xs) + static_cast<uint32_t>(wk * 256 + (t >> 1) * 128 + x_row * 16 + (t & 1) * 8);
    const uint32_t x_step = static_cast<uint32_t>(p.wk) * 256u;
    st.Run(p, tl, sg, [&](const Raw<kNvfp4, 1>& raw, int) {
      const uint2 xv = Lds64(x_rd);
      x_rd += x_step;
      if (slow) {
        ComputeStep<kNvfp4, true, 1>(acc, raw, xv.x, xv.y);
      } else {
        ComputeStep<kNvfp4, false, 1>(acc, raw, xv.x, xv.y);
      }
    });
  }
  Stamp(p, 3);
  if (p.trigger == 2) GridLaunchDependents();
  // all MMAs done before anybody reads the accumulators or reuses the ring as `red`
  if (!MbarWait(SmemAddr(&tc.done), 0)) tc.fault = 1;
  TcFenceAfter();
  __syncthreads();
  Stamp(p, 4);

  float* red = reinterpret_cast<float*>(smem);
  const int M = p.M;
  if (is_tc) {
    if (wk == 0) {
      // accumulators of this warp's 128 columns: TMEM lane 32 q + L of the group's four tiles, column n = x row
      uint32_t d[4][8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t ta = tmem + static_cast<uint32_t>(ng * 64 + i * 16) + (static_cast<uint32_t>(32 * q) << 16);
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(d[i][0]), "=r"(d[i][1]), "=r"(d[i][2]), "=r"(d[i][3]), "=r"(d[i][4]), "=r"(d[i][5]), "=r"(d[i][6]),
                       "=r"(d[i][7])
                     : "r"(ta));
      }
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      const int half = lane >> 4, l = lane & 15;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int j = 2 * i + half;  // fragment = MMA index of the direct kernel: columns 16 g' + 2 j (+ 1)
        const int c = wn * 128 + (l < 8 ? 16 * l + 2 * j : 16 * (l - 8) + 2 * j + 1);
#pragma unroll
        for (int m = 0; m < kMaxRows; ++m)
          if (m < M) red[m * TNc + RedCol(c, m)] = __uint_as_float(d[i][m]);
      }
    } else {
      for (int m = 0; m < M; ++m)
        for (int c = lane; c < 128; c += 32) red[(wk * M + m) * TNc + wn * 128 + c] = 0.f;
    }
  } else if (is_legacy) {
    if (warp_has_cols) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int cl = wn * 128 + g * 16 + 2 * j;
        const int m0 = 2 * t, m1 = 2 * t + 1;
        if (m0 < M) *reinterpret_cast<float2*>(&red[(wk * M + m0) * TNc + RedCol(cl, m0)]) = make_float2(acc[j][0], acc[j][2]);
        if (m1 < M) *reinterpret_cast<float2*>(&red[(wk * M + m1) * TNc + RedCol(cl, m1)]) = make_float2(acc[j][1], acc[j][3]);
      }
    } else {
      for (int m = 0; m < M; ++m)
        for (int c = lane; c < 128; c += 32) red[(wk * M + m) * TNc + wn * 128 + c] = 0.f;
    }
  }
  TcFenceBefore();
  __syncthreads();
  if (is_issuer) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(alloc_cols) : "memory");
  }
  if (p.fuse) {
    EpilogueTail<kNvfp4, true>(p, tl, smem, sh, p.wk, TNc);
  } else {
    EpilogueTail<kNvfp4>(p, tl, smem, sh, p.wk, TNc);
  }
  Stamp(p, 5);
}

// ------------------------------------------------------------------------------ ring kernel
template <int MODE>
__global__ void __launch_bounds__(kRingThreads, 2) SkinnyGemmRingKernel(const __grid_constant__ GemmParams p) {
  using G = Geom<MODE>;
  constexpr int NM = G::kMmas;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ SharedScratch sh;

  if (p.trigger == 1) GridLaunchDependents();

  const int tid = threadIdx.x;
  const int nthreads = blockDim.x;
  const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int wn = warp % p.wn, wk = warp / p.wn;
  const Tile tl = LocateTile(p);
  const Segment& sg = p.seg[tl.seg];
  const int N = sg.n, n0 = tl.n0, n1 = tl.n1, kbeg = tl.kbeg, kend = tl.kend, kslice = tl.kslice;
  const long long pitch = sg.pitch;
  const int R = 16 * p.wk * p.ks;
  const int nst = (kslice + R - 1) / R;

  const int TB = p.tile_row_bytes;
  const int SRB = p.scale_row_bytes;
  const uint32_t ring = SmemAddr(smem);
  const uint32_t swz_mask = static_cast<uint32_t>((TB / 16 - 1) & 6);

  // ---- producer geometry: weight bytes
  const int vec = sg.vec;
  const int ppr = TB / vec;
  const int lgp = CeilLog2(ppr);
  const int valid_row_bytes = (MODE == kBf16) ? (n1 - n0) * 2 : (MODE == kFp8) ? (n1 - n0) : (n1 - n0) / 2;
  const long long col_byte0 = (MODE == kBf16) ? static_cast<long long>(n0) * 2 : (MODE == kFp8) ? n0 : n0 / 2;
  const uint8_t* wbase = sg.w + col_byte0;
  // ---- producer geometry: NVFP4 scale bytes (an aligned superset of the tile's scale bytes)
  int svec = 4, sphase = 0, spps = 0, lgs = 0;
  long long srow_off = 0;
  if constexpr (MODE == kNvfp4) {
    svec = sg.svec;
    const long long soff = (N >> 1) + (n0 >> 4);
    srow_off = soff / svec * svec;
    sphase = static_cast<int>(soff - srow_off);
    spps = (sphase + ((n1 - n0) >> 4) + svec - 1) / svec;
    lgs = CeilLog2(spps);
  }

  auto issue_stage = [&](int stage) {
    const uint32_t slot = ring + static_cast<uint32_t>(stage % p.stages) * p.stage_bytes;
    const int row_base = kbeg + stage * R;
    {
      const int total = R << lgp;
      for (int i = tid; i < total; i += nthreads) {
        const int row = i >> lgp;
        const int c = i & ((1 << lgp) - 1);
        if (c >= ppr) continue;
        const int bo = c * vec;
        int bytes = min(vec, max(0, valid_row_bytes - bo));
        const int krow = row_base + row;
        if (krow >= kend) bytes = 0;
        const uint8_t* src = bytes > 0 ? wbase + static_cast<long long>(krow) * pitch + bo : sg.w;
        const uint32_t dst = slot + row * TB + ((((bo >> 4) ^ (((row >> 2) & 3) << 1 & swz_mask)) << 4) | (bo & 15));
        if (vec == 16) {
          CpAsync16(dst, src, bytes);
        } else if (vec == 8) {
          CpAsync8(dst, src, bytes);
        } else {
          CpAsync4(dst, src, bytes);
        }
      }
    }
    if constexpr (MODE == kNvfp4) {
      const uint32_t sslot = slot + R * TB;
      const int total = R << lgs;
      for (int i = tid; i < total; i += nthreads) {
        const int row = i >> lgs;
        const int c = i & ((1 << lgs) - 1);
        if (c >= spps) continue;
        const int krow = row_base + row;
        const long long pos = static_cast<long long>(krow) * pitch + srow_off + c * svec;
        int bytes = krow < kend ? static_cast<int>(min(static_cast<long long>(svec), sg.total_bytes - pos)) : 0;
        bytes = max(bytes, 0);
        const uint8_t* src = bytes > 0 ? sg.w + pos : sg.w;
        const uint32_t dst = sslot + row * SRB + c * svec;
        if (svec == 16) {
          CpAsync16(dst, src, bytes);
        } else if (svec == 8) {
          CpAsync8(dst, src, bytes);
        } else {
          CpAsync4(dst, src, bytes);
        }
      }
    }
  };

  // ---- prologue: fill the ring, then stage x while the first weights are in flight
  for (int st = 0; st < p.stages - 1; ++st) {
    if (st < nst) issue_stage(st);
    CpAsyncCommit();
  }
  if (p.pdl_wait) GridDependencyWait();

  uint16_t* xs = reinterpret_cast<uint16_t*>(smem + p.ring_bytes);
  const bool slow = p.fuse ? StageX<MODE, false, true, true>(p, tl, xs, sh) : StageX<MODE>(p, tl, xs, sh);

  float acc[NM][4];
#pragma unroll
  for (int j = 0; j < NM; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;

  const int cols_per_warp = 8 * G::kColsPerThread;
  const bool warp_has_cols = n0 + wn * cols_per_warp < n1;
  uint32_t w_off, s_off = 0;
  if constexpr (MODE == kNvfp4) {
    const uint32_t chunk = static_cast<uint32_t>(wn * 4 + (g >> 1));
    w_off = 4 * t * TB + (((chunk ^ ((t << 1) & swz_mask)) << 4) | ((g & 1) << 3));
    s_off = static_cast<uint32_t>(R * TB + 4 * t * SRB + sphase + wn * 8 + g);
  } else {
    const uint32_t chunk = static_cast<uint32_t>(wn * 8 + g);
    w_off = 4 * t * TB + ((chunk ^ ((t << 1) & swz_mask)) << 4);
  }
  const uint32_t xs_addr = SmemAddr(xs) + static_cast<uint32_t>((g * p.xpitch + 4 * t) * 2);
  const bool has_row = g < p.M;

  for (int it = 0; it < nst; ++it) {
    CpAsyncWait(p.stages - 2);
    __syncthreads();
    const int nxt = it + p.stages - 1;
    if (nxt < nst) issue_stage(nxt);
    CpAsyncCommit();
    if (warp_has_cols) {
      const uint32_t slot = ring + static_cast<uint32_t>(it % p.stages) * p.stage_bytes;
      for (int q = 0; q < p.ks; ++q) {
        const int step_in_stage = q * p.wk + wk;
        const int kstep = it * (p.wk * p.ks) + step_in_stage;
        if (kstep * 16 >= kslice) break;
        uint32_t b0 = 0, b1 = 0;
        if (has_row) {
          const uint2 xv = Lds64(xs_addr + static_cast<uint32_t>(kstep) * 32u);
          b0 = xv.x;
          b1 = xv.y;
        }
        const uint32_t wa = slot + static_cast<uint32_t>(step_in_stage * 16) * TB + w_off;
        Raw<MODE> raw;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if constexpr (MODE == kNvfp4) {
            raw.r[0][i] = Lds64(wa + static_cast<uint32_t>(i) * TB);
          } else {
            raw.r[i] = Lds128(wa + static_cast<uint32_t>(i) * TB);
          }
        }
        if constexpr (MODE == kNvfp4) {
          const uint32_t sa = slot + static_cast<uint32_t>(step_in_stage * 16) * SRB + s_off;
#pragma unroll
          for (int i = 0; i < 4; ++i) raw.s[0][i] = Lds8(sa + static_cast<uint32_t>(i) * SRB);
        }
        if constexpr (MODE == kBf16) {
          ComputeStep<MODE, false>(acc, raw, b0, b1);
        } else {
          if (slow) {
            ComputeStep<MODE, true>(acc, raw, b0, b1);
          } else {
            ComputeStep<MODE, false>(acc, raw, b0, b1);
          }
        }
      }
    }
  }
  CpAsyncWait(0);
  if (p.trigger == 2) GridLaunchDependents();
  __syncthreads();
  if (p.fuse) {
    Epilogue<MODE, 1, true>(p, tl, acc, smem, sh, warp_has_cols);
  } else {
    Epilogue<MODE>(p, tl, acc, smem, sh, warp_has_cols);
  }
}

// Largest dynamic shared-memory request any of the kernels accepts: the opt-in limit of the
// device minus the kernels' static shared memory.
int g_max_dynamic_smem = 0;

template <typename K>
cudaError_t ConfigureKernel(K kernel) {
  int dev = 0, optin = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  err = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (err != cudaSuccess) return err;
  cudaFuncAttributes fa;
  err = cudaFuncGetAttributes(&fa, kernel);
  if (err != cudaSuccess) return err;
  const int dyn = optin - static_cast<int>(fa.sharedSizeBytes);
  if (g_max_dynamic_smem == 0 || dyn < g_max_dynamic_smem) g_max_dynamic_smem = dyn;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn);
}

template <int MODE>
cudaError_t ConfigureDirect() {
  cudaError_t err = ConfigureKernel(SkinnyGemmDirectKernel<MODE, 2>);
  if (err == cudaSuccess) err = ConfigureKernel(SkinnyGemmDirectKernel<MODE, 3>);
  if (err == cudaSuccess) err = ConfigureKernel(SkinnyGemmDirectKernel<MODE, 4>);
  if (err == cudaSuccess) err = ConfigureKernel(SkinnyGemmDirectKernel<MODE, 2, true>);
  if (err == cudaSuccess) err = ConfigureKernel(SkinnyGemmDirectKernel<MODE, 3, true>);
  if (err == cudaSuccess) err = ConfigureKernel(SkinnyGemmDirectKernel<MODE, 4, true>);
  return err;
}

// the direct kernel is compiled for rings of 4, 6 and 8 k-steps (2, 3, 4 pairs)
template <int MODE>
cudaError_t LaunchDirect(const cudaLaunchConfig_t* cfg, int stages, const GemmParams& p) {
  if (p.fuse) {
    switch (stages) {
      case 4: return cudaLaunchKernelEx(cfg, SkinnyGemmDirectKernel<MODE, 2, true>, p);
      case 6: return cudaLaunchKernelEx(cfg, SkinnyGemmDirectKernel<MODE, 3, true>, p);
      case 8: return cudaLaunchKernelEx(cfg, SkinnyGemmDirectKernel<MODE, 4, true>, p);
      default: return cudaErrorInvalidValue;
    }
  }
  switch (stages) {
    case 4: return cudaLaunchKernelEx(cfg, SkinnyGemmDirectKernel<MODE, 2>, p);
    case 6: return cudaLaunchKernelEx(cfg, SkinnyGemmDirectKernel<MODE, 3>, p);
    case 8: return cudaLaunchKernelEx(cfg, SkinnyGemmDirectKernel<MODE, 4>, p);
    default: return cudaErrorInvalidValue;
  }
}

template <int MODE>
cudaError_t LaunchMode(const GemmParams& p, const Plan& plan, size_t smem, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(p.seg[p.nseg - 1].tile_begin + p.seg[p.nseg - 1].tiles),
                     static_cast<unsigned>(plan.cluster), 1);
  cfg.blockDim = dim3(static_cast<unsigned>(plan.threads()), 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n_attr = 0;
  if (plan.cluster > 1) {
    attr[n_attr].id = cudaLaunchAttributeClusterDimension;
    attr[n_attr].val.clusterDim.x = 1;
    attr[n_attr].val.clusterDim.y = static_cast<unsigned>(plan.cluster);
    attr[n_attr].val.clusterDim.z = 1;
    ++n_attr;
  }
  if (p.pdl_wait) {
    attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n_attr].val.programmaticStreamSerializationAllowed = 1;
    ++n_attr;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n_attr;
  if constexpr (MODE != kNvfp4) {
    if (plan.direct == 2) {
      return p.fuse ? cudaLaunchKernelEx(&cfg, SkinnyGemmRegKernel<MODE, true>, p) : cudaLaunchKernelEx(&cfg, SkinnyGemmRegKernel<MODE>, p);
    }
  }
  if (plan.direct) {
    if constexpr (MODE == kNvfp4) {
      if (plan.tc) {
        switch (plan.stages) {
          case 3: return cudaLaunchKernelEx(&cfg, SkinnyGemmTcKernel<3>, p);
          case 4: return cudaLaunchKernelEx(&cfg, SkinnyGemmTcKernel<4>, p);
          case 6: return cudaLaunchKernelEx(&cfg, SkinnyGemmTcKernel<6>, p);
          default: return cudaErrorInvalidValue;
        }
      }
    }
    return LaunchDirect<MODE>(&cfg, plan.stages, p);
  }
  return cudaLaunchKernelEx(&cfg, SkinnyGemmRingKernel<MODE>, p);
}

}  // namespace

int DeviceSmCount() {
  static int count = [] {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 148;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
    return n;
  }();
  return count;
}

// Co-resident clusters (CTAs for cluster == 1) of one launch shape on the current device; cached.
int QueryMaxActiveClusters(int mode, int direct, int threads, size_t smem, int cluster) {
  static std::mutex mu;
  static std::map<std::tuple<int, int, int, size_t, int>, int> cache;
  const size_t smem_key = (smem + 4095) & ~static_cast<size_t>(4095);
  const auto key = std::make_tuple(mode, direct, threads, smem_key, cluster);
  std::lock_guard<std::mutex> lock(mu);
  auto it = cache.find(key);
  if (it != cache.end()) return it->second;
  const void* fn = nullptr;
  switch (mode) {
    case kBf16:
      fn = direct == 4 ? (const void*)SkinnyGemmRegKernel<kBf16>
           : direct    ? (const void*)SkinnyGemmDirectKernel<kBf16, 2>
                       : (const void*)SkinnyGemmRingKernel<kBf16>;
      break;
    case kFp8:
      fn = direct == 4 ? (const void*)SkinnyGemmRegKernel<kFp8>
           : direct    ? (const void*)SkinnyGemmDirectKernel<kFp8, 2>
                       : (const void*)SkinnyGemmRingKernel<kFp8>;
      break;
    default:
      fn = direct == 3   ? (const void*)SkinnyGemmTcKernel<4>
           : direct >= 1 ? (const void*)SkinnyGemmDirectKernel<kNvfp4, 2>
                         : (const void*)SkinnyGemmRingKernel<kNvfp4>;
      break;
  }
  int result = 0;
  if (g_max_dynamic_smem > 0 && smem_key > static_cast<size_t>(g_max_dynamic_smem)) {
    result = 0;
  } else if (cluster <= 1) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem_key) == cudaSuccess) {
      result = per_sm * DeviceSmCount();
    }
  } else {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1, static_cast<unsigned>(cluster), 1);
    cfg.blockDim = dim3(static_cast<unsigned>(threads), 1, 1);
    cfg.dynamicSmemBytes = smem_key;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = static_cast<unsigned>(cluster);
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) == cudaSuccess) result = n;
  }
  cudaGetLastError();
  cache[key] = result;
  return result;
}

// Raises the dynamic shared-memory limit of the kernels once per process.  Called from the
// *_create entry points, i.e. outside any stream capture.
int g_configured_device = -1;

cudaError_t ConfigureSkinnyGemmKernels() {
  static std::once_flag once;
  static cudaError_t status = cudaSuccess;
  std::call_once(once, [] {
    status = cudaGetDevice(&g_configured_device);
    if (status == cudaSuccess) status = ConfigureDirect<kBf16>();
    if (status == cudaSuccess) status = ConfigureDirect<kFp8>();
    if (status == cudaSuccess) status = ConfigureDirect<kNvfp4>();
    if (status == cudaSuccess) status = ConfigureKernel(SkinnyGemmRegKernel<kBf16>);
    if (status == cudaSuccess) status = ConfigureKernel(SkinnyGemmRegKernel<kFp8>);
    if (status == cudaSuccess) status = ConfigureKernel(SkinnyGemmRegKernel<kBf16, true>);
    if (status == cudaSuccess) status = ConfigureKernel(SkinnyGemmRegKernel<kFp8, true>);
    if (status == cudaSuccess) status = ConfigureKernel(SkinnyGemmTcKernel<3>);
    if (status == cudaSuccess) status = ConfigureKernel(SkinnyGemmTcKernel<4>);
    if (status == cudaSuccess) status = ConfigureKernel(SkinnyGemmTcKernel<6>);
    if (status == cudaSuccess) status = ConfigureKernel(SkinnyGemmRingKernel<kBf16>);
    if (status == cudaSuccess) status = ConfigureKernel(SkinnyGemmRingKernel<kFp8>);
    if (status == cudaSuccess) status = ConfigureKernel(SkinnyGemmRingKernel<kNvfp4>);
    // without the kernel of skinny_stream.cu every call is these kernels'
    if (status == cudaSuccess && ConfigureStreamKernels() != cudaSuccess) cudaGetLastError();
  });
  return status;
}

// The kernels' attributes (shared-memory limits, co-resident cluster counts, SM count) were set up for one
// device: one process drives one GPU, and a call with another device current is refused rather than launched
// with the wrong limits.
cudaError_t CheckConfiguredDevice() {
  int dev = -1;
  if (g_configured_device >= 0 && (cudaGetDevice(&dev) != cudaSuccess || dev != g_configured_device)) return cudaErrorInvalidDevice;
  return cudaSuccess;
}

cudaError_t LaunchSkinnyGemm(int mode, GemmParams& p, const Plan& plan, cudaStream_t stream) {
  const cudaError_t device = CheckConfiguredDevice();
  if (device != cudaSuccess) return device;
  const ModeGeom geom = GeomOf(mode, plan.direct ? plan.wide : 1);
  p.wn = plan.wn;
  p.wk = plan.wk;
  p.ks = plan.ks;
  p.stages = plan.stages;
  p.cluster = plan.cluster;
  p.gran = plan.gran;
  p.tile_row_bytes = plan.wn * geom.bytes_per_warp;
  p.scale_row_bytes = mode == kNvfp4 ? (plan.wn * 8 + 16 + 15) & ~15 : 0;
  const int R = plan.rows_per_stage();
  p.stage_bytes = (R * (p.tile_row_bytes + p.scale_row_bytes) + 127) & ~127;
  const int TNc = PlanMaxCols(plan, mode);
  const int red_bytes = (plan.wk + (plan.cluster > 1 ? 1 : 0)) * p.M * TNc * 4;
  const int direct_slot = plan.tc ? DirectSlotBytes(mode, 1) : RingSlotBytes(mode);
  const int ring_warps = plan.tc ? plan.wn * plan.wk + plan.wk : plan.wn * plan.wk;
  const int ring = plan.direct == 2 ? 0 : plan.direct ? ring_warps * plan.stages * direct_slot : plan.stages * p.stage_bytes;
  p.ring_bytes = (std::max(ring, red_bytes) + 127) & ~127;
  const int ksteps = (p.K + 15) / 16;
  const int kslice_max = ((ksteps + plan.cluster - 1) / plan.cluster) * 16;
  p.xpitch = ((kslice_max + 63) & ~63) + 16;  // 32 bytes off a 128-byte multiple: rows land in distinct banks
  size_t smem = static_cast<size_t>(p.ring_bytes) + static_cast<size_t>(p.M) * p.xpitch * 2;
  if (plan.tc) {
    // x as the MMA operand: 256 bytes per k-step plus one spare step; at least 120 KB so that two CTAs,
    // each allocating up to all of tensor memory, can never share an SM
    smem = static_cast<size_t>(p.ring_bytes) + static_cast<size_t>(kslice_max / 16 + 1) * 256;
    if (smem < 120 * 1024) smem = 120 * 1024;
  }
  if (g_max_dynamic_smem > 0 && smem > static_cast<size_t>(g_max_dynamic_smem)) return cudaErrorInvalidConfiguration;
  p.scales_l1 = smem <= kL1UsableSmem ? 1 : 0;
  p.tail_groups = plan.tail;
  // K slices per shared group: at most kMaxTailSplit, one per CTA where there are enough CTAs, else one per idle warp
  p.tail_split = 1;
  p.tail_stride = 0;
  if (plan.tail > 0) {
    const int ctas = plan.tiles[0];
    if (ctas >= 2 * plan.tail) {
      p.tail_split = std::min(kMaxTailSplit, ctas / plan.tail);
      p.tail_stride = ctas / (plan.tail * p.tail_split);
    } else {
      p.tail_split = std::max(1, std::min(kMaxTailSplit, ctas * plan.wk / plan.tail));
    }
  }
  if (plan.tail > 0 && (!p.lm || p.lm_tail == nullptr || p.nseg != 1 || plan.cluster != 1)) return cudaErrorInvalidValue;
  int tiles = 0;
  for (int s = 0; s < p.nseg; ++s) {
    p.seg[s].tile_begin = tiles;
    p.seg[s].tiles = plan.tiles[s];
    p.seg[s].tail_cols = (s == 0) ? plan.tail * 128 : 0;
    p.seg[s].granules = (p.seg[s].n - p.seg[s].tail_cols + plan.gran - 1) / plan.gran;
    if (plan.tiles[s] < 1 || plan.tiles[s] > 65535) return cudaErrorInvalidValue;
    p.seg[s].gran_quot = p.seg[s].granules / plan.tiles[s];
    p.seg[s].gran_rem = p.seg[s].granules % plan.tiles[s];
    tiles += plan.tiles[s];
  }
  switch (mode) {
    case kBf16: return LaunchMode<kBf16>(p, plan, smem, stream);
    case kFp8: return LaunchMode<kFp8>(p, plan, smem, stream);
    case kNvfp4: return LaunchMode<kNvfp4>(p, plan, smem, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace qfg
