// Depthwise 5x5 (pad 2, stride 1) + bias + activation on bf16 NHWC, with three epilogues: bf16, dynamic MXFP8,
// static INT8. Operands and roundings follow FlashIM's torch reference (flashim/ops/conv.py:30-61): bf16 inputs and
// weights, exact products summed in fp32, bias added last in fp32.
//
// The sums run on the tensor cores (mma.sync m16n8k16, bf16 in, fp32 accumulators), one channel at a time:
//   M: 16 blocks of 2 rows x 4 columns of output pixels, N: the 8 pixels of a block, K: the 6 x 8 input patch of a block
//   (48 values, 3 K steps of two rows); B is the 5x5 kernel shifted to each of the 8 pixels (25 of its 48 rows non-zero).
// On the fp32 pipe the 25 multiply-adds per element alone take longer than the tensor's way through HBM. As MMAs they are
// a few percent of the tensor pipe; what the layout is chosen for is shared-memory bandwidth, the next bound:
//   - A warp sweeps down its strip, 32 columns wide, 4 output rows per step. M is 8 blocks side by side x 2 blocks one below the
//     other, so the two row pairs of the patch that a step shares with the step before, and the three that the two block
//     rows share, stay in registers: a step loads four input rows for four output rows, each value once per column block
//     that needs it (two), 16 bytes (8 channels) per lane and pixel.
//   - K is ordered (row, column pair) with patch columns q and q + 4 in one register: lane l reads pixels l and l + 4 of a
//     row, so the lanes of a shared-memory phase read neighbours, which the 64-byte TMA swizzle keeps free of conflicts.
//   - N is ordered (column, row): a lane ends up with four pixels of one column, column l of the tile, for 8 channels.
//   - A warp keeps to 8 channels, whose B fragments (48 registers) stay resident; four warps (a quad) cover the 32 channels
//     of an MX block, exchange block maxima through shared memory and fill one output panel for a TMA store. Storing 8
//     or 16 bytes per pixel from registers instead costs a shared-memory wavefront per lane.
//
// Measured against the fp32-pipe kernel before it (B200, inputs in L2 where they fit):
//   4x200x200x256: GELU -> bf16 68 -> 52 us, ReLU -> bf16 54 -> 42, GELU -> MXFP8 88 -> 85, ReLU -> INT8 87 -> 51
//   8x400x400x128: GELU -> bf16 232 -> 160, ReLU -> bf16 183 -> 127 (80 % of the HBM copy rate), GELU -> MXFP8 303 -> 281,
//   ReLU -> MXFP8 252 -> 198, ReLU -> INT8 299 -> 165
// What bounds the GELU and quantising forms now is what the schedulers can dispatch: packed FMAs, permutes, integer and conversion
// instructions take two cycles each and the MMAs of twelve warps 11.4, one after the other (MXFP8: about 90 % of the 1900 cycles per warp and
// step; bf16 GELU: 72 % of 1240). Sixteen warps with one set of B fragments per CTA were slower (bf16 GELU 57 -> 61 us). The same bytes as the chain (below) cost the MXFP8 form up to a quarter of its time: 225 and 178 us with a test that
// missed half of the codes that differ. Where the arguments of the GELU reach far into its left tail (a standard deviation of 1.5 and
// up) it takes 360 us, more than the fp32-pipe kernel.
//
// Precision: the tensor cores add the exact products into fp32 accumulators, as the fp32 chain of the reference does (ky-major FMA
// chain, bias last), but in another order; the two differ by up to about two fp32 ulp of the largest partial sum.
//   MXFP8: the bytes of the chain. Every value has two bounds, itself less and plus the largest difference (error_of); where their
//     codes differ (with normal data one in 1300) the output is summed again in the chain's order, at once and from shared memory.
//     Where the exponents of the two bounds of a block's maximum differ, the block is noted in a list of the quad. No code or scale
//     differed in 4 G of normal, wide, sparse, smooth, edge-filtered and heavy-tailed data.
//   bf16: outputs below 2**-14 of the sums in their column, where bias and products cancel, are noted (one in 30000). Others may
//     lie one ulp of bf16 from the chain's where its sum lies next to a rounding boundary: one in 200000 of normal data, up to one in
//     25000 where sums cancel.
//   INT8: likewise a code may lie one from the chain's: one in 4000000, up to one in 400000.
// The outputs and blocks of a list are summed again in the chain's order at the end of the quad's range or when the list fills up; a
// step with more of them, or with more open codes, than is worth doing one by one is summed again as a whole. The bits of all
// outputs thus depend on their own step alone, not on how the work is cut.
//
// A patch value outside an output's 5x5 window is multiplied by a zero of B, which an infinity or a not-a-number survives. A
// step that meets a sum which is not finite is therefore done again in the reference's order.
//
// Work: a strip is one (image, 32-column tile) over all rows, cut into steps of four output rows; a span is the part of a
// range of steps inside one strip. The quads of all CTAs (three per CTA, one CTA per SM) form groups of one quad per
// 32-channel tile, side by side on the SMs; the groups split the sequence of all steps evenly. The quads of a group thus read
// the 64-byte parts of the same lines at about the same time, so DRAM delivers every line once (channel tile by channel
// tile, 8x400x400x128 read twice its bytes: ReLU -> bf16 201 instead of 132 us), and a quad builds its B fragments once.
// Each quad has a ring of input chunks of its own: 4 rows x 36 columns x 32 channels, zero-filled outside the image by TMA.
// One named barrier per step orders all of it: behind it the step's chunk has been read by all four warps (and is
// refilled), their maxima are visible, and the output panel is complete.
#include <type_traits>

#include "common.cuh"
#include "flashim_sm100.h"
#include "flashim_sm100_tune.h"

namespace fim {
namespace {

constexpr int kTileX = 32, kStepRows = 4, kTileC = 32, kQuads = 3;
constexpr int kHaloX = kTileX + 4;
constexpr uint32_t kPixelBytes = kTileC * 2, kRowBytes = kHaloX * kPixelBytes, kChunkBytes = kStepRows * kRowBytes;
constexpr int kTaps = 25, kMaxStages = 6;
constexpr float kCancelled = 16384.0f;  // an output below 1 / kCancelled of the sums it comes from is summed again (bf16)
// MXFP8: how far a tensor-core sum may lie from the fp32 chain, as a share of the size that error_of forms: 2**-20.1. The largest
// difference in three times 46 M outputs of each of 88 kinds of data (normal, ReLU'd, positive, uniform, log-normal, smooth and flat
// images under random, positive, zero-sum, edge, Gaussian and log-normal taps) was 2**-20.6 of it, for edge filters on a smooth
// image; it is 2**-21.2 of the largest partial sum at most, and where sums cancel that is at most twice the size.
constexpr float kSumError = 8.9e-7f;
// The GELU passes on less than kGeluSlope of an argument's error (|GELU'| <= 1.129), and less than kGeluBase + kGeluGrowth * GELU
// (|GELU'| <= 0.5 + 1.6 GELU for every argument); both with a tenth for the rounding of the polynomial.
constexpr float kGeluSlope = 1.25f, kGeluBase = 0.55f, kGeluGrowth = 1.76f;
constexpr float kGeluUnderflow = 12.743085f;  // minus the argument at which 2**q of gelu_phi2 falls below 2**-126
// open codes that a warp corrects two by two (about 500 cycles); with more of them the quad does the step again (20000)
constexpr int kMostOpen = 32;
// The list of a quad: a header (count; flush and redo tags by step parity; MXFP8: error bounds of the four warps by step parity,
// the sizes of their taps and biases), then one word per entry: step of the range (20 bits) | row (2) | column (5) | channel (5; MXFP8:
// 0, for a block).
constexpr uint32_t kListHeader = 96, kListTags = 16, kListErrors = 32, kListSizes = 64, kFlushAt = 32;
// bf16: outputs that a lane notes in a step; with more of them the quad does the step again. A list below kFlushAt takes those of two
// steps, so which steps are done again is a matter of their own data alone, and so are the bits of the other outputs in them.
constexpr int kMostNoted = 2;
constexpr long long kMaxRange = 1 << 20;  // steps of a range that an entry can name
constexpr uint32_t kWeightBytes = kTaps * kTileC * 2, kBiasBytes = kTileC * 8;

enum { kOutBf16 = 0, kOutMx = 1, kOutInt8 = 2 };

__host__ __device__ constexpr uint32_t list_bytes(int mode) { return mode == kOutBf16 ? 3072u : 1024u; }
__host__ __device__ constexpr uint32_t list_entries(int mode) { return (list_bytes(mode) - kListHeader) / 4; }
static_assert(kFlushAt + 2 * 128 * kMostNoted <= list_entries(kOutBf16), "the notes of the step that fills the list, and of the next");

// shared memory of one quad: ring, two output panels (128 pixels x 32 channels), block maxima of two steps, list, B fragments,
// weights, bias. The MXFP8 form holds its values across a barrier and has no registers left for the B fragments (48): it reads
// them from shared memory, whose bandwidth it does not use up, at the price of a shorter ring. (Spilled to local memory, which
// the shared memory leaves hardly any L1 for, they cost a third of the kernel's time.)
__host__ __device__ constexpr uint32_t panel_bytes(int mode) { return mode == kOutBf16 ? 8192u : 4096u; }
__host__ __device__ constexpr uint32_t exchange_bytes(int mode) { return mode == kOutMx ? 4096u : 0u; }
__host__ __device__ constexpr bool shared_fragments(int mode) { return mode == kOutMx; }
// chunks of the ring that are kept after their products: MXFP8 corrects codes from the two of the step (it has two on the way then)
__host__ __device__ constexpr uint32_t kept_chunks(int mode) { return mode == kOutMx ? 2u : 0u; }
__host__ __device__ constexpr int stages(int mode) { return shared_fragments(mode) ? 4 : kMaxStages; }
__host__ __device__ constexpr uint32_t fragment_bytes(int mode) { return shared_fragments(mode) ? 4u * 12u * 512u : 0u; }
__host__ __device__ constexpr uint32_t quad_bytes(int mode) {
  return (stages(mode) * kChunkBytes + fragment_bytes(mode) + 2 * panel_bytes(mode) + exchange_bytes(mode) + list_bytes(mode) + kWeightBytes + kBiasBytes + 1023u) / 1024u * 1024u;
}

struct DwParams {
  const uint16_t* value;   // bf16 NHWC
  const uint32_t* weight;  // bf16x2 words, [25][C/2]
  const float* bias;
  uint8_t* out;
  uint8_t* scales;
  const float* scale;  // INT8
  int batch, height, width, channels;
  int tiles_x, channel_tiles;
  int strip_steps, total_steps;  // four-row steps per strip; all steps of one channel tile
  int groups, group_quads;       // quads of a group: min(channel tiles, quads of the grid), each takes every group_quads-th tile
  int cta_quads;                 // quads in use per CTA
  int swizzled;                  // 0: plain scales; else 1 + the padding groups behind the last one of a row
  int tma_out;                   // tma_out: the output can be the target of TMA stores (16-byte aligned)
  int* status;
};

// GELU(x) = x * Phi(x) on a pair of fp32 values, one packed FMA per Horner step of both. With p = Phi(-|x|) =
// 2**q(-|x|), q the degree-7 minimax polynomial of log2 Phi on [-5.5, 0] (relative error of p below 4e-6; q keeps falling
// beyond -5.5, so p underflows to 0 for large |x|), the value is max(x, 0) - |x| p for either sign. One MUFU per value. For
// x < -4.4 torch's own fp32 expression x * 0.5 * (1 + erf(x / sqrt 2)) is dominated by the rounding of 1 + erf; this form
// stays accurate there.
__device__ __forceinline__ uint64_t gelu_phi2(uint64_t x2) {
  float x0, x1;
  unpack2(x2, x0, x1);
  const uint64_t u = pack2(-fabsf(x0), -fabsf(x1));
  uint64_t q = pack2(1.793454771359393e-06f, 1.793454771359393e-06f);
  q = fma2(q, u, pack2(6.090417082305066e-05f, 6.090417082305066e-05f));
  q = fma2(q, u, pack2(0.000926029053516686f, 0.000926029053516686f));
  q = fma2(q, u, pack2(0.00849375780671835f, 0.00849375780671835f));
  q = fma2(q, u, pack2(0.053937844932079315f, 0.053937844932079315f));
  q = fma2(q, u, pack2(-0.45848050713539124f, -0.45848050713539124f));
  q = fma2(q, u, pack2(1.1512467861175537f, 1.1512467861175537f));
  q = fma2(q, u, pack2(-0.9999954700469971f, -0.9999954700469971f));
  float q0, q1;
  unpack2(q, q0, q1);
  return fma2(u, pack2(ex2_approx(q0), ex2_approx(q1)), pack2(fmaxf(x0, 0.0f), fmaxf(x1, 0.0f)));
}

template <int ACT>
__device__ __forceinline__ uint64_t activate2(uint64_t v) {
  if (ACT == kActNone) return v;
  if (ACT == kActGelu) return gelu_phi2(v);
  float lo, hi;
  unpack2(v, lo, hi);
  return pack2(fmaxf(lo, 0.0f), fmaxf(hi, 0.0f));
}

__device__ __forceinline__ void lds128(uint32_t addr, uint32_t (&v)[4]) {
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(addr));
}

// d += a b, or d = a b for the first K step
template <bool FIRST>
__device__ __forceinline__ void mma_16x8x16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if (FIRST) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
  } else {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
}

// max(|m|, |a|, |b|)
__device__ __forceinline__ float max_abs(float m, float a, float b) {
  float r;
  asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(m), "f"(a), "f"(b));
  return r;
}

// Two image rows of the patch for 8 channels, as A operands: [channel][row], patch columns q and q + 4 in one register.
// `at`: the lane's pixel in the upper row, its 16-byte piece chosen by the swizzle; in the odd row and four columns on, the
// swizzle phase differs in one bit.
struct RowPair {
  uint32_t a[8][2];
};
__device__ __forceinline__ void load_pair(uint32_t at, RowPair& p) {
  uint32_t v[4][4];
  lds128(at, v[0]);
  lds128((at ^ 32u) + 4 * kPixelBytes, v[1]);
  lds128((at ^ 32u) + kRowBytes, v[2]);
  lds128(at + kRowBytes + 4 * kPixelBytes, v[3]);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    p.a[2 * j][0] = __byte_perm(v[0][j], v[1][j], 0x5410);
    p.a[2 * j + 1][0] = __byte_perm(v[0][j], v[1][j], 0x7632);
    p.a[2 * j][1] = __byte_perm(v[2][j], v[3][j], 0x5410);
    p.a[2 * j + 1][1] = __byte_perm(v[2][j], v[3][j], 0x7632);
  }
}

// The largest magnitude of columns q + 4 in two row pairs, or `big`. As fp32 numbers the words are the values of their upper halves (and
// up to 2**-7 of them more), three to an instruction; packed bf16 maxima take five times as long.
__device__ __forceinline__ float size_of(const RowPair& p, const RowPair& q, float big) {
  float other = 0.0f;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    asm volatile("max.abs.f32 %0, %0, %1, %2;" : "+f"(big) : "f"(__uint_as_float(p.a[c][0])), "f"(__uint_as_float(p.a[c][1])));
    asm volatile("max.abs.f32 %0, %0, %1, %2;" : "+f"(other) : "f"(__uint_as_float(q.a[c][0])), "f"(__uint_as_float(q.a[c][1])));
  }
  return fmaxf(big, other);
}

// One K step for the 8 channels: the upper blocks (M rows 0-7) see row pair `upper` of the patch, the blocks below them the
// next pair.
template <bool FIRST>
__device__ __forceinline__ void multiply_step_shared(const RowPair& upper, const RowPair& lower, uint32_t fragments, float (&acc)[8][4]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint32_t b[4];
    lds128(fragments + j * 512, b);
    mma_16x8x16<FIRST>(acc[2 * j], upper.a[2 * j][0], lower.a[2 * j][0], upper.a[2 * j][1], lower.a[2 * j][1], b[0], b[1]);
    mma_16x8x16<FIRST>(acc[2 * j + 1], upper.a[2 * j + 1][0], lower.a[2 * j + 1][0], upper.a[2 * j + 1][1], lower.a[2 * j + 1][1], b[2], b[3]);
  }
}
template <bool FIRST>
__device__ __forceinline__ void multiply_step(const RowPair& upper, const RowPair& lower, const uint32_t (&b)[8][2], float (&acc)[8][4]) {
#pragma unroll
  for (int c = 0; c < 8; ++c) mma_16x8x16<FIRST>(acc[c], upper.a[c][0], lower.a[c][0], upper.a[c][1], lower.a[c][1], b[c][0], b[c][1]);
}

// The pre-activation value of one output as the reference sums it: an fp32 FMA chain over the taps, ky-major, bias last.
// `image`: the channel's first pixel, `weights`: the shared-memory address of its first tap. Five loads are in flight at a
// time; unrolling all 25 is slower, since the code runs once and is fetched as it runs.
__device__ __forceinline__ float chain_sum(const uint16_t* image, int height, int width, int channels, uint32_t weights, float bias, int y, int x) {
  float sum = 0.0f;
#pragma unroll 1
  for (int ky = 0; ky < 5; ++ky) {
    const int iy = y + ky - 2;
    const bool row_in = static_cast<unsigned>(iy) < static_cast<unsigned>(height);
    const uint16_t* row = image + static_cast<ptrdiff_t>(row_in ? iy : y) * width * channels;
    uint16_t v[5];
#pragma unroll
    for (int kx = 0; kx < 5; ++kx) {
      const int ix = x + kx - 2;
      const bool in = row_in && static_cast<unsigned>(ix) < static_cast<unsigned>(width);
      v[kx] = __ldg(row + static_cast<ptrdiff_t>(in ? ix : x) * channels);
      v[kx] = in ? v[kx] : static_cast<uint16_t>(0);
    }
#pragma unroll
    for (int kx = 0; kx < 5; ++kx) {
      uint16_t w;
      asm volatile("ld.shared.u16 %0, [%1];" : "=h"(w) : "r"(weights + (ky * 5 + kx) * (kTileC * 2)));
      sum = fmaf(bf16_lo(v[kx]), bf16_lo(w), sum);
    }
  }
  return sum + bias;
}

// The same for four neighbouring columns x .. x + 3 (those outside the image are of no use), eight loads in flight.
__device__ __forceinline__ float4 chain_sum4(const uint16_t* image, int height, int width, int channels, uint32_t weights, float bias, int y, int x) {
  float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 1
  for (int ky = 0; ky < 5; ++ky) {
    const int iy = y + ky - 2;
    const bool row_in = static_cast<unsigned>(iy) < static_cast<unsigned>(height);
    const uint16_t* row = image + static_cast<ptrdiff_t>(row_in ? iy : y) * width * channels;
    uint16_t v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int ix = x + j - 2;
      const bool in = row_in && static_cast<unsigned>(ix) < static_cast<unsigned>(width);
      v[j] = __ldg(row + static_cast<ptrdiff_t>(in ? ix : x) * channels);
      v[j] = in ? v[j] : static_cast<uint16_t>(0);
    }
#pragma unroll
    for (int kx = 0; kx < 5; ++kx) {
      uint16_t w;
      asm volatile("ld.shared.u16 %0, [%1];" : "=h"(w) : "r"(weights + (ky * 5 + kx) * (kTileC * 2)));
#pragma unroll
      for (int j = 0; j < 4; ++j) sum[j] = fmaf(bf16_lo(v[j + kx]), bf16_lo(w), sum[j]);
    }
  }
  return make_float4(sum[0] + bias, sum[1] + bias, sum[2] + bias, sum[3] + bias);
}

// Marks of a step in its tags (one pair for even and one for odd steps): flush - the quad empties the list one step later, redo - it
// does the whole step again then. `at`: the step's pair; `mark`: not 0, the value the readers look for.
__device__ __forceinline__ void tag_flush(uint32_t at, uint32_t mark) {
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(at), "r"(mark) : "memory");
}
__device__ __forceinline__ void tag_redo(uint32_t at, uint32_t mark) {
  asm volatile("st.shared.v2.b32 [%0], {%1, %1};" ::"r"(at), "r"(mark) : "memory");
}

// Notes an output (or the block it lies in) in the quad's list. A step whose entries do not fit is done again as a whole (MXFP8).
template <int MODE>
__device__ __forceinline__ void note(uint32_t list, uint32_t tags, uint32_t mark, uint32_t entry) {
  uint32_t at;
  asm volatile("atom.shared.add.u32 %0, [%1], 1;" : "=r"(at) : "r"(list) : "memory");
  if (at < list_entries(MODE)) {
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(list + kListHeader + at * 4), "r"(entry) : "memory");
    if (at >= kFlushAt) tag_flush(tags, mark);
  } else {
    tag_redo(tags, mark);
  }
}

// max(|a|, |b|, |c|), not a number if one of them is
__device__ __forceinline__ float max_abs_nan(float a, float b, float c) {
  float r;
  asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
// min(|a|, |b|, |c|)
__device__ __forceinline__ float min_abs(float a, float b, float c) {
  float r;
  asm("min.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float max3(float m, float a, float b) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(m), "f"(a), "f"(b));
  return r;
}
// the largest of numbers that are not negative (or a not-a-number), over the warp
__device__ __forceinline__ float warp_max(float v) { return __uint_as_float(redux_max(__float_as_uint(v), 0xffffffffu)); }

// four E4M3 codes, of max(value, 0) for a ReLU
template <int ACT>
__device__ __forceinline__ uint32_t codes_of(float a, float b, float c, float d) {
  if (ACT != kActRelu) return e4m3x4(a, b, c, d);
  uint16_t lo, hi;
  asm("cvt.rn.satfinite.relu.e4m3x2.f32 %0, %1, %2;" : "=h"(lo) : "f"(b), "f"(a));
  asm("cvt.rn.satfinite.relu.e4m3x2.f32 %0, %1, %2;" : "=h"(hi) : "f"(d), "f"(c));
  return static_cast<uint32_t>(lo) | (static_cast<uint32_t>(hi) << 16);
}

// Bound on the difference between a sum of the tensor cores plus bias and the same of the fp32 chain. Both err by ulps of
// their partial sums. `size` is the largest |sum| of the warp or, if that is larger, its largest |value| times twice the largest |tap| or
// a quarter of the sum of a channel's |taps|: where all sums cancel (flat areas under taps that sum to zero) only the second bounds the
// partial sums. The bias adds a rounding to an ulp of the result. Sums of zeros are equal. Near the subnormals ulps no longer shrink with the sums: nothing is
// assumed there.
__device__ __forceinline__ float error_of(float size, float bias) {
  const float total = fmaxf(size, bias);
  return size == 0.0f ? 0.0f : total < 1e-30f ? total : total * kSumError;
}

// E8M0 bytes and the factors 2**-e of four block maxima that are known to within `error`: e = E - 8 + (mantissa > 1.75), one
// carry away from the exponent field, unless one of them lies in the window above 1.75 where the reference's rule departs from
// that, is not finite, or the exponents of its two bounds differ. Returns a bit per maximum whose exponent is open.
__device__ __forceinline__ uint32_t block_scales(const float (&amax)[4], float error, uint32_t (&bytes)[4], float (&inv)[4]) {
  uint32_t unsure = 0;
  bool rare = false;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t low = __float_as_uint(fmaxf(amax[i] - error, 0.0f)), high = __float_as_uint(fmaxf(amax[i] + error, 0.0f));
    const uint32_t byte = (high + 0x1FFFFFu) >> 23;
    bytes[i] = static_cast<uint32_t>(max(static_cast<int>(byte) - 8, 0));
    inv[i] = __uint_as_float((254u - bytes[i]) << 23);
    rare |= ((low + 0x1FFFFFu) >> 23) != byte || ((low & 0x7FFFFFu) - 0x600001u) < 41u || high >= 0x7F800000u;
  }
  if (rare) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int e = e8m0_exponent(fmaxf(amax[i] + error, 0.0f));
      if (e8m0_exponent(fmaxf(amax[i] - error, 0.0f)) != e) unsure |= 1u << i;
      bytes[i] = static_cast<uint32_t>(e + 127);
      inv[i] = exp2_int(-e);
    }
  }
  return unsure;
}

// Where the steps of a quad start in the image.
struct Position {
  int k0, tx, b;
};
__device__ __forceinline__ Position position_of(const DwParams& p, int step) {
  Position at;
  int t = step / p.strip_steps;
  at.k0 = step - t * p.strip_steps;
  at.tx = t % p.tiles_x;
  at.b = t / p.tiles_x;
  return at;
}

template <int MODE, int ACT>
__global__ void __launch_bounds__(128 * kQuads, 1)
dw5x5_kernel(const __grid_constant__ CUtensorMap in_map, const __grid_constant__ CUtensorMap out_map, const DwParams p) {
  extern __shared__ uint8_t smem_raw[];
  constexpr int kStages = stages(MODE);
  __shared__ __align__(8) uint64_t full_bar[kQuads * kStages];
  __shared__ int abort_flag;

  // (the warp index through a shuffle: uniform to the compiler, and so is everything derived from it)
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int quad = warp >> 2, piece = warp & 3;  // piece: which 8 of the 32 channels
  const uint32_t ring = ((smem_u32(smem_raw) + 1023u) & ~1023u) + quad * quad_bytes(MODE);
  const uint32_t panels = ring + kStages * kChunkBytes, exchange = panels + 2 * panel_bytes(MODE);
  const uint32_t list = exchange + exchange_bytes(MODE), fragments = list + list_bytes(MODE) + piece * (12 * 512) + lane * 16;
  const uint32_t weights_at = list + list_bytes(MODE) + fragment_bytes(MODE), bias_at = weights_at + kWeightBytes;
  const uint32_t full0 = smem_u32(&full_bar[quad * kStages]);

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < kQuads * kStages; ++s) mbar_init(&full_bar[s], 1);
    mbar_fence_init();
    fence_async_proxy();
    tma_prefetch_desc(&in_map);
    tma_prefetch_desc(&out_map);
  }
  grid_release();
  grid_wait();
  __syncthreads();

  const int worker = blockIdx.x * p.cta_quads + quad, group = worker / p.group_quads, member = worker % p.group_quads;
  if (MODE == kOutMx && p.swizzled && blockIdx.x == gridDim.x - 1) {
    // the padding rows of the last scale tiles (the swizzled layout is zero there, and the caller's buffer need not be)
    const uint32_t rows = static_cast<uint32_t>(p.batch) * p.height * p.width, tiles = ((p.channels >> 5) + 3) / 4;
    const uint32_t pad_rows = (128u - rows % 128u) % 128u;
    for (uint32_t i = threadIdx.x; i < pad_rows * tiles; i += 128 * kQuads) {
      const uint32_t row = rows + i / tiles;
      uint8_t* to = p.scales + (static_cast<uint64_t>(row >> 7) * tiles + i % tiles) * 512 + (row & 31) * 16 + ((row & 127) >> 5) * 4;
      to[0] = to[1] = to[2] = to[3] = 0;
    }
  }
  const bool idle = quad >= p.cta_quads || group >= p.groups;
  const int s_begin = idle ? 0 : static_cast<int>(static_cast<long long>(group) * p.total_steps / p.groups);
  const int s_end = idle ? 0 : static_cast<int>(static_cast<long long>(group + 1) * p.total_steps / p.groups);
  const uint32_t quad_barrier = 1 + quad;

  // ---- copies: issued by one lane of the quad's first warp ----
  int copy_ct = member, copy_step = s_begin, copy_g = 0, copy_len = -1;  // next span's start; chunk and length of the span under way
  Position copy_at = {};
  uint32_t issued = 0, issue_slot = 0;
  auto issue_until = [&](uint32_t target) {
    while (issued < target) {
      if (copy_g > copy_len) {
        if (copy_step >= s_end) {  // the range once more for the quad's next channel tile
          copy_ct += p.group_quads, copy_step = s_begin;
        }
        if (copy_ct >= p.channel_tiles || copy_step >= s_end) return;
        copy_at = position_of(p, copy_step);
        copy_len = min(p.strip_steps - copy_at.k0, s_end - copy_step);
        copy_step += copy_len;
        copy_g = 0;
      }
      if (elect_one()) {
        mbar_expect_tx_addr(full0 + 8 * issue_slot, kChunkBytes);
        tma_load_4d_addr(ring + issue_slot * kChunkBytes, &in_map, full0 + 8 * issue_slot, copy_ct * kTileC, copy_at.tx * kTileX - 2,
                         (copy_at.k0 + copy_g) * kStepRows - 2, copy_at.b);
      }
      ++copy_g;
      ++issued;
      if (++issue_slot == kStages) issue_slot = 0;
    }
  };
  if (piece == 0) issue_until(kStages);

  const Int8Quantizer int8 = make_int8_quantizer(MODE == kOutInt8 ? __ldg(p.scale) : 1.0f);
  constexpr int kOutBytes = MODE == kOutBf16 ? 2 : 1;
  const uint32_t turn = static_cast<uint32_t>(piece ^ ((lane >> 1) & 3)) << 4;  // the 16-byte piece under the swizzle
  const uint32_t lane_at = ring + lane * kPixelBytes + turn;
  // from there to the lane's share of columns 0 - 3 of a chunk: row lane / 8, column lane / 2 % 4, four channels
  const uint32_t first_pixel = (lane >> 3) * kHaloX + ((lane >> 1) & 3);
  const uint32_t first_at = first_pixel * kPixelBytes + (((piece ^ (first_pixel >> 1)) & 3u) << 4) + (lane & 1) * 8 - (lane * kPixelBytes + turn);

  uint32_t taken = 0, slot = 0, parity = 0, flip = 0;  // chunks taken so far, the next one's ring position; panel in use
  bool alive = true;
  auto take_chunk = [&]() -> uint32_t {  // the lane's address in the next chunk, once it has arrived
    if (alive) alive = mbar_wait_warp(full0 + 8 * slot, parity, &abort_flag, p.status, kStatusWaitRows);
    const uint32_t at = lane_at + slot * kChunkBytes;
    ++taken;
    if (++slot == kStages) slot = 0, parity ^= 1u;
    return at;
  };
  uint32_t number = 0;  // MX: steps begun so far
  // MX panels are filled behind the step's barrier and stored behind the next one
  int stored_x = 0, stored_y = 0, stored_c = 0, stored_b = -1;
  auto store_panel = [&](uint32_t panel, int c, int x, int y, int b) {
    if (elect_one()) {
      tma_store_4d(&out_map, panel, c, x, y, b);
      bulk_commit();
    }
  };

  for (int ct = member; ct < p.channel_tiles && s_begin < s_end; ct += p.group_quads) {
    const int c0 = ct * kTileC;
    uint32_t bfrag[3][8][2];
    {  // weights through shared memory into the B fragments
      if (ct != member) named_barrier(quad_barrier, 128);  // every warp has read those of the tile before
      for (int i = threadIdx.x & 127; i < kTaps * (kTileC / 2); i += 128) {
        const uint32_t word = __ldg(p.weight + ((static_cast<size_t>(i >> 4) * p.channels + c0) >> 1) + (i & 15));
        asm volatile("st.shared.b32 [%0], %1;" ::"r"(weights_at + i * 4), "r"(word) : "memory");
      }
      if (piece == 0) {
        if (lane == 0) {
          asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(list), "r"(0u) : "memory");
          asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(list + kListTags), "r"(0u) : "memory");
        }
        const float bias = __ldg(p.bias + c0 + lane);
        asm volatile("st.shared.v2.f32 [%0], {%1, %1};" ::"r"(bias_at + lane * 8), "f"(bias) : "memory");
      }
      named_barrier(quad_barrier, 128);
      if (MODE == kOutMx) {  // the size of the taps (see error_of) and the largest |bias| of the warp's channels; four lanes per channel
        const uint32_t c = piece * 8 + (lane & 7);
        float bias, sum = 0.0f, most = 0.0f;
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(bias) : "r"(bias_at + c * 8));
#pragma unroll
        for (int i = 0; i < 7; ++i) {
          const int t = i * 4 + (lane >> 3);
          uint16_t tap = 0;
          if (t < kTaps) asm volatile("ld.shared.u16 %0, [%1];" : "=h"(tap) : "r"(weights_at + t * (kTileC * 2) + c * 2));
          sum += fabsf(bf16_lo(tap)), most = fmaxf(most, fabsf(bf16_lo(tap)));
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 8);
        sum += __shfl_xor_sync(0xffffffffu, sum, 16);
        const float tap_size = warp_max(fmaxf(2.0f * most, 0.25f * sum)), largest_bias = warp_max(fabsf(bias));
        if (lane == 0) asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(list + kListSizes + piece * 8), "f"(tap_size), "f"(largest_bias) : "memory");
        __syncwarp();
      }
      // B[k][n] = w[row - dy][column - dx] for patch position k = (row, column) and output pixel n = (dx, dy), else 0; this
      // lane holds columns q and q + 4 of pixel n
      const int q = lane & 3, dx = lane >> 3, dy = (lane >> 2) & 1;
      const bool lo_in = q >= dx, hi_in = q <= dx;
#pragma unroll
      for (int st = 0; st < 3; ++st) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int ky = 2 * st + h - dy;
          const bool in = ky >= 0 && ky < 5;
          uint32_t lo[4] = {}, hi[4] = {};  // 8 channels of the two taps
          const uint32_t tap = weights_at + (ky * 5 + q - dx) * (kTileC * 2) + piece * 16;
          if (in && lo_in) lds128(tap, lo);
          if (in && hi_in) lds128(tap + 4 * kTileC * 2, hi);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            bfrag[st][2 * j][h] = __byte_perm(lo[j], hi[j], 0x5410);
            bfrag[st][2 * j + 1][h] = __byte_perm(lo[j], hi[j], 0x7632);
          }
        }
        if (shared_fragments(MODE)) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(fragments + (st * 4 + j) * 512), "r"(bfrag[st][2 * j][0]),
                         "r"(bfrag[st][2 * j][1]), "r"(bfrag[st][2 * j + 1][0]), "r"(bfrag[st][2 * j + 1][1])
                         : "memory");  // (each lane reads back only what it wrote)
          }
        }
      }
    }

    // ---- the outputs in the list once more, and steps that are tagged as a whole, after the stores of their panels ----
    const auto sum_of = [&](int b, int y, int x, int c) {
      float bias;
      asm volatile("ld.shared.f32 %0, [%1];" : "=f"(bias) : "r"(bias_at + c * 8));
      return chain_sum(p.value + static_cast<size_t>(b) * p.height * p.width * p.channels + c0 + c, p.height, p.width, p.channels,
                       weights_at + c * 2, bias, y, x);
    };
    // one output per lane: channel c of image row `row` (of all images one below the other); MXFP8: a warp per block, c = lane
    const auto put = [&](uint32_t row, int px, int c, float sum) {
      float out, unused;
      unpack2(activate2<ACT>(pack2(sum, sum)), out, unused);
      const size_t pixel = static_cast<size_t>(row) * p.width + px, to = pixel * p.channels + c0 + c;
      if (MODE == kOutBf16) {
        reinterpret_cast<uint16_t*>(p.out)[to] = static_cast<uint16_t>(pack_bf16(out, 0.0f));
      } else if (MODE == kOutInt8) {
        p.out[to] = static_cast<uint8_t>(int8_exact(int8.scale, bf16_lo(pack_bf16(out, 0.0f))));
      } else {
        // (fmaxf drops a not-a-number, as the block maximum of a step does)
        const int e = e8m0_exponent(__uint_as_float(redux_max(__float_as_uint(fmaxf(fabsf(out), 0.0f)), 0xffffffffu)));
        p.out[to] = static_cast<uint8_t>(e4m3x2(out * exp2_int(-e), 0.0f));
        const int groups = p.channels >> 5;
        if (lane == 0) p.scales[p.swizzled ? swizzled_scale_offset(pixel, ct, (groups + 3) >> 2) : pixel * groups + ct] = static_cast<uint8_t>(e + 127);
      }
    };
    const auto redo_step = [&](const Position& at) {  // a row per warp, a channel per lane, four columns at a time
      const int row = at.k0 * kStepRows + piece, x0 = at.tx * kTileX, b = at.b;
      if (row >= p.height) return;
      float bias;
      asm volatile("ld.shared.f32 %0, [%1];" : "=f"(bias) : "r"(bias_at + lane * 8));
      const uint16_t* image = p.value + static_cast<size_t>(b) * p.height * p.width * p.channels + c0 + lane;
#pragma unroll 1
      for (int px = x0; px < min(x0 + kTileX, p.width); px += 4) {
        const float4 sums = chain_sum4(image, p.height, p.width, p.channels, weights_at + lane * 2, bias, row, px);
#pragma unroll 1
        for (int j = 0; j < min(4, p.width - px); ++j) {
          put(b * p.height + row, px + j, lane, j == 0 ? sums.x : j == 1 ? sums.y : j == 2 ? sums.z : sums.w);
        }
      }
    };
    const auto flush = [&](int step) {  // at the end of a step (flip is already the next one's)
      named_barrier(quad_barrier, 128);
      if (MODE == kOutMx) {
        if (piece == 0 && stored_b >= 0 && alive) store_panel(panels + (flip ^ 1u) * panel_bytes(MODE), stored_c, stored_x, stored_y, stored_b);
        stored_b = -1;
      }
      uint32_t count, redo, redo_before;
      asm volatile("ld.shared.b32 %0, [%1];" : "=r"(count) : "r"(list) : "memory");
      const uint32_t redo_tags = list + kListTags + (MODE == kOutInt8 ? 0u : 4u);
      asm volatile("ld.shared.b32 %0, [%1];" : "=r"(redo) : "r"(redo_tags + (flip ^ 1u) * 8) : "memory");
      asm volatile("ld.shared.b32 %0, [%1];" : "=r"(redo_before) : "r"(redo_tags + flip * 8) : "memory");
      const bool again = redo != 0 && (MODE != kOutMx || redo == number);
      const bool again_before = redo_before != 0 && (MODE != kOutMx || redo_before == number - 1u);
      if (count == 0 && !again && !again_before) return;
      if (piece == 0 && elect_one()) bulk_wait_all();
      named_barrier(quad_barrier, 128);  // (all of the quad have read the header)
      if ((threadIdx.x & 127) == 0) {
        asm volatile("st.shared.b32 [%0], %1;" ::"r"(list), "r"(0u) : "memory");
        asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(list + kListTags), "r"(0u) : "memory");
      }
      if (alive) {
        count = MODE == kOutInt8 ? 0 : min(count, list_entries(MODE));
#pragma unroll 1
        for (uint32_t i = MODE == kOutMx ? piece : threadIdx.x & 127; i < count; i += MODE == kOutMx ? 4 : 128) {
          uint32_t entry;
          asm volatile("ld.shared.b32 %0, [%1];" : "=r"(entry) : "r"(list + kListHeader + i * 4) : "memory");
          const Position at = position_of(p, s_begin + static_cast<int>(entry >> 12));
          const int row = at.k0 * kStepRows + static_cast<int>((entry >> 10) & 3u), px = at.tx * kTileX + static_cast<int>((entry >> 5) & 31u);
          const int c = MODE == kOutMx ? lane : static_cast<int>(entry & 31u);
          put(at.b * p.height + row, px, c, sum_of(at.b, row, px, c));
        }
#pragma unroll 1
        for (int s = again_before ? step - 1 : step; s <= (again ? step : step - 1); ++s) redo_step(position_of(p, s));
      }
      named_barrier(quad_barrier, 128);  // the entries have been read before new ones are noted
    };

    for (int s = s_begin; s < s_end;) {
      const Position at = position_of(p, s);
      const int len = min(p.strip_steps - at.k0, s_end - s);
      s += len;
      const int x0 = at.tx * kTileX, x = x0 + lane;
      // (rows of the scale matrix fit 32 bits: one more would be 256 GB of input)
      const uint32_t scale_row = (static_cast<uint32_t>(at.b) * p.height + piece) * p.width + x;
      const uint32_t scale_tile_bytes = ((p.channels >> 5) + 3) / 4 * 512, scale_at = (ct >> 2) * 512 + (ct & 3);
      // MX: the largest |value| of four channels of a pixel in the first four columns of a chunk, which size_of leaves out
      const auto first_columns = [&](uint32_t from) {
        uint32_t v[2];
        asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v[0]), "=r"(v[1]) : "r"(from + first_at));
        return max_abs(max_abs(0.0f, bf16_lo(v[0]), __uint_as_float(v[0])), bf16_lo(v[1]), __uint_as_float(v[1]));
      };
      RowPair r0, r1;  // the two row pairs above the ones a step brings
      float size_above = 0.0f;  // MX: the largest |value| that the lane has seen of their chunk
      {
        const uint32_t from = take_chunk();
        load_pair(from, r0);
        load_pair(from + 2 * kRowBytes, r1);
        if (MODE == kOutMx) size_above = size_of(r0, r1, first_columns(from));
      }
      for (int k = 0; k < len; ++k) {
        const int y = (at.k0 + k) * kStepRows;
        const int step = s - len + k;
        const uint32_t entry = static_cast<uint32_t>(step - s_begin) << 12 | static_cast<uint32_t>(lane) << 5;  // + row * 1024 + channel
        // The flush tag of the step before, in which all warps have to see the same. Dense and INT8 steps are noted ahead of their
        // barrier: the tag is read ahead of the next one, and the step after this one, which uses its place again, begins behind
        // that. MXFP8 steps are noted behind their barrier as well: the tag is read behind the next one, and a warp that is ahead may
        // have left the mark of the step after this one, which differs. (It then found no mark, and nor does this warp.)
        if (MODE == kOutMx) ++number;
        const uint32_t mark = MODE == kOutMx ? number : 1u, tags = list + kListTags + flip * 8, tags_before = list + kListTags + (flip ^ 1u) * 8;
        uint32_t tag = 0;
        const auto read_tag = [&]() {
          uint32_t redo;
          asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(tag), "=r"(redo) : "r"(tags_before) : "memory");
          if (MODE == kOutInt8) tag |= redo;  // (says nothing more; without it the compiler's schedule takes 182 instead of 172 us)
        };
        if (MODE != kOutMx) read_tag();
        const uint32_t from = take_chunk();
        const uint32_t panel = panels + flip * panel_bytes(MODE);
        float acc[8][4];
        float size_product = 0.0f, tap_size = 0.0f, largest_bias = 0.0f;  // MX: largest |value| that the lane knows of times the size of the taps
        {
          float first = 0.0f;
          if (MODE == kOutMx) {
            first = first_columns(from);
            asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(tap_size), "=f"(largest_bias) : "r"(list + kListSizes + piece * 8));
          }
          RowPair r2;
          const auto multiply = [&](auto first, const RowPair& upper, const RowPair& lower, int st) {
            if constexpr (shared_fragments(MODE)) {
              multiply_step_shared<decltype(first)::value>(upper, lower, fragments + st * (4 * 512), acc);
            } else {
              multiply_step<decltype(first)::value>(upper, lower, bfrag[st], acc);
            }
          };
          multiply(std::true_type{}, r0, r1, 0);
          load_pair(from, r2);
          multiply(std::false_type{}, r1, r2, 1);
          r0 = r2;
          load_pair(from + 2 * kRowBytes, r1);
          multiply(std::false_type{}, r0, r1, 2);
          if (MODE == kOutMx) {
            const float size = size_of(r0, r1, first), both = fmaxf(size, size_above);
            size_product = tap_size * both;
            if (size_product < 1e-36f && tap_size > 0.0f && both > 0.0f) size_product = 1e-36f;  // (underflow)
            size_above = size;
          }
        }
        // bias and activation: v[channel][0 / 1] = rows (0, 1) / (2, 3) of the lane's column
        uint64_t v[8][2];
        float margin = 0.0f, largest = 0.0f;
#pragma unroll
        for (int c = 0; c < 8; c += 2) {
          uint64_t bias[2];
          asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(bias[0]), "=l"(bias[1]) : "r"(bias_at + (piece * 8 + c) * 8));
          float slack[2];
#pragma unroll
          for (int d = 0; d < 2; ++d) {
            const float(&a)[4] = acc[c + d];
            v[c + d][0] = add2(pack2(a[0], a[1]), bias[d]);
            v[c + d][1] = add2(pack2(a[2], a[3]), bias[d]);
            if (MODE == kOutBf16) {
              float b, unused, f[4];
              unpack2(bias[d], b, unused);
              unpack2(v[c + d][0], f[0], f[1]);
              unpack2(v[c + d][1], f[2], f[3]);
              const float size = max_abs_nan(max_abs_nan(a[0], a[1], a[2]), a[3], b);
              largest = max_abs_nan(largest, size, size);
              slack[d] = fmaf(min_abs(min_abs(f[0], f[1], f[2]), f[3], f[3]), kCancelled, -size);
            }
          }
          if (MODE == kOutBf16) {
            margin = fminf(fminf(margin, slack[0]), slack[1]);
          } else {
#pragma unroll
            for (int d = 0; d < 2; ++d) {
              largest = max_abs_nan(largest, acc[c + d][0], acc[c + d][1]);
              largest = max_abs_nan(largest, acc[c + d][2], acc[c + d][3]);
            }
          }
        }
        float error = 0.0f;  // MX: a bound on the error of the warp's arguments
        float limit = __int_as_float(0x7F800000), reached = largest;
        if (MODE == kOutMx) {
          reached = warp_max(max_abs_nan(largest, size_product, size_product));
          error = error_of(reached, largest_bias);
          limit = 1e37f;  // (near the end of the range the chain may overflow where these sums do not)
        }
        if (!(reached < limit)) {
          if (MODE == kOutInt8) {
            tag_flush(tags, mark);  // (without a list the one tag says it all)
          } else {
            tag_redo(tags, mark);
          }
        }
        if (MODE == kOutBf16 && margin < 0.0f) {
          uint32_t cancelled = 0;  // bit 4 c + i
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            float f[4];
            unpack2(v[c][0], f[0], f[1]);
            unpack2(v[c][1], f[2], f[3]);
            // (the bias is part of the size as the difference of sum and product part)
            const float size = max_abs(max_abs(acc[c][0], acc[c][1], acc[c][2]), acc[c][3], f[0] - acc[c][0]) * (1.001f / kCancelled);
#pragma unroll
            for (int i = 0; i < 4; ++i) cancelled |= fabsf(f[i]) <= size ? 1u << (4 * c + i) : 0u;
          }
          if (__popc(cancelled) > kMostNoted) {
            tag_redo(tags, mark);
            cancelled = 0;
          }
#pragma unroll 1
          for (; cancelled != 0; cancelled &= cancelled - 1) {
            const int bit = __ffs(cancelled) - 1;
            if (x < p.width && y + (bit & 3) < p.height) note<MODE>(list, tags, mark, entry + (bit & 3) * 1024 + piece * 8 + (bit >> 2));
          }
        }
        // MX: whether the warp may hold many values in the left tail of the GELU. There they err by less than (1 + |x|) times the
        // argument's error *of themselves* (|GELU'| <= |x| |GELU|), far below the bound for all: the codes of values near zero would
        // look open everywhere. (Arguments of a standard deviation below 1.5 have fewer such values, at -4 and below, than looking
        // for them is worth.)
        constexpr bool kTails = MODE == kOutMx && ACT == kActGelu;
        uint32_t tails = 0;  // bit c * 4 + i * 4 + d, c = 0, 4: channel c + d of pixel i is below -1, before the activation
        uint32_t edge = 0;  // (as `pending` below) an argument at the underflow of Phi
        bool tail_warp = false;
        if (kTails) {
          tail_warp = error < 0.01f && __any_sync(0xffffffffu, largest + largest_bias > 5.0f);
          if (tail_warp) {
#pragma unroll
            for (int n = 7; n >= 0; --n) {
#pragma unroll
              for (int d = 3; d >= 0; --d) {
                float lo, hi;
                unpack2(add2(v[(n >> 2) * 4 + d][(n & 3) >> 1], pack2(1.0f, 1.0f)), lo, hi);
                tails = __funnelshift_l(__float_as_uint(n & 1 ? hi : lo), tails, 1);
              }
            }
            if (__any_sync(0xffffffffu, largest + largest_bias > 12.0f)) {
              // where Phi underflows the value goes from below zero to +0, and its code from 0x80 to 0x00
              float nearest = 1.0f;
#pragma unroll
              for (int c = 0; c < 8; ++c) {
                float f[4];
                unpack2(add2(v[c][0], pack2(kGeluUnderflow, kGeluUnderflow)), f[0], f[1]);
                unpack2(add2(v[c][1], pack2(kGeluUnderflow, kGeluUnderflow)), f[2], f[3]);
                nearest = min_abs(min_abs(nearest, f[0], f[1]), f[2], f[3]);
              }
              if (nearest < 2.0f * error + 1e-5f) {
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                  float f[4];
                  unpack2(v[c][0], f[0], f[1]);
                  unpack2(v[c][1], f[2], f[3]);
#pragma unroll
                  for (int i = 0; i < 4; ++i) {
                    edge |= fabsf(f[i] + kGeluUnderflow) < 2.0f * error + 1e-5f ? 1u << (8 * (c & 3) + 7 - (2 * i + (c >> 2))) : 0u;
                  }
                }
              }
            }
          }
        }
        // (the quantiser of a ReLU clips: its bounds lie on both sides of zero)
        if (MODE != kOutMx || ACT != kActRelu) {
#pragma unroll
          for (int c = 0; c < 8; ++c) v[c][0] = activate2<ACT>(v[c][0]), v[c][1] = activate2<ACT>(v[c][1]);
        }
        float inv[4];
        uint32_t unsure = 0;  // MX: bit i for a pixel whose block exponent is open
        if (MODE == kOutMx) {
          constexpr float kNone = ACT == kActRelu ? -__builtin_huge_valf() : 0.0f;
          float amax[4] = {kNone, kNone, kNone, kNone};  // (of a ReLU: the largest value, below zero as it is)
#pragma unroll
          for (int c = 0; c < 8; c += 2) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              float lo0, hi0, lo1, hi1;
              unpack2(v[c][h], lo0, hi0);
              unpack2(v[c + 1][h], lo1, hi1);
              amax[2 * h] = ACT == kActRelu ? max3(amax[2 * h], lo0, lo1) : max_abs(amax[2 * h], lo0, lo1);
              amax[2 * h + 1] = ACT == kActRelu ? max3(amax[2 * h + 1], hi0, hi1) : max_abs(amax[2 * h + 1], hi0, hi1);
            }
          }
          const uint32_t mine = exchange + flip * 2048 + lane * 16;
          asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(mine + piece * 512), "f"(amax[0]), "f"(amax[1]), "f"(amax[2]), "f"(amax[3])
                       : "memory");
          const uint32_t errors = list + kListErrors + flip * 16;
          if (lane == 0) asm volatile("st.shared.f32 [%0], %1;" ::"r"(errors + piece * 4), "f"(ACT == kActGelu ? error * kGeluSlope : error) : "memory");
          if (piece == 0 && elect_one()) bulk_wait_read<0>();  // the store of the panel before the last
          named_barrier(quad_barrier, 128);
          if (piece == 0) {
            if (stored_b >= 0) store_panel(panels + (flip ^ 1u) * panel_bytes(MODE), stored_c, stored_x, stored_y, stored_b);
            if (alive) issue_until(taken + kStages - kept_chunks(MODE));
          }
          stored_c = c0, stored_x = x0, stored_y = y, stored_b = p.tma_out ? at.b : -1;
          read_tag();
          float theirs[3][4];
#pragma unroll
          for (int other = 1; other < 4; ++other) {
            float(&t)[4] = theirs[other - 1];
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(t[0]), "=f"(t[1]), "=f"(t[2]), "=f"(t[3]) : "r"(mine + (piece ^ other) * 512));
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            amax[i] = fmaxf(ACT == kActRelu ? max3(amax[i], theirs[0][i], theirs[1][i]) : max_abs(amax[i], theirs[0][i], theirs[1][i]), theirs[2][i]);
          }
          uint32_t bytes[4];
          float e[4];
          asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(e[0]), "=f"(e[1]), "=f"(e[2]), "=f"(e[3]) : "r"(errors));
          unsure = block_scales(amax, fmaxf(max3(e[0], e[1], e[2]), e[3]), bytes, inv);
          if (alive && x < p.width && y + piece < p.height) {  // each warp stores the scales of one row
            const uint32_t byte = piece == 0 ? bytes[0] : piece == 1 ? bytes[1] : piece == 2 ? bytes[2] : bytes[3];
            const uint32_t row = scale_row + y * p.width, groups = p.channels >> 5;
            uint8_t* to = p.scales + (p.swizzled ? static_cast<uint64_t>(row >> 7) * scale_tile_bytes + (row & 31) * 16 + ((row & 127) >> 5) * 4 + scale_at
                                                 : static_cast<uint64_t>(row) * groups + ct);
            *to = static_cast<uint8_t>(byte);
            if (ct + 1 == p.channel_tiles) {  // the padding groups of a swizzled row
              for (int pad = 1; pad < p.swizzled; ++pad) to[pad] = 0;
            }
          }
        }
        // the lane's 8 channels of each of its four pixels, as they are stored
        constexpr int kWords = 2 * kOutBytes;
        uint32_t words[4][kWords];
        uint32_t pending = 0;  // MX: open codes of the lane: channel 4 j + b of pixel i in bit 8 b + 7 - (2 i + j)
        if (MODE == kOutMx) {
          // the codes of both bounds of every value; where they are the same it is the code of the fp32 chain, too
          uint32_t open[4][2];  // a byte other than 0 for a code that is open
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float tail_share[2] = {};
            if (kTails && tail_warp) {
              // (|GELU(x)| < exp(-x^2 / 2) / sqrt(2 pi) bounds |x| where the value is more than 2**-11 of the scale; below, both bounds
              // are zeros)
#pragma unroll
              for (int i = 0; i < 2; ++i) {
                const float far = fmaxf(1.3863f * static_cast<float>(static_cast<int>(__float_as_uint(inv[2 * h + i]) >> 23) - 127 + 11) - 1.83f, 0.0f);
                tail_share[i] = kGeluSlope * error * (2.0f + __fsqrt_rn(far));
              }
            }
#pragma unroll
            for (int c = 0; c < 8; c += 4) {
              uint32_t codes[2][2];
#pragma unroll
              for (int side = 0; side < 2; ++side) {
                const float bound = (side ? error : -error) * (ACT == kActGelu ? kGeluBase : 1.0f);
                const float grown = ACT == kActGelu ? 1.0f + (side ? error : -error) * kGeluGrowth : 1.0f;
                const uint64_t bounds = pack2(bound * inv[2 * h], bound * inv[2 * h + 1]), scale = pack2(grown * inv[2 * h], grown * inv[2 * h + 1]);
                float f[4][2];
#pragma unroll
                for (int d = 0; d < 4; ++d) unpack2(fma2(v[c + d][h], scale, bounds), f[d][0], f[d][1]);
#pragma unroll
                for (int i = 0; i < 2; ++i) codes[side][i] = codes_of<ACT>(f[0][i], f[1][i], f[2][i], f[3][i]);
              }
#pragma unroll
              for (int i = 0; i < 2; ++i) words[2 * h + i][c / 4] = codes[0][i], open[2 * h + i][c / 4] = codes[0][i] ^ codes[1][i];
              if (kTails && tail_warp) {
                // codes of the values themselves, and for those in the tail the bounds that hold there
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                  float f[4], low[4], up[4];
#pragma unroll
                  for (int d = 0; d < 4; ++d) {
                    float first, second;
                    unpack2(v[c + d][h], first, second);
                    f[d] = (i ? second : first) * inv[2 * h + i];
                    low[d] = fmaf(f[d], -tail_share[i], f[d]), up[d] = fmaf(f[d], tail_share[i], f[d]);
                  }
                  const uint32_t in_tail = ((tails >> (c * 4 + (2 * h + i) * 4) & 15u) * 0x204081u & 0x01010101u) * 0xFFu;
                  const uint32_t differ = codes_of<ACT>(low[0], low[1], low[2], low[3]) ^ codes_of<ACT>(up[0], up[1], up[2], up[3]);
                  open[2 * h + i][c / 4] = (open[2 * h + i][c / 4] & ~in_tail) | (differ & in_tail);
                  words[2 * h + i][c / 4] = codes_of<ACT>(f[0], f[1], f[2], f[3]);
                }
              }
            }
          }
          uint32_t any = edge;
#pragma unroll
          for (int i = 0; i < 4; ++i) any |= open[i][0] | open[i][1];
          if (__any_sync(0xffffffffu, any != 0)) {
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const uint32_t bytes = open[k >> 1][k & 1];
              pending |= ((((bytes & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | bytes) & 0x80808080u) >> k;
            }
            pending |= edge;
            const int rows = min(p.height - y, kStepRows);
            pending = x < p.width ? pending & ((0xFF00u >> (2 * rows) & 0xFFu) * 0x01010101u) : 0;
            if (__reduce_add_sync(0xffffffffu, __popc(pending)) > kMostOpen) {
              tag_redo(tags, mark);
              pending = 0;
            }
          }
          if (piece == 0 && unsure != 0 && x < p.width) {
#pragma unroll 1
            for (; unsure != 0; unsure &= unsure - 1) {
              const int i = __ffs(unsure) - 1;
              if (y + i < p.height) note<MODE>(list, tags, mark, entry + i * 1024);
            }
          }
        } else {
#pragma unroll
          for (int c = 0; c < 8; c += 4) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              float f[4];  // channels c .. c + 3 of pixel i
#pragma unroll
              for (int d = 0; d < 4; ++d) {
                float lo, hi;
                unpack2(v[c + d][i >> 1], lo, hi);
                f[d] = i & 1 ? hi : lo;
              }
              const uint32_t w0 = pack_bf16(f[0], f[1]), w1 = pack_bf16(f[2], f[3]);
              if (MODE == kOutBf16) {
                words[i][c / 2] = w0;
                words[i][(c / 2 + 1) % kWords] = w1;
              } else {
                words[i][c / 4] = int8_pack4(int8, bf16_lo(w0), bf16_hi(w0), bf16_lo(w1), bf16_hi(w1));
              }
            }
          }
        }
        if (p.tma_out) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t pixel = i * kTileX + lane;
            if (MODE == kOutBf16) {
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(panel + pixel * 64 + turn), "r"(words[i][0]), "r"(words[i][1]),
                           "r"(words[i][2 % kWords]), "r"(words[i][3 % kWords])
                           : "memory");
            } else {
              asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(panel + pixel * 32 + (((piece >> 1) ^ ((lane >> 2) & 1)) << 4) + (piece & 1) * 8),
                           "r"(words[i][0]), "r"(words[i][1])
                           : "memory");
            }
          }
        } else if (alive) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (x < p.width && y + i < p.height) {
              uint32_t* to = reinterpret_cast<uint32_t*>(
                  p.out + (((static_cast<size_t>(at.b) * p.height + y + i) * p.width + x) * p.channels + c0 + piece * 8) * kOutBytes);
#pragma unroll
              for (int j = 0; j < kWords; ++j) to[j] = words[i][j];
            }
          }
        }
        if (MODE == kOutMx) {
          // The sums of two outputs at a time as the chain forms them, from the two chunks of the ring that hold their windows: a product
          // per lane into the scratch, a chain in every lane, the codes from the lanes they belong to. One at a time takes 292 us for
          // GELU at 8x400x400x128 instead of 280, an output per lane without scratch 303. (Listed for the end of the range, when
          // the rows have left the L2, the corrections took three times as long.) Scratch is the warp's part of the exchange of the
          // step before: nobody else looks at it until the warp writes the next maxima.
          const uint32_t scratch = exchange + (flip ^ 1u) * 2048 + piece * 512;
          const uint32_t below = slot == 0 ? kStages - 1 : slot - 1, above = below == 0 ? kStages - 1 : below - 1;
#pragma unroll 1
          for (uint32_t holders; (holders = __ballot_sync(0xffffffffu, pending != 0)) != 0;) {
            // the first open codes of two lanes
            const uint32_t first = __ffs(holders) - 1, others = holders & (holders - 1), second = others != 0 ? __ffs(others) - 1 : first;
            const uint32_t mine = __ffs(pending) - 1;
            pending = lane == first || lane == second ? pending & (pending - 1) : pending;
            const auto channel = [&](uint32_t bit) { return piece * 8 + (~bit & 1u) * 4 + (bit >> 3); };
            const auto row_of = [&](uint32_t bit) { return (7 - (bit & 7u)) >> 1; };
            const auto products = [&](uint32_t owner, uint32_t to) {
              const uint32_t bit = __shfl_sync(0xffffffffu, mine, owner), c = channel(bit);
              if (lane < kTaps) {
                const uint32_t ky = lane / 5, row = row_of(bit) + ky, pixel = (row & 3u) * kHaloX + owner + (lane - ky * 5);
                uint16_t value, tap;
                asm volatile("ld.shared.u16 %0, [%1];" : "=h"(value) : "r"(ring + (row < 4 ? above : below) * kChunkBytes + pixel * kPixelBytes +
                                                                         (((c >> 3) ^ ((pixel >> 1) & 3u)) << 4) + (c & 7u) * 2));
                asm volatile("ld.shared.u16 %0, [%1];" : "=h"(tap) : "r"(weights_at + lane * (kTileC * 2) + c * 2));
                asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(to + lane * 8), "f"(bf16_lo(value)), "f"(bf16_lo(tap)) : "memory");
              }
            };
            products(first, scratch);
            if (others != 0) products(second, scratch + 208);
            const uint32_t from = lane == second && others != 0 ? scratch + 208 : scratch, c = channel(mine & 31u), i = row_of(mine & 31u);
            float bias;
            asm volatile("ld.shared.f32 %0, [%1];" : "=f"(bias) : "r"(bias_at + c * 8));
            __syncwarp();
            float sum = 0.0f;
#pragma unroll
            for (int t = 0; t < kTaps; t += 2) {
              uint32_t pair[4];
              lds128(from + t * 8, pair);
              sum = fmaf(__uint_as_float(pair[0]), __uint_as_float(pair[1]), sum);
              if (t + 1 < kTaps) sum = fmaf(__uint_as_float(pair[2]), __uint_as_float(pair[3]), sum);
            }
            __syncwarp();
            sum += bias;
            float out, unused;
            unpack2(activate2<ACT>(pack2(sum, sum)), out, unused);
            const uint32_t code = e4m3x2(out * (i == 0 ? inv[0] : i == 1 ? inv[1] : i == 2 ? inv[2] : inv[3]), 0.0f);
            if (lane == first || lane == second) {
              if (p.tma_out) {
                asm volatile("st.shared.u8 [%0], %1;" ::"r"(panel + (i * kTileX + lane) * 32 + (((piece >> 1) ^ ((lane >> 2) & 1)) << 4) + (c & 15u)), "r"(code) : "memory");
              } else if (alive) {
                p.out[((static_cast<size_t>(at.b) * p.height + y + i) * p.width + x) * p.channels + c0 + c] = static_cast<uint8_t>(code);
              }
            }
          }
        }
        if (p.tma_out) fence_async_proxy();
        if (MODE != kOutMx) {
          if (piece == 0 && elect_one()) bulk_wait_read<0>();  // the store of the other panel
          named_barrier(quad_barrier, 128);
          if (piece == 0) {
            if (p.tma_out && alive) store_panel(panel, c0 * kOutBytes, x0, y, at.b);
            if (alive) issue_until(taken + kStages);
          }
        }
        flip ^= 1u;
        if ((tag != 0 && (MODE != kOutMx || tag == number - 1u)) || step + 1 == s_end) flush(step);
      }
    }
  }
  if (piece == 0 && elect_one()) bulk_wait_read<0>();
  if (abort_flag) {
    // a wait ran out: give copies that are still in flight time to land before the shared memory is released
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
}

int g_dw_max_ctas = 0;

template <int MODE>
int launch_kernel(const CUtensorMap& in_map, const CUtensorMap& out_map, const DwParams& p, int act, unsigned grid, cudaStream_t s) {
  constexpr size_t kSmem = 1024 + kQuads * quad_bytes(MODE);
  static_assert(kSmem <= 227 * 1024, "shared memory of one CTA");
  auto kernel = dw5x5_kernel<MODE, kActRelu>;
  if constexpr (MODE != kOutInt8) {  // (the INT8 form always ends in a ReLU)
    if (act != kActRelu) kernel = act == kActGelu ? dw5x5_kernel<MODE, kActGelu> : dw5x5_kernel<MODE, kActNone>;
  }
  // every instantiation gets the opt-in limit once per device
  static bool configured[3][kMaxDevices] = {};
  const int device = current_device();
  if (device < 0 || device >= kMaxDevices || !configured[act][device]) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmem));
    if (e != cudaSuccess) return static_cast<int>(e);
    if (device >= 0 && device < kMaxDevices) configured[act][device] = true;
  }
  launch_dependent(kernel, grid, 128 * kQuads, kSmem, s, 1u, in_map, out_map, p);
  return static_cast<int>(cudaGetLastError());
}

template <int MODE>
int launch(const void* value, const void* weight, const float* bias, void* out, void* scales, const float* scale, int swizzled,
           int batch, int height, int width, int channels, int act, int* status, void* stream) {
  if (batch < 0 || height < 0 || width < 0 || channels <= 0 || act < 0 || act > 2) return kBadArgument;
  if (channels % 32) return kUnsupported;
  if (batch == 0 || height == 0 || width == 0) return kOk;
  if (value == nullptr || weight == nullptr || bias == nullptr || out == nullptr) return kBadArgument;
  if ((reinterpret_cast<uintptr_t>(value) & 15u) || (reinterpret_cast<uintptr_t>(weight) & 3u) ||
      (reinterpret_cast<uintptr_t>(out) & 3u)) {
    return kBadLayout;
  }
  DwParams p;
  p.value = static_cast<const uint16_t*>(value);
  p.weight = static_cast<const uint32_t*>(weight);
  p.bias = bias;
  p.out = static_cast<uint8_t*>(out);
  p.scales = static_cast<uint8_t*>(scales);
  p.scale = scale;
  p.batch = batch, p.height = height, p.width = width, p.channels = channels;
  p.tiles_x = ceil_div(width, kTileX);
  p.channel_tiles = channels / kTileC;
  p.strip_steps = ceil_div(height, kStepRows);
  p.swizzled = swizzled ? 1 + (4 - p.channel_tiles % 4) % 4 : 0, p.status = status;
  p.tma_out = (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
  const long long steps = static_cast<long long>(p.tiles_x) * batch * p.strip_steps;
  if (steps > 0x3fffffffLL || steps * p.channel_tiles > 0x3fffffffffLL) return kUnsupported;
  p.total_steps = static_cast<int>(steps);

  CUtensorMap in_map, out_map;
  {
    const uint64_t dims[4] = {static_cast<uint64_t>(channels), static_cast<uint64_t>(width), static_cast<uint64_t>(height),
                              static_cast<uint64_t>(batch)};
    const uint64_t row = static_cast<uint64_t>(channels) * 2;
    const uint64_t strides[3] = {row, width * row, static_cast<uint64_t>(height) * width * row};
    const uint32_t box[4] = {kTileC, kHaloX, kStepRows, 1};
    const int rc = make_tensor_map(&in_map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, value, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_64B,
                                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
    if (rc != kOk) return rc;
  }
  out_map = in_map;
  if (p.tma_out) {
    const int elem = MODE == kOutBf16 ? 2 : 1;
    const uint64_t row = static_cast<uint64_t>(channels) * elem;  // (in bytes, whatever the element)
    const uint64_t dims[4] = {row, static_cast<uint64_t>(width), static_cast<uint64_t>(height), static_cast<uint64_t>(batch)};
    const uint64_t strides[3] = {row, width * row, static_cast<uint64_t>(height) * width * row};
    const uint32_t box[4] = {static_cast<uint32_t>(kTileC * elem), kTileX, kStepRows, 1};
    const int rc = make_tensor_map(&out_map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, out, dims, strides, box,
                                   MODE == kOutBf16 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
    if (rc != kOk) return rc;
  }
  // one persistent CTA per SM with three quads; a small problem spreads over as many SMs as it has work for
  const int sms = g_dw_max_ctas > 0 && g_dw_max_ctas < sm_count() ? g_dw_max_ctas : sm_count();
  p.group_quads = p.channel_tiles < sms * kQuads ? p.channel_tiles : sms * kQuads;
  const long long most_groups = sms * kQuads / p.group_quads;
  p.groups = static_cast<int>(steps < most_groups ? steps : most_groups);
  const int quads = p.groups * p.group_quads;
  if (steps / p.groups >= kMaxRange) return kUnsupported;  // (on a whole GPU a tensor of more than its memory)
  p.cta_quads = ceil_div(quads, sms);
  const unsigned grid = static_cast<unsigned>(ceil_div(quads, p.cta_quads));
  return launch_kernel<MODE>(in_map, out_map, p, act, grid, static_cast<cudaStream_t>(stream));
}

}  // namespace
}  // namespace fim

using namespace fim;

extern "C" int fim_dw5x5_bf16(const void* value, const void* weight, const float* bias, void* out, int batch, int height,
                              int width, int channels, int act, int* status, void* stream) {
  return launch<kOutBf16>(value, weight, bias, out, nullptr, nullptr, 0, batch, height, width, channels, act, status, stream);
}

extern "C" int fim_dw5x5_mxfp8(const void* value, const void* weight, const float* bias, void* out, void* scales, int swizzled,
                               int batch, int height, int width, int channels, int act, int* status, void* stream) {
  if (scales == nullptr && batch > 0 && height > 0 && width > 0) return kBadArgument;
  return launch<kOutMx>(value, weight, bias, out, scales, nullptr, swizzled, batch, height, width, channels, act, status, stream);
}

extern "C" int fim_dw5x5_relu_int8(const void* value, const void* weight, const float* bias, const float* scale, void* out,
                                   int batch, int height, int width, int channels, int* status, void* stream) {
  if (scale == nullptr && batch > 0 && height > 0 && width > 0) return kBadArgument;
  return launch<kOutInt8>(value, weight, bias, out, nullptr, scale, 0, batch, height, width, channels, kActRelu, status, stream);
}

extern "C" void fim_dw_tune(int max_ctas, int /* reserved */) { g_dw_max_ctas = max_ctas; }

extern "C" int fim_abi_version(void) { return FIM_ABI_VERSION; }
