// GPTQ W3 group-128 planar weights times many activation rows (prompts, the dense fallback): y[T,O] = x[T,K] . W^T.
//
// One persistent kernel instead of chunks that were dequantised into L2 and read back by a library GEMM, two
// or three launches each.  A CTA owns 128 output rows of up to 256 tokens at a time; roles are warps:
//
//   warp 0         TMA: activations of a group, 128-byte swizzle, ring of four stages of up to 192 tokens, three of more
//   warp 2         TMA: plane tiles (three planes of 128 rows of a group), ring of four
//   warps 4..19    four warpgroups take turns on groups: a thread dequantises ITS row of the group and puts the 16-bit
//                  weights into tensor memory (tcgen05.st), where the MMA takes its A operand from: shared
//                  memory, which the B operand and its copies already load to two thirds, never sees them
//   warps 1, 3     tcgen05.mma, 128 x tokens x 16; up to 128 tokens they take turns on groups, each on an accumulator of its
//                  own, which the epilogue adds up; beyond, warp 3 has nothing to do
//   warps 20..27   epilogue: accumulator -> outputs
//
// Tensor memory: the accumulator (256 columns) and four operand slots of a group (64 columns each).  Two slots
// and two accumulators of 192 columns, which let the epilogue overlap the next tile, ran 10 % slower: the way
// from a finished MMA over the refilled slot to the next one is longer than an MMA.  A weight takes one of
// eight values per (row, group), scale * (code - zero) rounded in the scale's dtype and then in the
// activations'; they are looked up four at a time by byte permutes whose selector nibbles are the codes, or multiplied out.
//
// What bounds it: at 256 tokens a tile the MMA (tensor pipe 86 % active); up to 128 instruction issue of the dequantising warps, whatever the
// tokens.  Two warps issue there because one's course over a group (1000 clocks: two barriers 330, eight instructions 470, commits 120) would hold
// the four warpgroups up for 1500 of their 3500 clocks a group; with two they wait 300 to 500.  One issuer and two are kernels of their own: both
// loops in one took the MMAs' operands out of uniform registers (twice the time).  The values of a row come from 16-bit multiplications (200 clocks a
// group of a warpgroup, fp32 ones took 500); where scales and activations share a dtype there is no table but a code inside a magic number,
// on the idle multiply pipes.  The MMA warps look at both barriers with one instruction, their instructions are predicated on the elected lane, and
// where the activations' ring has as many stages as there are operand slots (up to 192 tokens) one commit releases both.
// us on a B200, weights cold, in a graph, fp16 / bf16 scales (in brackets with one issuer and a table of fp32 products): 12288 x 4096 at 64 tokens
// 16.3 / 16.9 (18.6 / 19.0), at 112 18.1 / 18.4 (19.6 / 20.0), at 333 32.9 / 31.7 (36.9 / 36.9), at 512 41.2 / 40.9 (43.0 / 43.0); 4096 x 12288 at 512
// 46.2 / 43.5 (48.0 / 48.5); 24576 x 4096 at 512 76.8 (79.9); chunks of the dense weight, 12288 x 4096 at 64 / 512: 39 / 62.
//
// A role whose wait expires gives up after two seconds in which the rings stood still, so what is in flight has landed when
// the CTA ends; it leaves with the status word set and the tensor memory freed.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <mutex>

#include "fb_common.cuh"

namespace {

using namespace fb;

constexpr int kRows = 128;
constexpr int kMaxTokens = 256;  // of a tile
constexpr int kDequant = 4;      // warpgroups that dequantise
constexpr int kEpilogue = 2;     // warpgroups that write outputs
constexpr int kThreads = 128 * (1 + kDequant + kEpilogue);
constexpr int kBBytes = 192 * 1024;  // ring of activation stages, a group each: four of up to 192 tokens, three of more
constexpr int kMaxBStages = 4;  // as many as operand slots
constexpr int kPlaneStages = 4;  // even: a stage always serves the same warpgroup (a wait by parity must not fall two phases behind)
constexpr int kPlaneStage = 3 * kRows * 16;
constexpr int kASlots = 4;             // weights of a group, 64 columns
static_assert(kMaxBStages == kASlots, "a full ring goes round with the operand slots");
constexpr int kAColumn = kMaxTokens;  // behind the accumulator
constexpr int kMaxMats = 4;
constexpr int kBars = 2 * kMaxBStages + 2 * kPlaneStages + 2 * kASlots + 2;
constexpr size_t kSmem = kBBytes + kPlaneStages * kPlaneStage + kBars * 8 + 16;

struct GemmMatrix {
  CUtensorMap plane_map;  // planes as uint32 [G*3][O/32][128], box 3 x 4 x 128
  const unsigned short* scales;
  const uint8_t* zeros;
  unsigned short* out;
  const unsigned short* addend;
  int O, tile_begin;  // first row tile
};

struct GemmParams {
  alignas(64) GemmMatrix mats[kMaxMats];
  CUtensorMap x_map;  // [T][K], box = tokens of a tile x 64
  unsigned* status;
  int n, T, G, ldo;
  int tokens, token_tiles, tiles, b_stages;
};

__device__ __forceinline__ void tcgen_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tcgen_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ bool elected() {
  uint32_t yes;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(yes));
  return yes != 0;
}
__device__ __forceinline__ void commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// 32 columns of this warp's 32 lanes
__device__ __forceinline__ void tmem_store32(uint32_t at, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, "
      "%23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(at),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]),
      "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]),
      "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
      : "memory");
}
__device__ __forceinline__ void tmem_load16(uint32_t at, uint32_t (&v)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
                 "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
               : "r"(at));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

template <bool BF16>
__device__ __forceinline__ uint32_t add2(uint32_t a, uint32_t b) {
  uint32_t d;
  if (BF16)
    asm("add.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  else
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
template <bool BF16>
__device__ __forceinline__ uint32_t mul2(uint32_t a, uint32_t b) {
  uint32_t d;
  if (BF16)
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  else
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
template <bool BF16>
__device__ __forceinline__ uint32_t fma2(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  if (BF16)
    asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  else
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
// {low, high} rounded to 16 bits
template <bool BF16>
__device__ __forceinline__ uint32_t pack2(float low, float high) {
  uint32_t d;
  if (BF16)
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(high), "f"(low));
  else
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(high), "f"(low));
  return d;
}
template <bool BF16>
__device__ __forceinline__ float widen(unsigned short bits) {
  return BF16 ? __uint_as_float((uint32_t)bits << 16) : __half2float(__ushort_as_half(bits));
}

// Bytes picked by a selector whose nibbles are below eight (__byte_perm would mask it first).
__device__ __forceinline__ uint32_t pick(uint32_t a, uint32_t b, uint32_t selector) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(selector));
  return d;
}
// (a & m) | (b & ~m)
__device__ __forceinline__ uint32_t blend(uint32_t a, uint32_t b, uint32_t m) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xE4;" : "=r"(d) : "r"(a), "r"(b), "r"(m));
  return d;
}

// 32 codes of a row (one word per plane, the high one inverted) -> 16 operand registers, inputs in order.  low, high: bytes
// of the values of the eight codes.  Neighbouring inputs share a byte of the selector words, so that what two look-ups
// pick is interleaved once and is in order then.
__device__ __forceinline__ void look_up(uint32_t p0, uint32_t p1, uint32_t p2, const uint32_t (&low)[2], const uint32_t (&high)[2], uint32_t* to) {
  // low two bits of the codes of inputs 0 2 4 6 of every byte, of 1 3 5 7, and from these of (0, 2 | 1, 3) and (4, 6 | 5, 7)
  const uint32_t even = blend(p0, p1 << 1, 0x55555555u), odd = blend(p0 >> 1, p1, 0x55555555u);
  const uint32_t first = blend(even, odd << 4, 0x0f0f0f0fu), last = blend(even >> 4, odd, 0x0f0f0f0fu);
  const uint32_t two[4] = {first, first >> 2, last, last >> 2};
  // bits 2 and 6: high bits of inputs 2 s and 2 s + 1
  const uint32_t top[4] = {blend(p2 << 2, p2 << 5, 0x0f0f0f0fu), blend(p2, p2 << 3, 0x0f0f0f0fu), blend(p2 >> 2, p2 << 1, 0x0f0f0f0fu), blend(p2 >> 4, p2 >> 1, 0x0f0f0f0fu)};
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    const uint32_t bits = two[s] & 0x33333333u;
    uint32_t codes;  // byte m: the codes of inputs 8 m + 2 s and 8 m + 2 s + 1
    asm("lop3.b32 %0, %1, %2, %3, 0xF4;" : "=r"(codes) : "r"(bits), "r"(0x44444444u), "r"(top[s]));  // bits | (0x4444... & ~top)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const uint32_t sel = half ? codes >> 16 : codes;
      const uint32_t l = pick(low[0], low[1], sel), h = pick(high[0], high[1], sel);
      to[8 * half + s] = pick(l, h, 0x5140u), to[8 * half + 4 + s] = pick(l, h, 0x7362u);
    }
  }
}

// The values of a row's eight codes, scale * (code - zero) rounded in the scale's dtype and then in the activations', split into
// low and high bytes.  A 16-bit multiplication rounds the exact product once, as the rounding of an fp32 product would.
template <bool SCALE_BF16, bool ACT_BF16>
__device__ __forceinline__ void value_table(uint32_t scale_bits, uint32_t zero, uint32_t (&low)[2], uint32_t (&high)[2]) {
  constexpr uint32_t kCodes[4] = {SCALE_BF16 ? 0x3f800000u : 0x3c000000u, SCALE_BF16 ? 0x40404000u : 0x42004000u, SCALE_BF16 ? 0x40a04080u : 0x45004400u,
                                  SCALE_BF16 ? 0x40e040c0u : 0x47004600u};  // (0, 1), (2, 3), (4, 5), (6, 7)
  const float minus_zero = -(float)zero;
  const uint32_t off = pack2<SCALE_BF16>(minus_zero, minus_zero), scale = scale_bits * 0x10001u;
  uint32_t v[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    v[q] = mul2<SCALE_BF16>(add2<SCALE_BF16>(kCodes[q], off), scale);
    if (SCALE_BF16 != ACT_BF16) v[q] = pack2<ACT_BF16>(widen<SCALE_BF16>((unsigned short)v[q]), widen<SCALE_BF16>((unsigned short)(v[q] >> 16)));
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) low[q] = pick(v[2 * q], v[2 * q + 1], 0x6420u), high[q] = pick(v[2 * q], v[2 * q + 1], 0x7531u);
}

// Scales and activations in one dtype: no table.  A code inside the mantissa of a magic number (128 in bf16, 1024 in fp16: its last
// place is one) is that number plus the code, or plus 16 times it: the published way to make 16-bit floats of small integers (Kim et al.,
// "Who Says Elephants Can't Run", 2022), here on words of three interleaved planes.  off, off16: -(magic + zero), -(magic / 16 + zero).
struct RowFactors {
  uint32_t off, off16, scale;
};
template <bool BF16>
__device__ __forceinline__ bool row_factors(uint32_t scale_bits, uint32_t zero, RowFactors& f) {
  f.off = zero * 0x10001u + (BF16 ? 0xc300c300u : 0xe400e400u);
  f.off16 = add2<BF16>(f.off, BF16 ? 0x42f042f0u : 0x63806380u);  // + 120, + 960
  f.scale = scale_bits * 0x10001u;
  return zero <= 100u;  // magic + zero has a last place of one
}

// 32 codes of a row (one word per plane, the high one inverted) -> 16 operand registers, inputs in order.  Nibble i of word j
// takes the code of input 4 i + j; bytes of two such words are put side by side.
template <bool BF16>
__device__ __forceinline__ void multiply(uint32_t p0, uint32_t p1, uint32_t p2, const RowFactors& f, uint32_t* to) {
  constexpr uint32_t kMagic = BF16 ? 0x43004300u : 0x64006400u, kSixteenth = BF16 ? 0x3d803d80u : 0x2c002c00u;
#pragma unroll
  for (int half = 0; half < 2; ++half) {  // inputs 4 i, 4 i + 1; 4 i + 2, 4 i + 3
    const uint32_t a = half ? p0 >> 2 : p0, b = half ? p1 >> 1 : p1 << 1, c = half ? p2 : p2 << 2;
    uint32_t even, odd;
    asm("lop3.b32 %0, %1, %2, %3, 0x72;" : "=r"(even) : "r"(blend(a, b, 0x11111111u)), "r"(c), "r"(0x44444444u));  // (a & ~m) | (~b & m)
    asm("lop3.b32 %0, %1, %2, %3, 0x72;" : "=r"(odd) : "r"(blend(a, b, 0x22222222u)), "r"(c), "r"(0x88888888u));
    odd >>= 1;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t w = pick(even, odd, 0x4400u + 0x1111u * k);
      uint32_t x0, x1;
      asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(x0) : "r"(w), "r"(0x00070007u), "n"(kMagic));  // (w & m) | magic
      asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(x1) : "r"(w), "r"(0x00700070u), "n"(kMagic));
      to[4 * k + half] = mul2<BF16>(add2<BF16>(x0, f.off), f.scale);
      to[4 * k + 2 + half] = mul2<BF16>(fma2<BF16>(x1, kSixteenth, f.off16), f.scale);
    }
  }
}

// TWO: both MMA warps issue.
template <bool SCALE_BF16, bool ACT_BF16, bool TWO>
__global__ void __launch_bounds__(kThreads, 1) w3_gemm_kernel(const __grid_constant__ GemmParams p) {
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char* const planes_s = smem + kBBytes;
  uint64_t* const bars = reinterpret_cast<uint64_t*>(planes_s + kPlaneStages * kPlaneStage);
  const uint32_t b_full = smem_u32(bars), b_empty = b_full + 8 * kMaxBStages;
  const uint32_t p_full = b_empty + 8 * kMaxBStages, p_empty = p_full + 8 * kPlaneStages;
  const uint32_t a_full = p_empty + 8 * kPlaneStages, a_empty = a_full + 8 * kASlots;
  const uint32_t d_full = a_empty + 8 * kASlots, d_empty = d_full + 8;
  uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(bars + kBars);
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);

  if (tid < kBars) {
    const int at = tid - 2 * kMaxBStages;
    const bool by_group = (at >= kPlaneStages && at < 2 * kPlaneStages + kASlots);  // p_empty, a_full: a dequantising warpgroup
    mbar_init(b_full + 8 * tid, tid == kBars - 1 ? 128 * kEpilogue : tid == kBars - 2 ? (TWO ? 2 : 1) : by_group ? 128 : 1);  // d_empty, d_full
    mbar_init_fence();
  }
  if (warp == 3) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen_before();
  __syncthreads();
  tcgen_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  const int G = p.G;
  const bool paired = p.b_stages == kASlots;
  bool dead = false;

  auto matrix_of = [&](int row_tile) {
    int j = 0;
    while (j + 1 < p.n && row_tile >= p.mats[j + 1].tile_begin) ++j;
    return j;
  };

  // What lies in x, the addends and the outputs belongs to the launches ahead; the weights do not.
  if (warp != 2) asm volatile("griddepcontrol.wait;" ::: "memory");

  if (warp == 0) {
    if (lane == 0) {
      unsigned stage = 0, phase = 0;
      bool first = true;  // round of the ring
      for (int tile = blockIdx.x; tile < p.tiles && !dead; tile += gridDim.x) {
        const int token0 = (tile % p.token_tiles) * p.tokens;
        for (int g = 0; g < G; ++g) {
          // with as many stages as operand slots the MMA's one commit of a group releases both
          if (!first && !mbar_wait_bounded((paired ? a_empty : b_empty) + 8 * stage, phase ^ 1u)) {
            dead = true;
            break;
          }
          mbar_expect_tx(b_full + 8 * stage, (uint32_t)p.tokens * 256u);
#pragma unroll
          for (int h = 0; h < 2; ++h)
            asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                             smem_u32(smem) + (uint32_t)((2 * stage + h) * p.tokens * 128)),
                         "l"(&p.x_map), "r"(g * 128 + h * 64), "r"(token0), "r"(b_full + 8 * stage)
                         : "memory");
          if (++stage == (unsigned)p.b_stages) stage = 0, phase ^= 1u, first = false;
        }
      }
    }
  } else if (warp == 2) {
    if (lane == 0) {
      unsigned step = 0;
      for (int tile = blockIdx.x; tile < p.tiles && !dead; tile += gridDim.x) {
        const int row_tile = tile / p.token_tiles, j = matrix_of(row_tile);
        const int unit = (row_tile - p.mats[j].tile_begin) * (kRows / 32);
        for (int g = 0; g < G; ++g, ++step) {
          const unsigned stage = step % kPlaneStages, use = step / kPlaneStages;
          if (use && !mbar_wait_bounded(p_empty + 8 * stage, (use - 1) & 1)) {
            dead = true;
            break;
          }
          mbar_expect_tx(p_full + 8 * stage, (uint32_t)kPlaneStage);
          asm volatile(
              "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
                  smem_u32(planes_s + stage * kPlaneStage)),
              "l"(&p.mats[j].plane_map), "r"(0), "r"(unit), "r"(3 * g), "r"(p_full + 8 * stage)
              : "memory");
        }
      }
    }
  } else if (warp == 1 || (TWO && warp == 3)) {
    // the whole warp walks the loop and one elected lane issues: operands known to be the same in all lanes go to the
    // tensor core's instructions as they are (issued from a lane's own branch, four of them took 480 clocks)
    // D fp32, A and B in the activation dtype, both K-major
    const uint32_t format = ACT_BF16 ? 1u : 0u;
    const uint32_t idesc = (1u << 4) | (format << 7) | (format << 10) | ((uint32_t)(p.tokens >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);
    // K-major, 128-byte swizzle: 8-row groups 1024 bytes apart; 16 inputs are 32 bytes of a row
    const uint64_t b_desc0 = (uint64_t)((smem_u32(smem) >> 4) & 0x3fffu) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
    // the groups of a tile that this warp takes: all, or every other one, on an accumulator that is its own
    constexpr int stride = TWO ? 2 : 1;
    const int first = TWO && warp == 3 ? 1 : 0;
    const uint32_t sums = tmem + (TWO && warp == 3 ? kMaxTokens / 2 : 0);
    unsigned step = 0, stage = 0, stage_phase = 0, it = 0;
    for (int tile = blockIdx.x; tile < p.tiles && !dead; tile += gridDim.x, ++it) {
      if (it && !__all_sync(0xffffffffu, mbar_wait_bounded(d_empty, (it - 1) & 1))) {
        dead = true;
        break;
      }
      if (TWO) step = it * G + first;
      for (int g = first; g < G; g += stride, step += stride) {
        const unsigned slot = step % kASlots, use = step / kASlots;
        if (TWO) stage = slot, stage_phase = use & 1;  // as many stages as slots
        // half of the lanes look at either barrier; a vote tells them that both have completed but orders no memory
        // between them, the __syncwarp does: the elected lane may then build on what the barrier of the others released
        const uint32_t full = lane & 1 ? a_full + 8 * slot : b_full + 8 * stage, parity = lane & 1 ? use & 1 : stage_phase;
        if (!__all_sync(0xffffffffu, mbar_try_wait(full, parity)) && !__all_sync(0xffffffffu, mbar_wait_bounded(full, parity))) {
          dead = true;
          break;
        }
        __syncwarp();
        tcgen_after();
        const uint64_t b_desc = b_desc0 + stage * (p.tokens * 16);
        const uint32_t a = tmem + kAColumn + slot * 64;
        const uint32_t a_done = a_empty + 8 * slot, b_done = b_empty + 8 * stage;
        // the elected lane's predicate sits on the instruction, not on a branch around it: operands stay uniform
        const uint32_t elect = elected() ? 1u : 0u, later = g > first ? 1u : 0u;
#pragma unroll
        for (int i = 0; i < 8; ++i)
          asm volatile(
              "{\n\t"
              ".reg .pred e, p;\n\t"
              "setp.ne.b32 e, %5, 0;\n\t"
              "setp.ne.b32 p, %4, 0;\n\t"
              "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
              "}\n" ::"r"(sums),
              "r"(a + 8 * i), "l"(b_desc + (i >> 2) * (p.tokens * 8) + 2 * (i & 3)), "r"(idesc), "r"(i ? 1u : later), "r"(elect)
              : "memory");
        if (elect) {
          commit(a_done);
          if (!TWO && !paired) commit(b_done);
          if (g + stride >= G) commit(d_full);
        }
        __syncwarp();
        if (!TWO && ++stage == (unsigned)p.b_stages) stage = 0, stage_phase ^= 1u;
      }
    }
  } else if (warp >= 4 && warp < 4 + 4 * kDequant) {
    const int group_of = (warp - 4) >> 2, row_in_tile = tid & 127;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    unsigned count = 0;  // groups of this CTA so far
    for (int tile = blockIdx.x; tile < p.tiles && !dead; tile += gridDim.x) {
      const int row_tile = tile / p.token_tiles, j = matrix_of(row_tile);
      const GemmMatrix& m = p.mats[j];
      const int row = (row_tile - m.tile_begin) * kRows + row_in_tile;
      // scale and zero point are requested one group of this warpgroup ahead; rows past O have weight zero
      uint32_t scale_next = 0, zero_next = 4;
      auto fetch = [&](int g) {
        scale_next = 0, zero_next = 4;
        if (row < m.O && g < G) {
          asm volatile("ld.global.nc.u16 %0, [%1];" : "=r"(scale_next) : "l"(m.scales + (size_t)g * m.O + row));
          if (m.zeros) asm volatile("ld.global.nc.u8 %0, [%1];" : "=r"(zero_next) : "l"(m.zeros + (size_t)g * m.O + row));
        }
      };
      int g = (int)((group_of - count) % kDequant);  // the warpgroups take turns, across tiles too
      fetch(g);
      for (; g < G; g += kDequant) {
        const unsigned at = count + g, stage = at % kPlaneStages;
        const uint32_t scale_bits = scale_next, zero = zero_next;
        fetch(g + kDequant);
        RowFactors factors;
        // one row of the warp that the short form does not cover sends it to the table
        const bool table = SCALE_BF16 != ACT_BF16 || !__all_sync(0xffffffffu, row_factors<ACT_BF16>(scale_bits, zero, factors));
        uint32_t low[2], high[2];
        if (table) value_table<SCALE_BF16, ACT_BF16>(scale_bits, zero, low, high);
        if (!__all_sync(0xffffffffu, mbar_wait_bounded(p_full + 8 * stage, (at / kPlaneStages) & 1))) {
          dead = true;
          break;
        }
        const uint4* const from = reinterpret_cast<const uint4*>(planes_s + stage * kPlaneStage) + row_in_tile;
        const uint4 w0 = from[0], w1 = from[kRows], w2 = from[2 * kRows];
        arrive(p_empty + 8 * stage);
        const unsigned slot = at % kASlots, use = at / kASlots;
        bool late = false;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t v[32];
          if (table) {
            look_up(h ? w0.z : w0.x, h ? w1.z : w1.x, h ? w2.z : w2.x, low, high, v);
            look_up(h ? w0.w : w0.y, h ? w1.w : w1.y, h ? w2.w : w2.y, low, high, v + 16);
          } else {
            multiply<ACT_BF16>(h ? w0.z : w0.x, h ? w1.z : w1.x, h ? w2.z : w2.x, factors, v);
            multiply<ACT_BF16>(h ? w0.w : w0.y, h ? w1.w : w1.y, h ? w2.w : w2.y, factors, v + 16);
          }
          if (h == 0) {
            late = use && !__all_sync(0xffffffffu, mbar_wait_bounded(a_empty + 8 * slot, (use - 1) & 1));
            if (late) break;
            tcgen_after();
          }
          tmem_store32(tmem + lanes + kAColumn + slot * 64 + h * 32, v);
        }
        if (late) {
          dead = true;
          break;
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tcgen_before();
        arrive(a_full + 8 * slot);
      }
      count += G;
    }
  } else if (warp >= 4 + 4 * kDequant) {
    const int row_in_tile = tid & 127, part = (warp - 4 - 4 * kDequant) >> 2;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    unsigned it = 0;
    for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x, ++it) {
      const int row_tile = tile / p.token_tiles, j = matrix_of(row_tile);
      const GemmMatrix& m = p.mats[j];
      const int row = (row_tile - m.tile_begin) * kRows + row_in_tile, token0 = (tile - row_tile * p.token_tiles) * p.tokens;
      const int tokens = min(p.tokens, p.T - token0);
      // addends are requested 16 tokens ahead, the first ones while the tile still accumulates
      unsigned short next[16];
      auto fetch = [&](int c) {
        if (!m.addend || row >= m.O) return;
        const unsigned short* from = m.addend + (size_t)(token0 + c) * p.ldo + row;
#pragma unroll
        for (int i = 0; i < 16; ++i, from += p.ldo)
          if (c + i < tokens) next[i] = *from;
      };
      fetch(16 * part);
      if (!__all_sync(0xffffffffu, mbar_wait_bounded(d_full, it & 1))) {
        dead = true;
        break;
      }
      tcgen_after();
      for (int c = 16 * part; c < tokens; c += 16 * kEpilogue) {
        uint32_t v[16];
        __syncwarp();
        tmem_load16(tmem + lanes + c, v);
        if (TWO) {
          uint32_t w[16];
          tmem_load16(tmem + lanes + kMaxTokens / 2 + c, w);
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) + __uint_as_float(w[i]));
        }
        if (m.addend) {
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) + widen<ACT_BF16>(next[i]));
          fetch(c + 16 * kEpilogue);
        }
        if (row < m.O) {
          unsigned short* to = m.out + (size_t)(token0 + c) * p.ldo + row;
#pragma unroll
          for (int i = 0; i < 16; ++i, to += p.ldo)
            if (c + i < tokens) *to = (unsigned short)pack2<ACT_BF16>(__uint_as_float(v[i]), 0.f);
        }
      }
      __syncwarp();
      tcgen_before();
      arrive(d_empty);
    }
  }
  if (dead) atomicExch(p.status, 3u);
  __syncwarp();
  tcgen_before();
  __syncthreads();
  tcgen_after();
  if (warp == 3) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

// Tokens of a tile: the tiles go round the SMs, and a round costs 190 + tokens.  Too steep a line for small tiles, but of the splits that fit it picks
// the best in all of eleven shapes from 2560 x 2560 to 25600 x 5120 at 100 to 700 tokens, with scales of either dtype (333 of 12288 x 4096: 112
// tokens 33.2 us, 176 39.0, 96 45.9; 512 of 6144 x 4096: 176 21.5, 256 25.6, 96 31.3; 512 of 24576 x 4096: 256 76.4, 176 79.7).
int token_tile(int T, int row_tiles, int sms) {
  int best = 0;
  long long best_cost = 0;
  const int fewest = (T + kMaxTokens - 1) / kMaxTokens;
  for (int n = fewest; n <= fewest + 12; ++n) {
    const int tokens = ((T + n - 1) / n + 15) / 16 * 16;
    const long long tiles = (long long)row_tiles * ((T + tokens - 1) / tokens), cost = (tiles + sms - 1) / sms * (190 + tokens);
    if (!best || cost < best_cost) best = tokens, best_cost = cost;
  }
  return best;
}

template <bool SCALE_BF16, bool ACT_BF16, bool TWO>
int launch(const GemmParams& p, int grid, cudaStream_t stream) {
  static std::mutex lock;
  static bool ready[64] = {};
  int device = 0;
  if (cudaError_t err = cudaGetDevice(&device); err != cudaSuccess) return cuda_fail(err, "cudaGetDevice");
  if (device < 0 || device >= 64) return fail(FB_ELIMIT, "device ordinal %d outside 0..63", device);
  {
    std::lock_guard<std::mutex> guard(lock);
    if (!ready[device]) {
      if (cudaError_t err = cudaFuncSetAttribute(w3_gemm_kernel<SCALE_BF16, ACT_BF16, TWO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem); err != cudaSuccess)
        return cuda_fail(err, "cudaFuncSetAttribute(w3_gemm_kernel)");
      ready[device] = true;
    }
  }
  return launch_pdl(w3_gemm_kernel<SCALE_BF16, ACT_BF16, TWO>, dim3(grid), dim3(kThreads), kSmem, stream, "w3_gemm_kernel launch", p);
}

}  // namespace

extern "C" int fb_w3_gemm(const void* x, int act_dtype, int tokens, const fb_w3_matrix_t* mats, int n_mats, int scale_dtype, int in_features, int out_stride,
                          void* scratch, size_t scratch_bytes, fb_stream_t stream) {
  if (!x || !mats) return fail(FB_EINVAL, "fb_w3_gemm: null pointer");
  if (n_mats < 1 || n_mats > kMaxMats) return fail(FB_ELIMIT, "fb_w3_gemm: %d matrices outside 1..%d", n_mats, kMaxMats);
  if ((act_dtype != FB_F16 && act_dtype != FB_BF16) || (scale_dtype != FB_F16 && scale_dtype != FB_BF16))
    return fail(FB_EINVAL, "fb_w3_gemm: dtype tags must be FB_F16 or FB_BF16");
  if (tokens < 1 || in_features < 128 || in_features % 128 || in_features / 128 > 255)
    return fail(FB_ELIMIT, "fb_w3_gemm: T=%d, K=%d: K must be a multiple of 128 with at most 255 groups", tokens, in_features);
  if (!aligned(x, 16)) return fail(FB_EINVAL, "fb_w3_gemm: x must be 16-byte aligned");
  if (!scratch || scratch_bytes < 256 || !aligned(scratch, 4)) return fail(FB_ESCRATCH, "fb_w3_gemm: scratch of 256 bytes needed, %zu given", scratch_bytes);
  const DeviceInfo* info = device_info();
  if (!info) return FB_ECUDA;
  if (kSmem > (size_t)info->max_smem_optin) return fail(FB_ELIMIT, "fb_w3_gemm: needs %zu bytes of shared memory", kSmem);
  GemmParams p;
  p.n = n_mats, p.T = tokens, p.G = in_features / 128, p.ldo = out_stride;
  p.status = static_cast<unsigned*>(scratch);
  int row_tiles = 0;
  for (int j = 0; j < n_mats; ++j) {
    const fb_w3_matrix_t& in = mats[j];
    if (!in.planes || !in.scales || !in.out) return fail(FB_EINVAL, "fb_w3_gemm: planes, scales and out must be non-null");
    if (in.out_features < 32 || in.out_features > 65536 || in.out_features % 32) return fail(FB_ELIMIT, "fb_w3_gemm: O=%d must be a multiple of 32 in 32..65536", in.out_features);
    if (out_stride < in.out_features) return fail(FB_EINVAL, "fb_w3_gemm: rows of out are %d apart, %d long", out_stride, in.out_features);
    if (!aligned(in.planes, 16) || !aligned(in.scales, 2) || !aligned(in.out, 2) || !aligned(in.residual, 2))
      return fail(FB_EINVAL, "fb_w3_gemm: planes must be 16-byte aligned, 16-bit tensors 2-byte aligned");
    const size_t out_bytes = ((size_t)(tokens - 1) * out_stride + in.out_features) * 2;
    if (overlaps(in.out, out_bytes, x, (size_t)tokens * in_features * 2)) return fail(FB_EALIAS, "fb_w3_gemm: out overlaps x");
    GemmMatrix& m = p.mats[j];
    if (!plane_tensor_map(in.planes, in.out_features, p.G, 32, kRows / 32, 3, &m.plane_map)) return FB_ECUDA;
    m.scales = static_cast<const unsigned short*>(in.scales), m.zeros = in.zeros;
    m.out = static_cast<unsigned short*>(in.out), m.addend = static_cast<const unsigned short*>(in.residual);
    m.O = in.out_features, m.tile_begin = row_tiles;
    row_tiles += (in.out_features + kRows - 1) / kRows;
  }
  p.tokens = token_tile(tokens, row_tiles, info->sm_count);
  p.token_tiles = (tokens + p.tokens - 1) / p.tokens;
  p.tiles = row_tiles * p.token_tiles;
  p.b_stages = kBBytes / (p.tokens * 256);
  if (p.b_stages > kMaxBStages) p.b_stages = kMaxBStages;
  if (!activation_tensor_map(x, tokens, in_features, p.tokens, &p.x_map)) return FB_ECUDA;

  const int grid = p.tiles < info->sm_count ? p.tiles : info->sm_count;
  const cudaStream_t on = static_cast<cudaStream_t>(stream);
  // two issuers where two accumulators fit and there are as many activation stages as operand slots
#define FB_LAUNCH(SCALE_BF16, ACT_BF16) \
  (p.tokens <= kMaxTokens / 2 && p.G > 1 ? launch<SCALE_BF16, ACT_BF16, true>(p, grid, on) : launch<SCALE_BF16, ACT_BF16, false>(p, grid, on))
  if (scale_dtype == FB_BF16) return act_dtype == FB_BF16 ? FB_LAUNCH(true, true) : FB_LAUNCH(true, false);
  return act_dtype == FB_BF16 ? FB_LAUNCH(false, true) : FB_LAUNCH(false, false);
#undef FB_LAUNCH
}
