// GPTQ W3 group-128 planar matrix times 1..16 activation rows (small batches, drafts, short prompts).
//
// HBM-bound byte work as for one row (fb_w3_gemv.cu), and the tables of that kernel grow with the rows; here the
// cost per weight hardly does.  What bounds it: turning three bit planes into operands (integer
// instructions), and at small sizes the chain launch - activations - weights - sums.  A form on
// tcgen05.mma needs its operand in shared memory: expanding the weights into it took 3300 instructions and
// as many shared-memory wavefronts per 128 x 128 tile.  This one takes no trip through shared memory.
// us on a B200, cold weights (before: tcgen05 form from five rows on, tables below), at 4 / 16 rows:
// 1024 x 4096 3.6 / 4.3 (8.3 / 10.5), 4096 x 4096 5.5 / 6.8 (10.1 / 11.4), 12288 x 4096 11.0 / 13.4 (22.4 / 22.5),
// 4096 x 12288 11.5 / 14.4 (24.7 / 22.5).
//
//  * The three planes of a group become operands of mma.sync.m16n8k16 in registers, without a table.  Two
//    bit-selects per word interleave them into 3-bit fields; a field inside the ten mantissa bits of an
//    fp16 IS the number code * 2^(b - 24), b = 0..7 its first bit, and one fma on a pair of them makes
//    (code - zero) * 2^-9: exact, and normal (the tensor cores keep the leading zeros of a subnormal
//    operand when they align products, which would cost the sums eight bits).  The K order inside a group is
//    free, so a lane's 32-bit plane word is its share of a row as it is.
//  * Activations are scaled per (group, row) by a power of two into fp16: the largest magnitude goes to
//    [2^14, 2^15), every bit of a bf16 down to 2^-21 of it survives (fp16: 2^-18), what is smaller is
//    rounded to 2^-39 of it, below the fp32 rounding of the sums.  An activation that dwarfs the rest of its
//    group (above 2^11 times their sum) or is not finite stays out of the MMA and is added in fp32 where
//    its signed code is not zero (one per group and row; a second one that is not finite makes the group's sums
//    NaN).  Finite activations of any size stay finite as long as the products with the weights do.
//  * Scales are applied per group in fp32: weights are never rounded.
//  * A cluster owns a slice of the output rows, its CTAs split K between them (four pairs of groups each
//    where there are enough: the activations of a CTA are converted once and stay in shared memory).  The
//    (32 rows x 2 groups) tasks of a CTA are dealt to its sixteen warps in contiguous, equally long runs;
//    a warp stages them through a private ring (tiled TMA copies, one mbarrier per slot) and puts its sums
//    down once per row unit it touches.  These are added up in ascending order, first over the warps,
//    then, through distributed shared memory (stores that count themselves in at the receiving
//    CTA), over the CTAs: no atomics, no barrier between units.
//  * The first staged items go out before griddepcontrol.wait, the rest of the ring behind the activations'
//    loads: a whole ring's requests ahead of those delay them by more than the early start is worth.
//  * A row's result does not depend on its neighbours: the plan does not look at the number of rows, so the
//    same sums are taken in the same order.
//
// The reference has no packed path for more than one row (csrc/w3_lut.cu:195); its dense fallback
// (w3_lut_deployment.py:343-359) is the oracle.  Scales, zero points and the rounding correction of the
// dequantised-weight arithmetic as in fb_w3_gemv.cu.
#include <mutex>
#include <new>

#include "fb_common.cuh"

namespace {

using namespace fb;

constexpr int kTileRows = 16;
constexpr int kTiles = 2;  // row tiles of a task: the operands of the activations are read once for both
constexpr int kUnitRows = kTiles * kTileRows;
constexpr int kRun = kTileRows * 16;  // 256 B: one plane of one group for a tile
constexpr int kWarps = 16;
constexpr int kThreads = kWarps * 32;
constexpr int kStages = 2;
constexpr int kMaxRows = 16;
constexpr int kMaxSplits = 8;  // CTAs of a cluster
constexpr int kSplitPairs = 4;
constexpr int kOperandBytes = 256;  // operands of one (group, row)

// A ring slot holds a task: planes [group][plane][tile][256 B], scales [group][row], zero points.
constexpr int kSlotPlanes = 6 * kTiles * kRun;
constexpr int kSlotZeros = kSlotPlanes + 128;
constexpr int kSlotBytes = kSlotZeros + 128;

struct RowsParams {
  alignas(64) CUtensorMap plane_map;  // planes as uint32 [G*3][O/16][64], box = the 256-byte runs of a task; groups beyond G read as zero
  CUtensorMap scale_map, zero_map;    // [G][O], box = the rows of a task x 2 groups
  const void* x;
  const int16_t* perm;
  void* out;
  const void* addend;  // [M, O], added in fp32 before the result is rounded; or null
  unsigned* status;
  const unsigned short* scales;  // for tensors that are not on a 16-byte boundary: no tiled copies of them
  const uint8_t* zero_points;
  int M, O, K, G;
  int act_dtype, scale_dtype, zeros;
  int direct;  // 1: scales and zero points do not come by tiled copies; 2: the column order is not aligned either
  int npairs, pairs_few, pairs_extra;  // pairs of groups: most and fewest of a CTA; CTAs of a cluster that have one more
  int units_few, units_extra;          // row units of a cluster likewise
  int batch;                           // most units between two cluster barriers
  unsigned rows_inv, pairs_inv, pairs_few_inv, splits_inv;  // ceil(2^16 / M) and so on: divisions of small numbers
  int out_aligned;     // outputs can be stored eight bytes at a time
};

__device__ __forceinline__ uint32_t lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ uint32_t lds8(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
template <int LUT>
__device__ __forceinline__ uint32_t lop3(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, %4;" : "=r"(d) : "r"(a), "r"(b), "r"(c), "n"(LUT));
  return d;
}
constexpr int kSelect = 0xE4;     // (a & c) | (b & ~c)
constexpr int kSelectNot = 0x72;  // (a & ~c) | (~b & c)

__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void mma16816_first(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t fma2(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

// Three plane words of one row (32 codes), interleaved: word 3 h + s holds the codes of input positions
// 8 h + b, b = s, s + 3, s + 6 below eight, at bits b, b + 1, b + 2 of each half (low half: positions
// 0..15, high half: 16..31).
__device__ __forceinline__ void interleave_codes(uint32_t p0, uint32_t p1, uint32_t p2, uint32_t (&t)[6]) {
  constexpr uint32_t first[3] = {0x00490049u, 0x00920092u, 0x00240024u};
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t a = h ? p0 >> 8 : p0, b = h ? p1 >> 7 : p1 << 1, c = h ? p2 >> 6 : p2 << 2;
#pragma unroll
    for (int s = 0; s < 3; ++s) t[3 * h + s] = lop3<kSelectNot>(lop3<kSelect>(a, b, first[s]), c, first[s] << 2);  // the high plane is stored inverted
  }
}

// Operand register r: (code - zero) * 2^-9 of input positions r and r + 16.
__device__ __forceinline__ uint32_t weight(const uint32_t (&t)[6], int r, uint32_t minus_zero) {
  const int b = r & 7;
  return fma2(t[3 * (r >> 3) + b % 3] & (0x00070007u << b), (uint32_t)(30 - b) * 0x04000400u, minus_zero);  // 2^(15 - b)
}

// An activation kept out of the MMA: its position in the group (-1: none) and its value.
struct Outlier {
  int k;
  float x;
};

// NT: column tiles of eight activation rows.
template <int NT, bool GATHER>
__global__ void __launch_bounds__(kThreads, 1) w3_rows_kernel(const __grid_constant__ RowsParams p) {
  extern __shared__ __align__(1024) unsigned char smem[];
  // the warp index through a shuffle: the compiler then knows that it is the same in all lanes
  const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const int gid = lane >> 2, tig = lane & 3, M = p.M;

  // ---- the cluster's row units [unit0, unit0 + count), this CTA's pairs of groups [pair0, pair0 + np) ----
  const int rank = (int)blockIdx.x, splits = (int)gridDim.x;
  const int pair0 = rank * p.pairs_few + min(rank, p.pairs_extra), np = p.pairs_few + (rank < p.pairs_extra ? 1 : 0);
  const int slice = (int)blockIdx.y, unit0 = slice * p.units_few + min(slice, p.units_extra), count = p.units_few + (slice < p.units_extra ? 1 : 0);
  const unsigned np_inv = np == p.npairs ? p.pairs_inv : p.pairs_few_inv;
  const int ng = 2 * np;  // groups, the last one possibly beyond G (zeros)

  // ---- shared memory: rings | operands | 2^ex | outliers | sums of the warps |
  // sums of the cluster's CTAs | barriers ----
  const int quarter = 8 * M;  // sums of eight rows: [activation row][8]
  unsigned char* const operands = smem + kWarps * kStages * kSlotBytes;
  float* const stat = reinterpret_cast<float*>(operands + 2 * p.npairs * M * kOperandBytes);  // [group][row]: 2^(ex - 5); rows padded to 8 NT
  Outlier* const outliers = reinterpret_cast<Outlier*>(stat + 2 * p.npairs * 8 * NT);
  float* const part = reinterpret_cast<float*>(outliers + 2 * p.npairs * M);  // slot (unit + warp): four quarters
  float* const inbox = part + (p.batch + kWarps - 1) * 4 * quarter;          // [quarter of this CTA][sender][quarter]
  uint64_t* const bars = reinterpret_cast<uint64_t*>(inbox + (4 * p.batch + splits) * quarter);
  const uint32_t inbox_bar = smem_u32(bars + kWarps * kStages);
  uchar2* const span = reinterpret_cast<uchar2*>(bars + kWarps * kStages + 1);  // per unit: the first and the last warp of its tasks
  const uint32_t ring_u32 = smem_u32(smem) + (uint32_t)(warp * kStages * kSlotBytes), bars_u32 = smem_u32(bars) + (uint32_t)(warp * kStages * 8);
  const uint32_t operands_u32 = smem_u32(operands);

  if (lane == 0) {
    if (warp == 0) mbar_init(inbox_bar, 1);
    for (int s = 0; s < kStages; ++s) mbar_init(bars_u32 + s * 8, 1);
    mbar_init_fence();
  }
  __syncwarp();
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");  // waited for before the first store into another CTA's shared memory

  // ---- tasks of a batch of units, unit-major: every warp has an equally long run (of at most one where there are few) ----
  auto run_of = [&](int units, int& t0, int& t1) {
    const int tasks = units * np;
    t0 = tasks < kWarps ? min(warp, tasks) : warp * tasks / kWarps, t1 = tasks < kWarps ? min(warp + 1, tasks) : (warp + 1) * tasks / kWarps;
  };
  auto unit_of = [&](int t) { return (int)((unsigned)t * np_inv >> 16); };
  // staging: lane 0 requests the planes, scales and zero points of this warp's tasks in order, each into the slot that
  // was read last
  int pf_first = -p.batch, pf_unit = 0, pf_pair = 0, pf_left = 0;
  auto pf_next_batch = [&]() {
    while (pf_left == 0 && pf_first + p.batch < count) {
      pf_first += p.batch;
      int t0, t1;
      run_of(min(p.batch, count - pf_first), t0, t1);
      pf_left = t1 - t0, pf_unit = unit_of(t0), pf_pair = t0 - pf_unit * np, pf_unit += pf_first;
    }
  };
  auto issue_next = [&](uint32_t dst, uint32_t bar) {
    const int g = 2 * (pair0 + pf_pair), unit = unit0 + pf_unit;
    if (p.direct) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const size_t at = (size_t)(g + i) * p.O + unit * kUnitRows + lane;
        const uint32_t scale = g + i < p.G ? p.scales[at] : 0u, zero = g + i < p.G && p.zeros ? p.zero_points[at] : 4u;
        asm volatile("st.shared.u16 [%0], %1;" ::"r"(dst + (uint32_t)(kSlotPlanes + (i * kUnitRows + lane) * 2)), "h"((unsigned short)scale) : "memory");
        asm volatile("st.shared.u8 [%0], %1;" ::"r"(dst + (uint32_t)(kSlotZeros + i * kUnitRows + lane)), "r"(zero) : "memory");
      }
      __syncwarp();
    }
    if (lane == 0) {
      mbar_expect_tx(bar, (uint32_t)(kSlotPlanes + (p.direct ? 0 : 4 * kUnitRows + (p.zeros ? 2 * kUnitRows : 0))));  // boxes are whole: what lies beyond G reads as zero
      asm volatile(
          "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
          "l"(&p.plane_map), "r"(0), "r"(unit * kTiles), "r"(3 * g), "r"(bar)
          : "memory");
      if (!p.direct)
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                         dst + (uint32_t)kSlotPlanes),
                   "l"(&p.scale_map), "r"(unit * kUnitRows), "r"(g), "r"(bar)
                   : "memory");
      if (p.zeros && !p.direct)
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                         dst + (uint32_t)kSlotZeros),
                     "l"(&p.zero_map), "r"(unit * kUnitRows), "r"(g), "r"(bar)
                     : "memory");
    }
    if (++pf_pair == np) pf_pair = 0, ++pf_unit;
    if (--pf_left == 0) pf_next_batch();
  };
  if (!p.zeros) {  // they are 4, and none are staged
    for (int s = 0; s < kStages; ++s)
      if (lane < kUnitRows / 2)
        asm volatile("st.shared.u32 [%0], %1;" ::"r"(ring_u32 + (uint32_t)(s * kSlotBytes + kSlotZeros + 4 * lane)), "r"(0x04040404u) : "memory");
    __syncwarp();
  }
  pf_next_batch();
  if (pf_left) issue_next(ring_u32, bars_u32);

  // ---- activations -> operands, eight threads per (group, row): thread (t, h) owns inputs 32 t + 8 h .. + 7 and the same
  // + 16, which are eight operand words (low half: first, high half: second) ----
  const int items_x = ng * M;
  const int k_in_group = (((int)threadIdx.x >> 1) & 3) * 32 + ((int)threadIdx.x & 1) * 8;
  // Through a column order row by row: the values that a CTA gathers of a row share sectors (four a sector at a quarter of 4096
  // inputs), which the L1 holds for a few rows but not for sixteen.  us, cold, in a graph, group by group / row by row, 16 rows: 1024x4096
  // 15.7 / 8.9, 4096x4096 15.9 / 11.6, 12288x4096 27.0 / 22.6, 4096x12288 38.2 / 33.9; 4 rows 4096x4096 7.2 / 6.8.  In identity order the rows
  // of a group come first: 2048x2048 at 16 rows 4.17 / 4.28, 4096x4096 6.71 / 6.59.
  auto locate = [&](int i, int& g, int& m) {
    if (GATHER)
      m = (int)((unsigned)(i >> 1) * np_inv >> 16), g = i - m * ng;
    else
      g = (int)((unsigned)i * p.rows_inv >> 16), m = i - g * M;
  };
  uint4 idx_lo = make_uint4(0u, 0u, 0u, 0u), idx_hi = idx_lo, raw_lo = idx_lo, raw_hi = idx_lo;
  auto fetch_idx = [&](int i) {  // the column order is part of the weights: no wait
    int g, m;
    locate(i, g, m);
    const int k = (2 * pair0 + g) * 128 + k_in_group;
    if (i < items_x && k < p.K) {
      if (p.direct > 1) {
        auto two = [&](int at) { return (uint32_t)(unsigned short)p.perm[k + at] | (uint32_t)(unsigned short)p.perm[k + at + 1] << 16; };
        idx_lo = make_uint4(two(0), two(2), two(4), two(6)), idx_hi = make_uint4(two(16), two(18), two(20), two(22));
      } else {
        idx_lo = *reinterpret_cast<const uint4*>(p.perm + k), idx_hi = *reinterpret_cast<const uint4*>(p.perm + k + 16);
      }
    }
  };
  auto fetch = [&](int i) {
    int g, m;
    locate(i, g, m);
    const int k = (2 * pair0 + g) * 128 + k_in_group;
    raw_lo = raw_hi = make_uint4(0u, 0u, 0u, 0u);
    if (i < items_x && k < p.K) {
      const unsigned short* const row = reinterpret_cast<const unsigned short*>(p.x) + (size_t)m * p.K;
      if (GATHER) {
        auto two = [&](uint32_t w) { return (uint32_t)row[w & 0xffffu] | (uint32_t)row[w >> 16] << 16; };
        raw_lo = make_uint4(two(idx_lo.x), two(idx_lo.y), two(idx_lo.z), two(idx_lo.w));
        raw_hi = make_uint4(two(idx_hi.x), two(idx_hi.y), two(idx_hi.z), two(idx_hi.w));
      } else {
        raw_lo = *reinterpret_cast<const uint4*>(row + k);
        raw_hi = *reinterpret_cast<const uint4*>(row + k + 16);
      }
    }
  };
  const int item0 = (int)threadIdx.x >> 3;
  constexpr int kItemStep = kThreads / 8;
  if (GATHER) fetch_idx(item0);

  // Everything below reads activations and writes outputs of this stream.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  fetch(item0);
  if (pf_left) issue_next(ring_u32 + (uint32_t)kSlotBytes, bars_u32 + 8u);

  int any_out = 0;
#pragma unroll 1
  for (int base = 0; base < items_x; base += kItemStep) {
    const int i = base + item0;
    const uint32_t words[8] = {raw_lo.x, raw_lo.y, raw_lo.z, raw_lo.w, raw_hi.x, raw_hi.y, raw_hi.z, raw_hi.w};
    if (base + kItemStep < items_x) {  // the next pass's loads fly while this one is converted
      if (GATHER) fetch_idx(i + kItemStep);
      fetch(i + kItemStep);
    }
    float v[16];  // inputs k .. k + 7, k + 16 .. k + 23
    if (p.act_dtype == FB_BF16) {
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = __uint_as_float((j & 1) ? words[j >> 1] & 0xffff0000u : words[j >> 1] << 16);
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = __half2float(__ushort_as_half((unsigned short)(words[j >> 1] >> (16 * (j & 1)))));
    }
    int g, m;
    locate(i, g, m);
    const bool live = i < items_x;
    // statistics over the eight threads of a (group, row)
    float top = 0.f, sum = 0.f;  // the sum in units of 2^8: 128 finite values do not overflow it
#pragma unroll
    for (int j = 0; j < 16; ++j) top = fmaxf(top, fabsf(v[j])), sum = fmaf(fabsf(v[j]), 0.00390625f, sum);
    float all_top = top, all_sum = sum;
#pragma unroll
    for (int d = 4; d >= 1; d >>= 1) all_top = fmaxf(all_top, __shfl_xor_sync(0xffffffffu, all_top, d)), all_sum += __shfl_xor_sync(0xffffffffu, all_sum, d);
    const float rest = all_sum - all_top * 0.00390625f;
    const bool wild = !(all_sum <= 3.4028235e38f);  // infinities, NaN
    // 2^-11 of the largest; a rest of zero may be one that the sum's rounding swallowed
    const bool ours = wild || rest < all_top * 1.9073486e-6f;
    bool lost = false;
    if (live && (lane & 7) == 0) outliers[g * M + m].k = -1;
    if (__any_sync(0xffffffffu, ours)) {  // rare
      __syncwarp();
      int large = 0, nonzero = 0;  // one value by itself needs no separate sum: nothing is rounded beside it
#pragma unroll
      for (int j = 0; j < 16; ++j) nonzero += v[j] != 0.f;
#pragma unroll
      for (int d = 4; d >= 1; d >>= 1) nonzero += __shfl_xor_sync(0xffffffffu, nonzero, d);
      top = 0.f;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const bool out = ours && (wild || nonzero > 1) && (wild ? !(fabsf(v[j]) <= 3.4028235e38f) : fabsf(v[j]) == all_top);
        if (out) {
          ++large;
          if (live) outliers[g * M + m].k = k_in_group + (j & 7) + (j >> 3) * 16, outliers[g * M + m].x = v[j], any_out = 1;
          v[j] = 0.f;
        }
        top = fmaxf(top, fabsf(v[j]));
      }
      all_top = top;
#pragma unroll
      for (int d = 4; d >= 1; d >>= 1) all_top = fmaxf(all_top, __shfl_xor_sync(0xffffffffu, all_top, d)), large += __shfl_xor_sync(0xffffffffu, large, d);
      lost = large > 1;
    }
    const int ex = max(-112, (int)(__float_as_uint(all_top) >> 23) - 127);
    if (live) {
      const float one = __uint_as_float((uint32_t)(141 - ex) << 23);  // 2^(14 - ex)
      uint32_t word[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(word[j]) : "f"(v[8 + j] * one), "f"(v[j] * one));
      // operand words of (group, row): [chunk of four][row][lane of a row]
      const uint32_t at = operands_u32 + (uint32_t)(((g * 4 + 2 * (lane & 1)) * M + m) * 64 + (k_in_group >> 5) * 16);
#pragma unroll
      for (int j = 0; j < 2; ++j)
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at + (uint32_t)(j * M * 64)), "r"(word[4 * j]), "r"(word[4 * j + 1]), "r"(word[4 * j + 2]),
                     "r"(word[4 * j + 3])
                     : "memory");
      if ((lane & 7) == 0) stat[g * 8 * NT + m] = lost ? __int_as_float(0x7fc00000) : __uint_as_float((uint32_t)(122 + ex) << 23);
    }
  }
  const bool has_outliers = __syncthreads_or(any_out) != 0;

  // the operand words of this lane's columns; columns beyond M repeat the last row
  uint32_t col_u32[NT];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) col_u32[nt] = operands_u32 + (uint32_t)(min(nt * 8 + gid, M - 1) * 64 + tig * 16);
  auto load_b = [&](int g, int nt, int c, uint32_t (&b)[4]) {
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3])
                 : "r"(col_u32[nt] + (uint32_t)((g * 4 + c) * M * 64)));
  };

  const bool scale_bf16 = p.scale_dtype == FB_BF16;
  uint32_t sa = ring_u32, bar = bars_u32, phase = 0;  // the slot at hand
  bool dead = false;
  float acc[kTiles][NT][4];
  // fp32 terms of the activations kept out of the MMA (rare): those of group g of the task at `sa`
  auto add_outliers = [&](int pair, int g) {
    for (int m = 0; m < M; ++m) {
      const Outlier o = outliers[(2 * pair + g) * M + m];
      if (o.k < 0) continue;
#pragma unroll
      for (int t = 0; t < kTiles; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t row = (uint32_t)(t * kTileRows + h * 8 + gid);
          const uint32_t at = sa + (uint32_t)(g * 3 * kTiles * kRun + (o.k >> 5) * 4) + row * 16u;
          const int bit = o.k & 31, zero = (int)lds8(sa + (uint32_t)(kSlotZeros + g * kUnitRows) + row);
          const int code = (int)((lds32(at) >> bit) & 1u) + 2 * (int)((lds32(at + kTiles * kRun) >> bit) & 1u) + 4 - 4 * (int)((lds32(at + 2 * kTiles * kRun) >> bit) & 1u) - zero;
          const uint32_t bits = lds16(sa + (uint32_t)(kSlotPlanes + g * 2 * kUnitRows) + row * 2u);
          const float term = code != 0 ? (float)code * bits_to_float((unsigned short)bits, p.scale_dtype) * o.x : 0.f;
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int c = 0; c < 2; ++c)
              if (m == nt * 8 + 2 * tig + c) acc[t][nt][2 * h + c] += term;
        }
    }
  };

  uint32_t inbox_phase = 0;
#pragma unroll 1
  for (int first = 0; first < count; first += p.batch) {
    const int units = min(p.batch, count - first);
    if (threadIdx.x == 0)  // the quarters that this CTA writes, from every CTA
      mbar_expect_tx(inbox_bar, ((unsigned)(4 * units - rank + splits - 1) * p.splits_inv >> 16) * (unsigned)(splits * quarter * 4));
    int t, t1;
    run_of(units, t, t1);
    int unit = unit_of(t), pair = t - unit * np;
    bool fresh = true;
#pragma unroll 1
    for (; t < t1; ++t) {
      if (!__all_sync(0xffffffffu, mbar_try_wait(bar, phase))) {
        if (dead || !__all_sync(0xffffffffu, mbar_wait_bounded(bar, phase))) {
          if (lane == 0) atomicExch(p.status, 1u);  // the copy never landed: give up, keep the barriers
          dead = true;
          break;
        }
      }
      if (fresh) {
#pragma unroll
        for (int tile = 0; tile < kTiles; ++tile)
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[tile][nt][q] = 0.f;
        fresh = false;
      }
      const uint32_t wa = sa + (uint32_t)(lane * 4);
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        const int gl = 2 * pair + g;
        float d[kTiles][NT][4];
        uint32_t ta[kTiles][6], tb[kTiles][6], za[kTiles], zb[kTiles];
#pragma unroll
        for (int tile = 0; tile < kTiles; ++tile) {
          uint32_t w[2][3];  // [row gid / gid + 8][plane]
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int pl = 0; pl < 3; ++pl) w[h][pl] = lds32(wa + (uint32_t)(((g * 3 + pl) * kTiles + tile) * kRun + h * 128));
          interleave_codes(w[0][0], w[0][1], w[0][2], ta[tile]);
          interleave_codes(w[1][0], w[1][1], w[1][2], tb[tile]);
          // a zero point in both halves is the subnormal z * 2^-24
          const uint32_t zero_at = sa + (uint32_t)(kSlotZeros + g * kUnitRows + tile * kTileRows + gid);
          za[tile] = fma2(lds8(zero_at) * 0x10001u, 0xf800f800u, 0u), zb[tile] = fma2(lds8(zero_at + 8u) * 0x10001u, 0xf800f800u, 0u);  // * -2^15
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t b[NT][4];
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) load_b(gl, nt, c, b[nt]);
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int r = 4 * c + 2 * q;
#pragma unroll
            for (int tile = 0; tile < kTiles; ++tile) {
              const uint32_t a0 = weight(ta[tile], r, za[tile]), a1 = weight(tb[tile], r, zb[tile]);
              const uint32_t a2 = weight(ta[tile], r + 1, za[tile]), a3 = weight(tb[tile], r + 1, zb[tile]);
#pragma unroll
              for (int nt = 0; nt < NT; ++nt)
                if (r == 0)
                  mma16816_first(d[tile][nt], a0, a1, a2, a3, b[nt][2 * q], b[nt][2 * q + 1]);
                else
                  mma16816(d[tile][nt], a0, a1, a2, a3, b[nt][2 * q], b[nt][2 * q + 1]);
            }
          }
        }
        // scale * 2^(ex - 5) * sum of the operands' products, the power of two first: a product on the way is as large as the
        // result, not as the sum of unscaled activations, which fp32 need not hold
        float sc[kTiles][2];
#pragma unroll
        for (int tile = 0; tile < kTiles; ++tile)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint32_t bits = lds16(sa + (uint32_t)(kSlotPlanes + (g * kUnitRows + tile * kTileRows + h * 8 + gid) * 2));
            sc[tile][h] = scale_bf16 ? __uint_as_float(bits << 16) : __half2float(__ushort_as_half((unsigned short)bits));
          }
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          const float2 st = *reinterpret_cast<const float2*>(&stat[gl * 8 * NT + nt * 8 + 2 * tig]);
#pragma unroll
          for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int tile = 0; tile < kTiles; ++tile) acc[tile][nt][q] = fmaf(sc[tile][q >> 1] * ((q & 1) ? st.y : st.x), d[tile][nt][q], acc[tile][nt][q]);
        }
      }
      if (has_outliers) add_outliers(pair, 0), add_outliers(pair, 1);
      // all lanes are done with the slot: it takes this warp's task kStages ahead
      __syncwarp();
      if (pf_left) issue_next(sa, bar);
      if (bar != bars_u32)
        sa = ring_u32, bar = bars_u32, phase ^= 1u;
      else
        sa += (uint32_t)kSlotBytes, bar += 8u;
      // the unit's end, or this warp's: put the sums down
      const bool last = pair + 1 == np;
      if (pair == 0 && lane == 0) span[unit].x = (unsigned char)warp;
      if (last && lane == 0) span[unit].y = (unsigned char)warp;
      if (last || t + 1 == t1) {
        float* const mine = part + (unit + warp) * 4 * quarter + gid;
#pragma unroll
        for (int tile = 0; tile < kTiles; ++tile)
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int m = nt * 8 + 2 * tig + (q & 1);
              if (m < M) mine[(2 * tile + (q >> 1)) * quarter + m * 8] = acc[tile][nt][q];
            }
        fresh = true;
      }
      pair = last ? 0 : pair + 1, unit += last ? 1 : 0;
    }
    const bool gave_up = __syncthreads_or(dead) != 0;

    // ---- per quarter unit: this CTA's sum over its warps, to the CTA that writes the quarter ----
    cluster_wait();  // the inboxes are free
    for (int i = warp; i < 4 * units; i += kWarps) {
      const int u = i >> 2, w0 = gave_up ? 0 : span[u].x, w1 = gave_up ? 0 : span[u].y, own = (int)((unsigned)i * p.splits_inv >> 16);
      if (lane < 2 * M) {
        const float4* from = reinterpret_cast<const float4*>(part + ((u + w0) * 4 + (i & 3)) * quarter) + lane;
        float4 v = *from;
        for (int w = w0; w < w1; ++w) {
          from += quarter;
          const float4 o = *from;
          v.x += o.x, v.y += o.y, v.z += o.z, v.w += o.w;
        }
        if (gave_up) v.x = v.y = v.z = v.w = __int_as_float(0x7fc00000);
        const uint32_t at = smem_u32(inbox + (own * splits + rank) * quarter + lane * 4);
        uint32_t there, there_bar;  // stores that count themselves in at the receiver: no fence, no cluster barrier
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(at), "r"(i - own * splits));
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there_bar) : "r"(inbox_bar), "r"(i - own * splits));
        asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(there), "f"(v.x), "f"(v.y),
                     "f"(v.z), "f"(v.w), "r"(there_bar)
                     : "memory");
      }
    }
    // Longer than a CTA of the cluster is held up by copies that do not land (one limit, then it sends NaN): none may leave
    // while another still stores into its shared memory.
    bool arrived = false;
    for (int limit = 0; limit < 3 && !arrived; ++limit) arrived = mbar_wait_bounded(inbox_bar, inbox_phase);
    inbox_phase ^= 1u;
    if (!arrived) atomicExch(p.status, 1u);
    for (int i = warp * splits + rank; i < 4 * units; i += kWarps * splits) {
      if (lane < 2 * M) {
        const float4* from = reinterpret_cast<const float4*>(inbox + (i - rank) * quarter) + lane;
        float4 v = *from;
        for (int s = 1; s < splits; ++s) {
          from += 2 * M;
          const float4 o = *from;
          v.x += o.x, v.y += o.y, v.z += o.z, v.w += o.w;
        }
        float r[4] = {v.x, v.y, v.z, v.w};
        if (!arrived) r[0] = r[1] = r[2] = r[3] = __int_as_float(0x7fc00000);
        const int at = (lane >> 1) * p.O + (unit0 + first) * kUnitRows + i * 8 + (lane & 1) * 4;
        if (p.addend)
          for (int q = 0; q < 4; ++q) r[q] += load_act(p.addend, p.act_dtype, at + q);
        unsigned short* const to = reinterpret_cast<unsigned short*>(p.out) + at;
        unsigned short h[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
          h[q] = p.act_dtype == FB_BF16 ? __bfloat16_as_ushort(__float2bfloat16_rn(r[q])) : __half_as_ushort(__float2half_rn(r[q]));
        if (p.out_aligned)
          *reinterpret_cast<uint2*>(to) = make_uint2((uint32_t)h[0] | (uint32_t)h[1] << 16, (uint32_t)h[2] | (uint32_t)h[3] << 16);
        else
          for (int q = 0; q < 4; ++q) to[q] = h[q];
      }
    }
    if (first + p.batch < count) {  // the next batch's sums overwrite these
      cluster_arrive();
      __syncthreads();
    }
  }
  if (dead) {  // the copies still in flight must not outlive the CTA's shared memory: wait for them, again bounded
    mbar_wait_bounded(bar, phase);
    mbar_wait_bounded(bar != bars_u32 ? bars_u32 : bars_u32 + 8u, bar != bars_u32 ? phase ^ 1u : phase);
  }
}

struct RowsPrepared : Prepared {
  RowsParams p;
  const uint8_t* planes;
  int rows, splits, slices;  // rows of the call; a launch takes 16, or 8
};

size_t shared_bytes(int rows, int npairs, int batch, int splits) {
  const size_t nt = rows <= 8 ? 1 : 2;
  return (size_t)kWarps * kStages * (kSlotBytes + 8) + 8 + 2 * batch + 2 * (size_t)npairs * (rows * (kOperandBytes + sizeof(Outlier)) + 8 * nt * sizeof(float)) +
         (size_t)((batch + kWarps - 1) * 4 + 4 * batch + splits) * 8 * rows * sizeof(float);
}

template <int NT, bool GATHER>
int launch(const RowsParams& p, const RowsPrepared& plan, size_t smem, bool pdl, cudaStream_t stream) {
  static std::mutex lock;
  static bool ready[64] = {};
  int device = 0;
  cudaError_t err = cudaGetDevice(&device);
  if (err != cudaSuccess) return cuda_fail(err, "cudaGetDevice");
  if (device < 0 || device >= 64) return fail(FB_ELIMIT, "device ordinal %d outside 0..63", device);
  {
    std::lock_guard<std::mutex> guard(lock);
    if (!ready[device]) {
      err = cudaFuncSetAttribute(w3_rows_kernel<NT, GATHER>, cudaFuncAttributeMaxDynamicSharedMemorySize, device_info()->max_smem_optin);
      if (err != cudaSuccess) return cuda_fail(err, "cudaFuncSetAttribute(w3_rows_kernel)");
      ready[device] = true;
    }
  }
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(plan.splits, plan.slices);
  config.blockDim = dim3(kThreads);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = plan.splits;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attr;
  config.numAttrs = pdl && pdl_allowed() ? 2 : 1;
  err = cudaLaunchKernelEx(&config, w3_rows_kernel<NT, GATHER>, p);
  return err == cudaSuccess ? FB_OK : cuda_fail(err, "w3_rows_kernel launch");
}

// Clusters of `splits` CTAs that the device runs at once (one CTA per SM; the SMs of a cluster lie in one GPC, so not
// every SM may find its place).  0 after recording an error.
int resident_clusters(int splits) {
  static std::mutex lock;
  static int known[64][kMaxSplits + 1] = {};
  int device = 0;
  if (cudaError_t err = cudaGetDevice(&device); err != cudaSuccess) return cuda_fail(err, "cudaGetDevice"), 0;
  if (device < 0 || device >= 64) return fail(FB_ELIMIT, "device ordinal %d outside 0..63", device), 0;
  std::lock_guard<std::mutex> guard(lock);
  int& answer = known[device][splits];
  if (answer) return answer;
  const auto kernel = w3_rows_kernel<1, false>;
  const int smem = device_info()->max_smem_optin;
  cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (err != cudaSuccess) return cuda_fail(err, "cudaFuncSetAttribute(w3_rows_kernel)"), 0;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(splits, 1024);
  config.blockDim = dim3(kThreads);
  config.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = splits;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  config.attrs = attr;
  config.numAttrs = 1;
  int clusters = 0;
  err = cudaOccupancyMaxActiveClusters(&clusters, kernel, &config);
  if (err != cudaSuccess) return cuda_fail(err, "cudaOccupancyMaxActiveClusters"), 0;
  return answer = clusters > 0 ? clusters : 1;
}

// How the work is dealt; the number of rows plays no part.  K over the CTAs of a cluster: kSplitPairs pairs of groups
// each, so that converting the activations costs little (4 KB of them per pair at 16 rows), or fewer where the row units
// alone would leave SMs idle.  Rows over the clusters that run at once.
int fill(RowsPrepared& made, int act_dtype, int m, const uint8_t* planes, const void* scales, int scale_dtype, const uint8_t* zeros, const int16_t* perm, int O,
         int K) {
  const DeviceInfo* info = device_info();
  if (!info) return FB_ECUDA;
  RowsParams& p = made.p;
  const int G = K / 128;
  p.O = O, p.K = K, p.G = G;
  p.scales = static_cast<const unsigned short*>(scales), p.zero_points = zeros;
  p.direct = perm && !aligned(perm, 16) ? 2 : (!aligned(scales, 16) || (zeros && !aligned(zeros, 16)) ? 1 : 0);
  p.act_dtype = act_dtype, p.scale_dtype = scale_dtype, p.zeros = zeros ? 1 : 0;
  p.perm = perm;
  const int pairs = (G + 1) / 2, units = O / kUnitRows;
  int splits = (pairs + kSplitPairs - 1) / kSplitPairs;
  if (splits < info->sm_count / units) splits = info->sm_count / units;
  if (splits > pairs) splits = pairs;
  if (splits > kMaxSplits) splits = kMaxSplits;
  made.splits = splits;
  made.slices = resident_clusters(splits);
  if (!made.slices) return FB_ECUDA;
  if (made.slices > units) made.slices = units;
  p.pairs_few = pairs / splits, p.pairs_extra = pairs % splits, p.npairs = p.pairs_few + (p.pairs_extra ? 1 : 0);
  p.units_few = units / made.slices, p.units_extra = units % made.slices;
  p.pairs_inv = (65536u + p.npairs - 1) / p.npairs, p.pairs_few_inv = (65536u + p.pairs_few - 1) / p.pairs_few;
  p.splits_inv = (65536u + splits - 1) / splits;
  // units between two cluster barriers: all, or as many as leave room beside the operands of a full launch
  const int most = p.npairs > 8 ? 8 : kMaxRows;
  p.batch = p.units_few + (p.units_extra ? 1 : 0);
  while (p.batch > 1 && shared_bytes(most, p.npairs, p.batch, splits) > (size_t)info->max_smem_optin) --p.batch;
  if (shared_bytes(most, p.npairs, p.batch, splits) > (size_t)info->max_smem_optin) return fail(FB_ELIMIT, "fb_w3_gemm_small: the plan does not fit in shared memory");
  if (!plane_tensor_map(planes, O, G, kTileRows, kTiles, 6, &p.plane_map)) return FB_ECUDA;
  p.scale_map = p.zero_map = p.plane_map;
  if (!p.direct && !group_row_tensor_map(scales, 2, O, G, kUnitRows, &p.scale_map)) return FB_ECUDA;
  if (!p.direct && zeros && !group_row_tensor_map(zeros, 1, O, G, kUnitRows, &p.zero_map)) return FB_ECUDA;
  made.planes = planes;
  made.rows = m;
  return FB_OK;
}

constexpr size_t kScratchBytes = 256;  // the status word

int run_add(const Prepared* base, const void* x, void* out, const void* addend, void* scratch, size_t scratch_bytes, unsigned flags, cudaStream_t stream) {
  const RowsPrepared& self = *static_cast<const RowsPrepared*>(base);
  RowsParams p = self.p;
  const size_t x_bytes = (size_t)self.rows * p.K * 2, out_bytes = (size_t)self.rows * p.O * 2;
  if (!aligned(out, 2) || !aligned(addend, 2) || !aligned(x, p.perm ? 2 : 16)) return fail(FB_EINVAL, "fb_w3_gemm_small: x must be 16-byte aligned, out 2-byte aligned");
  if (!scratch || scratch_bytes < kScratchBytes) return fail(FB_ESCRATCH, "fb_w3_gemm_small: scratch of %zu bytes needed, %zu given", kScratchBytes, scratch_bytes);
  if (!aligned(scratch, 256)) return fail(FB_EINVAL, "fb_w3_gemm_small: scratch must be 256-byte aligned");
  if (overlaps(out, out_bytes, x, x_bytes) || overlaps(scratch, kScratchBytes, out, out_bytes) || overlaps(scratch, kScratchBytes, x, x_bytes))
    return fail(FB_EALIAS, "fb_w3_gemm_small: out overlaps an input, or scratch overlaps x or out");
  if (overlaps(out, out_bytes, self.planes, (size_t)p.G * 3 * p.O * 16) || overlaps(out, out_bytes, p.scales, (size_t)p.G * p.O * 2))
    return fail(FB_EALIAS, "fb_w3_gemm_small: out overlaps an input");
  p.status = reinterpret_cast<unsigned*>(scratch);
  p.out_aligned = aligned(out, 8) ? 1 : 0;
  const bool pdl = (flags & FB_W3_NO_PDL) == 0;
  const int most = p.npairs > 8 ? 8 : kMaxRows;
  for (int row = 0; row < self.rows; row += most) {
    p.M = self.rows - row < most ? self.rows - row : most;
    p.rows_inv = (65536u + p.M - 1) / p.M;
    p.x = static_cast<const uint16_t*>(x) + (size_t)row * p.K;
    p.out = static_cast<uint16_t*>(out) + (size_t)row * p.O;
    p.addend = addend ? static_cast<const uint16_t*>(addend) + (size_t)row * p.O : nullptr;
    const size_t smem = shared_bytes(p.M, p.npairs, p.batch, self.splits);
    int rc;
    if (p.M > 8)
      rc = p.perm ? launch<2, true>(p, self, smem, pdl, stream) : launch<2, false>(p, self, smem, pdl, stream);
    else
      rc = p.perm ? launch<1, true>(p, self, smem, pdl, stream) : launch<1, false>(p, self, smem, pdl, stream);
    if (rc != FB_OK) return rc;
  }
  return FB_OK;
}

int run(const Prepared* base, const void* x, void* out, void* scratch, size_t scratch_bytes, unsigned flags, cudaStream_t stream) {
  return run_add(base, x, out, nullptr, scratch, scratch_bytes, flags, stream);
}

int check(int act_dtype, int m, const uint8_t* planes, const void* scales, int scale_dtype, const uint8_t* zeros, const int16_t* perm, int O, int K) {
  if (!planes || !scales) return fail(FB_EINVAL, "fb_w3_gemm_small: x, planes, scales and out must be non-null");
  if ((act_dtype != FB_F16 && act_dtype != FB_BF16) || (scale_dtype != FB_F16 && scale_dtype != FB_BF16))
    return fail(FB_EINVAL, "fb_w3_gemm_small: dtype tags must be FB_F16 or FB_BF16");
  if (m < 1 || m > kMaxRows) return fail(FB_ELIMIT, "fb_w3_gemm_small: M=%d outside 1..%d", m, kMaxRows);
  if (K < 128 || K % 128 || K / 128 > 255) return fail(FB_ELIMIT, "fb_w3_gemm_small: K=%d must be a multiple of 128 with at most 255 groups", K);
  if (O < 32 || O > 65536 || O % 32) return fail(FB_ELIMIT, "fb_w3_gemm_small: O=%d must be a multiple of 32 in 32..65536", O);
  if (!aligned(planes, 16) || !aligned(scales, 2) || !aligned(perm, 2))
    return fail(FB_EINVAL, "fb_w3_gemm_small: planes must be 16-byte aligned, 16-bit tensors 2-byte aligned");
  return FB_OK;
}

}  // namespace

extern "C" size_t fb_w3_gemm_small_scratch_bytes(int m, int out_features, int in_features) {
  return m < 1 || m > kMaxRows || out_features < 32 || in_features < 128 ? 0 : kScratchBytes;
}

extern "C" int fb_w3_prepare_small(int act_dtype, int m, const uint8_t* planes, const void* scales, int scale_dtype, const uint8_t* zeros,
                                   const int16_t* perm, int out_features, int in_features, fb_prepared_t** launch) {
  if (!launch) return fail(FB_EINVAL, "fb_w3_prepare_small: null result pointer");
  *launch = nullptr;
  int rc = check(act_dtype, m, planes, scales, scale_dtype, zeros, perm, out_features, in_features);
  if (rc != FB_OK) return rc;
  auto* made = new (std::nothrow) RowsPrepared;
  if (!made) return fail(FB_ELIMIT, "fb_w3_prepare_small: out of host memory");
  rc = fill(*made, act_dtype, m, planes, scales, scale_dtype, zeros, perm, out_features, in_features);
  if (rc != FB_OK) {
    delete made;
    return rc;
  }
  made->run = run;
  made->destroy = [](Prepared* self) { delete static_cast<RowsPrepared*>(self); };
  *launch = reinterpret_cast<fb_prepared_t*>(static_cast<Prepared*>(made));
  return FB_OK;
}

extern "C" int fb_w3_gemm_small(const void* x, int act_dtype, int m, const uint8_t* planes, const void* scales, int scale_dtype,
                                const uint8_t* zeros, const int16_t* perm, void* out, int out_features, int in_features,
                                void* scratch, size_t scratch_bytes, fb_stream_t stream) {
  return fb_w3_gemm_small_add(x, act_dtype, m, planes, scales, scale_dtype, zeros, perm, nullptr, out, out_features, in_features, scratch, scratch_bytes, stream);
}

extern "C" int fb_w3_gemm_small_add(const void* x, int act_dtype, int m, const uint8_t* planes, const void* scales, int scale_dtype,
                                    const uint8_t* zeros, const int16_t* perm, const void* addend, void* out, int out_features, int in_features,
                                    void* scratch, size_t scratch_bytes, fb_stream_t stream) {
  if (!x || !out) return fail(FB_EINVAL, "fb_w3_gemm_small: x, planes, scales and out must be non-null");
  int rc = check(act_dtype, m, planes, scales, scale_dtype, zeros, perm, out_features, in_features);
  if (rc != FB_OK) return rc;
  const size_t out_bytes = (size_t)m * out_features * 2;
  if (addend && overlaps(out, out_bytes, addend, out_bytes)) return fail(FB_EALIAS, "fb_w3_gemm_small: out overlaps the addend");
  RowsPrepared made;
  rc = fill(made, act_dtype, m, planes, scales, scale_dtype, zeros, perm, out_features, in_features);
  return rc != FB_OK ? rc : run_add(&made, x, out, addend, scratch, scratch_bytes, 0u, static_cast<cudaStream_t>(stream));
}
