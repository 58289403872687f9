// Two-base binary-basis GEMV, M = 1:  W ~ sum_b diag(row_b) * B_b * diag(col_b), B_b in {-1,+1},
// packed one bit per weight per base, in groups of 128 inputs.
//
// Same skeleton as the W3 GEMV (HBM-bound byte work, see fb_w3_gemv.cu): a K block is TWO groups
// (one for small matrices);
// a CTA holds 32 signed activation tables per group (2 bases x 16 chunks of 8 inputs, entries are
// sums of +/- x*col in ascending order) laid out entry-major so that the bank of a lookup is the
// table number; lane = output row; lanes walk the 32 (base, chunk) pairs of a group in a
// lane-rotated order so that lookups and staged-word reads are bank-conflict free; a warp's rows
// are, per group, one contiguous run of 32-byte code rows, staged by a bulk copy; the split over
// the K blocks is combined in the kernel by one 64-bit fixed-point atomic add per contribution
// (order-independent, repeat-exact).  Two groups per unit halve the fixed cost per byte of a unit
// (staging, scale loads, the returning atomic) and the atomics per output row.
//
// Two scale conventions:
//  * group mode (the reference's hybrid g128-s8 payload, deployment.py:23-27, kernel
//    csrc/m1_v5.cu:27-104): fp32 row scales per (group,row,base), fp32 column scales per
//    (group,input,base), plus a two-base refinement on 8 selected columns per group (two more
//    tables).  Codes may be planar [G,O,2,16] or interleaved [G,O,32]; interleaved words are unshuffled in
//    registers (16 instructions a word) and looked up like planar ones.
//  * global mode (matrix-wide fp16 scales r_b[O], c_b[K], planar codes, and `n_sal` dense bf16
//    residual columns): both groups of a unit share one sum per base; row scales are applied, and the residual
//    columns dealt, per contribution.
//
// What bounds it: the launch chain and, per unit, latencies; a unit carries two thirds of a W3 unit's bytes.  Only the codes are read
// ahead of the wait for the launch ahead, which may write everything else: scales, residual and refinement are brought to the L2
// before it and requested together with the activations behind it, a row's one unit ahead of their use.
// us on a B200, weights cold, in a graph, 1024x4096 / 4096x4096 / 12288x4096 / 4096x12288: matrix-wide scales 2.78 / 3.97 / 7.58 / 7.11,
// scales per group, planar 3.18 / 4.35 / 7.63 / 7.69, interleaved 3.26 / 5.36 / 10.6 / 10.6.  Read ahead of the wait they would take
// 2.78 / 3.82 / 7.32 / 6.98, 2.85 / 4.24 / 7.63 / 7.63 and 3.09 / 5.27 / 10.1 / 10.1; without the prefetch and the unit ahead, ring
// slots by a modulo and shares by 64-bit divisions it was 3.27 / 5.15 / 8.82 / 8.43, 4.02 / 6.26 / 9.96 / 9.97 and 4.37 / 8.52 / 16.5 / 16.6.
#include <mutex>
#include <new>

#include "fb_common.cuh"

namespace {

using namespace fb;

constexpr int kUnitRows = 32;
constexpr int kGroupBytes = kUnitRows * 32;  // 1 KB of codes per unit and group
constexpr int kWarps = 8;
constexpr int kCtasPerSm = 2;
constexpr int kGroupLutBytes = 32768;       // 256 entries x 32 tables x 4 B
constexpr int kGroupSparseBytes = 2048;     // 2 tables x 256 entries
constexpr int kMaxSalient = 256;            // residual columns

struct BBParams {
  const void* x;
  const uint8_t* codes;
  const float* rows;
  const float* cols;
  const uint8_t* sparse;
  const float* srows;
  const float* scols;
  const int16_t* indices;
  const __half* grow;
  const __half* gcol;
  const int32_t* sal_idx;
  const __nv_bfloat16* sal;
  void* out;
  unsigned long long* combine;  // [O] split-K accumulators, zero between launches
  unsigned* status;
  int O, K, G, nKB, nRU;
  int act_dtype, interleaved, global_mode, n_sal;
  int sal_most, sal_full;       // residual columns of a group whose activations are gathered: at most, and groups that have as many
  int sal_pairs;                // the residual values of two groups lie in one aligned 32-bit word
  int slots;                    // staged units per warp
  int units_few, units_extra;   // row units of a slice; slices that have one more
};

// Two words of eight sign bits per base, interleaved bit by bit, become [base 0: two bytes][base 1: two bytes]: the four
// steps of a perfect unshuffle (Warren, Hacker's Delight, 7-2).
__device__ __forceinline__ uint32_t unshuffle(uint32_t w) {
  uint32_t t;
  t = (w ^ (w >> 1)) & 0x22222222u, w ^= t ^ (t << 1);
  t = (w ^ (w >> 2)) & 0x0c0c0c0cu, w ^= t ^ (t << 2);
  t = (w ^ (w >> 4)) & 0x00f000f0u, w ^= t ^ (t << 4);
  t = (w ^ (w >> 8)) & 0x0000ff00u, w ^= t ^ (t << 8);
  return w;
}

// acc + {table entry at a0, table entry at a1}, each OFFSET bytes further: one packed add
template <int OFFSET>
__device__ __forceinline__ uint64_t add2_lds(uint64_t acc, uint32_t a0, uint32_t a1) {
  uint64_t r;
  asm volatile(
      "{\n\t.reg .f32 lo, hi;\n\t.reg .b64 both;\n\t"
      "ld.shared.f32 lo, [%2+%4];\n\t"
      "ld.shared.f32 hi, [%3+%4];\n\t"
      "mov.b64 both, {lo, hi};\n\t"
      "add.rn.f32x2 %0, %1, both;\n\t}"
      : "=l"(r)
      : "l"(acc), "r"(a0), "r"(a1), "n"(OFFSET));
  return r;
}
__device__ __forceinline__ void halves(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ float sum2(uint64_t v) {
  float lo, hi;
  halves(v, lo, hi);
  return lo + hi;
}
__device__ __forceinline__ uint32_t ldg16(const void* at) {
  uint32_t v;
  asm volatile("ld.global.u16 %0, [%1];" : "=r"(v) : "l"(at));
  return v;
}
__device__ __forceinline__ uint32_t ldg32(const void* at) {
  uint32_t v;
  asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(at));
  return v;
}
__device__ __forceinline__ float ldgf(const float* at) { return __uint_as_float(ldg32(at)); }
__device__ __forceinline__ float2 ldgf2(const float* at) {
  float2 v;
  asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(at));
  return v;
}
__device__ __forceinline__ void prefetch_l2(const void* at) { asm volatile("prefetch.global.L2 [%0];" ::"l"(at)); }
__device__ __forceinline__ float half_bits(uint32_t bits) { return __half2float(__ushort_as_half((unsigned short)bits)); }

// MORE (matrix-wide scales): a group carries several residual columns.
template <bool INTERLEAVED, bool GLOBAL, int GPB, bool MORE>
__global__ void __launch_bounds__(kWarps * 32, kCtasPerSm) bb_gemv_kernel(const BBParams p) {
  constexpr int kUnitBytes = GPB * kGroupBytes;  // staged per unit
  constexpr int kLutBytes = GPB * kGroupLutBytes, kSparseLutBytes = GLOBAL ? 0 : GPB * kGroupSparseBytes;
  extern __shared__ __align__(1024) unsigned char smem[];
  // the warp index through a shuffle, so that the compiler knows it is the same in all lanes (uniform registers)
  const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const int S = p.slots;
  unsigned char* const lut = smem;
  float* const sparse_lut = reinterpret_cast<float*>(smem + kLutBytes);
  const uint32_t ring_u32 = smem_u32(smem + kLutBytes + kSparseLutBytes) + (uint32_t)(warp * S * kUnitBytes);
  const uint32_t bars_u32 = smem_u32(smem + kLutBytes + kSparseLutBytes) + (uint32_t)(kWarps * S * kUnitBytes + warp * S * 8);
  // activations of the residual columns where a group carries several: [group][p.sal_most]
  float* const sal_x = reinterpret_cast<float*>(smem + kLutBytes + kSparseLutBytes + kWarps * S * (kUnitBytes + 8));

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  // ---- this CTA's K block and, dealt to its warps in turn, its row units ----
  const int kb = (int)blockIdx.y, slice = (int)blockIdx.x;
  const int first = slice * p.units_few + min(slice, p.units_extra) + warp;
  const int end = slice * p.units_few + min(slice, p.units_extra) + p.units_few + (slice < p.units_extra ? 1 : 0);
  const int ngroups = min(GPB, p.G - GPB * kb);

  if (lane == 0) {
    for (int s = 0; s < S; ++s) mbar_init(bars_u32 + s * 8, 1);
    mbar_init_fence();
  }
  __syncwarp();

  // ---- what the tables are made of beside the activations; lane = table (base = lane / 16, chunk = lane % 16).  A launch ahead may
  // still write it: ahead of the wait it is only brought to the L2, where such a write meets it ----
  const int base = lane >> 4, chunk = lane & 15;
  if (warp < ngroups) {
    const int g = GPB * kb + warp;
    if (GLOBAL) {  // 128 fp16 of either base, a sector per lane; a single residual column
      if (lane < 16) prefetch_l2(p.gcol + (size_t)(lane >> 3) * p.K + g * 128 + (lane & 7) * 16);
      if (!MORE && lane == 16 && g < p.n_sal) prefetch_l2(p.sal_idx + g);
    } else {
      prefetch_l2(p.cols + (size_t)g * 256 + lane * 8);
      if (lane < 2) prefetch_l2(p.scols + (size_t)g * 16 + lane * 8);
      if (lane == 2) prefetch_l2(p.indices + g * 8);
    }
  }
  // residual columns of a group's contribution, dealt round-robin: with MORE a thread gathers one of them, else all threads the first
  int sal_count[GPB];
  auto sal_column = [&](int gi) { return GPB * kb + gi + (MORE ? (int)threadIdx.x * p.G : 0); };
  auto gathers = [&](int gi) { return (MORE ? (int)threadIdx.x : 0) < sal_count[gi]; };
#pragma unroll
  for (int gi = 0; gi < GPB; ++gi) {
    sal_count[gi] = 0;
    if (GLOBAL && gi < ngroups) {
      sal_count[gi] = max(0, p.sal_most - (GPB * kb + gi < p.sal_full ? 0 : 1));
      if (MORE && (int)threadIdx.x < sal_count[gi]) prefetch_l2(p.sal_idx + sal_column(gi));
    }
  }

  // Staging of this warp's units in order, each into the slot that was read last: one bulk copy per group.  Rows past O in
  // the last unit are never copied (the copy is clipped) and never stored.
  int pf_ru = first, pf_slot = 0;
  auto issue_next = [&]() {
    if (lane == 0) {
      const uint32_t bar = bars_u32 + (uint32_t)(pf_slot * 8), dst = ring_u32 + (uint32_t)(pf_slot * kUnitBytes);
      const uint32_t bytes = (uint32_t)min(kUnitRows, p.O - pf_ru * kUnitRows) * 32u;
      const uint8_t* const src = p.codes + ((size_t)(GPB * kb) * p.O + (size_t)pf_ru * kUnitRows) * 32;
      mbar_expect_tx(bar, bytes * (uint32_t)ngroups);
      bulk_g2s(dst, src, bytes, bar);
      if (GPB == 2 && ngroups == 2) bulk_g2s(dst + kGroupBytes, src + (size_t)p.O * 32, bytes, bar);
    }
    pf_ru += kWarps;
    pf_slot = pf_slot + 1 == S ? 0 : pf_slot + 1;
  };
  if (pf_ru < end) issue_next();

  // Constants of a row in this K block, requested ONE UNIT AHEAD of their use (the first unit's together with the activations, brought
  // to the L2 before): requested where they were used, each unit of a warp waited for HBM once more.
  struct Constants {
    uint32_t r0, r1, sal[GPB];         // matrix-wide scales: fp16 row scales, bf16 residual values
    float2 rs[GPB], srs[GPB];          // scales per group: of the bases and of the refinement
    uint32_t sp[GPB];                  // refinement codes of both bases
  };
  auto request = [&](int ru, Constants& c) {
    const int row = min(ru * kUnitRows + lane, p.O - 1);
    if (GLOBAL) {
      c.r0 = ldg16(p.grow + row), c.r1 = ldg16(p.grow + (size_t)p.O + row);
      const __nv_bfloat16* const sal = p.sal + (size_t)row * p.n_sal + GPB * kb;
#pragma unroll
      for (int gi = 0; gi < GPB; ++gi) c.sal[gi] = 0u;
      if (GPB == 2 && p.sal_pairs) {
        if (GPB * kb < p.n_sal) {
          const uint32_t both = ldg32(sal);
          c.sal[0] = both << 16, c.sal[GPB - 1] = both & 0xffff0000u;
        }
      } else {
#pragma unroll
        for (int gi = 0; gi < GPB; ++gi)
          if (gi < ngroups && GPB * kb + gi < p.n_sal) c.sal[gi] = ldg16(sal + gi) << 16;
      }
    } else {
#pragma unroll
      for (int gi = 0; gi < GPB; ++gi) {
        c.rs[gi] = c.srs[gi] = make_float2(0.f, 0.f);
        c.sp[gi] = 0u;
        if (gi < ngroups) {
          const size_t at = (size_t)(GPB * kb + gi) * p.O + row;
          c.rs[gi] = ldgf2(p.rows + at * 2), c.srs[gi] = ldgf2(p.srows + at * 2), c.sp[gi] = ldg16(p.sparse + at * 2);
        }
      }
    }
  };
  if (first < end) {
    const int row = min(first * kUnitRows + lane, p.O - 1);
    if (GLOBAL) {
      prefetch_l2(p.grow + row), prefetch_l2(p.grow + (size_t)p.O + row);
      const __nv_bfloat16* const sal = p.sal + (size_t)row * p.n_sal;
      // A row's residual values are read one by one; up to four sectors of them are requested as a whole.  More would be in every CTA's way:
      // each K block asks for all of them, past the L1 (255 columns, with / without: 1024x8192 8.03 / 4.42 us, 4096x4096 12.1 / 8.8).
      if (MORE && p.n_sal <= 64) {
        for (int at = 0; at < p.n_sal; at += 16) prefetch_l2(sal + at);
      } else if (GPB * kb < p.n_sal) {
        prefetch_l2(sal + GPB * kb);
      }
    } else {
#pragma unroll
      for (int gi = 0; gi < GPB; ++gi)
        if (gi < ngroups) {
          const size_t at = ((size_t)(GPB * kb + gi) * p.O + row) * 2;
          prefetch_l2(p.rows + at), prefetch_l2(p.srows + at), prefetch_l2(p.sparse + at);
        }
    }
  }

  // Table addresses and word offsets of the rotated walk, the same for every unit.  Lookups use 32-bit shared-window
  // addresses: entry * 128 + table offset is ONE dp4a (a byte dot product whose only non-zero weight, 128, sits at the
  // wanted byte of the staged word).
  //  planar       row = [base 0: 16 bytes][base 1: 16 bytes]; word (h, ws) holds chunks 4 ws .. 4 ws + 3 of base h
  //  interleaved  row = 16 words of 16 bits, word c = chunk c of both bases; unshuffled, the 32-bit word w = 4 h + ws is
  //               [base 0: chunks 2 w, 2 w + 1][base 1: the same]
  const int rb = lane & 3, rw = (lane >> 2) & 3, rh = (lane >> 4) & 1;
  const uint32_t lut_u32 = smem_u32(lut);
  uint32_t sel[4], tables[2][4][4], woff[2][4];
#pragma unroll
  for (int b = 0; b < 4; ++b) sel[b] = 128u << (8 * ((b + rb) & 3));
#pragma unroll
  for (int jh = 0; jh < 2; ++jh)
#pragma unroll
    for (int jw = 0; jw < 4; ++jw) {
      const int h = jh ^ rh, ws = (jw + rw) & 3;
      woff[jh][jw] = (uint32_t)(h * 16 + ws * 4 + lane * 32);
      asm volatile("" : "+r"(woff[jh][jw]));
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int at = (b + rb) & 3;
        tables[jh][jw][b] = lut_u32 + (uint32_t)(INTERLEAVED ? 64 * (at >> 1) + 8 * (4 * h + ws) + 4 * (at & 1) : 64 * h + 16 * ws + 4 * at);
        asm volatile("" : "+r"(tables[jh][jw][b]));
      }
    }

  asm volatile("griddepcontrol.wait;" ::: "memory");

  // ---- activations, scales and the first unit's constants: all requests in one round trip ----
  uint4 xr[GPB];
  uint32_t col_half[GPB][4];
  float col[GPB][8];
#pragma unroll
  for (int gi = 0; gi < GPB; ++gi) {
    xr[gi] = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int j = 0; j < 8; ++j) col[gi][j] = 0.f;
    if (gi < ngroups) {
      const int k0 = (GPB * kb + gi) * 128 + chunk * 8;
      xr[gi] = *reinterpret_cast<const uint4*>(reinterpret_cast<const unsigned short*>(p.x) + k0);
      if (GLOBAL) {
        asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(col_half[gi][0]), "=r"(col_half[gi][1]), "=r"(col_half[gi][2]), "=r"(col_half[gi][3])
                     : "l"(p.gcol + (size_t)base * p.K + k0));
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) col[gi][j] = ldgf(p.cols + (size_t)(k0 + j) * 2 + base);
      }
    }
  }
  // the refinement's column and its scale: lane = (group, base, column)
  const int r_gi = GPB == 2 ? lane >> 4 : 0, r_base = (lane >> 3) & 1, r_j = lane & 7;
  const bool r_live = !GLOBAL && r_gi < ngroups && (GPB == 2 || lane < 16);
  int r_idx = 0;
  float r_col = 0.f;
  if (r_live) {
    const int g = GPB * kb + r_gi;
    r_idx = g * 128 + (int)ldg16(p.indices + g * 8 + r_j);
    r_col = ldgf(p.scols + (size_t)(g * 8 + r_j) * 2 + r_base);
  }
  int sal_at[GPB];
#pragma unroll
  for (int gi = 0; gi < GPB; ++gi) sal_at[gi] = gathers(gi) ? (int)ldg32(p.sal_idx + sal_column(gi)) : -1;
  Constants next;
  if (first < end) request(first, next);
  // The rest of the ring goes behind these and ahead of the gathers, which wait for the indices (scales per group, 12288x4096 7.60 us; behind
  // them 7.92).
  for (int s = 1; s < S && pf_ru < end; ++s) issue_next();
  // The residual columns' activations: where a group carries several, few warps gather them, ahead of the tables (12288x1024 4.53 us; behind them
  // 4.72, the first column by all warps 5.47).  A single one is gathered by all, behind the tables, which it would hold up (4096x4096
  // 4.05 us; ahead of them 4.13).
  float gathered[GPB];
  auto gather = [&]() {
#pragma unroll
    for (int gi = 0; gi < GPB; ++gi) gathered[gi] = sal_at[gi] >= 0 ? load_act(p.x, p.act_dtype, sal_at[gi]) : 0.f;
  };
  if (MORE) gather();
  float r_x = 0.f;
  if (r_live) r_x = load_act(p.x, p.act_dtype, r_idx);

  // ---- 32 signed tables per group ----
#pragma unroll
  for (int gi = 0; gi < GPB; ++gi) {
    const uint32_t xw[4] = {xr[gi].x, xr[gi].y, xr[gi].z, xr[gi].w};
    float v8[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float xv = bits_to_float((unsigned short)((xw[j >> 1] >> (16 * (j & 1))) & 0xffffu), p.act_dtype);
      v8[j] = GLOBAL ? __fmul_rn(xv, half_bits(col_half[gi][j >> 1] >> (16 * (j & 1)))) : __fmul_rn(xv, col[gi][j]);
      if (gi >= ngroups) v8[j] = 0.f;  // an odd number of groups: whatever lies in the empty half's slot finds zeros
    }
    // entry(p) = sum_b (bit b of p ? +v_b : -v_b) = low-nibble part + high-nibble part.  Warp w
    // owns the entries whose low nibble is 2w or 2w+1; the sixteen high-nibble parts come from
    // a tree (one add each), so an entry costs one add and one store.
    unsigned char* const column = lut + gi * kGroupLutBytes + lane * 4;
    float hi[16];
    hi[0] = ((-v8[4] - v8[5]) - v8[6]) - v8[7];
#pragma unroll
    for (int h = 1; h < 16; ++h) {
      const int top = h >= 8 ? 3 : (h >= 4 ? 2 : (h >= 2 ? 1 : 0));
      hi[h] = hi[h & ~(1 << top)] + 2.f * v8[4 + top];
    }
#pragma unroll
    for (int qq = 0; qq < 16 / kWarps; ++qq) {
      const int q = warp * (16 / kWarps) + qq;
      float lo = 0.f;
#pragma unroll
      for (int b = 0; b < 4; ++b) lo += ((q >> b) & 1) ? v8[b] : -v8[b];
#pragma unroll
      for (int h = 0; h < 16; ++h) *reinterpret_cast<float*>(column + (size_t)(h * 16 + q) * 128) = lo + hi[h];
    }
  }
  if (!GLOBAL) {
    // two refinement tables per group over its 8 selected columns; warp w fills entries 32w..32w+31
    const float sv = r_live ? __fmul_rn(r_x, r_col) : 0.f;
    const int pp = warp * 32 + lane;
#pragma unroll
    for (int t = 0; t < 2 * GPB; ++t) {  // (group, base)
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float one = __shfl_sync(0xffffffffu, sv, t * 8 + j);
        sum += ((pp >> j) & 1) ? one : -one;
      }
      sparse_lut[t * 256 + pp] = sum;
    }
  }
  if (!MORE) gather();
  if (MORE) {
#pragma unroll
    for (int gi = 0; gi < GPB; ++gi)
      if (sal_at[gi] >= 0) sal_x[gi * p.sal_most + (int)threadIdx.x] = gathered[gi];
  }
  __syncthreads();

  // Split over the K blocks: every contribution is ONE 64-bit atomic add carrying the scaled
  // partial sum in fixed point (steps of 2^-26, bits 16..63), an arrival count (bits 0..7) and a
  // count of partials that are not finite or too large for the format (bits 8..15).  Integer
  // adds commute, so the result is independent of arrival order; whoever reads back the last
  // count converts, writes the output and zeroes the word.  The answer is looked at one unit
  // later, so its round trip hides behind the next unit's lookups.
  unsigned long long pend_old = 0ull, pend_add = 0ull;
  int pend_row = -1;
  auto settle = [&]() {
    if (pend_row < 0) return;
    if (((unsigned)pend_old & 255u) == (unsigned)(p.nKB - 1)) {
      const unsigned long long total = pend_old + pend_add;
      float value = __ll2float_rn((long long)total >> 16) * 1.4901161193847656e-08f;  // 2^-26
      if ((total >> 8) & 255ull) value = __int_as_float(0x7fc00000);
      store_act(p.out, p.act_dtype, pend_row, value);
      p.combine[pend_row] = 0ull;
    }
    pend_row = -1;
  };

  int slot = 0;
  uint32_t phase = 0;
  for (int ru = first; ru < end; ru += kWarps) {
    Constants now = next;
    if (ru + kWarps < end) request(ru + kWarps, next);
    if (!__all_sync(0xffffffffu, mbar_wait_bounded(bars_u32 + (uint32_t)(slot * 8), phase))) {
      if (lane == 0) atomicExch(p.status, 1u);  // the copy never landed: give up
      break;
    }
    const uint32_t unit_u32 = ring_u32 + (uint32_t)(slot * kUnitBytes);
    constexpr int kSums = GLOBAL ? 1 : GPB;  // matrix-wide scales: the groups of a unit share their sums
    // planar: [sums of walk half jh]; interleaved: [byte steps 0 and 1 | 2 and 3]
    uint64_t acc[kSums][2] = {};
#pragma unroll
    for (int jh = 0; jh < 2; ++jh)
#pragma unroll
      for (int jw = 0; jw < 4; ++jw) {
        const uint32_t wa = unit_u32 + woff[jh][jw];
#pragma unroll
        for (int gi = 0; gi < GPB; ++gi) {
          uint32_t w, a[4];
          if (gi == 0)
            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w) : "r"(wa));
          else
            asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(w) : "r"(wa), "n"(kGroupBytes));
          if (INTERLEAVED) w = unshuffle(w);
#pragma unroll
          for (int b = 0; b < 4; ++b) asm("dp4a.u32.u32 %0, %1, %2, %3;" : "=r"(a[b]) : "r"(w), "r"(sel[b]), "r"(tables[jh][jw][b]));
          uint64_t& even = acc[GLOBAL ? 0 : gi][INTERLEAVED ? 0 : jh];
          uint64_t& odd = acc[GLOBAL ? 0 : gi][INTERLEAVED ? 1 : jh];
          even = gi == 0 ? add2_lds<0>(even, a[0], a[1]) : add2_lds<kGroupLutBytes>(even, a[0], a[1]);
          odd = gi == 0 ? add2_lds<0>(odd, a[2], a[3]) : add2_lds<kGroupLutBytes>(odd, a[2], a[3]);
        }
      }

    __syncwarp();
    if (pf_ru < end) issue_next();
    if (++slot == S) slot = 0, phase ^= 1u;

    float value = 0.f;
#pragma unroll
    for (int s = 0; s < kSums; ++s) {
      float d0, d1;  // the bases' sums
      if (INTERLEAVED) {
        float v[4];
        halves(acc[s][0], v[0], v[1]);
        halves(acc[s][1], v[2], v[3]);
        // byte step b served base ((b + rb) & 3) / 2
        const float near0 = (rb & 1) ? v[0] + v[3] : v[0] + v[1], near1 = (rb & 1) ? v[1] + v[2] : v[2] + v[3];
        d0 = (rb & 2) ? near1 : near0, d1 = (rb & 2) ? near0 : near1;
      } else {
        const float even = sum2(acc[s][0]), odd = sum2(acc[s][1]);
        d0 = rh ? odd : even, d1 = rh ? even : odd;
      }
      if (GLOBAL) {
        value = __fmaf_rn(half_bits(now.r0), d0, value);
        value = __fmaf_rn(half_bits(now.r1), d1, value);
      } else {
        const uint32_t sp = INTERLEAVED ? unshuffle(now.sp[s]) : now.sp[s];
        const uint32_t p0 = sp & 0xffu, p1 = INTERLEAVED ? sp >> 16 & 0xffu : sp >> 8;
        value = __fmaf_rn(now.rs[s].x, d0, value);
        value = __fmaf_rn(now.rs[s].y, d1, value);
        value = __fmaf_rn(now.srs[s].x, sparse_lut[s * 512 + p0], value);
        value = __fmaf_rn(now.srs[s].y, sparse_lut[s * 512 + 256 + p1], value);
      }
    }
    const int row = ru * kUnitRows + lane;
    if (GLOBAL) {
      // the dense residual columns are dealt round-robin over the groups' contributions
#pragma unroll
      for (int gi = 0; gi < GPB; ++gi) {
        if (sal_count[gi] > 0) value = __fmaf_rn(__uint_as_float(now.sal[gi]), MORE ? sal_x[gi * p.sal_most] : gathered[gi], value);
        if (MORE) {
          const __nv_bfloat16* const from = p.sal + (size_t)min(row, p.O - 1) * p.n_sal + GPB * kb + gi;
#pragma unroll 4
          for (int e = 1; e < sal_count[gi]; ++e) value = __fmaf_rn(__bfloat162float(from[e * p.G]), sal_x[gi * p.sal_most + e], value);
        } else if (p.n_sal > p.G && gi < ngroups && row < p.O) {  // one or two
          for (int at = GPB * kb + gi + p.G; at < p.n_sal; at += p.G)
            value = __fmaf_rn(__bfloat162float(p.sal[(size_t)row * p.n_sal + at]), load_act(p.x, p.act_dtype, p.sal_idx[at]), value);
        }
      }
    }
    settle();  // the previous unit's answer has long arrived
    if (row < p.O) {
      if (p.nKB == 1) {
        store_act(p.out, p.act_dtype, row, value);
      } else {
        const bool fits = fabsf(value) < GPB * 8192.f;  // 255 of one group, or 128 of two, stay inside 48 bits
        pend_add = fits ? ((unsigned long long)__float2ll_rn(value * 67108864.f) << 16) + 1ull : 257ull;
        asm volatile("atom.add.relaxed.gpu.global.u64 %0, [%1], %2;" : "=l"(pend_old) : "l"(p.combine + row), "l"(pend_add) : "memory");
        pend_row = row;
      }
    }
  }
  settle();
}

constexpr size_t kCombineOffset = 16384;  // after the status block: one 64-bit word per output row

template <bool INTERLEAVED, bool GLOBAL, int GPB, bool MORE>
int launch(const BBParams& p, dim3 grid, size_t smem, int max_smem, bool pdl, cudaStream_t stream) {
  static std::mutex lock;
  static bool ready[64] = {};
  int device = 0;
  cudaGetDevice(&device);
  {
    std::lock_guard<std::mutex> guard(lock);
    if (!ready[device]) {
      cudaError_t err = cudaFuncSetAttribute(bb_gemv_kernel<INTERLEAVED, GLOBAL, GPB, MORE>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
      if (err != cudaSuccess) return cuda_fail(err, "cudaFuncSetAttribute(bb_gemv_kernel)");
      ready[device] = true;
    }
  }
  cudaLaunchConfig_t config = {};
  config.gridDim = grid;
  config.blockDim = dim3(kWarps * 32);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attr;
  config.numAttrs = pdl && pdl_allowed() ? 1 : 0;
  cudaError_t err = cudaLaunchKernelEx(&config, bb_gemv_kernel<INTERLEAVED, GLOBAL, GPB, MORE>, p);
  if (err != cudaSuccess) return cuda_fail(err, "bb_gemv_kernel launch");
  return FB_OK;
}

// Two groups per K block halve the per-byte cost of a unit and double the tables to build ahead of the first: they pay once warps have
// units of one group to spare, more than one each with matrix-wide scales, more than four (interleaved: five) with scales per group, which
// bring more constants per unit either way.  us, one group / two, in brackets units of one group a warp: matrix-wide 2304x4096 (1.0) 3.29 / 3.59,
// 3072x4096 (1.3) 4.14 / 3.89, 3072x1024 (0.3) 3.02 / 3.81, 1024x12288 (1.3) 4.10 / 3.74; per group 2048x12288 (2.6) 5.53 / 6.04, 3072x12288 (3.9)
// 6.83 / 6.66, 9472x4096 (4.0) 6.99 / 7.32, 12288x4096 (5.2) 8.24 / 7.85; interleaved 5120x5120 (2.7) 6.91 / 7.45, 8192x5120 (4.3) 9.45 / 9.86,
// 12288x4096 (5.2) 10.79 / 10.79, 16384x4096 (6.9) 13.3 / 12.7.
int groups_per_block(int groups, int units, bool matrix_wide, bool interleaved, int sms) {
  return groups >= 2 && units * groups > kCtasPerSm * sms * kWarps * (matrix_wide ? 1 : interleaved ? 5 : 4) ? 2 : 1;
}

int run(BBParams& p, void* scratch, size_t scratch_bytes, unsigned flags, fb_stream_t stream, const char* who) {
  const size_t need = kCombineOffset + (size_t)p.O * sizeof(unsigned long long);
  if (!scratch || scratch_bytes < need) return fail(FB_ESCRATCH, "%s: scratch of %zu bytes needed, %zu given", who, need, scratch_bytes);
  if (!aligned(scratch, 256)) return fail(FB_EINVAL, "%s: scratch must be 256-byte aligned", who);
  const DeviceInfo* info = device_info();
  if (!info) return FB_ECUDA;
  unsigned char* base = static_cast<unsigned char*>(scratch);
  p.status = reinterpret_cast<unsigned*>(base);
  p.combine = reinterpret_cast<unsigned long long*>(base + kCombineOffset);
  p.nRU = (p.O + kUnitRows - 1) / kUnitRows;
  const int gpb = groups_per_block(p.G, p.nRU, p.global_mode, p.interleaved, info->sm_count);
  p.nKB = (p.G + gpb - 1) / gpb;
  int c = kCtasPerSm * info->sm_count / p.nKB;
  if (c < 1) c = 1;
  if (c > p.nRU) c = p.nRU;
  const dim3 grid(c, p.nKB);
  p.units_few = p.nRU / c, p.units_extra = p.nRU % c;
  p.sal_pairs = p.global_mode && p.n_sal % 2 == 0 && aligned(p.sal, 4) ? 1 : 0;
  const int per_warp = ((p.nRU + c - 1) / c + kWarps - 1) / kWarps;
  // Where a group carries three residual columns and more, their activations are gathered once per CTA; a second one is read where it is
  // used, which costs about the same.  us, gathered / as they are used: 32 columns 17x128 2.32 / 2.93, 512x512 (8 a group) 2.68 / 3.10, 16384x512 3.94 / 4.31, 512x1024 (4)
  // 2.70 / 2.93, 8192x1024 3.41 / 3.62, 8192x1280 (3.2) 4.20 / 4.94, 2048x2048 (2) 2.96 / 3.02, 5120x2560 (1.6) 4.17 / 4.17; 255 columns 2048x2048 (16) 5.51 / 5.86, 4096x4096
  // (8) 8.79 / 10.2.
  const bool more = p.global_mode && p.n_sal >= 3 * p.G;
  p.sal_most = !p.global_mode || p.n_sal == 0 ? 0 : more ? (p.n_sal - 1) / p.G + 1 : 1;
  p.sal_full = p.n_sal - (p.sal_most > 1 ? (p.sal_most - 1) * p.G : 0);
  const size_t sal_bytes = more ? (size_t)gpb * p.sal_most * sizeof(float) : 0;
  const int max_slots = gpb == 1 ? 4 : (p.global_mode && sal_bytes <= 512 ? 3 : 2);  // two CTAs per SM
  p.slots = per_warp < max_slots ? (per_warp < 1 ? 1 : per_warp) : max_slots;
  const size_t smem = (size_t)gpb * (kGroupLutBytes + (p.global_mode ? 0 : kGroupSparseBytes)) + (size_t)kWarps * p.slots * (gpb * kGroupBytes + 8) + sal_bytes;
  const bool pdl = (flags & FB_W3_NO_PDL) == 0;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (gpb == 2) {
    if (more) return launch<false, true, 2, true>(p, grid, smem, info->max_smem_optin, pdl, s);
    if (p.global_mode) return launch<false, true, 2, false>(p, grid, smem, info->max_smem_optin, pdl, s);
    if (p.interleaved) return launch<true, false, 2, false>(p, grid, smem, info->max_smem_optin, pdl, s);
    return launch<false, false, 2, false>(p, grid, smem, info->max_smem_optin, pdl, s);
  }
  if (more) return launch<false, true, 1, true>(p, grid, smem, info->max_smem_optin, pdl, s);
  if (p.global_mode) return launch<false, true, 1, false>(p, grid, smem, info->max_smem_optin, pdl, s);
  if (p.interleaved) return launch<true, false, 1, false>(p, grid, smem, info->max_smem_optin, pdl, s);
  return launch<false, false, 1, false>(p, grid, smem, info->max_smem_optin, pdl, s);
}

struct BBPrepared : Prepared {
  BBParams p;
};

int run_prepared(const Prepared* base, const void* x, void* out, void* scratch, size_t scratch_bytes, unsigned flags, cudaStream_t stream) {
  BBParams p = static_cast<const BBPrepared*>(base)->p;
  if (overlaps(out, (size_t)p.O * 2, x, (size_t)p.K * 2) || overlaps(out, (size_t)p.O * 2, p.codes, (size_t)p.G * p.O * 32))
    return fail(FB_EALIAS, "fb_bb_gemv: out overlaps an input");
  if (!aligned(x, 16)) return fail(FB_EINVAL, "fb_bb_gemv: x must be 16-byte aligned");
  if (flags & ~FB_W3_NO_PDL) return fail(FB_EINVAL, "fb_bb_gemv: unknown flag bits 0x%x", flags);
  p.x = x;
  p.out = out;
  return run(p, scratch, scratch_bytes, flags, stream, "fb_bb_gemv");
}

int check_common(const char* who, const void* x, int act_dtype, const uint8_t* codes, void* out, int O, int K) {
  if (!x || !codes || !out) return fail(FB_EINVAL, "%s: x, codes and out must be non-null", who);
  if (act_dtype != FB_F16 && act_dtype != FB_BF16) return fail(FB_EINVAL, "%s: activation dtype must be FB_F16 or FB_BF16", who);
  if (K < 128 || K % 128 || K / 128 > 255) return fail(FB_ELIMIT, "%s: K=%d must be a multiple of 128 with at most 255 groups", who, K);
  if (O < 1 || O > 65536) return fail(FB_ELIMIT, "%s: O=%d outside 1..65536", who, O);
  if (!aligned(codes, 16) || !aligned(x, 16)) return fail(FB_EINVAL, "%s: x and codes must be 16-byte aligned", who);
  if (overlaps(out, (size_t)O * 2, x, (size_t)K * 2) || overlaps(out, (size_t)O * 2, codes, (size_t)(K / 128) * O * 32))
    return fail(FB_EALIAS, "%s: out overlaps an input", who);
  return FB_OK;
}

}  // namespace

extern "C" size_t fb_bb_gemv_scratch_bytes(int out_features, int in_features, int global_scales) {
  if (out_features < 1 || in_features < 128) return 0;
  (void)global_scales;
  return kCombineOffset + (size_t)out_features * sizeof(unsigned long long);
}

extern "C" int fb_bb_gemv_block_groups(int out_features, int in_features, int planar, int global_scales) {
  if (out_features < 1 || in_features < 128 || in_features % 128) return fail(FB_ELIMIT, "fb_bb_gemv_block_groups: O=%d, K=%d", out_features, in_features);
  const DeviceInfo* info = device_info();
  if (!info) return FB_ECUDA;
  return groups_per_block(in_features / 128, (out_features + kUnitRows - 1) / kUnitRows, global_scales != 0, !planar, info->sm_count);
}

namespace {
int fill(BBParams& p, const void* x, int act_dtype, const uint8_t* codes, int planar, const float* rows, const float* cols, const uint8_t* sparse_codes,
         const float* sparse_rows, const float* sparse_cols, const int16_t* indices, void* out, int out_features, int in_features) {
  int rc = check_common("fb_bb_gemv", x, act_dtype, codes, out, out_features, in_features);
  if (rc) return rc;
  if (!rows || !cols || !sparse_codes || !sparse_rows || !sparse_cols || !indices)
    return fail(FB_EINVAL, "fb_bb_gemv: every payload tensor must be non-null");
  if (!aligned(rows, 8) || !aligned(sparse_rows, 8) || !aligned(sparse_codes, 2) || !aligned(cols, 4) || !aligned(sparse_cols, 4))
    return fail(FB_EINVAL, "fb_bb_gemv: scale tensors are misaligned");
  p = {};
  p.x = x; p.codes = codes; p.rows = rows; p.cols = cols; p.sparse = sparse_codes; p.srows = sparse_rows;
  p.scols = sparse_cols; p.indices = indices; p.out = out; p.O = out_features; p.K = in_features;
  p.G = in_features / 128; p.act_dtype = act_dtype; p.interleaved = planar ? 0 : 1; p.global_mode = 0;
  return FB_OK;
}
}  // namespace

extern "C" int fb_bb_gemv(const void* x, int act_dtype, const uint8_t* codes, int planar, const float* rows,
                          const float* cols, const uint8_t* sparse_codes, const float* sparse_rows,
                          const float* sparse_cols, const int16_t* indices, void* out, int out_features,
                          int in_features, void* scratch, size_t scratch_bytes, unsigned flags, fb_stream_t stream) {
  BBParams p;
  const int rc = fill(p, x, act_dtype, codes, planar, rows, cols, sparse_codes, sparse_rows, sparse_cols, indices, out, out_features, in_features);
  if (rc) return rc;
  if (flags & ~FB_W3_NO_PDL) return fail(FB_EINVAL, "fb_bb_gemv: unknown flag bits 0x%x", flags);
  return run(p, scratch, scratch_bytes, flags, stream, "fb_bb_gemv");
}

extern "C" int fb_bb_prepare(int act_dtype, const uint8_t* codes, int planar, const float* rows, const float* cols, const uint8_t* sparse_codes,
                             const float* sparse_rows, const float* sparse_cols, const int16_t* indices, int out_features, int in_features,
                             fb_prepared_t** launch) {
  if (!launch) return fail(FB_EINVAL, "fb_bb_prepare: null result pointer");
  auto* made = new (std::nothrow) BBPrepared;
  if (!made) return fail(FB_ELIMIT, "fb_bb_prepare: out of host memory");
  // addresses that no tensor has stand in for x and out, which come with each run
  const int rc = fill(made->p, reinterpret_cast<const void*>((uintptr_t)1 << 20), act_dtype, codes, planar, rows, cols, sparse_codes, sparse_rows, sparse_cols, indices,
                      reinterpret_cast<void*>(64), out_features, in_features);
  if (rc != FB_OK) {
    delete made;
    return rc;
  }
  made->run = run_prepared;
  made->destroy = [](Prepared* self) { delete static_cast<BBPrepared*>(self); };
  *launch = reinterpret_cast<fb_prepared_t*>(static_cast<Prepared*>(made));
  return FB_OK;
}

extern "C" int fb_bb_global_gemv(const void* x, int act_dtype, const uint8_t* codes, const void* row_scales,
                                 const void* col_scales, const int32_t* salient_idx, const void* salient,
                                 int n_salient, void* out, int out_features, int in_features, void* scratch,
                                 size_t scratch_bytes, unsigned flags, fb_stream_t stream) {
  int rc = check_common("fb_bb_global_gemv", x, act_dtype, codes, out, out_features, in_features);
  if (rc) return rc;
  if (!row_scales || !col_scales) return fail(FB_EINVAL, "fb_bb_global_gemv: scales must be non-null");
  if (!aligned(col_scales, 16)) return fail(FB_EINVAL, "fb_bb_global_gemv: column scales must be 16-byte aligned");
  if (n_salient < 0 || n_salient > kMaxSalient || (n_salient > 0 && (!salient_idx || !salient)))
    return fail(FB_EINVAL, "fb_bb_global_gemv: salient columns: 0..256 with index and value tensors");
  if (flags & ~FB_W3_NO_PDL) return fail(FB_EINVAL, "fb_bb_global_gemv: unknown flag bits 0x%x", flags);
  BBParams p = {};
  p.x = x; p.codes = codes; p.grow = static_cast<const __half*>(row_scales); p.gcol = static_cast<const __half*>(col_scales);
  p.sal_idx = salient_idx; p.sal = static_cast<const __nv_bfloat16*>(salient); p.n_sal = n_salient; p.out = out;
  p.O = out_features; p.K = in_features; p.G = in_features / 128; p.act_dtype = act_dtype; p.global_mode = 1;
  return run(p, scratch, scratch_bytes, flags, stream, "fb_bb_global_gemv");
}
