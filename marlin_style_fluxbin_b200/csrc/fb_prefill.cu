// Kernels of the many-token path (prefill, and the dense fallback of the packed Linear): the packed
// weights become 16-bit matrices for a dense GEMM, and the element-wise steps between the GEMMs take one
// launch each.
//
//   fb_w3_dequant           W3 planes -> 16-bit weight rows in group-sorted column order
//   fb_gather_columns       x[:, perm]: the activations in that order (cheaper than permuting the weight)
//   fb_qknorm_rope_prompt   per-head RMSNorm of q and k, rotary embedding, k / v into the cache, T tokens
//   fb_silu_mul_rows        SwiGLU gate of T rows whose gate and up halves lie side by side
//   fb_identity_order       whether a column order is the identity, told to the host without a wait
//
// Without them a 12288 x 4096 weight went through int32 and int64 tensors of its 50 M codes: 2.2 ms
// measured, against 0.02 ms for its 120 MB of traffic at the copy rate.
#include "fb_common.cuh"

namespace {

using namespace fb;

constexpr int kMaxDequant = 4;

struct DequantMatrix {
  const uint8_t* planes;
  const unsigned short* scales;
  const uint8_t* zeros;
  unsigned short* out;  // first requested row
  int O, row0, rows, block_begin;
};

struct DequantParams {
  DequantMatrix mats[kMaxDequant];
  int n, G, K, scale_dtype, out_dtype;
};

constexpr int kDequantRows = 64;   // per CTA: eight warps of eight rows
constexpr int kDequantGroups = 4;  // groups that a CTA walks

__device__ __forceinline__ unsigned short bits16(float v, int dtype) {
  return dtype == FB_BF16 ? __bfloat16_as_ushort(__float2bfloat16_rn(v)) : __half_as_ushort(__float2half_rn(v));
}

// Bound: the write of two bytes per weight (the planes are 3/16 of that).  Four lanes share a row of a
// group: each reads the row's 16 bytes of every plane and turns byte c of the four words into
// 4 x 8 consecutive weights, so a store instruction writes 64 contiguous bytes of eight rows.  A weight
// has one of eight values per (row, group); they are formed once, scale * (code - zero) rounded in the
// scale's dtype and then in the output's, split into tables of low and high bytes, and picked four at a
// time by byte permutes whose selector nibbles are the codes.
__global__ void __launch_bounds__(256) w3_dequant_kernel(const __grid_constant__ DequantParams p) {
  int j = 0;
  while (j + 1 < p.n && (int)blockIdx.x >= p.mats[j + 1].block_begin) ++j;
  const DequantMatrix& m = p.mats[j];
  const int lane = threadIdx.x & 31, c = lane & 3;
  const int local = ((int)blockIdx.x - m.block_begin) * kDequantRows + (threadIdx.x >> 5) * 8 + (lane >> 2);
  if (local >= m.rows) return;
  const int row = m.row0 + local;
  unsigned short* const out_row = m.out + (size_t)local * p.K;
  const uint32_t take = (uint32_t)(c | (c + 4) << 4);  // byte c of two words
  const int g_end = min(p.G, ((int)blockIdx.y + 1) * kDequantGroups);
#pragma unroll 2
  for (int g = blockIdx.y * kDequantGroups; g < g_end; ++g) {
    const uint4* const at = reinterpret_cast<const uint4*>(m.planes) + (size_t)(3 * g) * m.O + row;
    const uint4 w0 = __ldg(at), w1 = __ldg(at + m.O), w2 = __ldg(at + 2 * (size_t)m.O);
    const float scale = bits_to_float(m.scales[(size_t)g * m.O + row], p.scale_dtype);
    const int zero = m.zeros ? (int)m.zeros[(size_t)g * m.O + row] : 4;
    auto bytes = [&](const uint4& w) { return __byte_perm(__byte_perm(w.x, w.y, take), __byte_perm(w.z, w.w, take), 0x5410); };
    const uint32_t p0 = bytes(w0), p1 = bytes(w1), p2 = ~bytes(w2);  // the high plane is stored inverted
    uint32_t low[2], high[2];  // the eight values' low and high bytes
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      uint32_t v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = bits16(round_to(scale * (float)(4 * q + i - zero), p.scale_dtype), p.out_dtype);
      const uint32_t a = v[0] | v[1] << 16, b = v[2] | v[3] << 16;
      low[q] = __byte_perm(a, b, 0x6420), high[q] = __byte_perm(a, b, 0x7531);
    }
    // nibble n of codes[s]: the code of bit 4 * (n & 1) + s of byte n / 2
    uint32_t codes[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) codes[s] = ((p0 >> s) & 0x11111111u) | (((p1 >> s) & 0x11111111u) << 1) | (((p2 >> s) & 0x11111111u) << 2);
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      uint32_t x[4][2];  // [s]: values of nibbles 0, 1 and 2, 3
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const uint32_t sel = half ? codes[s] >> 16 : codes[s];
        const uint32_t l = __byte_perm(low[0], low[1], sel & 0xffffu), h = __byte_perm(high[0], high[1], sel & 0xffffu);
        x[s][0] = __byte_perm(l, h, 0x5140), x[s][1] = __byte_perm(l, h, 0x7362);
      }
#pragma unroll
      for (int b = 0; b < 2; ++b) {  // byte 2 * half + b of the plane word: word 2 * half + b of the row
        uint4 eight;
        eight.x = __byte_perm(x[0][b], x[1][b], 0x5410), eight.y = __byte_perm(x[2][b], x[3][b], 0x5410);
        eight.z = __byte_perm(x[0][b], x[1][b], 0x7632), eight.w = __byte_perm(x[2][b], x[3][b], 0x7632);
        *reinterpret_cast<uint4*>(out_row + g * 128 + (2 * half + b) * 32 + c * 8) = eight;
      }
    }
  }
}

// One CTA per row of x; K is a multiple of 128.
__global__ void __launch_bounds__(256) gather_columns_kernel(const unsigned short* __restrict__ x, const int16_t* __restrict__ perm,
                                                             unsigned short* __restrict__ out, int K) {
  const unsigned short* const row = x + (size_t)blockIdx.x * K;
  unsigned short* const to = out + (size_t)blockIdx.x * K;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  for (int k = threadIdx.x * 8; k < K; k += 256 * 8) {
    const uint4 idx = *reinterpret_cast<const uint4*>(perm + k);
    const uint32_t words[4] = {idx.x, idx.y, idx.z, idx.w};
    uint32_t v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = (uint32_t)row[words[i] & 0xffffu] | (uint32_t)row[words[i] >> 16] << 16;
    *reinterpret_cast<uint4*>(to + k) = make_uint4(v[0], v[1], v[2], v[3]);
  }
}

// A warp per (token, head), head_dim 128: a lane holds dims 2 l, 2 l + 1 and their partners + 64.  q heads
// go to q_out [T, q_heads, 128], k heads (normed, rotated) and v heads (as they are) to the cache rows.
__global__ void __launch_bounds__(256) qknorm_rope_prompt_kernel(const unsigned short* __restrict__ qkv, const unsigned short* __restrict__ q_weight,
                                                                 const unsigned short* __restrict__ k_weight, const unsigned short* __restrict__ cosv,
                                                                 const unsigned short* __restrict__ sinv, unsigned short* __restrict__ q_out,
                                                                 unsigned short* __restrict__ k_cache, unsigned short* __restrict__ v_cache,
                                                                 int tokens, int q_heads, int kv_heads, int max_positions, float eps, int dtype) {
  constexpr int D = 128;
  const int heads = q_heads + 2 * kv_heads, lane = threadIdx.x & 31;
  const int index = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (index >= tokens * heads) return;
  const int t = index / heads, head = index - t * heads;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const unsigned short* const src = qkv + ((size_t)t * heads + head) * D;
  const uint32_t a = *reinterpret_cast<const uint32_t*>(src + 2 * lane), b = *reinterpret_cast<const uint32_t*>(src + 64 + 2 * lane);
  if (head >= q_heads + kv_heads) {
    unsigned short* const dst = v_cache + ((size_t)(head - q_heads - kv_heads) * max_positions + t) * D;
    *reinterpret_cast<uint32_t*>(dst + 2 * lane) = a;
    *reinterpret_cast<uint32_t*>(dst + 64 + 2 * lane) = b;
    return;
  }
  const bool is_q = head < q_heads;
  const unsigned short* const weight = is_q ? q_weight : k_weight;
  unsigned short* const dst = is_q ? q_out + ((size_t)t * q_heads + head) * D : k_cache + ((size_t)(head - q_heads) * max_positions + t) * D;
  auto two = [&](uint32_t w, float (&f)[2]) { f[0] = bits_to_float((unsigned short)(w & 0xffffu), dtype), f[1] = bits_to_float((unsigned short)(w >> 16), dtype); };
  auto load2 = [&](const unsigned short* from, float (&f)[2]) { two(*reinterpret_cast<const uint32_t*>(from), f); };
  float lo[2], hi[2], wl[2], wh[2], cl[2], ch[2], sl[2], sh[2];
  two(a, lo), two(b, hi);
  load2(weight + 2 * lane, wl), load2(weight + 64 + 2 * lane, wh);
  load2(cosv + (size_t)t * D + 2 * lane, cl), load2(cosv + (size_t)t * D + 64 + 2 * lane, ch);
  load2(sinv + (size_t)t * D + 2 * lane, sl), load2(sinv + (size_t)t * D + 64 + 2 * lane, sh);
  float ss = lo[0] * lo[0] + lo[1] * lo[1] + hi[0] * hi[0] + hi[1] * hi[1];
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
  const float inv = rsqrtf(ss / (float)D + eps);
  uint32_t y0 = 0u, y1 = 0u;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float nlo = round_to(wl[i] * round_to(lo[i] * inv, dtype), dtype), nhi = round_to(wh[i] * round_to(hi[i] * inv, dtype), dtype);
    y0 |= (uint32_t)bits16(round_to(nlo * cl[i], dtype) - nhi * sl[i], dtype) << (16 * i);
    y1 |= (uint32_t)bits16(round_to(nhi * ch[i], dtype) + nlo * sh[i], dtype) << (16 * i);
  }
  *reinterpret_cast<uint32_t*>(dst + 2 * lane) = y0;
  *reinterpret_cast<uint32_t*>(dst + 64 + 2 * lane) = y1;
}

// out[t, i] = T(silu(gate_up[t, i])) * gate_up[t, width + i], eight elements per thread; a CTA's threads run along one row (a thread's
// row and column from its index took a 64-bit division: 10.5 us for 512 rows of 12288, 9.7 now, 3.9 TB/s of reads and writes that mostly stay in L2).
__global__ void __launch_bounds__(256) silu_mul_rows_kernel(const unsigned short* __restrict__ gate_up, unsigned short* __restrict__ out, int width, int out_stride,
                                                            int dtype) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const size_t t = blockIdx.x;
  for (long long at = ((long long)blockIdx.y * blockDim.x + threadIdx.x) * 8; at < width; at += (long long)gridDim.y * blockDim.x * 8) {
    const int i = (int)at;
    const uint4 g = *reinterpret_cast<const uint4*>(gate_up + (size_t)t * 2 * width + i), u = *reinterpret_cast<const uint4*>(gate_up + (size_t)t * 2 * width + width + i);
    const uint32_t gw[4] = {g.x, g.y, g.z, g.w}, uw[4] = {u.x, u.y, u.z, u.w};
    uint32_t v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      uint32_t both = 0u;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float gate = bits_to_float((unsigned short)(gw[k] >> (16 * h)), dtype), up = bits_to_float((unsigned short)(uw[k] >> (16 * h)), dtype);
        both |= (uint32_t)bits16(round_to(gate / (1.f + __expf(-gate)), dtype) * up, dtype) << (16 * h);
      }
      v[k] = both;
    }
    *reinterpret_cast<uint4*>(out + (size_t)t * out_stride + i) = make_uint4(v[0], v[1], v[2], v[3]);
  }
}

// *flag (device-visible host memory): 1 if perm is the identity, else 0.
__global__ void __launch_bounds__(1024) identity_order_kernel(const int16_t* __restrict__ perm, int K, int* flag) {
  int same = 1;
  for (int k = threadIdx.x; k < K; k += 1024) same &= perm[k] == k;
  same = __syncthreads_and(same);
  if (threadIdx.x == 0) {
    *flag = same;
    __threadfence_system();
  }
}

int launched(const char* what) {
  const cudaError_t err = cudaGetLastError();
  return err == cudaSuccess ? FB_OK : cuda_fail(err, what);
}
bool bad_dtype(int dtype) { return dtype != FB_F16 && dtype != FB_BF16; }
inline const unsigned short* u16(const void* p) { return static_cast<const unsigned short*>(p); }
inline unsigned short* u16(void* p) { return static_cast<unsigned short*>(p); }

}  // namespace

extern "C" int fb_w3_dequant(const fb_w3_matrix_t* matrices, int n_matrices, int row_begin, int row_count, int scale_dtype, int in_features, int out_dtype,
                             fb_stream_t stream) {
  if (!matrices) return fail(FB_EINVAL, "fb_w3_dequant: null matrix list");
  if (n_matrices < 1 || n_matrices > kMaxDequant) return fail(FB_ELIMIT, "fb_w3_dequant: %d matrices given, 1..%d supported", n_matrices, kMaxDequant);
  if (bad_dtype(scale_dtype) || bad_dtype(out_dtype)) return fail(FB_EINVAL, "fb_w3_dequant: dtype tags must be FB_F16 or FB_BF16");
  if (in_features < 128 || in_features % 128 || in_features / 128 > 255) return fail(FB_ELIMIT, "fb_w3_dequant: K=%d must be a multiple of 128 with at most 255 groups", in_features);
  DequantParams p = {};
  p.n = n_matrices;
  p.G = in_features / 128;
  p.K = in_features;
  p.scale_dtype = scale_dtype;
  p.out_dtype = out_dtype;
  int blocks = 0;
  for (int j = 0; j < n_matrices; ++j) {
    const fb_w3_matrix_t& in = matrices[j];
    const int O = in.out_features, rows = row_count > 0 ? row_count : O - row_begin;
    if (!in.planes || !in.scales || !in.out) return fail(FB_EINVAL, "fb_w3_dequant: planes, scales and out must be non-null");
    if (O < 1 || O > 65536 || row_begin < 0 || rows < 1 || row_begin + rows > O) return fail(FB_ELIMIT, "fb_w3_dequant: rows %d..%d of %d", row_begin, row_begin + rows, O);
    if (!aligned(in.planes, 16) || !aligned(in.out, 16) || !aligned(in.scales, 2)) return fail(FB_EINVAL, "fb_w3_dequant: planes and out must be 16-byte aligned");
    p.mats[j] = DequantMatrix{in.planes, u16(in.scales), in.zeros, u16(in.out), O, row_begin, rows, blocks};
    blocks += (rows + kDequantRows - 1) / kDequantRows;
  }
  w3_dequant_kernel<<<dim3(blocks, (p.G + kDequantGroups - 1) / kDequantGroups), 256, 0, static_cast<cudaStream_t>(stream)>>>(p);
  return launched("w3_dequant launch");
}

extern "C" int fb_gather_columns(const void* x, const int16_t* perm, void* out, int rows, int in_features, fb_stream_t stream) {
  if (!x || !perm || !out) return fail(FB_EINVAL, "fb_gather_columns: null pointer");
  if (rows < 1 || in_features < 128 || in_features % 128 || in_features > 32767) return fail(FB_ELIMIT, "fb_gather_columns: K=%d must be a multiple of 128 below 32768", in_features);
  if (!aligned(perm, 16) || !aligned(out, 16)) return fail(FB_EINVAL, "fb_gather_columns: perm and out must be 16-byte aligned");
  if (overlaps(out, (size_t)rows * in_features * 2, x, (size_t)rows * in_features * 2)) return fail(FB_EALIAS, "fb_gather_columns: out overlaps x");
  return launch_pdl(gather_columns_kernel, dim3(rows), dim3(256), 0, static_cast<cudaStream_t>(stream), "gather_columns launch", u16(x), perm, u16(out), in_features);
}

extern "C" int fb_qknorm_rope_prompt(const void* qkv, const void* q_weight, const void* k_weight, const void* cosv, const void* sinv, void* q_out, void* k_cache,
                                     void* v_cache, int tokens, int q_heads, int kv_heads, int head_dim, int max_positions, float eps, int dtype, fb_stream_t stream) {
  if (!qkv || !q_weight || !k_weight || !cosv || !sinv || !q_out || !k_cache || !v_cache) return fail(FB_EINVAL, "fb_qknorm_rope_prompt: null pointer");
  if (bad_dtype(dtype)) return fail(FB_EINVAL, "fb_qknorm_rope_prompt: dtype must be FB_F16 or FB_BF16");
  if (head_dim != 128) return fail(FB_ELIMIT, "fb_qknorm_rope_prompt: head_dim must be 128");
  if (q_heads < 1 || kv_heads < 1 || tokens < 1 || tokens > max_positions) return fail(FB_ELIMIT, "fb_qknorm_rope_prompt: %d tokens, cache of %d positions", tokens, max_positions);
  if (!aligned(qkv, 4) || !aligned(q_weight, 4) || !aligned(k_weight, 4) || !aligned(cosv, 4) || !aligned(sinv, 4) || !aligned(q_out, 4) || !aligned(k_cache, 4) ||
      !aligned(v_cache, 4))
    return fail(FB_EINVAL, "fb_qknorm_rope_prompt: tensors must be 4-byte aligned");
  const long long warps = (long long)tokens * (q_heads + 2 * kv_heads);
  if (warps > 0x7fffffff) return fail(FB_ELIMIT, "fb_qknorm_rope_prompt: too many tokens");
  return launch_pdl(qknorm_rope_prompt_kernel, dim3((unsigned)((warps + 7) / 8)), dim3(256), 0, static_cast<cudaStream_t>(stream), "qknorm_rope_prompt launch", u16(qkv),
                    u16(q_weight), u16(k_weight), u16(cosv), u16(sinv), u16(q_out), u16(k_cache), u16(v_cache), tokens, q_heads, kv_heads, max_positions, eps, dtype);
}

extern "C" int fb_silu_mul_rows(const void* gate_up, void* out, int rows, int width, int out_stride, int dtype, fb_stream_t stream) {
  if (!gate_up || !out) return fail(FB_EINVAL, "fb_silu_mul_rows: null pointer");
  if (bad_dtype(dtype)) return fail(FB_EINVAL, "fb_silu_mul_rows: dtype must be FB_F16 or FB_BF16");
  if (rows < 1 || width < 8 || width % 8 || out_stride < width || out_stride % 8) return fail(FB_ELIMIT, "fb_silu_mul_rows: width and stride must be multiples of 8");
  if (!aligned(gate_up, 16) || !aligned(out, 16)) return fail(FB_EINVAL, "fb_silu_mul_rows: tensors must be 16-byte aligned");
  const int per_row = width / 8, chunks = (per_row + 255) / 256 < 65535 ? (per_row + 255) / 256 : 65535;
  const int threads = chunks < 65535 ? ((per_row + chunks - 1) / chunks + 31) / 32 * 32 : 256;
  return launch_pdl(silu_mul_rows_kernel, dim3(rows, chunks), dim3(threads), 0, static_cast<cudaStream_t>(stream), "silu_mul_rows launch", u16(gate_up), u16(out), width,
                    out_stride, dtype);
}

extern "C" int fb_identity_order(const int16_t* perm, int in_features, int* flag, fb_stream_t stream) {
  if (!perm || !flag) return fail(FB_EINVAL, "fb_identity_order: null pointer");
  if (in_features < 1 || in_features > 32767) return fail(FB_ELIMIT, "fb_identity_order: K=%d outside 1..32767", in_features);
  identity_order_kernel<<<1, 1024, 0, static_cast<cudaStream_t>(stream)>>>(perm, in_features, flag);
  return launched("identity_order launch");
}
