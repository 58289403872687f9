// Host side of checkpoint preparation: raw GPTQ W3 words -> the planar layout, without the int64 tensors
// of single codes that the tensor-op form goes through (28 ms for a 1024 x 4096 Linear; its 3 MB in and out
// are about 0.3 ms of memory time on one core).
//
// A 3-bit code is cut out of one or two of the three 32-bit words of its block; 64 output columns at a time,
// eight input positions make one byte of each plane: the code's three bits are spread to bytes 0, 1 and 2 of a
// 32-bit lane by one multiplication, shifted to the position's bit and or-ed.  The compiler vectorises these
// loops over the columns (in the widest form the CPU has).  The layout wants the 16 bytes of a row together, so
// 16 x 16 byte blocks are transposed, with unpack instructions on x86; other hosts (the Arm ones of some B200 systems, or
// FB_PORTABLE) take the plain loops.  Groups are dealt to threads.
#if defined(__x86_64__) && !defined(FB_PORTABLE)
#include <emmintrin.h>
#define FB_X86 1
#define FB_CLONES __attribute__((target_clones("arch=skylake-avx512", "avx2", "default")))
#else
#define FB_X86 0
#define FB_CLONES
#endif
#include <stdint.h>
#include <string.h>

#include <atomic>
#include <thread>
#include <vector>

#include "../../include/fluxbin_b200.h"

namespace fb {
int fail(int code, const char* fmt, ...);
}

namespace {

constexpr int kColumns = 64;

// 16 rows of 16 bytes (row stride `stride`) -> 16 columns, written as 16 contiguous rows of 16 bytes.
inline void transpose16(const uint8_t* from, size_t stride, uint8_t* to) {
#if FB_X86
  __m128i a[16], b[16];
  for (int i = 0; i < 16; ++i) a[i] = _mm_loadu_si128(reinterpret_cast<const __m128i*>(from + i * stride));
  for (int round = 0; round < 4; ++round) {  // a perfect shuffle of the 256 bytes, four times, is the transpose
    for (int i = 0; i < 8; ++i) {
      b[2 * i] = _mm_unpacklo_epi8(a[i], a[i + 8]);
      b[2 * i + 1] = _mm_unpackhi_epi8(a[i], a[i + 8]);
    }
    memcpy(a, b, sizeof(a));
  }
  for (int i = 0; i < 16; ++i) _mm_storeu_si128(reinterpret_cast<__m128i*>(to + 16 * i), a[i]);
#else
  for (int i = 0; i < 16; ++i)
    for (int j = 0; j < 16; ++j) to[16 * j + i] = from[i * stride + j];
#endif
}

// Plane bytes of group g for columns [o0, o0 + n): n <= kColumns.
FB_CLONES void pack_block(const uint32_t* words, const int64_t* order, int O, int o0, int n, uint8_t (*bytes)[16][kColumns]) {
  for (int c = 0; c < 16; ++c) {
    uint32_t acc[kColumns] = {};
    for (int j = 0; j < 8; ++j) {
      const int64_t k = order[8 * c + j];
      const int bit = 3 * (int)(k & 31), shift = bit & 31;
      const uint32_t* const low = words + ((k >> 5) * 3 + (bit >> 5)) * O + o0;
      if (shift <= 29) {
        if (n == kColumns)
          for (int i = 0; i < kColumns; ++i) acc[i] |= ((((low[i] >> shift) & 7u) * 0x4081u) & 0x010101u) << j;
        else
          for (int i = 0; i < n; ++i) acc[i] |= ((((low[i] >> shift) & 7u) * 0x4081u) & 0x010101u) << j;
      } else {  // the code continues in the next word
        const uint32_t* const high = low + O;
        for (int i = 0; i < n; ++i) acc[i] |= (((((low[i] >> shift) | (high[i] << (32 - shift))) & 7u) * 0x4081u) & 0x010101u) << j;
      }
    }
    for (int p = 0; p < 3; ++p) {
      const uint8_t flip = p == 2 ? 0xff : 0;  // the high plane is stored inverted
      for (int i = 0; i < kColumns; ++i) bytes[p][c][i] = (uint8_t)(acc[i] >> (8 * p)) ^ flip;
    }
  }
}

void pack_groups(const uint32_t* words, const int64_t* order, int O, uint8_t* planes, int g_begin, int g_end) {
  alignas(32) uint8_t bytes[3][16][kColumns];
  alignas(16) uint8_t rows[256];
  for (int g = g_begin; g < g_end; ++g)
    for (int o0 = 0; o0 < O; o0 += kColumns) {
      const int n = O - o0 < kColumns ? O - o0 : kColumns;
      pack_block(words, order + 128 * (int64_t)g, O, o0, n, bytes);
      for (int p = 0; p < 3; ++p) {
        uint8_t* const out = planes + (((size_t)g * 3 + p) * O + o0) * 16;
        for (int i = 0; i < n; i += 16) {
          if (n - i >= 16) {
            transpose16(&bytes[p][0][i], kColumns, out + 16 * i);
          } else {
            transpose16(&bytes[p][0][i], kColumns, rows);
            memcpy(out + 16 * i, rows, (size_t)(n - i) * 16);
          }
        }
      }
    }
}

}  // namespace

extern "C" int fb_host_w3_order(const int32_t* g_idx, int in_features, int64_t* order) {
  if (!g_idx || !order || in_features < 128 || in_features % 128) return fb::fail(FB_EINVAL, "fb_host_w3_order: bad argument");
  if (in_features > 32767) return fb::fail(FB_ELIMIT, "fb_host_w3_order: K=%d: columns must be numbered by int16", in_features);
  const int G = in_features / 128;
  int next[255];
  for (int g = 0; g < G; ++g) next[g] = 128 * g;
  bool low = false, high = false, uneven = false;
  for (int k = 0; k < in_features; ++k) {
    const int g = g_idx[k];
    if (g < 0 || g >= G) return fb::fail(FB_ELIMIT, "fb_host_w3_order: group index outside the range");
    low |= g == 0, high |= g == G - 1;
    if (next[g] == 128 * (g + 1))
      uneven = true;
    else
      order[next[g]++] = k;
  }
  if (!low || !high) return fb::fail(FB_ELIMIT, "fb_host_w3_order: group index outside the range");
  return uneven ? fb::fail(FB_EINVAL, "fb_host_w3_order: groups of unequal size") : FB_OK;
}

extern "C" int fb_host_w3_planes(const uint32_t* qweight, const int64_t* order, int in_features, int out_features, uint8_t* planes, int threads) {
  if (!qweight || !order || !planes || in_features < 128 || in_features % 128 || out_features < 1)
    return fb::fail(FB_EINVAL, "fb_host_w3_planes: bad argument");
  const int G = in_features / 128;
  // a thread costs about 30 us to start, as much as packing 64 K codes
  const long long most = (long long)in_features * out_features / (256 * 1024);
  int n = threads < 1 ? 1 : threads;
  if (n > most) n = most < 1 ? 1 : (int)most;
  if (n > G) n = G;
  std::vector<std::thread> team;
  std::atomic<int> at{0};
  auto work = [&] {
    for (int g; (g = at.fetch_add(1)) < G;) pack_groups(qweight, order, out_features, planes, g, g + 1);
  };
  try {
    for (int t = 1; t < n; ++t) team.emplace_back(work);
  } catch (...) {  // no more threads to be had: this one does the rest
  }
  work();
  for (std::thread& t : team) t.join();
  return FB_OK;
}

extern "C" int fb_host_w3_zeros(const uint32_t* qzeros, int groups, int out_features, int plus, uint8_t* zeros, unsigned* seen) {
  if (!qzeros || !zeros || !seen || groups < 1 || out_features < 1 || out_features % 32) return fb::fail(FB_EINVAL, "fb_host_w3_zeros: bad argument");
  unsigned found = 0;
  const size_t blocks = (size_t)groups * out_features / 32;
  for (size_t b = 0; b < blocks; ++b) {
    const uint32_t* const w = qzeros + 3 * b;
    const uint64_t low = w[0] | (uint64_t)w[1] << 32, high = w[1] | (uint64_t)w[2] << 32;
    for (int i = 0; i < 32; ++i) {
      const unsigned zero = ((unsigned)((i <= 10 ? low >> (3 * i) : high >> (3 * i - 32)) + (unsigned)plus)) & 7u;
      zeros[32 * b + i] = (uint8_t)zero;
      found |= 1u << zero;
    }
  }
  *seen = found;
  return FB_OK;
}
