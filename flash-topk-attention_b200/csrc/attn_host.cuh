// Host side shared by the attention launchers: from a caller's problem
// (include/ftk_attn.h) to the grid of blocks the kernels work on.
#pragma once

#include <algorithm>

#include "../../include/ftk_attn.h"
#include "attn_common.cuh"
#include "ftk_host.cuh"

namespace ftk {

struct AttnGrid {
  int kd;                          // the kernels' head dim: 64, 128 or 256
  int g, kvb;                      // rows per q block / kv block in the kernels
  int q_pad_head, kv_pad_head;
  int QM, Mkv;                     // blocks of those sizes
  int64_t width;                   // blocks of that size a list can hold
  ListMap lm;
};

inline int attn_head_dim(int64_t d) { return d <= 64 ? 64 : d <= 128 ? 128 : 256; }

// Blocks of more than `limit` rows are worked on as parts of half the size,
// repeatedly if need be; the lists stay as they are (ListMap).  A block of n
// rows that starts at token j * n - pad is the two halves 2 j - s, 2 j - s + 1
// of a grid of n / 2 rows and pad head pad - s * n / 2, where s = 1 when the pad
// head covers the whole first half.
inline int attn_grid(const ftk_attn& a, int limit, AttnGrid* out) {
  if (!a.q || !a.k || !a.v || !a.lists) return FTK_ERR_BAD_ARG;
  if (a.B <= 0 || a.H <= 0 || a.N <= 0 || a.list_rows <= 0 || a.W <= 0) return FTK_ERR_BAD_ARG;
  if (a.dtype != FTK_DTYPE_F16 && a.dtype != FTK_DTYPE_BF16) return FTK_ERR_BAD_ARG;
  if (a.Hkv <= 0 || a.H % a.Hkv != 0) return FTK_ERR_BAD_ARG;
  if (a.q_block <= 0 || a.kv_block <= 0) return FTK_ERR_BAD_ARG;
  if (a.q_pad_head < 0 || a.q_pad_head >= a.q_block || a.kv_pad_head < 0 ||
      a.kv_pad_head >= a.kv_block)
    return FTK_ERR_BAD_ARG;
  if (static_cast<int64_t>(a.list_rows) * a.q_block < a.q_pad_head + a.N) return FTK_ERR_BAD_ARG;
  if (a.D <= 0 || a.D % 8 != 0 || a.D > 256) return FTK_ERR_UNSUPPORTED;
  if (a.q_block > 128 || a.kv_block > 128) return FTK_ERR_UNSUPPORTED;
  if (a.B * a.H > 65535) return FTK_ERR_BAD_ARG;
  AttnGrid r{};
  r.kd = attn_head_dim(a.D);
  r.g = a.q_block;
  r.kvb = a.kv_block;
  r.q_pad_head = a.q_pad_head;
  r.kv_pad_head = a.kv_pad_head;
  int64_t rows = a.list_rows;
  r.width = a.W;
  auto halve = [](int& block, int& pad, int& shift, int& off) {
    const int half = block / 2, s = pad >= half ? 1 : 0;
    pad -= s * half;
    off = 2 * off + s;
    shift++;
    block = half;
    return s;
  };
  while (r.kvb > limit) {
    if (r.kvb % 32 != 0) return FTK_ERR_UNSUPPORTED;
    halve(r.kvb, r.kv_pad_head, r.lm.kv_shift, r.lm.kv_off);
    r.width *= 2;
  }
  while (r.g > limit) {
    if (r.g % 32 != 0) return FTK_ERR_UNSUPPORTED;
    rows = 2 * rows - halve(r.g, r.q_pad_head, r.lm.q_shift, r.lm.q_off);
  }
  if (r.kvb % 16 != 0) return FTK_ERR_UNSUPPORTED;
  const int64_t mkv = (r.kv_pad_head + a.N + r.kvb - 1) / r.kvb;
  if (mkv > AT_MAX_BLOCKS) return FTK_ERR_UNSUPPORTED;
  if (rows > 0x7fffffffLL) return FTK_ERR_BAD_ARG;
  r.QM = static_cast<int>(rows);
  r.Mkv = static_cast<int>(mkv);
  *out = r;
  return FTK_OK;
}

// q and kv blocks of 64 or 32 rows are walked as 64-row tiles (see ColSpan)
inline bool tiles_of_64(int g, int kvb) {
  return (g == 64 || g == 32) && (kvb == 64 || kvb == 32);
}

// q blocks per 128-row tile
inline int attn_groups(int g) { return std::max(1, std::min(AT_MAX_GROUPS, 128 / g)); }

// 16-byte rows: what the kernels' vector loads and stores of a row need
inline bool aligned16(const void* p, int64_t sb, int64_t sn, int64_t sh) {
  return p && !(reinterpret_cast<uintptr_t>(p) & 15u) && !((sb | sn | sh) & 7);
}

}  // namespace ftk
