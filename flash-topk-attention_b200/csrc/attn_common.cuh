// Pieces shared by the sparse-attention kernels (forward, dQ, dK/dV).
//
// A CTA works on a 128-row tile made of G "groups" (q-blocks in the forward
// and dQ kernels, kv-blocks in the dK/dV kernel).  Each group brings its own
// list of partner blocks; the CTA walks the UNION of those lists in ascending
// block order and masks, per row, the partners its group does not list.  With
// 64-row blocks this fills the 128-row UMMA tile; where neighbouring groups
// list the same partners (the common case) no work is wasted.
#pragma once

#include "ftk_sm100.cuh"

namespace ftk {

constexpr int AT_MAX_GROUPS = 8;      // groups per 128-row tile
constexpr int AT_MAX_BLOCKS = 4096;   // partner blocks per slice
constexpr int AT_WORDS = AT_MAX_BLOCKS / 32;

struct UnionScratch {
  unsigned bm[AT_MAX_GROUPS][AT_WORDS];  // membership bitmaps
  unsigned uni[AT_WORDS];                // their union
  uint16_t pre[AT_WORDS];                // listed blocks below each word, within its warp's words
  uint16_t ids[AT_MAX_BLOCKS];           // union, ascending
  __align__(4) uint8_t masks[AT_MAX_BLOCKS];          // bit g set: group g lists the block
  int warp_tot[4];
};

// The tiles that a CTA walks are `sub` listed blocks wide, 1 or 2: blocks of 32 rows
// are walked two at a time as tiles of 64, with a mask byte for either half, since a
// 128 x 32 tile costs nearly what a 128 x 64 tile does (the barriers, TMEM accesses
// and UMMA overheads per tile are the same).

// What tile i of the union (its first token is tok0, `width` tokens) holds for a row
// of group `grp`: columns lo .. hi - 1, none unless `on`.  With sub 1 lo and hi are
// the same for all threads, and stay in uniform registers.
struct ColSpan {
  int lo, hi;
  bool on;
};
// `sub` as a template parameter of the kernels that walk 64-row tiles: the run-time
// choice cost 2 to 4 % of the dK/dV pair kernel.
__device__ __forceinline__ ColSpan col_span(const UnionScratch& u, int i, int sub, int grp, int tok0,
                                            int width, int N) {
  ColSpan c = {max(0, -tok0), min(width, N - tok0), true};
  if (sub == 1) {
    c.on = (u.masks[i] >> grp) & 1;
  } else {
    const unsigned m = *reinterpret_cast<const uint16_t*>(&u.masks[2 * i]) >> grp;
    if (!(m & 1u)) c.lo = max(c.lo, 32);
    if (!(m & 256u)) c.hi = min(c.hi, 32);
  }
  c.on = c.on && c.hi > c.lo;
  return c;
}

// How the caller's lists map to the blocks a kernel works on.  Lists over q
// blocks or kv blocks of more rows than the kernels take are read as lists over
// parts of 2^-shift of the size: part m of the q grid takes list row
// (m + q_off) >> q_shift, and listed block j stands for the 2^kv_shift parts
// from (j << kv_shift) - kv_off on (`off` parts before the grid's first token
// are not there).  Zero shifts and offsets: the lists as they are.
struct ListMap {
  int q_shift, q_off, kv_shift, kv_off;
};

// Lists the bits of u.bm in ascending order (ids, masks; `sub` bits make one
// entry).  All threads of the CTA call this, after a barrier behind the last write
// to u.bm.  Returns the number of entries.
// Expanding one bit per thread (128 threads walking a word each took as many
// serial steps as the densest word has bits) keeps this at four barriers.
__device__ __forceinline__ int list_union(UnionScratch& u, int words, int sub) {
  const int tid = threadIdx.x, nthr = blockDim.x;
  if (tid < AT_WORDS) {
    unsigned uni = 0;
    if (tid < words) {
#pragma unroll
      for (int g = 0; g < AT_MAX_GROUPS; g++) uni |= u.bm[g][tid];
      if (sub == 2) uni = (uni | (uni >> 1)) & 0x55555555u;
    }
    const int c = __popc(uni), lane = tid & 31;
    int inc = c;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, d);
      if (lane >= d) inc += v;
    }
    if (lane == 31) u.warp_tot[tid >> 5] = inc;
    u.uni[tid] = uni;
    u.pre[tid] = static_cast<uint16_t>(inc - c);
  }
  __syncthreads();
  const int t0 = u.warp_tot[0], t1 = u.warp_tot[1], t2 = u.warp_tot[2], t3 = u.warp_tot[3];
  for (int x = tid; x < words * 32; x += nthr) {
    const int wd = x >> 5, b = x & 31, wp = wd >> 5;
    const unsigned uni = u.uni[wd];
    if ((uni >> b) & 1u) {
      const int pos = u.pre[wd] + (wp > 0 ? t0 : 0) + (wp > 1 ? t1 : 0) + (wp > 2 ? t2 : 0) +
                      __popc(uni & ((1u << b) - 1u));
      unsigned mk = 0;   // both halves' bits when sub is 2: bits g and 8 + g
#pragma unroll
      for (int g = 0; g < AT_MAX_GROUPS; g++) {
        const unsigned bits = u.bm[g][wd] >> b;
        mk |= (bits & 1u) << g;
        if (sub == 2) mk |= (bits & 2u) << (7 + g);
      }
      if (sub == 1) {
        u.ids[pos] = static_cast<uint16_t>(x);
        u.masks[pos] = static_cast<uint8_t>(mk);
      } else {
        u.ids[pos] = static_cast<uint16_t>(x >> 1);
        *reinterpret_cast<uint16_t*>(&u.masks[2 * pos]) = static_cast<uint16_t>(mk);
      }
    }
  }
  __syncthreads();
  return t0 + t1 + t2 + t3;
}

__device__ __forceinline__ void clear_bitmaps(UnionScratch& u) {
  for (int i = threadIdx.x; i < AT_MAX_GROUPS * AT_WORDS; i += blockDim.x) (&u.bm[0][0])[i] = 0u;
}

// All threads of the CTA call this, after clear_bitmaps.  Groups first ..
// first + groups - 1 of the kernel's grid; `lists` is the slice's first list of
// `width` entries (or counts[g] of them when given); negative ids are skipped,
// ids >= num_blocks reported through `status`.  Returns the union size.
// FOLD: ascending lists have four ids in one word of the bitmap, and one atomic marks
// them.  In the one-CTA kernels, whose lists are short and whose unions weigh (lists of
// 16 blocks, B = 2, N = 4096, H = 32: forward 291 -> 288, dQ 380 -> 377 us; head dim 64,
// B = 2, N = 2048, H = 16: 70.4 -> 68.8 and 103.6 -> 101.1); the pairs and one
// CTA per SM at head dim 64 lose 1 to 2 %.
template <bool FOLD = false>
__device__ __forceinline__ int build_union(UnionScratch& u, const int32_t* lists, int first,
                                           int groups, int width, const int32_t* counts,
                                           int num_blocks, int sub, const ListMap& lm,
                                           int* status) {
  const int tid = threadIdx.x, nthr = blockDim.x;
  __syncthreads();
  auto row = [&](int g) {
    return lists + static_cast<int64_t>((first + g + lm.q_off) >> lm.q_shift) * width;
  };
  auto mark = [&](int g, int j) {
    if (j < 0) return;
    if (lm.kv_shift == 0) {
      if (j >= num_blocks) {
        if (status) atomicCAS(status, 0, FTK_DEV_BAD_INDEX);
        return;
      }
      atomicOr(&u.bm[g][j >> 5], 1u << (j & 31));
    } else if (j <= AT_MAX_BLOCKS) {
      const int s0 = (j << lm.kv_shift) - lm.kv_off;
      for (int i = 0; i < (1 << lm.kv_shift); i++) {
        const int x = s0 + i;
        if (x >= 0 && x < num_blocks) atomicOr(&u.bm[g][x >> 5], 1u << (x & 31));
      }
    }
  };
  if (!counts && (width & 3) == 0 && (reinterpret_cast<uintptr_t>(lists) & 15) == 0) {
    // lists are mostly -1 behind a prefix and wide (up to q block x topk): 16-byte
    // loads, four groups' in flight together
    const int quads = width >> 2;
    for (int g0 = 0; g0 < groups; g0 += 4) {
      for (int e = tid; e < quads; e += nthr) {
        int4 t[4];
#pragma unroll
        for (int x = 0; x < 4; x++)
          t[x] = g0 + x < groups ? reinterpret_cast<const int4*>(row(g0 + x))[e]
                                 : make_int4(-1, -1, -1, -1);
#pragma unroll
        for (int x = 0; x < 4; x++) {
          const int a = t[x].x, b = t[x].y, c = t[x].z, d = t[x].w;
          if (FOLD && (a & b & c & d) < 0) continue;
          if (FOLD && lm.kv_shift == 0 && ((a ^ b) | (a ^ c) | (a ^ d)) < 32 && (a | 31) < num_blocks &&
              ((a ^ b) | (a ^ c) | (a ^ d) | a) >= 0) {
            atomicOr(&u.bm[g0 + x][a >> 5],
                     (1u << (a & 31)) | (1u << (b & 31)) | (1u << (c & 31)) | (1u << (d & 31)));
            continue;
          }
          mark(g0 + x, t[x].x);
          mark(g0 + x, t[x].y);
          mark(g0 + x, t[x].z);
          mark(g0 + x, t[x].w);
        }
      }
    }
  } else {
    for (int g = 0; g < groups; g++) {
      const int cnt = counts ? min(counts[g], width) : width;
      const int32_t* r = row(g);
      for (int e = tid; e < cnt; e += nthr) mark(g, r[e]);
    }
  }
  __syncthreads();
  return list_union(u, (num_blocks + 31) >> 5, sub);
}

// What the dQ kernel leaves for the dK/dV kernel in place of a reverse index:
// one byte per (128-row q tile, kv block), bit i set when the tile's i-th
// q-block lists the kv block; `stride` bytes per tile, a multiple of 16.  Every
// CTA writes its own tile's whole row from the bitmaps it has just built, so
// nothing has to be cleared first, no atomics run, and the three launches of a
// separate reverse index (mark, list, sort) with their memset are not there.
__device__ __forceinline__ void write_tile_masks(const UnionScratch& u, uint8_t* row, int stride,
                                                 int g_first, int ng) {
  for (int x = threadIdx.x; x < (stride >> 2); x += blockDim.x) {
    const int wd = x >> 3, sh = (x & 7) * 4;
    unsigned out = 0;
    for (int i = 0; i < ng; i++) {
      const unsigned n = wd < AT_WORDS ? (u.bm[g_first + i][wd] >> sh) & 15u : 0u;
      out |= ((n & 1u) | ((n & 2u) << 7) | ((n & 4u) << 14) | ((n & 8u) << 21)) << i;
    }
    reinterpret_cast<unsigned*>(row)[x] = out;
  }
}

// The same union as build_union, for kv blocks j0 .. j0 + groups - 1, read off
// those bytes (after clear_bitmaps).  `masks` is the first tile's row of the
// first of `heads` query heads that share the kv head, `head_stride` bytes
// apart; listed blocks run over the heads: head * span + q-block.
__device__ __forceinline__ int build_union_masks(UnionScratch& u, const uint8_t* masks, int stride,
                                                 int tiles, int per_tile, int j0, int groups,
                                                 int heads, int64_t head_stride, int span, int sub) {
  const int tid = threadIdx.x, nthr = blockDim.x;
  // the bytes of a thread's (head, tile): words where the kv blocks fill whole ones
  const bool word = (groups & 3) == 0 && (j0 & 3) == 0;
  auto load = [&](int h, int t, int g) -> unsigned {
    const uint8_t* src = masks + h * head_stride + static_cast<int64_t>(t) * stride + j0 + g;
    return word ? *reinterpret_cast<const unsigned*>(src) : src[0];
  };
  const unsigned first = tid < tiles ? load(0, tid, 0) : 0u;   // under the clearing of the bitmaps
  __syncthreads();
  for (int h = 0; h < heads; h++) {
    for (int t = tid; t < tiles; t += nthr) {
      const int q = h * span + t * per_tile, wd = q >> 5, sh = q & 31;
      for (int g = 0; g < groups; g += word ? 4 : 1) {
        const unsigned b = h == 0 && t == tid && g == 0 ? first : load(h, t, g);
        if (word) {
#pragma unroll
          for (int x = 0; x < 4; x++) {
            const unsigned m = (b >> (8 * x)) & 255u;
            if (m) atomicOr(&u.bm[g + x][wd], m << sh);
          }
        } else if (b) {
          atomicOr(&u.bm[g][wd], b << sh);
        }
      }
    }
  }
  __syncthreads();
  return list_union(u, (heads * span) >> 5, sub);
}

// Up to four tiles of the union that between them hold, for every group with a
// list, at least one block of that list (the forward takes the rows' reference
// exponents from them): the tile that most groups list, then the one that most of
// the others list, and so on, ties to the first.  One warp calls this.  With wide
// lists one tile serves all groups.
struct CoverTiles {
  int n;                                 // tiles
  int entry[4];                          // their positions in the union
  int8_t of[AT_MAX_GROUPS];              // group -> which of them, -1: none
  int left;                              // groups with a list that none of the four holds
};
__device__ __forceinline__ void cover_tiles(const UnionScratch& u, int n, int groups, int sub,
                                            CoverTiles& c) {
  const int lane = threadIdx.x & 31;
  auto mask = [&](int i) -> unsigned {
    return sub == 1 ? u.masks[i] : u.masks[2 * i] | u.masks[2 * i + 1];
  };
  unsigned open = (1u << groups) - 1u;
  if (lane < AT_MAX_GROUPS) c.of[lane] = -1;
  __syncwarp();
  int e = 0;
  bool any = n > 0;
  for (; e < 4 && open && any; e++) {
    unsigned best = 0;   // groups served, then earlier first
    for (int i0 = 0; i0 < n; i0 += 32) {
      const int i = i0 + lane;
      const unsigned s = i < n ? __popc(mask(i) & open) : 0;
      best = max(best, s ? (s << 16) | (0xffffu - static_cast<unsigned>(i)) : 0u);
      if (__any_sync(0xffffffffu, (best >> 16) == __popc(open))) break;
    }
    best = __reduce_max_sync(0xffffffffu, best);
    any = best != 0;
    if (!any) break;
    const int i = static_cast<int>(0xffffu - (best & 0xffffu));
    const unsigned m = mask(i) & open;
    if (lane < AT_MAX_GROUPS && ((m >> lane) & 1u)) c.of[lane] = static_cast<int8_t>(e);
    if (lane == 0) c.entry[e] = i;
    open &= ~m;
  }
  // `open` groups: no list at all, or none of the four tiles holds one of its blocks
  unsigned listed = 0;
  if (open && any)
    for (int i = lane; i < n; i += 32) listed |= mask(i);
  listed = __reduce_or_sync(0xffffffffu, listed);
  if (lane == 0) {
    c.n = e;
    c.left = static_cast<int>(open & listed);
  }
  __syncwarp();
}

// two fp32 -> one 32-bit word of two 16-bit floats (element 0 in the low half)
__device__ __forceinline__ uint32_t pack2(float a, float b, int fmt) {
  if (fmt == 1) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  __half2 v = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}

__device__ __forceinline__ float2 unpack2(uint32_t w, int fmt) {
  if (fmt == 1) {
    return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&w));
  }
  return __half22float2(*reinterpret_cast<__half2*>(&w));
}

// 32 (or fewer) consecutive 16-bit results of one row, packed in pairs, columns
// c0 .. of a row of D: stored as they are or, for float32 callers, widened.
// Columns from D on are padding of the head dim and are not stored (D is a
// multiple of 8).
template <int NP>
__device__ __forceinline__ void store_row_part(uint8_t* row, int c0, int D,
                                               const uint32_t (&pk)[NP], int fmt, bool f32) {
#pragma unroll
  for (int x = 0; x < NP; x += 4) {
    if (c0 + 2 * x >= D) return;
    if (f32) {
      float4* dst = reinterpret_cast<float4*>(row + (c0 + 2 * x) * 4);
      const float2 a = unpack2(pk[x], fmt), b = unpack2(pk[x + 1], fmt),
                   c = unpack2(pk[x + 2], fmt), d = unpack2(pk[x + 3], fmt);
      dst[0] = make_float4(a.x, a.y, b.x, b.y);
      dst[1] = make_float4(c.x, c.y, d.x, d.y);
    } else {
      *reinterpret_cast<uint4*>(row + (c0 + 2 * x) * 2) =
          make_uint4(pk[x], pk[x + 1], pk[x + 2], pk[x + 3]);
    }
  }
}

}  // namespace ftk
