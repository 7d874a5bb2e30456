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
  uint8_t masks[AT_MAX_BLOCKS];          // bit g set: group g lists the block
  int warp_tot[4];
  int total;
};

// How the caller's lists map to the blocks a kernel works on.  Lists over q
// blocks or kv blocks of more rows than the kernels take are read as lists over
// parts of 2^-shift of the size: part m of the q grid takes list row
// (m + q_off) >> q_shift, and listed block j stands for the 2^kv_shift parts
// from (j << kv_shift) - kv_off on (`off` parts before the grid's first token
// are not there).  Zero shifts and offsets: the lists as they are.
struct ListMap {
  int q_shift, q_off, kv_shift, kv_off;
};

// Lists the bits of u.bm in ascending order (ids, masks, total).  All threads
// of the CTA call this, after a barrier behind the last write to u.bm.
// Expanding one bit per thread (128 threads walking a word each took as many
// serial steps as the densest word has bits) keeps this at four barriers.
__device__ __forceinline__ int list_union(UnionScratch& u, int words) {
  const int tid = threadIdx.x, nthr = blockDim.x;
  if (tid < AT_WORDS) {
    unsigned uni = 0;
    if (tid < words) {
#pragma unroll
      for (int g = 0; g < AT_MAX_GROUPS; g++) uni |= u.bm[g][tid];
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
      unsigned mk = 0;
#pragma unroll
      for (int g = 0; g < AT_MAX_GROUPS; g++) mk |= ((u.bm[g][wd] >> b) & 1u) << g;
      u.ids[pos] = static_cast<uint16_t>(x);
      u.masks[pos] = static_cast<uint8_t>(mk);
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
__device__ __forceinline__ int build_union(UnionScratch& u, const int32_t* lists, int first,
                                           int groups, int width, const int32_t* counts,
                                           int num_blocks, const ListMap& lm, int* status) {
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
          t[x] = g0 + x < groups ? __ldg(reinterpret_cast<const int4*>(row(g0 + x)) + e)
                                 : make_int4(-1, -1, -1, -1);
#pragma unroll
        for (int x = 0; x < 4; x++) {
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
  return list_union(u, (num_blocks + 31) >> 5);
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
// apart; entry ids run over the heads: head * span + q-block.
__device__ __forceinline__ int build_union_masks(UnionScratch& u, const uint8_t* masks, int stride,
                                                 int tiles, int per_tile, int j0, int groups,
                                                 int heads, int64_t head_stride, int span) {
  const int tid = threadIdx.x, nthr = blockDim.x;
  // the bytes of a thread's (head, tile): one word where four kv blocks lie in one
  const bool word = groups == 4 && (j0 & 3) == 0;
  auto load = [&](int h, int t) -> unsigned {
    const uint8_t* src = masks + h * head_stride + static_cast<int64_t>(t) * stride + j0;
    return word ? *reinterpret_cast<const unsigned*>(src) : src[0];
  };
  const unsigned first = tid < tiles ? load(0, tid) : 0u;   // under the clearing of the bitmaps
  __syncthreads();
  for (int h = 0; h < heads; h++) {
    for (int t = tid; t < tiles; t += nthr) {
      const int q = h * span + t * per_tile, wd = q >> 5, sh = q & 31;
      const unsigned b = h == 0 && t == tid ? first : load(h, t);
      if (word) {
#pragma unroll
        for (int g = 0; g < 4; g++) {
          const unsigned x = (b >> (8 * g)) & 255u;
          if (x) atomicOr(&u.bm[g][wd], x << sh);
        }
      } else {
        if (b) atomicOr(&u.bm[0][wd], b << sh);
        const uint8_t* src = masks + h * head_stride + static_cast<int64_t>(t) * stride + j0;
        for (int g = 1; g < groups; g++) {
          const unsigned x = src[g];
          if (x) atomicOr(&u.bm[g][wd], x << sh);
        }
      }
    }
  }
  __syncthreads();
  return list_union(u, (heads * span) >> 5);
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
