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

struct UnionScratch {
  uint16_t ids[AT_MAX_BLOCKS];                 // union, ascending
  __align__(4) uint8_t masks[AT_MAX_BLOCKS];   // bit g set: group g lists the block
  int warp_tot[32];
};

// The tiles that a CTA walks are `sub` listed blocks wide, 1 or 2: blocks of 32 rows
// are walked two at a time as tiles of 64, with a mask byte for either half, since a
// 128 x 32 tile costs nearly what a 128 x 64 tile does (the barriers, TMEM accesses
// and UMMA overheads per tile are the same).

// What tile i of the union (its first token is tok0, `width` tokens) holds for a row
// of group `grp`: columns lo .. hi - 1, none unless `on`.  With sub 1 lo and hi are
// the same for all threads, and stay in uniform registers.  Rows that do not exist are
// like the others: copies fill them with zeros.  What comes of that may be infinite or NaN
// (a zero query against an infinite key; 2^-lse against a small lse in dK / dV), but it
// stays in the row's own lane of every accumulator, and neither the stores nor the flags
// for the exact kernel look at such rows; nothing may add up over rows without leaving them
// out.  Told apart in the loop, they kept their warps off the path for full tiles in every
// tile (N = 3000, H = 12, head dim 96: forward 89 us, 61 without).
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

// What a list builder marks: one byte per (block, group), `stride` bytes per block, in
// dynamic shared memory that no TMA copy has been aimed at yet (the rings).  Bits would
// need atomics, and with few blocks the lanes of a warp all hit the same few words; bytes
// are plain stores, and the mask of a block comes out of one load.
__host__ __device__ constexpr int flag_stride(int groups) { return groups > 4 ? 8 : 4; }
__host__ __device__ constexpr int flag_blocks(int blocks) { return (blocks + 15) & ~15; }
__host__ __device__ constexpr size_t flag_bytes(int blocks, int groups) {
  return static_cast<size_t>(flag_blocks(blocks)) * flag_stride(groups);
}
__device__ __forceinline__ void clear_flags(uint8_t* flags, int blocks, int groups) {
  const int n = static_cast<int>(flag_bytes(blocks, groups) >> 4);
#pragma unroll 1
  for (int i = threadIdx.x; i < n; i += blockDim.x)
    reinterpret_cast<uint4*>(flags)[i] = make_uint4(0u, 0u, 0u, 0u);
}
// four bytes of 0 or 1 -> four bits (no two partial products meet in one place)
__device__ __forceinline__ unsigned bytes_to_bits(unsigned v) { return (v * 0x01020408u) >> 24; }

// Everything from here to a kernel's roles is run once per CTA, by warps that have
// nothing to overlap it with: a warp alone gets an instruction out every 4 to 5 cycles, so
// what counts is the number of instructions on its way.

// First half of listing a union: the WARPS warps of the CTA take consecutive runs of
// entries, mask_of(x) is the mask of entry x < n (its two halves' masks in two bytes when
// blocks are walked two at a time), and every warp counts its own.  The caller puts a
// barrier behind it and calls list_entries.  The mask of a thread's first entry (the only
// one up to 32 * WARPS) stays in a register.
struct ListRun {
  unsigned mask;
  int base, rounds;
};
template <int WARPS, typename Mask>
__device__ __forceinline__ ListRun count_entries(UnionScratch& u, int n, Mask&& mask_of) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  ListRun run;
  run.rounds = (n + 32 * WARPS - 1) / (32 * WARPS);
  run.base = warp * run.rounds * 32 + lane;
  run.mask = run.base < n ? mask_of(run.base) : 0u;
  int cnt = __popc(__ballot_sync(0xffffffffu, run.mask != 0u));
#pragma unroll 1
  for (int r = 1; r < run.rounds; r++) {
    const int x = run.base + r * 32;
    cnt += __popc(__ballot_sync(0xffffffffu, x < n && mask_of(x) != 0u));
  }
  if (lane == 0) u.warp_tot[warp] = cnt;
  return run;
}
// Second half: the entries in ascending order.  Returns their number.
template <int WARPS, typename Mask>
__device__ __forceinline__ int list_entries(UnionScratch& u, const ListRun& run, int n, int sub,
                                            Mask&& mask_of) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = lane < WARPS ? u.warp_tot[lane] : 0;
  const int total = __reduce_add_sync(0xffffffffu, t);
  int pos = __reduce_add_sync(0xffffffffu, lane < warp ? t : 0);
  unsigned m = run.mask;
  int x = run.base;
#pragma unroll 1
  for (int r = 0;;) {
    const unsigned b = __ballot_sync(0xffffffffu, m != 0u);
    if (m) {
      const int at = pos + __popc(b & ((1u << lane) - 1u));
      u.ids[at] = static_cast<uint16_t>(x);
      if (sub == 1) u.masks[at] = static_cast<uint8_t>(m);
      else *reinterpret_cast<uint16_t*>(&u.masks[2 * at]) = static_cast<uint16_t>(m);
    }
    if (++r >= run.rounds) break;
    pos += __popc(b);
    x += 32;
    m = x < n ? mask_of(x) : 0u;
  }
  return total;
}

// What the dQ kernel leaves for the dK/dV kernel in place of a reverse index:
// one byte per (128-row q tile, kv block), bit i set when the tile's i-th
// q-block lists the kv block; `flag_blocks(kv blocks)` bytes per tile.  Every
// CTA writes its own tile's whole row from the masks that it lists, so
// nothing has to be cleared first, no atomics run, and the three launches of a
// separate reverse index (mark, list, sort) with their memset are not there.
struct TileMaskRow {
  uint8_t* row = nullptr;      // null: none is written
  int first = 0, count = 0;    // the tile's q-blocks among the groups
};

// All threads of the CTA (WARPS warps) call this, after clear_flags(flags, num_blocks,
// groups).  Groups first .. first + groups - 1 of the kernel's grid; `lists` is the
// slice's first list of `width` entries (or counts[g] of them when given); negative ids
// are skipped, ids >= num_blocks reported through `status`.  Returns the union size.  The
// warp of thread 0, which issues the first copies, is dealt the last entries.
template <int WARPS>
__device__ __forceinline__ int build_union(UnionScratch& u, uint8_t* flags, const int32_t* lists,
                                           int first, int groups, int width, const int32_t* counts,
                                           int num_blocks, int sub, const ListMap& lm,
                                           int* status, TileMaskRow tile = TileMaskRow()) {
  constexpr int NTHR = 32 * WARPS;
  const int tid = threadIdx.x >= 32 ? threadIdx.x - 32 : threadIdx.x + NTHR - 32;
  const bool wide = groups > 4;
  const int shift = wide ? 3 : 2;
  auto row = [&](int g) {
    return lists + static_cast<int64_t>((first + g + lm.q_off) >> lm.q_shift) * width;
  };
  bool bad = false;
  auto mark = [&](int g, int j) {
    if (lm.kv_shift == 0) {
      if (static_cast<unsigned>(j) < static_cast<unsigned>(num_blocks)) flags[(j << shift) + g] = 1;
      else bad |= j >= 0;
    } else if (j >= 0 && j <= AT_MAX_BLOCKS) {
      const int s0 = (j << lm.kv_shift) - lm.kv_off;
#pragma unroll 1
      for (int i = 0; i < (1 << lm.kv_shift); i++) {
        const int x = s0 + i;
        if (x >= 0 && x < num_blocks) flags[(x << shift) + g] = 1;
      }
    }
  };
  if (!counts && (width & 3) == 0 && (reinterpret_cast<uintptr_t>(lists) & 15) == 0) {
    // lists are mostly -1 behind a prefix and wide (up to q block x topk): 16-byte
    // loads, four groups' in flight together and across the barrier behind the clearing
    const int quads = width >> 2;
    const uint32_t base = smem_u32(flags);
    int largest = -1;
    bool cleared = false;
#pragma unroll 1
    for (int g0 = 0; g0 < groups; g0 += 4) {
#pragma unroll 1
      for (int e = tid; e < quads || !cleared; e += NTHR) {
        int4 t[4];
#pragma unroll
        for (int x = 0; x < 4; x++)
          t[x] = g0 + x < groups && e < quads ? reinterpret_cast<const int4*>(row(g0 + x))[e]
                                              : make_int4(-1, -1, -1, -1);
        if (!cleared) {
          __syncthreads();
          cleared = true;
        }
#pragma unroll
        for (int x = 0; x < 4; x++) {
          if ((t[x].x & t[x].y & t[x].z & t[x].w) < 0) continue;
          const int j[4] = {t[x].x, t[x].y, t[x].z, t[x].w};
          if (lm.kv_shift == 0) {
            // four instructions a mark; with branches the 16 of a thread took 3300 cycles
#pragma unroll
            for (int y = 0; y < 4; y++)
              asm volatile(
                  "{\n\t.reg .pred p;\n\tsetp.lt.u32 p, %0, %1;\n\t@p st.shared.u8 [%2], %3;\n\t}" ::"r"(
                      j[y]),
                  "r"(num_blocks), "r"(base + g0 + x + (j[y] << shift)), "r"(1)
                  : "memory");
            largest = max(largest, max(max(j[0], j[1]), max(j[2], j[3])));
          } else {
#pragma unroll 1
            for (int y = 0; y < 4; y++)
              mark(g0 + x, y == 0 ? j[0] : y == 1 ? j[1] : y == 2 ? j[2] : j[3]);
          }
        }
      }
    }
    bad = lm.kv_shift == 0 && largest >= num_blocks;
  } else {
    __syncthreads();
#pragma unroll 1
    for (int g = 0; g < groups; g++) {
      const int cnt = counts ? min(counts[g], width) : width;
      const int32_t* r = row(g);
#pragma unroll 1
      for (int e = tid; e < cnt; e += NTHR) mark(g, r[e]);
    }
  }
  if (bad && status) atomicCAS(status, 0, FTK_DEV_BAD_INDEX);
  __syncthreads();
  auto one = [&](int x) -> unsigned {
    const uint8_t* f = flags + (x << shift);
    unsigned m = bytes_to_bits(*reinterpret_cast<const unsigned*>(f));
    if (wide) m |= bytes_to_bits(*reinterpret_cast<const unsigned*>(f + 4)) << 4;
    return m;
  };
  auto mask_of = [&](int x) -> unsigned {
    return sub == 1 ? one(x) : one(2 * x) | one(2 * x + 1) << 8;
  };
  const int n = flag_blocks(num_blocks) >> (sub - 1);
  const ListRun run = count_entries<WARPS>(u, n, [&](int x) -> unsigned {
    const unsigned m = mask_of(x);
    if (tile.row) {
      const unsigned keep = (1u << tile.count) - 1u;
      const unsigned mine = (m >> tile.first) & (keep | keep << 8);
      if (sub == 1) tile.row[x] = static_cast<uint8_t>(mine);
      else reinterpret_cast<uint16_t*>(tile.row)[x] = static_cast<uint16_t>(mine);
    }
    return m;
  });
  __syncthreads();
  const int total = list_entries<WARPS>(u, run, n, sub, mask_of);
  fence_async_smem();   // TMA copies are about to land where the flags were
  __syncthreads();
  return total;
}

// The same union for kv blocks j0 .. j0 + groups - 1 (groups a power of two up to 8, j0 a
// multiple of it; bytes behind the last kv block are 0), read off those bytes: an
// entry's mask is one load and a few shifts.  `masks` is the first tile's row of the
// first of `heads` query heads that share the kv head, `head_stride` bytes
// apart; listed blocks run over the heads: head * span + q-block.  per_tile q-blocks
// per row, a power of two, a multiple of `sub`.
template <int WARPS>
__device__ __forceinline__ int build_union_masks(UnionScratch& u, const uint8_t* masks, int stride,
                                                 int tiles, int per_tile, int j0, int groups,
                                                 int heads, int64_t head_stride, int span, int sub) {
  const int tile_shift = 31 - __clz(per_tile);
  auto mask_of = [&](int x) -> unsigned {
    const int q = x * sub;
    const int h = heads > 1 ? q / span : 0, at = q - h * span;
    const int t = at >> tile_shift, bit = at & (per_tile - 1);
    if (t >= tiles) return 0u;
    const uint8_t* src = masks + h * head_stride + static_cast<int64_t>(t) * stride + j0;
    unsigned w[2] = {0u, 0u};
    if (groups == 8) {
      const uint2 v = *reinterpret_cast<const uint2*>(src);
      w[0] = v.x;
      w[1] = v.y;
    } else if (groups == 4) {
      w[0] = *reinterpret_cast<const unsigned*>(src);
    } else if (groups == 2) {
      w[0] = *reinterpret_cast<const uint16_t*>(src);
    } else {
      w[0] = src[0];
    }
    auto bits = [&](int b) -> unsigned {
      const unsigned k = 0x01010101u;
      return bytes_to_bits((w[0] >> b) & k) | bytes_to_bits((w[1] >> b) & k) << 4;
    };
    return sub == 1 ? bits(bit) : bits(bit) | bits(bit + 1) << 8;
  };
  const int n = (heads * span) >> (sub - 1);
  const ListRun run = count_entries<WARPS>(u, n, mask_of);
  __syncthreads();
  const int total = list_entries<WARPS>(u, run, n, sub, mask_of);
  __syncthreads();
  return total;
}

// Up to `most` (at most 4) tiles of the union that between them hold, for every group
// with a list, at least one block of that list (the forward takes the rows' reference
// exponents from them): the tile that most groups list, then the one that most of
// the others list, and so on, ties to the first.  With wide lists one tile serves all
// groups.  Every warp works this out for itself: by one warp, behind a barrier for the
// others, it took 800 cycles.
// The union and its masks decide, not the order in which a list names its blocks: results
// do not depend on how a list is written.
struct CoverTiles {
  int n;                // tiles
  int e0, e1, e2, e3;   // their positions in the union
  unsigned of;          // four bits per group: which of them, 15: none
  int left;             // groups with a list that none of them holds
  __device__ __forceinline__ int entry(int e) const { return e == 0 ? e0 : e == 1 ? e1 : e == 2 ? e2 : e3; }
};
__device__ __forceinline__ CoverTiles cover_tiles(const UnionScratch& u, int n, int groups, int sub,
                                                  int most) {
  const int lane = threadIdx.x & 31;
  auto mask = [&](int i) -> unsigned {
    return sub == 1 ? u.masks[i] : u.masks[2 * i] | u.masks[2 * i + 1];
  };
  CoverTiles c = {0, 0, 0, 0, 0, 0xffffffffu, 0};
  unsigned open = (1u << groups) - 1u;
  bool any = n > 0;
  // as a rule one of the first tiles serves all
  const unsigned all = __ballot_sync(0xffffffffu, lane < n && mask(lane) == open);
  if (all) {
    c.n = 1;
    c.e0 = __ffs(all) - 1;
    c.of = 0;
    open = 0;
  }
  auto add = [&](int i) {
    if (c.n == 0) c.e0 = i;
    else if (c.n == 1) c.e1 = i;
    else if (c.n == 2) c.e2 = i;
    else c.e3 = i;
    c.n++;
  };
#pragma unroll 1
  while (c.n < most && open && any) {
    unsigned best = 0;   // groups served, then earlier first
#pragma unroll 1
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
#pragma unroll 1
    for (int g = 0; g < groups; g++)
      if ((m >> g) & 1u) c.of = (c.of & ~(15u << (4 * g))) | static_cast<unsigned>(c.n) << (4 * g);
    add(i);
    open &= ~m;
  }
  // `open` groups: no list at all, or none of the tiles holds one of its blocks
  unsigned listed = 0;
  if (open && any) {
#pragma unroll 1
    for (int i = lane; i < n; i += 32) listed |= mask(i);
    listed = __reduce_or_sync(0xffffffffu, listed);
  }
  c.left = static_cast<int>(open & listed);
  return c;
}

// Head dims between the kernels' own, of which D columns are there: the k-steps of 16 columns
// that a product over the head dim has, and the columns that a product of M = 256 across two CTAs
// yields (multiples of 32).  The others are zeros, or are not stored.
__device__ __forceinline__ int used_ksteps(int D) { return (D + 15) >> 4; }
__device__ __forceinline__ int used_columns(int D) { return (D + 31) & ~31; }

// Where a CTA's results go: worked out by one thread ahead of the loop over the tiles and
// kept in shared memory until the end of it, where a warp also asks for its number anew.
// Held in registers all along, they cost the loop's warps, which have 96, a few percent.
struct OutTile {
  int64_t off[2];    // elements to the slice's first row in the result (or in both)
  int row0, last;    // the tile's first row and the end of its rows that exist
};
__device__ __forceinline__ int late_tid() {
  int t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t)::"memory");
  return t;
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

// 32 (or 16) columns c0 .. of 32 rows, a row per lane packed in pairs, to global memory:
// as 16-bit values or, for float32 callers, widened.  Written straight from the lanes,
// each store instruction touches 32 rows, and the 32 KB of a tile took 3700 cycles; the
// detour over 2 KB of shared memory (`stage`, 16-byte aligned, the warp's own) leaves 8
// rows of 64 contiguous bytes per instruction.  `base` is the whole result, `o` where the
// tile lies in it, `which` picks the offset, `quarter` the 32 rows, `stride` in elements;
// columns below D (a multiple of 8) are stored.
template <int NP>
__device__ __forceinline__ void store_rows(uint8_t* stage, const uint32_t (&pk)[NP], void* base,
                                           const OutTile& o, int which, int quarter, int64_t stride,
                                           int c0, int D, int fmt, bool f32) {
  constexpr int CH = NP / 4;             // 16-byte chunks of a row
  static_assert(CH == 2 || CH == 4, "");
  const int lane = late_tid() & 31;
  const int row0 = o.row0 + 32 * quarter, first = -row0, last = o.last - row0;
  uint8_t* out = static_cast<uint8_t*>(base) + (f32 ? 4 : 2) * (o.off[which] + row0 * stride);
  // chunk j of row r sits at j ^ flip(r): both sides use every bank once per eight lanes
  auto flip = [](int r) { return (r >> (CH == 4 ? 1 : 2)) & (CH - 1); };
#pragma unroll
  for (int j = 0; j < CH; j++)
    *reinterpret_cast<uint4*>(stage + lane * (16 * CH) + ((j ^ flip(lane)) << 4)) =
        make_uint4(pk[4 * j], pk[4 * j + 1], pk[4 * j + 2], pk[4 * j + 3]);
  __syncwarp();
  if (!f32) {
    const int j = lane % CH;
    int r = lane / CH;
    out += 2 * (r * stride + c0 + 8 * j);
#pragma unroll
    for (int it = 0; it < CH; it++, r += 32 / CH, out += 2 * (32 / CH) * stride) {
      const uint4 v = *reinterpret_cast<const uint4*>(stage + r * (16 * CH) + ((j ^ flip(r)) << 4));
      if (r >= first && r < last && c0 + 8 * j < D) *reinterpret_cast<uint4*>(out) = v;
    }
  } else {
    const int hj = lane % (2 * CH), j = hj >> 1;
    int r = lane / (2 * CH);
    out += 4 * (r * stride + c0 + 4 * hj);
#pragma unroll
    for (int it = 0; it < 2 * CH; it++, r += 16 / CH, out += 4 * (16 / CH) * stride) {
      const uint2 v = *reinterpret_cast<const uint2*>(stage + r * (16 * CH) + ((j ^ flip(r)) << 4) +
                                                      (hj & 1) * 8);
      const float2 a = unpack2(v.x, fmt), b = unpack2(v.y, fmt);
      if (r >= first && r < last && c0 + 8 * j < D)
        *reinterpret_cast<float4*>(out) = make_float4(a.x, a.y, b.x, b.y);
    }
  }
  __syncwarp();
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
