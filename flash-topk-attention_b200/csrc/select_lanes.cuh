// Top-k select with one row per lane, for up to 32 picks of up to 128 entries: a warp works on
// 32 consecutive rows at once.
//
// A warp per row (select_row.cuh) spends its instructions on sorts across lanes, three per
// step and entry, and shuffles bound it.  Here a lane keeps the best entries of its own row
// sorted in registers: tiles of 32 rows x 16 or 32 entries come through shared memory (cp.async,
// one ahead), every lane sorts its part of the tile and merges it into its list, and a
// compare-exchange is one min and one max for 32 rows.
//
// The sorted keys are 32-bit, the average above the entry's position (lower ones first).  What
// is left for the average are its bits above a base, exactly over half of the range and without
// the lowest `pos_bits` beyond; the base lies a quarter of the range below the smallest one in
// the row's first tile, half an octave with 128 entries, so that the exact half is where the
// others of a row are as a rule (with the base at that one, 24828 rows of 17 entries and 16 picks,
// whose last picks lie below it, took 38 us; so 15).  Averages below the base have place 0.
// Averages that share a place there may come out in the wrong order; the values are read again for
// the result in any case, so neighbours that share one are compared in full and exchanged.  A row
// that this does not settle, or whose last pick shares its place with the first entry left out, is
// selected again by the warp from 64-bit keys; where many rows of a batch are like that, all of them
// are selected again first with a base right below that place.  Averages that are equal and have a
// place to themselves are in order: constant rows, such as zero queries leave, take less than others
// (131072 rows of 128 equal entries, 32 picks 54 us, a warp per row 232, 565 with each of these
// rows selected again; of multiples of 1/8, which tie at the cut, 126, 132 and 265).
//
// Everything but the networks is in loops: with one unrolled body per entry the code outgrew the
// instruction cache, and the same instructions took ten times as long.
// Kilocycles, a warp per row and a lane per row: 16384 rows of 16, 16 picks 16.5, 9.5; 32000 of
// 32, 8 picks 20.6, 13.2; 36000 of 47, 16 picks 32, 18; 131072 of 128, 32 picks 165, 116; 524288
// of 128, 16 picks 420, 276; 240000 of 118, 24 picks 300, 226.  It is the work per entry that
// grows with the row, where a warp per row sorts what is left of a filter: 960000 of 235, 24
// picks 1430, 1479, 131072 of 256, 32 picks 184, 244, and with lists of 64 131072 of 128, 64 picks
// 209, 216.  A queue per lane in front of the sort, for what passes the lane's threshold, was
// slower still (960000 of 235: 2060).
#pragma once

#include "select_row.cuh"

namespace ftk {

constexpr int SL_WARPS = 4;
constexpr int SL_MAX = 128, SL_PICKS = 32;   // entries of a row, picks
constexpr int SL_OUT = 33;    // words between the ranks of the results
constexpr int SL_AGAIN = 8;   // rows of a batch that are not settled: one by one below
// floats between the rows of a tile of kp columns (16-byte columns without bank conflicts)
__host__ __device__ constexpr int sl_pitch(int kp) { return kp + 4; }
__host__ __device__ constexpr int sl_tile(int kp) { return 32 * sl_pitch(kp); }
// keys and values of the picks, or candidates of reselect_row, in bytes
__host__ __device__ constexpr int sl_scratch(int kp) { return (2 * kp * SL_OUT * 4 + 255) & ~255; }
__host__ __device__ constexpr int sl_warp_bytes(int kp) { return 2 * sl_tile(kp) * 4 + sl_scratch(kp); }
// CTAs per SM that registers and shared memory are for
__host__ __device__ constexpr int sl_ctas(int kp) { return kp == 16 ? 5 : 3; }

__device__ __forceinline__ void exchange_desc(unsigned& a, unsigned& b) {
  const unsigned hi = max(a, b);
  b = min(a, b);
  a = hi;
}
// Batcher's odd-even merge sort, largest first: the step that compares at distance K while runs
// of P are merged, and those behind it
template <int P, int K, int N>
__device__ __forceinline__ void sort_lane_from(unsigned (&v)[N]) {
#pragma unroll
  for (int i = K % P; i + K < N; i++)
    if (((i - K % P) & K) == 0 && i / (2 * P) == (i + K) / (2 * P)) exchange_desc(v[i], v[i + K]);
  if constexpr (K > 1) sort_lane_from<P, K / 2>(v);
  else if constexpr (2 * P < N) sort_lane_from<2 * P, 2 * P>(v);
}
template <int N>
__device__ __forceinline__ void sort_lane(unsigned (&v)[N]) {
  sort_lane_from<1, 1>(v);
}
// a bitonic sequence, largest first
template <int N>
__device__ __forceinline__ void merge_lane(unsigned (&v)[N]) {
#pragma unroll
  for (int h = N / 2; h > 0; h >>= 1)
#pragma unroll
    for (int i = 0; i < N; i++)
      if ((i & h) == 0) exchange_desc(v[i], v[i + h]);
}

__device__ __forceinline__ void copy_async16(uint32_t dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async4(uint32_t dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}

// What an entry's average is: the sum over its tokens, of which the first and the last block
// have fewer.  Multiplying by the inverse of a power of two is exact.
struct BlockAverage {
  float inv_bsz;
  int bsz, last, pad_head, pad_tail;
  bool simple;   // a power of two, no padding
  __device__ __forceinline__ float operator()(float raw, int id) const {
    if (simple) return fmaxf(raw * inv_bsz, 0.f);   // NaN / negative: last among real blocks
    const int n = bsz - (id == 0 ? pad_head : 0) - (id == last ? pad_tail : 0);
    return fmaxf(__fdiv_rn(raw, static_cast<float>(n)), 0.f);
  }
};

// An average's place among the others of its row in 32 - pos_bits bits, and the smallest
// average that has it (none for place 0, which is also that of all below `base`).
struct PlaceOf {
  int half, shift;
  __device__ __forceinline__ unsigned operator()(unsigned bits, unsigned base) const {
    const int d = static_cast<int>(max(bits, base) - base);
    return static_cast<unsigned>(min(d, half + ((d - half) >> shift)));
  }
  __device__ __forceinline__ float lowest(unsigned place, unsigned base) const {
    if (place == 0u) return 0.f;
    const unsigned h = static_cast<unsigned>(half);
    return __uint_as_float(base + (place <= h ? place : h + ((place - h) << shift)));
  }
  // whether averages of this place may differ
  __device__ __forceinline__ bool shared(unsigned place, unsigned base) const {
    return place >= static_cast<unsigned>(half) || (place == 0u && base > 0u);
  }
};

// One row by the whole warp, from full keys: all of its entries whose average is at least `low`.
__device__ __noinline__ void reselect_row(const float* in, float inv_total, int M, int M_out,
                                          BlockAverage average, float low, float threshold,
                                          unsigned long long* cand, int32_t* oi, float* orw,
                                          float* oav) {
  static_assert(SL_MAX <= 128, "candidates that are sorted at once");
  const int lane = threadIdx.x & 31;
  int count = 0;
#pragma unroll 1
  for (int c0 = 0; c0 < M; c0 += 32) {
    const int id = c0 + lane;
    const float avg = average(id < M ? in[id] * inv_total : 0.f, id);
    const bool pass = id < M && avg >= low;
    const unsigned b = __ballot_sync(0xffffffffu, pass);
    if (pass)
      cand[count + __popc(b & ((1u << lane) - 1u))] =
          (static_cast<unsigned long long>(__float_as_uint(avg)) << 32) | (0xffffffffu - static_cast<unsigned>(id));
    count += __popc(b);
  }
  __syncwarp();
  if (count <= 64)
    sorted_emit<2, false>(cand, count, lane, in, inv_total, M_out, threshold, oi, orw, oav);
  else
    sorted_emit<4, false>(cand, count, lane, in, inv_total, M_out, threshold, oi, orw, oav);
  __syncwarp();
}

// KP: entries of a lane's list and columns of a tile, 16 or 32, at least M_out.
template <int KP>
__global__ void __launch_bounds__(SL_WARPS * 32, sl_ctas(KP))
topk_select_lanes_kernel(const float* scores, const float* row_scale, int64_t rows, int M, int M_out,
                         int bsz, int pad_head, int pad_tail, float threshold, int32_t* out_idx,
                         float* out_raw, float* out_avg) {
  constexpr int PITCH = sl_pitch(KP), TILE = sl_tile(KP);
  extern __shared__ __align__(16) uint8_t sl_smem[];
  pdl_wait();
  pdl_launch();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint8_t* mine = sl_smem + warp * sl_warp_bytes(KP);
  float* tile_s = reinterpret_cast<float*>(mine);
  unsigned* keys = reinterpret_cast<unsigned*>(mine + 2 * TILE * 4);   // of rank r at SL_OUT * r + lane
  float* vals = reinterpret_cast<float*>(keys + KP * SL_OUT);
  const int pos_bits = 32 - __clz(M);        // 2^pos_bits > M: no key of an entry is 0
  const unsigned pos_mask = (1u << pos_bits) - 1u;
  const PlaceOf place = {1 << (31 - pos_bits), pos_bits};
  const bool pow2 = (bsz & (bsz - 1)) == 0, pads = pad_head > 0 || pad_tail > 0;
  const BlockAverage average = {1.f / static_cast<float>(bsz), bsz, M - 1, pad_head, pad_tail, pow2 && !pads};
  const bool wide = (M & 3) == 0 && (reinterpret_cast<uintptr_t>(scores) & 15) == 0;
  const bool quads = (M_out & 3) == 0 &&
                     ((reinterpret_cast<uintptr_t>(out_idx) | reinterpret_cast<uintptr_t>(out_raw) |
                       reinterpret_cast<uintptr_t>(out_avg)) & 15) == 0;
  const int tiles = (M + KP - 1) / KP;
  const int64_t batches = (rows + 31) >> 5, nwarps = static_cast<int64_t>(gridDim.x) * SL_WARPS;

  // tile t of a batch's rows into buffer `buf`; rows and columns that are not there are left out
  auto fetch = [&](int64_t batch, int t, int buf) {
    if (batch < batches) {
      const int64_t row0 = batch * 32;
      const int left = static_cast<int>(min(static_cast<int64_t>(32), rows - row0));
      const uint32_t dst = smem_u32(tile_s + buf * TILE);
      if (wide) {
        constexpr int PER = KP / 4, STEP = 32 / PER;   // lanes per row, rows at once
        const int c = (lane % PER) * 4, r0 = lane / PER;
        const float* src = scores + (row0 + r0) * M + t * KP + c;
        if (t * KP + c < M) {
#pragma unroll
          for (int r = 0; r < 32; r += STEP)
            if (r0 + r < left) copy_async16(dst + ((r0 + r) * PITCH + c) * 4, src + r * M);
        }
      } else {
        constexpr int STEP = 32 / KP;
        const int c = lane % KP, r0 = lane / KP;
        const float* src = scores + (row0 + r0) * M + t * KP + c;
        if (t * KP + c < M) {
#pragma unroll 4
          for (int r = r0; r < left; r += STEP, src += STEP * M) copy_async4(dst + (r * PITCH + c) * 4, src);
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  int64_t batch = static_cast<int64_t>(blockIdx.x) * SL_WARPS + warp;
  int buf = 1;
  unsigned base = 0u;
  bool again = false;   // the batch once more, `base` is set
  fetch(batch, 0, 0);
#pragma unroll 1
  while (batch < batches) {
    const int64_t row0 = batch * 32;
    const int left = static_cast<int>(min(static_cast<int64_t>(32), rows - row0));
    const int64_t row = row0 + min(lane, left - 1);
    const float inv_total = row_scale ? __frcp_rn(row_scale[row]) : 1.f;
    const float* in = scores + row * M;
    // the two blocks whose averages may have another divisor
    float avg_first = 0.f, avg_last = 0.f;
    if (pads) {
      avg_first = average(in[0] * inv_total, 0);
      avg_last = average(in[M - 1] * inv_total, M - 1);
    }
    unsigned list[KP], rejected = 0u;
#pragma unroll
    for (int i = 0; i < KP; i++) list[i] = 0u;
#pragma unroll 1
    for (int t = 0; t < tiles; t++) {
      // the next tile, or the next batch's first, is under way while this one is worked on
      __syncwarp();   // the other buffer is free
      buf ^= 1;
      float* my = tile_s + buf * TILE + lane * PITCH;
      fetch(t + 1 < tiles ? batch : batch + nwarps, t + 1 < tiles ? t + 1 : 0, buf ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncwarp();
      const int id0 = t * KP, cols = min(KP, M - id0);
      if (!pow2) {   // divisions stay out of the unrolled code
#pragma unroll 1
        for (int j = 0; j < cols; j++) my[j] = average(my[j] * inv_total, id0 + j);
      }
      unsigned v[KP];
#pragma unroll
      for (int j = 0; j < KP; j += 4) {
        const float4 f = *reinterpret_cast<const float4*>(my + j);
        const float x[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
        for (int y = 0; y < 4; y++)
          v[j + y] = __float_as_uint(pow2 ? fmaxf(x[y] * inv_total * average.inv_bsz, 0.f) : x[y]);
      }
      const int at_last = pads ? M - 1 - id0 : -1;
      if (pads && t == 0) v[0] = __float_as_uint(avg_first);
#pragma unroll
      for (int j = 0; j < KP; j++) {
        v[j] = j == at_last ? __float_as_uint(avg_last) : v[j];
        v[j] = j < cols ? v[j] : 0xffffffffu;
      }
      if (t == 0) {
        unsigned lowest = 0xffffffffu;
#pragma unroll
        for (int j = 0; j < KP; j++) lowest = min(lowest, v[j]);
        const unsigned margin = static_cast<unsigned>(place.half) >> 1;
        lowest = lowest > margin ? lowest - margin : 0u;
        base = again ? base : lowest;
      }
#pragma unroll
      for (int j = 0; j < KP; j++)
        v[j] = j < cols ? place(v[j], base) << pos_bits | (pos_mask - static_cast<unsigned>(id0 + j)) : 0u;
      sort_lane<KP>(v);
      // the list against the tile, in opposite order
#pragma unroll
      for (int i = 0; i < KP; i++) {
        if (M_out == KP) rejected = max(rejected, min(list[i], v[KP - 1 - i]));
        list[i] = max(list[i], v[KP - 1 - i]);
      }
      merge_lane(list);
    }

    // ---- the picks' values, whether they are in order, and the running sum that the threshold cuts
    unsigned last = ~0u, next = rejected;
    __syncwarp();
#pragma unroll
    for (int r = 0; r < KP; r++) {
      keys[SL_OUT * r + lane] = list[r];
      if (r < M_out) last = min(last, list[r]);
      else next = max(next, list[r]);
    }
    bool close = false;
    unsigned before = 0u;
#pragma unroll 8
    for (int r = 0; r < M_out; r++) {
      const unsigned k = keys[SL_OUT * r + lane];
      vals[SL_OUT * r + lane] = in[min(pos_mask - (k & pos_mask), static_cast<unsigned>(M - 1))] * inv_total;
      close |= r > 0 && (k ^ before) <= pos_mask && place.shared(k >> pos_bits, base);
      before = k;
    }
    // the last pick and the first entry left out agree in their keys
    bool open = next != 0u && (last ^ next) <= pos_mask && place.shared(last >> pos_bits, base);
    if (__any_sync(0xffffffffu, close)) {
      bool moved = true;
#pragma unroll 1
      for (int pass = 0; pass < 4 && __any_sync(0xffffffffu, moved); pass++) {
        moved = false;
        unsigned k = keys[lane];   // what is carried along: bubbles down
        float f = vals[lane];
        bool have = false;
        float fa = 0.f;
#pragma unroll 1
        for (int r = 1; r < M_out; r++) {
          const unsigned k2 = keys[SL_OUT * r + lane];
          const bool same = (k ^ k2) <= pos_mask;
          if (__any_sync(0xffffffffu, same)) {
            const float f2 = vals[SL_OUT * r + lane];
            if (!have) fa = average(f, pos_mask - (k & pos_mask));
            const float fb = average(f2, pos_mask - (k2 & pos_mask));
            if (same && (fa < fb || (fa == fb && k < k2))) {
              keys[SL_OUT * (r - 1) + lane] = k2;
              vals[SL_OUT * (r - 1) + lane] = f2;
              keys[SL_OUT * r + lane] = k;
              vals[SL_OUT * r + lane] = f;
              moved = true;
            } else {
              k = k2;
              f = f2;
              fa = fb;
            }
            have = true;
          } else {
            k = k2;
            f = vals[SL_OUT * r + lane];
            have = false;
          }
        }
      }
      open |= moved;
    }
    int keep = M_out;
    float cum = 0.f;
#pragma unroll 8
    for (int r = 0; r < M_out; r++) {
      cum += vals[SL_OUT * r + lane];
      if (cum >= threshold) keep = min(keep, r + 1);
    }
    __syncwarp();
    // ---- out: the results of 32 rows are contiguous
    {
      const int64_t at = row0 * M_out;
      auto result = [&](int l, int r, int kept, int& id, float& raw, float& avg) {
        const unsigned k = keys[SL_OUT * r + l];
        const float f = vals[SL_OUT * r + l];
        const int i = static_cast<int>(pos_mask - (k & pos_mask));
        const bool on = r < kept;
        id = on ? i : -1;
        raw = on ? f : 0.f;
        avg = on ? average(f, i) : 0.f;
      };
      const int per = quads ? M_out >> 2 : M_out, n = left * per;
      const int drow = 32 / per, dcol = 32 - drow * per;
      int l = lane / per, c = lane - l * per;
#pragma unroll 1
      for (int e0 = 0; e0 < n; e0 += 32) {
        const int e = e0 + lane, kept = __shfl_sync(0xffffffffu, keep, l & 31);
        if (e < n) {
          if (quads) {
            int id[4];
            float raw[4], avg[4];
#pragma unroll
            for (int y = 0; y < 4; y++) result(l, 4 * c + y, kept, id[y], raw[y], avg[y]);
            reinterpret_cast<int4*>(out_idx + at)[e] = make_int4(id[0], id[1], id[2], id[3]);
            reinterpret_cast<float4*>(out_raw + at)[e] = make_float4(raw[0], raw[1], raw[2], raw[3]);
            reinterpret_cast<float4*>(out_avg + at)[e] = make_float4(avg[0], avg[1], avg[2], avg[3]);
          } else {
            result(l, c, kept, out_idx[at + e], out_raw[at + e], out_avg[at + e]);
          }
        }
        c += dcol;
        l += drow;
        if (c >= per) {
          c -= per;
          l++;
        }
      }
    }
    // ---- rows that are not settled
    unsigned rest = __ballot_sync(0xffffffffu, open && lane < left);
    if (!again && __popc(rest) >= SL_AGAIN) {
      // many that tie at the cut, all at once: with a base right below the place of the last pick
      // its averages have places of their own
      again = true;
      if (open) {
        const unsigned low = last >> pos_bits, reach = static_cast<unsigned>(place.half) - 1u;
        base = low ? __float_as_uint(place.lowest(low, base)) - 1u : base > reach ? base - reach : 0u;
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncwarp();
      fetch(batch, 0, buf ^ 1);
      continue;
    }
    again = false;
#pragma unroll 1
    while (rest) {
      __syncwarp();
      const int l = __ffs(rest) - 1;
      rest &= rest - 1;
      const float low = __shfl_sync(0xffffffffu, place.lowest(last >> pos_bits, base), l);
      const float inv = __shfl_sync(0xffffffffu, inv_total, l);
      const int64_t at = row0 + l;
      reselect_row(scores + at * M, inv, M, M_out, average, low, threshold,
                   reinterpret_cast<unsigned long long*>(keys), out_idx + at * M_out,
                   out_raw + at * M_out, out_avg + at * M_out);
    }
    __syncwarp();
    batch += nwarps;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

}  // namespace ftk
