// Top-k select of one row by one warp (used by topk_select_reg_kernel).
#pragma once

#include "ftk_sm100.cuh"

namespace ftk {

__device__ __forceinline__ int redux_max_s32(int v) {
  int r;
  asm volatile("redux.sync.max.s32 %0, %1, 0xffffffff;" : "=r"(r) : "r"(v));
  return r;
}
__device__ __forceinline__ int redux_min_s32(int v) {
  int r;
  asm volatile("redux.sync.min.s32 %0, %1, 0xffffffff;" : "=r"(r) : "r"(v));
  return r;
}
__device__ __forceinline__ unsigned redux_min_u32(unsigned v) {
  unsigned r;
  asm volatile("redux.sync.min.u32 %0, %1, 0xffffffff;" : "=r"(r) : "r"(v));
  return r;
}

// Bitonic network over 32*E values held E per lane (position p = r*32 + lane),
// sorted largest first.  Distances below 32 exchange across lanes, the others
// between registers of one lane; every index is a compile-time constant.
template <int E, typename T>
__device__ __forceinline__ void bitonic_desc(T (&v)[E], int lane) {
  constexpr int LOGN = (E == 1 ? 5 : E == 2 ? 6 : E == 4 ? 7 : 8);
#pragma unroll
  for (int lk = 1; lk <= LOGN; lk++) {
    const int k = 1 << lk;
#pragma unroll
    for (int lj = lk - 1; lj >= 0; lj--) {
      const int j = 1 << lj;
      if (j >= 32) {
        const int jr = j >> 5;
#pragma unroll
        for (int r = 0; r < E; r++) {
          if ((r & jr) == 0) {
            const bool desc = (((r * 32) & k) == 0);
            const T x = v[r], y = v[r | jr];
            const bool sw = desc ? (x < y) : (x > y);
            v[r] = sw ? y : x;
            v[r | jr] = sw ? x : y;
          }
        }
      } else {
#pragma unroll
        for (int r = 0; r < E; r++) {
          const T o = __shfl_xor_sync(0xffffffffu, v[r], j);
          const bool desc = (((r * 32 + lane) & k) == 0);
          const bool lower = (lane & j) == 0;
          const bool take_max = (desc == lower);
          const bool o_gt = o > v[r];
          v[r] = (take_max == o_gt) ? o : v[r];
        }
      }
    }
  }
}

// ---- 32 * E 32-bit keys, E per lane (position p = r*32 + lane), largest first
// A compare-exchange is one shuffle and one min or max.  In the mirrored form of
// the network (the first step of a merge pairs a lane with its mirror image) the
// lower lane of every pair keeps the larger key, so which of the two a lane does
// depends on one bit of its number.
__device__ __forceinline__ int keep_larger(int v, int lane_mask, bool lower) {
  const int o = __shfl_xor_sync(0xffffffffu, v, lane_mask);
  return lower ? max(v, o) : min(v, o);
}
__device__ __forceinline__ int merge32(int v, int lane) {   // bitonic input
#pragma unroll
  for (int j = 16; j > 0; j >>= 1) v = keep_larger(v, j, (lane & j) == 0);
  return v;
}
__device__ __forceinline__ int sort32(int v, int lane) {
#pragma unroll
  for (int k = 2; k <= 32; k <<= 1) {
    v = keep_larger(v, k - 1, (lane & (k >> 1)) == 0);
#pragma unroll
    for (int j = k >> 2; j > 0; j >>= 1) v = keep_larger(v, j, (lane & j) == 0);
  }
  return v;
}
// v[first .. first + COUNT), already a bitonic sequence of 32 * COUNT keys
template <int COUNT, int E>
__device__ __forceinline__ void merge_keys(int (&v)[E], int first, int lane) {
#pragma unroll
  for (int h = COUNT / 2; h > 0; h >>= 1)
#pragma unroll
    for (int r = 0; r < COUNT; r++)
      if ((r & h) == 0) {
        const int x = v[first + r], y = v[first + (r | h)];
        v[first + r] = max(x, y);
        v[first + (r | h)] = min(x, y);
      }
#pragma unroll
  for (int r = 0; r < COUNT; r++) v[first + r] = merge32(v[first + r], lane);
}
template <int E>
__device__ __forceinline__ void sort_keys(int (&v)[E], int lane) {
#pragma unroll
  for (int r = 0; r < E; r++) v[r] = sort32((r & 1) ? ~v[r] : v[r], lane);   // odd ones ascending
#pragma unroll
  for (int r = 1; r < E; r += 2) v[r] = ~v[r];
  if constexpr (E >= 2) {
#pragma unroll
    for (int r = 0; r < E; r += 2) {
      if (r & 2) {
        v[r] = ~v[r];
        v[r + 1] = ~v[r + 1];
        // ascending: the complement of a bitonic sequence is one
      }
      merge_keys<2>(v, r, lane);
      if (r & 2) {
        v[r] = ~v[r];
        v[r + 1] = ~v[r + 1];
      }
    }
  }
  if constexpr (E == 4) merge_keys<4>(v, 0, lane);
}

// Writes ranks 0 .. M_out - 1 <= 64 of a row: rank q*32 + lane holds the entry with
// key k[q] (average bits high, inverted block id low).  Raw scores are read again
// from the row (just loaded, so from L1).  The running sum that the threshold cuts
// is accumulated in rank order, one addition per rank, exactly like a sequential
// scan, but only where it can reach the threshold at all: the sum of the magnitudes
// in any order, with 2e-5 for rounding (64 additions of 2^-24 each way), bounds it.
template <int SLOTS>
__device__ __forceinline__ void emit_ranks(const unsigned long long (&k)[SLOTS], int lane,
                                           const float* in, float inv_total, int M_out,
                                           float threshold, int32_t* oi, float* orw, float* oav) {
  int id[SLOTS];
  float raw[SLOTS];
  float bound = 0.f;
#pragma unroll
  for (int q = 0; q < SLOTS; q++) {
    id[q] = static_cast<int>(0xffffffffu - static_cast<unsigned>(k[q]));
    raw[q] = 0.f;
    if (q * 32 + lane < M_out) raw[q] = in[id[q]] * inv_total;
    bound += fabsf(raw[q]);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) bound += __shfl_xor_sync(0xffffffffu, bound, d);
  int cutpos = 64;
  if (!(bound * 1.00002f < threshold)) {
    float cum = 0.f, mycum[SLOTS];
#pragma unroll
    for (int q = 0; q < SLOTS; q++) {
      mycum[q] = 0.f;
      for (int p = 0; p < min(M_out - q * 32, 32); p++) {
        cum += __shfl_sync(0xffffffffu, raw[q], p);
        if (p == lane) mycum[q] = cum;
      }
    }
    // first rank whose running sum reaches the threshold
#pragma unroll
    for (int q = SLOTS - 1; q >= 0; q--) {
      const unsigned m =
          __ballot_sync(0xffffffffu, (q * 32 + lane < M_out) && (mycum[q] >= threshold));
      if (m) cutpos = q * 32 + __ffs(m) - 1;
    }
  }
#pragma unroll
  for (int q = 0; q < SLOTS; q++) {
    const int rank = q * 32 + lane;
    if (rank < M_out) {
      const bool keep = rank <= cutpos;
      oi[rank] = keep ? id[q] : -1;
      orw[rank] = keep ? raw[q] : 0.f;
      oav[rank] = keep ? __int_as_float(static_cast<int>(k[q] >> 32)) : 0.f;
    }
  }
}

// Sort `count` <= 32 * E candidates and write the first M_out <= 64 of them.
// FAST: the keys are cut to 32 bits, average bits above the candidate's position, so
// that a compare-exchange is a shuffle and a min / max instead of two shuffles and a
// 64-bit compare and select.  Two candidates that agree in what is left of the
// average (17 mantissa bits at 64 candidates, so one row in a hundred) may come out
// in the wrong order: such a row is sorted again by its full keys.
template <int E, bool FAST>
__device__ __forceinline__ bool sorted_emit(const unsigned long long* cand, int count, int lane,
                                            const float* in, float inv_total, int M_out,
                                            float threshold, int32_t* oi, float* orw, float* oav) {
  constexpr int SLOTS = E >= 2 ? 2 : 1;
  unsigned long long top[SLOTS];
  if constexpr (FAST) {
    constexpr int POS = 32 * E - 1;
    int v[E];
#pragma unroll
    for (int r = 0; r < E; r++) {
      const int p = r * 32 + lane;
      const int hi = reinterpret_cast<const int*>(cand)[2 * p + 1];
      v[r] = p < count ? (hi & ~POS) | (POS - p) : -1;   // averages are >= 0
    }
    sort_keys<E>(v, lane);
    bool close = false;
#pragma unroll
    for (int r = 0; r < E; r++) {
      // the next rank's key; behind the last lane comes the next register's first
      const int src = (r + 1 < E && lane == 0) ? v[r + 1 < E ? r + 1 : r] : v[r];
      const int nx = __shfl_sync(0xffffffffu, src, (lane + 1) & 31);
      const bool has = (r + 1 < E || lane < 31) && nx >= 0;
      close |= has && ((v[r] ^ nx) & ~POS) == 0;
    }
    if (__any_sync(0xffffffffu, close)) return false;
#pragma unroll
    for (int q = 0; q < SLOTS; q++) top[q] = cand[POS - (v[q] & POS)];
  } else {
    unsigned long long v[E];
#pragma unroll
    for (int r = 0; r < E; r++) v[r] = (r * 32 + lane < count) ? cand[r * 32 + lane] : 0ull;
    bitonic_desc<E>(v, lane);
#pragma unroll
    for (int q = 0; q < SLOTS; q++) top[q] = v[q];
  }
  emit_ranks<SLOTS>(top, lane, in, inv_total, M_out, threshold, oi, orw, oav);
  return true;
}

// Top-k of one row with M <= 32 * IPT entries (IPT a compile-time constant), one
// warp: lane l holds entries l, l + 32, ... as average bit patterns in registers.
//
// Up to 64 picks: filter and sort.  Every lane takes the maxima of G groups of its
// slots: 32 * G distinct entries, so their M_out-th largest (or a smaller one of
// them) is a lower bound T of the M_out-th largest entry, and {average >= T} holds
// every entry the result can contain, ties included.  That set (about 42 of 512
// entries for 32 picks) is compacted, sorted and written.  Rows of at most 64
// entries are sorted as they are.  The kernel is bound by the integer pipe and by
// shuffles, so the sorts work on 32-bit keys with one min / max per step: 2^20 rows
// of 512 entries, 32 picks, take 0.96 ms (1.92 with 64-bit keys throughout), 2^18
// rows of 1024 entries, 64 picks, 0.78 (1.28).
// More picks, or more candidates than the scratch holds (flat rows): extraction,
// one warp-wide maximum per pick, with each lane's runner-up cached.
//
// `rawv` = the lane's slots of the row `in` (loaded by the caller so that it can
// have the next row's loads in flight; absent ones anything); `inv_total` is
// multiplied in first (scoring hands over unnormalised sums and one total per row;
// 1 otherwise).  `cand`: 256 keys of shared memory, the warp's own.
constexpr int SEL_CAND = 256;

template <int IPT>
__device__ __forceinline__ void select_row_reg(const float (&rawv)[IPT], const float* in,
                                               float inv_total, int M, int M_out, int bsz,
                                               int pad_head, int pad_tail, float threshold,
                                               unsigned long long* cand, int lane, int32_t* oi,
                                               float* orw, float* oav) {
  // dividing by a power of two is exact as a multiplication: same bits, no divide
  const bool pow2 = (bsz & (bsz - 1)) == 0;
  const float inv_bsz = 1.f / static_cast<float>(bsz);
  const int NEG = __float_as_int(-1.f);

  int a[IPT];   // average bit patterns (non-negative floats order as ints); NEG = absent
  if (pow2) {
#pragma unroll
    for (int i = 0; i < IPT; i++)   // NaN / negative input: ranks last among real blocks
      a[i] = __float_as_int(fmaxf(rawv[i] * inv_total * inv_bsz, 0.f));
    if (pad_head > 0 || pad_tail > 0) {   // the first and the last block hold fewer tokens
#pragma unroll
      for (int i = 0; i < IPT; i++) {
        const int j = i * 32 + lane;
        if ((i == 0 && j == 0) || j == M - 1) {
          const int n = bsz - (j == 0 ? pad_head : 0) - (j == M - 1 ? pad_tail : 0);
          a[i] = __float_as_int(fmaxf(__fdiv_rn(rawv[i] * inv_total, static_cast<float>(n)), 0.f));
        }
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < IPT; i++) {
      const int j = i * 32 + lane;
      const int n = bsz - (j == 0 ? pad_head : 0) - (j == M - 1 ? pad_tail : 0);
      a[i] = __float_as_int(fmaxf(__fdiv_rn(rawv[i] * inv_total, static_cast<float>(n)), 0.f));
    }
  }
#pragma unroll
  for (int i = IPT / 2; i < IPT; i++)   // M > 16 * IPT: only the upper slots can be absent
    if (i * 32 + lane >= M) a[i] = NEG;

  auto key64 = [&](int i) {
    return (static_cast<unsigned long long>(static_cast<unsigned>(a[i])) << 32) |
           (0xffffffffu - static_cast<unsigned>(i * 32 + lane));
  };
  if constexpr (IPT <= 2) {
    // every entry is a candidate, position = block id
    if (M_out <= 32 || IPT == 2) {
#pragma unroll
      for (int i = 0; i < IPT; i++) cand[i * 32 + lane] = key64(i);
      __syncwarp();
      if (!sorted_emit<IPT, true>(cand, M, lane, in, inv_total, M_out, threshold, oi, orw, oav))
        sorted_emit<IPT, false>(cand, M, lane, in, inv_total, M_out, threshold, oi, orw, oav);
      return;
    }
  } else if (M_out <= 64) {
    int T;
    if (M_out <= 16) {
      int g = a[0];
#pragma unroll
      for (int i = 1; i < IPT; i++) g = max(g, a[i]);
      T = __shfl_sync(0xffffffffu, sort32(g, lane), M_out - 1);
    } else if (M_out <= 32) {
      // the larger half of two sorted sets of 32: lane by lane the larger of one in
      // descending and the other in ascending order
      int g[2] = {NEG, NEG};
#pragma unroll
      for (int i = 0; i < IPT; i++) g[i >= IPT / 2] = max(g[i >= IPT / 2], a[i]);
      T = redux_min_s32(max(sort32(g[0], lane), ~sort32(~g[1], lane)));
    } else {
      int g[4] = {NEG, NEG, NEG, NEG};
#pragma unroll
      for (int i = 0; i < IPT; i++) g[(4 * i) / IPT] = max(g[(4 * i) / IPT], a[i]);
      int x[2] = {g[0], g[1]}, y[2] = {~g[2], ~g[3]};
      sort_keys<2>(x, lane);
      sort_keys<2>(y, lane);
      T = redux_min_s32(min(max(x[0], ~y[0]), max(x[1], ~y[1])));
    }
    T = max(T, 0);   // fewer real entries than picks among the maxima: all of them
    int mine = 0;
#pragma unroll
    for (int i = 0; i < IPT; i++) mine += a[i] >= T ? 1 : 0;
    int incl = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += v;
    }
    const int count = __shfl_sync(0xffffffffu, incl, 31);
    if (count <= SEL_CAND) {
      unsigned long long* dst = cand + (incl - mine);
#pragma unroll
      for (int i = 0; i < IPT; i++)
        if (a[i] >= T) *dst++ = key64(i);
      __syncwarp();
      bool done = false;
      if (count <= 32 && M_out <= 32)
        done = sorted_emit<1, true>(cand, count, lane, in, inv_total, M_out, threshold, oi, orw, oav);
      else if (count <= 64)
        done = sorted_emit<2, true>(cand, count, lane, in, inv_total, M_out, threshold, oi, orw, oav);
      else if (count <= 128)
        done = sorted_emit<4, true>(cand, count, lane, in, inv_total, M_out, threshold, oi, orw, oav);
      if (done) return;
      if (count <= 64)
        sorted_emit<2, false>(cand, count, lane, in, inv_total, M_out, threshold, oi, orw, oav);
      else if (count <= 128)
        sorted_emit<4, false>(cand, count, lane, in, inv_total, M_out, threshold, oi, orw, oav);
      else
        sorted_emit<8, false>(cand, count, lane, in, inv_total, M_out, threshold, oi, orw, oav);
      return;
    }
  }

  // best and runner-up of the lane; ties keep the lower slot (= lower id)
  int b1 = NEG, i1 = IPT, b2 = NEG, i2 = IPT;
  auto rescan = [&]() {
    b1 = NEG; i1 = IPT; b2 = NEG; i2 = IPT;
#pragma unroll
    for (int i = 0; i < IPT; i++) {
      const int v = a[i];
      if (v > b1) { b2 = b1; i2 = i1; b1 = v; i1 = i; }
      else if (v > b2) { b2 = v; i2 = i; }
    }
  };
  rescan();
  float cum = 0.f;
  bool cut = false;
  int hold_idx = -1;
  float hold_raw = 0.f, hold_avg = 0.f;
  for (int r = 0; r < M_out; r++) {
    int w_idx = -1;
    float w_raw = 0.f, w_avg = 0.f;
    if (!cut) {
      const int mx = redux_max_s32(b1);
      const unsigned mine =
          (b1 == mx) ? static_cast<unsigned>(i1 * 32 + lane) : 0xffffffffu;
      const unsigned win = redux_min_u32(mine);
      w_idx = static_cast<int>(win);
      w_raw = in[win] * inv_total;
      w_avg = __int_as_float(mx);
      cum += w_raw;
      if (cum >= threshold) cut = true;
      if ((win & 31u) == static_cast<unsigned>(lane)) {
        // pop: the slot is consumed; promote the runner-up, rescan only when
        // there is none cached
#pragma unroll
        for (int i = 0; i < IPT; i++)
          if (i == i1) a[i] = NEG;
        if (i2 < IPT) {
          b1 = b2; i1 = i2; b2 = NEG; i2 = IPT;
        } else {
          rescan();
        }
      }
    }
    if ((r & 31) == lane) { hold_idx = w_idx; hold_raw = w_raw; hold_avg = w_avg; }
    if ((r & 31) == 31 || r == M_out - 1) {
      const int base = r & ~31;
      if (base + lane <= r) {
        oi[base + lane] = hold_idx;
        orw[base + lane] = hold_raw;
        oav[base + lane] = hold_avg;
      }
    }
  }
}

}  // namespace ftk
