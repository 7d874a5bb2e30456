// Gathered-KV flash attention forward for sm_100a.
//
// Replaces sparse_attn_fwd_kernel of the reference
// (flash_topk_attn_v2/csrc/sparse_attn_kernel.cu:6-365).
//
// The exact running-maximum kernel below takes every supported shape and dtype.
// For q and kv blocks of 64 or 32 rows the pipelined fixed-reference kernels of
// sparse_fwd_pipe.cuh (one CTA per tile) and sparse_fwd_pipe2.cuh (pairs of SMs)
// run first, when the caller passes a workspace; the exact kernel then only
// redoes the tiles that they flag.
//
// One CTA owns 128 consecutive virtual query rows = G q-blocks of one (batch,
// head) slice and walks the union of their candidate KV blocks in ascending
// order (see attn_common.cuh).  Roles: warp 0 = TMA producer (Q once, then a
// ring of K/V block tiles), warp 1 = UMMA issuer, warps 2..9 = two softmax
// groups of 128 threads, one query row per thread in each group.
//   S = Q K^T      tcgen05 SS, both operands K-major, accumulator in TMEM
//   P = 2^(c S - m) rounded to the I/O dtype, written over the S columns
//   O += P V       tcgen05 with A = P from TMEM, B = V read MN-major from the
//                  same row-major tile TMA delivered
// Even union entries go through S buffer 0 / softmax group 0 / accumulator
// O0, odd entries through buffer 1 / group 1 / O1, so the two groups work
// concurrently and the tensor core alternates between them; each group keeps
// its own running maximum and sum and the two partial results are merged in
// the epilogue (split-KV merge).  A group raises its running maximum only
// when a block exceeds it by more than 2^8 (P stays inside fp16 range); its
// O accumulator is then rescaled in TMEM by the row owners.
#include <cfloat>
#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "attn_common.cuh"
#include "attn_host.cuh"
#include "ftk_host.cuh"
#include "ftk_sm100.cuh"

namespace ftk {

constexpr int FW_THREADS = 320;  // 2 + 2 x 4 warps
constexpr int FW_MAX_STAGES = 4;
// A redo CTA looks at the words of this many tiles at once, 16 bytes a load.
constexpr int REDO_LOADS = 8;
constexpr int REDO_LOOK = FW_THREADS * REDO_LOADS * 4;
constexpr int REDO_QUEUE = 128;   // and takes up to so many of them, where CTAs * REDO_QUEUE >= REDO_LOOK
// TMEM columns.  kv blocks of at most 64 rows: Q (16-bit pairs) 0..63, S[2]
// at 64 / 128, so the S UMMAs read their A operand from TMEM and shared-memory
// bandwidth is left to the K/V tiles (an SS UMMA of this shape spends more
// time fetching Q than multiplying).  Larger kv blocks: S[2] at 0 / 128 and Q
// stays in shared memory.  P is written over the S columns.  O[2] at 256 / 384.
constexpr int FW_COL_O = 256;

struct FwdParams {
  int N, H, QM, W, Mkv;
  int g, kvb, q_pad_head, kv_pad_head;
  int G, fmt, nstages;
  float scale_log2;
  const int32_t* merged;
  void* o;
  int64_t so_b, so_n, so_h;
  float* lse;
  int* status;
  int kv_hdiv;          // query heads per kv head (grouped-query attention), 1 otherwise
  int* redo_out;        // pipelined kernel: one word per 128-row tile, 1 = redo with the exact kernel
  const int* redo_in;   // exact kernel: when set, only tiles whose word is 1 are done
  int list_rows;        // rows of the caller's lists per slice
  int tiles_x, tiles;   // 128-row tiles per slice, and of all slices
  int D;                // columns of a row of O (the kernel's head dim less its padding)
  int out_f32;          // O is float32 (the 16-bit result, widened)
  int sub;              // listed kv blocks per tile (pipelined kernels)
  ListMap lm;
};

// What the exact kernel does: all tiles, or those that the pipelined one marked
enum : int { EXACT = 0, REDO_OWN = 1, REDO_DEAL = 2 };

// Where a redo CTA's look through the words stands, and the tiles that it found for itself.
struct RedoScan {
  int look, before;          // words looked at, marked tiles among them
  int warps[FW_THREADS / 32];
  int queue[REDO_QUEUE];
};
// REDO_DEAL: every CTA looks at all words, REDO_LOOK at a time, and does those of the marked tiles,
// counted as they come, whose number is its own (mod the CTAs).  Fills the queue with the next of
// them and returns how many there are, 0 behind the last; all threads call it.  A redone tile walks its
// whole list, 100 us for 7000 keys, and when a CTA looks at every gridDim.x-th word only, some have two
// or three marked tiles to do while most have none (fp16, 15000 tokens, H = 16, 17 to 109 of 1888
// tiles marked: 380 us, 221 dealt).  A thread counts the marked ones among its own words and
// knows from the counts before which of them the CTA does, so that marked tiles which others do
// cost nothing (1024 of 1024 tiles marked, lists of 2, head dim 64: forward 94 us, 285 with a walk
// over all of them).
__device__ __noinline__ int next_marked(const int* words, unsigned tiles, RedoScan* s, bool first) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, ctas = gridDim.x;
  const bool wide = (reinterpret_cast<uintptr_t>(words) & 15) == 0;
  if (first) {   // as a rule there are none
    int any = 0;
#pragma unroll 4
    for (unsigned t = 4u * tid; t < tiles; t += 4u * FW_THREADS) {
      if (wide && t + 4 <= tiles) {
        const int4 q = *reinterpret_cast<const int4*>(words + t);
        any |= q.x | q.y | q.z | q.w;
      } else {
        for (unsigned x = t; x < min(t + 4u, tiles); x++) any |= words[x];
      }
    }
    if (!__syncthreads_or(any)) return 0;
  }
  int before = first ? 0 : s->before;
#pragma unroll 1
  for (unsigned look = first ? 0u : s->look; look < tiles; look += REDO_LOOK) {
    unsigned mine = 0;   // bit 4 * k + x: word x of load k
#pragma unroll 4
    for (int k = 0; k < REDO_LOADS; k++) {
      const unsigned t = look + 4u * (k * FW_THREADS + tid);
      unsigned marks = 0;
      if (wide && t + 4 <= tiles) {
        const int4 q = *reinterpret_cast<const int4*>(words + t);
        marks = (q.x != 0 ? 1u : 0u) | (q.y != 0 ? 2u : 0u) | (q.z != 0 ? 4u : 0u) | (q.w != 0 ? 8u : 0u);
      } else {
        for (unsigned x = 0; x < 4 && t + x < tiles; x++) marks |= words[t + x] != 0 ? 1u << x : 0u;
      }
      mine |= marks << (4 * k);
    }
    if (!__syncthreads_or(mine != 0u)) continue;
    const int count = __popc(mine);
    int upto = count;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, upto, d);
      if (lane >= d) upto += o;
    }
    if (lane == 31) s->warps[warp] = upto;
    __syncthreads();
    int ahead = upto - count, total = 0;
#pragma unroll 1
    for (int x = 0; x < FW_THREADS / 32; x++) {
      const int n = s->warps[x];
      ahead += x < warp ? n : 0;
      total += n;
    }
    // CTAs of neighbouring numbers are neighbours on the chip, so that neighbouring tiles go to
    // distant ones (the factor has none in common with the number of CTAs): of the marked tiles of
    // this round, counted from 0, this CTA does `start`, `start` + ctas, ...
    const int own = static_cast<int>(blockIdx.x) * (ctas % 17 ? 17 : 19) % ctas;
    const int start = (own + ctas - before % ctas) % ctas;
    for (int at = ahead <= start ? 0 : (ahead - start + ctas - 1) / ctas; start + at * ctas < ahead + count; at++) {
      unsigned rest = mine;
#pragma unroll 1
      for (int skip = start + at * ctas - ahead; skip > 0; skip--) rest &= rest - 1;
      const int i = __ffs(rest) - 1;
      s->queue[at] = static_cast<int>(look + 4u * ((i >> 2) * FW_THREADS + tid) + (i & 3));
    }
    before += total;
    if (start < total) {
      if (tid == 0) {
        s->look = look + REDO_LOOK;
        s->before = before;
      }
      __syncthreads();
      return (total - start + ctas - 1) / ctas;
    }
    __syncthreads();   // the counts are read
  }
  return 0;
}

// D = head dim of the Q.K^T contraction, DV = columns of V / O.  Head dim 256: two 256-column accumulators do not
// fit TMEM next to S, so there is ONE accumulator (columns 256..511) and one
// softmax group with one running maximum drains both S buffers in turn; Q
// stays in shared memory.  The tile's UMMAs (16 + 4 k-steps) outlast its
// softmax, so one group keeps up.  The second group only helps in the epilogue.
//
// One CTA per 128-row tile; behind the pipelined kernel instead one CTA per
// SM that looks through that kernel's redo words and loops over its share of the
// tiles it finds (as a rule none): a grid of one CTA per tile, each leaving on
// its first instruction, took 69 us at 8192 tiles.
template <int D, int DV, int MODE>
__global__ void __launch_bounds__(FW_THREADS, 1)
sparse_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                  const __grid_constant__ CUtensorMap tm_v, const FwdParams p) {
  constexpr int NCH = D / 64;
  constexpr int NCV = DV / 64;
  constexpr bool SINGLE = DV > 128;     // one O accumulator, one softmax group
  constexpr int Q_BYTES = NCH * 128 * 128;
  constexpr bool REDO = MODE != EXACT;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem;
  uint8_t* sKV = smem + Q_BYTES;
  __shared__ UnionScratch un;
  __shared__ __align__(8) uint64_t bars[3 + 2 * FW_MAX_STAGES + 4];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_flag;
  __shared__ float s_m[2][128], s_l[2][128];
  __shared__ OutTile s_out;
  __shared__ std::conditional_t<MODE == REDO_DEAL, RedoScan, int> s_scan;
  __shared__ unsigned s_todo[(FW_THREADS + 31) / 32];

  pdl_wait();
  bool first_tile = true;
  uint32_t tmem = 0;
  // REDO_OWN: FW_THREADS redo words are looked at together, tiles blockIdx.x,
  // blockIdx.x + gridDim.x, ...; returns the next one to do, -1 behind the last
  int64_t base = blockIdx.x - static_cast<int64_t>(gridDim.x) * FW_THREADS;
  int word = FW_THREADS / 32;
  unsigned left = 0;
  auto next_tile = [&]() -> int {
    if constexpr (MODE == REDO_DEAL) {
      if (left == 0) left = next_marked(p.redo_in, p.tiles, &s_scan, first_tile);
      return left == 0 ? -1 : s_scan.queue[--left];
    }
    if (MODE == EXACT) return first_tile ? static_cast<int>(blockIdx.x) : -1;
    while (left == 0) {
      if (word < FW_THREADS / 32) {
        left = s_todo[word++];
        continue;
      }
      base += static_cast<int64_t>(gridDim.x) * FW_THREADS;
      if (base >= p.tiles) return -1;
      __syncthreads();
      const int64_t t = base + static_cast<int64_t>(threadIdx.x) * gridDim.x;
      const unsigned bal = __ballot_sync(0xffffffffu, t < p.tiles && p.redo_in[t] != 0);
      if ((threadIdx.x & 31) == 0) s_todo[threadIdx.x >> 5] = bal;
      __syncthreads();
      word = 0;
    }
    const int bit = __ffs(left) - 1;
    left &= left - 1;
    return static_cast<int>(base + static_cast<int64_t>((word - 1) * 32 + bit) * gridDim.x);
  };
  for (int tile = next_tile(); tile >= 0; tile = next_tile()) {
  // read anew for every tile: what is derived from it is not kept across the loop
  const int tid = REDO ? late_tid() : threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int bh = tile / p.tiles_x;
  const int m0 = (tile - bh * p.tiles_x) * p.G;
  const int b_idx = bh / p.H, h_idx = bh - b_idx * p.H;
  const int groups = min(p.G, p.QM - m0);
  const int tile_row0 = m0 * p.g - p.q_pad_head;
  const int kv_chunk_bytes = p.kvb * 128;
  const int stage_bytes = (NCH + NCV) * kv_chunk_bytes;
  const int NST = p.nstages;

  const uint32_t bar_q = smem_u32(&bars[0]);
  const uint32_t bar_final = smem_u32(&bars[1]);
  const uint32_t bar_qt = smem_u32(&bars[2]);   // Q copied into TMEM
  auto bar_kvfull = [&](int s) { return smem_u32(&bars[3 + s]); };
  auto bar_kvempty = [&](int s) { return smem_u32(&bars[3 + FW_MAX_STAGES + s]); };
  auto bar_sfull = [&](int s) { return smem_u32(&bars[3 + 2 * FW_MAX_STAGES + s]); };
  auto bar_pfull = [&](int s) { return smem_u32(&bars[3 + 2 * FW_MAX_STAGES + 2 + s]); };
  const bool q_tmem = D <= 128 && p.kvb <= 64;
  const uint32_t s_col0 = q_tmem ? 64u : 0u, s_stride = q_tmem ? 64u : 128u;

  if (tid == 0) {
    if (!REDO || first_tile) {
      abort_flag = 0;
    } else {
      for (auto& b : bars) mbar_inval(smem_u32(&b));
    }
    mbar_init(bar_q, 1);
    mbar_init(bar_final, 1);
    mbar_init(bar_qt, 4);
    for (int s = 0; s < FW_MAX_STAGES; s++) {
      mbar_init(bar_kvfull(s), 1);
      mbar_init(bar_kvempty(s), 1);
    }
    for (int s = 0; s < 2; s++) {
      mbar_init(bar_sfull(s), 1);
      mbar_init(bar_pfull(s), 4);  // one arrival per warp of the owning group
    }
    mbar_init_fence();
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
  }
  if (warp == 0 && (!REDO || first_tile)) {
    tmem_alloc(smem_u32(&tmem_base_s), 512);
    tmem_relinquish();
  }
  if (tid == 32)
    s_out = {{static_cast<int64_t>(b_idx) * p.so_b + static_cast<int64_t>(h_idx) * p.so_h, 0},
             tile_row0, min(p.N, tile_row0 + groups * p.g)};
  clear_flags(sKV, p.Mkv, groups);
  const int n = build_union<FW_THREADS / 32>(un, sKV, p.merged + static_cast<int64_t>(bh) * p.list_rows * p.W, m0, groups,
                            p.W, nullptr, p.Mkv, 1, p.lm, p.status);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (first_tile) pdl_launch();   // a REDO CTA without a tile by leaving
  first_tile = false;
  tmem = tmem_base_s;
  WaitCtx w{&abort_flag, p.status};

  if (warp == 0) {
    // ------------------------------------------------------- TMA producer
    if (lane == 0 && n > 0) {
      mbar_expect_tx(bar_q, Q_BYTES);
      for (int c = 0; c < NCH; c++)
        tma_load_4d(smem_u32(sQ) + c * 128 * 128, &tm_q, bar_q, c * 64, h_idx, tile_row0, b_idx);
      const int hk = h_idx / p.kv_hdiv;   // out of the loop: a division takes 150 cycles
      for (int i = 0; i < n; i++) {
        const int s = i % NST;
        const uint32_t ph = (i / NST) & 1;
        if (!mbar_wait(bar_kvempty(s), ph ^ 1, w, FTK_DEV_TIMEOUT_TMA)) break;
        const int tok0 = static_cast<int>(un.ids[i]) * p.kvb - p.kv_pad_head;
        const uint32_t base = smem_u32(sKV) + s * stage_bytes;
        mbar_expect_tx(bar_kvfull(s), stage_bytes);
        for (int c = 0; c < NCH; c++)
          tma_load_4d(base + c * kv_chunk_bytes, &tm_k, bar_kvfull(s), c * 64, hk,
                      tok0, b_idx);
        for (int c = 0; c < NCV; c++)
          tma_load_4d(base + (NCH + c) * kv_chunk_bytes, &tm_v, bar_kvfull(s), c * 64,
                      hk, tok0, b_idx);
      }
      // before the barriers are set up anew for another tile, every commit has arrived
      for (int i = max(0, n - NST); REDO && i < n; i++)
        if (!mbar_wait(bar_kvempty(i % NST), (i / NST) & 1, w, FTK_DEV_TIMEOUT_TMA)) break;
    }
  } else if (warp == 1) {
    // -------------------------------------------------------- UMMA issuer
    if (n > 0) {
      // the whole warp runs this path; one elected lane issues the UMMAs
      const uint32_t idesc_s = umma_idesc(128, p.kvb, p.fmt, 0, 0);
      const uint32_t idesc_pv = umma_idesc(128, DV, p.fmt, 0, 1);
      const uint64_t qdesc0 = smem_desc_sw128(smem_u32(sQ), 16, 1024);
      const uint64_t kdesc0 = smem_desc_sw128(smem_u32(sKV), 16, 1024);
      const uint64_t vdesc0 =
          smem_desc_sw128(smem_u32(sKV) + NCH * kv_chunk_bytes, kv_chunk_bytes, 1024);
      bool ok = mbar_wait(q_tmem ? bar_qt : bar_q, 0, w, FTK_DEV_TIMEOUT_MMA);
      tc_fence_after();
      auto issue_s = [&](int i) -> bool {
        const int s = i % NST;
        if (!mbar_wait(bar_kvfull(s), (i / NST) & 1, w, FTK_DEV_TIMEOUT_MMA)) return false;
        tc_fence_after();
        const uint64_t kdesc = desc_advance(kdesc0, s * stage_bytes);
        const uint32_t d_tmem = tmem + s_col0 + (i & 1) * s_stride;
        if (elect_one()) {
          if (q_tmem) {
#pragma unroll
            for (int ks = 0; ks < D / 16; ks++)
              umma_ts(d_tmem, tmem + ks * 8,
                      desc_advance(kdesc, (ks / 4) * kv_chunk_bytes + (ks % 4) * 32), idesc_s,
                      ks > 0);
          } else {
#pragma unroll
            for (int ks = 0; ks < D / 16; ks++)
              umma_ss(d_tmem, desc_advance(qdesc0, (ks / 4) * 128 * 128 + (ks % 4) * 32),
                      desc_advance(kdesc, (ks / 4) * kv_chunk_bytes + (ks % 4) * 32), idesc_s,
                      ks > 0);
          }
          umma_commit(bar_sfull(i & 1));
        }
        __syncwarp();
        return true;
      };
      if (ok) ok = issue_s(0);
      if (ok && n > 1) ok = issue_s(1);
      for (int i = 0; ok && i < n; i++) {
        const int s = i % NST, sb = i & 1;
        if (!mbar_wait(bar_pfull(sb), (i >> 1) & 1, w, FTK_DEV_TIMEOUT_MMA)) { ok = false; break; }
        tc_fence_after();
        const uint64_t vdesc = desc_advance(vdesc0, s * stage_bytes);
        const int ksteps = p.kvb / 16;
        if (elect_one()) {
          for (int ks = 0; ks < ksteps; ks++) {
            umma_ts(tmem + FW_COL_O + (SINGLE ? 0 : sb * 128),
                    tmem + s_col0 + sb * s_stride + ks * 8, desc_advance(vdesc, ks * 2048),
                    idesc_pv, (i >= (SINGLE ? 1 : 2)) || (ks > 0));
          }
          umma_commit(bar_kvempty(s));
        }
        __syncwarp();
        // S(i+2) overwrites the columns PV(i) reads P from; the tensor core
        // runs UMMAs in issue order, so issuing it after PV(i) is enough.
        if (i + 2 < n) ok = issue_s(i + 2);
      }
      if (ok && elect_one()) umma_commit(bar_final);
      __syncwarp();
    }
  } else {
    // ---------------------------------------------------- softmax threads
    const int grp_w = (warp - 2) >> 2;       // softmax group = S buffer it drains
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const int grp = r / p.g;
    const int qrow = tile_row0 + r;
    const bool row_valid = (grp < groups) && qrow >= 0 && qrow < p.N;
    const uint32_t lane_addr = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t o_addr = lane_addr + FW_COL_O + (SINGLE ? 0 : grp_w * 128);
    const float c = p.scale_log2;
    // a finite number also while no logit is: 2^(-inf - m_run) is 0, and the first finite one is above it
    float m_run = -FLT_MAX, l = 0.f;
    bool ok = true;

    if (q_tmem && n > 0 && grp_w == 0) {
      // group 0 moves the Q tile from (swizzled) shared memory into TMEM:
      // row r -> lane r, two 16-bit values per column
      ok = mbar_wait(bar_q, 0, w, FTK_DEV_TIMEOUT_CONSUMER);
      if (ok) {
#pragma unroll
        for (int ch = 0; ch < NCH; ch++) {
          uint32_t v[32];
#pragma unroll
          for (int j = 0; j < 8; j++) {
            const uint4 t4 =
                *reinterpret_cast<const uint4*>(sQ + ch * 128 * 128 + sw128_offset(r, j));
            v[j * 4 + 0] = t4.x;
            v[j * 4 + 1] = t4.y;
            v[j * 4 + 2] = t4.z;
            v[j * 4 + 3] = t4.w;
          }
          tmem_st32(lane_addr + ch * 32, v);
        }
        tmem_wait_st();
        tc_fence_before();
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_qt);
    }

    for (int i = SINGLE ? (grp_w == 0 ? 0 : n) : grp_w; ok && i < n; i += SINGLE ? 1 : 2) {
      // S(i) complete also means PV(i-2) has retired (same issue order), so
      // this buffer's P columns (and with two groups: this group's O
      // accumulator) are free to touch.
      const int sbuf = SINGLE ? (i & 1) : grp_w;
      const uint32_t s_addr = lane_addr + s_col0 + sbuf * s_stride;
      if (!mbar_wait(bar_sfull(sbuf), (i >> 1) & 1, w, FTK_DEV_TIMEOUT_CONSUMER)) {
        ok = false;
        break;
      }
      tc_fence_after();
      // One shared accumulator: PV(i-1) may still be adding to it.  A thread
      // that has to rescale it first waits until that UMMA has retired (the
      // commit that hands tile i-1's K / V stage back to the producer).
      auto o_quiet = [&]() -> bool {
        if (!SINGLE || i == 0) return true;
        const int sp = (i - 1) % NST;
        if (!mbar_wait(bar_kvempty(sp), ((i - 1) / NST) & 1, w, FTK_DEV_TIMEOUT_CONSUMER))
          return false;
        tc_fence_after();
        return true;
      };
      const int tok0 = static_cast<int>(un.ids[i]) * p.kvb - p.kv_pad_head;
      const int lo = max(0, -tok0), hi = min(p.kvb, p.N - tok0);
      const bool act = row_valid && ((un.masks[i] >> grp) & 1) && hi > lo;
      const bool any_act = __any_sync(0xffffffffu, act);
      const bool fast = __all_sync(0xffffffffu, act) && lo == 0 && hi == p.kvb;

      if (any_act && p.kvb == 64) {
        // ---- whole row of S in registers, one TMEM round trip
        uint32_t v0[32], v1[32];
        tmem_ld32(s_addr, v0);
        tmem_ld32(s_addr + 32, v1);
        tmem_wait_ld();
        float mt = -INFINITY;
        if (fast) {
#pragma unroll
          for (int x = 0; x < 32; x++)
            mt = fmaxf(mt, fmaxf(__uint_as_float(v0[x]), __uint_as_float(v1[x])));
        } else if (act) {
#pragma unroll
          for (int x = 0; x < 32; x++) {
            if (x >= lo && x < hi) mt = fmaxf(mt, __uint_as_float(v0[x]));
            if (x + 32 >= lo && x + 32 < hi) mt = fmaxf(mt, __uint_as_float(v1[x]));
          }
        }
        const float mt2 = act ? mt * c : -INFINITY;
        const bool grow = act && mt2 > m_run + 8.f;
        const float m_new = grow ? mt2 : m_run;
        const bool resc = grow && l > 0.f;
        if (__any_sync(0xffffffffu, resc)) {
          if (!o_quiet()) {
            ok = false;
            break;
          }
          const float alpha = resc ? fast_exp2(m_run - m_new) : 1.f;
          for (int c0 = 0; c0 < DV; c0 += 32) {
            uint32_t ov[32];
            tmem_ld32(o_addr + c0, ov);
            tmem_wait_ld();
#pragma unroll
            for (int x = 0; x < 32; x++) ov[x] = __float_as_uint(__uint_as_float(ov[x]) * alpha);
            tmem_st32(o_addr + c0, ov);
          }
          l *= alpha;
        }
        m_run = m_new;
        uint32_t pk[32];
        float l0 = 0.f, l1 = 0.f;
        if (fast) {
#pragma unroll
          for (int x = 0; x < 32; x += 2) {
            const float a0 = fast_exp2(fmaf(__uint_as_float(v0[x]), c, -m_run));
            const float a1 = fast_exp2(fmaf(__uint_as_float(v0[x + 1]), c, -m_run));
            const float b0 = fast_exp2(fmaf(__uint_as_float(v1[x]), c, -m_run));
            const float b1 = fast_exp2(fmaf(__uint_as_float(v1[x + 1]), c, -m_run));
            l0 += a0 + a1;
            l1 += b0 + b1;
            pk[x >> 1] = pack2(a0, a1, p.fmt);
            pk[16 + (x >> 1)] = pack2(b0, b1, p.fmt);
          }
        } else {
#pragma unroll
          for (int x = 0; x < 32; x += 2) {
            float a0 = 0.f, a1 = 0.f, b0 = 0.f, b1 = 0.f;
            if (act && x >= lo && x < hi) a0 = fast_exp2(fmaf(__uint_as_float(v0[x]), c, -m_run));
            if (act && x + 1 >= lo && x + 1 < hi)
              a1 = fast_exp2(fmaf(__uint_as_float(v0[x + 1]), c, -m_run));
            if (act && x + 32 >= lo && x + 32 < hi)
              b0 = fast_exp2(fmaf(__uint_as_float(v1[x]), c, -m_run));
            if (act && x + 33 >= lo && x + 33 < hi)
              b1 = fast_exp2(fmaf(__uint_as_float(v1[x + 1]), c, -m_run));
            l0 += a0 + a1;
            l1 += b0 + b1;
            pk[x >> 1] = pack2(a0, a1, p.fmt);
            pk[16 + (x >> 1)] = pack2(b0, b1, p.fmt);
          }
        }
        l += l0 + l1;
        tmem_st32(s_addr, pk);
      } else if (any_act) {
        // ---- generic block size: two passes over S in 16-column chunks.  P
        // chunk k lands on columns S has already been read from.
        float mt = -INFINITY;
        for (int c0 = 0; c0 < p.kvb; c0 += 16) {
          uint32_t v[16];
          tmem_ld16(s_addr + c0, v);
          tmem_wait_ld();
#pragma unroll
          for (int x = 0; x < 16; x++)
            if (c0 + x >= lo && c0 + x < hi) mt = fmaxf(mt, __uint_as_float(v[x]));
        }
        const float mt2 = act ? mt * c : -INFINITY;
        const bool grow = act && mt2 > m_run + 8.f;
        const float m_new = grow ? mt2 : m_run;
        const bool resc = grow && l > 0.f;
        if (__any_sync(0xffffffffu, resc)) {
          if (!o_quiet()) {
            ok = false;
            break;
          }
          const float alpha = resc ? fast_exp2(m_run - m_new) : 1.f;
          for (int c0 = 0; c0 < DV; c0 += 32) {
            uint32_t ov[32];
            tmem_ld32(o_addr + c0, ov);
            tmem_wait_ld();
#pragma unroll
            for (int x = 0; x < 32; x++) ov[x] = __float_as_uint(__uint_as_float(ov[x]) * alpha);
            tmem_st32(o_addr + c0, ov);
          }
          l *= alpha;
        }
        m_run = m_new;
        for (int c0 = 0; c0 < p.kvb; c0 += 16) {
          uint32_t v[16];
          tmem_ld16(s_addr + c0, v);
          tmem_wait_ld();
          uint32_t pk[8];
#pragma unroll
          for (int x = 0; x < 16; x += 2) {
            float p0 = 0.f, p1 = 0.f;
            if (act && c0 + x >= lo && c0 + x < hi)
              p0 = fast_exp2(fmaf(__uint_as_float(v[x]), c, -m_run));
            if (act && c0 + x + 1 >= lo && c0 + x + 1 < hi)
              p1 = fast_exp2(fmaf(__uint_as_float(v[x + 1]), c, -m_run));
            l += p0 + p1;
            pk[x >> 1] = pack2(p0, p1, p.fmt);
          }
          tmem_st8(s_addr + (c0 >> 1), pk);
        }
      } else {
        uint32_t z[8];
#pragma unroll
        for (int x = 0; x < 8; x++) z[x] = 0u;
        for (int c0 = 0; c0 < p.kvb; c0 += 16) tmem_st8(s_addr + (c0 >> 1), z);
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_pfull(sbuf));
    }

    // ------------------------------------------------------------ epilogue
    // merge the two groups' partial softmax states, then each group converts
    // and stores one half of the head dimension
    s_m[grp_w][r] = m_run;
    s_l[grp_w][r] = l;
    asm volatile("bar.sync 1, 256;" ::: "memory");
    if (ok && n > 0) ok = mbar_wait(bar_final, 0, w, FTK_DEV_TIMEOUT_EPILOGUE);
    if (ok) {
      tc_fence_after();
      const float ma = s_m[0][r], mb = s_m[1][r];
      const float la = s_l[0][r], lb = s_l[1][r];
      const float mm = fmaxf(ma, mb);
      const float fa = la > 0.f ? fast_exp2(ma - mm) : 0.f;
      const float fb = lb > 0.f ? fast_exp2(mb - mm) : 0.f;
      const float lt = la * fa + lb * fb;
      const bool have = (n > 0) && lt > 0.f;
      const float inv = have ? 1.f / lt : 0.f;
      const float wa = fa * inv, wb = fb * inv;
      constexpr int HALF = DV / 2;
#pragma unroll 1
      for (int c0 = grp_w * HALF; c0 < (grp_w + 1) * HALF; c0 += 32) {
        uint32_t va[32], vb[32];
        if (n > 0) tmem_ld32(lane_addr + FW_COL_O + c0, va);
        if (!SINGLE && n > 1) tmem_ld32(lane_addr + FW_COL_O + 128 + c0, vb);
        if (n > 0) tmem_wait_ld();
        uint32_t pk[16];
#pragma unroll
        for (int x = 0; x < 32; x += 2) {
          float a = 0.f, b = 0.f;
          if (have) {
            a = __uint_as_float(va[x]) * wa;
            b = __uint_as_float(va[x + 1]) * wa;
            if (!SINGLE && n > 1) {
              a = fmaf(__uint_as_float(vb[x]), wb, a);
              b = fmaf(__uint_as_float(vb[x + 1]), wb, b);
            }
          }
          pk[x >> 1] = pack2(a, b, p.fmt);
        }
        store_rows(smem + (warp - 2) * 2048, pk, p.o, s_out, 0, quarter, p.so_n, c0, p.D, p.fmt,
                   p.out_f32 != 0);
      }
      if (row_valid && grp_w == 0)
        p.lse[static_cast<int64_t>(bh) * p.N + qrow] =
            have ? (mm + log2f(lt)) * 0.6931471805599453f : -INFINITY;
    }
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (abort_flag) {
    for (int i = 0; i < 200; i++) __nanosleep(1000);
    break;   // uniform: barriers and TMEM are not in a state to go on with
  }
  }
  if (threadIdx.x < 32 && !first_tile) tmem_dealloc(tmem, 512);
}

}  // namespace ftk

#include "sparse_fwd_pipe.cuh"
#include "sparse_fwd_pipe2.cuh"

namespace ftk {

static int tmap_rows(CUtensorMap* out, const ftk_attn& a, char which, int rows) {
  const void* base = which == 'q' ? a.q : which == 'k' ? a.k : a.v;
  const int64_t sb = which == 'q' ? a.sq_b : which == 'k' ? a.sk_b : a.sv_b,
                sn = which == 'q' ? a.sq_n : which == 'k' ? a.sk_n : a.sv_n,
                sh = which == 'q' ? a.sq_h : which == 'k' ? a.sk_h : a.sv_h;
  return encode_tmap_bnhd(out, base, a.dtype, a.B, a.N, which == 'q' ? a.H : a.Hkv, a.D, sb, sn, sh,
                          64, rows);
}

template <int D, int NG>
static int launch_fwd_pipe(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
                           const FwdParams& p, int64_t BH, cudaStream_t st) {
  return choose<2>(p.fmt, [&](auto fmt) {
    return choose<3>(p.sub, [&](auto sub) {
      constexpr int F = decltype(fmt)::value, S = decltype(sub)::value == 2 ? 2 : 1;
      // A CTA that fits twice shall not share its SM while others are idle: behind a merge that is
      // still running on some SMs 128 tiles of 4096 keys, D = 64, took 52 us, 35 with this, 105 of
      // 13427 keys 155 and 100.
      const size_t smem = NG == 2 ? spread_smem(p.tiles, fp_smem(D, NG), FP_STATIC) : fp_smem(D, NG);
      if (int e = allow_smem<sparse_fwd_pipe_kernel<D, F, S, NG>>(smem)) return e;
      return launch_pdl(sparse_fwd_pipe_kernel<D, F, S, NG>,
                        dim3(p.tiles_x, static_cast<unsigned>(BH)), fp_threads(NG), smem, st, tq, tk, tv, p);
    });
  });
}

template <int D>
static int launch_fwd_pipe2(const CUtensorMap& tq, const CUtensorMap& tk32, const CUtensorMap& tv,
                            const FwdParams& p, int64_t BH, cudaStream_t st) {
  return choose<2>(p.fmt, [&](auto fmt) {
    return choose<3>(p.sub, [&](auto sub) {
      constexpr int F = decltype(fmt)::value, S = decltype(sub)::value == 2 ? 2 : 1;
      if (int e = allow_smem<sparse_fwd_pipe2_kernel<D, F, S>>(fp2_smem(D))) return e;
      return launch_pdl(sparse_fwd_pipe2_kernel<D, F, S>,
                        dim3(2 * ((p.tiles_x + 1) / 2), static_cast<unsigned>(BH)), FP2_THREADS,
                        fp2_smem(D), st, tq, tk32, tv, p);
    });
  });
}

template <int D>
static int launch_fwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
                      FwdParams p, cudaStream_t st) {
  constexpr int NCH = D / 64;
  const int stage_bytes = 2 * NCH * p.kvb * 128;
  // 227 KB per CTA less the static part (union scratch, softmax state: ~20 KB) and the Q tile
  const int ring_bytes = (227 - 21) * 1024 - NCH * 128 * 128;
  int nst = std::min(FW_MAX_STAGES, std::min(168 * 1024, ring_bytes) / stage_bytes);
  if (nst < 2) return FTK_ERR_UNSUPPORTED;
  p.nstages = nst;
  // the marks of the list union lie where the ring will be
  const size_t smem = 1024 + NCH * 128 * 128 +
                      std::max(static_cast<size_t>(nst) * stage_bytes, flag_bytes(p.Mkv, p.G));
  // Redo: as many CTAs as run at once, which find their tiles themselves.  Up to one tile per SM
  // they cannot meet, and with a few no CTA's share of the marked ones is long; beyond that the
  // marked ones are dealt, see next_marked.
  const bool deal = p.tiles > 4 * sm_count() && sm_count() * REDO_QUEUE >= REDO_LOOK;
  const int mode = !p.redo_in ? EXACT : deal ? REDO_DEAL : REDO_OWN;
  const int ctas = p.redo_in ? std::min(p.tiles, sm_count()) : p.tiles;
  return choose<3>(mode, [&](auto m) {
    constexpr auto kernel = sparse_fwd_kernel<D, D, decltype(m)::value>;
    if (int e = allow_smem<kernel>(smem)) return e;
    return launch_pdl(kernel, ctas, FW_THREADS, smem, st, tq, tk, tv, p);
  });
}

static size_t fwd_workspace(int64_t BH, int QM, int g) {
  const int G = attn_groups(g);
  return static_cast<size_t>(BH) * ((QM + G - 1) / G) * sizeof(int32_t);
}

static int attn_fwd(const ftk_attn& a, const AttnGrid& gr, void* o, int64_t so_b, int64_t so_n,
                    int64_t so_h, float* lse, void* workspace, size_t workspace_bytes,
                    int32_t* status, cudaStream_t st) {
  if (!aligned16(o, so_b, so_n, so_h) || !lse) return FTK_ERR_BAD_ARG;
  const int64_t BH = a.B * a.H;
  FwdParams p{};
  p.N = static_cast<int>(a.N);
  p.H = static_cast<int>(a.H);
  p.D = static_cast<int>(a.D);
  p.QM = gr.QM;
  p.W = a.W;
  p.list_rows = a.list_rows;
  p.Mkv = gr.Mkv;
  p.g = gr.g;
  p.kvb = gr.kvb;
  p.q_pad_head = gr.q_pad_head;
  p.kv_pad_head = gr.kv_pad_head;
  p.G = attn_groups(gr.g);
  p.fmt = a.dtype;
  p.out_f32 = a.out_f32;
  p.scale_log2 = a.scale * 1.4426950408889634f;
  p.merged = a.lists;
  p.lm = gr.lm;
  p.o = o;
  p.so_b = so_b;
  p.so_n = so_n;
  p.so_h = so_h;
  p.lse = lse;
  p.status = status;
  p.kv_hdiv = static_cast<int>(a.H / a.Hkv);
  p.tiles_x = (gr.QM + p.G - 1) / p.G;
  if (BH * p.tiles_x > 0x7fffffffLL) return FTK_ERR_BAD_ARG;
  p.tiles = static_cast<int>(BH * p.tiles_x);

  CUtensorMap tq, tk, tv;
  int e;
  if ((e = tmap_rows(&tq, a, 'q', 128))) return e;
  // q and kv blocks of 64 or 32 rows and a workspace: the pipelined kernel runs
  // first and the exact kernel redoes the tiles it flags.
  const char* env = getenv("FTK_FWD_PIPE");
  const bool pipe = tiles_of_64(gr.g, gr.kvb) && workspace &&
                    workspace_bytes >= fwd_workspace(BH, gr.QM, gr.g) && !(env && env[0] == '0');
  bool pairs = false;
  if (pipe) {
    p.sub = 64 / gr.kvb;
    p.kvb = 64;
    if ((e = tmap_rows(&tv, a, 'v', 64))) return e;
    p.redo_out = static_cast<int*>(workspace);
    const char* env2 = getenv("FTK_FWD_2CTA");
    // One CTA per SM, two, or pairs.  Pairs walk the union of four lists where one CTA walks that
    // of two, 0.9 of the time per tile; two CTAs per SM hide each other's unions, first loads and
    // last tiles, and two warps issue.  Kilocycles, pairs, then two CTAs per SM (head dim 128, blocks
    // of 64, lists as long as given of the blocks given): 32 of 32, 256 tiles 81, 73; 64 of 64, 1024
    // tiles 408, 383; 128 of 128 676, 685; 256 of 256 1226, 1342; 512 of 512, 2048 tiles 4843,
    // 5033; lists that are not full: 64 of 128 582, 470; 90 of 128 661, 608; 128 of 256 1070, 963.
    // So pairs take long lists that can name three quarters of the blocks and more.  (With q blocks
    // of 32 rows, one CTA per SM against pairs, the line is at half of the blocks.)
    // One CTA per SM against two: 2048 tiles, lists of 4 of 64 231, 143; of 16 376, 283; of 31 605,
    // 493; of 128 of 512, 1024 tiles 947, 919; 160 tiles 69, 61.  A grid of one wave has nothing
    // to hide: 128 tiles of 32 blocks 38, 44.  These two give the same bits; pairs do not where
    // lists differ (other reference tiles), so that line may not depend on the grid: the shards
    // of a problem would differ from the whole.
    // Head dim 256 takes pairs whatever the lists: four disjoint lists cost twice
    // the tiles of two, the one-CTA kernel three times the cycles per tile.
    // Head dim 64 with at most two q-blocks per tile: two CTAs per SM.
    pairs = gr.kd == 256;
    if (gr.kd == 128 && !(env2 && env2[0] == '0'))
      pairs = p.G <= 2 ? 4 * gr.width >= 3 * static_cast<int64_t>(gr.Mkv) &&
                             static_cast<int64_t>(gr.Mkv) * gr.kvb > 96 * 64
                       : 2 * gr.width >= gr.Mkv;
    // each CTA of a pair loads half of a tile's keys
    if ((e = tmap_rows(&tk, a, 'k', pairs ? 32 : 64))) return e;
    if (gr.kd == 256)
      e = launch_fwd_pipe2<256>(tq, tk, tv, p, BH, st);
    else if (pairs)
      e = launch_fwd_pipe2<128>(tq, tk, tv, p, BH, st);
    else if (gr.kd == 128)
      e = p.G <= 2 && p.tiles > sm_count() ? launch_fwd_pipe<128, 2>(tq, tk, tv, p, BH, st)
                                           : launch_fwd_pipe<128, 4>(tq, tk, tv, p, BH, st);
    else
      e = p.G <= 2 ? launch_fwd_pipe<64, 2>(tq, tk, tv, p, BH, st)
                   : launch_fwd_pipe<64, 4>(tq, tk, tv, p, BH, st);
    if (e) return e;
    p.redo_out = nullptr;
    p.redo_in = static_cast<const int*>(workspace);
  }
  p.sub = 1;
  p.kvb = gr.kvb;
  if (!pipe || pairs || gr.kvb != 64)   // else the tiles are the same
    if ((e = tmap_rows(&tk, a, 'k', gr.kvb))) return e;
  if (!pipe || gr.kvb != 64)
    if ((e = tmap_rows(&tv, a, 'v', gr.kvb))) return e;
  if (gr.kd == 64) return launch_fwd<64>(tq, tk, tv, p, st);
  if (gr.kd == 256) return launch_fwd<256>(tq, tk, tv, p, st);
  return launch_fwd<128>(tq, tk, tv, p, st);
}

}  // namespace ftk

using namespace ftk;

extern "C" int ftk_attn_parts(const ftk_attn* a, int limit, int32_t out[10]) {
  if (!a || !out || limit < 16) return FTK_ERR_BAD_ARG;
  AttnGrid gr;
  if (int e = attn_grid(*a, limit, &gr)) return e;
  const int32_t v[10] = {gr.g,          gr.kvb,       gr.q_pad_head, gr.kv_pad_head, gr.QM, gr.Mkv,
                         gr.lm.q_shift, gr.lm.q_off, gr.lm.kv_shift, gr.lm.kv_off};
  std::copy(v, v + 10, out);
  return FTK_OK;
}

// One redo word per tile of the pipelined kernel.
extern "C" size_t ftk_attn_fwd_workspace(const ftk_attn* a) {
  AttnGrid gr;
  if (!a || attn_grid(*a, 64, &gr)) return 0;
  return fwd_workspace(a->B * a->H, gr.QM, gr.g);
}

extern "C" int ftk_attn_fwd(const ftk_attn* a, void* o, int64_t so_b, int64_t so_n, int64_t so_h,
                            float* lse, void* workspace, size_t workspace_bytes, int32_t* status,
                            void* stream) {
  if (!a) return FTK_ERR_BAD_ARG;
  AttnGrid gr;
  if (int e = attn_grid(*a, 64, &gr)) return e;
  return attn_fwd(*a, gr, o, so_b, so_n, so_h, lse, workspace, workspace_bytes, status,
                  static_cast<cudaStream_t>(stream));
}

extern "C" size_t ftk_sparse_fwd_workspace(int64_t B, int64_t H, int QM, int q_block_size) {
  if (B <= 0 || H <= 0 || QM <= 0 || q_block_size <= 0) return 0;
  return fwd_workspace(B * H, QM, q_block_size);
}

extern "C" int ftk_sparse_fwd(const void* q, const void* k, const void* v, int dtype, int64_t B,
                              int64_t H, int64_t Hkv, int64_t N, int64_t D, int64_t sq_b, int64_t sq_n,
                              int64_t sq_h, int64_t sk_b, int64_t sk_n, int64_t sk_h, int64_t sv_b,
                              int64_t sv_n, int64_t sv_h, const int32_t* merged_idx, int QM, int W,
                              int q_block_size, int kv_block_size, int q_pad_head, int kv_pad_head,
                              float scale, void* o, int64_t so_b, int64_t so_n, int64_t so_h,
                              float* lse, void* workspace, size_t workspace_bytes,
                              int32_t* status, void* stream) {
  if (D != 64 && D != 128 && D != 256) return FTK_ERR_UNSUPPORTED;
  const ftk_attn a = {q,    k,    v,    dtype, 0,    B,    H,    Hkv <= 0 ? H : Hkv,
                      N,    D,    sq_b, sq_n,  sq_h, sk_b, sk_n, sk_h,
                      sv_b, sv_n, sv_h, merged_idx, QM, W, q_block_size, kv_block_size,
                      q_pad_head, kv_pad_head, scale};
  AttnGrid gr;
  if (int e = attn_grid(a, 128, &gr)) return e;   // blocks of up to 128 rows as they are
  return attn_fwd(a, gr, o, so_b, so_n, so_h, lse, workspace, workspace_bytes, status,
                  static_cast<cudaStream_t>(stream));
}
