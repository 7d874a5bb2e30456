// Block scoring for sm_100a: dense Q.K^T on tcgen05 with TMEM accumulators,
// K tiles staged by TMA, softmax mass accumulated per score block.
//
// Replaces block_score_kernel / block_normalize_kernel of the reference
// (flash_topk_attn_v2/csrc/block_score_kernel.cu:19-314).
//
// One CTA owns 256 query rows of one (batch, head) slice and streams every
// key tile once.  Roles: warp 0 = TMA producer, warp 1 = UMMA issuer, warps
// 2..17 = two groups of 256 softmax threads, one query row each (TMEM lane ==
// row).  Two 128x128 fp32 accumulators per stage (rows 0-127 / 128-255 share
// the K tile), two stages: 4 x 128 = 512 TMEM columns.  Group s drains stage
// s, so the groups work concurrently on consecutive tiles while the tensor
// core refills whichever accumulator was handed back.
//
// Softmax is single pass against a fixed per-row reference exponent `mref`
// (an integer in log2 units): sum_j[t] = sum_{i in block j} 2^(c*s_ti - mref),
// L[t] = sum_j sum_j[t]; the block score is sum_j / L.  mref comes from the
// row maximum over the first key tile (pass 0).  Should any later logit
// exceed it by more than the fp32 exponent range the row total overflows; a
// CTA that sees this walks its keys twice more (pass 1: exact row maximum,
// pass 2: sums against it).  The CTA owns its rows, so nobody else has to know:
// two follow-up launches and the clearing of their flag, which every call paid
// for (about 2 us of device time each at the smallest sizes, 6-7 us at the
// largest, and 3 of 5 launches), are not there.
//
// Where the grid has too few tiles of 256 rows to fill the SMs, or a last wave that
// is nearly empty, a cluster of 2, 4 or 8 CTAs shares a tile and splits its keys
// (score_split).  All take the reference exponents from the first key tile, so their
// block sums go out as they are; the row totals meet through the cluster's shared
// memory.  A total is always added up from the same SC_SEGS parts of the keys, so it
// does not depend on the split, bit for bit.  Of a grid of several waves only the tiles of
// the last one are split, in a launch of their own that fills the SMs as they become free.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>

#include "ftk_host.cuh"
#include "ftk_sm100.cuh"

namespace ftk {

constexpr int SC_QROWS = 256;      // query rows per CTA
constexpr int SC_KT = 128;         // key rows per tile (UMMA N)
constexpr int SC_STAGES = 4;       // K tile ring depth
constexpr int SC_THREADS = 576;    // 2 + 2 x 8 warps
constexpr int SC_SEGS = 8;         // parts of the keys that a row total is added up from
constexpr int SC_CHUNK_BYTES = 128 * 128;  // 128 rows x 64 16-bit elements
__host__ __device__ constexpr int score_ksplit(int d) { return d > 128 ? 2 : 1; }
__host__ __device__ constexpr int score_stages(int d) { return d > 128 ? 2 : SC_STAGES; }

struct ScoreParams {
  int N, M, D;
  int bsz, pad_head;          // score block size, virtual head padding
  int tile_rows;              // rows fetched per K tile (TMA box rows)
  int blocks_per_tile;        // bsz <= 128: whole blocks per tile, else 0
  int tiles_per_block;        // bsz > 128: tiles per block, else 0
  int num_tiles;
  int fmt;                    // 0 fp16, 1 bf16
  int H, bh_begin;
  int qtiles;                 // tiles of 256 query rows per slice
  int tile0;                  // first tile of this launch
  int behind;                 // runs beside the launch before it, which is part of the same call
  float scale_log2;           // log2(e) * softmax scale
  float* sums;                // [bh_count][N][M]   unnormalised block sums
  float* row_total;           // [bh_count][N]      L
  int* status;
};

struct TileInfo {
  int row0;     // first key token of the tile (may be negative)
  int used;     // accumulator columns that belong to score blocks
  int block0;   // score block of column 0
  int col_in_block0;  // position of column 0 inside that block
};

__device__ __forceinline__ TileInfo tile_info(const ScoreParams& p, int t) {
  TileInfo ti;
  if (p.blocks_per_tile > 0) {
    ti.block0 = t * p.blocks_per_tile;
    int nb = min(p.blocks_per_tile, p.M - ti.block0);
    ti.row0 = ti.block0 * p.bsz - p.pad_head;
    ti.used = nb * p.bsz;
    ti.col_in_block0 = 0;
  } else {
    int j = t / p.tiles_per_block, part = t - j * p.tiles_per_block;
    ti.block0 = j;
    ti.row0 = j * p.bsz - p.pad_head + part * SC_KT;
    ti.used = min(SC_KT, p.bsz - part * SC_KT);
    ti.col_in_block0 = part * SC_KT;
  }
  return ti;
}

// First tile of part s of the keys: whole score blocks, in order
__device__ __forceinline__ int seg_begin(const ScoreParams& p, int s) {
  const int per = max(1, p.tiles_per_block);
  return static_cast<int>(static_cast<int64_t>(s) * (p.num_tiles / per) / SC_SEGS) * per;
}

// Sum of 2^(c s - mref) over 16 columns, two per instruction for the scaling (fma.f32x2) and
// for the running sums (add.f32x2); the four partial sums are the same additions in the same
// order as scalar code.
__device__ __forceinline__ float sum16(const uint32_t (&r)[16], float c, float mref) {
  const float2 c2 = make_float2(c, c), nm2 = make_float2(-mref, -mref);
  auto exp2_of = [&](int i) {
    const float2 x = __ffma2_rn(make_float2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), c2, nm2);
    return make_float2(fast_exp2(x.x), fast_exp2(x.y));
  };
  float2 s01 = make_float2(0.f, 0.f), s23 = make_float2(0.f, 0.f);
#pragma unroll
  for (int i = 0; i < 16; i += 4) {
    s01 = __fadd2_rn(s01, exp2_of(i));
    s23 = __fadd2_rn(s23, exp2_of(i + 2));
  }
  return (s01.x + s01.y) + (s23.x + s23.y);
}

// SPLIT: launched as clusters that share a tile; its bookkeeping in the loop over the
// tiles took 4 % of the kernel where nothing is split.
template <int D, bool SPLIT>
__global__ void __launch_bounds__(SC_THREADS, 1)
score_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
             const ScoreParams p) {
  constexpr int NCH = D / 64;                       // 128-byte chunks per row
  constexpr int Q_BYTES = 2 * NCH * SC_CHUNK_BYTES; // 256 rows
  // Head dims above 128: a K tile travels as KSPLIT slices of the head dim,
  // one ring stage each (the 256-row Q tile leaves room for two 32 KB stages),
  // and the tile's UMMAs accumulate over the slices.
  constexpr int KSPLIT = score_ksplit(D);
  constexpr int NCHS = NCH / KSPLIT;                // chunks per stage
  constexpr int NSTG = score_stages(D);
  constexpr int K_STAGE_BYTES = NCHS * SC_CHUNK_BYTES;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem;
  uint8_t* sK = smem + Q_BYTES;
  __shared__ __align__(8) uint64_t bars[1 + 2 * SC_STAGES + 8 + 2];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_flag;
  __shared__ int s_redo, s_stop;
  __shared__ float s_mref[SC_QROWS];   // group 0 -> group 1: reference exponent / row maximum
  __shared__ float s_seg[2][SC_SEGS][SC_QROWS];   // totals per group and part (pass 1: maxima in part 0)

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int split = SPLIT ? static_cast<int>(cluster_nctas()) : 1,
            rank = SPLIT ? static_cast<int>(cluster_ctarank()) : 0;
  const int tile = p.tile0 + static_cast<int>(blockIdx.x) / split;
  const int bh_local = tile / p.qtiles;
  const int q0 = (tile - bh_local * p.qtiles) * SC_QROWS;
  const int bh = p.bh_begin + bh_local;
  const int b_idx = bh / p.H, h_idx = bh - b_idx * p.H;

  const uint32_t bar_q = smem_u32(&bars[0]);     // rows 0 .. 127 of Q
  auto bar_kfull = [&](int s) { return smem_u32(&bars[1 + s]); };
  auto bar_kempty = [&](int s) { return smem_u32(&bars[1 + SC_STAGES + s]); };
  // one full / empty pair per accumulator (stage s, row half h): the four
  // warps that drain an accumulator start as soon as its 8 UMMAs retire and
  // hand it back on their own
  auto bar_afull = [&](int s, int h) { return smem_u32(&bars[1 + 2 * SC_STAGES + s * 2 + h]); };
  auto bar_aempty = [&](int s, int h) {
    return smem_u32(&bars[1 + 2 * SC_STAGES + 4 + s * 2 + h]);
  };
  const uint32_t bar_mref = smem_u32(&bars[1 + 2 * SC_STAGES + 8]);
  const uint32_t bar_q1 = smem_u32(&bars[1 + 2 * SC_STAGES + 9]);   // rows 128 .. 255

  if (tid == 0) {
    abort_flag = 0;
    s_redo = s_stop = 0;
    mbar_init(bar_q, 1);
    mbar_init(bar_q1, 1);
    for (int s = 0; s < SC_STAGES; s++) {
      mbar_init(bar_kfull(s), 1);
      mbar_init(bar_kempty(s), 1);
    }
    for (int s = 0; s < 2; s++)
      for (int h = 0; h < 2; h++) {
        mbar_init(bar_afull(s, h), 1);
        mbar_init(bar_aempty(s, h), 4);  // one arrival per warp draining the accumulator
      }
    mbar_init(bar_mref, 8);
    mbar_init_fence();
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(&tmem_base_s), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_s;
  WaitCtx w{&abort_flag, p.status};
  // my tiles: t_first .. t_first + L - 1, and in pass 0 tile 0 ahead of them unless it
  // is mine (`pre`), for the reference exponents
  const int seg_first = rank * SC_SEGS / split, seg_last = (rank + 1) * SC_SEGS / split;
  const int t_first = SPLIT ? seg_begin(p, seg_first) : 0,
            L = SPLIT ? seg_begin(p, seg_last) - t_first : p.num_tiles;
  float mref = 0.f;    // softmax threads: the row's reference exponent
  // The second launch of a call starts when every block of the first one is past its wait, so
  // what came before the call is there.  It waits for the first one at its end: whoever
  // waits for this launch wants the results of both.  The wait must stand ahead of the trigger
  // (see pdl_wait()).
  if (!p.behind) pdl_wait();
  pdl_launch();

  // Pass 0 is all there is unless a row total overflows.  Every barrier's
  // phases run on from pass to pass: an accumulator and the K ring have been used
  // as often as the tiles of the passes before say.
  for (int pass = 0; pass < 3; pass++) {
  const int pre = SPLIT && pass == 0 && t_first > 0 ? 1 : 0;
  const int T = L + pre;
  const int done0 = pass > 0 ? L + (SPLIT && t_first > 0 ? 1 : 0) : 0;   // tiles of pass 0 ...
  const int done1 = pass > 1 ? L : 0;                                       // ... and of pass 1
  auto tile_of = [&](int u) { return u < pre ? 0 : t_first + u - pre; };
  auto used = [&](int a, int u) {   // uses of accumulator a before this pass's tile u
    return ((done0 + 1 - a) >> 1) + ((done1 + 1 - a) >> 1) + (u >> 1);
  };
  if (warp == 0) {
    // ------------------------------------------------------- TMA producer
    if (lane == 0) {
      // the first scores need half of Q and a key tile: those travel first
      auto load_q = [&](int half, uint32_t bar) {
        mbar_expect_tx(bar, Q_BYTES / 2);
        for (int c = 0; c < NCH; c++)
          tma_load_4d(smem_u32(sQ) + (half * NCH + c) * SC_CHUNK_BYTES, &tm_q, bar, c * 64, h_idx,
                      q0 + half * 128, b_idx);
      };
      if (pass == 0) load_q(0, bar_q);
      const uint32_t tile_bytes = static_cast<uint32_t>(p.tile_rows) * 128u * NCHS;
      const int u0 = (done0 + done1) * KSPLIT;
      for (int u = 0; u < T * KSPLIT; u++) {
        const int s = (u0 + u) % NSTG;
        const uint32_t ph = ((u0 + u) / NSTG) & 1;
        if (!mbar_wait(bar_kempty(s), ph ^ 1, w, FTK_DEV_TIMEOUT_TMA)) break;
        const int part = u % KSPLIT;
        const TileInfo ti = tile_info(p, tile_of(u / KSPLIT));
        mbar_expect_tx(bar_kfull(s), tile_bytes);
        for (int c = 0; c < NCHS; c++)
          tma_load_4d(smem_u32(sK) + s * K_STAGE_BYTES + c * SC_CHUNK_BYTES, &tm_k, bar_kfull(s),
                      (part * NCHS + c) * 64, h_idx, ti.row0, b_idx);
        if (pass == 0 && u == KSPLIT - 1) load_q(1, bar_q1);
      }
    }
  } else if (warp == 1) {
    // -------------------------------------------------------- UMMA issuer
    {
      // the whole warp runs this path; one elected lane issues the UMMAs
      const uint32_t idesc = umma_idesc(128, SC_KT, p.fmt, 0, 0);
      const uint64_t qdesc0 = smem_desc_sw128(smem_u32(sQ), 16, 1024);
      const uint64_t kdesc0 = smem_desc_sw128(smem_u32(sK), 16, 1024);
      bool ok = mbar_wait(bar_q, 0, w, FTK_DEV_TIMEOUT_MMA);
      for (int t = 0; ok && t < T; t++) {
        const int u0 = (done0 + done1 + t) * KSPLIT;
        const int a = t & 1;
        const uint32_t pa = used(a, t) & 1;
        // the three barriers of a tile are waited for together (a test of a
        // completed barrier still takes ~110 cycles) and the tile's UMMAs go
        // out as one batch, so the tensor core is not left idle in between
        const uint32_t wb[3] = {bar_kfull(u0 % NSTG), bar_aempty(a, 0), bar_aempty(a, 1)};
        const uint32_t wp[3] = {static_cast<uint32_t>((u0 / NSTG) & 1), pa ^ 1, pa ^ 1};
        if (!mbar_wait_all<3>(wb, wp, w, FTK_DEV_TIMEOUT_MMA)) break;
        tc_fence_after();
#pragma unroll
        for (int part = 0; part < KSPLIT; part++) {
          const int s = (u0 + part) % NSTG;
          if (part > 0) {
            if (!mbar_wait(bar_kfull(s), ((u0 + part) / NSTG) & 1, w, FTK_DEV_TIMEOUT_MMA)) {
              ok = false;
              break;
            }
            tc_fence_after();
          }
          const uint64_t kdesc = desc_advance(kdesc0, s * K_STAGE_BYTES);
          auto issue = [&](int half) {   // elected lane only
            const uint32_t d_tmem = tmem + static_cast<uint32_t>((a * 2 + half) * SC_KT);
            const uint64_t qdesc = desc_advance(qdesc0, (half * NCH + part * NCHS) * SC_CHUNK_BYTES);
#pragma unroll
            for (int ks = 0; ks < D / KSPLIT / 16; ks++) {
              const uint32_t off = (ks / 4) * SC_CHUNK_BYTES + (ks % 4) * 32;
              umma_ss(d_tmem, desc_advance(qdesc, off), desc_advance(kdesc, off), idesc,
                      part > 0 || ks > 0);
            }
            if (half == 1) umma_commit(bar_kempty(s));  // smem stage reusable once retired
            // this accumulator is readable
            if (part == KSPLIT - 1) umma_commit(bar_afull(a, half));
          };
          if (part == 0 && t == 0 && pass == 0) {   // the other half of Q may still be on its way
            if (elect_one()) issue(0);
            __syncwarp();
            ok = mbar_wait(bar_q1, 0, w, FTK_DEV_TIMEOUT_MMA);
            tc_fence_after();
            if (ok && elect_one()) issue(1);
          } else if (elect_one()) {
            issue(0);
            issue(1);
          }
          if (!ok) break;
          __syncwarp();
        }
      }
    }
  } else {
    // ---------------------------------------------------- softmax threads
    // Two groups of 8 warps, which take the CTA's tiles in turn and so run
    // concurrently on consecutive ones and hide each other's TMEM-load and barrier
    // latency.  A group is bound to one accumulator stage and meets every phase of
    // its barriers in order (a one-bit parity wait must never skip a phase).  When a
    // score block spans several tiles (block size > 128) one thread has to see all
    // of them, and group 0 takes every tile.
    const int cw = warp - 2;               // 0..15
    const int group = cw >> 3;
    const int half = (cw >> 2) & 1;        // which 128-row accumulator
    const int quarter = warp & 3;          // TMEM lane quarter this warp may read
    const int row_in_cta = half * 128 + quarter * 32 + lane;
    const int row = q0 + row_in_cta;
    const bool row_ok = row < p.N;
    const uint32_t lane_addr = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
    const size_t row_off = (static_cast<size_t>(bh_local) * p.N + (row_ok ? row : 0));
    float* out_row = p.sums + row_off * p.M;
    const float c = p.scale_log2;

    float run_max = -INFINITY;
    float total = 0.f;
    bool ok = true;

    if (pass == 2) mref = ceilf(s_mref[row_in_cta] * c);

    if (pass == 0) {
      if (group == 0) {
        // reference exponent from the row maximum over the first key tile
        ok = mbar_wait(bar_afull(0, half), 0, w, FTK_DEV_TIMEOUT_CONSUMER);
        if (ok) {
          tc_fence_after();
          const TileInfo ti = tile_info(p, 0);
          const int lo = max(0, -ti.row0), hi = min(ti.used, p.N - ti.row0);
          const float mx = tmem_row_max(lane_addr + static_cast<uint32_t>(half * SC_KT), ti.used, lo, hi);
          mref = ceilf(mx * c);
          if (!(fabsf(mref) < 1e30f)) mref = 0.f;
          if (pre) {   // not one of my tiles: hand the accumulator back
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_aempty(0, half));
          }
        }
        s_mref[row_in_cta] = mref;
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_mref);
      } else {
        ok = mbar_wait(bar_mref, 0, w, FTK_DEV_TIMEOUT_CONSUMER);
        mref = s_mref[row_in_cta];
      }
    }

    const bool whole = p.bsz % 64 == 0;
    float acc = 0.f;
    int j = 0, col_in_block = 0;
    // this group's tiles, part by part
    const int step = p.tiles_per_block > 1 ? 1 : 2;
    int u = step == 2 ? pre + ((group ^ pre) & 1) : (group == 0 ? pre : T);
    for (int seg = seg_first; seg < seg_last; seg++) {
    const int u_end = seg_begin(p, seg + 1) - t_first + pre;
    for (; ok && u < u_end; u += step) {
      const int t = tile_of(u), a = u & 1;
      const uint32_t pa = used(a, u) & 1;
      if (!mbar_wait(bar_afull(a, half), pa, w, FTK_DEV_TIMEOUT_CONSUMER)) { ok = false; break; }
      tc_fence_after();
      const TileInfo ti = tile_info(p, t);
      const int lo = max(0, -ti.row0), hi = min(ti.used, p.N - ti.row0);
      const bool full = (lo == 0 && hi == ti.used);
      if (ti.col_in_block0 == 0) { j = ti.block0; col_in_block = 0; }
      const uint32_t acc_addr = lane_addr + static_cast<uint32_t>((a * 2 + half) * SC_KT);
      auto flush = [&]() {   // block sums end on the 16-column grid
        if (col_in_block == p.bsz) {
          if (row_ok) out_row[j] = acc;
          total += acc;
          acc = 0.f;
          col_in_block = 0;
          j++;
        }
      };
      auto release = [&]() {
        // the tile's last columns are in registers: hand the accumulator back
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_aempty(a, half));
      };
      if (pass == 1) {
        run_max = fmaxf(run_max, tmem_row_max(acc_addr, ti.used, lo, hi));
        release();
      } else if (full && ti.used == SC_KT) {
        // Full tile: the next 16 columns are on their way while the last are summed.  Block
        // sizes of whole 64s (`whole`) look for the end of a block only there.  With 32-column
        // loads, a look every 16 columns and pass 1 in the same loop the exponentials ran at
        // 0.94 of the special-function unit's rate without the wait for the UMMAs, now at all
        // of it: N = 32768, H = 4 1239 -> 1200 us, 128-row blocks, N = 15000, H = 16 1135 ->
        // 1090, N = 2000, H = 16 34.8 -> 30.7.
        uint32_t ra[16], rb[16];
        if constexpr (D <= 128) tmem_ld16(acc_addr, ra);
#pragma unroll
        for (int c0 = 0; c0 < SC_KT; c0 += 32) {
          // The tensor core bounds head dim 256, and loads ahead of need get in its way: 32
          // columns at a time there.  With select, N = 8192, H = 16, blocks of 64 keys: 507 us with
          // 32 columns ahead, 483 with 16 at a time, 476 so; H = 8, blocks of 32: 319, 306, 292.
          if constexpr (D > 128) tmem_ld16(acc_addr + c0, ra);
          else tmem_wait_ld();
          tmem_ld16(acc_addr + c0 + 16, rb);
          if constexpr (D > 128) tmem_wait_ld();
          if (D > 128 && c0 + 32 == SC_KT) release();
          const float t0 = sum16(ra, c, mref);
          if constexpr (D <= 128) {
            tmem_wait_ld();
            if (c0 + 32 < SC_KT) tmem_ld16(acc_addr + c0 + 32, ra);
            else release();
          }
          const float t1 = sum16(rb, c, mref);
          acc += t0;
          if (!whole) { col_in_block += 16; flush(); }
          acc += t1;
          if (!whole) { col_in_block += 16; flush(); }
          else if (c0 & 32) { col_in_block += 64; flush(); }
        }
      } else if (D == 128 && full) {
        // Blocks that leave columns of the tile blank, 32 columns per wait: N = 8192, H = 8 with
        // select 288 -> 263 us for blocks of 48 keys, 274 -> 253 of 80.  At the other head dims a
        // wait per 16 columns was not the slower one (64: 253 us, 256 with 32; 256: 357, 362).
#pragma unroll 1
        for (int c0 = 0; c0 < ti.used; c0 += 32) {
          uint32_t ra[16], rb[16];
          tmem_ld16(acc_addr + c0, ra);
          tmem_ld16(acc_addr + c0 + 16, rb);   // the accumulator's own columns in any case
          tmem_wait_ld();
          if (c0 + 32 >= ti.used) release();
          acc += sum16(ra, c, mref);
          col_in_block += 16;
          flush();
          if (c0 + 16 < ti.used) {
            acc += sum16(rb, c, mref);
            col_in_block += 16;
            flush();
          }
        }
      } else {
#pragma unroll 1
        for (int c0 = 0; c0 < ti.used; c0 += 16) {
          uint32_t r[16];
          tmem_ld16(acc_addr + c0, r);
          tmem_wait_ld();
          if (c0 + 16 >= ti.used) release();
          float t = 0.f;
          if (full) {
            t = sum16(r, c, mref);
          } else if (c0 >= lo && c0 + 16 <= hi) {
            // partial tiles add up column by column, here without the comparisons
#pragma unroll
            for (int i = 0; i < 16; i++) t += fast_exp2(fmaf(__uint_as_float(r[i]), c, -mref));
          } else {
#pragma unroll
            for (int i = 0; i < 16; i++) {
              const int col = c0 + i;
              if (col >= lo && col < hi) t += fast_exp2(fmaf(__uint_as_float(r[i]), c, -mref));
            }
          }
          acc += t;
          col_in_block += 16;
          flush();
        }
      }
    }
    // publish this group's share of the part (pass 1: of the CTA's maximum)
    s_seg[group][pass == 1 ? 0 : seg][row_in_cta] = pass == 1 ? run_max : total;
    total = 0.f;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (split > 1) cluster_sync_all();
  if (tid < SC_QROWS) {
    // every CTA of the cluster adds up the same totals, so all come to the same decision
    if (pass == 1) {
      float mx = -INFINITY;
      for (int r = 0; r < split; r++)
        mx = fmaxf(mx, fmaxf(ld_cta(&s_seg[0][0][tid], r, split), ld_cta(&s_seg[1][0][tid], r, split)));
      s_mref[tid] = mx;
    } else {
      float tot = 0.f;
#pragma unroll
      for (int sg = 0; sg < SC_SEGS; sg++) {
        const int r = sg * split / SC_SEGS;
        tot += SPLIT ? ld_cta(&s_seg[0][sg][tid], r, split) + ld_cta(&s_seg[1][sg][tid], r, split)
                     : s_seg[0][sg][tid] + s_seg[1][sg][tid];
      }
      if (q0 + tid < p.N) {
        if (rank == 0) p.row_total[static_cast<size_t>(bh_local) * p.N + q0 + tid] = tot;
        if (pass == 0 && !(tot > 0.f && tot < 3.0e38f)) s_redo = 1;
      }
    }
  } else if (tid < SC_QROWS + split) {
    if (ld_cta(&abort_flag, tid - SC_QROWS, split)) s_stop = 1;
  }
  __syncthreads();
  const bool again = s_redo && !s_stop;
  if (split > 1) cluster_sync_all();   // nobody writes or leaves while a peer still reads
  if (!again) break;
  }

  // ------------------------------------------------------------- teardown
  if (abort_flag) {
    // give copies still in flight time to land before the smem is released
    for (int i = 0; i < 200; i++) __nanosleep(1000);
  }
  if (warp == 0) tmem_dealloc(tmem, 512);
  if (p.behind) pdl_wait();
}

// block_scores[r][j] = sums[r][j] / total[r]
__global__ void score_normalize_kernel(const float* __restrict__ sums,
                                       const float* __restrict__ total, float* __restrict__ out,
                                       int64_t rows, int M) {
  const int64_t n = rows * M;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = i / M;
    out[i] = sums[i] * __frcp_rn(total[r]);  // same arithmetic as the fused select path
  }
}

// How many CTAs share a tile of 256 query rows: the fewest waves of the shortest
// CTAs.  A CTA's time in key tiles is its share of them and about 3.5 to start and
// finish, 7.5 where it also has to fetch the first tile for the reference exponents
// and meet the others (512 tiles of 64 steps, D = 64: 4 waves unsplit 465 us, 7 waves of
// halves 476); the number of clusters that run at once is what the device says.
// 61 tiles of 122 steps: 203 -> 127 us with select, 32 of 32 steps: 59 -> 32 us.
// A grid of several waves leaves its last one as it is where that is full or nearly so; else
// its tiles are split like a small grid's, when that saves a tenth of the wave and three key tiles
// (a launch more for the host), or more than splitting all tiles does.
struct ScoreSplit {
  int cluster;   // CTAs per tile
  int tail;      // tiles of the last wave that are split, 0: none
  int tail_cluster;
};
template <int D>
static ScoreSplit score_split(int64_t tiles, int num_tiles, int units, size_t smem) {
  constexpr int MAX_DEVICES = 64;
  static std::atomic<int> resident[MAX_DEVICES][4];   // clusters of 1, 2, 4, 8
  ScoreSplit best = {1, 0, 1};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return best;
  auto clusters = [&](int i) {
    const int c = 1 << i;
    int n = resident[dev][i].load(std::memory_order_relaxed);
    if (n == 0) {
      n = c == 1 ? sm_count()
                 : allow_smem<score_kernel<D, true>>(smem) == FTK_OK
                       ? max_clusters(score_kernel<D, true>, c, SC_THREADS, smem)
                       : 0;
      resident[dev][i].store(n > 0 ? n : -1, std::memory_order_relaxed);
    }
    return n;
  };
  auto cost = [&](int64_t t, int i) {
    const int n = clusters(i), c = 1 << i;
    if (n <= 0) return 1e30;
    const double waves = static_cast<double>((t + n - 1) / n);
    return waves * (static_cast<double>(num_tiles) / c + (c > 1 ? 7.5 : 3.5));
  };
  double best_cost = cost(tiles, 0);
  for (int i = 1; i < 4 && (1 << i) <= units; i++) {
    const double x = cost(tiles, i);
    if (x < 0.95 * best_cost) {
      best.cluster = 1 << i;
      best_cost = x;
    }
  }
  const int n = clusters(0);
  if (n <= 0 || tiles <= n || tiles % n == 0) return best;
  const double wave = num_tiles + 3.5, full = static_cast<double>(tiles / n) * wave;
  if (best.cluster == 1) best_cost = full + std::min(0.9 * wave, wave - 3.);
  for (int i = 1; i < 4 && (1 << i) <= units; i++) {
    const double x = full + cost(tiles % n, i);
    if (x < best_cost) {
      best = {1, static_cast<int>(tiles % n), 1 << i};
      best_cost = x;
    }
  }
  return best;
}

template <int D>
static int launch_score_d(const CUtensorMap& tq, const CUtensorMap& tk, ScoreParams p,
                          int64_t bh_count, cudaStream_t st) {
  constexpr int NCH = D / 64;
  const size_t smem =
      1024 + (2 * NCH + score_stages(D) * (NCH / score_ksplit(D))) * SC_CHUNK_BYTES;
  if (int e = allow_smem<score_kernel<D, false>>(smem)) return e;
  p.qtiles = (p.N + SC_QROWS - 1) / SC_QROWS;
  const int64_t tiles = p.qtiles * bh_count;
  if (8 * tiles > 0x7fffffffLL) return FTK_ERR_BAD_ARG;
  const ScoreSplit split = score_split<D>(tiles, p.num_tiles, p.num_tiles / std::max(1, p.tiles_per_block), smem);
  const unsigned first = static_cast<unsigned>(tiles - split.tail);
  auto clusters = [&](unsigned n, int c) {
    if (int e = allow_smem<score_kernel<D, true>>(smem)) return e;
    return launch_clusters(score_kernel<D, true>, c, dim3(n * c), SC_THREADS, smem, st, tq, tk, p);
  };
  if (split.cluster > 1) return clusters(first, split.cluster);
  if (int e = launch_pdl(score_kernel<D, false>, dim3(first), SC_THREADS, smem, st, tq, tk, p)) return e;
  if (split.tail == 0) return FTK_OK;
  p.tile0 = static_cast<int>(first);
  p.behind = 1;
  return clusters(split.tail, split.tail_cluster);
}

struct ScoreWs {
  float* row_total;
  float* sums;
};

static size_t align256(size_t x) { return (x + 255) & ~static_cast<size_t>(255); }

static size_t score_ws_layout(int64_t bh_count, int64_t N, int64_t M, bool with_sums, char* base,
                              ScoreWs* ws) {
  size_t off = 0;
  const size_t rows = static_cast<size_t>(bh_count) * N;
  off += 256;
  if (ws) ws->row_total = reinterpret_cast<float*>(base + off);
  off += 2 * align256(rows * 4);   // the second row array is no longer used; the size is part of the ABI
  if (ws) ws->sums = reinterpret_cast<float*>(base + off);
  if (with_sums) off += align256(rows * static_cast<size_t>(M) * 4);
  return off;
}

// Validates arguments, encodes the tensor maps and launches the scoring kernel;
// sums go to `sums` ([bh_count][N][M]).
static int run_score(const void* q, const void* k, int dtype, int64_t B, int64_t H, int64_t N,
                     int64_t D, int64_t sq_b, int64_t sq_n, int64_t sq_h, int64_t sk_b,
                     int64_t sk_n, int64_t sk_h, int64_t bh_begin, int64_t bh_count, int bsz,
                     int pad_head, int pad_tail, float scale, float* sums, const ScoreWs& ws,
                     int32_t* status, cudaStream_t st) {
  if (!q || !k || B <= 0 || H <= 0 || N <= 0 || bsz <= 0 || !(scale > 0.f))
    return FTK_ERR_BAD_ARG;
  if (dtype != FTK_DTYPE_F16 && dtype != FTK_DTYPE_BF16) return FTK_ERR_BAD_ARG;
  if (pad_head < 0 || pad_tail < 0 || pad_head >= bsz || pad_tail >= bsz) return FTK_ERR_BAD_ARG;
  if ((pad_head + N + pad_tail) % bsz != 0) return FTK_ERR_BAD_ARG;
  if (bh_begin < 0 || bh_count <= 0 || bh_begin + bh_count > B * H) return FTK_ERR_BAD_ARG;
  // the tensor maps read columns beyond D as zeros: the kernels' head dims are 64, 128, 256
  if (D <= 0 || D % 8 != 0 || D > 256) return FTK_ERR_UNSUPPORTED;
  if (bsz % 16 != 0) return FTK_ERR_UNSUPPORTED;
  if (bh_count > 65535) return FTK_ERR_BAD_ARG;

  ScoreParams p{};
  p.N = static_cast<int>(N);
  p.M = static_cast<int>((pad_head + N + pad_tail) / bsz);
  p.D = static_cast<int>(D);
  p.bsz = bsz;
  p.pad_head = pad_head;
  if (bsz <= SC_KT) {
    p.blocks_per_tile = SC_KT / bsz;
    p.tiles_per_block = 0;
    p.tile_rows = p.blocks_per_tile * bsz;
    p.num_tiles = (p.M + p.blocks_per_tile - 1) / p.blocks_per_tile;
  } else {
    p.blocks_per_tile = 0;
    p.tiles_per_block = (bsz + SC_KT - 1) / SC_KT;
    p.tile_rows = SC_KT;
    p.num_tiles = p.M * p.tiles_per_block;
  }
  p.fmt = dtype;
  p.H = static_cast<int>(H);
  p.bh_begin = static_cast<int>(bh_begin);
  p.scale_log2 = static_cast<float>(1.4426950408889634 * static_cast<double>(scale));
  p.sums = sums;
  p.row_total = ws.row_total;
  p.status = status;

  CUtensorMap tq, tk;
  int e = encode_tmap_bnhd(&tq, q, dtype, B, N, H, D, sq_b, sq_n, sq_h, 64, 128);
  if (e) return e;
  e = encode_tmap_bnhd(&tk, k, dtype, B, N, H, D, sk_b, sk_n, sk_h, 64, p.tile_rows);
  if (e) return e;
  if (D <= 64) return launch_score_d<64>(tq, tk, p, bh_count, st);
  if (D > 128) return launch_score_d<256>(tq, tk, p, bh_count, st);
  return launch_score_d<128>(tq, tk, p, bh_count, st);
}

int select_launch(const float* block_scores, const float* row_scale, int64_t rows, int M,
                  int max_topk, int bsz, int pad_head, int pad_tail, float threshold,
                  int32_t* topk_idx, float* topk_raw, float* topk_avg, cudaStream_t st);

}  // namespace ftk

using namespace ftk;

extern "C" size_t ftk_block_score_workspace(int64_t bh_count, int64_t N) {
  return score_ws_layout(bh_count, N, 0, false, nullptr, nullptr);
}

extern "C" int ftk_block_score(const void* q, const void* k, int dtype, int64_t B, int64_t H,
                               int64_t N, int64_t D, int64_t sq_b, int64_t sq_n, int64_t sq_h,
                               int64_t sk_b, int64_t sk_n, int64_t sk_h, int64_t bh_begin,
                               int64_t bh_count, int score_block_size, int pad_head, int pad_tail,
                               float scale, float* block_scores, void* workspace,
                               size_t workspace_bytes,
                               int32_t* status, void* stream) {
  if (!block_scores) return FTK_ERR_BAD_ARG;
  if (bh_count <= 0 || N <= 0) return FTK_ERR_BAD_ARG;
  if (D != 64 && D != 128 && D != 256) return FTK_ERR_UNSUPPORTED;
  if (!workspace || workspace_bytes < ftk_block_score_workspace(bh_count, N))
    return FTK_ERR_WORKSPACE;
  if ((reinterpret_cast<uintptr_t>(workspace) & 255u) != 0) return FTK_ERR_BAD_ARG;
  ScoreWs ws;
  score_ws_layout(bh_count, N, 0, false, static_cast<char*>(workspace), &ws);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int e = run_score(q, k, dtype, B, H, N, D, sq_b, sq_n, sq_h, sk_b, sk_n, sk_h, bh_begin,
                    bh_count, score_block_size, pad_head, pad_tail, scale, block_scores, ws, status,
                    st);
  if (e) return e;
  const int M = static_cast<int>((pad_head + N + pad_tail) / score_block_size);
  const int64_t rows = bh_count * N;
  const int grid = static_cast<int>(std::min<int64_t>((rows * M + 255) / 256, 148 * 16));
  score_normalize_kernel<<<grid, 256, 0, st>>>(block_scores, ws.row_total, block_scores, rows, M);
  return launched(cudaGetLastError());
}

extern "C" size_t ftk_score_topk_workspace(int64_t bh_count, int64_t N, int64_t M) {
  return score_ws_layout(bh_count, N, M, true, nullptr, nullptr);
}

extern "C" int ftk_score_topk(const void* q, const void* k, int dtype, int64_t B, int64_t H,
                              int64_t N, int64_t D, int64_t sq_b, int64_t sq_n, int64_t sq_h,
                              int64_t sk_b, int64_t sk_n, int64_t sk_h, int64_t bh_begin,
                              int64_t bh_count, int score_block_size, int pad_head, int pad_tail,
                              float scale, int topk, float threshold, int32_t* topk_idx, float* topk_raw,
                              float* topk_avg, void* workspace, size_t workspace_bytes,
                              int32_t* status, void* stream) {
  if (!topk_idx || !topk_raw || !topk_avg || topk < 0) return FTK_ERR_BAD_ARG;
  if (bh_count <= 0 || N <= 0 || score_block_size <= 0) return FTK_ERR_BAD_ARG;
  const int64_t M = (pad_head + N + pad_tail) / score_block_size;
  if (M > 4096) return FTK_ERR_UNSUPPORTED;
  if (!workspace || workspace_bytes < ftk_score_topk_workspace(bh_count, N, M))
    return FTK_ERR_WORKSPACE;
  if ((reinterpret_cast<uintptr_t>(workspace) & 255u) != 0) return FTK_ERR_BAD_ARG;
  ScoreWs ws;
  score_ws_layout(bh_count, N, M, true, static_cast<char*>(workspace), &ws);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int e = run_score(q, k, dtype, B, H, N, D, sq_b, sq_n, sq_h, sk_b, sk_n, sk_h, bh_begin,
                    bh_count, score_block_size, pad_head, pad_tail, scale, ws.sums, ws, status, st);
  if (e) return e;
  return select_launch(ws.sums, ws.row_total, bh_count * N, static_cast<int>(M), topk,
                       score_block_size, pad_head, pad_tail, threshold, topk_idx, topk_raw,
                       topk_avg, st);
}
