// The pipelined forward kernel (sparse_fwd_pipe.cuh) on pairs of SMs (tcgen05
// cta_group::2), head dims 128 and 256.  Included by sparse_fwd.cu after it.
//
// A cluster of two CTAs owns 256 query rows (four q-blocks).  Each CTA keeps its
// own 128 rows of Q in TMEM, its own four S / P buffers, O accumulator and
// softmax warps, exactly as in the one-CTA kernel; both walk the union of the
// four q-blocks' candidate lists (and the up to four prologue blocks that give
// the rows their reference exponents).  Per kv block each CTA loads only
//   kv rows 32 r .. 32 r + 31 of K (all of d)    - its half of the B operand of
//        S = Q K^T (N = 64 kv rows split in two), and
//   d columns 64 r .. 64 r + 63 of V (all 64 rows) - its half of the B operand
//        of O += P V (N = 128 split in two),
// 16 KB per tile for twice the query rows (the one-CTA kernel loads 32 KB and
// is co-limited by the L2 -> SM path), and the M = 256 UMMAs cost 43 cycles at
// N = 64 and 64 at N = 128 for both CTAs together.  CTA 0 issues every UMMA;
// tcgen05.commit multicasts its arrivals; CTA 1's warp 1 forwards "my tiles
// have landed"; softmax warps of CTA 1 arrive on CTA 0's barriers through the
// cluster shared-memory window.  No TMA load is multicast.
//
// The issuing warp of CTA 0 bounds the loop: K of tile i + 4 and V of tile i share a
// stage, so that a round has three waits and two commits (a ring for either took five
// and three: 1.94 ms against 1.84 at B = 4, N = 8192, H = 16, head dim 128; 1.86
// against 1.80 at N = 15000 with 128-row blocks).
//
// Head dim 256: the 256-column O accumulator and the four S / P buffers fill
// TMEM, so Q stays in shared memory (an M = 256 UMMA with both operands there
// costs the same 43 cycles at N = 64) and the ring holds four stages of 32 KB.  Per tile 16 x 43 + 4 x 128 = 1200 cycles for 256 query rows,
// where the one-CTA exact kernel (16 x 75 + 4 x 138 for 128 rows, one softmax
// group, two stages) took 3700.
#pragma once

namespace ftk {

constexpr int FP2_THREADS = 576;   // TMA warp, UMMA warp, 4 softmax groups x 4 warps
constexpr int FP2_GROUPS = 4;
// Stages of the ring; a stage holds V of tile i and K of tile i + 4 (half of each).
__host__ __device__ constexpr int fp2_stages(int d) { return d > 128 ? 4 : 8; }
__host__ __device__ constexpr int fp2_tile(int d) { return d * 64; }           // bytes of either
__host__ __device__ constexpr size_t fp2_smem(int d) {
  return 1024 + static_cast<size_t>(d) * 256 + static_cast<size_t>(fp2_stages(d)) * 2 * fp2_tile(d);
}

template <int D, int FMT, int SUB>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(FP2_THREADS, 1)
sparse_fwd_pipe2_kernel(const __grid_constant__ CUtensorMap tm_q,
                        const __grid_constant__ CUtensorMap tm_k32,
                        const __grid_constant__ CUtensorMap tm_v, const FwdParams p) {
  constexpr bool BIG = D > 128;                // Q read from shared memory
  constexpr int NCH = D / 64;
  constexpr int Q_BYTES = NCH * 128 * 128;
  constexpr int KVB = 64;
  constexpr int TILE = fp2_tile(D);            // half a K tile (32 rows x D) or half a V tile
                                               // (64 rows x D / 2)
  constexpr int ST = fp2_stages(D), STAGE = 2 * TILE;
  constexpr uint32_t COL_S = BIG ? 0 : 64, COL_O = BIG ? 256 : 320;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem;
  uint8_t* sKV = smem + Q_BYTES;               // stage s: K half tile, then V half tile
  __shared__ UnionScratch un;
  __shared__ __align__(8) uint64_t bars[4 + 3 * ST + 2 * FP2_GROUPS];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_flag;
  __shared__ int s_ovf;
  __shared__ float s_l[FP2_GROUPS][128];
  __shared__ float s_mref[128];
  __shared__ OutTile s_out;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_ctarank();
  const int per = 128 / p.g;                  // q-blocks (of 64 or 32 rows) per CTA
  const int m0 = (blockIdx.x >> 1) * 2 * per; // first of the pair's q-blocks
  const int bh = blockIdx.y;
  const int b_idx = bh / p.H, h_idx = bh - b_idx * p.H;
  const int groups = min(2 * per, p.QM - m0);
  const int tile_row0 = m0 * p.g + 128 * static_cast<int>(rank) - p.q_pad_head;   // my 128 rows

  const uint32_t bar_q = smem_u32(&bars[0]);
  const uint32_t bar_final = smem_u32(&bars[1]);
  const uint32_t bar_qt = smem_u32(&bars[2]);    // CTA 0: Q of both CTAs copied into TMEM
                                                 // (BIG: CTA 1's Q has landed)
  const uint32_t bar_pro = smem_u32(&bars[3]);   // CTA 0: both CTAs' reference exponents are there
  auto bar_full = [&](int s) { return smem_u32(&bars[4 + s]); };
  auto bar_empty = [&](int s) { return smem_u32(&bars[4 + ST + s]); };
  auto bar_peer = [&](int s) { return smem_u32(&bars[4 + 2 * ST + s]); };   // CTA 0 only
  constexpr int BAR_S0 = 4 + 3 * ST;
  auto bar_sfull = [&](int b) { return smem_u32(&bars[BAR_S0 + b]); };
  auto bar_pfull = [&](int b) { return smem_u32(&bars[BAR_S0 + FP2_GROUPS + b]); };

  if (tid == 0) {
    abort_flag = 0;
    s_ovf = 0;
    mbar_init(bar_q, 1);
    mbar_init(bar_final, 1);
    mbar_init(bar_qt, BIG ? 1 : 8);        // the 4 copying warps of each CTA
    mbar_init(bar_pro, 8);                 // the 4 warps of group 0 of each CTA
    for (int s = 0; s < ST; s++) {
      mbar_init(bar_full(s), 1);
      mbar_init(bar_empty(s), 1);
      mbar_init(bar_peer(s), 1);
    }
    for (int b = 0; b < FP2_GROUPS; b++) {
      mbar_init(bar_sfull(b), 1);
      mbar_init(bar_pfull(b), 8);          // the group's 4 warps in each CTA
    }
    mbar_init_fence();
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k32);
    tma_prefetch_desc(&tm_v);
  }
  if (warp == 0) {
    tmem_alloc2(smem_u32(&tmem_base_s), 512);
    tmem_relinquish2();
  }
  if (tid == 32)
    s_out = {{static_cast<int64_t>(b_idx) * p.so_b + static_cast<int64_t>(h_idx) * p.so_h, 0},
             tile_row0, min(p.N, tile_row0 + (groups - per * static_cast<int>(rank)) * p.g)};
  clear_flags(sKV, p.Mkv, groups);
  tc_fence_before();
  cluster_arrive();
  pdl_wait();
  if (tid == 0) {   // under the building of the union
    mbar_expect_tx(bar_q, Q_BYTES);
    for (int c = 0; c < NCH; c++)
      tma_load_4d(smem_u32(sQ) + c * 128 * 128, &tm_q, bar_q, c * 64, h_idx, tile_row0, b_idx);
  }
  const int n = build_union<FP2_THREADS / 32>(
      un, sKV, p.merged + static_cast<int64_t>(bh) * p.list_rows * p.W, m0, groups, p.W, nullptr, p.Mkv,
      SUB, p.lm, p.status);
  pdl_launch();
  // tiles whose scores give the rows their reference exponents
  const CoverTiles pro = cover_tiles(un, n, groups, SUB, FP2_GROUPS);
  cluster_wait();            // barriers of both CTAs are initialised before anyone signals them
  tc_fence_after();
  const uint32_t tmem = tmem_base_s;
  WaitCtx w{&abort_flag, p.status};

  // prologue entry e goes through S buffer e
  const int npro = pro.n;
  auto pro_block = [&](int e) { return static_cast<int>(un.ids[pro.entry(e)]); };

  if (warp == 0) {
    // ------------------------------------------------------- TMA producer
    if (lane == 0 && n > 0) {
      // Stage rr holds K of tile rr and V of tile rr - 4; the first four, which
      // have no V, take the prologue's K tiles in its place.
      const int lead = min(n, FP2_GROUPS);
      const int hk = h_idx / p.kv_hdiv;   // out of the loop: a division takes 150 cycles
      const int dcol = D / 2 * static_cast<int>(rank), rsub = 32 * static_cast<int>(rank);
      for (int rr = 0; rr < n + FP2_GROUPS; rr++) {
        if (rr >= lead && rr < FP2_GROUPS) continue;
        const int s = rr % ST;
        if (!mbar_wait(bar_empty(s), ((rr / ST) & 1) ^ 1, w, FTK_DEV_TIMEOUT_TMA)) break;
        const bool has_k = rr < n, has_pro = rr < npro, has_v = rr >= FP2_GROUPS;
        const uint32_t kb = smem_u32(sKV) + s * STAGE, vb = kb + TILE;
        mbar_expect_tx(bar_full(s), (has_k && (has_pro || has_v)) ? STAGE : TILE);
        if (has_v) {
          const int tok0 = static_cast<int>(un.ids[rr - FP2_GROUPS]) * KVB - p.kv_pad_head;
#pragma unroll
          for (int c = 0; c < NCH / 2; c++)
            tma_load_4d(vb + c * 8192, &tm_v, bar_full(s), dcol + c * 64, hk, tok0, b_idx);
        }
        if (has_pro)
          for (int c = 0; c < NCH; c++)
            tma_load_4d(vb + c * 4096, &tm_k32, bar_full(s), c * 64, hk,
                        pro_block(rr) * KVB - p.kv_pad_head + rsub, b_idx);
        if (has_k) {
          const int tok0 = static_cast<int>(un.ids[rr]) * KVB - p.kv_pad_head + rsub;
          for (int c = 0; c < NCH; c++)
            tma_load_4d(kb + c * 4096, &tm_k32, bar_full(s), c * 64, hk, tok0, b_idx);
        }
      }
    }
  } else if (warp == 1 && rank == 1) {
    // ----------------------- CTA 1: tell CTA 0 when my tiles have landed
    if (BIG && n > 0) {
      const bool landed = mbar_wait(bar_q, 0, w, FTK_DEV_TIMEOUT_MMA);
      __syncwarp();
      if (landed && lane == 0) mbar_arrive_cta(bar_qt, 0);
    }
    for (int rr = 0; n > 0 && rr < n + FP2_GROUPS; rr++) {
      if (rr >= n && rr < FP2_GROUPS) continue;
      const int s = rr % ST;
      if (!mbar_wait(bar_full(s), (rr / ST) & 1, w, FTK_DEV_TIMEOUT_MMA)) break;
      __syncwarp();
      if (lane == 0) mbar_arrive_cta(bar_peer(s), 0);
    }
  } else if (warp == 1) {
    // ----------------------------- CTA 0: UMMA issuer for the CTA pair
    if (n > 0) {
      const uint32_t idesc_s = umma_idesc(256, KVB, FMT, 0, 0);
      const uint32_t idesc_pv = umma_idesc(256, D, FMT, 0, 1);
      const uint64_t kdesc0 = smem_desc_sw128(smem_u32(sKV), 16, 1024);
      const uint64_t vdesc0 = smem_desc_sw128(smem_u32(sKV) + TILE, 8192, 1024);
      const uint64_t qdesc0 = smem_desc_sw128(smem_u32(sQ), 16, 1024);
      bool ok = mbar_wait(bar_qt, 0, w, FTK_DEV_TIMEOUT_MMA);
      if (BIG && ok) ok = mbar_wait(bar_q, 0, w, FTK_DEV_TIMEOUT_MMA);
      tc_fence_after();
      // S = Q K^T for the K tile at `off` into S buffer `buf`; Q read from TMEM
      // (elected lane only)
      auto mma_s = [&](int off, int buf) {
        const uint64_t kdesc = desc_advance(kdesc0, off);
        const uint32_t d_tmem = tmem + COL_S + buf * 64;
#pragma unroll
        for (int ks = 0; ks < D / 16; ks++) {
          const uint64_t b = desc_advance(kdesc, (ks / 4) * 4096 + (ks % 4) * 32);
          if (BIG)
            umma2_ss(d_tmem, desc_advance(qdesc0, (ks / 4) * 128 * 128 + (ks % 4) * 32), b, idesc_s,
                     ks > 0);
          else
            umma2_ts(d_tmem, tmem + ks * 8, b, idesc_s, ks > 0);
        }
        umma2_commit(bar_sfull(buf), 3);
      };
      // the reference tiles' scores, then those of the first tiles whose buffers they do
      // not take, and the others once the references are there
      const int lead = min(n, FP2_GROUPS);
      for (int t = 0; ok && t < lead; t++) {
        const uint32_t wb[2] = {bar_full(t), bar_peer(t)};
        const uint32_t wp[2] = {0, 0};
        ok = mbar_wait_all<2>(wb, wp, w, FTK_DEV_TIMEOUT_MMA);
        tc_fence_after();
        if (ok && elect_one()) {
          if (t < npro) {
            mma_s(t * STAGE + TILE, t);
          } else {
            mma_s(t * STAGE, t);
            umma2_commit(bar_empty(t), 3);
          }
        }
        __syncwarp();
      }
      if (ok) ok = mbar_wait(bar_pro, 0, w, FTK_DEV_TIMEOUT_MMA);
      tc_fence_after();
      if (ok && elect_one())
        for (int t = 0; t < npro; t++) {
          mma_s(t * STAGE, t);
          umma2_commit(bar_empty(t), 3);
        }
      __syncwarp();
      // per round every barrier is waited for first (together), then P V of
      // tile i and S of tile i + 4 go out as one batch
      for (int q = 0; ok && q * FP2_GROUPS < n; q++) {
        const int s0 = ((q + 1) * FP2_GROUPS) % ST;
        const uint32_t full_ph = ((q + 1) * FP2_GROUPS / ST) & 1, p_ph = q & 1;
#pragma unroll
        for (int u = 0; u < FP2_GROUPS; u++) {
          const int i = q * FP2_GROUPS + u, s = s0 + u;
          if (i >= n) break;
          const uint32_t wb[3] = {bar_full(s), bar_peer(s), bar_pfull(u)};
          const uint32_t wp[3] = {full_ph, full_ph, p_ph};
          if (!mbar_wait_all<3>(wb, wp, w, FTK_DEV_TIMEOUT_MMA)) {
            ok = false;
            break;
          }
          tc_fence_after();
          if (elect_one()) {
            const uint64_t vdesc = desc_advance(vdesc0, s * STAGE);
#pragma unroll
            for (int ks = 0; ks < KVB / 16; ks++)
              umma2_ts(tmem + COL_O, tmem + COL_S + u * 64 + ks * 8,
                       desc_advance(vdesc, ks * 2048), idesc_pv, (i > 0) || (ks > 0));
            // S(i+4) lands on the columns PV(i) reads P from; UMMAs run in issue order
            if (i + FP2_GROUPS < n) mma_s(s * STAGE, u);
            umma2_commit(bar_empty(s), 3);
          }
          __syncwarp();
        }
      }
      if (elect_one()) umma2_commit(bar_final, 3);
      __syncwarp();
    }
  } else {
    // ---------------------------------------------------- softmax threads
    const int gw = (warp - 2) >> 2;          // softmax group = S buffer it drains
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const int grp = per * static_cast<int>(rank) + r / p.g;   // q-block of the pair (warp-uniform)
    const uint32_t lane_addr = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t s_addr = lane_addr + COL_S + gw * 64;
    const float c = p.scale_log2;
    float mref = 0.f, l = 0.f;
    bool ok = true, ovf = false;

    if (!BIG && n > 0 && gw == 0) {
      // group 0 moves the Q tile from (swizzled) shared memory into TMEM
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
      if (lane == 0) mbar_arrive_cta(bar_qt, 0);
    }

    if (n > 0) {
      // ---- reference exponent: scaled row maximum over the q-block's prologue tile.
      // Group 0 works it out; behind the barrier the others may rely on the first phase of
      // every prologue buffer being over, as their parity waits must.
      if (gw == 0) {
        for (int e = 0; ok && e < npro; e++)
          ok = mbar_wait(bar_sfull(e), 0, w, FTK_DEV_TIMEOUT_CONSUMER);
        tc_fence_after();
        float mx = -INFINITY;
        const int pb = (pro.of >> (4 * grp)) & 15;   // grp is the same for the warp's rows
        if (ok && pb != 15) {
          const ColSpan cs =
              col_span(un, pro.entry(pb), SUB, grp, pro_block(pb) * KVB - p.kv_pad_head, KVB, p.N);
          mx = tmem_row_max(lane_addr + COL_S + pb * 64, KVB, cs.lo, cs.hi);
          ovf = mx == -INFINITY;   // no reference for the row's other tiles: the exact kernel's
        }
        s_mref[r] = (mx > -INFINITY) ? mx * c : 0.f;
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cta(bar_pro, 0);
      }
      asm volatile("bar.sync 1, %0;" ::"n"(512) : "memory");
      mref = s_mref[r];
    }

    const float2 c2 = make_float2(c, c);
    const float2 nm = make_float2(-mref, -mref);
    for (int i = gw; ok && i < n; i += FP2_GROUPS) {
      // S(i) complete also means PV(i-4) has retired: the P columns are free
      const int u = (gw < npro ? 1 : 0) + (i / FP2_GROUPS);
      if (!mbar_wait(bar_sfull(gw), u & 1, w, FTK_DEV_TIMEOUT_CONSUMER)) {
        ok = false;
        break;
      }
      tc_fence_after();
      const int tok0 = static_cast<int>(un.ids[i]) * KVB - p.kv_pad_head;
      const ColSpan cs = col_span(un, i, SUB, grp, tok0, KVB, p.N);
      const int lo = cs.lo, hi = cs.hi;
      const bool fast = cs.on && lo == 0 && hi == KVB;   // the warp's rows are of one q-block

      if (cs.on) {
        uint32_t v0[32], v1[32];
        tmem_ld32(s_addr, v0);
        tmem_ld32(s_addr + 32, v1);
        tmem_wait_ld();
        uint32_t pk[16];
        float2 acc = make_float2(0.f, 0.f);
        if (fast) {
#pragma unroll
          for (int x = 0; x < 32; x += 2) {
            const float2 t = __ffma2_rn(
                make_float2(__uint_as_float(v0[x]), __uint_as_float(v0[x + 1])), c2, nm);
            const float2 e = make_float2(fast_exp2(t.x), fast_exp2(t.y));
            acc = __fadd2_rn(acc, e);
            pk[x >> 1] = pack16<FMT>(e.x, e.y);
          }
          tmem_st16(s_addr, pk);
#pragma unroll
          for (int x = 0; x < 32; x += 2) {
            const float2 t = __ffma2_rn(
                make_float2(__uint_as_float(v1[x]), __uint_as_float(v1[x + 1])), c2, nm);
            const float2 e = make_float2(fast_exp2(t.x), fast_exp2(t.y));
            acc = __fadd2_rn(acc, e);
            pk[x >> 1] = pack16<FMT>(e.x, e.y);
          }
          tmem_st16(s_addr + 16, pk);
        } else {
#pragma unroll
          for (int x = 0; x < 32; x += 2) {
            float a0 = 0.f, a1 = 0.f;
            if (x >= lo && x < hi) a0 = fast_exp2(fmaf(__uint_as_float(v0[x]), c, -mref));
            if (x + 1 >= lo && x + 1 < hi)
              a1 = fast_exp2(fmaf(__uint_as_float(v0[x + 1]), c, -mref));
            acc.x += a0;
            acc.y += a1;
            pk[x >> 1] = pack16<FMT>(a0, a1);
          }
          tmem_st16(s_addr, pk);
#pragma unroll
          for (int x = 0; x < 32; x += 2) {
            float b0 = 0.f, b1 = 0.f;
            if (x + 32 >= lo && x + 32 < hi)
              b0 = fast_exp2(fmaf(__uint_as_float(v1[x]), c, -mref));
            if (x + 33 >= lo && x + 33 < hi)
              b1 = fast_exp2(fmaf(__uint_as_float(v1[x + 1]), c, -mref));
            acc.x += b0;
            acc.y += b1;
            pk[x >> 1] = pack16<FMT>(b0, b1);
          }
          tmem_st16(s_addr + 16, pk);
        }
        const float lt = acc.x + acc.y;
        if (!(lt <= fp_overflow_bound<FMT>())) ovf = true;   // also catches NaN
        l += lt;
      } else {
        uint32_t z[16];
#pragma unroll
        for (int x = 0; x < 16; x++) z[x] = 0u;
        tmem_st16(s_addr, z);
        tmem_st16(s_addr + 16, z);
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cta(bar_pfull(gw), 0);
    }

    // ------------------------------------------------------------ epilogue
    // row sums of the four groups add up (same reference); each group converts
    // and stores a quarter of the head dimension
    const int ew = (late_tid() >> 5) - 2, er = ((ew + 2) & 3) * 32 + lane;   // warp, row
    s_l[ew >> 2][er] = l;
    const int qrow = s_out.row0 + er;
    const bool row_valid = qrow >= 0 && qrow < s_out.last;
    if (ovf && row_valid) atomicOr(&s_ovf, 1);
    asm volatile("bar.sync 1, 512;" ::: "memory");
    if (ok) ok = mbar_wait(n > 0 ? bar_final : bar_q, 0, w, FTK_DEV_TIMEOUT_EPILOGUE);
    if (ok) {
      tc_fence_after();
      const float lt = ((s_l[0][er] + s_l[1][er]) + s_l[2][er]) + s_l[3][er];
      const bool have = (n > 0) && lt > 0.f;
      const float inv = have ? 1.f / lt : 0.f;
      // every copy has landed and every UMMA has retired: the tiles make room for O
      constexpr int QUART = D / 4;   // 32 or 64 columns per group
#pragma unroll 1
      for (int c0 = (ew >> 2) * QUART, x0 = 0; x0 < QUART; c0 += 32, x0 += 32) {
        uint32_t ov[32], pk[16];
        if (n > 0) {
          tmem_ld32(lane_addr + COL_O + c0, ov);
          tmem_wait_ld();
        }
#pragma unroll
        for (int x = 0; x < 32; x += 2) {
          const float a = have ? __uint_as_float(ov[x]) * inv : 0.f;
          const float b = have ? __uint_as_float(ov[x + 1]) * inv : 0.f;
          pk[x >> 1] = pack16<FMT>(a, b);
        }
        store_rows(smem + ew * 2048, pk, p.o, s_out, 0, (ew + 2) & 3, p.so_n, c0, p.D, FMT,
                   p.out_f32 != 0);
      }
      if (row_valid && ew < 4)
        p.lse[static_cast<int64_t>(bh) * p.N + qrow] =
            have ? (mref + log2f(lt)) * 0.6931471805599453f : -INFINITY;
    }
  }

  tc_fence_before();
  __syncthreads();
  // the exact kernel redoes 128-row tiles: this CTA's rows are its tile 2 * pair + rank
  const int units_x = p.tiles_x;
  const int unit_x = static_cast<int>(blockIdx.x >> 1) * 2 + static_cast<int>(rank);
  if (tid == 0 && p.redo_out && unit_x < units_x)
    p.redo_out[blockIdx.y * units_x + unit_x] =
        s_ovf | (((pro.left >> (per * rank)) & ((1 << per) - 1)) != 0);
  if (abort_flag)
    for (int i = 0; i < 200; i++) __nanosleep(1000);
  // neither CTA may leave (or free TMEM) while the other can still touch it
  cluster_sync_all();
  if (warp == 0) tmem_dealloc2(tmem, 512);
}

}  // namespace ftk
