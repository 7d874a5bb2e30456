// Deeply pipelined forward kernel for q and kv blocks of 64 or 32 rows.  Included
// by sparse_fwd.cu (shares FwdParams).
//
// The exact kernel keeps a running maximum per softmax group, which ties every
// P tile to its group's accumulator: two groups, two O accumulators, two S
// buffers are all that fit in TMEM, and with two tiles in flight the tensor
// core idles while a group does its exponentials.  Here every row uses ONE
// fixed reference exponent for the whole list: the row's scaled maximum over one
// tile that its q-block lists, the tile that most of the CTA's q-blocks share
// (cover_tiles; a short prologue computes it).  P = 2^(c S - ref)
// then needs no rescaling, all tiles add into a single O accumulator, and NG
// softmax groups work on NG S buffers at once:
//   TMEM columns  Q, D / 2 | S/P buffers, 64 each | O, D
// With q-blocks of 32 rows (up to four reference tiles, each in an S buffer), and at head
// dim 128 in grids of one wave, a CTA has four groups and the SM to itself.  Otherwise
// it has two, 256 TMEM columns and half the shared memory, and
// two CTAs share an SM: as many tiles are in flight, the list union, first loads,
// reference tiles and last tiles of one CTA run under the tiles of the other, and two
// warps issue.  At head dim 128 Q then has no columns in TMEM and stays in shared memory, which
// leaves room for two stages.  A UMMA with both operands in shared memory takes 75 cycles instead
// of 42, but not beside another CTA's: a step takes 620 cycles (lists of 16 and 30 blocks alike for
// neighbours, B = 2, N = 4096, H = 32), 745 with the SM to itself, and 14000 cycles around the
// steps of a CTA are hidden.  The issuing warp bounds the loop otherwise: with 16 softmax warps beside
// it a round of 8 UMMAs, two commits and two waits takes it 600 cycles, the exponentials
// 512.  Forward at B = 1, H = 16,
// N = 8192, all pairs: 404 us with four groups, a K ring and a V ring; 388 with K and
// V in one ring (two waits and two commits per tile, were three and three) and
// addresses that the unrolled rounds share; 348 with two CTAs per SM.  Head dim 128,
// N = 8192, grouped heads: 312 -> 291 us from the ring.
// bf16 and fp32 share the exponent range, so a later block may exceed the
// reference by up to 2^80 before anything overflows (fp16: 2^15, P must stay
// below 65504); a row whose tile sum passes that bound marks its tile's word in
// `redo_out`, and the exact kernel, launched behind this one with a CTA per SM, looks
// through the words and recomputes exactly those tiles.  So does a row whose reference tile is
// all -inf: it has no reference for the others.
#pragma once

namespace ftk {

__host__ __device__ constexpr int fp_threads(int ng) { return 64 + 128 * ng; }   // TMA, UMMA warps
// Stages of the ring; a stage holds what one round of the issuing warp reads, V of
// tile i and K of tile i + ng.  A multiple of ng.
__host__ __device__ constexpr int fp_stages(int d, int ng) { return d == 64 && ng == 4 ? 8 : d == 128 && ng == 2 ? 2 : 4; }
constexpr size_t FP_STATIC = 16 * 1024;   // at most, beside the ring (checked in the kernel)
__host__ __device__ constexpr size_t fp_smem(int d, int ng) {
  return 1024 + (d / 64) * (128 * 128 + static_cast<size_t>(fp_stages(d, ng)) * 2 * 64 * 128);
}
// A tile's row sum of P above this marks the CTA for the exact kernel: 2^80 for
// bf16 (fp32 exponent range), 2^15 for fp16 (P itself must stay below 65504).
template <int FMT>
__device__ __forceinline__ float fp_overflow_bound() {
  return FMT == 1 ? 1.2089258196146292e24f : 32768.f;
}

template <int FMT>
__device__ __forceinline__ uint32_t pack16(float a, float b) {
  if (FMT == 1) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  __half2 v = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}

template <int D, int FMT, int SUB, int NG>
__global__ void __launch_bounds__(fp_threads(NG), 4 / NG)
sparse_fwd_pipe_kernel(const __grid_constant__ CUtensorMap tm_q,
                       const __grid_constant__ CUtensorMap tm_k,
                       const __grid_constant__ CUtensorMap tm_v, const FwdParams p) {
  constexpr int NCH = D / 64;
  constexpr int Q_BYTES = NCH * 128 * 128;
  constexpr int KVB = 64;
  constexpr int CHUNK = KVB * 128;             // one 64-wide chunk of a K or V tile
  constexpr int TILE = NCH * CHUNK;            // one K or V tile
  constexpr int ST = fp_stages(D, NG), STAGE = 2 * TILE;
  constexpr bool Q_S = D == 128 && NG == 2;                // Q stays in shared memory
  constexpr int SUMS = D == 128 ? 4 : NG;                  // parts of a row's sum (see below)
  constexpr int COL_S = Q_S ? 0 : D / 2, COL_O = COL_S + 64 * NG;   // Q in the columns before S
  constexpr int TMEM_COLS = NG == 2 ? 256 : 512;
  static_assert(COL_O + D <= TMEM_COLS, "TMEM columns");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem;
  uint8_t* sKV = smem + Q_BYTES;               // stage s: K tile, then V tile
  __shared__ UnionScratch un;
  __shared__ __align__(8) uint64_t bars[4 + 2 * ST + 2 * NG];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_flag;
  __shared__ int s_ovf;
  __shared__ float s_l[SUMS][128];
  __shared__ float s_mref[128];
  __shared__ OutTile s_out;
  static_assert(sizeof(un) + sizeof(bars) + sizeof(s_l) + sizeof(s_mref) + sizeof(s_out) +
                        sizeof(tmem_base_s) + sizeof(abort_flag) + sizeof(s_ovf) + 64 <= FP_STATIC,
                "static shared memory");
  static_assert(NG != 2 || 2 * (fp_smem(D, NG) + FP_STATIC + 1024) <= 228 * 1024, "two CTAs per SM");

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.x * p.G;
  const int bh = blockIdx.y;
  const int b_idx = bh / p.H, h_idx = bh - b_idx * p.H;
  const int groups = min(p.G, p.QM - m0);
  const int tile_row0 = m0 * p.g - p.q_pad_head;

  const uint32_t bar_q = smem_u32(&bars[0]);
  const uint32_t bar_final = smem_u32(&bars[1]);
  const uint32_t bar_qt = smem_u32(&bars[2]);    // Q copied into TMEM
  const uint32_t bar_pro = smem_u32(&bars[3]);   // the rows' reference exponents are there
  auto bar_full = [&](int s) { return smem_u32(&bars[4 + s]); };
  auto bar_empty = [&](int s) { return smem_u32(&bars[4 + ST + s]); };
  constexpr int BAR_S0 = 4 + 2 * ST;
  auto bar_sfull = [&](int b) { return smem_u32(&bars[BAR_S0 + b]); };
  auto bar_pfull = [&](int b) { return smem_u32(&bars[BAR_S0 + NG + b]); };

  if (tid == 0) {
    abort_flag = 0;
    s_ovf = 0;
    mbar_init(bar_q, 1);
    mbar_init(bar_final, 1);
    mbar_init(bar_qt, 4);
    mbar_init(bar_pro, 4);
    for (int s = 0; s < ST; s++) {
      mbar_init(bar_full(s), 1);
      mbar_init(bar_empty(s), 1);
    }
    for (int b = 0; b < NG; b++) {
      mbar_init(bar_sfull(b), 1);
      mbar_init(bar_pfull(b), 4);
    }
    mbar_init_fence();
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(&tmem_base_s), TMEM_COLS);
    tmem_relinquish();
  }
  if (tid == 32)
    s_out = {{static_cast<int64_t>(b_idx) * p.so_b + static_cast<int64_t>(h_idx) * p.so_h, 0},
             tile_row0, min(p.N, tile_row0 + groups * p.g)};
  clear_flags(sKV, p.Mkv, groups);
  tc_fence_before();
  pdl_wait();
  if (tid == 0) {   // under the building of the union
    mbar_expect_tx(bar_q, Q_BYTES);
    for (int c = 0; c < NCH; c++)
      tma_load_4d(smem_u32(sQ) + c * 128 * 128, &tm_q, bar_q, c * 64, h_idx, tile_row0, b_idx);
  }
  const int n = build_union<fp_threads(NG) / 32>(
      un, sKV, p.merged + static_cast<int64_t>(bh) * p.list_rows * p.W, m0, groups, p.W, nullptr, p.Mkv,
      SUB, p.lm, p.status);
  pdl_launch();
  tc_fence_after();
  // tiles whose scores give the rows their reference exponents
  const CoverTiles pro = cover_tiles(un, n, groups, SUB, NG);
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base_s, 0);
  WaitCtx w{&abort_flag, p.status};

  // prologue entry e goes through S buffer e
  const int npro = pro.n;
  auto pro_block = [&](int e) { return static_cast<int>(un.ids[pro.entry(e)]); };

  if (warp == 0) {
    // ------------------------------------------------------- TMA producer
    if (lane == 0 && n > 0) {
      // Stage rr holds K of tile rr and V of tile rr - NG; the first NG, which
      // have no V, take the prologue's K tiles in its place.
      const int lead = min(n, NG);
      const int hk = h_idx / p.kv_hdiv;   // out of the loop: a division takes 150 cycles
      for (int rr = 0; rr < n + NG; rr++) {
        if (rr >= lead && rr < NG) continue;
        const int s = rr % ST;
        if (!mbar_wait(bar_empty(s), ((rr / ST) & 1) ^ 1, w, FTK_DEV_TIMEOUT_TMA)) break;
        const bool has_k = rr < n, has_pro = rr < npro, has_v = rr >= NG;
        const uint32_t kb = smem_u32(sKV) + s * STAGE, vb = kb + TILE;
        mbar_expect_tx(bar_full(s), (has_k && (has_pro || has_v)) ? STAGE : TILE);
        if (has_v) {
          const int tok0 = static_cast<int>(un.ids[rr - NG]) * KVB - p.kv_pad_head;
          for (int c = 0; c < NCH; c++)
            tma_load_4d(vb + c * CHUNK, &tm_v, bar_full(s), c * 64, hk, tok0, b_idx);
        }
        if (has_pro)
          for (int c = 0; c < NCH; c++)
            tma_load_4d(vb + c * CHUNK, &tm_k, bar_full(s), c * 64, hk,
                        pro_block(rr) * KVB - p.kv_pad_head, b_idx);
        if (has_k) {
          const int tok0 = static_cast<int>(un.ids[rr]) * KVB - p.kv_pad_head;
          for (int c = 0; c < NCH; c++)
            tma_load_4d(kb + c * CHUNK, &tm_k, bar_full(s), c * 64, hk, tok0, b_idx);
        }
      }
    }
  } else if (warp == 1) {
    // -------------------------------------------------------- UMMA issuer
    if (n > 0) {
      const uint32_t idesc_s = umma_idesc(128, KVB, FMT, 0, 0);
      const uint32_t idesc_pv = umma_idesc(128, D, FMT, 0, 1);
      const uint64_t kdesc0 = smem_desc_sw128(smem_u32(sKV), 16, 1024);
      const uint64_t vdesc0 = smem_desc_sw128(smem_u32(sKV) + TILE, CHUNK, 1024);
      const uint64_t qdesc0 = smem_desc_sw128(smem_u32(sQ), 16, 1024);
      // head dim 128: without branches around what one lane issues (see elect_one)
      constexpr bool CONV = D == 128;
      const uint32_t el = CONV ? elect_one() : 1u;
      auto mine = [&]() { return CONV || elect_one(); };
      auto all = [&](bool x) { return CONV ? warp_all(x) : x; };
      bool ok = all(mbar_wait(Q_S ? bar_q : bar_qt, 0, w, FTK_DEV_TIMEOUT_MMA));
      tc_fence_after();
      // S = Q K^T for the K tile at `off` into S buffer `buf`; Q read from TMEM
      // (one lane)
      auto mma_s = [&](int off, int buf) {
        const uint64_t kdesc = desc_advance(kdesc0, off);
#pragma unroll
        for (int ks = 0; ks < D / 16; ks++) {
          const uint64_t b = desc_advance(kdesc, (ks / 4) * CHUNK + (ks % 4) * 32);
          if (Q_S)
            umma_ss(tmem + COL_S + buf * 64, desc_advance(qdesc0, (ks / 4) * 128 * 128 + (ks % 4) * 32), b,
                    idesc_s, ks > 0, el);
          else
            umma_ts(tmem + COL_S + buf * 64, tmem + ks * 8, b, idesc_s, ks > 0, el);
        }
        umma_commit(bar_sfull(buf), el);
      };
      // the reference tiles' scores, then those of the first tiles whose buffers they do
      // not take, and the others once the references are there
      const int lead = min(n, NG);
      for (int t = 0; ok && t < lead; t++) {
        ok = all(mbar_wait(bar_full(t), 0, w, FTK_DEV_TIMEOUT_MMA));
        tc_fence_after();
        if (ok && mine()) {
          if (t < npro) {
            mma_s(t * STAGE + TILE, t);
          } else {
            mma_s(t * STAGE, t);
            umma_commit(bar_empty(t), el);
          }
        }
        __syncwarp();
      }
      if (ok) ok = all(mbar_wait(bar_pro, 0, w, FTK_DEV_TIMEOUT_MMA));
      tc_fence_after();
      if (ok && mine())
        for (int t = 0; t < npro; t++) {
          mma_s(t * STAGE, t);
          umma_commit(bar_empty(t), el);
        }
      __syncwarp();
      // The tensor core runs dry whenever the issuing thread waits, so both
      // barriers of a round are waited for first and the round's UMMAs (P V of
      // tile i, then S of tile i + NG) go out as one uninterrupted batch.
      for (int q = 0; ok && q * NG < n; q++) {
        const int s0 = ((q + 1) * NG) % ST;
        const uint32_t full_ph = ((q + 1) * NG / ST) & 1, p_ph = q & 1;
#pragma unroll
        for (int u = 0; u < NG; u++) {
          const int i = q * NG + u, s = s0 + u;
          if (i >= n) break;
          const uint32_t wb[2] = {bar_full(s), bar_pfull(u)};
          const uint32_t wp[2] = {full_ph, p_ph};
          if (!all(mbar_wait_all<2>(wb, wp, w, FTK_DEV_TIMEOUT_MMA))) {
            ok = false;
            break;
          }
          tc_fence_after();
          if (mine()) {
            const uint64_t vdesc = desc_advance(vdesc0, s * STAGE);
#pragma unroll
            for (int ks = 0; ks < KVB / 16; ks++)
              umma_ts(tmem + COL_O, tmem + COL_S + u * 64 + ks * 8,
                      desc_advance(vdesc, ks * 2048), idesc_pv, (i > 0) || (ks > 0), el);
            // S(i + NG) lands on the columns PV(i) reads P from; UMMAs run in issue order
            if (i + NG < n) mma_s(s * STAGE, u);
            umma_commit(bar_empty(s), el);
          }
          __syncwarp();
        }
      }
      if (ok && mine()) umma_commit(bar_final, el);
      __syncwarp();
    }
  } else {
    // ---------------------------------------------------- softmax threads
    const int gw = (warp - 2) >> 2;          // softmax group = S buffer it drains
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const int grp = r / p.g;                 // warp-uniform: q-blocks are 64 or 32 rows
    const uint32_t lane_addr = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t s_addr = lane_addr + COL_S + gw * 64;
    const float c = p.scale_log2;
    // With two groups at head dim 128 each keeps two sums in turn, so that a row's is added up as
    // by four groups, here or on pairs: the size of the grid chooses the kernel, not the bits.
    float mref = 0.f, l = 0.f, l_next = 0.f;
    bool ok = true, ovf = false;

    if (!Q_S && n > 0 && gw == 0) {
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
      if (lane == 0) mbar_arrive(bar_qt);
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
        if (lane == 0) mbar_arrive(bar_pro);
      }
      asm volatile("bar.sync 1, %0;" ::"n"(128 * NG) : "memory");
      mref = s_mref[r];
    }

    const float2 c2 = make_float2(c, c);
    const float2 nm = make_float2(-mref, -mref);
    for (int i = gw; ok && i < n; i += NG) {
      // S(i) complete also means PV(i - NG) has retired: the P columns are free
      const int u = (gw < npro ? 1 : 0) + (i / NG);
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
      if (lane == 0) mbar_arrive(bar_pfull(gw));
      if (SUMS > NG) {
        const float t = l;
        l = l_next;
        l_next = t;
      }
    }
    if (SUMS > NG && n > gw && (((n - 1 - gw) / NG) & 1) == 0) {   // an odd number of tiles
      const float t = l;
      l = l_next;
      l_next = t;
    }

    // ------------------------------------------------------------ epilogue
    // row sums of the groups add up (same reference); each group converts
    // and stores a quarter of the head dimension
    const int ew = (late_tid() >> 5) - 2, er = ((ew + 2) & 3) * 32 + lane;   // warp, row
    s_l[ew >> 2][er] = l;
    if (SUMS > NG) s_l[NG + (ew >> 2)][er] = l_next;
    const int qrow = s_out.row0 + er;
    const bool row_valid = qrow >= 0 && qrow < s_out.last;
    if (ovf && row_valid) atomicOr(&s_ovf, 1);
    asm volatile("bar.sync 1, %0;" ::"n"(128 * NG) : "memory");
    if (ok) ok = mbar_wait(n > 0 ? bar_final : bar_q, 0, w, FTK_DEV_TIMEOUT_EPILOGUE);
    if (ok) {
      tc_fence_after();
      float lt = s_l[0][er];
#pragma unroll
      for (int x = 1; x < SUMS; x++) lt += s_l[x][er];
      const bool have = (n > 0) && lt > 0.f;
      const float inv = have ? 1.f / lt : 0.f;
      // every copy has landed and every UMMA has retired: the tiles make room for O
      constexpr int QUART = D / NG, PART = QUART < 32 ? QUART : 32;   // columns per group, at once
#pragma unroll 1
      for (int c0 = (ew >> 2) * QUART; c0 < (ew >> 2) * QUART + QUART; c0 += PART) {
        uint32_t ov[PART], pk[PART / 2];
        if (n > 0) {
          if constexpr (PART == 32) tmem_ld32(lane_addr + COL_O + c0, ov);
          else tmem_ld16(lane_addr + COL_O + c0, ov);
          tmem_wait_ld();
        }
#pragma unroll
        for (int x = 0; x < PART; x += 2) {
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
  if (tid == 0 && p.redo_out) p.redo_out[blockIdx.y * gridDim.x + blockIdx.x] = s_ovf | (pro.left != 0);
  if (abort_flag)
    for (int i = 0; i < 200; i++) __nanosleep(1000);
  if (warp == 0) tmem_dealloc(tmem, TMEM_COLS);
}

}  // namespace ftk
