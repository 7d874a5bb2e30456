// Sparse-attention backward for sm_100a: delta, dQ and dK/dV.
//
// Replaces preprocess_delta (flash_topk_attn_v2/sparse_attn_bwd.py:12-33),
// sparse_attn_bwd_dq_kernel (csrc/sparse_attn_bwd_dq_kernel.cu:6-419) and
// sparse_attn_bwd_dkv_sorted_kernel (csrc/sparse_attn_bwd_dkv_kernel.cu:6-435).
//
// Both kernels use the 128-row union tiles of attn_common.cuh and the same
// three roles as the forward: TMA producer warp, UMMA issuer warp, and 16
// compute warps in two groups (one per S / dP buffer); inside a group two
// warps share each TMEM lane quarter and take half of a tile's columns each.
// With P = 2^(c S - lse2):
//   dQ  kernel, per candidate KV block:  S = Q K^T, dP = dO V^T  (Q, dO in TMEM),
//        dS = P (dP - delta) rounded to the I/O dtype in TMEM, dQ += dS K
//        (A from TMEM, K read MN-major from the tile that fed S).
//   dKV kernel, per q-block of the reverse list: S^T = K Q^T, dP^T = V dO^T,
//        P^T and dS^T written over the S^T / dP^T columns they came from,
//        dV += P^T dO, dK += dS^T Q (dO, Q read MN-major).  One CTA owns its
//        128 kv rows, so dK/dV need no atomics.
#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "attn_common.cuh"
#include "attn_host.cuh"
#include "ftk_host.cuh"
#include "ftk_sm100.cuh"

namespace ftk {

constexpr int BW_THREADS = 576;  // 2 + 2 x 8 warps
constexpr int BW_MAX_STAGES = 4;
// A one-CTA kernel with ng groups of 8 warps; with one group two CTAs share an SM.
__host__ __device__ constexpr int bw_threads(int ng) { return 64 + 256 * ng; }
// dQ kernel: K tiles in the ring (held until dQ += dS K ran), V tiles (free once dP is computed)
__host__ __device__ constexpr int dq_kst(int ng) { return ng == 1 ? 6 : 7; }
constexpr int DQ_VST = 5;

struct BwdParams {
  int N, H, D, QM, W, Mkv;
  int g, kvb, q_pad_head, kv_pad_head;   // rows per group and per tile (sub * listed block)
  int G, fmt, nstages;
  float scale, scale_log2;
  const int32_t* lists;      // dQ: [BH][list_rows][W]; dKV: reverse_idx [BH][Mkv][QM] or null
  int list_rows;
  ListMap lm;
  const int32_t* counts;     // dKV with `lists`: reverse_counts [BH][Mkv]
  uint8_t* masks;            // [BH][mask_tiles][mask_stride]: dQ writes (when given), dKV reads
  int mask_stride, mask_tiles, mask_g;
  const float* lse;
  float* delta;              // [BH][N]: dQ writes, dKV reads
  const uint8_t* o;          // dQ: forward result and its gradient, for delta
  const uint8_t* dout;
  int64_t so_b, so_n, so_h, sd_b, sd_n, sd_h;
  void* out0;                // dQ kernel: dq ; dKV kernel: dk
  void* out1;                //                  dKV kernel: dv
  int64_t s0_b, s0_n, s0_h, s1_b, s1_n, s1_h;
  int out_f32;               // o, dq, dk, dv are float32
  int* status;
  int kv_hdiv;               // query heads per kv head (grouped-query attention), 1 otherwise
  int heads;                 // dKV: query heads one CTA walks (kv_hdiv, or 1: one result per query head)
  int span, span_tiles;      // dKV with heads > 1: q-blocks (a multiple of 32) and tiles per head
  int sub;                   // listed blocks per tile: kv blocks (dQ), q-blocks (dKV)
  const int32_t* order;      // dKV: kv blocks by fan-in, heaviest first ([BH][Mkv]) or null
  const int32_t* tile_order; // dKV: the CTAs' (pairs') tiles by number of q-blocks, heaviest first, or null
  const int32_t* pick;       // dKV: per slice, 1: the pair kernel does it, 0: the one-CTA kernel; or null
};

// ------------------------------------------------------------------- delta
// delta[row] = sum_d o * do for the 128 rows of a dQ tile, by the compute warps of the
// CTA (the others load and issue meanwhile), into shared memory (for the tile itself) and
// global memory (for dK/dV).
// kd / 8 lanes per row, each with one 16-byte load per tensor, so a warp covers
// 256 / kd rows at once and a thread has all of its loads in flight together.
// As a kernel of its own this cost a launch and 258 us at N = 32768, H = 32,
// D = 128 (122 us at B = 4, N = 8192, H = 16), reading O and dO at 4.2 TB/s;
// here the reads hide behind the other CTAs' UMMAs.
// Loaded and summed once Q and dO are on their way into TMEM, under the first UMMAs.  Issued
// before the union is built the loads stand in front of those of the lists, which the union waits
// for (6000 cycles of a CTA instead of 2900), and hold registers across it: lists of 16 of 64
// blocks, B = 2, N = 4096, H = 32 580 against 565 kilocycles, of 8 419 against 402.
template <int KD, int WARPS = 16>
struct TileDelta {
  static constexpr int LPR = KD / 8, RPW = 32 / LPR;
  static constexpr int STEPS = (128 + RPW * WARPS - 1) / (RPW * WARPS);
  uint4 vd[STEPS], vo[STEPS];   // vo of a float32 O: the first 4 of a lane's 8 columns

  __device__ __forceinline__ int row(int i) const {
    return (i * WARPS + (threadIdx.x >> 5) - 2) * RPW + (threadIdx.x & 31) / LPR;
  }
  __device__ __forceinline__ bool inside(const BwdParams& p, int r, int n, int rows) const {
    return r < rows && n >= 0 && n < p.N && (threadIdx.x & 31) % LPR * 8 < p.D;
  }
  __device__ __forceinline__ void load(const BwdParams& p, int b, int h, int tile_row0, int rows) {
    const int c = (threadIdx.x & 31) % LPR;
    const int64_t ob = static_cast<int64_t>(b) * p.so_b + static_cast<int64_t>(h) * p.so_h,
                  db = static_cast<int64_t>(b) * p.sd_b + static_cast<int64_t>(h) * p.sd_h;
#pragma unroll
    for (int i = 0; i < STEPS; i++) {
      const int r = row(i), n = tile_row0 + r;
      vd[i] = vo[i] = make_uint4(0u, 0u, 0u, 0u);
      if (!inside(p, r, n, rows)) continue;
      vd[i] = reinterpret_cast<const uint4*>(p.dout + 2 * (db + static_cast<int64_t>(n) * p.sd_n))[c];
      const int64_t oe = ob + static_cast<int64_t>(n) * p.so_n;
      vo[i] = p.out_f32 ? reinterpret_cast<const uint4*>(p.o + 4 * oe)[2 * c]
                        : reinterpret_cast<const uint4*>(p.o + 2 * oe)[c];
    }
  }
  __device__ __forceinline__ void finish(const BwdParams& p, float* s_delta, int bh, int b, int h,
                                         int tile_row0, int rows) {
    const int c = (threadIdx.x & 31) % LPR;
    float acc[STEPS];
#pragma unroll
    for (int i = 0; i < STEPS; i++) {
      const int r = row(i), n = tile_row0 + r;
      const uint32_t wd[4] = {vd[i].x, vd[i].y, vd[i].z, vd[i].w};
      float2 fo[4];
      if (p.out_f32) {
        // The second half lies in the sectors that `load` has fetched.  Loaded there as well
        // it would hold registers in 16-bit calls too.
        uint4 hi = make_uint4(0u, 0u, 0u, 0u);
        if (inside(p, r, n, rows)) {
          const int64_t oe = static_cast<int64_t>(b) * p.so_b + static_cast<int64_t>(h) * p.so_h +
                             static_cast<int64_t>(n) * p.so_n;
          hi = reinterpret_cast<const uint4*>(p.o + 4 * oe)[2 * c + 1];
        }
        fo[0] = make_float2(__uint_as_float(vo[i].x), __uint_as_float(vo[i].y));
        fo[1] = make_float2(__uint_as_float(vo[i].z), __uint_as_float(vo[i].w));
        fo[2] = make_float2(__uint_as_float(hi.x), __uint_as_float(hi.y));
        fo[3] = make_float2(__uint_as_float(hi.z), __uint_as_float(hi.w));
      } else {
        fo[0] = unpack2(vo[i].x, p.fmt);
        fo[1] = unpack2(vo[i].y, p.fmt);
        fo[2] = unpack2(vo[i].z, p.fmt);
        fo[3] = unpack2(vo[i].w, p.fmt);
      }
      acc[i] = 0.f;
#pragma unroll
      for (int x = 0; x < 4; x++) {
        const float2 gd = unpack2(wd[x], p.fmt);
        acc[i] = fmaf(fo[x].x, gd.x, acc[i]);
        acc[i] = fmaf(fo[x].y, gd.y, acc[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < STEPS; i++) {
      const int r = row(i), n = tile_row0 + r;
#pragma unroll
      for (int d = LPR >> 1; d > 0; d >>= 1) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], d);
      if (c == 0 && r < 128) {
        s_delta[r] = acc[i];
        if (inside(p, r, n, rows)) p.delta[static_cast<int64_t>(bh) * p.N + n] = acc[i];
      }
    }
  }
};

// dS = 2^(c s - lse2) (dp - delta) for 32 columns of one row, two columns per
// instruction (fma.f32x2, add.f32x2, mul.f32x2, one cvt per pair).
template <int FMT>
__device__ __forceinline__ void ds_pairs(const uint32_t (&sv)[32], const uint32_t (&dv)[32],
                                         uint32_t (&pk)[16], float c, float neg_lse2,
                                         float neg_delta) {
  const float2 c2 = make_float2(c, c), nl = make_float2(neg_lse2, neg_lse2),
               nd = make_float2(neg_delta, neg_delta);
#pragma unroll
  for (int x = 0; x < 32; x += 2) {
    const float2 t =
        __ffma2_rn(make_float2(__uint_as_float(sv[x]), __uint_as_float(sv[x + 1])), c2, nl);
    const float2 pr = make_float2(fast_exp2(t.x), fast_exp2(t.y));
    const float2 dd =
        __fadd2_rn(make_float2(__uint_as_float(dv[x]), __uint_as_float(dv[x + 1])), nd);
    const float2 ds = __fmul2_rn(pr, dd);
    if (FMT == 1) {
      __nv_bfloat162 v = __floats2bfloat162_rn(ds.x, ds.y);
      pk[x >> 1] = *reinterpret_cast<uint32_t*>(&v);
    } else {
      __half2 v = __floats2half2_rn(ds.x, ds.y);
      pk[x >> 1] = *reinterpret_cast<uint32_t*>(&v);
    }
  }
}

// P^T = 2^(c s - lse2) and dS^T = P^T (dp - delta) for 16 columns (= q rows) of
// one kv row, two columns per instruction; lse2 / delta of the columns come
// NEGATED from shared memory, one 16-byte broadcast load per four columns.
template <int FMT>
__device__ __forceinline__ void pt_pairs(const uint32_t (&sv)[16], const uint32_t (&dv)[16],
                                         const float4* nl4, const float4* nd4, float c,
                                         uint32_t (&pp)[8], uint32_t (&pd)[8]) {
  const float2 c2 = make_float2(c, c);
#pragma unroll
  for (int x = 0; x < 16; x += 4) {
    const float4 lq = nl4[x >> 2];
    const float4 dq = nd4[x >> 2];
#pragma unroll
    for (int y = 0; y < 4; y += 2) {
      const float2 nl = y == 0 ? make_float2(lq.x, lq.y) : make_float2(lq.z, lq.w);
      const float2 nd = y == 0 ? make_float2(dq.x, dq.y) : make_float2(dq.z, dq.w);
      const float2 t = __ffma2_rn(
          make_float2(__uint_as_float(sv[x + y]), __uint_as_float(sv[x + y + 1])), c2, nl);
      const float2 pr = make_float2(fast_exp2(t.x), fast_exp2(t.y));
      const float2 dd = __fadd2_rn(
          make_float2(__uint_as_float(dv[x + y]), __uint_as_float(dv[x + y + 1])), nd);
      const float2 ds = __fmul2_rn(pr, dd);
      if (FMT == 1) {
        __nv_bfloat162 a = __floats2bfloat162_rn(pr.x, pr.y), b = __floats2bfloat162_rn(ds.x, ds.y);
        pp[(x + y) >> 1] = *reinterpret_cast<uint32_t*>(&a);
        pd[(x + y) >> 1] = *reinterpret_cast<uint32_t*>(&b);
      } else {
        __half2 a = __floats2half2_rn(pr.x, pr.y), b = __floats2half2_rn(ds.x, ds.y);
        pp[(x + y) >> 1] = *reinterpret_cast<uint32_t*>(&a);
        pd[(x + y) >> 1] = *reinterpret_cast<uint32_t*>(&b);
      }
    }
  }
}

// The same where only columns lo .. hi - 1 are the row's.  A function: as a lambda of two callers
// it was not inlined well.  The exponential's argument is selected, not the exponential, which
// became a branch per value.  dK/dV of 4096 tokens, H = 16, blocks of 48, half of them listed: head
// dim 64 402 us, 264 like this, head dim 128 (with the early end of dP^T below) 680, 313.
__device__ __forceinline__ void pt_masked(const uint32_t (&sv)[16], const uint32_t (&dv)[16],
                                          const float4* nl4, const float4* nd4, float c, int lo, int hi,
                                          int fmt, uint32_t (&pp)[8], uint32_t (&pd)[8]) {
#pragma unroll
  for (int x = 0; x < 16; x += 4) {
    const float4 lq = nl4[x >> 2];
    const float4 dq = nd4[x >> 2];
    const float ls[4] = {lq.x, lq.y, lq.z, lq.w};
    const float ds[4] = {dq.x, dq.y, dq.z, dq.w};
    float pv[4], dsv[4];
#pragma unroll
    for (int y = 0; y < 4; y++) {
      const bool on = x + y >= lo && x + y < hi;
      const float pr = fast_exp2(on ? fmaf(__uint_as_float(sv[x + y]), c, ls[y]) : -INFINITY);
      pv[y] = pr;
      dsv[y] = pr * (__uint_as_float(dv[x + y]) + ds[y]);
    }
    pp[x >> 1] = pack2(pv[0], pv[1], fmt);
    pp[(x >> 1) + 1] = pack2(pv[2], pv[3], fmt);
    pd[x >> 1] = pack2(dsv[0], dsv[1], fmt);
    pd[(x >> 1) + 1] = pack2(dsv[2], dsv[3], fmt);
  }
}

// ---------------------------------------------------------------------- dQ
// TMEM columns: Q and dO, D / 2 each (16-bit pairs: the A operands of the
// S and dP UMMAs are read from TMEM, which leaves shared-memory bandwidth to
// the K/V tiles), S[NG] and dP[NG], 64 each (dS written over the first half of
// dP), dQ.
// Shared memory: the Q and dO tiles are dead once they sit in TMEM, so their
// 2 x 128 rows become four slots of the V ring (the fifth follows the K ring);
// K has its own ring.  K and V travel in
// separate rings because V is released after dP while K stays until dQ: the
// producer runs several tiles ahead, which is what lets the loads overlap the
// UMMAs instead of alternating with them.
// Both loads of a tile signal the K slot's barrier, so that the issuing warp has two
// waits per tile, not three (511 -> 503 us at head dim 64, N = 8192, H = 16; 377 -> 372
// with lists of 16 blocks at head dim 128, B = 2, N = 4096, H = 32).
// One group of warps (head dim 64): one S and one dP buffer, 256 TMEM columns, two CTAs
// per SM.  See one_group for when.
template <int D, int NG>
__global__ void __launch_bounds__(bw_threads(NG), 2 / NG)
sparse_bwd_dq_kernel(const __grid_constant__ CUtensorMap tm_q,
                     const __grid_constant__ CUtensorMap tm_do,
                     const __grid_constant__ CUtensorMap tm_k,
                     const __grid_constant__ CUtensorMap tm_v, const BwdParams p) {
  constexpr int NCH = D / 64;
  constexpr int ROW_TILE_BYTES = NCH * 128 * 128;
  // Head dim 256: Q and dO (128 TMEM columns each) no longer fit next to S, dP
  // and a 256-column dQ, so they stay in shared memory as SS operands; the
  // rings shrink to three K and two V tiles of at most 32 rows, all behind
  // the Q / dO tiles.  TMEM: S[2] 0/64, dP[2] 128/192, dQ 256..511.
  constexpr bool BIG = D > 128;
  constexpr int DQ_KST = dq_kst(NG);
  constexpr int KST = BIG ? 3 : DQ_KST, VST = BIG ? 2 : DQ_VST;
  constexpr uint32_t COL_S = BIG ? 0 : D, COL_DP = COL_S + 64 * NG, COL_DQ = COL_DP + 64 * NG;
  constexpr uint32_t TMEM_COLS = 256 * NG;
  static_assert(COL_DQ + D <= TMEM_COLS, "TMEM columns");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem;
  uint8_t* sDO = smem + ROW_TILE_BYTES;
  uint8_t* sV = smem;                          // over Q / dO once they are in TMEM
  uint8_t* sK = smem + 2 * ROW_TILE_BYTES;
  __shared__ UnionScratch un;
  __shared__ float s_delta[128];
  __shared__ OutTile s_out;
  __shared__ __align__(8) uint64_t bars[1 + 2 * DQ_KST + DQ_VST + 2 * NG + 2];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_flag;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.x * p.G;
  const int bh = blockIdx.y;
  const int b_idx = bh / p.H, h_idx = bh - b_idx * p.H;
  const int groups = min(p.G, p.QM - m0);
  const int tile_row0 = m0 * p.g - p.q_pad_head;
  const int kv_chunk_bytes = p.kvb * 128;
  const int tile_bytes = NCH * kv_chunk_bytes;   // one K or V tile
  auto v_slot = [&](int sv) {
    if (BIG) return smem_u32(sK) + (KST + sv) * tile_bytes;
    return sv < 4 ? smem_u32(sV) + sv * tile_bytes
                  : smem_u32(sK) + (DQ_KST + sv - 4) * tile_bytes;
  };

  const uint32_t bar_q = smem_u32(&bars[0]);
  auto bar_full = [&](int s) { return smem_u32(&bars[1 + s]); };   // of the K slot: K and V
  auto bar_kempty = [&](int s) { return smem_u32(&bars[1 + DQ_KST + s]); };
  auto bar_vempty = [&](int s) { return smem_u32(&bars[1 + 2 * DQ_KST + s]); };
  constexpr int BAR_A0 = 1 + 2 * DQ_KST + DQ_VST;
  auto bar_afull = [&](int s) { return smem_u32(&bars[BAR_A0 + s]); };
  auto bar_dsfull = [&](int s) { return smem_u32(&bars[BAR_A0 + NG + s]); };
  // arrives once, after the last UMMA of the CTA has retired
  const uint32_t bar_final = smem_u32(&bars[BAR_A0 + 2 * NG]);
  // Q and dO copied from shared memory into TMEM by the compute warps
  const uint32_t bar_qt = smem_u32(&bars[BAR_A0 + 2 * NG + 1]);

  if (tid == 0) {
    abort_flag = 0;
    mbar_init(bar_q, 1);
    for (int s = 0; s < DQ_KST; s++) {
      mbar_init(bar_full(s), 1);
      mbar_init(bar_kempty(s), 1);
    }
    for (int s = 0; s < DQ_VST; s++) {
      mbar_init(bar_vempty(s), 1);
    }
    for (int s = 0; s < NG; s++) {
      mbar_init(bar_afull(s), 1);
      mbar_init(bar_dsfull(s), 8);  // one arrival per warp of the owning group
    }
    mbar_init(bar_final, 1);
    mbar_init(bar_qt, 8);   // the 8 warps that copy Q / dO
    mbar_init_fence();
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_do);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(&tmem_base_s), TMEM_COLS);
    tmem_relinquish();
  }
  if (tid == 32)
    s_out = {{static_cast<int64_t>(b_idx) * p.s0_b + static_cast<int64_t>(h_idx) * p.s0_h, 0},
             tile_row0, min(p.N, tile_row0 + groups * p.g)};
  clear_flags(sK, p.Mkv, groups);
  tc_fence_before();
  pdl_wait();
  if (tid == 0) {   // under the building of the union
    mbar_expect_tx(bar_q, 2 * ROW_TILE_BYTES);
    for (int c = 0; c < NCH; c++) {
      tma_load_4d(smem_u32(sQ) + c * 128 * 128, &tm_q, bar_q, c * 64, h_idx, tile_row0, b_idx);
      tma_load_4d(smem_u32(sDO) + c * 128 * 128, &tm_do, bar_q, c * 64, h_idx, tile_row0, b_idx);
    }
  }
  TileDelta<D, 8 * NG> delta;
  float lse_mine = 0.f;   // of the row that a compute thread works on
  if (warp >= 2) {
    const int r = (warp & 3) * 32 + lane, qrow = tile_row0 + r;
    if (r < groups * p.g && qrow >= 0 && qrow < p.N) lse_mine = p.lse[static_cast<int64_t>(bh) * p.N + qrow];
  }
  const TileMaskRow mask_row = {
      p.masks ? p.masks + (static_cast<int64_t>(bh) * p.mask_tiles + blockIdx.x) * p.mask_stride : nullptr,
      0, groups};
  const int n = build_union<bw_threads(NG) / 32>(
      un, sK, p.lists + static_cast<int64_t>(bh) * p.list_rows * p.W, m0, groups, p.W, nullptr, p.Mkv,
      p.sub, p.lm, p.status, mask_row);
  pdl_launch();
  tc_fence_after();
  const uint32_t tmem = NG == 2 ? tmem_base_s : __shfl_sync(0xffffffffu, tmem_base_s, 0);
  WaitCtx w{&abort_flag, p.status};
  const bool split = (p.kvb % 32) == 0;   // kv columns of a tile shared by two warps per row

  if (warp == 0) {
    if (lane == 0 && n == 0) mbar_wait(bar_q, 0, w, FTK_DEV_TIMEOUT_TMA);   // lands before the exit
    if (lane == 0 && n > 0) {
      const int hk = h_idx / p.kv_hdiv;   // out of the loop: a division takes 150 cycles
      for (int i = 0; i < n; i++) {
        const int sk = i % KST, sv = i % VST;
        const int tok0 = static_cast<int>(un.ids[i]) * p.kvb - p.kv_pad_head;
        if (!mbar_wait(bar_kempty(sk), ((i / KST) & 1) ^ 1, w, FTK_DEV_TIMEOUT_TMA)) break;
        const uint32_t kb = smem_u32(sK) + sk * tile_bytes;
        mbar_expect_tx(bar_full(sk), 2 * tile_bytes);
        for (int c = 0; c < NCH; c++)
          tma_load_4d(kb + c * kv_chunk_bytes, &tm_k, bar_full(sk), c * 64, hk,
                      tok0, b_idx);
        // the V ring lies over the Q / dO tiles: wait until they sit in TMEM
        if (!BIG && i == 0 && !mbar_wait(bar_qt, 0, w, FTK_DEV_TIMEOUT_TMA)) break;
        if (!mbar_wait(bar_vempty(sv), ((i / VST) & 1) ^ 1, w, FTK_DEV_TIMEOUT_TMA)) break;
        const uint32_t vb = v_slot(sv);
        for (int c = 0; c < NCH; c++)
          tma_load_4d(vb + c * kv_chunk_bytes, &tm_v, bar_full(sk), c * 64, hk,
                      tok0, b_idx);
      }
    }
  } else if (warp == 1) {
    if (n > 0) {
      // the whole warp runs this path; one elected lane issues the UMMAs
      const uint32_t idesc_a = umma_idesc(128, p.kvb, p.fmt, 0, 0);
      const uint32_t idesc_b = umma_idesc(128, D, p.fmt, 0, 1);
      const uint64_t kdesc0 = smem_desc_sw128(smem_u32(sK), 16, 1024);
      const uint64_t kmn0 = smem_desc_sw128(smem_u32(sK), kv_chunk_bytes, 1024);
      // dS column of k-step ks: each half of the kv columns is written by its
      // own warps over the dP columns those warps read (see the compute part)
      // (kh is 1 or 2: shifts and masks only, the single issuing thread must
      // not spend longer between two UMMAs than the tensor core needs for one)
      const int kh = p.kvb / 32, kh_shift = kh >> 1, half_cols = p.kvb / 2;
      auto ds_col = [&](int ks) {
        return split ? (ks >> kh_shift) * half_cols + (ks & (kh - 1)) * 8 : ks * 8;
      };
      const uint64_t qdesc0 = smem_desc_sw128(smem_u32(sQ), 16, 1024);
      const uint64_t dodesc0 = smem_desc_sw128(smem_u32(sDO), 16, 1024);
      const uint32_t el = elect_one();
      bool ok = warp_all(mbar_wait(BIG ? bar_q : bar_qt, 0, w, FTK_DEV_TIMEOUT_MMA));
      tc_fence_after();
      // The tensor core runs dry whenever the issuing thread waits, so every
      // barrier of a round is waited for first and the round's UMMAs (dQ of
      // tile i, then S and dP of tile i + NG) go out as one uninterrupted batch.
      auto wait_kv = [&](int i) -> bool {
        return warp_all(mbar_wait(bar_full(i % KST), (i / KST) & 1, w, FTK_DEV_TIMEOUT_MMA));
      };
      auto mma_a = [&](int i) {   // elected lane only
        const int sk = i % KST, sv = i % VST;
        const uint64_t kdesc = desc_advance(kdesc0, sk * tile_bytes);
        const uint64_t vdesc = smem_desc_sw128(v_slot(sv), 16, 1024);
        const uint32_t sb = i % NG;
#pragma unroll
        for (int ks = 0; ks < D / 16; ks++) {
          const uint32_t koff = (ks / 4) * kv_chunk_bytes + (ks % 4) * 32;
          if (BIG)
            umma_ss(tmem + COL_S + sb * 64,
                    desc_advance(qdesc0, (ks / 4) * 128 * 128 + (ks % 4) * 32),
                    desc_advance(kdesc, koff), idesc_a, ks > 0, el);
          else
            umma_ts(tmem + COL_S + sb * 64, tmem + ks * 8, desc_advance(kdesc, koff), idesc_a,
                    ks > 0, el);
        }
#pragma unroll
        for (int ks = 0; ks < D / 16; ks++) {
          const uint32_t koff = (ks / 4) * kv_chunk_bytes + (ks % 4) * 32;
          if (BIG)
            umma_ss(tmem + COL_DP + sb * 64,
                    desc_advance(dodesc0, (ks / 4) * 128 * 128 + (ks % 4) * 32),
                    desc_advance(vdesc, koff), idesc_a, ks > 0, el);
          else
            umma_ts(tmem + COL_DP + sb * 64, tmem + D / 2 + ks * 8, desc_advance(vdesc, koff), idesc_a,
                    ks > 0, el);
        }
        umma_commit(bar_afull(sb), el);
        umma_commit(bar_vempty(sv), el);
      };
      auto mma_b = [&](int i) {   // elected lane only
        const int s = i % KST, sb = i % NG;
        const uint64_t kmn = desc_advance(kmn0, s * tile_bytes);
        if (p.kvb == 64) {
#pragma unroll
          for (int ks = 0; ks < 4; ks++)
            umma_ts(tmem + COL_DQ, tmem + COL_DP + sb * 64 + (ks >> 1) * 32 + (ks & 1) * 8,
                    desc_advance(kmn, ks * 2048), idesc_b, (i > 0) || (ks > 0), el);
        } else {
          for (int ks = 0; ks < p.kvb / 16; ks++)
            umma_ts(tmem + COL_DQ, tmem + COL_DP + sb * 64 + ds_col(ks), desc_advance(kmn, ks * 2048),
                    idesc_b, (i > 0) || (ks > 0), el);
        }
        umma_commit(bar_kempty(s), el);
      };
      if (ok) ok = wait_kv(0);
      if (ok && NG > 1 && n > 1) ok = wait_kv(1);
      tc_fence_after();
      if (ok) {
        mma_a(0);
        if (NG > 1 && n > 1) mma_a(1);
      }
      __syncwarp();
      for (int i = 0; ok && i < n; i++) {
        const bool more = i + NG < n;
        const int i2 = more ? i + NG : i;   // last rounds: the dS barrier stands in
        const uint32_t wb[2] = {bar_dsfull(i % NG), more ? bar_full(i2 % KST) : bar_dsfull(i % NG)};
        const uint32_t wp[2] = {static_cast<uint32_t>((i / NG) & 1),
                                static_cast<uint32_t>(more ? (i2 / KST) & 1 : (i / NG) & 1)};
        if (!warp_all(mbar_wait_all<2>(wb, wp, w, FTK_DEV_TIMEOUT_MMA))) break;
        tc_fence_after();
        mma_b(i);
        if (i + NG < n) mma_a(i + NG);
        __syncwarp();
      }
      if (ok) umma_commit(bar_final, el);
      __syncwarp();
    }
  } else {
    // NG groups of 8 warps; group w drains the buffers of tiles i = w (mod NG).
    // Inside a group two warps share each 32-row lane quarter and take one
    // half of the kv columns each, so a tile's latency-bound per-thread work
    // is 32 columns long and 4 compute warps per scheduler hide each other.
    const int cw = warp - 2;
    const int wg = cw >> 3;
    const int colhalf = (cw >> 2) & 1;
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const int grp = r / p.g;
    const int qrow = tile_row0 + r;
    const bool row_valid = (grp < groups) && qrow >= 0 && qrow < p.N;
    const uint32_t lane_addr = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t s_addr = lane_addr + COL_S + wg * 64;
    const uint32_t dp_addr = lane_addr + COL_DP + wg * 64;
    const int cbeg = split ? colhalf * (p.kvb / 2) : 0;
    const int cend = split ? cbeg + p.kvb / 2 : (colhalf == 0 ? p.kvb : 0);
    const float c = p.scale_log2;
    const float lse2 = lse_mine * 1.4426950408889634f;
    bool ok = true;
    const int copies = NG == 2 ? wg : colhalf;   // Q or dO
    if (!BIG && n > 0 && (NG == 1 || colhalf == 0)) {
      // group 0 moves the Q tile, group 1 the dO tile, from (swizzled) shared
      // memory into TMEM: row r -> lane r, two 16-bit values per column
      ok = mbar_wait(bar_q, 0, w, FTK_DEV_TIMEOUT_CONSUMER);
      if (ok) {
        const uint8_t* src = copies == 0 ? sQ : sDO;
#pragma unroll
        for (int ch = 0; ch < NCH; ch++) {
          uint32_t v[32];
#pragma unroll
          for (int j = 0; j < 8; j++) {
            const uint4 t4 = *reinterpret_cast<const uint4*>(src + ch * 128 * 128 +
                                                             sw128_offset(r, j));
            v[j * 4 + 0] = t4.x;
            v[j * 4 + 1] = t4.y;
            v[j * 4 + 2] = t4.z;
            v[j * 4 + 3] = t4.w;
          }
          tmem_st32(lane_addr + copies * (D / 2) + ch * 32, v);
        }
        tmem_wait_st();
        tc_fence_before();
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_qt);
    }
    // the sums run under the first UMMAs
    delta.load(p, b_idx, h_idx, tile_row0, groups * p.g);
    delta.finish(p, s_delta, bh, b_idx, h_idx, tile_row0, groups * p.g);
    asm volatile("bar.sync 1, %0;" ::"n"(256 * NG) : "memory");
    const float dl = row_valid ? s_delta[r] : 0.f;
    for (int i = wg; ok && i < n; i += NG) {
      // A(i) complete also means B(i - NG) has retired (same issue order), so the
      // dS columns of this buffer are free again.
      // what the tile's columns mean to this row: worked out before the wait
      const int tok0 = static_cast<int>(un.ids[i]) * p.kvb - p.kv_pad_head;
      const ColSpan cs = col_span(un, i, p.sub, grp, tok0, p.kvb, p.N);
      const int lo = cs.lo, hi = cs.hi;
      const bool act = cs.on;
      // all of this warp's columns, or none of them (of two listed blocks walked as one tile
      // each half of the warps has one)
      const bool fast = __all_sync(0xffffffffu, act && lo <= cbeg && hi >= cend);
      const bool none = !fast && !__any_sync(0xffffffffu, act && lo < cend && hi > cbeg);
      if (!mbar_wait(bar_afull(wg), (i / NG) & 1, w, FTK_DEV_TIMEOUT_CONSUMER)) {
        ok = false;
        break;
      }
      tc_fence_after();
      // dS of columns [c0, c0+w) is written over dP columns [cbeg + (c0-cbeg)/2, ..):
      // columns this thread has already read, never another warp's
      for (int c0 = cbeg; c0 < cend; c0 += 32) {
        const uint32_t ds_addr = dp_addr + cbeg + ((c0 - cbeg) >> 1);
        if (cend - c0 >= 32) {
          uint32_t sv[32], dv[32], pk[16];
          if (none) {   // the other group's block: dS = 0, nothing to read
#pragma unroll
            for (int x = 0; x < 16; x++) pk[x] = 0u;
            tmem_st16(ds_addr, pk);
            continue;
          }
          tmem_ld32(s_addr + c0, sv);
          tmem_ld32(dp_addr + c0, dv);
          tmem_wait_ld();
          if (fast) {
            if (p.fmt == 1) ds_pairs<1>(sv, dv, pk, c, -lse2, -dl);
            else ds_pairs<0>(sv, dv, pk, c, -lse2, -dl);
          } else {
#pragma unroll
            for (int x = 0; x < 32; x += 2) {
              float d0 = 0.f, d1 = 0.f;
              if (act && c0 + x >= lo && c0 + x < hi)
                d0 = fast_exp2(fmaf(__uint_as_float(sv[x]), c, -lse2)) *
                     (__uint_as_float(dv[x]) - dl);
              if (act && c0 + x + 1 >= lo && c0 + x + 1 < hi)
                d1 = fast_exp2(fmaf(__uint_as_float(sv[x + 1]), c, -lse2)) *
                     (__uint_as_float(dv[x + 1]) - dl);
              pk[x >> 1] = pack2(d0, d1, p.fmt);
            }
          }
          tmem_st16(ds_addr, pk);
        } else {
          uint32_t sv[16], dv[16], pk[8];
          tmem_ld16(s_addr + c0, sv);
          tmem_ld16(dp_addr + c0, dv);
          tmem_wait_ld();
#pragma unroll
          for (int x = 0; x < 16; x += 2) {
            float d0 = 0.f, d1 = 0.f;
            if (act && c0 + x >= lo && c0 + x < hi)
              d0 = fast_exp2(fmaf(__uint_as_float(sv[x]), c, -lse2)) *
                   (__uint_as_float(dv[x]) - dl);
            if (act && c0 + x + 1 >= lo && c0 + x + 1 < hi)
              d1 = fast_exp2(fmaf(__uint_as_float(sv[x + 1]), c, -lse2)) *
                   (__uint_as_float(dv[x + 1]) - dl);
            pk[x >> 1] = pack2(d0, d1, p.fmt);
          }
          tmem_st8(ds_addr, pk);
        }
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_dsfull(wg));
    }
    // epilogue: each group converts and stores one half of the head dimension
    if (ok) ok = mbar_wait(n > 0 ? bar_final : bar_q, 0, w, FTK_DEV_TIMEOUT_EPILOGUE);
    if (ok) {
      tc_fence_after();
      // every copy has landed and every UMMA has retired: the tiles make room for dQ
      const int ew = (late_tid() >> 5) - 2;   // 32-column chunks dealt to the warps of a lane quarter
      // 32-column chunks of the head dim are dealt round-robin to the four
      // warps of a lane quarter
#pragma unroll 1
      for (int c0 = (ew >> 2) * 32; c0 < D; c0 += 128) {
        uint32_t v[32];
        if (n > 0) {
          tmem_ld32(lane_addr + COL_DQ + c0, v);
          tmem_wait_ld();
        }
        uint32_t pk[16];
#pragma unroll
        for (int x = 0; x < 32; x += 2) {
          const float a = n > 0 ? __uint_as_float(v[x]) * p.scale : 0.f;
          const float b = n > 0 ? __uint_as_float(v[x + 1]) * p.scale : 0.f;
          pk[x >> 1] = pack2(a, b, p.fmt);
        }
        store_rows(smem + ew * 2048, pk, p.out0, s_out, 0, (ew + 2) & 3, p.s0_n, c0, p.D, p.fmt,
                 p.out_f32 != 0);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (abort_flag)
    for (int i = 0; i < 200; i++) __nanosleep(1000);
  if (warp == 0) tmem_dealloc(tmem, TMEM_COLS);
}

// -------------------------------------------------------------------- dK/dV
// Union of the lists of kv blocks j0 .. j0 + groups - 1 (`per` of them where the grid
// does not end), from the dQ kernel's tile masks or from a reverse index.  The caller has
// called pdl_wait.
__device__ __forceinline__ int dkv_union(UnionScratch& un, uint8_t* flags, const BwdParams& p, int bhq,
                                         int j0, int groups, int per) {
  int n;
  if (p.masks) {
    const int64_t per_head = static_cast<int64_t>(p.mask_tiles) * p.mask_stride;
    n = build_union_masks<BW_THREADS / 32>(un, p.masks + bhq * per_head, p.mask_stride, p.mask_tiles,
                                           p.mask_g, j0, per, p.heads, per_head, p.span, p.sub);
  } else {
    const int64_t kv_row = static_cast<int64_t>(bhq) * p.Mkv + j0;
    clear_flags(flags, p.QM, groups);
    n = build_union<BW_THREADS / 32>(un, flags, p.lists + kv_row * p.QM, 0, groups, p.QM,
                                     p.counts + kv_row, p.QM, p.sub, ListMap{0, 0, 0, 0}, p.status);
  }
  pdl_launch();   // the unions hold the barrier that follows the caller's tmem_alloc
  return n;
}

// Entry id of the union -> q tile, with the query head it belongs to (ids come
// in ascending order, head by head).  Without WALK ids are q-blocks.
template <bool WALK>
struct HeadWalk {
  int head = 0, first = 0;
  __device__ __forceinline__ int at(int id, const BwdParams& p) {
    while (WALK && id - first >= p.span_tiles) {
      first += p.span_tiles;
      head++;
    }
    return id - first;
  }
};

// The slice and the tile of launch position x of `tiles` in row blockIdx.y of the grid.
// With an order (see fan_in_kernel) the heaviest eighth of every slice's tiles comes first,
// those of all slices in turn, then the rest slice by slice, whose rows of Q and dO stay in
// L2 that way: sorted within the slices only, the last slice's heaviest tiles start late.
// Backward passes with none, a sixteenth, an eighth, a quarter, a half and all of them in
// turn, lists with a block that everybody reads: B = 2, N = 4096, H = 32, lists of 16 of 64
// 804, 771, 773, 777, 786, 792 us (four heads per kv head 857, 720, 718, 716, 716, 714);
// N = 16384, H = 8, lists of 32 855, 710, 710, 710, 712, 718; head dim 256, N = 8192,
// H = 16, lists of 24 1618, 1540, 1548, 1550, 1591, 1647, head dim 64 488, 433, 439, 436,
// 441, 419.  With windows or independent lists all are within 2 %.
struct KvTile {
  int slice, tile;
};
__device__ __forceinline__ KvTile kv_tile(const BwdParams& p, int x, int tiles) {
  KvTile t = {static_cast<int>(blockIdx.y), x};
  if (p.tile_order) {
    const int slices = gridDim.y, lead = (tiles + 7) >> 3, at = blockIdx.y * tiles + x;
    int rank;
    if (at < lead * slices) {
      rank = at / slices;
      t.slice = at - rank * slices;
    } else {
      const int rest = at - lead * slices;
      t.slice = rest / (tiles - lead);
      rank = lead + rest - t.slice * (tiles - lead);
    }
    pdl_wait();
    t.tile = p.tile_order[static_cast<int64_t>(t.slice) * tiles + rank];
  }
  return t;
}

// Both kernels are launched where the lists decide which is the faster (see fan_in_kernel);
// the CTAs of the other one leave at once, behind the wait for the decision, which also
// keeps the order of the launches for whoever waits for this one.
__device__ __forceinline__ bool other_kernel(const BwdParams& p, int slice, int mine) {
  if (!p.pick) return false;
  pdl_wait();
  return p.pick[slice] != mine;
}

// TMEM columns: S^T[2] 0/64 (P^T written over their first half), dP^T[2]
// 128/192 (dS^T likewise), dV 256.., dK 384..
// Head dim 128: K (192..255) is copied into TMEM, so that the S^T UMMAs (N = 64) take 42 cycles
// instead of the 75 with both operands in shared memory, 1528 cycles of UMMAs per tile instead of
// 1792, which they were bound by (1815 measured).  Its columns are those of a second dP^T buffer:
// dS^T goes beside P^T, over the S^T that both come from, and the one buffer is the next tile's as
// soon as its columns are in registers.  Between dP^T of two tiles the tensor core has dV and dK
// of the tile before and S^T of the one after, so it does not wait for that.  Kilocycles of a
// launch, before and now: lists of 16 of 64 blocks, B = 2, N = 4096, H = 32 on 8 kv heads 684,
// 612, lists of 128 of 512 at N = 32768, H = 4 2310, 2040.
// Head dim 64: K (320..351) and V (352..383) are copied into TMEM as well, so that the
// S^T and dP^T UMMAs (N = 64) take 42 cycles instead of the 75 that they take with both
// operands in shared memory: 672 cycles of UMMAs per tile instead of 936
// (774 -> 723 us at N = 8192, H = 16).
// MODE 0 (head dims up to 128) produces dV and dK in one launch.  At head dim
// 256 two 256-column accumulators do not fit TMEM next to S^T and dP^T, so the
// work goes in two launches with one accumulator at columns 256..511 each:
// MODE 1 = dV only (needs neither V nor dP^T: K alone stays resident, which
// leaves room for four ring stages), MODE 2 = dK only.
// WALK: see sparse_bwd_dkv2_kernel.
template <int D, int MODE, bool WALK>
__global__ void __launch_bounds__(BW_THREADS, 1)
sparse_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tm_q,
                      const __grid_constant__ CUtensorMap tm_do,
                      const __grid_constant__ CUtensorMap tm_k,
                      const __grid_constant__ CUtensorMap tm_v, const BwdParams p) {
  constexpr int NCH = D / 64;
  constexpr int ROW_TILE_BYTES = NCH * 128 * 128;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sK = smem;
  uint8_t* sV = smem + ROW_TILE_BYTES;
  uint8_t* sQD = smem + (MODE == 1 ? 1 : 2) * ROW_TILE_BYTES;
  constexpr uint32_t COL_DV = 256, COL_DK = MODE == 0 ? 384 : 256;
  constexpr bool K_T = D == 128;                 // K read from TMEM, one dP^T buffer
  constexpr bool ROWS_T = D == 64 || K_T;        // K (head dim 64: and V) read from TMEM
  constexpr uint32_t COL_K = K_T ? 192 : 320, COL_V = 352;
  __shared__ UnionScratch un;
  __shared__ __align__(8) uint64_t bars[1 + 2 * BW_MAX_STAGES + 7];
  __shared__ uint32_t tmem_base_s;
  __shared__ OutTile s_out;
  __shared__ int abort_flag;
  __shared__ __align__(16) float s_lse2[2][2][128], s_delta[2][2][128];  // [group][parity][q row]

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const KvTile at = kv_tile(p, blockIdx.x, gridDim.x);
  const int bh = at.slice;
  if (other_kernel(p, bh, 0)) return;
  int j0 = at.tile * p.G;                   // first kv block of the tile
  if (p.order && !p.tile_order) {
    // The same from a reverse index, which orders kv blocks: the grid has one CTA
    // per kv block, in the order of `order` (fan-in descending, ties by lower id);
    // the CTA whose block is the first of its tile in that order does the tile,
    // the others leave at once.
    pdl_wait();
    const int32_t* cnt = p.counts + static_cast<int64_t>(bh) * p.Mkv;
    const int j = p.order[static_cast<int64_t>(bh) * p.Mkv + blockIdx.x];
    if (j < 0 || j >= p.Mkv) return;
    j0 = (j / p.G) * p.G;
    const int cj = cnt[j];
    for (int jj = j0; jj < min(j0 + p.G, p.Mkv); jj++) {
      const int cc = cnt[jj];
      if (jj != j && (cc > cj || (cc == cj && jj < j))) return;
    }
  }
  // slice = (batch, first of the query heads this CTA walks)
  const int slices = WALK ? p.H / p.heads : p.H;
  const int b_idx = bh / slices, h_idx = (bh - b_idx * slices) * (WALK ? p.heads : 1);
  const int bhq = WALK ? b_idx * p.H + h_idx : bh;
  const int groups = min(p.G, p.Mkv - j0);
  const int tile_tok0 = j0 * p.kvb - p.kv_pad_head;
  const int q_chunk_bytes = p.g * 128;
  const int stage_bytes = 2 * NCH * q_chunk_bytes;
  // Four stages up to head dim 128.  Three divisions per tile by a number that only the
  // launch knew made the issuing warp the bound: 736 -> 675 us at N = 8192, H = 16,
  // head dim 64, all pairs.
  const int NST = D <= 128 ? BW_MAX_STAGES : p.nstages;

  const uint32_t bar_kv = smem_u32(&bars[0]);
  auto bar_qfull = [&](int s) { return smem_u32(&bars[1 + s]); };
  auto bar_qempty = [&](int s) { return smem_u32(&bars[1 + BW_MAX_STAGES + s]); };
  auto bar_afull = [&](int s) { return smem_u32(&bars[1 + 2 * BW_MAX_STAGES + s]); };
  auto bar_pfull = [&](int s) { return smem_u32(&bars[1 + 2 * BW_MAX_STAGES + 2 + s]); };
  // arrives once, after the last UMMA of the CTA has retired
  const uint32_t bar_final = smem_u32(&bars[1 + 2 * BW_MAX_STAGES + 4]);
  const uint32_t bar_kvt = smem_u32(&bars[1 + 2 * BW_MAX_STAGES + 5]);      // rows copied into TMEM
  const uint32_t bar_dpfree = smem_u32(&bars[1 + 2 * BW_MAX_STAGES + 6]);   // K_T: dP^T is in registers

  if (tid == 0) {
    abort_flag = 0;
    mbar_init(bar_kv, 1);
    mbar_init(bar_dpfree, 8);
    for (int s = 0; s < BW_MAX_STAGES; s++) {
      mbar_init(bar_qfull(s), 1);
      mbar_init(bar_qempty(s), 1);
    }
    for (int s = 0; s < 2; s++) {
      mbar_init(bar_afull(s), 1);
      mbar_init(bar_pfull(s), 8);  // one arrival per warp of the owning group
    }
    mbar_init(bar_kvt, 8);
    mbar_init(bar_final, 1);
    mbar_init_fence();
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_do);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(&tmem_base_s), 512);
    tmem_relinquish();
  }
  if (tid == 32) {
    const int64_t hk = WALK ? h_idx / p.heads : h_idx;
    s_out = {{static_cast<int64_t>(b_idx) * p.s0_b + hk * p.s0_h,
              static_cast<int64_t>(b_idx) * p.s1_b + hk * p.s1_h},
             tile_tok0, min(p.N, tile_tok0 + groups * p.kvb)};
  }
  tc_fence_before();
  pdl_wait();
  if (tid == 0) {   // under the building of the union
    mbar_expect_tx(bar_kv, (MODE == 1 ? 1 : 2) * ROW_TILE_BYTES);
    for (int c = 0; c < NCH; c++) {
      tma_load_4d(smem_u32(sK) + c * 128 * 128, &tm_k, bar_kv, c * 64, h_idx / p.kv_hdiv, tile_tok0,
                  b_idx);
      if (MODE != 1)
        tma_load_4d(smem_u32(sV) + c * 128 * 128, &tm_v, bar_kv, c * 64, h_idx / p.kv_hdiv, tile_tok0,
                    b_idx);
    }
  }
  const int n = dkv_union(un, sQD, p, bhq, j0, groups, p.G);
  tc_fence_after();
  const uint32_t tmem = tmem_base_s;
  WaitCtx w{&abort_flag, p.status};
  const bool split = (p.g % 32) == 0;   // q columns of a tile shared by two warps per row

  if (warp == 0) {
    if (lane == 0 && n > 0) {
      HeadWalk<WALK> hw;
      for (int i = 0; i < n; i++) {
        const int s = i % NST;
        if (!mbar_wait(bar_qempty(s), ((i / NST) & 1) ^ 1, w, FTK_DEV_TIMEOUT_TMA)) break;
        const int row0 = hw.at(un.ids[i], p) * p.g - p.q_pad_head;
        const uint32_t base = smem_u32(sQD) + s * stage_bytes;
        mbar_expect_tx(bar_qfull(s), stage_bytes);
        for (int c = 0; c < NCH; c++) {
          tma_load_4d(base + c * q_chunk_bytes, &tm_q, bar_qfull(s), c * 64, h_idx + hw.head, row0,
                      b_idx);
          tma_load_4d(base + (NCH + c) * q_chunk_bytes, &tm_do, bar_qfull(s), c * 64,
                      h_idx + hw.head, row0, b_idx);
        }
      }
    }
  } else if (warp == 1) {
    if (n > 0) {
      // the whole warp runs this path; one elected lane issues the UMMAs
      const uint32_t idesc_a = umma_idesc(128, p.g, p.fmt, 0, 0);
      const uint32_t idesc_b = umma_idesc(128, D, p.fmt, 0, 1);
      const uint64_t kdesc0 = smem_desc_sw128(smem_u32(sK), 16, 1024);
      const uint64_t vdesc0 = smem_desc_sw128(smem_u32(sV), 16, 1024);
      const uint64_t qdesc0 = smem_desc_sw128(smem_u32(sQD), 16, 1024);
      const uint64_t qmn0 = smem_desc_sw128(smem_u32(sQD), q_chunk_bytes, 1024);
      // P^T / dS^T column of k-step ks: each half of the q columns is written
      // by its own warps over the columns those warps read
      const int kh = p.g / 32, kh_shift = kh >> 1, half_cols = p.g / 2;
      auto pt_col = [&](int ks) {
        return split ? (ks >> kh_shift) * half_cols + (ks & (kh - 1)) * 8 : ks * 8;
      };
      // head dim 128: without branches around what one lane issues (see elect_one)
      const uint32_t el = K_T ? elect_one() : 1u;
      auto mine = [&]() { return K_T || elect_one(); };
      auto all = [&](bool x) { return K_T ? warp_all(x) : x; };
      bool ok = all(mbar_wait(ROWS_T ? bar_kvt : bar_kv, 0, w, FTK_DEV_TIMEOUT_MMA));
      tc_fence_after();
      auto wait_q = [&](int i) -> bool {
        return all(mbar_wait(bar_qfull(i % NST), (i / NST) & 1, w, FTK_DEV_TIMEOUT_MMA));
      };
      auto mma_s = [&](int i) {   // elected lane only, like the other three
        const uint64_t qdesc = desc_advance(qdesc0, (i % NST) * stage_bytes);
        const uint32_t sb = i & 1;
#pragma unroll
        for (int ks = 0; ks < D / 16; ks++) {
          const uint32_t aoff = (ks / 4) * 128 * 128 + (ks % 4) * 32;
          const uint32_t boff = (ks / 4) * q_chunk_bytes + (ks % 4) * 32;
          if (ROWS_T)
            umma_ts(tmem + sb * 64, tmem + COL_K + ks * 8, desc_advance(qdesc, boff), idesc_a, ks > 0, el);
          else
            umma_ss(tmem + sb * 64, desc_advance(kdesc0, aoff), desc_advance(qdesc, boff), idesc_a,
                    ks > 0, el);
        }
      };
      auto mma_dp = [&](int i) {
        const uint64_t dodesc = desc_advance(qdesc0, (i % NST) * stage_bytes + NCH * q_chunk_bytes);
        const uint32_t sb = i & 1, dp = tmem + 128 + (K_T ? 0 : sb * 64);
        if (MODE != 1) {
#pragma unroll
          for (int ks = 0; ks < D / 16; ks++) {
            const uint32_t aoff = (ks / 4) * 128 * 128 + (ks % 4) * 32;
            const uint32_t boff = (ks / 4) * q_chunk_bytes + (ks % 4) * 32;
            if (ROWS_T && !K_T)
              umma_ts(dp, tmem + COL_V + ks * 8, desc_advance(dodesc, boff), idesc_a, ks > 0, el);
            else
              umma_ss(dp, desc_advance(vdesc0, aoff), desc_advance(dodesc, boff), idesc_a, ks > 0, el);
          }
        }
        umma_commit(bar_afull(sb), el);
      };
      auto mma_a = [&](int i) {
        mma_s(i);
        mma_dp(i);
      };
      auto mma_b = [&](int i) {
        const int s = i % NST, sb = i & 1;
        const uint64_t qmn = desc_advance(qmn0, s * stage_bytes);
        const uint64_t domn = desc_advance(qmn, NCH * q_chunk_bytes);
        if (K_T) {   // P^T and dS^T of 16 q rows side by side over the S^T they came from
          auto step = [&](int ks) {
            const bool acc = (i > 0) || (ks > 0);
            const uint32_t col = tmem + sb * 64 + ks * 16;
            umma_ts(tmem + COL_DV, col, desc_advance(domn, ks * 2048), idesc_b, acc, el);
            umma_ts(tmem + COL_DK, col + 8, desc_advance(qmn, ks * 2048), idesc_b, acc, el);
          };
          if (p.g == 64) {
#pragma unroll
            for (int ks = 0; ks < 4; ks++) step(ks);
          } else {
            for (int ks = 0; ks < p.g / 16; ks++) step(ks);
          }
        } else if (p.g == 64) {
#pragma unroll
          for (int ks = 0; ks < 4; ks++) {
            const bool acc = (i > 0) || (ks > 0);
            const uint32_t col = sb * 64 + (ks >> 1) * 32 + (ks & 1) * 8;
            if (MODE != 2)
              umma_ts(tmem + COL_DV, tmem + col, desc_advance(domn, ks * 2048), idesc_b, acc, el);
            if (MODE != 1)
              umma_ts(tmem + COL_DK, tmem + 128 + col, desc_advance(qmn, ks * 2048), idesc_b, acc, el);
          }
        } else {
          for (int ks = 0; ks < p.g / 16; ks++) {
            const bool acc = (i > 0) || (ks > 0);
            if (MODE != 2)
              umma_ts(tmem + COL_DV, tmem + sb * 64 + pt_col(ks), desc_advance(domn, ks * 2048),
                      idesc_b, acc, el);
            if (MODE != 1)
              umma_ts(tmem + COL_DK, tmem + 128 + sb * 64 + pt_col(ks),
                      desc_advance(qmn, ks * 2048), idesc_b, acc, el);
          }
        }
        umma_commit(bar_qempty(s), el);
      };
      if (ok) ok = wait_q(0);
      if (ok && n > 1) ok = wait_q(1);
      tc_fence_after();
      if (ok && mine()) {
        mma_a(0);
        if (n > 1) {
          if (K_T) mma_s(1);
          else mma_a(1);
        }
      }
      __syncwarp();
      // At head dim 128 the next tile's loads (32 KB) are often still on their way: dV
      // and dK of tile i go out first and the wait for tile i + 2 runs under them.  At
      // head dim 64 (16 KB) they are there, and one wait and one batch are cheaper
      // (680 -> 675 us at N = 8192, H = 16).
      for (int i = 0; ok && i < n; i++) {
        if (D == 64) {
          const bool more = i + 2 < n;
          const int i2 = more ? i + 2 : i;
          const uint32_t wb[2] = {bar_pfull(i & 1), bar_qfull(i2 % NST)};
          const uint32_t wp[2] = {static_cast<uint32_t>((i >> 1) & 1),
                                  static_cast<uint32_t>((i2 / NST) & 1)};
          if (!mbar_wait_all<2>(wb, wp, w, FTK_DEV_TIMEOUT_MMA)) break;
          tc_fence_after();
          if (elect_one()) {
            mma_b(i);
            if (more) mma_a(i2);
          }
          __syncwarp();
          continue;
        }
        if (K_T && i + 1 < n) {
          if (!all(mbar_wait(bar_dpfree, i & 1, w, FTK_DEV_TIMEOUT_MMA))) break;
          tc_fence_after();
          mma_dp(i + 1);
          __syncwarp();
        }
        if (!all(mbar_wait(bar_pfull(i & 1), (i >> 1) & 1, w, FTK_DEV_TIMEOUT_MMA))) break;
        tc_fence_after();
        if (mine()) mma_b(i);
        __syncwarp();
        if (i + 2 < n) {
          if (!wait_q(i + 2)) break;
          tc_fence_after();
          if (mine()) {
            if (K_T) mma_s(i + 2);
            else mma_a(i + 2);
          }
          __syncwarp();
        }
      }
      if (ok && mine()) umma_commit(bar_final, el);
      __syncwarp();
    }
  } else {
    // Two groups of 8 warps; group w drains the buffers of tiles i = w (mod 2).
    // Inside a group two warps share each 32-row lane quarter and take one
    // half of the q columns each.
    const int cw = warp - 2;
    const int wg = cw >> 3;
    const int colhalf = (cw >> 2) & 1;
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const int ct = (tid - 64) & 255;         // index inside the group
    const int grp = r / p.kvb;
    const uint32_t lane_addr = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t st_addr = lane_addr + wg * 64;         // S^T, then P^T
    const uint32_t dp_addr = lane_addr + 128 + (K_T ? 0 : wg * 64);   // dP^T, then dS^T
    // (head dim 128, where 32 columns at most are kept while dP^T makes room: 48 as 32 and 16)
    const int part = K_T && p.g == 48 ? 32 : split ? p.g / 2 : p.g;
    const int cbeg = min(colhalf * part, p.g), cend = min(cbeg + part, p.g);
    const float c = p.scale_log2;
    bool ok = true;
    if (ROWS_T && n > 0 && colhalf == 0) {
      // group 0 moves the K tile, group 1 the V tile (head dim 128: each half of the K
      // tile), from (swizzled) shared memory into TMEM: row r -> lane r, two 16-bit values
      // per column
      ok = mbar_wait(bar_kv, 0, w, FTK_DEV_TIMEOUT_CONSUMER);
      if (ok) {
        const uint8_t* src = K_T ? sK + wg * 128 * 128 : wg == 0 ? sK : sV;
        uint32_t v[32];
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const uint4 t4 = *reinterpret_cast<const uint4*>(src + sw128_offset(r, j));
          v[j * 4 + 0] = t4.x;
          v[j * 4 + 1] = t4.y;
          v[j * 4 + 2] = t4.z;
          v[j * 4 + 3] = t4.w;
        }
        tmem_st32(lane_addr + (K_T ? COL_K + wg * 32 : wg == 0 ? COL_K : COL_V), v);
        tmem_wait_st();
        tc_fence_before();
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_kvt);
    }
    // every thread of a group runs all of the group's rounds (its named
    // barrier needs all 256); after a failed wait a thread only keeps the
    // barrier company and does no more work.
    HeadWalk<WALK> hw;
    for (int i = wg; i < n; i += 2) {
      const int pb = (i >> 1) & 1;           // per-group double buffer of lse / delta
      const int row0 = hw.at(un.ids[i], p) * p.g - p.q_pad_head;
      if (ct < p.g) {
        const int t = row0 + ct;
        float l2 = 0.f, dl = 0.f;
        if (t >= 0 && t < p.N) {   // staged negated: the packed fma / add take them as they are
          const int64_t e = static_cast<int64_t>(bhq + hw.head) * p.N + t;
          l2 = -p.lse[e] * 1.4426950408889634f;
          dl = -p.delta[e];
        }
        s_lse2[wg][pb][ct] = l2;
        s_delta[wg][pb][ct] = dl;
      }
      if (wg == 0)
        asm volatile("bar.sync 1, 256;" ::: "memory");
      else
        asm volatile("bar.sync 2, 256;" ::: "memory");
      const ColSpan cs = col_span(un, i, p.sub, grp, row0, p.g, p.N);
      const int lo = cs.lo, hi = cs.hi;
      const bool act = cs.on;
      // all of this warp's columns, or none of them (see the dQ kernel)
      const bool fast = __all_sync(0xffffffffu, act && lo <= cbeg && hi >= cend);
      const bool none = !fast && !__any_sync(0xffffffffu, act && lo < cend && hi > cbeg);
      if (!ok) continue;
      if (!mbar_wait(bar_afull(wg), (i >> 1) & 1, w, FTK_DEV_TIMEOUT_CONSUMER)) {
        ok = false;
        continue;
      }
      tc_fence_after();
      const float4* l4 = reinterpret_cast<const float4*>(s_lse2[wg][pb]);
      const float4* d4 = reinterpret_cast<const float4*>(s_delta[wg][pb]);
      // P^T / dS^T of columns [c0, c0+16) go over columns cbeg + (c0-cbeg)/2 ..
      // of the S^T / dP^T regions (head dim 128: over c0 .. and c0 + 8 .. of S^T): columns
      // this thread has already read
      const bool whole = cend - cbeg == 32;
      if (K_T && whole && fast) {
        // the dP^T buffer is the next tile's as soon as its columns are in registers
        uint32_t sv[2][16], dv[2][16];
        tmem_ld16(dp_addr + cbeg, dv[0]);
        tmem_ld16(dp_addr + cbeg + 16, dv[1]);
        tmem_ld16(st_addr + cbeg, sv[0]);
        tmem_ld16(st_addr + cbeg + 16, sv[1]);
        tmem_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_dpfree);
#pragma unroll
        for (int h = 0; h < 2; h++) {
          uint32_t pp[8], pd[8];
          const int c0 = cbeg + 16 * h;
          if (p.fmt == 1) pt_pairs<1>(sv[h], dv[h], l4 + (c0 >> 2), d4 + (c0 >> 2), c, pp, pd);
          else pt_pairs<0>(sv[h], dv[h], l4 + (c0 >> 2), d4 + (c0 >> 2), c, pp, pd);
          tmem_st8(st_addr + c0, pp);
          tmem_st8(st_addr + c0 + 8, pd);
        }
      } else if (K_T && whole && !none) {
        uint32_t sv[2][16], dv[2][16];
        tmem_ld16(dp_addr + cbeg, dv[0]);
        tmem_ld16(dp_addr + cbeg + 16, dv[1]);
        tmem_ld16(st_addr + cbeg, sv[0]);
        tmem_ld16(st_addr + cbeg + 16, sv[1]);
        tmem_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_dpfree);
#pragma unroll
        for (int h = 0; h < 2; h++) {
          uint32_t pp[8], pd[8];
          const int c0 = cbeg + 16 * h;
          pt_masked(sv[h], dv[h], l4 + (c0 >> 2), d4 + (c0 >> 2), c, act ? lo - c0 : 16, hi - c0, p.fmt, pp, pd);
          tmem_st8(st_addr + c0, pp);
          tmem_st8(st_addr + c0 + 8, pd);
        }
      } else
      for (int c0 = cbeg; c0 < cend; c0 += 16) {
        uint32_t sv[16], dv[16], pp[8], pd[8];
        const int oc = K_T ? c0 : cbeg + ((c0 - cbeg) >> 1);
        const uint32_t ds_addr = K_T ? st_addr + oc + 8 : dp_addr + oc;
        if (none) {   // the other group's q-block: P^T = dS^T = 0, nothing to read
#pragma unroll
          for (int x = 0; x < 8; x++) pp[x] = 0u;
          if (MODE != 2) tmem_st8(st_addr + oc, pp);
          if (MODE != 1) tmem_st8(ds_addr, pp);
          continue;
        }
        tmem_ld16(st_addr + c0, sv);
        if (MODE != 1) tmem_ld16(dp_addr + c0, dv);
        tmem_wait_ld();
        if (K_T) {   // 16 columns
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_dpfree);
        }
        if (MODE == 1) {   // no dP^T in this launch: dS^T is computed and dropped
#pragma unroll
          for (int x = 0; x < 16; x++) dv[x] = 0u;
        }
        if (fast) {
          if (p.fmt == 1) pt_pairs<1>(sv, dv, l4 + (c0 >> 2), d4 + (c0 >> 2), c, pp, pd);
          else pt_pairs<0>(sv, dv, l4 + (c0 >> 2), d4 + (c0 >> 2), c, pp, pd);
        } else {
          pt_masked(sv, dv, l4 + (c0 >> 2), d4 + (c0 >> 2), c, act ? lo - c0 : 16, hi - c0, p.fmt, pp, pd);
        }
        if (MODE != 2) tmem_st8(st_addr + oc, pp);
        if (MODE != 1) tmem_st8(ds_addr, pd);
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (K_T && (none || cbeg == cend)) mbar_arrive(bar_dpfree);
        mbar_arrive(bar_pfull(wg));
      }
    }
    if (ok) ok = mbar_wait(n > 0 ? bar_final : bar_kv, 0, w, FTK_DEV_TIMEOUT_EPILOGUE);
    if (ok) {
      tc_fence_after();
      // MODE 0: group 0 stores dV (TMEM 256..), group 1 stores dK (TMEM 384.., scaled);
      // otherwise both groups share the one accumulator's columns
      const int ew = (late_tid() >> 5) - 2;
      const int which = MODE == 0 ? ew >> 3 : MODE - 1;
      const float mul = which == 0 ? 1.f : p.scale;
      // every copy has landed and every UMMA has retired: the tiles make room for the results
      const int cfirst = MODE == 0 ? ((ew >> 2) & 1) * 32 : (ew >> 2) * 32;
#pragma unroll 1
      for (int c0 = cfirst; c0 < D; c0 += (MODE == 0 ? 64 : 128)) {
        uint32_t v[32];
        if (n > 0) {
          tmem_ld32(lane_addr + (which == 0 ? COL_DV : COL_DK) + c0, v);
          tmem_wait_ld();
        }
        uint32_t pk[16];
#pragma unroll
        for (int x = 0; x < 32; x += 2) {
          const float a = n > 0 ? __uint_as_float(v[x]) * mul : 0.f;
          const float b = n > 0 ? __uint_as_float(v[x + 1]) * mul : 0.f;
          pk[x >> 1] = pack2(a, b, p.fmt);
        }
        store_rows(smem + ew * 2048, pk, which == 0 ? p.out1 : p.out0, s_out, which == 0 ? 1 : 0,
                   (ew + 2) & 3, which == 0 ? p.s1_n : p.s0_n, c0, p.D, p.fmt, p.out_f32 != 0);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (abort_flag)
    for (int i = 0; i < 200; i++) __nanosleep(1000);
  if (warp == 0) tmem_dealloc(tmem, 512);
}

}  // namespace ftk

#include "sparse_bwd_dkv2.cuh"
#include "sparse_bwd_dq2.cuh"
#include "sparse_bwd_d256.cuh"

namespace ftk {

// ---------------------------------------------------- order of the dK/dV tiles
// Per slice: q-blocks that each kv tile (128 rows, or the 256 of a pair of CTAs: G kv
// blocks) has to walk, from the dQ kernel's tile masks, and the tiles sorted by that
// number, largest first (ties: lower tile).  With skewed lists a few tiles take many times
// the others' time; issued last they would run alone.  One CTA per slice, key = (count + 1, ~tile).
// `pick`: whether pairs of SMs should do the slice.  A step of the pair kernel is the shorter
// one, but it walks the q-blocks that list any of four kv blocks, not of two.  Twice the
// pairs' steps over the single tiles' steps is 1 where neighbouring blocks are listed together
// (windows, runs of blocks) and near 1.5 where lists of a quarter of the blocks are
// independent.  The line, 1.2, was drawn while the one-CTA kernel read K from shared memory (pairs 0.92
// to 0.98 of a backward pass at ratios up to 1.14, 1.01 at 1.25).  With K in tensor memory that kernel
// is the faster one for all lists: backward passes with the choice against without, N = 6400 to
// 32768, H = 4 to 32, lists of a quarter to a half: windows 1.04 to 1.10 of the time, runs of four
// blocks 1.03 to 1.07, lists that four q-blocks share 1.02 to 1.09, independent ones (which stay on
// single SMs) 1.00 to 1.02.  FTK_DKV_2CTA=0 leaves the choice out.
constexpr int FAN_THREADS = 1024;

__global__ void __launch_bounds__(FAN_THREADS)
fan_in_kernel(const uint8_t* masks, int stride, int tiles, int64_t head_stride, int heads,
              int slices_per_b, int H, int G, int cols, int colsp, int32_t* order, int32_t* pick) {
  extern __shared__ unsigned long long fan_keys[];
  unsigned* cnt = reinterpret_cast<unsigned*>(fan_keys + colsp);
  __shared__ unsigned single, pairs;   // q-blocks that all tiles, and all pairs of tiles, walk
  pdl_wait();
  pdl_launch();
  const int tid = threadIdx.x;
  const int slice = blockIdx.x;
  const int bhq = slice / slices_per_b * H + slice % slices_per_b * heads;
  if (tid == 0) single = pairs = 0u;
  for (int x = tid; x < colsp; x += FAN_THREADS) cnt[x] = 0u;
  __syncthreads();
  unsigned in_pairs = 0u, in_single = 0u;
  // 16 bytes = 16 / G kv tiles of one q tile per load, the q tiles dealt to as many
  // threads as there are (a byte per load and row took some 95 us longer at 403 q
  // tiles of 806 kv blocks, one slice)
  const int quads = stride >> 4, parts = max(1, FAN_THREADS / quads), rows = heads * tiles;
  for (int u = tid; u < quads * parts; u += FAN_THREADS) {
    const int quad = u % quads, part = u / quads;
    unsigned c[16];
#pragma unroll
    for (int x = 0; x < 16; x++) c[x] = 0;
#pragma unroll 4
    for (int r = part; r < rows; r += parts) {
      const int h = r / tiles;
      const uint4 t = *(reinterpret_cast<const uint4*>(
                            masks + (bhq + h) * head_stride +
                            static_cast<int64_t>(r - h * tiles) * stride) + quad);
      const unsigned w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
      for (int x = 0; x < 16; x++) {
        unsigned m = (w[x >> 2] >> (8 * (x & 3))) & 255u;
        if (G == 2) m |= (w[x >> 2] >> (8 * ((x & 3) ^ 1))) & 255u;
        if (G == 4 || G == 8) {
          m = w[x >> 2] | (G == 8 ? w[(x >> 2) ^ 1] : 0u);
          m = (m | (m >> 8) | (m >> 16) | (m >> 24)) & 255u;
        }
        if (x % G == 0) c[x] += __popc(m);
        if (pick && x % 4 == 0) {   // G is 2, a pair has four blocks
          const unsigned m4 = w[x >> 2];
          in_pairs += __popc((m4 | (m4 >> 8) | (m4 >> 16) | (m4 >> 24)) & 255u);
        }
      }
    }
#pragma unroll
    for (int x = 0; x < 16; x++) {
      const int col = (quad * 16 + x) / G;
      if (x % G == 0 && col < cols && c[x]) atomicAdd(&cnt[col], c[x]);
      if (x % G == 0) in_single += c[x];
    }
  }
  if (pick) {
    in_single = __reduce_add_sync(0xffffffffu, in_single);
    in_pairs = __reduce_add_sync(0xffffffffu, in_pairs);
    if ((tid & 31) == 0) {
      atomicAdd(&single, in_single);
      atomicAdd(&pairs, in_pairs);
    }
  }
  __syncthreads();
  if (pick && tid == 0) pick[slice] = 10 * pairs < 6 * single;
  for (int x = tid; x < colsp; x += FAN_THREADS)
    fan_keys[x] = x < cols ? (static_cast<unsigned long long>(cnt[x] + 1u) << 32) |
                                 (0xffffffffu - static_cast<unsigned>(x))
                           : 0ull;
  __syncthreads();
  for (int k = 2; k <= colsp; k <<= 1)
    for (int d = k >> 1; d > 0; d >>= 1) {
      for (int i = tid; i < colsp; i += FAN_THREADS) {
        const int o = i ^ d;
        if (o > i) {
          const unsigned long long a = fan_keys[i], b = fan_keys[o];
          if (((i & k) == 0) ? (a < b) : (a > b)) {
            fan_keys[i] = b;
            fan_keys[o] = a;
          }
        }
      }
      __syncthreads();
    }
  for (int x = tid; x < cols; x += FAN_THREADS)
    order[static_cast<int64_t>(slice) * cols + x] =
        static_cast<int32_t>(0xffffffffu - static_cast<unsigned>(fan_keys[x]));
}

// ------------------------------------------- sum over the heads of a kv head
// dk, dv of every query head ([B][N][H][D], 16-bit) -> one per kv head: the
// heads of a group added up in fp32, in order, and rounded once.  Bound by
// memory (2 * H * D * 2 B read per token, 16 bytes per thread and load); used
// where the grid is too small for one CTA to walk all heads of a group.
__global__ void __launch_bounds__(256)
head_sum_kernel(const uint8_t* dk_part, const uint8_t* dv_part, int fmt, int64_t N, int Hkv,
                int grp, int D, int64_t vecs, void* dk, int64_t k_b, int64_t k_n, int64_t k_h,
                void* dv, int64_t v_b, int64_t v_n, int64_t v_h, int f32) {
  pdl_wait();
  pdl_launch();
  const int dvec = D >> 3;
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= vecs) return;
  const uint4* src = reinterpret_cast<const uint4*>(blockIdx.y ? dv_part : dk_part);
  const int64_t head = i / dvec;                 // (b * N + n) * Hkv + hk
  const int c = static_cast<int>(i - head * dvec);
  const int64_t row = head / Hkv;
  const int hk = static_cast<int>(head - row * Hkv);
  const int64_t b = row / N, n = row - b * N;
  float acc[8];
#pragma unroll
  for (int x = 0; x < 8; x++) acc[x] = 0.f;
  const uint4* s = src + head * grp * dvec + c;
  for (int g = 0; g < grp; g++) {
    const uint4 t = s[static_cast<int64_t>(g) * dvec];
    const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
    for (int x = 0; x < 4; x++) {
      const float2 f = unpack2(w[x], fmt);
      acc[2 * x] += f.x;
      acc[2 * x + 1] += f.y;
    }
  }
  uint32_t pk[4];
#pragma unroll
  for (int x = 0; x < 4; x++) pk[x] = pack2(acc[2 * x], acc[2 * x + 1], fmt);
  uint8_t* out = static_cast<uint8_t*>(blockIdx.y ? dv : dk);
  const int64_t e = blockIdx.y ? b * v_b + n * v_n + hk * v_h : b * k_b + n * k_n + hk * k_h;
  store_row_part(out + (f32 ? 4 : 2) * e, c * 8, D, pk, fmt, f32 != 0);
}

// ------------------------------------------------------------------- host side
// What a backward pass shares between its two calls: the grid of blocks and
// where things lie in the workspace.
struct BwdPlan {
  AttnGrid gr;
  bool pair_dq, pair_dkv;    // kernels on pairs of SMs
  bool walk;                 // dK/dV: one CTA walks all query heads of its kv head
  int tiles, stride, span;   // tile masks (see TileMaskRow)
  int kv_tiles;              // kv tiles of a CTA (or a pair) per slice
  int tile_blocks;           // kv blocks of such a tile
  bool order;                // dK/dV tiles sorted by the work they have
  bool pick;                 // dK/dV: pairs or single SMs slice by slice, see fan_in_kernel
  size_t off_masks, off_order, off_pick, off_dk, off_dv, bytes;
};

static size_t up256(size_t x) { return (x + 255) & ~static_cast<size_t>(255); }

static bool env_off(const char* name) {
  const char* e = getenv(name);
  return e && e[0] == '0';
}

static int bwd_plan(const ftk_attn& a, BwdPlan* out) {
  BwdPlan b{};
  int e = attn_grid(a, 64, &b.gr);
  // head dim 256 with blocks other than 64 and 32 rows: the one-CTA kernels hold Q / dO
  // (dQ) or K / V (dK, dV) of 256 columns in shared memory and have room for 32-row
  // partner tiles only
  if (a.D > 128 && (e || !tiles_of_64(b.gr.g, b.gr.kvb))) e = attn_grid(a, 32, &b.gr);
  if (e) return e;
  const AttnGrid& gr = b.gr;
  const bool tiles64 = tiles_of_64(gr.g, gr.kvb);
  if (gr.g % 16 != 0) return FTK_ERR_UNSUPPORTED;
  if (gr.QM > AT_MAX_BLOCKS) return FTK_ERR_UNSUPPORTED;
  const int64_t BH = a.B * a.H;
  const int per = attn_groups(gr.g), G = attn_groups(gr.kvb);
  b.tiles = (gr.QM + per - 1) / per;
  b.stride = flag_blocks(gr.Mkv);
  b.span = (b.tiles * per + 31) & ~31;
  // Pairs walk the union of four lists.  dQ at head dim 128, kilocycles in pairs and without: all
  // blocks listed, 64 587, 609, 128 1050, 1112; lists of 40 of 64 545, 500, of 80 of 128 962, 880.
  // dK / dV on single SMs: K in tensor memory made them the faster ones whatever the lists
  // (backward passes: 64 of 64 blocks 1275, 1187, 128 of 128 2352, 2204, 512 of 512 8386, 8135, 47
  // of 47 274, 275; 64 of 128 2081, 1820, four heads per kv head 4155, 3338); `pick` still hands
  // some lists to pairs.  At head dim 256 the pair kernels are several times the faster per tile.
  b.pair_dq = tiles64 && (gr.kd == 256 || (gr.kd == 128 && 4 * gr.width >= 3 * static_cast<int64_t>(gr.Mkv)));
  b.pair_dkv = tiles64 && gr.kd == 256;
  // Query heads that share a kv head: walked one after the other by the CTA that
  // owns the kv rows, so that their sum stays in its fp32 accumulators, unless
  // that leaves SMs idle: waves of CTAs times heads per CTA against waves of one
  // CTA per head, with a quarter's lead for the per-head results that are then
  // neither written nor read again.
  const int64_t grp = a.H / a.Hkv, ctas = a.B * a.Hkv * ((gr.Mkv + G - 1) / G), sms = sm_count();
  auto waves = [&](int64_t n) { return (n + sms - 1) / sms; };
  b.walk = grp > 1 && grp * b.span <= AT_MAX_BLOCKS &&
           4 * grp * waves(ctas) <= 5 * waves(ctas * grp);
  const int64_t slices = b.walk ? a.B * a.Hkv : BH;
  // sorting pays once the tiles come in several waves; lists that can cover most blocks
  // give all tiles as much to do (head dim 128, backward passes in kilocycles, sorted and not: lists
  // of 64 of 128 1820, 1847, four heads per kv head 3338, 3577; 40 of 64 1062, 1048; 128 of 128
  // 2231, 2204)
  b.tile_blocks = b.pair_dkv ? 2 * G : G;
  b.kv_tiles = (gr.Mkv + b.tile_blocks - 1) / b.tile_blocks;
  b.order = b.pair_dkv ? 2 * gr.width < gr.Mkv && 2 * slices * b.kv_tiles >= 2 * sms
                       : slices * b.kv_tiles >= 2 * sms &&
                             !(tiles64 && gr.kd == 128 && 2 * gr.width > gr.Mkv);
  // Below that line the lists decide for dK / dV, where they can be such that pairs pay (see
  // fan_in_kernel, and there what they take now): from a quarter of the blocks on, and only if a kv
  // block is listed by 32 q-blocks or more on average.  CTAs that find the decision against them
  // take 7 to 24 us together.  Not where a CTA walks several heads, nor with blocks of 32 rows,
  // where two listed blocks share a tile's step and the ratio of the steps does not say which
  // is the faster.
  b.pick = b.order && !b.walk && gr.g == 64 && gr.kvb == 64 && gr.kd == 128 && !b.pair_dkv &&
           4 * gr.width >= gr.Mkv && 2 * gr.width < gr.Mkv &&
           gr.width * gr.QM >= 32 * static_cast<int64_t>(gr.Mkv) && !env_off("FTK_DKV_2CTA");
  size_t off = up256(static_cast<size_t>(BH) * a.N * 4);   // delta
  b.off_masks = off;
  off += up256(static_cast<size_t>(BH) * b.tiles * b.stride);
  b.off_order = off;
  if (b.order) off += up256(static_cast<size_t>(slices) * b.kv_tiles * 4);
  b.off_pick = off;
  if (b.pick) off += up256(static_cast<size_t>(slices) * 4);
  b.off_dk = b.off_dv = off;
  if (grp > 1 && !b.walk) {
    const size_t part = up256(static_cast<size_t>(BH) * a.N * a.D * 2);
    b.off_dv = off + part;
    off += 2 * part;
  }
  b.bytes = off;
  *out = b;
  return FTK_OK;
}

static BwdParams bwd_params(const ftk_attn& a, const AttnGrid& gr, const float* lse, float* delta,
                            int32_t* status) {
  BwdParams p{};
  p.N = static_cast<int>(a.N);
  p.H = static_cast<int>(a.H);
  p.D = static_cast<int>(a.D);
  p.QM = gr.QM;
  p.W = a.W;
  p.Mkv = gr.Mkv;
  p.g = gr.g;
  p.kvb = gr.kvb;
  p.q_pad_head = gr.q_pad_head;
  p.kv_pad_head = gr.kv_pad_head;
  p.fmt = a.dtype;
  p.scale = a.scale;
  p.scale_log2 = a.scale * 1.4426950408889634f;
  p.lse = lse;
  p.delta = delta;
  p.out_f32 = a.out_f32;
  p.status = status;
  p.kv_hdiv = static_cast<int>(a.H / a.Hkv);
  p.heads = 1;
  p.span = p.span_tiles = 1 << 30;
  return p;
}

struct Rows {   // a 16-bit tensor [b][n][h][d]
  const void* base;
  int64_t heads, sb, sn, sh;
};

static int tmap_of(CUtensorMap* t, const ftk_attn& a, const Rows& r, int rows) {
  return encode_tmap_bnhd(t, r.base, a.dtype, a.B, a.N, r.heads, a.D, r.sb, r.sn, r.sh, 64, rows);
}

// Two CTAs of one group per SM, or one CTA of two?  Two CTAs cover each other's list
// union, first loads and last tile, but go by twice the CTAs per wave.  A CTA's time
// with n tiles is put at 7 + 0.32 n us alone and 8.5 + 0.72 n us as one of two: fitted to
// which of the two was the faster in 44 backward passes (H N / 128 of 16 to 1024 CTAs,
// lists of 4 blocks to all), over which the rule is at most 0.8 % behind the better one.
// One against two groups: N = 1024, H = 32, all pairs 66.6, 70.6 us; N = 8192, H = 4, lists
// of 64 261, 251 and of 16 103, 105; H = 16, of 4 159, 173 and all pairs 1193, 1144.
static bool one_group(int64_t ctas, int tiles) {
  const int64_t sms = sm_count();
  return ((ctas + 2 * sms - 1) / (2 * sms)) * (8.5 + 0.72 * tiles) <
         ((ctas + sms - 1) / sms) * (7.0 + 0.32 * tiles);
}

static int launch_dq(const ftk_attn& a, const Rows& dout, BwdParams p, int kd, bool pair,
                     cudaStream_t st) {
  const Rows q = {a.q, a.H, a.sq_b, a.sq_n, a.sq_h}, k = {a.k, a.Hkv, a.sk_b, a.sk_n, a.sk_h},
             v = {a.v, a.Hkv, a.sv_b, a.sv_n, a.sv_h};
  const unsigned bh = static_cast<unsigned>(a.B * a.H);
  p.G = attn_groups(p.g);
  p.sub = tiles_of_64(p.g, p.kvb) && (pair || kd < 256) ? 64 / p.kvb : 1;
  p.kvb *= p.sub;
  CUtensorMap tq, tdo, tk, tv;
  int e;
  if ((e = tmap_of(&tq, a, q, 128)) || (e = tmap_of(&tdo, a, dout, 128)) ||
      (e = tmap_of(&tk, a, k, p.kvb)))
    return e;
  if (pair && (kd == 256 || !env_off("FTK_DQ_2CTA"))) {
    CUtensorMap tk32, tv32;
    if ((e = tmap_of(&tk32, a, k, 32)) || (e = tmap_of(&tv32, a, v, 32))) return e;
    const dim3 grid(2 * ((p.QM + 2 * p.G - 1) / (2 * p.G)), bh);
    auto go = [&](auto kernel_tag, size_t smem) -> int {
      constexpr auto kernel = decltype(kernel_tag)::kernel;
      if (int r = allow_smem<kernel>(smem)) return r;
      return launch_pdl(kernel, grid, BW_THREADS, smem, st, tq, tdo, tk, tk32, tv32, p);
    };
    return choose<2>(a.dtype, [&](auto fmt) {
      return choose<3>(p.sub, [&](auto sub) {
        constexpr int F = decltype(fmt)::value, S = decltype(sub)::value == 2 ? 2 : 1;
        return kd == 256
                   ? go(Kernel<sparse_bwd_dq256_kernel<F, S>>{},
                        1024 + 2 * B6_ROWS + static_cast<size_t>(DQ6_SLOTS) * B6_PIECE)
                   : go(Kernel<sparse_bwd_dq2_kernel<F, S>>{},
                        1024 + 2 * 2 * 128 * 128 + static_cast<size_t>(DQ2_STAGES) * 24576);
      });
    });
  }
  if ((e = tmap_of(&tv, a, v, p.kvb))) return e;
  const int nch = kd / 64;
  const dim3 grid((p.QM + p.G - 1) / p.G, bh);
  if (kd == 256) {
    // Q and dO resident, three K and two V tiles behind them: kv blocks of at most 32 rows
    if (p.kvb > 32) return FTK_ERR_UNSUPPORTED;
    const size_t smem =
        1024 + 2 * nch * 128 * 128 +
        std::max(static_cast<size_t>(3 + 2) * nch * p.kvb * 128, flag_bytes(p.Mkv, p.G));
    if ((e = allow_smem<sparse_bwd_dq_kernel<256, 2>>(smem))) return e;
    return launch_pdl(sparse_bwd_dq_kernel<256, 2>, grid, BW_THREADS, smem, st, tq, tdo, tk, tv, p);
  }
  auto go = [&](auto kernel_tag, int ng) -> int {
    constexpr auto kernel = decltype(kernel_tag)::kernel;
    // four V slots lie over the Q / dO tiles, the rest of the V ring behind the K ring; the
    // marks of the list union where the K ring will be
    const size_t smem = 1024 + 2 * nch * 128 * 128 +
                        std::max(static_cast<size_t>(dq_kst(ng) + DQ_VST - 4) * nch * p.kvb * 128,
                                 flag_bytes(p.Mkv, p.G));
    if (int r = allow_smem<kernel>(smem)) return r;
    return launch_pdl(kernel, grid, bw_threads(ng), smem, st, tq, tdo, tk, tv, p);
  };
  if (kd == 64)
    return one_group(static_cast<int64_t>(grid.x) * grid.y,
                     static_cast<int>(std::min(static_cast<int64_t>(p.G) * p.W,
                                               static_cast<int64_t>(p.Mkv / p.sub))))
               ? go(Kernel<sparse_bwd_dq_kernel<64, 1>>{}, 1)
               : go(Kernel<sparse_bwd_dq_kernel<64, 2>>{}, 2);
  return go(Kernel<sparse_bwd_dq_kernel<128, 2>>{}, 2);
}

static int launch_dkv(const ftk_attn& a, const Rows& dout, BwdParams p, int kd, bool pair,
                      cudaStream_t st) {
  const Rows q = {a.q, a.H, a.sq_b, a.sq_n, a.sq_h}, k = {a.k, a.Hkv, a.sk_b, a.sk_n, a.sk_h},
             v = {a.v, a.Hkv, a.sv_b, a.sv_n, a.sv_h};
  const unsigned slices = static_cast<unsigned>(a.B * a.H / p.heads);
  p.G = attn_groups(p.kvb);
  p.sub = tiles_of_64(p.g, p.kvb) && (pair || kd < 256) ? 64 / p.g : 1;
  p.g *= p.sub;
  p.span_tiles = p.span / p.sub;
  CUtensorMap tq, tdo, tk, tv;
  int e;
  if ((e = tmap_of(&tq, a, q, p.g)) || (e = tmap_of(&tdo, a, dout, p.g)) ||
      (e = tmap_of(&tk, a, k, 128)) || (e = tmap_of(&tv, a, v, 128)))
    return e;
  if (pair) {
    CUtensorMap tq32, tdo32;
    if ((e = tmap_of(&tq32, a, q, 32)) || (e = tmap_of(&tdo32, a, dout, 32))) return e;
    const dim3 grid(2 * ((p.Mkv + 2 * p.G - 1) / (2 * p.G)), slices);
    auto go = [&](auto kernel_tag, size_t smem) -> int {
      constexpr auto kernel = decltype(kernel_tag)::kernel;
      if (int r = allow_smem<kernel>(smem)) return r;
      return launch_pdl(kernel, grid, BW_THREADS, smem, st, tq, tdo, tq32, tdo32, tk, tv, p);
    };
    return choose<2>(a.dtype, [&](auto fmt) {
      constexpr int F = decltype(fmt)::value;
      if (kd == 128)   // 64-row blocks, one head per pair: see bwd_plan
        return go(Kernel<sparse_bwd_dkv2_kernel<F>>{},
                  1024 + 2 * 2 * 128 * 128 + static_cast<size_t>(DK2_STAGES) * 32768);
      return choose<3>(p.sub, [&](auto sub) {
        return choose<2>(p.heads > 1, [&](auto walk) {
          constexpr int S = decltype(sub)::value == 2 ? 2 : 1;
          constexpr bool W = decltype(walk)::value;
          int r = go(Kernel<sparse_bwd_dkv256_kernel<F, 1, W, S>>{},
                     1024 + B6_ROWS + static_cast<size_t>(DV6_SLOTS) * B6_PIECE);
          if (r) return r;
          return go(Kernel<sparse_bwd_dkv256_kernel<F, 2, W, S>>{},
                    1024 + 2 * B6_ROWS + static_cast<size_t>(DQ6_SLOTS) * B6_PIECE);
        });
      });
    });
  }
  const int nch = kd / 64;
  const int stage_bytes = 2 * nch * p.g * 128;
  const int tile_bytes = nch * 128 * 128;          // K or V of the CTA's 128 kv rows
  // 227 KB per CTA less the static part (union scratch, lse / delta staging: ~22 KB) and the
  // resident tiles; at head dim 256 that leaves two stages of q blocks of up to 32 rows next to
  // K and V, four next to K alone
  auto stages = [&](int resident) {
    const int ring_bytes = (227 - 23) * 1024 - resident * tile_bytes;
    return std::min(BW_MAX_STAGES, std::min(128 * 1024, ring_bytes) / stage_bytes);
  };
  auto smem_for = [&](int resident, int nst) {
    return static_cast<size_t>(1024) + static_cast<size_t>(resident) * tile_bytes +
           std::max(static_cast<size_t>(nst) * stage_bytes, p.masks ? 0 : flag_bytes(p.QM, p.G));
  };
  const dim3 grid(p.order ? p.Mkv : (p.Mkv + p.G - 1) / p.G, slices);
  auto go = [&](auto kernel_tag, int resident) -> int {
    constexpr auto kernel = decltype(kernel_tag)::kernel;
    p.nstages = stages(resident);
    if (p.nstages < (kd <= 128 ? BW_MAX_STAGES : 2)) return FTK_ERR_UNSUPPORTED;
    const size_t smem = smem_for(resident, p.nstages);
    if (int r = allow_smem<kernel>(smem)) return r;
    return launch_pdl(kernel, grid, BW_THREADS, smem, st, tq, tdo, tk, tv, p);
  };
  const bool walk = p.heads > 1;
  if (kd == 256) {
    if (stages(2) < 2) return FTK_ERR_UNSUPPORTED;
    if ((e = walk ? go(Kernel<sparse_bwd_dkv_kernel<256, 1, true>>{}, 1)
                  : go(Kernel<sparse_bwd_dkv_kernel<256, 1, false>>{}, 1)))
      return e;
    return walk ? go(Kernel<sparse_bwd_dkv_kernel<256, 2, true>>{}, 2)
                : go(Kernel<sparse_bwd_dkv_kernel<256, 2, false>>{}, 2);
  }
  if (kd == 64)
    return walk ? go(Kernel<sparse_bwd_dkv_kernel<64, 0, true>>{}, 2)
                : go(Kernel<sparse_bwd_dkv_kernel<64, 0, false>>{}, 2);
  return walk ? go(Kernel<sparse_bwd_dkv_kernel<128, 0, true>>{}, 2)
              : go(Kernel<sparse_bwd_dkv_kernel<128, 0, false>>{}, 2);
}

}  // namespace ftk

using namespace ftk;

extern "C" size_t ftk_attn_bwd_workspace(const ftk_attn* a) {
  BwdPlan b;
  return a && bwd_plan(*a, &b) == FTK_OK ? b.bytes : 0;
}

extern "C" int ftk_attn_bwd_dq(const ftk_attn* a, const void* o, int64_t so_b, int64_t so_n,
                               int64_t so_h, const void* dout, int64_t sdo_b, int64_t sdo_n,
                               int64_t sdo_h, const float* lse, void* workspace,
                               size_t workspace_bytes, void* dq, int64_t sdq_b, int64_t sdq_n,
                               int64_t sdq_h, int32_t* status, void* stream) {
  if (!a || !lse) return FTK_ERR_BAD_ARG;
  BwdPlan b;
  if (int e = bwd_plan(*a, &b)) return e;
  if (!aligned16(o, so_b, so_n, so_h) || !aligned16(dout, sdo_b, sdo_n, sdo_h) ||
      !aligned16(dq, sdq_b, sdq_n, sdq_h))
    return FTK_ERR_BAD_ARG;
  if (!workspace || workspace_bytes < b.bytes) return FTK_ERR_WORKSPACE;
  if (reinterpret_cast<uintptr_t>(workspace) & 255u) return FTK_ERR_BAD_ARG;
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  BwdParams p = bwd_params(*a, b.gr, lse, reinterpret_cast<float*>(ws), status);
  p.lists = a->lists;
  p.list_rows = a->list_rows;
  p.lm = b.gr.lm;
  p.masks = ws + b.off_masks;
  p.mask_stride = b.stride;
  p.mask_tiles = b.tiles;
  p.o = static_cast<const uint8_t*>(o);
  p.so_b = so_b;
  p.so_n = so_n;
  p.so_h = so_h;
  p.dout = static_cast<const uint8_t*>(dout);
  p.sd_b = sdo_b;
  p.sd_n = sdo_n;
  p.sd_h = sdo_h;
  p.out0 = dq;
  p.s0_b = sdq_b;
  p.s0_n = sdq_n;
  p.s0_h = sdq_h;
  return launch_dq(*a, Rows{dout, a->H, sdo_b, sdo_n, sdo_h}, p, b.gr.kd, b.pair_dq,
                   static_cast<cudaStream_t>(stream));
}

extern "C" int ftk_attn_bwd_dkv(const ftk_attn* a, const void* dout, int64_t sdo_b, int64_t sdo_n,
                                int64_t sdo_h, const float* lse, void* workspace,
                                size_t workspace_bytes, void* dk, int64_t sdk_b, int64_t sdk_n,
                                int64_t sdk_h, void* dv, int64_t sdv_b, int64_t sdv_n,
                                int64_t sdv_h, int32_t* status, void* stream) {
  if (!a || !lse) return FTK_ERR_BAD_ARG;
  BwdPlan b;
  if (int e = bwd_plan(*a, &b)) return e;
  if (!aligned16(dout, sdo_b, sdo_n, sdo_h) || !aligned16(dk, sdk_b, sdk_n, sdk_h) ||
      !aligned16(dv, sdv_b, sdv_n, sdv_h))
    return FTK_ERR_BAD_ARG;
  if (!workspace || workspace_bytes < b.bytes) return FTK_ERR_WORKSPACE;
  if (reinterpret_cast<uintptr_t>(workspace) & 255u) return FTK_ERR_BAD_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  BwdParams p = bwd_params(*a, b.gr, lse, reinterpret_cast<float*>(ws), status);
  p.masks = ws + b.off_masks;
  p.mask_stride = b.stride;
  p.mask_tiles = b.tiles;
  p.mask_g = attn_groups(b.gr.g);
  p.span = b.span;
  p.heads = b.walk ? p.kv_hdiv : 1;
  const bool parts = p.kv_hdiv > 1 && !b.walk;
  if (parts) {   // one 16-bit result per query head first
    const int64_t row = a->H * a->D;
    p.out0 = ws + b.off_dk;
    p.out1 = ws + b.off_dv;
    p.s0_b = p.s1_b = a->N * row;
    p.s0_n = p.s1_n = row;
    p.s0_h = p.s1_h = a->D;
    p.out_f32 = 0;
  } else {
    p.out0 = dk;
    p.s0_b = sdk_b;
    p.s0_n = sdk_n;
    p.s0_h = sdk_h;
    p.out1 = dv;
    p.s1_b = sdv_b;
    p.s1_n = sdv_n;
    p.s1_h = sdv_h;
  }
  if (b.order && !env_off("FTK_DKV_ORDER")) {
    int colsp = 32;
    while (colsp < b.kv_tiles) colsp <<= 1;
    const size_t smem = static_cast<size_t>(colsp) * 12;
    int32_t* order = reinterpret_cast<int32_t*>(ws + b.off_order);
    int32_t* pick = b.pick ? reinterpret_cast<int32_t*>(ws + b.off_pick) : nullptr;
    int e = allow_smem<fan_in_kernel>(smem);
    if (!e)
      e = launch_pdl(fan_in_kernel, static_cast<unsigned>(a->B * a->H / p.heads), FAN_THREADS, smem,
                     st, p.masks, b.stride, b.tiles,
                     static_cast<int64_t>(b.tiles) * b.stride, p.heads,
                     static_cast<int>(a->H / p.heads), static_cast<int>(a->H),
                     b.tile_blocks, b.kv_tiles, colsp, order, pick);
    if (e) return e;
    if (pick) {
      p.pick = pick;
      if ((e = launch_dkv(*a, Rows{dout, a->H, sdo_b, sdo_n, sdo_h}, p, b.gr.kd, true, st))) return e;
    }
    p.tile_order = order;
  }
  if (int e = launch_dkv(*a, Rows{dout, a->H, sdo_b, sdo_n, sdo_h}, p, b.gr.kd, b.pair_dkv, st))
    return e;
  if (!parts) return FTK_OK;
  const int64_t vecs = a->B * a->N * a->Hkv * (a->D / 8);
  if ((vecs + 255) / 256 > 0x7fffffffLL) return FTK_ERR_BAD_ARG;
  return launch_pdl(head_sum_kernel, dim3(static_cast<unsigned>((vecs + 255) / 256), 2), 256, 0, st,
                    ws + b.off_dk, ws + b.off_dv, a->dtype, a->N, static_cast<int>(a->Hkv),
                    p.kv_hdiv, static_cast<int>(a->D), vecs, dk, sdk_b, sdk_n, sdk_h, dv, sdv_b,
                    sdv_n, sdv_h, a->out_f32);
}

static int old_bwd_grid(const ftk_attn& a, AttnGrid* gr) {
  if (a.D != 64 && a.D != 128 && a.D != 256) return FTK_ERR_UNSUPPORTED;
  if (a.kv_block > 64) return FTK_ERR_UNSUPPORTED;
  return attn_grid(a, 128, gr);   // blocks as they are
}

extern "C" int ftk_sparse_bwd_dq(
    const void* q, const void* k, const void* v, const void* o, const void* dout, int dtype,
    int64_t B, int64_t H, int64_t Hkv, int64_t N, int64_t D, int64_t sq_b, int64_t sq_n, int64_t sq_h,
    int64_t sk_b, int64_t sk_n, int64_t sk_h, int64_t sv_b, int64_t sv_n, int64_t sv_h,
    int64_t so_b, int64_t so_n, int64_t so_h, int64_t sdo_b, int64_t sdo_n, int64_t sdo_h,
    const int32_t* merged_idx, int QM, int W, int q_block_size, int kv_block_size, int q_pad_head,
    int kv_pad_head, float scale, const float* lse, float* delta, void* dq, int64_t sdq_b,
    int64_t sdq_n, int64_t sdq_h, int32_t* status, void* stream) {
  const ftk_attn a = {q,    k,    v,    dtype, 0,    B,    H,    Hkv <= 0 ? H : Hkv,
                      N,    D,    sq_b, sq_n,  sq_h, sk_b, sk_n, sk_h,
                      sv_b, sv_n, sv_h, merged_idx, QM, W, q_block_size, kv_block_size,
                      q_pad_head, kv_pad_head, scale};
  AttnGrid gr;
  if (int e = old_bwd_grid(a, &gr)) return e;
  if (!lse || !delta || !aligned16(o, so_b, so_n, so_h) || !aligned16(dout, sdo_b, sdo_n, sdo_h) ||
      !aligned16(dq, sdq_b, sdq_n, sdq_h))
    return FTK_ERR_BAD_ARG;
  BwdParams p = bwd_params(a, gr, lse, delta, status);
  p.lists = merged_idx;
  p.list_rows = QM;
  p.o = static_cast<const uint8_t*>(o);
  p.so_b = so_b;
  p.so_n = so_n;
  p.so_h = so_h;
  p.dout = static_cast<const uint8_t*>(dout);
  p.sd_b = sdo_b;
  p.sd_n = sdo_n;
  p.sd_h = sdo_h;
  p.out0 = dq;
  p.s0_b = sdq_b;
  p.s0_n = sdq_n;
  p.s0_h = sdq_h;
  const bool pair = D == 128 && q_block_size == 64 && kv_block_size == 64 &&
                    4 * static_cast<int64_t>(W) >= 3 * static_cast<int64_t>(gr.Mkv);
  return launch_dq(a, Rows{dout, H, sdo_b, sdo_n, sdo_h}, p, gr.kd, pair,
                   static_cast<cudaStream_t>(stream));
}

extern "C" int ftk_sparse_bwd_dkv(
    const void* q, const void* k, const void* v, const void* dout, int dtype, int64_t B, int64_t H,
    int64_t Hkv, int64_t N, int64_t D, int64_t sq_b, int64_t sq_n, int64_t sq_h, int64_t sk_b, int64_t sk_n,
    int64_t sk_h, int64_t sv_b, int64_t sv_n, int64_t sv_h, int64_t sdo_b, int64_t sdo_n,
    int64_t sdo_h, const int32_t* reverse_idx, const int32_t* reverse_counts,
    const int32_t* sorted_kv, int QM, int M, int q_block_size, int kv_block_size, int q_pad_head,
    int kv_pad_head, float scale, const float* lse, const float* delta, void* dk, int64_t sdk_b,
    int64_t sdk_n, int64_t sdk_h, void* dv, int64_t sdv_b, int64_t sdv_n, int64_t sdv_h,
    int fwd_list_width, int32_t* status, void* stream) {
  const ftk_attn a = {q,    k,    v,    dtype, 0,    B,    H,    Hkv <= 0 ? H : Hkv,
                      N,    D,    sq_b, sq_n,  sq_h, sk_b, sk_n, sk_h,
                      sv_b, sv_n, sv_h, reverse_idx, QM, QM, q_block_size, kv_block_size,
                      q_pad_head, kv_pad_head, scale};
  AttnGrid gr;
  if (int e = old_bwd_grid(a, &gr)) return e;
  if (q_block_size % 16 != 0 || q_block_size > 64) return FTK_ERR_UNSUPPORTED;
  if (QM > AT_MAX_BLOCKS) return FTK_ERR_UNSUPPORTED;
  if (M <= 0 || static_cast<int64_t>(M) * kv_block_size < kv_pad_head + N) return FTK_ERR_BAD_ARG;
  if (!reverse_counts || !lse || !delta || !aligned16(dout, sdo_b, sdo_n, sdo_h) ||
      !aligned16(dk, sdk_b, sdk_n, sdk_h) || !aligned16(dv, sdv_b, sdv_n, sdv_h))
    return FTK_ERR_BAD_ARG;
  BwdParams p = bwd_params(a, gr, lse, const_cast<float*>(delta), status);
  p.Mkv = M;
  p.lists = reverse_idx;
  p.counts = reverse_counts;
  p.out0 = dk;
  p.s0_b = sdk_b;
  p.s0_n = sdk_n;
  p.s0_h = sdk_h;
  p.out1 = dv;
  p.s1_b = sdv_b;
  p.s1_n = sdv_n;
  p.s1_h = sdv_h;
  // tiles in order of fan-in when the caller brings the order and the lists are not wide
  const bool wide = D == 128 && q_block_size == 64 && kv_block_size == 64 &&
                    (fwd_list_width <= 0 || 2 * static_cast<int64_t>(fwd_list_width) > M);
  p.order = sorted_kv && !wide && !env_off("FTK_DKV_ORDER") ? sorted_kv : nullptr;
  return launch_dkv(a, Rows{dout, H, sdo_b, sdo_n, sdo_h}, p, gr.kd, false,
                    static_cast<cudaStream_t>(stream));
}
