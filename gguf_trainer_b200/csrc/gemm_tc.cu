// Tensor-core matrix product for sm_100a: tcgen05.mma (kind::tf32, f32 operands read straight from
// shared memory, f32 accumulators in TMEM), operands staged by TMA into 128B-swizzled tiles, a 5/6-stage
// mbarrier pipeline, persistent CTAs (one per SM) with two TMEM accumulators: one elected thread issues TMA, one
// issues MMA, four warps drain the finished accumulator while the next tile is being accumulated.
// Covers the three layouts of WebGPUBackend.gemm (src/backend/webgpu.ts:1654-1671; srcGemm
// src/backend/wgsl.ts:87-196): NT (forward y = x.W^T), NN (dX += dY.W), TN (dW += dY^T.X), with ragged
// edges handled by TMA zero fill and guarded stores, `accum` by a read-modify-write epilogue, and split-K
// (f32 reductions in L2) when a product has few output tiles and a deep K (the dW product, K = rows).
//
// Every wait on an mbarrier is bounded in wall time; on expiry the CTA records a code in a device flag
// the host checks at the next sync, skips its stores, releases its TMEM and exits.
#include <cuda.h>

#include <string.h>

#include <mutex>
#include <unordered_map>

#include "common.cuh"
#include "tc_common.cuh"

using namespace tc;

namespace {

constexpr int BM1 = 128;         // UMMA M (cta_group::1): accumulator row i lives in TMEM lane i
constexpr int BK = 32;           // f32 elements per stage along K: 128 bytes = one swizzle row
constexpr int UMMA_K = 8;        // tf32: 32 bytes of K per instruction

// Tile shapes. MT = 1: 128 x BN output tile, two TMEM accumulators, so the epilogue of a tile runs under the
// main loop of the next. MT = 2: 256 x BN, two 128-row halves that share every B tile and fill the tensor memory
// (no second buffer: the epilogue is exposed). With 4-byte operands the main loop is bound by shared-memory
// bandwidth, not by the tensor pipe: every stage is written once by TMA and read by the MMAs once per 128-row
// half, at 128 B/clk. A 256-row tile moves fewer bytes per flop (the B tile is fetched once for both halves), which
// pays when the tile count still fills the SMs evenly; the host picks per product.
// SUB epilogue warps share the rows of a TMEM lane quadrant and take turns at its column blocks: one for plain outputs, whose
// epilogue hides under the next tile's main loop; three where the epilogue computes (the gated unit, the rotation): with one
// it took 10 us a tile against 6 us of main loop at K 576 and set the pace (gate, up and the unit at 16384 rows: 137 us).
template <int BN, int MT, int SUB = 1>
struct Smem {
  static constexpr int BM = BM1 * MT;
  static constexpr int A_BYTES = BM * BK * 4;   // 16 / 32 KB
  static constexpr int B_BYTES = BN * BK * 4;
  static constexpr int STAGE = A_BYTES + B_BYTES;
  static constexpr int STAGES = MT == 2 ? 3 : (BN <= 128 ? 5 : 4);
  static constexpr int EPI_WARPS = 4 * MT * SUB;
  static constexpr int EPI_TILES = MT == 2 || SUB > 1 ? 1 : 2;   // 32x32 f32 staging tiles per epilogue warp for the TMA store
  static constexpr int EPI_BYTES = EPI_WARPS * EPI_TILES * 4096;
  static constexpr int TOTAL = STAGES * STAGE + EPI_BYTES + 1024 /*alignment slack*/ + 256 /*barriers*/;
  static constexpr uint32_t TMEM_COLS = 2 * BN <= 256 ? 256 : 512;   // two accumulators (MT = 1) or two halves (MT = 2)
  static constexpr int THREADS = 64 + 32 * EPI_WARPS;   // warp 0: TMA, warp 1: MMA + TMEM owner, then the epilogue warps
  static_assert(TOTAL <= 232448, "shared memory");
};

// Persistent: each CTA walks output tiles t = blockIdx.x, blockIdx.x + gridDim.x, ... (n fastest, then m, then the
// split-K slice), so CTAs running at the same time share their A row-blocks in L2.
// A_K: A is K-major in memory (NT, NN); else MN-major ([K, M], TN). B_K: B is K-major (NT); else [K, N] (NN, TN).
// Operands of one launch: up to MAX_PARTS products A_p.B_p of the same layout, K_p deep, summed into the same output
// tiles. kb_end[p] is the number of K blocks of parts 0..p; only the TMA producer looks at it.
constexpr int MAX_PARTS = 8;
struct PartMaps {
  CUtensorMap a[MAX_PARTS], b[MAX_PARTS];
  int kb_end[MAX_PARTS];
  int nparts;
  // Grouped form (ngroups > 1, one part): group g is its own product A_g.B_g -> C_g of gM[g] x gN[g], all of one
  // layout and one K; its tiles are units [unit_end[g-1], unit_end[g]) of the launch (n fastest, then m, then the
  // split-K slice). c[g] is its output map (c[0] the only one when ngroups == 1).
  CUtensorMap c[MAX_PARTS];
  int ngroups;
  int gM[MAX_PARTS], gN[MAX_PARTS], g_accum[MAX_PARTS], unit_end[MAX_PARTS];
  // Rotary form (EPI_ROPE): the outputs of the groups with g_rope[g] set are rotated as they are written (see the kernel).
  int g_rope[MAX_PARTS];
  float* cp[MAX_PARTS];     // the outputs themselves (gemm_tf32_small_kernel stores without a tensor map)
  const float2* rope_tab;   // [rope_period][32] (cos, sin) of the 32 pairs of a 64-wide head
  int rope_period;          // positions per sequence: row r is position r % rope_period
  CeArgs ce;                // readout forms (EPI_CE_STATS, EPI_CE_GRAD)
};
constexpr int EPI_ROPE = 8;   // values of the kernel's GLU argument that are neither activation
constexpr int EPI_CE_STATS = 16, EPI_CE_GRAD = 32, EPI_CE_BOTH = 64;

// GLU != 0 (GT_EW_SILU or GT_EW_GELU; NT layout, BN = 192 only): the gated unit of the FFN in the projection that
// feeds it. B is two weight matrices: the tile's first 96 columns are rows [n0/2, n0/2 + 96) of b[0] (gate), the other 96
// the same rows of b[1] (up). The epilogue writes the gate and up projections (backward needs them) through c[0] and
// c[1] and act(gate) * up through c[2], so the separate pass that read both and wrote the product is not launched.
// N_ is 2 x the FFN width.
// GLU == EPI_ROPE (grouped NT launches, BN = 192, heads 64 wide): the rotary embedding that follows the q and k
// projections (src/arch/llama.ts:195-199 records `rope(linear(x, Wq))`) applied to the accumulator on its way out. A
// 192-column tile is three whole heads; the thread that owns a row loads the two 32-column halves of a head, rotates
// pair (j, j + 32) by the angle of (row's position, j) from the table, and both halves go out as they would have.
// The unrotated projection is never written.
// GLU == EPI_CE_STATS, EPI_CE_GRAD (NT layout, one product, no split): the logits of one vocabulary span of the chunked
// readout loss. STATS keeps, per row, the maximum and the sum of exponentials of the tile's columns (one pair per epilogue
// thread, merged by ce_merge_kernel) and the target's logit, and writes no logits at all; GRAD turns the logits into the
// loss's gradient on their way out. The passes over [rows, span] that did this (a read; a read and a write) are bound by
// HBM: at 8192 x 32768 157 and 552 us beside a product of 1.3 ms.
// EPI_CE_BOTH writes the logits of a whole vocabulary and takes their statistics (the loss that keeps its logits): the pass
// over them costs 239 us at 8192 x 49152.
// (epilogue warps per lane quadrant: three where the epilogue computes and runs beside the main loop)
template <int MT, int GLU>
struct EpiSub { static constexpr int N = MT == 1 && GLU != 0 ? 3 : 1; };
// What one epilogue warp does with its share of a finished accumulator: 32 rows (a TMEM lane quadrant), every SUB-th column
// block. Outputs are staged as 32x32 blocks in shared memory (128-byte rows, 16-byte chunks XOR (row mod 8), the layout the
// store's tensor map expects) and written by TMA: whole 128-byte rows, clipped at M and N, as a plain store or, when
// accumulating or combining split-K slices, as an f32 reduce-add performed in L2. Shared by the kernels below.
struct CeRow { uint32_t tg; float m, inv, sc; };   // readout forms: what the row needs of the loss
template <int GLU>
__device__ __forceinline__ CeRow ce_row(const PartMaps& maps, int row, int M) {
  CeRow r = {0xffffffffu, 0.f, 0.f, 0.f};
  if (GLU >= EPI_CE_STATS && row < M) {
    r.tg = __ldg(maps.ce.targets + row);
    if (GLU == EPI_CE_GRAD) {
      r.m = __ldg(maps.ce.run + (size_t)row * 3);
      r.inv = 1.f / __ldg(maps.ce.run + (size_t)row * 3 + 1);
      r.sc = __ldg(maps.ce.gloss) * __ldg(maps.ce.inv_kept + row / maps.ce.T) / (float)maps.ce.nseq;
    }
  }
  return r;
}
struct Drain {           // of one tile
  const CUtensorMap* mapC;
  float* C;
  int bi, g, n0, row0, M, N, ksplit, accum, use_tma_store;   // row0: first row of this warp's 32
  float out_scale;
  bool dead;             // a wait has expired: nothing is stored
};
template <int BN, int GLU, int SUB, int TILES>
__device__ __forceinline__ void drain_tile(const PartMaps& maps, const Drain& d, const CeRow& ce, uint8_t* smem_raw, uint32_t stage,
                                           uint32_t tacc, int sub, int lane, uint32_t& nst) {
  constexpr bool IS_GLU = GLU == GT_EW_SILU || GLU == GT_EW_GELU;
  const int M = d.M, N = d.N, n0 = d.n0, row = d.row0 + lane;
  auto put = [&](const float* v, const CUtensorMap* map, int col0) {
    const uint32_t tile = stage + (nst % TILES) * 4096u;
    if (nst >= TILES) tma_wait_read<TILES - 1>();   // the tile's previous contents have been read out
    __syncwarp();
    uint8_t* tp = smem_raw + (tile - smem_u32(smem_raw)) + lane * 128;
#pragma unroll
    for (int c4 = 0; c4 < 8; c4++)
      *reinterpret_cast<float4*>(tp + ((c4 ^ (lane & 7)) * 16)) = make_float4(v[4 * c4], v[4 * c4 + 1], v[4 * c4 + 2], v[4 * c4 + 3]);
    fence_async_smem();
    __syncwarp();
    if (lane == 0 && !d.dead && d.row0 < M) {
      if (!IS_GLU && (d.ksplit > 1 || d.accum)) tma_reduce_add_3d(map, tile, col0, d.row0, d.bi);
      else tma_store_3d(map, tile, col0, d.row0, d.bi);
    }
    if (lane == 0) tma_commit_group();
    nst++;
  };
  if (GLU == EPI_CE_STATS || GLU == EPI_CE_BOTH) {
    float m = -3.0e38f, s = 0.f;
    const uint32_t tcol = ce.tg - (uint32_t)maps.ce.v0;   // the target's column of the span, if it is below N
#pragma unroll 1
    for (int c = sub; c < BN / 32; c += SUB) {
      const int col0 = n0 + c * 32;
      if (col0 >= N) break;   // uniform across the warp
      float v[32];
      tmem_ld32(tacc + (uint32_t)(c * 32), v);
      float mb = m;
#pragma unroll
      for (int j = 0; j < 32; j++) {
        v[j] = col0 + j < N ? v[j] * d.out_scale : -3.0e38f;
        mb = fmaxf(mb, v[j]);
      }
      if (GLU == EPI_CE_BOTH) put(v, d.mapC, col0);
      float t[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int j = 0; j < 32; j++) t[j & 3] += __expf(v[j] - mb);
      s = s * __expf(m - mb) + ((t[0] + t[1]) + (t[2] + t[3]));
      m = mb;
      if (ce.tg != 0xffffffffu && tcol - (uint32_t)col0 < 32u && tcol < (uint32_t)N && !d.dead) {
#pragma unroll
        for (int j = 0; j < 32; j++)
          if (tcol == (uint32_t)(col0 + j)) maps.ce.run[(size_t)row * 3 + 2] = v[j];
      }
    }
    if (row < M && !d.dead) maps.ce.part[(size_t)((n0 / BN) * SUB + sub) * M + row] = make_float2(m, s);
  } else if (IS_GLU) {
    // gate | up halves of the accumulator: three outputs per 32-column block, each through its own tensor map
#pragma unroll 1
    for (int c = sub; c < BN / 64; c += SUB) {
      const int col0 = (n0 >> 1) + c * 32;
      if (col0 >= (N >> 1)) break;   // uniform across the warp
      float vg[32], vu[32];
      tmem_ld32_issue(tacc + (uint32_t)(c * 32), vg);
      tmem_ld32_issue(tacc + (uint32_t)(c * 32) + BN / 2, vu);
      tmem_wait_ld();
#pragma unroll
      for (int j = 0; j < 32; j++) { vg[j] *= d.out_scale; vu[j] *= d.out_scale; }
      put(vg, &maps.c[0], col0);
      put(vu, &maps.c[1], col0);
#pragma unroll
      for (int j = 0; j < 32; j++) {
        const float a = vg[j];
        float act;
        if (GLU == GT_EW_SILU) act = a / (1.f + __expf(-a));
        else act = 0.5f * a * (1.f + tanhf(0.7978845608028654f * (a + 0.044715f * a * a * a)));
        vg[j] = act * vu[j];
      }
      put(vg, &maps.c[2], col0);
    }
  } else if (GLU == EPI_ROPE && maps.g_rope[d.g]) {
    // (cos, sin) of this row's position, pairs 0..31; rows past M are clipped by the store and read row M - 1's.
    // (adding into the output is allowed: a rotation is linear)
    const float4* tab4 = reinterpret_cast<const float4*>(maps.rope_tab + (size_t)((row < M ? row : M - 1) % maps.rope_period) * 32);
#pragma unroll 1
    for (int c = sub; c < BN / 64; c += SUB) {
      const int col0 = n0 + c * 64;
      if (col0 >= N) break;   // uniform across the warp
      float v0[32], v1[32];
      tmem_ld32_issue(tacc + (uint32_t)(c * 64), v0);
      tmem_ld32_issue(tacc + (uint32_t)(c * 64) + 32, v1);
      tmem_wait_ld();
#pragma unroll
      for (int j = 0; j < 32; j += 2) {
        const float4 cs = __ldg(tab4 + (j >> 1));   // cos, sin of pair j; cos, sin of pair j + 1
        const float a0 = v0[j] * d.out_scale, a1 = v1[j] * d.out_scale, b0 = v0[j + 1] * d.out_scale, b1 = v1[j + 1] * d.out_scale;
        v0[j] = a0 * cs.x - a1 * cs.y;
        v1[j] = a0 * cs.y + a1 * cs.x;
        v0[j + 1] = b0 * cs.z - b1 * cs.w;
        v1[j + 1] = b0 * cs.w + b1 * cs.z;
      }
      put(v0, d.mapC, col0);
      put(v1, d.mapC, col0 + 32);
    }
  } else {
    const bool vec = (N & 3) == 0;
#pragma unroll 1
    for (int c = sub; c < BN / 32; c += SUB) {
      const int col0 = n0 + c * 32;
      if (col0 >= N) break;   // uniform across the warp
      float v[32];
      tmem_ld32(tacc + (uint32_t)(c * 32), v);
#pragma unroll
      for (int j = 0; j < 32; j++) v[j] *= d.out_scale;   // the caller's factor times the truncation compensation
      if (GLU == EPI_CE_GRAD) {
        const uint32_t tcol = ce.tg - (uint32_t)(maps.ce.v0 + col0);
#pragma unroll
        for (int j = 0; j < 32; j++) {
          const float g = ce.sc * (__expf(v[j] - ce.m) * ce.inv - (tcol == (uint32_t)j ? 1.f : 0.f));
          v[j] = ce.tg == 0xffffffffu ? 0.f : g;
        }
      }
      if (d.use_tma_store) {
        put(v, d.mapC, col0);
      } else if (row < M && !d.dead) {
        float* dst = d.C + (size_t)d.bi * M * N + (size_t)row * N + col0;
        if (vec && col0 + 32 <= N) {
          if (d.ksplit > 1) {
#pragma unroll
            for (int j = 0; j < 32; j += 4) atomicAdd(reinterpret_cast<float4*>(dst + j), make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]));
          } else if (d.accum) {
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
              float4 o = *reinterpret_cast<float4*>(dst + j);
              o.x += v[j]; o.y += v[j + 1]; o.z += v[j + 2]; o.w += v[j + 3];
              *reinterpret_cast<float4*>(dst + j) = o;
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; j += 4) *reinterpret_cast<float4*>(dst + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; j++) {
            if (col0 + j < N) {
              if (d.ksplit > 1) atomicAdd(dst + j, v[j]);
              else dst[j] = d.accum ? dst[j] + v[j] : v[j];
            }
          }
        }
      }
    }
  }
}

// Where tile t of a launch lies: batch matrix (or group), first column, first row, K slice (n fastest, then m, then the slice).
struct Where { int bi, g, n0, m0, z; };
template <int BM, int BN>
__device__ __forceinline__ Where tile_at(const PartMaps& maps, int t, int tiles_n, int tiles_m, int per_mat) {
  Where w;
  if (maps.ngroups > 1) {
    int g = 0;
    while (t >= maps.unit_end[g]) g++;
    const int tt = t - (g ? maps.unit_end[g - 1] : 0);
    const int tn = (maps.gN[g] + BN - 1) / BN, tmn = tn * ((maps.gM[g] + BM - 1) / BM);
    const int rem = tt % tmn;
    w.bi = 0; w.g = g; w.z = tt / tmn; w.n0 = (rem % tn) * BN; w.m0 = (rem / tn) * BM;
  } else {
    const int tt = t % per_mat;
    w.bi = t / per_mat; w.g = 0; w.n0 = (tt % tiles_n) * BN; w.m0 = ((tt / tiles_n) % tiles_m) * BM; w.z = tt / (tiles_n * tiles_m);
  }
  return w;
}

template <bool A_K, bool B_K, int BN, int MT, int GLU = 0>
__global__ void __launch_bounds__(Smem<BN, MT, EpiSub<MT, GLU>::N>::THREADS, 1)
gemm_tf32_kernel(const __grid_constant__ PartMaps maps, float* __restrict__ C, int M_, int N_,
                 int accum_, int ksplit, int use_tma_store, int batch, float out_scale, int* __restrict__ flag) {
  pdl_wait();
  extern __shared__ uint8_t smem_raw[];
  constexpr int SUB = EpiSub<MT, GLU>::N;
  using S = Smem<BN, MT, SUB>;
  const int M = M_, N = N_;   // (of the single product; a grouped launch takes each group's from `maps`)
  constexpr int STAGES = S::STAGES, BM = S::BM;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t epi = base + STAGES * S::STAGE;    // staging tiles of the epilogue warps
  const uint32_t bars = epi + S::EPI_BYTES;         // full[STAGES], empty[STAGES], acc_full[2], acc_empty[2], tmem slot
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (STAGES + s); };
  auto acc_full = [&](int b) { return bars + 8u * (2 * STAGES + b); };
  auto acc_empty = [&](int b) { return bars + 8u * (2 * STAGES + 2 + b); };
  const uint32_t tmem_slot = bars + 8u * (2 * STAGES + 4);
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));

  constexpr bool IS_GLU = GLU == GT_EW_SILU || GLU == GT_EW_GELU;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_n = (N + BN - 1) / BN, tiles_m = (M + BM - 1) / BM;
  const int per_mat = tiles_n * tiles_m * ksplit;
  const int ngroups = maps.ngroups;
  const int ntiles = ngroups > 1 ? maps.unit_end[ngroups - 1] : per_mat * batch;   // the matrices of a batch are just more tiles
  auto where = [&](int t) { return tile_at<BM, BN>(maps, t, tiles_n, tiles_m, per_mat); };
  // Further products of the same layout are accumulated into the same tiles: their K blocks simply follow those of
  // the first in the main loop, read through their own tensor maps.
  const int kblocks = maps.kb_end[maps.nparts - 1];
  const int per = (kblocks + ksplit - 1) / ksplit;   // K blocks per split-K slice
  // TMEM slot of a 128-row accumulator and the parity of its hand-over barriers: with MT = 1 the tiles alternate
  // between two slots, with MT = 2 slot h holds half h of every tile.
  auto slot_of = [&](uint32_t tl, int h) { return MT == 2 ? h : (int)(tl & 1); };
  auto par_of = [&](uint32_t tl) { return MT == 2 ? (tl & 1) : ((tl >> 1) & 1); };

  if (threadIdx.x == 0) {
    for (int p = 0; p < maps.nparts; p++) { tma_prefetch_map(&maps.a[p]); tma_prefetch_map(&maps.b[p]); }
    for (int g = 1; g < ngroups; g++) { tma_prefetch_map(&maps.a[g]); tma_prefetch_map(&maps.b[g]); }
    if (use_tma_store)
      for (int g = 0; g < ngroups; g++) tma_prefetch_map(&maps.c[g]);
    for (int s = 0; s < STAGES; s++) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    for (int b = 0; b < 2; b++) { mbar_init(acc_full(b), 1); mbar_init(acc_empty(b), 128 * SUB); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tmem_slot, S::TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot_ptr;
  bool dead = false;   // set once a bounded wait has expired: later waits are skipped, control flow stays the same
  auto wait = [&](uint32_t bar, uint32_t parity, int code) {
    if (dead) return;
    if (!mbar_wait(bar, parity)) { dead = true; atomicExch(flag, code); }
  };

  if (warp == 0) {
    if (lane == 0) {
      // ---- TMA producer ----
      uint32_t it = 0;
      for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const Where wh = where(t);
        const int bi = wh.bi, n0 = wh.n0, m0 = wh.m0, z = wh.z;
        const int kb0 = z * per, kb1 = min(kblocks, kb0 + per);
        int part = wh.g;        // (a grouped launch has one K range per group: the group's operands)
        for (int kb = kb0; kb < kb1; kb++, it++) {
          const int s = it % STAGES;
          wait(empty_bar(s), ((it / STAGES) & 1) ^ 1, 1);
          const uint32_t a_dst = base + s * S::STAGE, b_dst = a_dst + S::A_BYTES;
          if (ngroups == 1) while (kb >= maps.kb_end[part]) part++;
          const CUtensorMap* pa = &maps.a[part];
          const CUtensorMap* pb = &maps.b[part];
          const int k0 = (ngroups == 1 ? kb - (part ? maps.kb_end[part - 1] : 0) : kb) * BK;
          mbar_expect_tx(full_bar(s), S::STAGE);
          if (A_K) tma_load_3d(a_dst, pa, k0, m0, bi, full_bar(s));
          else
            for (int c = 0; c < BM / 32; c++) tma_load_3d(a_dst + c * 4096, pa, m0 + 32 * c, k0, bi, full_bar(s));
          if (IS_GLU) {
            tma_load_3d(b_dst, &maps.b[0], k0, n0 >> 1, bi, full_bar(s));
            tma_load_3d(b_dst + (BN / 2) * 128, &maps.b[1], k0, n0 >> 1, bi, full_bar(s));
          } else if (B_K) tma_load_3d(b_dst, pb, k0, n0, bi, full_bar(s));
          else
            for (int c = 0; c < BN / 32; c++) tma_load_3d(b_dst + c * 4096, pb, n0 + 32 * c, k0, bi, full_bar(s));
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // ---- MMA issuer ----
      constexpr uint32_t idesc = idesc_tf32(!A_K, !B_K, BM1, BN);
      const uint64_t a_desc0 = A_K ? desc_kmajor(base) : desc_mnmajor(base);
      const uint64_t b_desc0 = B_K ? desc_kmajor(base + S::A_BYTES) : desc_mnmajor(base + S::A_BYTES);
      constexpr uint32_t A_STEP = A_K ? 32 : 1024, B_STEP = B_K ? 32 : 1024;   // bytes per K = 8 step
      uint32_t it = 0, tl = 0;
      for (int t = blockIdx.x; t < ntiles; t += gridDim.x, tl++) {
        const int z = where(t).z;
        const int kb0 = z * per, kb1 = min(kblocks, kb0 + per);
        const uint32_t par = par_of(tl) ^ 1;
        wait(acc_empty(slot_of(tl, 0)), par, 4);   // the epilogue has drained this accumulator
        if (MT == 2 && kb0 >= kb1) wait(acc_empty(1), par, 4);
        tc_fence_after();
        for (int kb = kb0; kb < kb1; kb++, it++) {
          const int s = it % STAGES;
          wait(full_bar(s), (it / STAGES) & 1, 2);
          tc_fence_after();
          const uint32_t soff = (uint32_t)(s * S::STAGE) >> 4;
#pragma unroll
          for (int h = 0; h < MT; h++) {
            if (h == 1 && kb == kb0) {             // the second half's accumulator is drained a little later
              wait(acc_empty(1), par, 4);
              tc_fence_after();
            }
            const uint32_t d_tmem = tmem + slot_of(tl, h) * BN;
#pragma unroll
            for (int j = 0; j < BK / UMMA_K; j++)
              umma_tf32(d_tmem, a_desc0 + soff + ((h * 16384 + j * A_STEP) >> 4), b_desc0 + soff + ((j * B_STEP) >> 4), idesc,
                        (kb > kb0 || j > 0) ? 1u : 0u);
            if (kb == kb1 - 1) umma_commit(acc_full(slot_of(tl, h)));   // this accumulator is complete
          }
          umma_commit(empty_bar(s));   // the stage is free once these MMAs have read it
        }
      }
    }
  } else {
    // ---- epilogue: warp w may touch TMEM lanes [32*(w%4), 32*(w%4)+32) ----
    const int q = warp & 3, ew = warp - 2, half = MT == 2 ? ew >> 2 : 0, sub = MT == 2 ? 0 : ew >> 2;
    uint32_t tl = 0, nst = 0;   // nst: TMA stores issued by this warp
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x, tl++) {
      const Where wh = where(t);
      const int M = ngroups > 1 ? maps.gM[wh.g] : M_, N = ngroups > 1 ? maps.gN[wh.g] : N_;
      const int b = slot_of(tl, half), row0 = wh.m0 + half * BM1 + q * 32;
      const CeRow ce = ce_row<GLU>(maps, row0 + lane, M);   // (fetched while the tile is being made)
      const bool have = wh.z * per < kblocks;     // an empty split-K slice issues no MMA and contributes nothing
      if (have) wait(acc_full(b), par_of(tl), 3);
      dead = __any_sync(0xffffffffu, dead);
      tc_fence_after();
      if (have) {
        const Drain d = {&maps.c[wh.g], C, wh.bi, wh.g, wh.n0, row0, M, N, ksplit, ngroups > 1 ? maps.g_accum[wh.g] : accum_, use_tma_store, out_scale, dead};
        drain_tile<BN, GLU, SUB, S::EPI_TILES>(maps, d, ce, smem_raw, epi + (uint32_t)(ew * S::EPI_TILES) * 4096u,
                                               tmem + b * BN + ((uint32_t)(q * 32) << 16), sub, lane, nst);
      }
      tc_fence_before();
      mbar_arrive(acc_empty(b));
    }
    if (lane == 0) tma_wait_all<0>();   // every store of this warp has landed before the CTA's shared memory goes away
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, S::TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------------------------
// The same product on CTA pairs (cta_group::2): a cluster of two CTAs on neighbouring SMs owns a 256 x BN output
// tile. Each CTA stages its 128 rows of A and HALF of the B tile (the pair's tensor cores read both halves), so a
// K block costs each SM 16 KB + BN/2 x 128 B of shared-memory writes and as many reads, against 16 KB + BN x 128 B
// for a CTA working alone: with 4-byte operands that traffic, not the tensor pipe, bounds the main loop. Each
// CTA holds its 128 rows of the accumulator, twice (the epilogue of a tile runs under the next tile's main loop).
// Roles per CTA as above; the MMAs are issued by the even CTA only. Barriers: the TMA copies of both CTAs count
// their bytes on the even CTA's `full`; `empty` and `acc_full` receive the MMA completions in both CTAs (multicast
// commit); the epilogue threads of both CTAs arrive on the even CTA's `acc_empty`.
// ---------------------------------------------------------------------------------------------
// A 256 wide tile holds four blocks of a gated unit or four heads, a 192 wide one three: the computing epilogues have a warp
// per lane quadrant for each (two per quadrant instead of four: 241 against 173 us for gate, up and the unit at
// 16384 x 640 x 2*2048, where a block waits for its stores and then computes). The readout forms have eight blocks and two.
template <int BN, int GLU>
struct PairSub { static constexpr int N = GLU == 0 ? 1 : GLU >= EPI_CE_STATS ? 2 : BN / 64; };
template <int BN, int GLU = 0>
struct SmemPair {
  static constexpr int BH = BN / 2;                 // rows of the B tile staged by each CTA
  static constexpr int A_BYTES = BM1 * BK * 4;      // 16 KB
  static constexpr int B_BYTES = BH * BK * 4;
  static constexpr int STAGE = A_BYTES + B_BYTES;
  static constexpr int SUB = PairSub<BN, GLU>::N;
  static constexpr int EPI_TILES = SUB == 1 ? 2 : 1;
  static constexpr int EPI_BYTES = 4 * SUB * EPI_TILES * 4096;
  static constexpr int STAGES = (232448 - EPI_BYTES - 1024 - 256) / STAGE;   // 6 (7 for BN = 192)
  static constexpr int TOTAL = STAGES * STAGE + EPI_BYTES + 1024 + 256;
  static constexpr uint32_t TMEM_COLS = 2 * BN <= 256 ? 256 : 512;
  static constexpr int THREADS = 64 + 128 * SUB;
  static_assert(BH % 32 == 0 && STAGES >= 3 && 8 * (2 * STAGES + 5) <= 256, "tile");
};

template <bool A_K, bool B_K, int BN, int GLU = 0>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(SmemPair<BN, GLU>::THREADS, 1)
gemm_tf32_pair_kernel(const __grid_constant__ PartMaps maps, float* __restrict__ C, int M_, int N_, int accum_, int ksplit,
                      int use_tma_store, int batch, float out_scale, int* __restrict__ flag) {
  pdl_wait();
  extern __shared__ uint8_t smem_raw[];
  using S = SmemPair<BN, GLU>;
  constexpr bool IS_GLU = GLU == GT_EW_SILU || GLU == GT_EW_GELU;
  constexpr int STAGES = S::STAGES, BM = 2 * BM1;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t epi = base + STAGES * S::STAGE;
  const uint32_t bars = epi + S::EPI_BYTES;         // full[STAGES], empty[STAGES], acc_full[2], acc_empty[2], tmem slot
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (STAGES + s); };
  auto acc_full = [&](int b) { return bars + 8u * (2 * STAGES + b); };
  auto acc_empty = [&](int b) { return bars + 8u * (2 * STAGES + 2 + b); };
  const uint32_t tmem_slot = bars + 8u * (2 * STAGES + 4);
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank();          // 0: issues the MMAs; both stage operands and drain their rows
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  const int tiles_n = (N_ + BN - 1) / BN, tiles_m = (M_ + BM - 1) / BM;
  const int per_mat = tiles_n * tiles_m * ksplit;
  const int ngroups = maps.ngroups;
  const int ntiles = ngroups > 1 ? maps.unit_end[ngroups - 1] : per_mat * batch;
  auto where = [&](int t) { return tile_at<BM, BN>(maps, t, tiles_n, tiles_m, per_mat); };
  const int kblocks = maps.kb_end[maps.nparts - 1];
  const int per = (kblocks + ksplit - 1) / ksplit;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    for (int b = 0; b < 2; b++) { mbar_init(acc_full(b), 1); mbar_init(acc_empty(b), 256 * S::SUB); }   // the epilogue threads of both CTAs
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc_pair(tmem_slot, S::TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();            // the peer's barriers exist before anything is signalled to them
  tc_fence_after();
  const uint32_t tmem = *tmem_slot_ptr;
  bool dead = false;
  auto wait = [&](uint32_t bar, uint32_t parity, int code) {
    if (dead) return;
    if (!mbar_wait(bar, parity)) { dead = true; atomicExch(flag, code); }
  };

  if (warp == 0) {
    if (lane == 0) {
      // ---- TMA producer (both CTAs) ----
      uint32_t it = 0;
      for (int t = pair; t < ntiles; t += npairs) {
        const Where wh = where(t);
        const int bi = wh.bi, n0 = wh.n0 + rank * S::BH, m0 = wh.m0 + rank * BM1;
        const int kb0 = wh.z * per, kb1 = min(kblocks, kb0 + per);
        int part = wh.g;
        for (int kb = kb0; kb < kb1; kb++, it++) {
          const int s = it % STAGES;
          wait(empty_bar(s), ((it / STAGES) & 1) ^ 1, 1);
          const uint32_t a_dst = base + s * S::STAGE, b_dst = a_dst + S::A_BYTES;
          if (ngroups == 1) while (kb >= maps.kb_end[part]) part++;
          const CUtensorMap* pa = &maps.a[part];
          const CUtensorMap* pb = &maps.b[IS_GLU ? rank : part];   // (gated unit: the even CTA stages the gate's rows, the odd one up's)
          const int k0 = (ngroups == 1 ? kb - (part ? maps.kb_end[part - 1] : 0) : kb) * BK;
          if (rank == 0) mbar_expect_tx(full_bar(s), 2 * S::STAGE);   // both CTAs' stages
          if (A_K) tma_load_3d_pair(a_dst, pa, k0, m0, bi, full_bar(s));
          else
            for (int c = 0; c < BM1 / 32; c++) tma_load_3d_pair(a_dst + c * 4096, pa, m0 + 32 * c, k0, bi, full_bar(s));
          if (B_K) tma_load_3d_pair(b_dst, pb, k0, IS_GLU ? wh.n0 >> 1 : n0, bi, full_bar(s));
          else
            for (int c = 0; c < S::BH / 32; c++) tma_load_3d_pair(b_dst + c * 4096, pb, n0 + 32 * c, k0, bi, full_bar(s));
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      // ---- MMA issuer (even CTA) ----
      constexpr uint32_t idesc = idesc_tf32(!A_K, !B_K, BM, BN);
      const uint64_t a_desc0 = A_K ? desc_kmajor(base) : desc_mnmajor(base);
      const uint64_t b_desc0 = B_K ? desc_kmajor(base + S::A_BYTES) : desc_mnmajor(base + S::A_BYTES);
      constexpr uint32_t A_STEP = A_K ? 32 : 1024, B_STEP = B_K ? 32 : 1024;
      uint32_t it = 0, tl = 0;
      for (int t = pair; t < ntiles; t += npairs, tl++) {
        const int z = where(t).z;
        const int kb0 = z * per, kb1 = min(kblocks, kb0 + per);
        const int b = tl & 1;
        wait(acc_empty(b), ((tl >> 1) & 1) ^ 1, 4);   // both CTAs have drained this accumulator
        tc_fence_after();
        const uint32_t d_tmem = tmem + b * BN;
        for (int kb = kb0; kb < kb1; kb++, it++) {
          const int s = it % STAGES;
          wait(full_bar(s), (it / STAGES) & 1, 2);
          tc_fence_after();
          const uint32_t soff = (uint32_t)(s * S::STAGE) >> 4;
#pragma unroll
          for (int j = 0; j < BK / UMMA_K; j++)
            umma_tf32_pair(d_tmem, a_desc0 + soff + ((j * A_STEP) >> 4), b_desc0 + soff + ((j * B_STEP) >> 4), idesc,
                           (kb > kb0 || j > 0) ? 1u : 0u);
          umma_commit_pair(empty_bar(s), 3);   // the stage is free in both CTAs once these MMAs have read it
        }
        if (kb1 > kb0) umma_commit_pair(acc_full(b), 3);
      }
    }
  } else {
    // ---- epilogue (both CTAs): this CTA's 128 rows ----
    const int q = warp & 3, ew = warp - 2, sub = ew >> 2;
    uint32_t tl = 0, nst = 0;
    for (int t = pair; t < ntiles; t += npairs, tl++) {
      const Where wh = where(t);
      const int M = ngroups > 1 ? maps.gM[wh.g] : M_, N = ngroups > 1 ? maps.gN[wh.g] : N_;
      const int b = tl & 1, row0 = wh.m0 + rank * BM1 + q * 32;
      const CeRow ce = ce_row<GLU>(maps, row0 + lane, M);
      const bool have = wh.z * per < kblocks;
      if (have) wait(acc_full(b), (tl >> 1) & 1, 3);
      dead = __any_sync(0xffffffffu, dead);
      tc_fence_after();
      if (have) {
        const Drain d = {&maps.c[wh.g], C, wh.bi, wh.g, wh.n0, row0, M, N, ksplit, ngroups > 1 ? maps.g_accum[wh.g] : accum_, use_tma_store, out_scale, dead};
        drain_tile<BN, GLU, S::SUB, S::EPI_TILES>(maps, d, ce, smem_raw, epi + (uint32_t)(ew * S::EPI_TILES) * 4096u,
                                                  tmem + b * BN + ((uint32_t)(q * 32) << 16), sub, lane, nst);
      }
      tc_fence_before();
      mbar_arrive_leader(acc_empty(b));
    }
    if (lane == 0) tma_wait_all<0>();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();            // neither CTA leaves (or frees tensor memory) while the other may still signal it
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem, S::TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------------------------
// The same products when their tiles do not fill the SMs: decoding and short sequences (M of a few dozen to a few hundred
// rows), weight gradients of short batches, the thin products of adapters. One tile of 128 x BN per CTA, BN 32, 64 or
// 128, the contraction cut over a cluster of up to 8 CTAs. Each leaves its partial tile in shared memory and finishes its
// share of the rows over all of them, in rank order, so that C is written once: no clear before the launch, no reduce-adds in
// L2, and the result does not depend on which slice came first. What bounds these launches is latency (start-up, first
// copies, the last products, the hand-over), so nothing is persistent and all four warps drain the accumulator.
// At 512 rows, K 576: 5 us a launch where the persistent kernel with its clear took 8 + 1.5 us; gate, up and the gated unit
// of a decode step (40 rows, 7 MB of weights) 28.6 -> 6 us.
// ---------------------------------------------------------------------------------------------
template <int BN>
struct SmallSmem {
  static constexpr int A_BYTES = BM1 * BK * 4, B_BYTES = BN * BK * 4, STAGE = A_BYTES + B_BYTES;
  static constexpr int STAGES = 4;                    // two CTAs per SM at BN 32 and 64
  static constexpr int PITCH = BN + 4;                // of the partial tile (reuses the stages)
  static constexpr int TOTAL = STAGES * STAGE + 1024 + 128;
  static constexpr uint32_t TMEM_COLS = BN;
  static constexpr int THREADS = 256;
  static_assert(BM1 * PITCH * 4 <= STAGES * STAGE && TOTAL <= 232448, "shared memory");
};

// EPI: 0, GT_EW_SILU, GT_EW_GELU (gate, up and the gated unit) or EPI_ROPE, as in gemm_tf32_kernel. gridDim.x = tiles x ksplit,
// the slices of a tile adjacent and one cluster.
template <bool A_K, bool B_K, int BN, int EPI>
__global__ void __launch_bounds__(SmallSmem<BN>::THREADS)
gemm_tf32_small_kernel(const __grid_constant__ PartMaps maps, int M_, int N_, int accum_, int ksplit, float out_scale, int* __restrict__ flag) {
  pdl_wait();
  extern __shared__ uint8_t smem_raw[];
  using S = SmallSmem<BN>;
  constexpr int STAGES = S::STAGES;
  constexpr bool IS_GLU = EPI == GT_EW_SILU || EPI == GT_EW_GELU;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t bars = base + STAGES * S::STAGE;     // full[STAGES], empty[STAGES], acc_full, tmem slot
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (STAGES + s); };
  const uint32_t acc_full = bars + 8u * (2 * STAGES), tmem_slot = acc_full + 8;
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int z = (int)blockIdx.x % ksplit;
  int t = (int)blockIdx.x / ksplit, g = 0, bi = 0;
  if (maps.ngroups > 1) {
    while (t >= maps.unit_end[g]) g++;
    if (g) t -= maps.unit_end[g - 1];
  }
  const int M = maps.ngroups > 1 ? maps.gM[g] : M_, N = maps.ngroups > 1 ? maps.gN[g] : N_;
  const int accum = maps.ngroups > 1 ? maps.g_accum[g] : accum_;
  const int tn = (N + BN - 1) / BN, tmn = tn * ((M + BM1 - 1) / BM1);
  bi = t / tmn;                                       // matrix of a batch
  t -= bi * tmn;
  const int n0 = (t % tn) * BN, m0 = (t / tn) * BM1;
  const int kblocks = maps.kb_end[maps.nparts - 1];
  const int per = (kblocks + ksplit - 1) / ksplit;
  const int kb0 = min(kblocks, z * per), kb1 = min(kblocks, kb0 + per);

  bool dead = false;
  auto wait = [&](uint32_t bar, uint32_t parity, int code) {
    if (dead) return;
    if (!mbar_wait(bar, parity)) { dead = true; atomicExch(flag, code); }
  };
  int part = maps.ngroups > 1 ? g : 0;
  auto load = [&](int kb) {                           // K block kb of this slice (called in order, by thread 0)
    const int s = (kb - kb0) % STAGES;
    const uint32_t a_dst = base + s * S::STAGE, b_dst = a_dst + S::A_BYTES;
    if (maps.ngroups == 1) while (kb >= maps.kb_end[part]) part++;
    const CUtensorMap* pa = &maps.a[part];
    const CUtensorMap* pb = &maps.b[part];
    const int k0 = (maps.ngroups == 1 ? kb - (part ? maps.kb_end[part - 1] : 0) : kb) * BK;
    mbar_expect_tx(full_bar(s), S::STAGE);
    if (A_K) tma_load_3d(a_dst, pa, k0, m0, bi, full_bar(s));
    else
      for (int c = 0; c < BM1 / 32; c++) tma_load_3d(a_dst + c * 4096, pa, m0 + 32 * c, k0, bi, full_bar(s));
    if (IS_GLU) {
      tma_load_3d(b_dst, &maps.b[0], k0, n0 >> 1, bi, full_bar(s));
      tma_load_3d(b_dst + (BN / 2) * 128, &maps.b[1], k0, n0 >> 1, bi, full_bar(s));
    } else if (B_K) tma_load_3d(b_dst, pb, k0, n0, bi, full_bar(s));
    else
      for (int c = 0; c < BN / 32; c++) tma_load_3d(b_dst + c * 4096, pb, n0 + 32 * c, k0, bi, full_bar(s));
  };
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    mbar_init(acc_full, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_async_smem();
    for (int kb = kb0; kb < min(kb1, kb0 + STAGES); kb++) load(kb);   // the first copies start before anything else is set up
  }
  if (warp == 1) tmem_alloc(tmem_slot, S::TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot_ptr;

  if (warp == 0) {
    if (lane == 0)
      for (int kb = kb0 + STAGES; kb < kb1; kb++) {
        wait(empty_bar((kb - kb0) % STAGES), (((kb - kb0) / STAGES) & 1) ^ 1, 5);
        load(kb);
      }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = idesc_tf32(!A_K, !B_K, BM1, BN);
      const uint64_t a_desc0 = A_K ? desc_kmajor(base) : desc_mnmajor(base);
      const uint64_t b_desc0 = B_K ? desc_kmajor(base + S::A_BYTES) : desc_mnmajor(base + S::A_BYTES);
      constexpr uint32_t A_STEP = A_K ? 32 : 1024, B_STEP = B_K ? 32 : 1024;
      for (int kb = kb0, it = 0; kb < kb1; kb++, it++) {
        const int s = it % STAGES;
        wait(full_bar(s), (it / STAGES) & 1, 6);
        tc_fence_after();
        const uint32_t soff = (uint32_t)(s * S::STAGE) >> 4;
#pragma unroll
        for (int j = 0; j < BK / UMMA_K; j++)
          umma_tf32(tmem, a_desc0 + soff + ((j * A_STEP) >> 4), b_desc0 + soff + ((j * B_STEP) >> 4), idesc, (kb > kb0 || j > 0) ? 1u : 0u);
        umma_commit(empty_bar(s));
      }
      if (kb1 > kb0) umma_commit(acc_full);
    }
  }
  __syncwarp();
  const bool have = kb1 > kb0;
  if (have) wait(acc_full, 0, 7);      // every product has completed: the stages are free, the accumulator is whole
  dead = __any_sync(0xffffffffu, dead);
  tc_fence_after();
  // the partial tile, row by row: warps w and w + 4 take accumulator rows 32 (w mod 4) .. + 31, every other 32 columns each
  {
    const int qd = warp & 3;
    float* tile = reinterpret_cast<float*>(smem_raw + (base - smem_u32(smem_raw))) + (qd * 32 + lane) * S::PITCH;
#pragma unroll 1
    for (int c = warp >> 2; c < BN / 32; c += 2) {
      float v[32];
      if (have) tmem_ld32(tmem + ((uint32_t)(qd * 32) << 16) + (uint32_t)(c * 32), v);
#pragma unroll
      for (int j = 0; j < 32; j += 4)
        *reinterpret_cast<float4*>(tile + c * 32 + j) = have ? make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  tc_fence_before();
  if (ksplit > 1) cluster_sync_all(); else __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, S::TMEM_COLS);
  }
  const int mrows = min(BM1, M - m0);
  // four columns of a row over the slices, scaled; every slice's load is issued before the first is used
  auto sum = [&](int r, int col) {
    const uint32_t at = base + (uint32_t)(r * S::PITCH + col) * 4u;
    float4 v[8];
    if (ksplit == 1) v[0] = *reinterpret_cast<const float4*>(smem_raw + (at - smem_u32(smem_raw)));
    else {
#pragma unroll
      for (int k = 0; k < 8; k++)
        if (k < ksplit) v[k] = ld_cluster_f32x4(cluster_addr_of(at, k));
    }
    float4 s = v[0];
#pragma unroll
    for (int k = 1; k < 8; k++)
      if (k < ksplit) { s.x += v[k].x; s.y += v[k].y; s.z += v[k].z; s.w += v[k].w; }
    s.x *= out_scale; s.y *= out_scale; s.z *= out_scale; s.w *= out_scale;
    return s;
  };
  auto put = [&](float* C, int pitch, int row, int col, int ncols, float4 v, int acc) {
    if (col >= ncols || dead) return;
    float* d = C + (size_t)row * pitch + col;
    if ((pitch & 3) == 0 && col + 4 <= ncols && (((uintptr_t)C) & 15) == 0) {
      if (acc) { const float4 o = *reinterpret_cast<const float4*>(d); v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w; }
      *reinterpret_cast<float4*>(d) = v;
      return;
    }
    d[0] = acc ? d[0] + v.x : v.x;
    if (col + 1 < ncols) d[1] = acc ? d[1] + v.y : v.y;
    if (col + 2 < ncols) d[2] = acc ? d[2] + v.z : v.z;
    if (col + 3 < ncols) d[3] = acc ? d[3] + v.w : v.w;
  };
  float* C = maps.cp[IS_GLU ? 0 : g] + (size_t)bi * M * N;
  if constexpr (IS_GLU) {
    const int ffn = maps.gN[0];
    for (int q = z * S::THREADS + threadIdx.x; q < mrows * (BN / 8); q += ksplit * S::THREADS) {
      const int r = q / (BN / 8), c = (q % (BN / 8)) * 4, col = (n0 >> 1) + c;
      if (col >= ffn) continue;
      const float4 a = sum(r, c), u = sum(r, c + BN / 2);
      auto act = [](float x) {
        if (EPI == GT_EW_SILU) return x / (1.f + __expf(-x));
        return 0.5f * x * (1.f + tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x)));
      };
      put(maps.cp[0], ffn, m0 + r, col, ffn, a, 0);
      put(maps.cp[1], ffn, m0 + r, col, ffn, u, 0);
      put(maps.cp[2], ffn, m0 + r, col, ffn, make_float4(act(a.x) * u.x, act(a.y) * u.y, act(a.z) * u.z, act(a.w) * u.w), 0);
    }
  } else if (EPI == EPI_ROPE && maps.g_rope[g]) {
    // heads of 64 columns, BN a multiple of 64: quads j and j + 32 of a head are rotated together
    for (int q = z * S::THREADS + threadIdx.x; q < mrows * (BN / 8); q += ksplit * S::THREADS) {
      const int r = q / (BN / 8), e = q % (BN / 8), c = (e / 8) * 64 + (e % 8) * 4;
      if (n0 + c >= N) continue;
      const float4* tab = reinterpret_cast<const float4*>(maps.rope_tab + (size_t)((m0 + r) % maps.rope_period) * 32 + (e % 8) * 4);
      const float4 a = sum(r, c), b = sum(r, c + 32), t0 = __ldg(tab), t1 = __ldg(tab + 1);   // (cos, sin) of four pairs
      put(C, N, m0 + r, n0 + c, N, make_float4(a.x * t0.x - b.x * t0.y, a.y * t0.z - b.y * t0.w, a.z * t1.x - b.z * t1.y, a.w * t1.z - b.w * t1.w), accum);
      put(C, N, m0 + r, n0 + c + 32, N, make_float4(a.x * t0.y + b.x * t0.x, a.y * t0.w + b.y * t0.z, a.z * t1.y + b.z * t1.x, a.w * t1.w + b.w * t1.z), accum);
    }
  } else {
    const int end = mrows * (BN / 4), step = ksplit * S::THREADS;
    for (int q = z * S::THREADS + threadIdx.x; q < end; q += 2 * step) {     // two quads at a time, their loads together
      const int q1 = q + step < end ? q + step : q;
      const int r = q / (BN / 4), c = (q % (BN / 4)) * 4, r1 = q1 / (BN / 4), c1 = (q1 % (BN / 4)) * 4;
      const float4 v = sum(r, c), v1 = sum(r1, c1);
      if (n0 + c < N) put(C, N, m0 + r, n0 + c, N, v, accum);
      if (q1 != q && n0 + c1 < N) put(C, N, m0 + r1, n0 + c1, N, v1, accum);
    }
  }
  __syncwarp();
  if (ksplit > 1) cluster_sync_all();                 // nobody leaves while its tile may still be read
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
int* g_flag[64] = {};

template <bool A_K, bool B_K, int BN, int EPI>
gt_status launch_small(gt_ctx* ctx, const PartMaps& maps, long tiles, int M, int N, int accum, int ksplit, float out_scale) {
  auto kern = gemm_tf32_small_kernel<A_K, B_K, BN, EPI>;
  using S = SmallSmem<BN>;
  static bool attr_set[64] = {};
  if (!attr_set[ctx->device]) {
    GT_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::TOTAL));
    attr_set[ctx->device] = true;
  }
  GT_CUDA(ctx, gt_launch(ctx, ksplit, kern, dim3((unsigned)(tiles * ksplit)), S::THREADS, S::TOTAL, maps, M, N, accum, ksplit, out_scale, g_flag[ctx->device]));
  GT_LAUNCHED(ctx, "gemm_tf32_small_kernel");
  return GT_OK;
}

template <int BN, int EPI = 0>
gt_status launch_small_kind(gt_ctx* ctx, int kind, const PartMaps& maps, long tiles, int M, int N, int accum, int ksplit, float out_scale) {
  if (kind == GT_GEMM_NT) return launch_small<true, true, BN, EPI>(ctx, maps, tiles, M, N, accum, ksplit, out_scale);
  if constexpr (EPI == 0) {
    if (kind == GT_GEMM_NN) return launch_small<true, false, BN, EPI>(ctx, maps, tiles, M, N, accum, ksplit, out_scale);
    return launch_small<false, false, BN, EPI>(ctx, maps, tiles, M, N, accum, ksplit, out_scale);
  }
  return GT_ERR_ARG;
}

// CTAs that can be resident at once, one per SM, when they come in clusters of `c` (clusters lie inside a group of SMs, and the
// groups are not all of one size).
int cluster_room(gt_ctx* ctx, int c) {
  static int room[64][9] = {};
  int& r = room[ctx->device][c];
  if (r == 0) {
    auto kern = gemm_tf32_small_kernel<true, true, 128, 0>;
    int n = 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(ctx->sm_count / c * c), 1, 1);
    cfg.blockDim = dim3(SmallSmem<128>::THREADS, 1, 1);
    cfg.dynamicSmemBytes = SmallSmem<128>::TOTAL;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = c;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SmallSmem<128>::TOTAL) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    r = n > 0 ? n * c : c;
    if (gt_env("GT_GEMM_TILE")) fprintf(stderr, "[gguftrain] resident CTAs in clusters of %d: %d\n", c, r);
  }
  return r;
}

// Predicted times in microseconds, fitted to 919 launches of 154 products (16 to 16384 rows, outputs 576 to 49152 wide, depths
// 576 to 49152; the fit's rms error is 4 %): a launch costs a fixed part and, per wave of tiles, its K blocks and what of
// the epilogue is not hidden. A K block costs the larger of its shared-memory traffic (written once by TMA, read once per 128-row half by the MMAs,
// 128 B/clk for all of it) and its MMAs; MN-major operands cost CTA pairs more than that.
struct Shape { int mt, bn; double per_kb[3], epilogue; };   // mt 1, 2: 128 / 256 rows on one CTA; mt 3: 256 rows on a CTA pair; per_kb by layout
constexpr Shape SHAPES[6] = {{1, 192, {0.345, 0.400, 0.465}, 1.67}, {1, 128, {0.312, 0.358, 0.429}, 0.76}, {2, 256, {0.651, 0.631, 0.638}, 5.35},
                             {2, 192, {0.550, 0.543, 0.621}, 3.90}, {3, 192, {0.330, 0.392, 0.502}, 0.89}, {3, 256, {0.334, 0.428, 0.529}, 1.75}};
constexpr double FIXED = 4.3, FIXED_PAIR = 6.1;   // what a launch costs beside its tiles
constexpr double SLICE = 0.52;                    // per wave when slices of K are added up in L2
constexpr double CLEAR = 4.6;                     // the clear before a launch whose slices meet in L2: itself, and a node that nothing overlaps
double shape_cost(const Shape& h, int kind, long units, long workers, int kblocks, int ks) {
  return (h.mt == 3 ? FIXED_PAIR : FIXED) + gt_cdiv(units, workers) * (gt_cdiv(kblocks, ks) * h.per_kb[kind] + h.epilogue + (ks > 1 ? SLICE : 0.0));
}

// The best shape of the one-tile-per-CTA kernel for `tiles(bn)` tiles of 128 x bn and its predicted time. A K block costs
// its shared-memory traffic; resident CTAs of an SM share that. (Measured in cycles, CYCLE us each.)
constexpr double SMALL_FIXED = 10500.0, SMALL_WAVE = 8500.0, CYCLE = 0.00067;
struct SmallPick { int bn = 0, ks = 1; double cost = 1e30; };
template <typename F>
SmallPick pick_small(gt_ctx* ctx, int kind, int kblocks, F tiles, int min_bn) {
  const long workers = ctx->sm_count - ctx->sm_reserved;
  SmallPick p;
  for (int bn = min_bn; bn <= 128; bn *= 2) {
    const long n = tiles(bn);
    if (n > 4 * workers) continue;
    const double per_kb = 2.0 * (BM1 + bn) * BK * 4 / 128.0 * (kind == GT_GEMM_NT ? 1.0 : 1.25);   // (MN-major stages come in more copies)
    for (int ks = 1; ks <= 8 && ks <= kblocks; ks++) {
      const int per = gt_cdiv(kblocks, ks);
      if ((long)(ks - 1) * per >= kblocks) continue;   // (an empty slice)
      const long room = ks == 1 ? workers : max((long)ks, (long)cluster_room(ctx, ks) - ctx->sm_reserved);   // two CTAs of up to 64 columns share an SM
      const double share = n * ks > room && bn <= 64 ? 2.0 : 1.0;
      const double waves = ceil((double)(n * ks) / (room * share));
      const double cost = waves * (per * per_kb * share + SMALL_WAVE) + (SMALL_FIXED - SMALL_WAVE) + (share > 1.0 ? 5000.0 : 0.0) + 6.0 * bn + (ks > 1 ? 2000.0 : 0.0);
      if (cost * CYCLE < p.cost) { p.cost = cost * CYCLE; p.bn = bn; p.ks = ks; }
    }
  }
  return p;
}

template <bool A_K, bool B_K, int BN, int MT, int GLU = 0>
gt_status launch(gt_ctx* ctx, const PartMaps& maps, long ntiles, int tma_store, float* c, int M, int N, int accum, int ksplit,
                 int batch, float out_scale) {
  auto kern = gemm_tf32_kernel<A_K, B_K, BN, MT, GLU>;
  using S = Smem<BN, MT, EpiSub<MT, GLU>::N>;
  static bool attr_set[64] = {};
  if (!attr_set[ctx->device]) {
    GT_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::TOTAL));
    attr_set[ctx->device] = true;
  }
  dim3 grid((unsigned)min((long)(ctx->sm_count - ctx->sm_reserved), ntiles), 1, 1);
  GT_CUDA(ctx, gt_launch(ctx, 1, kern, grid, S::THREADS, S::TOTAL, maps, c, M, N, accum, ksplit, tma_store, batch, out_scale, g_flag[ctx->device]));
  GT_LAUNCHED(ctx, "gemm_tf32_kernel");
  return GT_OK;
}

template <bool A_K, bool B_K, int BN, int GLU = 0>
gt_status launch_pair(gt_ctx* ctx, const PartMaps& maps, long ntiles, int tma_store, float* c, int M, int N, int accum, int ksplit,
                      int batch, int npairs, float out_scale) {
  auto kern = gemm_tf32_pair_kernel<A_K, B_K, BN, GLU>;
  using S = SmemPair<BN, GLU>;
  static bool attr_set[64] = {};
  if (!attr_set[ctx->device]) {
    GT_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::TOTAL));
    attr_set[ctx->device] = true;
  }
  dim3 grid(2u * (unsigned)min((long)npairs, ntiles), 1, 1);
  GT_CUDA(ctx, gt_launch(ctx, 1, kern, grid, S::THREADS, S::TOTAL, maps, c, M, N, accum, ksplit, tma_store, batch, out_scale, g_flag[ctx->device]));
  GT_LAUNCHED(ctx, "gemm_tf32_pair_kernel");
  return GT_OK;
}

template <int BN>
gt_status launch_pair_kind(gt_ctx* ctx, int kind, const PartMaps& maps, long ntiles, int tma_store, float* c, int M, int N, int accum,
                           int ksplit, int batch, int npairs, float out_scale) {
  if (kind == GT_GEMM_NT) return launch_pair<true, true, BN>(ctx, maps, ntiles, tma_store, c, M, N, accum, ksplit, batch, npairs, out_scale);
  if (kind == GT_GEMM_NN) return launch_pair<true, false, BN>(ctx, maps, ntiles, tma_store, c, M, N, accum, ksplit, batch, npairs, out_scale);
  return launch_pair<false, false, BN>(ctx, maps, ntiles, tma_store, c, M, N, accum, ksplit, batch, npairs, out_scale);
}

// CTA pairs that can be resident at once (two neighbouring SMs each); 0 when the device cannot run the pair kernel.
int pair_capacity(gt_ctx* ctx) {
  static int cap[64];
  static bool known[64] = {};
  if (!known[ctx->device]) {
    auto kern = gemm_tf32_pair_kernel<true, true, 192>;
    int n = 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2u * (unsigned)ctx->sm_count, 1, 1);
    cfg.blockDim = dim3(SmemPair<192>::THREADS, 1, 1);
    cfg.dynamicSmemBytes = SmemPair<192>::TOTAL;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SmemPair<192>::TOTAL) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    cap[ctx->device] = n;
    known[ctx->device] = true;
    if (gt_env("GT_GEMM_TILE")) fprintf(stderr, "[gguftrain] resident CTA pairs: %d\n", n);
  }
  return cap[ctx->device];
}

int pair_workers(gt_ctx* ctx) { return max(0, pair_capacity(ctx) - (ctx->sm_reserved + 1) / 2); }

template <int BN, int MT>
gt_status launch_kind(gt_ctx* ctx, int kind, const PartMaps& maps, long ntiles, int tma_store, float* c, int M, int N, int accum,
                      int ksplit, int batch, float out_scale) {
  if (kind == GT_GEMM_NT) return launch<true, true, BN, MT>(ctx, maps, ntiles, tma_store, c, M, N, accum, ksplit, batch, out_scale);
  if (kind == GT_GEMM_NN) return launch<true, false, BN, MT>(ctx, maps, ntiles, tma_store, c, M, N, accum, ksplit, batch, out_scale);
  return launch<false, false, BN, MT>(ctx, maps, ntiles, tma_store, c, M, N, accum, ksplit, batch, out_scale);
}

}  // namespace

namespace {
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn g_encode = nullptr;
std::once_flag g_encode_once;

EncodeTiledFn encode_fn() {
  std::call_once(g_encode_once, [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) == cudaSuccess && qres == cudaDriverEntryPointSuccess)
      g_encode = (EncodeTiledFn)fn;
  });
  return g_encode;
}

// 2-D f32 tensor [outer, inner] with `inner` contiguous; box [box_outer, 32]; out-of-range reads give 0.
// kmajor: the tile's rows are K runs (128-byte swizzle); else its rows are MN runs (128-byte swizzle, 32-byte atoms).
}  // namespace

namespace {
// Encoded maps are a pure function of their arguments, and a training or decoding loop asks for the same ones again and
// again (weights stay where they are, recycled activations come back to the same blocks): a few thousand are kept per thread.
struct MapKey {
  uint64_t v[8];
  bool operator==(const MapKey& o) const { return memcmp(v, o.v, sizeof v) == 0; }
};
struct WordsHash {
  template <typename K>
  size_t operator()(const K& k) const {
    uint64_t h = 0x9e3779b97f4a7c15ull;
    for (auto x : k.v) h = (h ^ (uint64_t)x) * 0xff51afd7ed558ccdull, h ^= h >> 29;
    return (size_t)h;
  }
};
template <typename F>
bool cached_map(CUtensorMap* map, const MapKey& key, F encode) {
  thread_local std::unordered_map<MapKey, CUtensorMap, WordsHash> maps;
  auto it = maps.find(key);
  if (it == maps.end()) {
    if (!encode(map)) return false;
    if (maps.size() >= 4096) maps.clear();
    maps.emplace(key, *map);
    return true;
  }
  *map = it->second;
  return true;
}
}  // namespace

bool tc::make_map_3d(CUtensorMap* map, const float* ptr, uint64_t inner, uint64_t outer, uint64_t batch, uint64_t row_pitch_elems,
                     uint64_t batch_stride_elems, uint32_t box_outer, bool kmajor) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return false;
  cuuint64_t dims[3] = {inner, outer, batch};
  cuuint64_t strides[2] = {row_pitch_elems * sizeof(float), batch_stride_elems * sizeof(float)};
  cuuint32_t box[3] = {32, box_outer, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return cached_map(map, {{(uint64_t)(uintptr_t)ptr, inner, outer, batch, row_pitch_elems, batch_stride_elems, box_outer, kmajor ? 1ull : 2ull}}, [&](CUtensorMap* map) { return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             kmajor ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS; });
}

bool tc::make_map_atoms(CUtensorMap* map, const float* ptr, uint64_t inner, uint64_t outer, uint64_t row_pitch_elems,
                        uint32_t box_outer, uint32_t atoms, bool kmajor) {
  EncodeTiledFn enc = encode_fn();
  if (!enc || inner % 32 != 0) return false;
  cuuint64_t dims[3] = {32, outer, inner / 32};
  cuuint64_t strides[2] = {row_pitch_elems * sizeof(float), 32 * sizeof(float)};
  cuuint32_t box[3] = {32, box_outer, atoms};
  cuuint32_t estr[3] = {1, 1, 1};
  return cached_map(map, {{(uint64_t)(uintptr_t)ptr, inner, outer, atoms, row_pitch_elems, 0, box_outer, kmajor ? 3ull : 4ull}}, [&](CUtensorMap* map) { return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             kmajor ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS; });
}

bool tc::make_map_2d(CUtensorMap* map, const float* ptr, uint64_t inner, uint64_t outer, uint64_t row_pitch_elems,
                     uint32_t box_outer, bool kmajor) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return false;
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {row_pitch_elems * sizeof(float)};
  cuuint32_t box[2] = {32, box_outer};
  cuuint32_t estr[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             kmajor ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int* tc::device_flag(gt_ctx* ctx) {
  if (ctx->device < 0 || ctx->device >= 64) return nullptr;
  if (!g_flag[ctx->device]) {
    if (ctx->capturing) return nullptr;
    if (cudaMalloc(&g_flag[ctx->device], 65536) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    cudaMemsetAsync(g_flag[ctx->device], 0, 65536, ctx->stream);
  }
  return g_flag[ctx->device];
}

// Self-test of the bounded wait every pipeline kernel relies on: one thread waits on an mbarrier that nothing will
// ever arrive on, with a caller-chosen limit instead of the kernels' 2 s, gives up when the limit has passed, raises
// the device flag like a pipeline kernel would (code 99) and returns. Nothing spins beyond the limit and the context
// stays usable; the next gt_sync reports the expiry.
__global__ void bounded_wait_selftest_kernel(unsigned long long limit_ns, int* __restrict__ flag) {
  __shared__ __align__(8) unsigned long long bar_storage;
  const uint32_t bar = smem_u32(&bar_storage);
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    const uint64_t t0 = gtimer();
    bool arrived = mbar_try(bar, 0);
    while (!arrived && gtimer() - t0 <= limit_ns) arrived = mbar_try(bar, 0);
    if (!arrived) atomicExch(flag, 99);
  }
}

extern "C" gt_status gt_selftest_bounded_wait(gt_ctx* ctx, int32_t limit_us) {
  GT_DRAIN(ctx);
  GT_REQUIRE(ctx, limit_us >= 1 && limit_us <= 1000000, "gt_selftest_bounded_wait: limit %d us (1..1000000)", limit_us);
  if (ctx->capturing) return gt_fail(ctx, GT_ERR_STATE, "gt_selftest_bounded_wait inside a graph capture");
  int* flag = device_flag(ctx);
  if (!flag) return gt_fail(ctx, GT_ERR_CUDA, "gt_selftest_bounded_wait: cannot allocate the device flag");
  bounded_wait_selftest_kernel<<<1, 32, 0, ctx->stream>>>((unsigned long long)limit_us * 1000ull, flag);
  GT_LAUNCHED(ctx, "bounded_wait_selftest_kernel");
  return GT_OK;
}

// The device flag the kernels raise when a bounded wait expires: gt_sync reads it with its other latched words.
int* gt_gemm_tc_word(gt_ctx* ctx) { return g_flag[ctx->device]; }
gt_status gt_gemm_tc_answer(gt_ctx* ctx, int code) {
  if (code == 0) return GT_OK;
  cudaMemsetAsync(g_flag[ctx->device], 0, sizeof(int), ctx->stream);
  return gt_fail(ctx, GT_ERR_CUDA, "tensor-core kernel: a pipeline wait expired (code %d); results of that launch are invalid", code);
}

struct Plan { int mt = 0, bn = 0, ks = 1; bool small = false; };   // mt 0: not for the tensor cores
struct PlanKey {
  int v[8 + MAX_PARTS] = {};
  bool operator==(const PlanKey& o) const { return memcmp(v, o.v, sizeof v) == 0; }
};
static std::unordered_map<PlanKey, Plan, WordsHash>& plan_cache() {
  thread_local std::unordered_map<PlanKey, Plan, WordsHash> plans;
  if (plans.size() > 4096) plans.clear();
  return plans;
}
static Plan choose_plan(gt_ctx* ctx, int kind, int accum, int M, int N, int kblocks, int batch, const char* force, const char* ds) {
  // Tile shape and split-K factor: the cheapest under the model above.
  const bool deep_split = !(ds && ds[0] == '0');
  const int npairs = pair_workers(ctx);
  int best = -1, ksplit = 1;
  double best_cost = 1e30;
  int best_deep = 0, ks_deep = 1;      // the best choice that also cuts a product with enough tiles along K (see below)
  double cost_deep = 1e30;
  for (int i = 0; i < 6; i++) {
    const Shape& h = SHAPES[i];
    const int bm = h.mt == 1 ? BM1 : 2 * BM1;
    if (h.mt == 3 && npairs < 8) continue;
    if (force) {
      int fm = 0, fb = 0;
      if (sscanf(force, "%d,%d", &fm, &fb) == 2 && (fm != h.mt || fb != h.bn)) continue;
    }
    const long workers = h.mt == 3 ? npairs : ctx->sm_count - ctx->sm_reserved;
    const long tiles = (long)gt_cdiv(N, h.bn) * gt_cdiv(M, bm) * batch;
    // split K when the output has few tiles and K is deep (dW: K = rows); partial sums meet in L2 with f32 adds
    int ks = 1;
    if (tiles < workers && kblocks >= 16) {
      ks = (int)min((long)(workers / tiles), (long)(kblocks / 8));
      if (ks < 1) ks = 1;
    }
    const double cost = shape_cost(h, kind, tiles * ks, workers, kblocks, ks) + (ks > 1 && !accum ? CLEAR : 0.0);
    if (cost < best_cost) { best_cost = cost; best = i; ksplit = ks; }
    // A deep product whose tiles fill the SMs unevenly (the readout's dX: 384 tiles of 128 x 192 on 148 SMs are 2.6
    // waves, run as 3) may be cut along K as well when that evens the waves out: as 192 tiles of 256 x 192 in three
    // slices it is 576 units = 3.9 waves of a third of the length. The clear before it and the reduce-adds are
    // charged; the candidate is taken after the loop only if it is predicted well ahead. Measured at rows 16384: the
    // readout's dX (K 49152) 1890 -> 1292 us, dX of gate and up (K 3072) 128 -> 106 us; at K 1536 the same choice
    // measured slower (60.5 -> 67.9 us), hence the depth limit of 64 K blocks.
    if (ks == 1 && tiles >= workers && kblocks >= 64 && deep_split) {
      double best_w = (double)gt_cdiv(tiles, workers);
      int k2best = 1;
      for (int k2 = 2; k2 <= 4; k2++) {
        const double w2 = (double)gt_cdiv(tiles * k2, workers) / k2;
        if (w2 < best_w - 0.05) { best_w = w2; k2best = k2; }
      }
      if (k2best > 1) {
        const double c2 = shape_cost(h, kind, tiles * k2best, workers, kblocks, k2best) + CLEAR + 2.0;
        if (c2 < cost_deep) { cost_deep = c2; best_deep = i; ks_deep = k2best; }
      }
    }
  }
  if (cost_deep < 0.92 * best_cost) { best_cost = cost_deep; best = best_deep; ksplit = ks_deep; }
  int fm = -1, fb = 0;
  if (force && sscanf(force, "%d,%d", &fm, &fb) < 1) fm = -1;
  SmallPick small;
  if (fm <= 0)
    small = pick_small(ctx, kind, kblocks, [&](int b) { return (fm == 0 && fb && b != fb) ? 1l << 40 : (long)gt_cdiv(N, b) * gt_cdiv(M, BM1) * batch; }, 32);
  const bool use_small = small.bn && small.cost < best_cost;
  if (best < 0 && !use_small) return {};
  if (use_small) return {1, small.bn, small.ks, true};
  return {SHAPES[best].mt, SHAPES[best].bn, ksplit, false};
}

// `batch` independent products of the same shape, matrix i of each operand `M*K`, `N*K`, `M*N` elements after matrix i-1.
// With nparts > 1 (batch 1 only): c (+)= sum_p op(a_p).op(b_p), every product of the same kind, K_p deep.
static gt_status gemm_tc_dispatch(gt_ctx* ctx, int kind, int accum, int M, int N, int nparts, const int* Ks, const float* const* as,
                                  const float* const* bs, float* c, int batch, float alpha, bool* handled) {
  *handled = false;
  if (batch < 1 || nparts < 1 || nparts > MAX_PARTS || (nparts > 1 && batch != 1)) return GT_OK;
  // Small or oddly aligned products stay on the f32 kernel: TMA needs 16-byte row pitches and bases.
  const bool a_k = kind != GT_GEMM_TN, b_k = kind == GT_GEMM_NT;
  if (M < 16 || N < 16 || Ks[0] < 16) return GT_OK;   // (rows of a tile past M or N are zero-filled by TMA and clipped on store)
  if (((uintptr_t)c) & 15) return GT_OK;
  int kblocks = 0;
  for (int p = 0; p < nparts; p++) {
    const int a_inner = a_k ? Ks[p] : M, b_inner = b_k ? Ks[p] : N;
    if (Ks[p] < 1 || (a_inner & 3) || (b_inner & 3) || ((((uintptr_t)as[p]) | ((uintptr_t)bs[p])) & 15)) return GT_OK;
    kblocks += gt_cdiv(Ks[p], BK);
  }
  if (ctx->device < 0 || ctx->device >= 64) return GT_OK;
  if (!device_flag(ctx)) return GT_OK;
  const char* force = gt_env("GT_GEMM_TILE");   // "mt,bn": forces one tile shape (read per call so tests can switch it); mt 0: one tile per CTA
  const char* ds = gt_env("GT_GEMM_DEEP_SPLIT");   // "0": never cut a product that already fills the SMs along K (for comparison)
  // the choice is made once per shape
  Plan plan;
  PlanKey key = {{kind, accum ? 1 : 0, M, N, batch, ctx->device, ctx->sm_reserved, nparts}};
  for (int p = 0; p < nparts; p++) key.v[8 + p] = Ks[p];
  auto& plans = plan_cache();
  auto found = force || ds ? plans.end() : plans.find(key);
  if (found != plans.end()) plan = found->second;
  else {
    plan = choose_plan(ctx, kind, accum, M, N, kblocks, batch, force, ds);
    if (!force && !ds) plans.emplace(key, plan);
  }
  if (!plan.mt) return GT_OK;
  const bool use_small = plan.small;
  const int ksplit = plan.ks, mt = plan.mt, bn = plan.bn;
  const int a_box = mt == 2 ? 2 * BM1 : BM1, b_box = mt == 3 ? bn / 2 : bn;   // rows one TMA copy brings
  PartMaps maps;
  maps.nparts = nparts;
  int kb_sum = 0;
  for (int p = 0; p < nparts; p++) {
    const int K = Ks[p];
    const uint64_t sa = (uint64_t)M * K, sb = (uint64_t)N * K;
    const bool oka = a_k ? make_map_3d(&maps.a[p], as[p], K, M, batch, K, sa, a_box, true) : make_map_3d(&maps.a[p], as[p], M, K, batch, M, sa, BK, false);
    const bool okb = b_k ? make_map_3d(&maps.b[p], bs[p], K, N, batch, K, sb, b_box, true) : make_map_3d(&maps.b[p], bs[p], N, K, batch, N, sb, BK, false);
    if (!oka || !okb) return GT_OK;
    kb_sum += gt_cdiv(K, BK);
    maps.kb_end[p] = kb_sum;
  }
  for (int p = nparts; p < MAX_PARTS; p++) { maps.a[p] = maps.a[0]; maps.b[p] = maps.b[0]; maps.kb_end[p] = kb_sum; }
  // the output goes through TMA (32x32 blocks of whole 128-byte rows) whenever its row pitch allows a tensor map
  const uint64_t sc = (uint64_t)M * N;
  maps.ngroups = 1;
  if (use_small) {
    maps.cp[0] = c;
    const long tiles = (long)gt_cdiv(N, bn) * gt_cdiv(M, BM1) * batch;
    gt_status s = bn == 32 ? launch_small_kind<32>(ctx, kind, maps, tiles, M, N, accum, ksplit, alpha * TRUNC_COMP)
                : bn == 64 ? launch_small_kind<64>(ctx, kind, maps, tiles, M, N, accum, ksplit, alpha * TRUNC_COMP)
                           : launch_small_kind<128>(ctx, kind, maps, tiles, M, N, accum, ksplit, alpha * TRUNC_COMP);
    if (s) return s;
    *handled = true;
    return GT_OK;
  }
  maps.c[0] = maps.a[0];
  const int tma_store = ((N & 3) == 0 && make_map_3d(&maps.c[0], c, N, M, batch, N, sc, 32, true)) ? 1 : 0;
  for (int p = 1; p < MAX_PARTS; p++) maps.c[p] = maps.c[0];
  for (int p = 0; p < MAX_PARTS; p++) { maps.gM[p] = M; maps.gN[p] = N; maps.g_accum[p] = accum; maps.unit_end[p] = 0; }
  if (ksplit > 1 && !accum) GT_CUDA(ctx, cudaMemsetAsync(c, 0, sizeof(float) * (size_t)M * N * batch, ctx->stream));
  const float out_scale = alpha * TRUNC_COMP;
  const long ntiles = (long)gt_cdiv(N, bn) * gt_cdiv(M, mt == 1 ? BM1 : 2 * BM1) * ksplit * batch;
  gt_status s;
  const int npairs = pair_workers(ctx);
  if (mt == 3 && bn == 192) s = launch_pair_kind<192>(ctx, kind, maps, ntiles, tma_store, c, M, N, accum, ksplit, batch, npairs, out_scale);
  else if (mt == 3) s = launch_pair_kind<256>(ctx, kind, maps, ntiles, tma_store, c, M, N, accum, ksplit, batch, npairs, out_scale);
  else if (mt == 1 && bn == 192) s = launch_kind<192, 1>(ctx, kind, maps, ntiles, tma_store, c, M, N, accum, ksplit, batch, out_scale);
  else if (mt == 1) s = launch_kind<128, 1>(ctx, kind, maps, ntiles, tma_store, c, M, N, accum, ksplit, batch, out_scale);
  else if (bn == 256) s = launch_kind<256, 2>(ctx, kind, maps, ntiles, tma_store, c, M, N, accum, ksplit, batch, out_scale);
  else s = launch_kind<192, 2>(ctx, kind, maps, ntiles, tma_store, c, M, N, accum, ksplit, batch, out_scale);
  if (s) return s;
  *handled = true;
  return GT_OK;
}

struct GroupKey {
  int v[6 + 3 * MAX_PARTS] = {};
  bool operator==(const GroupKey& o) const { return memcmp(v, o.v, sizeof v) == 0; }
};
static std::unordered_map<GroupKey, Plan, WordsHash>& group_cache() {
  thread_local std::unordered_map<GroupKey, Plan, WordsHash> plans;
  if (plans.size() > 4096) plans.clear();
  return plans;
}
static Plan choose_group_plan(gt_ctx* ctx, int kind, int ngroups, const int* Ms, const int* Ns, int kblocks, const int* accums, bool any_rope,
                              const char* force) {
  int clears = 0;      // (one clear per product that does not accumulate)
  for (int g = 0; g < ngroups; g++) clears += !accums[g];
  // The tile shape and the split-K factor (one for the whole launch) with the least predicted time, among slices of at
  // least 8 K blocks and at most 8 partial sums per output element.
  int best = -1, best_ks = 1;
  double best_cost = 1e30;
  const int npairs = pair_workers(ctx);
  for (int i = 0; i < 6; i++) {
    const Shape& h = SHAPES[i];
    if ((h.mt == 3 && npairs < 8) || h.bn == 128 || (any_rope && h.mt == 2)) continue;
    if (force) { int fm = 0, fb = 0; if (sscanf(force, "%d,%d", &fm, &fb) == 2 && (fm != h.mt || fb != h.bn)) continue; }
    long tiles = 0;
    for (int g = 0; g < ngroups; g++) tiles += (long)gt_cdiv(Ns[g], h.bn) * gt_cdiv(Ms[g], h.mt == 1 ? BM1 : 2 * BM1);
    const long workers = h.mt == 3 ? npairs : ctx->sm_count - ctx->sm_reserved;
    for (int ks = 1; ks <= 8 && (ks == 1 || kblocks / ks >= 8); ks++) {
      const double cost = shape_cost(h, kind, tiles * ks, workers, kblocks, ks) + (ks > 1 ? clears * CLEAR : 0.0);
      if (cost < best_cost) { best_cost = cost; best = i; best_ks = ks; }
    }
  }
  int fm = -1, fb = 0;
  if (force && sscanf(force, "%d,%d", &fm, &fb) < 1) fm = -1;
  // (outputs that could be whole heads take the tiles a rotation needs whether it is applied or not: its values then do not
  // depend on where it runs)
  bool heads64 = kind == GT_GEMM_NT;
  for (int g = 0; g < ngroups; g++) heads64 = heads64 && (Ns[g] & 63) == 0;
  SmallPick small;
  if (fm <= 0)
    small = pick_small(ctx, kind, kblocks, [&](int b) {
      if (fm == 0 && fb && b != fb) return 1l << 40;
      long n = 0;
      for (int g = 0; g < ngroups; g++) n += (long)gt_cdiv(Ns[g], b) * gt_cdiv(Ms[g], BM1);
      return n;
    }, any_rope || heads64 ? 64 : 32);
  const bool use_small = small.bn && small.cost < best_cost;
  if (best < 0 && !use_small) return {};
  return use_small ? Plan{1, small.bn, small.ks, true} : Plan{SHAPES[best].mt, SHAPES[best].bn, best_ks, false};
}

// ngroups independent products of one layout and one K, each with its own operands, extents and accumulate flag, as
// ONE launch: the weight gradients dW_g = dY_g^T.X_g of several projections (K = rows for all of them). Their tiles
// are so few per product that each would need its own split-K launch with its own tail; together they fill the SMs.
static gt_status gemm_tc_grouped(gt_ctx* ctx, int kind, int ngroups, const int* Ms, const int* Ns, int K, const float* const* as,
                                 const float* const* bs, float* const* cs, const int* accums, const int* ropes, const float2* rope_tab,
                                 int rope_period, float alpha, bool* handled) {
  *handled = false;
  if (ngroups < 2 || ngroups > MAX_PARTS || K < 16) return GT_OK;
  bool any_rope = false;
  for (int g = 0; ropes && g < ngroups; g++) {
    if (!ropes[g]) continue;
    if (kind != GT_GEMM_NT || (Ns[g] & 63) || !rope_tab || rope_period <= 0) return GT_OK;
    any_rope = true;
  }
  const bool a_k = kind != GT_GEMM_TN, b_k = kind == GT_GEMM_NT;
  for (int g = 0; g < ngroups; g++) {
    const int a_inner = a_k ? K : Ms[g], b_inner = b_k ? K : Ns[g];
    if (Ms[g] < 16 || Ns[g] < 16 || (a_inner & 3) || (b_inner & 3) || (Ns[g] & 3)) return GT_OK;
    if ((((uintptr_t)as[g]) | ((uintptr_t)bs[g]) | ((uintptr_t)cs[g])) & 15) return GT_OK;
  }
  if (ctx->device < 0 || ctx->device >= 64 || !device_flag(ctx)) return GT_OK;
  const int kblocks = gt_cdiv(K, BK);
  const char* force = gt_env("GT_GEMM_TILE");
  GroupKey key = {{kind, K, ngroups, any_rope ? 1 : 0, ctx->device, ctx->sm_reserved}};
  for (int g = 0; g < ngroups; g++) { key.v[6 + 3 * g] = Ms[g]; key.v[7 + 3 * g] = Ns[g]; key.v[8 + 3 * g] = accums[g] ? 1 : 0; }
  auto& plans = group_cache();
  auto found = force ? plans.end() : plans.find(key);
  Plan plan;
  if (found != plans.end()) plan = found->second;
  else {
    plan = choose_group_plan(ctx, kind, ngroups, Ms, Ns, kblocks, accums, any_rope, force);
    if (!force) plans.emplace(key, plan);
  }
  if (!plan.mt) return GT_OK;
  const bool use_small = plan.small;
  const int mt = plan.mt, ksplit = plan.ks, bm = mt == 1 ? BM1 : 2 * BM1, bn = plan.bn;
  const int a_box = mt == 2 ? 2 * BM1 : BM1, b_box = mt == 3 ? bn / 2 : bn;   // rows one TMA copy brings
  PartMaps maps;
  maps.nparts = 1;
  maps.ngroups = ngroups;
  int units = 0;
  for (int g = 0; g < ngroups; g++) {
    const int M = Ms[g], N = Ns[g];
    const bool oka = a_k ? make_map_3d(&maps.a[g], as[g], K, M, 1, K, (uint64_t)M * K, a_box, true) : make_map_3d(&maps.a[g], as[g], M, K, 1, M, (uint64_t)M * K, BK, false);
    const bool okb = b_k ? make_map_3d(&maps.b[g], bs[g], K, N, 1, K, (uint64_t)N * K, b_box, true) : make_map_3d(&maps.b[g], bs[g], N, K, 1, N, (uint64_t)N * K, BK, false);
    const bool okc = use_small || make_map_3d(&maps.c[g], cs[g], N, M, 1, N, (uint64_t)M * N, 32, true);
    if (!oka || !okb || !okc) return GT_OK;
    maps.cp[g] = cs[g];
    units += gt_cdiv(N, bn) * gt_cdiv(M, bm) * (use_small ? 1 : ksplit);
    maps.unit_end[g] = units;
    maps.gM[g] = M; maps.gN[g] = N; maps.g_accum[g] = accums[g];
    maps.g_rope[g] = any_rope ? ropes[g] : 0;
    maps.kb_end[g] = kblocks;
  }
  maps.rope_tab = rope_tab;
  maps.rope_period = rope_period;
  if (use_small) {
    const float scale = alpha * TRUNC_COMP;
    gt_status s = any_rope ? (bn == 64 ? launch_small_kind<64, EPI_ROPE>(ctx, kind, maps, units, 0, 0, 0, ksplit, scale)
                                       : launch_small_kind<128, EPI_ROPE>(ctx, kind, maps, units, 0, 0, 0, ksplit, scale))
                : bn == 32 ? launch_small_kind<32>(ctx, kind, maps, units, 0, 0, 0, ksplit, scale)
                : bn == 64 ? launch_small_kind<64>(ctx, kind, maps, units, 0, 0, 0, ksplit, scale)
                           : launch_small_kind<128>(ctx, kind, maps, units, 0, 0, 0, ksplit, scale);
    if (s) return s;
    *handled = true;
    return GT_OK;
  }
  for (int g = ngroups; g < MAX_PARTS; g++) {
    maps.a[g] = maps.a[0]; maps.b[g] = maps.b[0]; maps.c[g] = maps.c[0];
    maps.unit_end[g] = units; maps.gM[g] = Ms[0]; maps.gN[g] = Ns[0]; maps.g_accum[g] = accums[0]; maps.kb_end[g] = kblocks;
    maps.g_rope[g] = 0;
  }
  if (ksplit > 1)
    for (int g = 0; g < ngroups; g++)
      if (!accums[g]) GT_CUDA(ctx, cudaMemsetAsync(cs[g], 0, sizeof(float) * (size_t)Ms[g] * Ns[g], ctx->stream));
  gt_status s;
  const float scale = alpha * TRUNC_COMP;
  const int npairs = pair_workers(ctx);
  if (any_rope)
    s = mt == 1 ? launch<true, true, 192, 1, EPI_ROPE>(ctx, maps, units, 1, cs[0], Ms[0], Ns[0], accums[0], ksplit, 1, scale)
        : bn == 192 ? launch_pair<true, true, 192, EPI_ROPE>(ctx, maps, units, 1, cs[0], Ms[0], Ns[0], accums[0], ksplit, 1, npairs, scale)
                    : launch_pair<true, true, 256, EPI_ROPE>(ctx, maps, units, 1, cs[0], Ms[0], Ns[0], accums[0], ksplit, 1, npairs, scale);
  else
    s = mt == 1 ? launch_kind<192, 1>(ctx, kind, maps, units, 1, cs[0], Ms[0], Ns[0], accums[0], ksplit, 1, scale)
        : mt == 2 && bn == 256 ? launch_kind<256, 2>(ctx, kind, maps, units, 1, cs[0], Ms[0], Ns[0], accums[0], ksplit, 1, scale)
        : mt == 2 ? launch_kind<192, 2>(ctx, kind, maps, units, 1, cs[0], Ms[0], Ns[0], accums[0], ksplit, 1, scale)
        : bn == 192 ? launch_pair_kind<192>(ctx, kind, maps, units, 1, cs[0], Ms[0], Ns[0], accums[0], ksplit, 1, npairs, scale)
                    : launch_pair_kind<256>(ctx, kind, maps, units, 1, cs[0], Ms[0], Ns[0], accums[0], ksplit, 1, npairs, scale);
  if (s) return s;
  *handled = true;
  return GT_OK;
}

// gate = x.Wg^T, up = x.Wu^T and out = act(gate) * up as one launch (see the GLU form of the kernel).
gt_status gt_glu_linear_tc(gt_ctx* ctx, int op, int rows, int ffn, int in, const float* x, const float* wg, const float* wu, float* gate,
                           float* up, float* out, bool* handled) {
  *handled = false;
  if (rows < 16 || ffn < 96 || in < 16 || (in & 3) || (ffn & 3)) return GT_OK;
  if ((((uintptr_t)x) | ((uintptr_t)wg) | ((uintptr_t)wu) | ((uintptr_t)gate) | ((uintptr_t)up) | ((uintptr_t)out)) & 15) return GT_OK;
  if (ctx->device < 0 || ctx->device >= 64 || !device_flag(ctx)) return GT_OK;
  PartMaps maps;
  maps.nparts = 1;
  maps.ngroups = 1;
  const int kblocks = gt_cdiv(in, BK);
  const long workers = ctx->sm_count - ctx->sm_reserved;
  const int npairs = pair_workers(ctx);
  // (the unit's epilogue is not hidden: 3 us a 192 wide tile, 6.5 us a 256 wide pair of them)
  const Shape s1 = {1, 192, {SHAPES[0].per_kb[0]}, 5.0}, s3 = {3, 256, {SHAPES[5].per_kb[0]}, 5.5};
  double cost = shape_cost(s1, 0, (long)gt_cdiv(ffn, 96) * gt_cdiv(rows, BM1), workers, kblocks, 1);
  const double cost_pair = npairs < 8 ? 1e30 : shape_cost(s3, 0, (long)gt_cdiv(ffn, 128) * gt_cdiv(rows, 2 * BM1), npairs, kblocks, 1);
  bool pair = cost_pair < cost;
  cost = min(cost, cost_pair);
  const SmallPick small = pick_small(ctx, GT_GEMM_NT, kblocks, [&](int b) { return (long)gt_cdiv(ffn, b / 2) * gt_cdiv(rows, BM1); }, 32);
  const char* force = gt_env("GT_GEMM_TILE");
  if (small.bn && small.cost < cost && (!force || force[0] == '0')) {
    const int bn = small.bn;
    if (!make_map_3d(&maps.a[0], x, in, rows, 1, in, (uint64_t)rows * in, BM1, true) ||
        !make_map_3d(&maps.b[0], wg, in, ffn, 1, in, (uint64_t)ffn * in, bn / 2, true) ||
        !make_map_3d(&maps.b[1], wu, in, ffn, 1, in, (uint64_t)ffn * in, bn / 2, true))
      return GT_OK;
    maps.kb_end[0] = kblocks;
    maps.gN[0] = ffn;
    maps.cp[0] = gate; maps.cp[1] = up; maps.cp[2] = out;
    const long tiles = (long)gt_cdiv(ffn, bn / 2) * gt_cdiv(rows, BM1);
    const int n2 = 2 * gt_cdiv(ffn, bn / 2) * (bn / 2);
    gt_status s = GT_OK;
#define GT_SMALL_GLU(B) s = op == GT_EW_SILU ? launch_small<true, true, B, GT_EW_SILU>(ctx, maps, tiles, rows, n2, 0, small.ks, TRUNC_COMP) \
                                             : launch_small<true, true, B, GT_EW_GELU>(ctx, maps, tiles, rows, n2, 0, small.ks, TRUNC_COMP)
    if (bn == 32) GT_SMALL_GLU(32);
    else if (bn == 64) GT_SMALL_GLU(64);
    else GT_SMALL_GLU(128);
#undef GT_SMALL_GLU
    if (s) return s;
    *handled = true;
    return GT_OK;
  }
  if (force && !strcmp(force, "1,192")) pair = false;
  if (force && !strcmp(force, "3,256") && npairs >= 8) pair = true;
  const int bn = pair ? 256 : 192, bm = pair ? 2 * BM1 : BM1;
  bool ok = make_map_3d(&maps.a[0], x, in, rows, 1, in, (uint64_t)rows * in, BM1, true);
  ok = ok && make_map_3d(&maps.b[0], wg, in, ffn, 1, in, (uint64_t)ffn * in, bn / 2, true);
  ok = ok && make_map_3d(&maps.b[1], wu, in, ffn, 1, in, (uint64_t)ffn * in, bn / 2, true);
  ok = ok && make_map_3d(&maps.c[0], gate, ffn, rows, 1, ffn, (uint64_t)rows * ffn, 32, true);
  ok = ok && make_map_3d(&maps.c[1], up, ffn, rows, 1, ffn, (uint64_t)rows * ffn, 32, true);
  ok = ok && make_map_3d(&maps.c[2], out, ffn, rows, 1, ffn, (uint64_t)rows * ffn, 32, true);
  if (!ok) return GT_OK;
  for (int p = 0; p < MAX_PARTS; p++) {
    if (p > 0) maps.a[p] = maps.a[0];
    if (p > 1) maps.b[p] = maps.b[0];
    if (p > 2) maps.c[p] = maps.c[0];
    maps.kb_end[p] = kblocks; maps.gM[p] = rows; maps.gN[p] = 2 * ffn; maps.g_accum[p] = 0; maps.unit_end[p] = 0;
  }
  const int N2 = 2 * gt_cdiv(ffn, bn / 2) * (bn / 2);   // whole tiles of two halves; the maps clip at ffn
  const long ntiles = (long)gt_cdiv(N2, bn) * gt_cdiv(rows, bm);
  gt_status s;
  if (pair) s = op == GT_EW_SILU ? launch_pair<true, true, 256, GT_EW_SILU>(ctx, maps, ntiles, 1, out, rows, N2, 0, 1, 1, npairs, TRUNC_COMP)
                                 : launch_pair<true, true, 256, GT_EW_GELU>(ctx, maps, ntiles, 1, out, rows, N2, 0, 1, 1, npairs, TRUNC_COMP);
  else s = op == GT_EW_SILU ? launch<true, true, 192, 1, GT_EW_SILU>(ctx, maps, ntiles, 1, out, rows, N2, 0, 1, 1, TRUNC_COMP)
                            : launch<true, true, 192, 1, GT_EW_GELU>(ctx, maps, ntiles, 1, out, rows, N2, 0, 1, 1, TRUNC_COMP);
  if (s) return s;
  *handled = true;
  return GT_OK;
}

// One vocabulary span of the chunked readout loss: logits = hidden.w^T with their statistics or their gradient taken in
// the epilogue (see the kernel). `parts` is the number of (max, sum) pairs per row that the statistics form leaves in
// ce.part (two per 256 columns, or part of a tile of them).
gt_status gt_readout_tc(gt_ctx* ctx, int form, int rows, int n, int h, const float* hidden, const float* w, float* chunk, const CeArgs& ce,
                        int* parts, bool* handled) {
  *handled = false;
  const bool store = form != GT_READOUT_STATS;
  if (rows < 16 || n < 256 || h < 16 || (h & 3) || (store && (n & 3))) return GT_OK;
  if ((((uintptr_t)hidden) | ((uintptr_t)w) | ((uintptr_t)chunk)) & 15) return GT_OK;
  if (ctx->device < 0 || ctx->device >= 64 || !device_flag(ctx)) return GT_OK;
  const int kblocks = gt_cdiv(h, BK);
  const int npairs = pair_workers(ctx);
  // Spans with few tiles go through the product that cuts its contraction, and a pass that then finds them in L2. The CTA
  // pair hides most of this epilogue: 665 (statistics) and 763 us (gradient) at 8192 x 32768 x 1024, against 731 and 893 on
  // 256-row tiles of one CTA.
  const long tiles = (long)gt_cdiv(n, 256) * gt_cdiv(rows, 2 * BM1);
  if (npairs < 8 || 2 * tiles < npairs) return GT_OK;
  const char* force = gt_env("GT_GEMM_TILE");
  if (force && strcmp(force, "3,256")) return GT_OK;
  PartMaps maps;
  maps.nparts = maps.ngroups = 1;
  if (!make_map_3d(&maps.a[0], hidden, h, rows, 1, h, (uint64_t)rows * h, BM1, true) ||
      !make_map_3d(&maps.b[0], w, h, n, 1, h, (uint64_t)n * h, 128, true))
    return GT_OK;
  maps.c[0] = maps.a[0];
  if (store && !make_map_3d(&maps.c[0], chunk, n, rows, 1, n, (uint64_t)rows * n, 32, true)) return GT_OK;
  maps.kb_end[0] = kblocks;
  maps.ce = ce;
  *parts = gt_cdiv(n, 256) * PairSub<256, EPI_CE_STATS>::N;
  gt_status s = form == GT_READOUT_GRAD ? launch_pair<true, true, 256, EPI_CE_GRAD>(ctx, maps, tiles, 1, chunk, rows, n, 0, 1, 1, npairs, TRUNC_COMP)
                : form == GT_READOUT_BOTH ? launch_pair<true, true, 256, EPI_CE_BOTH>(ctx, maps, tiles, 1, chunk, rows, n, 0, 1, 1, npairs, TRUNC_COMP)
                     : launch_pair<true, true, 256, EPI_CE_STATS>(ctx, maps, tiles, 0, chunk, rows, n, 0, 1, 1, npairs, TRUNC_COMP);
  if (s) return s;
  *handled = true;
  return GT_OK;
}

gt_status gt_gemm_tc_grouped(gt_ctx* ctx, int kind, int ngroups, const int* Ms, const int* Ns, int K, const float* const* as,
                             const float* const* bs, float* const* cs, const int* accums, const int* ropes, const float2* rope_tab,
                             int rope_period, float alpha, bool* handled) {
  return gemm_tc_grouped(ctx, kind, ngroups, Ms, Ns, K, as, bs, cs, accums, ropes, rope_tab, rope_period, alpha, handled);
}

gt_status gt_gemm_tc_batched(gt_ctx* ctx, int kind, int accum, int M, int N, int K, const float* a, const float* b, float* c, int batch,
                             bool* handled) {
  return gemm_tc_dispatch(ctx, kind, accum, M, N, 1, &K, &a, &b, c, batch, 1.f, handled);
}

gt_status gt_gemm_tc(gt_ctx* ctx, int kind, int accum, int M, int N, int K, const float* a, const float* b, float* c, float alpha,
                     bool* handled) {
  return gemm_tc_dispatch(ctx, kind, accum, M, N, 1, &K, &a, &b, c, 1, alpha, handled);
}

gt_status gt_gemm_tc_multi(gt_ctx* ctx, int kind, int accum, int M, int N, int nparts, const int* Ks, const float* const* as,
                           const float* const* bs, float* c, bool* handled) {
  return gemm_tc_dispatch(ctx, kind, accum, M, N, nparts, Ks, as, bs, c, 1, 1.f, handled);
}
