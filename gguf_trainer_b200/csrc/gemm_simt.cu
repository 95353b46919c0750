// Strict-f32 matrix product: f32 loads, FFMA, f32 accumulate. This is the precision mode whose results
// must stay within 1e-5 relative L2 of the reference's f64-accumulating loops (src/model/autograd.ts:348-377);
// the tensor-core path lives in gemm_tc.cu. Covers the three operand layouts of WebGPUBackend.gemm
// (src/backend/webgpu.ts:1654-1671) with ragged edges in every dimension, sums of products written once and groups of
// independent products in one launch.
#include <cooperative_groups.h>
#include <math.h>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace {

// Tile of a CTA: BM x BN outputs, BK deep per stage, TM x TN outputs per thread (as 4-row and 4-column strips, so that a
// warp's shared-memory reads are 16-byte, conflict-free or broadcast).
// What bounds it is the FMA pipe (128 per clock and SM) and, below a few hundred tiles, the number of SMs at work.
//  * 128 x 128: 64 FMAs per four 16-byte shared-memory reads and thread; for products whose tiles fill the SMs.
//  * 64 x 64: a quarter of the tile, for everything else; the contraction is cut over a cluster of up to 8 CTAs, which add
//    their tiles through distributed shared memory in rank order (no atomics, no scratch, the same bits on every run).
// Both keep one stage in registers on its way from global memory while the stage before it is multiplied, and write
// shared memory double-buffered: one barrier per stage. Two FMAs issue as one packed instruction (fma.rn.f32x2): the same
// IEEE operations at half the issue slots.
template <int BM_, int BN_, int BK_, int TM_, int TN_>
struct Tile {
  static constexpr int BM = BM_, BN = BN_, BK = BK_, TM = TM_, TN = TN_;
  static constexpr int THREADS = (BM / TM) * (BN / TN);
  static constexpr int STAGE = BK * (BM + BN);
  static constexpr int SMEM = (2 * STAGE > BM * BN ? 2 * STAGE : BM * BN) * 4;   // (the reduction reuses it for a whole tile)
  static constexpr int QA = BM * BK / 4 / THREADS, QB = BN * BK / 4 / THREADS;   // 16-byte loads per thread and stage
};
using Big = Tile<128, 128, 16, 8, 8>;
using Small = Tile<64, 64, 32, 8, 4>;

// Stages are [BK][R] with column r of row k at r ^ swz(k): an operand that is contiguous along K is transposed on its way
// into shared memory, and with this the 32 lanes of a warp, which hold four rows' worth of k for 128 / BK columns,
// store to 32 different banks; quads of columns stay together, so reads are 16-byte loads as before.
template <int BK>
__device__ __forceinline__ constexpr int swz(int k) { return ((k / 4) % (BK / 4)) * (128 / BK); }

constexpr int MAX_PARTS = 8;
struct F32Args {
  const float* a[MAX_PARTS];
  const float* b[MAX_PARTS];
  float* c[MAX_PARTS];
  int K[MAX_PARTS];
  int M[MAX_PARTS], N[MAX_PARTS], accum[MAX_PARTS];
  int tile_end[MAX_PARTS];   // grouped: group g owns tiles [tile_end[g-1], tile_end[g])
  int nparts, ngroups;       // one of the two is 1: products summed into c[0], or independent products of one K
  float alpha;
};

// a quad of four consecutive floats along the contiguous axis, zero outside [0, n) x [0, m)
template <bool VEC>
__device__ __forceinline__ float4 quad(const float* __restrict__ p, long row, int ld, int i, int n, bool row_ok) {
  if (!row_ok || i >= n) return make_float4(0.f, 0.f, 0.f, 0.f);
  const float* s = p + row * ld + i;
  if (VEC) return __ldg(reinterpret_cast<const float4*>(s));   // (n is a multiple of 4: the whole quad is inside)
  float4 v = make_float4(__ldg(s), 0.f, 0.f, 0.f);
  if (i + 1 < n) v.y = __ldg(s + 1);
  if (i + 2 < n) v.z = __ldg(s + 2);
  if (i + 3 < n) v.w = __ldg(s + 3);
  return v;
}

// One operand's stage in registers: R rows (the M or N extent) x BK. KC: the operand is [R, K] with K contiguous, else [K, R].
template <int R, int BK, int Q, int THREADS, bool KC, bool VEC>
struct Operand {
  float4 v[Q];
  __device__ __forceinline__ void load(const float* __restrict__ p, int rows, int K, int r0, int k0) {
#pragma unroll
    for (int i = 0; i < Q; i++) {
      const int idx = threadIdx.x + i * THREADS;
      if (KC) {
        const int kq = idx % (BK / 4), r = idx / (BK / 4);
        v[i] = quad<VEC>(p, r0 + r, K, k0 + kq * 4, K, r0 + r < rows);
      } else {
        const int rq = idx % (R / 4), k = idx / (R / 4);
        v[i] = quad<VEC>(p, k0 + k, rows, r0 + rq * 4, rows, k0 + k < K);
      }
    }
  }
  __device__ __forceinline__ void store(float* s) const {
#pragma unroll
    for (int i = 0; i < Q; i++) {
      const int idx = threadIdx.x + i * THREADS;
      if (KC) {
        const int kq = idx % (BK / 4), r = idx / (BK / 4);
        float* d = s + kq * 4 * R + (r ^ swz<BK>(kq * 4));
        d[0] = v[i].x; d[R] = v[i].y; d[2 * R] = v[i].z; d[3 * R] = v[i].w;
      } else {
        const int rq = idx % (R / 4), k = idx / (R / 4);
        *reinterpret_cast<float4*>(s + k * R + ((rq * 4) ^ swz<BK>(k))) = v[i];
      }
    }
  }
};

__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

// gridDim.x = tiles x ksplit, the ksplit CTAs of a tile adjacent and, when there are several, one cluster.
template <class T, bool A_K, bool B_K, bool VEC>
__global__ void __launch_bounds__(T::THREADS) gemm_f32_kernel(const __grid_constant__ F32Args p, int ksplit) {
  pdl_wait();
  extern __shared__ __align__(16) float sm[];
  constexpr int BM = T::BM, BN = T::BN, BK = T::BK, TM = T::TM, TN = T::TN;
  constexpr int TX = BN / TN, TY = BM / TM;
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const int z = blockIdx.x % ksplit;
  int t = blockIdx.x / ksplit, g = 0;
  if (p.ngroups > 1) {
    while (t >= p.tile_end[g]) g++;
    if (g) t -= p.tile_end[g - 1];
  }
  const int M = p.M[g], N = p.N[g];
  const int tn = (N + BN - 1) / BN, n0 = (t % tn) * BN, m0 = (t / tn) * BM;
  int kblocks = 0;
  for (int i = 0; i < p.nparts; i++) kblocks += (p.K[g + i] + BK - 1) / BK;
  const int per = (kblocks + ksplit - 1) / ksplit;
  const int kb0 = min(kblocks, z * per), kb1 = min(kblocks, kb0 + per);

  unsigned long long acc[TM / 2][TN];      // pairs of rows: only the TN values of B need duplicating per K row
#pragma unroll
  for (int i = 0; i < TM / 2; i++)
#pragma unroll
    for (int j = 0; j < TN; j++) acc[i][j] = 0ull;

  Operand<BM, BK, T::QA, T::THREADS, A_K, VEC> oa;
  Operand<BN, BK, T::QB, T::THREADS, B_K, VEC> ob;
  // K block kb lies in product `part`, from its row k0 on
  int part = g, k0 = kb0 * BK;
  while (part < g + p.nparts - 1 && k0 >= (p.K[part] + BK - 1) / BK * BK) { k0 -= (p.K[part] + BK - 1) / BK * BK; part++; }
  auto fetch = [&] {
    oa.load(p.a[part], M, p.K[part], m0, k0);
    ob.load(p.b[part], N, p.K[part], n0, k0);
    k0 += BK;
    if (k0 >= p.K[part] && part < g + p.nparts - 1) { k0 = 0; part++; }
  };
  if (kb0 < kb1) {
    fetch();
    oa.store(sm); ob.store(sm + BK * BM);
  }
  __syncthreads();
  for (int kb = kb0; kb < kb1; kb++) {
    const float* As = sm + ((kb - kb0) & 1) * T::STAGE;
    const float* Bs = As + BK * BM;
    if (kb + 1 < kb1) fetch();
#pragma unroll
    for (int kk = 0; kk < BK; kk++) {
      unsigned long long av[TM / 2];
      float bv[TN];
#pragma unroll
      for (int i = 0; i < TM / 4; i++) {
        const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(As + kk * BM + ((i * (4 * TY) + ty * 4) ^ swz<BK>(kk)));
        av[2 * i] = w.x; av[2 * i + 1] = w.y;
      }
#pragma unroll
      for (int j = 0; j < TN / 4; j++)
        *reinterpret_cast<float4*>(&bv[4 * j]) = *reinterpret_cast<const float4*>(Bs + kk * BN + ((j * (4 * TX) + tx * 4) ^ swz<BK>(kk)));
#pragma unroll
      for (int j = 0; j < TN; j++) {
        const unsigned long long bb = pack2(bv[j], bv[j]);
#pragma unroll
        for (int i = 0; i < TM / 2; i++) fma2(acc[i][j], av[i], bb);
      }
    }
    if (kb + 1 < kb1) {
      float* d = sm + ((kb + 1 - kb0) & 1) * T::STAGE;
      oa.store(d); ob.store(d + BK * BM);
    }
    __syncthreads();
  }

  auto quad_of = [&](int i, int j) {           // row i, columns 4 j .. 4 j + 3 of this thread's outputs
    float v[4];
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const float2 u = unpack2(acc[i / 2][4 * j + e]);
      v[e] = (i & 1) ? u.y : u.x;
    }
    return make_float4(v[0], v[1], v[2], v[3]);
  };
  float* C = p.c[g];
  const int accum = p.accum[g];
  const bool vecC = (N & 3) == 0 && (((uintptr_t)C) & 15) == 0;
  auto put = [&](int m, int n, float4 v) {     // four outputs of a row
    if (m >= M || n >= N) return;
    float* d = C + (long)m * N + n;
    v.x *= p.alpha; v.y *= p.alpha; v.z *= p.alpha; v.w *= p.alpha;
    if (vecC) {
      if (accum) { const float4 o = *reinterpret_cast<const float4*>(d); v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w; }
      *reinterpret_cast<float4*>(d) = v;
      return;
    }
    d[0] = accum ? d[0] + v.x : v.x;
    if (n + 1 < N) d[1] = accum ? d[1] + v.y : v.y;
    if (n + 2 < N) d[2] = accum ? d[2] + v.z : v.z;
    if (n + 3 < N) d[3] = accum ? d[3] + v.w : v.w;
  };
  if (ksplit == 1) {
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
      for (int j = 0; j < TN / 4; j++) put(m0 + (i / 4) * (4 * TY) + ty * 4 + i % 4, n0 + j * (4 * TX) + tx * 4, quad_of(i, j));
    return;
  }
  // the cluster's slices: every CTA leaves its tile in shared memory and adds up its share of the rows over all of them
#pragma unroll
  for (int i = 0; i < TM; i++)
#pragma unroll
    for (int j = 0; j < TN / 4; j++)
      *reinterpret_cast<float4*>(sm + ((i / 4) * (4 * TY) + ty * 4 + i % 4) * BN + j * (4 * TX) + tx * 4) = quad_of(i, j);
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  for (int q = z * T::THREADS + tid; q < BM * BN / 4; q += ksplit * T::THREADS) {
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int r = 0; r < ksplit; r++) {
      const float4 v = *(reinterpret_cast<const float4*>(cluster.map_shared_rank(sm, r)) + q);
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    put(m0 + q / (BN / 4), n0 + (q % (BN / 4)) * 4, s);
  }
  cluster.sync();      // (nobody leaves while its tile may still be read)
}

template <class T, bool A_K, bool B_K, bool VEC>
gt_status launch(gt_ctx* ctx, const F32Args& p, long tiles, int ksplit) {
  auto kern = gemm_f32_kernel<T, A_K, B_K, VEC>;
  static bool attr_set[64] = {};
  if (ctx->device >= 0 && ctx->device < 64 && !attr_set[ctx->device]) {
    GT_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, T::SMEM));
    attr_set[ctx->device] = true;
  }
  GT_CUDA(ctx, gt_launch(ctx, ksplit, kern, dim3((unsigned)(tiles * ksplit)), T::THREADS, T::SMEM, p, ksplit));
  GT_LAUNCHED(ctx, "gemm_f32_kernel");
  return GT_OK;
}

template <class T, bool VEC>
gt_status launch_kind(gt_ctx* ctx, int kind, const F32Args& p, long tiles, int ksplit) {
  if (kind == GT_GEMM_NT) return launch<T, true, true, VEC>(ctx, p, tiles, ksplit);
  if (kind == GT_GEMM_NN) return launch<T, true, false, VEC>(ctx, p, tiles, ksplit);
  return launch<T, false, false, VEC>(ctx, p, tiles, ksplit);
}

template <class T>
long tiles_of(F32Args& p) {
  long n = 0;
  for (int g = 0; g < p.ngroups; g++) {
    n += (long)gt_cdiv(p.M[g], T::BM) * gt_cdiv(p.N[g], T::BN);
    p.tile_end[g] = (int)n;
  }
  return n;
}

// Tile and slices by predicted cycles of the SM with the most work: CTAs there x K rows each x cycles per K row, plus what
// a CTA costs whatever its depth. A K row of a tile is BM x BN / 128 cycles of the FMA pipe; `eff` is the part of that rate
// that the resident CTAs reach together (one 64 x 64 CTA, four warps, 0.44; four of them 0.68; 128 x 128, eight warps,
// 0.62 and 0.74). Clusters of four and more land unevenly on the SMs when there are few. Fitted on eleven shapes from
// 512 x 128 x 128 to 8192 x 8192 x 1024, where it picks the fastest choice or one within 15 %: 53 TFLOP/s at the largest
// (128 x 128), 57 us for 512 x 576 x 1536 in one slice against 31 in eight.
template <class T>
double cost_of(gt_ctx* ctx, const F32Args& p, long tiles, int ksplit) {
  double rows = 0;
  for (int i = 0; i < p.nparts; i++) rows += gt_cdiv(p.K[i], T::BK) * T::BK;
  const double per = gt_cdiv((long)rows / T::BK, ksplit) * T::BK;
  const double share = (double)tiles * ksplit / ctx->sm_count;
  const double ctas = share <= 0.5 ? 1.0 : ceil(share * (ksplit >= 4 && share < 4.0 ? 1.25 : 1.0));
  const double eff = T::THREADS >= 256 ? (ctas < 2 ? 0.62 : 0.74) : (ctas < 2 ? 0.44 : ctas < 3 ? 0.54 : ctas < 4 ? 0.60 : 0.68);
  return per * ctas * (T::BM * T::BN / 128.0) / eff + 3500.0 + (ksplit > 1 ? 1000.0 + 500.0 * ksplit : 0.0) + 600.0 * (ctas - 1);
}

gt_status run(gt_ctx* ctx, int kind, F32Args& p) {
  bool vec = true;
  for (int i = 0; i < p.nparts + p.ngroups - 1; i++) {
    const int m = p.M[p.ngroups > 1 ? i : 0], n = p.N[p.ngroups > 1 ? i : 0];
    const int ia = kind == GT_GEMM_TN ? m : p.K[i], ib = kind == GT_GEMM_NT ? p.K[i] : n;
    vec = vec && ((ia | ib) & 3) == 0 && ((((uintptr_t)p.a[i]) | ((uintptr_t)p.b[i])) & 15) == 0;
  }
  // Weight gradients of a model's projections are launched in whatever groups the backward pass gives (they differ with and
  // without recompute), and a strict-f32 result may not depend on that: their slices follow from the depth alone.
  if (kind == GT_GEMM_TN && p.nparts == 1) {
    bool projection = true;
    for (int g = 0; g < p.ngroups; g++) projection = projection && (long)gt_cdiv(p.M[g], Small::BM) * gt_cdiv(p.N[g], Small::BN) <= 1024;
    if (projection) {
      const int ks = p.K[0] >= 2048 ? 8 : p.K[0] >= 512 ? 4 : p.K[0] >= 256 ? 2 : 1;
      const long n = tiles_of<Small>(p);
      return vec ? launch_kind<Small, true>(ctx, kind, p, n, ks) : launch_kind<Small, false>(ctx, kind, p, n, ks);
    }
  }
  const long big = tiles_of<Big>(p);
  double best = cost_of<Big>(ctx, p, big, 1);
  int ksplit = 0;            // 0: the big tile
  const long small = tiles_of<Small>(p);
  for (int ks = 1; ks <= 8; ks *= 2) {
    const double c = cost_of<Small>(ctx, p, small, ks);
    if (c < best) { best = c; ksplit = ks; }
  }
  if (ksplit) return vec ? launch_kind<Small, true>(ctx, kind, p, small, ksplit) : launch_kind<Small, false>(ctx, kind, p, small, ksplit);
  tiles_of<Big>(p);
  return vec ? launch_kind<Big, true>(ctx, kind, p, big, 1) : launch_kind<Big, false>(ctx, kind, p, big, 1);
}

bool kind_ok(int kind) { return kind == GT_GEMM_NT || kind == GT_GEMM_NN || kind == GT_GEMM_TN; }

}  // namespace

// c (+)= alpha * sum_p op(a_p).op(b_p)
static gt_status f32_multi(gt_ctx* ctx, int kind, int accum, int M, int N, int nparts, const int* Ks, const float* const* as,
                           const float* const* bs, float* c, float alpha) {
  if (!kind_ok(kind)) return gt_fail(ctx, GT_ERR_ARG, "gt_gemm: unknown kind %d", kind);
  F32Args p = {};
  p.nparts = nparts; p.ngroups = 1; p.alpha = alpha;
  p.M[0] = M; p.N[0] = N; p.accum[0] = accum; p.c[0] = c;
  for (int i = 0; i < nparts; i++) { p.a[i] = as[i]; p.b[i] = bs[i]; p.K[i] = Ks[i]; }
  return run(ctx, kind, p);
}

static gt_status f32_grouped(gt_ctx* ctx, int kind, int ngroups, const int* Ms, const int* Ns, int K, const float* const* as,
                             const float* const* bs, float* const* cs, const int* accums, float alpha) {
  if (!kind_ok(kind)) return gt_fail(ctx, GT_ERR_ARG, "gt_gemm: unknown kind %d", kind);
  F32Args p = {};
  p.nparts = 1; p.ngroups = ngroups; p.alpha = alpha;
  for (int g = 0; g < ngroups; g++) {
    p.a[g] = as[g]; p.b[g] = bs[g]; p.c[g] = cs[g]; p.K[g] = K;
    p.M[g] = Ms[g]; p.N[g] = Ns[g]; p.accum[g] = accums[g];
  }
  return run(ctx, kind, p);
}

gt_status gt_gemm_simt(gt_ctx* ctx, int kind, int accum, int M, int N, int K, const float* a, const float* b, float* c, float alpha) {
  return f32_multi(ctx, kind, accum, M, N, 1, &K, &a, &b, c, alpha);
}

gt_status gt_gemm_batched(gt_ctx* ctx, int kind, int accum, int M, int N, int K, const float* a, const float* b, float* c, int batch) {
  if (ctx->precision != GT_PREC_FP32) {
    bool handled = false;
    gt_status s = gt_gemm_tc_batched(ctx, kind, accum, M, N, K, a, b, c, batch, &handled);
    if (s != GT_OK || handled) return s;
  }
  for (int i0 = 0; i0 < batch; i0 += MAX_PARTS) {     // eight matrices to a launch
    const int n = min(MAX_PARTS, batch - i0);
    const float* pa[MAX_PARTS];
    const float* pb[MAX_PARTS];
    float* pc[MAX_PARTS];
    int m[MAX_PARTS], nn[MAX_PARTS], acc[MAX_PARTS];
    for (int i = 0; i < n; i++) {
      pa[i] = a + (size_t)(i0 + i) * M * K; pb[i] = b + (size_t)(i0 + i) * N * K; pc[i] = c + (size_t)(i0 + i) * M * N;
      m[i] = M; nn[i] = N; acc[i] = accum;
    }
    gt_status s = f32_grouped(ctx, kind, n, m, nn, K, pa, pb, pc, acc, 1.f);
    if (s) return s;
  }
  return GT_OK;
}

// c (+)= alpha * op(a).op(b): the factor is applied to the f32 accumulator when it is written out
extern "C" gt_status gt_gemm_scaled(gt_ctx* ctx, int32_t kind, int32_t accum, int32_t M, int32_t N, int32_t K, gt_buf a, gt_buf b, gt_buf c,
                                    float alpha) {
  GT_REQUIRE(ctx, M > 0 && N > 0 && K > 0, "gt_gemm: empty product %dx%dx%d", M, N, K);
  GT_REQUIRE(ctx, a && b && c, "gt_gemm: null operand");
  if (ctx->precision != GT_PREC_FP32) {
    bool handled = false;
    gt_status s = gt_gemm_tc(ctx, kind, accum, M, N, K, gt_ptr<const float>(a), gt_ptr<const float>(b), gt_ptr<float>(c), alpha, &handled);
    if (s != GT_OK || handled) return s;
  }
  return gt_gemm_simt(ctx, kind, accum, M, N, K, gt_ptr<const float>(a), gt_ptr<const float>(b), gt_ptr<float>(c), alpha);
}

extern "C" gt_status gt_gemm(gt_ctx* ctx, int32_t kind, int32_t accum, int32_t M, int32_t N, int32_t K, gt_buf a, gt_buf b, gt_buf c) {
  return gt_gemm_scaled(ctx, kind, accum, M, N, K, a, b, c, 1.f);
}

// c (+)= sum_p op(a_p).op(b_p): one launch on the tensor-core path (each product's K blocks follow the previous one's in
// the main loop), accumulating products otherwise.
extern "C" gt_status gt_gemm_multi(gt_ctx* ctx, int32_t kind, int32_t accum, int32_t M, int32_t N, int32_t nparts, const int32_t* Ks,
                                   const gt_buf* as, const gt_buf* bs, gt_buf c) {
  GT_REQUIRE(ctx, M > 0 && N > 0 && nparts >= 1 && nparts <= 8 && Ks && as && bs && c, "gt_gemm_multi: %dx%d, %d products (1..8)", M, N, nparts);
  const float* pa[8];
  const float* pb[8];
  int k[8];
  for (int p = 0; p < nparts; p++) {
    GT_REQUIRE(ctx, Ks[p] > 0 && as[p] && bs[p], "gt_gemm_multi: product %d is empty or has a null operand", p);
    pa[p] = gt_ptr<const float>(as[p]); pb[p] = gt_ptr<const float>(bs[p]); k[p] = Ks[p];
  }
  if (ctx->precision != GT_PREC_FP32) {
    bool handled = false;
    gt_status s = gt_gemm_tc_multi(ctx, kind, accum, M, N, nparts, k, pa, pb, gt_ptr<float>(c), &handled);
    if (s != GT_OK || handled) return s;
  }
  if (ctx->precision == GT_PREC_FP32) return f32_multi(ctx, kind, accum, M, N, nparts, k, pa, pb, gt_ptr<float>(c), 1.f);
  for (int p = 0; p < nparts; p++) {
    gt_status s = gt_gemm(ctx, kind, p ? 1 : accum, M, N, k[p], as[p], bs[p], c);
    if (s) return s;
  }
  return GT_OK;
}

// ngroups products of one layout and one depth K, each with its own operands, extents and accumulate flag: one launch
// on the tensor-core path, one product after the other otherwise. alpha multiplies every product.
extern "C" gt_status gt_gemm_grouped_scaled(gt_ctx* ctx, int32_t kind, int32_t ngroups, const int32_t* Ms, const int32_t* Ns, int32_t K,
                                            const gt_buf* as, const gt_buf* bs, const gt_buf* cs, const int32_t* accums, float alpha) {
  GT_REQUIRE(ctx, ngroups >= 1 && ngroups <= 8 && K > 0 && Ms && Ns && as && bs && cs && accums, "gt_gemm_grouped: %d products (1..8), K %d", ngroups, K);
  const float* pa[8];
  const float* pb[8];
  float* pc[8];
  int m[8], n[8], acc[8];
  for (int g = 0; g < ngroups; g++) {
    GT_REQUIRE(ctx, Ms[g] > 0 && Ns[g] > 0 && as[g] && bs[g] && cs[g], "gt_gemm_grouped: product %d is empty or has a null operand", g);
    pa[g] = gt_ptr<const float>(as[g]); pb[g] = gt_ptr<const float>(bs[g]); pc[g] = gt_ptr<float>(cs[g]);
    m[g] = Ms[g]; n[g] = Ns[g]; acc[g] = accums[g];
  }
  if (ctx->precision != GT_PREC_FP32 && ngroups > 1) {
    bool handled = false;
    gt_status s = gt_gemm_tc_grouped(ctx, kind, ngroups, m, n, K, pa, pb, pc, acc, nullptr, nullptr, 0, alpha, &handled);
    if (s != GT_OK || handled) return s;
  }
  if (ctx->precision == GT_PREC_FP32) return f32_grouped(ctx, kind, ngroups, m, n, K, pa, pb, pc, acc, alpha);
  for (int g = 0; g < ngroups; g++) {
    gt_status s = gt_gemm_scaled(ctx, kind, acc[g], m[g], n[g], K, as[g], bs[g], cs[g], alpha);
    if (s) return s;
  }
  return GT_OK;
}

extern "C" gt_status gt_gemm_grouped(gt_ctx* ctx, int32_t kind, int32_t ngroups, const int32_t* Ms, const int32_t* Ns, int32_t K,
                                     const gt_buf* as, const gt_buf* bs, const gt_buf* cs, const int32_t* accums) {
  return gt_gemm_grouped_scaled(ctx, kind, ngroups, Ms, Ns, K, as, bs, cs, accums, 1.f);
}

// Projections y_g = x.W_g^T of one input launched together, the rotary embedding applied to the outputs that take one
// (heads[g] > 0) as their tiles are written; elsewhere each product followed by the rotation as a pass over its output.
extern "C" gt_status gt_linear_rope_grouped(gt_ctx* ctx, int32_t ngroups, int32_t rows, int32_t K, gt_buf x, const int32_t* Ns,
                                            const gt_buf* ws, const gt_buf* ys, const int32_t* heads, int32_t hd, double base,
                                            int32_t pos_offset) {
  GT_REQUIRE(ctx, ngroups >= 1 && ngroups <= 8 && rows > 0 && K > 0 && x && Ns && ws && ys && heads, "gt_linear_rope_grouped: %d projections (1..8), rows %d, K %d",
             ngroups, rows, K);
  GT_REQUIRE(ctx, hd > 0 && hd % 2 == 0, "gt_linear_rope_grouped: head size %d (must be even)", hd);
  const float* pa[8];
  const float* pb[8];
  float* pc[8];
  int m[8], n[8], acc[8], rp[8];
  bool any = false;
  for (int g = 0; g < ngroups; g++) {
    GT_REQUIRE(ctx, Ns[g] > 0 && ws[g] && ys[g], "gt_linear_rope_grouped: projection %d is empty or has a null operand", g);
    GT_REQUIRE(ctx, heads[g] == 0 || heads[g] * hd == Ns[g], "gt_linear_rope_grouped: projection %d is %d wide, not %d heads of %d", g, Ns[g], heads[g], hd);
    pa[g] = gt_ptr<const float>(x); pb[g] = gt_ptr<const float>(ws[g]); pc[g] = gt_ptr<float>(ys[g]);
    m[g] = rows; n[g] = Ns[g]; acc[g] = 0; rp[g] = heads[g] > 0;
    any = any || rp[g];
  }
  const float2* tab = nullptr;
  int period = 0;
  if (any) {
    gt_status s = gt_rope_table(ctx, rows, hd, base, pos_offset, &tab, &period);
    if (s) return s;
  }
  if (ctx->precision != GT_PREC_FP32 && ngroups > 1 && (!any || hd == 64)) {
    bool handled = false;
    gt_status s = gt_gemm_tc_grouped(ctx, GT_GEMM_NT, ngroups, m, n, K, pa, pb, pc, acc, rp, tab, period, 1.f, &handled);
    if (s != GT_OK || handled) return s;
  }
  if (ctx->precision == GT_PREC_FP32) {
    gt_status s = f32_grouped(ctx, GT_GEMM_NT, ngroups, m, n, K, pa, pb, pc, acc, 1.f);
    for (int g = 0; g < ngroups && !s; g++)
      if (rp[g]) s = gt_rope_apply(ctx, false, rows, heads[g], hd, base, pos_offset, pc[g], pc[g], 0);
    return s;
  }
  for (int g = 0; g < ngroups; g++) {
    gt_status s = gt_gemm(ctx, GT_GEMM_NT, 0, rows, n[g], K, x, ws[g], ys[g]);
    if (s) return s;
    if (rp[g]) s = gt_rope_apply(ctx, false, rows, heads[g], hd, base, pos_offset, pc[g], pc[g], 0);
    if (s) return s;
  }
  return GT_OK;
}

extern "C" gt_status gt_gemm2(gt_ctx* ctx, int32_t kind, int32_t accum, int32_t M, int32_t N, int32_t K, gt_buf a, gt_buf b, int32_t K2,
                              gt_buf a2, gt_buf b2, gt_buf c) {
  GT_REQUIRE(ctx, M > 0 && N > 0 && K > 0 && K2 > 0, "gt_gemm2: empty product %dx%dx(%d+%d)", M, N, K, K2);
  GT_REQUIRE(ctx, a && b && a2 && b2 && c, "gt_gemm2: null operand");
  const int32_t Ks[2] = {K, K2};
  const gt_buf as[2] = {a, a2}, bs[2] = {b, b2};
  return gt_gemm_multi(ctx, kind, accum, M, N, 2, Ks, as, bs, c);
}
