// Causal grouped-query attention with optional sliding window, forward and backward, for any head
// dimension up to 256 (src/model/autograd.ts:640-729; srcAttnFwd/BwdD/BwdDq/BwdDkv src/backend/wgsl.ts:657-918).
// f32 FMA throughout. This is the strict-precision path and the one that covers head dimensions the
// tensor-core kernels do not (the reference's tests use hd 4, 6, 12, 24).
// Same formulation as the reference's flash kernels: scores in the exp2 domain
// (SCALE2 = log2(e)/sqrt(hd)), running max with sentinel -3e38, LSE[h,row] = m + log2(l) as the only
// side buffer, backward recomputing p = exp2(q.k*SCALE2 - LSE).
//
// A CTA owns R rows of the output and walks the other axis in tiles of C, every operand tile as stored ([row][head], row
// pitch HDP + 4 floats, zeros past the sequence and the head size). The products run from shared memory with 4 columns and
// R C / 4 NT rows per thread. Thread (ty, tx) takes rows ty + TY i and columns tx + TX j of a score tile, so that its 16-byte
// reads along the head dimension start in different banks for neighbouring lanes, and the TX lanes that share a row are one
// aligned group of a warp: row maxima, sums and the hand-over of P from one product to the next stay inside it. Score sums
// are kept as pairs (even and odd head positions), which the packed FMA takes without moving registers.
// What bounds these kernels is the FMA pipe at long sequences and, at short ones, the chain of tiles of the CTA with most
// of them: rows per CTA are 32 instead of 64 while that leaves SMs idle. At 512 rows of 9/3 heads of 64 a warp per row took
// 230 us forward and 690 us backward.
// No atomics: one CTA owns its rows (dQ), or the CTAs of a cluster, one per query head of the group, add their dK and dV
// through distributed shared memory in rank order. The same bits on every run.
#include <cooperative_groups.h>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr float NEG = -3.0e38f;

typedef unsigned long long pair_t;
__device__ __forceinline__ pair_t pack2(float x, float y) {
  pair_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 unpack2(pair_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ void fma2(pair_t& d, pair_t a, pair_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }

template <int HDP_, int R_, int C_, int NT_>
struct Geo {
  static constexpr int HDP = HDP_, R = R_, C = C_, NT = NT_;
  static constexpr int TX = C / 4, TY = NT / TX, TR = R / TY;     // column lanes, row lanes, rows per thread
  static constexpr int P = HDP + 4, PP = C + 4;                   // row pitches of operand and probability tiles
  static constexpr int OC = HDP / TX, VW = OC < 4 ? OC : 4, OG = OC / VW;   // output columns per thread: OG runs of VW
  static constexpr int FWD_SMEM = ((R + 2 * C) * P + R * PP) * 4;
  static constexpr int BWD_SMEM = ((2 * R + 2 * C) * P + 2 * R * PP) * 4;
  static_assert(TX <= 32 && 32 % TX == 0 && TR * TY == R && (OC == 2 || OC % 4 == 0), "geometry");
  static_assert(FWD_SMEM <= 232448 && BWD_SMEM <= 232448, "shared memory");
};

// rows [r0, r0 + ROWS) of one head of a [rows, stride] matrix; zeros from `last` on and past hd
template <class G, int ROWS>
__device__ __forceinline__ void load_tile(float* dst, const float* __restrict__ src, int r0, int last, size_t stride, int hd, bool vec) {
  constexpr int Q = G::HDP / 4;
  for (int i = threadIdx.x; i < ROWS * Q; i += G::NT) {
    const int r = i / Q, d = (i % Q) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r0 + r < last && d < hd) {
      const float* s = src + (size_t)(r0 + r) * stride + d;
      if (vec) v = __ldg(reinterpret_cast<const float4*>(s));
      else {
        v.x = __ldg(s);
        if (d + 1 < hd) v.y = __ldg(s + 1);
        if (d + 2 < hd) v.z = __ldg(s + 2);
        if (d + 3 < hd) v.w = __ldg(s + 3);
      }
    }
    *reinterpret_cast<float4*>(dst + r * G::P + d) = v;
  }
}

// s[i][j] = A[ty + TY i] . B[tx + TX j] over the head dimension
template <class G>
__device__ __forceinline__ void dots(const float* A, const float* B, int ty, int tx, float (&s)[G::TR][4]) {
  pair_t acc[G::TR][4];
#pragma unroll
  for (int i = 0; i < G::TR; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = 0ull;
#pragma unroll 8
  for (int d = 0; d < G::HDP; d += 4) {
    ulonglong2 a[G::TR], b[4];
#pragma unroll
    for (int i = 0; i < G::TR; i++) a[i] = *reinterpret_cast<const ulonglong2*>(A + (ty + G::TY * i) * G::P + d);
#pragma unroll
    for (int j = 0; j < 4; j++) b[j] = *reinterpret_cast<const ulonglong2*>(B + (tx + G::TX * j) * G::P + d);
#pragma unroll
    for (int i = 0; i < G::TR; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) { fma2(acc[i][j], a[i].x, b[j].x); fma2(acc[i][j], a[i].y, b[j].y); }
  }
#pragma unroll
  for (int i = 0; i < G::TR; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) { const float2 v = unpack2(acc[i][j]); s[i][j] = v.x + v.y; }
}

// o[i][..] += W[ty + TY i][0..C) . B[0..C)[this thread's columns]
template <class G>
__device__ __forceinline__ void accumulate(const float* W, const float* B, int ty, int tx, pair_t (&o)[G::TR][G::OC / 2]) {
#pragma unroll 4
  for (int c = 0; c < G::C; c += 4) {
    float4 w[G::TR];
#pragma unroll
    for (int i = 0; i < G::TR; i++) w[i] = *reinterpret_cast<const float4*>(W + (ty + G::TY * i) * G::PP + c);
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const float* b = B + (c + e) * G::P + tx * G::VW;
      pair_t bv[G::OC / 2];
#pragma unroll
      for (int g = 0; g < G::OG; g++) {
        if constexpr (G::VW == 4) {
          const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(b + g * 4 * G::TX);
          bv[2 * g] = t.x; bv[2 * g + 1] = t.y;
        } else {
          bv[g] = *reinterpret_cast<const pair_t*>(b + g * 2 * G::TX);
        }
      }
#pragma unroll
      for (int i = 0; i < G::TR; i++) {
        const float we = e == 0 ? w[i].x : e == 1 ? w[i].y : e == 2 ? w[i].z : w[i].w;
        const pair_t ww = pack2(we, we);
#pragma unroll
        for (int g = 0; g < G::OC / 2; g++) fma2(o[i][g], ww, bv[g]);
      }
    }
  }
}

// column of this thread's output pair g
template <class G>
__device__ __forceinline__ int out_col(int tx, int g) { return (g / (G::VW / 2)) * G::VW * G::TX + tx * G::VW + (g % (G::VW / 2)) * 2; }

template <class G>
__global__ void __launch_bounds__(G::NT) attn_fwd_f32_kernel(int rows, int T, int Hq, int Hkv, int hd, int window, float scale2,
                                                             const float* __restrict__ q, const float* __restrict__ k,
                                                             const float* __restrict__ v, float* __restrict__ out,
                                                             float* __restrict__ lse, int vec) {
  pdl_wait();
  extern __shared__ __align__(16) float sm[];
  constexpr int R = G::R, C = G::C, TR = G::TR, TX = G::TX;
  float* Qs = sm;
  float* Ks = Qs + R * G::P;
  float* Vs = Ks + C * G::P;
  float* Ps = Vs + C * G::P;
  const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
  const int q0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * R;     // late queries read the most keys: heaviest first
  const int h = blockIdx.x % Hq, seq = blockIdx.x / Hq, kvh = h / (Hq / Hkv), row0 = seq * T;
  const size_t qS = (size_t)Hq * hd, kS = (size_t)Hkv * hd;
  const float* qp = q + (size_t)row0 * qS + (size_t)h * hd;
  const float* kp = k + (size_t)row0 * kS + (size_t)kvh * hd;
  const float* vp = v + (size_t)row0 * kS + (size_t)kvh * hd;
  load_tile<G, R>(Qs, qp, q0, T, qS, hd, vec);
  const int q_last = min(q0 + R - 1, T - 1);
  const int lo = (window > 0 && q0 - window + 1 > 0) ? (q0 - window + 1) / C : 0, hi = q_last / C;
  float m[TR], l[TR];
  pair_t o[TR][G::OC / 2];
#pragma unroll
  for (int i = 0; i < TR; i++) {
    m[i] = NEG; l[i] = 0.f;
#pragma unroll
    for (int g = 0; g < G::OC / 2; g++) o[i][g] = 0ull;
  }
  for (int kb = lo; kb <= hi; kb++) {
    __syncthreads();                       // everyone has read the tiles of the block before
    load_tile<G, C>(Ks, kp, kb * C, T, kS, hd, vec);
    load_tile<G, C>(Vs, vp, kb * C, T, kS, hd, vec);
    __syncthreads();
    float s[TR][4];
    dots<G>(Qs, Ks, ty, tx, s);
#pragma unroll
    for (int i = 0; i < TR; i++) {
      const int tq = q0 + ty + G::TY * i;
      float mx = NEG;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int kg = kb * C + tx + TX * j;
        const bool keep = kg <= tq && kg < T && (window == 0 || kg > tq - window);
        s[i][j] = keep ? s[i][j] * scale2 : NEG;
        mx = fmaxf(mx, s[i][j]);
      }
#pragma unroll
      for (int d = TX / 2; d > 0; d >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d));
      const float mn = fmaxf(m[i], mx), alpha = exp2f(m[i] - mn);
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const float p = s[i][j] > -1.0e38f ? exp2f(s[i][j] - mn) : 0.f;
        Ps[(ty + G::TY * i) * G::PP + tx + TX * j] = p;
        sum += p;
      }
#pragma unroll
      for (int d = TX / 2; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
      l[i] = l[i] * alpha + sum;
      m[i] = mn;
#pragma unroll
      for (int g = 0; g < G::OC / 2; g++) { const float2 x = unpack2(o[i][g]); o[i][g] = pack2(x.x * alpha, x.y * alpha); }
    }
    __syncwarp();                          // (a row of P is written and read by the same lanes)
    accumulate<G>(Ps, Vs, ty, tx, o);
  }
#pragma unroll
  for (int i = 0; i < TR; i++) {
    const int tq = q0 + ty + G::TY * i;
    if (tq >= T) continue;
    const float inv = 1.f / l[i];
    float* dst = out + (size_t)(row0 + tq) * qS + (size_t)h * hd;
#pragma unroll
    for (int g = 0; g < G::OC / 2; g++) {
      const int d = out_col<G>(tx, g);
      const float2 x = unpack2(o[i][g]);
      if (d < hd) dst[d] = x.x * inv;
      if (d + 1 < hd) dst[d + 1] = x.y * inv;
    }
    if (tx == 0) lse[(size_t)h * rows + row0 + tq] = m[i] + log2f(l[i]);
  }
}

// D[h,row] = sum_d dO*O   (srcAttnBwdD)
__global__ void attn_bwd_d_kernel(int rows, int Hq, int hd, const float* __restrict__ go, const float* __restrict__ o,
                                  float* __restrict__ D) {
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const long w = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= (long)rows * Hq) return;
  const int h = (int)(w % Hq);
  const long row = w / Hq;
  const size_t b = (size_t)row * Hq * hd + (size_t)h * hd;
  float acc = 0.f;
  for (int d = lane; d < hd; d += 32) acc = fmaf(go[b + d], o[b + d], acc);
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
  if (lane == 0) D[(size_t)h * rows + row] = acc;
}

struct BwdArgs {
  int rows, T, Hq, Hkv, hd, window;
  float scale2, scale;
  const float *q, *k, *v, *go, *lse, *D;
  float *gq, *gk, *gv;
  int accum_q, accum_k, accum_v, vec;
  int ntiles, dq_ctas, cs;     // row tiles per sequence, CTAs of the dQ part, CTAs that share a dK/dV tile
};

// dQ of R query rows of one head   (srcAttnBwdDq)
template <class G>
__device__ void bwd_dq(const BwdArgs& p, float* sm, int item) {
  constexpr int R = G::R, C = G::C, TR = G::TR, TX = G::TX;
  float* Qs = sm;
  float* Gs = Qs + R * G::P;
  float* Ks = Gs + R * G::P;
  float* Vs = Ks + C * G::P;
  float* Ws = Vs + C * G::P;
  const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
  const int heads = p.Hq * (p.rows / p.T);
  const int q0 = (p.ntiles - 1 - item / heads) * R;
  const int h = (item % heads) % p.Hq, row0 = (item % heads) / p.Hq * p.T, kvh = h / (p.Hq / p.Hkv);
  const size_t qS = (size_t)p.Hq * p.hd, kS = (size_t)p.Hkv * p.hd;
  const size_t qo = (size_t)row0 * qS + (size_t)h * p.hd, ko = (size_t)row0 * kS + (size_t)kvh * p.hd;
  load_tile<G, R>(Qs, p.q + qo, q0, p.T, qS, p.hd, p.vec);
  load_tile<G, R>(Gs, p.go + qo, q0, p.T, qS, p.hd, p.vec);
  float L[TR], Dr[TR];
  pair_t o[TR][G::OC / 2];
#pragma unroll
  for (int i = 0; i < TR; i++) {
    const int tq = min(q0 + ty + G::TY * i, p.T - 1);
    L[i] = p.lse[(size_t)h * p.rows + row0 + tq];
    Dr[i] = p.D[(size_t)h * p.rows + row0 + tq];
#pragma unroll
    for (int g = 0; g < G::OC / 2; g++) o[i][g] = 0ull;
  }
  const int q_last = min(q0 + R - 1, p.T - 1);
  const int lo = (p.window > 0 && q0 - p.window + 1 > 0) ? (q0 - p.window + 1) / C : 0, hi = q_last / C;
  for (int kb = lo; kb <= hi; kb++) {
    __syncthreads();
    load_tile<G, C>(Ks, p.k + ko, kb * C, p.T, kS, p.hd, p.vec);
    load_tile<G, C>(Vs, p.v + ko, kb * C, p.T, kS, p.hd, p.vec);
    __syncthreads();
    float s[TR][4], dp[TR][4];
    dots<G>(Qs, Ks, ty, tx, s);
    dots<G>(Gs, Vs, ty, tx, dp);
#pragma unroll
    for (int i = 0; i < TR; i++) {
      const int tq = q0 + ty + G::TY * i;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int kg = kb * C + tx + TX * j;
        const bool keep = kg <= tq && tq < p.T && (p.window == 0 || kg > tq - p.window);
        Ws[(ty + G::TY * i) * G::PP + tx + TX * j] = keep ? exp2f(s[i][j] * p.scale2 - L[i]) * (dp[i][j] - Dr[i]) * p.scale : 0.f;
      }
    }
    __syncwarp();
    accumulate<G>(Ws, Ks, ty, tx, o);
  }
#pragma unroll
  for (int i = 0; i < TR; i++) {
    const int tq = q0 + ty + G::TY * i;
    if (tq >= p.T) continue;
    float* dst = p.gq + (size_t)(row0 + tq) * qS + (size_t)h * p.hd;
#pragma unroll
    for (int g = 0; g < G::OC / 2; g++) {
      const int d = out_col<G>(tx, g);
      const float2 x = unpack2(o[i][g]);
      if (d < p.hd) dst[d] = p.accum_q ? dst[d] + x.x : x.x;
      if (d + 1 < p.hd) dst[d + 1] = p.accum_q ? dst[d + 1] + x.y : x.y;
    }
  }
}

// dK and dV of R key rows of one kv head: CTA `r` of the cs that share them takes the query heads r, r + cs, ... of the
// group, then every CTA adds up its share of the rows over all of them   (srcAttnBwdDkv)
template <class G>
__device__ void bwd_dkv(const BwdArgs& p, float* sm, int item) {
  constexpr int R = G::R, C = G::C, TR = G::TR, TX = G::TX;
  float* Ks = sm;
  float* Vs = Ks + R * G::P;
  float* Qs = Vs + R * G::P;
  float* Gs = Qs + C * G::P;
  float* Ps = Gs + C * G::P;
  float* Ws = Ps + R * G::PP;
  const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
  const int rank = item % p.cs, tile = item / p.cs;
  const int heads = p.Hkv * (p.rows / p.T), group = p.Hq / p.Hkv;
  const int k0 = tile / heads * R;                        // early keys are read by the most queries: heaviest first
  const int kvh = (tile % heads) % p.Hkv, row0 = (tile % heads) / p.Hkv * p.T;
  const size_t qS = (size_t)p.Hq * p.hd, kS = (size_t)p.Hkv * p.hd;
  const size_t ko = (size_t)row0 * kS + (size_t)kvh * p.hd;
  load_tile<G, R>(Ks, p.k + ko, k0, p.T, kS, p.hd, p.vec);
  load_tile<G, R>(Vs, p.v + ko, k0, p.T, kS, p.hd, p.vec);
  pair_t dk[TR][G::OC / 2], dv[TR][G::OC / 2];
#pragma unroll
  for (int i = 0; i < TR; i++)
#pragma unroll
    for (int g = 0; g < G::OC / 2; g++) dk[i][g] = dv[i][g] = 0ull;
  const int k_last = min(k0 + R - 1, p.T - 1);
  const int lo = k0 / C, hi = (p.window > 0 ? min(p.T - 1, k_last + p.window - 1) : p.T - 1) / C;
  for (int h = kvh * group + rank; h < (kvh + 1) * group; h += p.cs) {
    const size_t qo = (size_t)row0 * qS + (size_t)h * p.hd;
    for (int qb = lo; qb <= hi; qb++) {
      __syncthreads();
      load_tile<G, C>(Qs, p.q + qo, qb * C, p.T, qS, p.hd, p.vec);
      load_tile<G, C>(Gs, p.go + qo, qb * C, p.T, qS, p.hd, p.vec);
      float L[4], Dr[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int tq = min(qb * C + tx + TX * j, p.T - 1);
        L[j] = p.lse[(size_t)h * p.rows + row0 + tq];
        Dr[j] = p.D[(size_t)h * p.rows + row0 + tq];
      }
      __syncthreads();
      float s[TR][4], dp[TR][4];
      dots<G>(Ks, Qs, ty, tx, s);
      dots<G>(Vs, Gs, ty, tx, dp);
#pragma unroll
      for (int i = 0; i < TR; i++) {
        const int kg = k0 + ty + G::TY * i;
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const int tq = qb * C + tx + TX * j;
          const bool keep = kg <= tq && tq < p.T && (p.window == 0 || kg > tq - p.window);
          const float w = keep ? exp2f(s[i][j] * p.scale2 - L[j]) : 0.f;
          const int at = (ty + G::TY * i) * G::PP + tx + TX * j;
          Ps[at] = w;
          Ws[at] = w * (dp[i][j] - Dr[j]) * p.scale;
        }
      }
      __syncwarp();
      accumulate<G>(Ps, Gs, ty, tx, dv);
      accumulate<G>(Ws, Qs, ty, tx, dk);
    }
  }
  auto put = [&](int r, int d, float2 a, float2 b) {     // (dk, dv) of columns d and d + 1 of row r
    if (k0 + r >= p.T) return;
    const size_t at = (size_t)(row0 + k0 + r) * kS + (size_t)kvh * p.hd + d;
    if (d < p.hd) {
      if (p.gk) p.gk[at] = p.accum_k ? p.gk[at] + a.x : a.x;
      if (p.gv) p.gv[at] = p.accum_v ? p.gv[at] + b.x : b.x;
    }
    if (d + 1 < p.hd) {
      if (p.gk) p.gk[at + 1] = p.accum_k ? p.gk[at + 1] + a.y : a.y;
      if (p.gv) p.gv[at + 1] = p.accum_v ? p.gv[at + 1] + b.y : b.y;
    }
  };
  if (p.cs == 1) {
#pragma unroll
    for (int i = 0; i < TR; i++)
#pragma unroll
      for (int g = 0; g < G::OC / 2; g++) put(ty + G::TY * i, out_col<G>(tx, g), unpack2(dk[i][g]), unpack2(dv[i][g]));
    return;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < TR; i++)                            // (K and V have been read for the last time: their tiles take dK and dV)
#pragma unroll
    for (int g = 0; g < G::OC / 2; g++) {
      const int at = (ty + G::TY * i) * G::P + out_col<G>(tx, g);
      *reinterpret_cast<pair_t*>(Ks + at) = dk[i][g];
      *reinterpret_cast<pair_t*>(Vs + at) = dv[i][g];
    }
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  for (int e = rank * G::NT + threadIdx.x; e < R * G::HDP / 2; e += p.cs * G::NT) {
    const int r = e / (G::HDP / 2), d = e % (G::HDP / 2) * 2;
    float2 a = make_float2(0.f, 0.f), b = a;
    for (int c = 0; c < p.cs; c++) {
      const float2 x = *reinterpret_cast<const float2*>(cluster.map_shared_rank(Ks, c) + r * G::P + d);
      const float2 y = *reinterpret_cast<const float2*>(cluster.map_shared_rank(Vs, c) + r * G::P + d);
      a.x += x.x; a.y += x.y; b.x += y.x; b.y += y.y;
    }
    put(r, d, a, b);
  }
  cluster.sync();                                         // (nobody leaves while its tiles may still be read)
}

// One launch for both: the dK/dV tiles first (the longer ones), then the dQ tiles.
template <class G>
__global__ void __launch_bounds__(G::NT) attn_bwd_f32_kernel(const __grid_constant__ BwdArgs p) {
  pdl_wait();
  extern __shared__ __align__(16) float sm[];
  const int dkv = (int)gridDim.x - p.dq_ctas;
  if ((int)blockIdx.x < dkv) bwd_dkv<G>(p, sm, blockIdx.x);
  else bwd_dq<G>(p, sm, blockIdx.x - dkv);
}

template <class G>
gt_status launch_fwd(gt_ctx* ctx, int rows, int T, int Hq, int Hkv, int hd, int window, const float* q, const float* k, const float* v,
                     float* out, float* lse, int vec) {
  static bool done[64] = {};
  if (!done[ctx->device]) {
    GT_CUDA(ctx, cudaFuncSetAttribute(attn_fwd_f32_kernel<G>, cudaFuncAttributeMaxDynamicSharedMemorySize, G::FWD_SMEM));
    done[ctx->device] = true;
  }
  const float scale2 = 1.4426950408889634f / sqrtf((float)hd);
  GT_CUDA(ctx, gt_launch(ctx, 1, attn_fwd_f32_kernel<G>, dim3(Hq * (rows / T), gt_cdiv(T, G::R)), G::NT, G::FWD_SMEM, rows, T, Hq, Hkv, hd, window, scale2, q, k, v, out, lse, vec));
  GT_LAUNCHED(ctx, "attn_fwd_f32_kernel");
  return GT_OK;
}

template <class G>
gt_status launch_bwd(gt_ctx* ctx, BwdArgs p) {
  static bool done[64] = {};
  if (!done[ctx->device]) {
    GT_CUDA(ctx, cudaFuncSetAttribute(attn_bwd_f32_kernel<G>, cudaFuncAttributeMaxDynamicSharedMemorySize, G::BWD_SMEM));
    done[ctx->device] = true;
  }
  const int nseq = p.rows / p.T, group = p.Hq / p.Hkv;
  p.ntiles = gt_cdiv(p.T, G::R);
  p.cs = 1;
  if (p.gk || p.gv)
    for (int c = 2; c <= 8; c++)
      if (group % c == 0) p.cs = c;
  const long dkv = p.gk || p.gv ? (long)p.ntiles * p.Hkv * nseq * p.cs : 0;
  p.dq_ctas = p.gq ? p.ntiles * p.Hq * nseq : 0;           // (a multiple of cs: Hq is)
  GT_CUDA(ctx, gt_launch(ctx, p.cs, attn_bwd_f32_kernel<G>, dim3((unsigned)(dkv + p.dq_ctas)), G::NT, G::BWD_SMEM, p));
  GT_LAUNCHED(ctx, "attn_bwd_f32_kernel");
  return GT_OK;
}

// 64 rows to a CTA where that still gives every SM one, else 32 (their chain of tiles is as long, each half the work)
bool tall(gt_ctx* ctx, int rows, int T, int Hq) { return (long)Hq * (rows / T) * gt_cdiv(T, 64) >= ctx->sm_count; }

}  // namespace

gt_status gt_attention_fwd_simt(gt_ctx* ctx, int rows, int T, int Hq, int Hkv, int hd, int window, const float* q,
                                const float* k, const float* v, float* out, float* lse) {
  const int vec = (hd & 3) == 0 && ((((uintptr_t)q) | ((uintptr_t)k) | ((uintptr_t)v)) & 15) == 0;
  GT_REQUIRE(ctx, ctx->device >= 0 && ctx->device < 64, "gt_attention_fwd: device index %d out of range", ctx->device);
  const bool big = tall(ctx, rows, T, Hq);
#define GT_FWD(...) launch_fwd<Geo<__VA_ARGS__>>(ctx, rows, T, Hq, Hkv, hd, window, q, k, v, out, lse, vec)
  if (hd <= 32) return big ? GT_FWD(32, 64, 64, 256) : GT_FWD(32, 32, 64, 128);
  if (hd <= 64) return big ? GT_FWD(64, 64, 64, 256) : GT_FWD(64, 32, 64, 128);
  if (hd <= 128) return big ? GT_FWD(128, 64, 64, 256) : GT_FWD(128, 32, 64, 128);
  return GT_FWD(256, 32, 32, 128);
#undef GT_FWD
}

gt_status gt_attention_bwd_simt_scratch(gt_ctx* ctx, float* D, int rows, int T, int Hq, int Hkv, int hd, int window,
                                        const float* q, const float* k, const float* v, const float* out, const float* lse,
                                        const float* go, float* gq, int accum_q, float* gk, int accum_k, float* gv,
                                        int accum_v);

gt_status gt_attention_bwd_simt(gt_ctx* ctx, int rows, int T, int Hq, int Hkv, int hd, int window, const float* q,
                                const float* k, const float* v, const float* out, const float* lse, const float* go,
                                float* gq, int accum_q, float* gk, int accum_k, float* gv, int accum_v) {
  float* D = nullptr;
  gt_status s = gt_scratch(ctx, sizeof(float) * (size_t)rows * Hq, &D);
  if (s) return s;
  return gt_attention_bwd_simt_scratch(ctx, D, rows, T, Hq, Hkv, hd, window, q, k, v, out, lse, go, gq, accum_q, gk, accum_k, gv,
                                       accum_v);
}

// The backward launches with the row-dot scratch D supplied by the caller: the context's growable scratch block
// (gt_attention_bwd_simt above) or the fixed array of the entry point that must not allocate.
gt_status gt_attention_bwd_simt_scratch(gt_ctx* ctx, float* D, int rows, int T, int Hq, int Hkv, int hd, int window,
                                        const float* q, const float* k, const float* v, const float* out, const float* lse,
                                        const float* go, float* gq, int accum_q, float* gk, int accum_k, float* gv,
                                        int accum_v) {
  GT_REQUIRE(ctx, ctx->device >= 0 && ctx->device < 64, "gt_attention_bwd: device index %d out of range", ctx->device);
  const long warps = (long)rows * Hq;
  GT_CUDA(ctx, gt_launch(ctx, 1, attn_bwd_d_kernel, gt_cdiv(warps * 32, 256), 256, 0, rows, Hq, hd, go, out, D));
  GT_LAUNCHED(ctx, "attn_bwd_d_kernel");
  BwdArgs p = {};
  p.rows = rows; p.T = T; p.Hq = Hq; p.Hkv = Hkv; p.hd = hd; p.window = window;
  p.scale = 1.f / sqrtf((float)hd);
  p.scale2 = 1.4426950408889634f * p.scale;
  p.q = q; p.k = k; p.v = v; p.go = go; p.lse = lse; p.D = D;
  p.gq = gq; p.gk = gk; p.gv = gv;
  p.accum_q = accum_q; p.accum_k = accum_k; p.accum_v = accum_v;
  p.vec = (hd & 3) == 0 && ((((uintptr_t)q) | ((uintptr_t)k) | ((uintptr_t)v) | ((uintptr_t)go)) & 15) == 0;
  const bool big = tall(ctx, rows, T, Hq);
  if (hd <= 32) return big ? launch_bwd<Geo<32, 64, 64, 256>>(ctx, p) : launch_bwd<Geo<32, 32, 64, 128>>(ctx, p);
  if (hd <= 64) return big ? launch_bwd<Geo<64, 64, 64, 256>>(ctx, p) : launch_bwd<Geo<64, 32, 64, 128>>(ctx, p);
  if (hd <= 128) return big ? launch_bwd<Geo<128, 64, 64, 256>>(ctx, p) : launch_bwd<Geo<128, 32, 64, 128>>(ctx, p);
  return launch_bwd<Geo<256, 32, 32, 128>>(ctx, p);
}
