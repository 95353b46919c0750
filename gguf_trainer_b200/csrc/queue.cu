// The launch queue: the ops of a context are launched by a thread of its own, in the order in which they were called.
//
// A launch costs the host 4 to 5 us in the driver, and the code that records the ops (a training loop outside a graph,
// scoring, decoding) spends about as long again on each of them. Done by one thread the two add up, and at model sizes
// where a kernel takes 5 us that sum is what a step takes; on two threads the longer of them is.
// Measured: 4 tokens decoded by 30 layers of 576 13.1 -> 9.9 ms, two sequences of 512 scored by 15 layers 3.1 -> 2.4 ms, a
// loop over micro-batches of a tiny model 7.4 -> 5.7 ms.
//
// What the public names of these ops do: check the arguments, copy them (arrays included) into a ring of records and
// return. Every other entry point waits for the ring to be empty first (gt_drain), so reads, waits, graph recordings and
// replays, events, collectives and optimizer steps see the stream as they would without it. Wrong arguments are refused by the
// call that has them, as before; what can only go wrong in the launch (a failed launch, no memory for scratch) is
// reported by the next call on the context, and the ops behind it in the ring are not launched. Not used while a graph is being
// recorded, on hosts with one processor, nor while a development switch (GT_GEMM_*, GT_ATTN_*) is set: those are read at
// the launch. GT_QUEUE=0 switches it off.
#define GT_QUEUE_FRONT
#include "common.cuh"

#include <sched.h>
#include <string.h>

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <mutex>
#include <new>
#include <thread>
#include <type_traits>


extern char** environ;

namespace {
thread_local bool t_worker = false;      // this thread launches for a context
inline void cpu_pause() {
#if defined(__x86_64__)
  __builtin_ia32_pause();
#else
  std::this_thread::yield();
#endif
}
}  // namespace

struct GtQueue {
  static constexpr uint64_t SLOTS = 1024;
  static constexpr size_t ROOM = 496;
  // A thread that finds the ring empty keeps looking for this long before it sleeps: waking it takes longer than the ops of
  // a running loop are apart.
  static constexpr std::chrono::microseconds PATIENCE{500};
  struct alignas(64) Slot {
    gt_status (*run)(void*);
    alignas(16) char room[ROOM];
  };
  Slot* slots = new Slot[SLOTS];
  alignas(64) std::atomic<uint64_t> head{0};       // records written
  alignas(64) std::atomic<uint64_t> tail{0};       // records done
  alignas(64) std::atomic<int> failed{0};          // status of the op that failed: those behind it are dropped until it is reported
  std::string err;                                 // its message (written by the thread, read once the ring is empty)
  std::atomic<bool> asleep{false}, stop{false};
  std::atomic_flag writing = ATOMIC_FLAG_INIT;
  std::mutex m;
  std::condition_variable cv;
  std::thread thread;

  explicit GtQueue(int device) : thread([this, device] { work(device); }) {}
  ~GtQueue() {
    {
      std::lock_guard<std::mutex> l(m);
      stop = true;
    }
    cv.notify_all();
    thread.join();
    delete[] slots;
  }
  void work(int device) {
    t_worker = true;
    cudaSetDevice(device);
    uint64_t t = 0;
    for (;;) {
      if (head.load(std::memory_order_acquire) == t) {
        const auto t0 = std::chrono::steady_clock::now();
        while (head.load(std::memory_order_acquire) == t && !stop && std::chrono::steady_clock::now() - t0 < PATIENCE) cpu_pause();
        if (head.load(std::memory_order_acquire) == t) {
          std::unique_lock<std::mutex> l(m);
          asleep.store(true);
          cv.wait(l, [&] { return stop || head.load() != t; });
          asleep.store(false);
          if (head.load() == t) return;   // (stopping)
        }
      }
      Slot& s = slots[t % SLOTS];
      const gt_status st = s.run(s.room);
      if (st) failed.store(st);
      tail.store(++t, std::memory_order_release);
    }
  }
  template <typename F>
  gt_status put(const F& f) {
    static_assert(sizeof(F) <= ROOM && std::is_trivially_destructible<F>::value, "record");
    while (writing.test_and_set(std::memory_order_acquire)) cpu_pause();
    const uint64_t h = head.load(std::memory_order_relaxed);
    while (h - tail.load(std::memory_order_acquire) >= SLOTS) cpu_pause();
    Slot& s = slots[h % SLOTS];
    new (s.room) F(f);
    s.run = [](void* p) { return (*static_cast<F*>(p))(); };
    head.store(h + 1);
    writing.clear(std::memory_order_release);
    if (asleep.load()) {
      std::lock_guard<std::mutex> l(m);
      cv.notify_one();
    }
    return GT_OK;
  }
  void wait() {
    const uint64_t h = head.load();
    while (tail.load(std::memory_order_acquire) < h) cpu_pause();
  }
};

const char* gt_env(const char* name) { return t_worker ? nullptr : getenv(name); }
std::string& gt_error_text(gt_ctx* ctx) { return t_worker && ctx->queue ? ctx->queue->err : ctx->err; }
bool gt_skip_queued(gt_ctx* ctx) { return ctx->queue->failed.load(std::memory_order_relaxed) != 0; }

gt_status gt_drain(gt_ctx* ctx) {
  if (!ctx || !ctx->queue || t_worker) return GT_OK;
  ctx->queue->wait();
  const int st = ctx->queue->failed.exchange(0);
  if (!st) return GT_OK;
  ctx->err = ctx->queue->err;
  return (gt_status)st;
}

void gt_queue_destroy(gt_ctx* ctx) {
  delete ctx->queue;
  ctx->queue = nullptr;
}

namespace {
// the queue if the op may go through it
GtQueue* queue_of(gt_ctx* ctx, bool valid) {
  if (!ctx || !valid || ctx->capturing || t_worker) return nullptr;
  for (char** e = environ; e && *e; e++)
    if ((*e)[0] == 'G' && (!strncmp(*e, "GT_GEMM_", 8) || !strncmp(*e, "GT_ATTN_", 8) || !strcmp(*e, "GT_QUEUE=0"))) return nullptr;
  if (!ctx->queue) {
    static const bool several = [] {
      cpu_set_t set;
      return sched_getaffinity(0, sizeof set, &set) == 0 && CPU_COUNT(&set) > 1;
    }();
    if (!several) return nullptr;
    ctx->queue = new GtQueue(ctx->device);
  }
  return ctx->queue;
}
bool in_batch(const gt_ctx* ctx, int rows) { return !ctx->batch || rows == ctx->batch * ctx->seq_len; }
bool heads(int rows, int Hq, int Hkv, int hd, int window) {
  return rows > 0 && Hq > 0 && Hkv > 0 && hd > 0 && hd <= 256 && window >= 0 && Hq % Hkv == 0;
}
bool unit(int op) { return op == GT_EW_SILU || op == GT_EW_GELU; }
template <typename... A>
bool aligned(A... a) { return ((a | ...) & 15) == 0; }
}  // namespace

// A valid call becomes a record; any other is made at once, behind everything queued, and gives its own error.
#define GT_QUEUED(ctx, valid, ...)                                                                      \
  if (GtQueue* q_ = queue_of(ctx, valid)) {                                                             \
    if (q_->failed.load(std::memory_order_relaxed)) return gt_drain(ctx);                               \
    return q_->put([=]() -> gt_status { return gt_skip_queued(ctx) ? GT_OK : __VA_ARGS__; });           \
  }                                                                                                     \
  const gt_status s_ = gt_drain(ctx);                                                                   \
  return s_ ? s_ : __VA_ARGS__

extern "C" {
decltype(gt_gemm) now_gt_gemm;
decltype(gt_gemm_scaled) now_gt_gemm_scaled;
decltype(gt_gemm2) now_gt_gemm2;
decltype(gt_ew_fwd) now_gt_ew_fwd;
decltype(gt_ew_bwd) now_gt_ew_bwd;
decltype(gt_glu_fwd) now_gt_glu_fwd;
decltype(gt_glu_linear_fwd) now_gt_glu_linear_fwd;
decltype(gt_glu_bwd) now_gt_glu_bwd;
decltype(gt_rmsnorm_fwd) now_gt_rmsnorm_fwd;
decltype(gt_add_rmsnorm_fwd) now_gt_add_rmsnorm_fwd;
decltype(gt_rmsnorm_heads_rope_fwd) now_gt_rmsnorm_heads_rope_fwd;
decltype(gt_rmsnorm_bwd) now_gt_rmsnorm_bwd;
decltype(gt_rmsnorm_bwd_add) now_gt_rmsnorm_bwd_add;
decltype(gt_embedding_fwd) now_gt_embedding_fwd;
decltype(gt_embedding_bwd) now_gt_embedding_bwd;
decltype(gt_rope_fwd) now_gt_rope_fwd;
decltype(gt_rope_bwd) now_gt_rope_bwd;
decltype(gt_attention_fwd) now_gt_attention_fwd;
decltype(gt_attention_bwd) now_gt_attention_bwd;
decltype(gt_attention_bwd_rope) now_gt_attention_bwd_rope;
decltype(gt_ce_fwd) now_gt_ce_fwd;
decltype(gt_ce_bwd) now_gt_ce_bwd;
decltype(gt_ce_chunk_stats) now_gt_ce_chunk_stats;
decltype(gt_ce_loss_from_stats) now_gt_ce_loss_from_stats;
decltype(gt_ce_chunk_grad) now_gt_ce_chunk_grad;
decltype(gt_readout_ce_fwd) now_gt_readout_ce_fwd;
decltype(gt_readout_ce_stats) now_gt_readout_ce_stats;
decltype(gt_readout_ce_grad) now_gt_readout_ce_grad;
decltype(gt_soft_ce_fwd) now_gt_soft_ce_fwd;
decltype(gt_soft_ce_bwd) now_gt_soft_ce_bwd;
decltype(gt_zero) now_gt_zero;
decltype(gt_copy) now_gt_copy;
decltype(gt_gemm_multi) now_gt_gemm_multi;
decltype(gt_gemm_grouped) now_gt_gemm_grouped;
decltype(gt_gemm_grouped_scaled) now_gt_gemm_grouped_scaled;
decltype(gt_linear_rope_grouped) now_gt_linear_rope_grouped;
decltype(gt_write) now_gt_write;

gt_status gt_gemm(gt_ctx* ctx, int32_t kind, int32_t accum, int32_t M, int32_t N, int32_t K, gt_buf a, gt_buf b, gt_buf c) {
  GT_QUEUED(ctx, M > 0 && N > 0 && K > 0 && a && b && c, now_gt_gemm(ctx, kind, accum, M, N, K, a, b, c));
}
gt_status gt_gemm_scaled(gt_ctx* ctx, int32_t kind, int32_t accum, int32_t M, int32_t N, int32_t K, gt_buf a, gt_buf b, gt_buf c,
            float alpha) {
  GT_QUEUED(ctx, M > 0 && N > 0 && K > 0 && a && b && c, now_gt_gemm_scaled(ctx, kind, accum, M, N, K, a, b, c, alpha));
}
gt_status gt_gemm2(gt_ctx* ctx, int32_t kind, int32_t accum, int32_t M, int32_t N, int32_t K, gt_buf a, gt_buf b, int32_t K2, gt_buf a2,
            gt_buf b2, gt_buf c) {
  GT_QUEUED(ctx, M > 0 && N > 0 && K > 0 && K2 > 0 && a && b && a2 && b2 && c, now_gt_gemm2(ctx, kind, accum, M, N, K, a, b, K2, a2, b2,
            c));
}
gt_status gt_ew_fwd(gt_ctx* ctx, int32_t op, uint64_t n, gt_buf a, gt_buf b, float c, gt_buf out) {
  GT_QUEUED(ctx, a && out && aligned(a, b, out) && op >= GT_EW_ADD && op <= GT_EW_SCALE && (b || op > GT_EW_MUL), now_gt_ew_fwd(ctx, op, n,
            a, b, c, out));
}
gt_status gt_ew_bwd(gt_ctx* ctx, int32_t op, uint64_t n, gt_buf a, gt_buf b, float c, gt_buf gout, gt_buf ga, int32_t accum_a, gt_buf gb,
            int32_t accum_b) {
  GT_QUEUED(ctx, gout && aligned(a, b, gout, ga, gb) && op >= GT_EW_ADD && op <= GT_EW_SCALE &&
            (a || op == GT_EW_ADD || op == GT_EW_SCALE) && (b || op != GT_EW_MUL), now_gt_ew_bwd(ctx, op, n, a, b, c, gout, ga, accum_a,
            gb, accum_b));
}
gt_status gt_glu_fwd(gt_ctx* ctx, int32_t op, uint64_t n, gt_buf x, gt_buf u, gt_buf out) {
  GT_QUEUED(ctx, x && u && out && aligned(x, u, out) && unit(op), now_gt_glu_fwd(ctx, op, n, x, u, out));
}
gt_status gt_glu_linear_fwd(gt_ctx* ctx, int32_t op, int32_t rows, int32_t ffn, int32_t in, gt_buf x, gt_buf wg, gt_buf wu, gt_buf gate,
            gt_buf up, gt_buf out) {
  GT_QUEUED(ctx, rows > 0 && ffn > 0 && in > 0 && x && wg && wu && gate && up && out && unit(op), now_gt_glu_linear_fwd(ctx, op, rows, ffn,
            in, x, wg, wu, gate, up, out));
}
gt_status gt_glu_bwd(gt_ctx* ctx, int32_t op, uint64_t n, gt_buf x, gt_buf u, gt_buf gout, gt_buf gx, int32_t accum_x, gt_buf gu,
            int32_t accum_u) {
  GT_QUEUED(ctx, x && u && gout && aligned(x, u, gout, gx, gu) && unit(op) && (!gx || gx != gu), now_gt_glu_bwd(ctx, op, n, x, u, gout, gx,
            accum_x, gu, accum_u));
}
gt_status gt_rmsnorm_fwd(gt_ctx* ctx, int32_t rows, int32_t d, gt_buf x, gt_buf w, float eps, gt_buf y, gt_buf rinv) {
  GT_QUEUED(ctx, rows > 0 && d > 0 && d <= 2048 && x && w && y && rinv, now_gt_rmsnorm_fwd(ctx, rows, d, x, w, eps, y, rinv));
}
gt_status gt_add_rmsnorm_fwd(gt_ctx* ctx, int32_t rows, int32_t d, gt_buf a, gt_buf b, gt_buf w, float eps, gt_buf sum, gt_buf y,
            gt_buf rinv) {
  GT_QUEUED(ctx, rows > 0 && d > 0 && d <= 2048 && a && b && w && sum && y && rinv, now_gt_add_rmsnorm_fwd(ctx, rows, d, a, b, w, eps, sum,
            y, rinv));
}
gt_status gt_rmsnorm_heads_rope_fwd(gt_ctx* ctx, int32_t rows, int32_t H, int32_t hd, gt_buf x, gt_buf w, float eps, gt_buf y, gt_buf rinv,
            double base, int32_t pos_offset) {
  GT_QUEUED(ctx, rows > 0 && H > 0 && hd > 0 && hd <= 2048 && hd % 2 == 0 && x && w && y && rinv && in_batch(ctx, rows),
            now_gt_rmsnorm_heads_rope_fwd(ctx, rows, H, hd, x, w, eps, y, rinv, base, pos_offset));
}
gt_status gt_rmsnorm_bwd(gt_ctx* ctx, int32_t rows, int32_t d, gt_buf x, gt_buf w, gt_buf rinv, gt_buf gy, gt_buf gx, int32_t accum_x,
            gt_buf gw, int32_t accum_w) {
  GT_QUEUED(ctx, rows > 0 && d > 0 && d <= 2048 && x && w && rinv && gy, now_gt_rmsnorm_bwd(ctx, rows, d, x, w, rinv, gy, gx, accum_x, gw,
            accum_w));
}
gt_status gt_rmsnorm_bwd_add(gt_ctx* ctx, int32_t rows, int32_t d, gt_buf x, gt_buf w, gt_buf rinv, gt_buf gy, gt_buf gadd, gt_buf gx,
            gt_buf gw, int32_t accum_w) {
  GT_QUEUED(ctx, rows > 0 && d > 0 && d <= 2048 && x && w && rinv && gy && gadd && gx, now_gt_rmsnorm_bwd_add(ctx, rows, d, x, w, rinv, gy,
            gadd, gx, gw, accum_w));
}
gt_status gt_embedding_fwd(gt_ctx* ctx, int32_t rows, int32_t d, gt_buf w, gt_buf ids, gt_buf out) {
  GT_QUEUED(ctx, rows > 0 && d > 0 && w && ids && out, now_gt_embedding_fwd(ctx, rows, d, w, ids, out));
}
gt_status gt_embedding_bwd(gt_ctx* ctx, int32_t rows, int32_t d, gt_buf gy, gt_buf ids, gt_buf gw) {
  GT_QUEUED(ctx, rows > 0 && d > 0 && gy && ids, now_gt_embedding_bwd(ctx, rows, d, gy, ids, gw));
}
gt_status gt_rope_fwd(gt_ctx* ctx, int32_t rows, int32_t H, int32_t hd, double base, int32_t pos_offset, gt_buf x, gt_buf y) {
  GT_QUEUED(ctx, rows > 0 && H > 0 && hd > 0 && hd % 2 == 0 && x && y && in_batch(ctx, rows), now_gt_rope_fwd(ctx, rows, H, hd, base,
            pos_offset, x, y));
}
gt_status gt_rope_bwd(gt_ctx* ctx, int32_t rows, int32_t H, int32_t hd, double base, int32_t pos_offset, gt_buf gy, gt_buf gx,
            int32_t accum) {
  GT_QUEUED(ctx, rows > 0 && H > 0 && hd > 0 && hd % 2 == 0 && gy && gx && in_batch(ctx, rows), now_gt_rope_bwd(ctx, rows, H, hd, base,
            pos_offset, gy, gx, accum));
}
gt_status gt_attention_fwd(gt_ctx* ctx, int32_t rows, int32_t Hq, int32_t Hkv, int32_t hd, int32_t window, gt_buf q, gt_buf k, gt_buf v,
            gt_buf out, gt_buf lse) {
  GT_QUEUED(ctx, heads(rows, Hq, Hkv, hd, window) && in_batch(ctx, rows) && q && k && v && out && lse, now_gt_attention_fwd(ctx, rows, Hq,
            Hkv, hd, window, q, k, v, out, lse));
}
gt_status gt_attention_bwd(gt_ctx* ctx, int32_t rows, int32_t Hq, int32_t Hkv, int32_t hd, int32_t window, gt_buf q, gt_buf k, gt_buf v,
            gt_buf out, gt_buf lse, gt_buf gout, gt_buf gq, int32_t accum_q, gt_buf gk, int32_t accum_k, gt_buf gv, int32_t accum_v) {
  GT_QUEUED(ctx, heads(rows, Hq, Hkv, hd, window) && in_batch(ctx, rows) && q && k && v && out && lse && gout, now_gt_attention_bwd(ctx,
            rows, Hq, Hkv, hd, window, q, k, v, out, lse, gout, gq, accum_q, gk, accum_k, gv, accum_v));
}
gt_status gt_attention_bwd_rope(gt_ctx* ctx, int32_t rows, int32_t Hq, int32_t Hkv, int32_t hd, int32_t window, gt_buf q, gt_buf k,
            gt_buf v, gt_buf out, gt_buf lse, gt_buf gout, gt_buf gq, int32_t accum_q, gt_buf gk, int32_t accum_k, gt_buf gv,
            int32_t accum_v, double base, int32_t pos_offset) {
  GT_QUEUED(ctx, heads(rows, Hq, Hkv, hd, window) && hd % 2 == 0 && in_batch(ctx, rows) && q && k && v && out && lse && gout,
            now_gt_attention_bwd_rope(ctx, rows, Hq, Hkv, hd, window, q, k, v, out, lse, gout, gq, accum_q, gk, accum_k, gv, accum_v, base,
            pos_offset));
}
gt_status gt_ce_fwd(gt_ctx* ctx, int32_t rows, int32_t V, gt_buf logits, gt_buf targets, gt_buf stats, gt_buf loss, gt_buf inv_kept) {
  GT_QUEUED(ctx, rows > 0 && V > 0 && in_batch(ctx, rows) && logits && targets && stats && loss && inv_kept, now_gt_ce_fwd(ctx, rows, V,
            logits, targets, stats, loss, inv_kept));
}
gt_status gt_ce_bwd(gt_ctx* ctx, int32_t rows, int32_t V, gt_buf logits, gt_buf targets, gt_buf stats, gt_buf inv_kept, gt_buf gloss,
            gt_buf glogits, int32_t accum) {
  GT_QUEUED(ctx, rows > 0 && V > 0 && logits && targets && stats && inv_kept && gloss, now_gt_ce_bwd(ctx, rows, V, logits, targets, stats,
            inv_kept, gloss, glogits, accum));
}
gt_status gt_ce_chunk_stats(gt_ctx* ctx, int32_t rows, int32_t n, int32_t v0, int32_t first, gt_buf chunk, gt_buf targets, gt_buf run) {
  GT_QUEUED(ctx, rows > 0 && n > 0 && v0 >= 0 && chunk && targets && run, now_gt_ce_chunk_stats(ctx, rows, n, v0, first, chunk, targets,
            run));
}
gt_status gt_ce_loss_from_stats(gt_ctx* ctx, int32_t rows, gt_buf run, gt_buf targets, gt_buf loss, gt_buf inv_kept) {
  GT_QUEUED(ctx, rows > 0 && in_batch(ctx, rows) && run && targets && loss && inv_kept, now_gt_ce_loss_from_stats(ctx, rows, run, targets,
            loss, inv_kept));
}
gt_status gt_ce_chunk_grad(gt_ctx* ctx, int32_t rows, int32_t n, int32_t v0, gt_buf chunk, gt_buf targets, gt_buf run, gt_buf inv_kept,
            gt_buf gloss) {
  GT_QUEUED(ctx, rows > 0 && n > 0 && chunk && targets && run && inv_kept && gloss, now_gt_ce_chunk_grad(ctx, rows, n, v0, chunk, targets,
            run, inv_kept, gloss));
}
gt_status gt_readout_ce_fwd(gt_ctx* ctx, int32_t rows, int32_t V, int32_t h, gt_buf hidden, gt_buf w, gt_buf logits, gt_buf targets,
            gt_buf stats, gt_buf loss, gt_buf inv_kept) {
  GT_QUEUED(ctx, rows > 0 && V > 0 && h > 0 && in_batch(ctx, rows) && hidden && w && logits && targets && stats && loss && inv_kept,
            now_gt_readout_ce_fwd(ctx, rows, V, h, hidden, w, logits, targets, stats, loss, inv_kept));
}
gt_status gt_readout_ce_stats(gt_ctx* ctx, int32_t rows, int32_t n, int32_t h, int32_t v0, int32_t first, gt_buf hidden, gt_buf w,
            gt_buf chunk, gt_buf targets, gt_buf run) {
  GT_QUEUED(ctx, rows > 0 && n > 0 && h > 0 && v0 >= 0 && hidden && w && chunk && targets && run, now_gt_readout_ce_stats(ctx, rows, n, h,
            v0, first, hidden, w, chunk, targets, run));
}
gt_status gt_readout_ce_grad(gt_ctx* ctx, int32_t rows, int32_t n, int32_t h, int32_t v0, gt_buf hidden, gt_buf w, gt_buf chunk,
            gt_buf targets, gt_buf run, gt_buf inv_kept, gt_buf gloss) {
  GT_QUEUED(ctx, rows > 0 && n > 0 && h > 0 && v0 >= 0 && hidden && w && chunk && targets && run && inv_kept && gloss,
            now_gt_readout_ce_grad(ctx, rows, n, h, v0, hidden, w, chunk, targets, run, inv_kept, gloss));
}
gt_status gt_soft_ce_fwd(gt_ctx* ctx, int32_t rows, int32_t V, int32_t k, gt_buf logits, gt_buf tids, gt_buf tprobs, gt_buf stats,
            gt_buf loss, gt_buf inv_kept) {
  GT_QUEUED(ctx, rows > 0 && V > 0 && k > 0 && in_batch(ctx, rows) && logits && tids && tprobs && stats && loss && inv_kept,
            now_gt_soft_ce_fwd(ctx, rows, V, k, logits, tids, tprobs, stats, loss, inv_kept));
}
gt_status gt_soft_ce_bwd(gt_ctx* ctx, int32_t rows, int32_t V, int32_t k, gt_buf logits, gt_buf tids, gt_buf tprobs, gt_buf stats,
            gt_buf inv_kept, gt_buf gloss, gt_buf glogits, int32_t accum) {
  GT_QUEUED(ctx, rows > 0 && V > 0 && k > 0 && logits && tids && tprobs && stats && inv_kept && gloss, now_gt_soft_ce_bwd(ctx, rows, V, k,
            logits, tids, tprobs, stats, inv_kept, gloss, glogits, accum));
}
gt_status gt_zero(gt_ctx* ctx, gt_buf buf, uint64_t bytes) {
  GT_QUEUED(ctx, true, now_gt_zero(ctx, buf, bytes));
}
gt_status gt_copy(gt_ctx* ctx, gt_buf dst, gt_buf src, uint64_t bytes) {
  GT_QUEUED(ctx, true, now_gt_copy(ctx, dst, src, bytes));
}

// ---- entry points with arrays: copied into the record ----
gt_status gt_gemm_multi(gt_ctx* ctx, int32_t kind, int32_t accum, int32_t M, int32_t N, int32_t nparts, const int32_t* Ks, const gt_buf* as,
                        const gt_buf* bs, gt_buf c) {
  struct { int32_t k[8]; gt_buf a[8], b[8]; } v = {};
  bool ok = M > 0 && N > 0 && nparts >= 1 && nparts <= 8 && Ks && as && bs && c;
  for (int p = 0; ok && p < nparts; p++) {
    ok = Ks[p] > 0 && as[p] && bs[p];
    v.k[p] = Ks[p]; v.a[p] = as[p]; v.b[p] = bs[p];
  }
  if (!ok) {
    const gt_status s = gt_drain(ctx);
    return s ? s : now_gt_gemm_multi(ctx, kind, accum, M, N, nparts, Ks, as, bs, c);
  }
  GT_QUEUED(ctx, true, now_gt_gemm_multi(ctx, kind, accum, M, N, nparts, v.k, v.a, v.b, c));
}
gt_status gt_gemm_grouped_scaled(gt_ctx* ctx, int32_t kind, int32_t ngroups, const int32_t* Ms, const int32_t* Ns, int32_t K, const gt_buf* as,
                                 const gt_buf* bs, const gt_buf* cs, const int32_t* accums, float alpha) {
  struct { int32_t m[8], n[8], acc[8]; gt_buf a[8], b[8], c[8]; } v = {};
  bool ok = ngroups >= 1 && ngroups <= 8 && K > 0 && Ms && Ns && as && bs && cs && accums;
  for (int g = 0; ok && g < ngroups; g++) {
    ok = Ms[g] > 0 && Ns[g] > 0 && as[g] && bs[g] && cs[g];
    v.m[g] = Ms[g]; v.n[g] = Ns[g]; v.acc[g] = accums[g]; v.a[g] = as[g]; v.b[g] = bs[g]; v.c[g] = cs[g];
  }
  if (!ok) {
    const gt_status s = gt_drain(ctx);
    return s ? s : now_gt_gemm_grouped_scaled(ctx, kind, ngroups, Ms, Ns, K, as, bs, cs, accums, alpha);
  }
  GT_QUEUED(ctx, true, now_gt_gemm_grouped_scaled(ctx, kind, ngroups, v.m, v.n, K, v.a, v.b, v.c, v.acc, alpha));
}
gt_status gt_gemm_grouped(gt_ctx* ctx, int32_t kind, int32_t ngroups, const int32_t* Ms, const int32_t* Ns, int32_t K, const gt_buf* as,
                          const gt_buf* bs, const gt_buf* cs, const int32_t* accums) {
  return gt_gemm_grouped_scaled(ctx, kind, ngroups, Ms, Ns, K, as, bs, cs, accums, 1.f);
}
gt_status gt_linear_rope_grouped(gt_ctx* ctx, int32_t ngroups, int32_t rows, int32_t K, gt_buf x, const int32_t* Ns, const gt_buf* ws,
                                 const gt_buf* ys, const int32_t* hs, int32_t hd, double base, int32_t pos_offset) {
  struct { int32_t n[8], h[8]; gt_buf w[8], y[8]; } v = {};
  bool ok = ngroups >= 1 && ngroups <= 8 && rows > 0 && K > 0 && x && Ns && ws && ys && hs && hd > 0 && hd % 2 == 0 && in_batch(ctx, rows);
  for (int g = 0; ok && g < ngroups; g++) {
    ok = Ns[g] > 0 && ws[g] && ys[g] && (hs[g] == 0 || hs[g] * hd == Ns[g]);
    v.n[g] = Ns[g]; v.h[g] = hs[g]; v.w[g] = ws[g]; v.y[g] = ys[g];
  }
  if (!ok) {
    const gt_status s = gt_drain(ctx);
    return s ? s : now_gt_linear_rope_grouped(ctx, ngroups, rows, K, x, Ns, ws, ys, hs, hd, base, pos_offset);
  }
  GT_QUEUED(ctx, true, now_gt_linear_rope_grouped(ctx, ngroups, rows, K, x, v.n, v.w, v.y, v.h, hd, base, pos_offset));
}
// Small writes (token ids, targets) keep their place among the ops through a copy of their own; large ones are made at once.
gt_status gt_write(gt_ctx* ctx, gt_buf dst, const void* host, uint64_t bytes) {
  GtQueue* q = queue_of(ctx, dst && host && bytes > 0 && bytes <= (256u << 10));
  char* copy = q && !q->failed.load(std::memory_order_relaxed) ? (char*)malloc(bytes) : nullptr;
  if (!copy) {
    const gt_status s = gt_drain(ctx);
    return s ? s : now_gt_write(ctx, dst, host, bytes);
  }
  memcpy(copy, host, bytes);
  return q->put([=]() -> gt_status {
    const gt_status s = gt_skip_queued(ctx) ? GT_OK : now_gt_write(ctx, dst, copy, bytes);
    free(copy);
    return s;
  });
}

}  // extern "C"
