// gb_serve.cu -- a request loop for Boolean operators on layers resident in HBM.
//
// Layers are added once and binned into a long-lived context.  Requests
// (AND / NOT / OR / XOR / GROW / SIZE on one or two resident layers) arrive on
// a schedule; the loop admits an arrived request as soon as an execution slot
// is free and the estimated device memory of all requests in flight fits the
// budget, runs it asynchronously on the slot's own stream and arena (so the
// work of concurrent requests overlaps on the GPU), and retires requests as
// their completion events fire.  Requests that arrive while others run are
// admitted as slots and memory free up: batching is continuous, not a queue
// drained in rounds.  Latency = completion - arrival, on the host clock.
#include <algorithm>
#include <chrono>
#include <cstring>
#include <deque>
#include <thread>
#include <vector>

#include "gbool.h"
#include "gb_internal.h"

using namespace gbi;

// What a request leaves for the host, written to pinned memory by its last
// kernel: nothing is copied and no stream is waited for when it retires.
struct gb_served {
  long long count;  // strips of the result
  int err;          // GB_* status of the slot's context
};

struct gb_server_slot {
  gb_context* ctx = nullptr;
  cudaEvent_t done = nullptr;
  int req = -1;
  unsigned long long mark = 0;  // the slot's empty arena, for its lifetime
  long long est = 0;
  gb_layer* out = nullptr;
  gb_served* back = nullptr;  // pinned
};

struct gb_server {
  int device = 0;
  unsigned long long budget = 0;
  gb_context* home = nullptr;  // owns the resident (binned) layers
  std::vector<gb_layer*> raw, binned;
  std::vector<long long> nbox;
  std::vector<gb_server_slot> slots;
  std::vector<std::vector<c_box>> kept;  // results copied out when requested
};

namespace {

// rewind (may be null): the arena goes back there, the result is not needed.
__global__ void k_served(const DLayer* L, DStatus* st, gb_served* back, const unsigned long long* rewind) {
  back->count = L->cell_count ? L->cell_count[0] : -1;
  back->err = st->err;
  if (rewind) st->arena_off = *rewind;
}

long long estimate(const gb_server* S, const gb_request& r) {
  long long n = S->nbox[r.a] + (r.op <= GB_OP_NOT ? S->nbox[r.b] : 0);
  if (r.op == GB_REQ_SIZE && r.amount < 0) n *= 3;  // erosion runs two Booleans on the complement
  return 48ll * n + (4ll << 20);
}

// CTAs that a request's operators may share tiles with when k requests are in flight or waiting for a slot.  CTAs that
// share a tile repeat its ranking, which pays on idle SMs only: all of them for one request, fewer the more run beside
// it.  40 requests (us; 8 slots with a burst / 3 slots with a burst / one at a time) by this rule, with half of the
// chip whatever k, the whole chip, none: on 20000 boxes 731 / 1276 / 3082, 749 / 1275 / 3242, 1028 / 1386 / 3095, 677 /
// 1390 / 3836; on 60000 1062 / 1599 / 3734, 1113 / 1610 / 3975, 1332 / 1730 / 3782, 1027 / 1527 / 3967; on 2000 all but
// none (1278 us with 3 slots, 3553 one at a time) within 3% of 637 / 1157 / 2950.
int shared_ctas(int full, int k) { return full * 2 / (k + 1) / 8 * 8; }

gb_layer* issue(gb_server* S, gb_server_slot& sl, const gb_request& r, int* status) {
  gb_layer* O = nullptr;
  int e = GB_ERR_ARG;
  gb_layer* A = S->binned[r.a];
  switch (r.op) {
    case GB_OP_XOR:
    case GB_OP_OR:
    case GB_OP_AND:
    case GB_OP_NOT:
      e = gb_op_bool(sl.ctx, r.op, A, S->binned[r.b], &O);
      break;
    case GB_REQ_GROW:
      e = gb_op_grow(sl.ctx, A, r.amount, r.amount, r.amount, r.amount, &O);
      break;
    case GB_REQ_SIZE:
      e = gb_op_size(sl.ctx, A, r.amount, &O);
      break;
    default:
      break;
  }
  *status = e;
  return e ? nullptr : O;
}

}  // namespace

extern "C" int gb_serve_create(int device, unsigned long long budget_bytes, int slots,
                               unsigned long long slot_arena_bytes, gb_server** out) {
  if (!out || slots < 1 || slots > 64) return GB_ERR_ARG;
  gb_server* S = new gb_server();
  S->device = device;
  S->budget = budget_bytes;
  int e = gb_context_create(device, slot_arena_bytes, &S->home);
  if (e) { delete S; return e; }
  for (int i = 0; i < slots; ++i) {
    gb_server_slot sl;
    e = gb_context_create(device, slot_arena_bytes, &sl.ctx);
    if (!e) e = gb_set_tile_scratch(sl.ctx, 4ull << 20);
    if (!e && cudaEventCreateWithFlags(&sl.done, cudaEventDisableTiming) != cudaSuccess) e = GB_ERR_OOM;
    // written by kernels: without it no request may run
    if (!e && cudaMallocHost(&sl.back, sizeof(gb_served)) != cudaSuccess) e = GB_ERR_OOM;
    if (e) {
      S->slots.push_back(sl);  // what it has is freed with the others
      break;
    }
    sl.mark = gb_arena_mark(sl.ctx);
    S->slots.push_back(sl);
  }
  if (e) {
    cudaGetLastError();
    gb_serve_destroy(S);
    return e;
  }
  *out = S;
  return GB_OK;
}

extern "C" int gb_serve_add_layer(gb_server* S, const c_box* boxes, unsigned long long n, int* id) {
  if (!S || !id) return GB_ERR_ARG;
  gb_layer* L = nullptr;
  int e = gb_layer_from_host(S->home, boxes, n, nullptr, 1, &L);
  if (e) return e;
  // bin once; the binned form lives in the home context's arena for the server's lifetime
  gb_layer* B = binned_of(S->home, L, 16);
  if (!B) {
    gb_layer_free(S->home, L);  // not recorded: gb_serve_destroy would never free it
    return GB_ERR_CAPACITY;
  }
  e = gb_sync(S->home, nullptr);
  if (e) {
    gb_layer_free(S->home, B);
    gb_layer_free(S->home, L);
    return e;
  }
  *id = (int)S->raw.size();
  S->raw.push_back(L);
  S->binned.push_back(B);
  S->nbox.push_back((long long)n);
  return GB_OK;
}

extern "C" int gb_serve_run(gb_server* S, const gb_request* reqs, int nreq, gb_result* res, int keep_outputs) {
  if (!S || (nreq && (!reqs || !res))) return GB_ERR_ARG;
  using clk = std::chrono::steady_clock;
  const auto t0 = clk::now();
  auto now_s = [&]() { return std::chrono::duration<double>(clk::now() - t0).count(); };
  if (keep_outputs) S->kept.assign(nreq, {});
  for (int i = 0; i < nreq; ++i) {
    res[i] = gb_result{};
    res[i].status = -1;
    if (reqs[i].a < 0 || reqs[i].a >= (int)S->raw.size() ||
        (reqs[i].op <= GB_OP_NOT && (reqs[i].b < 0 || reqs[i].b >= (int)S->raw.size())))
      res[i].status = GB_ERR_ARG;
  }
  std::deque<int> waiting;
  int next = 0, done = 0;
  long long inflight = 0;
  while (done < nreq) {
    const double t = now_s();
    while (next < nreq && reqs[next].arrival_s <= t) waiting.push_back(next++);
    // retire finished requests
    for (gb_server_slot& sl : S->slots) {
      if (sl.req < 0 || cudaEventQuery(sl.done) != cudaSuccess) continue;
      const int i = sl.req;
      const int e = cudaGetLastError() != cudaSuccess ? GB_ERR_CUDA : sl.back->err;  // a failed launch leaves no status
      res[i].status = e;
      res[i].count = sl.back->count;
      if (!e && keep_outputs && sl.out) {
        unsigned long long n = 0;
        gb_layer_to_host(sl.ctx, sl.out, nullptr, 0, &n, nullptr);
        S->kept[i].resize(n);
        gb_layer_to_host(sl.ctx, sl.out, S->kept[i].data(), n, &n, nullptr);
      }
      res[i].end_s = now_s();
      res[i].latency_ms = (res[i].end_s - reqs[i].arrival_s) * 1e3;
      if (e) gb_clear_status(sl.ctx);
      arena_rewind(sl.ctx, sl.mark, keep_outputs != 0);
      inflight -= sl.est;
      sl.req = -1;
      sl.out = nullptr;
      ++done;
    }
    // admit arrived requests in order while a slot is free and the budget allows
    while (!waiting.empty()) {
      const int i = waiting.front();
      if (res[i].status == GB_ERR_ARG) {
        waiting.pop_front();
        res[i].end_s = now_s();
        ++done;
        continue;
      }
      const long long est = estimate(S, reqs[i]);
      if (est > (long long)S->budget) {  // can never fit: refuse
        waiting.pop_front();
        res[i].status = GB_ERR_CAPACITY;
        res[i].end_s = now_s();
        ++done;
        continue;
      }
      gb_server_slot* free_slot = nullptr;
      for (gb_server_slot& sl : S->slots)
        if (sl.req < 0) { free_slot = &sl; break; }
      if (!free_slot || inflight + est > (long long)S->budget) break;
      waiting.pop_front();
      gb_server_slot& sl = *free_slot;
      res[i].start_s = now_s();
      int st = 0;
      int k = 1 + (int)waiting.size();
      for (const gb_server_slot& o : S->slots) k += o.req >= 0;
      sl.ctx->c.split_ctas = shared_ctas(S->home->c.split_ctas, std::min(k, (int)S->slots.size()));
      sl.out = issue(S, sl, reqs[i], &st);
      if (!sl.out) {
        res[i].status = st;
        res[i].end_s = now_s();
        arena_rewind(sl.ctx, sl.mark, true);
        ++done;
        continue;
      }
      k_served<<<1, 1, 0, sl.ctx->c.stream>>>(sl.out->d, sl.ctx->c.st, sl.back,
                                              keep_outputs ? nullptr : mark_word(sl.ctx, sl.mark));
      cudaEventRecord(sl.done, sl.ctx->c.stream);
      sl.req = i;
      sl.est = est;
      inflight += est;
    }
    if (done < nreq) {
      bool busy = false;
      for (gb_server_slot& sl : S->slots) busy |= sl.req >= 0;
      if (!busy && waiting.empty() && next < nreq) {
        const double wait = reqs[next].arrival_s - now_s();
        if (wait > 0) std::this_thread::sleep_for(std::chrono::duration<double>(std::min(wait, 0.001)));
      } else {
        std::this_thread::yield();
      }
    }
  }
  return GB_OK;
}

extern "C" int gb_serve_result_boxes(gb_server* S, int i, c_box* out, unsigned long long cap,
                                     unsigned long long* n) {
  if (!S || !n || i < 0 || i >= (int)S->kept.size()) return GB_ERR_ARG;
  *n = S->kept[i].size();
  if (*n > cap) return GB_ERR_CAPACITY;
  if (*n && out) memcpy(out, S->kept[i].data(), *n * sizeof(c_box));
  return GB_OK;
}

extern "C" void gb_serve_destroy(gb_server* S) {
  if (!S) return;
  for (gb_server_slot& sl : S->slots) {
    if (sl.ctx) gb_sync(sl.ctx, nullptr);
    if (sl.done) cudaEventDestroy(sl.done);
    if (sl.back) cudaFreeHost(sl.back);
    if (sl.ctx) gb_context_destroy(sl.ctx);
  }
  for (gb_layer* L : S->raw) gb_layer_free(S->home, L);
  if (S->home) gb_context_destroy(S->home);
  delete S;
}
