// extern "C" surface of libb200llm.so (include/b200_llm.h).
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <vector>

#include "graph.h"

using namespace b200;

struct b200_model { Model m; };
struct b200_graph { Graph g; };

namespace {
struct Scratch {   // device temporaries of one call
  std::vector<void*> ptrs;
  ~Scratch() { for (void* p : ptrs) cudaFree(p); }
  template <class T> int get(T** out, size_t bytes) {
    void* p = nullptr;
    cudaError_t e = cudaMalloc(&p, bytes ? bytes : 1);
    if (e != cudaSuccess) { set_error(std::string("device allocation of ") + std::to_string(bytes) + " bytes failed: " + cudaGetErrorString(e)); return ENOMEM_; }
    ptrs.push_back(p);
    *out = (T*)p;
    return OK;
  }
};

// Pinned host blocks for results (b200_host_acquire). One cache per process, because what is expensive is pinning the
// pages (about a millisecond per four megabytes), not handing a block out: blocks go back to it and serve whichever
// graph asks next. Bounded: at most POOL_MAX bytes exist at a time, in use or not, and at most POOL_IDLE of them idle.
struct HostPool {
  static constexpr size_t POOL_MAX = (size_t)1 << 30, POOL_IDLE = (size_t)256 << 20;
  std::mutex mu;
  struct Block { size_t size; bool idle; };
  std::multimap<size_t, void*> idle;
  std::map<void*, Block> blocks;
  size_t total = 0, idle_bytes = 0;

  void drop_largest() {   // mu held
    auto it = std::prev(idle.end());
    cudaFreeHost(it->second);
    total -= it->first; idle_bytes -= it->first;
    blocks.erase(it->second);
    idle.erase(it);
  }
  void* acquire(size_t bytes) {
    const size_t unit = bytes > ((size_t)1 << 20) ? (size_t)1 << 20 : (size_t)64 << 10, want = (bytes + unit - 1) / unit * unit;
    std::lock_guard<std::mutex> lock(mu);
    auto it = idle.lower_bound(want);
    if (it != idle.end() && it->first <= 2 * want) {
      void* p = it->second;
      idle_bytes -= it->first;
      idle.erase(it);
      blocks[p].idle = false;
      return p;
    }
    while (!idle.empty() && total + want > POOL_MAX) drop_largest();
    void* p = nullptr;
    if (total + want > POOL_MAX || cudaHostAlloc(&p, want, cudaHostAllocPortable) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    total += want;
    blocks[p] = Block{want, false};
    return p;
  }
  bool owns(const void* p) {
    std::lock_guard<std::mutex> lock(mu);
    auto it = blocks.find(const_cast<void*>(p));
    return it != blocks.end() && !it->second.idle;
  }
  void release(void* p) {
    std::lock_guard<std::mutex> lock(mu);
    auto it = blocks.find(p);
    if (it == blocks.end() || it->second.idle) return;   // not a block, or given back already
    it->second.idle = true;
    idle.emplace(it->second.size, p);
    idle_bytes += it->second.size;
    while (idle_bytes > POOL_IDLE) drop_largest();
  }
};
HostPool& host_pool() {
  static HostPool* pool = new HostPool;   // never destroyed: arrays may be given back while the process ends
  return *pool;
}

// The output buffers a caller has set hold for one call, however it ends: made before the call looks at its arguments.
struct OutputsForOneCall {
  b200_graph* g;
  explicit OutputsForOneCall(b200_graph* graph) : g(graph) {}
  ~OutputsForOneCall() {
    if (g == nullptr) return;
    g->g.out_logits = g->g.out_resid = nullptr;
    g->g.out_logits_cap = g->g.out_resid_cap = 0;
  }
};
}  // namespace

extern "C" {

const char* b200_last_error(void) { return last_error(); }

int32_t b200_device_count(void) {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess) return 0;
  return n;
}

int32_t b200_model_new(const b200_config* cfg, int32_t device, b200_model** out) {
  if (!cfg || !out) { set_error("model_new: null argument"); return EINVAL_; }
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) { set_error("no CUDA device: this library has no CPU path"); return ECUDA; }
  if (device < 0 || device >= n) { set_error("model_new: no such device"); return EINVAL_; }
  auto* m = new (std::nothrow) b200_model();
  if (!m) return ENOMEM_;
  m->m.c = *cfg; m->m.device = device;
  *out = m;
  return OK;
}
int32_t b200_model_add_tensor(b200_model* m, const char* name, uint32_t type, uint32_t n_dims, const int64_t* dims, const void* host) {
  if (!m || !name || !dims || !host) { set_error("add_tensor: null argument"); return EINVAL_; }
  return m->m.add_host(name, type, n_dims, dims, host);
}
int32_t b200_model_add_synthetic(b200_model* m, const char* name, uint32_t type, uint32_t n_dims, const int64_t* dims, uint64_t seed, int32_t rule, float p0, float p1) {
  if (!m || !name || !dims) { set_error("add_synthetic: null argument"); return EINVAL_; }
  return m->m.add_synthetic(name, type, n_dims, dims, seed, rule, p0, p1);
}
int32_t b200_model_finalize(b200_model* m) { if (!m) { set_error("null model"); return EINVAL_; } return m->m.finalize(); }
int32_t b200_model_open_gguf(const char* path, int32_t device, b200_model** out) {
  if (!path || !out) { set_error("open_gguf: null argument"); return EINVAL_; }
  auto* bm = new (std::nothrow) b200_model();
  if (!bm) return ENOMEM_;
  int s = load_gguf_into(path, device, &bm->m);
  if (s != OK) { delete bm; return s; }
  *out = bm;
  return OK;
}
int32_t b200_model_config(const b200_model* m, b200_config* out) { if (!m || !out) return EINVAL_; *out = m->m.c; return OK; }
int64_t b200_model_weight_bytes(const b200_model* m) { return m ? m->m.weight_bytes : 0; }
int64_t b200_model_tensor_bytes(const b200_model* m, const char* name) {
  if (!m || !name) return -1;
  auto it = m->m.tensors.find(name);
  if (it == m->m.tensors.end()) return -1;
  return gguf_row_bytes(it->second.type, it->second.k) * it->second.rows;
}
int32_t b200_model_read_tensor(const b200_model* m, const char* name, void* dst, int64_t nbytes) {
  if (!m || !name || !dst) { set_error("read_tensor: null argument"); return EINVAL_; }
  return m->m.read_tensor(name, dst, nbytes);
}
void b200_model_free(b200_model* m) { delete m; }

int32_t b200_graph_create(b200_model* m, const b200_graph_opts* opts, b200_graph** out) {
  if (!m || !opts || !out) { set_error("graph_create: null argument"); return EINVAL_; }
  auto* g = new (std::nothrow) b200_graph();
  if (!g) return ENOMEM_;
  int s = g->g.init(&m->m, *opts);
  if (s != OK) { delete g; return s; }
  *out = g;
  return OK;
}
void b200_graph_destroy(b200_graph* g) { delete g; }
int32_t b200_graph_slots(const b200_graph* g) { return g ? g->g.o.slots : 0; }
int32_t b200_graph_nkv(const b200_graph* g) { return g ? g->g.o.n_kv : 0; }
int32_t b200_graph_use_slot(b200_graph* g, int32_t slot) {
  if (!g) return EINVAL_;
  if (slot < 0 || slot >= g->g.o.slots) { set_error("use_slot: slot " + std::to_string(slot) + " does not exist"); return EINVAL_; }
  g->g.cur = slot; g->g.dcur = slot; g->g.spec_n = 0;
  return OK;
}
int32_t b200_graph_reset(b200_graph* g) { if (!g) return EINVAL_; return g->g.reset_slot(g->g.cur); }
int32_t b200_graph_set_past(b200_graph* g, int32_t past) {
  if (!g) return EINVAL_;
  if (past < 0 || past > g->g.o.n_kv) { set_error("set_past: position outside the slot's context"); return EINVAL_; }
  g->g.past[g->g.cur] = past; g->g.spec_n = 0;
  return OK;
}
int32_t b200_graph_past(const b200_graph* g) { return g ? g->g.past[g->g.cur] : 0; }

void* b200_host_acquire(b200_graph* g, int64_t bytes) {
  if (!g || bytes <= 0 || cudaSetDevice(g->g.m->device) != cudaSuccess) return nullptr;
  return host_pool().acquire((size_t)bytes);
}
void b200_host_release(void* p) { if (p) host_pool().release(p); }
int32_t b200_graph_set_outputs(b200_graph* g, float* logits, int64_t logit_floats, float* residual, int64_t residual_floats) {
  if (!g) { set_error("set_outputs: null argument"); return EINVAL_; }
  g->g.out_logits = logits; g->g.out_logits_cap = logits ? logit_floats : 0;
  g->g.out_resid = residual; g->g.out_resid_cap = residual ? residual_floats : 0;
  g->g.out_logits_mapped = logits && host_pool().owns(logits); g->g.out_resid_mapped = residual && host_pool().owns(residual);
  return OK;
}
int32_t b200_graph_forward(b200_graph* g, const int32_t* ids, int32_t n, const float** logits, const float** hidden) {
  OutputsForOneCall once(g);
  if (!g || !ids) { set_error("forward: null argument"); return EINVAL_; }
  B200_TRY(g->g.outputs_fit(g->g.m->c.vocab, 0));
  B200_TRY(g->g.reset_slot(g->g.cur));
  PassFlags f;
  return g->g.extend(ids, n, f, logits, hidden);
}
int32_t b200_graph_extend(b200_graph* g, const int32_t* ids, int32_t n, const float** logits, const float** hidden) {
  OutputsForOneCall once(g);
  if (!g || !ids) { set_error("extend: null argument"); return EINVAL_; }
  PassFlags f;
  return g->g.extend(ids, n, f, logits, hidden);
}
int32_t b200_graph_extend_input(b200_graph* g, const b200_input* in, const float** logits, const float** hidden) {
  OutputsForOneCall once(g);
  if (!g || !in || !in->ids) { set_error("extend_input: null argument"); return EINVAL_; }
  if (in->n_images != 0) { set_error("extend_input: this library has no vision tower; inputs with images are refused"); return EINVAL_; }
  PassFlags f;
  return g->g.extend(in->ids, in->n, f, logits, hidden);
}
int32_t b200_graph_extend_rows(b200_graph* g, const int32_t* ids, int32_t n, const float** logits, const float** residual) {
  OutputsForOneCall once(g);
  if (!g || !ids) { set_error("extend_rows: null argument"); return EINVAL_; }
  PassFlags f; f.want_all_logits = true; f.want_residual = true; f.spec = g->g.speculating;
  return g->g.extend(ids, n, f, logits, residual);
}
int32_t b200_graph_extend_residual(b200_graph* g, const int32_t* ids, int32_t n, const float** logits, const float** residual) {
  OutputsForOneCall once(g);
  if (!g || !ids) { set_error("extend_residual: null argument"); return EINVAL_; }
  PassFlags f; f.want_residual = true;
  return g->g.extend(ids, n, f, logits, residual);
}
int32_t b200_graph_decode_rows(b200_graph* g, const int32_t* slots, const int32_t* ids, int32_t n, const float** logits) {
  OutputsForOneCall once(g);
  if (!g || !slots || !ids) { set_error("decode_rows: null argument"); return EINVAL_; }
  return g->g.decode_rows(slots, ids, n, logits);
}
int32_t b200_graph_checkpoint(b200_graph* g, int32_t* handle) { if (!g || !handle) return EINVAL_; return g->g.checkpoint(handle); }
int32_t b200_graph_restore(b200_graph* g, int32_t handle) { if (!g) return EINVAL_; return g->g.restore(handle); }
int32_t b200_graph_checkpoint_free(b200_graph* g, int32_t handle) {
  if (!g) return EINVAL_;
  auto it = g->g.ckpts.find(handle);
  if (it == g->g.ckpts.end()) { set_error("checkpoint_free: unknown checkpoint"); return EINVAL_; }
  cudaSetDevice(g->g.m->device);
  for (float* p : it->second.state) cudaFree(p);
  for (float* p : it->second.ring) cudaFree(p);
  g->g.ckpts.erase(it);
  return OK;
}
int32_t b200_graph_speculate(b200_graph* g, int32_t on) {
  if (!g) return EINVAL_;
  if (on && !g->g.o.speculative) { set_error("speculate: the graph was created with speculative = 0"); return ESTATE; }
  g->g.speculating = on != 0;
  return OK;
}
int32_t b200_graph_speculating(const b200_graph* g) { return g && g->g.speculating ? 1 : 0; }
int32_t b200_graph_speculate_first(b200_graph* g, int32_t on) {
  if (!g) return EINVAL_;
  if (g->g.spec_n > 0) { set_error("speculate_first: a speculative pass is in flight; commit or rewind it first"); return ESTATE; }
  g->g.spec_first = on != 0;
  return OK;
}
int32_t b200_graph_keep(b200_graph* g, int32_t k) { if (!g) return EINVAL_; return g->g.keep(k); }
int32_t b200_graph_keep_first(b200_graph* g) { if (!g) return EINVAL_; return g->g.keep(1); }
int32_t b200_graph_commit(b200_graph* g) { if (!g) return EINVAL_; return g->g.keep(g->g.spec_n); }
int32_t b200_graph_rewind(b200_graph* g) {
  if (!g) return EINVAL_;
  // with SpeculateFirst on, row 0 of a pass is a token already emitted: the pass ends by Commit or KeepFirst (llm/graph.go:1166-1178)
  if (g->g.spec_first && g->g.spec_n > 0) { set_error("rewind: with speculate_first on a pass is ended by commit or keep_first"); return ESTATE; }
  return g->g.keep(0);
}
int32_t b200_graph_residual_row(b200_graph* g, int32_t r, float* dst) { if (!g || !dst) { set_error("residual_row: null argument"); return EINVAL_; } return g->g.residual_row(r, dst); }
int32_t b200_graph_pass_experts(b200_graph* g, int32_t* out) { if (!g || !out) { set_error("pass_experts: null argument"); return EINVAL_; } return g->g.pass_experts(out); }
uint32_t b200_graph_fp16_weight_mask(const b200_graph* g, int32_t rows, int32_t logit_rows) { return g ? g->g.fp16_weight_mask(rows, logit_rows) : 0; }
int32_t b200_graph_stats_get(const b200_graph* g, b200_graph_stats* out) {
  if (!g || !out) return EINVAL_;
  *out = g->g.stats;
  int64_t dev = 0;
  cudaSetDevice(g->g.m->device);
  if (cudaMemcpy(&dev, g->g.distinct_dev, sizeof(dev), cudaMemcpyDeviceToHost) != cudaSuccess) { set_error("stats: cannot read the device counter"); return ECUDA; }
  out->expert_streams = dev + g->g.single_row_layers * g->g.m->c.n_expert_used;
  return OK;
}
int32_t b200_graph_stats_reset(b200_graph* g) {
  if (!g) return EINVAL_;
  g->g.stats = b200_graph_stats{}; g->g.single_row_layers = 0;
  cudaSetDevice(g->g.m->device);
  if (cudaMemset(g->g.distinct_dev, 0, sizeof(int64_t)) != cudaSuccess) { set_error("stats: cannot clear the device counter"); return ECUDA; }
  return OK;
}
int32_t b200_graph_ep_export(b200_graph* g, int32_t rank, int32_t world, b200_ep_handle* out) { if (!g || !out) return EINVAL_; return g->g.ep_export(rank, world, out->bytes); }
int32_t b200_graph_ep_attach(b200_graph* g, const b200_ep_handle* handles) { if (!g || !handles) return EINVAL_; return g->g.ep_attach(handles); }
int32_t b200_graph_ep_prepare(b200_graph* g, int32_t rank, int32_t world) { if (!g) return EINVAL_; return g->g.ep_prepare(rank, world); }
int32_t b200_graph_ep_attach_local(b200_graph* g, b200_graph* const* graphs, int32_t world) {
  if (!g || !graphs || world < 1 || world > EP_MAX_RANKS) { set_error("ep_attach_local: bad argument"); return EINVAL_; }
  Graph* peers[EP_MAX_RANKS] = {};
  for (int i = 0; i < world; i++) peers[i] = graphs[i] ? &graphs[i]->g : nullptr;
  return g->g.ep_attach_local(peers, world);
}
int32_t b200_graph_ep_enable(b200_graph* g, int32_t on) {
  if (!g) return EINVAL_;
  if (on && !g->g.ep_ready) { set_error("ep_enable: attach the peers first"); return ESTATE; }
  g->g.ep_on = on != 0;
  return OK;
}
int32_t b200_graph_synth_context(b200_graph* g, int32_t cells, uint64_t seed) { if (!g) return EINVAL_; return g->g.synth_context(g->g.cur, cells, seed); }
int32_t b200_graph_inject_wait_timeout(b200_graph* g) { if (!g) return EINVAL_; return g->g.inject_wait_timeout(); }

int32_t b200_graph_generate_greedy(b200_graph* g, const int32_t* slots, const int32_t* first_ids, int32_t n, int32_t steps, int32_t* out_ids) {
  if (!g || !slots || !first_ids || !out_ids) { set_error("generate_greedy: null argument"); return EINVAL_; }
  return g->g.generate_greedy(slots, first_ids, n, steps, out_ids);
}
float b200_graph_last_device_ms(const b200_graph* g) { return g ? g->g.last_ms : 0.f; }
int32_t b200_graph_last_launches(const b200_graph* g) { return g ? g->g.last_launches : 0; }
int32_t b200_graph_timeline(b200_graph* g, int64_t* dst, int32_t max_launches) {
  if (!g || !dst) return -1;
  if (!g->g.timeline) return 0;
  cudaSetDevice(g->g.m->device);
  int n = g->g.last_launches < g->g.timeline_cap ? g->g.last_launches : g->g.timeline_cap;
  if (n > max_launches) n = max_launches;
  if (cudaMemcpy(dst, g->g.timeline, (size_t)n * 8 * sizeof(long long), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
  return n;
}
int64_t b200_graph_trace(b200_graph* g, int32_t what, void* dst, int64_t nbytes) { if (!g || !dst) return -EINVAL_; return g->g.trace(what, dst, nbytes); }

int32_t b200_draft_rows(b200_graph* g, const float* hs, const int32_t* ids, int32_t n, int32_t vocab_k, const float** residual, const float** logits) {
  OutputsForOneCall once(g);
  if (!g || !hs || !ids) { set_error("draft_rows: null argument"); return EINVAL_; }
  return g->g.draft_rows(hs, ids, n, vocab_k, residual, logits);
}
int32_t b200_draft_past(const b200_graph* g) { return g ? g->g.draft_past[g->g.dcur] : 0; }
int32_t b200_draft_rewind(b200_graph* g, int32_t past) {
  if (!g) return EINVAL_;
  if (past < 0 || past > g->g.draft_past[g->g.dcur]) { set_error("draft_rewind: position outside the draft cache"); return EINVAL_; }
  g->g.draft_past[g->g.dcur] = past;
  return OK;
}
int32_t b200_draft_set_vocab(b200_graph* g, int32_t k) {
  if (!g) return EINVAL_;
  if (k < 0 || k % 16 || k > g->g.m->c.vocab) { set_error("draft_set_vocab: a multiple of 16 up to the vocabulary size, or 0 for all of it"); return EINVAL_; }
  g->g.draft_vocab_default = k == g->g.m->c.vocab ? 0 : k;
  return OK;
}
int32_t b200_draft_use_slot(b200_graph* g, int32_t slot) {
  if (!g) return EINVAL_;
  if (slot < 0 || slot >= g->g.o.slots) { set_error("draft_use_slot: draft cache slot " + std::to_string(slot) + " of " + std::to_string(g->g.o.slots)); return EINVAL_; }
  g->g.dcur = slot;
  return OK;
}
int32_t b200_draft_slots(const b200_graph* g) { return g && g->g.m->c.has_draft ? g->g.o.slots : 0; }
int32_t b200_draft_reset(b200_graph* g) { if (!g) return EINVAL_; g->g.draft_past[g->g.dcur] = 0; return OK; }
int32_t b200_draft_max_rows(const b200_graph* g) { return g ? g->g.LR : 0; }
int32_t b200_draft_wide(const b200_graph* g) { return g ? g->g.m->c.n_embd : 0; }

// ---- unit entry points --------------------------------------------------------------------
// They run on the device that is current in the calling thread and free what they allocate on
// every path out.
static int need_device() {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) { set_error("no CUDA device: this library has no CPU path"); return ECUDA; }
  return OK;
}


int32_t b200_dequantize(uint32_t type, const void* host_data, int64_t n, float* host_out) {
  B200_TRY(need_device());
  int e, nb;
  if (!host_data || !host_out || !block_geometry(type, &e, &nb) || n % e || n <= 0) { set_error("dequantize: bad type or element count"); return EINVAL_; }
  const int64_t bytes = gguf_row_bytes(type, n);
  DTensor t; t.type = type; t.k = n; t.rows = 1; t.stride = device_row_stride(type, n);
  Scratch sc;
  uint8_t* src = nullptr; float* out = nullptr;
  B200_TRY(sc.get(&src, (size_t)bytes)); B200_TRY(sc.get(&t.data, (size_t)t.stride + 256)); B200_TRY(sc.get(&out, (size_t)n * sizeof(float)));
  B200_CUDA(cudaMemcpy(src, host_data, (size_t)bytes, cudaMemcpyHostToDevice));
  B200_TRY(repack_rows(type, n, 1, src, t.data, 0));
  B200_TRY(dequant_rows(t, 0, 1, out, 0));
  B200_CUDA(cudaMemcpy(host_out, out, (size_t)n * sizeof(float), cudaMemcpyDeviceToHost));
  return OK;
}

// weights in device layout, activations as fp16 rows, an error word: what both projection entry points stage
static int stage_projection(Scratch& sc, uint32_t type, const void* host_w, int64_t rows, int64_t k, const float* host_x, int32_t mrows,
                            DTensor* t, __half** x16, float** y, int** err) {
  const int64_t rb = gguf_row_bytes(type, k);
  if (rb < 0) { set_error("projection: bad type or row length"); return EINVAL_; }
  t->type = type; t->k = k; t->rows = rows; t->stride = device_row_stride(type, k);
  uint8_t* src = nullptr; float* xf = nullptr;
  B200_TRY(sc.get(&src, (size_t)(rb * rows))); B200_TRY(sc.get(&t->data, (size_t)(t->stride * rows) + 256));
  B200_TRY(sc.get(&xf, (size_t)mrows * k * sizeof(float))); B200_TRY(sc.get(x16, (size_t)mrows * k * sizeof(__half)));
  B200_TRY(sc.get(y, (size_t)mrows * rows * sizeof(float))); B200_TRY(sc.get(err, sizeof(int)));
  B200_CUDA(cudaMemset(*err, 0, sizeof(int)));
  B200_CUDA(cudaMemcpy(src, host_w, (size_t)(rb * rows), cudaMemcpyHostToDevice));
  B200_CUDA(cudaMemcpy(xf, host_x, (size_t)mrows * k * sizeof(float), cudaMemcpyHostToDevice));
  B200_TRY(repack_rows(type, k, rows, src, t->data, 0));
  B200_TRY(quantize_rows_device(T_F16, xf, mrows, k, (uint8_t*)*x16, 0));
  return OK;
}
static int finish_projection(const char* who, const float* y, const int* err, int64_t n, float* host_y) {
  int herr = 0;
  B200_CUDA(cudaMemcpy(&herr, err, sizeof(int), cudaMemcpyDeviceToHost));
  if (herr != 0) { set_error(std::string(who) + ": a bounded wait gave up"); return ETIMEOUT; }
  if (n > 0) B200_CUDA(cudaMemcpy(host_y, y, (size_t)n * sizeof(float), cudaMemcpyDeviceToHost));
  return OK;
}

int32_t b200_qgemv(uint32_t type, const void* host_w, int64_t rows, int64_t k, const float* host_x, int32_t mrows, float* host_y) {
  B200_TRY(need_device());
  if (!host_w || !host_x || !host_y || rows <= 0 || mrows <= 0) { set_error("qgemv: bad argument"); return EINVAL_; }
  Scratch sc; DTensor t; __half* x16 = nullptr; float* y = nullptr; int* err = nullptr;
  B200_TRY(stage_projection(sc, type, host_w, rows, k, host_x, mrows, &t, &x16, &y, &err));
  if (mrows > QG_MAXCOLS && tgemm_type(type)) {   // as the passes of more than eight rows do
    __half* sx = nullptr;
    B200_TRY(sc.get(&sx, (size_t)mrows * (k / 256) * TG_SX * sizeof(__half)));
    TGemmMaps maps{};
    B200_TRY(make_w_tensor_map(type, t.data, rows, t.stride, 128, &maps.w));
    B200_TRY(make_rows_map(x16, mrows, (int)k, tgemm_cols(mrows), &maps.x));
    B200_TRY(make_rows_map(sx, mrows, (int)(k / 256 * TG_SX), tgemm_cols(mrows), &maps.sx));
    maps.w2 = maps.w;
    B200_TRY(launch_row_sums(x16, mrows, (int)k, sx, false, 0));
    TGemmParams g{};
    g.K = (int)k; g.N = (int)rows; g.M = mrows; g.seg_end = (int)rows; g.ksplit = 1; g.y = y; g.ldy = rows; g.err = err;
    B200_TRY(launch_tgemm(type, tgemm_cols(mrows), g, maps, false, 0));
    return finish_projection("qgemv", y, err, (int64_t)mrows * rows, host_y);
  }
  QGemvParams p{};
  p.w[0] = t.data; p.seg_end[0] = (int)rows; p.nseg = 1; p.stride = t.stride; p.K = (int)k; p.N = (int)rows; p.M = mrows; p.xcols = mrows < QG_MAXCOLS ? mrows : QG_MAXCOLS;
  p.x = x16; p.ldx = k; p.y = y; p.ldy = rows; p.x_div = 1; p.err = err;
  QGemvMaps maps{};
  B200_TRY(make_qgemv_map(type, t.data, rows, t.stride, &maps.w[0]));
  B200_TRY(launch_qgemv(type, PRO_F16, EPI_STORE, false, false, p, maps, false, 0));
  return finish_projection("qgemv", y, err, (int64_t)mrows * rows, host_y);
}

int32_t b200_qgemm(uint32_t type, const void* host_w, int64_t rows, int64_t k, const float* host_x, int32_t mrows, int32_t tile_rows, float* host_y) {
  B200_TRY(need_device());
  if (!host_w || !host_x || !host_y || rows <= 0 || mrows <= 0) { set_error("qgemm: bad argument"); return EINVAL_; }
  Scratch sc; DTensor t; __half* x16 = nullptr; float* y = nullptr; int* err = nullptr;
  B200_TRY(stage_projection(sc, type, host_w, rows, k, host_x, mrows, &t, &x16, &y, &err));
  if (tile_rows != 64 && tile_rows != 128 && tile_rows != 256) { set_error("qgemm: activation tile must be 64, 128 or 256 rows"); return EINVAL_; }
  if (!wgemm_type(type) || (type == T_Q8_0 && tile_rows != 64)) { set_error("qgemm: weight type has no tensor-core projection kernel (Q4_K, Q5_K, Q6_K; Q8_0 with 64-row tiles)"); return EINVAL_; }
  WGemmMaps maps{};
  B200_TRY(make_wmap(type, t.data, rows, t.stride, 128, &maps.w));
  B200_TRY(make_rows_map(x16, mrows, (int)k, 64, &maps.x));
  WGemmParams p{};
  p.one = GemmProblem{0, 0, mrows, 0}; p.n_problems = 1; p.max_count = mrows; p.K = (int)k; p.N = (int)rows; p.ksplit = 1; p.y = y; p.ldy = rows; p.err = err;
  B200_TRY(launch_wgemm(type, WG_STORE, tile_rows, p, maps, false, 0));
  return finish_projection("qgemm", y, err, (int64_t)mrows * rows, host_y);
}

int32_t b200_qgemv_static(uint32_t type, const void* dev_w, int64_t rows, int64_t k, const float* dev_x, int32_t m, float* dev_y) {
  B200_TRY(need_device());
  return qgemv_static(type, dev_w, rows, k, dev_x, m, dev_y);
}

int32_t b200_attention(int32_t n_head, int32_t n_head_kv, int32_t head_dim, int32_t rows, int32_t cells, int32_t parts, const float* q, const float* k,
                       const float* v, const float* gate, float* out) {
  B200_TRY(need_device());
  if (!q || !k || !v || !gate || !out) { set_error("attention: null argument"); return EINVAL_; }
  if (n_head < 1 || n_head_kv < 1 || n_head % n_head_kv || !attn_tc_shape(n_head, n_head_kv, head_dim) || rows < 16 || rows > 4096 || cells < rows || cells > (1 << 20) || parts < 1 || parts > 64) {
    set_error("attention: 16..4096 rows, rows..2^20 cells, 8 query heads per KV head of 256 dims or 4 of 128, 1..64 parts");
    return EINVAL_;
  }
  const size_t M = rows, N = cells, Hq = n_head, Hkv = n_head_kv, hd = head_dim;
  Scratch sc;
  auto half_rows = [&](const float* src, size_t r, size_t w, __half** dst) -> int {
    float* f = nullptr;
    B200_TRY(sc.get(&f, r * w * sizeof(float))); B200_TRY(sc.get(dst, r * w * sizeof(__half)));
    B200_CUDA(cudaMemcpy(f, src, r * w * sizeof(float), cudaMemcpyHostToDevice));
    return quantize_rows_device(T_F16, f, (int64_t)r, (int64_t)w, (uint8_t*)*dst, 0);
  };
  AttnParams p{};
  B200_TRY(half_rows(q, M, Hq * hd, &p.q16)); B200_TRY(half_rows(k, N, Hkv * hd, &p.kcache)); B200_TRY(half_rows(v, N, Hkv * hd, &p.vcache));
  std::vector<float> proj(M * Hq * 2 * hd, 0.f);   // per head q | gate
  for (size_t i = 0; i < M * Hq; i++) memcpy(&proj[(2 * i + 1) * hd], gate + i * hd, hd * sizeof(float));
  std::vector<int> at(2 * M, 0);                   // slots, then positions
  for (size_t i = 0; i < M; i++) at[M + i] = (int)(N - M + i);
  float* d_proj = nullptr; int *d_at = nullptr, *err = nullptr;
  B200_TRY(sc.get(&d_proj, proj.size() * sizeof(float))); B200_TRY(sc.get(&d_at, at.size() * sizeof(int))); B200_TRY(sc.get(&err, sizeof(int)));
  B200_TRY(sc.get(&p.ctx16, M * Hq * hd * sizeof(__half)));
  const int64_t room = parts > 1 ? (int64_t)(M * Hq * (hd + 2)) * parts : 0;
  B200_TRY(sc.get(&p.partial, (size_t)room * sizeof(float)));
  B200_CUDA(cudaMemcpy(d_proj, proj.data(), proj.size() * sizeof(float), cudaMemcpyHostToDevice));
  B200_CUDA(cudaMemcpy(d_at, at.data(), at.size() * sizeof(int), cudaMemcpyHostToDevice));
  B200_CUDA(cudaMemset(err, 0, sizeof(int)));
  p.proj = d_proj; p.ldp = (int64_t)(Hq * 2 * hd); p.slot_stride = (int64_t)(N * Hkv * hd); p.row_slot = d_at; p.row_pos = d_at + M;
  p.M = rows; p.Hq = n_head; p.Hkv = n_head_kv; p.hd = head_dim; p.n_kv = cells; p.err = err;
  AttnTcMaps maps{};
  B200_TRY(make_attn_maps(p.q16, rows, n_head, p.kcache, p.vcache, cells, n_head_kv, head_dim, &maps));
  B200_TRY(launch_attn_tc(p, maps, cells - 1, room, false, 0));
  if (p.nsplit > 0) B200_TRY(launch_attn_merge(p, false, 0));
  std::vector<__half> h(M * Hq * hd);
  B200_TRY(finish_projection("attention", nullptr, err, 0, nullptr));
  B200_CUDA(cudaMemcpy(h.data(), p.ctx16, h.size() * sizeof(__half), cudaMemcpyDeviceToHost));
  for (size_t i = 0; i < h.size(); i++) out[i] = __half2float(h[i]);
  return OK;
}

int32_t b200_deltanet(int32_t heads_k, int32_t heads_v, int32_t n_embd, int32_t rows, const float* proj, const float* x, const float* alpha_w,
                      const float* beta_w, const float* conv_w, const float* ssm_a, const float* dt_bias, float* state, float* out) {
  B200_TRY(need_device());
  if (!proj || !x || !alpha_w || !beta_w || !conv_w || !ssm_a || !dt_bias || !state || !out) { set_error("deltanet: null argument"); return EINVAL_; }
  if (heads_k < 1 || heads_v < 1 || heads_v > 256 || heads_v % heads_k || n_embd < 256 || n_embd % 256 || rows < 2 || rows > 4096) { set_error("deltanet: 2..4096 rows, heads_v a multiple of heads_k, n_embd of 256"); return EINVAL_; }
  const size_t D = 128, Hk = heads_k, Hv = heads_v, M = rows, H = n_embd, cw = (2 * Hk + Hv) * D, ld = cw + Hv * D;
  Scratch sc;
  auto in = [&](const float* src, size_t n, float** dst) -> int {
    B200_TRY(sc.get(dst, n * sizeof(float)));
    B200_CUDA(cudaMemcpy(*dst, src, n * sizeof(float), cudaMemcpyHostToDevice));
    return (int)OK;
  };
  float *d_proj, *d_x, *d_a, *d_b, *d_conv, *d_ssm, *d_dt, *d_state, *d_norm;
  B200_TRY(in(proj, M * ld, &d_proj)); B200_TRY(in(x, M * H, &d_x)); B200_TRY(in(alpha_w, Hv * H, &d_a)); B200_TRY(in(beta_w, Hv * H, &d_b));
  B200_TRY(in(conv_w, cw * 4, &d_conv)); B200_TRY(in(ssm_a, Hv, &d_ssm)); B200_TRY(in(dt_bias, Hv, &d_dt)); B200_TRY(in(state, Hv * D * D, &d_state));
  const std::vector<float> ones(D, 1.f);
  B200_TRY(in(ones.data(), D, &d_norm));
  DnStepParams p{};
  __half* x16 = nullptr; SeqDesc* seqs = nullptr;
  B200_TRY(sc.get(&x16, M * H * sizeof(__half))); B200_TRY(sc.get(&p.y16, M * Hv * D * sizeof(__half))); B200_TRY(sc.get(&seqs, sizeof(SeqDesc)));
  p.ring_slot_stride = (int64_t)(Hv * 4 * DN_RING * DN_RING_W);
  B200_TRY(sc.get(&p.ring, p.ring_slot_stride * sizeof(float))); B200_TRY(sc.get(&p.pre, M * (Hk * 256 + Hv * 130) * sizeof(float)));
  B200_TRY(sc.get(&p.wy, M * Hv * 192 * sizeof(float))); B200_TRY(sc.get(&p.o_raw, M * Hv * D * sizeof(float))); B200_TRY(sc.get(&p.ab, M * 2 * Hv * sizeof(float)));
  const SeqDesc seq{0, 0, rows, 0};
  B200_CUDA(cudaMemcpy(seqs, &seq, sizeof(seq), cudaMemcpyHostToDevice));
  B200_TRY(quantize_rows_device(T_F16, d_x, rows, n_embd, (uint8_t*)x16, 0));
  p.proj = d_proj; p.ldp = (int64_t)ld; p.xn = x16; p.alpha_w = d_a; p.beta_w = d_b; p.conv_w = d_conv; p.ssm_a = d_ssm; p.dt_bias = d_dt;
  p.state = d_state; p.state_slot_stride = (int64_t)(Hv * D * D); p.seqs = seqs; p.n_seq = 1; p.norm_w = d_norm; p.pre_rows = rows;
  p.H = n_embd; p.Hk = heads_k; p.Hv = heads_v; p.D = 128; p.conv = 4; p.eps = 1e-6f;
  int launches = 0;
  B200_TRY(launch_dn_scan(p, rows, rows, &launches, false, 0));
  B200_CUDA(cudaMemcpy(out, p.o_raw, M * Hv * D * sizeof(float), cudaMemcpyDeviceToHost));
  B200_CUDA(cudaMemcpy(state, d_state, Hv * D * D * sizeof(float), cudaMemcpyDeviceToHost));
  return OK;
}

int32_t b200_quantize(uint32_t type, const float* host_src, int64_t rows, int64_t k, void* host_dst) {
  B200_TRY(need_device());
  const int64_t rb = gguf_row_bytes(type, k);
  if (!host_src || !host_dst || rb < 0 || rows <= 0) { set_error("quantize: bad argument"); return EINVAL_; }
  Scratch sc; float* f = nullptr; uint8_t* q = nullptr;
  B200_TRY(sc.get(&f, (size_t)rows * k * sizeof(float))); B200_TRY(sc.get(&q, (size_t)(rb * rows)));
  B200_CUDA(cudaMemcpy(f, host_src, (size_t)rows * k * sizeof(float), cudaMemcpyHostToDevice));
  B200_TRY(quantize_rows_device(type, f, rows, k, q, 0));
  B200_CUDA(cudaMemcpy(host_dst, q, (size_t)(rb * rows), cudaMemcpyDeviceToHost));
  return OK;
}

}  // extern "C"
