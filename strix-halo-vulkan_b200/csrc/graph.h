// The token-loop graph: per-slot sequence state, pass scheduling, CUDA-graph replay.
// Host half of the reference's llm.Graph (llm/graph.go:184-289), re-designed for one
// device arena and one captured CUDA graph per decode step.
#pragma once
#include <map>
#include <vector>

#include "attn_tc.cuh"
#include "ep.cuh"
#include "kernels.cuh"
#include "model.h"

namespace b200 {

struct PassFlags {
  bool want_all_logits = false;   // logits for every row, else the last row only
  bool want_residual = false;     // copy every row's residual to the host
  bool spec = false;              // speculative: write per-row state planes, leave the state untouched
  bool greedy = false;            // argmax + advance on the device (no host traffic)
  bool draft = false;             // the pass runs the draft layer only
  bool want_hidden = true;        // copy the last row's residual to the host (when not every row's)
  const float* hs = nullptr;      // draft: the rows' previous residuals, host memory
};

struct Graph {
  Model* m = nullptr;
  b200_graph_opts o{};
  cudaStream_t st = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  int MR = 0;           // rows per pass
  int LR = 0;           // rows whose logits one pass can return
  int attn_rows = 0;    // rows a pass may send through the split-KV attention kernel (its partial results are per row)
  int n_dn = 0, n_attn = 0;
  std::vector<int> dn_index, attn_index;  // layer -> index among its kind (draft layer = last attention)
  // activations
  float *h = nullptr, *proj = nullptr, *attn_partial = nullptr, *down = nullptr, *logits = nullptr, *e_buf = nullptr, *hs_buf = nullptr;
  __half *xn16 = nullptr, *q16 = nullptr, *ctx16 = nullptr, *act16 = nullptr, *y16 = nullptr, *xcat16 = nullptr;
  float *dn_pre = nullptr, *dn_wy = nullptr, *dn_oraw = nullptr, *dn_ab = nullptr;   // many-token DeltaNet: scan inputs (q | k per key head, v and decay | beta per value head), raw outputs [rows][Hv*D]
  int pass_max_n = 1;                            // longest sequence of the pass being enqueued
  __half* xperm16 = nullptr;   // [rows * (used + 1)][H]: activation rows in expert-sorted order, the shared expert's last
  // tensor maps of every weight matrix and of the activation rows (tgemm, qlist, wgemm), sub-block sums of the rows
  struct LayerMaps {
    TMap gate, up, down, gate_sh, up_sh, down_sh;                 // boxes of 16 rows (qlist)
    WMap wgate, wup, wdown, wgate_sh, wup_sh, wdown_sh, qkv, z, out, q, k, v, o, router;   // boxes of 64 (gate, up) and 128 rows
  };
  std::vector<LayerMaps> wmaps;
  std::map<const uint8_t*, TMap> row_maps;   // by weight: the maps of the projections of at most eight rows
  WMap head_map{};
  TMap tx_xperm{}, tx_act{};   // expert-sorted rows and their activations, boxes of 64 rows
  TMap tx_xn[3], ts_xn[3], tx_y16[3], ts_y16[3], tx_ctx[3], ts_ctx[3];   // activation rows and their sums, boxes of 16 / 32 / 64 rows
  __half *sx_xn = nullptr, *sx_act = nullptr, *sx_y = nullptr, *sx_ctx = nullptr, *sx_ep = nullptr;
  int4* gprob = nullptr;       // [n_expert + 1] GEMM problem per expert, the shared expert's last
  float* ss_part = nullptr;   // [rows][SS_LD] partial sums of squares of the residual rows
  float *r_logits = nullptr, *topk_w = nullptr, *margin = nullptr;
  int32_t *topk = nullptr, *ids_dev = nullptr, *next_ids = nullptr, *history = nullptr;
  int *r_ticket = nullptr, *pair_counts = nullptr, *pair_pos = nullptr, *err_flag = nullptr, *n_entries = nullptr, *cols = nullptr, *row_slot = nullptr, *row_pos = nullptr, *logit_rows = nullptr, *hist_len = nullptr;
  int4* entries = nullptr;
  int64_t* distinct_dev = nullptr;     // experts streamed by the work lists built so far (device counter)
  int n_rows_moe = 0;                  // layers (without the draft's) whose experts a fused pass selects inside the expert kernel
  int64_t single_row_layers = 0;       // (row, layer) pairs of fused passes in those layers
  SeqDesc* seqs = nullptr;
  float* rope = nullptr;
  int proj_ld = 0, max_entries = 0, nsplit = 0, split_cells = 0;
  // sequence state
  std::vector<float*> dn_state, dn_ring, dn_mid;   // per DeltaNet layer
  std::vector<AttnTcMaps> attn_maps;               // per attention layer: query rows and its caches
  int64_t attn_partial_floats = 0;
  int pass_last_pos = 0;                           // passes of one sequence: position of the last row
  std::vector<__half*> kcache, vcache;             // per attention layer (+ draft)
  int64_t state_slot_stride = 0, ring_slot_stride = 0, kv_slot_stride = 0, mid_seq_stride = 0;
  std::vector<int> past, draft_past;
  int cur = 0;
  // speculation
  bool speculating = false, spec_first = false;
  int spec_pos0 = -1, spec_n = 0;
  int dcur = 0;        // slot whose draft cache the draft calls read and write (MTPHead.UseSlot)
  // running totals over the passes this graph ran (the reference's GraphStats: llm/graph.go:527-589)
  b200_graph_stats stats{};
  // host staging (pinned) and its image on the device: PassOut | ids | slots | positions | logit rows | sequences, one copy per pass
  uint8_t *stage = nullptr, *stage_dev = nullptr;
  // results land in the graph's own pinned buffers (grown to what calls ask for: a pass may return hundreds of
  // megabytes of logits) or, for one call, where b200_graph_set_outputs points
  float *logits_host = nullptr, *resid_host = nullptr, *hidden_host = nullptr;
  int64_t logits_host_cap = 0, resid_host_cap = 0;
  float *out_logits = nullptr, *out_resid = nullptr;
  int64_t out_logits_cap = 0, out_resid_cap = 0;
  bool out_logits_mapped = false, out_resid_mapped = false;   // blocks the device can write
  int32_t* ids_host = nullptr;
  // trace
  float *tr_mid = nullptr, *tr_out = nullptr, *tr_w = nullptr, *tr_margin = nullptr;
  int32_t* tr_topk = nullptr;
  int last_rows = 0;
  // replay
  std::map<int, cudaGraphExec_t> decode_graphs, greedy_graphs;
  long long* timeline = nullptr;  // [launch][8] phase timestamps when B200_TIMELINE is set
  int timeline_cap = 0;
  int launches = 0, last_launches = 0, draft_vocab = 0, draft_vocab_default = 0, resid_off = 0;
  float last_ms = 0.f;
  // expert parallelism (ep.cuh): exchange arena, peers' arenas as mapped here, switch
  EpParams ep{};
  uint8_t* ep_arena = nullptr;
  size_t ep_arena_bytes = 0;
  int* ep_epoch = nullptr;
  std::vector<void*> ep_mapped;
  bool ep_ready = false, ep_on = false;
  // checkpoints: DeltaNet state + rings of a slot at a token boundary
  struct Ckpt { int slot, past; std::vector<float*> state, ring; };
  std::map<int, Ckpt> ckpts;
  int next_ckpt = 1;
  std::vector<void*> allocs;

  ~Graph();
  int init(Model* model, const b200_graph_opts& opts);
  int enqueue_pass(int M, int n_seq, int n_logit_rows, const PassFlags& f);
  int entry_cols(int M, bool stream) const;
  int max_entries_for(int M, bool stream) const;
  bool dense_tg(uint32_t type, int M, int N) const;
  bool direct_out(const PassFlags& f, int M, int n_logit_rows) const;
  bool rows_moe(const LayerW& L) const;
  bool experts_stream(const LayerW& L, int M) const;
  int make_weight_maps();
  uint32_t fp16_weight_mask(int M, int n_logit_rows) const;
  int run_rows(const int32_t* ids, const int* slots, const int* pos, int M, const std::vector<SeqDesc>& sq, const std::vector<int>& lrows, const PassFlags& f);
  int extend(const int32_t* ids, int n, const PassFlags& f, const float** logits_out, const float** hidden_out);
  int decode_rows(const int32_t* slots, const int32_t* ids, int n, const float** logits_out);
  int generate_greedy(const int32_t* slots, const int32_t* first, int n, int steps, int32_t* out);
  int draft_rows(const float* hs, const int32_t* ids, int n, int vocab_k, const float** resid, const float** logits_out);
  int reset_slot(int slot);
  int keep(int k);
  int checkpoint(int* handle);
  int restore(int handle);
  int64_t trace(int what, void* dst, int64_t nbytes);
  int residual_row(int r, float* dst);
  int pass_experts(int* out);
  int inject_wait_timeout();
  int finish_pass();
  void place_stage(int M);
  int upload_stage(int M);
  int outputs_fit(int64_t logit_floats, int64_t resid_floats) const;
  int result_buffers(int64_t logit_floats, int64_t resid_floats, float** lg, float** rs);
  int ep_prepare(int rank, int world);
  int ep_export(int rank, int world, void* handle64);
  int ep_attach(const void* handles64);
  int ep_attach_local(Graph* const* peers, int world);
  int synth_context(int slot, int cells, uint64_t seed);
  template <class T> int dalloc(T** p, size_t n, bool zero = true);
};

}  // namespace b200
