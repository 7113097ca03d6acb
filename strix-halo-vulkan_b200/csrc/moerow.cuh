// The MoE block of a pass of at most QG_FUSED_ROWS rows: every row is routed, computed and finished on its own, by the same
// kernels whatever the number of rows, so a pass of several rows gives each the single-row result bit for bit. See moerow.cu.
#pragma once
#include "qgemv.cuh"

namespace b200 {

// gate and up projections of the selected experts and the shared one, SwiGLU; selects the experts from the router's logits
struct MoeGateParams {
  RouterParams route;       // logits in; topk, topk_w and margin out
  int K, N, M;              // N: rows of one expert's gate (= up) matrix
  const __half* x;          // [M][K]
  __half* act;              // [M][used + 1][N]
  const uint8_t *down, *down_sh;   // the down projection's weights, brought to L2 on the way: [expert][down_bytes]
  int64_t down_bytes;       // of one expert
  const uint8_t* ahead[6];  // the next layer's dense weights, likewise
  int64_t ahead_bytes[6];
  int n_ahead;
  int* err;
  Timeline tl;
};
struct MoeGateMaps { TMap gate, up, gate_sh, up_sh; };   // boxes of 16 rows (make_w_tensor_map)

// down projections, routing weights, shared expert and residual: h[row] += sum_s w_s (W_s act_s) + gate * shared
struct MoeDownParams {
  int K, N, used;
  const int32_t* topk;      // [rows][used]
  const float* topk_w;      // [rows][used + 1]
  const __half* act;        // [rows][used + 1][K]
  float* h;                 // [rows][N]
  float* ss_out;            // [rows][SS_LD] sums of squares, part = tile of 16 rows
  int* err;
  Timeline tl;
};
struct MoeDownMaps { TMap w, ws; };

// whether both kernels take these weights (Q4_K and Q5_K, gate and up alike, the shared expert as the routed ones)
bool moe_rows_fit(uint32_t gate_type, uint32_t down_type, int H, int ffn, int n_expert, int used);
int launch_moe_gate(uint32_t type, const MoeGateParams& p, const MoeGateMaps& maps, bool pdl, cudaStream_t st);
int launch_moe_down(uint32_t type, const MoeDownParams& p, const MoeDownMaps& maps, int rows, bool pdl, cudaStream_t st);

}  // namespace b200
