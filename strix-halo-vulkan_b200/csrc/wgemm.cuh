// Many-row K-quant projections as a tensor-core GEMM (tcgen05 / TMEM) with fp16-rounded weights:
//
//   Y[t][n] = sum_k fp16(W[n][k]) * X16[t][k]
//
// the reference's prefill projection and prefill expert kernels (shaders/llm_gemm.comp MODE 2, shaders/llm_moe_gemm.comp:1-110).
// See wgemm.cu for the pipeline and for how a weight is rounded.
#pragma once
#include "common.cuh"
#include "tgemm.cuh"

namespace b200 {

enum { WG_STORE = 0, WG_SWIGLU = 1 };

// One problem of a launch (a dense projection has one; the expert kernels one per expert, the shared expert last).
struct GemmProblem {
  int expert;          // weight rows start at expert * N; < 0: the shared expert's matrices
  int x_row0;          // first activation row (into the tensor map's row axis)
  int count;           // activation rows
  int y_row0;          // first output row
};

struct WGemmParams {
  const GemmProblem* problems;  // device array of n_problems; null: the single problem `one`
  int n_problems;
  GemmProblem one;
  int max_count;                // upper bound of the activation rows of all problems together
  int K, N;
  int ksplit;                   // parts the contraction is cut into (one problem, WG_STORE); part i writes plane i
  float* y; int64_t ldy, plane; // WG_STORE: f32 [.][ldy]
  __half* y16;                  // WG_SWIGLU: fp16 [.][ldy] of silu(gate) * up
  const int* y_rows;            // optional: row y_row0 + i is written to y_rows[y_row0 + i]
  int* err;
};

struct WMap { TMap m[4]; };     // a weight matrix: one map, or one per plane of the re-laid types
struct WGemmMaps { WMap w, w2, ws, ws2; TMap x; };   // WG_SWIGLU: w gate, w2 up; ws, ws2 the shared expert's

bool wgemm_type(uint32_t type);
// columns of a tile for M activation rows against N weight rows, and how many parts to cut K into
int wgemm_cols(int M, int N);
int wgemm_ksplit(int M, int N, int K);
int launch_wgemm(uint32_t type, int epi, int cols, const WGemmParams& p, const WGemmMaps& maps, bool pdl, cudaStream_t st);
// box_rows: 128, or 64 for the matrices of a gated pair
int make_wmap(uint32_t type, const uint8_t* w, int64_t rows, int64_t stride, int box_rows, WMap* out);

}  // namespace b200
