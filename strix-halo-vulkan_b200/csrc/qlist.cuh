// Expert projections over a work list of few columns per expert (passes of 9 rows up to some hundreds), weights exact:
// the arithmetic of qgemv.cuh, with warps that stream their own weights. See qlist.cu.
#pragma once
#include "common.cuh"
#include "tgemm.cuh"

namespace b200 {

enum { QL_STORE = 0, QL_SWIGLU = 1 };

struct QListParams {
  const int4* entries; const int* n_entries; const int* cols;   // {expert (< 0: shared), first column, columns, 0}; column -> pair id
  int x_div;                 // activation row = pair id / x_div
  int K, N;
  const __half* x;           // [.][K]
  const __half* sx;          // [.][K / 256][TG_SX] sub-block sums
  float* y; int64_t ldy;     // QL_STORE: f32 rows by pair id
  __half* y16;               // QL_SWIGLU: fp16 rows by pair id, and their sub-block sums
  __half* sx_out;
  int* err;
};

// Tensor maps (make_w_tensor_map, boxes of 16 rows) of the routed weights [experts * N][K] and of the shared expert's
struct QListMaps { TMap w, w2, ws, ws2; };   // QL_SWIGLU: w gate, w2 up

bool qlist_type(uint32_t type);
bool qlist_fits(int K, int N, int max_entries);
// cols: columns an entry may have, 8 or 16
int launch_qlist(uint32_t type, int epi, int cols, const QListParams& p, const QListMaps& maps, bool pdl, cudaStream_t st);

}  // namespace b200
