// K-quant projections of some tens of activation rows on the 5th-generation tensor cores, with the weights exact:
// the product the column-tiled kernel (qgemv.cuh) forms, for the dense projections of passes of 9 rows and more.
//
//   y[c][n] = sum_b ( d[n][b] * sum_k (sc q)[n][k] x[c][k]  -  dmin[n][b] * sum_s m[n][s] X[c][s] )      b: super-blocks
//
// (sc q) and m are integers below 2048, exact in fp16; X are the sums of x over the sub-blocks of 32, as fp16 hi + lo; d and
// dmin are applied in f32 once per super-block. See tgemm.cu for the pipeline.
#pragma once
#include "common.cuh"

namespace b200 {

constexpr int TG_SX = 64;   // halves kept per row and super-block of the sub-block sums: 8 hi, 8 lo, padding to a 128-byte row

struct TMap { alignas(64) unsigned char b[128]; };   // a CUtensorMap

struct TGemmParams {
  int K, N, M;          // N weight rows, M activation rows
  int seg_end;          // weight rows from here on come from the second matrix (N when there is one)
  int ksplit;           // parts the contraction is cut into; part i writes plane i
  float* y; int64_t ldy, plane;
  int* err;
};

// Tensor maps of a launch: weights (w2: the second segment), activation rows, their sub-block sums
struct TGemmMaps { TMap w, w2, x, sx; };

bool tgemm_type(uint32_t type);
// columns of a tile for a pass of M rows: 16, 32 or 64
int tgemm_cols(int M);
int tgemm_ksplit(int K, int N, int M, int cols);
int launch_tgemm(uint32_t type, int cols, const TGemmParams& p, const TGemmMaps& maps, bool pdl, cudaStream_t st);
// weight rows of `stride` bytes for boxes of one super-block x box_rows
int make_w_tensor_map(uint32_t type, const uint8_t* w, int64_t rows, int64_t stride, int box_rows, TMap* out);
// fp16 rows of K elements for boxes of 64 elements x box_rows
int make_rows_map(const __half* x, int64_t rows, int K, int box_rows, TMap* out);
// sub-block sums of fp16 rows, for rows that no kernel of this library leaves them with
int launch_row_sums(const __half* x, int rows, int K, __half* sx, bool pdl, cudaStream_t st);

#ifdef __CUDACC__
// where the sum of sub-block s (of 32 elements) of a row goes, hi + lo
__device__ __forceinline__ void store_sub_sum(__half* sx_row, int s, float sum) {
  const __half hi = __float2half_rn(sum);
  __half* p = sx_row + (size_t)(s >> 3) * TG_SX + (s & 7);
  p[0] = hi;
  p[8] = __float2half_rn(sum - __half2float(hi));
}
#endif

}  // namespace b200
