// The token loop's non-projection kernels: embedding gather, router + routing, gated
// DeltaNet step, attention pre-pass and split-KV decode attention, MoE combine, argmax,
// and the Q6_K / Q8_0 row re-layout.
#include "kernels.cuh"

#include <cooperative_groups.h>

#include <cmath>

namespace cg = cooperative_groups;

namespace b200 {

// =========================================================================================
// Row layout
// =========================================================================================
bool block_geometry(uint32_t t, int* e, int* b) {
  switch (t) {
    case T_F32: *e = 1; *b = 4; return true;
    case T_F16: case T_BF16: *e = 1; *b = 2; return true;
    case T_Q4_1: *e = 32; *b = 20; return true;
    case T_Q5_0: *e = 32; *b = 22; return true;
    case T_Q5_1: *e = 32; *b = 24; return true;
    case T_Q8_0: *e = 32; *b = 34; return true;
    case T_IQ4_NL: *e = 32; *b = 18; return true;
    case T_Q4_K: *e = 256; *b = 144; return true;
    case T_Q5_K: *e = 256; *b = 176; return true;
    case T_Q6_K: *e = 256; *b = 210; return true;
  }
  return false;
}
int64_t gguf_row_bytes(uint32_t t, int64_t n) {
  int e, b;
  if (!block_geometry(t, &e, &b) || n % e) return -1;
  return n / e * b;
}
int64_t device_row_stride(uint32_t t, int64_t k) {
  int64_t rb = gguf_row_bytes(t, k);
  if (rb < 0) return -1;
  if (t == T_Q6_K || t == T_Q8_0) return (rb + 15) / 16 * 16;
  return rb;
}

// One thread per block. Q6_K: ql | qh | scales | d planes; Q8_0: qs | d planes.
__global__ void repack_kernel(uint32_t type, int64_t nb, int64_t rows, int64_t stride, const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, int inverse) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nb * rows) return;
  int64_t r = i / nb, b = i - r * nb;
  uint8_t* drow = dst + (inverse ? 0 : r * stride);
  const uint8_t* srow = src + (inverse ? r * stride : 0);
  if (type == T_Q6_K) {
    const int64_t g = (r * nb + b) * 210;
    uint8_t* gq = inverse ? dst + g : nullptr;
    const uint8_t* gs = inverse ? nullptr : src + g;
    uint8_t* pql = (inverse ? const_cast<uint8_t*>(srow) : drow) + b * 128;
    uint8_t* pqh = (inverse ? const_cast<uint8_t*>(srow) : drow) + nb * 128 + b * 64;
    uint8_t* psc = (inverse ? const_cast<uint8_t*>(srow) : drow) + nb * 192 + b * 16;
    uint8_t* pd = (inverse ? const_cast<uint8_t*>(srow) : drow) + nb * 208 + b * 2;
    if (!inverse) {
      for (int j = 0; j < 128; j++) pql[j] = gs[j];
      for (int j = 0; j < 64; j++) pqh[j] = gs[128 + j];
      for (int j = 0; j < 16; j++) psc[j] = gs[192 + j];
      pd[0] = gs[208]; pd[1] = gs[209];
    } else {
      for (int j = 0; j < 128; j++) gq[j] = pql[j];
      for (int j = 0; j < 64; j++) gq[128 + j] = pqh[j];
      for (int j = 0; j < 16; j++) gq[192 + j] = psc[j];
      gq[208] = pd[0]; gq[209] = pd[1];
    }
  } else {  // Q8_0
    const int64_t g = (r * nb + b) * 34;
    uint8_t* base = inverse ? const_cast<uint8_t*>(srow) : drow;
    uint8_t* pq = base + b * 32;
    uint8_t* pd = base + nb * 32 + b * 2;
    if (!inverse) {
      pd[0] = src[g]; pd[1] = src[g + 1];
      for (int j = 0; j < 32; j++) pq[j] = src[g + 2 + j];
    } else {
      dst[g] = pd[0]; dst[g + 1] = pd[1];
      for (int j = 0; j < 32; j++) dst[g + 2 + j] = pq[j];
    }
  }
}

int repack_rows(uint32_t type, int64_t k, int64_t rows, const uint8_t* gguf_dev, uint8_t* dst_dev, cudaStream_t st) {
  int64_t rb = gguf_row_bytes(type, k);
  if (rb < 0) { set_error("repack: bad type or row length"); return EINVAL_; }
  if (type != T_Q6_K && type != T_Q8_0) {
    B200_CUDA(cudaMemcpyAsync(dst_dev, gguf_dev, (size_t)(rb * rows), cudaMemcpyDeviceToDevice, st));
    return OK;
  }
  int64_t nb = k / (type == T_Q6_K ? 256 : 32), n = nb * rows;
  repack_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(type, nb, rows, device_row_stride(type, k), gguf_dev, dst_dev, 0);
  B200_CUDA(cudaGetLastError());
  return OK;
}
int unpack_rows(uint32_t type, int64_t k, int64_t rows, const uint8_t* dev, uint8_t* gguf_dev, cudaStream_t st) {
  int64_t rb = gguf_row_bytes(type, k);
  if (rb < 0) { set_error("unpack: bad type or row length"); return EINVAL_; }
  if (type != T_Q6_K && type != T_Q8_0) {
    B200_CUDA(cudaMemcpyAsync(gguf_dev, dev, (size_t)(rb * rows), cudaMemcpyDeviceToDevice, st));
    return OK;
  }
  int64_t nb = k / (type == T_Q6_K ? 256 : 32), n = nb * rows;
  repack_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(type, nb, rows, device_row_stride(type, k), dev, gguf_dev, 1);
  B200_CUDA(cudaGetLastError());
  return OK;
}

// =========================================================================================
// Exact element dequantisation (reference: gguf/dequant.go:128-356), device layout
// =========================================================================================
__device__ __forceinline__ float ld_f16(const uint8_t* p) { return __half2float(*reinterpret_cast<const __half*>(p)); }

__device__ __forceinline__ void k4_scale_min(int j, const uint8_t* q, int* sc, int* m) {
  if (j < 4) { *sc = q[j] & 63; *m = q[j + 4] & 63; }
  else { *sc = (q[j + 4] & 0xF) | ((q[j - 4] >> 6) << 4); *m = (q[j + 4] >> 4) | ((q[j] >> 6) << 4); }
}

// value of element k of a device row. __fmul_rn / __fsub_rn keep the reference's
// unfused `d*sc*q - dmin*m` so the result is bit-identical to the CPU dequantiser.
__device__ float dequant_elem(uint32_t type, const uint8_t* row, int64_t K, int64_t k) {
  switch (type) {
    case T_F32: return reinterpret_cast<const float*>(row)[k];
    case T_F16: return ld_f16(row + 2 * k);
    case T_BF16: return __uint_as_float((uint32_t)reinterpret_cast<const unsigned short*>(row)[k] << 16);
    case T_Q8_0: {
      int64_t nb = K / 32, b = k / 32;
      float d = ld_f16(row + nb * 32 + b * 2);
      return __fmul_rn((float)(int8_t)row[k], d);
    }
    case T_Q4_K: {
      const uint8_t* blk = row + (k / 256) * 144;
      int e = (int)(k % 256), grp = e / 64, in = e % 64, hi = in / 32, l = in % 32;
      float d = ld_f16(blk), dmin = ld_f16(blk + 2);
      int sc, m; k4_scale_min(2 * grp + hi, blk + 4, &sc, &m);
      int q = hi ? (blk[16 + 32 * grp + l] >> 4) : (blk[16 + 32 * grp + l] & 0xF);
      return __fsub_rn(__fmul_rn(__fmul_rn(d, (float)sc), (float)q), __fmul_rn(dmin, (float)m));
    }
    case T_Q5_K: {
      const uint8_t* blk = row + (k / 256) * 176;
      int e = (int)(k % 256), grp = e / 64, in = e % 64, hi = in / 32, l = in % 32;
      float d = ld_f16(blk), dmin = ld_f16(blk + 2);
      int sc, m; k4_scale_min(2 * grp + hi, blk + 4, &sc, &m);
      int q = hi ? (blk[48 + 32 * grp + l] >> 4) : (blk[48 + 32 * grp + l] & 0xF);
      if (blk[16 + l] & (1 << (2 * grp + hi))) q += 16;
      return __fsub_rn(__fmul_rn(__fmul_rn(d, (float)sc), (float)q), __fmul_rn(dmin, (float)m));
    }
    case T_Q6_K: {
      int64_t nb = K / 256, b = k / 256;
      int e = (int)(k % 256), hf = e / 128, in = e % 128, quarter = in / 32, l = in % 32;
      const uint8_t* ql = row + b * 128 + 64 * hf + 32 * (quarter & 1) + l;
      const uint8_t* qh = row + nb * 128 + b * 64 + 32 * hf + l;
      int8_t sc = (int8_t)row[nb * 192 + b * 16 + 8 * hf + l / 16 + 2 * quarter];
      float d = ld_f16(row + nb * 208 + b * 2);
      int nib = quarter >= 2 ? (*ql >> 4) : (*ql & 0xF);
      int q = (nib | (((*qh >> (2 * quarter)) & 3) << 4)) - 32;
      return __fmul_rn(__fmul_rn(d, (float)sc), (float)q);
    }
  }
  return 0.f;
}

__global__ void dequant_rows_kernel(DTensor t, int64_t row0, int64_t rows, float* out) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows * t.k) return;
  int64_t r = i / t.k, k = i - r * t.k;
  out[i] = dequant_elem(t.type, t.data + (row0 + r) * t.stride, t.k, k);
}
int dequant_rows(const DTensor& t, int64_t row0, int64_t rows, float* out, cudaStream_t st) {
  int64_t n = rows * t.k;
  dequant_rows_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(t, row0, rows, out);
  B200_CUDA(cudaGetLastError());
  return OK;
}

// Embedding gather on the device (the reference dequantises the row on the host and
// uploads it: llm/model.go:125-144), fused with the first layer's input norm.
__global__ void __launch_bounds__(QG_THREADS) embed_norm_kernel(EmbedParams p) {
  __shared__ float scratch[2 * QG_WARPS];
  const int n = blockIdx.x;
  const int64_t id = p.ids[n];
  const uint8_t* row = p.embd.data + id * p.embd.stride;
  float* h = p.h + (size_t)n * p.H;
  float sq = 0.f;
  for (int k = threadIdx.x; k < p.H; k += blockDim.x) { const float v = dequant_elem(p.embd.type, row, p.H, k); h[k] = v; sq += v * v; }
  if (p.ss_out != nullptr) {  // the first projection normalises from this
    sq = warp_sum(sq);
    if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = sq;
    __syncthreads();
    if (threadIdx.x == 0) {
      float t = 0.f;
      for (int w = 0; w < QG_WARPS; w++) t += scratch[w];
      p.ss_out[(size_t)n * SS_LD] = t;
    }
  }
  if (p.gamma != nullptr) {
    __syncthreads();
    row_rmsnorm_f16(h, p.gamma, p.eps, p.H, p.xn + (size_t)n * p.H, scratch, p.sx != nullptr ? p.sx + (size_t)n * (p.H / 256 * TG_SX) : nullptr);
  }
}
int launch_embed(const EmbedParams& p, cudaStream_t st) {
  embed_norm_kernel<<<p.M, QG_THREADS, 0, st>>>(p);
  B200_CUDA(cudaGetLastError());
  return OK;
}

// =========================================================================================
// PDL launch helper
// =========================================================================================
template <class... KArgs, class... Args>
static int launch_k(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, bool pdl, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = pdl ? 1 : 0;
  B200_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
  return OK;
}

// =========================================================================================
// Router: ffn_norm + router GEMV (exact f32 dequant) + softmax + top-k + work list
// (reference: llm/moe.go:219-282; shaders/llm_moe_router.comp, llm_moe_route_decode.comp)
// =========================================================================================
constexpr int RT_ROWS = 4;  // router rows per CTA: two warps to a row, half of its contraction each, so that 513 rows reach every SM

// Expert work list of a pass from its routing, by one CTA of 256 threads: pair id = n*(used+1) + slot,
// slot == used is the shared expert; entries of at most 8 columns per expert for the column-tiled kernels,
// one GEMM problem per expert for the tensor-core kernels, cols = pairs in expert-sorted order.
__device__ void build_work_list(const RouterParams& p, int* counts, int* offs, int* eoff) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, M = p.M, nE = p.nE, used = p.used;
  const int EC = p.ecols > 0 ? p.ecols : 8;  // columns per entry
  // work list: pair id = n*(used+1) + slot; slot == used is the shared expert
  if (M == 1) {
    if (tid < used) { p.entries[tid] = make_int4(p.topk[tid], tid, 1, 0); p.cols[tid] = tid; }
    if (tid == used) { p.entries[used] = make_int4(-1, used, 1, 0); p.cols[used] = used; *p.n_entries = used + 1; }
    if (tid == 0 && p.distinct != nullptr) *p.distinct += used;
    tl_mark(p.tl, 6, true);
    return;
  }
  const int e_lo = p.e_hi > 0 ? p.e_lo : 0, e_hi = p.e_hi > 0 ? p.e_hi : nE;
  const int sh_lo = p.sh_hi > 0 ? p.sh_lo : 0, sh_hi = p.sh_hi > 0 ? p.sh_hi : M;
  const bool counted = p.pair_pos != nullptr;   // the routing has counted the pairs and placed each among its expert's
  for (int i = tid; i <= nE; i += 256) {
    counts[i] = counted && i < nE ? __ldcg(p.pair_counts + i) : 0;
    if (counted && i < nE) p.pair_counts[i] = 0;
  }
  __syncthreads();
  if (!counted) {
    for (int i = tid; i < M * used; i += 256) {
      const int e = __ldcg(p.topk + i);
      if (e >= e_lo && e < e_hi) atomicAdd(&counts[e], 1);
    }
    __syncthreads();
  }
  if (p.distinct != nullptr) {   // experts this pass streams (what a step's byte count needs)
    int mine = 0;
    for (int e = tid; e < nE; e += 256) mine += counts[e] > 0;
    mine = __reduce_add_sync(0xffffffffu, mine);
    if (lane == 0 && mine > 0) atomicAdd(reinterpret_cast<unsigned long long*>(p.distinct), (unsigned long long)mine);
  }
  if (warp == 0) {  // exclusive scans of the pair counts and of the entry counts (EC columns per entry)
    const int per = (nE + 31) / 32;
    int c = 0, en = 0;
    for (int i = 0; i < per; i++) { const int e = lane * per + i; if (e < nE) { c += counts[e]; en += (counts[e] + EC - 1) / EC; } }
    int cs = c, es = en;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int a = __shfl_up_sync(0xffffffffu, cs, o), b = __shfl_up_sync(0xffffffffu, es, o);
      if (lane >= o) { cs += a; es += b; }
    }
    int co = cs - c, eo = es - en;
    for (int i = 0; i < per; i++) {
      const int e = lane * per + i;
      if (e < nE) { offs[e] = co; eoff[e] = eo; co += counts[e]; eo += (counts[e] + EC - 1) / EC; }
    }
    const int tot_c = __shfl_sync(0xffffffffu, cs, 31), tot_e = __shfl_sync(0xffffffffu, es, 31);
    if (lane == 0) { offs[nE] = tot_c; eoff[nE] = tot_e; }
  }
  __syncthreads();
  for (int e = tid; e < nE; e += 256) {
    for (int c = 0, i = 0; c < counts[e]; c += EC, i++)
      if (eoff[e] + i < p.max_entries) p.entries[eoff[e] + i] = make_int4(e, offs[e] + c, min(EC, counts[e] - c), 0);
  }
  // one GEMM problem per expert for the tensor-core expert kernels: rows [offs, offs + count) of the expert-sorted order
  if (p.gprob != nullptr) for (int e = tid; e <= nE; e += 256) p.gprob[e] = e < nE ? make_int4(e, offs[e], counts[e], offs[e]) : make_int4(-1, offs[nE], M, offs[nE]);
  const int nshr = sh_hi - sh_lo, nsh = (nshr + EC - 1) / EC;
  for (int i = tid; i < nsh; i += 256)
    if (eoff[nE] + i < p.max_entries) p.entries[eoff[nE] + i] = make_int4(-1, offs[nE] + EC * i, min(EC, nshr - EC * i), 0);
  if (tid == 0) { *p.n_entries = min(eoff[nE] + nsh, p.max_entries); if (p.n_pairs != nullptr) *p.n_pairs = offs[nE] + nshr; }
  if (counted && p.gprob != nullptr) return;     // the gather kernel writes cols as it places the rows
  if (counted) {
#pragma unroll 4
    for (int i = tid; i < M * used; i += 256) {
      const int n = i / used;
      p.cols[offs[__ldcg(p.topk + i)] + __ldcg(p.pair_pos + i)] = n * (used + 1) + i - n * used;
    }
  } else {
    __syncthreads();
    for (int i = tid; i <= nE; i += 256) counts[i] = 0;
    __syncthreads();
    for (int i = tid; i < M * used; i += 256) {
      const int e = __ldcg(p.topk + i), n = i / used, k = i - n * used;
      if (e < e_lo || e >= e_hi) continue;
      const int pos = atomicAdd(&counts[e], 1);
      p.cols[offs[e] + pos] = n * (used + 1) + k;
    }
  }
  for (int n = tid; n < nshr; n += 256) p.cols[offs[nE] + n] = (sh_lo + n) * (used + 1) + used;
}

// Work list of an expert-parallel pass: the gathered routing of every rank's rows, restricted to the experts
// this rank owns. One CTA.
__global__ void __launch_bounds__(256) ep_worklist_kernel(RouterParams p) {
  __shared__ int counts[1025], offs[1025], eoff[1025];
  pdl_wait();
  pdl_launch();
  build_work_list(p, counts, offs, eoff);
}
int launch_ep_worklist(const RouterParams& p, bool pdl, cudaStream_t st) {
  if (p.nE > 1024 || p.used > 32 || p.M < 2) { set_error("ep_worklist: shape outside kernel limits"); return ECAPACITY; }
  return launch_k(ep_worklist_kernel, dim3(1), dim3(256), 0, pdl, st, p);
}

// Router logits by per-row dot products, and the shared expert's gate; weights exact. Selection is the next kernel's.
__global__ void __launch_bounds__(256) router_kernel(RouterParams p) {
  __shared__ float half_sum[8][8];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, H = p.H, M = p.M;
  const int row = blockIdx.x * RT_ROWS + (warp >> 1), half = warp & 1;  // of the nE + 1 outputs; the last is the shared-expert gate
  const int k_lo = half * (H / 2), k_hi = half ? H : H / 2;
  tl_mark(p.tl, 0);
  const bool q8 = p.router.type == T_Q8_0 && H % 512 == 0 && H <= 4096;
  // the row's weights do not depend on the producer kernel: fetch them first
  uint4 wq[4]; float wd[4];
  if (row < p.nE && q8) {
    const uint8_t* wr = p.router.data + (size_t)row * p.router.stride;
    const int nb = H / 32;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int k0 = k_lo + lane * 16 + i * 512;
      if (k0 < k_hi) { wq[i] = ldg_stream(wr + k0); wd[i] = ld_f16(wr + nb * 32 + (k0 / 32) * 2); }
    }
  }
  const bool staged = p.h != nullptr;
  float4 hpre[2], gpre[2];
  if (staged) {  // the norm weights do not depend on the producer kernel either
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const int k = tid * 4 + i * 1024;
      if (k < H) gpre[i] = *reinterpret_cast<const float4*>(p.gamma + k);
    }
  }
  pdl_wait();
  pdl_launch();
  tl_mark(p.tl, 1);
  extern __shared__ __align__(16) __half rxs[];  // [M][H] when the rows are normalised here
  __shared__ float rscale[8];
  if (staged) {  // ffn_norm fused into the router (M <= 8): every CTA normalises the rows, CTA 0 keeps a copy
    // the first row's values do not depend on the scale: fetch them before reducing the partials
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const int k = tid * 4 + i * 1024;
      if (k < H) hpre[i] = __ldcg(reinterpret_cast<const float4*>(p.h + k));
    }
    if (warp < M) {
      const float sc = scale_from_parts(p.ss_in, p.ss_n, warp, H, p.eps);
      if (lane == 0) rscale[warp] = sc;
    }
    __syncthreads();
    auto put = [&](int n, int k, const float4& hv, const float4& g, float scale) {
      __half2 a = __floats2half2_rn(hv.x * scale * g.x, hv.y * scale * g.y), b = __floats2half2_rn(hv.z * scale * g.z, hv.w * scale * g.w);
      const uint2 o = make_uint2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b));
      *reinterpret_cast<uint2*>(rxs + (size_t)n * H + k) = o;
      if (blockIdx.x == 0 && p.xn_out != nullptr) *reinterpret_cast<uint2*>(p.xn_out + (size_t)n * H + k) = o;
    };
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const int k = tid * 4 + i * 1024;
      if (k < H) put(0, k, hpre[i], gpre[i], rscale[0]);
    }
    for (int n = 0; n < M; n++) {
      const float scale = rscale[n];
      for (int k = tid * 4 + (n == 0 ? 2048 : 0); k < H; k += 1024)
        put(n, k, __ldcg(reinterpret_cast<const float4*>(p.h + (size_t)n * H + k)), *reinterpret_cast<const float4*>(p.gamma + k), scale);
    }
    __syncthreads();
  }
  if (row <= p.nE) {
    // rows of the pass are spread over blockIdx.y in groups of 8 so a many-slot pass fills the machine
    const int n_lo = blockIdx.y * 8, n_hi = min(M, n_lo + 8);
    for (int n = n_lo; n < n_hi; n++) {
      const __half* x = staged ? rxs + (size_t)n * H : p.xn + (size_t)n * H;
      float acc = 0.f;
      if (row == p.nE) {
        for (int k = k_lo + lane * 8; k < k_hi; k += 256) {
          uint4 xv = *reinterpret_cast<const uint4*>(x + k);
          const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
          float4 g0 = *reinterpret_cast<const float4*>(p.sh_gate + k), g1 = *reinterpret_cast<const float4*>(p.sh_gate + k + 4);
          acc = fmaf(g0.x, h2f_lo(xw[0]), acc); acc = fmaf(g0.y, h2f_hi(xw[0]), acc); acc = fmaf(g0.z, h2f_lo(xw[1]), acc); acc = fmaf(g0.w, h2f_hi(xw[1]), acc);
          acc = fmaf(g1.x, h2f_lo(xw[2]), acc); acc = fmaf(g1.y, h2f_hi(xw[2]), acc); acc = fmaf(g1.z, h2f_lo(xw[3]), acc); acc = fmaf(g1.w, h2f_hi(xw[3]), acc);
        }
      } else if (q8) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int k0 = k_lo + lane * 16 + i * 512;
          if (k0 < k_hi) {
            uint4 xa = *reinterpret_cast<const uint4*>(x + k0), xb = *reinterpret_cast<const uint4*>(x + k0 + 8);
            const uint32_t xw[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
            const uint32_t w[4] = {wq[i].x, wq[i].y, wq[i].z, wq[i].w};
#pragma unroll
            for (int j = 0; j < 16; j++) {
              const float wv = __fmul_rn((float)(int8_t)((w[j >> 2] >> (8 * (j & 3))) & 0xFF), wd[i]);  // gguf/dequant.go:128-137
              const float xv = (j & 1) ? h2f_hi(xw[j >> 1]) : h2f_lo(xw[j >> 1]);
              acc = fmaf(wv, xv, acc);
            }
          }
        }
      } else {
        const uint8_t* wr = p.router.data + (size_t)row * p.router.stride;
        for (int k = k_lo + lane; k < k_hi; k += 32) acc = fmaf(dequant_elem(p.router.type, wr, H, k), __half2float(x[k]), acc);
      }
      acc = warp_sum(acc);
      if (lane == 0) half_sum[n - n_lo][warp] = acc;
    }
  }
  __syncthreads();
  if (tid < 8 * RT_ROWS) {
    const int n = blockIdx.y * 8 + tid / RT_ROWS, w = tid % RT_ROWS, e = blockIdx.x * RT_ROWS + w;
    if (n < M && e <= p.nE) {
      const float v = half_sum[tid / RT_ROWS][2 * w] + half_sum[tid / RT_ROWS][2 * w + 1];
      if (e == p.nE) p.topk_w[(size_t)n * (p.used + 1) + p.used] = sigmoid_acc(v);
      else p.logits[(size_t)n * p.nE + e] = v;
    }
  }
  tl_mark(p.tl, 4);
}

__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

// Router logits of a pass of some tens to hundreds of rows (batched decode): too few rows for the 128-row
// tensor-memory tiles to fill the device (512 experts are four tiles), too many for the per-row dot products
// above. A CTA takes 16 experts x 64 rows; each warp an eighth of the hidden dimension, with the experts on the
// M axis of mma.m16n8k16 and eight column tiles reusing every dequantised fragment. Q8_0 weights become
// fp16(d * q), as in the tensor-core GEMM the longer passes use. A lane reads 16 contiguous weight bytes and the
// matching 32 bytes of an activation row; the k-slots of the four mma steps are assigned to those bytes in A
// and B alike. Warp partials are summed in warp order. grid (nE / 16, ceil(M / 64)), block 256.
__global__ void __launch_bounds__(256) router_mma_kernel(RouterParams p) {
  __shared__ float part[8][16][65];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int H = p.H, M = p.M, e0 = blockIdx.x * 16, n0 = blockIdx.y * 64;
  const int ks = H / 8, nc = ks / 64, k_lo = warp * ks + 16 * t;
  const uint8_t* wa = p.router.data + (size_t)(e0 + g) * p.router.stride;
  const uint8_t* wb = p.router.data + (size_t)(e0 + g + 8) * p.router.stride;
  // the weights do not depend on the producer kernel: fetch them first
  uint4 qa[8], qb[8]; float da[8], db[8];
#pragma unroll
  for (int c = 0; c < 8; c++) {
    if (c < nc) {
      const int k0 = k_lo + 64 * c;
      qa[c] = ldg_stream(wa + k0); qb[c] = ldg_stream(wb + k0);
      da[c] = ld_f16(wa + H + (k0 / 32) * 2); db[c] = ld_f16(wb + H + (k0 / 32) * 2);
    }
  }
  pdl_wait();
  pdl_launch();
  float acc[8][4];
#pragma unroll
  for (int nt = 0; nt < 8; nt++) { acc[nt][0] = 0.f; acc[nt][1] = 0.f; acc[nt][2] = 0.f; acc[nt][3] = 0.f; }
  auto deq2 = [](uint32_t w, int sh, float d) {  // bytes sh, sh + 1 of w as fp16(d * q) pairs
    const float lo = __fmul_rn((float)(int8_t)((w >> (8 * sh)) & 0xFF), d), hi = __fmul_rn((float)(int8_t)((w >> (8 * sh + 8)) & 0xFF), d);
    return pack_half2(lo, hi);
  };
#pragma unroll
  for (int c = 0; c < 8; c++) {
    if (c < nc) {
      const int k0 = k_lo + 64 * c;
      const uint32_t wav[4] = {qa[c].x, qa[c].y, qa[c].z, qa[c].w}, wbv[4] = {qb[c].x, qb[c].y, qb[c].z, qb[c].w};
      uint32_t a[4][4];
#pragma unroll
      for (int s = 0; s < 4; s++) {
        a[s][0] = deq2(wav[s], 0, da[c]); a[s][1] = deq2(wbv[s], 0, db[c]);
        a[s][2] = deq2(wav[s], 2, da[c]); a[s][3] = deq2(wbv[s], 2, db[c]);
      }
#pragma unroll
      for (int nt = 0; nt < 8; nt++) {
        const int row = min(n0 + nt * 8 + g, M - 1);  // rows past the end are not written
        const __half* x = p.xn + (size_t)row * H + k0;
        const uint4 x0 = *reinterpret_cast<const uint4*>(x), x1 = *reinterpret_cast<const uint4*>(x + 8);
        mma16816(acc[nt], a[0], x0.x, x0.y);
        mma16816(acc[nt], a[1], x0.z, x0.w);
        mma16816(acc[nt], a[2], x1.x, x1.y);
        mma16816(acc[nt], a[3], x1.z, x1.w);
      }
    }
  }
#pragma unroll
  for (int nt = 0; nt < 8; nt++) {
    part[warp][g][nt * 8 + 2 * t] = acc[nt][0]; part[warp][g][nt * 8 + 2 * t + 1] = acc[nt][1];
    part[warp][g + 8][nt * 8 + 2 * t] = acc[nt][2]; part[warp][g + 8][nt * 8 + 2 * t + 1] = acc[nt][3];
  }
  __syncthreads();
  for (int i = tid; i < 16 * 64; i += 256) {
    const int e = i & 15, n = i >> 4;
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < 8; w++) v += part[w][e][n];
    if (n0 + n < M) p.logits[(size_t)(n0 + n) * p.nE + e0 + e] = v;
  }
}
bool router_mma_fits(const RouterParams& p) {
  return p.router.type == T_Q8_0 && p.H % 512 == 0 && p.H <= 4096 && p.nE % 16 == 0 && p.xn != nullptr;
}
int launch_router_mma(const RouterParams& p, bool pdl, cudaStream_t st) {
  if (!router_mma_fits(p)) { set_error("router_mma: shape outside kernel limits"); return EINVAL_; }
  return launch_k(router_mma_kernel, dim3(p.nE / 16, (p.M + 63) / 64), dim3(256), 0, pdl, st, p);
}

// Selection for every row of a pass from its logits, a CTA per row (route_row_cta), with the shared expert's gate (f32 weights
// against the fp16 row) where the router has not left it. Every pair also takes its place among its expert's pairs, so that the last
// CTA has only the experts to go over for the work list. (A warp per row, and one CTA that counted and placed all pairs, took 22 us
// for 64 rows and 57 for 2048, most of it that CTA's walk over the pairs.) grid M, block 256.
template <int VPT>
__global__ void __launch_bounds__(256) route_rows_kernel(RouterParams p) {
  __shared__ int is_last;
  __shared__ RouteSmem rs;
  __shared__ float gate[8];
  __shared__ int counts[1025], offs[1025], eoff[1025];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, H = p.H, n = blockIdx.x, used = p.used;
  pdl_wait();
  pdl_launch();
  float l[VPT];
#pragma unroll
  for (int i = 0; i < VPT; i++) l[i] = tid + 256 * i < p.nE ? __ldcg(p.logits + (size_t)n * p.nE + tid + 256 * i) : -INFINITY;
  if (!p.gate_done) {
    const __half* x = p.xn + (size_t)n * H;
    float acc = 0.f;
    for (int k = tid * 8; k < H; k += 2048) {
      uint4 xv = *reinterpret_cast<const uint4*>(x + k);
      const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
      float4 g0 = *reinterpret_cast<const float4*>(p.sh_gate + k), g1 = *reinterpret_cast<const float4*>(p.sh_gate + k + 4);
      acc = fmaf(g0.x, h2f_lo(xw[0]), acc); acc = fmaf(g0.y, h2f_hi(xw[0]), acc); acc = fmaf(g0.z, h2f_lo(xw[1]), acc); acc = fmaf(g0.w, h2f_hi(xw[1]), acc);
      acc = fmaf(g1.x, h2f_lo(xw[2]), acc); acc = fmaf(g1.y, h2f_hi(xw[2]), acc); acc = fmaf(g1.z, h2f_lo(xw[3]), acc); acc = fmaf(g1.w, h2f_hi(xw[3]), acc);
    }
    acc = warp_sum(acc);
    if (lane == 0) gate[warp] = acc;   // read after the selection's barriers
  }
  route_row_cta<VPT>(p, n, l, true, -1, rs);
  if (!p.gate_done && tid == 0) p.topk_w[(size_t)n * (used + 1) + used] = sigmoid_acc(((gate[0] + gate[1]) + (gate[2] + gate[3])) + ((gate[4] + gate[5]) + (gate[6] + gate[7])));
  if (p.entries == nullptr) return;   // routing only (expert-parallel passes build their list from the gathered routing)
  if (warp == 0 && p.M > 1) {
    __syncwarp();                     // the row's experts were written by other lanes
    if (lane < used) p.pair_pos[(size_t)n * used + lane] = atomicAdd(p.pair_counts + __ldcg(p.topk + (size_t)n * used + lane), 1);
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) is_last = (atomicAdd(p.ticket, 1) == (int)gridDim.x - 1);
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  if (tid == 0) *p.ticket = 0;
  build_work_list(p, counts, offs, eoff);
}
// The same with a warp per row, for passes whose rows fill the device anyway: a CTA per row spends more instructions, most of them
// repeated in its eight warps. grid ceil(M / 8), block 256.
__global__ void __launch_bounds__(256) route_many_kernel(RouterParams p) {
  __shared__ int is_last;
  __shared__ float2 cand[8][32];
  __shared__ int counts[1025], offs[1025], eoff[1025];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, H = p.H, n = blockIdx.x * 8 + warp, used = p.used;
  pdl_wait();
  pdl_launch();
  if (n < p.M) {
    if (!p.gate_done) {
      const __half* x = p.xn + (size_t)n * H;
      float acc = 0.f;
      for (int k = lane * 8; k < H; k += 256) {
        uint4 xv = *reinterpret_cast<const uint4*>(x + k);
        const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
        float4 g0 = *reinterpret_cast<const float4*>(p.sh_gate + k), g1 = *reinterpret_cast<const float4*>(p.sh_gate + k + 4);
        acc = fmaf(g0.x, h2f_lo(xw[0]), acc); acc = fmaf(g0.y, h2f_hi(xw[0]), acc); acc = fmaf(g0.z, h2f_lo(xw[1]), acc); acc = fmaf(g0.w, h2f_hi(xw[1]), acc);
        acc = fmaf(g1.x, h2f_lo(xw[2]), acc); acc = fmaf(g1.y, h2f_hi(xw[2]), acc); acc = fmaf(g1.z, h2f_lo(xw[3]), acc); acc = fmaf(g1.w, h2f_hi(xw[3]), acc);
      }
      acc = warp_sum(acc);
      if (lane == 0) p.topk_w[(size_t)n * (used + 1) + used] = sigmoid_acc(acc);
    }
    if (p.nE <= 512) route_token<16>(p, n, lane, true, cand[warp]);
    else route_token<32>(p, n, lane, true, cand[warp]);
    __syncwarp();
    if (p.entries != nullptr && lane < used) p.pair_pos[(size_t)n * used + lane] = atomicAdd(p.pair_counts + __ldcg(p.topk + (size_t)n * used + lane), 1);
  }
  if (p.entries == nullptr) return;
  __threadfence();
  __syncthreads();
  if (tid == 0) is_last = (atomicAdd(p.ticket, 1) == (int)gridDim.x - 1);
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  if (tid == 0) *p.ticket = 0;
  build_work_list(p, counts, offs, eoff);
}
// Rows from which a warp per row fills the device. Whole prompts of the 512-expert shape, 12 layers, a CTA or a warp per row: 200 rows 4889 or
// 4936 us, 300 rows 6814 or 6743, 512 rows 8080 or 8000, 2048 rows 13825 or 13532.
constexpr int ROUTE_MANY_FROM = 512;
int launch_route_rows(const RouterParams& p, bool pdl, cudaStream_t st) {
  if (p.nE > 1024 || p.used > 32 || p.H % 8 || p.xn == nullptr || p.pair_pos == nullptr) { set_error("route_rows: shape outside kernel limits"); return ECAPACITY; }
  if (p.M >= ROUTE_MANY_FROM) return launch_k(route_many_kernel, dim3((p.M + 7) / 8), dim3(256), 0, pdl, st, p);
  return p.nE <= 512 ? launch_k(route_rows_kernel<2>, dim3(p.M), dim3(256), 0, pdl, st, p) : launch_k(route_rows_kernel<4>, dim3(p.M), dim3(256), 0, pdl, st, p);
}

int launch_router(const RouterParams& p, bool pdl, cudaStream_t st) {
  if (p.nE > 1024 || p.used > 32 || p.H % 16) { set_error("router: shape outside kernel limits"); return ECAPACITY; }
  int grid = (p.nE + 1 + RT_ROWS - 1) / RT_ROWS;
  size_t smem = 0;
  if (p.h != nullptr) {
    if (p.M > 8) { set_error("router: the fused norm handles at most 8 rows"); return EINVAL_; }
    smem = (size_t)p.M * p.H * sizeof(__half);
    B200_ONCE_PER_DEVICE(cudaFuncSetAttribute(router_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    if (smem > 200 * 1024) { set_error("router: rows too long for shared memory"); return ECAPACITY; }
  }
  return launch_k(router_kernel, dim3(grid, p.h != nullptr ? 1 : (p.M + 7) / 8), dim3(256), smem, pdl, st, p);
}

// Expert-sorted copy of the activation rows for the tensor-core expert kernels (the reference's
// shaders/llm_moe_perm.comp): sorted row i holds the row of token cols[i] / (used + 1).
__global__ void __launch_bounds__(256) moe_gather_kernel(const __half* xn, RouterParams p, __half* xperm) {
  pdl_wait();
  pdl_launch();
  const int slots1 = p.used + 1, n = blockIdx.x / slots1, s = blockIdx.x - n * slots1;
  const int i = s < p.used ? p.gprob[p.topk[n * p.used + s]].y + p.pair_pos[n * p.used + s] : p.gprob[p.nE].y + n;
  if (threadIdx.x == 0) p.cols[i] = blockIdx.x;
  const uint4* src = reinterpret_cast<const uint4*>(xn + (size_t)n * p.H);
  uint4* dst = reinterpret_cast<uint4*>(xperm + (size_t)i * p.H);
  for (int k = threadIdx.x; k < p.H / 8; k += 256) dst[k] = __ldcg(src + k);
}
int launch_moe_gather(const __half* xn, const RouterParams& p, __half* xperm, bool pdl, cudaStream_t st) {
  return launch_k(moe_gather_kernel, dim3(p.M * (p.used + 1)), dim3(256), 0, pdl, st, xn, p, xperm);
}

// Row kernels, one CTA per row, for passes of more than QG_FUSED_ROWS rows: RMSNorm, or MoE combine + RMSNorm.
__global__ void __launch_bounds__(QG_THREADS) row_tail_kernel(TailParams tp) {
  __shared__ float scratch[2 * QG_WARPS];
  pdl_wait();
  pdl_launch();
  const int n = blockIdx.x, slots1 = tp.used + 1;
  float* hrow = tp.h + (size_t)n * tp.H;
  if (tp.mode == 2) {
    row_moe_combine(hrow, tp.down + (size_t)n * slots1 * tp.H, tp.topk_w + (size_t)n * slots1, tp.used, tp.H);
    __syncthreads();
  }
  if (tp.n_parts > 0) {   // (a thread normalises the elements it adds here)
    for (int k = threadIdx.x * 4; k < tp.H; k += QG_THREADS * 4) {
      float4 v = *reinterpret_cast<float4*>(hrow + k), a = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int i = 0; i < tp.n_parts; i++) {
        const float4 d = __ldcg(reinterpret_cast<const float4*>(tp.parts + i * tp.part_plane + (size_t)n * tp.H + k));
        a.x += d.x; a.y += d.y; a.z += d.z; a.w += d.w;
      }
      v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
      *reinterpret_cast<float4*>(hrow + k) = v;
    }
  }
  row_rmsnorm_f16(hrow, tp.gamma, tp.eps, tp.H, tp.xn + (size_t)n * tp.H, scratch, tp.sx != nullptr ? tp.sx + (size_t)n * (tp.H / 256 * TG_SX) : nullptr,
                  tp.ss_out != nullptr ? tp.ss_out + (size_t)n * SS_LD : nullptr);
}
int launch_row_tail(const TailParams& tp, bool pdl, cudaStream_t st) {
  return launch_k(row_tail_kernel, dim3(tp.M), dim3(QG_THREADS), 0, pdl, st, tp);
}

// Draft seed input: xcat[n] = fp16(rms(embd[n], enorm)) | fp16(rms(h_prev[n], hnorm))  (llm/mtp.go:352-384)
__global__ void __launch_bounds__(QG_THREADS) concat_norm_kernel(const float* e, const float* hs, const float* enorm, const float* hnorm, float eps, int H, __half* xcat) {
  __shared__ float scratch[2 * QG_WARPS];
  pdl_wait();
  pdl_launch();
  const int n = blockIdx.x;
  row_rmsnorm_f16(e + (size_t)n * H, enorm, eps, H, xcat + (size_t)n * 2 * H, scratch);
  __syncthreads();
  row_rmsnorm_f16(hs + (size_t)n * H, hnorm, eps, H, xcat + (size_t)n * 2 * H + H, scratch);
}
int launch_concat_norm(const float* e, const float* hs, const float* enorm, const float* hnorm, float eps, int H, int M, __half* xcat, bool pdl, cudaStream_t st) {
  return launch_k(concat_norm_kernel, dim3(M), dim3(QG_THREADS), 0, pdl, st, e, hs, enorm, hnorm, eps, H, xcat);
}

// =========================================================================================
// Gated DeltaNet step: alpha/beta projections, causal conv + SiLU, L2 norm, gates, the
// delta-rule state update and read-out (reference: llm/deltanet.go:263-321, 365-455;
// shaders/llm_dn_conv.comp, llm_dn_scan.comp, llm_seq_hist.comp).
// grid (Hv * 4, n_seq): a CTA owns 32 of the 128 state rows of one value head of one
// sequence, keeps them in registers and walks the sequence's tokens in order. The four CTAs
// of a head form a thread-block cluster: the gated RMSNorm over the head's 128 outputs
// (reference: llm/deltanet.go:326-341, shaders/llm_dn_norm.comp) needs their four partial
// sums of squares, exchanged through distributed shared memory.
// =========================================================================================
__device__ __forceinline__ float softplus_ref(float x) {  // llm/deltanet.go:450-455
  if (x > 20.f) return x;
  return logf(1.0f + expf(x));
}
__device__ __forceinline__ float silu_acc(float x) { return x * sigmoid_acc(x); }
// Sums of eight values over the warp's lanes, every lane getting all eight: halves of the values change hands at each of the first
// three steps, so 17 shuffles instead of 40, and every sum is the one the plain butterfly from 16 down to 1 forms.
__device__ __forceinline__ void warp_sum8(float (&v)[8]) {
  const int lane = threadIdx.x & 31;
  float a[4], b[2];
  const bool h4 = lane & 16, h2 = lane & 8, h1 = lane & 4;
#pragma unroll
  for (int i = 0; i < 4; i++) a[i] = (h4 ? v[i + 4] : v[i]) + __shfl_xor_sync(0xffffffffu, h4 ? v[i] : v[i + 4], 16);
#pragma unroll
  for (int i = 0; i < 2; i++) b[i] = (h2 ? a[i + 2] : a[i]) + __shfl_xor_sync(0xffffffffu, h2 ? a[i] : a[i + 2], 8);
  float c = (h1 ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, h1 ? b[0] : b[1], 4);
  c += __shfl_xor_sync(0xffffffffu, c, 2);
  c += __shfl_xor_sync(0xffffffffu, c, 1);
#pragma unroll
  for (int r = 0; r < 8; r++) v[r] = __shfl_sync(0xffffffffu, c, 4 * r);   // row r sits in the lanes whose bits 4, 3, 2 spell it
}

// (Passes of 16 sequences and more use dn_head_kernel below instead.)
// OCC: CTAs per SM it is compiled for. One or two sequences leave an SM two CTAs at most, and everything that is fetched before the
// wait stays in registers; from three on, five to an SM keep a pass in one wave (18 us against 10 for five sequences).
template <int OCC>
__global__ void __cluster_dims__(4, 1, 1) __launch_bounds__(128, OCC) dn_step_kernel(DnStepParams p) {
  cg::cluster_group cluster = cg::this_cluster();
  const int D = 128, RB = 4;
  const int h = blockIdx.x / RB, rb = blockIdx.x % RB, hk = h % p.Hk;
  const SeqDesc sq = p.seqs[blockIdx.y];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int qk = p.Hk * D, H = p.H;
  __shared__ float qs[128], ks[128], vs[32], red[16], wss[4], cta_ss[2][4];  // cta_ss[token parity][row block]
  const int ch_q = hk * D + tid, ch_k = qk + hk * D + tid, ch_v = 2 * qk + h * D + rb * 32 + (tid & 31);
  const float4 cwq = *reinterpret_cast<const float4*>(p.conv_w + (size_t)ch_q * 4);
  const float4 cwk = *reinterpret_cast<const float4*>(p.conv_w + (size_t)ch_k * 4);
  const float4 cwv = *reinterpret_cast<const float4*>(p.conv_w + (size_t)ch_v * 4);
  const float a_h = p.ssm_a[h], dtb = p.dt_bias[h];
  // everything that does not depend on the producer kernel is fetched before waiting for it:
  // the first token's alpha / beta weight slices, the conv history and the state rows
  float4 pwa[4], pwb[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int k = tid * 4 + 512 * i;
    pwa[i] = k < p.H ? *reinterpret_cast<const float4*>(p.alpha_w + (size_t)h * p.H + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    pwb[i] = k < p.H ? *reinterpret_cast<const float4*>(p.beta_w + (size_t)h * p.H + k) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  // conv history: the three inputs before pos0, zeros before the sequence start
  // Every CTA keeps a private ring of its own 288 conv inputs (q 128 | k 128 | v 32), indexed
  // by position, so no CTA ever reads what another one writes.
  float* ring = p.ring + (size_t)sq.slot * p.ring_slot_stride + (size_t)blockIdx.x * (DN_RING * DN_RING_W);
  float hq[3], hkk[3], hv[3];
#pragma unroll
  for (int j = 0; j < 3; j++) {
    const int pos = sq.pos0 - 3 + j;
    const float* r = ring + (size_t)(pos & (DN_RING - 1)) * DN_RING_W;
    hq[j] = pos >= 0 ? r[tid] : 0.f;
    hkk[j] = pos >= 0 ? r[128 + tid] : 0.f;
    hv[j] = pos >= 0 ? r[256 + (tid & 31)] : 0.f;
  }
  // state rows of this warp: j = rb*32 + warp*8 + r, four floats per lane
  float* S = p.state + (size_t)sq.slot * p.state_slot_stride + (size_t)h * D * D;
  const int j0 = rb * 32 + warp * 8;
  float4 s[8];
#pragma unroll
  for (int r = 0; r < 8; r++) s[r] = *reinterpret_cast<const float4*>(S + (size_t)(j0 + r) * D + lane * 4);
  const float oscale = 1.0f / sqrtf((float)D);
  const float nw = lane < 8 ? p.norm_w[j0 + lane] : 0.f;  // gated-norm weight of the row this lane writes
  tl_mark(p.tl, 0);
  pdl_wait();
  pdl_launch();
  tl_mark(p.tl, 1);

  for (int i = 0; i < sq.n; i++) {
    const int row = sq.row0 + i, pos = sq.pos0 + i;
    const float* pr = p.proj + (size_t)row * p.ldp;
    // alpha / beta: F32 weights against the fp16-rounded block input
    const __half* xn = p.xn + (size_t)row * H;
    float pa = 0.f, pb = 0.f;
    auto ab_dot = [&](int k, const float4& wa, const float4& wb) {
      const __half2 x01 = *reinterpret_cast<const __half2*>(xn + k), x23 = *reinterpret_cast<const __half2*>(xn + k + 2);
      const float2 f01 = __half22float2(x01), f23 = __half22float2(x23);
      pa += wa.x * f01.x + wa.y * f01.y + wa.z * f23.x + wa.w * f23.y;
      pb += wb.x * f01.x + wb.y * f01.y + wb.z * f23.x + wb.w * f23.y;
    };
#pragma unroll
    for (int ki = 0; ki < 4; ki++) {
      const int k = tid * 4 + 512 * ki;
      if (k < H) {
        if (i == 0) ab_dot(k, pwa[ki], pwb[ki]);
        else ab_dot(k, *reinterpret_cast<const float4*>(p.alpha_w + (size_t)h * H + k), *reinterpret_cast<const float4*>(p.beta_w + (size_t)h * H + k));
      }
    }
    for (int k = tid * 4 + 2048; k < H; k += 512)
      ab_dot(k, *reinterpret_cast<const float4*>(p.alpha_w + (size_t)h * H + k), *reinterpret_cast<const float4*>(p.beta_w + (size_t)h * H + k));
    // conv + SiLU for q, k (whole head) and this CTA's 32 v channels
    const float cq = pr[ch_q], ck = pr[ch_k], cv = pr[ch_v];
    const float zz = lane < 8 ? pr[2 * qk + p.Hv * D + h * D + j0 + lane] : 0.f;  // the gate, asked for with the other inputs
    const float q = silu_acc(hq[0] * cwq.x + hq[1] * cwq.y + hq[2] * cwq.z + cq * cwq.w);
    const float k = silu_acc(hkk[0] * cwk.x + hkk[1] * cwk.y + hkk[2] * cwk.z + ck * cwk.w);
    const float v = silu_acc(hv[0] * cwv.x + hv[1] * cwv.y + hv[2] * cwv.z + cv * cwv.w);
    hq[0] = hq[1]; hq[1] = hq[2]; hq[2] = cq;
    hkk[0] = hkk[1]; hkk[1] = hkk[2]; hkk[2] = ck;
    hv[0] = hv[1]; hv[1] = hv[2]; hv[2] = cv;
    // the ring keeps every token's conv input by position (rollback = moving `past` back)
    {
      float* rw = ring + (size_t)(pos & (DN_RING - 1)) * DN_RING_W;
      rw[tid] = cq; rw[128 + tid] = ck;
      if (tid < 32) rw[256 + tid] = cv;
    }
    float sq2 = warp_sum(q * q), sk2 = warp_sum(k * k);
    pa = warp_sum(pa); pb = warp_sum(pb);
    __syncthreads();
    if (lane == 0) { red[warp] = sq2; red[4 + warp] = sk2; red[8 + warp] = pa; red[12 + warp] = pb; }
    if (tid < 32) vs[tid] = v;
    __syncthreads();
    const float qn = 1.0f / sqrtf(red[0] + red[1] + red[2] + red[3] + p.eps);
    const float kn = 1.0f / sqrtf(red[4] + red[5] + red[6] + red[7] + p.eps);
    const float alpha = red[8] + red[9] + red[10] + red[11], betar = red[12] + red[13] + red[14] + red[15];
    qs[tid] = q * qn;
    ks[tid] = k * kn;
    __syncthreads();
    const float g = expf(softplus_ref(alpha + dtb) * a_h);
    const float beta = sigmoid_acc(betar);
    const float4 k4 = *reinterpret_cast<const float4*>(ks + lane * 4);
    const float4 q4 = *reinterpret_cast<const float4*>(qs + lane * 4);
    float kv[8], oo[8];
#pragma unroll
    for (int r = 0; r < 8; r++) {
      s[r].x *= g; s[r].y *= g; s[r].z *= g; s[r].w *= g;
      kv[r] = s[r].x * k4.x + s[r].y * k4.y + s[r].z * k4.z + s[r].w * k4.w;
    }
    warp_sum8(kv);
#pragma unroll
    for (int r = 0; r < 8; r++) {
      const float dj = (vs[warp * 8 + r] - kv[r]) * beta;
      s[r].x += dj * k4.x; s[r].y += dj * k4.y; s[r].z += dj * k4.z; s[r].w += dj * k4.w;
      oo[r] = s[r].x * q4.x + s[r].y * q4.y + s[r].z * q4.z + s[r].w * q4.w;
    }
    warp_sum8(oo);
    // gated norm: sum of squares over the head's 128 outputs = four CTA partials, added in rank order
    float ov = oo[0] * oscale, ss = 0.f;
#pragma unroll
    for (int r = 0; r < 8; r++) {
      const float orr = oo[r] * oscale;
      ss += orr * orr;
      ov = lane == r ? orr : ov;
    }
    if (lane == 0) wss[warp] = ss;
    __syncthreads();
    // each CTA pushes its partial into the four CTAs' shared memory (thread r writes to rank r), one cluster
    // barrier, then everyone adds the four local copies in rank order: no CTA reads a peer's memory, so none
    // has to outlive a peer's reads
    if (tid < 4) *cluster.map_shared_rank(&cta_ss[i & 1][rb], tid) = wss[0] + wss[1] + wss[2] + wss[3];
    cluster.sync();
    float tot = 0.f;
#pragma unroll
    for (int r = 0; r < 4; r++) tot += cta_ss[i & 1][r];
    if (lane < 8) {
      const int j = j0 + lane;
      const float nsc = 1.0f / sqrtf(tot / (float)D + p.eps);
      p.y16[(size_t)row * (p.Hv * D) + h * D + j] = __float2half_rn(ov * nsc * nw * sigmoid_acc(zz));
    }
    if (p.mid != nullptr) {  // state after token i, for keep-prefix speculation
      float* Sm = p.mid + (size_t)blockIdx.y * p.mid_seq_stride + (size_t)i * p.mid_stride + (size_t)h * D * D;
#pragma unroll
      for (int r = 0; r < 8; r++) *reinterpret_cast<float4*>(Sm + (size_t)(j0 + r) * D + lane * 4) = s[r];
    }
    __syncthreads();
  }
  if (p.mid == nullptr) {
#pragma unroll
    for (int r = 0; r < 8; r++) *reinterpret_cast<float4*>(S + (size_t)(j0 + r) * D + lane * 4) = s[r];
  }
  tl_mark(p.tl, 4);
}

// -----------------------------------------------------------------------------------------
// Many sequences of one or a few tokens (batched decode): one CTA of sixteen warps per (value head,
// sequence) instead of a cluster of four. The alpha / beta projections and the q / k convolutions are
// computed once per head rather than once per row block, the gated norm's sum of squares is a
// shared-memory reduction rather than a cluster barrier, and the state rows, the conv rings and the
// grouping of every partial sum are those of dn_step_kernel (warp W here is warp W % 4 of row block W / 4).
// -----------------------------------------------------------------------------------------
__global__ void __launch_bounds__(512, 2) dn_head_kernel(DnStepParams p) {
  const int D = 128, RB = 4;
  const int h = blockIdx.x, hk = h % p.Hk;
  const SeqDesc sq = p.seqs[blockIdx.y];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int qk = p.Hk * D, H = p.H;
  __shared__ float qs[128], ks[128], vs[128], red[40], wss[16];
  // conv roles: threads 0..127 the q channels, 128..255 k, 256..383 the head's v channels; the rest idle there
  const int role = tid >> 7, c = tid & 127;
  const int ch = role == 0 ? hk * D + c : role == 1 ? qk + hk * D + c : 2 * qk + h * D + c;
  // ring of row block rb: [pos][q 128 | k 128 | v 32]; q and k are kept in all four, read from the first
  float* ring0 = p.ring + (size_t)sq.slot * p.ring_slot_stride + (size_t)(h * RB) * (DN_RING * DN_RING_W);
  const int ring_off = role == 0 ? c : role == 1 ? 128 + c : (c >> 5) * (DN_RING * DN_RING_W) + 256 + (c & 31);
  float4 cw = make_float4(0.f, 0.f, 0.f, 0.f);
  float hist[3] = {0.f, 0.f, 0.f};
  if (role < 3) {
    cw = *reinterpret_cast<const float4*>(p.conv_w + (size_t)ch * 4);
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const int pos = sq.pos0 - 3 + j;
      hist[j] = pos >= 0 ? ring0[(size_t)(pos & (DN_RING - 1)) * DN_RING_W + ring_off] : 0.f;
    }
  }
  const float a_h = p.ssm_a[h], dtb = p.dt_bias[h];
  // state rows of this warp: j = warp*8 + r, four floats per lane
  float* S = p.state + (size_t)sq.slot * p.state_slot_stride + (size_t)h * D * D;
  const int j0 = warp * 8;
  float4 s[8];
#pragma unroll
  for (int r = 0; r < 8; r++) s[r] = *reinterpret_cast<const float4*>(S + (size_t)(j0 + r) * D + lane * 4);
  const float oscale = 1.0f / sqrtf((float)D);
  tl_mark(p.tl, 0);
  pdl_wait();
  pdl_launch();
  tl_mark(p.tl, 1);

  for (int i = 0; i < sq.n; i++) {
    const int row = sq.row0 + i, pos = sq.pos0 + i;
    const float* pr = p.proj + (size_t)row * p.ldp;
    const __half* xn = p.xn + (size_t)row * H;
    float pa = 0.f, pb = 0.f;
    for (int k = tid * 4; k < H; k += 2048) {
      const float4 wa = *reinterpret_cast<const float4*>(p.alpha_w + (size_t)h * H + k), wb = *reinterpret_cast<const float4*>(p.beta_w + (size_t)h * H + k);
      const __half2 x01 = *reinterpret_cast<const __half2*>(xn + k), x23 = *reinterpret_cast<const __half2*>(xn + k + 2);
      const float2 f01 = __half22float2(x01), f23 = __half22float2(x23);
      pa += wa.x * f01.x + wa.y * f01.y + wa.z * f23.x + wa.w * f23.y;
      pb += wb.x * f01.x + wb.y * f01.y + wb.z * f23.x + wb.w * f23.y;
    }
    float cv = 0.f, act = 0.f;
    if (role < 3) {
      cv = pr[ch];
      act = silu_acc(hist[0] * cw.x + hist[1] * cw.y + hist[2] * cw.z + cv * cw.w);
      hist[0] = hist[1]; hist[1] = hist[2]; hist[2] = cv;
      // the rings keep every token's conv input by position (rollback = moving `past` back)
      float* rw = ring0 + (size_t)(pos & (DN_RING - 1)) * DN_RING_W + ring_off;
      if (role == 2) rw[0] = cv;
      else {
#pragma unroll
        for (int rb = 0; rb < RB; rb++) rw[(size_t)rb * (DN_RING * DN_RING_W)] = cv;
      }
    }
    const float a2 = warp_sum(act * act);  // warps 0..3: q, 4..7: k
    pa = warp_sum(pa); pb = warp_sum(pb);
    __syncthreads();
    if (lane == 0) { red[warp] = pa; red[16 + warp] = pb; if (warp < 8) red[32 + warp] = a2; }
    if (role == 2) vs[c] = act;
    __syncthreads();
    const float qn = 1.0f / sqrtf(red[32] + red[33] + red[34] + red[35] + p.eps);
    const float kn = 1.0f / sqrtf(red[36] + red[37] + red[38] + red[39] + p.eps);
    float alpha = 0.f, betar = 0.f;
#pragma unroll
    for (int w = 0; w < 16; w++) { alpha += red[w]; betar += red[16 + w]; }
    if (role == 0) qs[c] = act * qn;
    if (role == 1) ks[c] = act * kn;
    __syncthreads();
    const float g = expf(softplus_ref(alpha + dtb) * a_h);
    const float beta = sigmoid_acc(betar);
    const float4 k4 = *reinterpret_cast<const float4*>(ks + lane * 4);
    const float4 q4 = *reinterpret_cast<const float4*>(qs + lane * 4);
    float kv[8], oo[8];
#pragma unroll
    for (int r = 0; r < 8; r++) {
      s[r].x *= g; s[r].y *= g; s[r].z *= g; s[r].w *= g;
      kv[r] = s[r].x * k4.x + s[r].y * k4.y + s[r].z * k4.z + s[r].w * k4.w;
    }
    warp_sum8(kv);
#pragma unroll
    for (int r = 0; r < 8; r++) {
      const float dj = (vs[j0 + r] - kv[r]) * beta;
      s[r].x += dj * k4.x; s[r].y += dj * k4.y; s[r].z += dj * k4.z; s[r].w += dj * k4.w;
      oo[r] = s[r].x * q4.x + s[r].y * q4.y + s[r].z * q4.z + s[r].w * q4.w;
    }
    warp_sum8(oo);
    // gated norm: sum of squares over the head's 128 outputs, warp partials grouped by four as the row blocks were
    float ov = oo[0] * oscale, ss = 0.f;
#pragma unroll
    for (int r = 0; r < 8; r++) {
      const float orr = oo[r] * oscale;
      ss += orr * orr;
      ov = lane == r ? orr : ov;
    }
    if (lane == 0) wss[warp] = ss;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int rb = 0; rb < RB; rb++) tot += wss[4 * rb] + wss[4 * rb + 1] + wss[4 * rb + 2] + wss[4 * rb + 3];
    if (lane < 8) {
      const int j = j0 + lane;
      const float nsc = 1.0f / sqrtf(tot / (float)D + p.eps);
      const float zz = pr[2 * qk + p.Hv * D + h * D + j];
      p.y16[(size_t)row * (p.Hv * D) + h * D + j] = __float2half_rn(ov * nsc * p.norm_w[j] * sigmoid_acc(zz));
    }
    if (p.mid != nullptr) {  // state after token i, for keep-prefix speculation
      float* Sm = p.mid + (size_t)blockIdx.y * p.mid_seq_stride + (size_t)i * p.mid_stride + (size_t)h * D * D;
#pragma unroll
      for (int r = 0; r < 8; r++) *reinterpret_cast<float4*>(Sm + (size_t)(j0 + r) * D + lane * 4) = s[r];
    }
    __syncthreads();
  }
  if (p.mid == nullptr) {
#pragma unroll
    for (int r = 0; r < 8; r++) *reinterpret_cast<float4*>(S + (size_t)(j0 + r) * D + lane * 4) = s[r];
  }
  tl_mark(p.tl, 4);
}

// -----------------------------------------------------------------------------------------
// The same layer for sequences of many tokens (prefill), as three kernels: everything that does not
// depend on the recurrent state (alpha / beta, conv + SiLU, L2 norms, gates) is computed for all tokens
// in parallel and packed per (head, row block) and token; the scan then walks the tokens with no
// block-wide synchronisation at all; the gated norm runs per token afterwards.
// -----------------------------------------------------------------------------------------
// State-independent inputs of the many-token recurrence, written once per pass by dn_pre_kernel and read by every
// CTA that needs them (the four row blocks of a head share its v, decay and beta; the value heads of a key head
// share its q and k): [Hk][rows][256] normalised q | k, then [Hv][rows][128] v, then [Hv][rows][2] decay | beta.
__device__ __forceinline__ float* dn_pre_qk(const DnStepParams& p, int hk, int64_t row) { return p.pre + ((size_t)hk * p.pre_rows + row) * 256; }
__device__ __forceinline__ float* dn_pre_v(const DnStepParams& p, int h, int64_t row) { return p.pre + (size_t)p.Hk * p.pre_rows * 256 + ((size_t)h * p.pre_rows + row) * 128; }
__device__ __forceinline__ float* dn_pre_gb(const DnStepParams& p, int h, int64_t row) {
  return p.pre + (size_t)p.pre_rows * ((size_t)p.Hk * 256 + (size_t)p.Hv * 128) + ((size_t)h * p.pre_rows + row) * 2;
}
constexpr int DN_PRE_TOKENS = 64;
constexpr int DN_CHUNK_FROM = 64;   // sequences of this many tokens and more run the chunked recurrence, shorter ones the token-by-token scan

// alpha / beta projections of all rows of a pass (llm/deltanet.go:305-318): out[row][o], o = head for alpha, Hv + head for
// beta. A CTA keeps 16 rows of the normalised input in shared memory and takes its share of the 2*Hv weight rows; a warp takes two of
// them at a time, or, where the CTA has fewer pairs than warps, a slice of the contraction of two. Few rows are cut finely (12 CTAs
// that each walked 16 weight rows left a 37-row pass waiting for 20 us), many coarsely, since every CTA reads its 16 rows.
// grid (ceil(M / 16), cut), block 256, dynamic shared memory 16 * H halves.
constexpr int DN_AB_ROWS = 16;
__global__ void __launch_bounds__(256) dn_ab_kernel(DnStepParams p, int M) {
  extern __shared__ __align__(16) uint8_t dn_ab_smem[];
  __half* xs = reinterpret_cast<__half*>(dn_ab_smem);
  __shared__ float part[8][33];
  const int H = p.H, r0 = blockIdx.x * DN_AB_ROWS, nr = min(DN_AB_ROWS, M - r0);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  pdl_wait();
  pdl_launch();
  for (int i = tid; i < DN_AB_ROWS * H / 8; i += 256) {
    const int r = i / (H / 8), c = i - r * (H / 8);
    reinterpret_cast<uint4*>(xs)[i] = r < nr ? __ldcg(reinterpret_cast<const uint4*>(p.xn + (size_t)(r0 + r) * H) + c) : make_uint4(0, 0, 0, 0);
  }
  __syncthreads();
  auto row = [&](int o) { return o < p.Hv ? p.alpha_w + (size_t)o * H : p.beta_w + (size_t)(o - p.Hv) * H; };
  const int n_out = 2 * p.Hv, per = (n_out + gridDim.y - 1) / gridDim.y, o0 = blockIdx.y * per, o_end = min(n_out, o0 + per);
  const int pairs = (per + 1) / 2, ks = pairs >= 8 ? 1 : pairs >= 4 ? 2 : pairs >= 2 ? 4 : 8;   // warps that share a pair of weight rows
  const int kn = (H / 128 + ks - 1) / ks * 128, k0 = (warp % ks) * kn, k1 = min(H, k0 + kn);
  for (int b = o0; b < o_end; b += 2 * (8 / ks)) {
    const int o = b + 2 * (warp / ks);
    const bool one = o < o_end, two = o + 1 < o_end;
    const float *wa = row(one ? o : o0), *wb = row(two ? o + 1 : o0);
    float acc[32];   // [weight row][row]
#pragma unroll
    for (int r = 0; r < 32; r++) acc[r] = 0.f;
    for (int k = k0 + lane * 4; k < k1; k += 128) {
      const float4 va = *reinterpret_cast<const float4*>(wa + k), vb = *reinterpret_cast<const float4*>(wb + k);
#pragma unroll
      for (int r = 0; r < DN_AB_ROWS; r++) {
        const uint2 xv = *reinterpret_cast<const uint2*>(xs + (size_t)r * H + k);
        const float2 f01 = __half22float2(*reinterpret_cast<const __half2*>(&xv.x)), f23 = __half22float2(*reinterpret_cast<const __half2*>(&xv.y));
        acc[r] = fmaf(va.w, f23.y, fmaf(va.z, f23.x, fmaf(va.y, f01.y, fmaf(va.x, f01.x, acc[r]))));
        acc[16 + r] = fmaf(vb.w, f23.y, fmaf(vb.z, f23.x, fmaf(vb.y, f01.y, fmaf(vb.x, f01.x, acc[16 + r]))));
      }
    }
    // sums over the lanes: halves of the values change hands at each step, lane i ends with value i
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
      const bool up = lane & s;
#pragma unroll
      for (int i = 0; i < s; i++) acc[i] = (up ? acc[i + s] : acc[i]) + __shfl_xor_sync(0xffffffffu, up ? acc[i] : acc[i + s], s);
    }
    part[warp][lane] = acc[0];
    __syncthreads();
    if (warp % ks == 0) {
      float v = 0.f;
      for (int w = 0; w < ks; w++) v += part[warp + w][lane];
      const int r = lane & 15, h = lane >> 4;
      if (r < nr && (h ? two : one)) p.ab[(size_t)(r0 + r) * n_out + o + h] = v;
    }
    __syncthreads();
  }
}

// conv + SiLU of q, k and v, L2 norm of q and k, decay and beta: a warp takes one 128-channel head of q, k or v over eight
// tokens, four channels per lane, so the norm is a warp sum and nothing waits at a barrier (one CTA per head and 16 tokens
// with two barriers per token measured 148 us at 4096 rows; the bytes take 41). Conv inputs of the positions before this
// pass come from the rings the decode kernels keep per (head, row block). grid (2 Hk + Hv, n_seq, 64-token groups), block 256.
__global__ void __launch_bounds__(256) dn_pre_kernel(DnStepParams p) {
  constexpr int D = 128, RB = 4;
  const int kind = (int)blockIdx.x < p.Hk ? 0 : (int)blockIdx.x < 2 * p.Hk ? 1 : 2;      // q, k, v
  const int hd = blockIdx.x - (kind == 0 ? 0 : kind == 1 ? p.Hk : 2 * p.Hk);             // key head or value head
  const SeqDesc sq = p.seqs[blockIdx.y];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c = 4 * lane;
  const int i0 = blockIdx.z * DN_PRE_TOKENS + warp * 8, i1 = min(sq.n, i0 + 8);
  if (i0 >= sq.n) return;
  const int ch = kind * p.Hk * D + hd * D + c;                                           // channel of the projection row
  float4 w[4];
#pragma unroll
  for (int k = 0; k < 4; k++) w[k] = *reinterpret_cast<const float4*>(p.conv_w + (size_t)(ch + k) * 4);
  // ring of the decode kernels' CTA (head, row block): q at 0..127 and k at 128..255 of any CTA of a head whose key head
  // this is (head hd, block 0 is one), v at 256..287 of the block that owns the channel
  const float* ring = p.ring + (size_t)sq.slot * p.ring_slot_stride + (size_t)(kind < 2 ? hd * RB : hd * RB + (c >> 5)) * (DN_RING * DN_RING_W) + (kind < 2 ? 128 * kind + c : 256 + (c & 31));
  const float a_h = kind == 2 ? p.ssm_a[hd] : 0.f, dtb = kind == 2 ? p.dt_bias[hd] : 0.f;
  pdl_wait();
  pdl_launch();
  auto input = [&](int ii) {   // conv inputs of token index ii (negative: before this pass)
    if (ii >= 0) return __ldcg(reinterpret_cast<const float4*>(p.proj + (size_t)(sq.row0 + ii) * p.ldp + ch));
    const int pos = sq.pos0 + ii;
    return pos >= 0 ? *reinterpret_cast<const float4*>(ring + (size_t)(pos & (DN_RING - 1)) * DN_RING_W) : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  float4 x[11];
#pragma unroll
  for (int u = 0; u < 11; u++) x[u] = i0 - 3 + u < i1 ? input(i0 - 3 + u) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int u = 0; u < 8; u++) {
    if (i0 + u >= i1) break;
    const int row = sq.row0 + i0 + u;
    float4 v;
    v.x = silu_acc(x[u].x * w[0].x + x[u + 1].x * w[0].y + x[u + 2].x * w[0].z + x[u + 3].x * w[0].w);
    v.y = silu_acc(x[u].y * w[1].x + x[u + 1].y * w[1].y + x[u + 2].y * w[1].z + x[u + 3].y * w[1].w);
    v.z = silu_acc(x[u].z * w[2].x + x[u + 1].z * w[2].y + x[u + 2].z * w[2].z + x[u + 3].z * w[2].w);
    v.w = silu_acc(x[u].w * w[3].x + x[u + 1].w * w[3].y + x[u + 2].w * w[3].z + x[u + 3].w * w[3].w);
    if (kind < 2) {
      const float n = 1.0f / sqrtf(warp_sum((v.x * v.x + v.y * v.y) + (v.z * v.z + v.w * v.w)) + p.eps);
      v.x *= n; v.y *= n; v.z *= n; v.w *= n;
      *reinterpret_cast<float4*>(dn_pre_qk(p, hd, row) + 128 * kind + c) = v;
    } else {
      *reinterpret_cast<float4*>(dn_pre_v(p, hd, row) + c) = v;
    }
  }
  if (kind == 2 && lane < 8 && i0 + lane < i1) {   // decay and beta of the eight tokens, a lane each (one lane for all of them took half of the kernel)
    const int row = sq.row0 + i0 + lane;
    const float alpha = __ldcg(p.ab + (size_t)row * 2 * p.Hv + hd), betar = __ldcg(p.ab + (size_t)row * 2 * p.Hv + p.Hv + hd);
    *reinterpret_cast<float2*>(dn_pre_gb(p, hd, row)) = make_float2(expf(softplus_ref(alpha + dtb) * a_h), sigmoid_acc(betar));
  }
}

// The recurrence itself. A thread owns a quarter (32 of the 128 key dims) of one of the CTA's 32 state
// rows, in registers; per token it needs that quarter of k and q (fetched one token ahead), 32-term dot
// products as four interleaved partial sums, and two shuffles over the four lanes of a row. No shared
// memory and no barrier: every group of four lanes advances on its own. (The summation order differs from
// dn_step_kernel's, so the two forms agree to rounding, not to the bit.)
__global__ void __launch_bounds__(128) dn_scan_kernel(DnStepParams p) {
  const int D = 128, RB = 4;
  const int h = blockIdx.x / RB, rb = blockIdx.x % RB;
  const SeqDesc sq = p.seqs[blockIdx.y];
  const int tid = threadIdx.x, jl = tid >> 2, part = tid & 3;
  const int j = rb * 32 + jl;
  float* Srow = p.state + (size_t)sq.slot * p.state_slot_stride + (size_t)h * D * D + (size_t)j * D + 32 * part;
  float s[32];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const float4 v = *reinterpret_cast<const float4*>(Srow + 4 * i);
    s[4 * i] = v.x; s[4 * i + 1] = v.y; s[4 * i + 2] = v.z; s[4 * i + 3] = v.w;
  }
  const float oscale = 1.0f / sqrtf((float)D);
  pdl_wait();
  pdl_launch();
  const float* pqk = dn_pre_qk(p, h % p.Hk, sq.row0);
  const float* pv = dn_pre_v(p, h, sq.row0) + rb * 32;
  const float* pgb = dn_pre_gb(p, h, sq.row0);
  float4 kq[16], nkq[16];  // k quarter (8 float4) then q quarter
  float vv, nvv = 0.f; float2 gb, ngb = make_float2(0.f, 0.f);
  auto fetch = [&](int i, float4 (&dst)[16], float& v, float2& g) {
    const float* t = pqk + (size_t)i * 256;
#pragma unroll
    for (int u = 0; u < 8; u++) {
      dst[u] = __ldcg(reinterpret_cast<const float4*>(t + 128 + 32 * part + 4 * u));
      dst[8 + u] = __ldcg(reinterpret_cast<const float4*>(t + 32 * part + 4 * u));
    }
    v = __ldcg(pv + (size_t)i * 128 + jl);
    g = __ldcg(reinterpret_cast<const float2*>(pgb + (size_t)i * 2));
  };
  fetch(0, kq, vv, gb);
  for (int i = 0; i < sq.n; i++) {
    if (i + 1 < sq.n) fetch(i + 1, nkq, nvv, ngb);
    const float g = gb.x, beta = gb.y;
    float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll
    for (int u = 0; u < 8; u++) {
      a0 = fmaf(s[4 * u], kq[u].x, a0); a1 = fmaf(s[4 * u + 1], kq[u].y, a1);
      a2 = fmaf(s[4 * u + 2], kq[u].z, a2); a3 = fmaf(s[4 * u + 3], kq[u].w, a3);
    }
    float kv = (a0 + a1) + (a2 + a3);
    kv += __shfl_xor_sync(0xffffffffu, kv, 1);
    kv += __shfl_xor_sync(0xffffffffu, kv, 2);
    // S *= g; u = (v - S^T k) * beta; S += k u^T   (llm/deltanet.go:365-418), with g factored out of the dot
    const float dj = (vv - g * kv) * beta;
    float o0 = 0.f, o1 = 0.f, o2 = 0.f, o3 = 0.f;
#pragma unroll
    for (int u = 0; u < 8; u++) {
      s[4 * u] = fmaf(dj, kq[u].x, s[4 * u] * g); s[4 * u + 1] = fmaf(dj, kq[u].y, s[4 * u + 1] * g);
      s[4 * u + 2] = fmaf(dj, kq[u].z, s[4 * u + 2] * g); s[4 * u + 3] = fmaf(dj, kq[u].w, s[4 * u + 3] * g);
      o0 = fmaf(s[4 * u], kq[8 + u].x, o0); o1 = fmaf(s[4 * u + 1], kq[8 + u].y, o1);
      o2 = fmaf(s[4 * u + 2], kq[8 + u].z, o2); o3 = fmaf(s[4 * u + 3], kq[8 + u].w, o3);
    }
    float ov = (o0 + o1) + (o2 + o3);
    ov += __shfl_xor_sync(0xffffffffu, ov, 1);
    ov += __shfl_xor_sync(0xffffffffu, ov, 2);
    if (part == 0) p.o_raw[(size_t)(sq.row0 + i) * (p.Hv * D) + h * D + j] = ov * oscale;
#pragma unroll
    for (int u = 0; u < 16; u++) kq[u] = nkq[u];
    vv = nvv; gb = ngb;
  }
#pragma unroll
  for (int i = 0; i < 8; i++) *reinterpret_cast<float4*>(Srow + 4 * i) = make_float4(s[4 * i], s[4 * i + 1], s[4 * i + 2], s[4 * i + 3]);
  // the ring keeps the last positions' conv inputs (written here, after every read of the old ring)
  {
    const int hk = h % p.Hk, qk = p.Hk * D;
    const int ch_q = hk * D + tid, ch_k = qk + hk * D + tid, ch_v = 2 * qk + h * D + rb * 32 + (tid & 31);
    float* ring = p.ring + (size_t)sq.slot * p.ring_slot_stride + (size_t)blockIdx.x * (DN_RING * DN_RING_W);
    for (int i = max(0, sq.n - DN_RING); i < sq.n; i++) {
      const float* pr = p.proj + (size_t)(sq.row0 + i) * p.ldp;
      float* rw = ring + (size_t)((sq.pos0 + i) & (DN_RING - 1)) * DN_RING_W;
      rw[tid] = pr[ch_q]; rw[128 + tid] = pr[ch_k];
      if (tid < 32) rw[256 + tid] = pr[ch_v];
    }
  }
}

// -----------------------------------------------------------------------------------------
// The recurrence in chunks of 64 tokens (the WY form of the gated delta rule). Within a chunk the per-token updates
// s_j <- g_t s_j + beta_t (v_t[j] - g_t s_j . k_t) k_t  are solved for all tokens at once: with L_t = sum_{r<=t} log g_r,
// Gamma_t = exp(L_t) and ratio(t, r) = exp(L_t - L_r),
//   A[t][r] = beta_t ratio(t, r) (k_t . k_r)  (r < t),   T = (I + A)^-1,   W[t][r] = ratio(t, r) (q_t . k_r)  (r <= t),
//   U = T (beta V),   Y = T (beta Gamma K),   D = U - Y S0^T,
//   o_t = (Gamma_t S0 q_t + sum_r W[t][r] D[r]) / sqrt(128),   S_C = Gamma_C S0 + sum_r ratio(C, r) D[r] k_r^T,
// the token-by-token recurrence re-associated (llm/deltanet.go:365-418 is the sequential form; the reference has no chunked
// one, llm/gpu_deltanet.go:48-52). Everything up to Y needs no state: dn_wy_kernel forms it for every chunk in parallel and
// leaves dn_chunk_kernel, which walks the chunks, three products against the 32 state rows a CTA owns.
//
// The state and the recurrence are f32 throughout in the reference's device path, so the products run as split TF32: every
// operand is hi + lo with hi rounded to TF32 and lo the exact rest, and hi hi + (hi lo + lo hi) is accumulated in f32; the
// logarithms L are summed and subtracted in f64, since their differences are what exp magnifies. Against the recurrence in f64 (2048
// tokens, 32 heads, relative 2-norm of the outputs / of the state): 2.3e-7 / 1.7e-7 with decays as config.py draws them, 2.6e-7 / 3.1e-7
// with a hundredth of their logarithms. The form before (f32 on the FMA pipe, f32 logarithms): 8.9e-7 / 6.3e-7 and 2.4e-7 / 3.1e-7; hi hi
// summed by the tensor core: 4.4e-7 / 1.7e-7 and 4.7e-7 / 4.1e-7. mma.sync TF32 runs at 500 multiply-adds per cycle and SM, three to one
// here: 1.3 times the FMA pipe, at a tenth of its shared-memory reads, which is what bounded the register-tiled form.
// 4096 tokens, 32 heads: 1706 us as one kernel on the FMA pipe.
// -----------------------------------------------------------------------------------------
constexpr int DN_C = 64;                            // tokens per chunk
// pitches (floats) of shared-memory rows: 16-byte reads of rows g at 16 kk + 4 t want 16 mod 32, 4-byte reads of rows t at
// column g want 8, of rows g at column t want 4
constexpr int DN_P16 = 144, DN_P8 = 136, DN_P4 = 68, DN_PD = 40, DN_PU = 36;

__device__ __forceinline__ void tf_split(float x, uint32_t& hi, uint32_t& lo) {
  hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
  lo = __float_as_uint(x - __uint_as_float(hi));
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
struct TfA { uint32_t hi[4], lo[4]; };
struct TfB { uint32_t hi[2], lo[2]; };
__device__ __forceinline__ TfA tf_a(float a0, float a1, float a2, float a3) {
  TfA r;
  tf_split(a0, r.hi[0], r.lo[0]); tf_split(a1, r.hi[1], r.lo[1]); tf_split(a2, r.hi[2], r.lo[2]); tf_split(a3, r.hi[3], r.lo[3]);
  return r;
}
__device__ __forceinline__ TfB tf_b(float b0, float b1) {
  TfB r;
  tf_split(b0, r.hi[0], r.lo[0]); tf_split(b1, r.hi[1], r.lo[1]);
  return r;
}
// main += hi hi, cross += hi lo + lo hi. The large term's sum is an f32 addition, not the tensor core's own, which rounds towards zero.
__device__ __forceinline__ void mma_split(float (&main)[4], float (&cross)[4], const TfA& a, const TfB& b) {
  float m[4] = {0.f, 0.f, 0.f, 0.f};
  mma_tf32(m, a.hi, b.hi[0], b.hi[1]);
#pragma unroll
  for (int i = 0; i < 4; i++) main[i] += m[i];
  mma_tf32(cross, a.hi, b.lo[0], b.lo[1]);
  mma_tf32(cross, a.lo, b.hi[0], b.hi[1]);
}
// One 16 x 8*NT tile over 128 (float4 steps of 16): X rows m0 + g, + 8 and Y rows n0 + 8 nt + g, both at pitch DN_P16. A lane
// takes four consecutive elements of each row; the mma's k slots are whatever those are, in X and Y alike.
template <int NT>
__device__ __forceinline__ void rows_by_rows(const float* X, const float* Y, int g, int t, float (&main)[NT][4], float (&cross)[NT][4], int live = NT) {
#pragma unroll
  for (int n = 0; n < NT; n++)
#pragma unroll
    for (int i = 0; i < 4; i++) { main[n][i] = 0.f; cross[n][i] = 0.f; }
#pragma unroll 2
  for (int kk = 0; kk < 8; kk++) {
    const float4 xa = *reinterpret_cast<const float4*>(X + g * DN_P16 + 16 * kk + 4 * t), xb = *reinterpret_cast<const float4*>(X + (g + 8) * DN_P16 + 16 * kk + 4 * t);
    const TfA a0 = tf_a(xa.x, xb.x, xa.y, xb.y), a1 = tf_a(xa.z, xb.z, xa.w, xb.w);
#pragma unroll
    for (int n = 0; n < NT; n++) {
      if (n < live) {
        const float4 y = *reinterpret_cast<const float4*>(Y + (8 * n + g) * DN_P16 + 16 * kk + 4 * t);
        mma_split(main[n], cross[n], a0, tf_b(y.x, y.y));
        mma_split(main[n], cross[n], a1, tf_b(y.z, y.w));
      }
    }
  }
}
__device__ __forceinline__ float* dn_y(const DnStepParams& p, int h, int64_t row) { return p.wy + ((size_t)h * p.pre_rows + row) * 128; }
__device__ __forceinline__ float* dn_w(const DnStepParams& p, int h, int64_t row) { return p.wy + (size_t)p.Hv * p.pre_rows * 128 + ((size_t)h * p.pre_rows + row) * 64; }

// What a chunk needs before its state is known. A CTA takes one chunk of one key head: K K^T and Q K^T once, then for each of
// the value heads that read this key head A, T, W, U (in place of V), Y, and (Gamma, ratio(C, .)) in place of (decay, beta).
// T by blocks of 16: the diagonal ones by substitution (a lane per column, in registers), the rest block row by block row.
// grid (chunks, Hk, n_seq), block 512.
constexpr size_t DN_WY_SMEM = sizeof(float) * (2 * DN_C * DN_P16 + DN_C * DN_P8 + 4 * DN_C * DN_P4 + 4 * DN_C);
__global__ void __launch_bounds__(512, 1) dn_wy_kernel(DnStepParams p) {
  const SeqDesc sq = p.seqs[blockIdx.z];
  const int hk = blockIdx.y, c0 = blockIdx.x * DN_C, n = min(DN_C, sq.n - c0);
  if (n <= 0) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3, w8 = warp & 7;
  const int64_t row0 = sq.row0 + c0;
  extern __shared__ __align__(16) float dn_smem[];
  float* Ks = dn_smem;                          // [64][P16]
  float* Qs = Ks + DN_C * DN_P16;               // [64][P16]
  float* Vs = Qs + DN_C * DN_P16;               // [64][P8]
  float* KK = Vs + DN_C * DN_P8;                // [64][P4] each
  float* QK = KK + DN_C * DN_P4;
  float* Am = QK + DN_C * DN_P4;
  float* Tm = Am + DN_C * DN_P4;                // lower blocks: T; upper blocks: scratch
  double* Lg = reinterpret_cast<double*>(Tm + DN_C * DN_P4);   // [64] cumulative log decay
  float* Bt = Tm + DN_C * DN_P4 + 2 * DN_C;     // [64] beta
  float* Gm = Bt + DN_C;                        // [64] beta Gamma
  pdl_wait();
  pdl_launch();
  for (int i = tid; i < DN_C * 64; i += 512) {
    const int r = i >> 6, c = i & 63;           // 64 float4 per token: 32 of q, 32 of k
    const float4 v = r < n ? __ldcg(reinterpret_cast<const float4*>(dn_pre_qk(p, hk, row0 + r) + 4 * c)) : make_float4(0.f, 0.f, 0.f, 0.f);
    *reinterpret_cast<float4*>((c < 32 ? Qs : Ks) + r * DN_P16 + 4 * (c & 31)) = v;
  }
  __syncthreads();
  {
    // lower triangles only: 20 tiles of 16 x 8 for each product, at most three to a warp
    const int mt = w8 < 3 ? 3 : w8 < 5 ? 2 : w8 < 7 ? 1 : 0, nt0 = w8 == 1 || w8 == 4 ? 3 : w8 == 2 ? 6 : w8 == 6 ? 2 : 0, nts = w8 == 0 || w8 == 1 || w8 == 3 || w8 == 4 ? 3 : 2;
    float m[3][4], x[3][4];
    rows_by_rows<3>((warp >= 8 ? Qs : Ks) + mt * 16 * DN_P16, Ks + nt0 * 8 * DN_P16, g, t, m, x, nts);
    float* out = (warp >= 8 ? QK : KK) + (mt * 16 + g) * DN_P4 + nt0 * 8 + 2 * t;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      if (i < nts) {
        *reinterpret_cast<float2*>(out + 8 * i) = make_float2(m[i][0] + x[i][0], m[i][1] + x[i][1]);
        *reinterpret_cast<float2*>(out + 8 * DN_P4 + 8 * i) = make_float2(m[i][2] + x[i][2], m[i][3] + x[i][3]);
      }
    }
  }
  for (int h = hk; h < p.Hv; h += p.Hk) {
    if (warp == 0) {                            // cumulative log decay of the chunk: two tokens per lane
      const int t0 = 2 * lane, t1 = t0 + 1;
      float2 e0 = make_float2(1.f, 0.f), e1 = e0;
      if (t0 < n) e0 = __ldcg(reinterpret_cast<const float2*>(dn_pre_gb(p, h, row0 + t0)));
      if (t1 < n) e1 = __ldcg(reinterpret_cast<const float2*>(dn_pre_gb(p, h, row0 + t1)));
      const double l0 = fmaxf(logf(e0.x), -87.f), l1 = fmaxf(logf(e1.x), -87.f);
      double run = l0 + l1;                     // inclusive scan over the lanes' pair sums
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const double up = __shfl_up_sync(0xffffffffu, run, o); if (lane >= o) run += up; }
      const double total = __shfl_sync(0xffffffffu, run, 31), la = run - l1;
      Lg[t0] = la; Lg[t1] = run; Bt[t0] = e0.y; Bt[t1] = e1.y; Gm[t0] = e0.y * expf((float)la); Gm[t1] = e1.y * expf((float)run);
      if (t0 < n) *reinterpret_cast<float2*>(dn_pre_gb(p, h, row0 + t0)) = make_float2(expf((float)la), expf((float)(total - la)));
      if (t1 < n) *reinterpret_cast<float2*>(dn_pre_gb(p, h, row0 + t1)) = make_float2(expf((float)run), expf((float)(total - run)));
    }
    for (int i = tid; i < DN_C * 32; i += 512) {
      const int r = i >> 5, c = i & 31;
      const float4 v = r < n ? __ldcg(reinterpret_cast<const float4*>(dn_pre_v(p, h, row0 + r) + 4 * c)) : make_float4(0.f, 0.f, 0.f, 0.f);
      *reinterpret_cast<float4*>(Vs + r * DN_P8 + 4 * c) = v;
    }
    __syncthreads();
    for (int i = tid; i < DN_C * DN_C; i += 512) {
      const int r = i >> 6, c = i & 63;
      const float ratio = c <= r ? expf((float)(Lg[r] - Lg[c])) : 0.f;
      Am[r * DN_P4 + c] = c < r ? Bt[r] * ratio * KK[r * DN_P4 + c] : 0.f;
      if (r < n) dn_w(p, h, row0 + r)[c] = c <= r ? ratio * QK[r * DN_P4 + c] : 0.f;
    }
    __syncthreads();
    if (warp < 4 && lane < 16) {                // diagonal blocks of T: column `lane` of block `warp`
      const float* a = Am + 16 * warp * (DN_P4 + 1);
      float* o = Tm + 16 * warp * (DN_P4 + 1) + lane;
      float x[16];
#pragma unroll
      for (int r = 0; r < 16; r++) {
        float v = r == lane ? 1.f : 0.f;
#pragma unroll
        for (int c = 0; c < 16; c++)
          if (c < r) v -= a[r * DN_P4 + c] * x[c];
        x[r] = v;
        o[r * DN_P4] = v;
      }
    }
    __syncthreads();
    for (int lv = 1; lv < 4; lv++) {            // T_ba = -T_bb sum_{a <= c < b} A_bc T_ca for b = a + lv; the sums wait in block (a, b)
      for (int i = tid; i < (4 - lv) * 256; i += 512) {
        const int a = i >> 8, b = a + lv, r = (i >> 4) & 15, c = i & 15;
        const float* ar = Am + (16 * b + r) * DN_P4 + 16 * a;
        const float* tc = Tm + 16 * a * DN_P4 + 16 * a + c;
        float s = 0.f;
        for (int k = 0; k < 16 * lv; k++) s = fmaf(ar[k], tc[k * DN_P4], s);
        Tm[(16 * a + r) * DN_P4 + 16 * b + c] = s;
      }
      __syncthreads();
      for (int i = tid; i < (4 - lv) * 256; i += 512) {
        const int a = i >> 8, b = a + lv, r = (i >> 4) & 15, c = i & 15;
        const float* tr = Tm + (16 * b + r) * DN_P4 + 16 * b;
        const float* xc = Tm + 16 * a * DN_P4 + 16 * b + c;
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < 16; k++) s = fmaf(tr[k], xc[k * DN_P4], s);
        Tm[(16 * b + r) * DN_P4 + 16 * a + c] = -s;
      }
      __syncthreads();
    }
    {
      // U (first eight warps) and Y: all 64 rows x 16 columns per warp, contraction up to the diagonal block
      const bool second = warp >= 8;
      const float* B = second ? Ks : Vs;
      const int bp = second ? DN_P16 : DN_P8;
      const float* sc = second ? Gm : Bt;
      float m[4][2][4], x[4][2][4];
#pragma unroll
      for (int a = 0; a < 32; a++) { (&m[0][0][0])[a] = 0.f; (&x[0][0][0])[a] = 0.f; }
#pragma unroll
      for (int k8 = 0; k8 < 8; k8++) {
        const int ka = k8 * 8 + t, kb = ka + 4;
        const float sa = sc[ka], sb = sc[kb];
        TfB b[2];
#pragma unroll
        for (int nt = 0; nt < 2; nt++) b[nt] = tf_b(B[ka * bp + w8 * 16 + nt * 8 + g], B[kb * bp + w8 * 16 + nt * 8 + g]);
#pragma unroll
        for (int mt = 0; mt < 4; mt++) {
          if (mt >= (k8 >> 1)) {
            const float* tr = Tm + (mt * 16 + g) * DN_P4;
            const TfA a = tf_a(tr[ka] * sa, tr[8 * DN_P4 + ka] * sa, tr[kb] * sb, tr[8 * DN_P4 + kb] * sb);
#pragma unroll
            for (int nt = 0; nt < 2; nt++) mma_split(m[mt][nt], x[mt][nt], a, b[nt]);
          }
        }
      }
#pragma unroll
      for (int mt = 0; mt < 4; mt++)
#pragma unroll
        for (int nt = 0; nt < 2; nt++)
#pragma unroll
          for (int hh = 0; hh < 2; hh++) {
            const int r = mt * 16 + g + 8 * hh;
            if (r < n) *reinterpret_cast<float2*>((second ? dn_y(p, h, row0 + r) : dn_pre_v(p, h, row0 + r)) + w8 * 16 + nt * 8 + 2 * t) = make_float2(m[mt][nt][2 * hh] + x[mt][nt][2 * hh], m[mt][nt][2 * hh + 1] + x[mt][nt][2 * hh + 1]);
          }
    }
    __syncthreads();                            // V, A and T are free for the next head
  }
}

// The walk over the chunks. A CTA owns 32 of a head's 128 state rows: kept as f32 in the registers of the warps that update
// them, with a copy in shared memory for the products that read them. Per chunk two phases: warps 0..7 form D while warps
// 8..15 form Gamma Q S^T; then warps 0..7 update the state while warps 8..15 add W D and write the outputs. What a phase has
// read is refilled for the next chunk by asynchronous copies under the other phase. grid (Hv * 4, n_seq), block 512.
constexpr size_t DN_CHUNK_SMEM = sizeof(float) * (2 * DN_C * DN_P16 + DN_C * DN_P8 + DN_C * DN_P4 + DN_C * DN_PU + 32 * DN_P16 + DN_C * DN_PD + 4 * DN_C);
__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool live) {   // zeros when not live
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__global__ void __launch_bounds__(512, 1) dn_chunk_kernel(DnStepParams p) {
  constexpr int D = 128, RB = 4;
  const int h = blockIdx.x / RB, rb = blockIdx.x % RB, hk = h % p.Hk;
  const SeqDesc sq = p.seqs[blockIdx.y];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3, w8 = warp & 7;
  const bool second = warp >= 8;
  extern __shared__ __align__(16) float dn_smem[];
  float* Ys = dn_smem;                          // [64][P16]
  float* Qs = Ys + DN_C * DN_P16;               // [64][P16]
  float* Ks = Qs + DN_C * DN_P16;               // [64][P8]
  float* Ws = Ks + DN_C * DN_P8;                // [64][P4]
  float* Us = Ws + DN_C * DN_P4;                // [64][PU]
  float* ST = Us + DN_C * DN_PU;                // [32][P16] the state rows
  float* Ds = ST + 32 * DN_P16;                 // [64][PD]
  float* gam = Ds + DN_C * DN_PD;               // [2][64][2] (Gamma_t, ratio(C, t)) of this chunk and the next
  float* Sg = p.state + (size_t)sq.slot * p.state_slot_stride + (size_t)h * D * D + (size_t)(rb * 32) * D;
  // the state block does not depend on the producer kernel
  float s[2][2][4];                             // warps 0..7: rows 16 mt + g (+ 8), columns 16 w8 + 8 nt + 2t (+ 1)
  for (int i = tid; i < 32 * 32; i += 512) *reinterpret_cast<float4*>(ST + (i >> 5) * DN_P16 + 4 * (i & 31)) = *reinterpret_cast<const float4*>(Sg + 4 * i);
  if (!second) {
#pragma unroll
    for (int mt = 0; mt < 2; mt++)
#pragma unroll
      for (int nt = 0; nt < 2; nt++)
#pragma unroll
        for (int hh = 0; hh < 2; hh++) {
          const float2 v = *reinterpret_cast<const float2*>(Sg + (size_t)(16 * mt + g + 8 * hh) * D + 16 * w8 + 8 * nt + 2 * t);
          s[mt][nt][2 * hh] = v.x; s[mt][nt][2 * hh + 1] = v.y;
        }
  }
  const float oscale = 1.0f / sqrtf((float)D);
  pdl_wait();
  pdl_launch();
  const float *pqk = dn_pre_qk(p, hk, sq.row0), *pu = dn_pre_v(p, h, sq.row0) + rb * 32, *pg = dn_pre_gb(p, h, sq.row0), *py = dn_y(p, h, sq.row0), *pw = dn_w(p, h, sq.row0);
  auto load_first = [&](int c0, int buf) {      // what phase 1 reads (and the factors)
    for (int i = tid; i < DN_C * 32; i += 512) {
      const int r = i >> 5, c = 4 * (i & 31);
      const bool live = c0 + r < sq.n;
      const int64_t row = live ? c0 + r : 0;
      cp_async16(Ys + r * DN_P16 + c, py + row * 128 + c, live);
      cp_async16(Qs + r * DN_P16 + c, pqk + row * 256 + c, live);
    }
    { const int r = tid >> 3, c = 4 * (tid & 7); const bool live = c0 + r < sq.n; cp_async16(Us + r * DN_PU + c, pu + (live ? (int64_t)(c0 + r) * 128 : 0) + c, live); }
    if (tid < 64) {
      const bool live = c0 + tid < sq.n;
      const float2 v = live ? __ldcg(reinterpret_cast<const float2*>(pg + (int64_t)(c0 + tid) * 2)) : make_float2(0.f, 0.f);
      *reinterpret_cast<float2*>(gam + buf * 128 + 2 * tid) = v;
    }
  };
  auto load_second = [&](int c0) {              // what phase 2 reads
    for (int i = tid; i < DN_C * 32; i += 512) {
      const int r = i >> 5, c = 4 * (i & 31);
      const bool live = c0 + r < sq.n;
      cp_async16(Ks + r * DN_P8 + c, pqk + (live ? (int64_t)(c0 + r) * 256 : 0) + 128 + c, live);
    }
    for (int i = tid; i < DN_C * 16; i += 512) {
      const int r = i >> 4, c = 4 * (i & 15);
      const bool live = c0 + r < sq.n;
      cp_async16(Ws + r * DN_P4 + c, pw + (live ? (int64_t)(c0 + r) * 64 : 0) + c, live);
    }
  };
  load_first(0, 0);
  cp_async_wait_all();
  __syncthreads();
  load_second(0);
  const int mt4 = w8 & 3, nh = w8 >> 2;         // 16-token tile and 16-column half of the products with 64 x 32 results
  int buf = 0;
  for (int c0 = 0; c0 < sq.n; c0 += DN_C, buf ^= 1) {
    const int n = min(DN_C, sq.n - c0);
    const float* gm = gam + buf * 128;
    float o[2][4];
    {
      float m[2][4], x[2][4];
      rows_by_rows<2>((second ? Qs : Ys) + mt4 * 16 * DN_P16, ST + nh * 16 * DN_P16, g, t, m, x);
#pragma unroll
      for (int nt = 0; nt < 2; nt++)
#pragma unroll
        for (int hh = 0; hh < 2; hh++) {
          const int r = mt4 * 16 + g + 8 * hh, c = nh * 16 + 8 * nt + 2 * t;
          const float v0 = m[nt][2 * hh] + x[nt][2 * hh], v1 = m[nt][2 * hh + 1] + x[nt][2 * hh + 1];
          if (second) {
            const float gr = gm[2 * r];
            o[nt][2 * hh] = gr * v0; o[nt][2 * hh + 1] = gr * v1;
          } else {
            const float2 u = *reinterpret_cast<const float2*>(Us + r * DN_PU + c);
            *reinterpret_cast<float2*>(Ds + r * DN_PD + c) = make_float2(u.x - v0, u.y - v1);
          }
        }
    }
    cp_async_wait_all();
    __syncthreads();                            // D is there, this chunk's K and W have landed, Y, Q and U are free
    if (c0 + DN_C < sq.n) load_first(c0 + DN_C, buf ^ 1);
    if (second) {
      float x[2][4];
#pragma unroll
      for (int i = 0; i < 8; i++) (&x[0][0])[i] = 0.f;
      for (int k8 = 0; k8 < 2 * (mt4 + 1); k8++) {
        const int ka = 8 * k8 + t, kb = ka + 4;
        const float* w = Ws + (mt4 * 16 + g) * DN_P4;
        const TfA a = tf_a(w[ka], w[8 * DN_P4 + ka], w[kb], w[8 * DN_P4 + kb]);
#pragma unroll
        for (int nt = 0; nt < 2; nt++) mma_split(o[nt], x[nt], a, tf_b(Ds[ka * DN_PD + nh * 16 + 8 * nt + g], Ds[kb * DN_PD + nh * 16 + 8 * nt + g]));
      }
#pragma unroll
      for (int nt = 0; nt < 2; nt++)
#pragma unroll
        for (int hh = 0; hh < 2; hh++) {
          const int r = mt4 * 16 + g + 8 * hh;
          if (r < n) *reinterpret_cast<float2*>(p.o_raw + (size_t)(sq.row0 + c0 + r) * (p.Hv * D) + h * D + rb * 32 + nh * 16 + 8 * nt + 2 * t) =
              make_float2((o[nt][2 * hh] + x[nt][2 * hh]) * oscale, (o[nt][2 * hh + 1] + x[nt][2 * hh + 1]) * oscale);
        }
    } else {
      const float gc = gm[2 * (n - 1)];
      float x[2][2][4];
#pragma unroll
      for (int i = 0; i < 16; i++) { (&s[0][0][0])[i] *= gc; (&x[0][0][0])[i] = 0.f; }
#pragma unroll 2
      for (int k8 = 0; k8 < 8; k8++) {
        const int ka = 8 * k8 + t, kb = ka + 4;
        const float ca = gm[2 * ka + 1], cb = gm[2 * kb + 1];
        TfB b[2];
#pragma unroll
        for (int nt = 0; nt < 2; nt++) b[nt] = tf_b(Ks[ka * DN_P8 + 16 * w8 + 8 * nt + g], Ks[kb * DN_P8 + 16 * w8 + 8 * nt + g]);
#pragma unroll
        for (int mt = 0; mt < 2; mt++) {
          const float *da = Ds + ka * DN_PD + 16 * mt + g, *db = Ds + kb * DN_PD + 16 * mt + g;
          const TfA a = tf_a(da[0] * ca, da[8] * ca, db[0] * cb, db[8] * cb);
#pragma unroll
          for (int nt = 0; nt < 2; nt++) mma_split(s[mt][nt], x[mt][nt], a, b[nt]);
        }
      }
#pragma unroll
      for (int mt = 0; mt < 2; mt++)
#pragma unroll
        for (int nt = 0; nt < 2; nt++)
#pragma unroll
          for (int hh = 0; hh < 2; hh++) {
            float* sv = &s[mt][nt][2 * hh];
            sv[0] += x[mt][nt][2 * hh]; sv[1] += x[mt][nt][2 * hh + 1];
            *reinterpret_cast<float2*>(ST + (16 * mt + g + 8 * hh) * DN_P16 + 16 * w8 + 8 * nt + 2 * t) = make_float2(sv[0], sv[1]);
          }
    }
    cp_async_wait_all();
    __syncthreads();                            // the state is there, the next Y, Q and U have landed, K, W and D are free
    if (c0 + DN_C < sq.n) load_second(c0 + DN_C);
  }
  if (!second) {
#pragma unroll
    for (int mt = 0; mt < 2; mt++)
#pragma unroll
      for (int nt = 0; nt < 2; nt++)
#pragma unroll
        for (int hh = 0; hh < 2; hh++)
          *reinterpret_cast<float2*>(Sg + (size_t)(16 * mt + g + 8 * hh) * D + 16 * w8 + 8 * nt + 2 * t) = make_float2(s[mt][nt][2 * hh], s[mt][nt][2 * hh + 1]);
  }
  // the ring keeps the last positions' conv inputs (written here, after every read of the old ring by the pre-pass)
  if (tid < 128) {
    const int qk = p.Hk * D;
    const int ch_q = hk * D + tid, ch_k = qk + hk * D + tid, ch_v = 2 * qk + h * D + rb * 32 + (tid & 31);
    float* ring = p.ring + (size_t)sq.slot * p.ring_slot_stride + (size_t)blockIdx.x * (DN_RING * DN_RING_W);
    for (int i = max(0, sq.n - DN_RING); i < sq.n; i++) {
      const float* pr = p.proj + (size_t)(sq.row0 + i) * p.ldp;
      float* rw = ring + (size_t)((sq.pos0 + i) & (DN_RING - 1)) * DN_RING_W;
      rw[tid] = pr[ch_q]; rw[128 + tid] = pr[ch_k];
      if (tid < 32) rw[256 + tid] = pr[ch_v];
    }
  }
}

// gated RMSNorm of a token's heads, a warp per (row, head), four of its 128 outputs per lane. grid ceil(M * Hv / 8), block 256.
__global__ void __launch_bounds__(256) dn_post_kernel(DnStepParams p, int M) {
  constexpr int D = 128;
  const int w = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int row = w / p.Hv, h = w - row * p.Hv;
  if (row >= M) return;
  const float4 z = *reinterpret_cast<const float4*>(p.proj + (size_t)row * p.ldp + 2 * p.Hk * D + p.Hv * D + h * D + 4 * lane);   // written three kernels back
  const float4 nw = *reinterpret_cast<const float4*>(p.norm_w + 4 * lane);
  pdl_wait();
  pdl_launch();
  const float4 o = __ldcg(reinterpret_cast<const float4*>(p.o_raw + (size_t)row * (p.Hv * D) + h * D + 4 * lane));
  const float sc = 1.0f / sqrtf(warp_sum((o.x * o.x + o.y * o.y) + (o.z * o.z + o.w * o.w)) / (float)D + p.eps);
  const uint2 v = make_uint2(pack_half2(o.x * sc * nw.x * sigmoid_acc(z.x), o.y * sc * nw.y * sigmoid_acc(z.y)), pack_half2(o.z * sc * nw.z * sigmoid_acc(z.z), o.w * sc * nw.w * sigmoid_acc(z.w)));
  *reinterpret_cast<uint2*>(p.y16 + (size_t)row * (p.Hv * D) + h * D + 4 * lane) = v;
}

int launch_dn_scan(const DnStepParams& p, int M, int max_n, int* n_launches, bool pdl, cudaStream_t st) {
  if (p.D != 128 || p.conv != 4) { set_error("dn_scan: head dim must be 128 and conv kernel 4"); return EINVAL_; }
  if (p.mid != nullptr || p.pre == nullptr || p.o_raw == nullptr) { set_error("dn_scan: not available for speculative passes"); return EINVAL_; }
  if (p.ab == nullptr || p.H % 128 != 0 || (size_t)DN_AB_ROWS * p.H * 2 > 200 * 1024) { set_error("dn_scan: row length must be a multiple of 128 (at most 6400)"); return EINVAL_; }
  const int ab_smem = DN_AB_ROWS * p.H * 2;
  B200_ONCE_PER_DEVICE(cudaFuncSetAttribute(dn_ab_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
  // the weight rows cut in 16 or in 8, prompts of 12 layers: 128 rows 4271 or 4299 us, 256 rows 6372 or 6379, 701 rows 9685 or 9667, 2048 rows 13593 or 13531
  B200_TRY(launch_k(dn_ab_kernel, dim3((M + DN_AB_ROWS - 1) / DN_AB_ROWS, M <= 256 ? 16 : 8), dim3(256), ab_smem, pdl, st, p, M));
  B200_TRY(launch_k(dn_pre_kernel, dim3(2 * p.Hk + p.Hv, p.n_seq, (max_n + DN_PRE_TOKENS - 1) / DN_PRE_TOKENS), dim3(256), 0, true, st, p));
  *n_launches = 4;
  if (max_n >= DN_CHUNK_FROM) {
    // long sequences: the recurrence in chunks of 64 tokens
    if (p.wy == nullptr) { set_error("dn_scan: no buffer for the chunked form"); return EINVAL_; }
    B200_ONCE_PER_DEVICE(cudaFuncSetAttribute(dn_wy_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DN_WY_SMEM));
    B200_ONCE_PER_DEVICE(cudaFuncSetAttribute(dn_chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DN_CHUNK_SMEM));
    B200_TRY(launch_k(dn_wy_kernel, dim3((max_n + DN_C - 1) / DN_C, p.Hk, p.n_seq), dim3(512), DN_WY_SMEM, true, st, p));
    B200_TRY(launch_k(dn_chunk_kernel, dim3(p.Hv * 4, p.n_seq), dim3(512), DN_CHUNK_SMEM, true, st, p));
    *n_launches = 5;
  } else {
    B200_TRY(launch_k(dn_scan_kernel, dim3(p.Hv * 4, p.n_seq), dim3(128), 0, true, st, p));
  }
  return launch_k(dn_post_kernel, dim3((M * p.Hv + 7) / 8), dim3(256), 0, true, st, p, M);
}

int launch_dn_step(const DnStepParams& p, bool pdl, cudaStream_t st) {
  if (p.D != 128 || p.conv != 4) { set_error("dn_step: head dim must be 128 and conv kernel 4"); return EINVAL_; }
  // (passes of at most 8 sequences stay on dn_step_kernel: they give every row the single-row pass's bits)
  if (p.n_seq >= 16) return launch_k(dn_head_kernel, dim3(p.Hv, p.n_seq), dim3(512), 0, pdl, st, p);
  // five CTAs to an SM or one, batched steps of 12 layers: 2 sequences 768 or 746 us, 3 sequences 900 or 909, 5 sequences 1123 or 1148
  if (p.n_seq > 2) return launch_k(dn_step_kernel<5>, dim3(p.Hv * 4, p.n_seq), dim3(128), 0, pdl, st, p);
  return launch_k(dn_step_kernel<1>, dim3(p.Hv * 4, p.n_seq), dim3(128), 0, pdl, st, p);
}

// =========================================================================================
// Attention pre-pass: per-head RMSNorm of q and k, NeoX partial rotary from a host-built
// table, fp16 K/V into the cache (reference: llm/attn.go:144-184, 510-586;
// shaders/llm_attn_pack.comp). A warp per (row, head): the norm is a warp sum and the rotary partner comes from shared
// memory of the warp's own (a CTA per head and two barriers took 66 us for 2048 rows). grid (ceil((Hq + 2 Hkv) / 4), M), block 128.
// =========================================================================================
template <int HD>
__global__ void __launch_bounds__(128) attn_pack_kernel(AttnParams p) {
  constexpr int V = HD / 32;                         // dims of a lane: lane * V ..
  const int n = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, which = blockIdx.x * 4 + warp, d0 = lane * V;
  __shared__ __align__(16) float buf[4][HD];
  tl_mark(p.tl, 0);
  // what the producer kernel does not write (position, slot, norm weight, rotary entries) is fetched before waiting for it
  const int pos = p.row_pos[n], slot = p.row_slot[n], half = p.rope_dims / 2;
  const float* gamma = which < p.Hq ? p.q_norm : which < p.Hq + p.Hkv ? p.k_norm : nullptr;
  float ga[V];
  float2 cs[V];
#pragma unroll
  for (int i = 0; i < V; i++) {
    const int d = d0 + i;
    ga[i] = gamma != nullptr ? gamma[d] : 0.f;
    cs[i] = gamma != nullptr && d < p.rope_dims ? *reinterpret_cast<const float2*>(p.rope + ((size_t)(pos + p.rope_off) * half + (d < half ? d : d - half)) * 2) : make_float2(1.f, 0.f);
  }
  pdl_wait();
  pdl_launch();
  tl_mark(p.tl, 1);
  if (which >= p.Hq + 2 * p.Hkv) return;
  const float* pr = p.proj + (size_t)n * p.ldp + (which < p.Hq ? which * 2 * HD : p.Hq * 2 * HD + (which - p.Hq) * HD);   // q | gate per head, then k, then v
  float x[V];
#pragma unroll
  for (int i = 0; i < V; i += 4) *reinterpret_cast<float4*>(x + i) = *reinterpret_cast<const float4*>(pr + d0 + i);
  if (gamma != nullptr) {
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < V; i++) ss += x[i] * x[i];
    const float sc = 1.0f / sqrtf(warp_sum(ss) / (float)HD + p.eps);
#pragma unroll
    for (int i = 0; i < V; i++) { x[i] = x[i] * sc * ga[i]; buf[warp][d0 + i] = x[i]; }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < V; i++) {
      const int d = d0 + i;
      if (d < p.rope_dims) x[i] = d < half ? x[i] * cs[i].x - buf[warp][d + half] * cs[i].y : buf[warp][d - half] * cs[i].y + x[i] * cs[i].x;
    }
  }
  __half* dst;
  if (which < p.Hq) dst = p.q16 + ((size_t)n * p.Hq + which) * HD;
  else {
    const bool isk = which < p.Hq + p.Hkv;
    const int kh = isk ? which - p.Hq : which - p.Hq - p.Hkv;
    dst = (isk ? p.kcache : p.vcache) + (size_t)slot * p.slot_stride + ((size_t)pos * p.Hkv + kh) * HD;
  }
#pragma unroll
  for (int i = 0; i < V; i += 4) *reinterpret_cast<uint2*>(dst + d0 + i) = make_uint2(pack_half2(x[i], x[i + 1]), pack_half2(x[i + 2], x[i + 3]));
}
int launch_attn_pack(const AttnParams& p, bool pdl, cudaStream_t st) {
  const dim3 grid((p.Hq + 2 * p.Hkv + 3) / 4, p.M);
  if (p.hd == 256) return launch_k(attn_pack_kernel<256>, grid, dim3(128), 0, pdl, st, p);
  if (p.hd == 128) return launch_k(attn_pack_kernel<128>, grid, dim3(128), 0, pdl, st, p);
  set_error("attn_pack: head dim must be 128 or 256");
  return EINVAL_;
}

// =========================================================================================
// Split-KV decode attention (reference: llm/attn.go:190-217, 444-496;
// shaders/llm_attn_wmma.comp -DSPLITK, llm_attn_combine.comp). grid (nsplit, Hkv, M):
// a CTA of 4 warps covers `split_cells` cells of one KV head for the G query heads that
// share it.
// =========================================================================================
// -----------------------------------------------------------------------------------------
// Tensor-core form of the same split-KV decode attention. A warp walks 16 cells at a time:
//   S = Q K^T   as mma.m16n8k16 with the G query heads of the KV group on the M axis (the reference's
//               HROWS idea, shaders/llm_attn_wmma.comp:161-190) and 8 cells on N; a lane reads 16 bytes
//               of a K row (the dot product does not care which head dims share a k-slot, so the k-slots
//               are assigned to whatever 8 dims a lane's load covers, in Q and K alike);
//   P = exp(S * scale - m), rounded to fp16 (reference: shaders/llm_attn_wmma.comp:860);
//   O += P V    with the score tile's C registers reused as the A fragment, and V pairs of two cells
//               packed per dim with byte permutes (an in-register transpose; no shared-memory staging).
// Online softmax per warp, warps merged in shared memory, splits merged by attn_merge_kernel.
// -----------------------------------------------------------------------------------------

template <int HD, int G>
__global__ void __launch_bounds__(128) attn_mma_kernel(AttnParams p) {
  constexpr int KS = HD / 16;   // k-steps of the score mma
  constexpr int NB = HD / 64;   // 64-dim blocks of the value mma
  const int split = blockIdx.x, kvh = blockIdx.y, n = blockIdx.z;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  __shared__ float sm_m[4][G], sm_l[4][G], sm_f[4][G];
  __shared__ __align__(16) float sm_o[4][G][HD + 4];  // padded: the 16-byte stores of a quarter warp spread over the banks
  tl_mark(p.tl, 0);
  // The row's position and slot were written before this pass began. When every sequence has one row in the pass,
  // every cell but the newest was written by earlier passes too: both can be read before the producer kernel
  // (which writes the newest cell and the query) is known to be complete. A warp whose first block lies wholly
  // below the newest cell fetches its keys now.
  const int pos = p.row_pos[n], slot = p.row_slot[n];
  const int ncell = pos + 1;
  const int c0 = split * p.split_cells, c1 = min(ncell, c0 + p.split_cells);
  const float scale = 1.0f / sqrtf((float)HD);
  const size_t cell_stride = (size_t)p.Hkv * HD;
  const __half* kbase = p.kcache + (size_t)slot * p.slot_stride + (size_t)kvh * HD;
  const __half* vbase = p.vcache + (size_t)slot * p.slot_stride + (size_t)kvh * HD;
  uint4 ka4[KS / 2], kb4[KS / 2];
  auto fetch_k = [&](int cb) {
    const int ka = min(cb + g, c1 - 1), kb = min(cb + 8 + g, c1 - 1);  // clamped rows are masked below
    const __half* kra = kbase + (size_t)ka * cell_stride;
    const __half* krb = kbase + (size_t)kb * cell_stride;
#pragma unroll
    for (int j = 0; j < KS / 2; j++) {
      ka4[j] = ldg_stream(kra + 8 * (t + 4 * j));
      kb4[j] = ldg_stream(krb + 8 * (t + 4 * j));
    }
  };
  const int cb_first = c0 + warp * 16;
  const bool early = p.one_row_per_seq && cb_first + 16 <= pos;   // (then also cb_first < c1)
  if (early) fetch_k(cb_first);
  pdl_wait();
  pdl_launch();
  tl_mark(p.tl, 1);
  // query A fragments: head g of the group on row g; rows 8..15 stay zero
  uint32_t qa[KS][2];
#pragma unroll
  for (int j = 0; j < KS / 2; j++) {
    uint4 v = make_uint4(0, 0, 0, 0);
    if (g < G) v = *reinterpret_cast<const uint4*>(p.q16 + ((size_t)n * p.Hq + kvh * G + g) * HD + 8 * (t + 4 * j));
    qa[2 * j][0] = v.x; qa[2 * j][1] = v.y; qa[2 * j + 1][0] = v.z; qa[2 * j + 1][1] = v.w;
  }
  float o[HD / 8][2];
#pragma unroll
  for (int i = 0; i < HD / 8; i++) { o[i][0] = 0.f; o[i][1] = 0.f; }
  float m = -INFINITY, l = 0.f;
  for (int cb = c0 + warp * 16; cb < c1; cb += 64) {
    // ---- scores of 16 cells ----
    float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
    if (!(early && cb == cb_first)) fetch_k(cb);
    // the value rows do not depend on the scores: the first two 64-dim blocks are fetched while the score mma
    // runs, the rest as soon as the key registers are free, so every value load is in flight before the softmax
    const int cell_a = cb + 2 * t, cell_c = cb + 8 + 2 * t;
    const int va_c = min(cell_a, c1 - 1), vb_c = min(cell_a + 1, c1 - 1), vc_c = min(cell_c, c1 - 1), vd_c = min(cell_c + 1, c1 - 1);
    uint4 vv[NB][4];
    auto fetch_v = [&](int b) {
      const int doff = 8 * (g + 8 * b);
      vv[b][0] = ldg_stream(vbase + (size_t)va_c * cell_stride + doff); vv[b][1] = ldg_stream(vbase + (size_t)vb_c * cell_stride + doff);
      vv[b][2] = ldg_stream(vbase + (size_t)vc_c * cell_stride + doff); vv[b][3] = ldg_stream(vbase + (size_t)vd_c * cell_stride + doff);
    };
#pragma unroll
    for (int b = 0; b < NB && b < 2; b++) fetch_v(b);
#pragma unroll
    for (int j = 0; j < KS / 2; j++) {
      const uint32_t a0[4] = {qa[2 * j][0], 0u, qa[2 * j][1], 0u}, a1[4] = {qa[2 * j + 1][0], 0u, qa[2 * j + 1][1], 0u};
      mma16816(s0, a0, ka4[j].x, ka4[j].y);
      mma16816(s0, a1, ka4[j].z, ka4[j].w);
      mma16816(s1, a0, kb4[j].x, kb4[j].y);
      mma16816(s1, a1, kb4[j].z, kb4[j].w);
    }
#pragma unroll
    for (int b = 2; b < NB; b++) fetch_v(b);
    // row g, cells cb + 2t, +1 (tile 0) and cb + 8 + 2t, +1 (tile 1)
    float sc[4] = {s0[0] * scale, s0[1] * scale, s1[0] * scale, s1[1] * scale};
    const int cell[4] = {cb + 2 * t, cb + 2 * t + 1, cb + 8 + 2 * t, cb + 9 + 2 * t};
#pragma unroll
    for (int i = 0; i < 4; i++) if (cell[i] >= c1) sc[i] = -INFINITY;
    float mx = fmaxf(fmaxf(sc[0], sc[1]), fmaxf(sc[2], sc[3]));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float mn = fmaxf(m, mx);                       // finite: a block always holds at least one live cell
    const float corr = expf(m - mn);
    float pv[4];
#pragma unroll
    for (int i = 0; i < 4; i++) pv[i] = expf(sc[i] - mn);
    l = l * corr + ((pv[0] + pv[1]) + (pv[2] + pv[3]));
    m = mn;
    const uint32_t pa[4] = {pack_half2(pv[0], pv[1]), 0u, pack_half2(pv[2], pv[3]), 0u};
    // ---- O = O * corr + P V ----
#pragma unroll
    for (int b = 0; b < NB; b++) {
      const uint4 wa = vv[b][0], wb = vv[b][1], wc = vv[b][2], wd = vv[b][3];
      const uint32_t ra[4] = {wa.x, wa.y, wa.z, wa.w}, rb[4] = {wb.x, wb.y, wb.z, wb.w}, rc[4] = {wc.x, wc.y, wc.z, wc.w}, rd[4] = {wd.x, wd.y, wd.z, wd.w};
#pragma unroll
      for (int j = 0; j < 4; j++) {
        float acc_e[4] = {o[b * 8 + 2 * j][0] * corr, o[b * 8 + 2 * j][1] * corr, 0.f, 0.f};
        float acc_o[4] = {o[b * 8 + 2 * j + 1][0] * corr, o[b * 8 + 2 * j + 1][1] * corr, 0.f, 0.f};
        mma16816(acc_e, pa, __byte_perm(ra[j], rb[j], 0x5410), __byte_perm(rc[j], rd[j], 0x5410));
        mma16816(acc_o, pa, __byte_perm(ra[j], rb[j], 0x7632), __byte_perm(rc[j], rd[j], 0x7632));
        o[b * 8 + 2 * j][0] = acc_e[0]; o[b * 8 + 2 * j][1] = acc_e[1];
        o[b * 8 + 2 * j + 1][0] = acc_o[0]; o[b * 8 + 2 * j + 1][1] = acc_o[1];
      }
    }
  }
  // row sums live as per-lane partials over the four t lanes
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);
  // n-tile (b, i) column n' holds dim 8 * (n' + 8b) + i; this lane has columns 2t and 2t + 1 of head g
  if (g < G) {
    if (t == 0) { sm_m[warp][g] = m; sm_l[warp][g] = l; }
#pragma unroll
    for (int b = 0; b < NB; b++) {
      float* d0 = &sm_o[warp][g][8 * (2 * t + 8 * b)];
      float* d1 = &sm_o[warp][g][8 * (2 * t + 1 + 8 * b)];
      *reinterpret_cast<float4*>(d0) = make_float4(o[b * 8 + 0][0], o[b * 8 + 1][0], o[b * 8 + 2][0], o[b * 8 + 3][0]);
      *reinterpret_cast<float4*>(d0 + 4) = make_float4(o[b * 8 + 4][0], o[b * 8 + 5][0], o[b * 8 + 6][0], o[b * 8 + 7][0]);
      *reinterpret_cast<float4*>(d1) = make_float4(o[b * 8 + 0][1], o[b * 8 + 1][1], o[b * 8 + 2][1], o[b * 8 + 3][1]);
      *reinterpret_cast<float4*>(d1 + 4) = make_float4(o[b * 8 + 4][1], o[b * 8 + 5][1], o[b * 8 + 6][1], o[b * 8 + 7][1]);
    }
  }
  __syncthreads();
  // the warps' factors exp(m_w - m*) once per head, not once per output element
  if (tid < 4 * G) {
    const int w = tid / G, hh = tid - w * G;
    const float mm = fmaxf(fmaxf(sm_m[0][hh], sm_m[1][hh]), fmaxf(sm_m[2][hh], sm_m[3][hh]));
    sm_f[w][hh] = sm_m[w][hh] == -INFINITY ? 0.f : expf(sm_m[w][hh] - mm);
  }
  __syncthreads();
  const int PW = HD + 2;
  for (int i = tid; i < G * HD; i += 128) {
    const int hh = i / HD, d = i - hh * HD;
    float ov = 0.f;
#pragma unroll
    for (int w = 0; w < 4; w++) ov += sm_o[w][hh][d] * sm_f[w][hh];
    float* part = p.partial + (((size_t)n * p.Hq + kvh * G + hh) * p.nsplit + split) * PW;
    part[d] = ov;
    if (d == 0) {
      float lv = 0.f;
#pragma unroll
      for (int w = 0; w < 4; w++) lv += sm_l[w][hh] * sm_f[w][hh];
      part[HD] = fmaxf(fmaxf(sm_m[0][hh], sm_m[1][hh]), fmaxf(sm_m[2][hh], sm_m[3][hh]));
      part[HD + 1] = lv;
    }
  }
  tl_mark(p.tl, 4);
}

// -----------------------------------------------------------------------------------------
// Long-split form of the same kernel: eight warps, and the key and value rows reach shared memory by
// bulk copies (one per 16-cell tile row, completing on an mbarrier) instead of passing through registers.
// A warp owns a ring of three tile slots and keeps a whole block (16 keys + 16 values) in flight ahead of
// the block it computes on, so the bytes in flight per SM no longer depend on registers or on which phase
// the warps are in. Row pitches are padded (keys +64 bytes, values +16) so the 16-byte fragment reads of
// a quarter warp fall on distinct banks. Arithmetic and fragment layout are those of attn_mma_kernel.
// -----------------------------------------------------------------------------------------
template <int HD, int G>
__global__ void __launch_bounds__(256, 1) attn_ring_kernel(AttnParams p) {
  constexpr int KS = HD / 16, NB = HD / 64, NW = 8, NSLOT = 3;
  constexpr int KP = HD * 2 + 64, VP = HD * 2 + 16;  // row pitches in bytes
  constexpr int SLOT = 16 * KP;                      // a slot holds the key or the value rows of 16 cells
  extern __shared__ __align__(128) uint8_t ar_ring[];  // [NW][NSLOT][SLOT]; reused for the warps' outputs at the end
  __shared__ uint64_t bars[NW][NSLOT];
  __shared__ float sm_m[NW][G], sm_l[NW][G], sm_f[NW][G];
  const int split = blockIdx.x, kvh = blockIdx.y, n = blockIdx.z;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  tl_mark(p.tl, 0);
  if (lane == 0) {
#pragma unroll
    for (int s = 0; s < NSLOT; s++) mbar_init(&bars[warp][s], 1);
    mbar_fence_init();
  }
  __syncwarp();
  pdl_wait();
  pdl_launch();
  tl_mark(p.tl, 1);
  const int pos = p.row_pos[n], slot = p.row_slot[n];
  const int ncell = pos + 1;
  const int c0 = split * p.split_cells, c1 = min(ncell, c0 + p.split_cells);
  const float scale = 1.0f / sqrtf((float)HD);
  const size_t cell_stride = (size_t)p.Hkv * HD;
  const __half* kbase = p.kcache + (size_t)slot * p.slot_stride + (size_t)kvh * HD;
  const __half* vbase = p.vcache + (size_t)slot * p.slot_stride + (size_t)kvh * HD;
  uint8_t* ring = ar_ring + (size_t)warp * NSLOT * SLOT;
  const int cb0 = c0 + warp * 16;
  // tile j of this warp: keys (j even) or values (j odd) of block j / 2, in slot j % 3
  auto issue = [&](int j) {
    const int cb = cb0 + (NW * 16) * (j >> 1);
    if (cb >= c1) return;
    const bool isv = j & 1;
    uint64_t* bar = &bars[warp][j % NSLOT];
    uint8_t* dst = ring + (j % NSLOT) * SLOT;
    if (lane == 0) mbar_expect_tx(bar, 16 * HD * 2);
    __syncwarp();  // every lane is done with the slot's previous tile, and the byte count is posted
    if (lane < 16) {
      const int row = min(cb + lane, c1 - 1);  // clamped rows are masked below
      bulk_copy_g2s(dst + lane * (isv ? VP : KP), (isv ? vbase : kbase) + (size_t)row * cell_stride, HD * 2, bar);
    }
  };
  issue(0); issue(1); issue(2);
  uint32_t qa[KS][2];
#pragma unroll
  for (int j = 0; j < KS / 2; j++) {
    uint4 v = make_uint4(0, 0, 0, 0);
    if (g < G) v = *reinterpret_cast<const uint4*>(p.q16 + ((size_t)n * p.Hq + kvh * G + g) * HD + 8 * (t + 4 * j));
    qa[2 * j][0] = v.x; qa[2 * j][1] = v.y; qa[2 * j + 1][0] = v.z; qa[2 * j + 1][1] = v.w;
  }
  float o[HD / 8][2];
#pragma unroll
  for (int i = 0; i < HD / 8; i++) { o[i][0] = 0.f; o[i][1] = 0.f; }
  float m = -INFINITY, l = 0.f;
  bool lost = false;
  for (int i = 0, cb = cb0; cb < c1; i++, cb += NW * 16) {
    // ---- scores of 16 cells ----
    const int jk = 2 * i, jv = 2 * i + 1;
    if (!mbar_wait(&bars[warp][jk % NSLOT], (jk / NSLOT) & 1)) { lost = true; break; }
    const uint8_t* kt = ring + (jk % NSLOT) * SLOT + g * KP + t * 16;
    float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < KS / 2; j++) {
      const uint4 ka = lds128(kt + j * 64), kb = lds128(kt + 8 * KP + j * 64);
      const uint32_t a0[4] = {qa[2 * j][0], 0u, qa[2 * j][1], 0u}, a1[4] = {qa[2 * j + 1][0], 0u, qa[2 * j + 1][1], 0u};
      mma16816(s0, a0, ka.x, ka.y);
      mma16816(s0, a1, ka.z, ka.w);
      mma16816(s1, a0, kb.x, kb.y);
      mma16816(s1, a1, kb.z, kb.w);
    }
    issue(jk + 3);  // the next block's values, into the slot the keys just left
    // row g, cells cb + 2t, +1 (tile 0) and cb + 8 + 2t, +1 (tile 1)
    float sc[4] = {s0[0] * scale, s0[1] * scale, s1[0] * scale, s1[1] * scale};
    const int cell[4] = {cb + 2 * t, cb + 2 * t + 1, cb + 8 + 2 * t, cb + 9 + 2 * t};
#pragma unroll
    for (int u = 0; u < 4; u++) if (cell[u] >= c1) sc[u] = -INFINITY;
    float mx = fmaxf(fmaxf(sc[0], sc[1]), fmaxf(sc[2], sc[3]));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float mn = fmaxf(m, mx);                       // finite: a block always holds at least one live cell
    const float corr = expf(m - mn);
    float pv[4];
#pragma unroll
    for (int u = 0; u < 4; u++) pv[u] = expf(sc[u] - mn);
    l = l * corr + ((pv[0] + pv[1]) + (pv[2] + pv[3]));
    m = mn;
    const uint32_t pa[4] = {pack_half2(pv[0], pv[1]), 0u, pack_half2(pv[2], pv[3]), 0u};
    // ---- O = O * corr + P V ----
    if (!mbar_wait(&bars[warp][jv % NSLOT], (jv / NSLOT) & 1)) { lost = true; break; }
    const uint8_t* vt = ring + (jv % NSLOT) * SLOT + (2 * t) * VP + g * 16;
#pragma unroll
    for (int b = 0; b < NB; b++) {
      const uint4 wa = lds128(vt + b * 128), wb = lds128(vt + VP + b * 128), wc = lds128(vt + 8 * VP + b * 128), wd = lds128(vt + 9 * VP + b * 128);
      const uint32_t ra[4] = {wa.x, wa.y, wa.z, wa.w}, rb[4] = {wb.x, wb.y, wb.z, wb.w}, rc[4] = {wc.x, wc.y, wc.z, wc.w}, rd[4] = {wd.x, wd.y, wd.z, wd.w};
#pragma unroll
      for (int j = 0; j < 4; j++) {
        float acc_e[4] = {o[b * 8 + 2 * j][0] * corr, o[b * 8 + 2 * j][1] * corr, 0.f, 0.f};
        float acc_o[4] = {o[b * 8 + 2 * j + 1][0] * corr, o[b * 8 + 2 * j + 1][1] * corr, 0.f, 0.f};
        mma16816(acc_e, pa, __byte_perm(ra[j], rb[j], 0x5410), __byte_perm(rc[j], rd[j], 0x5410));
        mma16816(acc_o, pa, __byte_perm(ra[j], rb[j], 0x7632), __byte_perm(rc[j], rd[j], 0x7632));
        o[b * 8 + 2 * j][0] = acc_e[0]; o[b * 8 + 2 * j][1] = acc_e[1];
        o[b * 8 + 2 * j + 1][0] = acc_o[0]; o[b * 8 + 2 * j + 1][1] = acc_o[1];
      }
    }
    issue(jv + 3);  // the keys two blocks ahead, into the slot the values just left
  }
  if (lost && lane == 0) report_error(p.err);  // a copy never landed: report; the result is void
  // row sums live as per-lane partials over the four t lanes
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);
  __syncthreads();  // every warp has consumed what it issued: the ring becomes the warps' output buffer
  float (*sm_o)[G][HD + 4] = reinterpret_cast<float (*)[G][HD + 4]>(ar_ring);  // padded like attn_mma_kernel's
  if (g < G) {
    if (t == 0) { sm_m[warp][g] = m; sm_l[warp][g] = l; }
#pragma unroll
    for (int b = 0; b < NB; b++) {
      float* d0 = &sm_o[warp][g][8 * (2 * t + 8 * b)];
      float* d1 = &sm_o[warp][g][8 * (2 * t + 1 + 8 * b)];
      *reinterpret_cast<float4*>(d0) = make_float4(o[b * 8 + 0][0], o[b * 8 + 1][0], o[b * 8 + 2][0], o[b * 8 + 3][0]);
      *reinterpret_cast<float4*>(d0 + 4) = make_float4(o[b * 8 + 4][0], o[b * 8 + 5][0], o[b * 8 + 6][0], o[b * 8 + 7][0]);
      *reinterpret_cast<float4*>(d1) = make_float4(o[b * 8 + 0][1], o[b * 8 + 1][1], o[b * 8 + 2][1], o[b * 8 + 3][1]);
      *reinterpret_cast<float4*>(d1 + 4) = make_float4(o[b * 8 + 4][1], o[b * 8 + 5][1], o[b * 8 + 6][1], o[b * 8 + 7][1]);
    }
  }
  __syncthreads();
  // the warps' factors exp(m_w - m*) once per head, not once per output element
  if (tid < NW * G) {
    const int w = tid / G, hh = tid - w * G;
    float mm = -INFINITY;
#pragma unroll
    for (int v = 0; v < NW; v++) mm = fmaxf(mm, sm_m[v][hh]);
    sm_f[w][hh] = sm_m[w][hh] == -INFINITY ? 0.f : expf(sm_m[w][hh] - mm);
  }
  __syncthreads();
  const int PW = HD + 2;
  for (int i = tid; i < G * HD; i += 256) {
    const int hh = i / HD, d = i - hh * HD;
    float ov = 0.f;
#pragma unroll
    for (int w = 0; w < NW; w++) ov += sm_o[w][hh][d] * sm_f[w][hh];
    float* part = p.partial + (((size_t)n * p.Hq + kvh * G + hh) * p.nsplit + split) * PW;
    part[d] = ov;
    if (d == 0) {
      float mm = -INFINITY, lv = 0.f;
#pragma unroll
      for (int w = 0; w < NW; w++) { mm = fmaxf(mm, sm_m[w][hh]); lv += sm_l[w][hh] * sm_f[w][hh]; }
      part[HD] = mm; part[HD + 1] = lv;
    }
  }
  tl_mark(p.tl, 4);
}

// Merge of the splits: O = sum_s O_s * exp(m_s - m*), divide by the merged row sum, times
// sigmoid(gate), to fp16 (reference: shaders/llm_attn_combine.comp:43-102). grid (Hq, M), block hd.
__global__ void attn_merge_kernel(AttnParams p) {
  const int head = blockIdx.x, n = blockIdx.y, d = threadIdx.x, hd = p.hd, PW = hd + 2;
  extern __shared__ float mg_f[];  // [nsplit] factors exp(m_s - m*), then [nsplit] row sums
  __shared__ float mg_red[8];
  tl_mark(p.tl, 0);
  // the row's position and its gate (written by the in-projection, three kernels back) do not wait for the splits
  const int nlive = (p.row_pos[n] + 1 + p.split_cells - 1) / p.split_cells;
  const float gate = p.proj[(size_t)n * p.ldp + head * 2 * hd + hd + d];
  pdl_wait();
  pdl_launch();
  tl_mark(p.tl, 1);
  const float* part = p.partial + ((size_t)n * p.Hq + head) * p.nsplit * PW;
  // one round of loads for every split's maximum and row sum, shared through shared memory
  float mloc = -INFINITY;
  for (int sp = d; sp < nlive; sp += blockDim.x) {
    const float ms = __ldcg(part + (size_t)sp * PW + hd);
    mg_f[sp] = ms; mg_f[p.nsplit + sp] = __ldcg(part + (size_t)sp * PW + hd + 1);
    mloc = fmaxf(mloc, ms);
  }
  mloc = warp_max(mloc);
  if ((d & 31) == 0) mg_red[d >> 5] = mloc;
  __syncthreads();
  float mm = -INFINITY;
  for (int w = 0; w < (int)(blockDim.x + 31) / 32; w++) mm = fmaxf(mm, mg_red[w]);
  float ov = 0.f, lv = 0.f;
  int sp = 0;
  for (; sp + 16 <= nlive; sp += 16) {  // sixteen independent loads in flight, summed in split order
    float a[16];
#pragma unroll
    for (int u = 0; u < 16; u++) a[u] = __ldcg(part + (size_t)(sp + u) * PW + d);
#pragma unroll
    for (int u = 0; u < 16; u++) {
      const float ms = mg_f[sp + u];
      const float e = ms == -INFINITY ? 0.f : expf(ms - mm);
      ov += a[u] * e; lv += mg_f[p.nsplit + sp + u] * e;
    }
  }
  for (; sp < nlive; sp++) {
    const float ms = mg_f[sp];
    const float e = ms == -INFINITY ? 0.f : expf(ms - mm);
    ov += __ldcg(part + (size_t)sp * PW + d) * e; lv += mg_f[p.nsplit + sp] * e;
  }
  p.ctx16[(size_t)n * p.Hq * hd + head * hd + d] = __float2half_rn(ov / lv * sigmoid_acc(gate));
  tl_mark(p.tl, 6, true);
}

int launch_attn_decode(const AttnParams& p, bool pdl, cudaStream_t st) {
  const int G = p.Hq / p.Hkv;
  dim3 grid(p.nsplit, p.Hkv, p.M), block(128);
  int s;
  if (p.split_cells >= 256 && ((p.hd == 256 && G == 8) || (p.hd == 128 && G == 4))) {
    // long splits: eight warps fed by bulk copies
    const size_t smem = (size_t)8 * 3 * 16 * (p.hd * 2 + 64);
    B200_ONCE_PER_DEVICE(cudaFuncSetAttribute(attn_ring_kernel<256, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, 8 * 3 * 16 * (256 * 2 + 64)));
    B200_ONCE_PER_DEVICE(cudaFuncSetAttribute(attn_ring_kernel<128, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, 8 * 3 * 16 * (128 * 2 + 64)));
    return p.hd == 256 ? launch_k(attn_ring_kernel<256, 8>, grid, dim3(256), smem, pdl, st, p)
                       : launch_k(attn_ring_kernel<128, 4>, grid, dim3(256), smem, pdl, st, p);
  }
  if (p.hd == 256 && G == 8) s = launch_k(attn_mma_kernel<256, 8>, grid, block, 0, pdl, st, p);
  else if (p.hd == 128 && G == 4) s = launch_k(attn_mma_kernel<128, 4>, grid, block, 0, pdl, st, p);
  else if (p.hd == 128 && G == 8) s = launch_k(attn_mma_kernel<128, 8>, grid, block, 0, pdl, st, p);
  else if (p.hd == 256 && G == 4) s = launch_k(attn_mma_kernel<256, 4>, grid, block, 0, pdl, st, p);
  else { set_error("attn_decode: unsupported head_dim / group size (128 or 256 dims, 4 or 8 query heads per KV head)"); return EINVAL_; }
  return s;
}
int launch_attn_merge(const AttnParams& p, bool pdl, cudaStream_t st) {
  return launch_k(attn_merge_kernel, dim3(p.Hq, p.M), dim3(p.hd), (size_t)2 * p.nsplit * sizeof(float), pdl, st, p);
}

// =========================================================================================
// Greedy sampling: argmax with ties to the lowest id (reference: llm/sample.go:359-367)
// =========================================================================================
__global__ void __launch_bounds__(1024) argmax_kernel(const float* logits, int V, int32_t* out) {
  __shared__ float bv[32];
  __shared__ int bi[32];
  pdl_wait();
  pdl_launch();
  const float* lg = logits + (size_t)blockIdx.x * V;
  float v = -INFINITY; int idx = 0x7fffffff;
  if ((V & 3) == 0 && (reinterpret_cast<uintptr_t>(lg) & 15) == 0) {
    // four independent 16-byte loads in flight per thread; a thread's indices still rise, so `>` keeps the lowest
    const float4* lg4 = reinterpret_cast<const float4*>(lg);
    const int V4 = V >> 2;
    for (int i0 = threadIdx.x; i0 < V4; i0 += 4 * 1024) {
      float4 x[4];
#pragma unroll
      for (int u = 0; u < 4; u++) { const int i = i0 + u * 1024; x[u] = i < V4 ? __ldcg(lg4 + i) : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY); }
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int e = 4 * (i0 + u * 1024);
        if (x[u].x > v) { v = x[u].x; idx = e; }
        if (x[u].y > v) { v = x[u].y; idx = e + 1; }
        if (x[u].z > v) { v = x[u].z; idx = e + 2; }
        if (x[u].w > v) { v = x[u].w; idx = e + 3; }
      }
    }
  } else {
    for (int i = threadIdx.x; i < V; i += 1024) {
      float x = lg[i];
      if (x > v) { v = x; idx = i; }
    }
  }
  auto better = [](float a, int ai, float b, int bi2) { return a > b || (a == b && ai < bi2); };
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    float ov = __shfl_xor_sync(0xffffffffu, v, o);
    int oi = __shfl_xor_sync(0xffffffffu, idx, o);
    if (better(ov, oi, v, idx)) { v = ov; idx = oi; }
  }
  if ((threadIdx.x & 31) == 0) { bv[threadIdx.x >> 5] = v; bi[threadIdx.x >> 5] = idx; }
  __syncthreads();
  if (threadIdx.x < 32) {
    v = bv[threadIdx.x]; idx = bi[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      float ov = __shfl_xor_sync(0xffffffffu, v, o);
      int oi = __shfl_xor_sync(0xffffffffu, idx, o);
      if (better(ov, oi, v, idx)) { v = ov; idx = oi; }
    }
    if (threadIdx.x == 0) out[blockIdx.x] = idx == 0x7fffffff ? 0 : idx;
  }
}
int launch_argmax(const float* logits, int M, int V, int32_t* out, bool pdl, cudaStream_t st) {
  return launch_k(argmax_kernel, dim3(M), dim3(1024), 0, pdl, st, logits, V, out);
}

__global__ void advance_kernel(int32_t* ids, const int32_t* next, int* row_pos, SeqDesc* seqs, int M, int32_t* history, int* hist_len) {
  const int i = threadIdx.x;
  if (i < M) {
    ids[i] = next[i];
    row_pos[i] += 1;
    seqs[i].pos0 += 1;
    if (history != nullptr) history[(size_t)(*hist_len) * M + i] = next[i];
  }
  __syncthreads();
  if (i == 0 && hist_len != nullptr) *hist_len += 1;
}
int launch_advance(int32_t* ids, const int32_t* next, int* row_pos, SeqDesc* seqs, int M, int32_t* history, int* hist_len, cudaStream_t st) {
  if (M > 1024) { set_error("advance: too many rows"); return ECAPACITY; }
  advance_kernel<<<1, 1024, 0, st>>>(ids, next, row_pos, seqs, M, history, hist_len);
  B200_CUDA(cudaGetLastError());
  return OK;
}

// =========================================================================================
// Failure-detection probe: a bounded wait that nothing can satisfy. The barrier expects 16 bytes of
// copies and none is issued, so the wait runs out, the error word is set and the kernel returns; no
// copy is in flight and nothing faults. The host then sees the word exactly as it would after a real
// copy that never landed.
// =========================================================================================
__global__ void wait_timeout_probe_kernel(int* err, uint32_t limit) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_fence_init();
    mbar_expect_tx(&bar, 16);
    if (!mbar_wait(&bar, 0, limit)) report_error(err);
  }
}
int launch_wait_timeout_probe(int* err, cudaStream_t st) {
  wait_timeout_probe_kernel<<<1, 32, 0, st>>>(err, 1u << 16);
  B200_CUDA(cudaGetLastError());
  return OK;
}

}  // namespace b200
