// Expert projections of passes of at most eight rows (see moerow.cuh).
//
// What bounds them is latency and instruction issue, not DRAM: a row's eleven experts are 13 MB of gate and up weights (2 us of
// memory time) behind a selection that has to come first. So the selection is spread over a CTA (route_row_cta), each warp
// brings its own 16 x 256 weights as one TMA box as soon as the expert is known, and a second matrix's box flies meanwhile.
#include <algorithm>

#include "kernels.cuh"
#include "moerow.cuh"

namespace b200 {

namespace {

template <int TYPE> __host__ __device__ constexpr int mr_blk() { return TYPE == T_Q4_K ? 144 : 176; }
template <int TYPE> __host__ __device__ constexpr int mr_raw() { return 16 * mr_blk<TYPE>(); }

__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) { asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory"); }

int slices(int nb) { return nb >= 8 ? 8 : nb >= 4 ? 4 : nb >= 2 ? 2 : 1; }   // warps that share a tile's contraction

// A CTA serves one (row, slot): blockIdx.y. Its eight warps share out tiles of 16 gate + 16 up rows, `slices` warps to a tile, one
// super-block each at a time. grid (CTAs per slot, M * (used + 1)), three CTAs to an SM: a row's 352 CTAs of the benchmark's shape
// are resident at once; passes of more rows walk several tiles per CTA, each warp refilling its boxes as soon as it has read them.
template <int TYPE, int VPT>
__global__ void __launch_bounds__(256, 3) moe_gate_kernel(const __grid_constant__ MoeGateMaps maps, const MoeGateParams p, int wpt) {
  constexpr int BLK = mr_blk<TYPE>(), RAW = mr_raw<TYPE>();
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ __align__(8) uint64_t bars[8][2];
  __shared__ RouteSmem rs;
  __shared__ float red[2][2][8][16];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int K = p.K, nb = K / 256, used = p.route.used, slots1 = used + 1, row = blockIdx.y / slots1, slot = blockIdx.y - row * slots1;
  const int tpc = 8 / wpt, tiles = p.N / 16, lt = warp / wpt, ks = warp % wpt;
  uint8_t* raw = smem + warp * (2 * RAW);
  uint8_t* xs = smem + 8 * 2 * RAW;
  __half* sxs = reinterpret_cast<__half*>(xs + qg_xstride(K));
  tl_mark(p.tl, 0);
  if (lane < 2) mbar_init(&bars[warp][lane], 1);
  if (lane == 0) mbar_fence_init();
  __syncwarp();
  pdl_wait();   // logits and normalised rows come from the router kernel
  pdl_launch();
  float l[VPT];
#pragma unroll
  for (int i = 0; i < VPT; i++) l[i] = tid + 256 * i < p.route.nE ? __ldcg(p.route.logits + (size_t)row * p.route.nE + tid + 256 * i) : -INFINITY;
  copy_x_row(p.x + (int64_t)row * K, K, xs, sxs, sxs + K / 32, tid, 256);
  int ex = -1;
  if (slot < used) ex = route_row_cta<VPT>(p.route, row, l, blockIdx.x == 0 && slot == 0, slot, rs);
  else __syncthreads();
  tl_mark(p.tl, 1);
  // what this warp computes: blocks ks, ks + wpt, ... of tiles lt, lt + tpc * gridDim.x, ...
  const int bpt = nb > ks ? (nb - ks + wpt - 1) / wpt : 0;
  auto fetch = [&](int tile, int b) {
    if (elect_one()) {
      const int r = (ex >= 0 ? ex * p.N : 0) + tile * 16;
#pragma unroll
      for (int m = 0; m < 2; m++) {
        mbar_expect_tx(&bars[warp][m], RAW);
        const TMap* map = ex >= 0 ? (m ? &maps.up : &maps.gate) : (m ? &maps.up_sh : &maps.gate_sh);
        tma_box_2d(raw + m * RAW, map, (ks + b * wpt) * BLK, r, &bars[warp][m]);
      }
    }
  };
  const int step = tpc * gridDim.x, tile0 = blockIdx.x * tpc + lt;
  if (tile0 < tiles && bpt > 0) fetch(tile0, 0);
  // Once this CTA's first weights are here: its share of the slot's down weights, and of the next layer's dense weights, on their way
  // to L2. The chain of latencies leaves memory idle, and the kernels that need them next find them there.
  auto bring = [&]() {
    if (warp == 0 && lane == 0) {
      const int64_t share = p.down_bytes / gridDim.x & ~(int64_t)15;
      prefetch_l2((ex >= 0 ? p.down + ex * p.down_bytes : p.down_sh) + blockIdx.x * share, (uint32_t)share);
    }
    if (warp == 1 && lane < p.n_ahead) {
      const int64_t n = (int64_t)gridDim.x * gridDim.y, c = (int64_t)blockIdx.y * gridDim.x + blockIdx.x, units = p.ahead_bytes[lane] / 16;
      const int64_t from = units * c / n, to = units * (c + 1) / n;
      if (to > from) prefetch_l2(p.ahead[lane] + from * 16, (uint32_t)((to - from) * 16));
    }
  };
  tl_mark(p.tl, 2);
  int phase = 0, buf = 0;
  bool lost = false;
  const uint32_t ra = (uint32_t)__cvta_generic_to_shared(raw) + 2 * g * BLK;
  const __half* sp = sxs + (t & 1) * (K / 32) + 2 * (t >> 1);
  for (int base = blockIdx.x * tpc; base < tiles; base += step, buf ^= 1) {
    const int tile = base + lt;
    float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    if (tile < tiles && !lost) {
      for (int b = 0; b < bpt; b++, phase ^= 1) {
        const int blk = ks + b * wpt;
        const uint32_t s0 = *reinterpret_cast<const uint32_t*>(sp + 8 * blk), s1 = *reinterpret_cast<const uint32_t*>(sp + 8 * blk + 4);
#pragma unroll
        for (int m = 0; m < 2; m++) {
          if (warp_wait(&bars[warp][m], phase)) k45_accumulate<TYPE>(acc[m], ra + m * RAW, ra + m * RAW + BLK, xs + 576 * blk, s0, s1, t);
          else lost = true;
        }
        if (lost) {   // a copy never landed: report, the results are void; no more are asked for, and those in flight land before the CTA leaves
          if (lane == 0) report_error(p.err);
          for (int m = 0; m < 2; m++) mbar_wait(&bars[warp][m], phase, 1u << 18);
          break;
        }
        __syncwarp();
        const bool more = b + 1 < bpt;
        if (more || tile + step < tiles) { fence_proxy_async(); fetch(more ? tile : tile + step, more ? b + 1 : 0); }
      }
    }
    if (base == (int)blockIdx.x * tpc) bring();
    if (t == 0) {   // every column holds the one activation row
#pragma unroll
      for (int m = 0; m < 2; m++) *reinterpret_cast<float2*>(&red[buf][m][warp][2 * g]) = make_float2(acc[m][0], acc[m][2]);
    }
    __syncthreads();
    if (tid < tpc * 16) {
      const int l2 = tid >> 4, r = tid & 15;
      float v = 0.f, v2 = 0.f;
      for (int w = 0; w < wpt; w++) { v += red[buf][0][l2 * wpt + w][r]; v2 += red[buf][1][l2 * wpt + w][r]; }
      // SwiGLU rounded to fp16 (reference: shaders/llm_moe_gemv.comp:777-781)
      if (base + l2 < tiles) p.act[(size_t)blockIdx.y * p.N + (base + l2) * 16 + r] = __float2half_rn(v * sigmoid_acc(v) * v2);
    }
  }
  tl_mark(p.tl, 4);
}

// The MoE block's end (reference: llm/moe.go:347-357, 403-406; shaders/llm_moe_combine.comp:48-63), with the sum of squares of each
// tile's rows for the norm that follows. A CTA owns 16 rows of h of one row of the pass; its warps take (slot, super-block) units,
// each of which has a buffer of its own, so all copies are asked for at once; w_s times the units' sums are added in unit order.
// The form before (8 warps, staging for the whole CTA, three partial rows that every CTA of the next projection added up again)
// took 8 us and 3 us more of that projection's staging. grid (N / 16, rows).
constexpr int MD_MAXWARPS = 24;
constexpr int MD_X = 4 * 144 + 32;     // one super-block of a staged row, its eight sums as hi | lo

template <int TYPE>
__global__ void __launch_bounds__(MD_MAXWARPS * 32) moe_down_kernel(const __grid_constant__ MoeDownMaps maps, const MoeDownParams p) {
  constexpr int BLK = mr_blk<TYPE>(), RAW = mr_raw<TYPE>();
  extern __shared__ __align__(128) uint8_t smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3, warps = blockDim.x >> 5;
  const int nb = p.K / 256, slots1 = p.used + 1, units = slots1 * nb, tile = blockIdx.x, row = blockIdx.y, ld = ((units + 3) & ~3) + 4;
  uint8_t* xs0 = smem + units * RAW;
  float* yv = reinterpret_cast<float*>(xs0 + units * MD_X);   // [16][ld]
  uint64_t* bars = reinterpret_cast<uint64_t*>(yv + 16 * ld);
  tl_mark(p.tl, 0);
  for (int u = warp; u < units; u += warps)
    if (lane == 0) mbar_init(&bars[u], 1);
  if (lane == 0) mbar_fence_init();
  __syncwarp();
  pdl_wait();   // the selection and the activations come from the kernel before
  pdl_launch();
  tl_mark(p.tl, 1);
  const float hv = tid < 16 ? __ldcg(p.h + (size_t)row * p.N + tile * 16 + tid) : 0.f;
  for (int u = warp; u < units; u += warps) {
    const int s = u / nb, blk = u - s * nb;
    const int e = s < p.used ? __ldcg(p.topk + (size_t)row * p.used + s) : -1;
    if (elect_one()) {
      mbar_expect_tx(&bars[u], RAW);
      tma_box_2d(smem + u * RAW, e >= 0 ? &maps.w : &maps.ws, blk * BLK, (e >= 0 ? e * p.N : 0) + tile * 16, &bars[u]);
    }
  }
  for (int u = warp; u < units; u += warps) {
    const int s = u / nb, blk = u - s * nb;
    uint8_t* xs = xs0 + u * MD_X;
    __half* sx = reinterpret_cast<__half*>(xs + 4 * 144);
    const float w = __ldcg(p.topk_w + (size_t)row * slots1 + s);
    const uint4 v = __ldcg(reinterpret_cast<const uint4*>(p.act + ((size_t)row * slots1 + s) * p.K + blk * 256 + 8 * lane));
    const uint4 o = make_uint4(__byte_perm(v.x, v.y, 0x5410), __byte_perm(v.x, v.y, 0x7632), __byte_perm(v.z, v.w, 0x5410), __byte_perm(v.z, v.w, 0x7632));
    *reinterpret_cast<uint4*>(xs + 16 * lane + 16 * (lane >> 3)) = o;
    put_sx<4>(sum4_h2(o.x, o.y) + sum4_h2(o.z, o.w), sx, sx + 8, lane >> 2);
    __syncwarp();
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    if (warp_wait(&bars[u], 0)) {
      const uint32_t ra = (uint32_t)__cvta_generic_to_shared(smem + u * RAW) + 2 * g * BLK;
      const __half* sp = sx + ((t & 1) ? 8 : 0) + 2 * (t >> 1);
      k45_accumulate<TYPE>(acc, ra, ra + BLK, xs, *reinterpret_cast<const uint32_t*>(sp), *reinterpret_cast<const uint32_t*>(sp + 4), t);
    } else {   // a copy never landed: report, the results are void; leave once it has, or its limit has run out again
      if (lane == 0) report_error(p.err);
      mbar_wait(&bars[u], 0, 1u << 18);
    }
    if (t == 0) { yv[2 * g * ld + u] = w * acc[0]; yv[(2 * g + 1) * ld + u] = w * acc[2]; }   // every column holds the one activation row
  }
  tl_mark(p.tl, 3);
  __syncthreads();
  if (tid < 16) {
    float acc = 0.f;
#pragma unroll 8
    for (int u = 0; u < units; u++) acc += yv[tid * ld + u];
    const float r = hv + acc;
    p.h[(size_t)row * p.N + tile * 16 + tid] = r;
    float sq = r * r;
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) sq += __shfl_xor_sync(0xffffu, sq, o);
    if (tid == 0) p.ss_out[(size_t)row * SS_LD + tile] = sq;
  }
  tl_mark(p.tl, 4);
}

template <class Kernel, class Params, class... Extra>
int launch(Kernel kernel, dim3 grid, int threads, size_t smem, bool pdl, cudaStream_t st, const Params& p, Extra... extra) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = dim3(threads); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = pdl ? 1 : 0;
  B200_CUDA(cudaLaunchKernelEx(&cfg, kernel, p, extra...));
  return OK;
}

size_t gate_smem(uint32_t type, int K) { return (size_t)16 * 16 * (type == T_Q4_K ? 144 : 176) + qg_xstride(K) + (size_t)K / 32 * 2 * sizeof(__half); }
size_t down_smem(uint32_t type, int K, int used) {
  const size_t units = (size_t)(used + 1) * (K / 256);
  return units * (16 * (type == T_Q4_K ? 144 : 176) + MD_X + sizeof(uint64_t)) + 16 * (((units + 3) & ~(size_t)3) + 4) * sizeof(float);
}

template <int TYPE, int VPT>
int launch_gate(const MoeGateParams& p, const MoeGateMaps& maps, bool pdl, cudaStream_t st) {
  auto kernel = moe_gate_kernel<TYPE, VPT>;
  const size_t smem = gate_smem(TYPE, p.K);
  B200_ONCE_PER_DEVICE(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
  const int sms = sm_count_current();
  if (sms <= 0) return ECUDA;
  const int wpt = slices(p.K / 256), tpc = 8 / wpt, groups = (p.N / 16 + tpc - 1) / tpc, ny = p.M * (p.route.used + 1);
  // as many CTAs per slot as are resident together (three to an SM), each walking the same number of tile groups
  const int cap = std::max(1, 3 * sms / ny), rounds = (groups + cap - 1) / cap, gx = (groups + rounds - 1) / rounds;
  return launch(kernel, dim3(gx, ny), 256, smem, pdl, st, maps, p, wpt);
}
template <int TYPE>
int launch_down(const MoeDownParams& p, const MoeDownMaps& maps, int rows, bool pdl, cudaStream_t st) {
  auto kernel = moe_down_kernel<TYPE>;
  B200_ONCE_PER_DEVICE(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
  // one row: a warp per unit where they fit; more rows: half as many warps, so that two CTAs share an SM
  const int units = (p.used + 1) * (p.K / 256), most = rows == 1 ? MD_MAXWARPS : MD_MAXWARPS / 2;
  const int rounds = (units + most - 1) / most, warps = (units + rounds - 1) / rounds;
  return launch(kernel, dim3(p.N / 16, rows), warps * 32, down_smem(TYPE, p.K, p.used), pdl, st, maps, p);
}

}  // namespace

bool moe_rows_fit(uint32_t gate_type, uint32_t down_type, int H, int ffn, int n_expert, int used) {
  auto k45 = [](uint32_t t) { return t == T_Q4_K || t == T_Q5_K; };
  return k45(gate_type) && k45(down_type) && H % 256 == 0 && ffn % 256 == 0 && H / 16 <= SS_LD && n_expert <= 1024 && used < 32 && used <= n_expert &&
         gate_smem(gate_type, H) <= 72 * 1024 && down_smem(down_type, ffn, used) <= 200 * 1024;
}
int launch_moe_gate(uint32_t type, const MoeGateParams& p, const MoeGateMaps& maps, bool pdl, cudaStream_t st) {
  if (p.K % 256 != 0 || p.N % 16 != 0 || p.route.nE > 1024 || p.M < 1 || p.M > QG_FUSED_ROWS || gate_smem(type, p.K) > 72 * 1024) { set_error("moe_gate: shape outside kernel limits"); return EINVAL_; }
  const bool few = p.route.nE <= 512;
  if (type == T_Q4_K) return few ? launch_gate<T_Q4_K, 2>(p, maps, pdl, st) : launch_gate<T_Q4_K, 4>(p, maps, pdl, st);
  if (type == T_Q5_K) return few ? launch_gate<T_Q5_K, 2>(p, maps, pdl, st) : launch_gate<T_Q5_K, 4>(p, maps, pdl, st);
  set_error("moe_gate: weight type has no kernel (Q4_K, Q5_K)");
  return EINVAL_;
}
int launch_moe_down(uint32_t type, const MoeDownParams& p, const MoeDownMaps& maps, int rows, bool pdl, cudaStream_t st) {
  if (p.K % 256 != 0 || p.N % 16 != 0 || p.N / 16 > SS_LD || p.used >= 32 || rows < 1 || rows > QG_FUSED_ROWS || down_smem(type, p.K, p.used) > 200 * 1024) { set_error("moe_down: shape outside kernel limits"); return EINVAL_; }
  if (type == T_Q4_K) return launch_down<T_Q4_K>(p, maps, rows, pdl, st);
  if (type == T_Q5_K) return launch_down<T_Q5_K>(p, maps, rows, pdl, st);
  set_error("moe_down: weight type has no kernel (Q4_K, Q5_K)");
  return EINVAL_;
}

}  // namespace b200
