// Causal attention of a many-row pass of one sequence: query tiles x key tiles with an online softmax (the reference's flash form:
// shaders/llm_attn_wmma.comp:102-117 QT/BM query tiles, :161-190 HROWS), both products on tcgen05.
//
// The 128 rows of an accumulator are 128 / G query rows times the G query heads of one KV head. Tensor memory holds O (HD columns) and
// two score tiles of 128 cells; a score tile becomes, in place, the fp16 probabilities that are the A operand of the second product. Six warps:
//   warp 0     TMA: the query tile once, then keys and values in pieces of 32 KB through a ring of four;
//   warp 1     one thread issues S = Q K^T of tile k + 1, then O += P V of tile k, so the tensor core works while tile k's softmax runs;
//   warps 2-5  a thread per row: maximum, exponentials, row sum, and the result.
// O is rescaled whenever a row's maximum has grown, after the tile's exponentials, while the tensor core forms the next scores: the largest
// probability is then exactly 1, which fp16 carries without error, and the row sum is of the probabilities as fp16 carries them, so that
// part of what rounds them drops out of the quotient. Against f64 with peaked scores 2.17e-4 (fp16 of the exact result: 2.08e-4); with a
// maximum kept until it had grown by 2^8, and the unrounded sum, 2.71e-4 (and 117 us).
// What bounds it: a step of 128 rows x 128 cells is 2500 cycles of tcgen05.mma and 128 KB of keys and values out of L2, about as long
// (the KV heads' tiles are read once per query tile). With mma.sync (16 rows a warp, keys and values through shared memory for every
// warp) 2048 rows over 2 to 4 thousand cells took 752 us, this takes 128; 46 us are the tensor core's floor.
#include <algorithm>

#include "attn_tc.cuh"
#include "tcgen.cuh"

namespace b200 {

namespace {

using namespace tc;

constexpr int AT_THREADS = 192, AT_PIECE = 32768, AT_NP = 4, AT_CELLS = 128;

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t half2_of(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

template <int HD, int G>
__global__ void __launch_bounds__(AT_THREADS, 1) attn_tc_kernel(const __grid_constant__ AttnTcMaps maps, const AttnParams p) {
  constexpr int QR = 128 / G, KPC = HD / 128;                 // query rows of a tile, key pieces (128 cells x 128 dims) of a tile
  constexpr int VC = AT_PIECE / (2 * HD), VPC = AT_CELLS / VC;   // cells of a value piece (all dims), value pieces of a tile
  constexpr int TO = 0, TS = 256;                             // tensor memory columns: O, score tiles
  extern __shared__ uint8_t at_smem[];
  uint8_t* q_s = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(at_smem) + 1023) & ~(uintptr_t)1023);
  uint8_t* pc = q_s + 128 * HD * 2;
  __shared__ __align__(8) uint64_t q_full, full[AT_NP], empty[AT_NP], s_full[2], p_full[2], pv_done;
  __shared__ uint32_t tmem_sm;
  __shared__ volatile int failed;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tile = (int)gridDim.x - 1 - (int)blockIdx.x;      // long rows first
  const int kvh = blockIdx.y, n0 = tile * QR;
  if (tid == 0) {
    mbar_init(&q_full, 1); mbar_init(&pv_done, 1);
    for (int i = 0; i < AT_NP; i++) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    for (int i = 0; i < 2; i++) { mbar_init(&s_full[i], 1); mbar_init(&p_full[i], 4); }
    mbar_fence_init();
    failed = 0;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_addr(&tmem_sm)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tm = tmem_sm;
  pdl_wait();
  pdl_launch();
  const int slot = p.row_slot[n0], pos0 = p.row_pos[n0];      // rows of one sequence at consecutive positions
  const int rows = min(QR, p.M - n0), ncell = pos0 + rows;    // cells the tile's last row sees
  const int c_lo = (int)blockIdx.z * p.split_cells, c_hi = min(ncell, c_lo + p.split_cells);   // this part of them
  const int nt = c_hi > c_lo ? (c_hi - c_lo + AT_CELLS - 1) / AT_CELLS : 0;
  auto give_up = [&]() { report_error(p.err); failed = 1; };
  auto stopped = [&]() { return __any_sync(0xffffffffu, failed); };
  // pieces in the order they are needed: K(0), then for every tile k: K(k + 1), V(k)
  auto v_piece = [&](int k) { return KPC * (min(k + 1, nt - 1) + 1) + VPC * k; };

  if (warp == 0) {
    if (nt > 0 && elect_one()) {
      mbar_expect_tx(&q_full, 128 * HD * 2);
      for (int j = 0; j < HD / 64; j++) tma_box3(q_s + j * 16384, &maps.q, 64 * j, kvh * G, n0, &q_full);
    }
    __syncwarp();
    uint32_t it = 0;
    const int base = slot * p.n_kv + c_lo;
    auto next = [&](auto boxes) {
      const int s = it % AT_NP;
      if (!warp_wait(&empty[s], ((it / AT_NP) & 1) ^ 1)) { give_up(); return false; }
      if (elect_one()) {
        mbar_expect_tx(&full[s], AT_PIECE);
        boxes(pc + s * AT_PIECE, &full[s]);
      }
      __syncwarp();
      it++;
      return true;
    };
    auto keys = [&](int k) {
      for (int h = 0; h < KPC; h++)
        if (!next([&](uint8_t* d, uint64_t* bar) { for (int j = 0; j < 2; j++) tma_box3(d + j * 16384, &maps.k, 128 * h + 64 * j, kvh, base + k * AT_CELLS, bar); })) return false;
      return true;
    };
    bool ok = nt == 0 || keys(0);
    for (int k = 0; k < nt && ok && !stopped(); k++) {
      if (k + 1 < nt) ok = keys(k + 1);
      for (int h = 0; h < VPC && ok; h++)
        ok = next([&](uint8_t* d, uint64_t* bar) { for (int j = 0; j < HD / 64; j++) tma_box3(d + j * (VC * 128), &maps.v, 64 * j, kvh, base + k * AT_CELLS + h * VC, bar); });
    }
    if (failed) {                                             // leave only once the copies in flight have landed
      if (nt > 0) mbar_wait(&q_full, 0);
      for (uint32_t i = it > (uint32_t)AT_NP ? it - AT_NP : 0; i < it; i++) mbar_wait(&full[i % AT_NP], (i / AT_NP) & 1);
    }
  } else if (warp == 1) {
    uint32_t it = 0;
    bool ok = nt == 0 || warp_wait(&q_full, 0);
    if (!ok) give_up();
    const uint32_t q_a = smem_addr(q_s), p_a = smem_addr(pc);
    auto scores = [&](int k) {
      for (int h = 0; h < KPC; h++, it++) {
        const int s = it % AT_NP;
        if (!warp_wait(&full[s], (it / AT_NP) & 1)) { give_up(); return false; }
        fence_after();
        if (elect_one()) {
#pragma unroll
          for (int i = 0; i < 8; i++)
            mma_ss(tm + TS + (k & 1) * AT_CELLS, desc_sw128(q_a + (2 * h + (i >> 2)) * 16384) + 2 * (i & 3), desc_sw128(p_a + s * AT_PIECE + (i >> 2) * 16384) + 2 * (i & 3), idesc_n(AT_CELLS),
                   (h | i) != 0);
          commit(&empty[s]);
          if (h == KPC - 1) commit(&s_full[k & 1]);
        }
        __syncwarp();
      }
      return true;
    };
    ok = ok && (nt == 0 || scores(0));
    for (int k = 0; k < nt && ok && !stopped(); k++) {
      if (k + 1 < nt) ok = scores(k + 1);
      if (!ok || !(ok = warp_wait(&p_full[k & 1], (k >> 1) & 1))) { give_up(); break; }
      for (int h = 0; h < VPC; h++, it++) {
        const int s = it % AT_NP;
        if (!(ok = warp_wait(&full[s], (it / AT_NP) & 1))) { give_up(); break; }
        fence_after();
        if (elect_one()) {
#pragma unroll
          for (int i = 0; i < VC / 16; i++)
            mma_ts(tm + TO, tm + TS + (k & 1) * AT_CELLS + h * (VC / 2) + 8 * i, desc_mn_sw128(p_a + s * AT_PIECE + i * 2048, VC * 128), idesc_n(HD) | IDESC_B_MN, (k | h | i) != 0);
          commit(&empty[s]);
          if (h == VPC - 1) commit(&pv_done);
        }
        __syncwarp();
      }
    }
  } else {
    const int q = warp & 3, r = q * 32 + lane, n = n0 + r / G, head = kvh * G + r % G;
    const uint32_t lanes = tm + ((uint32_t)(q * 32) << 16);
    const int pos = pos0 + min(r / G, rows - 1);
    const float scale = 1.0f / sqrtf((float)HD), c = scale * 1.4426950408889634f;
    float m = -INFINITY, l = 0.f;
    bool ok = true;
    for (int k = 0; k < nt && ok; k++) {
      if (!(ok = warp_wait(&s_full[k & 1], (k >> 1) & 1)) || stopped()) { ok = false; give_up(); break; }
      fence_after();
      float s[4][32];
#pragma unroll
      for (int i = 0; i < 4; i++) tmem_ld32(lanes + TS + (k & 1) * AT_CELLS + 32 * i, s[i]);
      tmem_ld_wait();
      const int cb = c_lo + k * AT_CELLS;
      if (cb + AT_CELLS - 1 > pos0) {                         // cells past a row's own position
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
          for (int j = 0; j < 32; j++) if (cb + 32 * i + j > pos || cb + 32 * i + j >= c_hi) s[i][j] = -INFINITY;
      }
      float mx[4] = {s[0][0], s[1][0], s[2][0], s[3][0]};
#pragma unroll
      for (int j = 1; j < 32; j++)
#pragma unroll
        for (int i = 0; i < 4; i++) mx[i] = fmaxf(mx[i], s[i][j]);
      const float mn = fmaxf(m, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])));
      const bool grown = mn > m;
      const float f = grown ? ex2((m - mn) * c) : 1.f;
      m = mn;
      const float mc = m == -INFINITY ? 0.f : m * c;
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int hf = 0; hf < 2; hf++) {
        uint32_t w[32];
#pragma unroll
        for (int j = 0; j < 32; j++) {
          const float a = ex2(fmaf(s[2 * hf + (j >> 4)][(2 * j) & 31], c, -mc)), b = ex2(fmaf(s[2 * hf + (j >> 4)][((2 * j) & 31) + 1], c, -mc));
          w[j] = half2_of(a, b);
          const float2 r = __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
          sum[j & 3] += r.x + r.y;
        }
        tmem_st32(lanes + TS + (k & 1) * AT_CELLS + 32 * hf, w);
      }
      l = fmaf(l, f, (sum[0] + sum[1]) + (sum[2] + sum[3]));
      // The tile before is in O, and every warp has seen so: a wait by parity would take the product before last for the last one, at the
      // end and for the pieces below. (Free: the tensor core has the scores of the next tile to form after it.)
      if (k > 0 && !(ok = warp_wait(&pv_done, (k - 1) & 1))) { give_up(); break; }
      if (k > 0 && __any_sync(0xffffffffu, grown)) {
        fence_after();
#pragma unroll 1
        for (int j = 0; j < HD; j += 32) {
          float o[32];
          tmem_ld32(lanes + TO + j, o);
          tmem_ld_wait();
          uint32_t w[32];
#pragma unroll
          for (int i = 0; i < 32; i++) w[i] = __float_as_uint(o[i] * f);
          tmem_st32(lanes + TO + j, w);
        }
      }
      if (cb + AT_CELLS > c_hi) {
        // value rows past the end hold whatever the cache held: weight zero is not enough against an infinity
        const int live = c_hi - cb;
        for (int h = 0; h < VPC && ok; h++) {
          const uint32_t v = v_piece(k) + h;
          if (!(ok = warp_wait(&full[v % AT_NP], (v / AT_NP) & 1))) { give_up(); break; }
          uint8_t* d = pc + (v % AT_NP) * AT_PIECE;
          for (int i = tid - 64; i < AT_PIECE / 16; i += 128)
            if (h * VC + ((i >> 3) % VC) >= live) *reinterpret_cast<uint4*>(d + i * 16) = make_uint4(0, 0, 0, 0);
        }
        fence_proxy_async();
      }
      tmem_st_wait();
      fence_before();
      __syncwarp();
      if (lane == 0) arrive(&p_full[k & 1]);
    }
    if (ok && nt > 0 && warp_wait(&pv_done, (nt - 1) & 1)) {
      fence_after();
      const bool whole = p.nsplit == 0, live = r / G < rows;
      const float* gate = p.proj + (size_t)n * p.ldp + (size_t)head * 2 * HD + HD;
      __half* dst = p.ctx16 + (size_t)n * p.Hq * HD + (size_t)head * HD;
      float* part = p.partial + (((size_t)n * p.Hq + head) * p.nsplit + blockIdx.z) * (HD + 2);
      // The gates are a row's own 128 bytes per 32 columns: asked for ahead of their use. O / l * sigmoid(gate)
      // (reference: shaders/llm_attn_combine.comp:100-102) is one quotient, O / (l (1 + exp(-gate))).
      float4 gn[8];
      auto ask = [&](int j) {
#pragma unroll
        for (int i = 0; i < 8; i++) gn[i] = *reinterpret_cast<const float4*>(gate + j + 4 * i);
      };
      if (whole && live) ask(0);
#pragma unroll 1
      for (int j = 0; j < HD; j += 32) {
        float o[32];
        tmem_ld32(lanes + TO + j, o);
        tmem_ld_wait();
        if (!live) continue;
        if (whole) {
          float g[32];
#pragma unroll
          for (int i = 0; i < 8; i++) { g[4 * i] = gn[i].x; g[4 * i + 1] = gn[i].y; g[4 * i + 2] = gn[i].z; g[4 * i + 3] = gn[i].w; }
          if (j + 32 < HD) ask(j + 32);
#pragma unroll
          for (int i = 0; i < 32; i++) o[i] = o[i] / fmaf(l, expf(-g[i]), l);
#pragma unroll
          for (int i = 0; i < 32; i += 8)
            *reinterpret_cast<uint4*>(dst + j + i) = make_uint4(half2_of(o[i], o[i + 1]), half2_of(o[i + 2], o[i + 3]), half2_of(o[i + 4], o[i + 5]), half2_of(o[i + 6], o[i + 7]));
        } else {
#pragma unroll
          for (int i = 0; i < 32; i += 2) *reinterpret_cast<float2*>(part + j + i) = make_float2(o[i], o[i + 1]);
        }
      }
      if (live && !whole) { part[HD] = m * scale; part[HD + 1] = l; }
    } else if (nt > 0) {
      give_up();
    }
  }
  fence_before();
  __syncthreads();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tm) : "memory");
}

template <int HD, int G>
int launch_t(const AttnParams& p, const AttnTcMaps& maps, int nz, bool pdl, cudaStream_t st) {
  auto kernel = attn_tc_kernel<HD, G>;
  constexpr int smem = 128 * HD * 2 + AT_NP * AT_PIECE + 1024;
  B200_ONCE_PER_DEVICE(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((p.M + 128 / G - 1) / (128 / G), p.Hkv, nz); cfg.blockDim = dim3(AT_THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = pdl ? 1 : 0;
  B200_CUDA(cudaLaunchKernelEx(&cfg, kernel, maps, p));
  return OK;
}

}  // namespace

bool attn_tc_shape(int Hq, int Hkv, int hd) {
  const int G = Hkv > 0 ? Hq / Hkv : 0;
  return (G == 8 && hd == 256) || (G == 4 && hd == 128);
}

int make_attn_maps(const __half* q16, int64_t rows, int Hq, const __half* kcache, const __half* vcache, int64_t cells, int Hkv, int hd, AttnTcMaps* out) {
  const int G = Hq / Hkv;
  const int64_t qd[3] = {hd, Hq, rows}, qs[2] = {hd * 2, (int64_t)Hq * hd * 2}, cd[3] = {hd, Hkv, cells}, cs[2] = {hd * 2, (int64_t)Hkv * hd * 2};
  const int qb[3] = {64, G, 128 / G}, kb[3] = {64, 1, AT_CELLS}, vb[3] = {64, 1, AT_PIECE / (2 * hd)};
  B200_TRY(encode_nd(CU_TENSOR_MAP_DATA_TYPE_FLOAT16, q16, 3, qd, qs, qb, CU_TENSOR_MAP_SWIZZLE_128B, &out->q));
  B200_TRY(encode_nd(CU_TENSOR_MAP_DATA_TYPE_FLOAT16, kcache, 3, cd, cs, kb, CU_TENSOR_MAP_SWIZZLE_128B, &out->k));
  return encode_nd(CU_TENSOR_MAP_DATA_TYPE_FLOAT16, vcache, 3, cd, cs, vb, CU_TENSOR_MAP_SWIZZLE_128B, &out->v);
}

int launch_attn_tc(AttnParams& p, const AttnTcMaps& maps, int last_pos, int64_t partial_floats, bool pdl, cudaStream_t st) {
  if (!attn_tc_fits(p)) { set_error("attn_tc: 8 query heads per KV head of 256 dims, or 4 of 128"); return EINVAL_; }
  const int QR = 128 * p.Hkv / p.Hq, ctas = (p.M + QR - 1) / QR * p.Hkv, tiles = (last_pos + AT_CELLS) / AT_CELLS;
  // cut the keys while the query tiles leave SMs idle, into parts of four tiles at least (a part costs its write and the merge)
  const int64_t room = partial_floats / ((int64_t)p.M * p.Hq * (p.hd + 2));
  int nz = (int)std::min<int64_t>(std::min(sm_count_current() / std::max(ctas, 1), tiles / 4), room);
  if (nz < 2) nz = 1;
  p.split_cells = (tiles + nz - 1) / nz * AT_CELLS;
  nz = (tiles * AT_CELLS + p.split_cells - 1) / p.split_cells;
  p.nsplit = nz > 1 ? nz : 0;
  return p.hd == 256 ? launch_t<256, 8>(p, maps, nz, pdl, st) : launch_t<128, 4>(p, maps, nz, pdl, st);
}

}  // namespace b200
