// Exact K-quant projections on tcgen05 (see tgemm.cuh).
//
// A CTA of fourteen warps walks units of 128 weight rows x at most NMAX activation rows. Per super-block of 256 elements:
//   warp 0        one TMA box of the 128 rows' quant blocks and five of the activation rows' 256 elements and sums into a ring
//                 of stages;
//   warps 2..9    a thread per weight row and half block: quants -> fp16 integers sc * (q - centre) in registers -> tensor memory
//                 (tcgen05.st), where the A operand is read from: no trip through shared memory, no swizzle;
//   warp 1        one thread issues sixteen tcgen05.mma (M 128, N the columns in use, K 16) into a fresh accumulator, and
//                 one more into it and one for the min term over the sub-block sums;
//   warps 10..13  a thread per weight row: reads both accumulators back and adds d * C - dmin * Cm to its f32 registers, so
//                 the block scales are applied in f32 as the column-tiled kernel applies them; epilogue at the unit's end.
// The roles meet only through mbarriers (every wait bounded), so loads, dequantisation, tensor core and drain of different
// blocks overlap, across units too.
#include <algorithm>
#include <cstring>
#include <string>

#include "tcgen.cuh"

namespace b200 {

namespace {

constexpr int TG_THREADS = 448, TG_TILE = 128;
constexpr int TG_DQ0 = 2, TG_DR0 = 10;               // first dequantising and first draining warp
constexpr int TG_ASLOT = 64, TG_NA = 3;              // tensor-memory columns of half a block's A operand, ring of three
constexpr int TG_MIN = TG_ASLOT * TG_NA;             // min operands: 8 columns, ring of two
constexpr int TG_CEN = TG_MIN + 16;                  // scales times the centre: the same
constexpr int TG_ACC = 256;                          // accumulators: C and Cm of NMAX columns each, ring of two
constexpr int TG_ND = 8;                             // block scales on their way from the dequantising to the draining warps

template <int TYPE> __host__ __device__ constexpr int tg_blk() { return TYPE == T_Q4_K ? 144 : 176; }
template <int TYPE, int NMAX> __host__ __device__ constexpr int tg_stage() { return NMAX * 640 + TG_TILE * tg_blk<TYPE>(); }
template <int TYPE, int NMAX> __host__ __device__ constexpr int tg_stages() { return (NMAX == 64 ? 190 : 200) * 1024 / tg_stage<TYPE, NMAX>(); }

using namespace tc;

__device__ __forceinline__ uint32_t h2c(float v) {
  __half2 h = __float2half2_rn(v);
  return *reinterpret_cast<uint32_t*>(&h);
}

// Quants enter less their centre, and the centre comes back as one more product over the sub-block sums: the tensor core's running sums
// round towards zero, in proportion to their size, and about the centre they are a third of the size (relative error of a
// projection 5.3e-7 to 7.7e-7 without, 3.0e-7 to 3.5e-7 with; mma.sync with whole quants had 3.1e-7 to 4.1e-7). With its bits at the top of a byte, 0x54 above them makes a Q4_K quant the half
// 64 + q and 0x58 a Q5_K one 128 + q; both products below are exact.
template <int TYPE> __device__ __forceinline__ constexpr float tg_centre() { return TYPE == T_Q4_K ? 8.f : 16.f; }
__device__ __forceinline__ uint32_t bytes_to_h2(uint32_t four, uint32_t sel) { return hadd2_u(__byte_perm(four, 0x64646464u, sel), h2c(-1024.f)); }   // two bytes picked by sel

// Group `grp` (64 elements: low nibbles, then high nibbles of 32 bytes) of a block as 32 columns of tensor memory.
template <int TYPE>
__device__ __forceinline__ void dequant_group(const uint4& qa, const uint4& qb, const uint32_t (&fifth)[8], int grp, uint32_t scales, int byte, uint32_t (&out)[32]) {
  constexpr uint32_t MAGIC = TYPE == T_Q4_K ? 0x54545454u : 0x58585858u;
  constexpr float BASE = TYPE == T_Q4_K ? 64.f : 128.f;
  const uint32_t w[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
  const uint32_t s_lo = bytes_to_h2(scales, 0x4040u | (uint32_t)byte | (uint32_t)(byte << 8)), s_hi = bytes_to_h2(scales, 0x4040u | (uint32_t)(byte + 1) | (uint32_t)((byte + 1) << 8));
  const uint32_t o_lo = hmul2_u(s_lo, h2c(-(BASE + tg_centre<TYPE>()))), o_hi = hmul2_u(s_hi, h2c(-(BASE + tg_centre<TYPE>())));
#pragma unroll
  for (int i = 0; i < 8; i++) {
    uint32_t l, h;
    if constexpr (TYPE == T_Q4_K) {
      l = (w[i] << 4) & 0xF0F0F0F0u;
      h = w[i] & 0xF0F0F0F0u;
    } else {   // bit 2 grp of a fifth-bit byte belongs to the low nibble, the next one to the high
      const uint32_t f = fifth[i] >> (2 * grp);   // bits of the other bytes move in above and are masked away
      l = ((w[i] << 3) & 0x78787878u) | ((f << 7) & 0x80808080u);
      h = ((w[i] >> 1) & 0x78787878u) | ((f << 6) & 0x80808080u);
    }
    out[2 * i] = hfma2_u(__byte_perm(l, MAGIC, 0x4140), s_lo, o_lo); out[2 * i + 1] = hfma2_u(__byte_perm(l, MAGIC, 0x4342), s_lo, o_lo);
    out[16 + 2 * i] = hfma2_u(__byte_perm(h, MAGIC, 0x4140), s_hi, o_hi); out[16 + 2 * i + 1] = hfma2_u(__byte_perm(h, MAGIC, 0x4342), s_hi, o_hi);
  }
}

struct Unit { int tile, col_off, cnt, sb0, nsb, ks; };

template <int TYPE, int NMAX>
__global__ void __launch_bounds__(TG_THREADS, 1) tgemm_kernel(const __grid_constant__ TGemmMaps maps, const TGemmParams p) {
  constexpr int BLK = tg_blk<TYPE>(), STAGE = tg_stage<TYPE, NMAX>(), NS = tg_stages<TYPE, NMAX>(), RAW = NMAX * 640;
  extern __shared__ uint8_t tg_smem[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(tg_smem) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full[NS], empty[NS], a_full[TG_NA], a_empty[TG_NA], c_full[2], c_empty[2], d_full[TG_ND];
  __shared__ float2 dd[TG_ND][TG_TILE];
  __shared__ uint32_t tmem_sm;
  __shared__ volatile int failed;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (int s = 0; s < NS; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 9); }
    for (int s = 0; s < TG_NA; s++) { mbar_init(&a_full[s], 4); mbar_init(&a_empty[s], 1); }
    for (int s = 0; s < 2; s++) { mbar_init(&c_full[s], 1); mbar_init(&c_empty[s], 4); }
    for (int s = 0; s < TG_ND; s++) mbar_init(&d_full[s], 4);
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

  const int nb = p.K / 256, tiles = (p.N + TG_TILE - 1) / TG_TILE, coltiles = (p.M + NMAX - 1) / NMAX;
  auto give_up = [&]() { report_error(p.err); failed = 1; };
  auto stopped = [&]() { return __any_sync(0xffffffffu, failed); };
  auto unit_at = [&](int u) {
    Unit t;
    t.ks = u % p.ksplit;
    const int v = u / p.ksplit;
    t.tile = v % tiles; t.col_off = v / tiles * NMAX; t.cnt = min(NMAX, p.M - t.col_off);
    t.sb0 = t.ks * nb / p.ksplit; t.nsb = (t.ks + 1) * nb / p.ksplit - t.sb0;
    return t;
  };
  // the quant blocks of super-block sb of a unit's 128 rows, and the unit's activation rows
  constexpr uint32_t TX = TG_TILE * BLK + RAW;
  auto load_raw = [&](const Unit& t, int sb, int s) {
    const int row = t.tile * TG_TILE;
    mbar_expect_tx(&full[s], TX);
    tma_box(smem + (size_t)s * STAGE + RAW, reinterpret_cast<const CUtensorMap*>(row < p.seg_end ? &maps.w : &maps.w2), sb * BLK, row < p.seg_end ? row : row - p.seg_end, &full[s]);
  };
  auto load_x = [&](const Unit& t, int sb, int s) {
    uint8_t* bt = smem + (size_t)s * STAGE;
    for (int c = 0; c < 4; c++) tma_box(bt + c * (NMAX * 128), reinterpret_cast<const CUtensorMap*>(&maps.x), sb * 256 + c * 64, t.col_off, &full[s]);
    tma_box(bt + 4 * (NMAX * 128), reinterpret_cast<const CUtensorMap*>(&maps.sx), sb * TG_SX, t.col_off, &full[s]);
  };

  // A CTA's share of units does not depend on the kernel before it, nor do its weights: the first stages of quants are
  // asked for while that kernel still runs.
  const long long U = (long long)coltiles * tiles * p.ksplit;
  const int u0 = (int)(blockIdx.x * U / gridDim.x), u1 = (int)((blockIdx.x + 1) * U / gridDim.x);
  uint32_t early = 0;
  if (warp == 0) {
    for (int u = u0; u < u1 && early < (uint32_t)NS; u++) {
      const Unit t = unit_at(u);
      for (int b = 0; b < t.nsb && early < (uint32_t)NS; b++, early++)
        if (elect_one()) load_raw(t, t.sb0 + b, early);
    }
  }
  pdl_wait();
  pdl_launch();

  if (warp == 0) {
    // ---- loads --------------------------------------------------------------------------------
    uint32_t it = 0;
    for (int u = u0; u < u1 && !stopped(); u++) {
      const Unit t = unit_at(u);
      for (int b = 0; b < t.nsb; b++, it++) {
        const int s = it % NS;
        if (it >= early && !warp_wait(&empty[s], ((it / NS) & 1) ^ 1)) { give_up(); break; }
        if (elect_one()) {
          if (it >= early) load_raw(t, t.sb0 + b, s);
          load_x(t, t.sb0 + b, s);
        }
        __syncwarp();
      }
    }
    // a CTA that gave up leaves only once its copies have landed
    if (failed)
      for (uint32_t k = it > (uint32_t)NS ? it - NS : 0; k < it; k++) mbar_wait(&full[k % NS], (k / NS) & 1);
  } else if (warp == 1) {
    // ---- tensor core --------------------------------------------------------------------------
    uint32_t it = 0, hx = 0, cx = 0;
    bool ok = true;
    for (int u = u0; u < u1 && ok && !stopped(); u++) {
      const Unit t = unit_at(u);
      const uint32_t id = idesc_n((t.cnt + 15) & ~15);
      for (int b = 0; b < t.nsb && ok; b++, it++, cx++) {
        const int s = it % NS, cs = cx & 1;
        const uint32_t acc = tm + TG_ACC + cs * 2 * NMAX;
        if (!warp_wait(&full[s], (it / NS) & 1) || !warp_wait(&c_empty[cs], ((cx >> 1) & 1) ^ 1)) { give_up(); ok = false; break; }
        const uint32_t bt = smem_addr(smem + (size_t)s * STAGE);
#pragma unroll
        for (int h = 0; h < 2; h++, hx++) {
          const int as = hx % TG_NA;
          if (!warp_wait(&a_full[as], (hx / TG_NA) & 1)) { give_up(); ok = false; break; }
          fence_after();
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < 8; k++)
              mma_ts(acc, tm + as * TG_ASLOT + 8 * k, desc_sw128(bt + (2 * h + (k >> 2)) * (NMAX * 128)) + 2 * (k & 3), id, (h | k) != 0);
            if (h == 1) {
              mma_ts(acc, tm + TG_CEN + (it & 1) * 8, desc_sw128(bt + 4 * (NMAX * 128)), id, 1);
              mma_ts(acc + NMAX, tm + TG_MIN + (it & 1) * 8, desc_sw128(bt + 4 * (NMAX * 128)), id, 0);
            }
            commit(&a_empty[as]);
            if (h == 1) { commit(&empty[s]); commit(&c_full[cs]); }
          }
          __syncwarp();
        }
      }
    }
  } else if (warp < TG_DR0) {
    // ---- dequantisation -----------------------------------------------------------------------
    const int half = warp >= TG_DQ0 + 4, q = warp & 3, row = q * 32 + lane;
    const uint32_t lane_base = tm + ((uint32_t)(q * 32) << 16);
    uint32_t it = 0;
    bool ok = true;
    for (int u = u0; u < u1 && ok && !stopped(); u++) {
      const Unit t = unit_at(u);
      for (int b = 0; b < t.nsb; b++, it++) {
        const int s = it % NS;
        const uint32_t hx = 2 * it + half;
        const int as = hx % TG_NA;
        if (!warp_wait(&full[s], (it / NS) & 1)) { give_up(); ok = false; break; }
        const uint8_t* blk = smem + (size_t)s * STAGE + RAW + row * BLK;
        const uint4 hdr = lds128(blk);
        uint4 qv[4];
        uint32_t fifth[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if constexpr (TYPE == T_Q5_K) {
          const uint4 fa = lds128(blk + 16), fb = lds128(blk + 32);
          fifth[0] = fa.x; fifth[1] = fa.y; fifth[2] = fa.z; fifth[3] = fa.w; fifth[4] = fb.x; fifth[5] = fb.y; fifth[6] = fb.z; fifth[7] = fb.w;
        }
#pragma unroll
        for (int i = 0; i < 4; i++) qv[i] = lds128(blk + (TYPE == T_Q4_K ? 16 : 48) + 64 * half + 16 * i);
        __syncwarp();
        if (lane == 0) arrive(&empty[s]);
        // 6-bit scales and mins of this half's four sub-blocks (gguf/dequant.go:238-243)
        const uint32_t sc = half ? (hdr.w & 0x0F0F0F0Fu) | ((hdr.y >> 2) & 0x30303030u) : hdr.y & 0x3F3F3F3Fu;
        const uint32_t mn = half ? ((hdr.w >> 4) & 0x0F0F0F0Fu) | ((hdr.z >> 2) & 0x30303030u) : hdr.z & 0x3F3F3F3Fu;
        const uint32_t m01 = bytes_to_h2(mn, 0x4140), m23 = bytes_to_h2(mn, 0x4342), c2 = h2c(tg_centre<TYPE>()), c01 = hmul2_u(bytes_to_h2(sc, 0x4140), c2), c23 = hmul2_u(bytes_to_h2(sc, 0x4342), c2);
        uint32_t out[32];
        dequant_group<TYPE>(qv[0], qv[1], fifth, 2 * half, sc, 0, out);
        if (!warp_wait(&a_empty[as], ((hx / TG_NA) & 1) ^ 1)) { give_up(); ok = false; break; }
        fence_after();
        tmem_st32(lane_base + as * TG_ASLOT, out);
        const uint32_t mcol = lane_base + TG_MIN + (it & 1) * 8 + 2 * half;
        tmem_st2(mcol, m01, m23);
        tmem_st2(mcol + 4, m01, m23);
        tmem_st2(mcol + TG_CEN - TG_MIN, c01, c23);
        tmem_st2(mcol + TG_CEN - TG_MIN + 4, c01, c23);
        dequant_group<TYPE>(qv[2], qv[3], fifth, 2 * half + 1, sc, 2, out);
        tmem_st32(lane_base + as * TG_ASLOT + 32, out);
        if (!half) dd[it % TG_ND][row] = make_float2(h2f_lo(hdr.x), h2f_hi(hdr.x));
        tmem_st_wait();
        fence_before();
        __syncwarp();
        if (lane == 0) { arrive(&a_full[as]); if (!half) arrive(&d_full[it % TG_ND]); }
      }
    }
  } else {
    // ---- drain and epilogue -------------------------------------------------------------------
    const int q = warp & 3, row = q * 32 + lane;
    const uint32_t lane_base = tm + ((uint32_t)(q * 32) << 16) + TG_ACC;
    uint32_t it = 0;
    bool ok = true;
    for (int u = u0; u < u1 && ok && !stopped(); u++) {
      const Unit t = unit_at(u);
      float acc[NMAX];
#pragma unroll
      for (int c = 0; c < NMAX; c++) acc[c] = 0.f;
      for (int b = 0; b < t.nsb; b++, it++) {
        const int cs = it & 1;
        if (!warp_wait(&d_full[it % TG_ND], (it / TG_ND) & 1) || !warp_wait(&c_full[cs], (it >> 1) & 1)) { give_up(); ok = false; break; }
        fence_after();
        const float2 dm = dd[it % TG_ND][row];
#pragma unroll
        for (int c0 = 0; c0 < NMAX; c0 += 16) {
          if (c0 < t.cnt) {
            uint32_t v[16], m[16];
            tmem_ld16(lane_base + cs * 2 * NMAX + c0, v);
            tmem_ld16(lane_base + cs * 2 * NMAX + NMAX + c0, m);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; i++) acc[c0 + i] += fmaf(dm.x, __uint_as_float(v[i]), -(dm.y * __uint_as_float(m[i])));
          }
        }
        fence_before();
        __syncwarp();
        if (lane == 0) arrive(&c_empty[cs]);
      }
      if (!ok) break;
      const int orow = t.tile * TG_TILE + row;
      if (orow < p.N) {
        float* y = p.y + (int64_t)t.ks * p.plane + (int64_t)t.col_off * p.ldy + orow;
#pragma unroll
        for (int c = 0; c < NMAX; c++)
          if (c < t.cnt) y[(int64_t)c * p.ldy] = acc[c];
      }
    }
  }
  fence_before();
  __syncthreads();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tm) : "memory");
}

template <int TYPE, int NMAX>
int launch_t(const TGemmParams& p, const TGemmMaps& maps, bool pdl, cudaStream_t st) {
  auto kernel = tgemm_kernel<TYPE, NMAX>;
  constexpr int smem = tg_stages<TYPE, NMAX>() * tg_stage<TYPE, NMAX>() + 1024;
  B200_ONCE_PER_DEVICE(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const int sms = sm_count_current();
  if (sms <= 0) return ECUDA;
  const int64_t units = (int64_t)((p.M + NMAX - 1) / NMAX) * ((p.N + TG_TILE - 1) / TG_TILE) * p.ksplit;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)std::min<int64_t>(units, sms)); cfg.blockDim = dim3(TG_THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = pdl ? 1 : 0;
  B200_CUDA(cudaLaunchKernelEx(&cfg, kernel, maps, p));
  return OK;
}
template <int TYPE>
int launch_n(int cols, const TGemmParams& p, const TGemmMaps& maps, bool pdl, cudaStream_t st) {
  if (cols == 16) return launch_t<TYPE, 16>(p, maps, pdl, st);
  if (cols == 32) return launch_t<TYPE, 32>(p, maps, pdl, st);
  if (cols == 64) return launch_t<TYPE, 64>(p, maps, pdl, st);
  set_error("tgemm: tiles have 16, 32 or 64 columns");
  return EINVAL_;
}

// A warp per (row, sub-block), lane = element. grid (rows, ceil(K / 256)), block 256.
__global__ void __launch_bounds__(256) row_sums_kernel(const __half* x, int K, __half* sx) {
  pdl_wait();
  pdl_launch();
  const int s = blockIdx.y * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (s * 32 >= K) return;
  const float sum = warp_sum(__half2float(x[(size_t)blockIdx.x * K + s * 32 + lane]));
  if (lane == 0) store_sub_sum(sx + (size_t)blockIdx.x * (K / 256 * TG_SX), s, sum);
}

}  // namespace

typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                             CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

int encode_nd(CUtensorMapDataType type, const void* base, int rank, const int64_t* dims_, const int64_t* strides_, const int* box_, CUtensorMapSwizzle swizzle, TMap* out) {
  static std::atomic<EncodeFn> encode{nullptr};
  EncodeFn fn = encode.load();
  if (fn == nullptr) {
    void* q = nullptr;
    cudaDriverEntryPointQueryResult res;
    B200_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &q, cudaEnableDefault, &res));
    if (q == nullptr || res != cudaDriverEntryPointSuccess) { set_error("the driver does not export cuTensorMapEncodeTiled"); return ECUDA; }
    fn = (EncodeFn)q;
    encode.store(fn);
  }
  cuuint64_t dims[3], strides[2];
  cuuint32_t box[3], estr[3] = {1, 1, 1};
  for (int i = 0; i < rank; i++) { dims[i] = (cuuint64_t)dims_[i]; box[i] = (cuuint32_t)box_[i]; if (i + 1 < rank) strides[i] = (cuuint64_t)strides_[i]; }
  const CUresult r = fn(reinterpret_cast<CUtensorMap*>(out->b), type, rank, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled failed with code " + std::to_string((int)r)); return ECUDA; }
  return OK;
}
int encode_2d(CUtensorMapDataType type, const void* base, int64_t inner, int64_t rows, int64_t stride, int box_inner, int box_rows, CUtensorMapSwizzle swizzle, TMap* out) {
  const int64_t dims[2] = {inner, rows};
  const int box[2] = {box_inner, box_rows};
  return encode_nd(type, base, 2, dims, &stride, box, swizzle, out);
}

bool tgemm_type(uint32_t type) { return type == T_Q4_K || type == T_Q5_K; }

int tgemm_cols(int rows) { return rows <= 16 ? 16 : rows <= 32 ? 32 : 64; }

// As many parts of the contraction as keep every SM busy with at least two super-blocks each.
int tgemm_ksplit(int K, int N, int M, int cols) {
  const int units = (N + TG_TILE - 1) / TG_TILE * ((M + cols - 1) / cols);
  return std::max(1, std::min(148 / std::max(units, 1), K / 512));
}

int make_w_tensor_map(uint32_t type, const uint8_t* w, int64_t rows, int64_t stride, int box_rows, TMap* out) {
  if (!tgemm_type(type)) { set_error("tgemm: weight type has no kernel"); return EINVAL_; }
  return encode_2d(CU_TENSOR_MAP_DATA_TYPE_UINT8, w, stride, rows, stride, type == T_Q4_K ? 144 : 176, box_rows, CU_TENSOR_MAP_SWIZZLE_NONE, out);
}
int make_rows_map(const __half* x, int64_t rows, int K, int box_rows, TMap* out) {
  return encode_2d(CU_TENSOR_MAP_DATA_TYPE_FLOAT16, x, K, rows, (int64_t)K * 2, 64, box_rows, CU_TENSOR_MAP_SWIZZLE_128B, out);
}

int launch_row_sums(const __half* x, int rows, int K, __half* sx, bool pdl, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(rows, (K + 255) / 256); cfg.blockDim = dim3(256); cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = pdl ? 1 : 0;
  B200_CUDA(cudaLaunchKernelEx(&cfg, row_sums_kernel, x, K, sx));
  return OK;
}

int launch_tgemm(uint32_t type, int cols, const TGemmParams& p, const TGemmMaps& maps, bool pdl, cudaStream_t st) {
  if (p.K % 256 != 0 || p.K <= 0 || p.N <= 0 || p.M <= 0 || p.ksplit < 1 || p.ksplit > p.K / 256) { set_error("tgemm: row length must be a multiple of 256"); return EINVAL_; }
  if (p.seg_end < p.N && p.seg_end % TG_TILE != 0) { set_error("tgemm: the first segment must be whole tiles"); return EINVAL_; }
  if (type == T_Q4_K) return launch_n<T_Q4_K>(cols, p, maps, pdl, st);
  if (type == T_Q5_K) return launch_n<T_Q5_K>(cols, p, maps, pdl, st);
  set_error("tgemm: weight type has no kernel (Q4_K, Q5_K)");
  return EINVAL_;
}

}  // namespace b200
