// Work-list expert projections with warps that work alone.
//
// Few columns per expert make this a stream of weights: 1.8 MB per expert, each weight used for one to sixteen columns. What
// bounded the column-tiled kernel here was not DRAM but what it did per 16-row tile around the arithmetic: eight warps shared
// a tile's super-blocks, met at a barrier, added their partial sums through shared memory and refilled a ring that one thread
// fed. Here a warp owns 32 gate + 32 up rows (or 64 rows of the down projection) over the whole contraction: its sums never
// leave its registers, the four 16-row tiles share every activation fragment, and it feeds a ring of its own with TMA boxes of
// 16 rows x one super-block: two super-blocks of four boxes deep for Q4_K (18 KB per warp, 216 KB in flight per SM), one for Q5_K
// (11 KB). Warps meet only once, to read the CTA's part of the list. Activations come through L1, which all twelve warps share.
// Now it is instruction issue: 343 per box with one column group and 453 with two (12 and 701 rows of the 512-expert shape), half
// of them integer ones; 38 us for 124 MB of gate and up weights, 55 % of the issue slots.
#include <algorithm>

#include "qgemv.cuh"
#include "qlist.cuh"

namespace b200 {

namespace {

constexpr int QL_ENT = 64;   // entries one CTA's share may touch

template <int TYPE, int NC> struct QlCfg {
  static constexpr int BLK = TYPE == T_Q4_K ? 144 : 176, BYTES = 16 * BLK;   // a ring slot: 16 rows x one super-block, rows BLK apart
  static constexpr int WARPS = 12;                                           // 168 registers a thread; sixteen warps of 128 measured the same
  static constexpr int AHEAD = 216 * 1024 / WARPS / BYTES >= 8 ? 2 : 1;      // super-blocks (four chunks) in the ring
  static constexpr int SLOTS = 4 * AHEAD;
};

__device__ __forceinline__ void tma_box(uint32_t dst, const void* tm, int c0, int c1, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(tm), "r"(c0), "r"(c1),
               "r"((uint32_t)__cvta_generic_to_shared(bar))
               : "memory");
}

template <int TYPE, int NC, int EPI>
__global__ void __launch_bounds__(QlCfg<TYPE, NC>::WARPS * 32, 1) qlist_kernel(const __grid_constant__ QListMaps maps, const QListParams p) {
  using Cf = QlCfg<TYPE, NC>;
  constexpr bool PAIR = EPI == QL_SWIGLU;
  constexpr int UROWS = PAIR ? 32 : 64;      // output rows of a unit; its four chunks are gate, up, gate, up rows or four times 16 rows
  constexpr int SLOTS = Cf::SLOTS, THREADS = Cf::WARPS * 32, QOFF = Cf::BLK - 128;
  extern __shared__ __align__(128) uint8_t ql_smem[];
  __shared__ int4 ent[QL_ENT];
  __shared__ int ids[QL_ENT][8 * NC];
  __shared__ __align__(8) uint64_t bars[Cf::WARPS][SLOTS];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int nb = p.K / 256, upe = p.N / UROWS;   // units per entry
  if (lane == 0) {
    for (int i = 0; i < SLOTS; i++) mbar_init(&bars[warp][i], 1);
    mbar_fence_init();
  }
  pdl_wait();
  pdl_launch();
  const int n_ent = *p.n_entries;
  const long long U = (long long)n_ent * upe;
  const int u0 = (int)(blockIdx.x * U / gridDim.x), u1 = (int)((blockIdx.x + 1) * U / gridDim.x);
  if (u0 >= u1) return;
  const int e0 = u0 / upe, ne = (u1 - 1) / upe - e0 + 1;
  for (int i = tid; i < ne * 8 * NC; i += THREADS) {
    const int e = i / (8 * NC), c = i - e * (8 * NC);
    const int4 v = p.entries[e0 + e];
    if (c == 0) ent[e] = v;
    ids[e][c] = p.cols[v.y + min(c, v.z - 1)];   // columns past the end repeat the last one and are not written
  }
  __syncthreads();

  const uint32_t ring = (uint32_t)__cvta_generic_to_shared(ql_smem) + warp * (SLOTS * Cf::BYTES);
  const int n_units = u0 + warp < u1 ? (u1 - u0 - warp + Cf::WARPS - 1) / Cf::WARPS : 0;
  // ---- the copy side walks the super-blocks AHEAD of the arithmetic; a chunk's slot and its place in the unit are constants of j ----
  int f_left = n_units * nb, f_unit = u0 + warp, f_sb = 0, f_row = 0;
  const void *fa = nullptr, *fb = nullptr;
  auto locate = [&]() {   // the unit that is fetched from now on
    const int e = min(f_unit, u1 - 1) / upe, ex = ent[e - e0].x;
    f_row = (ex >= 0 ? ex * p.N : 0) + (f_unit - e * upe) * UROWS;
    fa = ex >= 0 ? &maps.w : &maps.ws;
    fb = !PAIR ? fa : ex >= 0 ? &maps.w2 : &maps.ws2;
  };
  auto fetch = [&](int slot, int j, bool reused) {   // chunk j of super-block f_sb
    if (f_left > 0 && elect_one()) {
      if (reused) fence_proxy_async();
      mbar_expect_tx(&bars[warp][slot], Cf::BYTES);
      tma_box(ring + slot * Cf::BYTES, (j & 1) ? fb : fa, f_sb * Cf::BLK, f_row + (PAIR ? j >> 1 : j) * 16, &bars[warp][slot]);
    }
  };
  auto fetched = [&]() {   // a super-block's four chunks are on their way
    if (f_left > 0) { f_left--; if (++f_sb == nb) { f_sb = 0; f_unit += Cf::WARPS; if (f_left > 0) locate(); } }
  };
  if (n_units > 0) locate();
  for (int i = 0; i < Cf::AHEAD; i++) {
    for (int j = 0; j < 4; j++) fetch(4 * i + j, j, false);
    fetched();
  }

  // mma row g is row 2g of a chunk, mma row g + 8 row 2g + 1: at a pitch of 144 or 176 bytes the eight-byte reads of four
  // neighbouring g then fall on distinct banks
  const uint32_t row_off = 2 * g * Cf::BLK;
  const uint32_t min_sel = 0x4040u | (2 * (t >> 1)) | ((2 * (t >> 1) + 1) << 8);   // two mins of this thread's pair as magic halves
  uint32_t done = 0;   // super-blocks
  for (int i = 0; i < n_units; i++) {
    const int u = u0 + warp + i * Cf::WARPS, e = u / upe, tile = u - e * upe, le = e - e0, cnt = ent[le].z;
    const __half *xp[NC], *sp[NC];
#pragma unroll
    for (int nc = 0; nc < NC; nc++) {
      const int64_t row = ids[le][nc * 8 + g] / p.x_div;
      xp[nc] = p.x + row * p.K + 8 * t;
      sp[nc] = p.sx + row * (nb * TG_SX) + ((t & 1) ? 8 : 0) + 2 * (t >> 1);   // even t: the hi parts, odd t: the lo parts
    }
    const bool wide = NC > 1 && cnt > 8;
    float acc[4][NC][4];
#pragma unroll
    for (int a = 0; a < 4 * NC * 4; a++) (&acc[0][0][0])[a] = 0.f;
    // activation fragments of a super-block: sub-block s, words (0, 2), (1, 3), (4, 6), (5, 7) of the thread's eight elements
    uint4 b[NC][8];
    auto load_b = [&](int sb, int s0, int s1) {
#pragma unroll
      for (int nc = 0; nc < NC; nc++)
        if (nc == 0 || wide) {
#pragma unroll
          for (int s = s0; s < s1; s++) b[nc][s] = *reinterpret_cast<const uint4*>(xp[nc] + sb * 256 + s * 32);
        }
    };
    load_b(0, 0, 8);
#pragma unroll 1
    for (int sb = 0; sb < nb; sb++, done++) {
      const int slot0 = Cf::AHEAD == 2 ? (done & 1) * 4 : 0, phase = Cf::AHEAD == 2 ? (done >> 1) & 1 : done & 1;
      uint32_t sx0[NC], sx1[NC];
#pragma unroll
      for (int nc = 0; nc < NC; nc++) {
        sx0[nc] = *reinterpret_cast<const uint32_t*>(sp[nc] + sb * TG_SX);
        sx1[nc] = *reinterpret_cast<const uint32_t*>(sp[nc] + sb * TG_SX + 4);
      }
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int slot = slot0 + j;
        if (!warp_wait(&bars[warp][slot], phase)) {   // a copy never landed: report, the results are void
          if (lane == 0) report_error(p.err);
          // leave with no copy in flight: this super-block's other chunks, the next one's before this
          for (int k = 0; k < SLOTS; k++) {
            const bool ahead = Cf::AHEAD == 2 && (k >> 2) != (slot0 >> 2);
            mbar_wait(&bars[warp][k], ahead ? (done + 1) >> 1 & 1 : k - slot0 < j ? phase ^ 1 : phase, 1u << 18);
          }
          return;
        }
        const uint32_t base = ring + slot * Cf::BYTES + row_off;
        const uint4 h0 = ld_s128(base), h1 = ld_s128(base + Cf::BLK);
        // 6-bit scales of the two rows, four sub-blocks to a word (gguf/dequant.go:238-243)
        const uint32_t scl[2][2] = {{h0.y & 0x3F3F3F3Fu, (h0.w & 0x0F0F0F0Fu) | ((h0.y >> 2) & 0x30303030u)}, {h1.y & 0x3F3F3F3Fu, (h1.w & 0x0F0F0F0Fu) | ((h1.y >> 2) & 0x30303030u)}};
        float sum[NC][4];   // sub-block scale x (q . x), without d
#pragma unroll
        for (int a = 0; a < NC * 4; a++) (&sum[0][0])[a] = 0.f;
#pragma unroll
        for (int G = 0; G < 4; G++) {
          const uint32_t qa = base + QOFF + 32 * G + 8 * t;
          const uint2 q0 = ld_s64(qa), q1 = ld_s64(qa + Cf::BLK);
          uint2 f0 = make_uint2(0, 0), f1 = f0;
          if constexpr (TYPE == T_Q5_K) { f0 = ld_s64(base + 16 + 8 * t); f1 = ld_s64(base + Cf::BLK + 16 + 8 * t); }
          if (j == 0) {   // first use of the fragments: into pair order
#pragma unroll
            for (int nc = 0; nc < NC; nc++)
              if (nc == 0 || wide) {
#pragma unroll
                for (int k = 0; k < 2; k++) {
                  const uint4 x = b[nc][2 * G + k];
                  b[nc][2 * G + k] = make_uint4(__byte_perm(x.x, x.y, 0x5410), __byte_perm(x.x, x.y, 0x7632), __byte_perm(x.z, x.w, 0x5410), __byte_perm(x.z, x.w, 0x7632));
                }
              }
          }
          uint32_t al[2][4], ah[2][4];
          unpack_word<TYPE>(q0.x, f0.x, G, al[0][0], al[0][2], ah[0][0], ah[0][2]);
          unpack_word<TYPE>(q1.x, f1.x, G, al[0][1], al[0][3], ah[0][1], ah[0][3]);
          unpack_word<TYPE>(q0.y, f0.y, G, al[1][0], al[1][2], ah[1][0], ah[1][2]);
          unpack_word<TYPE>(q1.y, f1.y, G, al[1][1], al[1][3], ah[1][1], ah[1][3]);
          float s0[2], s1[2];    // scales of sub-blocks 2G, 2G + 1 of the two rows
          sub_scales<TYPE>(scl[0][G >> 1], G & 1, s0);
          sub_scales<TYPE>(scl[1][G >> 1], G & 1, s1);
#pragma unroll
          for (int nc = 0; nc < NC; nc++)
            if (nc == 0 || wide) {
              float C[4], D[4];
              const uint4 xl = b[nc][2 * G], xh = b[nc][2 * G + 1];
              mma16816_z(C, al[0], xl.x, xl.y); mma16816(C, al[1], xl.z, xl.w);
              mma16816_z(D, ah[0], xh.x, xh.y); mma16816(D, ah[1], xh.z, xh.w);
              float* a = sum[nc];
              a[0] = fmaf(s0[0], C[0], a[0]); a[1] = fmaf(s0[0], C[1], a[1]); a[2] = fmaf(s1[0], C[2], a[2]); a[3] = fmaf(s1[0], C[3], a[3]);
              a[0] = fmaf(s0[1], D[0], a[0]); a[1] = fmaf(s0[1], D[1], a[1]); a[2] = fmaf(s1[1], D[2], a[2]); a[3] = fmaf(s1[1], D[3], a[3]);
            }
          if (j == 3 && sb + 1 < nb) load_b(sb + 1, 2 * G, 2 * G + 2);   // the next super-block's, as soon as these are done with
        }
        // min term (sub-blocks 2 (t / 2), + 1 and 4 + these), then the block scales
        const uint32_t am[4] = {hadd2_u(__byte_perm(h0.z & 0x3F3F3F3Fu, 0x64646464u, min_sel), half2_const(-1024.f)), hadd2_u(__byte_perm(h1.z & 0x3F3F3F3Fu, 0x64646464u, min_sel), half2_const(-1024.f)),
                                hadd2_u(__byte_perm(((h0.w >> 4) & 0x0F0F0F0Fu) | ((h0.z >> 2) & 0x30303030u), 0x64646464u, min_sel), half2_const(-1024.f)),
                                hadd2_u(__byte_perm(((h1.w >> 4) & 0x0F0F0F0Fu) | ((h1.z >> 2) & 0x30303030u), 0x64646464u, min_sel), half2_const(-1024.f))};
        const float d0 = h2f_lo(h0.x) * unit_scale<TYPE>(), n0 = h2f_hi(h0.x), d1 = h2f_lo(h1.x) * unit_scale<TYPE>(), n1 = h2f_hi(h1.x);
#pragma unroll
        for (int nc = 0; nc < NC; nc++) {
          if (nc == 0 || wide) {
            float Cm[4];
            mma16816_z(Cm, am, sx0[nc], sx1[nc]);
            float* a = acc[j][nc];
            a[0] = fmaf(-n0, Cm[0], fmaf(d0, sum[nc][0], a[0])); a[1] = fmaf(-n0, Cm[1], fmaf(d0, sum[nc][1], a[1]));
            a[2] = fmaf(-n1, Cm[2], fmaf(d1, sum[nc][2], a[2])); a[3] = fmaf(-n1, Cm[3], fmaf(d1, sum[nc][3], a[3]));
          }
        }
        __syncwarp();   // every lane has read the chunk
        fetch(slot, j, true);
      }
      fetched();
    }
    if constexpr (PAIR) {
      // SwiGLU (shaders/llm_moe_gemv.comp:777-781); the 32 rows are one sub-block of the down projection's input
#pragma unroll
      for (int nc = 0; nc < NC; nc++) {
        if (nc == 0 || wide) {
          float s[2] = {0.f, 0.f};
#pragma unroll
          for (int pr = 0; pr < 2; pr++)
#pragma unroll
            for (int k = 0; k < 2; k++) {
              const float g0 = acc[2 * pr][nc][k], g1 = acc[2 * pr][nc][k + 2];
              const __half2 hv = __floats2half2_rn(g0 * sigmoid_acc(g0) * acc[2 * pr + 1][nc][k], g1 * sigmoid_acc(g1) * acc[2 * pr + 1][nc][k + 2]);
              const float2 fv = __half22float2(hv);
              s[k] += fv.x + fv.y;
              const int c = nc * 8 + 2 * t + k;
              if (c < cnt) *reinterpret_cast<__half2*>(p.y16 + (int64_t)ids[le][c] * p.ldy + tile * 32 + pr * 16 + 2 * g) = hv;
            }
#pragma unroll
          for (int k = 0; k < 2; k++) {
            s[k] += __shfl_xor_sync(0xffffffffu, s[k], 4); s[k] += __shfl_xor_sync(0xffffffffu, s[k], 8); s[k] += __shfl_xor_sync(0xffffffffu, s[k], 16);
            const int c = nc * 8 + 2 * t + k;
            if (g == 0 && c < cnt) store_sub_sum(p.sx_out + (int64_t)ids[le][c] * (p.ldy / 256 * TG_SX), tile, s[k]);
          }
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; j++)
#pragma unroll
        for (int nc = 0; nc < NC; nc++)
#pragma unroll
          for (int k = 0; k < 2; k++) {
            const int c = nc * 8 + 2 * t + k;
            if (c < cnt) *reinterpret_cast<float2*>(p.y + (int64_t)ids[le][c] * p.ldy + tile * 64 + j * 16 + 2 * g) = make_float2(acc[j][nc][k], acc[j][nc][k + 2]);
          }
    }
  }
}

template <int TYPE, int NC, int EPI>
int launch_t(const QListParams& p, const QListMaps& maps, bool pdl, cudaStream_t st) {
  using Cf = QlCfg<TYPE, NC>;
  auto kernel = qlist_kernel<TYPE, NC, EPI>;
  constexpr int smem = Cf::WARPS * Cf::SLOTS * Cf::BYTES;
  B200_ONCE_PER_DEVICE(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const int sms = sm_count_current();
  if (sms <= 0) return ECUDA;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(sms); cfg.blockDim = dim3(Cf::WARPS * 32); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = pdl ? 1 : 0;
  B200_CUDA(cudaLaunchKernelEx(&cfg, kernel, maps, p));
  return OK;
}
template <int TYPE>
int launch_c(int epi, int cols, const QListParams& p, const QListMaps& maps, bool pdl, cudaStream_t st) {
  if (cols == 8) return epi == QL_SWIGLU ? launch_t<TYPE, 1, QL_SWIGLU>(p, maps, pdl, st) : launch_t<TYPE, 1, QL_STORE>(p, maps, pdl, st);
  if (cols == 16) return epi == QL_SWIGLU ? launch_t<TYPE, 2, QL_SWIGLU>(p, maps, pdl, st) : launch_t<TYPE, 2, QL_STORE>(p, maps, pdl, st);
  set_error("qlist: entries have at most 8 or 16 columns");
  return EINVAL_;
}

}  // namespace

bool qlist_type(uint32_t type) { return type == T_Q4_K || type == T_Q5_K; }
// whole units, and a CTA's share of the list must fit its table of entries
bool qlist_fits(int K, int N, int max_entries) { return K % 256 == 0 && N % 64 == 0 && max_entries / 100 + 2 <= QL_ENT; }

int launch_qlist(uint32_t type, int epi, int cols, const QListParams& p, const QListMaps& maps, bool pdl, cudaStream_t st) {
  if (p.K % 256 != 0 || p.N % 64 != 0 || (epi == QL_SWIGLU && p.ldy % 256 != 0)) { set_error("qlist: shape outside kernel limits"); return EINVAL_; }
  if (sm_count_current() < 100) { set_error("qlist: the list's shares assume at least 100 SMs"); return ECAPACITY; }
  if (type == T_Q4_K) return launch_c<T_Q4_K>(epi, cols, p, maps, pdl, st);
  if (type == T_Q5_K) return launch_c<T_Q5_K>(epi, cols, p, maps, pdl, st);
  set_error("qlist: weight type has no kernel (Q4_K, Q5_K)");
  return EINVAL_;
}

}  // namespace b200
