// tcgen05 GEMM over K-quant weights rounded to fp16 (see wgemm.cuh).
//
// A CTA of 19 or 23 warps walks items of 128 weight rows (or 64 gate + 64 up rows) x NT activation rows:
//   warp 0        TMA boxes of the rows' quant blocks, one super-block per ring stage;
//   the last warp TMA boxes of the activation rows, 128 elements per ring stage (64 for NT 256), only as many rows as the problem has;
//   warps 2..     three groups of four: a group turns half a super-block of the 128 rows (a thread per row) into fp16 and puts
//                 it into tensor memory with tcgen05.st; the groups take the halves in turn;
//   warp 1        one thread issues eight tcgen05.mma (M 128, N NT, K 16) per half, A from tensor memory, B from shared memory;
//   the others    epilogue, one or two groups of four warps.
// What bounds it: a tcgen05.mma with M 128 and K 16 takes 68 cycles for every N up to 128 (measured), 32 weights per cycle
// and SM, so 512 experts of 3 M weights take 180 us whatever their rows; NT 256 doubles the work per cycle. The form before
// this one (eight dequantising warps that loaded their rows from global memory and stored the fp16 tile swizzled into shared
// memory) took 1190 us at 40 rows per expert and 1366 us at 80, waiting on latencies.
// At 40 rows per expert it issues on 67 % of the cycles, 5.4 thread instructions per gate or up weight and 7.4 per down weight
// (counters); turning a quant into fp16 is about 2.8 of these, the rest are waits that poll, the epilogue and the items' set-up.
//
// How a weight is rounded: the quants become exact fp16 integers q; the factors d * sc and dmin * m are carried as fp16 hi + lo
// pairs (hi the rounded product, lo the exact rest from one fma), and the weight is fma(q, dh, -mh) + fma(q, dl, -ml). Against
// one rounding of the f32 value this differs by at most one fp16 ulp, independently per weight (a single fp16 factor would put
// the same error on all 32 weights of a sub-block).
#include <algorithm>
#include <cstring>
#include <string>

#include "tcgen.cuh"
#include "wgemm.cuh"

namespace b200 {

namespace {

using namespace tc;

constexpr int WG_TILE = 128, WG_MAXPROB = 1025;
constexpr int WG_DQ0 = 2, WG_GROUPS = 3, WG_NA = 4, WG_ASLOT = 64;   // tensor memory: four half-block operands of 64 columns, then the accumulators
// Two accumulators (one of 256 columns). Items of few half blocks, the down projections', are bound by draining them: a group of four
// epilogue warps each (228 us against 198 for 2048 rows). The gated pair's items are four times as long, and there the registers of
// more warps cost more than they gave (288 us against 323 with a fourth dequantising group and six operands instead of the second
// accumulator): one group serves both.
template <int NT> __host__ __device__ constexpr int wg_nacc() { return NT == 256 ? 1 : 2; }
template <int NT, int EPI> __host__ __device__ constexpr int wg_epg() { return EPI == WG_SWIGLU ? 1 : wg_nacc<NT>(); }
template <int NT, int EPI> __host__ __device__ constexpr int wg_threads() { return 32 * (WG_DQ0 + 4 * WG_GROUPS + 4 * wg_epg<NT, EPI>() + 1); }

template <int TYPE> __host__ __device__ constexpr int wg_raw() { return WG_TILE * (TYPE == T_Q4_K ? 144 : TYPE == T_Q5_K ? 176 : TYPE == T_Q6_K ? 224 : 272); }
// stages of raw weights: 256 columns need the room for activations, whose 64 KB per super-block set the pace there (83 us against 76)
template <int NT> __host__ __device__ constexpr int wg_nr() { return NT == 256 ? 2 : 3; }
// A group has a half in two super-blocks of three. A wait by parity takes a stage's copy before last for the wanted one while the copy
// between them is on its way, so a group has to see every copy of the stages it waits on. With as many stages as groups all that
// it skips lies in one stage, which it never waits on; with another number every group waits for every super-block and gives its stage back.
template <int NT> __host__ __device__ constexpr bool wg_all_wait() { return wg_nr<NT>() != WG_GROUPS; }
__host__ __device__ constexpr uint32_t wg_half(uint32_t it, uint32_t grp) { return (grp + (WG_GROUPS - 2) * it) % WG_GROUPS; }   // group grp's half of super-block `it`; none if above 1
__host__ __device__ constexpr bool wg_sees_all(int nr, bool all_wait) {
  for (int g = 0; g < WG_GROUPS; g++)
    for (int it = nr; it < nr + nr * WG_GROUPS; it++)
      if (!all_wait && wg_half(it, g) < 2 && wg_half(it - nr, g) > 1) return false;
  return true;
}
template <int NT> __host__ __device__ constexpr int wg_xc() { return NT == 256 ? 1 : 2; }   // chunks of 64 elements per activation stage
template <int TYPE, int NT> __host__ __device__ constexpr int wg_nx() {                     // activation stages in what the raw stages leave
  return (204 * 1024 - wg_nr<NT>() * wg_raw<TYPE>()) / (NT * 128 * wg_xc<NT>()) < 8 ? (204 * 1024 - wg_nr<NT>() * wg_raw<TYPE>()) / (NT * 128 * wg_xc<NT>()) : 8;
}

__device__ __forceinline__ uint32_t h2c(float v) {
  __half2 h = __float2half2_rn(v);
  return *reinterpret_cast<uint32_t*>(&h);
}
constexpr uint32_t SIGN2 = 0x80008000u;
// four bytes of 0..63 -> two half2 of the exact integers less `off` (1024 and the format's centre)
__device__ __forceinline__ void bytes_h2(uint32_t w, uint32_t off, uint32_t& p01, uint32_t& p23) {
  p01 = hadd2_u(__byte_perm(w, 0x64646464u, 0x4140), off);
  p23 = hadd2_u(__byte_perm(w, 0x64646464u, 0x4342), off);
}

// Half a super-block (128 elements) of one row: read from its ring stage, then formed 32 elements (16 columns) at a time.
template <int TYPE> struct HalfBlock;

template <int TYPE> struct HalfBlockK4 {
  uint4 hdr, q[4], f[2];
  __device__ __forceinline__ void load(const uint8_t* raw, int row, int half, int) {
    constexpr int BLK = TYPE == T_Q4_K ? 144 : 176;
    const uint8_t* b = raw + row * BLK;
    hdr = lds128(b);
    if constexpr (TYPE == T_Q5_K) { f[0] = lds128(b + 16); f[1] = lds128(b + 32); }
#pragma unroll
    for (int i = 0; i < 4; i++) q[i] = lds128(b + BLK - 128 + 64 * half + 16 * i);
  }
  template <class Put> __device__ __forceinline__ void form(int half, Put put) const {
    // 6-bit scales and mins of the half's four sub-blocks (gguf/dequant.go:238-243)
    const uint32_t sc = half ? (hdr.w & 0x0F0F0F0Fu) | ((hdr.y >> 2) & 0x30303030u) : hdr.y & 0x3F3F3F3Fu;
    const uint32_t mn = half ? ((hdr.w >> 4) & 0x0F0F0F0Fu) | ((hdr.z >> 2) & 0x30303030u) : hdr.z & 0x3F3F3F3Fu;
    const uint32_t d = __byte_perm(hdr.x, 0, 0x1010), nd = __byte_perm(hdr.x, 0, 0x3232) ^ SIGN2, m1024 = h2c(-1024.f);
    const uint32_t fw[8] = {f[0].x, f[0].y, f[0].z, f[0].w, f[1].x, f[1].y, f[1].z, f[1].w};
#pragma unroll
    for (int gi = 0; gi < 2; gi++) {             // 64 elements: low nibbles of 32 bytes, then their high nibbles
      uint32_t s2, s2b, n2, n2b;
      bytes_h2(sc, m1024, s2, s2b); bytes_h2(mn, m1024, n2, n2b);
      if (gi) { s2 = s2b; n2 = n2b; }
      const uint32_t dh = hmul2_u(d, s2), dl = hfma2_u(d, s2, dh ^ SIGN2), nh = hmul2_u(nd, n2), nl = hfma2_u(nd, n2, nh ^ SIGN2);
      const uint32_t w[8] = {q[2 * gi].x, q[2 * gi].y, q[2 * gi].z, q[2 * gi].w, q[2 * gi + 1].x, q[2 * gi + 1].y, q[2 * gi + 1].z, q[2 * gi + 1].w};
#pragma unroll
      for (int hi = 0; hi < 2; hi++) {
        const uint32_t sel = hi ? 0x3232 : 0x1010;
        const uint32_t DH = __byte_perm(dh, 0, sel), DL = __byte_perm(dl, 0, sel), NH = __byte_perm(nh, 0, sel), NL = __byte_perm(nl, 0, sel);
        uint32_t out[16];
#pragma unroll
        for (int i = 0; i < 8; i++) {
          uint32_t a, b;
          if constexpr (TYPE == T_Q4_K) {
            if (hi) {                            // 16 q: (1024 + 16 q) / 16 - 64
              const uint32_t v = w[i] & 0xF0F0F0F0u;
              a = hfma2_u(__byte_perm(v, 0x64646464u, 0x4140), h2c(0.0625f), h2c(-64.f)); b = hfma2_u(__byte_perm(v, 0x64646464u, 0x4342), h2c(0.0625f), h2c(-64.f));
            } else {
              bytes_h2(w[i] & 0x0F0F0F0Fu, m1024, a, b);
            }
          } else {                               // fifth bits: bit 2 G of a byte belongs to its low nibble, the next to its high one
            const uint32_t fb = fw[i] >> (4 * half + 2 * gi);
            bytes_h2(hi ? ((w[i] >> 4) & 0x0F0F0F0Fu) | ((fb & 0x02020202u) << 3) : (w[i] & 0x0F0F0F0Fu) | ((fb & 0x01010101u) << 4), m1024, a, b);
          }
          out[2 * i] = hadd2_u(hfma2_u(a, DH, NH), hfma2_u(a, DL, NL));
          out[2 * i + 1] = hadd2_u(hfma2_u(b, DH, NH), hfma2_u(b, DL, NL));
        }
        put(2 * gi + hi, out);
      }
    }
  }
};
template <> struct HalfBlock<T_Q4_K> : HalfBlockK4<T_Q4_K> {};
template <> struct HalfBlock<T_Q5_K> : HalfBlockK4<T_Q5_K> {};

template <> struct HalfBlock<T_Q6_K> {           // planes: ql (128-byte swizzle) | qh (64-byte swizzle) | scales | the 16 bytes that hold d
  uint4 ql[4], qh[2];
  uint2 sc;
  float d;
  __device__ __forceinline__ void load(const uint8_t* raw, int row, int half, int d_off) {
#pragma unroll
    for (int i = 0; i < 4; i++) ql[i] = lds128(raw + row * 128 + (((4 * half + i) ^ (row & 7)) << 4));
#pragma unroll
    for (int i = 0; i < 2; i++) qh[i] = lds128(raw + 16384 + row * 64 + (((2 * half + i) ^ ((row >> 1) & 3)) << 4));
    sc = *reinterpret_cast<const uint2*>(raw + 24576 + row * 16 + 8 * half);
    d = __half2float(*reinterpret_cast<const __half*>(raw + 26624 + row * 16 + d_off));
  }
  template <class Put> __device__ __forceinline__ void form(int, Put put) const {
    const uint32_t m1056 = h2c(-1056.f);
    const uint32_t lw[16] = {ql[0].x, ql[0].y, ql[0].z, ql[0].w, ql[1].x, ql[1].y, ql[1].z, ql[1].w, ql[2].x, ql[2].y, ql[2].z, ql[2].w, ql[3].x, ql[3].y, ql[3].z, ql[3].w};
    const uint32_t hw[8] = {qh[0].x, qh[0].y, qh[0].z, qh[0].w, qh[1].x, qh[1].y, qh[1].z, qh[1].w};
#pragma unroll
    for (int c = 0; c < 4; c++) {                // quarter c: bytes 32 (c & 1) .. of ql, low or high nibbles; scale per 16 elements
      uint32_t out[16];
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const uint32_t word = (c >> 1) ? sc.y : sc.x;
        const float v = __fmul_rn(d, (float)(int)(int8_t)((word >> (8 * (2 * (c & 1) + (i >> 2)))) & 0xFF));
        const __half hh = __float2half_rn(v);
        const uint32_t ds = h2c(__half2float(hh)), dl = h2c(v - __half2float(hh));
        const uint32_t nib = (c >= 2 ? lw[8 * (c & 1) + i] >> 4 : lw[8 * (c & 1) + i]) & 0x0F0F0F0Fu;
        uint32_t a, b;
        bytes_h2(nib | (((hw[i] >> (2 * c)) & 0x03030303u) << 4), m1056, a, b);
        out[2 * i] = hfma2_u(a, ds, hmul2_u(a, dl)); out[2 * i + 1] = hfma2_u(b, ds, hmul2_u(b, dl));
      }
      put(c, out);
    }
  }
};
template <> struct HalfBlock<T_Q8_0> {           // planes: int8 quants in two 128-byte-swizzled boxes | eight fp16 d
  uint4 q[8];
  uint2 d;
  __device__ __forceinline__ void load(const uint8_t* raw, int row, int half, int) {
#pragma unroll
    for (int i = 0; i < 8; i++) q[i] = lds128(raw + half * 16384 + row * 128 + ((i ^ (row & 7)) << 4));
    d = *reinterpret_cast<const uint2*>(raw + 32768 + row * 16 + 8 * half);
  }
  template <class Put> __device__ __forceinline__ void form(int, Put put) const {
    const uint32_t m1152 = h2c(-1152.f);         // sign bit flipped: b + 128, plus the 1024
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const uint32_t ds = __byte_perm(c >> 1 ? d.y : d.x, 0, c & 1 ? 0x3232 : 0x1010);
      const uint32_t w[8] = {q[2 * c].x, q[2 * c].y, q[2 * c].z, q[2 * c].w, q[2 * c + 1].x, q[2 * c + 1].y, q[2 * c + 1].z, q[2 * c + 1].w};
      uint32_t out[16];
#pragma unroll
      for (int i = 0; i < 8; i++) {
        uint32_t a, b;
        bytes_h2(w[i] ^ 0x80808080u, m1152, a, b);
        out[2 * i] = hmul2_u(a, ds); out[2 * i + 1] = hmul2_u(b, ds);
      }
      put(c, out);
    }
  }
};

__device__ __forceinline__ bool bar_and(int id, int threads, bool v) {
  uint32_t r;
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\nbarrier.cta.red.and.pred q, %2, %3, p;\nselp.u32 %0, 1, 0, q;\n}" : "=r"(r) : "r"((uint32_t)v), "r"(id), "r"(threads) : "memory");
  return r != 0;
}

struct Item { int expert, cnt, x_row, y_row, nt, ks; };

template <int TYPE, int NT, int EPI>
__global__ void __launch_bounds__(wg_threads<NT, EPI>(), 1) wgemm_kernel(const __grid_constant__ WGemmMaps maps, const WGemmParams p) {
  constexpr bool PAIR = EPI == WG_SWIGLU;
  constexpr int TROWS = PAIR ? 64 : 128;             // output rows of a tile
  constexpr int NR = wg_nr<NT>(), NX = wg_nx<TYPE, NT>(), RAW = wg_raw<TYPE>(), XC = wg_xc<NT>(), XST = NT * 128 * XC;
  constexpr int NACC = wg_nacc<NT>(), EPG = wg_epg<NT, EPI>(), EP0 = WG_DQ0 + 4 * WG_GROUPS, XW = EP0 + 4 * EPG, ACC = WG_NA * WG_ASLOT;
  static_assert(NX >= 2, "two activation stages at least");
  static_assert(wg_sees_all(NR, wg_all_wait<NT>()), "a group would wait on a stage whose copy before last it has not seen");
  extern __shared__ uint8_t wg_smem[];
  uint8_t* raw0 = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(wg_smem) + 1023) & ~(uintptr_t)1023);
  uint8_t* x0 = raw0 + NR * RAW;
  __shared__ __align__(8) uint64_t r_full[NR], r_empty[NR], x_full[NX], x_empty[NX], a_full[WG_NA], a_empty[WG_NA], c_full[NACC], c_empty[NACC];
  __shared__ float ex[PAIR ? 2 * 128 * 17 : 1];
  __shared__ int stile[WG_MAXPROB + 1];              // activation tiles before each problem (exclusive scan)
  __shared__ uint32_t tmem_sm;
  __shared__ volatile int failed;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (int s = 0; s < NR; s++) { mbar_init(&r_full[s], 1); mbar_init(&r_empty[s], wg_all_wait<NT>() ? 4 * WG_GROUPS : 8); }
    for (int s = 0; s < NX; s++) { mbar_init(&x_full[s], 1); mbar_init(&x_empty[s], 1); }
    for (int s = 0; s < WG_NA; s++) { mbar_init(&a_full[s], 4); mbar_init(&a_empty[s], 1); }
    for (int s = 0; s < NACC; s++) { mbar_init(&c_full[s], 1); mbar_init(&c_empty[s], 4); }
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
  const int nb = p.K / 256, n_tiles = (p.N + TROWS - 1) / TROWS;
  pdl_wait();
  pdl_launch();
  // Items: (problem, activation tile, part of K, weight-row tile), the weight tile fastest, over the tiles the problems really
  // have: a scan of ceil(count / NT) per problem turns an item index into its problem by bisection.
  const int n_prob = p.problems != nullptr ? p.n_problems : 1;
  if (p.problems == nullptr) {
    if (tid == 0) { stile[0] = 0; stile[1] = (p.one.count + NT - 1) / NT; }
  } else if (warp == 0) {
    const int per = (n_prob + 31) / 32;
    int c = 0;
    for (int i = 0; i < per; i++) { const int e = lane * per + i; if (e < n_prob) c += (p.problems[e].count + NT - 1) / NT; }
    int cs = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int up = __shfl_up_sync(0xffffffffu, cs, o); if (lane >= o) cs += up; }
    int run = cs - c;
    for (int i = 0; i < per; i++) { const int e = lane * per + i; if (e < n_prob) { stile[e] = run; run += (p.problems[e].count + NT - 1) / NT; } }
    if (lane == 31) stile[n_prob] = cs;
  }
  __syncthreads();
  const int total = stile[n_prob] * p.ksplit * n_tiles;
  // A warp works its CTA's next 32 items out at once, one per lane, and takes them by shuffles.
  Item mine{};
  auto item = [&](int n) {
    if ((n & 31) == 0) {
      const int64_t idx = blockIdx.x + (int64_t)(n + lane) * gridDim.x;
      if (idx < total) {
        const int v = (int)idx / n_tiles, tile = v / p.ksplit;
        int lo = 0, hi = n_prob - 1;                 // the last problem whose first tile is not after `tile`
        while (lo < hi) { const int mid = (lo + hi + 1) >> 1; if (stile[mid] <= tile) lo = mid; else hi = mid - 1; }
        const GemmProblem pr = p.problems != nullptr ? p.problems[lo] : p.one;
        const int c0 = (tile - stile[lo]) * NT;
        mine = Item{pr.expert, min(NT, pr.count - c0), pr.x_row0 + c0, pr.y_row0 + c0, (int)idx - v * n_tiles, v - tile * p.ksplit};
      }
    }
    const int l = n & 31;
    auto from = [&](int v) { return __shfl_sync(0xffffffffu, v, l); };
    return Item{from(mine.expert), from(mine.cnt), from(mine.x_row), from(mine.y_row), from(mine.nt), from(mine.ks)};
  };
  const int n_items = blockIdx.x < total ? (total - 1 - blockIdx.x) / gridDim.x + 1 : 0;
  auto sb_begin = [&](int ks) { return ks * nb / p.ksplit; };
  auto give_up = [&]() { report_error(p.err); failed = 1; };
  auto stopped = [&]() { return __any_sync(0xffffffffu, failed); };

  if (warp == 0) {
    // ---- weights --------------------------------------------------------------------------------
    uint32_t it = 0;
    for (int n = 0; n < n_items && !stopped(); n++) {
      const Item t = item(n);
      const int row = (t.expert > 0 ? t.expert * p.N : 0) + t.nt * TROWS, sb1 = sb_begin(t.ks + 1);
      const WMap &wa = t.expert >= 0 ? maps.w : maps.ws, &wb = t.expert >= 0 ? maps.w2 : maps.ws2;
      for (int sb = sb_begin(t.ks); sb < sb1; sb++, it++) {
        const int s = it % NR;
        if (!warp_wait(&r_empty[s], ((it / NR) & 1) ^ 1)) { give_up(); break; }
        if (elect_one()) {
          mbar_expect_tx(&r_full[s], RAW);
#pragma unroll
          for (int h = 0; h < (PAIR ? 2 : 1); h++) {
            const CUtensorMap* m = reinterpret_cast<const CUtensorMap*>(h ? &wb : &wa);
            uint8_t* d = raw0 + s * RAW;
            auto box = [&](int map, int pitch, int base, int col) { tma_box(d + base + h * 64 * pitch, m + map, col, row, &r_full[s]); };
            if constexpr (TYPE == T_Q4_K) box(0, 144, 0, sb * 144);
            else if constexpr (TYPE == T_Q5_K) box(0, 176, 0, sb * 176);
            else if constexpr (TYPE == T_Q6_K) { box(0, 128, 0, sb * 128); box(1, 64, 16384, nb * 128 + sb * 64); box(2, 16, 24576, nb * 192 + sb * 16); box(2, 16, 26624, (nb * 208 + sb * 2) & ~15); }
            else { box(0, 128, 0, sb * 256); box(0, 128, 16384, sb * 256 + 128); box(1, 16, 32768, p.K + sb * 16); }
          }
        }
        __syncwarp();
      }
    }
    if (failed)                                      // leave only once the copies in flight have landed
      for (uint32_t k = it > (uint32_t)NR ? it - NR : 0; k < it; k++) mbar_wait(&r_full[k % NR], (k / NR) & 1);
  } else if (warp == XW) {
    // ---- activation rows ------------------------------------------------------------------------
    uint32_t it = 0;
    for (int n = 0; n < n_items && !stopped(); n++) {
      const Item t = item(n);
      const int boxes = (t.cnt + 63) / 64, c1 = 4 * sb_begin(t.ks + 1);
      for (int c = 4 * sb_begin(t.ks); c < c1; c += XC, it++) {
        const int s = it % NX;
        if (!warp_wait(&x_empty[s], ((it / NX) & 1) ^ 1)) { give_up(); break; }
        if (elect_one()) {
          mbar_expect_tx(&x_full[s], boxes * 8192 * XC);
#pragma unroll
          for (int k = 0; k < XC; k++)
            for (int b = 0; b < boxes; b++) tma_box(x0 + s * XST + k * (NT * 128) + b * 8192, reinterpret_cast<const CUtensorMap*>(&maps.x), (c + k) * 64, t.x_row + 64 * b, &x_full[s]);
        }
        __syncwarp();
      }
    }
    if (failed)
      for (uint32_t k = it > (uint32_t)NX ? it - NX : 0; k < it; k++) mbar_wait(&x_full[k % NX], (k / NX) & 1);
  } else if (warp == 1) {
    // ---- tensor core ------------------------------------------------------------------------------
    uint32_t hx = 0, xi = 0, ci = 0;
    bool ok = true;
    for (int n = 0; n < n_items && ok && !stopped(); n++, ci++) {
      const Item t = item(n);
      const int n_half = 2 * (sb_begin(t.ks + 1) - sb_begin(t.ks));
      const uint32_t id = idesc_n((t.cnt + 15) & ~15);
      const uint32_t acc = tm + ACC + (ci % NACC) * NT;
      if (!warp_wait(&c_empty[ci % NACC], ((ci / NACC) & 1) ^ 1)) { give_up(); break; }
      for (int h = 0; h < n_half && ok; h++, hx++) {
        const int as = hx % WG_NA;
#pragma unroll
        for (int c = 0; c < 2; c += XC, xi++) {
          // even lanes wait for the weights, odd ones for the activations: one latency of a ready barrier instead of two
          const int xs = xi % NX;
          const bool wa = c == 0 && (lane & 1) == 0;
          ok = __all_sync(0xffffffffu, mbar_wait(wa ? &a_full[as] : &x_full[xs], wa ? (hx / WG_NA) & 1 : (xi / NX) & 1));
          if (!ok) { give_up(); break; }
          fence_after();
          if (elect_one()) {
            const uint64_t bd = desc_sw128(smem_addr(x0 + xs * XST));
#pragma unroll
            for (int k = 0; k < 4 * XC; k++) mma_ts(acc, tm + as * WG_ASLOT + 32 * c + 8 * k, bd + (k >> 2) * (NT * 8) + 2 * (k & 3), id, (h | c | k) != 0);
            commit(&x_empty[xs]);
            if (c + XC == 2) commit(&a_empty[as]);
            if (c + XC == 2 && h == n_half - 1) commit(&c_full[ci % NACC]);
          }
          __syncwarp();
        }
      }
    }
  } else if (warp < EP0) {
    // ---- dequantisation ---------------------------------------------------------------------------
    const int grp = (warp - WG_DQ0) >> 2, q = warp & 3, row = q * 32 + lane;
    const uint32_t lane_base = tm + ((uint32_t)(q * 32) << 16);
    uint32_t it = 0;                                 // super-blocks of all items
    bool ok = true;
    for (int n = 0; n < n_items && ok && !stopped(); n++) {
      const Item t = item(n);
      const int sb0 = sb_begin(t.ks), sb1 = sb_begin(t.ks + 1);
      for (int sb = sb0; sb < sb1; sb++, it++) {
        const int s = it % NR, half = wg_half(it, grp);
        if (half > 1 && !wg_all_wait<NT>()) continue;
        if (!warp_wait(&r_full[s], (it / NR) & 1)) { give_up(); ok = false; break; }
        if (half > 1) {
          if (lane == 0) arrive(&r_empty[s]);
          continue;
        }
        const uint32_t hx = 2 * it + half;
        const int as = hx % WG_NA;
        HalfBlock<TYPE> v;
        v.load(raw0 + s * RAW, row, half, (nb * 208 + sb * 2) & 15);
        __syncwarp();
        if (lane == 0) arrive(&r_empty[s]);
        bool waited = false;
        v.form(half, [&](int sub, const uint32_t (&out)[16]) {
          if (!waited) {
            ok = warp_wait(&a_empty[as], ((hx / WG_NA) & 1) ^ 1);
            fence_after();
            waited = true;
          }
          if (ok) tmem_st16(lane_base + as * WG_ASLOT + 16 * sub, out);
        });
        if (!ok) { give_up(); break; }
        tmem_st_wait();
        fence_before();
        __syncwarp();
        if (lane == 0) arrive(&a_full[as]);
      }
    }
  } else if (warp < XW) {
    // ---- epilogue -----------------------------------------------------------------------------------
    const int q = warp & 3, eg = (warp - EP0) >> 2;    // with two groups, group eg drains accumulator eg
    const uint32_t lane_base = tm + ((uint32_t)(q * 32) << 16) + ACC;
    int exb = 0;
    for (int n = 0; n < n_items; n++) {
      const Item t = item(n);
      if (EPG == 2 && (n & 1) != eg) continue;
      const uint32_t ci = n;
      const int cnt = t.cnt;
      // output row of column c0 + lane, fetched by the lanes side by side ahead of its use and handed round by shuffles
      auto row_of = [&](int c0) {
        const int r = t.y_row + min(c0 + lane, cnt - 1);
        return p.y_rows != nullptr ? __ldg(p.y_rows + r) : r;
      };
      int next_row = row_of(0);
      bool ok = warp_wait(&c_full[ci % NACC], (ci / NACC) & 1);
      if (!ok) give_up();
      if constexpr (PAIR) ok = bar_and(1, 128, ok);   // the four warps meet again below: all leave or none
      if (!ok) break;
      fence_after();
#pragma unroll 1
      for (int c0 = 0; c0 < cnt; c0 += 32) {
        const int my_row = next_row;
        uint32_t v[32];
        tmem_ld16(lane_base + (ci % NACC) * NT + c0, *reinterpret_cast<uint32_t (*)[16]>(v));
        tmem_ld16(lane_base + (ci % NACC) * NT + c0 + 16, *reinterpret_cast<uint32_t (*)[16]>(v + 16));
        tmem_ld_wait();
        if (c0 + 32 < cnt) {
          next_row = row_of(c0 + 32);
        } else {                                     // the accumulator is free for the item after the next
          fence_before();
          __syncwarp();
          if (lane == 0) arrive(&c_empty[ci % NACC]);
        }
        const int live = min(32, cnt - c0);
        if constexpr (PAIR) {
          // SwiGLU (shaders/llm_moe_gemv.comp:777-781): the gate rows' warps take the first 16 columns and get the up values,
          // the up rows' warps take the others and get the gates
          const int up = q >> 1, r = (q & 1) * 32 + lane, orow = t.nt * 64 + r;
          float* e = ex + exb * (128 * 17);
          exb ^= 1;
#pragma unroll
          for (int i = 0; i < 16; i++) e[((up ^ 1) * 64 + r) * 17 + i] = __uint_as_float(up ? v[i] : v[16 + i]);
          asm volatile("bar.sync 1, 128;" ::: "memory");
#pragma unroll
          for (int i = 0; i < 16; i++) {
            const float o = e[(up * 64 + r) * 17 + i], own = __uint_as_float(up ? v[16 + i] : v[i]);
            const float gv = up ? o : own, uv = up ? own : o;
            const int yr = __shfl_sync(0xffffffffu, my_row, up * 16 + i);
            if (up * 16 + i < live && orow < p.N) p.y16[(uint64_t)(uint32_t)yr * (uint32_t)p.ldy + orow] = __float2half_rn(gv * sigmoid_acc(gv) * uv);
          }
        } else {
          const int orow = t.nt * 128 + q * 32 + lane;
          float* y = p.y + (int64_t)t.ks * p.plane + orow;
#pragma unroll
          for (int i = 0; i < 32; i++) {
            const int yr = __shfl_sync(0xffffffffu, my_row, i);
            if (i < live && orow < p.N) y[(uint64_t)(uint32_t)yr * (uint32_t)p.ldy] = __uint_as_float(v[i]);
          }
        }
      }
    }
  }
  fence_before();
  __syncthreads();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tm) : "memory");
}

template <int TYPE, int NT, int EPI>
int launch_t(const WGemmParams& p, const WGemmMaps& maps, bool pdl, cudaStream_t st) {
  auto kernel = wgemm_kernel<TYPE, NT, EPI>;
  constexpr int smem = wg_nr<NT>() * wg_raw<TYPE>() + wg_nx<TYPE, NT>() * NT * 128 * wg_xc<NT>() + 1024;
  B200_ONCE_PER_DEVICE(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const int sms = sm_count_current();
  if (sms <= 0) return ECUDA;
  const int n_tiles = (p.N + (EPI == WG_SWIGLU ? 63 : 127)) / (EPI == WG_SWIGLU ? 64 : 128);
  const int64_t total = ((int64_t)(p.max_count + NT - 1) / NT + (p.problems != nullptr ? p.n_problems : 0)) * n_tiles * p.ksplit;   // every problem rounds up once at most
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)std::max<int64_t>(1, std::min<int64_t>(total, sms))); cfg.blockDim = dim3(wg_threads<NT, EPI>()); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = pdl ? 1 : 0;
  B200_CUDA(cudaLaunchKernelEx(&cfg, kernel, maps, p));
  return OK;
}
template <int TYPE>
int launch_n(int epi, int cols, const WGemmParams& p, const WGemmMaps& maps, bool pdl, cudaStream_t st) {
  if (epi == WG_STORE) {
    if (cols == 64) return launch_t<TYPE, 64, WG_STORE>(p, maps, pdl, st);
    if (cols == 128) return launch_t<TYPE, 128, WG_STORE>(p, maps, pdl, st);
    if (cols == 256) return launch_t<TYPE, 256, WG_STORE>(p, maps, pdl, st);
  } else if constexpr (TYPE != T_Q8_0) {
    if (cols == 64) return launch_t<TYPE, 64, WG_SWIGLU>(p, maps, pdl, st);
    if (cols == 128) return launch_t<TYPE, 128, WG_SWIGLU>(p, maps, pdl, st);
  }
  set_error("wgemm: tiles have 64, 128 or 256 columns (128 at most for the gated pair)");
  return EINVAL_;
}

}  // namespace

bool wgemm_type(uint32_t type) { return type == T_Q4_K || type == T_Q5_K || type == T_Q6_K || type == T_Q8_0; }

// 128 columns cost the tensor core what fewer cost; 256 cost twice that and halve the dequantisation per column, which pays
// once the device is full of them
int wgemm_cols(int M, int N) {
  const int tiles = (N + 127) / 128;
  return M <= 64 ? 64 : tiles * ((M + 255) / 256) >= 3 * 148 / 2 ? 256 : 128;
}
int wgemm_ksplit(int M, int N, int K) {
  const int units = (N + 127) / 128 * ((M + 127) / 128);
  return std::max(1, std::min(std::min(148 / std::max(units, 1), K / 512), 8));
}

int make_wmap(uint32_t type, const uint8_t* w, int64_t rows, int64_t stride, int box_rows, WMap* out) {
  auto u8 = [&](int inner, CUtensorMapSwizzle swizzle, TMap* m) { return encode_2d(CU_TENSOR_MAP_DATA_TYPE_UINT8, w, stride, rows, stride, inner, box_rows, swizzle, m); };
  switch (type) {
    case T_Q4_K: return u8(144, CU_TENSOR_MAP_SWIZZLE_NONE, &out->m[0]);
    case T_Q5_K: return u8(176, CU_TENSOR_MAP_SWIZZLE_NONE, &out->m[0]);
    case T_Q6_K:
      B200_TRY(u8(128, CU_TENSOR_MAP_SWIZZLE_128B, &out->m[0]));
      B200_TRY(u8(64, CU_TENSOR_MAP_SWIZZLE_64B, &out->m[1]));
      return u8(16, CU_TENSOR_MAP_SWIZZLE_NONE, &out->m[2]);
    case T_Q8_0:
      B200_TRY(u8(128, CU_TENSOR_MAP_SWIZZLE_128B, &out->m[0]));
      return u8(16, CU_TENSOR_MAP_SWIZZLE_NONE, &out->m[1]);
  }
  set_error("wgemm: weight type has no kernel (Q4_K, Q5_K, Q6_K, Q8_0)");
  return EINVAL_;
}

int launch_wgemm(uint32_t type, int epi, int cols, const WGemmParams& p, const WGemmMaps& maps, bool pdl, cudaStream_t st) {
  if (p.K % 256 != 0 || p.K <= 0 || p.N <= 0) { set_error("wgemm: row length must be a multiple of 256"); return EINVAL_; }
  if (p.ksplit < 1 || p.ksplit > p.K / 256 || (p.ksplit > 1 && (p.problems != nullptr || epi != WG_STORE))) { set_error("wgemm: only a single plain projection can be cut along K"); return EINVAL_; }
  if (p.problems != nullptr && (p.n_problems < 1 || p.n_problems > WG_MAXPROB || p.N % (epi == WG_SWIGLU ? 64 : 128) != 0)) { set_error("wgemm: problem list outside its limits"); return EINVAL_; }
  switch (type) {
    case T_Q4_K: return launch_n<T_Q4_K>(epi, cols, p, maps, pdl, st);
    case T_Q5_K: return launch_n<T_Q5_K>(epi, cols, p, maps, pdl, st);
    case T_Q6_K: return launch_n<T_Q6_K>(epi, cols, p, maps, pdl, st);
    case T_Q8_0: return launch_n<T_Q8_0>(epi, cols, p, maps, pdl, st);
  }
  set_error("wgemm: weight type has no kernel (Q4_K, Q5_K, Q6_K, Q8_0)");
  return EINVAL_;
}

}  // namespace b200
