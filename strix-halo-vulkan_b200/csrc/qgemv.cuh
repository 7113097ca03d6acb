// Fused K-quant dequant "GEMV" for 1..8 activation rows per launch column-tile.
//
// y[n][r] = sum_k W[r][k] * x16[n][k], W read as the checkpoint's own K-quant blocks.
//
// Replaces the reference's dense decode projection and decode expert FFN kernels
// (shaders/llm_gemv.comp:116-263, shaders/llm_moe_gemv.comp:586-786), keeping their
// arithmetic: activations staged as fp16, weights never rounded, f32 accumulation.
//
// Design (B200): a CTA of 8 warps owns 16-row weight tiles; its warps split K by
// super-block, and each brings its own 16 x 256 weights ahead of the arithmetic. The quants
// enter mma.sync.m16n8k16 as fp16 subnormals, the bare integers, one mask per pair; the <= 8
// activation rows are the B-fragments, read from shared memory; sub-block scales are applied
// to the f32 result of a sub-block's two mma steps, d and the min term
// dmin * sum_s m_s * sum_{k in s} x_k (itself one more mma over the eight sub-block sums,
// split into fp16 hi + lo parts) per super-block. What bounds it is instructions and the
// chain from the producer's rows to the partial sums, not DRAM: with the scale multiplied
// into every fragment, one copying warp and a barrier per tile, a single row's largest
// projection took 12 us of its layer, now 10 of 38.
// Partial sums of the K-slices are added in warp order (deterministic), and a column's
// result depends on that column alone, so a batched pass equals each row stepped alone.
//
// Q6_K has no integer sub-scale small enough: sc*(q-32) can reach 4064 and is rounded to
// fp16 above 2048 (relative error <= 2^-12 on those weights).
#pragma once
#include "common.cuh"
#include "router.cuh"
#include "tgemm.cuh"
#ifdef __CUDACC__
#include <cooperative_groups.h>
#endif

namespace b200 {

constexpr int QG_WARPS = 8;
constexpr int QG_THREADS = QG_WARPS * 32;
constexpr int QG_MAXCOLS = 8;
constexpr int QG_FUSED_ROWS = 8;       // passes of at most this many rows fold norms into the staging of the consumers
constexpr int QG_FUSED_MAX_K = 2048;   // ... of residual rows up to this long

enum { EPI_STORE = 0, EPI_RESID = 1, EPI_SWIGLU = 2 };
enum { PRO_F16 = 0, PRO_NORM = 1 };
constexpr int SS_LD = 512;  // partial sums of squares kept per activation row

// Where a pass of few rows leaves its results, read on the device so that a replayed pass can change them: host memory the device can
// write (or the graph's own device buffer), and the residual rows of the columns from h_first on (nullptr: not wanted).
struct PassOut { float* logits; float* h; int h_first, pad; };

struct QGemvParams {
  // weights: up to 4 row segments of one fused projection (same type and K)
  const uint8_t* w[4];
  const uint8_t* w2[4];      // DUAL: the second tensor (up), same shape as w
  int seg_end[4];            // exclusive end row of each segment
  int nseg;
  int64_t stride;            // bytes per row
  int K, N;
  // grouped (per-expert) mode: entries[e] = {expert (<0: shared expert, uses ws/ws2), col_off, col_cnt, 0}
  const int4* entries;
  const int* n_entries;
  const int* cols;           // column -> x / y row ids
  int64_t expert_stride;     // bytes between consecutive experts
  const uint8_t* ws;         // shared expert weights (grouped mode)
  const uint8_t* ws2;
  int x_div;                 // grouped: x row = cols[c] / x_div
  // plain mode columns: rows [ztile*8, ztile*8+8) of M
  int M;
  int xcols;                 // columns the shared-memory layout is sized for (1..8)
  int nstage;                // weight pipeline stages in shared memory (1..QG_MAX_STAGES)
  int* err;                  // device error word: set when a bounded wait gives up
  Timeline tl;
  const int* row_ids;        // optional: plain mode column c reads row row_ids[c] and writes row c
  // activations. PRO_F16: fp16 rows in natural order. PRO_NORM: the f32 residual rows `hsrc`, normalised
  // while they are staged: x = fp16(h * gamma / sqrt(sum(ss_in[row][0..ss_n)) / K + eps)); the sums of
  // squares arrive as per-CTA partials from the kernel that wrote h, added in a fixed order
  const __half* x;
  int64_t ldx;
  const float* hsrc;
  const float* gamma;
  const float* ss_in;
  int ss_n;
  float eps;
  __half* xn_out;            // PRO_NORM: optional copy of the normalised rows, [.][K], written by CTA 0
  float* ss_out;             // STORE / RESID: optional partial sums of squares of the rows written, [.][SS_LD], part = tile of 16 rows
  const PassOut* out;        // the head of a pass of few rows: y and the residual copy come from here
  // epilogue
  float* y;                  // STORE / RESID: float [.][ldy]
  int64_t ldy;
  __half* y16;               // SWIGLU: half [.][ldy]
};

// Q4_K and Q5_K, plain mode: tensor maps of the row segments, boxes of 16 rows x one super-block (make_w_tensor_map)
struct QGemvMaps { TMap w[4]; };
// whether a launch reads its weights through QGemvMaps
__host__ __device__ constexpr bool qg_boxed(uint32_t type, bool grouped) { return !grouped && (type == T_Q4_K || type == T_Q5_K); }

__host__ __device__ inline int qg_xstride(int K) {
  int base = 2 * K + 16 * (K / 64);
  int pad = (64 - base % 128 + 128) % 128;
  return base + pad;
}
constexpr int QG_MAX_STAGES = 8;
constexpr size_t QG_SMEM_MAX = 222 * 1024;   // dynamic shared memory of a CTA that has its SM alone
// pitch of a weight row in shared memory (see mma_row), and bytes of one pipeline stage: the tiles one CTA works on per iteration
__host__ __device__ inline int64_t qg_pitch(uint32_t type, int64_t stride, bool grouped) { return type != T_Q6_K && grouped ? stride + 16 : stride; }
__host__ __device__ inline size_t qg_stage_bytes(int K, int64_t stride, bool dual) {
  const int nb = K / 256;
  const int wpt = nb >= 8 ? 8 : nb >= 4 ? 4 : nb >= 2 ? 2 : 1;
  return (size_t)(QG_WARPS / wpt) * 16 * (size_t)stride * (dual ? 2 : 1);
}
__host__ __device__ inline size_t qg_fixed_smem(int K, int xcols, bool dual) {
  size_t xs = (size_t)xcols * qg_xstride(K);
  size_t sx = (size_t)xcols * (K / 32) * 2 * sizeof(__half);  // hi and lo planes
  size_t red = (size_t)2 * QG_WARPS * 16 * 8 * sizeof(float);  // partial sums: two units of eight columns, or one of a pair of matrices
  return ((xs + ((sx + 15) & ~(size_t)15) + red) + 127) & ~(size_t)127;
}

// byte offset of activation element k inside a staged row: 4-groups hold [x0,x2,x1,x3]
// (the order the nibble unpack produces pairs in), 16 bytes of padding per 64 elements.
__device__ __forceinline__ int xs_off(int k) {
  int k4 = k & 3;
  int p = (k4 == 1) ? 2 : (k4 == 2) ? 1 : k4;
  return 2 * ((k & ~3) | p) + 16 * (k >> 6);
}

__device__ __forceinline__ uint4 ld_s128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ uint2 ld_s64(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}

__device__ __forceinline__ uint32_t half2_const(float v) {
  __half2 h = __float2half2_rn(v);
  return *reinterpret_cast<uint32_t*>(&h);
}

// ---- Q4_K, Q5_K -------------------------------------------------------------------------
// Block: d, dmin (fp16), 12 bytes of packed 6-bit (scale, min), for Q5_K 32 bytes of fifth bits, 128 bytes of nibbles
// (reference: gguf/dequant.go:238-318); 32 bytes of nibbles hold two sub-blocks, the even one low. Thread t of a quad takes
// bytes 8t .. 8t + 7 of each such group, so that one mma step lies within one sub-block.
// Quants enter the tensor core as they are: four or five bits below a half's exponent are a subnormal q * 2^-s, exactly,
// so a pair of weights costs one mask and no conversion, no multiply; the sub-block scale is applied to the f32 result of
// the sub-block's two mma steps, the 2^s (and the 16 of a high nibble left where it is) with the block scale.
// How far below matters: the tensor core aligns products by the operands' exponents and a subnormal's bits lie under its own, so at
// 2^-24 an mma has an error of 4.1e-7, at 2^-22 of 5e-8 and from 2^-20 on of 8e-9 (16 products of 0..15 with normal values). Q4_K
// takes 2^-22 and 2^-18 with one shift more per word than 2^-24 and 2^-20, Q5_K 2^-21.
// lo: sub-block 2G, hi: 2G + 1; of a word's four bytes the pairs are (0, 2) and (1, 3).
template <int TYPE>
__device__ __forceinline__ void unpack_word(uint32_t w, uint32_t fifth, int G, uint32_t& l02, uint32_t& l13, uint32_t& h02, uint32_t& h13) {
  if constexpr (TYPE == T_Q4_K) {
    const uint32_t even = w << 2, odd = w >> 6;
    l02 = even & 0x003C003Cu; h02 = even & 0x03C003C0u; l13 = odd & 0x003C003Cu; h13 = odd & 0x03C003C0u;
  } else {   // fifth bits: bit 2G of a byte belongs to its low nibble, bit 2G + 1 to the high one
    const uint32_t f = fifth >> (2 * G);
    const uint32_t lo = ((w << 3) & 0x78787878u) | ((f << 7) & 0x80808080u), hi = ((w >> 1) & 0x78787878u) | ((f << 6) & 0x80808080u);
    l02 = lo & 0x00F800F8u; l13 = (lo >> 8) & 0x00F800F8u; h02 = hi & 0x00F800F8u; h13 = (hi >> 8) & 0x00F800F8u;
  }
}
template <int TYPE> __device__ __forceinline__ constexpr float unit_scale() { return TYPE == T_Q4_K ? 4194304.f : 2097152.f; }   // 2^s of a low nibble
// D = A B, no accumulator in
__device__ __forceinline__ void mma16816_z(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// scales (bytes 2 pair, 2 pair + 1 of a word) of a low- and a high-nibble sub-block as f32
template <int TYPE>
__device__ __forceinline__ void sub_scales(uint32_t four, int pair, float (&s)[2]) {
  const uint32_t h2 = hadd2_u(__byte_perm(four, 0x64646464u, pair ? 0x4342 : 0x4140), half2_const(-1024.f));
  s[0] = h2f_lo(h2);
  s[1] = h2f_hi(TYPE == T_Q4_K ? hmul2_u(h2, half2_const(0.0625f)) : h2);
}

// two bytes (b0, b1) of each pair picked by sel -> half2(b0, b1), exact
__device__ __forceinline__ uint32_t mins_half2(uint32_t four, uint32_t sel) { return hadd2_u(__byte_perm(four, 0x64646464u, sel), half2_const(-1024.f)); }

// One super-block of the rows of mma rows g (at smem address ra) and g + 8 (rb), added to acc (C layout: [0], [1] row g, columns
// 2t, 2t + 1; [2], [3] row g + 8). x: this lane's column of the staged activations at the super-block (xs_off layout); sx0, sx1:
// its pairs of sub-block sums 2 (t / 2), + 1 and 4 + these, hi parts for even t and lo parts for odd t.
template <int TYPE>
__device__ __forceinline__ void k45_accumulate(float (&acc)[4], uint32_t ra, uint32_t rb, const uint8_t* x, uint32_t sx0, uint32_t sx1, int t) {
  constexpr int QOFF = TYPE == T_Q4_K ? 16 : 48;
  const uint4 h0 = ld_s128(ra), h1 = ld_s128(rb);
  // 6-bit scales of the two rows, four sub-blocks to a word (gguf/dequant.go:238-243)
  const uint32_t scl[2][2] = {{h0.y & 0x3F3F3F3Fu, (h0.w & 0x0F0F0F0Fu) | ((h0.y >> 2) & 0x30303030u)}, {h1.y & 0x3F3F3F3Fu, (h1.w & 0x0F0F0F0Fu) | ((h1.y >> 2) & 0x30303030u)}};
  uint2 f0 = make_uint2(0, 0), f1 = f0;
  if constexpr (TYPE == T_Q5_K) { f0 = ld_s64(ra + 16 + 8 * t); f1 = ld_s64(rb + 16 + 8 * t); }
  float a[4] = {0.f, 0.f, 0.f, 0.f};   // sub-block scale x (q . x), without d
#pragma unroll
  for (int G = 0; G < 4; G++) {
    const uint2 q0 = ld_s64(ra + QOFF + 32 * G + 8 * t), q1 = ld_s64(rb + QOFF + 32 * G + 8 * t);
    uint32_t al[2][4], ah[2][4];
    unpack_word<TYPE>(q0.x, f0.x, G, al[0][0], al[0][2], ah[0][0], ah[0][2]);
    unpack_word<TYPE>(q1.x, f1.x, G, al[0][1], al[0][3], ah[0][1], ah[0][3]);
    unpack_word<TYPE>(q0.y, f0.y, G, al[1][0], al[1][2], ah[1][0], ah[1][2]);
    unpack_word<TYPE>(q1.y, f1.y, G, al[1][1], al[1][3], ah[1][1], ah[1][3]);
    float s0[2], s1[2];
    sub_scales<TYPE>(scl[0][G >> 1], G & 1, s0);
    sub_scales<TYPE>(scl[1][G >> 1], G & 1, s1);
    const uint4 xl = *reinterpret_cast<const uint4*>(x + 144 * G + 16 * t), xh = *reinterpret_cast<const uint4*>(x + 144 * G + 64 + 16 * t);
    float C[4], D[4];
    mma16816_z(C, al[0], xl.x, xl.y); mma16816(C, al[1], xl.z, xl.w);
    mma16816_z(D, ah[0], xh.x, xh.y); mma16816(D, ah[1], xh.z, xh.w);
    a[0] = fmaf(s0[0], C[0], a[0]); a[1] = fmaf(s0[0], C[1], a[1]); a[2] = fmaf(s1[0], C[2], a[2]); a[3] = fmaf(s1[0], C[3], a[3]);
    a[0] = fmaf(s0[1], D[0], a[0]); a[1] = fmaf(s0[1], D[1], a[1]); a[2] = fmaf(s1[1], D[2], a[2]); a[3] = fmaf(s1[1], D[3], a[3]);
  }
  // min term: one mma over the eight sub-block sums, then the block scales
  const uint32_t sel = 0x4040u | (2 * (t >> 1)) | ((2 * (t >> 1) + 1) << 8);
  const uint32_t am[4] = {mins_half2(h0.z & 0x3F3F3F3Fu, sel), mins_half2(h1.z & 0x3F3F3F3Fu, sel), mins_half2(((h0.w >> 4) & 0x0F0F0F0Fu) | ((h0.z >> 2) & 0x30303030u), sel),
                          mins_half2(((h1.w >> 4) & 0x0F0F0F0Fu) | ((h1.z >> 2) & 0x30303030u), sel)};
  float Cm[4];
  mma16816_z(Cm, am, sx0, sx1);
  const float d0 = h2f_lo(h0.x) * unit_scale<TYPE>(), n0 = h2f_hi(h0.x), d1 = h2f_lo(h1.x) * unit_scale<TYPE>(), n1 = h2f_hi(h1.x);
  acc[0] = fmaf(-n0, Cm[0], fmaf(d0, a[0], acc[0])); acc[1] = fmaf(-n0, Cm[1], fmaf(d0, a[1], acc[1]));
  acc[2] = fmaf(-n1, Cm[2], fmaf(d1, a[2], acc[2])); acc[3] = fmaf(-n1, Cm[3], fmaf(d1, a[3], acc[3]));
}

// ---- Q6_K (row planes, see DTensor) ---------------------------------------------------
// Per block: ql[128], qh[64], 16 int8 scales, fp16 d (reference: gguf/dequant.go:331-356).
// Unit u = t (+4): half hf = u>>2, lh = (u>>1)&1, l0 = 16*(u&1): low nibbles are quarter lh,
// high nibbles quarter lh+2, of elements l0..l0+15; element k = 128*hf + 32*quarter + l.
struct Q6KRow {
  uint4 qla, qlb, qha, qhb, sc;
  uint32_t d;
};
__device__ __forceinline__ void q6k_issue(Q6KRow& r, const uint8_t* row, int nb, int blk, int t) {
  const uint8_t* ql = row + (size_t)blk * 128;
  const uint8_t* qh = row + (size_t)nb * 128 + (size_t)blk * 64;
  const uint8_t* sc = row + (size_t)nb * 192 + (size_t)blk * 16;
  const uint8_t* d = row + (size_t)nb * 208 + (size_t)blk * 2;
  r.qla = lds128(ql + 16 * t);
  r.qlb = lds128(ql + 64 + 16 * t);
  r.qha = lds128(qh + 16 * (t & 1));
  r.qhb = lds128(qh + 32 + 16 * (t & 1));
  r.sc = lds128(sc);
  r.d = *reinterpret_cast<const unsigned short*>(d);
}
__device__ __forceinline__ int q6_scale(const uint4& sc, int idx) {  // int8 scale idx of the block
  uint32_t w = idx < 4 ? sc.x : idx < 8 ? sc.y : idx < 12 ? sc.z : sc.w;
  return (int)(int8_t)((w >> (8 * (idx & 3))) & 0xFF);
}
__device__ __forceinline__ void q6_unpack_word(uint32_t w, uint32_t qh, int lh, uint32_t sc_lo2, uint32_t sc_hi2, uint32_t& lo02, uint32_t& lo13,
                                               uint32_t& hi02, uint32_t& hi13) {
  // 2-bit field of quarter c sits at bits 2c..2c+1 of the qh byte; move it to bits 4..5
  uint32_t rl = __funnelshift_r(qh, qh, (2 * lh - 4) & 31);
  uint32_t rh = __funnelshift_r(qh, qh, (2 * lh) & 31);  // quarter lh+2: (2*(lh+2) - 4)
  uint32_t lo = lop3_or_andb(w & 0x0F0F0F0Fu, rl, 0x30303030u);
  uint32_t hi = lop3_or_andb((w >> 4) & 0x0F0F0F0Fu, rh, 0x30303030u);
  const uint32_t off = half2_const(-1056.f);  // 1024 magic + 32 centre
  lo02 = hmul2_u(hadd2_u(__byte_perm(lo, 0x64646464u, 0x4240), off), sc_lo2);
  lo13 = hmul2_u(hadd2_u(__byte_perm(lo, 0x64646464u, 0x4341), off), sc_lo2);
  hi02 = hmul2_u(hadd2_u(__byte_perm(hi, 0x64646464u, 0x4240), off), sc_hi2);
  hi13 = hmul2_u(hadd2_u(__byte_perm(hi, 0x64646464u, 0x4341), off), sc_hi2);
}

// 8 mmas of one quad pair (rows g and g+8): words w0/w1, activations at element base kb
// (low nibbles) and kb+hi_off (high nibbles).
template <class Unpack0, class Unpack1>
__device__ __forceinline__ void quad_mmas(float (&C)[4], const uint8_t* xrow, bool live, int kb, int hi_off, const uint4& q0, const uint4& q1,
                                          Unpack0 un0, Unpack1 un1) {
  const uint32_t w0[4] = {q0.x, q0.y, q0.z, q0.w}, w1[4] = {q1.x, q1.y, q1.z, q1.w};
  uint4 xl0 = make_uint4(0, 0, 0, 0), xl1 = xl0, xh0 = xl0, xh1 = xl0;
  if (live) {
    const uint8_t* pl = xrow + 2 * kb + 16 * (kb >> 6);
    const uint8_t* ph = xrow + 2 * (kb + hi_off) + 16 * ((kb + hi_off) >> 6);
    xl0 = *reinterpret_cast<const uint4*>(pl);
    xl1 = *reinterpret_cast<const uint4*>(pl + 16);
    xh0 = *reinterpret_cast<const uint4*>(ph);
    xh1 = *reinterpret_cast<const uint4*>(ph + 16);
  }
  const uint32_t bl[8] = {xl0.x, xl0.y, xl0.z, xl0.w, xl1.x, xl1.y, xl1.z, xl1.w};
  const uint32_t bh[8] = {xh0.x, xh0.y, xh0.z, xh0.w, xh1.x, xh1.y, xh1.z, xh1.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    uint32_t a_lo[4], a_hi[4];
    un0(i, w0[i], a_lo[0], a_lo[2], a_hi[0], a_hi[2]);
    un1(i, w1[i], a_lo[1], a_lo[3], a_hi[1], a_hi[3]);
    mma16816(C, a_lo, bl[2 * i], bl[2 * i + 1]);
    mma16816(C, a_hi, bh[2 * i], bh[2 * i + 1]);
  }
}

// One super-block of rows g and g + 8 into acc (C layout as in k45_accumulate)
__device__ __forceinline__ void q6_accumulate(float (&acc)[4], const Q6KRow& r0, const Q6KRow& r1, const uint8_t* xrow, bool live, int blk, int t) {
  const int th = t >> 1, hb = t & 1;
  float C[4] = {0.f, 0.f, 0.f, 0.f}, C2[4] = {0.f, 0.f, 0.f, 0.f};
  // unit a = t: hf 0, lh = th, l0 = 16*hb; unit b = t+4: hf 1
  const int sia = hb + 2 * th, sib = 8 + hb + 2 * th;  // scale index of the low-nibble quarter; high is +4
  auto sc2 = [](int s) { return half2_const((float)s); };
  const uint32_t sla0 = sc2(q6_scale(r0.sc, sia)), sha0 = sc2(q6_scale(r0.sc, sia + 4));
  const uint32_t slb0 = sc2(q6_scale(r0.sc, sib)), shb0 = sc2(q6_scale(r0.sc, sib + 4));
  const uint32_t sla1 = sc2(q6_scale(r1.sc, sia)), sha1 = sc2(q6_scale(r1.sc, sia + 4));
  const uint32_t slb1 = sc2(q6_scale(r1.sc, sib)), shb1 = sc2(q6_scale(r1.sc, sib + 4));
  const uint32_t ha0[4] = {r0.qha.x, r0.qha.y, r0.qha.z, r0.qha.w}, hb0[4] = {r0.qhb.x, r0.qhb.y, r0.qhb.z, r0.qhb.w};
  const uint32_t ha1[4] = {r1.qha.x, r1.qha.y, r1.qha.z, r1.qha.w}, hb1[4] = {r1.qhb.x, r1.qhb.y, r1.qhb.z, r1.qhb.w};
  const int ka = blk * 256 + 32 * th + 16 * hb, kb = ka + 128;
  quad_mmas(C, xrow, live, ka, 64, r0.qla, r1.qla,
            [&](int i, uint32_t w, uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d) { q6_unpack_word(w, ha0[i], th, sla0, sha0, a, b, c, d); },
            [&](int i, uint32_t w, uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d) { q6_unpack_word(w, ha1[i], th, sla1, sha1, a, b, c, d); });
  quad_mmas(C2, xrow, live, kb, 64, r0.qlb, r1.qlb,
            [&](int i, uint32_t w, uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d) { q6_unpack_word(w, hb0[i], th, slb0, shb0, a, b, c, d); },
            [&](int i, uint32_t w, uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d) { q6_unpack_word(w, hb1[i], th, slb1, shb1, a, b, c, d); });
#pragma unroll
  for (int i = 0; i < 4; i++) C[i] += C2[i];
  const float d0 = __half2float(__ushort_as_half((unsigned short)r0.d)), d1 = __half2float(__ushort_as_half((unsigned short)r1.d));
  acc[0] = fmaf(d0, C[0], acc[0]);
  acc[1] = fmaf(d0, C[1], acc[1]);
  acc[2] = fmaf(d1, C[2], acc[2]);
  acc[3] = fmaf(d1, C[3], acc[3]);
}

// The tile row that mma row g (second = false) or g + 8 stands for. Q4_K and Q5_K rows are read in eight-byte pieces at a pitch of a
// block (144 or 176 bytes) or of the row's length + 16: with mma row g on row 2g, g + 8 on 2g + 1, a warp's reads fall on distinct banks.
template <int TYPE> __device__ __forceinline__ int mma_row(int g, bool second) { return TYPE == T_Q6_K ? g + (second ? 8 : 0) : 2 * g + (second ? 1 : 0); }
// row0, row1: the rows' blocks `blk` (Q4_K, Q5_K), or the rows (Q6_K, whose blocks are spread over planes)
template <int TYPE>
__device__ __forceinline__ void block_accumulate(float (&acc)[4], const uint8_t* row0, const uint8_t* row1, const uint8_t* xrow, const __half* sxrow, bool live, int nb, int blk, int t) {
  if constexpr (TYPE == T_Q6_K) {
    Q6KRow a0, a1;
    q6k_issue(a0, row0, nb, blk, t);
    q6k_issue(a1, row1, nb, blk, t);
    q6_accumulate(acc, a0, a1, xrow, live, blk, t);
  } else {   // a column past the last repeats the first: its results are not stored
    const __half* sp = sxrow + blk * 8 + 2 * (t >> 1);
    k45_accumulate<TYPE>(acc, (uint32_t)__cvta_generic_to_shared(row0), (uint32_t)__cvta_generic_to_shared(row1), xrow + 576 * blk, *reinterpret_cast<const uint32_t*>(sp),
                         *reinterpret_cast<const uint32_t*>(sp + 4), t);
  }
}

// ---- row-level helpers -------------------------------------------------------------------
// Executed by one whole CTA (QG_THREADS threads) for one activation row: the row kernels of passes of
// more than QG_FUSED_ROWS rows, the embedding gather and the draft head's input use them.

// xn[k] = fp16(h[k] * gamma[k] / sqrt(mean(h^2) + eps))   (reference: llm/hc.go:176-190)
// and, when asked, the sums of the rounded values over every 32 of them (the eight threads of a sub-block are neighbours)
__device__ __forceinline__ void row_rmsnorm_f16(const float* h, const float* gamma, float eps, int H, __half* xn, float* scratch, __half* sx = nullptr, float* ss_out = nullptr) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  float s = 0.f;
  for (int k = tid * 4; k < H; k += QG_THREADS * 4) {
    float4 v = *reinterpret_cast<const float4*>(h + k);
    s += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
  }
  s = warp_sum(s);
  __syncthreads();
  if (lane == 0) scratch[warp] = s;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int w = 0; w < QG_WARPS; w++) tot += scratch[w];
  if (ss_out != nullptr && tid == 0) *ss_out = tot;
  const float scale = 1.0f / sqrtf(tot / (float)H + eps);
  for (int k = tid * 4; k < H; k += QG_THREADS * 4) {
    float4 v = *reinterpret_cast<const float4*>(h + k);
    float4 g = *reinterpret_cast<const float4*>(gamma + k);
    __half2 a = __floats2half2_rn(v.x * scale * g.x, v.y * scale * g.y), b = __floats2half2_rn(v.z * scale * g.z, v.w * scale * g.w);
    *reinterpret_cast<uint2*>(xn + k) = make_uint2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b));
    if (sx != nullptr) {   // H is a multiple of 256: whole warps take part
      const float2 fa = __half22float2(a), fb = __half22float2(b);
      float sum = (fa.x + fa.y) + (fb.x + fb.y);
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if ((lane & 7) == 0) store_sub_sum(sx, k >> 5, sum);
    }
  }
}

// h += sum_k w_k * down_k (slot order) + sigmoid(gate) * shared   (reference: llm/moe.go:347-357, 403-406)
__device__ __forceinline__ void row_moe_combine(float* h, const float* down, const float* w, int used, int H) {
  for (int j = threadIdx.x * 4; j < H; j += QG_THREADS * 4) {
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = 0; k < used; k++) {
      const float wk = w[k];
      float4 d = __ldcg(reinterpret_cast<const float4*>(down + (size_t)k * H + j));
      acc.x += d.x * wk; acc.y += d.y * wk; acc.z += d.z * wk; acc.w += d.w * wk;
    }
    const float sg = w[used];
    float4 sh = __ldcg(reinterpret_cast<const float4*>(down + (size_t)used * H + j));
    float4 hv = *reinterpret_cast<float4*>(h + j);
    hv.x += acc.x + sh.x * sg; hv.y += acc.y + sh.y * sg; hv.z += acc.z + sh.z * sg; hv.w += acc.w + sh.w * sg;
    *reinterpret_cast<float4*>(h + j) = hv;
  }
}

// Row kernels (row_tail_kernel) for passes of more than QG_FUSED_ROWS rows
struct TailParams {
  int mode;             // 1 rmsnorm, 2 MoE combine + rmsnorm
  float* h;             // [M][H] residual stream
  const float* down;    // [M][used+1][H]
  const float* topk_w;  // [M][used+1]
  int used, H, M;
  const float* gamma;
  __half* xn;
  float eps;
  // mode 1: first h += parts[0] + parts[1] + ... (the planes of a projection whose contraction was cut), in plane order
  const float* parts;
  int n_parts;
  int64_t part_plane;
  __half* sx;           // optional: sub-block sums of the normalised rows, [M][H / 256][TG_SX]
  float* ss_out;        // optional: [M][SS_LD] sum of squares of the row, as one part
};

// ---- activation staging ------------------------------------------------------------------
// Activation rows go to shared memory as fp16 in the permuted, padded layout the B fragments are read in, with the sums of every
// 32 of them (fp16 hi + lo planes, [plane(2)][xcols][K/32] halves) for the min term. The threads that hold a sub-block are
// neighbours and add it up by shuffles: (x0 + x1) + (x2 + x3) per four elements, then a tree over the eight fours, whoever stages.
__device__ __forceinline__ float sum4_h2(uint32_t x02, uint32_t x13) { return (h2f_lo(x02) + h2f_lo(x13)) + (h2f_hi(x02) + h2f_hi(x13)); }
template <int LANES>   // that share a sub-block: 8 of four elements each, or 4 of eight
__device__ __forceinline__ void put_sx(float sum, __half* sx_hi, __half* sx_lo, int sub) {
  const int lane = threadIdx.x & 31;
  const uint32_t mask = ((1u << LANES) - 1) << (lane & ~(LANES - 1));
#pragma unroll
  for (int o = 1; o < LANES; o <<= 1) sum += __shfl_xor_sync(mask, sum, o);
  if ((lane & (LANES - 1)) == 0) {
    const __half hi = __float2half_rn(sum);
    sx_hi[sub] = hi;
    sx_lo[sub] = __float2half_rn(sum - __half2float(hi));
  }
}

// one fp16 row into the permuted layout, by threads t of nt (nt a multiple of 8, t and the thread's lane alike in their low bits)
__device__ __forceinline__ void copy_x_row(const __half* src, int K, uint8_t* dst, __half* sx_hi, __half* sx_lo, int t, int nt) {
  // every CTA reads the same row: each starts at another 128-byte line so the L2 slices are not all asked for
  // the same line at the same moment
  t = (t + 8 * (int)((blockIdx.x + blockIdx.y) % (unsigned)(nt / 8))) % nt;
  for (int k = t * 8; k < K; k += nt * 8) {
    uint4 v = __ldcg(reinterpret_cast<const uint4*>(src + k));
    uint4 o;
    o.x = __byte_perm(v.x, v.y, 0x5410); o.y = __byte_perm(v.x, v.y, 0x7632);
    o.z = __byte_perm(v.z, v.w, 0x5410); o.w = __byte_perm(v.z, v.w, 0x7632);
    *reinterpret_cast<uint4*>(dst + 2 * k + 16 * (k >> 6)) = o;
    put_sx<4>(sum4_h2(o.x, o.y) + sum4_h2(o.z, o.w), sx_hi, sx_lo, k >> 5);
  }
}
__device__ __forceinline__ void stage_x_f16(const __half* x, int64_t ldx, int K, int xcols, uint8_t* xs, __half* sxs, int ncols, const int* xrows, int xstride) {
  const int nsub = K / 32;
  for (int c = 0; c < ncols; c++)
    copy_x_row(x + (int64_t)xrows[c] * ldx, K, xs + (size_t)c * xstride, sxs + (size_t)c * nsub, sxs + (size_t)(xcols + c) * nsub, threadIdx.x, QG_THREADS);
  __syncthreads();
}

// 1 / sqrt(mean(h^2) + eps) of row `row` from the partial sums its producer left, by one warp
__device__ __forceinline__ float scale_from_parts(const float* ss_in, int ss_n, int64_t row, int K, float eps) {
  float s = 0.f;
  for (int i = threadIdx.x & 31; i < ss_n; i += 32) s += __ldcg(ss_in + row * SS_LD + i);
  s = warp_sum(s);
  return 1.0f / sqrtf(s / (float)K + eps);
}

// RMSNorm fused into the staging (reference: llm/hc.go:176-190): each CTA normalises the rows it needs
__device__ __forceinline__ void stage_x_norm(const QGemvParams& p, uint8_t* xs, __half* sxs, float* scratch, int ncols, const int* xrows, int xstride,
                                             bool write_xn) {
  const int warp = threadIdx.x >> 5, K = p.K;
  float* hout = p.out != nullptr && blockIdx.x == 0 && blockIdx.z == 0 ? p.out->h : nullptr;
  const int h_first = hout != nullptr ? p.out->h_first : 0;
  // element index of this thread, rotated by whole 128-byte lines per CTA (every CTA reads the same rows)
  const int tid = (threadIdx.x + 8 * (int)((blockIdx.x + blockIdx.y) & 31)) & (QG_THREADS - 1);
  // the residual values do not depend on the scale: fetch the first batch before reducing the partials
  constexpr int PRE = 2;
  float4 hpre[PRE], gpre[PRE];
  const float* src0 = p.hsrc + (int64_t)xrows[0] * K;
#pragma unroll
  for (int i = 0; i < PRE; i++) {
    const int k = tid * 4 + i * QG_THREADS * 4;
    if (k < K) { hpre[i] = __ldcg(reinterpret_cast<const float4*>(src0 + k)); gpre[i] = *reinterpret_cast<const float4*>(p.gamma + k); }
  }
  if (warp < ncols) {
    const float sc = scale_from_parts(p.ss_in, p.ss_n, xrows[warp], K, p.eps);
    if ((threadIdx.x & 31) == 0) scratch[warp] = sc;
  }
  __syncthreads();
  for (int c = 0; c < ncols; c++) {
    const int64_t row = xrows[c];
    const float* src = p.hsrc + row * (int64_t)K;
    const float scale = scratch[c];
    uint8_t* dst = xs + (size_t)c * xstride;
    int i = 0;
    for (int k = tid * 4; k < K; k += QG_THREADS * 4, i++) {
      float4 h, g;
      if (c == 0 && i < PRE) { h = hpre[i < PRE ? i : 0]; g = gpre[i < PRE ? i : 0]; }
      else { h = __ldcg(reinterpret_cast<const float4*>(src + k)); g = *reinterpret_cast<const float4*>(p.gamma + k); }
      const float v0 = h.x * scale * g.x, v1 = h.y * scale * g.y, v2 = h.z * scale * g.z, v3 = h.w * scale * g.w;
      __half2 a = __floats2half2_rn(v0, v2), b = __floats2half2_rn(v1, v3);  // stored order [x0,x2,x1,x3]
      *reinterpret_cast<uint2*>(dst + 2 * k + 16 * (k >> 6)) = make_uint2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b));
      if (hout != nullptr && c >= h_first) *reinterpret_cast<float4*>(hout + (size_t)(c - h_first) * K + k) = h;
      if (write_xn) {
        __half2 n0 = __floats2half2_rn(v0, v1), n1 = __floats2half2_rn(v2, v3);
        *reinterpret_cast<uint2*>(p.xn_out + row * K + k) = make_uint2(*reinterpret_cast<uint32_t*>(&n0), *reinterpret_cast<uint32_t*>(&n1));
      }
      put_sx<8>(sum4_h2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b)), sxs + (size_t)c * (K / 32), sxs + (size_t)(p.xcols + c) * (K / 32), k >> 5);
    }
  }
  __syncthreads();
}

// ---- the kernel ----------------------------------------------------------------------------
// grid.x: persistent CTAs walking the row-tile groups; grid.z: column tile of 8 activation rows (plain mode).
// A grouped launch over a work list is one row of CTAs that share the list's (entry, group) units evenly.
//
// Weights reach the SM as whole tiles (16 consecutive rows are one contiguous run of the
// checkpoint's own blocks) through cp.async.bulk into a ring of shared-memory stages, each
// completing on its mbarrier, so many tiles are in flight per SM without holding registers.
template <int TYPE, int PRO, int EPI, bool DUAL, bool GROUPED>
__global__ void __launch_bounds__(QG_THREADS, (GROUPED || TYPE == T_Q6_K) ? 3 : 2) qgemv_kernel(const __grid_constant__ QGemvMaps maps, const QGemvParams p) {
  extern __shared__ __align__(128) uint8_t smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int K = p.K, nb = K / 256;
  const int wpt = nb >= 8 ? 8 : nb >= 4 ? 4 : nb >= 2 ? 2 : 1;  // warps per tile (K-slices)
  const int tpc = QG_WARPS / wpt;                               // tiles per CTA and iteration
  const int xstride = qg_xstride(K);
  uint8_t* xs = smem;
  __half* sxs = reinterpret_cast<__half*>(smem + (size_t)p.xcols * xstride);
  float* red = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(sxs) + (((size_t)p.xcols * (K / 32) * 2 * sizeof(__half) + 15) & ~(size_t)15));
  uint8_t* stages = smem + qg_fixed_smem(K, p.xcols, DUAL);
  constexpr bool BOXED = qg_boxed(TYPE, GROUPED);
  constexpr int BLK = TYPE == T_Q4_K ? 144 : TYPE == T_Q5_K ? 176 : 0;   // bytes of a super-block where a row's lie side by side
  const size_t pitch = (size_t)qg_pitch(TYPE, p.stride, GROUPED), tile_bytes = 16 * pitch;
  const size_t stage_bytes = (size_t)tpc * tile_bytes * (DUAL ? 2 : 1);
  const int NS = p.nstage;
  __shared__ float scratch[4 * QG_WARPS];
  __shared__ int col_rows[QG_MAXCOLS], xrows[QG_MAXCOLS];
  __shared__ __align__(8) uint64_t full_bar[BOXED ? QG_WARPS : 1][QG_MAX_STAGES];

  const int tiles = (p.N + 15) / 16;
  const int ngroups = (tiles + tpc - 1) / tpc;
  const int lt = warp / wpt, kslice = warp % wpt;

  tl_mark(p.tl, 0);
  if constexpr (BOXED) {
    if (lane < NS) mbar_init(&full_bar[warp][lane], 1);
    if (lane == 0) mbar_fence_init();
    __syncwarp();
  } else {
    if (tid == 0) {
      for (int s = 0; s < NS; s++) mbar_init(&full_bar[0][s], 1);
      mbar_fence_init();
    }
    __syncthreads();
  }

  // What this CTA walks is a sequence of units, each one row-tile group of one weight matrix. Plain launches take the groups blockIdx.x, blockIdx.x + gridDim.x, ... of the one matrix they
  // are given. Launches over a work list cut the whole list, entries * groups units, into one contiguous run per CTA:
  // every CTA gets the same share whatever the list's length (known only on the device), a run stages the activation
  // rows of an entry once, and the weight ring runs ahead across the entries' boundaries.
  int ncols = 0, col_off = 0, n_units = 0;
  long long u0 = 0;
  if constexpr (GROUPED) {
    pdl_wait();  // the entries are written by the router kernel
    const long long U = (long long)*p.n_entries * ngroups, c = blockIdx.x;
    u0 = c * U / gridDim.x;
    n_units = (int)((c + 1) * U / gridDim.x - u0);
  } else {
    ncols = p.M - (int)blockIdx.z * QG_MAXCOLS;
    if (ncols > QG_MAXCOLS) ncols = QG_MAXCOLS;
    col_off = (int)blockIdx.z * QG_MAXCOLS;
    n_units = (int)blockIdx.x < ngroups ? (ngroups - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
  }
  // BOXED: each warp brings its own super-blocks of its own tile, 16 x 256 weights to a box at a pitch of a block, and refills them
  // alone. Else warp 0 is the producer: one bulk copy per tile row, or per tile where rows lie as in memory.
  auto issue_boxes = [&](int it) {
    const int tile = ((int)blockIdx.x + it * (int)gridDim.x) * tpc + lt, s = it % NS;
    if (tile >= tiles || kslice >= nb) return;
    if (elect_one()) {
      int sg = 0;
      while (sg + 1 < p.nseg && tile * 16 >= p.seg_end[sg]) sg++;
      const int r = tile * 16 - (sg > 0 ? p.seg_end[sg - 1] : 0);
      uint8_t* dst = stages + (size_t)s * stage_bytes + (size_t)lt * tile_bytes;
      mbar_expect_tx(&full_bar[BOXED ? warp : 0][s], (uint32_t)((nb - kslice + wpt - 1) / wpt * 16 * BLK));
      for (int blk = kslice; blk < nb; blk += wpt) tma_box_2d(dst + blk * (16 * BLK), &maps.w[sg], blk * BLK, r, &full_bar[BOXED ? warp : 0][s]);
    }
    __syncwarp();
  };
  auto issue_group = [&](int grp, int s, const uint8_t* ga, const uint8_t* gb) {
    if (lane == 0) {
      uint32_t total = 0;
      for (int l = 0; l < tpc; l++) {
        const int tile = grp * tpc + l;
        if (tile < tiles) total += (uint32_t)(min(16, p.N - tile * 16) * p.stride) * (DUAL ? 2 : 1);
      }
      mbar_expect_tx(&full_bar[0][s], total);
    }
    __syncwarp();
    for (int l = 0; l < tpc; l++) {
      const int tile = grp * tpc + l;
      if (tile >= tiles) continue;
      const int nrows = min(16, p.N - tile * 16);
      const uint8_t *base = ga, *base2 = gb;
      int seg_r0 = 0;
      if constexpr (!GROUPED) {
        int sg = 0;
        while (sg + 1 < p.nseg && tile * 16 >= p.seg_end[sg]) sg++;
        seg_r0 = sg > 0 ? p.seg_end[sg - 1] : 0;
        base = p.w[sg];
        if constexpr (DUAL) base2 = p.w2[sg];
      }
      uint8_t* dst = stages + (size_t)s * stage_bytes + (size_t)l * tile_bytes * (DUAL ? 2 : 1);
      const int64_t off = (int64_t)(tile * 16 - seg_r0) * p.stride;
      if constexpr (TYPE == T_Q6_K) {
        if (lane == 0) {
          bulk_copy_g2s(dst, base + off, (uint32_t)(nrows * p.stride), &full_bar[0][s]);
          if constexpr (DUAL) bulk_copy_g2s(dst + tile_bytes, base2 + off, (uint32_t)(nrows * p.stride), &full_bar[0][s]);
        }
      } else {
        const int r = lane & 15;
        if (r < nrows && lane < (DUAL ? 32 : 16)) bulk_copy_g2s(dst + (lane >> 4) * tile_bytes + r * pitch, (lane < 16 ? base : base2) + off + r * p.stride, (uint32_t)p.stride, &full_bar[0][s]);
      }
    }
  };
  // unit j of this CTA goes to ring stage j % NS
  auto issue_unit = [&](int j) {
    if constexpr (GROUPED) {
      const long long u = u0 + j;
      const int en = (int)(u / ngroups), grp = (int)(u - (long long)en * ngroups);
      const int ex = p.entries[en].x;
      const uint8_t* ga = ex >= 0 ? p.w[0] + (size_t)ex * p.expert_stride : p.ws;
      const uint8_t* gb = nullptr;
      if constexpr (DUAL) gb = ex >= 0 ? p.w2[0] + (size_t)ex * p.expert_stride : p.ws2;
      issue_group(grp, j % NS, ga, gb);
    } else {
      issue_group((int)blockIdx.x + j * (int)gridDim.x, j % NS, nullptr, nullptr);
    }
  };
  if constexpr (BOXED) {
    for (int k = 0; k < NS && k < n_units; k++) issue_boxes(k);
  } else if (warp == 0) {
    for (int k = 0; k < NS && k < n_units; k++) issue_unit(k);
  }
  if constexpr (!GROUPED) pdl_wait();
  pdl_launch();
  tl_mark(p.tl, 1);

  float* const y = p.out != nullptr ? p.out->logits : p.y;
  bool live = false;
  const uint8_t* xrow = xs;
  const __half* sxrow = sxs;
  // the activation rows of the current entry (or of this launch's column tile) into shared memory
  auto stage_rows = [&]() {
    if (tid < QG_MAXCOLS) {
      const int c = tid < ncols ? tid : 0;
      int id;
      if constexpr (GROUPED) id = p.cols[col_off + c];
      else id = p.row_ids ? p.row_ids[col_off + c] : col_off + c;
      col_rows[tid] = id;
      xrows[tid] = GROUPED ? id / p.x_div : id;
    }
    __syncthreads();
    if constexpr (PRO == PRO_NORM) stage_x_norm(p, xs, sxs, scratch, ncols, xrows, xstride, p.xn_out != nullptr && blockIdx.x == 0 && blockIdx.y == 0);
    else stage_x_f16(p.x, p.ldx, K, p.xcols, xs, sxs, ncols, xrows, xstride);
    live = g < ncols;
    xrow = xs + (size_t)(live ? g : 0) * xstride;
    sxrow = sxs + (size_t)((t & 1) * p.xcols + (live ? g : 0)) * (K / 32);
  };
  if constexpr (!GROUPED) { stage_rows(); tl_mark(p.tl, 2); }

  // Units go through in chunks: every warp leaves its partial sums of a chunk's units, [unit][warp][column][row], one barrier, and
  // the CTA adds them up in warp order. (A barrier per unit left the warps waiting for one another three times in a decode step's
  // largest projection.) A chunk is what the ring and 8 KB of partial sums hold.
  const int xc = GROUPED ? QG_MAXCOLS : p.xcols, chunk = GROUPED ? 1 : min(NS, 2 * QG_MAXCOLS / xc);
  const size_t plane2 = QG_WARPS * 16 * QG_MAXCOLS;   // DUAL: the second matrix's sums
  int cur = -1;
  bool lost = false;
  // a copy never landed: the results are void, and no more are asked for; those in flight land (or run out their limit too) before the CTA leaves
  auto land = [&](uint64_t* bars, int it) {
    for (int k = it; k < it + NS && k < n_units; k++) mbar_wait(&bars[k % NS], (uint32_t)((k / NS) & 1), 1u << 18);
  };
  for (int it0 = 0; it0 < n_units; it0 += chunk) {
    const int cnt = min(chunk, n_units - it0);
    if (it0 > 0) __syncthreads();   // the sums before are read; GROUPED: every warp is done with the rows of the entry before
    if constexpr (GROUPED) {
      const int en = (int)((u0 + it0) / ngroups);
      if (en != cur) {
        const int4 e = p.entries[en];
        col_off = e.y; ncols = e.z; cur = en;
        stage_rows();
      }
    }
    auto group_of = [&](int it) {
      if constexpr (GROUPED) return (int)((u0 + it) % ngroups);
      else return (int)blockIdx.x + it * (int)gridDim.x;
    };
    for (int u = 0; u < cnt; u++) {
      const int it = it0 + u, s = it % NS;
      const int tile = group_of(it) * tpc + lt;
      float acc[4] = {0.f, 0.f, 0.f, 0.f}, acc2[4] = {0.f, 0.f, 0.f, 0.f};
      if constexpr (BOXED) {
        if (tile < tiles && kslice < nb && !lost) {
          if (!warp_wait(&full_bar[BOXED ? warp : 0][s], (uint32_t)((it / NS) & 1))) {
            if (lane == 0) report_error(p.err);
            lost = true;
            land(full_bar[BOXED ? warp : 0], it);
          } else {
            if (it == 0) tl_mark(p.tl, 3);
            const uint8_t* row0 = stages + (size_t)s * stage_bytes + (size_t)lt * tile_bytes + 2 * g * BLK;
            for (int blk = kslice; blk < nb; blk += wpt) block_accumulate<TYPE>(acc, row0 + blk * (16 * BLK), row0 + blk * (16 * BLK) + BLK, xrow, sxrow, live, nb, blk, t);
          }
          __syncwarp();
          if (it + NS < n_units && !lost) { fence_proxy_async(); issue_boxes(it + NS); }
        }
      } else {
        if (!mbar_wait(&full_bar[0][s], (uint32_t)((it / NS) & 1))) {
          if (tid == 0) report_error(p.err);
          land(full_bar[0], it);
          return;
        }
        if (it == 0) tl_mark(p.tl, 3);
        if (tile < tiles) {
          const int nrows = min(16, p.N - tile * 16);
          const uint8_t* tb = stages + (size_t)s * stage_bytes + (size_t)lt * tile_bytes * (DUAL ? 2 : 1);
          const uint8_t *row0 = tb + min(mma_row<TYPE>(g, false), nrows - 1) * pitch, *row1 = tb + min(mma_row<TYPE>(g, true), nrows - 1) * pitch;
          for (int blk = kslice; blk < nb; blk += wpt) {
            const int off = blk * BLK;
            block_accumulate<TYPE>(acc, row0 + off, row1 + off, xrow, sxrow, live, nb, blk, t);
            if constexpr (DUAL) block_accumulate<TYPE>(acc2, row0 + tile_bytes + off, row1 + tile_bytes + off, xrow, sxrow, live, nb, blk, t);
          }
        }
      }
      auto leave = [&](float* my, const float (&a)[4]) {
        const int m0 = mma_row<TYPE>(g, false), m1 = mma_row<TYPE>(g, true);
        if (2 * t < xc) { my[2 * t * 16 + m0] = a[0]; my[2 * t * 16 + m1] = a[2]; }
        if (2 * t + 1 < xc) { my[(2 * t + 1) * 16 + m0] = a[1]; my[(2 * t + 1) * 16 + m1] = a[3]; }
      };
      leave(red + (size_t)(u * QG_WARPS + warp) * 16 * xc, acc);
      if constexpr (DUAL) leave(red + plane2 + (size_t)(u * QG_WARPS + warp) * 16 * xc, acc2);
    }
    __syncthreads();
    // every warp is done with these stages: refill them with the units NS iterations ahead
    if constexpr (!BOXED) {
      if (warp == 0)
        for (int u = 0; u < cnt; u++)
          if (it0 + u + NS < n_units) { fence_proxy_async(); issue_unit(it0 + u + NS); }
    }
    // sixteen threads per (unit, tile, column), one row each
    const int r = tid & 15, sets = cnt * tpc, inv = 65535 / sets + 1;
    for (int q = tid >> 4; q < sets * ncols; q += QG_THREADS / 16) {
      const int c = (q * inv) >> 16, ul = q - c * sets, u = ul / tpc, l2 = ul - u * tpc;
      const int tile = group_of(it0 + u) * tpc + l2, grow = tile * 16 + r;
      const float* rb = red + ((size_t)(u * QG_WARPS + l2 * wpt) * xc + c) * 16 + r;
      float v = 0.f, v2 = 0.f, sq = 0.f;
      for (int w = 0; w < wpt; w++) {
        v += rb[w * 16 * xc];
        if constexpr (DUAL) v2 += rb[plane2 + w * 16 * xc];
      }
      const int64_t orow = (!GROUPED && p.row_ids != nullptr) ? col_off + c : col_rows[c];
      if (grow < p.N) {
        if constexpr (EPI == EPI_STORE) { y[orow * p.ldy + grow] = v; sq = v * v; }
        else if constexpr (EPI == EPI_RESID) { const float nv = y[orow * p.ldy + grow] + v; y[orow * p.ldy + grow] = nv; sq = nv * nv; }
        else p.y16[orow * p.ldy + grow] = __float2half_rn(v * sigmoid_acc(v) * v2);  // SwiGLU of (gate, up) rounded to fp16 (reference: shaders/llm_moe_gemv.comp:777-781)
      }
      if constexpr (EPI != EPI_SWIGLU && !GROUPED) {
        if (p.ss_out != nullptr) {  // sum of squares of this tile's rows per column, in a fixed order
#pragma unroll
          for (int o = 1; o < 16; o <<= 1) sq += __shfl_xor_sync(0xffffu << (lane & 16), sq, o);
          if (r == 0 && tile < tiles) p.ss_out[orow * SS_LD + tile] = sq;
        }
      }
    }
  }
  tl_mark(p.tl, 4);
}

}  // namespace b200
