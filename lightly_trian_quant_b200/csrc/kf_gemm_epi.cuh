// Shared pieces of the block-scaled GEMM kernels: argument block, per-format traits and the fused epilogues
// (PLAIN / RES / ROPE / QUANT) as one device function that works on a 32-row x 64-column piece of the accumulator held in
// registers.  Epilogue math per infer-opt/round13_mxfp8_full/impl/mgx_core.cu:308-426 and
// infer-opt/round14_fp4_full/impl/fp4g_core.cu:309-382.
//
// Every epilogue works in the layout tcgen05.ld delivers: thread `lane` of a warp owns 64 consecutive columns of ONE
// output row.  That is 128 contiguous bytes of a 16-bit output (exactly one [token, head] row of the q/k/v layout) or
// 256 contiguous bytes of an fp32 one, which the thread moves with 256-bit global loads / stores (ld/st.global.v8): every
// access is a whole 32-byte sector.  Two forms exchange data to move whole 128-byte lines instead: ROPE transposes the pieces of every
// four rows between lanes (store_rows128), as PLAIN does with bf16; RES on CTA pairs, and RES launches of many rounds and a short K, update
// the residual in shared memory, where it comes and goes as TMA boxes (epilogue_res_tma).  Shared memory also holds the bias (and LayerScale) values, the whole vector of
// the launch, loaded once per CTA, or a 64-value slice per warp and tile where the operand ring leaves no room for the vector, and
// for ROPE the rotary-table rows of the tile.
#pragma once
#include "kf_sm100_pair.cuh"

namespace kf {

constexpr int KIND_MX8 = KF_FMT_MX8, KIND_NV4 = KF_FMT_NV4, KIND_MX4 = KF_FMT_MX4, KIND_BF16 = KF_FMT_BF16;
constexpr int BM = 128, BKB = 128;                     // tile rows, K bytes per stage
constexpr int A_BYTES = BM * BKB;
// Column-tile widths BN = 256 and BN = 128 (kf_gemm.cu says when which): bytes of one operand stage (16 KB of A, then 32 or
// 16 KB of W), bytes of its scale atoms (up to 4 for A, then up to 4 for every 128 rows of W), accumulators that fit the 256
// tensor-memory columns in front of the scale factors, and columns of one epilogue warp (16 warps = 4 row quarters x 4).
template <int BN>
struct Tile {
  static constexpr int BYTES = (BM + BN) * BKB;
  static constexpr int SF_BYTES = (1 + BN / 128) * 4 * 512;
  static constexpr int ACCS = 256 / BN;
  static constexpr int CW = BN / 4;
};
constexpr int EPI_WARPS = 16;
constexpr int EPI_WARP0 = 4;                           // warps 0..3: TMA producer, MMA issuer, two spares
constexpr int GEMM_THREADS = 32 * (EPI_WARP0 + EPI_WARPS);
constexpr int SF_BUFS = 4;                             // scale-factor buffers in TMEM, 48 columns each (A at +0, W at +16)
constexpr int SF_BUF_COLS = 48;
constexpr int TMEM_COLS = 512;
constexpr int TMEM_SF_COL = 256;                       // accumulator: columns [0,256); scale factors from 256
constexpr int SLICE_FLOATS = 128;                      // per epilogue warp: 64 bias values, then 64 LayerScale values (RES)
constexpr int ROPE_SLAB_FLOATS = 32 * 64;              // per TMEM lane quarter: 32 rows x (32 sin | 32 cos) values of the rotary tables
static_assert(TMEM_SF_COL + SF_BUFS * SF_BUF_COLS <= TMEM_COLS, "TMEM budget");

struct GemmArgs {
  const uint8_t *sfa, *sfw;
  const float *ts_a, *ts_w, *bias, *gamma, *R, *sin, *cos, *tso;
  void* C;
  uint8_t *Qo, *SFo;
  int M, N, K;
  int Ntok, prefix, H, d;
  int out_dtype, flags, out_fmt;
  int m_tiles, n_tiles, k_tiles, nkb4, stages;
  int full_tiles, items;                   // work items: full_tiles whole tiles, then the remaining tiles of the last round as two 128-column halves each
  int row_group, row_stride, row_offset;   // PLAIN, RES: output row = (m / group) * stride + offset + m % group (group 0: identity)
  int m_tiles_pb, a_rows_pb, w_rows_pb;    // batched products (m_tiles_pb > 0): row tiles, A rows and W rows per product
  int vec_floats;                          // > 0: the whole bias vector (and for RES the LayerScale vector behind it) sits in shared memory for the launch
  int res_tma;                             // RES, BN = 128 or CTA pairs: the residual goes through shared memory by TMA boxes (epilogue_res_tma)
  float* y_dbg;                            // QUANT: optional export of the values that were quantised (fp32 [M, N])
  unsigned int* err;
};

template <int KIND>
struct KindTraits;
template <>
struct KindTraits<KIND_MX8> { static constexpr int ATOMS = 1; };   // 128 elements per stage = 4 k-blocks of 32
template <>
struct KindTraits<KIND_NV4> { static constexpr int ATOMS = 4; };   // 256 elements per stage = 16 k-blocks of 16
template <>
struct KindTraits<KIND_MX4> { static constexpr int ATOMS = 2; };   // 256 elements per stage = 8 k-blocks of 32
template <>
struct KindTraits<KIND_BF16> { static constexpr int ATOMS = 0; };

// ------------------------------------------------------------------------------------------------ 256-bit global accesses
struct F8 {
  float v[8];
};
__device__ __forceinline__ F8 ldg8_stream(const float* p) {   // 32-byte aligned; read once: do not keep the line in L1
  F8 r;
  asm volatile("ld.global.L1::no_allocate.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(r.v[0]), "=f"(r.v[1]), "=f"(r.v[2]), "=f"(r.v[3]), "=f"(r.v[4]), "=f"(r.v[5]), "=f"(r.v[6]), "=f"(r.v[7])
               : "l"(p));
  return r;
}
__device__ __forceinline__ float4 ldg4_nc(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ void stg8(void* p, float a, float b, float c, float d, float e, float f, float g, float h) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d), "f"(e), "f"(f), "f"(g), "f"(h)
               : "memory");
}
// two fp32 -> one 32-bit word of two bf16 / f16 values (first value in the low half)
__device__ __forceinline__ uint32_t pack2(float a, float b, int out_dtype) {
  if (out_dtype == KF_BF16) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

// Stores the warp's 32 rows of 128 bytes (lane = row, w = its four 32-byte pieces) as whole lines: inside every four lanes the pieces are
// transposed (4 x 4), then a store instruction covers eight rows of 128 bytes instead of 32 pieces of 32 bytes in 32 lines, whose
// look-ups had L1 71 % busy in the ROPE epilogue, the unit the operand ring fills through (qkv NVFP4 M = 22 470: 66 -> 60 us, MXFP8
// x 768 55 -> 52 us).  PLAIN bf16 NVFP4 x 4096: 78 -> 64 us together with the forms
// below.  For the residual of RES (level) it did not pay.
// base: the 128 bytes of row 0; rows from `rows` on are not written.
__device__ __forceinline__ void store_rows128(uint32_t (&w)[32], uint8_t* base, size_t row_bytes, int rows, int lane) {
  const bool b0 = lane & 1, b1 = lane & 2;
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int q = 0; q < 8; ++q) {                  // -> w[8 * (2j + e)]: piece 2j + b0 of row e of the lane's pair
      const uint32_t a = w[16 * j + q], b = w[16 * j + 8 + q];
      const uint32_t got = __shfl_xor_sync(0xffffffffu, b0 ? a : b, 1);
      w[16 * j + q] = b0 ? got : a;
      w[16 * j + 8 + q] = b0 ? b : got;
    }
#pragma unroll
  for (int e = 0; e < 2; ++e)
#pragma unroll
    for (int q = 0; q < 8; ++q) {                  // -> w[8 * k]: piece 2 * b1 + b0 of row k of the lane's four
      const uint32_t a = w[8 * e + q], b = w[16 + 8 * e + q];
      const uint32_t got = __shfl_xor_sync(0xffffffffu, b1 ? a : b, 2);
      w[8 * e + q] = b1 ? got : a;
      w[16 + 8 * e + q] = b1 ? b : got;
    }
  const int row0 = lane & ~3;
  uint8_t* p = base + (size_t)row0 * row_bytes + (lane & 3) * 32;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (row0 + k < rows) stg8w(p + k * row_bytes, &w[8 * k]);
}
// ------------------------------------------------------------------------------------------------ QUANT
// QUANT epilogue of one 32-column chunk: the thread owns columns n0..n0+31 of row m = two nv4 blocks or one mx block, so
// block maxima need no shuffles and the per-block scale arithmetic is paid once per 16 / 32 values.
// The codes and scale bytes are the bit specification's quantisation (IEEE divisions, as in the row quantiser) of the
// values gelu(acc*ts + bias), optionally rounded to bf16, which y_dbg exports for the parity tests.

// values 16*h .. 16*h+15 of the chunk: bias + GELU (+ bf16 rounding), exported when asked; returns their maximum magnitude
// FAST: rounding to bf16, no export (the forms of the model), without a test per value
template <bool FAST>
__device__ __forceinline__ float quant_values16(const GemmArgs& g, const uint32_t (&r)[32], int h, float ts, const float* bsm, float* dbg, float (&v)[16]) {
  const float2 ts2 = splat2(ts);
#pragma unroll
  for (int q4 = 0; q4 < 4; ++q4) {
    const int k = 16 * h + 4 * q4;
    const float4 bb = *reinterpret_cast<const float4*>(bsm + k);   // zeros without a bias
    float2 a = gelu_erf2(fma2(make_float2(__uint_as_float(r[k]), __uint_as_float(r[k + 1])), ts2, make_float2(bb.x, bb.y)));
    float2 b = gelu_erf2(fma2(make_float2(__uint_as_float(r[k + 2]), __uint_as_float(r[k + 3])), ts2, make_float2(bb.z, bb.w)));
    if (FAST || (g.flags & KF_Q_ROUND_BF16)) {
      a = bf16_round2(a);
      b = bf16_round2(b);
    }
    v[4 * q4] = a.x;
    v[4 * q4 + 1] = a.y;
    v[4 * q4 + 2] = b.x;
    v[4 * q4 + 3] = b.y;
    if (!FAST && dbg) *reinterpret_cast<float4*>(dbg + k) = make_float4(a.x, a.y, b.x, b.y);
  }
  float am = 0.f;
#pragma unroll
  for (int k = 0; k < 16; k += 2) am = max3(am, fabsf(v[k]), fabsf(v[k + 1]));
  return am;
}

// FMT: the output format, or -1 for the one in the arguments (with all options)
template <int FMT>
__device__ __forceinline__ void quant_chunk(const GemmArgs& g, const uint32_t (&r)[32], float ts, const Nv4Scale& sco /* per-tensor scale of an nv4 output */, int m, int n0,
                                            const float* bsm /* the chunk's 32 bias values in shared memory */) {
  const bool div_true = !(g.flags & KF_Q_RECIP_DIV);
  const bool ok = m < g.M;
  constexpr bool FAST = FMT >= 0;
  const int out_fmt = FAST ? FMT : g.out_fmt;
  float* dbg = (!FAST && g.y_dbg != nullptr && ok) ? g.y_dbg + (size_t)m * g.N + n0 : nullptr;
  int by0, by1;
  if (out_fmt == KF_FMT_NV4) {
    uint32_t o[4];
    float va[16], vb[16];
    const float am0 = quant_values16<FAST>(g, r, 0, ts, bsm, dbg, va), am1 = quant_values16<FAST>(g, r, 1, ts, bsm, dbg, vb);
    if (!FAST && (g.flags & KF_Q_FAST_NV4)) {
      quant_nv4_fast<16>(va, am0, sco.ts, sco.rcp_ts, o, by0);
      quant_nv4_fast<16>(vb, am1, sco.ts, sco.rcp_ts, o + 2, by1);
    } else {
      quant_nv4_pair16(va, am0, vb, am1, sco, div_true, o, by0, by1);
    }
    if (ok) *reinterpret_cast<uint4*>(g.Qo + (size_t)m * (g.N >> 1) + (n0 >> 1)) = make_uint4(o[0], o[1], o[2], o[3]);
    // two scale bytes of this row for the chunk (rows beyond M inside the last tile get zeros)
    *reinterpret_cast<uint16_t*>(g.SFo + sf_offset(m, n0 >> 4, g.N >> 6)) = ok ? (uint16_t)(by0 | (by1 << 8)) : (uint16_t)0;
    return;
  }
  float va[16], vb[16];
  const float am = amax_nan(quant_values16<FAST>(g, r, 0, ts, bsm, dbg, va), quant_values16<FAST>(g, r, 1, ts, bsm, dbg, vb));
  if (out_fmt == KF_FMT_MX8) {
    uint32_t o[8];
    quant_mx8<16>(va, am, div_true, o, by0);
    quant_mx8<16>(vb, am, div_true, o + 4, by0);
    if (ok) stg8w(g.Qo + (size_t)m * g.N + n0, o);
    g.SFo[sf_offset(m, n0 >> 5, g.N >> 7)] = ok ? (uint8_t)by0 : (uint8_t)0;
  } else {
    uint32_t o[4];
    quant_mx4<16>(va, am, div_true, o, by0);
    quant_mx4<16>(vb, am, div_true, o + 2, by0);
    if (ok) *reinterpret_cast<uint4*>(g.Qo + (size_t)m * (g.N >> 1) + (n0 >> 1)) = make_uint4(o[0], o[1], o[2], o[3]);
    g.SFo[sf_offset(m, n0 >> 5, g.N >> 7)] = ok ? (uint8_t)by0 : (uint8_t)0;
  }
}

// ------------------------------------------------------------------------------------------------ PLAIN
// PLAIN epilogue of one 32-column chunk: the thread writes 64 (16-bit) or 128 (fp32) contiguous bytes of its row.  One value pair of it:
// MODE -1 tests the flags for every pair; the modes of the model (bf16 out) are compiled for themselves: without the tests the epilogue
// of a 128 x 256 tile takes a third of the instructions (NVFP4, M = 22 470, N = 4096, K = 1024, bf16 out: 78 -> 64 us).
constexpr int PL_BF16 = 0, PL_GELU = 1, PL_GELU_PRE = 2;
template <int MODE>
__device__ __forceinline__ float2 plain_pair(const GemmArgs& g, float2 a, float2 ts2, float2 bb) {
  const bool pre = MODE < 0 ? (g.flags & KF_G_PRE_ROUND_BF16) != 0 : MODE == PL_GELU_PRE;
  const bool gelu = MODE < 0 ? (g.flags & KF_G_GELU) != 0 : MODE != PL_BF16;
  float2 x = pre ? add2(bf16_round2(mul2(a, ts2)), bb) : fma2(a, ts2, bb);   // the result may be rounded to bf16 before the bias
  if (gelu) x = gelu_erf_pair(x);
  if (MODE < 0 && (g.flags & KF_G_ROUND_BF16)) x = bf16_round2(x);
  return x;
}
__device__ __forceinline__ void plain_chunk(const GemmArgs& g, const uint32_t (&r)[32], float ts, uint8_t* dst_row, int n0, const float* bsm /* the chunk's 32 bias values in shared memory, zeros without a bias */) {
  const float2 ts2 = splat2(ts);
#pragma unroll
  for (int q = 0; q < 2; ++q) {                 // 16 columns at a time
    float v[16];
#pragma unroll
    for (int h = 0; h < 8; ++h) {               // packed pairs
      const int k = 16 * q + 2 * h;
      const float2 x = plain_pair<-1>(g, make_float2(__uint_as_float(r[k]), __uint_as_float(r[k + 1])), ts2, *reinterpret_cast<const float2*>(bsm + k));
      v[2 * h] = x.x;
      v[2 * h + 1] = x.y;
    }
    if (dst_row) {
      if (g.out_dtype == KF_F32) {
        float* d = reinterpret_cast<float*>(dst_row) + n0 + 16 * q;
        stg8(d, v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]);
        stg8(d + 8, v[8], v[9], v[10], v[11], v[12], v[13], v[14], v[15]);
      } else {
        uint32_t w[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) w[e] = pack2(v[2 * e], v[2 * e + 1], g.out_dtype);
        stg8w(dst_row + (size_t)(n0 + 16 * q) * 2, w);
      }
    }
  }
}
// bf16 output without a row mapping: the warp's 32 rows x W columns; W = 64 leaves as whole lines
template <int MODE, int W>
__device__ __forceinline__ void plain_rows(const GemmArgs& g, const uint32_t (&r)[W], float ts, int rbase, int n0, const float* bsm, int lane, int m_end) {
  const float2 ts2 = splat2(ts);
  uint32_t w[W / 2];
#pragma unroll
  for (int k = 0; k < W; k += 4) {
    const float4 bb = *reinterpret_cast<const float4*>(bsm + k);
    const float2 x = plain_pair<MODE>(g, make_float2(__uint_as_float(r[k]), __uint_as_float(r[k + 1])), ts2, make_float2(bb.x, bb.y));
    const float2 y = plain_pair<MODE>(g, make_float2(__uint_as_float(r[k + 2]), __uint_as_float(r[k + 3])), ts2, make_float2(bb.z, bb.w));
    w[k / 2] = pack2(x.x, x.y, KF_BF16);
    w[k / 2 + 1] = pack2(y.x, y.y, KF_BF16);
  }
  uint8_t* base = static_cast<uint8_t*>(g.C) + ((size_t)rbase * g.N + n0) * 2;
  if constexpr (W == 64) {
    store_rows128(w, base, (size_t)g.N * 2, m_end - rbase, lane);
  } else {
    if (rbase + lane < m_end) {
      stg8w(base + (size_t)lane * g.N * 2, w);
      stg8w(base + (size_t)lane * g.N * 2 + 32, w + 8);
    }
  }
}

// Fallback when the launch has no room for the whole vectors: the bias values (and for RES the LayerScale values) of the
// warp's 64 columns go to its shared-memory slice with one coalesced load per tile (the kernel's shared memory leaves
// little L1: a load inside the chunk loops would be an L2 round trip); the chunk loops then read them as broadcast
// float4s.  The store into the slice waits for the load, an L2 round trip at the head of the tile.
template <int EPI, int COUNT /* 64 or 32 values */>
__device__ __forceinline__ void epilogue_slice_stage(const GemmArgs& g, int n0, float* slice, int lane) {
  if (n0 >= g.N) return;
  const bool on = 2 * lane < COUNT;
  float2 b2 = make_float2(0.f, 0.f), g2 = make_float2(0.f, 0.f);
  if (on && g.bias) b2 = __ldg(reinterpret_cast<const float2*>(g.bias + n0) + lane);
  if (on && EPI == KF_EPI_RES) g2 = __ldg(reinterpret_cast<const float2*>(g.gamma + n0) + lane);
  __syncwarp();                                // every lane has finished reading the previous tile's values
  if (on) {
    reinterpret_cast<float2*>(slice)[lane] = b2;
    if (EPI == KF_EPI_RES) reinterpret_cast<float2*>(slice + 64)[lane] = g2;
  }
  __syncwarp();
}

// ------------------------------------------------------------------------------------------------ ROPE table slab
// Rotary tables whose columns 32..63 repeat columns 0..31 (KF_G_ROPE_HALF; true for the axial tables of DINOv3, where the
// angle vector is concatenated with itself): the 4 warps that share a TMEM lane quarter (the 4 heads of a 256-column tile)
// need the same 32 table rows.  Together they fetch them with coalesced loads BEFORE the wait for the accumulator (the L2
// latency runs under that wait, 4 float4 per thread held in registers), then park them in the quarter's slab:
// row j = [sin 0..31 | cos 0..31] of token rbase + j, 16-byte pieces XOR-swizzled by the row so that the row-layout reads
// of the epilogue (lane = row) are free of bank conflicts.
struct RopeSlabRegs {
  float4 v[4];
};
__device__ __forceinline__ void rope_slab_fetch(const GemmArgs& g, int rbase, int tid /* 0..127 within the quarter */, RopeSlabRegs& x) {
  const int f = tid & 15;                                            // piece of the row: 0..7 sin, 8..15 cos
  const float* tab = (f < 8 ? g.sin : g.cos) + ((f & 7) << 2);
  int t = (rbase + (tid >> 4)) % g.Ntok;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int m = rbase + (tid >> 4) + 8 * u;
    x.v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (u != 0) {
      t += 8;
      if (t >= g.Ntok) t = t - g.Ntok < g.Ntok ? t - g.Ntok : t % g.Ntok;
    }
    if (m < g.M) {
      if (t >= g.prefix) x.v[u] = __ldg(reinterpret_cast<const float4*>(tab + (size_t)(t - g.prefix) * 64));
    }
  }
}
__device__ __forceinline__ void rope_slab_store(float* slab, int tid, const RopeSlabRegs& x) {
  const int f = tid & 15;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int row = (tid >> 4) + 8 * u;
    *reinterpret_cast<float4*>(slab + row * 64 + ((f ^ (row & 7)) << 2)) = x.v[u];
  }
}
__device__ __forceinline__ void quarter_barrier(int quarter) { asm volatile("bar.sync %0, 128;" ::"r"(1 + quarter) : "memory"); }

// ------------------------------------------------------------------------------------------------ the fused epilogues
// One epilogue warp's share of a tile: rows rbase..rbase+31 (thread `lane` holds row rbase + lane of the accumulator) and W
// columns in r.  W = 64: columns n0..n0+63.  W = 32: columns n0..n0+31; ROPE then holds half of the rotation pairs of the
// head that starts at n0, columns j0..j0+15 in r[0..15] and 32+j0..32+j0+15 in r[16..31].
// `slice` / `gslice` point at the bias / LayerScale values of the columns from n0 in shared memory.
template <int EPI, int W, int MODE = -1>
__device__ __forceinline__ void epilogue_math(const GemmArgs& g, uint32_t (&r)[W], float ts, const Nv4Scale& sco, int rbase, int n0, int j0,
                                              const float* slice, const float* gslice /* RES: the LayerScale values of the warp's columns */,
                                              const float* slab /* ROPE: the quarter's table rows in shared memory, or null */, int lane,
                                              int m_end /* first row past the product: M, or the end of the tile's product in a batched launch */,
                                              const F8* res_ahead /* RES, W = 32: the row's residual values, already requested */) {
  const int m = rbase + lane;
  if (EPI == KF_EPI_ROPE) {
    // the 64 columns of this warp are one head of q, k or v and the thread's 64 values are one [token, head] row of the
    // output: first half of r = first, second half = second columns of the rotation pairs, so the rotary embedding needs no data exchange:
    //   lo' = lo*cos_lo - hi*sin_lo (tables of columns 0..31), hi' = hi*cos_hi + lo*sin_hi (tables of columns 32..63).
    // With KF_G_ROPE_HALF the table row of every token of the warp's quarter is already in shared memory (rope_slab_*).
    if (W == 32 && m >= g.M) return;            // W = 64: all lanes take part in the stores
    const int which = n0 / g.d, h = (n0 - which * g.d) >> 6;
    const int b = m / g.Ntok, t = m - b * g.Ntok;
    const bool rot = which < 2 && t >= g.prefix && m < g.M;
    const float* srow = slab + lane * 64;
    uint32_t wo[W == 64 ? 32 : 16];             // packed output: the columns of the first half, then those of the second
    const float2 ts2 = splat2(ts);
    // FORM 0: no rotation (v columns), 1: every row rotates, tables in the slab, 2: row by row
    auto columns = [&](auto form) {
      constexpr int FORM = decltype(form)::value;
      const float* sn = g.sin + (size_t)(rot ? t - g.prefix : 0) * 64;
      const float* cs = g.cos + (size_t)(rot ? t - g.prefix : 0) * 64;
#pragma unroll
      for (int c = 0; c < W / 8; ++c) {           // 4 rotation pairs at a time (few values live: the thread already holds W accumulators)
        const float4 bl = *reinterpret_cast<const float4*>(slice + j0 + 4 * c), bh = *reinterpret_cast<const float4*>(slice + 32 + j0 + 4 * c);
        const int j = 4 * c;
        const float2 lo[2] = {fma2(make_float2(__uint_as_float(r[j]), __uint_as_float(r[j + 1])), ts2, make_float2(bl.x, bl.y)),
                              fma2(make_float2(__uint_as_float(r[j + 2]), __uint_as_float(r[j + 3])), ts2, make_float2(bl.z, bl.w))};
        const float2 hi[2] = {fma2(make_float2(__uint_as_float(r[W / 2 + j]), __uint_as_float(r[W / 2 + j + 1])), ts2, make_float2(bh.x, bh.y)),
                              fma2(make_float2(__uint_as_float(r[W / 2 + j + 2]), __uint_as_float(r[W / 2 + j + 3])), ts2, make_float2(bh.z, bh.w))};
        float2 ol[2] = {lo[0], lo[1]}, oh[2] = {hi[0], hi[1]};
        if (FORM == 1 || (FORM == 2 && rot)) {
          const int ct = (j0 >> 2) + c;           // 16-byte piece of the table row
          float4 s4, c4;                          // sin / cos of the 4 pairs: first for the lo outputs, then for the hi outputs
          if (FORM == 1 || slab != nullptr) {     // both halves of the tables are the same 32 values
            s4 = *reinterpret_cast<const float4*>(srow + ((ct ^ (lane & 7)) << 2));
            c4 = *reinterpret_cast<const float4*>(srow + (((ct + 8) ^ (lane & 7)) << 2));
          } else {
            s4 = ldg4_nc(sn + 4 * ct);
            c4 = ldg4_nc(cs + 4 * ct);
          }
          ol[0] = fma2(mul2(hi[0], splat2(-1.f)), make_float2(s4.x, s4.y), mul2(lo[0], make_float2(c4.x, c4.y)));   // -hi: one packed product, exact
          ol[1] = fma2(mul2(hi[1], splat2(-1.f)), make_float2(s4.z, s4.w), mul2(lo[1], make_float2(c4.z, c4.w)));
          if (FORM == 2 && slab == nullptr) {
            s4 = ldg4_nc(sn + 32 + 4 * ct);
            c4 = ldg4_nc(cs + 32 + 4 * ct);
          }
          oh[0] = fma2(hi[0], make_float2(c4.x, c4.y), mul2(lo[0], make_float2(s4.x, s4.y)));
          oh[1] = fma2(hi[1], make_float2(c4.z, c4.w), mul2(lo[1], make_float2(s4.z, s4.w)));
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          wo[2 * c + e] = pack2(ol[e].x, ol[e].y, g.out_dtype);
          wo[W / 4 + 2 * c + e] = pack2(oh[e].x, oh[e].y, g.out_dtype);
        }
      }
    };
    // Which form is the same for a warp: a test per value and per-row branches around the rotation doubled the instructions of the epilogue
    // (871 per warp and 128 x 256 tile; the rows of the cls / register tokens and of the general tables still take them)
    if (which == 2) columns(std::integral_constant<int, 0>{});
    else if (slab != nullptr && __all_sync(W == 64 ? 0xffffffffu : __activemask(), rot || m >= g.M)) columns(std::integral_constant<int, 1>{});
    else columns(std::integral_constant<int, 2>{});
    if constexpr (W == 64) {                    // rows of the output are [token, head] rows: row m of a third of q / k / v is b * Ntok + t = m
      store_rows128(wo, static_cast<uint8_t*>(g.C) + (((size_t)which * g.M + rbase) * g.H + h) * 128, (size_t)g.H * 128, g.M - rbase, lane);
    } else {
      uint8_t* dst = static_cast<uint8_t*>(g.C) + ((((size_t)which * (g.M / g.Ntok) + b) * g.Ntok + t) * g.H + h) * 128;
      stg8w(dst + 2 * j0, wo);
      stg8w(dst + 64 + 2 * j0, wo + 8);
    }
  } else if (EPI == KF_EPI_RES) {
    // out = R + gamma * (acc*ts + bias) on the thread's 256 (or 128) contiguous bytes of the fp32 residual row: 32-byte pieces,
    // four residual loads in flight ahead of the arithmetic (W = 32: all of them since before the accumulator was complete).
    if (m >= g.M) return;
    const float* rrow = g.R + (size_t)m * g.N + n0;
    const int64_t orow = g.row_group > 0 ? (int64_t)(m / g.row_group) * g.row_stride + g.row_offset + m % g.row_group : m;   // the output may be a longer stream
    float* crow = static_cast<float*>(g.C) + (size_t)orow * g.N + n0;
    const float2 ts2 = splat2(ts);
    F8 rr[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) rr[c] = W == 32 ? res_ahead[c] : ldg8_stream(rrow + 8 * c);
#pragma unroll
    for (int c = 0; c < W / 8; ++c) {
      const uint32_t* acc = &r[8 * c];
      const F8 cur = rr[c & 3];
      if (c + 4 < W / 8) rr[c & 3] = ldg8_stream(rrow + 8 * (c + 4));
      float o[8];
#pragma unroll
      for (int e = 0; e < 8; e += 2) {
        const float2 bb = *reinterpret_cast<const float2*>(slice + 8 * c + e), gg = *reinterpret_cast<const float2*>(gslice + 8 * c + e);
        const float2 v = fma2(make_float2(__uint_as_float(acc[e]), __uint_as_float(acc[e + 1])), ts2, bb);
        const float2 w = fma2(gg, v, make_float2(cur.v[e], cur.v[e + 1]));
        o[e] = w.x;
        o[e + 1] = w.y;
      }
      stg8(crow + 8 * c, o[0], o[1], o[2], o[3], o[4], o[5], o[6], o[7]);
    }
  } else if (EPI == KF_EPI_PLAIN && MODE >= 0) {
    plain_rows<(MODE < 0 ? 0 : MODE), W>(g, r, ts, rbase, n0, slice, lane, m_end);
  } else if (EPI == KF_EPI_PLAIN) {
    uint8_t* dst_row = nullptr;
    if (m < m_end) {
      const int64_t orow = g.row_group > 0 ? (int64_t)(m / g.row_group) * g.row_stride + g.row_offset + m % g.row_group : m;
      dst_row = static_cast<uint8_t*>(g.C) + (size_t)orow * g.N * (g.out_dtype == KF_F32 ? 4 : 2);
    }
#pragma unroll
    for (int c = 0; c < W; c += 32) plain_chunk(g, reinterpret_cast<const uint32_t(&)[32]>(r[c]), ts, dst_row, n0 + c, slice + c);
  } else {   // KF_EPI_QUANT: gelu(acc*ts + bias) -> codes + blocked scales of format out_fmt
#pragma unroll
    for (int c = 0; c < W; c += 32) quant_chunk<MODE>(g, reinterpret_cast<const uint32_t(&)[32]>(r[c]), ts, sco, m, n0 + c, slice + c);
  }
}

// RES through shared memory: 32 rows x 32 columns of the residual (all of a warp's columns where BN = 128) come as one TMA box (128-byte rows, swizzled),
// are updated in place in shared memory and leave as one box.  Every request is then a whole 128-byte line: a read-modify-write of
// 22 470 x 1024 fp32 takes 33.0 us this way and 39.9 us with the 32-byte accesses of the row layout (copy: 32.7 us).
constexpr int RES_BOX_BYTES = 32 * 128;
constexpr int PACE_POLLS = 1000;                        // a turn that does not come within about 100 us is taken anyway: order, not correctness, hangs on it
__device__ __forceinline__ void epilogue_res_tma(const GemmArgs& g, const uint32_t (&r)[32], float ts, const float* slice, const float* gslice, uint8_t* box, int lane) {
  const float2 ts2 = splat2(ts);
  uint8_t* row = box + lane * 128;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    float4* q = reinterpret_cast<float4*>(row + ((c ^ (lane & 7)) << 4));
    const float4 bb = *reinterpret_cast<const float4*>(slice + 4 * c), gg = *reinterpret_cast<const float4*>(gslice + 4 * c), x = *q;
    const float2 v0 = fma2(make_float2(__uint_as_float(r[4 * c]), __uint_as_float(r[4 * c + 1])), ts2, make_float2(bb.x, bb.y));
    const float2 v1 = fma2(make_float2(__uint_as_float(r[4 * c + 2]), __uint_as_float(r[4 * c + 3])), ts2, make_float2(bb.z, bb.w));
    const float2 o0 = fma2(make_float2(gg.x, gg.y), v0, make_float2(x.x, x.y)), o1 = fma2(make_float2(gg.z, gg.w), v1, make_float2(x.z, x.w));
    *q = make_float4(o0.x, o0.y, o1.x, o1.y);
  }
}

// First A / C row of row tile m_blk and the first row past its product (batched launches: row tiles never straddle two
// products, the last tile of a product is cut at the product's end); the first W row of the column tile that starts at n0.
__device__ __forceinline__ int tile_row0(const GemmArgs& g, int m_blk, int& row_end) {
  if (g.m_tiles_pb > 0) {
    const int b = m_blk / g.m_tiles_pb, mt = m_blk - b * g.m_tiles_pb;
    row_end = (b + 1) * g.a_rows_pb;
    return b * g.a_rows_pb + mt * BM;
  }
  row_end = g.M;
  return m_blk * BM;
}
__device__ __forceinline__ int tile_wrow0(const GemmArgs& g, int m_blk, int n0) { return (g.m_tiles_pb > 0 ? (m_blk / g.m_tiles_pb) * g.w_rows_pb : 0) + n0; }

// ------------------------------------------------------------------------------------------------ tile schedules and the epilogue warps' loop
// Work item idx of a launch: columns n0 .. n0 + cols - 1 of row tile m_blk.  Items are the tiles in row-major order; the tiles of a
// last round that would leave more than half of the SMs empty come as two halves of 128 columns (BN = 256, kf_gemm.cu).
struct WorkItem {
  int m_blk, n0, cols;
};
template <int BN>
__device__ __forceinline__ WorkItem work_item(const GemmArgs& g, int idx) {
  int tile = idx, half = 0, cols = BN;
  if (BN == 256 && idx >= g.full_tiles) {
    tile = g.full_tiles + ((idx - g.full_tiles) >> 1);
    half = (idx - g.full_tiles) & 1;
    cols = 128;
  }
  WorkItem w;
  w.m_blk = tile / g.n_tiles;
  w.n0 = (tile - w.m_blk * g.n_tiles) * BN + half * 128;
  w.cols = cols;
  return w;
}

// The form of a launch's options that has an epilogue, and a kernel, of its own, or -1 (all options).  QUANT: the output format, whatever the
// operands are; one kernel with all options for outputs of another format than the operands': NVFP4 in, MXFP8 out, 22 470 x 1024 x 4096 70.8 -> 90.7 us,
// MXFP8 in, NVFP4 out, 1605 x 768 x 3072 10.1 -> 12.6, bf16 in, NVFP4 out 12.0 -> 13.6.
static int epilogue_form(int epi, const GemmArgs& g) {
  if (epi == KF_EPI_PLAIN) {
    const int f = g.flags & (KF_G_PRE_ROUND_BF16 | KF_G_GELU | KF_G_ROUND_BF16);
    if (g.row_group > 0 || g.out_dtype != KF_BF16) return -1;
    return f == 0 ? PL_BF16 : f == KF_G_GELU ? PL_GELU : f == (KF_G_GELU | KF_G_PRE_ROUND_BF16) ? PL_GELU_PRE : -1;
  }
  if (epi == KF_EPI_QUANT) return g.y_dbg == nullptr && (g.flags & (KF_Q_ROUND_BF16 | KF_Q_FAST_NV4)) == KF_Q_ROUND_BF16 ? g.out_fmt : -1;
  return -1;
}
// run(epilogue, form) with the launch's constants as types
template <typename Run>
static int with_epilogue(int epi, const GemmArgs& g, Run&& run) {
  constexpr std::integral_constant<int, -1> any{};
  constexpr std::integral_constant<int, KF_EPI_PLAIN> plain{};
  constexpr std::integral_constant<int, KF_EPI_QUANT> quant{};
  const int form = epilogue_form(epi, g);
  switch (epi) {
    case KF_EPI_PLAIN:
      switch (form) {
        case PL_BF16: return run(plain, std::integral_constant<int, PL_BF16>{});
        case PL_GELU: return run(plain, std::integral_constant<int, PL_GELU>{});
        case PL_GELU_PRE: return run(plain, std::integral_constant<int, PL_GELU_PRE>{});
        default: return run(plain, any);
      }
    case KF_EPI_RES: return run(std::integral_constant<int, KF_EPI_RES>{}, any);
    case KF_EPI_ROPE: return run(std::integral_constant<int, KF_EPI_ROPE>{}, any);
    default:
      switch (form) {
        case KF_FMT_MX8: return run(quant, std::integral_constant<int, KF_FMT_MX8>{});
        case KF_FMT_NV4: return run(quant, std::integral_constant<int, KF_FMT_NV4>{});
        case KF_FMT_MX4: return run(quant, std::integral_constant<int, KF_FMT_MX4>{});
        default: return run(quant, any);
      }
  }
}

// Body of the 16 epilogue warps (warp = (TMEM lane quarter, 64- or 32-column group)): per tile, stage the bias slice (and fetch
// the rotary-table rows), wait for the accumulator, take the warp's piece into registers, hand TMEM back at once and
// run the fused epilogue on the registers while the next tile's main loop fills the accumulator again.
// PAIR (CTA pairs, BN = 256): work items are counted per pair and name row tiles 2 * m_blk and 2 * m_blk + 1, one per CTA; the
// accumulator is handed back to the leader's MMA warp.
template <int EPI, int BN, bool PAIR, int FORM>
__device__ __forceinline__ void epilogue_warps(const GemmArgs& g, uint32_t tmem_base, uint64_t* tfull, uint64_t* tempty, float* slices,
                                               float* slabs, uint8_t* boxes, uint64_t* box_full, const volatile uint32_t* issued /* PAIR, RES: operand stages requested so far */, const CUtensorMap* tmR, const CUtensorMap* tmC, const WaitCtx& ctx, int warp,
                                               int lane) {
  constexpr int W = Tile<BN>::CW, ACCS = Tile<BN>::ACCS;
  constexpr bool PAIRS = EPI == KF_EPI_ROPE && W == 32;       // two warps share a head: its column pairs 0..15 and 16..31
  const int quarter = warp & 3;                 // TMEM lanes 32*quarter .. +31 are the ones this warp may read
  const int cg = (warp - EPI_WARP0) >> 2;       // which column group of the tile
  float* slice = slices + (warp - EPI_WARP0) * SLICE_FLOATS;
  // Where the launch left room for it, the bias vector (and the LayerScale vector) is brought into shared memory once per
  // CTA instead of 64 values per warp and tile: that load was an L2 round trip (400-700 clk) at the head of every tile of
  // warps that are the busy role of these kernels.
  const bool vec = g.vec_floats > 0;
  if (vec) {
    const int tid = (warp - EPI_WARP0) * 32 + lane;
    for (int i = tid; i < g.N; i += EPI_WARPS * 32) {
      slices[i] = g.bias ? __ldg(g.bias + i) : 0.f;
      if (EPI == KF_EPI_RES) slices[g.N + i] = __ldg(g.gamma + i);
    }
    asm volatile("bar.sync 5, %0;" ::"r"(EPI_WARPS * 32) : "memory");
  }
  float ts = 1.f;
  if (g.ts_a) ts *= __ldg(g.ts_a);
  if (g.ts_w) ts *= __ldg(g.ts_w);
  const Nv4Scale sco = nv4_scale((EPI == KF_EPI_QUANT && g.out_fmt == KF_FMT_NV4) ? __ldg(g.tso) : 1.f);   // once per CTA: every global load here is an L2 round trip
  const int col = PAIRS ? (cg >> 1) * 64 : cg * W, j0 = PAIRS ? (cg & 1) * 16 : 0;
  const uint32_t taddr0 = tmem_base + ((uint32_t)(quarter * 32) << 16) + col + j0;
  // RES through shared memory: this warp's box and its barrier; the box of the next tile is requested when the present one has left
  constexpr bool BOXES = EPI == KF_EPI_RES && (W == 32 || PAIR);
  const bool boxed = BOXES && g.res_tma != 0;
  const int first = PAIR ? (int)blockIdx.x >> 1 : (int)blockIdx.x, stride = PAIR ? (int)gridDim.x >> 1 : (int)gridDim.x, rank = PAIR ? (int)cluster_ctarank() : 0;
  auto row_tile = [&](const WorkItem& w) { return PAIR ? 2 * w.m_blk + rank : w.m_blk; };
  const uint32_t leader_tempty = PAIR ? map_to_rank(tempty, 0) : 0;
  uint8_t* box = boxes + (warp - EPI_WARP0) * RES_BOX_BYTES;
  uint64_t* bfull = box_full + (warp - EPI_WARP0);
  uint32_t bph = 0;
  auto box_load = [&](int idx) {
    if (idx >= g.items) return;
    const WorkItem w = work_item<BN>(g, idx);
    const int row = row_tile(w) * BM + quarter * 32;
    if (row < g.M && col < w.cols && lane == 0) {
      mbar_expect_tx(bfull, RES_BOX_BYTES);
      tma_load_2d(box, tmR, (w.n0 + col) * 4, row, bfull);
    }
  };
  if (boxed) box_load(first);
  int lt = 0;
  // A warp takes one decision at every wait, and one whose wait for an accumulator ran out does not leave: it keeps company at the barriers
  // of its remaining tiles, which have no limit (ROPE: the four warps of a quarter meet at named ones, as often in all four: they depend
  // on the tile only), and stores nothing.
  bool live = true;
  for (int idx = first; idx < g.items; idx += stride, ++lt) {
    const WorkItem item = work_item<BN>(g, idx);
    int row_end;
    const int rbase = tile_row0(g, row_tile(item), row_end) + quarter * 32;
    const int n0 = item.n0 + col;               // first column of this warp's group (or of its head)
    const int acc = lt % ACCS;
    const uint32_t taddr = taddr0 + acc * BN;
    uint32_t r[W];
    if (!vec) epilogue_slice_stage<EPI, PAIRS ? 64 : W>(g, n0, slice, lane);
    const float* bsl = vec ? slices + n0 : slice;
    const float* gsl = vec ? slices + g.N + n0 : slice + 64;
    // ROPE with half tables: the quarter's table rows are fetched now and parked in shared memory after the wait
    const bool use_slab = EPI == KF_EPI_ROPE && (g.flags & KF_G_ROPE_HALF) != 0 && item.n0 < 2 * g.d;   // the tile holds q or k columns
    RopeSlabRegs tab;
    if (EPI == KF_EPI_ROPE && use_slab) rope_slab_fetch(g, rbase, cg * 32 + lane, tab);
    F8 res[4];
    if (EPI == KF_EPI_RES && W == 32 && !boxed && rbase + lane < g.M) {  // the residual's latency runs under the main loop
#pragma unroll
      for (int c = 0; c < 4; ++c) res[c] = ldg8_stream(g.R + (size_t)(rbase + lane) * g.N + n0 + 8 * c);
    }
    live = live && mbar_wait_warp(&tfull[acc], (lt / ACCS) & 1, ctx, 4);
    tc_fence_after();
    __syncwarp();
    if constexpr (W == 64) {
      tmem_ld32(taddr, reinterpret_cast<uint32_t(&)[32]>(r[0]));
      tmem_ld32(taddr + 32, reinterpret_cast<uint32_t(&)[32]>(r[32]));
    } else if constexpr (PAIRS) {
      tmem_ld16(taddr, reinterpret_cast<uint32_t(&)[16]>(r[0]));
      tmem_ld16(taddr + 32, reinterpret_cast<uint32_t(&)[16]>(r[16]));
    } else {
      tmem_ld32(taddr, r);
    }
    tmem_ld_wait();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) {                                          // the accumulator is in registers: hand TMEM back
      if (PAIR) mbar_arrive_remote(leader_tempty);
      else mbar_arrive(&tempty[acc]);
    }
    float* slab = nullptr;
    if (EPI == KF_EPI_ROPE && use_slab) {                      // all 4 warps of the quarter take this path together (it depends on the tile only)
      slab = slabs + quarter * ROPE_SLAB_FLOATS;
      quarter_barrier(quarter);                                // the previous tile's rows have been read by all four warps
      rope_slab_store(slab, cg * 32 + lane, tab);
      quarter_barrier(quarter);
    }
    if (!live || n0 >= g.N || col >= item.cols) continue;      // column group past N in the last column tile, or past a half tile
    if (PAIR && rbase >= g.m_tiles * BM) continue;             // the follower's row tile past the last one
    if constexpr (BOXES) {
      if (boxed) {
        // The column groups take turns over the next tile's main loop: 16 warps' boxes at once (64 KB of loads, then of stores, twice a
        // tile) held up the operand loads in the same queue.  A turn is a fifth of the main loop, counted in the stages its producer has
        // requested (which run a ring ahead of the products), so it is the same part of it in every format and at every clock.  None -> turns of
        // 75 ns a stage -> a fifth, us: NVFP4 22 470 x 4096 x 1024 62.9 -> 60.4 -> 58.4, 51 360 rows 132.8 -> 124.7 -> 120.3, MXFP4 129.5 -> 118.1 -> 114.9,
        // MXFP8 22 470 95.7 -> 91.2 -> 88.5, bf16 153.1 -> 151.0 -> 149.5; an eighth: NVFP4 60.2, 123.8, a third: 61.6, 126.7.  Not for a CTA's last
        // tile, where it would only come later.
        if (PAIR && cg != 0 && idx + stride < g.items) {
          const uint32_t turn = (uint32_t)((lt + 1) * g.k_tiles + min(g.k_tiles, g.stages + cg * g.k_tiles / 5));
          if (lane == 0)
            for (int i = 0; i < PACE_POLLS && (int32_t)(*issued - turn) < 0 && !*ctx.abort_flag; ++i) __nanosleep(100);
          __syncwarp();
        }
        bool lost = false;
        if (rbase < g.M) {
#pragma unroll
          for (int c = 0; c < W; c += 32) {                      // W = 64: two boxes, one after the other through the same 4 KB
            if (c != 0 && lane == 0) {
              mbar_expect_tx(bfull, RES_BOX_BYTES);
              tma_load_2d(box, tmR, (n0 + c) * 4, rbase, bfull);
            }
            if (!mbar_wait_warp(bfull, bph, ctx, 5)) {
              lost = true;
              break;
            }
            bph ^= 1;
            epilogue_res_tma(g, reinterpret_cast<const uint32_t(&)[32]>(r[c]), ts, bsl + c, gsl + c, box, lane);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              tma_store_2d(tmC, box, (n0 + c) * 4, rbase);
              bulk_commit();
              bulk_wait_read();
            }
          }
        }
        if (lost) break;
        box_load(idx + stride);
        __syncwarp();
        continue;
      }
    }
    epilogue_math<EPI, W, FORM>(g, r, ts, sco, rbase, n0, j0, bsl, gsl, slab, lane, row_end, res);
  }
  if (boxed && lane == 0) bulk_wait_all();
}

constexpr int REGS_LEAN = 40, REGS_EPI = 104;          // 128 * 40 + 512 * 104 <= 640 * 96, the allocation at launch
constexpr int REGS_LEAN_ROPE = 32, REGS_EPI_ROPE = 112; // the ROPE epilogue spills at 104 registers (64 accumulators + packed outputs + table values)

}  // namespace kf
