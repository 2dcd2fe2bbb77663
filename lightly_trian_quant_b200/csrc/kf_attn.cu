// FlashAttention-style forward on the sm_100a tensor cores (tcgen05.mma kind::f16, fp32 S and O in TMEM), head
// dimension 64, no mask, RoPE already applied by the qkv epilogue.
//
//   input    qkv [3, B, N, H, 64] bf16 | f16 (the physical layout the qkv GEMM epilogue writes)
//   output   O [B, N, H*64] bf16 | f16, or directly the quantised operand of the proj GEMM (kf_attn_fwd_quant)
//   CTA      persistent, two per SM; an item is 128 query rows of one (batch, head), key tiles of 96; a CTA takes the
//            items blockIdx.x, blockIdx.x + gridDim.x, ... and keeps every barrier phase running across them
//   roles    warps 0..3: softmax, one query row per thread (tcgen05.ld of the S row, running max / sum in fp32,
//            P -> 16 bit -> tensor memory by tcgen05.st); warp 4: TMA producer (Q in two buffers, K and V in 3-deep
//            rings, 4-D tensor maps so rows past N read zero); warp 5 issues the products (S = Q K^T: 4 MMAs of K=16
//            from shared memory; O += P V: 6 MMAs of K=16 with P as the A operand from tensor memory and V as the
//            MN-major B operand); warps 6 and 7 idle (they complete the second warp group, whose registers setmaxnreg
//            hands to the softmax warps: 208 against 48).
//   pipeline two S buffers in tensor memory, P(j) written over the first half of S(j); O accumulates over all key
//            tiles.  One thread issues PV(j) and then S(j+2) into the same buffer: the tensor core runs them in order,
//            so nothing waits for PV(j) to complete, also across the end of an item (the next item's Q and first K tiles
//            are loaded by then).  The softmax warps request two thirds of the next S row when two thirds of the present one
//            are used up, and ask for its barrier a third of a step before they look at the answer.  What bounds the kernel is their
//            instruction stream: two of them per scheduler take 1242 clk per 96-key step in a loop of nothing else (the
//            exponentials' unit: 1152), ~1660 here, where waits, S loads, the check of the row sum and the hand-over of P add
//            ~400 clk to every step of a warp, whatever its width.  That is why a step has 96 keys: with 64 (three S buffers, S two steps
//            ahead, the same tensor memory) a third more of them were paid; 128 leave no room for a second S buffer, and a last
//            tile of 128 pads the model's token counts more (1605 keys: 1632 with tiles of 96, 1664 with 64 or 128).
//            The exponentials of a tile
//            use the running maximum as it is; the tile's own row sum tells whether that was safe (below 2^15 no
//            element exceeded 2^15), so no maximum is tracked in the common case; only a row whose sum came out larger
//            finds its maximum, recomputes its P and has its O rescaled (TMEM load, multiply, store), which happens on
//            the first tiles and then almost never; the O barriers are waited only then and at the end of an item.
//            Measured, tiles of 64 -> 96 keys (B 14, H 16, N 1605, bf16 out / NVFP4 out; N 1805, NVFP4 out; B 8, N 4101, f16,
//            MXFP4 out; B 1, N 1605, NVFP4 out): 199 -> 186 / 204 -> 194 / 250 -> 239 / 667 -> 636 / 24.7 -> 23.6 us; 256-bit stores of the output
//            where it is 32-byte aligned: 186 -> 184.3 / 191.1 -> 190.5 / 236.2 -> 235.4 us (16-byte pieces of a row per lane cost twice the look-ups).
//            Few tokens paid for the wider tiles (B 1, H 12, N 261, MXFP8 out 6.5 -> 6.7 us, captured) until the quantising forms stopped spilling: 6.15.
//            Not kept: the barrier asked for only where it is waited on (198 us against 194), the next row requested at the end of the
//            step (199), five of sixteen pairs or none of every third 32 off the special-function unit (202, 202), an item's output behind the
//            first step of the next one (203: the waits it hides are fewer than the registers it takes from the loop); with
//            tiles of 64: four CTAs per SM with one S buffer each, two softmax warps per row with an O each, the end of a step
//            spread over the exponentials of the next one (level or slower).
//   numerics softmax scale 1/8 folded into exp2 (fp32; three of every four element pairs by the special-function unit,
//            the fourth by a cubic on the FMA pipe: the unit is shared by the softmax warps of both CTAs and is the
//            busiest pipe of the step; more than a quarter costs more issue slots than it frees); the exponent
//            arguments and the row sums as packed fp32 pairs; m, l, O in fp32; P rounded to the input 16-bit type.
//            Every mbarrier wait is bounded.
//
// Replaces a16::fwd_kernel / attn16_fwd (infer-opt/round12_lowp_stack/impl/attn16o.cu:126-404; mma.sync m16n8k16 +
// TMA on sm_120).  The power-of-two Q pre-scale `pre` of the reference protects its fp16 accumulators
// (attn16o.cu:184-194); with fp32 accumulation it is mathematically neutral and is accepted but not applied.
#include <type_traits>

#include "kf_sm100.cuh"

namespace kf {

constexpr int AT_BM = 128, AT_BN = 96, AT_D = 64;
constexpr int AT_THREADS = 256;                        // warps 0..3 softmax, 4 TMA, 5 MMA issuer, 6 and 7 idle
constexpr int AT_REGS_SOFTMAX = 208, AT_REGS_LEAN = 48; // 128 * 208 + 128 * 48 <= 256 * 128, the allocation at launch
constexpr int AT_KV = 3;                               // K / V ring depth
constexpr int AT_QTILE = AT_BM * AT_D * 2;             // 16 KB
constexpr int AT_KTILE = AT_BN * AT_D * 2;             // 12 KB
constexpr int AT_OFF_Q = 0, AT_OFF_K = 2 * AT_QTILE, AT_OFF_V = AT_OFF_K + AT_KV * AT_KTILE, AT_OFF_BAR = AT_OFF_V + AT_KV * AT_KTILE;
constexpr size_t AT_SMEM = (size_t)AT_OFF_BAR + 256;
constexpr float AT_SUM_LIMIT = 32768.f;                  // a tile's row sum above this sends the row to the exact-maximum path (the largest finite f16 is 65504)
constexpr int AT_POLY_K = 3;                             // element pairs AT_POLY_K .. 3 of every four take the polynomial exponential
constexpr int AT_SBUF = 2;                               // S buffers in tensor memory
constexpr int AT_TMEM_COLS = 256, AT_COL_S = 0, AT_COL_O = AT_SBUF * AT_BN;   // P (16-bit pairs, 48 columns) replaces the first half of its S buffer
static_assert(AT_COL_O + AT_D <= AT_TMEM_COLS, "TMEM budget");

struct AttnArgs {
  void* O;
  int B, N, H;
  int f16;          // 0 = bf16, 1 = f16
  float scale_log2; // softmax scale * log2(e)
  unsigned int* err;
  // optional fused quantisation of the output (the proj GEMM's A operand): out_fmt < 0 = off
  int out_fmt, flags;
  int wide;         // the output is 32-byte aligned: 256-bit stores
  uint8_t *Qo, *SFo;
  const float* tso;
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// 2^t for a pair without the special-function unit: t = n + f with n = round(t) taken from the low mantissa bits of
// t + 1.5 * 2^23 and f in [-0.5, 0.5]; 2^f by a cubic (minimax for the relative error on that interval: 7.6e-5, far
// below the rounding of the 16-bit P it feeds); n goes into the exponent field by an integer add.  t is clamped at -126
// (the result is then 2^-126 instead of 0: it vanishes in the 16-bit P and in the row sum alike) and at 127, behind which the add
// would wrap to anything, a small or a negative number too: a row with such an element has a sum that no limit lets pass.  A t that
// is no number passes the clamps and the add makes a huge element of it, with the same effect (a clamp that drops it would drop the key).  All of it runs on the
// FMA and integer pipes, as packed pairs where the operation exists.
// Clamps and no check of the largest t: that costs an instruction less, but a register through the key loop (captured, us: B 14, H 12, N 1605, MXFP8 out
// 137.5 against 135.3; B 1, H 16, N 1605 22.2 against 21.9).
__device__ __forceinline__ float clamp_ex2(float t) {
  asm("max.NaN.f32 %0, %0, 0fC2FC0000;\n\tmin.NaN.f32 %0, %0, 0f42FE0000;" : "+f"(t));   // [-126, 127]
  return t;
}
__device__ __forceinline__ float2 ex2_poly2(float2 t) {
  t.x = clamp_ex2(t.x);
  t.y = clamp_ex2(t.y);
  const float2 r = add2(t, splat2(12582912.f));
  const float2 n = add2(r, splat2(-12582912.f));
  const float2 f = fma2(n, splat2(-1.f), t);
  float2 p = fma2(f, splat2(0x1.c43e56p-5f), splat2(0x1.f0df98p-3f));
  p = fma2(p, f, splat2(0x1.62f24ap-1f));
  p = fma2(p, f, splat2(0x1.fff686p-1f));
  return make_float2(__int_as_float(__float_as_int(p.x) + (__float_as_int(r.x) << 23)), __int_as_float(__float_as_int(p.y) + (__float_as_int(r.y) << 23)));
}

__device__ __forceinline__ uint32_t pack16(float a, float b, int f16) {
  if (f16) {
    __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

// F16: 16-bit type of q / k / v / P / O (0 = bf16); OUT: -1 = plain 16-bit output, else the KF_FMT_* of the fused
// output quantisation.  Compile-time so that the softmax loop carries one copy of its code.
template <int F16, int OUT>
__global__ void __launch_bounds__(AT_THREADS, 2)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                const __grid_constant__ AttnArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + AT_OFF_BAR);
  uint64_t *q_full = bars, *q_empty = bars + 2, *k_full = bars + 4, *k_empty = k_full + AT_KV, *v_full = k_empty + AT_KV, *v_empty = v_full + AT_KV,
           *s_full = v_empty + AT_KV, *p_full = s_full + AT_SBUF, *o_full = p_full + AT_SBUF;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(o_full + AT_SBUF);
  volatile uint32_t* abort_flag = tmem_holder + 1;

  pdl_launch_dependents();                               // the next kernel of the stream may take the SMs this grid leaves
  const int warp = warp_index(), lane = threadIdx.x & 31;
  // Persistent: this CTA works through the (image, head, query tile) items blockIdx.x, blockIdx.x + gridDim.x, ...  All
  // barriers keep running across items: K / V ring stages, S / P buffers and the O barriers are indexed by the CTA's global
  // key-tile count G, the two Q buffers by the item count, so the loads and the first S products of the next item are
  // under way while the current one finishes and writes its output.
  const int q_tiles = (a.N + AT_BM - 1) / AT_BM;
  const int n_kt = (a.N + AT_BN - 1) / AT_BN;
  const int items = a.B * a.H * q_tiles;
  const int n_my = (int)blockIdx.x < items ? (items - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
  struct Item {
    int qt, h, b;
  };
  auto item_of = [&](int it) {
    const int item = blockIdx.x + it * gridDim.x;
    Item r;
    r.qt = item % q_tiles;
    const int bh = item / q_tiles;
    r.h = bh % a.H;
    r.b = bh / a.H;
    return r;
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
    }
    for (int i = 0; i < AT_KV; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 1);
    }
    for (int i = 0; i < AT_SBUF; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 128);
      mbar_init(&o_full[i], 1);                           // PV(G) completes o_full[G % 2]: a waiter is never more than one phase behind
    }
    *abort_flag = 0u;
    fence_mbar_init();
  }
  if (warp == 5) {
    tmem_alloc(tmem_holder, AT_TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();                                            // set-up done: from here on global memory of the predecessors is read and written
  const uint32_t tmem_base = *tmem_holder;
  const WaitCtx ctx{abort_flag, a.err};
  const bool bad_align = (smem_u32(smem) & 1023u) != 0;  // the swizzled tiles need a 1024-byte aligned base; the same answer in every thread
  if (bad_align && threadIdx.x == 0 && atomicCAS(&a.err[0], 0u, 99u) == 0u) {
    a.err[1] = 100;
    a.err[2] = blockIdx.x;
  }

  if (warp >= 4) {
  setmaxnreg_dec<AT_REGS_LEAN>();
  if (bad_align) {
    // nothing was issued; fall through to the teardown
  } else if (warp == 4) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      prefetch_tmap(&tmQ);
      prefetch_tmap(&tmK);
      prefetch_tmap(&tmV);
    }
    uint32_t st = 0, ph = 1;                                                      // ring slot and the parity of its release
    // Has an earlier launch failed?  The producer alone looks, once: without its loads the other roles' waits end with the abort flag.
    bool ok = !__any_sync(0xffffffffu, *static_cast<volatile unsigned int*>(a.err) != 0u);
    if (!ok) *abort_flag = 1u;
    for (int it = 0; it < n_my && ok; ++it) {
      const Item I = item_of(it);
      const int qb = it & 1;
      if (!mbar_wait_warp(&q_empty[qb], ((it >> 1) & 1) ^ 1, ctx, 10)) break;       // the S products of item it - 2 are done with this buffer
      if (elect_one()) {
        mbar_expect_tx(&q_full[qb], AT_QTILE);
        tma_load_4d(smem + AT_OFF_Q + qb * AT_QTILE, &tmQ, 0, I.h, I.qt * AT_BM, I.b, &q_full[qb]);
      }
      for (int j = 0; j < n_kt; ++j) {
        if (!mbar_wait_warp(&k_empty[st], ph, ctx, 11)) { ok = false; break; }      // S(G - AT_KV) is complete
        if (elect_one()) {
          mbar_expect_tx(&k_full[st], AT_KTILE);
          tma_load_4d(smem + AT_OFF_K + st * AT_KTILE, &tmK, 0, I.h, j * AT_BN, I.b, &k_full[st]);
        }
        __syncwarp();
        if (!mbar_wait_warp(&v_empty[st], ph, ctx, 15)) { ok = false; break; }      // PV(G - AT_KV) is complete
        if (elect_one()) {
          mbar_expect_tx(&v_full[st], AT_KTILE);
          tma_load_4d(smem + AT_OFF_V + st * AT_KTILE, &tmV, 0, I.h, j * AT_BN, I.b, &v_full[st]);
        }
        __syncwarp();
        if (++st == AT_KV) {
          st = 0;
          ph ^= 1;
        }
      }
    }
  } else if (warp == 5) {
    // ------------------------------------------------------------------ MMA issuer
    // S(0), S(1), then PV(G) and S(G + 2) for every step.  All come from one thread, so the tensor core runs them in
    // order: S(G + 2) overwrites the buffer of P(G) behind PV(G) without a wait for its completion.  A softmax that sees
    // S(G + 2) complete knows that PV(G) is.  S(G + 2) comes ~700 clk after the hand-over of P(G); the softmax asks for it ~1000 clk
    // into step G + 1.
    const uint32_t idesc_s = idesc_f16(F16 ? 0u : 1u, AT_BN);
    const uint32_t idesc_o = idesc_f16(F16 ? 0u : 1u, AT_D) | (1u << 16);     // B (= V) is MN-major
    const uint32_t t_o = tmem_base + AT_COL_O;
    const uint32_t total = (uint32_t)n_my * (uint32_t)n_kt;                  // key-tile steps of this CTA over all its items
    const bool leader = elect_one();
    uint32_t s_it = 0, s_j = 0;                                              // item and key tile of the next S product
    uint32_t k_st = 0, k_ph = 0;                                             // its slot in the K ring and the parity of the load
    auto issue_s = [&](uint32_t buf) {
      const uint64_t qdesc = smem_desc_sw128(smem_u32(smem + AT_OFF_Q + (s_it & 1) * AT_QTILE));
      const uint64_t kdesc = smem_desc_sw128(smem_u32(smem + AT_OFF_K + k_st * AT_KTILE));
      const uint32_t t_s = tmem_base + AT_COL_S + buf * AT_BN;
      const bool last = s_j + 1 == (uint32_t)n_kt;
      if (leader) {
#pragma unroll
        for (int kk = 0; kk < AT_D / 16; ++kk) mma_f16(t_s, qdesc + 2 * kk, kdesc + 2 * kk, idesc_s, kk != 0);
        tc_commit(&s_full[buf]);
        tc_commit(&k_empty[k_st]);
        if (last) tc_commit(&q_empty[s_it & 1]);                             // the item's last S product: its Q buffer is free once it completes
      }
      __syncwarp();
      if (++s_j == (uint32_t)n_kt) {
        s_j = 0;
        ++s_it;
      }
      if (++k_st == AT_KV) {
        k_st = 0;
        k_ph ^= 1;
      }
    };
    bool ok = true;
    for (uint32_t G = 0; G < AT_SBUF && G < total && ok; ++G) {
      ok = (s_j != 0 || mbar_wait_warp(&q_full[s_it & 1], (s_it >> 1) & 1, ctx, 12)) && mbar_wait_warp(&k_full[k_st], k_ph, ctx, 13);
      tc_fence_after();
      if (ok) issue_s(G);
    }
    uint32_t j = 0, buf = 0, pph = 0;                                        // buffer of step G and the parity of its P barrier
    uint32_t st = 0, vph = 0;                                                // V ring
    for (uint32_t G = 0; G < total && ok; ++G) {
      const bool more = G + AT_SBUF < total;
      if (more && s_j == 0 && !mbar_wait_warp(&q_full[s_it & 1], (s_it >> 1) & 1, ctx, 12)) break;
      // P(G), V(G) and the K tile of S(G + 2), asked for together: a barrier costs a round trip of 60 clk also when its phase is complete
      if (more) {
        if (!mbar_wait_warp3(&p_full[buf], pph, &v_full[st], vph, &k_full[k_st], k_ph, ctx, 14)) break;
      } else {
        if (!mbar_wait_warp3(&p_full[buf], pph, &v_full[st], vph, &v_full[st], vph, ctx, 14)) break;
      }
      tc_fence_after();
      const uint32_t t_p = tmem_base + AT_COL_S + buf * AT_BN;
      const uint64_t vdesc = smem_desc_sw128(smem_u32(smem + AT_OFF_V + st * AT_KTILE));
      if (leader) {
#pragma unroll
        for (int kk = 0; kk < AT_BN / 16; ++kk)  // A: 16 keys = 8 TMEM columns of P; B: 16 key rows of V = two 8-row groups of 1024 bytes
          mma_f16_ta(t_o, t_p + 8 * kk, vdesc + (uint64_t)(kk * (2048 >> 4)), idesc_o, (j | (uint32_t)kk) != 0);
        tc_commit(&o_full[buf]);
        tc_commit(&v_empty[st]);
      }
      __syncwarp();
      if (more) issue_s(buf);
      if (++j == (uint32_t)n_kt) j = 0;
      if (++buf == AT_SBUF) {
        buf = 0;
        pph ^= 1;
      }
      if (++st == AT_KV) {
        st = 0;
        vph ^= 1;
      }
    }
  }   // warps 6 and 7 are idle: they complete the second warp group, whose registers go to the softmax warps
  } else {
    setmaxnreg_inc<AT_REGS_SOFTMAX>();
    if (!bad_align) {
    // ------------------------------------------------------------------ softmax: thread = query row
    const int row = warp * 32 + lane;
    const uint32_t t_lane = tmem_base + ((uint32_t)(warp * 32) << 16);
    const float sc = a.scale_log2;
    bool ok = true;
    uint32_t buf = 0, sph = 0;                                   // the next step's S buffer and the parity of its barriers
    // per-tensor scale of an NVFP4 output, its reciprocal and range check: one L2 round trip per CTA, not per item
    const Nv4Scale tsc = nv4_scale(OUT == KF_FMT_NV4 ? __ldg(a.tso) : 1.f);
    const float2 sc2 = splat2(sc);
    // P = exp2(s*sc + mneg) of 32 keys as 16-bit pairs; adds the row sum to s0 / s1.  The exponent arguments and the row
    // sums run as packed pairs: half the issue slots of the scalar form.
    auto exp_half = [&](const uint32_t (&r)[32], uint32_t* w, float2 mn2, float2& s0, float2& s1) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float2 p[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float2 t = fma2(make_float2(__uint_as_float(r[8 * i + 2 * k]), __uint_as_float(r[8 * i + 2 * k + 1])), sc2, mn2);
          p[k] = k >= AT_POLY_K ? ex2_poly2(t) : make_float2(ex2(t.x), ex2(t.y));   // one pair in four off the special-function unit
        }
        s0 = add2(s0, add2(p[0], p[1]));
        s1 = add2(s1, add2(p[2], p[3]));
#pragma unroll
        for (int k = 0; k < 4; ++k) w[4 * i + k] = pack16(p[k].x, p[k].y, F16);
      }
    };
    auto row_max = [](const uint32_t (&r)[32], float mx) {
      float m4[4] = {mx, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < 16; ++i) m4[i & 3] = max3(m4[i & 3], __uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
      return amax_nan(amax_nan(m4[0], m4[1]), amax_nan(m4[2], m4[3]));
    };
    auto store32 = [&](uint8_t* dst, const uint32_t* w) {
      if (a.wide) {
        stg8w(dst, w);
      } else {
        reinterpret_cast<uint4*>(dst)[0] = make_uint4(w[0], w[1], w[2], w[3]);
        reinterpret_cast<uint4*>(dst)[1] = make_uint4(w[4], w[5], w[6], w[7]);
      }
    };
    auto mask_tail = [&](uint32_t (&r)[32], int key0) {          // columns past N never win the max and give P = 0
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (key0 + i >= a.N) r[i] = 0xff800000u;
    };
    for (int it = 0; it < n_my && ok; ++it) {
    float m_run = 0.f, l_run = 0.f;
    uint32_t ra[32], rb[32], rc[32];                             // the S row of this step: keys 0..31, 32..63 and 64..95 of the tile
    ok = mbar_wait_warp(&s_full[buf], sph, ctx, 17);
    if (!ok) break;
    tc_fence_after();
    tmem_ld32(t_lane + AT_COL_S + buf * AT_BN, ra);
    tmem_ld32(t_lane + AT_COL_S + buf * AT_BN + 32, rb);
    tmem_ld32(t_lane + AT_COL_S + buf * AT_BN + 64, rc);
    for (int j = 0; j < n_kt; ++j) {
      const uint32_t t_s = t_lane + AT_COL_S + buf * AT_BN, cur = buf, cph = sph;
      if (++buf == AT_SBUF) {
        buf = 0;
        sph ^= 1;
      }
      const bool prefetch = j + 1 < n_kt;                        // the next step of this item
      const int kbase = j * AT_BN;
      tmem_ld_wait();
      tmem_ld_fence(ra);
      tmem_ld_fence(rb);
      tmem_ld_fence(rc);
      if (kbase + AT_BN > a.N) {
        mask_tail(ra, kbase);
        mask_tail(rb, kbase + 32);
        mask_tail(rc, kbase + 64);
      }
      if (j == 0) m_run = row_max(rb, row_max(ra, -INFINITY));
      const float2 mn2 = splat2(-m_run * sc);
      float2 s0 = make_float2(0.f, 0.f), s1 = s0;
      uint32_t w[48];
      exp_half(ra, w, mn2, s0, s1);
      // asked for here, looked at a third of a step later: S(G + 1) was issued at the end of the last step
      const bool ready = mbar_test_wait(&s_full[buf], sph);
      exp_half(rb, w + 16, mn2, s0, s1);
      // The next step's S row is requested as soon as the registers of this one are free
      if (prefetch) {
        if (!__all_sync(0xffffffffu, ready) && !mbar_wait_warp(&s_full[buf], sph, ctx, 17)) { ok = false; break; }
        tc_fence_after();
        tmem_ld32(t_lane + AT_COL_S + buf * AT_BN, ra);
        tmem_ld32(t_lane + AT_COL_S + buf * AT_BN + 32, rb);
      }
      exp_half(rc, w + 32, mn2, s0, s1);
      if (prefetch) tmem_ld32(t_lane + AT_COL_S + buf * AT_BN + 64, rc);
      // Lazy maximum without a maximum: the exponentials of tile j > 0 use the running maximum as it is, and the tile's
      // own row sum tells whether that was safe: while it stays below 2^15 no element exceeded 2^15 (bf16 / f16 P, the
      // fp32 sums and O have room for that), so the maximum of the tile is not needed at all.  That holds for the special-function unit,
      // whose results only grow (to infinity), and for the polynomial, whose argument is clamped.  Only a row whose sum came out larger (or infinite,
      // or no number) finds its maximum, raises the running maximum, recomputes its P and has its O rescaled.
      // The first tile has no running maximum yet and takes that of its first 64 keys (the 96 of the tile would do: the 64 leave the
      // bits of P what they were with tiles of 64).
      float sum = (s0.x + s0.y) + (s1.x + s1.y), alpha = 1.f;
      const bool need = !(sum <= AT_SUM_LIMIT);
      if (__any_sync(0xffffffffu, need)) {                    // warp-uniform; S is still in tensor memory: P replaces it only below
        uint32_t r[32];
        float mx = m_run;
#pragma unroll 1
        for (int c = 0; c < AT_BN / 32; ++c) {
          tmem_ld32(t_s + 32 * c, r);
          tmem_ld_wait();
          tmem_ld_fence(r);
          if (kbase + AT_BN > a.N) mask_tail(r, kbase + 32 * c);
          mx = row_max(r, mx);
        }
        if (need) {
          alpha = ex2((m_run - mx) * sc);
          m_run = mx;
        }
        s0 = s1 = make_float2(0.f, 0.f);
#pragma unroll 1
        for (int c = 0; c < AT_BN / 32; ++c) {
          tmem_ld32(t_s + 32 * c, r);
          tmem_ld_wait();
          tmem_ld_fence(r);
          if (kbase + AT_BN > a.N) mask_tail(r, kbase + 32 * c);
          if (c == 0) exp_half(r, w, splat2(-m_run * sc), s0, s1);
          else if (c == 1) exp_half(r, w + 16, splat2(-m_run * sc), s0, s1);
          else exp_half(r, w + 32, splat2(-m_run * sc), s0, s1);
        }
        sum = (s0.x + s0.y) + (s1.x + s1.y);
        // rescale O in tensor memory, where there is one: PV(G - 1) must have landed first.  Its barrier's previous completion,
        // PV(G - 3), is covered by S(G), which this step has read.
        if (j > 0) {
          const uint32_t pb = cur == 0 ? AT_SBUF - 1 : cur - 1;
          if (!mbar_wait_warp(&o_full[pb], cur == 0 ? cph ^ 1 : cph, ctx, 18)) { ok = false; break; }
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < 2; ++c) {
            tmem_ld32(t_lane + AT_COL_O + 32 * c, r);
            tmem_ld_wait();
            tmem_ld_fence(r);
#pragma unroll
            for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
            tmem_st32(t_lane + AT_COL_O + 32 * c, r);
          }
        }
      }
      l_run = l_run * alpha + sum;
      tmem_st32(t_s, *reinterpret_cast<const uint32_t(*)[32]>(w));   // the A operand of the PV product: 96 keys = 48 columns of 16-bit pairs
      tmem_st16(t_s + 32, w + 32);
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(&p_full[cur]);
    }
    // Where the item's rows go is worked out here and not before its key loop: with three values more in that the quantising forms spill
    // (B 1, N 261, H 12, MXFP8 / NVFP4 / MXFP4 out 6.28 / 6.41 / 6.55 -> 6.15 / 6.34 / 6.41 us, captured; the plain form has registers to spare
    // and takes the same time either way).
    const Item I = item_of(it);
    const int qt = I.qt, h = I.h, b = I.b;
    // the item's last PV product; its barrier's previous completion, PV(G - 3), is covered by S(G - 1), which has been read
    if (ok) ok = mbar_wait_warp(&o_full[buf == 0 ? AT_SBUF - 1 : buf - 1], buf == 0 ? sph ^ 1 : sph, ctx, 19);
    const int n = qt * AT_BM + row;
    if (ok) {
      tc_fence_after();
      uint32_t r0[32], r1[32];
      tmem_ld32(t_lane + AT_COL_O, r0);
      tmem_ld32(t_lane + AT_COL_O + 32, r1);
      tmem_ld_wait();
      if (n < a.N && OUT >= 0) {
        // O row of this head (64 values) -> rounded to the 16-bit type -> 4 nv4 blocks or 2 mx blocks, written as the
        // codes and scale bytes of row b*N + n, columns h*64.. of the [B*N, H*64] operand
        const float inv = 1.0f / l_run;
        const bool div_true = !(a.flags & KF_Q_RECIP_DIV);
        float v[64];
        const float2 inv2 = splat2(inv);
        auto norm_round = [&](auto is_f16) {                       // O / l rounded to the 16-bit type, as packed pairs
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            float2 x = mul2(make_float2(__uint_as_float(r0[i]), __uint_as_float(r0[i + 1])), inv2);
            float2 y = mul2(make_float2(__uint_as_float(r1[i]), __uint_as_float(r1[i + 1])), inv2);
            if (decltype(is_f16)::value) {
              x = __half22float2(__float22half2_rn(x));
              y = __half22float2(__float22half2_rn(y));
            } else {
              x = bf16_round2(x);
              y = bf16_round2(y);
            }
            v[i] = x.x;
            v[i + 1] = x.y;
            v[32 + i] = y.x;
            v[33 + i] = y.y;
          }
        };
        norm_round(std::integral_constant<int, F16>{});
        const size_t m = (size_t)b * a.N + n;
        const int d = a.H * AT_D;
        if (OUT == KF_FMT_NV4) {
          uint32_t o[8];
          float am[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            am[k] = 0.f;
#pragma unroll
            for (int i = 0; i < 16; i += 2) am[k] = max3(am[k], fabsf(v[16 * k + i]), fabsf(v[16 * k + i + 1]));
          }
          int by[4];
#pragma unroll
          for (int k = 0; k < 4; k += 2) {                       // two blocks at a time: their scalars on packed pairs
            const float(&b0)[16] = *reinterpret_cast<const float(*)[16]>(&v[16 * k]);
            const float(&b1)[16] = *reinterpret_cast<const float(*)[16]>(&v[16 * k + 16]);
            quant_nv4_pair16(b0, am[k], b1, am[k + 1], tsc, div_true, o + 2 * k, by[k], by[k + 1]);
          }
          const uint32_t word = (uint32_t)by[0] | ((uint32_t)by[1] << 8) | ((uint32_t)by[2] << 16) | ((uint32_t)by[3] << 24);
          store32(a.Qo + m * (d >> 1) + h * 32, o);
          *reinterpret_cast<uint32_t*>(a.SFo + sf_offset((int)m, h * 4, d >> 6)) = word;
        } else {
          uint32_t half = 0;
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const float(&va)[16] = *reinterpret_cast<const float(*)[16]>(&v[32 * k]);
            const float(&vb)[16] = *reinterpret_cast<const float(*)[16]>(&v[32 * k + 16]);
            float am = 0.f;
#pragma unroll
            for (int i = 0; i < 32; i += 2) am = max3(am, fabsf(v[32 * k + i]), fabsf(v[32 * k + i + 1]));
            int by;
            if (OUT == KF_FMT_MX8) {
              uint32_t o[8];
              quant_mx8<16>(va, am, div_true, o, by);
              quant_mx8<16>(vb, am, div_true, o + 4, by);
              store32(a.Qo + m * d + h * 64 + k * 32, o);
            } else {
              uint32_t o[4];
              quant_mx4<16>(va, am, div_true, o, by);
              quant_mx4<16>(vb, am, div_true, o + 2, by);
              *reinterpret_cast<uint4*>(a.Qo + m * (d >> 1) + h * 32 + k * 16) = make_uint4(o[0], o[1], o[2], o[3]);
            }
            half |= (uint32_t)by << (8 * k);
          }
          *reinterpret_cast<uint16_t*>(a.SFo + sf_offset((int)m, h * 2, d >> 7)) = (uint16_t)half;
        }
      } else if (n < a.N) {
        const float inv = 1.0f / l_run;
        uint32_t w[32];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          w[i] = pack16(__uint_as_float(r0[2 * i]) * inv, __uint_as_float(r0[2 * i + 1]) * inv, F16);
          w[16 + i] = pack16(__uint_as_float(r1[2 * i]) * inv, __uint_as_float(r1[2 * i + 1]) * inv, F16);
        }
        uint8_t* dst = static_cast<uint8_t*>(a.O) + (((size_t)b * a.N + n) * a.H + h) * (AT_D * 2);
#pragma unroll
        for (int i = 0; i < 4; ++i) store32(dst + 32 * i, w + 8 * i);
      }
    }
    }   // items
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag && !bad_align) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
  }
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc(tmem_base, AT_TMEM_COLS);
  }
}

// 4-D tensor map over one of q / k / v: dims (64, H, N, B) of 16-bit elements, box (64, 1, rows, 1), 128-byte swizzle;
// rows past N are out of bounds in their own dimension and read as zero.  Encoding costs about a microsecond of host time and
// a layer stack asks for the same few maps over and over: kept per thread, direct-mapped by their arguments.
static int make_tmap_qkv(CUtensorMap* map, const void* base, int B, int N, int H, int box_rows) {
  struct Slot {
    const void* base;
    int B, N, H, box_rows;
    CUtensorMap map;
  };
  constexpr int SLOTS = 64;
  static thread_local Slot cache[SLOTS] = {};
  const uintptr_t h = (reinterpret_cast<uintptr_t>(base) >> 8) * 0x9E3779B97F4A7C15ull + (uintptr_t)N * 31 + (uintptr_t)B * 7 + (uintptr_t)box_rows;
  Slot& slot = cache[(h >> 32 ^ h) % SLOTS];
  if (slot.base == base && slot.B == B && slot.N == N && slot.H == H && slot.box_rows == box_rows) {
    *map = slot.map;
    return KF_OK;
  }
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) {
    set_error("cuTensorMapEncodeTiled is not available from the driver");
    return KF_ERR_UNSUPPORTED;
  }
  cuuint64_t dims[4] = {64, (cuuint64_t)H, (cuuint64_t)N, (cuuint64_t)B};
  cuuint64_t strides[3] = {128, (cuuint64_t)H * 128, (cuuint64_t)N * H * 128};
  cuuint32_t box[4] = {64, 1, (cuuint32_t)box_rows, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 4, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled (qkv) failed with CUresult %d", (int)r);
    return KF_ERR_BAD_ARGUMENT;
  }
  slot = Slot{base, B, N, H, box_rows, *map};
  return KF_OK;
}

}  // namespace kf

using namespace kf;

static int attn_launch(int dtype, const void* qkv, void* O, int B, int N, int H, int out_fmt, void* Qo, void* SFo, const float* tso, int flags,
                       void* stream) {
  KF_REQUIRE(dtype == KF_BF16 || dtype == KF_F16, "kf_attn_fwd: dtype must be bf16 or f16");
  KF_REQUIRE(B >= 0 && N > 0 && H > 0, "kf_attn_fwd: bad shape B=%d N=%d H=%d", B, N, H);
  if (B == 0) return KF_OK;
  KF_REQUIRE(qkv && (reinterpret_cast<uintptr_t>(qkv) & 15) == 0, "kf_attn_fwd: qkv must be non-null and 16-byte aligned");
  if (out_fmt < 0) {
    KF_REQUIRE(O && (reinterpret_cast<uintptr_t>(O) & 15) == 0, "kf_attn_fwd: O must be non-null and 16-byte aligned");
  } else {
    KF_REQUIRE(out_fmt == KF_FMT_MX8 || out_fmt == KF_FMT_NV4 || out_fmt == KF_FMT_MX4, "kf_attn_fwd_quant: bad output format %d", out_fmt);
    KF_REQUIRE(Qo && SFo && (reinterpret_cast<uintptr_t>(Qo) & 15) == 0 && (reinterpret_cast<uintptr_t>(SFo) & 15) == 0,
               "kf_attn_fwd_quant: Qo and SFo must be non-null and 16-byte aligned");
    KF_REQUIRE(out_fmt != KF_FMT_NV4 || tso, "kf_attn_fwd_quant: nv4 needs the per-tensor scale");
    KF_REQUIRE((H * 64) % 128 == 0, "kf_attn_fwd_quant: H*64 must be a multiple of 128");
  }
  const size_t plane = (size_t)B * N * H * 64 * 2;
  const uint8_t* base = static_cast<const uint8_t*>(qkv);
  CUtensorMap tq, tk, tv;
  int st = make_tmap_qkv(&tq, base, B, N, H, AT_BM);
  if (st != KF_OK) return st;
  st = make_tmap_qkv(&tk, base + plane, B, N, H, AT_BN);
  if (st != KF_OK) return st;
  st = make_tmap_qkv(&tv, base + 2 * plane, B, N, H, AT_BN);
  if (st != KF_OK) return st;
  // one instantiation per 16-bit type and output form
  using KernelFn = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, AttnArgs);
  static const KernelFn table[2][4] = {
      {attn_fwd_kernel<0, -1>, attn_fwd_kernel<0, KF_FMT_MX8>, attn_fwd_kernel<0, KF_FMT_NV4>, attn_fwd_kernel<0, KF_FMT_MX4>},
      {attn_fwd_kernel<1, -1>, attn_fwd_kernel<1, KF_FMT_MX8>, attn_fwd_kernel<1, KF_FMT_NV4>, attn_fwd_kernel<1, KF_FMT_MX4>}};
  const int oi = out_fmt < 0 ? 0 : out_fmt == KF_FMT_MX8 ? 1 : out_fmt == KF_FMT_NV4 ? 2 : 3;
  const KernelFn kern = table[dtype == KF_F16 ? 1 : 0][oi];
  static PerDevice<bool> attr_set[2][4];
  int dev = 0;
  cudaGetDevice(&dev);
  PerDevice<bool>& ready = attr_set[dtype == KF_F16 ? 1 : 0][oi];
  if (!ready.get(dev)) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)AT_SMEM);
    if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute(attn_fwd_kernel)");
    ready.put(dev, true);
  }
  AttnArgs a{};
  a.O = O; a.B = B; a.N = N; a.H = H; a.f16 = dtype == KF_F16;
  a.scale_log2 = 0.125f * 1.4426950408889634f;
  a.err = dev_error_ptr();
  a.out_fmt = out_fmt; a.flags = flags; a.Qo = static_cast<uint8_t*>(Qo); a.SFo = static_cast<uint8_t*>(SFo); a.tso = tso;
  a.wide = (reinterpret_cast<uintptr_t>(out_fmt < 0 ? O : Qo) & 31) == 0;
  KF_REQUIRE(a.err != nullptr, "kf_attn_fwd: device error word unavailable");
  const int q_tiles = (N + AT_BM - 1) / AT_BM;
  const long long items = (long long)B * H * q_tiles;
  KF_REQUIRE(items < (1ll << 30), "kf_attn_fwd: too many (image, head, query tile) items");
  int sms = 0;
  const int sst = device_sm_count(&sms);
  if (sst != KF_OK) return sst;
  const int slots = 2 * sms;                                  // two CTAs are resident per SM
  const int grid = items < slots ? (int)items : slots;
  return cuda_status(launch_maybe_pdl((int64_t)B * N, kern, dim3(grid), dim3(AT_THREADS), (size_t)AT_SMEM, static_cast<cudaStream_t>(stream), tq, tk, tv, a),
                     "kf_attn_fwd launch");
}

extern "C" int kf_attn_fwd(int dtype, const void* qkv, void* O, int B, int N, int H, float pre, void* stream) {
  (void)pre;
  return attn_launch(dtype, qkv, O, B, N, H, -1, nullptr, nullptr, nullptr, 0, stream);
}

extern "C" int kf_attn_fwd_quant(int dtype, const void* qkv, int B, int N, int H, float pre, int out_fmt, void* Qo, void* SFo, const float* tso, int flags,
                                 void* stream) {
  (void)pre;
  return attn_launch(dtype, qkv, nullptr, B, N, H, out_fmt, Qo, SFo, tso, flags, stream);
}
