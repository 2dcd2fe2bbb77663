// Memory-bound producers of the block-scaled operands: the stand-alone row quantiser (optionally bias + GELU first),
// LayerNorm fused with quantisation, and LayerNorm to a 16-bit tensor.  All three stream each input element once
// from HBM with 16-byte loads issued up front, keep the row segment in registers and write codes with 8/16-byte
// stores and scale factors as whole 32-bit words of the 128x4 blocked layout.
//
// Bit rules (identical to the reference's torch quantiser, infer-opt/round10_lowp_probe/impl/quant_ref.py:92-154):
//   mx8  byte = min(exp(fl32(amax/448)) + (mant != 0), 255);  q = e4m3_rn_sat(clamp(x * 2^(127 - max(byte,1)), +-448))
//   mx4  byte = min(exp(fl32(amax/6))   + (mant != 0), 254);  q = e2m1_rn_sat(x * 2^(127 - byte))
//   nv4  sf = e4m3_rn(min((amax/6)/ts, 448));  q = e2m1_rn_sat(x / (float(sf) * ts)), 0 when the scale is 0
// LN + quant is persistent (warps stride over the rows) with the LayerNorm weight and bias of the lane's columns held
// in registers, so the only per-row loads are the row itself.
#include "kf_sm100.cuh"

namespace kf {

// ------------------------------------------------------------------------------------------------ loads
// 32 bytes of read-once input as eight words: one 256-bit load where the address allows it (`wide`), else two of 128 bits.
__device__ __forceinline__ void load32b(const void* p, bool wide, uint32_t* w) {
  if (wide) {
    asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
                 : "l"(p));
  } else {
    const uint4 a = __ldg(static_cast<const uint4*>(p)), b = __ldg(static_cast<const uint4*>(p) + 1);
    w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w; w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
  }
}
// two 16-bit values (first one in the low half) as floats
template <typename T>
__device__ __forceinline__ float2 unpack2(uint32_t w) {
  if constexpr (std::is_same<T, __half>::value) return __half22float2(*reinterpret_cast<__half2*>(&w));
  else return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
}

// 32 consecutive elements: all loads issued together, converted when they are needed
template <typename T>
constexpr int LOAD32_WORDS = 8 * (int)sizeof(T);          // 32-byte pieces: 4 of fp32, 2 of a 16-bit type
template <typename T>
__device__ __forceinline__ void load32_raw(const T* p, bool wide, uint32_t (&w)[LOAD32_WORDS<T>]) {
#pragma unroll
  for (int i = 0; i < (int)sizeof(T); ++i) load32b(reinterpret_cast<const uint8_t*>(p) + 32 * i, wide, w + 8 * i);
}
template <typename T>
__device__ __forceinline__ void unpack32(const uint32_t (&w)[LOAD32_WORDS<T>], float (&v)[32]) {
  if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(w[i]);
  } else {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float2 f = unpack2<T>(w[i]);
      v[2 * i] = f.x;
      v[2 * i + 1] = f.y;
    }
  }
}
template <typename T>
__device__ __forceinline__ void load32(const T* p, bool wide, float (&v)[32]) {
  uint32_t w[LOAD32_WORDS<T>];
  load32_raw<T>(p, wide, w);
  unpack32<T>(w, v);
}

// Gathers the scale bytes of 4 consecutive k-blocks (held by lanes lane0, lane0+STEP, ...) into one word on lane0.
template <int STEP>
__device__ __forceinline__ uint32_t gather_sf_word(int byte, int lane) {
  int base = lane & ~(4 * STEP - 1);
  uint32_t b0 = __shfl_sync(0xffffffffu, byte, base);
  uint32_t b1 = __shfl_sync(0xffffffffu, byte, base + STEP);
  uint32_t b2 = __shfl_sync(0xffffffffu, byte, base + 2 * STEP);
  uint32_t b3 = __shfl_sync(0xffffffffu, byte, base + 3 * STEP);
  return (b0 & 0xFF) | ((b1 & 0xFF) << 8) | ((b2 & 0xFF) << 16) | ((b3 & 0xFF) << 24);
}

// ------------------------------------------------------------------------------------------------ row quantiser
// One thread = 32 consecutive elements of one row: one mx block, or two nv4 blocks whose scalars go through the packed-pair
// quantiser of the GEMM epilogue.  No maximum crosses lanes; two (nv4) or four (mx) lanes share one scale word.
// Bound by HBM.  With 16 elements per thread (two lanes per mx block, the nv4 divisions scalar) the NVFP4 form was bound by
// instruction issue: 51 360 x 4096 bf16 139 us = 3.9 TB/s, then 103 us.  16-bit inputs: the grid is what is resident at once and a thread
// requests its next item before it quantises the present one (half of a thread's life had no load in flight): NVFP4 103 -> 86 us = 6.3 TB/s,
// MXFP8 102 -> 97, MXFP4 92 -> 84; 22 470 x 1024 16.5 -> 14.4; 6420 x 3072 12.8 -> 11.3.  fp32 inputs have twice the words in flight already
// and lose the residency to the second set of registers (22 470 x 1024 20.6 -> 24.5 us): one item per thread.
template <typename T, int FMT>
__global__ void __launch_bounds__(256) quant_rows_kernel(const T* __restrict__ x, int64_t ldx, int M, int K, const float* __restrict__ ts_ptr,
                                                         const float* __restrict__ bias, int flags, int wide, uint8_t* __restrict__ q,
                                                         uint8_t* __restrict__ sf, int64_t items_valid, int64_t items_total) {
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const uint32_t per_row = (uint32_t)K >> 5;
  // 32-bit index arithmetic (the host checks that the item count fits); a power-of-two row length needs no division
  const bool pow2 = (per_row & (per_row - 1)) == 0;
  const int log2_row = 31 - __clz((int)per_row);
  auto place = [&](uint32_t w, int& row, int& c32) {
    row = (int)(pow2 ? w >> log2_row : w / per_row);
    c32 = (int)(pow2 ? w & (per_row - 1) : w - (uint32_t)row * per_row);
  };
  const Nv4Scale ts = nv4_scale(FMT == KF_FMT_NV4 ? __ldg(ts_ptr) : 1.f);
  // Rows up to items_total exist in the blocked scale layout, those from items_valid on only get zero scale bytes.  Both counts are multiples
  // of a row, and a warp's 32 items lie on one side of items_total as a whole (128 rows of it): whole warps run the loop.
  const uint32_t valid_end = (uint32_t)items_valid, end = (uint32_t)items_total, stride = gridDim.x * 256u;
  uint32_t w32 = blockIdx.x * 256u + threadIdx.x;
  int row, c32;
  place(w32, row, c32);
  constexpr bool AHEAD = sizeof(T) == 2;
  uint32_t raw[LOAD32_WORDS<T>];
  if (AHEAD && w32 < valid_end) load32_raw<T>(x + (int64_t)row * ldx + c32 * 32, wide != 0, raw);
  for (;;) {
    const bool valid = w32 < valid_end, in_pad = w32 < end;
    float v[32];
    if (valid) {
      if (AHEAD) unpack32<T>(raw, v);
      else load32<T>(x + (int64_t)row * ldx + c32 * 32, wide != 0, v);
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = 0.f;
    }
    // 16-bit inputs: the next item's loads travel while this one is quantised
    const uint32_t next = w32 + stride;
    const bool more = AHEAD && __any_sync(0xffffffffu, next < end && next >= stride);
    int nrow = 0, nc32 = 0;
    if (more) {
      place(next, nrow, nc32);
      if (next < valid_end) load32_raw<T>(x + (int64_t)nrow * ldx + nc32 * 32, wide != 0, raw);
    }
    if constexpr (FMT == KF_FMT_NV4 && std::is_same<T, __half>::value) {
      // The corrected quotient of a negative zero is a positive one (code 0, the bit rule says 8).  fp16 inputs reach -0 by
      // underflow of ordinary values; a magnitude below any fp16 one takes its place.
      if (!(flags & KF_Q_GELU)) {
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(v[i]) == 0x80000000u ? -1e-20f : v[i];
      }
    }
    if ((flags & KF_Q_GELU) && valid) {
      const float4* b4 = reinterpret_cast<const float4*>(bias + c32 * 32);
#pragma unroll
      for (int i = 0; i < 32; i += 4) {
        const float4 bb = __ldg(b4 + (i >> 2));
        const float2 a = gelu_erf_pair(add2(make_float2(v[i], v[i + 1]), make_float2(bb.x, bb.y)));
        const float2 c = gelu_erf_pair(add2(make_float2(v[i + 2], v[i + 3]), make_float2(bb.z, bb.w)));
        v[i] = a.x;
        v[i + 1] = a.y;
        v[i + 2] = c.x;
        v[i + 3] = c.y;
      }
    }
    if (flags & KF_Q_ROUND_BF16) {
#pragma unroll
      for (int i = 0; i < 32; i += 2) {
        const float2 a = bf16_round2(make_float2(v[i], v[i + 1]));
        v[i] = a.x;
        v[i + 1] = a.y;
      }
    }
    float am0 = 0.f, am1 = 0.f;
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
      am0 = max3(am0, fabsf(v[i]), fabsf(v[i + 1]));
      am1 = max3(am1, fabsf(v[16 + i]), fabsf(v[17 + i]));
    }
    const bool div_true = !(flags & KF_Q_RECIP_DIV);
    const float(&va)[16] = *reinterpret_cast<const float(*)[16]>(&v[0]);
    const float(&vb)[16] = *reinterpret_cast<const float(*)[16]>(&v[16]);
    if constexpr (FMT == KF_FMT_NV4) {
      uint32_t o[4];
      int by0, by1;
      quant_nv4_pair16(va, am0, vb, am1, ts, div_true, o, by0, by1);
      if (valid) *reinterpret_cast<uint4*>(q + (int64_t)row * (K >> 1) + c32 * 16) = make_uint4(o[0], o[1], o[2], o[3]);
      const uint32_t pk = valid ? (uint32_t)(by0 | (by1 << 8)) : 0u;
      const uint32_t up = __shfl_xor_sync(0xffffffffu, pk, 1);           // on an even lane: the bytes of the word's other two blocks
      if (in_pad && (lane & 1) == 0) *reinterpret_cast<uint32_t*>(sf + sf_offset(row, 2 * c32, K >> 6)) = pk | (up << 16);
    } else {
      const float amax = amax_nan(am0, am1);
      int byte;
      if constexpr (FMT == KF_FMT_MX8) {
        uint32_t o[8];
        quant_mx8<16>(va, amax, div_true, o, byte);
        quant_mx8<16>(vb, amax, div_true, o + 4, byte);
        if (valid) {
          uint4* dst = reinterpret_cast<uint4*>(q + (int64_t)row * K + c32 * 32);
          dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
          dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
        }
      } else {
        uint32_t o[4];
        quant_mx4<16>(va, amax, div_true, o, byte);
        quant_mx4<16>(vb, amax, div_true, o + 2, byte);
        if (valid) *reinterpret_cast<uint4*>(q + (int64_t)row * (K >> 1) + c32 * 16) = make_uint4(o[0], o[1], o[2], o[3]);
      }
      if (!valid) byte = 0;
      const uint32_t word = gather_sf_word<1>(byte, lane);
      if (in_pad && (lane & 3) == 0) *reinterpret_cast<uint32_t*>(sf + sf_offset(row, c32, K >> 7)) = word;
    }
    if (!AHEAD || !more) break;
    w32 = next;
    row = nrow;
    c32 = nc32;
  }
}

// ------------------------------------------------------------------------------------------------ dynamic per-tensor scale
// The per-tensor scale of an NVFP4 operand measured on the values about to be quantised: ts = factor * max|v| (1 when that is
// zero or NaN), in one launch: block maxima meet in an atomic maximum on the bit patterns (non-negative floats order as
// integers, a NaN above them all), the last block writes ts and leaves the workspace (two words, zero before the first
// use) as it found it.  As six to nine elementwise launches with fp32 copies it was most of a swapped block: 6420 rows of
// ViT-B, four Linears: 457 -> 178 us.
__device__ __forceinline__ void amax_finish(float am, float factor, float* ts, uint32_t* ws) {
  __shared__ uint32_t part[32];
  uint32_t bits = __float_as_uint(am);
  bits = __reduce_max_sync(0xffffffffu, bits);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  if (lane == 0) part[warp] = bits;
  __syncthreads();
  if (warp != 0) return;
  bits = __reduce_max_sync(0xffffffffu, lane < nwarps ? part[lane] : 0u);
  if (lane != 0) return;
  atomicMax(&ws[0], bits);
  __threadfence();
  if (atomicAdd(&ws[1], 1u) == gridDim.x - 1) {
    const float peak = __uint_as_float(atomicExch(&ws[0], 0u));
    ws[1] = 0;
    *ts = peak > 0.f ? peak * factor : 1.f;
  }
}

// |gelu(x)| with the exact-erf definition, in the form the framework's eager GELU evaluates
__device__ __forceinline__ float gelu_abs(float x) { return fabsf(x * 0.5f * (1.0f + erff(x * 0.70710678118654752440f))); }

// max |v| or max |gelu(v)| over a matrix.  GELU rises for v >= 0 and stays within 0.17 of zero below, so of 32 values only the largest is
// evaluated, and the negative ones only while nothing above 0.17 has been seen (the GELU of 20 M values takes longer than reading
// them: 6420 x 3072 bf16 28 us with a test per value).  NaN and -Inf give NaN, as the eager GELU does.
constexpr float GELU_NEG_MAX = 0.17f;                      // above |gelu(-0.7518)| = 0.16997
__device__ __forceinline__ float min3(float a, float b, float c) {
  float y;
  asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
  return y;
}
template <typename T, bool GELU>
__global__ void __launch_bounds__(256) amax_scale_kernel(const T* __restrict__ x, int64_t ldx, int M, int K, int wide, float factor, float* __restrict__ ts,
                                                         uint32_t* __restrict__ ws) {
  pdl_wait();
  const uint32_t per_row = K >> 5, total = (uint32_t)M * per_row;
  float am = 0.f;
  for (uint32_t i = blockIdx.x * 256u + threadIdx.x; i < total; i += gridDim.x * 256u) {
    const uint32_t row = i / per_row, c = i - row * per_row;
    float v[32];
    load32<T>(x + (int64_t)row * ldx + c * 32, wide != 0, v);
    if (GELU) {
      float top = v[0], low = v[0];
#pragma unroll
      for (int j = 0; j < 32; j += 2) {
        top = max3(top, v[j], v[j + 1]);
        low = min3(low, v[j], v[j + 1]);
      }
      if (!(low >= -3.402823466e38f)) {
        am = __int_as_float(0x7fc00000);
      } else {
        if (top > am) am = fmaxf(am, gelu_abs(top));
        if (am < GELU_NEG_MAX && -low > am) {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (-v[j] > am) am = fmaxf(am, gelu_abs(v[j]));
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; j += 2) am = max3(am, fabsf(v[j]), fabsf(v[j + 1]));
    }
  }
  amax_finish(fabsf(am), factor, ts, ws);
}

// ------------------------------------------------------------------------------------------------ LayerNorm (+ quant)
// One warp per row; lane l holds the 8 consecutive elements [i*256 + l*8, +8) for i < NV (d = NV*256), as two pieces of
// four.  With BLK16 the lane's chunks pair up into runs of 16 consecutive elements (whole NVFP4 blocks): chunks 2h and
// 2h + 1 are [h*512 + l*16, +16).  The lane then reads the four pieces of a run in the rotated order
// (k + (l >> 1)) & 3, k = 0..3: with a lane stride of 64 bytes the eight lanes of a 128-bit shared-memory access would
// otherwise meet in two bank groups (four passes per load); rotated they cover all eight.  LayerNorm does not care about
// the order, the affine parameters are loaded in the same order, and the quantiser undoes it on its packed output.
// LAY_SWAP is the chunk layout read from shared memory: lanes 4..7 of every eight take the two pieces of a chunk in the
// other order (at a lane stride of 32 bytes lanes l and l + 4 would otherwise share their banks: two passes per load).
constexpr int LAY_CHUNK = 0, LAY_BLK16 = 1, LAY_SWAP = 2;
template <int LAY>
__device__ __forceinline__ int ln_piece_offset(int i, int half, int lane) {
  if (LAY == LAY_BLK16) return (i >> 1) * 512 + lane * 16 + (((2 * (i & 1) + half) + ((lane >> 1) & 3)) & 3) * 4;
  if (LAY == LAY_SWAP) return i * 256 + lane * 8 + (half ^ ((lane >> 2) & 1)) * 4;
  return i * 256 + lane * 8 + half * 4;
}

template <int NV, int LAY = LAY_CHUNK>
__device__ __forceinline__ void ln_affine_load(const float* __restrict__ w, const float* __restrict__ b, int lane, float (&ww)[NV][8], float (&bb)[NV][8]) {
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const float4 w0 = __ldg(reinterpret_cast<const float4*>(w + ln_piece_offset<LAY>(i, 0, lane)));
    const float4 w1 = __ldg(reinterpret_cast<const float4*>(w + ln_piece_offset<LAY>(i, 1, lane)));
    const float4 b0 = __ldg(reinterpret_cast<const float4*>(b + ln_piece_offset<LAY>(i, 0, lane)));
    const float4 b1 = __ldg(reinterpret_cast<const float4*>(b + ln_piece_offset<LAY>(i, 1, lane)));
    ww[i][0] = w0.x; ww[i][1] = w0.y; ww[i][2] = w0.z; ww[i][3] = w0.w; ww[i][4] = w1.x; ww[i][5] = w1.y; ww[i][6] = w1.z; ww[i][7] = w1.w;
    bb[i][0] = b0.x; bb[i][1] = b0.y; bb[i][2] = b0.z; bb[i][3] = b0.w; bb[i][4] = b1.x; bb[i][5] = b1.y; bb[i][6] = b1.z; bb[i][7] = b1.w;
  }
}

// four consecutive values of a row: 16 bytes of fp32 or 8 of bf16
template <bool FROM_SMEM, typename TI>
__device__ __forceinline__ float4 ln_load4(const TI* p) {
  if constexpr (sizeof(TI) == 4) {
    return FROM_SMEM ? *reinterpret_cast<const float4*>(p) : __ldg(reinterpret_cast<const float4*>(p));
  } else {
    const uint2 u = FROM_SMEM ? *reinterpret_cast<const uint2*>(p) : __ldg(reinterpret_cast<const uint2*>(p));
    const float2 a = unpack2<TI>(u.x), b = unpack2<TI>(u.y);
    return make_float4(a.x, a.y, b.x, b.y);
  }
}

// LayerNorm of one row with the affine parameters already in registers (the persistent kernels load them once per
// warp: re-reading them per row doubles the load instructions of a kernel that is otherwise one pass over x).
template <int NV, bool FROM_SMEM = false, int LAY = LAY_CHUNK, typename TI = float>
__device__ __forceinline__ void ln_row(const TI* xr, const float (&ww)[NV][8], const float (&bb)[NV][8], float eps,
                                       int lane, bool valid, float (&v)[NV][8]) {
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    if (valid) {
      const float4 a = ln_load4<FROM_SMEM>(xr + ln_piece_offset<LAY>(i, 0, lane)), c = ln_load4<FROM_SMEM>(xr + ln_piece_offset<LAY>(i, 1, lane));
      v[i][0] = a.x; v[i][1] = a.y; v[i][2] = a.z; v[i][3] = a.w; v[i][4] = c.x; v[i][5] = c.y; v[i][6] = c.z; v[i][7] = c.w;
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[i][j] = 0.f;
    }
  }
  // statistics and affine step on packed pairs, the sums in one chain per 256-element group
  constexpr float inv_d = 1.0f / (NV * 256);
  float2 sp[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    sp[i] = add2(add2(make_float2(v[i][0], v[i][1]), make_float2(v[i][2], v[i][3])), add2(make_float2(v[i][4], v[i][5]), make_float2(v[i][6], v[i][7])));
  }
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) s += sp[i].x + sp[i].y;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  const float mean = s * inv_d;
  const float2 nmean = splat2(-mean);
  float2 c[NV][4], qp[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
#pragma unroll
    for (int j = 0; j < 4; ++j) c[i][j] = add2(make_float2(v[i][2 * j], v[i][2 * j + 1]), nmean);
    qp[i] = mul2(c[i][0], c[i][0]);
#pragma unroll
    for (int j = 1; j < 4; ++j) qp[i] = fma2(c[i][j], c[i][j], qp[i]);
  }
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) ss += qp[i].x + qp[i].y;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  const float2 rstd = splat2(rsqrtf(ss * inv_d + eps));
#pragma unroll
  for (int i = 0; i < NV; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 y = fma2(mul2(c[i][j], rstd), make_float2(ww[i][2 * j], ww[i][2 * j + 1]), make_float2(bb[i][2 * j], bb[i][2 * j + 1]));
      v[i][2 * j] = y.x;
      v[i][2 * j + 1] = y.y;
    }
}

// Rows are streamed through shared memory: each warp owns a ring of LNQ_RING row buffers filled by 1-D bulk copies
// (cp.async.bulk + mbarrier), so one to two rows per warp (4-8 KB) are in flight while the warp normalises and
// quantises the current one; with 16 warps per SM that keeps about 100 KB of HBM reads outstanding per SM, which
// register-staged loads cannot (they stop while the warp computes).  A third row only costs (22 470 rows, us, 3 -> 2: NVFP4 1024 24.7 -> 22.6, 768
// 26.7 -> 25.5; MXFP8 26.8 -> 26.1, 21.2 -> 20.6); five or six CTAs per SM spill the affine parameters (28.8, 35.1).
constexpr int LNQ_RING = 2;

template <int NV, int FMT, typename TI>
__global__ void __launch_bounds__(128, NV <= 4 ? 4 : 1) ln_quant_kernel(const TI* __restrict__ x, const float* __restrict__ w, const float* __restrict__ b, float eps,
                                                       int M, int rows_pad, const float* __restrict__ ts_ptr, int flags, uint8_t* __restrict__ q,
                                                       uint8_t* __restrict__ sf, float* __restrict__ y_dbg, unsigned int* err) {
  constexpr int D = NV * 256;
  extern __shared__ __align__(128) uint8_t lsm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  TI* ring = reinterpret_cast<TI*>(lsm) + (size_t)warp * LNQ_RING * D;
  uint64_t* bars = reinterpret_cast<uint64_t*>(lsm + (size_t)4 * LNQ_RING * D * sizeof(TI)) + warp * LNQ_RING;
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(lsm + (size_t)4 * LNQ_RING * D * sizeof(TI) + 4 * LNQ_RING * 8);
  pdl_launch_dependents();                        // the next kernel of the stream may take the SMs this grid leaves
  if (threadIdx.x == 0) *abort_flag = 0;
  if (lane == 0) {
    for (int i = 0; i < LNQ_RING; ++i) mbar_init(&bars[i], 1);
    fence_mbar_init();
  }
  __syncthreads();
  constexpr bool BLK16 = FMT == KF_FMT_NV4 && NV == 4;   // d = 1024 in NVFP4: a lane owns whole 16-value blocks
  constexpr int LAY = BLK16 ? LAY_BLK16 : LAY_SWAP;
  float ww[NV][8], bb[NV][8];
  // affine parameters whose writes the caller vouches for: their L2 round trip runs under the predecessor's end
  const bool early = (flags & KF_Q_STATIC_AFFINE) != 0;
  if (early) ln_affine_load<NV, LAY>(w, b, lane, ww, bb);
  pdl_wait();                                     // from here on global memory of the predecessors is read and written
  const WaitCtx ctx{abort_flag, err};
  const int W = gridDim.x * 4, gw = blockIdx.x * 4 + warp;
  auto issue = [&](int k) {                       // lane 0: start the copy of this warp's k-th row into slot k % RING
    const int r = gw + k * W;
    if (r < M) {
      mbar_expect_tx(&bars[k % LNQ_RING], D * sizeof(TI));
      bulk_load_1d(ring + (size_t)(k % LNQ_RING) * D, x + (int64_t)r * D, D * sizeof(TI), &bars[k % LNQ_RING]);
    }
  };
  if (lane == 0)
    for (int k = 0; k < LNQ_RING; ++k) issue(k);
  if (!early) ln_affine_load<NV, LAY>(w, b, lane, ww, bb);
  const Nv4Scale ts = nv4_scale(FMT == KF_FMT_NV4 ? __ldg(ts_ptr) : 1.f);
  const bool div_true = !(flags & KF_Q_RECIP_DIV);
  const bool rb = flags & KF_Q_ROUND_BF16;
  // persistent: warp gw of the grid takes rows gw, gw + W, gw + 2W, ... (rows M..rows_pad only get zero scale words)
  int k = 0;
  for (int row = gw; row < rows_pad; row += W, ++k) {
  const bool valid = row < M;
  const int slot = k % LNQ_RING;
  if (valid && !mbar_wait_warp(&bars[slot], (k / LNQ_RING) & 1, ctx, 30)) break;
  float v[NV][8];
  ln_row<NV, true, LAY>(ring + (size_t)slot * D, ww, bb, eps, lane, valid, v);
  __syncwarp();                                   // every lane has its part of the row: the slot can be refilled
  if (lane == 0) {
    fence_proxy_async_smem();
    issue(k + LNQ_RING);
  }
  if constexpr (BLK16) {
    // d = 1024 in NVFP4 (the block path of the model).  The lane holds two whole blocks: elements [16 l, +16) in chunks
    // 0 and 1 and [512 + 16 l, +16) in chunks 2 and 3, so the block maxima and scalars need no exchange between lanes.
    // Both blocks are quantised together, their scalars on packed pairs; the two scale bytes of a lane are the same
    // byte of two scale words, put together over the four lanes of a word with two shuffles.
    float am[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      am[h] = 0.f;
#pragma unroll
      for (int i = 2 * h; i < 2 * h + 2; ++i) {
        if (rb) {
#pragma unroll
          for (int j = 0; j < 8; j += 2) {
            const float2 t = bf16_round2(make_float2(v[i][j], v[i][j + 1]));
            v[i][j] = t.x;
            v[i][j + 1] = t.y;
          }
        }
        if (y_dbg && valid) {
          *reinterpret_cast<float4*>(y_dbg + (int64_t)row * D + ln_piece_offset<LAY_BLK16>(i, 0, lane)) = make_float4(v[i][0], v[i][1], v[i][2], v[i][3]);
          *reinterpret_cast<float4*>(y_dbg + (int64_t)row * D + ln_piece_offset<LAY_BLK16>(i, 1, lane)) = make_float4(v[i][4], v[i][5], v[i][6], v[i][7]);
        }
#pragma unroll
        for (int j = 0; j < 8; j += 2) am[h] = max3(am[h], fabsf(v[i][j]), fabsf(v[i][j + 1]));
      }
    }
    const float(&blk0)[16] = *reinterpret_cast<const float(*)[16]>(&v[0][0]);
    const float(&blk1)[16] = *reinterpret_cast<const float(*)[16]>(&v[2][0]);
    uint32_t o[4];
    int by0, by1;
    quant_nv4_pair16(blk0, am[0], blk1, am[1], ts, div_true, o, by0, by1);
    {
      // piece k of the registers is piece (k + s) & 3 of the block: rotate the four 16-bit code groups of each block left by s
      const int sr = (lane >> 1) & 3;
      const uint32_t sh = (uint32_t)(sr & 1) * 16;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t lo = (sr & 2) ? o[2 * h + 1] : o[2 * h], hi = (sr & 2) ? o[2 * h] : o[2 * h + 1];
        o[2 * h] = __funnelshift_l(hi, lo, sh);
        o[2 * h + 1] = __funnelshift_l(lo, hi, sh);
      }
    }
    if (valid) {
      uint8_t* qr = q + (int64_t)row * (D / 2) + lane * 8;
      *reinterpret_cast<uint2*>(qr) = make_uint2(o[0], o[1]);
      *reinterpret_cast<uint2*>(qr + D / 4) = make_uint2(o[2], o[3]);
    }
    // lanes 4g .. 4g+3 hold the bytes of k-blocks 4g .. 4g+3 (first half of the row) and 32 + 4g .. (second half)
    uint32_t pk = valid ? ((uint32_t)by0 | ((uint32_t)by1 << 16)) : 0u;              // byte 0: first word, byte 2: second
    pk |= __shfl_xor_sync(0xffffffffu, pk, 1) << 8;                                   // on even lanes: the bytes of lanes l, l + 1
    const uint32_t up = __shfl_xor_sync(0xffffffffu, pk, 2);                          // on lane 4g: the pairs of lanes 4g + 2, 4g + 3
    if ((lane & 3) == 0) {
      const uint32_t w0 = __byte_perm(pk, up, 0x5410), w1 = __byte_perm(pk, up, 0x7632);
      *reinterpret_cast<uint32_t*>(sf + sf_offset(row, lane, D >> 6)) = w0;
      *reinterpret_cast<uint32_t*>(sf + sf_offset(row, 32 + lane, D >> 6)) = w1;
    }
  } else {
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    if (rb) {
#pragma unroll
      for (int j = 0; j < 8; j += 2) {
        const float2 t = bf16_round2(make_float2(v[i][j], v[i][j + 1]));
        v[i][j] = t.x;
        v[i][j + 1] = t.y;
      }
    }
    if (y_dbg && valid) {
      *reinterpret_cast<float4*>(y_dbg + (int64_t)row * D + ln_piece_offset<LAY_SWAP>(i, 0, lane)) = make_float4(v[i][0], v[i][1], v[i][2], v[i][3]);
      *reinterpret_cast<float4*>(y_dbg + (int64_t)row * D + ln_piece_offset<LAY_SWAP>(i, 1, lane)) = make_float4(v[i][4], v[i][5], v[i][6], v[i][7]);
    }
    const bool swapped = (lane >> 2) & 1;                            // this lane holds the two pieces of the chunk in the other order
    float amax = 0.f;
#pragma unroll
    for (int j = 0; j < 8; j += 2) amax = max3(amax, fabsf(v[i][j]), fabsf(v[i][j + 1]));
    amax = amax_nan(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    if (FMT != KF_FMT_NV4) amax = amax_nan(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    int byte;
    const int col = i * 256 + lane * 8;
    if (FMT == KF_FMT_MX8) {
      uint32_t o[2];
      quant_mx8<8>(v[i], amax, div_true, o, byte);
      if (valid) *reinterpret_cast<uint2*>(q + (int64_t)row * D + col) = swapped ? make_uint2(o[1], o[0]) : make_uint2(o[0], o[1]);
    } else if (FMT == KF_FMT_MX4) {
      uint32_t o[1];
      quant_mx4<8>(v[i], amax, div_true, o, byte);
      if (valid) *reinterpret_cast<uint32_t*>(q + (int64_t)row * (D / 2) + (col >> 1)) = swapped ? __funnelshift_l(o[0], o[0], 16) : o[0];
    } else {
      uint32_t o[1];
      quant_nv4<8>(v[i], amax, ts, div_true, o, byte);
      if (valid) *reinterpret_cast<uint32_t*>(q + (int64_t)row * (D / 2) + (col >> 1)) = swapped ? __funnelshift_l(o[0], o[0], 16) : o[0];
    }
    if (!valid) byte = 0;
    constexpr int STEP = (FMT == KF_FMT_NV4) ? 2 : 4;               // lanes per k-block
    uint32_t word = gather_sf_word<STEP>(byte, lane);
    if ((lane & (4 * STEP - 1)) == 0) {
      int kb = col / ((FMT == KF_FMT_NV4) ? 16 : 32);
      constexpr int nkb4 = (FMT == KF_FMT_NV4) ? (D >> 6) : (D >> 7);
      *reinterpret_cast<uint32_t*>(sf + sf_offset(row, kb, nkb4)) = word;
    }
  }
  }
  }
}

// Dynamic per-tensor scale of the LayerNorm of x, rounded to bf16 as the quantiser behind it will see it (no output tensor).
template <int NV, typename TI>
__global__ void __launch_bounds__(128) ln_amax_kernel(const TI* __restrict__ x, const float* __restrict__ w, const float* __restrict__ b, float eps, int M, float factor,
                                                      float* __restrict__ ts, uint32_t* __restrict__ ws) {
  pdl_wait();
  constexpr int D = NV * 256;
  const int lane = threadIdx.x & 31;
  float ww[NV][8], bb[NV][8], v[NV][8], am = 0.f;
  ln_affine_load<NV>(w, b, lane, ww, bb);
  for (int row = blockIdx.x * 4 + (threadIdx.x >> 5); row < M; row += gridDim.x * 4) {
    ln_row<NV>(x + (int64_t)row * D, ww, bb, eps, lane, true, v);
#pragma unroll
    for (int i = 0; i < NV; ++i)
#pragma unroll
      for (int j = 0; j < 8; j += 2) am = max3(am, fabsf(v[i][j]), fabsf(v[i][j + 1]));
  }
  amax_finish(bf16_round(am), factor, ts, ws);               // rounding is monotone: the maximum of the rounded values
}

template <int NV, typename TO>
__global__ void __launch_bounds__(128) ln_rows_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ b, float eps,
                                                      int M, TO* __restrict__ y) {
  pdl_wait();
  constexpr int D = NV * 256;
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (row >= M) return;
  float v[NV][8], ww[NV][8], bb[NV][8];
  ln_affine_load<NV>(w, b, lane, ww, bb);
  ln_row<NV>(x + (int64_t)row * D, ww, bb, eps, lane, true, v);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if constexpr (sizeof(TO) == 2 && std::is_same<TO, __nv_bfloat16>::value) {
        __nv_bfloat162 h = __floats2bfloat162_rn(v[i][2 * j], v[i][2 * j + 1]);
        o[j] = *reinterpret_cast<uint32_t*>(&h);
      } else {
        __half2 h = __floats2half2_rn(v[i][2 * j], v[i][2 * j + 1]);
        o[j] = *reinterpret_cast<uint32_t*>(&h);
      }
    }
    *reinterpret_cast<uint4*>(y + (int64_t)row * D + i * 256 + lane * 8) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

// Final LayerNorm of the token stream [B, Ntok, D] with the row gather of the EoMT head: the first Q rows of every
// image (queries) go to qb [B*Q, D], rows >= Q + npre (patch tokens) go to xb [B*(Ntok-Q-npre), D], the cls / register
// rows in between are skipped.
template <int NV>
__global__ void __launch_bounds__(128) ln_tail_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ b, float eps,
                                                      int M, int Ntok, int Q, int npre, __nv_bfloat16* __restrict__ qb, __nv_bfloat16* __restrict__ xb,
                                                      const __nv_bfloat16* __restrict__ wcls, const float* __restrict__ bcls, int ncls1,
                                                      __nv_bfloat16* __restrict__ cl) {
  pdl_wait();
  constexpr int D = NV * 256;
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (row >= M) return;
  const int img = row / Ntok, t = row - img * Ntok;
  if (t >= Q && t < Q + npre) return;
  float v[NV][8], ww[NV][8], bb[NV][8];
  ln_affine_load<NV>(w, b, lane, ww, bb);
  ln_row<NV>(x + (int64_t)row * D, ww, bb, eps, lane, true, v);
  const int P = Ntok - Q - npre;
  __nv_bfloat16* y = t < Q ? qb + ((int64_t)img * Q + t) * D : xb + ((int64_t)img * P + (t - Q - npre)) * D;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      __nv_bfloat162 h = __floats2bfloat162_rn(v[i][2 * j], v[i][2 * j + 1]);
      o[j] = *reinterpret_cast<uint32_t*>(&h);
      const float2 r = __bfloat1622float2(h);          // the class head sees the bf16 values that were stored
      v[i][2 * j] = r.x;
      v[i][2 * j + 1] = r.y;
    }
    *reinterpret_cast<uint4*>(y + i * 256 + lane * 8) = make_uint4(o[0], o[1], o[2], o[3]);
  }
  // class head on the query rows: logits[c] = bf16(sum_k q[k] * W[c][k] + bias[c]), fp32 accumulation
  if (wcls != nullptr && t < Q) {
    for (int c = 0; c < ncls1; ++c) {
      float acc = 0.f;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const uint4 wq = __ldg(reinterpret_cast<const uint4*>(wcls + (int64_t)c * D + i * 256 + lane * 8));
        const uint32_t wv[4] = {wq.x, wq.y, wq.z, wq.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&wv[j]));
          acc = fmaf(v[i][2 * j], f.x, acc);
          acc = fmaf(v[i][2 * j + 1], f.y, acc);
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (lane == 0) cl[((int64_t)img * Q + t) * ncls1 + c] = __float2bfloat16_rn(acc + bcls[c]);
    }
  }
}

// Copies a block of fp32 rows into every image of a token stream: dst[b, row_offset + r, :] = src[r, :] for r < R.
// The query rows that join the stream for the last blocks and the cls / register rows in front of the patch tokens.
__global__ void __launch_bounds__(256) broadcast_rows_kernel(const float4* __restrict__ src, float4* __restrict__ dst, int R, int d4, int B, int64_t img_stride4,
                                                             int64_t row_offset4) {
  pdl_wait();
  const int64_t n = (int64_t)R * d4;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n * B; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t bimg = i / n, e = i - bimg * n;
    dst[bimg * img_stride4 + row_offset4 + e] = __ldg(src + e);
  }
}

// ------------------------------------------------------------------------------------------------ host launchers
static int rows_32b_aligned(const void* x, int64_t pitch_bytes) { return ((reinterpret_cast<uintptr_t>(x) | (uintptr_t)pitch_bytes) & 31) == 0; }   // 256-bit loads

template <typename T>
static int launch_amax_scale(const void* x, int64_t ldx, int M, int K, bool gelu, float factor, float* ts, void* ws, cudaStream_t st) {
  const int64_t total = (int64_t)M * (K / 32);
  KF_REQUIRE(total + (1 << 20) < (1ll << 32), "kf_amax_scale: M*K/32 = %lld work items do not fit the 32-bit index", (long long)total);
  int sms = 0;
  const int rc = device_sm_count(&sms);
  if (rc != KF_OK) return rc;
  // one round of resident blocks at most: every block ends with one atomic on the same word
  const unsigned grid = (unsigned)((total + 255) / 256 < 4 * sms ? (total + 255) / 256 : 4 * sms);
  const int wide = rows_32b_aligned(x, ldx * (int64_t)sizeof(T));
  const T* xp = static_cast<const T*>(x);
  cudaError_t e;
  if (gelu) e = launch_maybe_pdl(M, amax_scale_kernel<T, true>, dim3(grid), dim3(256), 0, st, xp, ldx, M, K, wide, factor, ts, static_cast<uint32_t*>(ws));
  else e = launch_maybe_pdl(M, amax_scale_kernel<T, false>, dim3(grid), dim3(256), 0, st, xp, ldx, M, K, wide, factor, ts, static_cast<uint32_t*>(ws));
  return cuda_status(e, "kf_amax_scale launch");
}

template <typename T>
static int launch_quant_rows(int fmt, const void* x, int64_t ldx, int M, int K, const float* ts, const float* bias, int flags, void* q, void* sf,
                             cudaStream_t st) {
  int64_t per_row = K / 32;
  int64_t valid = (int64_t)M * per_row, total = (int64_t)((M + 127) / 128 * 128) * per_row;
  KF_REQUIRE(total + 256 < (1ll << 32), "kf_quant_rows: M*K/32 = %lld work items do not fit the 32-bit index", (long long)total);
  int sms = 0, dev = 0;
  const int rc = device_sm_count(&sms);
  if (rc != KF_OK) return rc;
  cudaGetDevice(&dev);
  const T* xp = static_cast<const T*>(x);
  const int wide = rows_32b_aligned(x, ldx * (int64_t)sizeof(T));
  uint8_t *qp = static_cast<uint8_t*>(q), *sp = static_cast<uint8_t*>(sf);
  static PerDevice<int> resident[3];                     // CTAs per SM, per format of this input type
  auto go = [&](auto kern) {
    const int64_t blocks = (total + 255) / 256;
    int64_t rounds = 1;
    if (sizeof(T) == 2) {
      int per_sm = resident[fmt].get(dev);
      if (per_sm == 0) {
        const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 256, 0);
        if (e != cudaSuccess) return cuda_status(e, "cudaOccupancyMaxActiveBlocksPerMultiprocessor(quant_rows_kernel)");
        if (per_sm < 1) per_sm = 1;
        resident[fmt].put(dev, per_sm);
      }
      const int64_t slots = (int64_t)sms * per_sm;
      rounds = (blocks + slots - 1) / slots;
    }
    const unsigned grid = (unsigned)((blocks + rounds - 1) / rounds);   // equal shares
    return cuda_status(launch_maybe_pdl(M, kern, dim3(grid), dim3(256), 0, st, xp, ldx, M, K, ts, bias, flags, wide, qp, sp, valid, total), "kf_quant_rows launch");
  };
  if (fmt == KF_FMT_MX8) return go(quant_rows_kernel<T, KF_FMT_MX8>);
  if (fmt == KF_FMT_NV4) return go(quant_rows_kernel<T, KF_FMT_NV4>);
  return go(quant_rows_kernel<T, KF_FMT_MX4>);
}

template <int NV, typename TI>
static int launch_ln_quant(int fmt, const TI* x, const float* w, const float* b, float eps, int M, const float* ts, int flags, void* q, void* sf,
                           float* y_dbg, cudaStream_t st) {
  int rows_pad = (M + 127) / 128 * 128;
  int sms = 0;
  int rc = device_sm_count(&sms);                        // of the CURRENT device
  if (rc != KF_OK) return rc;
  int dev = 0;
  cudaGetDevice(&dev);
  unsigned grid = (unsigned)((rows_pad + 3) / 4);
  uint8_t *qp = static_cast<uint8_t*>(q), *sp = static_cast<uint8_t*>(sf);
  unsigned int* err = dev_error_ptr();
  KF_REQUIRE(err != nullptr, "kf_ln_quant: device error word unavailable");
  const size_t smem = (size_t)4 * LNQ_RING * NV * 256 * sizeof(TI) + 4 * LNQ_RING * 8 + 16;
  static PerDevice<int> resident[3];                     // CTAs per SM, per format of this row width
  auto go = [&](auto kern) {
    // persistent: as many CTAs of 4 warps as are resident at once (4 per SM up to d = 1024, fewer for wider rows); a
    // grid beyond that would run its surplus as a second, nearly empty wave.  The attribute and the occupancy query are
    // per (kernel instance, device): worked out at the first call and kept.
    int per_sm = resident[fmt].get(dev);
    if (per_sm == 0) {
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute(ln_quant_kernel)");
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 128, smem);
      if (e != cudaSuccess) return cuda_status(e, "cudaOccupancyMaxActiveBlocksPerMultiprocessor(ln_quant_kernel)");
      if (per_sm < 1) per_sm = 1;
      if (per_sm > 4) per_sm = 4;
      resident[fmt].put(dev, per_sm);
    }
    if (grid > (unsigned)(sms * per_sm)) grid = (unsigned)(sms * per_sm);
    return cuda_status(launch_maybe_pdl(M, kern, dim3(grid), dim3(128), smem, st, x, w, b, eps, M, rows_pad, ts, flags, qp, sp, y_dbg, err), "kf_ln_quant launch");
  };
  if (fmt == KF_FMT_MX8) return go(ln_quant_kernel<NV, KF_FMT_MX8, TI>);
  if (fmt == KF_FMT_NV4) return go(ln_quant_kernel<NV, KF_FMT_NV4, TI>);
  return go(ln_quant_kernel<NV, KF_FMT_MX4, TI>);
}

template <int NV, typename TI>
static int launch_ln_amax(const TI* x, const float* w, const float* b, float eps, int M, float factor, float* ts, void* ws, cudaStream_t st) {
  int sms = 0;
  const int rc = device_sm_count(&sms);
  if (rc != KF_OK) return rc;
  const int grid = (M + 3) / 4 < 4 * sms ? (M + 3) / 4 : 4 * sms;
  const cudaError_t e = launch_maybe_pdl(M, ln_amax_kernel<NV, TI>, dim3(grid), dim3(128), 0, st, x, w, b, eps, M, factor, ts, static_cast<uint32_t*>(ws));
  return cuda_status(e, "kf_ln_amax_scale launch");
}

template <int NV>
static int launch_ln_rows(const float* x, const float* w, const float* b, float eps, int M, int out_dtype, void* y, cudaStream_t st) {
  unsigned grid = (unsigned)((M + 3) / 4);
  cudaError_t e;
  if (out_dtype == KF_BF16) e = launch_maybe_pdl(M, ln_rows_kernel<NV, __nv_bfloat16>, dim3(grid), dim3(128), 0, st, x, w, b, eps, M, static_cast<__nv_bfloat16*>(y));
  else e = launch_maybe_pdl(M, ln_rows_kernel<NV, __half>, dim3(grid), dim3(128), 0, st, x, w, b, eps, M, static_cast<__half*>(y));
  return cuda_status(e, "kf_ln_rows launch");
}

template <int NV>
static int launch_ln_tail(const float* x, const float* w, const float* b, float eps, int M, int Ntok, int Q, int npre, void* qb, void* xb, const void* wcls,
                          const float* bcls, int ncls1, void* cl, cudaStream_t st) {
  const cudaError_t e = launch_maybe_pdl(M, ln_tail_kernel<NV>, dim3((M + 3) / 4), dim3(128), 0, st, x, w, b, eps, M, Ntok, Q, npre, static_cast<__nv_bfloat16*>(qb), static_cast<__nv_bfloat16*>(xb),
                                                              static_cast<const __nv_bfloat16*>(wcls), bcls, ncls1, static_cast<__nv_bfloat16*>(cl));
  return cuda_status(e, "kf_ln_tail launch");
}

template <typename TI>
static int ln_quant_width(int fmt, const TI* x, const float* w, const float* b, float eps, int M, int d, const float* ts, int flags, void* q, void* sf, float* y_dbg,
                          cudaStream_t st) {
  switch (d / 256) {
    case 1: return launch_ln_quant<1, TI>(fmt, x, w, b, eps, M, ts, flags, q, sf, y_dbg, st);
    case 2: return launch_ln_quant<2, TI>(fmt, x, w, b, eps, M, ts, flags, q, sf, y_dbg, st);
    case 3: return launch_ln_quant<3, TI>(fmt, x, w, b, eps, M, ts, flags, q, sf, y_dbg, st);
    case 4: return launch_ln_quant<4, TI>(fmt, x, w, b, eps, M, ts, flags, q, sf, y_dbg, st);
    case 5: return launch_ln_quant<5, TI>(fmt, x, w, b, eps, M, ts, flags, q, sf, y_dbg, st);
    case 6: return launch_ln_quant<6, TI>(fmt, x, w, b, eps, M, ts, flags, q, sf, y_dbg, st);
    case 7: return launch_ln_quant<7, TI>(fmt, x, w, b, eps, M, ts, flags, q, sf, y_dbg, st);
    default: return launch_ln_quant<8, TI>(fmt, x, w, b, eps, M, ts, flags, q, sf, y_dbg, st);
  }
}

template <typename TI>
static int ln_amax_width(const TI* x, const float* w, const float* b, float eps, int M, int d, float factor, float* ts, void* ws, cudaStream_t st) {
  switch (d / 256) {
    case 1: return launch_ln_amax<1, TI>(x, w, b, eps, M, factor, ts, ws, st);
    case 2: return launch_ln_amax<2, TI>(x, w, b, eps, M, factor, ts, ws, st);
    case 3: return launch_ln_amax<3, TI>(x, w, b, eps, M, factor, ts, ws, st);
    case 4: return launch_ln_amax<4, TI>(x, w, b, eps, M, factor, ts, ws, st);
    case 5: return launch_ln_amax<5, TI>(x, w, b, eps, M, factor, ts, ws, st);
    case 6: return launch_ln_amax<6, TI>(x, w, b, eps, M, factor, ts, ws, st);
    case 7: return launch_ln_amax<7, TI>(x, w, b, eps, M, factor, ts, ws, st);
    default: return launch_ln_amax<8, TI>(x, w, b, eps, M, factor, ts, ws, st);
  }
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace kf

using namespace kf;

extern "C" int kf_quant_rows(int fmt, int in_dtype, const void* x, int64_t ldx, int M, int K, const float* ts, const float* bias, int flags, void* q,
                             void* sf, void* stream) {
  KF_REQUIRE(fmt == KF_FMT_MX8 || fmt == KF_FMT_NV4 || fmt == KF_FMT_MX4, "kf_quant_rows: unknown format %d", fmt);
  KF_REQUIRE(in_dtype == KF_F32 || in_dtype == KF_BF16 || in_dtype == KF_F16, "kf_quant_rows: unknown input dtype %d", in_dtype);
  KF_REQUIRE(M >= 0 && K > 0 && K % 128 == 0, "kf_quant_rows: K=%d must be a positive multiple of 128 (M=%d)", K, M);
  if (M == 0) return KF_OK;
  KF_REQUIRE(x && q && sf, "kf_quant_rows: null tensor pointer");
  KF_REQUIRE(ldx >= K && ldx % 8 == 0, "kf_quant_rows: row stride %lld must be >= K and a multiple of 8", (long long)ldx);
  KF_REQUIRE(aligned16(x) && aligned16(q) && aligned16(sf), "kf_quant_rows: tensors must be 16-byte aligned");
  KF_REQUIRE(fmt != KF_FMT_NV4 || ts, "kf_quant_rows: nv4 needs the per-tensor scale pointer");
  KF_REQUIRE(!(flags & KF_Q_GELU) || (bias && aligned16(bias)), "kf_quant_rows: KF_Q_GELU needs a 16-byte aligned bias");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (in_dtype == KF_F32) return launch_quant_rows<float>(fmt, x, ldx, M, K, ts, bias, flags, q, sf, st);
  if (in_dtype == KF_BF16) return launch_quant_rows<__nv_bfloat16>(fmt, x, ldx, M, K, ts, bias, flags, q, sf, st);
  return launch_quant_rows<__half>(fmt, x, ldx, M, K, ts, bias, flags, q, sf, st);
}

extern "C" int kf_ln_quant(int fmt, const float* x, const float* w, const float* b, float eps, int M, int d, const float* ts, int flags, void* q,
                           void* sf, float* y_dbg, void* stream) {
  KF_REQUIRE(fmt == KF_FMT_MX8 || fmt == KF_FMT_NV4 || fmt == KF_FMT_MX4, "kf_ln_quant: unknown format %d", fmt);
  KF_REQUIRE(M >= 0 && d > 0 && d % 256 == 0 && d <= 2048, "kf_ln_quant: d=%d must be a multiple of 256 up to 2048", d);
  if (M == 0) return KF_OK;
  KF_REQUIRE(x && w && b && q && sf, "kf_ln_quant: null tensor pointer");
  KF_REQUIRE(aligned16(x) && aligned16(w) && aligned16(b) && aligned16(q) && aligned16(sf) && aligned16(y_dbg), "kf_ln_quant: tensors must be 16-byte aligned");
  KF_REQUIRE(fmt != KF_FMT_NV4 || ts, "kf_ln_quant: nv4 needs the per-tensor scale pointer");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (flags & KF_Q_IN_BF16) return ln_quant_width(fmt, reinterpret_cast<const __nv_bfloat16*>(x), w, b, eps, M, d, ts, flags, q, sf, y_dbg, st);
  return ln_quant_width(fmt, x, w, b, eps, M, d, ts, flags, q, sf, y_dbg, st);
}

extern "C" int kf_amax_scale(int in_dtype, const void* x, int64_t ldx, int M, int K, int flags, float factor, float* ts, void* ws, void* stream) {
  KF_REQUIRE(in_dtype == KF_F32 || in_dtype == KF_BF16 || in_dtype == KF_F16, "kf_amax_scale: unknown input dtype %d", in_dtype);
  KF_REQUIRE(M > 0 && K > 0 && K % 32 == 0, "kf_amax_scale: K=%d must be a positive multiple of 32 and M=%d positive", K, M);
  KF_REQUIRE(x && ts && ws && aligned16(x), "kf_amax_scale: tensors must be non-null and x 16-byte aligned");
  KF_REQUIRE(ldx >= K && ldx % 8 == 0, "kf_amax_scale: row stride %lld must be >= K and a multiple of 8", (long long)ldx);
  KF_REQUIRE((flags & ~KF_Q_GELU) == 0, "kf_amax_scale: only KF_Q_GELU is a valid flag");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool gelu = flags & KF_Q_GELU;
  if (in_dtype == KF_F32) return launch_amax_scale<float>(x, ldx, M, K, gelu, factor, ts, ws, st);
  if (in_dtype == KF_BF16) return launch_amax_scale<__nv_bfloat16>(x, ldx, M, K, gelu, factor, ts, ws, st);
  return launch_amax_scale<__half>(x, ldx, M, K, gelu, factor, ts, ws, st);
}

extern "C" int kf_ln_amax_scale(int in_dtype, const void* x, const float* w, const float* b, float eps, int M, int d, float factor, float* ts, void* ws, void* stream) {
  KF_REQUIRE(in_dtype == KF_F32 || in_dtype == KF_BF16, "kf_ln_amax_scale: x must be f32 or bf16");
  KF_REQUIRE(M > 0 && d > 0 && d % 256 == 0 && d <= 2048, "kf_ln_amax_scale: d=%d must be a multiple of 256 up to 2048 and M=%d positive", d, M);
  KF_REQUIRE(x && w && b && ts && ws && aligned16(x) && aligned16(w) && aligned16(b), "kf_ln_amax_scale: tensors must be non-null and 16-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (in_dtype == KF_BF16) return ln_amax_width(static_cast<const __nv_bfloat16*>(x), w, b, eps, M, d, factor, ts, ws, st);
  return ln_amax_width(static_cast<const float*>(x), w, b, eps, M, d, factor, ts, ws, st);
}

extern "C" int kf_ln_rows(const float* x, const float* w, const float* b, float eps, int M, int d, int out_dtype, void* y, void* stream) {
  KF_REQUIRE(out_dtype == KF_BF16 || out_dtype == KF_F16, "kf_ln_rows: output dtype must be bf16 or f16");
  KF_REQUIRE(M >= 0 && d > 0 && d % 256 == 0 && d <= 2048, "kf_ln_rows: d=%d must be a multiple of 256 up to 2048", d);
  if (M == 0) return KF_OK;
  KF_REQUIRE(x && w && b && y, "kf_ln_rows: null tensor pointer");
  KF_REQUIRE(aligned16(x) && aligned16(w) && aligned16(b) && aligned16(y), "kf_ln_rows: tensors must be 16-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (d / 256) {
    case 1: return launch_ln_rows<1>(x, w, b, eps, M, out_dtype, y, st);
    case 2: return launch_ln_rows<2>(x, w, b, eps, M, out_dtype, y, st);
    case 3: return launch_ln_rows<3>(x, w, b, eps, M, out_dtype, y, st);
    case 4: return launch_ln_rows<4>(x, w, b, eps, M, out_dtype, y, st);
    case 5: return launch_ln_rows<5>(x, w, b, eps, M, out_dtype, y, st);
    case 6: return launch_ln_rows<6>(x, w, b, eps, M, out_dtype, y, st);
    case 7: return launch_ln_rows<7>(x, w, b, eps, M, out_dtype, y, st);
    default: return launch_ln_rows<8>(x, w, b, eps, M, out_dtype, y, st);
  }
}

extern "C" int kf_ln_tail(const float* x, const float* w, const float* b, float eps, int B, int Ntok, int Q, int npre, int d, void* qb, void* xb,
                          const void* wcls, const float* bcls, int ncls1, void* cl, void* stream) {
  KF_REQUIRE(B >= 0 && Ntok > 0 && Q >= 0 && npre >= 0 && Q + npre <= Ntok, "kf_ln_tail: bad token counts Ntok=%d Q=%d npre=%d", Ntok, Q, npre);
  KF_REQUIRE(d > 0 && d % 256 == 0 && d <= 2048, "kf_ln_tail: d=%d must be a multiple of 256 up to 2048", d);
  if (B == 0) return KF_OK;
  KF_REQUIRE(x && w && b && xb && (qb || Q == 0), "kf_ln_tail: null tensor pointer");
  KF_REQUIRE(aligned16(x) && aligned16(w) && aligned16(b) && aligned16(qb) && aligned16(xb), "kf_ln_tail: tensors must be 16-byte aligned");
  KF_REQUIRE(wcls == nullptr || (bcls && cl && ncls1 > 0 && ncls1 <= 64 && aligned16(wcls)), "kf_ln_tail: the class head needs wcls (16-byte aligned), bcls, cl and 1..64 logits");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int M = B * Ntok;
  switch (d / 256) {
    case 1: return launch_ln_tail<1>(x, w, b, eps, M, Ntok, Q, npre, qb, xb, wcls, bcls, ncls1, cl, st);
    case 2: return launch_ln_tail<2>(x, w, b, eps, M, Ntok, Q, npre, qb, xb, wcls, bcls, ncls1, cl, st);
    case 3: return launch_ln_tail<3>(x, w, b, eps, M, Ntok, Q, npre, qb, xb, wcls, bcls, ncls1, cl, st);
    case 4: return launch_ln_tail<4>(x, w, b, eps, M, Ntok, Q, npre, qb, xb, wcls, bcls, ncls1, cl, st);
    case 5: return launch_ln_tail<5>(x, w, b, eps, M, Ntok, Q, npre, qb, xb, wcls, bcls, ncls1, cl, st);
    case 6: return launch_ln_tail<6>(x, w, b, eps, M, Ntok, Q, npre, qb, xb, wcls, bcls, ncls1, cl, st);
    case 7: return launch_ln_tail<7>(x, w, b, eps, M, Ntok, Q, npre, qb, xb, wcls, bcls, ncls1, cl, st);
    default: return launch_ln_tail<8>(x, w, b, eps, M, Ntok, Q, npre, qb, xb, wcls, bcls, ncls1, cl, st);
  }
}

extern "C" int kf_broadcast_rows(const float* src, float* dst, int R, int d, int B, int64_t img_stride, int64_t row_offset, void* stream) {
  KF_REQUIRE(R >= 0 && B >= 0 && d > 0 && d % 4 == 0, "kf_broadcast_rows: d=%d must be a positive multiple of 4", d);
  KF_REQUIRE(img_stride % 4 == 0 && row_offset >= 0 && row_offset + (int64_t)R <= img_stride / d, "kf_broadcast_rows: rows %lld..%lld do not fit an image of %lld values",
             (long long)row_offset, (long long)(row_offset + R), (long long)img_stride);
  if (R == 0 || B == 0) return KF_OK;
  KF_REQUIRE(src && dst && aligned16(src) && aligned16(dst), "kf_broadcast_rows: tensors must be non-null and 16-byte aligned");
  const int64_t n = (int64_t)R * (d / 4) * B;
  int grid = (int)((n + 255) / 256);
  if (grid > 148 * 8) grid = 148 * 8;
  const cudaError_t e = launch_maybe_pdl(img_stride / d * B, broadcast_rows_kernel, dim3(grid), dim3(256), 0, static_cast<cudaStream_t>(stream), reinterpret_cast<const float4*>(src), reinterpret_cast<float4*>(dst), R, d / 4, B, img_stride / 4,
                                                                            row_offset * (d / 4));
  return cuda_status(e, "kf_broadcast_rows launch");
}
