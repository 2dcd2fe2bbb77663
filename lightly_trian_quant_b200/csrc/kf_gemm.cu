// Block-scaled GEMM  C[M,N] = A[M,K] * W[N,K]^T  on the sm_100a tensor cores (tcgen05.mma, fp32 accumulators in
// TMEM) with the epilogues of the ViT block fused in.
//
//   operands   K-major codes: e4m3 bytes (mx8), packed e2m1 nibbles (nv4 / mx4) or plain bf16; scale factors in
//              the 128x4 blocked layout, one 512-byte atom per 128 rows x 4 k-blocks
//   tile       128 x 256 output tile per CTA step (128 x 128 for launches of a few tiles: gemm_columns) (one MMA instruction is 128 x 256 x 32 K-bytes), 128 bytes of K per
//              pipeline stage.  The tile shape is set by shared-memory bandwidth: a 128 x 128 MMA reads its 8 KB of
//              operands in the ~68 clk it executes, which alone saturates the 128 B/clk of the shared-memory array,
//              and the TMA writes of the next stages need the same array (measured: main loop at half the instruction
//              rate).  At 128 x 256 an MMA reads 12 KB per ~136 clk.
//   pipeline   20 warps.  Warp group 0: warp 0 = TMA producer (operand tiles by tensor map, scale atoms by 1-D bulk copy),
//              warp 1 = MMA issuer (per stage: the scale atoms smem -> TMEM by tcgen05.cp, then 4 MMAs; one thread issues
//              both, in order, and the hardware overlaps them), warps 2 and 3 idle.  Both issuing warps run warp-uniform
//              loops with one elected lane per instruction (kf_sm100.cuh): with one-lane loops and the copies issued by a
//              warp of their own a stage of NVFP4 took 1090 clk on an otherwise idle SM, now 610 (its MMAs: 544); M = 1605,
//              K = 4096, N = 1024: 14.8 -> 10.6 us, M = 22 470: fc2 75 -> 67 us, plain 69 -> 67 us.  Warp groups
//              1..4 = 16 epilogue warps.  Registers are re-balanced between the roles (setmaxnreg, per epilogue kind): the issuing
//              roles give theirs up and every epilogue thread holds its 64 accumulator values plus loads in flight
//              without spilling.
//              One 256-column accumulator in TMEM: each epilogue warp takes (32-row TMEM quarter, 64 columns) into
//              registers and hands TMEM back at once, so the next tile's main loop runs under the epilogue math;
//              persistent CTAs, one per SM, static round-robin over tiles
//   epilogues  PLAIN  out = act(acc*ts + bias)                       -> f32 | bf16 | f16 [M,N]
//              RES    out = R + gamma * (acc*ts + bias)              -> f32 [M,N]         (proj, fc2)
//              ROPE   bias + rotary embedding of q,k + relayout      -> bf16 | f16 [3,B,Ntok,H,64]   (qkv)
//              QUANT  gelu(acc*ts + bias) quantised again            -> codes [M,N] + blocked scales (fc1 -> fc2)
//              all four work in the TMEM row layout (a thread owns 64 consecutive columns of one row) and touch global
//              memory in whole 32-byte sectors or 128-byte lines (kf_gemm_epi.cuh)
//
// Replaces (reference checkout paths): infer-opt/round13_mxfp8_full/impl/mgx_core.cu:118-444 (MXFP8, mma.sync) and
// infer-opt/round14_fp4_full/impl/fp4g_core.cu:153-470 (NVFP4 / MXFP4, mma.sync); epilogue math per
// mgx_core.cu:308-426 and fp4g_core.cu:309-382.
#include "kf_gemm_epi.cuh"

namespace kf {

// Depth of the operand ring, chosen per launch.  BN = 256: a fourth stage (54 KB) helps where the main loop is the longer chain
// (measured at M = 22 470: fc2 K 4096 79 -> 76 us, MXFP8 fc2 116 -> 108 us, PLAIN 73 -> 69 us) and hurts where the epilogue is
// (proj 51 -> 53 us, fc1 93 -> 98 us: the stage's shared memory comes out of the L1 the epilogue's global accesses use);
// the ROPE kernel's table slabs leave no room for one.  BN = 128: the launches of a few tiles, where the fill rate is the bytes in
// flight over the L2 latency, so all of K up to six stages (36 KB each).
constexpr int MAX_STAGES = 6;
template <int BN>
static int gemm_stages(int epi, int k_tiles, int flags, bool res_tma) {
  if (BN == 128) {
    const int most = epi == KF_EPI_ROPE ? 5 : res_tma ? 4 : 6;
    return k_tiles < 2 ? 2 : k_tiles < most ? k_tiles : most;
  }
  if (epi == KF_EPI_PLAIN) return (flags & KF_G_GELU) ? 3 : 4;      // PLAIN with GELU (the head's ConvTranspose GEMMs) is epilogue-bound too
  if (epi == KF_EPI_RES && k_tiles >= 8) return 4;
  return 3;
}
constexpr size_t GEMM_SMEM_MAX = 227 * 1024;
// operand ring + scale atoms + bias slices or vectors (+ the rotary-table slabs, + the residual boxes) + barriers
template <int EPI, int BN>
constexpr size_t gemm_smem(int stages, int vec_floats = 0, bool res_tma = false) {
  const size_t sl = (size_t)(vec_floats > EPI_WARPS * SLICE_FLOATS ? vec_floats : EPI_WARPS * SLICE_FLOATS) * 4;
  return (size_t)stages * (Tile<BN>::BYTES + Tile<BN>::SF_BYTES) + sl + (EPI == KF_EPI_ROPE ? 4 * ROPE_SLAB_FLOATS * 4 : 0) +
         (res_tma ? EPI_WARPS * RES_BOX_BYTES : 0) + 384;
}
static_assert(gemm_smem<KF_EPI_ROPE, 256>(3) <= GEMM_SMEM_MAX && gemm_smem<KF_EPI_RES, 256>(4) <= GEMM_SMEM_MAX && gemm_smem<KF_EPI_ROPE, 128>(5) <= GEMM_SMEM_MAX &&
                  gemm_smem<KF_EPI_RES, 128>(6) <= GEMM_SMEM_MAX &&
                  gemm_smem<KF_EPI_RES, 128>(4, 0, true) <= GEMM_SMEM_MAX,
              "shared memory of the deepest rings");

// ------------------------------------------------------------------------------------------------ the kernel
// FORM: epilogue_form of the launch.  A kernel of its own for each: with all of them in one the code that a short launch fetches is scattered
// (ViT-B 256 px: captured 575 -> 569 us, eager 615 -> 610).
template <int KIND, int EPI, int BN, int FORM>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmR,
            const __grid_constant__ CUtensorMap tmC, const GemmArgs g) {
  constexpr int ATOMS = KindTraits<KIND>::ATOMS;
  constexpr bool SCALED = KIND != KIND_BF16;
  constexpr int TILE_BYTES = Tile<BN>::BYTES, SF_STAGE_BYTES = Tile<BN>::SF_BYTES, ACCS = Tile<BN>::ACCS;
  const int STAGES = g.stages;                            // the ring depth this launch was given shared memory for

  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* tiles = smem;
  uint8_t* boxes = smem + (size_t)STAGES * TILE_BYTES;                                  // RES through shared memory only; 1024-byte aligned
  uint8_t* sfs = boxes + (EPI == KF_EPI_RES && BN == 128 && g.res_tma ? EPI_WARPS * RES_BOX_BYTES : 0);
  float* slices = reinterpret_cast<float*>(sfs + (size_t)STAGES * SF_STAGE_BYTES);
  float* slabs = slices + (g.vec_floats > EPI_WARPS * SLICE_FLOATS ? g.vec_floats : EPI_WARPS * SLICE_FLOATS);   // ROPE only
  uint64_t* bars = reinterpret_cast<uint64_t*>(slabs + (EPI == KF_EPI_ROPE ? 4 * ROPE_SLAB_FLOATS : 0));
  uint64_t *full = bars, *empty = bars + MAX_STAGES, *tfull = bars + 2 * MAX_STAGES, *tempty = tfull + 2;
  uint64_t* box_full = tempty + 2;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(box_full + EPI_WARPS);
  volatile uint32_t* abort_flag = tmem_holder + 1;

  const int warp = warp_index(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < ACCS; ++a) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], EPI_WARPS);
    }
    if (EPI == KF_EPI_RES && BN == 128)
      for (int w = 0; w < EPI_WARPS; ++w) mbar_init(&box_full[w], 1);
    *abort_flag = 0u;
    fence_mbar_init();
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmW);
  }
  if (warp == 1) {
    tmem_alloc(tmem_holder, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // Set-up done: from here on global memory of the predecessors is read and written.  Ahead of the wait the producer reads only the
  // error word and weights that KF_G_W_STATIC vouches for.
  const bool w_early = (g.flags & KF_G_W_STATIC) != 0;
  if (warp != 0 || !w_early) pdl_wait();
  const uint32_t tmem_base = *tmem_holder;
  const WaitCtx ctx{abort_flag, g.err};
  const bool bad_align = (smem_u32(smem) & 1023u) != 0;   // the swizzled operand tiles need a 1024-byte aligned base; the same answer in every thread
  if (bad_align && threadIdx.x == 0 && atomicCAS(&g.err[0], 0u, (unsigned)(-KF_ERR_DEVICE_WAIT)) == 0u) {
    g.err[1] = 100;
    g.err[2] = blockIdx.x;
  }

  if (warp < EPI_WARP0) {
    setmaxnreg_dec<EPI == KF_EPI_ROPE ? REGS_LEAN_ROPE : REGS_LEAN>();
    if (bad_align) {
      if (warp == 0 && w_early) pdl_wait();              // nothing is issued; fall through to the teardown
    } else if (warp == 0) {
      // ------------------------------------------------------------------ TMA producer
      uint32_t s = 0, ph = 0;
      // Has an earlier launch failed?  The producer alone looks, once, before it requests anything: without its loads no barrier of the
      // other roles completes and the abort flag ends their waits.  A look of every warp at a word that another launch may write
      // in between would let some roles run and others not.
      bool ok = !__any_sync(0xffffffffu, *static_cast<volatile unsigned int*>(g.err) != 0u);
      if (!ok) {
        *abort_flag = 1u;
        if (w_early) pdl_wait();
      }
      // Weights whose writes the host has seen complete (KF_G_W_STATIC): the W part of the first tile's stages is requested before the
      // wait for the predecessor, so its way from HBM runs under the predecessor's end.
      int early = 0;
      auto load_w = [&](uint32_t st, int kt, const WorkItem& w, int w_halves, uint32_t tx) {
        mbar_expect_tx(&full[st], tx);
        // rows past the end of W are filled with zeros; a half tile has a map of its own with boxes of 128 rows
        tma_load_2d(tiles + (size_t)st * TILE_BYTES + A_BYTES, BN == 256 && w.cols == 128 ? &tmR : &tmW, kt * BKB, tile_wrow0(g, w.m_blk, w.n0), &full[st]);
        if (SCALED) {
          uint8_t* sa = sfs + (size_t)st * SF_STAGE_BYTES;
          for (int h = 0; h < w_halves; ++h)
            bulk_load_1d(sa + (1 + h) * ATOMS * 512, g.sfw + ((size_t)(w.n0 / 128 + h) * g.nkb4 + (size_t)kt * ATOMS) * 512, ATOMS * 512, &full[st]);
        }
      };
      for (int idx = blockIdx.x; idx < g.items && ok; idx += gridDim.x) {
        const WorkItem w = work_item<BN>(g, idx);
        const int w_halves = (BN == 256 && w.cols == BN && w.n0 + 128 < g.N) ? 2 : 1;   // the last column tile of 256 may hold only 128 columns
        int row_end;
        const int a_row0 = tile_row0(g, w.m_blk, row_end);
        const uint32_t tx = A_BYTES + w.cols * BKB + (SCALED ? (1 + w_halves) * ATOMS * 512 : 0);
        if (w_early && idx == (int)blockIdx.x) {
          early = g.k_tiles < STAGES ? g.k_tiles : STAGES;
          if (elect_one())
            for (int kt = 0; kt < early; ++kt) load_w(kt, kt, w, w_halves, tx);
          __syncwarp();
          pdl_wait();
        }
        for (int kt = 0; kt < g.k_tiles; ++kt) {
          if (!mbar_wait_warp(&empty[s], ph ^ 1, ctx, 1)) { ok = false; break; }
          if (elect_one()) {
            if (kt >= early) load_w(s, kt, w, w_halves, tx);
            tma_load_2d(tiles + (size_t)s * TILE_BYTES, &tmA, kt * BKB, a_row0, &full[s]);
            if (SCALED) bulk_load_1d(sfs + (size_t)s * SF_STAGE_BYTES, g.sfa + ((size_t)w.m_blk * g.nkb4 + (size_t)kt * ATOMS) * 512, ATOMS * 512, &full[s]);
          }
          __syncwarp();
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
        early = 0;
      }
    } else if (warp == 1) {
      // ------------------------------------------------------------------ MMA issuer
      // Per stage: the scale-factor atoms into one of the SF_BUFS tensor-memory buffers (tcgen05.cp), then four MMAs of 32
      // K-bytes.  One thread issues both, so the hardware runs them in order (an MMA sees the copies in front of it, a copy
      // does not overtake the MMAs that read the buffer's previous contents) and overlaps them: twelve copies and four
      // MMAs take the time of the MMAs alone.
      constexpr auto idesc_n = [](int n) {
        return KIND == KIND_BF16 ? idesc_f16(1, n) : KIND == KIND_MX8 ? idesc_bs(0, 1, n) : KIND == KIND_NV4 ? idesc_bs(1, 0, n) : idesc_bs(1, 1, n);
      };
      uint32_t s = 0, ph = 0, lt = 0, sb = 0;
      bool ok = true;
      for (int idx = blockIdx.x; idx < g.items && ok; idx += gridDim.x, ++lt) {
        const WorkItem w = work_item<BN>(g, idx);
        const bool two = BN == 256 && w.cols == BN && w.n0 + 128 < g.N;
        const uint32_t IDESC = w.cols == BN ? idesc_n(BN) : idesc_n(128);
        const uint32_t ac = lt % ACCS;
        if (!mbar_wait_warp(&tempty[ac], ((lt / ACCS) & 1) ^ 1, ctx, 2)) break;   // the epilogue has taken this accumulator's previous tile out of TMEM
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + ac * BN;
        for (int kt = 0; kt < g.k_tiles; ++kt) {
          if (!mbar_wait_warp(&full[s], ph, ctx, 3)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a_addr = smem_u32(tiles + (size_t)s * TILE_BYTES);
          const uint64_t adesc = smem_desc_sw128(a_addr), bdesc = smem_desc_sw128(a_addr + A_BYTES);
          // scale factors of this stage: A at +0 (4 columns per atom), W at +16 (BN = 256: 8 columns per atom pair, the atom of
          // columns 0..127 of the tile, then the atom of columns 128..255; BN = 128: 4 columns per atom)
          constexpr uint32_t WS = 4 * (BN / 128);
          const uint32_t sf_t = tmem_base + TMEM_SF_COL + sb * SF_BUF_COLS;
          const uint32_t sa = smem_u32(sfs + (size_t)s * SF_STAGE_BYTES);
          if (elect_one()) {
            if (SCALED) {
#pragma unroll
              for (int a = 0; a < ATOMS; ++a) {
                tc_cp_sf(sf_t + 4 * a, smem_desc_sf(sa + a * 512));
                tc_cp_sf(sf_t + 16 + WS * a, smem_desc_sf(sa + (ATOMS + a) * 512));
                if (two) tc_cp_sf(sf_t + 16 + WS * a + 4, smem_desc_sf(sa + (2 * ATOMS + a) * 512));
              }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {                                       // 32 K-bytes per MMA
              const uint32_t acc = (kt | j) != 0;
              const uint64_t ad = adesc + 2 * j, bd = bdesc + 2 * j;
              if (KIND == KIND_BF16) {
                mma_f16(d_tmem, ad, bd, IDESC, acc);
              } else if (KIND == KIND_MX8) {      // one scale per row per MMA: byte j of the atom's 32-bit word
                mma_mxf8(d_tmem, ad, bd, idesc_with_sf_id(IDESC, j, j), acc, sf_t, sf_t + 16);
              } else if (KIND == KIND_NV4) {      // four scales per row per MMA: atom j
                mma_nvf4(d_tmem, ad, bd, IDESC, acc, sf_t + 4 * j, sf_t + 16 + WS * j);
              } else {                            // two scales per row per MMA: half-word (j & 1) of atom j / 2
                mma_mxf4(d_tmem, ad, bd, idesc_with_sf_id(IDESC, 2 * (j & 1), 2 * (j & 1)), acc, sf_t + 4 * (j >> 1), sf_t + 16 + WS * (j >> 1));
              }
            }
            tc_commit(&empty[s]);
            if (kt == g.k_tiles - 1) tc_commit(&tfull[ac]);
          }
          __syncwarp();
          if (SCALED && ++sb == SF_BUFS) sb = 0;
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue: 16 warps, warp = (TMEM lane quarter, 64-column group)
    setmaxnreg_inc<EPI == KF_EPI_ROPE ? REGS_EPI_ROPE : REGS_EPI>();
    if (!bad_align) {
      epilogue_warps<EPI, BN, false, FORM>(g, tmem_base, tfull, tempty, slices, slabs, boxes, box_full, nullptr, &tmR, &tmC, ctx, warp, lane);
    }
  }

  pdl_launch_dependents();                               // only now: see kf_common.cuh
  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {                 // a wait ran out: give copies still in flight time to land before the CTA exits
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------------------------ host side
EncodeTiledFn encode_tiled_fn() {
  static const EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    const bool found = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess;
    return found ? reinterpret_cast<EncodeTiledFn>(p) : nullptr;
  }();
  return fn;
}

// Encoding a tensor map costs about a microsecond of host time; an eager caller (the Linear swap) issues the same few
// (pointer, shape) combinations over and over, so the encoded maps are kept in a small per-thread direct-mapped cache.
struct TmapKey {
  const void* base;
  uint64_t rows, row_bytes, pitch_bytes;
  uint32_t box_rows;
  bool atoms;                                            // rows of 128 words without a swizzle (scale atoms) instead of 128-byte boxes
  bool operator==(const TmapKey& o) const {
    return base == o.base && rows == o.rows && row_bytes == o.row_bytes && pitch_bytes == o.pitch_bytes && box_rows == o.box_rows && atoms == o.atoms;
  }
};
struct TmapSlot {
  TmapKey key;
  CUtensorMap map;
  bool used;
};

static int make_tmap_cached(CUtensorMap* map, const TmapKey& key) {
  constexpr int SLOTS = 256;
  static thread_local TmapSlot cache[SLOTS] = {};
  uint64_t h = reinterpret_cast<uintptr_t>(key.base) >> 8;
  h ^= key.rows * 0x9E3779B97F4A7C15ull;
  h ^= (key.row_bytes << 7) ^ key.box_rows;
  TmapSlot& slot = cache[(h ^ (h >> 17)) % SLOTS];
  if (slot.used && slot.key == key) {
    *map = slot.map;
    return KF_OK;
  }
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) {
    set_error("cuTensorMapEncodeTiled is not available from the driver");
    return KF_ERR_UNSUPPORTED;
  }
  cuuint64_t dims[2] = {key.atoms ? 128 : key.row_bytes, key.rows};
  cuuint64_t strides[1] = {key.pitch_bytes};
  cuuint32_t box[2] = {128, key.box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, key.atoms ? CU_TENSOR_MAP_DATA_TYPE_UINT32 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(key.base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, key.atoms ? CU_TENSOR_MAP_SWIZZLE_NONE : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed with CUresult %d (base %p rows %llu row_bytes %llu)", (int)r, key.base, (unsigned long long)key.rows,
              (unsigned long long)key.row_bytes);
    return KF_ERR_BAD_ARGUMENT;
  }
  slot.key = key;
  slot.map = *map;
  slot.used = true;
  return KF_OK;
}
int make_tmap_2d_bytes(CUtensorMap* map, const void* base, uint64_t rows, uint64_t row_bytes, uint64_t pitch_bytes, uint32_t box_rows) {
  return make_tmap_cached(map, TmapKey{base, rows, row_bytes, pitch_bytes, box_rows, false});
}
int make_tmap_atoms(CUtensorMap* map, const void* base, uint64_t n_atoms, uint32_t atoms) {
  return make_tmap_cached(map, TmapKey{base, n_atoms, 512, 512, atoms, true});
}

int device_sm_count(int* sms) {
  static PerDevice<int> cached;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_status(e, "cudaGetDevice");
  int n = cached.get(dev);
  if (n != 0) {
    *sms = n;
    return KF_OK;
  }
  e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return cuda_status(e, "cudaDeviceGetAttribute");
  cached.put(dev, n);
  *sms = n;
  return KF_OK;
}

int launch_gemm_pair(const kf_gemm_params* p, uint64_t kbytes, uint64_t w_rows, GemmArgs& g, int sms, cudaStream_t st);   // kf_gemm_pair.cu

struct GemmMaps {
  CUtensorMap A, W, R, C;                                 // R, C: the residual and the output of a RES launch through shared memory; R: W in boxes of 128 rows for half tiles
};

template <int KIND, int EPI, int BN, int FORM>
static int launch_gemm(const GemmMaps& tm, const GemmArgs& g, int grid, cudaStream_t st) {
  static PerDevice<bool> attr_set;
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set.get(dev)) {
    cudaError_t e = cudaFuncSetAttribute(gemm_kernel<KIND, EPI, BN, FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GEMM_SMEM_MAX);
    if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute(gemm_kernel)");
    attr_set.put(dev, true);
  }
  return cuda_status(launch_maybe_pdl(g.M, gemm_kernel<KIND, EPI, BN, FORM>, dim3(grid), dim3(GEMM_THREADS), gemm_smem<EPI, BN>(g.stages, g.vec_floats, g.res_tma != 0), st, tm.A, tm.W, tm.R, tm.C, g), "kf_gemm_bs launch");
}

template <int KIND, int BN>
static int launch_gemm_epi(int epi, const GemmMaps& tm, const GemmArgs& g, int grid, cudaStream_t st) {
  return with_epilogue(epi, g, [&](auto e, auto form) { return launch_gemm<KIND, decltype(e)::value, BN, decltype(form)::value>(tm, g, grid, st); });
}

// A last round of 256-column tiles that fills at most half of the SMs is cut into halves of 128 columns: the round then takes about
// 0.6 of its time (one frame's 13 x 16 tiles are 1.6 rounds instead of 2, M = 22 470 x 3072 14.6 instead of 15).  Number of tiles cut.
static int split_tiles(int total, int N, int sms) {
  const int rest = total % sms;
  return total > sms && 2 * rest <= sms && N % 256 == 0 ? rest : 0;
}

template <int BN>
static int launch_gemm_fmt(int fmt, int epi, const GemmMaps& tm, GemmArgs& g, int sms, cudaStream_t st) {
  g.n_tiles = (g.N + BN - 1) / BN;
  const int total = g.m_tiles * g.n_tiles, grid = total < sms ? total : sms;
  const int split = BN == 256 ? split_tiles(total, g.N, sms) : 0;
  g.full_tiles = total - split;
  g.items = total + split;
  g.stages = gemm_stages<BN>(epi, g.k_tiles, g.flags, g.res_tma != 0);
  // The whole bias (+ LayerScale) vector in shared memory where a CTA works on several tiles and the ring depth leaves room for it
  const int want = (g.bias || epi == KF_EPI_RES) ? g.N * (epi == KF_EPI_RES ? 2 : 1) : 0;
  const size_t with = epi == KF_EPI_ROPE ? gemm_smem<KF_EPI_ROPE, BN>(g.stages, want) : gemm_smem<KF_EPI_RES, BN>(g.stages, want, g.res_tma != 0);
  g.vec_floats = (want > 0 && total > grid && with <= GEMM_SMEM_MAX) ? want : 0;
  switch (fmt) {
    case KF_FMT_MX8: return launch_gemm_epi<KIND_MX8, BN>(epi, tm, g, grid, st);
    case KF_FMT_NV4: return launch_gemm_epi<KIND_NV4, BN>(epi, tm, g, grid, st);
    case KF_FMT_MX4: return launch_gemm_epi<KIND_MX4, BN>(epi, tm, g, grid, st);
    default: return launch_gemm_epi<KIND_BF16, BN>(epi, tm, g, grid, st);
  }
}

// Column-tile width of a launch.  256 columns need the least operand traffic per product (the tile shape comment above) and win
// wherever there are many tiles; 128 columns cut the launch finer, take twice the SMs where the tiles do not fill the
// chip, and keep two accumulators in tensor memory.  A round of 128-column tiles takes about 0.6 of a round of 256-column tiles
// (0.7 for PLAIN, whose epilogue is too short to hide the larger operand traffic: MXFP8 1605 x 1024 x 4096 13.4 us in 3 rounds
// against 12.8 in 2; 0.505 for QUANT on 4-bit operands, which is as slow as its epilogue in either form, M = 22 470 92.6 -> 90.2 us),
// so 128 wins where its rounds are the shorter sum: one frame's 13 row tiles x 1024 columns are one round either way (104 SMs instead
// of 52: proj / fc2 NVFP4 13.9 -> 8.8 us on average).
static int gemm_columns(int fmt, int epi, int m_tiles, int N, int sms) {
  const int t256 = m_tiles * ((N + 255) / 256), t128 = m_tiles * (N / 128);
  const bool fp4 = fmt == KF_FMT_NV4 || fmt == KF_FMT_MX4;
  const int permille = epi == KF_EPI_PLAIN ? 700 : epi == KF_EPI_QUANT && fp4 ? 505 : 600;
  const int64_t cost256 = 1000 * (int64_t)(t256 / sms) + (t256 % sms == 0 ? 0 : split_tiles(t256, N, sms) ? 600 : 1000), cost128 = (int64_t)permille * ((t128 + sms - 1) / sms);
  return cost128 <= cost256 ? 128 : 256;
}

// RES launches that move the residual through shared memory on 128-column tiles: those of many rounds, where its bandwidth counts
// and the box of the next tile travels under the present one.
// Not for a long K: the 128-column tiles then cost more operand traffic than the boxes save.  256-column tiles without boxes -> 128-column
// tiles with boxes, in place, operands from HBM, us at M = 9630, 22 470 and 51 360:
//    4 stages  NVFP4 1024 x 1024   26.8 -> 20.8   47.4 -> 37.3   97.6 -> 76.8
//    6 stages  MXFP8  768 x  768   24.7 -> 21.1   41.3 -> 36.6   80.5 -> 70.8
//    8 stages  MXFP8 1024 x 1024   30.7 -> 30.0   55.6 -> 56.2  116.8 -> 112.4     NVFP4 1024 x 2048  33.6 -> 32.5  60.5 -> 61.2  120.4 -> 116.6
//   10 stages  MXFP8 1024 x 1280   33.9 -> 34.1   62.6 -> 63.8  127.8 -> 130.2
// and against CTA pairs (captured; these boxes -> pairs; 9630, 22 470, 51 360): 4 stages NVFP4 1024 x 1024 17.6 -> 19.3, 36.1 -> 38.3, 75.1 -> 86.9;
// 6 stages MXFP8 768 x 768 15.3 -> 16.4, 34.1 -> 33.9, 67.2 -> 70.7; 8 stages MXFP8 1024 x 1024 27.8 -> 23.9, 53.2 -> 44.3, 106.4 -> 86.1.
// The line lies after 6 stages where pairs are possible, after 8 where they are not.
static bool gemm_res_boxes(int k_tiles, int m_tiles, int N, int sms) {
  return k_tiles <= (N % 256 == 0 ? 6 : 8) && (int64_t)m_tiles * (N / 128) >= 3 * (int64_t)sms;
}

// Launches that run on CTA pairs (kf_gemm_pair.cu).  A tile of a pair is twice as much to lose in a last round, and a launch of pairs starts
// about a microsecond later (cluster launch, hand-shakes); what a pair gains is operand traffic, so it gains with the length of the main loop
// beside the epilogue.  The line lies by row tiles and K, in stages of 128 bytes.  One CTA -> pairs, captured launches, us at 3210, 4815, 6420 and 9630 rows:
//    PLAIN  4 stages   NVFP4 1024 x 4096   11.1 -> 10.8  14.4 -> 13.5  20.5 -> 18.2  30.7 -> 25.6     3  NVFP4  768 x 3072   8.1 -> 8.5  10.3 -> 10.7  14.3 -> 13.9  19.5 -> 18.3
//           6          MXFP8  768 x 3072   10.6 ->  9.9  14.5 -> 12.7  20.2 -> 16.6  30.6 -> 25.2    16  NVFP4 4096 x 1024   9.9 -> 10.2 15.1 -> 14.1  17.9 -> 16.1  26.9 -> 24.3
//    QUANT  3          NVFP4  768 x 3072   13.2 -> 13.5  17.1 -> 17.1  22.4 -> 21.9  30.1 -> 29.1     4  NVFP4 1024 x 4096  15.0 -> 15.6 21.3 -> 21.2  27.0 -> 27.2  40.6 -> 36.9
//           6          MXFP8  768 x 3072   13.0 -> 14.1  16.7 -> 17.5  21.8 -> 22.6  31.5 -> 30.6     8  MXFP8 1024 x 4096  18.1 -> 16.6 28.6 -> 25.2  33.2 -> 32.5  47.0 -> 46.2
//          12          bf16   768 x 3072   17.5 -> 16.6  24.3 -> 23.1  33.4 -> 28.6  44.1 -> 39.6
//    ROPE   4          NVFP4 1024 x 3072   11.5 -> 12.4  14.9 -> 16.3  20.2 -> 19.9  26.5 -> 26.2     6  MXFP8  768 x 2304  10.5 -> 11.0 13.1 -> 13.8  19.0 -> 18.0  24.3 -> 22.3
//           8          MXFP8 1024 x 3072   14.0 -> 14.7  19.2 -> 19.0  25.2 -> 24.4  39.0 -> 33.7    12  bf16   768 x 2304  15.1 -> 14.1 18.7 -> 16.8  26.0 -> 22.6  36.9 -> 31.2
//    RES    1          NVFP4  256 x 1024    9.4 ->  8.8  12.1 -> 11.0  15.1 -> 13.3                  16  NVFP4 4096 x 1024  16.3 -> 15.4 20.9 -> 20.1  24.8 -> 24.2  34.5 -> 31.1   (the residual as boxes)
// Under 3 stages the epilogue is all there is: pairs lose in ROPE (256 x 3072, 6420 rows: MXFP8 19.4 -> 22.0, NVFP4 17.5 -> 18.6), in QUANT on 8-bit
// operands (9630: 29.2 -> 34.9) and in PLAIN (256 x 1024, 22 470: NVFP4 12.0 -> 12.8) but for many rounds (256 x 4096, 22 470: MXFP8 46.2 -> 43.3); QUANT on
// 4-bit operands, as slow as its epilogue in either form, stays by its rows (256 x 4096, 9630: 35.5 -> 34.3).
// Not where the tiles do not fill the pairs (for RES half of them: without pairs its residual goes in 32-byte pieces), nor for what
// gemm_res_boxes takes.  Few rows against many columns (the mask product: two row tiles an image, 8 x 200 x 65 536 x 1024 340 -> 261 us) count from four
// rounds on, but for QUANT with a short K (MXFP8 768 x 3072, 6420 rows, is that already); a batched product needs its row tiles in twos.
static bool gemm_pairs(int fmt, int epi, int k_tiles, int m_tiles, int m_tiles_pb, int N, int sms) {
  if (N % 256 != 0 || m_tiles_pb % 2 != 0) return false;
  const int64_t tiles = (int64_t)((m_tiles + 1) / 2) * (N / 256), pairs = sms / 2;
  if (epi == KF_EPI_RES) return m_tiles >= 24 && 2 * tiles > pairs;
  const bool fp4 = fmt == KF_FMT_NV4 || fmt == KF_FMT_MX4;
  if (k_tiles < 3 && (epi == KF_EPI_PLAIN ? tiles < 8 * pairs : epi == KF_EPI_ROPE || !fp4)) return false;
  const bool long_k = k_tiles >= (epi == KF_EPI_PLAIN ? 6 : epi == KF_EPI_QUANT ? 8 : 12);
  const int rows = long_k ? 24 : epi == KF_EPI_QUANT && !fp4 ? 64 : 48;
  return tiles >= pairs && (m_tiles >= rows || (tiles >= 4 * pairs && (long_k || epi != KF_EPI_QUANT)));
}

static bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
static bool al32(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 31) == 0; }   // 256-bit global accesses of the epilogues

}  // namespace kf

using namespace kf;

extern "C" int kf_gemm_bs(const kf_gemm_params* p, void* stream) {
  KF_REQUIRE(p != nullptr, "kf_gemm_bs: null parameter block");
  const int fmt = p->fmt, epi = p->epi;
  KF_REQUIRE(fmt >= KF_FMT_MX8 && fmt <= KF_FMT_BF16, "kf_gemm_bs: unknown operand format %d", fmt);
  KF_REQUIRE(epi >= KF_EPI_PLAIN && epi <= KF_EPI_QUANT, "kf_gemm_bs: unknown epilogue %d", epi);
  KF_REQUIRE(p->M >= 0 && p->N > 0 && p->K > 0, "kf_gemm_bs: bad shape M=%d N=%d K=%d", p->M, p->N, p->K);
  KF_REQUIRE(p->N % 128 == 0, "kf_gemm_bs: N=%d must be a multiple of 128", p->N);
  const int kelems = fmt == KF_FMT_MX8 ? 128 : (fmt == KF_FMT_BF16 ? 64 : 256);   // K elements per 128-byte stage
  KF_REQUIRE(p->K % kelems == 0, "kf_gemm_bs: K=%d must be a multiple of %d for this format", p->K, kelems);
  if (p->M == 0) return KF_OK;
  KF_REQUIRE(p->A && p->W && al16(p->A) && al16(p->W), "kf_gemm_bs: A and W must be non-null and 16-byte aligned");
  if (fmt != KF_FMT_BF16) KF_REQUIRE(p->SFA && p->SFW && al16(p->SFA) && al16(p->SFW), "kf_gemm_bs: scale tensors must be non-null and 16-byte aligned");
  KF_REQUIRE(!p->bias || al16(p->bias), "kf_gemm_bs: bias must be 16-byte aligned");
  if (epi == KF_EPI_PLAIN) {
    KF_REQUIRE(p->C && al32(p->C), "kf_gemm_bs: PLAIN needs a 32-byte aligned output C");
    KF_REQUIRE(p->out_row_group >= 0 && (p->out_row_group == 0 || (p->out_row_stride >= p->out_row_group && p->out_row_offset >= 0)),
               "kf_gemm_bs: bad output row mapping group=%d stride=%d offset=%d", p->out_row_group, p->out_row_stride, p->out_row_offset);
    KF_REQUIRE(p->out_dtype == KF_F32 || p->out_dtype == KF_BF16 || p->out_dtype == KF_F16, "kf_gemm_bs: bad out_dtype %d", p->out_dtype);
  } else if (epi == KF_EPI_RES) {
    KF_REQUIRE(p->C && p->R && p->gamma && al32(p->C) && al32(p->R) && al16(p->gamma), "kf_gemm_bs: RES needs 32-byte aligned C and R and a 16-byte aligned gamma");
    KF_REQUIRE(p->out_row_group >= 0 && (p->out_row_group == 0 || (p->out_row_stride >= p->out_row_group && p->out_row_offset >= 0)),
               "kf_gemm_bs: bad output row mapping group=%d stride=%d offset=%d", p->out_row_group, p->out_row_stride, p->out_row_offset);
    KF_REQUIRE(p->out_row_group == 0 || p->C != p->R, "kf_gemm_bs: RES with an output row mapping cannot run in place");
  } else if (epi == KF_EPI_ROPE) {
    KF_REQUIRE(p->C && al32(p->C) && p->sin && p->cos && al32(p->sin) && al32(p->cos), "kf_gemm_bs: ROPE needs 32-byte aligned C, sin and cos");
    KF_REQUIRE(p->out_dtype == KF_BF16 || p->out_dtype == KF_F16, "kf_gemm_bs: ROPE output must be bf16 or f16");
    KF_REQUIRE(p->H > 0 && p->N == 3 * p->H * 64, "kf_gemm_bs: ROPE needs N = 3*H*64 (N=%d, H=%d)", p->N, p->H);
    KF_REQUIRE(p->Ntok > 0 && p->M % p->Ntok == 0 && p->prefix >= 0 && p->prefix <= p->Ntok, "kf_gemm_bs: ROPE needs M %% Ntok == 0 and 0 <= prefix <= Ntok");
  } else {
    KF_REQUIRE(p->out_fmt == KF_FMT_MX8 || p->out_fmt == KF_FMT_NV4 || p->out_fmt == KF_FMT_MX4, "kf_gemm_bs: bad quantise-out format %d", p->out_fmt);
    KF_REQUIRE(p->Qo && p->SFo && al32(p->Qo) && al16(p->SFo), "kf_gemm_bs: QUANT needs a 32-byte aligned Qo and a 16-byte aligned SFo");
    KF_REQUIRE(p->out_fmt != KF_FMT_NV4 || p->tso, "kf_gemm_bs: nv4 quantise-out needs the per-tensor scale tso");
    KF_REQUIRE(!p->y_dbg || al16(p->y_dbg), "kf_gemm_bs: y_dbg must be 16-byte aligned");
  }
  KF_REQUIRE(p->batch >= 0, "kf_gemm_bs: negative batch");
  if (p->batch > 0) {
    KF_REQUIRE(fmt == KF_FMT_BF16 && epi == KF_EPI_PLAIN && p->out_row_group == 0, "kf_gemm_bs: batched products need bf16 operands, the PLAIN epilogue and no output row mapping");
    KF_REQUIRE(p->a_rows_per_batch > 0 && (long long)p->batch * p->a_rows_per_batch == p->M && p->w_rows_per_batch >= p->N,
               "kf_gemm_bs: batched products need M = batch * a_rows_per_batch and w_rows_per_batch >= N (batch=%d, rows=%d, M=%d, w rows=%d, N=%d)",
               p->batch, p->a_rows_per_batch, p->M, p->w_rows_per_batch, p->N);
  }
  const uint64_t kbytes = fmt == KF_FMT_MX8 ? (uint64_t)p->K : (fmt == KF_FMT_BF16 ? 2ull * p->K : (uint64_t)p->K / 2);
  const uint64_t w_rows = p->batch > 0 ? (uint64_t)p->batch * p->w_rows_per_batch : (uint64_t)p->N;
  const int m_tiles = p->batch > 0 ? p->batch * ((p->a_rows_per_batch + BM - 1) / BM) : (p->M + BM - 1) / BM;
  int sms = 0;
  int st = device_sm_count(&sms);
  if (st != KF_OK) return st;
  const bool res_tma = epi == KF_EPI_RES && p->out_row_group == 0 && gemm_res_boxes((int)(kbytes / BKB), m_tiles, p->N, sms);
  const int m_tiles_pb = p->batch > 0 ? (p->a_rows_per_batch + BM - 1) / BM : 0;
  const bool pair = !res_tma && gemm_pairs(fmt, epi, (int)(kbytes / BKB), m_tiles, m_tiles_pb, p->N, sms);
  const int bn = res_tma ? 128 : gemm_columns(fmt, epi, m_tiles, p->N, sms);
  GemmArgs g{};
  g.sfa = static_cast<const uint8_t*>(p->SFA);
  g.sfw = static_cast<const uint8_t*>(p->SFW);
  g.ts_a = p->ts_a; g.ts_w = p->ts_w; g.bias = p->bias; g.gamma = p->gamma; g.R = p->R; g.sin = p->sin; g.cos = p->cos; g.tso = p->tso;
  g.C = p->C; g.Qo = static_cast<uint8_t*>(p->Qo); g.SFo = static_cast<uint8_t*>(p->SFo);
  g.M = p->M; g.N = p->N; g.K = p->K;
  g.Ntok = p->Ntok; g.prefix = p->prefix; g.H = p->H; g.d = p->H * 64;
  g.out_dtype = p->out_dtype; g.flags = p->flags; g.out_fmt = p->out_fmt;
  g.m_tiles = m_tiles; g.k_tiles = (int)(kbytes / BKB);
  if (p->batch > 0) {
    g.m_tiles_pb = m_tiles_pb;
    g.a_rows_pb = p->a_rows_per_batch;
    g.w_rows_pb = p->w_rows_per_batch;
  }
  g.nkb4 = fmt == KF_FMT_BF16 ? 0 : p->K / (4 * fmt_vec(fmt));
  const bool maps_rows = epi == KF_EPI_PLAIN || epi == KF_EPI_RES;
  g.row_group = maps_rows ? p->out_row_group : 0; g.row_stride = p->out_row_stride; g.row_offset = p->out_row_offset;
  g.res_tma = res_tma;
  g.y_dbg = epi == KF_EPI_QUANT ? p->y_dbg : nullptr;
  g.err = dev_error_ptr();
  KF_REQUIRE(g.err != nullptr, "kf_gemm_bs: device error word unavailable");
  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  if (pair) return launch_gemm_pair(p, kbytes, w_rows, g, sms, cs);
  GemmMaps tm;
  st = make_tmap_2d_bytes(&tm.A, p->A, (uint64_t)p->M, kbytes, kbytes, BM);
  if (st != KF_OK) return st;
  st = make_tmap_2d_bytes(&tm.W, p->W, w_rows, kbytes, kbytes, bn);
  if (st != KF_OK) return st;
  tm.R = tm.C = tm.A;
  if (bn == 256 && split_tiles(m_tiles * ((p->N + 255) / 256), p->N, sms)) {
    st = make_tmap_2d_bytes(&tm.R, p->W, w_rows, kbytes, kbytes, 128);   // the half tiles' W boxes
    if (st != KF_OK) return st;
  }
  if (res_tma) {
    st = make_tmap_2d_bytes(&tm.R, p->R, (uint64_t)p->M, 4ull * p->N, 4ull * p->N, 32);
    if (st != KF_OK) return st;
    st = make_tmap_2d_bytes(&tm.C, p->C, (uint64_t)p->M, 4ull * p->N, 4ull * p->N, 32);
    if (st != KF_OK) return st;
  }
  return bn == 128 ? launch_gemm_fmt<128>(fmt, epi, tm, g, sms, cs) : launch_gemm_fmt<256>(fmt, epi, tm, g, sms, cs);
}
