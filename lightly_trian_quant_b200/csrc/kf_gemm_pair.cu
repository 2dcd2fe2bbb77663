// Block-scaled GEMM on CTA pairs (tcgen05 cta_group::2): a cluster of two CTAs computes one 256 x 256 output tile.  Each CTA loads its
// own 128 rows of A and half of the tile's W rows per stage, the leader issues one M = 256, N = 256 MMA per 32 K-bytes, and every SM
// accumulates its 128 rows x 256 columns in its own tensor memory.  Formats, epilogues and the C-ABI are those of kf_gemm.cu, whose
// gemm_pairs says which launches come here: those of many rows.
//
//   why        an SM writes 32 KB of operands to shared memory per stage and the tensor core reads 32 KB, against 48 + 48 KB with a 128 x 256
//              tile of its own: of the 128 bytes a clock that shared memory moves, the bf16 main loop at full rate (512 clk a stage) takes 128
//              instead of 190.  The ring has 4 to 7 stages instead of 3 or 4, the residual of RES always has room for its boxes.
//   hand-over  full[s]   leader: the loads of BOTH CTAs complete on it (cta_group::2 loads may signal a barrier of either CTA)
//              empty[s]  per CTA: one commit of the leader's MMA warp arrives on both; tfull likewise
//              tempty    leader: the 32 epilogue warps of both CTAs have the accumulator in registers.  They arrive RELAXED: the
//                        accumulator has been read (tcgen05.wait::ld) and nothing else is handed over, while a release at cluster scope
//                        waits for the global stores of the tile before: 1350-1900 clk per tile from the accumulator to its hand-over instead of
//                        110-160, which had the pair level with one CTA
//   measured   one CTA -> pair, captured launches, M = 22 470, K x N of ViT-L (us): bf16 qkv 127 -> 107, fc1 169 -> 143, fc2 161 -> 153; MXFP8
//              qkv 79 -> 71, proj 53 -> 44, fc1 102 -> 90, fc2 96 -> 90; NVFP4 fc1 84 -> 79, fc2 65 -> 58, plain 62 -> 55
//   forms      a kernel for each (epilogue_form), as in kf_gemm.cu.  With all of them in one the bf16 kernels of PLAIN and QUANT spilled (24 and 96 bytes
//              of loads): bf16 22 400 x 1024 x 4096 GELU 143.1 -> 140.0 us, 4815 x 768 x 3072 plain 19.9 -> 19.3, GELU 22.5 -> 20.9; MXFP8 QUANT
//              22 470 x 768 x 3072 61.8 -> 61.1; NVFP4 QUANT and the one-form epilogues level
//
// No load is a multicast; the two cluster barriers (start, teardown) are reached by every thread on every path, every other wait is bounded.
// Replaces the same reference kernels as kf_gemm.cu: infer-opt/round13_mxfp8_full/impl/mgx_core.cu:118-444 and
// infer-opt/round14_fp4_full/impl/fp4g_core.cu:153-470.
#include "kf_gemm_epi.cuh"

namespace kf {

constexpr int PAIR_MAX_STAGES = 7;
constexpr int PAIR_TILE_BYTES = 2 * A_BYTES;             // 16 KB of A rows + 16 KB of W rows per CTA and stage
template <int KIND>
constexpr int pair_sf_bytes() { return 3 * KindTraits<KIND>::ATOMS * 512; }   // scale atoms of a stage: this CTA's A rows, then all 256 W rows
constexpr size_t PAIR_SMEM_MAX = 227 * 1024;
constexpr int PAIR_BAR_BYTES = 384;

template <int KIND, int EPI>
constexpr size_t pair_smem(int stages, int vec_floats, bool boxes) {
  return (size_t)stages * (PAIR_TILE_BYTES + pair_sf_bytes<KIND>()) + (boxes ? EPI_WARPS * RES_BOX_BYTES : 0) +
         (size_t)(vec_floats > EPI_WARPS * SLICE_FLOATS ? vec_floats : EPI_WARPS * SLICE_FLOATS) * 4 + (EPI == KF_EPI_ROPE ? 4 * ROPE_SLAB_FLOATS * 4 : 0) + PAIR_BAR_BYTES;
}

struct PairMaps {
  CUtensorMap A, W, Wh, SA, SW, R, C;                    // Wh: W in boxes of 64 rows for half tiles; R, C: the residual and the output of RES
};

template <int KIND, int EPI, int FORM>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ PairMaps tm, const GemmArgs g) {
  constexpr int ATOMS = KindTraits<KIND>::ATOMS;
  constexpr bool SCALED = KIND != KIND_BF16;
  constexpr int SF_BYTES = pair_sf_bytes<KIND>();
  const int STAGES = g.stages;

  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* tiles = smem;
  uint8_t* boxes = smem + (size_t)STAGES * PAIR_TILE_BYTES;                             // 1024-byte aligned
  uint8_t* sfs = boxes + (EPI == KF_EPI_RES && g.res_tma ? EPI_WARPS * RES_BOX_BYTES : 0);
  float* slices = reinterpret_cast<float*>(sfs + (size_t)STAGES * SF_BYTES);
  float* slabs = slices + (g.vec_floats > EPI_WARPS * SLICE_FLOATS ? g.vec_floats : EPI_WARPS * SLICE_FLOATS);   // ROPE only
  uint64_t* bars = reinterpret_cast<uint64_t*>(slabs + (EPI == KF_EPI_ROPE ? 4 * ROPE_SLAB_FLOATS : 0));
  uint64_t *full = bars, *empty = bars + PAIR_MAX_STAGES, *tfull = bars + 2 * PAIR_MAX_STAGES, *tempty = tfull + 1;
  uint64_t* box_full = tempty + 1;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(box_full + EPI_WARPS);
  volatile uint32_t* abort_flag = tmem_holder + 1;
  volatile uint32_t* issued = tmem_holder + 2;             // stages this CTA's producer has requested: what the residual boxes are paced by

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();                 // 0 = leader (issues the MMAs), 1 = follower
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);                              // the leader's: the loads of BOTH CTAs complete on it
      mbar_init(&empty[s], 1);                             // per CTA: the leader commits to both
    }
    mbar_init(tfull, 1);                                   // per CTA, like empty
    mbar_init(tempty, 2 * EPI_WARPS);                      // the leader's: the epilogue warps of both CTAs
    if (EPI == KF_EPI_RES)
      for (int w = 0; w < EPI_WARPS; ++w) mbar_init(&box_full[w], 1);
    *abort_flag = 0u;
    *issued = 0u;
    fence_mbar_init();
    prefetch_tmap(&tm.A);
    prefetch_tmap(&tm.W);
    if (SCALED) {
      prefetch_tmap(&tm.SA);
      prefetch_tmap(&tm.SW);
    }
  }
  if (warp == 1) {
    tmem_alloc2(tmem_holder, TMEM_COLS);
    tmem_relinquish2();
  }
  tc_fence_before();
  cluster_sync_all();                                      // both CTAs' barriers exist before anything arrives on them from outside
  tc_fence_after();
  pdl_wait();                                              // set-up done: from here on global memory of the predecessors is read and written
  const uint32_t tmem_base = *tmem_holder;
  const WaitCtx ctx{abort_flag, g.err};
  const bool bad_align = (smem_u32(smem) & 1023u) != 0;    // the same answer in every thread of both CTAs
  if (bad_align && threadIdx.x == 0 && atomicCAS(&g.err[0], 0u, (unsigned)(-KF_ERR_DEVICE_WAIT)) == 0u) {
    g.err[1] = 100;
    g.err[2] = blockIdx.x;
  }
  const int first = (int)blockIdx.x >> 1, stride = (int)gridDim.x >> 1;

  if (warp < EPI_WARP0) {
    setmaxnreg_dec<EPI == KF_EPI_ROPE ? REGS_LEAN_ROPE : REGS_LEAN>();
    if (bad_align) {
      // nothing is issued; fall through to the teardown
    } else if (warp == 0) {
      // ------------------------------------------------------------------ TMA producer (each CTA its own part)
      uint32_t s = 0, ph = 0, n_issued = 0;
      // Has an earlier launch failed?  The leader's producer alone looks, once, and raises the flag of both CTAs: without its arrivals no
      // stage completes, and the flags end the waits of all other roles.
      bool ok = true;
      if (rank == 0 && __any_sync(0xffffffffu, *static_cast<volatile unsigned int*>(g.err) != 0u)) {
        ok = false;
        *abort_flag = 1u;
        st_shared_cluster_u32(map_to_rank(const_cast<const uint32_t*>(abort_flag), 1), 1u);
      }
      const uint32_t leader_full = map_to_rank(&full[0], 0);
      for (int idx = first; idx < g.items && ok; idx += stride) {
        const WorkItem w = work_item<256>(g, idx);
        const bool half = w.cols == 128;
        const int m_blk = 2 * w.m_blk + (int)rank, w_halves = half ? 1 : 2;
        const int m_sf = m_blk < g.m_tiles ? m_blk : g.m_tiles - 1;             // a row tile past M has no scale atoms: any do, its codes read as zeros
        const uint32_t tx = 2 * (A_BYTES + (half ? A_BYTES / 2 : A_BYTES) + (SCALED ? (1 + w_halves) * ATOMS * 512 : 0));   // of both CTAs
        int row_end;
        const int a_row = tile_row0(g, m_blk, row_end), w_row = tile_wrow0(g, m_blk, w.n0) + (int)rank * (half ? 64 : 128);
        for (int kt = 0; kt < g.k_tiles; ++kt) {
          if (!mbar_wait_warp(&empty[s], ph ^ 1, ctx, 1)) { ok = false; break; }
          if (elect_one()) {
            if (rank == 0) mbar_expect_tx(&full[s], tx);
            if (EPI == KF_EPI_RES) *issued = n_issued + 1;
            const uint32_t bar = leader_full + s * 8;
            uint8_t* ta = tiles + (size_t)s * PAIR_TILE_BYTES;
            tma_load_2d_pair(ta, &tm.A, kt * BKB, a_row, bar);              // rows past M read as zeros
            tma_load_2d_pair(ta + A_BYTES, half ? &tm.Wh : &tm.W, kt * BKB, w_row, bar);
            if (SCALED) {
              uint8_t* sa = sfs + (size_t)s * SF_BYTES;
              tma_load_2d_pair(sa, &tm.SA, 0, m_sf * g.nkb4 + kt * ATOMS, bar);
              for (int h = 0; h < w_halves; ++h) tma_load_2d_pair(sa + (1 + h) * ATOMS * 512, &tm.SW, 0, (w.n0 / 128 + h) * g.nkb4 + kt * ATOMS, bar);
            }
          }
          __syncwarp();
          ++n_issued;
          if (++s == (uint32_t)STAGES) { s = 0; ph ^= 1; }
        }
      }
      // The leader's commits to the empty barriers reach both CTAs on their own time, those of the last stages too: this CTA stays until the
      // last one has arrived in every slot (a slot that was never filled is open from the start).
      for (int i = 0; i < STAGES && ok; ++i) {
        ok = mbar_wait_warp(&empty[s], ph ^ 1, ctx, 6);
        if (++s == (uint32_t)STAGES) { s = 0; ph ^= 1; }
      }
    } else if (warp == 1 && rank == 0) {
      // ------------------------------------------------------------------ MMA issuer (leader): the scale atoms of a stage, then its four MMAs
      constexpr auto idesc_n = [](int n) {
        return idesc_pair(KIND == KIND_BF16 ? idesc_f16(1, n) : KIND == KIND_MX8 ? idesc_bs(0, 1, n) : KIND == KIND_NV4 ? idesc_bs(1, 0, n) : idesc_bs(1, 1, n));
      };
      uint32_t s = 0, ph = 0, lt = 0, sb = 0;
      bool ok = true;
      for (int idx = first; idx < g.items && ok; idx += stride, ++lt) {
        const WorkItem w = work_item<256>(g, idx);
        const bool two = w.cols == 256;
        const uint32_t IDESC = two ? idesc_n(256) : idesc_n(128);
        if (!mbar_wait_cluster_warp(tempty, (lt & 1) ^ 1, ctx, 2)) break;         // both CTAs' epilogues have taken the previous tile out of TMEM
        tc_fence_after();
        for (int kt = 0; kt < g.k_tiles; ++kt) {
          if (!mbar_wait_warp(&full[s], ph, ctx, 3)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a_addr = smem_u32(tiles + (size_t)s * PAIR_TILE_BYTES);
          const uint64_t adesc = smem_desc_sw128(a_addr), bdesc = smem_desc_sw128(a_addr + A_BYTES);
          const uint32_t sf_t = tmem_base + TMEM_SF_COL + sb * SF_BUF_COLS;       // A at +0 (4 columns per atom), W at +16 (8 columns per atom pair)
          const uint32_t sa = smem_u32(sfs + (size_t)s * SF_BYTES);
          if (elect_one()) {
            if (SCALED) {
#pragma unroll
              for (int a = 0; a < ATOMS; ++a) {
                tc_cp_sf2(sf_t + 4 * a, smem_desc_sf(sa + a * 512));
                tc_cp_sf2(sf_t + 16 + 8 * a, smem_desc_sf(sa + (ATOMS + a) * 512));
                if (two) tc_cp_sf2(sf_t + 16 + 8 * a + 4, smem_desc_sf(sa + (2 * ATOMS + a) * 512));
              }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {                                       // 32 K-bytes per MMA
              const uint32_t acc = (kt | j) != 0;
              const uint64_t ad = adesc + 2 * j, bd = bdesc + 2 * j;
              if (KIND == KIND_BF16) mma2_f16(tmem_base, ad, bd, IDESC, acc);
              else if (KIND == KIND_MX8) mma2_mxf8(tmem_base, ad, bd, idesc_with_sf_id(IDESC, j, j), acc, sf_t, sf_t + 16);
              else if (KIND == KIND_NV4) mma2_nvf4(tmem_base, ad, bd, IDESC, acc, sf_t + 4 * j, sf_t + 16 + 8 * j);
              else mma2_mxf4(tmem_base, ad, bd, idesc_with_sf_id(IDESC, 2 * (j & 1), 2 * (j & 1)), acc, sf_t + 4 * (j >> 1), sf_t + 16 + 8 * (j >> 1));
            }
            tc_commit_both(&empty[s]);                                          // the stage is free again, in both CTAs
            if (kt == g.k_tiles - 1) tc_commit_both(tfull);
          }
          __syncwarp();
          if (SCALED && ++sb == SF_BUFS) sb = 0;
          if (++s == (uint32_t)STAGES) { s = 0; ph ^= 1; }
        }
      }
    }
  } else {
    setmaxnreg_inc<EPI == KF_EPI_ROPE ? REGS_EPI_ROPE : REGS_EPI>();
    if (!bad_align) epilogue_warps<EPI, 256, true, FORM>(g, tmem_base, tfull, tempty, slices, slabs, boxes, box_full, issued, &tm.R, &tm.C, ctx, warp, lane);
  }

  pdl_launch_dependents();
  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {                 // a wait ran out: give copies still in flight time to land before the CTA exits
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
  }
  cluster_sync_all();                // no arrival, load or MMA of the pair may target a CTA that has left: rings drained, accumulators read
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc2(tmem_base, TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------------------------ host side
template <int KIND, int EPI, int FORM>
static int launch_pair(const PairMaps& tm, GemmArgs& g, int pairs, bool want_vec, cudaStream_t st) {
  static PerDevice<bool> attr_set;
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set.get(dev)) {
    cudaError_t e = cudaFuncSetAttribute(gemm_pair_kernel<KIND, EPI, FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PAIR_SMEM_MAX);
    if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute(gemm_pair_kernel)");
    attr_set.put(dev, true);
  }
  const int vec = want_vec ? g.N * (EPI == KF_EPI_RES ? 2 : 1) : 0;
  g.vec_floats = pair_smem<KIND, EPI>(3, vec, g.res_tma != 0) <= PAIR_SMEM_MAX ? vec : 0;
  g.stages = 2;
  while (g.stages < PAIR_MAX_STAGES && pair_smem<KIND, EPI>(g.stages + 1, g.vec_floats, g.res_tma != 0) <= PAIR_SMEM_MAX) ++g.stages;
  return cuda_status(launch_maybe_pdl(g.M, gemm_pair_kernel<KIND, EPI, FORM>, dim3(2 * pairs), dim3(GEMM_THREADS), pair_smem<KIND, EPI>(g.stages, g.vec_floats, g.res_tma != 0), st, tm, g),
                     "kf_gemm_bs (pair) launch");
}

template <int KIND>
static int launch_pair_epi(int epi, const PairMaps& tm, GemmArgs& g, int pairs, bool want_vec, cudaStream_t st) {
  return with_epilogue(epi, g, [&](auto e, auto form) { return launch_pair<KIND, decltype(e)::value, decltype(form)::value>(tm, g, pairs, want_vec, st); });
}

// Called by kf_gemm_bs with validated arguments, N a multiple of 256 and, in a batched product, an even number of row tiles per product.
int launch_gemm_pair(const kf_gemm_params* p, uint64_t kbytes, uint64_t w_rows, GemmArgs& g, int sms, cudaStream_t st) {
  const int fmt = p->fmt, epi = p->epi;
  PairMaps tm;
  int rc = make_tmap_2d_bytes(&tm.A, p->A, (uint64_t)p->M, kbytes, kbytes, BM);
  if (rc != KF_OK) return rc;
  rc = make_tmap_2d_bytes(&tm.W, p->W, w_rows, kbytes, kbytes, 128);
  if (rc != KF_OK) return rc;
  g.n_tiles = p->N / 256;
  const int total = (g.m_tiles + 1) / 2 * g.n_tiles, most = sms / 2, pairs = total < most ? total : most;
  const int rest = total % most, split = total > most && 2 * rest <= most ? rest : 0;
  g.full_tiles = total - split;
  g.items = total + split;
  tm.Wh = tm.W;
  if (split) {
    rc = make_tmap_2d_bytes(&tm.Wh, p->W, w_rows, kbytes, kbytes, 64);
    if (rc != KF_OK) return rc;
  }
  tm.SA = tm.SW = tm.R = tm.C = tm.A;
  if (fmt != KF_FMT_BF16) {
    const uint32_t atoms = fmt == KF_FMT_NV4 ? 4 : fmt == KF_FMT_MX4 ? 2 : 1;
    rc = make_tmap_atoms(&tm.SA, p->SFA, (uint64_t)g.m_tiles * g.nkb4, atoms);
    if (rc != KF_OK) return rc;
    rc = make_tmap_atoms(&tm.SW, p->SFW, (uint64_t)(p->N / 128) * g.nkb4, atoms);
    if (rc != KF_OK) return rc;
  }
  g.res_tma = epi == KF_EPI_RES && p->out_row_group == 0;
  if (g.res_tma) {
    rc = make_tmap_2d_bytes(&tm.R, p->R, (uint64_t)p->M, 4ull * p->N, 4ull * p->N, 32);
    if (rc != KF_OK) return rc;
    rc = make_tmap_2d_bytes(&tm.C, p->C, (uint64_t)p->M, 4ull * p->N, 4ull * p->N, 32);
    if (rc != KF_OK) return rc;
  }
  const bool want_vec = (g.bias || epi == KF_EPI_RES) && total > pairs;
  switch (fmt) {
    case KF_FMT_MX8: return launch_pair_epi<KIND_MX8>(epi, tm, g, pairs, want_vec, st);
    case KF_FMT_NV4: return launch_pair_epi<KIND_NV4>(epi, tm, g, pairs, want_vec, st);
    case KF_FMT_MX4: return launch_pair_epi<KIND_MX4>(epi, tm, g, pairs, want_vec, st);
    default: return launch_pair_epi<KIND_BF16>(epi, tm, g, pairs, want_vec, st);
  }
}

}  // namespace kf
