// Prompt-sized bf16 GEMM on pairs of SMs (tcgen05.mma cta_group::2), behind the interface of gemm_sm100.cu.
//
//   out[token, feature] = sum_k W[group * rows_per_group + feature, k] * X[token, k]       (dense or grouped, optional gate/up)
//
// A pair of CTAs multiplies 256 weight rows with BN tokens: each CTA holds 128 of the rows and half of the tokens in shared
// memory, and the accumulators of its rows (all BN tokens) in its tensor memory. One CTA by itself (128 x 256 tile) moves 12 KB
// of operands per 128 cycles of products into shared memory and reads them again, 187 bytes per cycle against the 128 that
// shared memory gives, and reached 1.08 PFLOP/s; the pair's tile halves the token side of that.
// Gate and up rows of the same 64 features lie in one CTA's tile (rows 0..63 and 64..127), so the activation needs no
// exchange between the CTAs and no second accumulator.
// Work items run in bands of BAND token tiles, all features of a band before the next: the pairs that run side by side
// share both operands in L2, and the weights are fetched once per band instead of once per token tile.
//
// Roles per CTA (320 threads, persistent): warp 0 TMA producer of the own tiles (both CTAs' copies are counted on the first
// CTA's barrier), warp 1 of the first CTA issues the products for both, warps 2..5 and 6..9 epilogue, on alternate blocks
// of 32 tokens (one warpgroup takes longer for a tile than its products do at K = 2048). Every wait is bounded.
#include "act_type.cuh"
#include "cluster_pair.cuh"
#include "gemm_sm100.h"
#include "tmap.cuh"

namespace lb {
namespace {

constexpr int BM = 128, BK = 64, BAND = 8;

template <int BN>
struct PairCfg {
  static constexpr int W_BYTES = BM * BK * 2;
  static constexpr int X_BYTES = BN / 2 * BK * 2;
  static constexpr int STAGE_BYTES = W_BYTES + X_BYTES;
  static constexpr int STAGES = BN == 256 ? 6 : 8;
  static constexpr int NACC = 512 / BN;     // all of tensor memory: the columns lie alike in both CTAs
  static constexpr int EPI_BYTES = 2 * 32 * BM * 4;     // one staging tile per epilogue warpgroup
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + EPI_BYTES + 1024 + 256;
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory budget");
};

struct PairItem { int group, tok0, out0, ntok, feat0; };      // feat0: first feature of this CTA

template <int BN, bool DUAL>
__device__ __forceinline__ bool pair_item(const WgemmArgs& a, int w, int n_tok_tiles, int rank, PairItem& it) {
  const int fb = (a.n_feat + (DUAL ? 127 : 255)) / (DUAL ? 128 : 256);
  const int band = w / (BAND * fb);
  const int here = min(BAND, n_tok_tiles - band * BAND);
  if (here <= 0) return false;
  const int r = w - band * BAND * fb;
  const int f = r / here;
  if (f >= fb) return false;
  const int tt = band * BAND + r - f * here;
  it.feat0 = (f * 2 + rank) * (DUAL ? 64 : 128);
  if (a.tile_group) {
    it.group = a.tile_group[tt];
    it.tok0 = a.tile_tok0[tt];
    it.out0 = a.tile_out0 ? a.tile_out0[tt] : it.tok0;
    it.ntok = a.tile_ntok[tt];
  } else {
    it.group = 0;
    it.tok0 = tt * BN;
    it.out0 = it.tok0;
    it.ntok = min(BN, a.n_tok - it.tok0);
  }
  return true;
}

template <int BN, bool DUAL>
__global__ void __launch_bounds__(320, 1)
pair_gemm_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const WgemmArgs a) {
  using Cfg = PairCfg<BN>;
  constexpr int STAGES = Cfg::STAGES, NACC = Cfg::NACC;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* stage = reinterpret_cast<float*>(smem + STAGES * Cfg::STAGE_BYTES);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * Cfg::STAGE_BYTES + Cfg::EPI_BYTES);     // the first CTA's count
  uint64_t* empty = full + STAGES;
  uint64_t* tfull = empty + STAGES;
  uint64_t* tempty = tfull + NACC;                                                                     // the first CTA's count
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + NACC);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = int(cluster_rank());
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int i = 0; i < NACC; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], 16);         // the epilogue warps of both CTAs
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    pair_tmem_alloc(tmem_slot);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();                        // barriers and tensor memory of both CTAs are set up
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  griddep_wait();
  griddep_launch();

  const int n_tok_tiles = a.tile_group ? min(*a.n_tiles_dev, a.n_tok_tiles_max) : (a.n_tok + BN - 1) / BN;
  const int num_kb = (a.K + BK - 1) / BK;
  const int w0 = blockIdx.x >> 1, step = gridDim.x >> 1;

  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&tmW);
      tma_prefetch_desc(&tmX);
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      PairItem it;
      for (int w = w0; ok && pair_item<BN, DUAL>(a, w, n_tok_tiles, rank, it); w += step) {
        const int wrow = it.group * a.rows_per_group + it.feat0;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(&empty[s], ph ^ 1, abort_flag)) {
            *abort_flag = 1;
            atomicCAS(a.status, 0, ST_TIMEOUT_EMPTY | SITE_GEMM);
            ok = false;
            break;
          }
          uint8_t* st = smem + s * Cfg::STAGE_BYTES;
          if (rank == 0) mbar_expect_tx(&full[s], 2 * Cfg::STAGE_BYTES);
          const uint32_t bar = in_first(&full[s]);
          pair_load_2d(st, &tmW, bar, kb * BK, wrow);
          if (DUAL) pair_load_2d(st + Cfg::W_BYTES / 2, &tmW, bar, kb * BK, wrow + a.dual_offset);
          pair_load_2d(st + Cfg::W_BYTES, &tmX, bar, kb * BK, it.tok0 + rank * (BN / 2));
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
      }
      // the products' signals to this CTA have all arrived before it may leave
      for (int i = 0; ok && i < STAGES; ++i) {
        ok = mbar_wait(&empty[s], ph ^ 1, abort_flag);
        if (++s == STAGES) { s = 0; ph ^= 1; }
      }
      if (!ok) {                         // copies in flight get a bounded time to land
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 2000000ull) {}
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      constexpr uint32_t idesc = umma_idesc(2 * BM, BN, 1, 1, 0, 0);
      int s = 0, acc = 0;
      uint32_t ph = 0, acc_ph = 0;
      bool ok = true;
      PairItem it;
      for (int w = w0; ok && pair_item<BN, DUAL>(a, w, n_tok_tiles, rank, it); w += step) {
        if (!mbar_wait(&tempty[acc], acc_ph ^ 1, abort_flag)) {
          *abort_flag = 1;
          atomicCAS(a.status, 0, ST_TIMEOUT_TMEM_EMPTY | SITE_GEMM);
          break;
        }
        tc_fence_after();
        const uint32_t d0 = tmem_base + acc * BN;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(&full[s], ph, abort_flag)) {
            *abort_flag = 1;
            atomicCAS(a.status, 0, ST_TIMEOUT_FULL | SITE_GEMM);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + s * Cfg::STAGE_BYTES);
          const uint64_t dw = umma_desc_k_sw128(sa), dx = umma_desc_k_sw128(sa + Cfg::W_BYTES);
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            pair_mma(d0, dw + uint64_t(k * 2), dx + uint64_t(k * 2), idesc, (kb | k) ? 1u : 0u);
          pair_commit(&empty[s]);
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
        if (!ok) break;
        pair_commit(&tfull[acc]);
        if (++acc == NACC) { acc = 0; acc_ph ^= 1; }
      }
    }
  } else {
    const int q = warp & 3, row = q * 32 + lane, eset = (warp - 2) >> 2, etid = threadIdx.x - 64 - eset * 128;
    stage += eset * (32 * BM);
    constexpr int TPR = DUAL ? 8 : 16;               // threads per output row of 8 features each
    constexpr int RPP = 128 / TPR;                   // rows per pass
    const int f8 = (etid % TPR) * 8;
    int acc = 0;
    uint32_t acc_ph = 0;
    PairItem it;
    for (int w = w0; pair_item<BN, DUAL>(a, w, n_tok_tiles, rank, it); w += step) {
      if (!__all_sync(0xffffffffu, mbar_wait(&tfull[acc], acc_ph, abort_flag))) {
        *abort_flag = 1;
        atomicCAS(a.status, 0, ST_TIMEOUT_TMEM_FULL | SITE_GEMM);
        break;
      }
      tc_fence_after();
      const uint32_t t0 = tmem_base + (uint32_t(q * 32) << 16) + acc * BN;
      const int feat8 = it.feat0 + f8;
#pragma unroll 1
      for (int c = eset * 32; c < BN; c += 64) {
        if (c >= it.ntok) break;
        uint32_t r[32];
        tmem_ld32(t0 + c, r);
        // output rows of this thread's passes, asked for before the first store could be in their way
        long orows[32 / RPP];
#pragma unroll
        for (int p = 0; p < 32 / RPP; ++p) {
          const int t = c + p * RPP + etid / TPR;
          orows[p] = t < it.ntok && feat8 < a.n_feat ? (a.out_rows ? long(a.out_rows[it.out0 + t]) : long(it.out0 + t)) : -1;
        }
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) stage[j * BM + row] = __uint_as_float(r[j]);
        asm volatile("bar.sync %0, 128;" ::"r"(2 + eset) : "memory");
#pragma unroll
        for (int p = 0; p < 32 / RPP; ++p) {
          const int j = p * RPP + etid / TPR;
          if (orows[p] < 0) continue;
          const float4 v0 = *reinterpret_cast<const float4*>(&stage[j * BM + f8]);
          const float4 v1 = *reinterpret_cast<const float4*>(&stage[j * BM + f8 + 4]);
          float v[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
          if (DUAL) {
            const float4 u0 = *reinterpret_cast<const float4*>(&stage[j * BM + 64 + f8]);
            const float4 u1 = *reinterpret_cast<const float4*>(&stage[j * BM + 64 + f8 + 4]);
            const float u[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = gate_act(v[e], a.act) * u[e];
          }
          if (a.tok_scale) {
            const float sc = a.tok_scale[it.out0 + c + j];
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] *= sc;
          }
          if (a.residual) {
            const uint4 rr = *reinterpret_cast<const uint4*>(a.residual + orows[p] * a.ldr + feat8);
            const __nv_bfloat162* r2 = reinterpret_cast<const __nv_bfloat162*>(&rr);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float2 f = __bfloat1622float2(r2[e]);
              v[2 * e] += f.x;
              v[2 * e + 1] += f.y;
            }
          }
          uint4 o;
          o.x = pack_bf16x2(v[0], v[1]); o.y = pack_bf16x2(v[2], v[3]);
          o.z = pack_bf16x2(v[4], v[5]); o.w = pack_bf16x2(v[6], v[7]);
          *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(a.out) + orows[p] * a.ldo + feat8) = o;
        }
        asm volatile("bar.sync %0, 128;" ::"r"(2 + eset) : "memory");
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) arrive_first(&tempty[acc]);
      if (++acc == NACC) { acc = 0; acc_ph ^= 1; }
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync();                        // nobody signals the other CTA's shared memory any more
  if (warp == 1) {
    tc_fence_after();
    pair_tmem_dealloc(tmem_base);
  }
}

template <int BN, bool DUAL>
int start(const WgemmHost& h, const WgemmArgs& a, int grid, cudaStream_t stream, const char** err) {
  using Cfg = PairCfg<BN>;
  const CUtensorMap* tmW = tmap_2d(h.w, uint64_t(h.w_rows), uint64_t(h.K), uint64_t(h.ldw) * 2, DUAL ? 64 : 128, BK, TM_BF16, true);
  const CUtensorMap* tmX = tmap_2d(h.x, uint64_t(h.x_rows), uint64_t(h.K), uint64_t(h.ldx) * 2, BN / 2, BK, TM_BF16, true);
  if (!tmW || !tmX) {
    *err = tmap_last_error();
    return 1;
  }
  auto kfn = pair_gemm_kernel<BN, DUAL>;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES) != cudaSuccess) {
      *err = "cannot set the shared memory size";
      return 1;
    }
    attr_set = true;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(320);
  cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kfn, *tmW, *tmX, a);
  if (e != cudaSuccess) *err = cudaGetErrorString(e);
  return e != cudaSuccess;
}

}  // namespace

bool wgemm_pair_ok(const WgemmHost& h, const WgemmArgs& a, int sms) {
  if (h.out_f32 || h.w_scales || h.w_bscale || h.xielu || h.relu2 || h.bias || h.comm.enabled || h.head.enabled ||
      h.n_out_peer > 0 || h.x_group_col != 0 || h.n_groups > 0 || a.split_k > 1 || !a.vec_ok || h.K < 512)
    return false;
  // grouped tiles of 128 tokens are bound by what L2 delivers, 48 KB per k block and pair or CTA. 128 experts of 2048 x 768,
  // 44,000 token rows: down projection 222 us on pairs, 317 us by single CTAs; gate and up 372 and 291
  if (h.tile_group) return h.bn == 128 && !h.dual && h.n_tok_tiles_max >= 64;
  // enough tiles for every pair; below that more and smaller ones do better (the dispatch's rule for the tile is the same)
  if (h.bn != (h.dual ? 128 : 256) || h.n_tok <= 128) return false;
  const long items = long((h.n_tok + 255) / 256) * ((h.n_feat + (h.dual ? 127 : 255)) / (h.dual ? 128 : 256));
  return items >= sms / 2;
}

int wgemm_pair_launch(const WgemmHost& h, const WgemmArgs& a, int sms, cudaStream_t stream, const char** err) {
  const int bn = h.tile_group ? 128 : 256;
  const long tiles = h.tile_group ? h.n_tok_tiles_max : (h.n_tok + bn - 1) / bn;
  const long items = tiles * ((h.n_feat + (h.dual ? 127 : 255)) / (h.dual ? 128 : 256));
  const int grid = 2 * int(items < sms / 2 ? items : sms / 2);
  if (bn == 128) return start<128, false>(h, a, grid, stream, err);
  return h.dual ? start<256, true>(h, a, grid, stream, err) : start<256, false>(h, a, grid, stream, err);
}

}  // namespace lb
