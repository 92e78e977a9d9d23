// Paged causal prompt attention on pairs of SMs (tcgen05.mma cta_group::2), behind the interface of attn_prefill_sm100.cu.
//
// A pair of CTAs takes 256 query rows of one (sequence, query head), 128 each, and 128 keys at a time: each CTA fetches half
// of the keys and half of the value columns, and the products of both read both halves. A CTA by itself, with 64 keys at
// a time, moves twice the keys and values per row and reads its queries from shared memory twice as often, and its four
// softmax warps wait for one another's steps most of the time. 4096 tokens, single CTAs / pairs: 40 heads of 128 over 8 key heads 318 /
// 277 us (540 / 620 TFLOP/s), 32 heads of 192 (values 128) 486 / 232 us (354 / 740). Bound by the softmax (exponentials
// and its chain of tensor-memory and barrier latencies), not by the products. Where it wins: attn_on_pairs in ops/sm100.py.
//   warp 0, lane 0   TMA: queries and keys (both CTAs' copies are counted on the first CTA's barriers)
//   warp 10, lane 0  TMA: values
//   warp 1, lane 0   of the first CTA: all products; S(i + 1) = Q K^T is issued ahead of the softmax of block i, in the other of
//                    two score buffers, O += P V when P is there
//   warps 2..9       softmax, two threads per query row (64 keys of a block each, their maxima exchanged through shared
//                    memory); P goes over the scores in tensor memory, O is rescaled there when a maximum grew by more than 2^8
// Lengths, offsets and block tables are data; every wait is bounded, and a softmax warp whose wait ran out goes on through
// the barriers without touching tensor memory, so that nobody is left behind.
#include "cluster_pair.cuh"
#include "kernels.h"
#include "pair_launch.h"
#include "tmap.cuh"

namespace lb {
namespace {

constexpr int BKV = 128;
constexpr float RESCALE_LOG2 = 8.f;

struct PairAttnArgs {
  const int* cu_q; const int* ctx_lens; const int* block_table;
  int table_width, page, Hq, Hkv;
  float scale_log2;
  __nv_bfloat16* out;      // [T, Hq, dv]
  int dk, dv;
  int* status;
};

template <int DK, int DV>
struct PairAttnCfg {
  static constexpr int HALVES = DK / 64, VH = DV / 128;      // 64-column parts of a query or key row; of a CTA's value columns
  static constexpr int Q_BYTES = HALVES * 128 * 128;
  static constexpr int K_BYTES = HALVES * 64 * 128;          // 64 of the block's keys
  static constexpr int V_BYTES = VH * BKV * 128;             // half of the value columns of all its keys
  static constexpr int KS = 4, VS = 4;                       // blocks in flight
  static constexpr int RING = Q_BYTES + KS * K_BYTES + VS * V_BYTES;
  static constexpr int SMEM = RING + (2 * 2 + 1) * 128 * 4 + 512;
  static_assert(SMEM <= 227 * 1024, "shared memory budget");
};

__device__ __forceinline__ void st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// packed fp32 pairs and the three-input maximum: the softmax is bound by instruction issue next to the exponentials
__device__ __forceinline__ uint64_t pk2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void un2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

template <int DK, int DV>
__global__ void __launch_bounds__(352, 1)
pair_attn_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, const PairAttnArgs a) {
  using Cfg = PairAttnCfg<DK, DV>;
  constexpr int KS = Cfg::KS, VS = Cfg::VS;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int seq = blockIdx.z, head = blockIdx.y;
  const int q0 = a.cu_q[seq], q_len = a.cu_q[seq + 1] - q0;
  // the last rows of a sequence see the most keys: tiles are handed out from the last to the first
  const int pair_row0 = (int(gridDim.x >> 1) - 1 - int(blockIdx.x >> 1)) * 256;
  // (both CTAs of a pair decide alike: swizzled tiles need the alignment)
  if (pair_row0 >= q_len) return;
  if (smem_u32(smem) & 1023u) {
    if (threadIdx.x == 0) atomicCAS(a.status, 0, ST_BAD_ARGS);
    return;
  }
  uint8_t* q_s = smem;
  uint8_t* k_s = q_s + Cfg::Q_BYTES;
  uint8_t* v_s = k_s + KS * Cfg::K_BYTES;
  float* mxs = reinterpret_cast<float*>(smem + Cfg::RING);       // [parity][warpgroup][row]
  float* sums = mxs + 2 * 2 * 128;                               // [row], of the second warpgroup's keys
  uint64_t* q_full = reinterpret_cast<uint64_t*>(sums + 128);
  uint64_t* k_full = q_full + 1;       // [4]  counted in the first CTA, as q_full, v_full and p_ready
  uint64_t* k_empty = k_full + 4;      // [4]  in both, as the rest
  uint64_t* v_full = k_empty + 4;      // [4]
  uint64_t* v_empty = v_full + 4;      // [4]
  uint64_t* s_full = v_empty + 4;      // [2]
  uint64_t* p_ready = s_full + 2;      // [2]
  uint64_t* o_done = p_ready + 2;      // [2] even / odd blocks: a softmax warp looks at them only when it rescales
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_done + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = int(cluster_rank());
  const int tile_row0 = pair_row0 + rank * 128;
  const int ctx = a.ctx_lens[seq];
  const int kvh = head / (a.Hq / a.Hkv);
  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < 4; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_ready[i], 16);      // the softmax warps of both CTAs
      mbar_init(&o_done[i], 1);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) pair_tmem_alloc(tmem_slot);
  tc_fence_before();
  __syncthreads();
  cluster_sync();
  tc_fence_after();
  const uint32_t tmem_S = *tmem_slot, tmem_O = tmem_S + 2 * BKV;

  const int pos0 = ctx - q_len + tile_row0;                                   // absolute position of the tile's row 0
  const int rows_here = max(0, min(128, q_len - tile_row0));
  const int kv_hi = min(ctx, ctx - q_len + min(q_len, pair_row0 + 256));      // keys that the pair's last row sees
  const int n_blk = kv_hi > 0 ? (kv_hi + BKV - 1) / BKV : 0;                  // 0: a context shorter than the rows behind this tile
  const int* bt = a.block_table + long(seq) * a.table_width;

  if (warp == 0 || warp == 10) {
    if (lane == 0) {
      const bool values = warp == 10;
      const CUtensorMap* tm = values ? &tmV : &tmK;
      const int stages = values ? VS : KS, bytes = values ? Cfg::V_BYTES : Cfg::K_BYTES;
      uint8_t* ring = values ? v_s : k_s;
      uint64_t* full = values ? v_full : k_full;
      uint64_t* empty = values ? v_empty : k_empty;
      const int parts = values ? Cfg::VH : Cfg::HALVES, rows = values ? BKV : 64;
      const int col0 = values ? rank * (DV / 2) : 0, key_off = values ? 0 : rank * 64;
      tma_prefetch_desc(tm);
      bool ok = true;
      if (!values) {
        if (rank == 0) mbar_expect_tx(q_full, 2 * Cfg::Q_BYTES);
        for (int h = 0; h < Cfg::HALVES; ++h)
          pair_load_3d(q_s + h * (128 * 128), &tmQ, in_first(q_full), h * 64, head, q0 + tile_row0);
      }
      int s = 0;
      uint32_t ph = 0;
      for (int i = 0; ok && i < n_blk; ++i) {
        if (!mbar_wait(&empty[s], ph ^ 1, abort_flag)) {
          *abort_flag = 1;
          atomicCAS(a.status, 0, ST_TIMEOUT_EMPTY | SITE_PREFILL_ATTN);
          ok = false;
          break;
        }
        if (rank == 0) mbar_expect_tx(&full[s], 2 * bytes);
        const uint32_t bar = in_first(&full[s]);
        uint8_t* dst = ring + s * bytes;
        for (int p = 0; p * a.page < rows; ++p) {
          const int tok = i * BKV + key_off + p * a.page;
          // pages past the end of the sequence read a valid page: masked later
          const int cell = (tok < ctx ? bt[tok / a.page] : bt[0]) * a.page;
          for (int h = 0; h < parts; ++h)
            pair_load_3d(dst + h * (rows * 128) + p * a.page * 128, tm, bar, col0 + h * 64, kvh, cell);
        }
        if (++s == stages) { s = 0; ph ^= 1; }
      }
      // the products' signals to this CTA have all arrived before it may leave
      for (int i = 0; ok && i < stages; ++i) {
        ok = mbar_wait(&empty[s], ph ^ 1, abort_flag);
        if (++s == stages) { s = 0; ph ^= 1; }
      }
      if (!ok) {
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 2000000ull) {}
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      constexpr uint32_t idesc_s = umma_idesc(256, BKV, 1, 1, 0, 0);
      constexpr uint32_t idesc_o = umma_idesc(256, DV, 1, 1, 0, 1);           // V is MN-major
      const uint32_t qa = smem_u32(q_s);
      auto fail = [&](int code) {
        *abort_flag = 1;
        atomicCAS(a.status, 0, code | SITE_PREFILL_ATTN);
        return false;
      };
      auto issue_s = [&](int j) -> bool {
        const int st = j % KS;
        if (!mbar_wait(&k_full[st], uint32_t(j / KS) & 1u, abort_flag)) return fail(ST_TIMEOUT_FULL);
        tc_fence_after();
        const uint32_t ka = smem_u32(k_s + st * Cfg::K_BYTES);
#pragma unroll
        for (int h = 0; h < Cfg::HALVES; ++h) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if (h * 64 + k * 16 >= a.dk) break;
            pair_mma(tmem_S + uint32_t(j & 1) * BKV, umma_desc_k_sw128(qa + h * (128 * 128) + k * 32),
                     umma_desc_k_sw128(ka + h * (64 * 128) + k * 32), idesc_s, (h | k) ? 1u : 0u);
          }
        }
        pair_commit(&s_full[j & 1]);
        pair_commit(&k_empty[st]);
        return true;
      };
      bool ok = mbar_wait(q_full, 0, abort_flag) || fail(ST_TIMEOUT_FULL);
      if (n_blk > 0) ok = ok && issue_s(0);
      for (int i = 0; ok && i < n_blk; ++i) {
        // buffer (i + 1) & 1 held P(i - 1), whose products have been issued: they run in order
        if (i + 1 < n_blk && !issue_s(i + 1)) break;
        if (!mbar_wait(&p_ready[i & 1], uint32_t(i >> 1) & 1u, abort_flag)) { fail(ST_TIMEOUT_FLAG); break; }
        const int st = i % VS;
        if (!mbar_wait(&v_full[st], uint32_t(i / VS) & 1u, abort_flag)) { fail(ST_TIMEOUT_FULL); break; }
        tc_fence_after();
        const uint32_t va = smem_u32(v_s + st * Cfg::V_BYTES), tp = tmem_S + uint32_t(i & 1) * BKV;
#pragma unroll
        for (int k = 0; k < BKV / 16; ++k)
          pair_mma_ts(tmem_O, tp + k * 8, umma_desc_mn_sw128(va + k * 16 * 128, BKV * 128, 1024), idesc_o, (i | k) ? 1u : 0u);
        pair_commit(&o_done[i & 1]);
        pair_commit(&v_empty[st]);
      }
    }
  } else {
    // two threads per row: warpgroup wg works on keys wg * 64 .. of a block and on half of the output columns
    const int wg = (warp - 2) >> 2, row = (warp & 3) * 32 + lane;
    const uint32_t lane_off = uint32_t((warp & 3) * 32) << 16;
    const int qpos = pos0 + row;
    const int hi = row < rows_here ? min(ctx, qpos + 1) : 0;                  // keys that the row sees
    constexpr int OC = DV / 2;
    const uint32_t my_O = tmem_O + lane_off + wg * OC;
    float m = -INFINITY, l = 0.f, alpha = 1.f, sum = 0.f;
    // the first warpgroup adds both halves of the block before to the row's sum, in the order of the keys
    auto add_sums = [&]() { l = l * alpha + sum; l += sums[row]; };
    bool ok = true;
    auto fail = [&](int code) { *abort_flag = 1; atomicCAS(a.status, 0, code | SITE_PREFILL_ATTN); ok = false; };
    for (int i = 0; i < n_blk; ++i) {
      if (ok && !__all_sync(0xffffffffu, mbar_wait(&s_full[i & 1], uint32_t(i >> 1) & 1u, abort_flag))) fail(ST_TIMEOUT_TMEM_FULL);
      const uint32_t S = tmem_S + uint32_t(i & 1) * BKV + lane_off;
      const int key0 = i * BKV + wg * 64;
      uint32_t r[64];
      if (ok) {
        tc_fence_after();
        tmem_ld32(S + wg * 64, *reinterpret_cast<uint32_t(*)[32]>(&r[0]));
        tmem_ld32(S + wg * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(&r[32]));
        tmem_ld_wait();
      }
      const bool inner = rows_here == 128 && key0 + 64 <= min(ctx, pos0 + 1);    // every row sees all of these keys
      float mx = -INFINITY;
      if (inner) {
        float m0 = -INFINITY, m1 = m0, m2 = m0, m3 = m0;
#pragma unroll
        for (int j = 0; j < 64; j += 8) {
          m0 = max3(m0, __uint_as_float(r[j]), __uint_as_float(r[j + 1]));
          m1 = max3(m1, __uint_as_float(r[j + 2]), __uint_as_float(r[j + 3]));
          m2 = max3(m2, __uint_as_float(r[j + 4]), __uint_as_float(r[j + 5]));
          m3 = max3(m3, __uint_as_float(r[j + 6]), __uint_as_float(r[j + 7]));
        }
        mx = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
      } else {
#pragma unroll
        for (int j = 0; j < 64; ++j)
          if (key0 + j < hi) mx = fmaxf(mx, __uint_as_float(r[j]));
      }
      // both halves' maxima; past this barrier the scores have been read and P may go over them
      float* ex = mxs + (i & 1) * 256;
      ex[wg * 128 + row] = mx;
      tc_fence_before();
      asm volatile("bar.sync 1, 256;" ::: "memory");
      tc_fence_after();
      const float other = ex[(wg ^ 1) * 128 + row];
      if (i >= 1 && wg == 0) {
        add_sums();
        asm volatile("bar.arrive 2, 256;" ::: "memory");
      }
      alpha = 1.f;
      // the reference moves as it would over blocks of 64 keys, and the sums are added in that order. Not the single CTA's bits where the
      // second 64 keys raise the reference: the first ones' probabilities are rounded against the later one here, and against
      // their own (and rescaled) there; either way an error of 2^-9 each
      auto follow = [&](float half) {
        const float h = half * a.scale_log2;
        if (h > m + RESCALE_LOG2 || (m == -INFINITY && h != -INFINITY)) {
          alpha = (m == -INFINITY) ? 0.f : alpha * exp2f(m - h);
          m = h;
        }
      };
      follow(wg == 0 ? mx : other);
      follow(wg == 0 ? other : mx);
      const float neg_m = (m == -INFINITY) ? 0.f : -m;
      uint32_t packed[32];
      if (inner) {
        const uint64_t sc2 = pk2(a.scale_log2, a.scale_log2), nm2 = pk2(neg_m, neg_m);
        uint64_t acc0 = pk2(0.f, 0.f), acc1 = acc0;
#pragma unroll
        for (int j = 0; j < 64; j += 4) {
          float x0, x1, x2, x3;
          un2(fma2(pk2(__uint_as_float(r[j]), __uint_as_float(r[j + 1])), sc2, nm2), x0, x1);
          un2(fma2(pk2(__uint_as_float(r[j + 2]), __uint_as_float(r[j + 3])), sc2, nm2), x2, x3);
          const float p0 = exp2f(x0), p1 = exp2f(x1), p2 = exp2f(x2), p3 = exp2f(x3);
          acc0 = add2(acc0, pk2(p0, p1));
          acc1 = add2(acc1, pk2(p2, p3));
          packed[j / 2] = pack_bf16x2(p0, p1);
          packed[j / 2 + 1] = pack_bf16x2(p2, p3);
        }
        float s0, s1, s2, s3;
        un2(acc0, s0, s1);
        un2(acc1, s2, s3);
        sum = (s0 + s1) + (s2 + s3);
      } else {
        sum = 0.f;
#pragma unroll
        for (int j = 0; j < 64; j += 2) {
          float p0 = exp2f(fmaf(__uint_as_float(r[j]), a.scale_log2, neg_m));
          float p1 = exp2f(fmaf(__uint_as_float(r[j + 1]), a.scale_log2, neg_m));
          if (key0 + j >= hi) p0 = 0.f;
          if (key0 + j + 1 >= hi) p1 = 0.f;
          // sum what the tensor core will see, to keep numerator and denominator of short rows consistent
          const __nv_bfloat162 b = __floats2bfloat162_rn(p0, p1);
          const float2 f = __bfloat1622float2(b);
          sum += f.x + f.y;
          packed[j / 2] = *reinterpret_cast<const uint32_t*>(&b);
        }
      }
      if (wg == 1) {
        if (i >= 1) asm volatile("bar.sync 2, 256;" ::: "memory");      // the sum before this one has been read
        sums[row] = sum;
      }
      if (ok) {
        // cell c of the row holds keys 2 c (low half) and 2 c + 1
        st16(S + wg * 32, &packed[0]);
        st16(S + wg * 32 + 16, &packed[16]);
      }
      if (i >= 1 && __any_sync(0xffffffffu, alpha != 1.f)) {
        // O may be touched once the products of the block before are done; those of this block wait for p_ready
        if (ok && !__all_sync(0xffffffffu, mbar_wait(&o_done[(i - 1) & 1], uint32_t((i - 1) >> 1) & 1u, abort_flag)))
          fail(ST_TIMEOUT_TMEM_EMPTY);
        if (ok) {
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < OC; c += 16) {
            uint32_t o[16];
            tmem_ld16(my_O + c, o);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
            st16(my_O + c, o);
          }
        }
      }
      if (ok) st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) arrive_first(&p_ready[i & 1]);
    }
    if (ok && n_blk > 0 &&
        !__all_sync(0xffffffffu, mbar_wait(&o_done[(n_blk - 1) & 1], uint32_t((n_blk - 1) >> 1) & 1u, abort_flag)))
      fail(ST_TIMEOUT_TMEM_FULL);
    asm volatile("bar.sync 1, 256;" ::: "memory");
    if (wg == 0) {
      if (n_blk > 0) add_sums();
      mxs[row] = l;                    // (past the barrier nobody reads maxima)
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");
    l = mxs[row];
    if (ok) {
      tc_fence_after();
      const float inv = l > 0.f ? 1.f / l : 0.f;
      __nv_bfloat16* orow = a.out + (long(q0 + tile_row0 + row) * a.Hq + head) * a.dv + wg * OC;
#pragma unroll 1
      for (int c = 0; c < OC; c += 32) {
        uint32_t o[32];
        if (n_blk > 0) {
          tmem_ld32(my_O + c, o);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) o[j] = 0;
        }
        if (row < rows_here) {
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            uint4 u;
            u.x = pack_bf16x2(__uint_as_float(o[8 * v + 0]) * inv, __uint_as_float(o[8 * v + 1]) * inv);
            u.y = pack_bf16x2(__uint_as_float(o[8 * v + 2]) * inv, __uint_as_float(o[8 * v + 3]) * inv);
            u.z = pack_bf16x2(__uint_as_float(o[8 * v + 4]) * inv, __uint_as_float(o[8 * v + 5]) * inv);
            u.w = pack_bf16x2(__uint_as_float(o[8 * v + 6]) * inv, __uint_as_float(o[8 * v + 7]) * inv);
            if (wg * OC + c + 8 * v < a.dv) *reinterpret_cast<uint4*>(orow + c + 8 * v) = u;
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();                      // nobody signals the other CTA's shared memory any more
  if (warp == 1) {
    tc_fence_after();
    pair_tmem_dealloc(tmem_S);
  }
}

template <int DK, int DV>
int start(const CUtensorMap* tq, const CUtensorMap* tk, const CUtensorMap* tv, const PairAttnArgs& a, dim3 grid, cudaStream_t s) {
  constexpr int smem = PairAttnCfg<DK, DV>::SMEM;
  auto kfn = pair_attn_kernel<DK, DV>;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return 1;
    attr_set = true;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(352);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kfn, *tq, *tk, *tv, a) != cudaSuccess;
}

}  // namespace

int pair_attn_launch(const CUtensorMap* tq, const CUtensorMap* tk, const CUtensorMap* tv, const int* cu_q, const int* ctx_lens,
                     const int* block_table, int table_width, int page, int n_seqs, int max_q_len, int Hq, int Hkv, int dk,
                     int dv, float scale_log2, void* out, int* status, cudaStream_t s) {
  // head sizes above 192 stay on single CTAs: the rounding against a later reference (above) becomes 3% of the outputs of models
  // with 4-bit activations after 32768 tokens, and those are the ones with such heads (pairs were twice as fast there)
  if (64 % page || dk <= 64 || dv <= 64 || dk > 192 || dv > 128 || (reinterpret_cast<uintptr_t>(out) & 15)) return -1;
  PairAttnArgs a{cu_q, ctx_lens, block_table, table_width, page, Hq, Hkv, scale_log2, static_cast<__nv_bfloat16*>(out), dk, dv,
                 status};
  const dim3 grid(2 * ((max_q_len + 255) / 256), Hq, n_seqs);
  return dk <= 128 ? start<128, 128>(tq, tk, tv, a, grid, s) : start<192, 128>(tq, tk, tv, a, grid, s);
}

}  // namespace lb
