// Persistent form of the tcgen05 products for many tokens: pairs of CTAs (cta_group::2) walk the output tiles.
//
// The one-tile-per-CTA kernel (gemm_kernel.cuh) is not bound by a pipe at many tokens: tensor pipe 61 % active at 2048 tokens
// on 34816 x 5120, shared-memory reads 30 %, L2 to SM 29 % (int8) and 43 % (bf16) of their peaks.  What is missing is
// overlap: filling the ring, the epilogue and the launch of the next CTA stand between two main loops.  Here
//   * a pair of CTAs owns a tile of 256 weight rows x NT tokens (32 or 64 in batched decode).  One tcgen05.mma of M = 256 reads
//     128 weight rows and half of the tokens from each CTA's shared memory, so a CTA fetches 32 KB per 128 bytes of k for 128 x
//     256 accumulator columns;
//   * the accumulators (256 TMEM columns: NT = 256 tokens of a bf16 product, or two limbs of NT = 128 tokens of an int8 one)
//     are double-buffered: the epilogue of a tile runs beside the main loop of the next one;
//   * the ring of stages runs on across tiles.
// Tiles are dealt statically, `group_m` token tiles by all weight tiles at a time: the 74 tiles in flight then span about as
// many bytes of weights as of activations, and both stay in L2.  Where the last round of tiles would leave half of the pairs
// or more without one, its tiles are cut along k: the fp32 partial results meet in a workspace, and the last CTA of a tile's
// half to arrive adds them in the order of the slices and runs the epilogue.
//
// Roles per CTA (384 threads): warps 0 and 2 copy (alternate stages), warps 4..11 run the epilogue of this CTA's 128 rows (two
// warps per 32 rows, alternate blocks of 16 tokens; residual rows are requested a block ahead), warp 1 of the first CTA issues
// the MMAs of both.  Barriers: `full` (first CTA: bytes of both), `empty` and `acc_full` (both CTAs, arrived on by
// tcgen05.commit), `acc_empty` (first CTA: one arrival per epilogue warp of both).  Every wait is bounded.
#pragma once
#include "gemm_kernel.cuh"

namespace ti {

template <int NT, bool BF16> struct PairGeom {
  static constexpr int kStageB = (BF16 ? 1 : 2) * (NT / 2) * kBK * kKS;       // this CTA's half of the tokens (both limb planes)
  static constexpr int kStageBytes = kStageA + kStageB;
  static constexpr int kStages = 192 * 1024 / kStageBytes;
  static constexpr int kAccCols = (BF16 ? 1 : 2) * NT;
  static constexpr int kEpiBytes = 8 * 16 * 36 * 4;                           // 16 tokens x 32 rows of results per epilogue warp
  static constexpr size_t kSmem = (size_t)kStages * kStageBytes + kEpiBytes + 16 * kStages + 64 + 1024;
};
constexpr int kPairs = 74;                                                    // pairs of SMs of a B200
constexpr int kPairThreads = 384, kPairProducerB = 2, kPairEpilogue = 4;      // second copying warp, first epilogue warp

// instruction descriptors of idesc_i8 / idesc_bf16 with M = 256
template <int BN> TI_DEVICE constexpr uint32_t idesc_pair_i8(bool b_signed) {
  return (2u << 4) | (1u << 7) | ((b_signed ? 1u : 0u) << 10) | ((uint32_t)(BN >> 3) << 17) | (16u << 24);
}
template <int BN> TI_DEVICE constexpr uint32_t idesc_pair_bf16() {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | (16u << 24);
}

// What the plan of a launch says about its work: `whole` tiles with all of k, then `cut` tiles in `slices` slices of
// kb_per_split stages each.  A pair takes units pair, pair + pairs, ...
struct PairUnit {
  int m, n, kb0, kb1, slice, r;      // tile; its stages of k; slice and number of a cut tile, or slice -1
};
TI_HOST_DEVICE PairUnit pair_unit(int u, int tiles_m, int tiles_n, int group_m, int KB, int whole, int cut, int kb_per_split) {
  PairUnit x;
  int tile = u;
  x.slice = -1;
  x.r = 0;
  x.kb0 = 0;
  x.kb1 = KB;
  if (u >= whole) {
    x.slice = (u - whole) / cut;
    x.r = u - whole - x.slice * cut;
    tile = whole + x.r;
    x.kb0 = x.slice * kb_per_split;
    x.kb1 = x.kb0 + kb_per_split < KB ? x.kb0 + kb_per_split : KB;
  }
  const int per = group_m * tiles_n, grp = tile / per, rem = tile - grp * per;
  const int gm = tiles_m - grp * group_m < group_m ? tiles_m - grp * group_m : group_m;
  x.n = rem / gm;
  x.m = grp * group_m + rem - x.n * gm;
  return x;
}

template <int NT, bool BF16>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1) gemm_pair_kernel(const __grid_constant__ GemmParams p) {
  using G = PairGeom<NT, BF16>;
  constexpr int kStages = G::kStages, kStageBytes = G::kStageBytes, kPlane = (NT / 2) * kBK * kKS;
  constexpr uint32_t kCols = 2 * G::kAccCols;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const uint32_t stage0 = smem_u32(smem);
  uint8_t* after = smem + kStages * kStageBytes;                  // epilogue blocks, then the barriers
  const uint32_t full0 = smem_u32(after + G::kEpiBytes), empty0 = full0 + 8 * kStages;
  const uint32_t acc_full = empty0 + 8 * kStages, acc_empty = acc_full + 16, tmem_slot = acc_empty + 16;
  uint32_t* tmem_slot_ptr = reinterpret_cast<uint32_t*>(after + G::kEpiBytes + 16 * kStages + 32);
  __shared__ int s_last;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int tiles_m = (p.M + NT - 1) / NT, KB = (p.K + kBK * kKS - 1) / (kBK * kKS);
  const int units = p.whole + p.cut * p.slices, mine = pair < units ? (units - 1 - pair) / pairs + 1 : 0;
  auto unit = [&](int i) { return pair_unit(pair + i * pairs, tiles_m, p.tiles_n, p.group_m, KB, p.whole, p.cut, p.kb_per_split); };

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full + 8 * b, 1);
      mbar_init(acc_empty + 8 * b, 16);
    }
    fence_mbar_init();
  }
  if (warp == 1) tmem_alloc_pair(tmem_slot, kCols);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;

  pdl_trigger();
  if (warp == 0 || warp == kPairProducerB) {
    // ------------------------------------------------------------ copies: every other stage of this pair's sequence
    const int first = warp == 0 ? 0 : 1;
    const uint32_t full_of = map_to_rank(full0, 0);                // the bytes of both CTAs are counted on the first one's
    int n_pre = 0;
    // weights do not depend on the preceding kernel: those of the first ring fill are requested before the wait
    if (mine > 0) {
      const PairUnit x = unit(0);
      n_pre = min(kStages, x.kb1 - x.kb0);
      if (elect_one()) {
        for (int it = first; it < n_pre; it += 2) {
          if (rank == 0) mbar_expect_tx(full0 + 8 * it, 2 * kStageBytes);
          tma_pair_4d(stage0 + it * kStageBytes, &p.map_w, 0, 0, (x.kb0 + it) * kKS, x.n * 32 + (int)rank * 16, full_of + 8 * it);
        }
      }
      __syncwarp();
    }
    pdl_wait();
    if (elect_one()) {
      const int row = (int)rank * (NT / 2);
      bool ok = true;
      int it = 0;
      for (int i = 0; i < mine && ok; ++i) {
        const PairUnit x = unit(i);
        for (int kb = x.kb0; kb < x.kb1; ++kb, ++it) {
          if ((it & 1) != first) continue;
          const int s = it % kStages;
          const uint32_t dst = stage0 + s * kStageBytes, bar = full_of + 8 * s;
          if (it >= n_pre) {
            if (it >= kStages) ok = mbar_wait(empty0 + 8 * s, ((it / kStages) & 1) ^ 1, kGemmWaitNs, p.status);
            if (!ok) break;
            if (rank == 0) mbar_expect_tx(full0 + 8 * s, 2 * kStageBytes);
            tma_pair_4d(dst, &p.map_w, 0, 0, kb * kKS, x.n * 32 + (int)rank * 16, bar);
          }
          tma_pair_2d(dst + kStageA, &p.map_xh, kb * kBK * kKS, x.m * NT + row, bar);
          if (!BF16) tma_pair_2d(dst + kStageA + kPlane, &p.map_xl, kb * kBK * kKS, x.m * NT + row, bar);
        }
      }
      // Before a CTA leaves, the commits on its `empty` barriers for the last ring fill have to arrive: nobody else waits for
      // them, and those of both CTAs come from the first one's MMAs.  After a wait that ran out the copies already issued have
      // to land; the first CTA counts the bytes of both and holds the second at the closing cluster barrier.
      const int last = max(0, it - kStages);
      for (int k = last; k < it && ok; ++k)
        if ((k & 1) == first) ok = mbar_wait(empty0 + 8 * (k % kStages), (k / kStages) & 1, kGemmWaitNs, p.status);
      if (!ok && rank == 0)
        for (int k = last; k < it; ++k)
          if ((k & 1) == first) mbar_wait(full0 + 8 * (k % kStages), (k / kStages) & 1, kPairDrainNs, p.status);
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMAs of both CTAs
    pdl_wait();
    if (rank == 0 && elect_one()) {
      bool ok = true;
      int it = 0;
      for (int i = 0; i < mine && ok; ++i) {
        const int b = i & 1;
        const PairUnit x = unit(i);
        ok = mbar_wait_cluster(acc_empty + 8 * b, ((i >> 1) & 1) ^ 1, 2 * kGemmWaitNs, p.status);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d = tmem_base + (uint32_t)(b * G::kAccCols);
        for (int kb = x.kb0; kb < x.kb1; ++kb, ++it) {
          const int s = it % kStages;
          ok = mbar_wait(full0 + 8 * s, (it / kStages) & 1, kGemmWaitNs, p.status);
          if (!ok) break;
          tc_fence_after();
          const uint32_t a = stage0 + s * kStageBytes, bh = a + kStageA;
#pragma unroll
          for (int j = 0; j < 2 * kKS; ++j) {                     // four 32-byte k steps (operand layouts: gemm_kernel.cuh)
            const uint32_t acc = (kb > x.kb0 || j > 0) ? 1u : 0u;
            const uint64_t da = smem_desc_sw64_sbo(a + (j >> 1) * 512 + (j & 1) * 32, 1024);
            if (BF16) {
              umma_pair_bf16(d, da, smem_desc_sw128(bh + j * 32), idesc_pair_bf16<NT>(), acc);
            } else {
              umma_pair_i8(d, da, smem_desc_sw128(bh + j * 32), idesc_pair_i8<NT>(true), acc);
              umma_pair_i8(d + NT, da, smem_desc_sw128(bh + kPlane + j * 32), idesc_pair_i8<NT>(false), acc);
            }
          }
          umma_commit_pair(empty0 + 8 * s);
        }
        umma_commit_pair(acc_full + 8 * b);
      }
    }
    __syncwarp();
  } else if (warp >= kPairEpilogue) {
    // ------------------------------------------------------------ epilogue of this CTA's 128 rows (warp & 3: TMEM lane quarter)
    const int quarter = warp & 3, half = (warp - kPairEpilogue) >> 2;
    float* stage_t = reinterpret_cast<float*>(after) + (warp - kPairEpilogue) * (16 * 36);
    const uint32_t acc_empty_of = map_to_rank(acc_empty, 0);
    const int tk = lane >> 2, c8 = (lane & 3) * 8;                // stores: token of eight, first of eight adjacent rows
    const bool pre = gemm_resid_vec(p);
    pdl_wait();
    bool ok = true;
    for (int i = 0; i < mine; ++i) {
      const int b = i & 1;
      const PairUnit x = unit(i);
      const int m0 = x.m * NT, n0 = x.n * 256 + (int)rank * kBM + quarter * 32, n = n0 + lane, ns = n0 + c8;
      const float ws = n < p.N ? (BF16 ? 1.f : __bfloat162float(p.wscale[n])) : 0.f;
      // this lane's rows of the workspace of a cut tile: [slice][cut tile][token][256]
      float* part = p.part + ((size_t)max(x.slice, 0) * p.cut + x.r) * (NT * 256) + (ns - x.n * 256);
      ResidPre r[2] = {};
      if (pre && x.slice < 0)
#pragma unroll
        for (int u = 0; u < 2; ++u)
          if (m0 + half * 16 + tk + 8 * u < p.M && ns + 8 <= p.N) r[u] = gemm_resid_load(p, m0 + half * 16 + tk + 8 * u, ns);
      ok = ok && mbar_wait(acc_full + 8 * b, (i >> 1) & 1, 4 * kGemmWaitNs, p.status);
      ok = __all_sync(0xffffffffu, ok);
      if (ok) {
        tc_fence_after();
        const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(b * G::kAccCols);
        for (int c0 = half * 16; c0 < NT; c0 += 32) {
          if (m0 + c0 >= p.M) break;
          uint32_t hi[16], lo[16];
          tmem_ld16(taddr + c0, hi);
          if (!BF16) tmem_ld16(taddr + NT + c0, lo);
          ResidPre rn[2] = {};
          if (pre && x.slice < 0 && c0 + 32 < NT)                 // the next block's residual rows
#pragma unroll
            for (int u = 0; u < 2; ++u)
              if (m0 + c0 + 32 + tk + 8 * u < p.M && ns + 8 <= p.N) rn[u] = gemm_resid_load(p, m0 + c0 + 32 + tk + 8 * u, ns);
          const int m_lane = m0 + c0 + (lane & 15);
          const float xs_lane = (!BF16 && m_lane < p.M) ? p.xscale[m_lane] : 0.f;
          tmem_ld_wait();
          __syncwarp();                                           // the previous block has been written out
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float xs = __shfl_sync(0xffffffffu, xs_lane, j);
            stage_t[j * 36 + lane] = BF16 ? __uint_as_float(hi[j]) : ((float)(int)hi[j] * 256.f + (float)(int)lo[j]) * xs * ws;
          }
          __syncwarp();
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int tok = tk + 8 * u, m = m0 + c0 + tok;
            const float4 va = *reinterpret_cast<const float4*>(stage_t + tok * 36 + c8);
            const float4 vb = *reinterpret_cast<const float4*>(stage_t + tok * 36 + c8 + 4);
            if (x.slice >= 0) {
              float4* dst = reinterpret_cast<float4*>(part + (c0 + tok) * 256);
              __stcg(dst, va);
              __stcg(dst + 1, vb);
            } else if (m < p.M && ns < p.N) {
              gemm_store8(p, m, ns, va, vb, 1, 0, pre, r[u]);
            }
          }
          r[0] = rn[0];
          r[1] = rn[1];
        }
        tc_fence_before();
        __syncwarp();                                             // every lane's TMEM loads have returned
        if (lane == 0) mbar_arrive_cluster(acc_empty_of + 8 * b);
      }
      if (x.slice >= 0) {                                         // also after a wait that ran out: the counters stay in step
        __threadfence();
        asm volatile("bar.sync 1, 256;\n" ::: "memory");
        if (threadIdx.x == 32 * kPairEpilogue) {
          unsigned* count = p.tile_count + 2 * x.r + rank;
          s_last = atomicAdd(count, 1u) + 1 == (unsigned)p.slices;
          if (s_last) *count = 0;                                 // ready for the next launch
          __threadfence();
        }
        asm volatile("bar.sync 1, 256;\n" ::: "memory");
        if (s_last) {
          const float* base = p.part + (size_t)x.r * (NT * 256) + (ns - x.n * 256);
          for (int c0 = half * 16; c0 < NT; c0 += 32) {
            if (m0 + c0 >= p.M) break;
            float4 va[2], vb[2];
            ResidPre rr[2] = {};
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              va[u] = vb[u] = make_float4(0.f, 0.f, 0.f, 0.f);
              if (pre && m0 + c0 + tk + 8 * u < p.M && ns + 8 <= p.N) rr[u] = gemm_resid_load(p, m0 + c0 + tk + 8 * u, ns);
            }
            for (int z0 = 0; z0 < p.slices; z0 += 4) {            // the loads of four slices are in flight together
              float4 a[2][4], c[2][4];
#pragma unroll
              for (int z = 0; z < 4; ++z)
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                  const float4* src = reinterpret_cast<const float4*>(base + (size_t)(z0 + z) * p.cut * (NT * 256) + (c0 + tk + 8 * u) * 256);
                  a[u][z] = c[u][z] = make_float4(0.f, 0.f, 0.f, 0.f);
                  if (z0 + z < p.slices) {
                    a[u][z] = __ldcg(src);
                    c[u][z] = __ldcg(src + 1);
                  }
                }
#pragma unroll
              for (int z = 0; z < 4; ++z)
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                  va[u] = make_float4(va[u].x + a[u][z].x, va[u].y + a[u][z].y, va[u].z + a[u][z].z, va[u].w + a[u][z].w);
                  vb[u] = make_float4(vb[u].x + c[u][z].x, vb[u].y + c[u][z].y, vb[u].z + c[u][z].z, vb[u].w + c[u][z].w);
                }
            }
#pragma unroll
            for (int u = 0; u < 2; ++u)
              if (m0 + c0 + tk + 8 * u < p.M && ns < p.N) gemm_store8(p, m0 + c0 + tk + 8 * u, ns, va[u], vb[u], 1, 0, pre, rr[u]);
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                             // neither CTA leaves before the copying warps of both are through
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, kCols);
  }
}

struct PairPlan {
  int whole, cut, slices, kb_per_split;
  float rounds;                      // rounds of whole tiles that the launch takes (cut tiles count as their longest slice)
};
// Cutting the tiles of the last round along k costs a round trip of partial results through L2: about as long as 40 stages (of
// 128 bytes of k) of an int8 tile of 128 tokens, 50 of a bf16 one of 256, 64 of a bf16 one of 128, whose stages are shorter.  So it has
// to save 66 stages of that round, where each of the three gains.  N = 5120, us uncut / cut: int8 at 128 tokens K = 6144 (saves 32)
// 21.0 / 22.9, 8192 (42) 25.7 / 24.8, 17408 (90) 46.6 / 35.2, at 1060 tokens K = 6144 (24) 49 / 51, 17408 (68) 132 / 125; bf16 at 128
// tokens K = 4096 (42) 19.5 / 21.8, 6144 (64) 25.5 / 25.1, 17408 (181) 57.9 / 44.1, at 1060 tokens K = 6144 (48) 63.6 / 64.8, 8192 (64)
// 83.2 / 80.6.  Tiles of 32 and 64 tokens carry a quarter or half of the partial results through L2 and are bound by the weights'
// arrival, which a cut shares among more SMs: 30 stages.  int8 5120 x 6144 (saves 32) at 32 / 64 tokens 14.4 / 13.8, 15.4 / 17.0, 4096 x
// 8192 (48) 17.5 / 14.7, 18.7 / 18.2, 5120 x 17408 (90) 32.6 / 22.4, 33.9 / 27.0: tiles of 64 gain from about 40 on.
static PairPlan pair_plan(int M, int n_tiles, int KS, int NT, bool may_cut) {
  PairPlan q;
  const int tiles = (n_tiles * 8 + 255) / 256 * ((M + NT - 1) / NT);
  q.cut = tiles % kPairs;
  q.slices = q.cut == 0 || !may_cut ? 1 : std::max(1, std::min(std::min(kPairs / q.cut, KS / 16), 8));
  q.kb_per_split = (KS + q.slices - 1) / q.slices;
  q.slices = (KS + q.kb_per_split - 1) / q.kb_per_split;       // no empty slice
  if (KS - q.kb_per_split < (NT <= 64 ? 30 : 66)) q.slices = 1;
  if (q.slices == 1) q.cut = 0;
  q.whole = tiles - q.cut;
  q.rounds = (q.whole + kPairs - 1) / kPairs + (q.cut ? (float)q.kb_per_split / KS : 0.f);
  return q;
}
// workspace for every unit of one round of cut tiles, and a counter for each half of a cut tile
static bool pair_may_cut(const void* part, size_t part_bytes, const void* tile_count, int n_count) {
  return part != nullptr && tile_count != nullptr && part_bytes >= (size_t)kPairs * 256 * 256 * 4 && n_count >= kPairs;
}
// Tokens of a pair's tile.
//   * Batched decode: as few as hold the batch.
//   * bf16 products of many tokens: tiles of 128 tokens cost 0.62 of those of 256 (34816 x 5120 at 4096 tokens: 1143 us against 917), but
//     may leave fewer pairs idle in the last round.
//   * A few hundred tokens of few weight tiles: 64, where that gives more pairs work in the one round there is: a tile of 64 takes about 0.7
//     of one of 128.  us with the larger tiles / 64, int8: 5120 x 6144 at 65 / 128 / 192 tokens 19.4 / 15.4, 21.4 / 16.3, 21.9 / 16.7, 2048 x 6144 at
//     128 / 512 20.8 / 14.6, 21.3 / 16.9, 6176 x 2048 at 128 12.2 / 9.7; bf16: 5120 x 6144 at 128 24.7 / 22.8, 2048 x 6144 at 512 33.3 / 23.3.  Not where tiles
//     of 128 would be cut along k instead, nor long products where those of 256 would: their partial results cost about 103 stages, a
//     stage of a tile of 64 0.8 of theirs, since the weights' arrival bounds both (bf16, 256 cut / 64: 5120 x 17408 at 129 / 192 tokens 49.2 / 53.4,
//     53.8 / 55.3, 5120 x 14336 43.7 / 45.1, 48.0 / 46.3, 5120 x 10240 36.5 / 34.1, 40.7 / 34.7, 2048 x 8192 at 129 / 256 30.0 / 19.9, 43.5 / 22.7).
static int pair_tokens(bool bf16, int M, int n_tiles, int KS, bool may_cut) {
  if (M <= 64) return M <= 32 ? 32 : 64;
  const PairPlan q128 = pair_plan(M, n_tiles, KS, 128, may_cut), q256 = pair_plan(M, n_tiles, KS, 256, may_cut);
  const bool wide = bf16 && M > 128 && 0.62f * q128.rounds >= q256.rounds;
  const int tn = (n_tiles * 8 + 255) / 256, t64 = tn * ((M + 63) / 64);
  const bool cut = wide ? q256.slices > 1 && 0.8f * KS >= q256.kb_per_split + 103 : q128.slices > 1;
  if (t64 <= kPairs && t64 > tn * ((M + 127) / 128) && !cut) return 64;
  return wide ? 256 : 128;
}
// Products with tiles enough for every SM without a k split.
static bool pair_many(int M, int n_tiles) { return (n_tiles * 8 + 255) / 256 * ((M + 127) / 128) >= 120; }
// Which products the pairs take.  Not
//   * short ones, unless they have many tiles: the launch of a pair and its first ring fill take about 4 us longer (8192 x 512 at 70
//     tokens 11.1 us on one CTA per tile against 14.5, at 250 15.8 / 15.3, at 512 28.8 -> 16.8; with many tiles, 30976 x 320 at 8 / 64 /
//     128 / 1024 tokens int8 6.3 -> 6.6, 11.0 -> 9.4, 19.7 -> 13.3, 115 -> 71, bf16 at 16 / 64 / 128 / 1024 6.9 -> 7.7, 10.9 -> 9.3, 18.2 -> 12.1,
//     69 -> 51);
//   * a single tile of weight rows (routers), which would leave half of each pair idle;
//   * bf16 products of up to 8 tokens, where weights alone are streamed, twice as many bytes as in int8 (5120 x 17408 at 4 tokens 33.3
//     us against 35.7, a step of 3 decodes 757 / 763; at 14 decodes 841 -> 827, at 32 934 -> 908).
// One tile per CTA -> pairs, us, on N x K: 34816 x 5120 at 64 / 128 / 1060 / 4096 tokens int8 37.8 -> 34.0, 56 -> 39, 327 -> 239,
// 1085 -> 810, bf16 61 -> 61, 70 -> 62, 379 -> 298, 1238 -> 917; 5120 x 17408 at 64 tokens int8 28.2 -> 24.9, bf16 43.2 -> 40.9;
// 5120 x 6144 int8 18.9 -> 16.1, 30 -> 27, 95 -> 60, 366 -> 186; 2048 x 2048 at 64 / 128 / 1060 tokens int8 12.2 -> 9.6, 18 -> 13, 19 -> 15.
// At 4 tokens an int8 product alone gains nothing (18.5 -> 17.7, 10.6 -> 11.3, 8.9 -> 9.8), nor does a bf16 one at 12 to 24 (12288 x
// 2048 12.3 -> 13.8, 4096 x 4096 11.8 -> 12.8); a decode step does, since the next product's weights are requested earlier: 2 decodes
// of the 27B layers 551 -> 515 us, 5 599 -> 557, 12 652 -> 591, 64 1038 -> 976.  The other four families' steps of 2 to 64 decodes (widths 2048
// and 4096) with this rule against one tile per CTA: int8 0.6 to 10.2 % faster, bf16 at 12 and more between 1.0 %
// slower (one step, within what runs differ by) and 11.6 % faster.
static bool pair_serves(bool bf16, int M, int n_tiles, int N, int KS) {
  return N > 128 && !(bf16 && M <= 8) && (KS >= 16 || M > 256 || pair_many(M, n_tiles));
}

static void pair_apply(GemmParams& p, const PairPlan& q, int n_tiles, int NT, void* part, void* tile_count) {
  p.tiles_n = (n_tiles * 8 + 255) / 256;
  p.group_m = 2048 / NT;             // 2048 tokens by 74 / group_m weight tiles in flight (down at 4096 tokens, int8: 453 us; all 4096: 469)
  p.whole = q.whole;
  p.cut = q.cut;
  p.slices = q.slices;
  p.kb_per_split = q.kb_per_split;
  p.part = (float*)part;
  p.tile_count = (unsigned*)tile_count;
}

template <int NT, bool BF16>
static int launch_pair(const GemmParams& p, cudaStream_t st) {
  static bool configured = false;
  auto k = gemm_pair_kernel<NT, BF16>;
  if (!configured) {
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PairGeom<NT, BF16>::kSmem);
    configured = true;
  }
  const cudaError_t e = launch_kernel(k, dim3(2 * std::min(kPairs, p.whole + p.cut * p.slices)), dim3(kPairThreads), PairGeom<NT, BF16>::kSmem, st, true, p);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

}  // namespace ti
