// The swap-AB GEMM for many rows (prompts): a pair of SMs works on one tile of 256 features x up to 256 tokens with tcgen05.mma.cta_group::2.
//
// What bounds it: at 128 x 256 per SM the operands of a k-block (48 KB) cross from L2 to the SM in the time of its products only at ~96 B / clk / SM,
// more than the SM takes in, and the tensor pipe idles a third of the time.  In a pair each SM holds its own 128 weight rows and HALF of the token
// tile, and the products read the other half from the neighbour's shared memory: 32 KB per k-block (64 B / clk), or 48 KB per two products for the
// gate / up form (48 B / clk).  Beside that
//   * tiles are walked in groups of 8 token tiles, token tile fastest, so the ~74 tiles in flight share ~17 operand panels instead of re-reading
//     the whole weight per token tile (235 MB per token tile for the gate / up weights of Llama-3-8B);
//   * grouped (mixture-of-experts) launches walk the tiles that exist (a prefix sum over the experts' tile counts), not the tiles that could;
//   * the N extent of the products is that of the tile's rows (multiples of 32): ragged last tiles and small experts cost what they hold;
//   * 8 epilogue warps; features lie along the lanes, so rows leave the registers as 64-byte (bf16, two rows per store) or 128-byte (fp32) runs: no
//     staging in shared memory, no barrier; the residual is added in fp32 before the only rounding.
// Roles (384 threads per CTA): warp 0 TMA, warp 1 MMA (leader CTA) + TMEM, warps 4..11 epilogue.
// B200, whole blocks, one-SM tiles -> pairs: Llama-3-8B feed-forward on 8 k tokens (power-capped) 2804 -> 2432 us, its attention on 4 k tokens 533 -> 461 us,
// DeepSeek-V2-Lite attention on 64 x ~128 tokens 382 -> 333 us, Gemma-2-9B attention on 2 k tokens 273 -> 248 us.  A launch costs ~4 us more than one of the
// one-SM kernel, and the gate / up epilogue is exposed (one accumulator set of 512 columns): pair_pays below.  Up to 256 rows the one-SM kernel is as
// good (it streams the weight once either way), and results that go to peer memory (stage hand-off, expert-parallel return) stay with it.
#include <algorithm>

#include "gemm_cluster.cuh"
#include "gemm_tmap.h"
#include "launch.h"

namespace b200 {

using namespace gemm;

namespace {

constexpr int kPairThreads = 384;
constexpr int kPairTok = 256;                  // tokens of a tile
constexpr int kPairFeat = 2 * kTileM;          // features of a tile
constexpr int kPairGroup = 8;                  // token tiles that are walked together
constexpr int kPairMaxExperts = 256;
constexpr int kXHalfBytes = (kPairTok / 2) * kBlockK * 2;

__host__ __device__ constexpr int pair_stage_bytes(bool dual) { return kATileBytes * (dual ? 2 : 1) + kXHalfBytes; }
__host__ __device__ constexpr int pair_stages(bool dual) { return dual ? 4 : 6; }
__host__ __device__ constexpr int pair_smem(bool dual) { return pair_stages(dual) * pair_stage_bytes(dual) + 1024 + 256 + 2 * (kPairMaxExperts + 1) * 4; }

B200_DEVICE void pair_tma(uint32_t dst, const CUtensorMap* m, uint32_t leader_bar, int c0, int c1, uint64_t hint) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4}], [%2], %5;" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(leader_bar), "r"(c0), "r"(c1), "l"(hint)
      : "memory");
}
B200_DEVICE void pair_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b),
               "r"(idesc), "r"(accumulate)
               : "memory");
}
// arrives on the barrier at this offset in both CTAs once all products issued so far have completed
B200_DEVICE void pair_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "h"(static_cast<uint16_t>(3))
               : "memory");
}
B200_DEVICE void pair_remote_arrive(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

struct PairTile {
  int n0, w_row, row_base, rows;
};

// tile t of the walk (the same for every role of both CTAs)
__device__ __forceinline__ PairTile pair_tile(const GemmParams& p, const int* s_cum, const int* s_off, int num_experts, int t, int tiles_n, int tiles_m) {
  PairTile ti;
  if (num_experts > 0) {
    int lo = 0, hi = num_experts;              // s_cum[lo] <= t < s_cum[hi]
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (s_cum[mid] <= t) lo = mid; else hi = mid;
    }
    const int r = t - s_cum[lo], mt = r / tiles_n;
    ti.n0 = (r % tiles_n) * kPairFeat;
    ti.row_base = s_off[lo] + mt * kPairTok;
    ti.rows = s_off[lo + 1] - ti.row_base;
    ti.w_row = lo * p.n + ti.n0;
  } else {
    const int span = kPairGroup * tiles_n, g = t / span, m0 = g * kPairGroup, gm = min(kPairGroup, tiles_m - m0), r = t - g * span;
    ti.n0 = (r / gm) * kPairFeat;
    ti.row_base = (m0 + r % gm) * kPairTok;
    ti.rows = p.m - ti.row_base;
    ti.w_row = ti.n0;
  }
  if (ti.rows > kPairTok) ti.rows = kPairTok;
  return ti;
}
__device__ __forceinline__ int pair_cols(int rows) { return (rows + 31) & ~31; }      // N extent of the products

}  // namespace

template <bool DUAL, typename OutT>
__global__ void __launch_bounds__(kPairThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_w2, const __grid_constant__ CUtensorMap tmap_x,
                 const GemmParams p, const int tiles_n, const int tiles_m, const int num_experts, const WaitBound bound) {
  constexpr int ST = pair_stages(DUAL), STAGE = pair_stage_bytes(DUAL), NUM_ACC = DUAL ? 1 : 2;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + ST * STAGE);      // leader's: both CTAs' copies
  uint64_t* empty_bar = full_bar + ST;                                      // each CTA's own
  uint64_t* tfull_bar = empty_bar + ST;                                     // [2], each CTA's own
  uint64_t* tempty_bar = tfull_bar + 2;                                     // [2], leader's: the epilogue warps of both CTAs
  uint32_t* tmem_base_smem = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  uint32_t* dead = tmem_base_smem + 1;
  int* s_cum = reinterpret_cast<int*>(smem + ST * STAGE + 256);             // [E + 1] tiles of the experts in front
  int* s_off = s_cum + kPairMaxExperts + 1;                                 // [E + 1] first rows

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int cid = blockIdx.x >> 1, ncl = gridDim.x >> 1;
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_x);
    if (DUAL) tma_prefetch_desc(&tmap_w2);
    *dead = 0u;
    for (int s = 0; s < ST; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&tfull_bar[a], 1); mbar_init(&tempty_bar[a], 16); }
    mbar_fence_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_base_smem)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  pdl_launch_dependents();
  pdl_wait();
  if (num_experts > 0 && warp == 2) {                                       // prefix sum of the experts' tile counts
    int base = 0;
    for (int e0 = 0; e0 < num_experts; e0 += 32) {
      const int e = e0 + lane;
      const int lo = e < num_experts ? __ldcg(p.expert_offsets + e) : 0, hi = e < num_experts ? __ldcg(p.expert_offsets + e + 1) : 0;
      int incl = (hi - lo + kPairTok - 1) / kPairTok * tiles_n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
      }
      if (e < num_experts) { s_cum[e + 1] = base + incl; s_off[e] = lo; s_off[e + 1] = hi; }
      base += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) s_cum[0] = 0;
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                                       // both CTAs' barriers and TMEM exist
  tc_fence_after();
  const uint32_t tmem_base = *tmem_base_smem;
  const int total = num_experts > 0 ? s_cum[num_experts] : tiles_n * tiles_m;
  const int kb_total = (p.k + kBlockK - 1) / kBlockK;
  // A CTA whose wait gives up signals nothing more; its neighbour's waits then run out by themselves, and both meet at the end.
  auto wait = [&](uint64_t* bar, uint32_t parity) { return mbar_wait_bounded(bar, parity, dead, bound.spins); };
  bool alive = true;

  if (warp == 0) {
    // ============================================================== TMA producer: own weight rows, own half of the tokens
    if (elect_one()) {
      uint32_t it = 0;
      for (int t = cid; alive && t < total; t += ncl) {
        const PairTile ti = pair_tile(p, s_cum, s_off, num_experts, t, tiles_n, tiles_m);
        const int x_row = ti.row_base + (int)rank * (pair_cols(ti.rows) >> 1), w_row = ti.w_row + (int)rank * kTileM;
        for (int kb = 0; kb < kb_total; ++kb, ++it) {
          const uint32_t s = it % ST, ph = (it / ST) & 1;
          alive = wait(&empty_bar[s], ph ^ 1);
          if (!alive) break;
          if (rank == 0) mbar_arrive_expect_tx(&full_bar[s], 2 * STAGE);
          const uint32_t st = smem_u32(smem + s * STAGE), bar = mapa_shared(smem_u32(&full_bar[s]), 0);
          const int kc = kb * kBlockK;
          pair_tma(st, &tmap_w, bar, kc, w_row, kEvictNormal);
          if (DUAL) pair_tma(st + kATileBytes, &tmap_w2, bar, kc, w_row, kEvictNormal);
          pair_tma(st + kATileBytes * (DUAL ? 2 : 1), &tmap_x, bar, kc, x_row, kEvictNormal);
        }
      }
      // the leader's commits to this CTA's barriers have all arrived before the CTA may go
      for (int i = 0; alive && i < ST; ++i, ++it) alive = wait(&empty_bar[it % ST], ((it / ST) & 1) ^ 1);
    }
  } else if (warp == 1) {
    // ============================================================== MMA issuer of the pair
    if (rank == 0 && elect_one()) {
      uint32_t it = 0, tc = 0;
      for (int t = cid; alive && t < total; t += ncl, ++tc) {
        const PairTile ti = pair_tile(p, s_cum, s_off, num_experts, t, tiles_n, tiles_m);
        const uint32_t idesc = umma_idesc_bf16(2 * kTileM, (uint32_t)pair_cols(ti.rows));
        const uint32_t ab = tc % NUM_ACC, aph = (tc / NUM_ACC) & 1;
        alive = wait(&tempty_bar[ab], aph ^ 1);
        tc_fence_after();
        const uint32_t acc = tmem_base + ab * kPairTok;
        for (int kb = 0; alive && kb < kb_total; ++kb, ++it) {
          const uint32_t s = it % ST, ph = (it / ST) & 1;
          alive = wait(&full_bar[s], ph);
          if (!alive) break;
          tc_fence_after();
          const uint32_t a0 = smem_u32(smem + s * STAGE);
          const uint64_t ad = umma_desc_sw128(a0), ad2 = umma_desc_sw128(a0 + kATileBytes), bd = umma_desc_sw128(a0 + kATileBytes * (DUAL ? 2 : 1));
#pragma unroll
          for (int kk = 0; kk < kBlockK / kUmmaK; ++kk) {
            pair_mma(acc, ad + 2 * kk, bd + 2 * kk, idesc, (kb | kk) ? 1u : 0u);
            if (DUAL) pair_mma(acc + kPairTok, ad2 + 2 * kk, bd + 2 * kk, idesc, (kb | kk) ? 1u : 0u);
          }
          pair_commit(&empty_bar[s]);
        }
        if (alive) pair_commit(&tfull_bar[ab]);
      }
    }
  } else if (warp >= 4) {
    // ============================================================== epilogue: lane = feature, columns = tokens
    const int q = warp & 3, half = (warp - 4) >> 2;
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    uint32_t tc = 0;
    for (int t = cid; t < total; t += ncl, ++tc) {
      const PairTile ti = pair_tile(p, s_cum, s_off, num_experts, t, tiles_n, tiles_m);
      const uint32_t ab = tc % NUM_ACC, aph = (tc / NUM_ACC) & 1;
      const int f = ti.n0 + (int)rank * kTileM + q * 32 + lane;
      const bool f_ok = f < p.n;
      const float bias = (p.bias != nullptr && f_ok) ? __bfloat162float(p.bias[f]) : 0.0f;
      if (!__all_sync(0xffffffffu, wait(&tfull_bar[ab], aph))) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + lane_addr + ab * kPairTok;
#pragma unroll 1
      for (int c = half * 32; c < ti.rows; c += 64) {
        uint32_t v[32], u[DUAL ? 32 : 1];
        tmem_ld32(taddr + c, v);
        if constexpr (DUAL) tmem_ld32(taddr + kPairTok + c, u);
        const int row0 = ti.row_base + c, left = ti.rows - c;
        if constexpr (sizeof(OutT) == 2) {
          // two rows at a time: the even lane takes row 2j, its odd neighbour row 2j + 1, each with both lanes' features
          uint32_t res[16];
          const __nv_bfloat16* rp = p.residual == nullptr ? nullptr : p.residual + (size_t)(row0 + (lane & 1)) * p.ld_res + (f & ~1);
#pragma unroll
          for (int j = 0; j < 16; ++j)
            res[j] = rp != nullptr && f_ok && 2 * j + (lane & 1) < left ? *reinterpret_cast<const uint32_t*>(rp + (size_t)(2 * j) * p.ld_res) : 0u;
          tmem_ld_wait();
          __nv_bfloat16* op = reinterpret_cast<__nv_bfloat16*>(p.out) + (size_t)(row0 + (lane & 1)) * p.ld_out + (f & ~1);
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            float y[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              float g = __uint_as_float(v[2 * j + e]) + bias;
              if constexpr (DUAL) g = gated_act(p.act, p.act_limit, g, __uint_as_float(u[2 * j + e]));
              else if (p.act == kActRelu2) { g = fmaxf(g, 0.f); g *= g; }
              if (p.softcap > 0.f) g = p.softcap * tanhf(g / p.softcap);
              y[e] = g;
            }
            const bool odd = lane & 1;
            const float got = __shfl_xor_sync(0xffffffffu, odd ? y[0] : y[1], 1);
            const float lo = (odd ? got : y[0]) + bf16_lo(res[j]), hi = (odd ? y[1] : got) + bf16_hi(res[j]);
            if (f_ok && 2 * j + (lane & 1) < left) *reinterpret_cast<uint32_t*>(op + (size_t)(2 * j) * p.ld_out) = pack_bf16(lo, hi);
          }
        } else {
          tmem_ld_wait();
          float* op = reinterpret_cast<float*>(p.out) + (size_t)row0 * p.ld_out + f;
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            float y = __uint_as_float(v[j]) + bias;
            if (p.act == kActRelu2) { y = fmaxf(y, 0.f); y *= y; }
            if (p.softcap > 0.f) y = p.softcap * tanhf(y / p.softcap);
            if (f_ok && j < left) {
              if (p.residual != nullptr) y += __bfloat162float(p.residual[(size_t)(row0 + j) * p.ld_res + f]);
              op[(size_t)j * p.ld_out] = y;
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) pair_remote_arrive(mapa_shared(smem_u32(&tempty_bar[ab]), 0));
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (*reinterpret_cast<volatile uint32_t*>(dead) != 0u) report_dead(bound, kWaitPairGemm);
  cluster_sync_all();                                                       // nobody reads or signals this CTA any more
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
  }
}

namespace {

template <bool DUAL, typename OutT>
cudaError_t pair_launch_one(const CUtensorMap& tw, const CUtensorMap& tw2, const CUtensorMap& tx, const GemmParams& p, int tiles_n, int tiles_m, int experts,
                            long long tiles, const WaitBound& wait, cudaStream_t stream) {
  constexpr int smem = pair_smem(DUAL);
  static_assert(smem <= 227 * 1024, "shared memory budget exceeded");
  auto kern = gemm_pair_kernel<DUAL, OutT>;
  static int fit = 0;                          // pairs that run at once (a GPC with an odd number of SMs leaves one out)
  if (fit == 0) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(2); cfg.blockDim = dim3(kPairThreads); cfg.dynamicSmemBytes = smem; cfg.attrs = at; cfg.numAttrs = 1;
    int n = 0;
    e = cudaOccupancyMaxActiveClusters(&n, kern, &cfg);
    if (e != cudaSuccess) return e;
    fit = n > 0 ? n : 1;
  }
  const int clusters = static_cast<int>(std::min<long long>(tiles, fit));
  (void)launch_pdl_cluster(kern, dim3(2 * clusters), dim3(kPairThreads), smem, stream, dim3(2), tw, tw2, tx, p, tiles_n, tiles_m, experts, wait);
  return cudaGetLastError();
}

}  // namespace

// Where pairs are faster.  Both kernels walk their tiles in rounds of the chip; times from products with both kernels in turn in one process, weights from HBM,
// 257 to 8192 rows, us, single SMs / pairs, kb = k-blocks of 64:
//   bf16:        single SMs 2.6 + rounds (2.5 + 0.355 kb), pairs 6.7 + rounds (0.95 + 0.327 kb), at least 6.5 a round (the epilogue); the single SMs' partly filled
//                last token tile costs in proportion.  3648 x 2048: 1024 rows 17.3 / 19.2, 4096 rows 53 / 49; 4096 x 512: 8192 rows 43 / 52; 6144 x 4096: 512 rows 31 / 33,
//                2048 rows 81 / 72; 10944 x 2048: 384 rows 27 / 29, 8192 rows 312 / 245.  Below a gain of 3 % the smaller launch stays.
//   + residual:  pairs (with one, single SMs take 6 us more a round): 256 x 2048 21 / 18, 2048 x 2048 at 257 rows 23 / 19, 8192 rows 112 / 56
//   fp32:        pairs' last epilogue is exposed: single SMs 1 + rounds (2.5 + 0.38 kb), pairs 14 + rounds (3 + 0.31 kb).  4096 x 2048: 1024 rows 21 / 29, 8192 rows
//                118 / 115; 2048 x 4096: 2048 rows 28 / 35, 8192 rows 115 / 105
//   gate and up: 256 x 256 of both weights fill TMEM, so every epilogue is exposed (8 us a round more); worth it only where single SMs read weights that L2
//                (126 MB) does not keep again for every token tile.  10944 x 2048 (90 MB): 257 rows 51 / 70, 2048 rows 157 / 177, 8192 rows 632 / 646; 4096 x 4096: 1024 rows
//                56 / 63, 8192 rows 386 / 407; 14336 x 4096 (235 MB): 512 rows 108 / 114, 513 rows 147 / 138, 1024 rows 216 / 213, 2048 rows 412 / 378, 4096 rows 799 / 738
// Experts (E of them, r rows each on average): a pair's products are as wide as the rows that a tile holds and its list holds the tiles that exist; single SMs' are 256
// wide and their list holds every tile that could exist, so theirs is the less even one where tiles are few or many.
//   gate and up: kb >= 56 pairs (8 x 14336 x 4096: r 128 435 / 366, r 1024 1843 / 1728; 16 x 4096 x 4096: r 200 375 / 249), kb < 24 not (32 x 2048 x 1024: r 200 82 / 108).
//                Between, with kb = 32: E 8 r 150 79 / 39, r 325 85 / 74, r 400 64 / 78, r 512 89 / 106, r 2048 244 / 276; E 32 r 128 61 / 68, r 512 175 / 173; E 64 r 96
//                171 / 161, r 384 386 / 344, r 562 519 / 554 (1408 x 2048), two of 66 with all rows: r 248 260 / 246, r 496 468 / 423, r 727 655 / 699
//   down (fp32): kb >= 48 pairs (8 x 4096 x 14336: r 256 374 / 275), kb < 20 not (32 x 2048 x 1024: r 200 45 / 60; 64 x 2048 x 768: r 256 96 / 129).  Between: E 8 x 2048 x 2048
//                r 150 42 / 26, r 400 36 / 41, r 750 73 / 55; E 32 x 1024 x 2048 r 200 39 / 46, r 375 73 / 66; E 64 x 2048 x 1408 r 96 96 / 76, r 768 369 / 330
static bool pair_pays(const GemmArgs& a) {
  auto up = [](long long x, long long y) { return (x + y - 1) / y; };
  const int kb = static_cast<int>(up(a.k, kBlockK));
  if (a.expert_offsets != nullptr) {
    const double r = static_cast<double>(a.m) / a.num_experts;
    const int few = 16, many = 48;
    if (a.w2 != nullptr) {
      if (kb >= 56 || kb < 24) return kb >= 56;
      return a.num_experts <= few ? r <= 340 : a.num_experts >= many && r <= 512;
    }
    if (kb >= 48 || kb < 20) return kb >= 48;
    return a.num_experts >= many || (a.num_experts <= few ? r <= 340 || r >= 700 : r >= 350);
  }
  if (a.w2 != nullptr) return 4ll * a.n * a.k > (126ll << 20) && a.m > 512;
  if (a.residual != nullptr) return true;
  constexpr int kSms = 148;                                                                      // of the measured chip: rounds
  const double pairs = static_cast<double>(up(up(a.n, kPairFeat) * up(a.m, kPairTok), kSms / 2));
  const double ones = static_cast<double>(up(up(a.n, kTileM) * a.m, static_cast<long long>(kPairTok) * kSms));
  if (a.out_fp32) return 14 + pairs * (3 + 0.31 * kb) < 0.97 * (1 + ones * (2.5 + 0.38 * kb));
  return 6.7 + pairs * std::max(6.5, 0.95 + 0.327 * kb) < 0.97 * (2.6 + ones * (2.5 + 0.355 * kb));
}

bool gemm_pair_takes(const GemmArgs& a) {
  const bool grouped = a.expert_offsets != nullptr;
  if (a.signal_flag != nullptr || a.signal_peers != nullptr || a.row_dst != nullptr || a.ep_arrive != nullptr) return false;
  if (grouped ? (a.expert_stride > 0 || a.num_experts > kPairMaxExperts || a.bn != kPairTok) : a.m <= kPairTok) return false;
  if (a.n <= kTileM || (reinterpret_cast<uintptr_t>(a.out) & 3) != 0 || (reinterpret_cast<uintptr_t>(a.residual) & 3) != 0) return false;
  if (a.pair == 0 || (a.pair < 0 && !pair_pays(a))) return false;
  return (a.k % 8) == 0 && (a.n % 8) == 0 && (a.ld_out % 2) == 0 && (a.residual == nullptr || (a.ld_res % 2) == 0) && !(a.w2 != nullptr && a.out_fp32);
}

cudaError_t gemm_pair_launch(const GemmArgs& a, cudaStream_t stream) {
  const bool dual = a.w2 != nullptr, grouped = a.expert_offsets != nullptr;
  CUtensorMap tw, tw2, tx;
  const uint64_t w_rows = static_cast<uint64_t>(a.n) * (grouped ? a.num_experts : 1);
  if (!gemm_make_tmap(&tw, a.w, w_rows, a.k, a.ld_w, kTileM)) return cudaErrorUnknown;
  tw2 = tw;
  if (dual && !gemm_make_tmap(&tw2, a.w2, w_rows, a.k, a.ld_w, kTileM)) return cudaErrorUnknown;
  if (!gemm_make_tmap(&tx, a.x, a.x_rows, a.k, a.ld_x, kPairTok / 2)) return cudaErrorUnknown;
  GemmParams p = {};
  p.m = a.m; p.n = a.n; p.k = a.k; p.splits = 1;
  p.expert_offsets = a.expert_offsets;
  p.out = a.out; p.ld_out = a.ld_out;
  p.residual = static_cast<const __nv_bfloat16*>(a.residual); p.ld_res = a.ld_res;
  p.bias = static_cast<const __nv_bfloat16*>(a.bias); p.act = a.act; p.act_limit = a.act_limit; p.softcap = a.softcap;
  const int tiles_n = (a.n + kPairFeat - 1) / kPairFeat, tiles_m = (a.max_rows + kPairTok - 1) / kPairTok;
  const long long most = static_cast<long long>(tiles_n) * tiles_m * (grouped ? a.num_experts : 1);
  const int experts = grouped ? a.num_experts : 0;
  if (a.out_fp32) return pair_launch_one<false, float>(tw, tw2, tx, p, tiles_n, tiles_m, experts, most, a.wait, stream);
  if (dual) return pair_launch_one<true, __nv_bfloat16>(tw, tw2, tx, p, tiles_n, tiles_m, experts, most, a.wait, stream);
  return pair_launch_one<false, __nv_bfloat16>(tw, tw2, tx, p, tiles_n, tiles_m, experts, most, a.wait, stream);
}

}  // namespace b200
