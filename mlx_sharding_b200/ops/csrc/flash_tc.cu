// Causal flash attention of prompts and portions of prompts on tcgen05 / TMEM, against the paged cache (ragged batches, any context in front).
//
// The reference materialises a dense additive [T, T] mask and calls mx.fast.scaled_dot_product_attention on a contiguous cache
// (shard/server/model/llama.py:48-59, gemma2.py:47-58, deepseek_v2.py:47-57).
//
// What bounds it: 4 * d flops per (query, visible key, head) against one exponential; the warp-level mma.sync form of this kernel reached 160
// TFLOP/s on 2 x 2 k tokens of Llama-3-8B.  Here
//   * a CTA owns up to 256 query rows of one kv head as two *streams* of 128 (two query heads of a group on the same rows, or two row tiles of
//     one head): every K / V tile that TMA brings feeds both, which halves the L2 traffic (a stream alone would ask for ~46 B / clk / SM);
//   * tiles of 64 keys = one page: S = Q K^T [128 x 64] (operands in shared memory), P V with P read from TMEM and V as an MN-major operand
//     straight from its page: no transposition, no copy of P through shared memory;
//   * CTAs are persistent: a CTA that came and went per 256 rows spent ~9 us on its set-up, first loads and drain (75 us for 64 prompts of 128 tokens).
//     The grid holds a CTA per (row tile, head) item, a sequence's longest first, and a running CTA that is done takes the next one that has not
//     started out of the launch queue (clusterlaunchcontrol): one resident CTA per SM, dynamic balance, no counter in memory.  Rings, score buffers
//     and barriers run on across items, so the next item's queries, keys and first scores arrive while the last one is normalised and stored;
//   * S is double buffered, the scores of each stream and the second products have an issuing thread of their own (issuing, not the tensor pipe, was
//     what one thread for all was bound by: ~100 cycles per product), so scores run a tile ahead of the softmax warps; P overwrites its own score buffer.  A buffer is written again only after the product that reads
//     it has completed (its commit is waited for);
//   * one thread per row: no shuffles; the accumulator in TMEM is rescaled when a row of the warp has a new maximum, after the tile's
//     exponentials, so that the last product has had their time to complete (rescaled before them: 1 x 8 k tokens 579 us, here 549);
//   * capped scores, heads of 256 and SINK (fp32 probabilities, or queries, before): probabilities enter the second product as two bf16 terms (error 2^-17 of
//     each; a visible infinity in V gives NaN, as the low term may be 0 or of the other sign), and the maximum may lag by 2^8 before a rescale.  The plain modes
//     have one term, and with it the exact maximum, as the mma.sync form: the dominant probability is then 1 and rounds to itself, which the lag would
//     lose.  Error of the op against 64 bits at scores with a spread of 2: mma.sync form 1.838e-3, one term and the lag 2.104e-3, one term and the exact maximum
//     1.838e-3, two terms 1.647e-3 (the rounding of the result: 1.645e-3).  B200, whole blocks, lag / exact / two terms: Llama-3-8B 4 k tokens of prompts 428 / 442
//     / 450 us, DeepSeek-V2-Lite 2 k behind 6 k 297 / 299 / 340 us, 64 x ~128 312 / 307 / 318 us (the low terms cost tensor time and, under the power cap, clock);
//   * heads of 256 (Gemma-2): the accumulator takes 256 columns, so there is one stream, whose rows' 64 scores are shared by two threads, and
//     three score buffers;
//   * MLA: the decompressed keys / values are read where the kv_b product left them ([rows, heads * (nope + v)]), the shared rotary key from
//     the latent pool's pages: no per-head K / V pool is assembled.
//   * SINK (windowed attention of the hybrid stacks, sinkattn.cu): only tiles with visible keys are walked; the fp32 queries enter the first product
//     as two bf16 terms (the softmax warps lay them out in shared memory), a sink joins the denominator, gates multiply the result.
// Rows of V behind the last key are zeroed in shared memory (what lies there may be anything, and 0 * inf is not 0).
// B200, the kernel alone, one CTA per item with one issuing thread and a lagging maximum -> this form: Llama-3-8B heads, 1 x 8 k tokens 753 -> 549 us
// (1002 TFLOP/s), 2 x 2 k 145 -> 122 us, 64 x 128 75 -> 54 us; DeepSeek-V2-Lite 2 k behind 6 k 213 -> 166 us; windowed
// attention with a sink (mma.sync form before), 4 k tokens of 16 heads, window 1024, 241 -> 89 us.  Before that, the mma.sync form: 1 x 8 k tokens 2869 us, 2 x 2 k
// 439 us, the portion 864 us; capped scores ran on the decode kernel (2 x 1 k tokens of Gemma-2-9B 1814 us, here 52 us).
#include <cuda.h>

#include "gemm_tmap.h"
#include "kernels.h"
#include "launch.h"
#include "ptx.cuh"
#include "sinkattn.h"

namespace b200 {

namespace {

constexpr int kRows = 128;                    // query rows of a stream (UMMA M)
constexpr int kKeys = 64;                     // keys of a tile
constexpr int kFlashThreads = 384;            // warps 0..7: softmax, 8: TMA + item list, 9 / 10: S of a stream (9: TMEM too), 11: P V
constexpr int kSlots = 4;                     // items that the producer may be ahead
constexpr float kLazy = 8.f;                  // how far (log2) the maximum may lag where probabilities are two terms

constexpr int kMaxSeqs = 512;                 // sequences of a step that the item table holds

enum : int { kMla = 1, kCap = 2, kSink = 4 };

struct FlashTcParams {
  const int* block_tables; int max_blocks;
  const int* cu_seqlens; const int* context_lens;
  int num_seqs, q_heads, kv_heads, page, box_rows;
  long long lin_stride;                        // MLA: first row of a sequence in the linear keys / values (< 0: its first token's row)
  float scale, softcap;
  __nv_bfloat16* out; long long o_ld_t;
  // SINK
  const float* q32;                            // [T, q_heads, DK]
  const float* sink; const __nv_bfloat16* gate; long long ld_gate;
  int gate_elem, block, window, keep;
  float out_mult;
  WaitBound wait;
};

// probabilities in two terms and a maximum that may lag, or in one and the exact maximum
__host__ __device__ constexpr bool ft_split(int dv, int mode) { return dv > 128 || (mode & (kCap | kSink)) != 0; }
__host__ __device__ constexpr int ft_streams(int dv) { return dv > 128 ? 1 : 2; }
__host__ __device__ constexpr int ft_bufs(int dv) { return dv > 128 ? 3 : 2; }
__host__ __device__ constexpr int ft_stages(int dk, int dv, int mode) { return (mode & kSink) || dk + dv > 320 ? 2 : dk + dv > 256 ? 3 : 4; }
__host__ __device__ constexpr int ft_q_bytes(int dk, int mode) { return kRows * dk * 2 * ((mode & kSink) ? 2 : 1); }
__host__ __device__ constexpr int ft_smem(int dk, int dv, int mode) {
  return ft_streams(dv) * ft_q_bytes(dk, mode) + ft_stages(dk, dv, mode) * kKeys * (dk + dv) * 2 + 1024 + 1024 + 4 * kMaxSeqs * 3 + (dv > 128 ? 3 * 2 * kRows * 4 : 0);
}

__host__ __device__ constexpr uint32_t ft_idesc(uint32_t M, uint32_t N, uint32_t b_mn_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (b_mn_major << 16) | ((N >> 3) << 17) | ((M >> 4) << 24);
}
// A operand from TMEM (row = lane, two bf16 per 32-bit column), B from shared memory
B200_DEVICE void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
               ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
B200_DEVICE void ft_tma_2d(uint32_t dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0), "r"(c1) : "memory");
}
B200_DEVICE void tmem_st16(uint32_t taddr, const uint32_t* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr), "r"(v[0]),
      "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]),
      "r"(v[14]), "r"(v[15])
      : "memory");
}
// Takes a CTA that has not started out of this grid's launch queue; the answer (16 bytes) arrives on the barrier
B200_DEVICE void ft_try_cancel(uint4* answer, uint64_t* bar) {
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(smem_u32(answer)), "r"(smem_u32(bar))
               : "memory");
}
B200_DEVICE int ft_canceled_cta(const uint4* answer, int none) {               // blockIdx.x of the CTA, `none` where none was left
  uint32_t ok, x;
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b128 r;\n\t"
      "ld.shared.b128 r, [%2];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\n\t"
      "selp.u32 %0, 1, 0, p;\n\tmov.u32 %1, 0;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, r;\n\t}"
      : "=r"(ok), "=r"(x) : "r"(smem_u32(answer)) : "memory");
  return ok != 0u ? (int)x : none;
}

// What an item is: up to two streams of 128 rows on one kv head
struct FlashItem {
  int seq, tok_base, hk, n_max, nkept, w0;     // n_max < 0: the list ends
  int rows[2], pos[2], n[2], head[2], tok[2], end[2];
  __device__ __forceinline__ int tile(int j) const { return j < nkept ? j : w0 + j - nkept; }      // key tile of step j
};

__device__ __forceinline__ int ft_first_key(const FlashTcParams& p, int pos) {                     // SINK: the first window / block key of a query
  int lo = p.block > 0 ? pos / p.block * p.block : 0;
  if (p.window > 0) lo = max(lo, pos - p.window + 1);
  return lo;
}

template <int NS, int MODE>
__device__ __forceinline__ FlashItem ft_item(const FlashTcParams& p, const int* s_cum, const int* s_start, const int* s_ctx, int w, int total, int heads,
                                                 bool pair_heads) {
  FlashItem it = {};
  const int t = total - 1 - w / heads, y = w % heads;                        // a sequence's last rows see the most keys: they come first
  int lo = 0, hi = p.num_seqs - 1;
  while (lo < hi) {                                                          // the first sequence with more than t tiles up to it
    const int mid = (lo + hi) >> 1;
    if (s_cum[mid] > t) hi = mid; else lo = mid + 1;
  }
  it.seq = lo;
  it.tok_base = s_start[lo];
  const int span = NS == 2 && !pair_heads ? 2 * kRows : kRows, q0 = (t - (lo > 0 ? s_cum[lo - 1] : 0)) * span;
  const int qlen = s_start[lo + 1] - it.tok_base, ctx = s_ctx[lo];
  it.hk = (pair_heads ? 2 * y : y) / (p.q_heads / p.kv_heads);
  it.n_max = 0;
  it.nkept = 0;
  it.w0 = 0;
  if constexpr ((MODE & kSink) != 0) {
    const int first = ft_first_key(p, ctx - qlen + q0);
    it.nkept = (min(p.keep, first) + kKeys - 1) / kKeys;
    it.w0 = max(it.nkept, first / kKeys);
  }
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    const int r0 = q0 + (pair_heads ? 0 : s * kRows);
    it.rows[s] = max(0, min(kRows, qlen - r0));
    it.head[s] = pair_heads ? 2 * y + s : y;
    it.tok[s] = it.tok_base + r0;
    it.pos[s] = ctx - qlen + r0;
    it.end[s] = min(ctx, it.pos[s] + it.rows[s]);                            // causal: keys 0 .. the last row's position
    const int tiles = (it.end[s] + kKeys - 1) / kKeys;
    it.n[s] = it.rows[s] > 0 ? it.nkept + max(0, tiles - it.w0) : 0;
    it.n_max = max(it.n_max, it.n[s]);
  }
  if (NS == 1) it.end[1] = it.end[0];
  return it;
}

template <int DK, int DV, int MODE>
__global__ void __launch_bounds__(kFlashThreads, 1)
flash_tc_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                const __grid_constant__ CUtensorMap tmap_pe, const FlashTcParams p) {
  constexpr bool MLA = (MODE & kMla) != 0, CAP = (MODE & kCap) != 0, SINK = (MODE & kSink) != 0, SPLIT = ft_split(DV, MODE);
  constexpr int NS = ft_streams(DV), NB = ft_bufs(DV), ST = ft_stages(DK, DV, MODE);
  constexpr int CK = DK / 64, CV = DV / 64;
  constexpr int QB = ft_q_bytes(DK, MODE), KB = kKeys * DK * 2, VB = kKeys * DV * 2, CHUNK = kKeys * 128;
  constexpr uint32_t O_COL = NS * NB * 64;
  constexpr float LAG = SPLIT ? kLazy : 0.f;
  static_assert(O_COL + NS * DV <= 512, "TMEM budget exceeded");
  constexpr uint32_t IDESC_S = ft_idesc(kRows, kKeys, 0), IDESC_O = ft_idesc(kRows, DV, 1);
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* q_smem = smem;
  uint8_t* k_smem = q_smem + NS * QB;
  uint8_t* v_smem = k_smem + ST * KB;
  uint64_t* bars = reinterpret_cast<uint64_t*>(v_smem + ST * VB);
  uint64_t* q_full = bars;                    // [2]
  uint64_t* q_empty = bars + 2;               // [2]
  uint64_t* o_free = bars + 4;                // [2]
  uint64_t* k_full = bars + 6;                // [ST]
  uint64_t* k_empty = k_full + ST;
  uint64_t* v_full = k_empty + ST;
  uint64_t* v_empty = v_full + ST;
  uint64_t* s_full = v_empty + ST;            // [NS][NB]
  uint64_t* p_ready = s_full + NS * NB;       // [NS][NB]: softmax may be a tile ahead of the issuer, so a barrier per buffer
  uint64_t* o_done = p_ready + NS * NB;       // [NS][NB]
  uint64_t* w_full = o_done + NS * NB;        // [kSlots]
  uint64_t* w_empty = w_full + kSlots;        // [kSlots]: the issuers and the softmax warps
  uint32_t* tmem_base_smem = reinterpret_cast<uint32_t*>(w_empty + kSlots);
  uint32_t* dead = tmem_base_smem + 1;
  FlashItem* s_item = reinterpret_cast<FlashItem*>(bars + 64);          // [kSlots]
  uint64_t* clc_bar = bars + 48;
  uint4* s_clc = reinterpret_cast<uint4*>(bars + 50);                   // answer of the launch queue (16-byte aligned)
  int* s_cum = reinterpret_cast<int*>(v_smem + ST * VB + 960);          // [num_seqs] row tiles of the sequences up to this one
  int* s_start = s_cum + kMaxSeqs;                                      // [num_seqs + 1] first rows
  int* s_ctx = s_start + kMaxSeqs + 16;                                 // [num_seqs] tokens in the cache after this step
  float* s_red = reinterpret_cast<float*>(s_ctx + kMaxSeqs);            // NS == 1: [parity, or 2: sums][half][row]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 8 && lane == 0) {
    if (!SINK) tma_prefetch_desc(&tmap_q);
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
    *dead = 0u;
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], SINK ? 128 : 1);
      mbar_init(&q_empty[i], 1);
      mbar_init(&o_free[i], NS == 2 ? 128 : 256);
    }
    for (int i = 0; i < ST; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], NS); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); }
    for (int i = 0; i < NS * NB; ++i) { mbar_init(&s_full[i], 1); mbar_init(&p_ready[i], NS == 2 ? 128 : 256); mbar_init(&o_done[i], 1); }
    for (int i = 0; i < kSlots; ++i) { mbar_init(&w_full[i], 1); mbar_init(&w_empty[i], 9 + NS); }
    mbar_init(clc_bar, 1);
    mbar_fence_init();
  }
  if (warp == 9) tmem_alloc(tmem_base_smem, 512);
  pdl_launch_dependents();
  pdl_wait();  // queries, cache and step metadata are written by predecessor kernels

  const bool pair_heads = NS == 2 && (p.q_heads / p.kv_heads) % 2 == 0;
  const int heads = pair_heads ? p.q_heads / 2 : p.q_heads;
  if (warp == 0) {
    const int span = NS == 2 && !pair_heads ? 2 * kRows : kRows;              // rows of a sequence that an item covers
    int base = 0;
    for (int b0 = 0; b0 < p.num_seqs; b0 += 32) {
      const int b = b0 + lane;
      const bool in = b < p.num_seqs;
      const int start = in ? __ldcg(p.cu_seqlens + b) : 0, stop = in ? __ldcg(p.cu_seqlens + b + 1) : 0;
      int incl = (stop - start + span - 1) / span;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
      }
      if (in) {
        s_cum[b] = base + incl;
        s_start[b] = start;
        s_start[b + 1] = stop;
        s_ctx[b] = __ldcg(p.context_lens + b);
      }
      base += __shfl_sync(0xffffffffu, incl, 31);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_base_smem;
  const int total = s_cum[p.num_seqs - 1], items = total * heads;
  auto wait = [&](uint64_t* bar, uint32_t parity) { return mbar_wait_bounded(bar, parity, dead, p.wait.spins); };
  // the i-th item of this CTA, as the producer drew and laid it out; false at the end of the list, or where a wait gave up
  auto item_at = [&](uint32_t i, FlashItem& it) {
    const bool here = wait(&w_full[i % kSlots], (i / kSlots) & 1);
    it = s_item[i % kSlots];
    return here && it.n_max >= 0 && *reinterpret_cast<volatile uint32_t*>(dead) == 0u;
  };

  if (warp == 8) {
    // ============================================================== TMA producer
    if (elect_one()) {
      uint32_t kv = 0, qn[NS];
#pragma unroll
      for (int s = 0; s < NS; ++s) qn[s] = 0;
      int w = blockIdx.x;
      bool alive = true;                                                        // a copy is armed only on a barrier whose last one has been waited for
      for (uint32_t i = 0; alive; ++i) {
        if (i > 0) {                                                            // the item of a CTA that was taken out of the launch queue
          if (!wait(clc_bar, (i - 1) & 1)) break;
          w = ft_canceled_cta(s_clc, items);
        }
        const bool more = w < items;
        FlashItem it = {};
        it.n_max = -1;
        if (more) it = ft_item<NS, MODE>(p, s_cum, s_start, s_ctx, w, total, heads, pair_heads);
        if (!wait(&w_empty[i % kSlots], ((i / kSlots) & 1) ^ 1)) break;
        s_item[i % kSlots] = it;
        mbar_arrive(&w_full[i % kSlots]);
        if (!more) break;
        fence_proxy_async_smem();                                               // (the last answer has been read)
        mbar_arrive_expect_tx(clc_bar, 16);
        ft_try_cancel(s_clc, clc_bar);                                          // on its way while this item's copies are issued
        const int* bt = p.block_tables + (size_t)it.seq * p.max_blocks;
        const int R = p.box_rows, per = kKeys / R, kv_end = max(it.end[0], it.end[1]);
        const long long lin0 = MLA ? (p.lin_stride < 0 ? (long long)it.tok_base : p.lin_stride * it.seq) : 0;
        // cache rows of a tile's boxes (pages behind the last key are not in the table); looked up a tile ahead, so that the table's latency
        // lies behind the waits below
        auto rows_of = [&](int j, int (&row)[4]) {
          const int key0 = it.tile(j) * kKeys;
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            const int key = key0 + b * R;
            if (b < per && key < kv_end) row[b] = MLA ? bt[key / p.page] * p.page + key % p.page : (bt[key / p.page] * p.kv_heads + it.hk) * p.page + key % p.page;
          }
        };
        int row[4] = {0, 0, 0, 0};
        rows_of(0, row);
        if constexpr (!SINK) {
#pragma unroll
          for (int s = 0; s < NS; ++s) {
            if (it.n[s] == 0) continue;
            alive = alive && wait(&q_empty[s], (qn[s] & 1) ^ 1);
            if (!alive) continue;
            mbar_arrive_expect_tx(&q_full[s], QB);
            for (int c = 0; c < CK; ++c) tma_load_3d(q_smem + s * QB + c * kRows * 128, &tmap_q, &q_full[s], c * 64, it.head[s], it.tok[s]);
            ++qn[s];
          }
        }
        for (int j = 0; alive && j < it.n_max; ++j, ++kv) {
          const int st = kv % ST;
          const uint32_t ph = (kv / ST) & 1;
          const int key0 = it.tile(j) * kKeys, nbox = min(per, (kv_end - key0 + R - 1) / R);
          const uint32_t kd = smem_u32(k_smem + st * KB), vd = smem_u32(v_smem + st * VB);
          int ahead[4] = {0, 0, 0, 0};
          if (j + 1 < it.n_max) rows_of(j + 1, ahead);
          alive = wait(&k_empty[st], ph ^ 1);
          if (!alive) break;
          if constexpr (MLA) {
            const int lin = (int)(lin0 + key0);
            mbar_arrive_expect_tx(&k_full[st], KB);
            for (int c = 0; c < CK - 1; ++c) ft_tma_2d(kd + c * CHUNK, &tmap_k, &k_full[st], it.head[0] * (DK - 64 + DV) + c * 64, lin);
            ft_tma_2d(kd + (CK - 1) * CHUNK, &tmap_pe, &k_full[st], 512, row[0]);
            alive = wait(&v_empty[st], ph ^ 1);
            if (!alive) break;
            mbar_arrive_expect_tx(&v_full[st], VB);
            for (int c = 0; c < CV; ++c) ft_tma_2d(vd + c * CHUNK, &tmap_k, &v_full[st], it.head[0] * (DK - 64 + DV) + DK - 64 + c * 64, lin);
          } else {
            mbar_arrive_expect_tx(&k_full[st], nbox * R * DK * 2);
#pragma unroll
            for (int b = 0; b < 4; ++b)
              if (b < nbox)
                for (int c = 0; c < CK; ++c) ft_tma_2d(kd + c * CHUNK + b * R * 128, &tmap_k, &k_full[st], c * 64, row[b]);
            alive = wait(&v_empty[st], ph ^ 1);
            if (!alive) break;
            mbar_arrive_expect_tx(&v_full[st], nbox * R * DV * 2);
#pragma unroll
            for (int b = 0; b < 4; ++b)
              if (b < nbox)
                for (int c = 0; c < CV; ++c) ft_tma_2d(vd + c * CHUNK + b * R * 128, &tmap_v, &v_full[st], c * 64, row[b]);
          }
#pragma unroll
          for (int b = 0; b < 4; ++b) row[b] = ahead[b];
        }
      }
    }
  } else if (warp == 9 || (NS == 2 && warp == 10)) {
    // ============================================================== S = Q K^T of one stream
    // (Issuing a product costs a thread more than the tensor pipe takes for 128 x 64 x 16, so every stream's scores have an issuer of their own.)
    if (elect_one()) {
      const int s = warp - 9;
      uint32_t kv = 0, g = 0, cnt = 0;                                          // key tiles of the CTA, tiles and items of the stream so far
      const uint32_t qa = smem_u32(q_smem + s * QB);
      FlashItem it;
      bool alive = true;
      for (uint32_t i = 0; alive && item_at(i, it); ++i) {
        mbar_arrive(&w_empty[i % kSlots]);
        const int n = s ? it.n[1] : it.n[0];
        if (n > 0) alive = wait(&q_full[s], cnt & 1);
        for (int j = 0; alive && j < it.n_max; ++j, ++kv) {
          alive = wait(&k_full[kv % ST], (kv / ST) & 1);
          if (!alive) break;
          if (j >= n) {                                                         // (rows in pairs: the first tile sees fewer keys)
            mbar_arrive(&k_empty[kv % ST]);
            continue;
          }
          if (g >= NB) alive = wait(&o_done[s * NB + g % NB], (g / NB - 1) & 1);                   // the product that read this buffer's P
          if (!alive) break;
          tc_fence_after();
          const uint32_t ka = smem_u32(k_smem + (kv % ST) * KB), d = tmem_base + (s * NB + g % NB) * 64;
#pragma unroll
          for (int c = 0; c < CK; ++c) {
            const uint64_t ad = umma_desc_sw128(qa + c * kRows * 128), bd = umma_desc_sw128(ka + c * CHUNK);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) umma_f16(d, ad + 2 * kk, bd + 2 * kk, IDESC_S, (c | kk) ? 1u : 0u);
            if constexpr (SINK) {                                               // what the rounding of the queries left
              const uint64_t al = umma_desc_sw128(qa + (CK + c) * kRows * 128);
#pragma unroll
              for (int kk = 0; kk < 4; ++kk) umma_f16(d, al + 2 * kk, bd + 2 * kk, IDESC_S, 1u);
            }
          }
          umma_commit(&s_full[s * NB + g % NB]);
          umma_commit(&k_empty[kv % ST]);
          if (j + 1 == n) umma_commit(&q_empty[s]);
          ++g;
        }
        cnt += n > 0 ? 1 : 0;
      }
    }
  } else if (warp == 11) {
    // ============================================================== O += P V of every stream
    if (elect_one()) {
      uint32_t kv = 0, g[2] = {0, 0}, cnt[2] = {0, 0};
      FlashItem it;
      bool alive = true;
      for (uint32_t i = 0; alive && item_at(i, it); ++i) {
        mbar_arrive(&w_empty[i % kSlots]);
        for (int j = 0; alive && j < it.n_max; ++j, ++kv) {
          alive = wait(&v_full[kv % ST], (kv / ST) & 1);
#pragma unroll
          for (int s = 0; s < NS; ++s) {
            if (j >= it.n[s]) continue;
            if (j == 0 && cnt[s] > 0) alive = alive && wait(&o_free[s], (cnt[s] - 1) & 1);        // the last item's result has been read
            alive = alive && wait(&p_ready[s * NB + g[s] % NB], (g[s] / NB) & 1);
            if (!alive) continue;
            tc_fence_after();
            const uint32_t va = smem_u32(v_smem + (kv % ST) * VB), pa = tmem_base + (s * NB + g[s] % NB) * 64, d = tmem_base + O_COL + s * DV;
#pragma unroll
            for (int ks = 0; ks < kKeys / 16; ++ks) {
              const uint64_t bd = umma_desc_mn_sw128(va + ks * 2048, CHUNK, 1024);
              umma_f16_ts(d, pa + 8 * ks, bd, IDESC_O, (j | ks) ? 1u : 0u);
              if constexpr (SPLIT) umma_f16_ts(d, pa + 32 + 8 * ks, bd, IDESC_O, 1u);
            }
            umma_commit(&o_done[s * NB + g[s] % NB]);
            ++g[s];
          }
          umma_commit(&v_empty[kv % ST]);
        }
#pragma unroll
        for (int s = 0; s < NS; ++s) cnt[s] += it.n[s] > 0 ? 1 : 0;
      }
    }
  } else if (warp < 8) {
    // ============================================================== softmax: one row per thread (NS == 1: two threads per row, 32 columns each)
    constexpr int COLS = NS == 2 ? kKeys : kKeys / 2;
    constexpr int PAIRS = COLS / 2;
    constexpr float kLog2e = 1.4426950408889634f;
    const int s = NS == 2 ? warp >> 2 : 0, half = NS == 2 ? 0 : warp >> 2;
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const float sl2 = SINK ? kLog2e : (CAP ? p.softcap : p.scale) * kLog2e;      // scores -> base-2 domain
    const float cap_in = CAP ? p.scale / p.softcap : 0.f;
    const uint32_t o_addr = tmem_base + lane_addr + O_COL + s * DV + (NS == 1 ? half * (DV / 2) : 0);
    constexpr int OCOLS = NS == 2 ? DV : DV / 2;                                 // accumulator columns that this thread rescales and stores
    uint32_t g = 0, kv0 = 0, cnt = 0;                                            // tiles of the stream, key tiles of the CTA, items of the stream so far
    FlashItem it;
    for (uint32_t i = 0;; ++i) {
      // threads that meet at a barrier, a shuffle or a warp-wide access to TMEM below leave at the same item.  (Where a wait gives up inside an
      // item its later ones fall through, and the item is walked to its end.)
      const bool on = item_at(i, it);
      __syncwarp();
      if constexpr (NS == 1) {
        if (!named_bar_and(3, 256, on)) break;
      } else {
        if (!__all_sync(0xffffffffu, on)) break;
      }
      if (lane == 0) mbar_arrive(&w_empty[i % kSlots]);
      const int n = s ? it.n[1] : it.n[0], pos0 = s ? it.pos[1] : it.pos[0], rows = s ? it.rows[1] : it.rows[0], kv_end = s ? it.end[1] : it.end[0];
      const int tok = s ? it.tok[1] : it.tok[0], head = s ? it.head[1] : it.head[0];
      const int qpos = pos0 + row, v_end = max(it.end[0], it.end[1]);
      if (n == 0) {                                                              // (rows in pairs: the second tile holds none)
        kv0 += it.n_max;
        continue;
      }
      if constexpr (SINK) {
        // this row's query as two bf16 terms, in the K-major 128B-swizzled layout that TMA writes
        wait(&q_empty[s], (cnt & 1) ^ 1);
        constexpr int LPR = DK / 4, RPI = 32 / LPR;                              // lanes of a row, rows of an instruction: whole rows, coalesced
        const int c4 = lane % LPR;
#pragma unroll 8
        for (int r0 = 0; r0 < 32; r0 += RPI) {
          const int r = (warp & 3) * 32 + r0 + lane / LPR;
          float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
          if (r < rows) f = *reinterpret_cast<const float4*>(p.q32 + ((size_t)(tok + r) * p.q_heads + head) * DK + c4 * 4);
          f.x *= p.scale; f.y *= p.scale; f.z *= p.scale; f.w *= p.scale;
          const uint32_t h0 = pack_bf16(f.x, f.y), h1 = pack_bf16(f.z, f.w);
          uint8_t* d = q_smem + s * QB + r * 128 + (c4 >> 4) * kRows * 128 + ((((c4 >> 1) & 7) ^ (r & 7)) << 4) + (c4 & 1) * 8;
          *reinterpret_cast<uint2*>(d) = make_uint2(h0, h1);
          *reinterpret_cast<uint2*>(d + CK * kRows * 128) = make_uint2(pack_bf16(f.x - bf16_lo(h0), f.y - bf16_hi(h0)), pack_bf16(f.z - bf16_lo(h1), f.w - bf16_hi(h1)));
        }
        fence_proxy_async_smem();
        mbar_arrive(&q_full[s]);
      }
      const int lo_key = SINK ? ft_first_key(p, qpos) : 0, lo_last = SINK ? ft_first_key(p, pos0 + rows - 1) : 0;
      float m = -INFINITY, l = 0.f;

      for (int j = 0; j < n; ++j, ++g) {
        const uint32_t buf = tmem_base + lane_addr + (s * NB + g % NB) * 64;
        wait(&s_full[s * NB + g % NB], (g / NB) & 1);
        tc_fence_after();
        uint32_t v[COLS];
#pragma unroll
        for (int c = 0; c < COLS; c += 32) tmem_ld32(buf + half * COLS + c, v + c);
        tmem_ld_wait();
        float* x = reinterpret_cast<float*>(v);
        if constexpr (CAP) {
#pragma unroll
          for (int c = 0; c < COLS; ++c) x[c] = tanhf(x[c] * cap_in);
        }
        const int tile0 = it.tile(j) * kKeys, key0 = tile0 + half * COLS;
        // tiles that some row does not see as a whole
        if (key0 + COLS - 1 > pos0 || key0 + COLS > kv_end || (SINK && key0 < lo_last && key0 + COLS > p.keep)) {
          const int lim = min(qpos, kv_end - 1) - key0;                          // last visible column
#pragma unroll
          for (int c = 0; c < COLS; ++c) x[c] = c <= lim && (!SINK || key0 + c >= lo_key || key0 + c < p.keep) ? x[c] : -INFINITY;
        }
        float mx[4] = {x[0], x[1], x[2], x[3]};
#pragma unroll
        for (int c = 4; c < COLS; c += 4) {
#pragma unroll
          for (int e = 0; e < 4; ++e) mx[e] = fmaxf(mx[e], x[c + e]);
        }
        float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
        if constexpr (NS == 1) {                                                 // the row's other half
          float* red = s_red + (g & 1) * 2 * kRows;
          red[half * kRows + row] = top;
          named_bar_sync(1, 256);
          top = fmaxf(top, red[(half ^ 1) * kRows + row]);
        }
        top *= sl2;
        const bool moved = __any_sync(0xffffffffu, top > m + LAG);               // (m = -inf: the row's first visible tile)
        float corr = 1.f;
        if (moved) {
          const float mn = top > m + LAG ? top : m;
          corr = mn == -INFINITY ? 1.f : exp2f(m - mn);
          m = mn;
          l *= corr;
        }
        const float sub = m == -INFINITY ? 0.f : -m;
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
        uint32_t hi[PAIRS], lo[SPLIT ? PAIRS : 1];
#pragma unroll
        for (int c = 0; c < PAIRS; ++c) {
          const float a = exp2f(fmaf(x[2 * c], sl2, sub)), b = exp2f(fmaf(x[2 * c + 1], sl2, sub));
          sum[c & 3] += a + b;
          hi[c] = pack_bf16(a, b);
          if constexpr (SPLIT) lo[c] = pack_bf16(a - bf16_lo(hi[c]), b - bf16_hi(hi[c]));
        }
        l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
        if constexpr (NS == 1) named_bar_sync(2, 256);                           // P overwrites the scores: both halves of a row have been read
#pragma unroll
        for (int c = 0; c < PAIRS; c += 16) {
          tmem_st16(buf + half * PAIRS + c, hi + c);
          if constexpr (SPLIT) tmem_st16(buf + 32 + half * PAIRS + c, lo + c);
        }
        if (moved && j > 0) {
          // the accumulator follows the maximum; here the last tile's product has had the time of the exponentials to complete
          wait(&o_done[s * NB + (g - 1) % NB], ((g - 1) / NB) & 1);
          tc_fence_after();
          constexpr int W = OCOLS % 64 == 0 ? 64 : 32;
#pragma unroll 1
          for (int c = 0; c < OCOLS; c += W) {
            uint32_t o[W];
#pragma unroll
            for (int e = 0; e < W; e += 32) tmem_ld32(o_addr + c + e, o + e);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < W; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * corr);
#pragma unroll
            for (int e = 0; e < W; e += 16) tmem_st16(o_addr + c + e, o + e);
          }
        }
        tmem_st_wait();
        const int vend = v_end - tile0;
        if (vend < kKeys) {
          // the tile's rows of V behind the last key that any stream sees: zeros (both streams write the same zeros)
          const uint32_t kv = kv0 + j;
          wait(&v_full[kv % ST], (kv / ST) & 1);
          const int r = threadIdx.x & 63;
          if (r >= vend) {
            for (int c = 0; c < CV; ++c)
#pragma unroll
              for (int e = 0; e < 8; ++e)
                *reinterpret_cast<uint4*>(v_smem + (kv % ST) * VB + c * CHUNK + r * 128 + e * 16) = make_uint4(0u, 0u, 0u, 0u);
          }
          fence_proxy_async_smem();
        }
        tc_fence_before();
        mbar_arrive(&p_ready[s * NB + g % NB]);
      }
      kv0 += it.n_max;
      ++cnt;
      // ---- normalise and store
      if constexpr (NS == 1) {
        float* red = s_red + 2 * 2 * kRows;
        red[half * kRows + row] = l;
        named_bar_sync(1, 256);
        l += red[(half ^ 1) * kRows + row];
      }
      float inv = 1.f;
      if constexpr (SINK) {
        if (p.sink != nullptr) l += exp2f(fmaf(p.sink[head], kLog2e, -m));
        inv = p.out_mult;
        if (p.gate != nullptr && !p.gate_elem && row < rows) inv *= 1.f / (1.f + expf(-__bfloat162float(p.gate[(size_t)(tok + row) * p.ld_gate + head])));
      }
      inv = l > 0.f ? inv / l : 0.f;
      wait(&o_done[s * NB + (g - 1) % NB], ((g - 1) / NB) & 1);
      tc_fence_after();
      if (*reinterpret_cast<volatile uint32_t*>(dead) != 0u) inv = __int_as_float(0x7fffffff);
      const int col0 = head * DV + (NS == 1 ? half * (DV / 2) : 0);
#pragma unroll 1
      for (int c = 0; c < OCOLS; c += 32) {
        uint32_t o[32];
        tmem_ld32(o_addr + c, o);
        tmem_ld_wait();
        if (c + 32 >= OCOLS) {
          tc_fence_before();
          mbar_arrive(&o_free[s]);
        }
        float f[32];
#pragma unroll
        for (int e = 0; e < 32; ++e) f[e] = __uint_as_float(o[e]) * inv;
        if constexpr (SINK) {
          if (p.gate != nullptr && p.gate_elem && row < rows) {
            const __nv_bfloat16* gp = p.gate + (size_t)(tok + row) * p.ld_gate + col0 + c;
#pragma unroll
            for (int e = 0; e < 32; ++e) f[e] *= 1.f / (1.f + expf(-__bfloat162float(gp[e])));
          }
        }
        // a row's 64 bytes lie in one lane; four lanes exchange 16-byte pieces, so that a store writes 64 bytes of 8 rows and not 16 of 32
        uint32_t w[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) w[e] = pack_bf16(f[2 * e], f[2 * e + 1]);
        const bool b0 = lane & 1, b1 = lane & 2;
#pragma unroll
        for (int e = 0; e < 4; ++e) {                                            // pieces 0 <-> 1 and 2 <-> 3 with the neighbour
          const uint32_t x0 = __shfl_xor_sync(0xffffffffu, b0 ? w[e] : w[4 + e], 1), x1 = __shfl_xor_sync(0xffffffffu, b0 ? w[8 + e] : w[12 + e], 1);
          if (b0) { w[e] = x0; w[8 + e] = x1; } else { w[4 + e] = x0; w[12 + e] = x1; }
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {                                            // pairs of pieces with the lane two away
          const uint32_t x0 = __shfl_xor_sync(0xffffffffu, b1 ? w[e] : w[8 + e], 2);
          if (b1) w[e] = x0; else w[8 + e] = x0;
        }
        const int quad_row = (warp & 3) * 32 + (lane & ~3);
#pragma unroll
        for (int k = 0; k < 4; ++k)                                              // lane q of the quad now holds piece q of its four rows
          if (quad_row + k < rows)
            *reinterpret_cast<uint4*>(p.out + (size_t)(tok + quad_row + k) * p.o_ld_t + col0 + c + (lane & 3) * 8) =
                make_uint4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]);
      }
    }
    tc_fence_before();
  }
  __syncthreads();
  if (*reinterpret_cast<volatile uint32_t*>(dead) != 0u) report_dead(p.wait, kWaitPromptAttention);     // before the CTA's memory goes
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

bool ft_map_2d(CUtensorMap* m, const void* ptr, uint64_t cols, uint64_t rows, uint64_t ld, uint32_t box_rows) {
  const cuuint64_t dims[2] = {cols, rows}, strides[1] = {ld * 2};
  const cuuint32_t box[2] = {64, box_rows}, one[2] = {1, 1};
  return tensor_map_encoder()(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
bool ft_map_q(CUtensorMap* m, const void* ptr, uint64_t dk, uint64_t heads, uint64_t tokens, uint64_t ld_h, uint64_t ld_t) {
  const cuuint64_t dims[3] = {dk, heads, tokens}, strides[2] = {ld_h * 2, ld_t * 2};
  const cuuint32_t box[3] = {64, 1, kRows}, one[3] = {1, 1, 1};
  return tensor_map_encoder()(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int DK, int DV, int MODE>
cudaError_t launch_flash_tc(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tpe, const FlashTcParams& p,
                            int tokens, cudaStream_t s) {
  constexpr int smem = ft_smem(DK, DV, MODE);
  static_assert(smem <= 227 * 1024, "shared memory budget exceeded");
  auto kern = flash_tc_kernel<DK, DV, MODE>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    configured = true;
  }
  const bool pair_heads = ft_streams(DV) == 2 && (p.q_heads / p.kv_heads) % 2 == 0;
  const int span = ft_streams(DV) == 2 && !pair_heads ? 2 * kRows : kRows;
  const long long most = (long long)(tokens / span + p.num_seqs) * (pair_heads ? p.q_heads / 2 : p.q_heads);   // at most one ragged tile per sequence
  if (most > 0x7fffffffLL) return cudaErrorInvalidValue;
  (void)launch_pdl(kern, dim3((unsigned)most), dim3(kFlashThreads), smem, s, tq, tk, tv, tpe, p);
  return cudaGetLastError();
}

bool ft_aligned(const void* ptr) { return (reinterpret_cast<uintptr_t>(ptr) & 15) == 0; }
bool ft_pages(int page) { return page % kKeys == 0 || page == 16 || page == 32; }

}  // namespace

bool flash_tc_supported(const FlashPrefillArgs& a) {
  const bool dims = (a.dk_ == 128 && a.dv_ == 128) || (a.dk_ == 192 && a.dv_ == 128) || (a.dk_ == 64 && a.dv_ == 64) || (a.dk_ == 256 && a.dv_ == 256);
  return dims && ft_pages(a.page) && a.q_heads % a.kv_heads == 0 && a.q_ld_t % 8 == 0 && a.q_ld_h % 8 == 0 && ft_aligned(a.q) && ft_aligned(a.kpool) &&
         ft_aligned(a.vpool) && ft_aligned(a.out) && a.o_ld_t % 8 == 0 && a.num_seqs <= kMaxSeqs && a.pool_rows < (1LL << 31) && tensor_map_encoder() != nullptr;
}

cudaError_t flash_tc_launch(const FlashPrefillArgs& a, cudaStream_t s) {
  if (a.num_seqs == 0 || a.tokens == 0) return cudaSuccess;
  if (!flash_tc_supported(a)) return cudaErrorInvalidValue;
  FlashTcParams p = {};
  p.block_tables = a.block_tables; p.max_blocks = a.max_blocks; p.cu_seqlens = a.cu_seqlens; p.context_lens = a.context_lens; p.num_seqs = a.num_seqs;
  p.q_heads = a.q_heads; p.kv_heads = a.kv_heads; p.page = a.page; p.box_rows = a.page % kKeys == 0 ? kKeys : a.page; p.lin_stride = -1;
  p.wait = a.wait;
  p.scale = a.scale; p.softcap = a.softcap; p.out = static_cast<__nv_bfloat16*>(a.out); p.o_ld_t = a.o_ld_t;
  CUtensorMap tq, tk, tv;
  if (!ft_map_q(&tq, a.q, a.dk_, a.q_heads, a.tokens, a.q_ld_h, a.q_ld_t) || !ft_map_2d(&tk, a.kpool, a.dk_, a.pool_rows, a.dk_, p.box_rows) ||
      !ft_map_2d(&tv, a.vpool, a.dv_, a.pool_rows, a.dv_, p.box_rows))
    return cudaErrorInvalidValue;
  if (a.softcap > 0.f) {
    if (a.dk_ == 256) return launch_flash_tc<256, 256, kCap>(tq, tk, tv, tk, p, a.tokens, s);
    if (a.dk_ == 192) return launch_flash_tc<192, 128, kCap>(tq, tk, tv, tk, p, a.tokens, s);
    if (a.dk_ == 128) return launch_flash_tc<128, 128, kCap>(tq, tk, tv, tk, p, a.tokens, s);
    return launch_flash_tc<64, 64, kCap>(tq, tk, tv, tk, p, a.tokens, s);
  }
  if (a.dk_ == 256) return launch_flash_tc<256, 256, 0>(tq, tk, tv, tk, p, a.tokens, s);
  if (a.dk_ == 192) return launch_flash_tc<192, 128, 0>(tq, tk, tv, tk, p, a.tokens, s);
  if (a.dk_ == 128) return launch_flash_tc<128, 128, 0>(tq, tk, tv, tk, p, a.tokens, s);
  return launch_flash_tc<64, 64, 0>(tq, tk, tv, tk, p, a.tokens, s);
}

bool flash_mla_supported(int num_seqs) { return num_seqs <= kMaxSeqs; }

cudaError_t flash_mla_launch(const FlashMlaArgs& a, cudaStream_t s) {
  if (a.num_seqs == 0 || a.tokens == 0) return cudaSuccess;
  if (a.page % kKeys != 0 || a.q_ld_t % 8 != 0 || a.q_ld_h % 8 != 0 || a.kv_ld % 8 != 0 || !ft_aligned(a.q) || !ft_aligned(a.kv) || !ft_aligned(a.pool) ||
      !ft_aligned(a.out) || a.o_ld_t % 8 != 0 || a.kv_rows >= (1LL << 31) || a.pool_rows >= (1LL << 31) || a.num_seqs > kMaxSeqs || tensor_map_encoder() == nullptr)
    return cudaErrorInvalidValue;
  FlashTcParams p = {};
  p.block_tables = a.block_tables; p.max_blocks = a.max_blocks; p.cu_seqlens = a.cu_seqlens; p.context_lens = a.context_lens; p.num_seqs = a.num_seqs;
  p.q_heads = p.kv_heads = a.heads; p.page = a.page; p.box_rows = kKeys; p.lin_stride = a.lin_stride; p.scale = a.scale; p.wait = a.wait;
  p.out = static_cast<__nv_bfloat16*>(a.out); p.o_ld_t = a.o_ld_t;
  CUtensorMap tq, tk, tpe;
  if (!ft_map_q(&tq, a.q, 192, a.heads, a.tokens, a.q_ld_h, a.q_ld_t) || !ft_map_2d(&tk, a.kv, (uint64_t)a.heads * 256, a.kv_rows, a.kv_ld, kKeys) ||
      !ft_map_2d(&tpe, a.pool, 576, a.pool_rows, 576, kKeys))
    return cudaErrorInvalidValue;
  return launch_flash_tc<192, 128, kMla>(tq, tk, tk, tpe, p, a.tokens, s);
}

bool flash_sink_takes(const SinkAttnArgs& a, long long pool_rows) {
  const bool dims = (a.D == 128 && a.V == 128) || (a.D == 64 && a.V == 64);
  return dims && a.slopes == nullptr && a.bias == nullptr && ft_pages(a.page) && a.H % a.G == 0 && a.B > 0 && a.B <= kMaxSeqs && ft_aligned(a.q) &&
         ft_aligned(a.kpool) && ft_aligned(a.vpool) && ft_aligned(a.out) && a.ld_out % 8 == 0 && pool_rows < (1LL << 31) && tensor_map_encoder() != nullptr;
}

cudaError_t flash_sink_launch(const SinkAttnArgs& a, const int* context_lens, long long pool_rows, int tokens, const WaitBound& wait, cudaStream_t s) {
  if (!flash_sink_takes(a, pool_rows)) return cudaErrorInvalidValue;
  FlashTcParams p = {};
  p.wait = wait;
  p.block_tables = a.block_tables; p.max_blocks = a.max_blocks; p.cu_seqlens = a.cu; p.context_lens = context_lens; p.num_seqs = a.B;
  p.q_heads = a.H; p.kv_heads = a.G; p.page = a.page; p.box_rows = a.page % kKeys == 0 ? kKeys : a.page; p.lin_stride = -1;
  p.scale = a.scale; p.out = static_cast<__nv_bfloat16*>(a.out); p.o_ld_t = a.ld_out;
  p.q32 = a.q; p.sink = a.sink; p.gate = static_cast<const __nv_bfloat16*>(a.gate); p.ld_gate = a.ld_gate; p.gate_elem = a.gate_elem ? 1 : 0;
  p.block = a.block; p.window = a.window; p.keep = a.keep; p.out_mult = a.out_mult;
  CUtensorMap tk, tv;
  if (!ft_map_2d(&tk, a.kpool, a.D, pool_rows, a.D, p.box_rows) || !ft_map_2d(&tv, a.vpool, a.V, pool_rows, a.V, p.box_rows)) return cudaErrorInvalidValue;
  if (a.D == 128) return launch_flash_tc<128, 128, kSink>(tk, tk, tv, tk, p, tokens, s);
  return launch_flash_tc<64, 64, kSink>(tk, tk, tv, tk, p, tokens, s);
}

}  // namespace b200
