// Paged-KV attention of decode steps (and of ragged batches that the tensor-core prefill kernels do not take): split-KV flash-decoding with
// online softmax on the warp-level tensor path.
//
// The reference runs `mx.fast.scaled_dot_product_attention` over one contiguous, ever-growing KVCache
// with a dense additive mask (shard/server/model/llama.py:48-59 via mlx_lm) for exactly one sequence.
// This kernel serves a ragged batch against a *paged* cache: every query token carries its own causal
// limit (kv_len = position + 1) and its sequence's block table, so the same kernel handles decode
// micro-batches and mixed batches.  d_qk != d_v (MLA 192/128), GQA and Gemma-2 logit soft-capping are supported.
//
// What bounds it: the K / V bytes (512 B per key and kv head at d = 128), read once per (token, kv head).  A form that splits a head over the
// lanes spends ~100 issue slots per key on shuffle trees and on a serial softmax per head (0.7 TB/s measured); here 16 keys meet all G heads
// of the group in one product:
//   * CTA = (query token, kv head, split), 4 warps (1 for short contexts); every warp walks its own 16-key tiles through a private cp.async ring, so the main loop has
//     no CTA barrier and 2 CTAs per SM keep ~130 KB in flight;
//   * S[16 (G used), 16 keys] = Q K^T and O^T[dv, 8 heads] += V^T P^T with mma.m16n8k16: the score fragment IS the B operand of the second
//     product (no shuffle), and the second product has no padded rows;
//   * probabilities enter the second product as two bf16 terms, p = hi + lo (error 2^-17 of p; the sums are fp32), where the form on the CUDA cores held
//     them in fp32.  Error of the op against 64 bits, ragged contexts of 100 to 7000 keys: 1.65859e-3 with either (the rounding of the result); a third
//     term takes 17.5 to 19.2 us for 64 sequences of 256 keys.  A visible infinity in V gives NaN (0 * inf in the low term), where it gave infinity;
//   * splits: 16-key tiles are dealt round-robin to (split, warp), so ragged contexts share out evenly; the last CTA of a (token, kv head)
//     to arrive (ticket) merges the splits' partials -- no second kernel.
// B200, 32 sequences x ~4 k tokens, 8 kv heads x 128, G = 4 (537 MB of cache): the whole attention block 782 -> 139 us; a Llama-3-8B decode step of
// one sequence at 512 tokens 4494 -> 3117 us (the block's combine kernel is gone).
#include <algorithm>

#include "kernels.h"
#include "launch.h"
#include "ptx.cuh"

namespace b200 {

namespace {

constexpr int kDecWarps = 4;
constexpr int kDecKeys = 16;      // keys of a warp's tile (the K extent of one mma of the second product)
constexpr int kDecHeads = 8;      // query heads per kv head that a tile holds

__host__ __device__ constexpr int dec_tile_bytes(int dk, int dv) { return kDecKeys * (dk + dv) * 2; }
// ring depth: two CTAs of up to ~100 KB per SM; heads of 256 take one CTA per SM
__host__ __device__ constexpr int dec_stages(int dk, int dv) { return dk + dv <= 128 ? 4 : dk + dv <= 256 ? 3 : dk + dv <= 320 ? 2 : 3; }
__host__ __device__ constexpr int dec_smem(int dk, int dv, int warps, int stages) {
  const int ring = warps * stages * dec_tile_bytes(dk, dv);
  const int merge = warps * kDecHeads * (dv + 4) * 4;
  return ring > merge ? ring : merge;
}

template <int DK, int DV, int WARPS, int STAGES>
__global__ void __launch_bounds__(WARPS * 32)
paged_decode_kernel(const __nv_bfloat16* __restrict__ q, long long q_ld_t, long long q_ld_h, const __nv_bfloat16* __restrict__ kpool,
                    const __nv_bfloat16* __restrict__ vpool, const int* __restrict__ block_tables, int max_blocks,
                    const int* __restrict__ positions, const int* __restrict__ token_seq, int kv_heads, int G, int page, float scale,
                    float softcap, int nsplit, __nv_bfloat16* __restrict__ out, long long o_ld_t, float* __restrict__ part_acc,
                    float* __restrict__ part_ml, unsigned int* __restrict__ tickets) {
  pdl_sync();  // PDL: predecessor's writes visible; let the successor start its prologue
  constexpr int TILE = dec_tile_bytes(DK, DV);
  constexpr int CK = DK / 8, CV = DV / 8;                     // 16-byte chunks of a row (multiples of 8: the swizzle stays inside 128 bytes)
  static_assert(DK % 64 == 0 && DV % 64 == 0, "head dims must be multiples of 64");
  constexpr float kLog2e = 1.4426950408889634f;
  extern __shared__ __align__(128) uint8_t dec_smem_raw[];
  const int t = blockIdx.x, hk = blockIdx.y, sp = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int kv_len = positions[t] + 1;
  const int* bt = block_tables + (size_t)token_seq[t] * max_blocks;
  const int ntile = (kv_len + kDecKeys - 1) / kDecKeys;
  const int first = sp * WARPS + warp, stride = nsplit * WARPS;
  const int n = first < ntile ? (ntile - 1 - first) / stride + 1 : 0;

  // cache row of this lane's key (lane & 15) of the warp's i-th tile; keys behind the end repeat the last one and are masked below
  auto row_of = [&](int i) -> uint32_t {
    const int pos = min((first + i * stride) * kDecKeys + (lane & 15), kv_len - 1);
    return ((uint32_t)bt[pos / page] * kv_heads + hk) * page + pos % page;
  };
  const uint32_t ring = smem_u32(dec_smem_raw) + warp * STAGES * TILE;
  auto load = [&](uint32_t rows, int buf) {
    const uint32_t base = ring + buf * TILE;
#pragma unroll
    for (int j = 0; j < kDecKeys * CK / 32; ++j) {
      const int idx = j * 32 + lane, r = idx / CK, c = idx % CK;
      const uint32_t row = __shfl_sync(0xffffffffu, rows, r);
      cp_async16(base + r * DK * 2 + ((c ^ (r & 7)) << 4), kpool + (size_t)row * DK + c * 8);
    }
#pragma unroll
    for (int j = 0; j < kDecKeys * CV / 32; ++j) {
      const int idx = j * 32 + lane, r = idx / CV, c = idx % CV;
      const uint32_t row = __shfl_sync(0xffffffffu, rows, r);
      cp_async16(base + kDecKeys * DK * 2 + r * DV * 2 + ((c ^ (r & 7)) << 4), vpool + (size_t)row * DV + c * 8);
    }
  };
  uint32_t next = n > 0 ? row_of(0) : 0u;
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < n) {
      load(next, s);
      if (s + 1 < n) next = row_of(s + 1);
    }
    cp_async_commit();
  }

  // queries: A operand, rows 0..7 = heads of the group (zeros behind G), rows 8..15 unused
  uint32_t qa[DK / 16][2];
  {
    const __nv_bfloat16* qp = q + (size_t)t * q_ld_t + (size_t)(hk * G + min(g, G - 1)) * q_ld_h;
#pragma unroll
    for (int ks = 0; ks < DK / 16; ++ks) {
      qa[ks][0] = g < G ? *reinterpret_cast<const uint32_t*>(qp + ks * 16 + t4 * 2) : 0u;
      qa[ks][1] = g < G ? *reinterpret_cast<const uint32_t*>(qp + ks * 16 + 8 + t4 * 2) : 0u;
    }
  }
  float o[DV / 16][4];                                        // O^T: dims mt*16 + g (+8), heads 2*t4, 2*t4 + 1
#pragma unroll
  for (int i = 0; i < DV / 16; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  float m = -INFINITY, l = 0.f;                               // of head g, in the base-2 domain; l: this lane's keys
  // ldmatrix lanes: 0-7 keys 0..7, first chunk; 8-15 the same keys, second chunk; 16-31 keys 8..15
  const int lk = (lane & 7) + ((lane >> 4) << 3), lc = (lane >> 3) & 1;

  for (int i = 0; i < n; ++i) {
    if (i + STAGES - 1 < n) {
      load(next, (i + STAGES - 1) % STAGES);
      if (i + STAGES < n) next = row_of(i + STAGES);
    }
    cp_async_commit();
    cp_async_wait<STAGES - 1>();
    __syncwarp();
    const uint32_t kb = ring + (i % STAGES) * TILE, vb = kb + kDecKeys * DK * 2;
    float sc[2][4];
#pragma unroll
    for (int e = 0; e < 4; ++e) sc[0][e] = sc[1][e] = 0.f;
#pragma unroll
    for (int ks = 0; ks < DK / 16; ++ks) {
      uint32_t r[4];
      ldmatrix_x4(r, kb + lk * DK * 2 + (((2 * ks + lc) ^ (lane & 7)) << 4));
      mma_m16n8k16(sc[0], qa[ks][0], 0u, qa[ks][1], 0u, r[0], r[1]);
      mma_m16n8k16(sc[1], qa[ks][0], 0u, qa[ks][1], 0u, r[2], r[3]);
    }
    const int key0 = (first + i * stride) * kDecKeys + t4 * 2;
    float p[4];                                               // keys key0, key0 + 1, key0 + 8, key0 + 9 of head g
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float s = sc[e >> 1][e & 1] * scale;
      if (softcap > 0.f) s = softcap * tanhf(s / softcap);
      p[e] = key0 + (e >> 1) * 8 + (e & 1) < kv_len ? s * kLog2e : -INFINITY;
    }
    float mx = fmaxf(fmaxf(p[0], p[1]), fmaxf(p[2], p[3]));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float mn = fmaxf(m, mx);                            // finite: a tile holds at least one visible key (unless the scores themselves overflow)
    const float corr = mn == -INFINITY ? 1.f : exp2f(m - mn);
#pragma unroll
    for (int e = 0; e < 4; ++e) p[e] = mn == -INFINITY ? 0.f : exp2f(p[e] - mn);
    l = l * corr + ((p[0] + p[1]) + (p[2] + p[3]));
    m = mn;
    if (__any_sync(0xffffffffu, corr != 1.f)) {
      const float c0 = __shfl_sync(0xffffffffu, corr, t4 * 8), c1 = __shfl_sync(0xffffffffu, corr, t4 * 8 + 4);
#pragma unroll
      for (int d = 0; d < DV / 16; ++d) { o[d][0] *= c0; o[d][1] *= c1; o[d][2] *= c0; o[d][3] *= c1; }
    }
    const uint32_t h0 = pack_bf16(p[0], p[1]), h1 = pack_bf16(p[2], p[3]);
    const uint32_t l0 = pack_bf16(p[0] - bf16_lo(h0), p[1] - bf16_hi(h0)), l1 = pack_bf16(p[2] - bf16_lo(h1), p[3] - bf16_hi(h1));
#pragma unroll
    for (int d = 0; d < DV / 16; ++d) {
      uint32_t r[4];
      ldmatrix_x4_trans(r, vb + lk * DV * 2 + (((2 * d + lc) ^ (lane & 7)) << 4));
      mma_m16n8k16(o[d], r[0], r[1], r[2], r[3], h0, h1);
      mma_m16n8k16(o[d], r[0], r[1], r[2], r[3], l0, l1);
    }
    __syncwarp();                                             // the slot is refilled by the next iteration
  }
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);

  // ---- merge the warps through shared memory (the rings are idle: every issued copy has been waited for)
  cp_async_wait<0>();
  __syncthreads();
  __shared__ float s_m[WARPS][kDecHeads], s_l[WARPS][kDecHeads];
  __shared__ int s_last;
  float* s_acc = reinterpret_cast<float*>(dec_smem_raw);      // [warp][head][DV + 4]
  constexpr int AS = DV + 4;
  if (t4 == 0) { s_m[warp][g] = m; s_l[warp][g] = l; }
#pragma unroll
  for (int d = 0; d < DV / 16; ++d)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      s_acc[(warp * kDecHeads + t4 * 2 + (e & 1)) * AS + d * 16 + g + (e >> 1) * 8] = o[d][e];
  __syncthreads();
  const int Hq = kv_heads * G;
  for (int idx = threadIdx.x; idx < G * DV; idx += WARPS * 32) {
    const int h = idx / DV, d = idx % DV;
    float mm = -INFINITY;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) mm = fmaxf(mm, s_m[w][h]);
    float ll = 0.f, a = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const float c = s_m[w][h] == -INFINITY ? 0.f : exp2f(s_m[w][h] - mm);
      ll += s_l[w][h] * c;
      a += s_acc[(w * kDecHeads + h) * AS + d] * c;
    }
    const int hq = hk * G + h;
    if (nsplit == 1) {
      out[(size_t)t * o_ld_t + (size_t)hq * DV + d] = __float2bfloat16_rn(ll > 0.f ? a / ll : 0.f);
    } else {
      const size_t pidx = ((size_t)t * Hq + hq) * nsplit + sp;
      if (mm != -INFINITY) part_acc[pidx * DV + d] = a;
      if (d == 0) { part_ml[pidx * 2] = mm; part_ml[pidx * 2 + 1] = ll; }
    }
  }
  if (nsplit == 1) return;
  // ---- the last split of this (token, kv head) to arrive merges them
  __syncthreads();
  if (threadIdx.x == 0) {                                     // the barriers on both sides and one thread's fences order the whole CTA's partials
    unsigned int* tk = tickets + (size_t)t * kv_heads + hk;
    __threadfence();
    const bool last = atomicAdd(tk, 1u) == (unsigned int)(nsplit - 1);
    __threadfence();
    if (last) *tk = 0u;                                       // for the next launch
    s_last = last;
  }
  __syncthreads();
  if (!s_last) return;
  float* s_w = s_acc;                                         // [G][nsplit] weight of every split, normalised
  if (threadIdx.x < G) {
    const float* ml = part_ml + (((size_t)t * Hq + hk * G + threadIdx.x) * nsplit) * 2;
    float mm = -INFINITY, ll = 0.f;
    for (int s = 0; s < nsplit; ++s) mm = fmaxf(mm, __ldcg(ml + 2 * s));
    for (int s = 0; s < nsplit; ++s) {
      const float ms = __ldcg(ml + 2 * s), c = ms == -INFINITY ? 0.f : exp2f(ms - mm);
      s_w[threadIdx.x * nsplit + s] = c;
      ll += __ldcg(ml + 2 * s + 1) * c;
    }
    s_l[0][threadIdx.x] = ll > 0.f ? 1.f / ll : 0.f;
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < G * DV; idx += WARPS * 32) {
    const int h = idx / DV, d = idx % DV;
    const float* pa = part_acc + (((size_t)t * Hq + hk * G + h) * nsplit) * DV + d;
    float a = 0.f;
#pragma unroll 8
    for (int s = 0; s < nsplit; ++s) {
      const float c = s_w[h * nsplit + s];
      if (c != 0.f) a += __ldcg(pa + (size_t)s * DV) * c;      // (a split without keys stored nothing)
    }
    out[(size_t)t * o_ld_t + (size_t)(hk * G + h) * DV + d] = __float2bfloat16_rn(a * s_l[0][h]);
  }
}

// Contexts of a few keys with one or two query heads per kv head: of the products above at most an eighth is useful, and a tile is always 16 keys.  Here lanes
// split the head dimension, a warp takes four keys at a time in registers, products are finished with shuffles, and nothing goes through shared memory
// but the merge of the four warps.  One split.
constexpr int kVecKeys = 4;
template <int DK, int DV, int G>
__global__ void __launch_bounds__(128)
paged_vector_kernel(const __nv_bfloat16* __restrict__ q, long long q_ld_t, long long q_ld_h, const __nv_bfloat16* __restrict__ kpool,
                    const __nv_bfloat16* __restrict__ vpool, const int* __restrict__ block_tables, int max_blocks, const int* __restrict__ positions,
                    const int* __restrict__ token_seq, int kv_heads, int page, float scale, float softcap, __nv_bfloat16* __restrict__ out, long long o_ld_t) {
  pdl_sync();  // PDL: predecessor's writes visible; let the successor start its prologue
  constexpr int PK = DK / 64, PV = DV / 64, WARPS = 4;          // bf16 pairs of a row that a lane holds
  const int t = blockIdx.x, hk = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kv_len = positions[t] + 1;
  const int* bt = block_tables + (size_t)token_seq[t] * max_blocks;
  float qf[G][2 * PK], m[G], l[G], acc[G][2 * PV];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const __nv_bfloat16* qp = q + (size_t)t * q_ld_t + (size_t)(hk * G + g) * q_ld_h;
#pragma unroll
    for (int i = 0; i < PK; ++i) {
      const uint32_t u = reinterpret_cast<const uint32_t*>(qp)[lane + 32 * i];
      qf[g][2 * i] = bf16_lo(u) * scale;
      qf[g][2 * i + 1] = bf16_hi(u) * scale;
    }
    m[g] = -INFINITY; l[g] = 0.f;
#pragma unroll
    for (int i = 0; i < 2 * PV; ++i) acc[g][i] = 0.f;
  }
  for (int base = warp * kVecKeys; base < kv_len; base += WARPS * kVecKeys) {
    uint32_t kreg[kVecKeys][PK], vreg[kVecKeys][PV];
#pragma unroll
    for (int j = 0; j < kVecKeys; ++j) {
      const int pos = min(base + j, kv_len - 1);                // behind the end: the last key, left out below
      const size_t row = ((size_t)bt[pos / page] * kv_heads + hk) * page + pos % page;
      const uint32_t* kp = reinterpret_cast<const uint32_t*>(kpool + row * DK);
      const uint32_t* vp = reinterpret_cast<const uint32_t*>(vpool + row * DV);
#pragma unroll
      for (int i = 0; i < PK; ++i) kreg[j][i] = kp[lane + 32 * i];
#pragma unroll
      for (int i = 0; i < PV; ++i) vreg[j][i] = vp[lane + 32 * i];
    }
#pragma unroll
    for (int j = 0; j < kVecKeys; ++j) {
#pragma unroll
      for (int g = 0; g < G; ++g) {
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < PK; ++i) {
          s += qf[g][2 * i] * bf16_lo(kreg[j][i]);
          s += qf[g][2 * i + 1] * bf16_hi(kreg[j][i]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (softcap > 0.f) s = softcap * tanhf(s / softcap);
        if (base + j < kv_len) {
          const float mn = fmaxf(m[g], s), corr = __expf(m[g] - mn), p = __expf(s - mn);
          l[g] = l[g] * corr + p;
#pragma unroll
          for (int i = 0; i < PV; ++i) {
            acc[g][2 * i] = acc[g][2 * i] * corr + p * bf16_lo(vreg[j][i]);
            acc[g][2 * i + 1] = acc[g][2 * i + 1] * corr + p * bf16_hi(vreg[j][i]);
          }
          m[g] = mn;
        }
      }
    }
  }
  __shared__ float s_m[WARPS][G], s_l[WARPS][G], s_acc[WARPS][G][DV];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    if (lane == 0) { s_m[warp][g] = m[g]; s_l[warp][g] = l[g]; }
#pragma unroll
    for (int i = 0; i < PV; ++i) {
      s_acc[warp][g][2 * (lane + 32 * i)] = acc[g][2 * i];
      s_acc[warp][g][2 * (lane + 32 * i) + 1] = acc[g][2 * i + 1];
    }
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < G * DV; idx += 128) {
    const int g = idx / DV, d = idx % DV;
    float mm = -INFINITY, ll = 0.f, a = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) mm = fmaxf(mm, s_m[w][g]);
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const float c = s_m[w][g] == -INFINITY ? 0.f : __expf(s_m[w][g] - mm);
      ll += s_l[w][g] * c;
      a += s_acc[w][g][d] * c;
    }
    out[(size_t)t * o_ld_t + (size_t)(hk * G + g) * DV + d] = __float2bfloat16_rn(ll > 0.f ? a / ll : 0.f);
  }
}

template <int DK, int DV, int G>
cudaError_t launch_vector(const PagedAttnArgs& a, cudaStream_t s) {
  (void)launch_pdl(paged_vector_kernel<DK, DV, G>, dim3(a.T, a.kv_heads), dim3(128), 0, s, static_cast<const __nv_bfloat16*>(a.q), a.q_ld_t, a.q_ld_h,
                   static_cast<const __nv_bfloat16*>(a.kpool), static_cast<const __nv_bfloat16*>(a.vpool), a.block_tables, a.max_blocks, a.positions,
                   a.token_seq, a.kv_heads, a.page, a.scale, a.softcap, static_cast<__nv_bfloat16*>(a.out), a.o_ld_t);
  return cudaGetLastError();
}

// Where the vector form is faster.  B200, us, vector / matrix form, by the bound of the contexts: one query head per kv head, 16 heads of 192 / 128, 1 token
// 2.2 / 2.7 (up to 16 keys; 17: 3.2 / 2.7), 8 tokens 2.4 / 2.8 (16; 17: 3.3 / 3.2), 64 tokens 3.0 / 3.7 (1), 3.9 / 3.8 (8), 5.1 / 3.8 (16), 256 tokens 8.5 / 11.1 (8), 11.7 / 11.1 (16),
// 1024 tokens 42.8 / 45.7 (16), 54.2 / 53.6 (17); 32 heads of 128, 1 token 2.3 / 2.5 (16), 8 tokens 2.5 / 2.7 (8), 2.8 / 2.6 (16), 64 tokens 4.9 / 5.0 (8), 256 tokens 11.7 / 12.9 (1), 14.1 / 12.9 (8);
// 16 heads of 256, 8 tokens 2.6 / 3.0 (16), 64 tokens 3.8 / 4.5 (8), 5.2 / 4.5 (16), 6.0 / 7.5 (17), 8.0 / 7.5 (32), 1024 tokens 71 / 77 (17), 96 / 90 (32); two query heads
// per kv head, 8 of 256, 64 tokens 4.3 / 4.5 (8), 5.0 / 4.5 (16), 256 tokens 10.6 / 8.4 (8).  Heads of 64 and larger groups: the matrix form is as fast or faster from one key on.
bool vector_form(int dk, int G, int max_ctx, long long pairs) {
  if (max_ctx <= 0 || max_ctx > 24) return false;
  if (G == 2 && dk == 256) return max_ctx <= 8 && pairs <= 512;
  if (G != 1 || dk < 128) return false;
  if (max_ctx <= 8) return dk > 128 || pairs <= 2048 || max_ctx <= 2;
  if (max_ctx <= 16) return pairs <= (dk > 128 ? 128 : 32) || (dk == 192 && pairs >= 8192);
  return dk == 256 && pairs >= 1024;
}

template <int DK, int DV, int WARPS, int STAGES>
cudaError_t launch_decode_ring(const PagedAttnArgs& a, cudaStream_t s) {
  constexpr int smem = dec_smem(DK, DV, WARPS, STAGES);
  auto kern = paged_decode_kernel<DK, DV, WARPS, STAGES>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    configured = true;
  }
  dim3 grid(a.T, a.kv_heads, a.nsplit);
  (void)launch_pdl(kern, grid, dim3(WARPS * 32), smem, s, static_cast<const __nv_bfloat16*>(a.q), a.q_ld_t, a.q_ld_h,
                   static_cast<const __nv_bfloat16*>(a.kpool), static_cast<const __nv_bfloat16*>(a.vpool), a.block_tables, a.max_blocks,
                   a.positions, a.token_seq, a.kv_heads, a.q_heads / a.kv_heads, a.page, a.scale, a.softcap, a.nsplit,
                   static_cast<__nv_bfloat16*>(a.out), a.o_ld_t, a.part_acc, a.part_ml, a.tickets);
  return cudaGetLastError();
}

// Short contexts: a warp of its own per (token, kv head) where that fills the chip or one tile is all there is (no merge of warps, three times the CTAs per SM);
// one tile per warp needs no ring.  B200, four warps with rings / this rule: Gemma-2-9B heads, 1024 tokens of up to 16 keys 73 / 26 us, 64 sequences of 100 keys
// 15.5 / 12.2; Llama-3-8B, 256 sequences of 64 keys 16.9 / 12.7, 1000 keys no gain.  Every form is right for any context; the rule is about time only.
template <int DK, int DV>
cudaError_t launch_decode(const PagedAttnArgs& a, cudaStream_t s) {
  if (a.max_ctx > 0 && a.max_ctx <= kDecKeys) return launch_decode_ring<DK, DV, 1, 1>(a, s);
  if (a.max_ctx > 0 && a.max_ctx <= 256 * a.nsplit && (long long)a.T * a.kv_heads * a.nsplit >= 512) return launch_decode_ring<DK, DV, 1, 2>(a, s);
  if (a.max_ctx > 0 && a.max_ctx <= kDecKeys * kDecWarps * a.nsplit) return launch_decode_ring<DK, DV, kDecWarps, 1>(a, s);
  return launch_decode_ring<DK, DV, kDecWarps, dec_stages(DK, DV)>(a, s);
}

}  // namespace

// Splits of the KV range.  A split costs a pair of (token, kv head) ~5 us, whatever its length (partials, a fence, the ticket, the merge), and a CTA ~5 us of start
// and end; four warps walk 64 keys in 0.6 us.  So contexts up to 768 keys stay whole, longer ones are cut into pieces of 256 keys (512 above 4096: fewer partials to merge) or more while the CTAs
// fit the chip in one round, and beyond one round only long contexts are cut (four rounds even ragged ones out).  B200, Llama-3-8B heads, before (64-key pieces
// to fill a round, 256-key pieces up to four) / this rule: 8 sequences of 127 keys 8.8 / 4.4 us, 511 16.6 / 8.6; 32 of 1000 45.8 / 23.1, 32 of 4000 103 / 81.7, of 1000 to
// 4000 70 / 61.0; 4 of 8000 66 / 30.7; one of 2000 18.6 / 11.1.
int paged_attention_splits(int T, int kv_heads, int dk, int dv, int max_ctx, int sms) {
  if (max_ctx <= 768) return 1;
  const long long pairs = (long long)T * kv_heads;
  const long long slots = (long long)sms * (dk + dv > 320 ? 1 : 2);   // heads of 256: one CTA per SM
  auto up = [](long long a, long long b) { return (a + b - 1) / b; };
  const long long one_round = std::min(slots / pairs, up(max_ctx, max_ctx <= 4096 ? 256 : 512)), four_rounds = std::min(up(4 * slots, pairs), up(max_ctx, dk + dv <= 128 ? 1024 : 16 * (dk + dv)));
  const long long n = std::max(one_round, four_rounds);
  return n < 1 ? 1 : n > 64 ? 64 : (int)n;
}

cudaError_t paged_attention_launch(const PagedAttnArgs& a, cudaStream_t s) {
  if (a.T == 0) return cudaSuccess;
  const uintptr_t kv = reinterpret_cast<uintptr_t>(a.kpool) | reinterpret_cast<uintptr_t>(a.vpool);
  if ((kv & 15) || (reinterpret_cast<uintptr_t>(a.q) & 3)) return cudaErrorInvalidValue;      // cp.async of 16 bytes; queries in pairs
  if ((a.q_ld_t % 2) || (a.q_ld_h % 2) || a.nsplit < 1 || a.nsplit > 64) return cudaErrorInvalidValue;
  if (a.nsplit > 1 && (a.part_acc == nullptr || a.part_ml == nullptr || a.tickets == nullptr)) return cudaErrorInvalidValue;
  const int G = a.q_heads / a.kv_heads;
  const bool pow2 = G == 1 || G == 2 || G == 4 || G == 8;
  if (a.nsplit == 1 && a.q_heads == G * a.kv_heads && vector_form(a.dk_, G, a.max_ctx, (long long)a.T * a.kv_heads)) {
    if (a.dk_ == 192 && a.dv_ == 128) return launch_vector<192, 128, 1>(a, s);
    if (a.dk_ == 128 && a.dv_ == 128) return launch_vector<128, 128, 1>(a, s);
    if (a.dk_ == 256 && a.dv_ == 256) return G == 1 ? launch_vector<256, 256, 1>(a, s) : launch_vector<256, 256, 2>(a, s);
  }
  if (a.dk_ == 192 && a.dv_ == 128 && G == 1) return launch_decode<192, 128>(a, s);       // DeepSeek-V2 MLA, decompressed cache
  if (a.dk_ == 128 && a.dv_ == 128 && pow2) return launch_decode<128, 128>(a, s);         // Llama-3-8B: 32 q heads / 8 kv heads
  if (a.dk_ == 256 && a.dv_ == 256 && pow2 && G <= 2) return launch_decode<256, 256>(a, s);   // Gemma-2-9B
  if (a.dk_ == 64 && a.dv_ == 64 && pow2 && G <= 4) return launch_decode<64, 64>(a, s);
  return cudaErrorNotSupported;
}

}  // namespace b200
