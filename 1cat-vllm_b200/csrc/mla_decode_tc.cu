// Latent-attention decode on tcgen05 tensor cores (latents of 512, key part of up to 64): the absorbed form of mla.cu for 128 (head,
// query-token) rows at a time.
//
// Rows of one request's tokens and heads share the keys, so a CTA owns 128 of them, one split of the context and one half of the 256 + 256
// output columns:
//   S = Q K^T      tcgen05.mma over the whole row of 512 + 64, S [128 x 64 keys] in TMEM (fp32, double-buffered)
//   P = softmax    four warps, one thread per row; P replaces S in its TMEM columns as bf16
//   O += P V       operand A from TMEM, V = this CTA's 256 latent columns of the same key tile as an MN-major operand, O [128 x 256] in TMEM
// Both halves compute all scores (576 + 256 instead of 576 / 2 + 256 products per key): that keeps O in half of the tensor memory, where the
// whole of it would leave no room for S, and needs no exchange between CTAs. The second CTA's key tiles come from L2. The two sum a score in
// different orders, so one may take a new reference where the other keeps its own: each hands its (reference, sum) to the merge of the splits.
// Operand Q does not fit beside two key tiles (144 of 227 KB), so the 256 columns of it that meet this CTA's value columns live in TMEM, and
// the other 256 + 64 in shared memory. A key tile (64 keys, 72 KB) is loaded in two groups, each with barriers of its own: group A (the five
// column chunks only scores need) is free again after the scores, group B (the four chunks that are also values) after the value product.
// The accumulator is rescaled only when a row's maximum has grown by more than 2^8 since its reference (the sums are exact either way: the
// weights' reference cancels in the division), by the softmax warps, which then wait for the value products issued so far.
// Roles: warp 0 TMA producer, warp 1 MMA issue, warps 2-5 queries, softmax and epilogue. Every wait is bounded (see common.cuh).
//
// Bound: 128 x 64 x (576 + 256) = 6.8 M products per key tile and CTA, about 1980 cycles at 32 cycles per 128 x 64 x 16 product and 48 where operand
// A comes from shared memory (its reads then need 6 KB per instruction at 128 bytes a cycle). A tile takes about 4900: one softmax warp per scheduler and
// the tensor pipe (37 % busy) hand scores and weights to each other. Measured (kernel and merge): 32 requests x 4096 keys x 128 heads 99 us, two splits on
// 128 of 148 SMs, where the mma.sync kernel takes 730; the cache's 150 MB alone are 23 us of memory.
// (reference: csrc/attention/mla/sm100_cutlass_mla_kernel.cu)
#include "common.cuh"
#include "kernels.h"

namespace oc {
namespace {

constexpr int TM = 128;                      // rows of a CTA = UMMA M
constexpr int TK = 64;                       // keys per tile
constexpr int DV = 512, HV = DV / 2;         // latent width, output columns of a CTA
constexpr int kKChunk = TK * 128;            // bytes of 64 columns of a key tile
constexpr int kQChunk = TM * 128;
constexpr int kNA = 5, kNB = 4;              // column chunks of the two load groups (A: the other half of the latent, the key part)
constexpr int kStage = (kNA + kNB) * kKChunk;
constexpr int kSmem = kNA * kQChunk + 2 * kStage + 512 + 1024;   // queries, two key tiles, barriers, alignment
constexpr int kThreads = 192;
constexpr uint32_t kColO = 0, kColS = 256, kColQ = 384;          // TMEM columns: O | S0 | S1 | Q of group B
constexpr float kLazy = 8.f;                 // growth of a maximum (log2) that is left in the weights

// V as operand B, MN-major: 64 columns x 8 keys form a 1024-byte swizzle atom; the next 8 keys are 1024 bytes on, the next 64 columns a chunk on
__device__ __forceinline__ uint64_t desc_v(uint32_t smem_addr) { return umma_desc_sw128_mn(smem_addr, kKChunk); }

// element j of a rotated row (see mla.cu)
__device__ __forceinline__ float rotated(const __nv_bfloat16* x, int j, int n, const float* cs, int interleaved) {
  const int h = n / 2, i = interleaved ? j >> 1 : (j < h ? j : j - h);
  const bool second = interleaved ? (j & 1) : j >= h;
  const float u = __bfloat162float(x[interleaved ? 2 * i : i]), v = __bfloat162float(x[interleaved ? 2 * i + 1 : i + h]), c = cs[i], s = cs[h + i];
  return second ? v * c + u * s : u * c - v * s;
}

__global__ void __launch_bounds__(kThreads, 1)
mla_decode_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const MlaParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;                        // group A's chunks of the queries
  uint8_t* sK = smem + kNA * kQChunk;        // per stage: group A's chunks, group B's chunks
  uint64_t* bars = reinterpret_cast<uint64_t*>(sK + 2 * kStage);
  uint64_t* q_full = bars;                   // queries of group A by TMA
  uint64_t* q_ready = bars + 1;              // rotated part and TMEM columns written by the softmax warps
  uint64_t* full_a = bars + 2;               // [2]
  uint64_t* full_b = bars + 4;
  uint64_t* empty_a = bars + 6;
  uint64_t* empty_b = bars + 8;              // also: the value product of the tile is complete
  uint64_t* s_full = bars + 10;              // [2] scores complete
  uint64_t* p_ready = bars + 12;             // [2] weights written
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 14);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int half = blockIdx.x & 1, row0 = (blockIdx.x >> 1) * TM, r = blockIdx.y, split = blockIdx.z;
  pdl_trigger();
  pdl_wait();
  const int qs = p.query_start_loc[r], qlen = p.query_start_loc[r + 1] - qs, S = p.seq_lens[r];
  if (qlen <= 0 || S <= 0 || (p.skip_min_len > 0 && qlen >= p.skip_min_len)) return;
  const int total_rows = qlen * p.H;         // row = token * H + head
  if (row0 >= total_rows) return;
  const int nrows = min(TM, total_rows - row0);
  const int ctx0 = S - qlen;
  const int kv_end = min(S, ctx0 + (row0 + nrows - 1) / p.H + 1);
  const int ntiles = (kv_end + TK - 1) / TK;
  int lo = 0, hi = ntiles;
  if (p.splits > 1) {
    const int per = (ntiles + p.splits - 1) / p.splits;
    lo = min(split * per, ntiles);
    hi = min(ntiles, lo + per);
  }
  const int n = hi - lo;                     // tiles of this CTA
  if (n <= 0) {                              // an empty split: a sum of nothing (the merge skips its columns)
    if (threadIdx.x < nrows) {
      float* wm = p.ws_ml + (((size_t)split * p.T * p.H + (size_t)qs * p.H + row0 + threadIdx.x) * 2 + half) * 2;
      wm[0] = -INFINITY;
      wm[1] = 0.f;
    }
    return;
  }

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    mbar_init(q_ready, 4);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&full_a[i], 1);
      mbar_init(&full_b[i], 1);
      mbar_init(&empty_a[i], 1);
      mbar_init(&empty_b[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&p_ready[i], 4);
    }
    *abort_flag = 0;
    mbar_fence_init();
    prefetch_tmap(&tmQ);
    prefetch_tmap(&tmK);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int col_b = half * HV, col_a = HV - col_b;   // first latent column of group B (values) and of group A

  if (warp == 0) {
    // ------------------------------------------------------------------ producer: lane -> (chunk of 64 columns, 16 keys of the tile)
    if (lane == 0) {
      mbar_expect_tx(q_full, 4 * kQChunk);
      // rows past the end of the tensor are zero-filled; rows of other requests are computed and never stored
      for (int c = 0; c < 4; ++c) tma_load_2d(sQ + c * kQChunk, &tmQ, col_a + c * 64, qs * p.H + row0, q_full);
    }
    const int* bt = p.block_table + (size_t)r * p.bt_stride;
    const int piece = lane & 3;
    bool ok = true;
    for (int j = 0; j < n && ok; ++j) {
      const int s = j & 1;
      const uint32_t ph = ((j >> 1) & 1) ^ 1;
      const int key = (lo + j) * TK + piece * 16;    // pieces past the sequence lie past the tensor: the copy fills them with zeros
      const int row = key < S ? bt[key >> p.bs_shift] * p.bs + (key & (p.bs - 1)) : p.num_blocks * p.bs;
      uint8_t* dst = sK + s * kStage + piece * 2048;
      for (int g = 0; g < 2 && ok; ++g) {
        uint64_t* full = g == 0 ? &full_a[s] : &full_b[s];
        if (lane == 0) {
          ok = mbar_wait(g == 0 ? &empty_a[s] : &empty_b[s], ph, abort_flag);
          if (ok) mbar_expect_tx(full, (g == 0 ? kNA : kNB) * kKChunk);
        }
        ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
        if (!ok) break;
        const int c = lane >> 2;                     // lanes 0-15: the four latent chunks of the group, lanes 16-19: the key part
        if (g == 0 && c < kNA) tma_load_2d(dst + c * kKChunk, &tmK, c < 4 ? col_a + c * 64 : DV, row, full);
        if (g == 1 && c < kNB) tma_load_2d(dst + (kNA + c) * kKChunk, &tmK, col_b + c * 64, row, full);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issue (uniform control flow, one elected lane)
    const uint32_t idesc_qk = umma_idesc_bf16(TM, TK);
    const uint32_t idesc_pv = umma_idesc_bf16(TM, HV) | (1u << 16);   // operand B (V) is MN-major
    const uint32_t q_addr = smem_u32(sQ), k_addr = smem_u32(sK);
    bool ok = mbar_wait(q_full, 0, abort_flag);
    if (ok) ok = mbar_wait(q_ready, 0, abort_flag);
    ok = __all_sync(0xffffffffu, ok);
    auto scores = [&](int j) {
      const int s = j & 1;
      const uint32_t ph = (j >> 1) & 1;
      const uint32_t d = tmem_base + kColS + s * TK, ka = k_addr + s * kStage;
      ok = mbar_wait(&full_a[s], ph, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) return;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int c = 0; c < kNA; ++c) {
          const uint64_t da = umma_desc_sw128(q_addr + c * kQChunk), db = umma_desc_sw128(ka + c * kKChunk);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_bf16(d, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc_qk, (c | k) ? 1u : 0u);
        }
        umma_commit(&empty_a[s]);
      }
      __syncwarp();
      ok = mbar_wait(&full_b[s], ph, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) return;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int c = 0; c < kNB; ++c) {
          const uint64_t db = umma_desc_sw128(ka + (kNA + c) * kKChunk);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_bf16_ts(d, tmem_base + kColQ + c * 32 + k * 8, db + (uint64_t)(k * 2), idesc_qk, 1u);
        }
        umma_commit(&s_full[s]);
      }
      __syncwarp();
    };
    if (ok) scores(0);
    for (int j = 0; j < n && ok; ++j) {
      // S of tile j + 1 takes the columns of tile j - 1, whose value product was issued before (products run in order)
      if (j + 1 < n) scores(j + 1);
      if (!ok) break;
      const int s = j & 1;
      ok = mbar_wait(&p_ready[s], (j >> 1) & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        const uint32_t va = k_addr + s * kStage + kNA * kKChunk;
#pragma unroll
        for (int k = 0; k < TK / 16; ++k)
          umma_bf16_ts(tmem_base + kColO, tmem_base + kColS + s * TK + k * 8, desc_v(va + k * 2048), idesc_pv, (j | k) ? 1u : 0u);
        umma_commit(&empty_b[s]);
      }
      __syncwarp();
    }
  } else {
    // ------------------------------------------------------------------ queries, softmax, epilogue: one thread per row
    const int q4 = warp & 3, row = q4 * 32 + lane;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(q4 * 32) << 16);
    const int gr = row0 + row, tok = gr / p.H, hd = gr - tok * p.H;
    const bool live = row < nrows;
    const size_t orow = (size_t)qs * p.H + gr;
    // the rotated part -> shared memory (128-byte swizzle), zeros past its width and for rows past the end
    {
      const __nv_bfloat16* x = reinterpret_cast<const __nv_bfloat16*>(p.q_rope) + (size_t)(qs + tok) * p.qr_st + (size_t)hd * p.qr_sh;
      const float* cs = p.cos_sin != nullptr && live ? p.cos_sin + (size_t)(ctx0 + tok) * p.rope : nullptr;
      const uint32_t base = smem_u32(sQ) + 4 * kQChunk + row * 128;
#pragma unroll 1
      for (int c = 0; c < 8; ++c) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float v[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int j = c * 8 + i * 2 + e;
            v[e] = !live || j >= p.rope ? 0.f : (cs != nullptr ? rotated(x, j, p.rope, cs, p.interleaved) : __bfloat162float(x[j]));
          }
          const __nv_bfloat162 b = __floats2bfloat162_rn(v[0], v[1]);
          w[i] = *reinterpret_cast<const uint32_t*>(&b);
        }
        sts128(base + ((c ^ (row & 7)) << 4), make_uint4(w[0], w[1], w[2], w[3]));
      }
      fence_proxy_async_smem();
    }
    // group B's query columns -> TMEM
    {
      const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(p.q_abs) + orow * DV + col_b);
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t w[32];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint4 v = live ? src[c * 8 + i] : make_uint4(0, 0, 0, 0);
          w[4 * i] = v.x;
          w[4 * i + 1] = v.y;
          w[4 * i + 2] = v.z;
          w[4 * i + 3] = v.w;
        }
        tmem_st_32x32(lane_addr + kColQ + c * 32, w);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(q_ready);
    }
    const float sl2 = p.scale * 1.4426950408889634f;
    const int limit = live ? min(S, ctx0 + tok + 1) : kv_end;   // keys [0, limit) are visible to this row
    float m = -INFINITY, l = 0.f;            // reference of the weights (a maximum of some tile so far), their sum
    bool ok = true;
    for (int j = 0; j < n && ok; ++j) {
      const int s = j & 1, k0 = (lo + j) * TK;
      const uint32_t s_addr = lane_addr + kColS + s * TK;
      ok = mbar_wait(&s_full[s], (j >> 1) & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      uint32_t v[2][32];
      tmem_ld_32x32(s_addr, v[0]);
      tmem_ld_32x32(s_addr + 32, v[1]);
      tmem_ld_wait();
      if (k0 + TK > limit) {
#pragma unroll
        for (int i = 0; i < TK; ++i)
          if (k0 + i >= limit) v[i >> 5][i & 31] = 0xff800000u;
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < TK; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(v[i >> 5][i & 31]));
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * sl2;
      const bool grown = mx > m + kLazy || m == -INFINITY;
      float alpha = 1.f;
      if (grown && mx != -INFINITY) {
        alpha = m == -INFINITY ? 0.f : ex2(m - mx);
        m = mx;
        l *= alpha;
      }
      if (j > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
        // the products of tile j - 1 are the last that were issued: once they are done, this warp's rows of O are its own
        ok = mbar_wait(&empty_b[s ^ 1], ((j - 1) >> 1) & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < HV; c += 32) {
          uint32_t o[32];
          tmem_ld_32x32(lane_addr + kColO + c, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_st_32x32(lane_addr + kColO + c, o);
        }
      }
      const float m_use = m == -INFINITY ? 0.f : m;
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
      uint32_t pk[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const float a = ex2(fmaf(__uint_as_float(v[i >> 4][(2 * i) & 31]), sl2, -m_use)), b = ex2(fmaf(__uint_as_float(v[i >> 4][(2 * i + 1) & 31]), sl2, -m_use));
        sum[i & 3] += a + b;
        const __nv_bfloat162 w = __floats2bfloat162_rn(a, b);
        pk[i] = *reinterpret_cast<const uint32_t*>(&w);
      }
      l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
      tmem_st_32x32(s_addr, pk);
      if (k0 + TK > S && (S & 15)) {
        // the rest of the sequence's last page may hold anything: weights of zero must meet zeros. The scores have read the tile (s_full),
        // the value product waits for p_ready.
        const int first = S - k0, rows = 16 - (S & 15);
        const uint32_t base = smem_u32(sK) + s * kStage + kNA * kKChunk + first * 128;
        for (int i = threadIdx.x - 64; i < rows * kNB * 8; i += 128) sts128(base + (i / (rows * 8)) * kKChunk + (i % (rows * 8)) * 16, make_uint4(0, 0, 0, 0));
        fence_proxy_async_smem();
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_ready[s]);
    }
    if (ok) ok = mbar_wait(&empty_b[(n - 1) & 1], ((n - 1) >> 1) & 1, abort_flag);
    ok = __all_sync(0xffffffffu, ok);
    if (ok) {
      tc_fence_after();
      const bool part = p.splits > 1;
      float inv = 1.f;
      if (!part && live) {
        const float den = l + (p.sinks != nullptr ? ex2(p.sinks[hd] * 1.4426950408889634f - m) : 0.f);
        const float gate = p.gate != nullptr
                               ? 1.f / (1.f + expf(-__bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p.gate)[(size_t)(qs + tok) * p.gate_st + hd])))
                               : 1.f;
        inv = den > 0.f ? gate / den : 0.f;
      }
      float* wo = part ? p.ws_o + ((size_t)split * p.T * p.H + orow) * DV + col_b : nullptr;
      __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.out) + orow * DV + col_b;
#pragma unroll 1
      for (int c = 0; c < HV; c += 32) {
        uint32_t o[32];
        tmem_ld_32x32(lane_addr + kColO + c, o);
        tmem_ld_wait();
        if (!live) continue;
        if (part) {
#pragma unroll
          for (int i = 0; i < 32; i += 4) *reinterpret_cast<uint4*>(wo + c + i) = make_uint4(o[i], o[i + 1], o[i + 2], o[i + 3]);
        } else {
          uint32_t w[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const __nv_bfloat162 b = __floats2bfloat162_rn(__uint_as_float(o[2 * i]) * inv, __uint_as_float(o[2 * i + 1]) * inv);
            w[i] = *reinterpret_cast<const uint32_t*>(&b);
          }
#pragma unroll
          for (int i = 0; i < 16; i += 4) *reinterpret_cast<uint4*>(dst + c + 2 * i) = make_uint4(w[i], w[i + 1], w[i + 2], w[i + 3]);
        }
      }
      if (part && live) {                      // of this half: the other CTA may have another reference
        float* wm = p.ws_ml + (((size_t)split * p.T * p.H + orow) * 2 + half) * 2;
        wm[0] = m;
        wm[1] = l;
      }
    }
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) {
    // give copies that are still in flight a bounded chance to land before the CTA's shared memory is released
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) {}
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace

// What this kernel can run: DeepSeek's latent width, weights in one term, pages of whole 16-key pieces (a TMA box) and positive scales
// (the maximum is taken before scaling). Callers choose (plan_mla in ops/cuda.py): with 16 rows of heads a request seven eighths of a tile are
// padding and it is mostly still the faster one (32 requests x 4096 keys: 89 us against 122; one request x 1000 keys: 30 against 46), since the
// tensor core reads a key tile once where mma.sync kept four warps busy with fragments.
bool mla_decode_tc_takes(int kv_lora, int rope_pad, int bs, int fine, float scale) {
  return kv_lora == DV && rope_pad <= 64 && rope_pad % 8 == 0 && !fine && scale > 0.f && bs >= 16 && (bs & (bs - 1)) == 0;
}

int mla_decode_tc_launch(const MlaParams& p, cudaStream_t st) {
  if (((uintptr_t)p.q_abs & 15) || ((uintptr_t)p.cache & 15) || ((uintptr_t)p.out & 15) || p.num_blocks <= 0) return -1;
  CUtensorMap tmQ, tmK;
  if (make_tmap_bf16(&tmQ, p.q_abs, (uint64_t)p.T * p.H, DV, DV, TM)) return -2;
  if (make_tmap_bf16(&tmK, p.cache, (uint64_t)p.num_blocks * p.bs, (uint64_t)(DV + p.rope_pad), (uint64_t)(DV + p.rope_pad), 16)) return -3;
  static bool configured_dev[kMaxDevices] = {};
  bool& configured = configured_dev[current_device_slot()];  // the limit is an attribute of (kernel, device)
  if (!configured) {
    if (cudaFuncSetAttribute(mla_decode_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess) return -4;
    configured = true;
  }
  const dim3 grid(2 * (unsigned)(((long long)p.max_q_len * p.H + TM - 1) / TM), p.R, p.splits);
  return launch_k(mla_decode_tc_kernel, grid, dim3(kThreads), (size_t)kSmem, st, true, tmQ, tmK, p) == cudaSuccess ? 0 : -5;
}

unsigned int* mla_decode_tc_status_word() { return status_word_tu(); }

}  // namespace oc
