// Paged flash-attention prefill on tcgen05 tensor cores (head size 128, causal with prefix, GQA).
//
// One CTA owns 256 consecutive query tokens of one request for one query head, as two tiles of 128, and walks the keys in tiles of 128:
//   S_w = Q_w K^T    tcgen05.mma, both operands in shared memory (TMA, 128-byte swizzle), S_w in TMEM (fp32)
//   P_w = softmax    four warps per tile, one thread per query row: tcgen05.ld of the row's 128 scores, running maximum and sum in registers;
//                    P_w replaces S_w in its TMEM columns as bf16
//   O_w += P_w V     operand A from TMEM, V as an MN-major shared-memory operand straight from the paged cache layout [key][d]; O_w in TMEM
// The two tiles take turns: while one's scores are exponentiated the tensor pipe multiplies the other's, and both read every key tile from one copy
// in shared memory. The products of a tile are issued value product first, next scores second, so scores that have arrived mean that the
// accumulator is at rest; a row whose maximum has grown by more than 2^8 since its reference rescales it then (smaller growth stays in
// the weights: their reference cancels in the division). Query tiles go out longest first, all heads of a tile together.
// Bound: 1024 tensor cycles per 128 x 128 tile, and as many for its 16384 exponentials at 16 a cycle. Measured: 8192
// tokens x 40 heads 650 us (1.06 PFLOP/s; one tile of 128 rows per CTA with its results summed in registers took 1520); a prompt of 1024 tokens
// 47 us for 63. Handing the weights over in two halves, so that the value product starts earlier, was no faster.
// Roles: warp 0 = TMA producer (the 16 page loads of a K or V tile are issued by 16 lanes at once), warp 1 = MMA issue, warps 2-5 and 6-9 =
// softmax and epilogue of the two query tiles.
// Every wait is bounded; on expiry the CTA raises the status word and tears down (see common.cuh).
//
// Role in the reference's terms: the paged prefill of Flash-V100 / FA2 (reference: flash-attention-v100/kernel/
// fused_mha_forward_paged.cu:364,3297; vllm/v1/attention/backends/flash_attn.py) for D = 128; D = 256 stays on the mma.sync kernel.
#include "common.cuh"
#include "kernels.h"

namespace oc {

namespace {

constexpr int TQ = 128;   // query rows per tile = UMMA M; two tiles per CTA
constexpr int TK = 128;   // keys per tile = UMMA N of S and the k extent of P V
constexpr int HD = 128;   // head size
constexpr int kHalf = TK * 128;          // bytes of one 64-column half of a 128-row operand tile (rows of 128 bytes)
constexpr int kTile = 2 * kHalf;         // 32 KB: one Q tile, one K tile, or one V tile
constexpr int kSlots = 5;                // ring of K0, V0, K1, V1, ...
constexpr int kSmem = (2 + kSlots) * kTile + 1024;
constexpr int kThreads = 320;
constexpr uint32_t kColS = 0, kColO = 256;   // TMEM columns: S0 | S1 | O0 | O1
constexpr float kLazy = 8.f;             // growth of a maximum (log2) that is left in the weights

// two fp32 operations in one instruction
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 x, y, z, w;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\tfma.rn.f32x2 w, x, y, z;\n\tmov.b64 {%0, %1}, w;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 x, y, w;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.f32x2 w, x, y;\n\tmov.b64 {%0, %1}, w;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// V tile as UMMA operand B, MN-major (d contiguous): 64 d-values x 8 keys form a 1024-byte swizzle atom; the next 8 keys are
// 1024 bytes on (stride byte offset), the next 64 d-values are in the other half of the tile (leading byte offset).
__device__ __forceinline__ uint64_t umma_desc_sw128_mn(uint32_t smem_addr, uint32_t lbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

__global__ void __launch_bounds__(kThreads, 1)
attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmKV, const AttnParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sKV = smem + 2 * kTile;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (2 + kSlots) * kTile);
  uint64_t* q_full = bars;                // [2]
  uint64_t* full = q_full + 2;            // [kSlots]
  uint64_t* empty = full + kSlots;        // [kSlots]
  uint64_t* s_full = empty + kSlots;      // [2] scores complete (and the value product before them)
  uint64_t* p_ready = s_full + 2;         // [2] weights written
  uint64_t* o_full = p_ready + 2;         // [2] the last value product is complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* s_req = const_cast<int*>(reinterpret_cast<volatile int*>(tmem_slot + 2));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = blockIdx.x;
  const int G = p.Hq / p.Hkv;
  const int hkv = h / G;

  if (threadIdx.x == 0) {
    // which request and which 256 of its tokens this CTA owns (short queries belong to the decode kernel)
    int b = p.num_q_tiles - 1 - blockIdx.y, found = -1, t0 = 0;
    for (int i = 0; i < p.R; ++i) {
      const int ql = p.query_start_loc[i + 1] - p.query_start_loc[i];
      const int nt = (ql > p.short_q_len) ? (ql + 2 * TQ - 1) / (2 * TQ) : 0;
      if (b < nt) { found = i; t0 = b * 2 * TQ; break; }
      b -= nt;
    }
    s_req[0] = found;
    s_req[1] = t0;
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&p_ready[i], 4);
      mbar_init(&o_full[i], 1);
    }
    for (int i = 0; i < kSlots; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    *abort_flag = 0;
    mbar_fence_init();
    prefetch_tmap(&tmQ);
    prefetch_tmap(&tmKV);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int r = s_req[0], tq0 = s_req[1];

  // key tiles that the two query tiles walk: the last row of a tile sees the keys up to its own position; a tile past the query has none
  int nt0 = 0, nt1 = 0, qs = 0, qlen = 0, S = 0, ctx0 = 0;
  if (r >= 0) {
    qs = p.query_start_loc[r];
    qlen = p.query_start_loc[r + 1] - qs;
    S = p.seq_lens[r];
    ctx0 = S - qlen;
    nt0 = (min(S, ctx0 + min(tq0 + TQ, qlen)) + TK - 1) / TK;
    if (tq0 + TQ < qlen) nt1 = (min(S, ctx0 + min(tq0 + 2 * TQ, qlen)) + TK - 1) / TK;
  }
  const int ntiles = max(nt0, nt1);

  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    if (ntiles > 0) {
      if (lane == 0) {
        for (int w = 0; w < (nt1 > 0 ? 2 : 1); ++w) {
          mbar_expect_tx(&q_full[w], kTile);
          // rows past the end of the tensor are zero-filled; rows of the next request are loaded and never stored
          tma_load_2d(sQ + w * kTile, &tmQ, h * HD, qs + tq0 + w * TQ, &q_full[w]);
          tma_load_2d(sQ + w * kTile + kHalf, &tmQ, h * HD + 64, qs + tq0 + w * TQ, &q_full[w]);
        }
      }
      const int* bt = p.block_table + (size_t)r * p.bt_stride;
      // lane -> (column half, 16-key chunk)
      const int half = (lane >> 3) & 1, chunk = lane & 7;
      Ring st;
      bool ok = true;
      for (int j = 0; j < 2 * ntiles && ok; ++j) {   // K and V tiles in turn
        const int is_v = j & 1, key0 = (j >> 1) * TK + chunk * 16;
        int page = 0, off = 0;  // keys past the sequence read the null block
        if (key0 < S) {
          page = bt[key0 >> p.bs_shift];
          off = key0 & (p.bs - 1);
        }
        const int row = ((page * 2 + is_v) * p.Hkv + hkv) * p.bs + off;
        if (lane == 0) {
          ok = mbar_wait(&empty[st.idx], st.phase ^ 1, abort_flag);
          if (ok) mbar_expect_tx(&full[st.idx], kTile);
        }
        ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
        if (!ok) break;
        if (lane < 16) tma_load_2d(sKV + st.idx * kTile + half * kHalf + chunk * 2048, &tmKV, half * 64, row, &full[st.idx]);
        st.advance(kSlots);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issue (uniform control flow, one elected lane)
    if (ntiles > 0) {
      const uint32_t idesc_qk = umma_idesc_bf16(TQ, TK);
      const uint32_t idesc_pv = umma_idesc_bf16(TQ, HD) | (1u << 16);  // operand B (V) is MN-major
      const uint32_t q_addr = smem_u32(sQ), kv_addr = smem_u32(sKV);
      bool ok = true;
      auto wait = [&](uint64_t* bar, uint32_t parity) {
        if (ok) ok = mbar_wait(bar, parity, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
      };
      // tile index of the ring (K of j: 2 j, V of j: 2 j + 1) -> slot and parity
      auto slot_of = [](int i) { return i % kSlots; };
      auto parity_of = [](int i) { return (uint32_t)((i / kSlots) & 1); };
      auto issue_qk = [&](int w, int j, bool last) {   // last: no other product reads this K tile
        const int s = slot_of(2 * j);
        wait(&full[s], parity_of(2 * j));
        if (!ok) return;
        tc_fence_after();
        if (elect_one()) {
          const uint32_t d = tmem_base + kColS + w * TK, qa = q_addr + w * kTile, ka = kv_addr + s * kTile;
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
            const uint64_t da = umma_desc_sw128(qa + hf * kHalf), db = umma_desc_sw128(ka + hf * kHalf);
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) umma_bf16(d, da + (uint64_t)(jj * 2), db + (uint64_t)(jj * 2), idesc_qk, (hf | jj) ? 1u : 0u);
          }
          umma_commit(&s_full[w]);
          if (last) umma_commit(&empty[s]);
        }
        __syncwarp();
      };
      wait(&q_full[0], 0);
      if (nt1 > 0) wait(&q_full[1], 0);
      if (ok) issue_qk(0, 0, nt1 == 0);
      if (ok && nt1 > 0) issue_qk(1, 0, true);
      for (int j = 0; j < ntiles && ok; ++j) {
        const int s = slot_of(2 * j + 1);
#pragma unroll
        for (int w = 0; w < 2; ++w) {
          const int n = w == 0 ? nt0 : nt1, other = w == 0 ? nt1 : nt0;
          if (j >= n) continue;
          wait(&p_ready[w], j & 1);
          wait(&full[s], parity_of(2 * j + 1));
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
            const uint32_t va = kv_addr + s * kTile, pa = tmem_base + kColS + w * TK;
#pragma unroll
            for (int jj = 0; jj < TK / 16; ++jj)   // 16 keys per MMA: 8 TMEM columns of P, two 8-key groups (2048 bytes) of V
              umma_bf16_ts(tmem_base + kColO + w * HD, pa + jj * 8, umma_desc_sw128_mn(va + jj * 2048, kHalf), idesc_pv, (j | jj) ? 1u : 0u);
            if (w == 1 || j >= other) umma_commit(&empty[s]);
            if (j + 1 == n) umma_commit(&o_full[w]);
          }
          __syncwarp();
          if (j + 1 < n) issue_qk(w, j + 1, w == 1 || j + 1 >= other);
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax + epilogue: one thread per query row
    const int q4 = warp & 3;                 // TMEM lane quarter this warp may touch
    const int w = (warp - 2) >> 2;           // query tile
    const int row = q4 * 32 + lane;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(q4 * 32) << 16);
    const uint32_t s_addr = lane_addr + kColS + w * TK, o_addr = lane_addr + kColO + w * HD;
    const float sl2 = p.scale * 1.4426950408889634f;
    const int tq = tq0 + w * TQ + row;              // query token inside the request
    const int limit = min(S, ctx0 + tq + 1);        // keys [0, limit) are visible to this row
    const int limit0 = __shfl_sync(0xffffffffu, limit, 0);   // the warp's smallest
    const int n = w == 0 ? nt0 : nt1;
    float m = -INFINITY, l = 0.f;            // reference of the weights (a maximum of some tile so far), their sum
    bool ok = true;
    for (int j = 0; j < n && ok; ++j) {
      ok = mbar_wait(&s_full[w], j & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      uint32_t v[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32(s_addr + c * 32, v[c]);
      tmem_ld_wait();
      const int k0 = j * TK;
      if (k0 + TK > limit0) {
#pragma unroll
        for (int i = 0; i < TK; ++i)
          if (k0 + i >= limit) v[i >> 5][i & 31] = 0xff800000u;
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < TK; i += 2) mx4[(i >> 1) & 3] = fmaxf(mx4[(i >> 1) & 3], fmaxf(__uint_as_float(v[i >> 5][i & 31]), __uint_as_float(v[i >> 5][(i + 1) & 31])));
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * sl2;
      float alpha = 1.f;
      if (mx != -INFINITY && (m == -INFINITY || mx > m + kLazy)) {
        alpha = m == -INFINITY ? 0.f : ex2(m - mx);
        m = mx;
        l *= alpha;
      }
      if (j > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
#pragma unroll 1
        for (int c = 0; c < HD; c += 16) {
          uint32_t o[16];
          tmem_ld_32x16(o_addr + c, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_st_32x16(o_addr + c, o);
        }
      }
      const float m_use = m == -INFINITY ? 0.f : m;   // a row that sees no key yet keeps zeros
      const float2 sc = make_float2(sl2, sl2), off = make_float2(-m_use, -m_use);
      float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float2 y = fma2(make_float2(__uint_as_float(v[c][2 * i]), __uint_as_float(v[c][2 * i + 1])), sc, off);
          const __nv_bfloat162 b = __floats2bfloat162_rn(ex2(y.x), ex2(y.y));
          pk[i] = *reinterpret_cast<const uint32_t*>(&b);
          sum[i & 1] = add2(sum[i & 1], make_float2(__uint_as_float(pk[i] << 16), __uint_as_float(pk[i] & 0xffff0000u)));   // what the tensor core will multiply
        }
        tmem_st_32x16(s_addr + c * 16, pk);
      }
      l += (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_ready[w]);
    }
    if (n > 0 && ok) {
      ok = mbar_wait(&o_full[w], 0, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
    }
    if (n > 0 && ok) {
      tc_fence_after();
      const float inv = l > 0.f ? 1.f / l : 0.f;
      const size_t orow = (size_t)(qs + tq) * p.Hq + h;
#pragma unroll
      for (int c = 0; c < HD; c += 32) {
        uint32_t o[32];
        tmem_ld_32x32(o_addr + c, o);
        tmem_ld_wait();
        if (tq < qlen) {
          uint4* dst = reinterpret_cast<uint4*>(p.out + orow * HD + c);
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            uint32_t b[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const __nv_bfloat162 x = __floats2bfloat162_rn(__uint_as_float(o[i + 2 * e]) * inv, __uint_as_float(o[i + 2 * e + 1]) * inv);
              b[e] = *reinterpret_cast<const uint32_t*>(&x);
            }
            dst[i >> 3] = make_uint4(b[0], b[1], b[2], b[3]);
          }
        }
      }
      if (p.lse != nullptr && tq < qlen) p.lse[orow] = (m + log2f(l)) * 0.6931471805599453f;
    }
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) {
    // give copies that are still in flight a bounded chance to land before the CTA's shared memory is released
    uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) {}
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres);
    fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}

// bf16 [rows][cols] with a row pitch in bytes -> boxes of {64 columns, box_rows rows}, 128-byte swizzle, zero fill
int make_tmap(CUtensorMap* tm, const void* base, uint64_t rows, uint64_t cols, uint64_t pitch_bytes, uint32_t box_rows) {
  EncodeTiledFn enc = get_encode_fn();
  if (!enc) return -1;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {pitch_bytes};
  cuuint32_t box[2] = {64, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : (int)r;
}

}  // namespace

// Prefill attention of every request with more than `short_q_len` query tokens. `num_q_tiles` = sum over those requests of
// ceil(q_len / 256); `num_blocks` = pages in the cache. Needs D == 128, the heads of a token contiguous in q (q_sh == D),
// 16-byte aligned bases and pitches, and a positive scale (maxima are taken and keys masked ahead of it).
int attention_prefill_tc_launch(const AttnParams& p, long long num_blocks, cudaStream_t st) {
  if (p.D != HD || p.q_sh != HD || !(p.scale > 0.f) || p.Hq % p.Hkv || p.bs < 16 || (p.bs & (p.bs - 1))) return -1;
  if (((uintptr_t)p.q & 15) || ((uintptr_t)p.kv_cache & 15) || ((uintptr_t)p.out & 15) || (p.q_st * 2) % 16) return -1;
  if (p.num_q_tiles <= 0) return 0;
  if (p.num_q_tiles > 65535) return -1;
  CUtensorMap tmQ, tmKV;
  if (make_tmap(&tmQ, p.q, (uint64_t)p.T, (uint64_t)p.Hq * HD, (uint64_t)p.q_st * 2, TQ)) return -2;
  if (make_tmap(&tmKV, p.kv_cache, (uint64_t)num_blocks * 2 * p.Hkv * p.bs, HD, HD * 2, 16)) return -3;
  static bool configured_dev[kMaxDevices] = {};
  bool& configured = configured_dev[current_device_slot()];  // the limit is an attribute of (kernel, device)
  if (!configured) {
    if (cudaFuncSetAttribute(attn_prefill_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem + 1024) != cudaSuccess) return -4;
    configured = true;
  }
  dim3 grid(p.Hq, p.num_q_tiles);   // at most 65535 tiles of 256 tokens
  attn_prefill_tc_kernel<<<grid, kThreads, kSmem + 1024, st>>>(tmQ, tmKV, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

unsigned int* attention_tc_status_word() { return status_word_tu(); }

}  // namespace oc
