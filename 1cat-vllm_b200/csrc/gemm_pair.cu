// out[t, n] = sum_k X[t, k] * W[n, k], bf16, for many tokens: tcgen05 products over pairs of SMs.
//
// Two CTAs of a cluster work on one tile of 256 tokens x 256 output features (cta_group::2): each loads its 128 tokens and its 128 weight rows, and
// the product reads both halves of the weights from both SMs' shared memory. Per product an SM then reads 8 KB of operands from shared memory
// instead of the 12 KB that a 128 x 256 tile of its own takes (gemm_sm100.cu), and the pair loads a third less from L2: long products run under
// the power limit, where that is clock.
//   warp 0      producer: TMA copies of this CTA's halves; both CTAs' copies are counted by the first CTA's barrier
//   warp 1      MMA issue, in the first CTA of the pair only
//   warps 2-5   epilogue of this CTA's 128 tokens: a thread owns a token, its accumulator row holds neighbouring features, so gate and up rows
//               (interleaved in blocks of 16) meet inside a thread and results leave as 16-byte vectors without a transpose
// Two accumulators of 256 columns: the epilogue of a tile overlaps the products of the next. Tiles go out in groups of eight token tiles, feature
// tiles outside, so that what is in flight at a time shares both operands in L2.
// Every wait is bounded (see common.cuh); when a role gives up in one CTA, the other CTA's waits run out too, and both meet at the end.
// Bound by the tensor pipe (95 % busy), in long products by power. Measured against the single-CTA tiles of gemm_sm100.cu: 8192 x 34816 x 5120 1781 to
// 1858 us (1.57 to 1.64 PFLOP/s) for 2343, 1024 x 34816 x 5120 235 for 301, 8192 x 5120 x 5120 277 for 356, 300 x 16384 x 5120 83 for 114.
// (reference: cuBLAS for unquantised layers)
#include "common.cuh"
#include "gemm_sm100.h"

namespace oc {
namespace {

constexpr int kTok = 256, kFeat = 256;            // tile of the pair
constexpr int kHalfBytes = 128 * 128;             // 128 rows x 64 k of bf16
constexpr int kStage = 2 * kHalfBytes, kStages = 6;
constexpr int kThreads = 192;
constexpr int kSmem = kStages * kStage + 1024 + 1024;
constexpr int kWidenTokens = 1024;                // see gemm_widen_takes
constexpr int kGroup = 8;                         // token tiles of a group

// TMA copy into this CTA's shared memory, counted by a barrier of either CTA of the pair (a shared::cluster address)
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* tm, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(smem_u32(smem_dst)), "l"(tm), "r"(bar), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap* tm, int x, int y) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(tm), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void umma_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrives on the barrier at this offset in both CTAs once the products issued so far are done
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((uint16_t)3)
               : "memory");
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const GemmParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStages * kStage);
  uint64_t* full = bars;                  // [kStages] first CTA: both CTAs' operands of a stage are in place
  uint64_t* empty = full + kStages;       // [kStages] the products have read the stage
  uint64_t* tfull = empty + kStages;      // [2] accumulator complete
  uint64_t* tempty = tfull + 2;           // [2] first CTA: accumulator drained by both CTAs' epilogues
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank();

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], 8);           // one arrival per epilogue warp of the pair
    }
    *abort_flag = 0;
    mbar_fence_init();
    prefetch_tmap(&tmX);
    prefetch_tmap(&tmW);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                     // both CTAs' barriers exist before either is signalled from the other
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_trigger();
  pdl_wait();

  const int tt_all = p.num_t_tiles, nt_all = p.num_n_tiles, ktiles = p.K / 64;
  const int total = tt_all * nt_all, clusters = gridDim.x >> 1;
  auto decode = [&](int w, int& tt, int& nt) {
    const int g = w / (kGroup * nt_all), rows = min(kGroup, tt_all - g * kGroup), i = w - g * kGroup * nt_all;
    nt = i / rows;
    tt = g * kGroup + i - nt * rows;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    if (lane == 0) {
      Ring st;
      bool ok = true;
      for (int w = blockIdx.x >> 1; w < total && ok; w += clusters) {
        int tt, nt;
        decode(w, tt, nt);
        const int y0 = tt * kTok + rank * 128, y1 = nt * kFeat + rank * 128;
        // Rows of long k lie far apart, and a k tile at a time is 128 bytes from each: there the group's first pair brings the weights of eight k
        // tiles at a time to L2 (17408 k, 5120 features: 512 tokens 155 -> 130 us, 4096 685 -> 544; at 5120 k it costs 8 %, and at 8192
        // tokens the other operand sets the pace).
        const bool lead = p.K >= 8192 && tt_all <= 2 * kGroup && tt % kGroup == 0 && y1 < p.n_rows;   // a half past the rows has nothing to bring
        for (int kt = 0; kt < ktiles; ++kt) {
          if (lead && kt % 8 == 0) {
            const int k1 = min(kt + 16, ktiles);
            for (int k = kt == 0 ? 0 : kt + 8; k < k1; ++k) tma_prefetch_2d(&tmW, k * 64, y1);
          }
          ok = mbar_wait(&empty[st.idx], st.phase ^ 1, abort_flag);
          if (!ok) break;
          if (rank == 0) mbar_expect_tx(&full[st.idx], 2 * kStage);   // the other CTA's bytes too; they may land before this
          const uint32_t bar = mapa_shared(smem_u32(&full[st.idx]), 0);
          uint8_t* dst = smem + st.idx * kStage;
          tma_load_2d_pair(dst, &tmX, kt * 64, y0, bar);              // rows past the tensors are zero-filled
          tma_load_2d_pair(dst + kHalfBytes, &tmW, kt * 64, y1, bar);
          st.advance(kStages);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issue (uniform control flow, one elected lane)
    if (rank == 0) {
      const uint32_t idesc = umma_idesc_bf16(kTok, kFeat), base = smem_u32(smem);
      Ring st;
      uint32_t tile_i = 0;
      bool ok = true;
      for (int w = blockIdx.x >> 1; w < total && ok; w += clusters, ++tile_i) {
        const int acc = tile_i & 1;
        ok = mbar_wait_cluster(&tempty[acc], ((tile_i >> 1) & 1) ^ 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        for (int kt = 0; kt < ktiles; ++kt) {
          ok = mbar_wait(&full[st.idx], st.phase, abort_flag);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
            const uint64_t da = umma_desc_sw128(base + st.idx * kStage), db = umma_desc_sw128(base + st.idx * kStage + kHalfBytes);
#pragma unroll
            for (int j = 0; j < 4; ++j) umma_pair(tmem_base + acc * kFeat, da + (uint64_t)(j * 2), db + (uint64_t)(j * 2), idesc, (kt | j) ? 1u : 0u);
            umma_commit_pair(&empty[st.idx]);
            if (kt + 1 == ktiles) umma_commit_pair(&tfull[acc]);
          }
          __syncwarp();
          st.advance(kStages);
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue: one thread per token of this CTA's half
    const int q = warp & 3;               // TMEM lane quarter this warp may read
    const bool gated = p.epi == EPI_SILU_MUL || p.epi == EPI_GELU_MUL;
    uint32_t tile_i = 0;
    bool ok = true;
    for (int w = blockIdx.x >> 1; w < total && ok; w += clusters, ++tile_i) {
      int tt, nt;
      decode(w, tt, nt);
      const int acc = tile_i & 1;
      ok = mbar_wait(&tfull[acc], (tile_i >> 1) & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const int t = tt * kTok + rank * 128 + q * 32 + lane;
      const uint32_t taddr = tmem_base + acc * kFeat + ((uint32_t)(q * 32) << 16);
#pragma unroll 1
      for (int c = 0; c < kFeat; c += 32) {
        uint32_t v[32];
        tmem_ld_32x32(taddr + c, v);
        tmem_ld_wait();
        if (c + 32 == kFeat) {            // the accumulator is in registers: the next tile but one may start on it
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(&tempty[acc]), 0));
        }
        const int n0 = nt * kFeat + c;
        if (t >= p.T || n0 >= p.n_rows) continue;
        float a[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) a[i] = __uint_as_float(v[i]);
        if (gated) {
#pragma unroll
          for (int i = 0; i < 16; ++i) a[i] = (p.epi == EPI_SILU_MUL ? a[i] / (1.f + __expf(-a[i])) : gelu_tanh(a[i])) * a[16 + i];
        } else {
          if (p.bias != nullptr) {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (n0 + i < p.N) a[i] += __bfloat162float(p.bias[n0 + i]);
          }
          if (p.epi == EPI_GELU_TANH) {
#pragma unroll
            for (int i = 0; i < 32; ++i) a[i] = gelu_tanh(a[i]);
          }
        }
        const int o0 = gated ? n0 / 2 : n0, cnt = gated ? 16 : 32, lim = gated ? p.n_out : p.N;
        if (p.out_f32 != nullptr) {
          float* dst = p.out_f32 + (size_t)t * p.ldo + o0;
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (o0 + i < lim) dst[i] = a[i];
          continue;
        }
        __nv_bfloat16* dst = p.out + (size_t)t * p.ldo + o0;
        if (p.vec_ok && o0 + cnt <= lim) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            if (i >= cnt) break;
            uint32_t b[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const __nv_bfloat162 x = __floats2bfloat162_rn(a[i + 2 * e], a[i + 2 * e + 1]);
              b[e] = *reinterpret_cast<const uint32_t*>(&x);
            }
            *reinterpret_cast<uint4*>(dst + i) = make_uint4(b[0], b[1], b[2], b[3]);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (i < cnt && o0 + i < lim) dst[i] = __float2bfloat16(a[i]);
        }
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
  cluster_sync_all();                     // the other CTA may still signal this one's barriers or read its operands
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
  }
}

}  // namespace

// Takes more than 128 tokens (fewer leave half of a tile empty) with tiles for at least half of the pairs; below that the split k ranges of
// gemm_sm100.cu keep more SMs busy (256 tokens x 5120 x 17408, 20 tiles: 83 us; 300 tokens, 40 tiles: 138 there, 130 here).
bool gemm_pair_takes(const GemmParams& p, int num_sms) {
  if (p.work != nullptr || p.n_push != 0) return false;
  const long long tiles = (long long)((p.T + kTok - 1) / kTok) * ((p.n_rows + kFeat - 1) / kFeat);
  return p.T > 128 && tiles >= num_sms / 4;
}

int gemm_pair_launch(const GemmParams& p_in, const void* x, int ldx, const void* w, int ldw, int num_sms, cudaStream_t st) {
  GemmParams p = p_in;
  if (p.K % 64 || p.K <= 0) return -1;
  CUtensorMap tmX, tmW;
  if (make_tmap_bf16(&tmX, x, (uint64_t)p.T, (uint64_t)p.K, (uint64_t)ldx, 128)) return -2;
  if (make_tmap_bf16(&tmW, w, (uint64_t)p.n_rows, (uint64_t)p.K, (uint64_t)ldw, 128)) return -3;
  p.num_t_tiles = (p.T + kTok - 1) / kTok;
  p.num_n_tiles = (p.n_rows + kFeat - 1) / kFeat;
  p.vec_ok = p.out != nullptr && (p.ldo % 8 == 0) && ((uintptr_t)p.out & 15) == 0;
  static bool configured_dev[kMaxDevices] = {};
  bool& configured = configured_dev[current_device_slot()];  // the limit is an attribute of (kernel, device)
  if (!configured) {
    if (cudaFuncSetAttribute(gemm_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess) return -4;
    configured = true;
  }
  const long long total = (long long)p.num_t_tiles * p.num_n_tiles;
  const int clusters = (int)(total < num_sms / 2 ? total : num_sms / 2);
  if (launch_k(gemm_pair_kernel, dim3(2 * clusters), dim3(kThreads), (size_t)kSmem, st, true, tmX, tmW, p) != cudaSuccess) return -10;
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

// ---- packed weights, many tokens: rows [row0, row0 + rows) widened to bf16 [rows][K], a thread per eight neighbouring k. The numbers are those of
// the widening inside gemm_sm100.cu.
namespace {

template <int WKIND>
__global__ void __launch_bounds__(256) widen_kernel(const uint8_t* __restrict__ w, const uint32_t* __restrict__ sz, __nv_bfloat16* __restrict__ out, int row0,
                                                    int K, int n_pad, int gk) {
  constexpr int kTileBytes = WKIND == 2 ? 8192 : 4096, kScaleWords = WKIND == 4 ? 2 : 1, U = 4;
  pdl_trigger();
  pdl_wait();                             // the slab may still be read by the product before
  const int c = threadIdx.x & 7, local = blockIdx.x * 32 + (threadIdx.x >> 3), row = row0 + local, ktiles = K / 64;
  const int kt0 = blockIdx.y * U, rt = row & 127;
  const uint8_t* src = w + (size_t)(row >> 7) * ktiles * kTileBytes + (WKIND == 2 ? (c >> 1) * 2048 + rt * 16 + (c & 1) * 8 : (c >> 2) * 2048 + rt * 16 + (c & 3) * 4);
  uint32_t q[U][2], s[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int kt = min(kt0 + u, ktiles - 1);
    if constexpr (WKIND == 2) {
      const uint2 v = __ldcs(reinterpret_cast<const uint2*>(src + (size_t)kt * kTileBytes));
      q[u][0] = v.x;
      q[u][1] = v.y;
    } else {
      q[u][0] = __ldcs(reinterpret_cast<const uint32_t*>(src + (size_t)kt * kTileBytes));
    }
    s[u] = __ldg(sz + ((size_t)(kt / gk) * n_pad + row) * kScaleWords + (WKIND == 4 ? c >> 2 : 0));
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (kt0 + u >= ktiles) break;
    // the scale of these k: int4 and fp8 one per tile, MXFP4 one per half, NVFP4 one per two words
    const bool upper = WKIND == 3 ? c >= 4 : (WKIND == 4 ? (c & 2) : false);
    const uint32_t sc = upper ? __byte_perm(s[u], 0, 0x3232) : __byte_perm(s[u], 0, 0x1010), z = __byte_perm(s[u], 0, 0x3232);
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint32_t v;
      if constexpr (WKIND == 1) {
        const uint32_t x = ((q[u][0] >> (4 * i)) & 0x000f000fu) | 0x43004300u;
        const __nv_bfloat162 d = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&x), *reinterpret_cast<const __nv_bfloat162*>(&z));
        v = *reinterpret_cast<const uint32_t*>(&d);
      } else if constexpr (WKIND == 2) {
        const uint32_t t = __byte_perm(q[u][i >> 1], 0, (i & 1) ? 0x3424 : 0x1404);
        v = (t & 0x80008000u) | ((t >> 4) & 0x07f007f0u);
      } else {
        const uint32_t x = q[u][0] >> (4 * i);
        v = ((x & 0x00080008u) << 12) | ((x & 0x00070007u) << 6);
      }
      const __nv_bfloat162 r = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&v), *reinterpret_cast<const __nv_bfloat162*>(&sc));
      o[i] = *reinterpret_cast<const uint32_t*>(&r);
    }
    *reinterpret_cast<uint4*>(out + (size_t)local * K + (kt0 + u) * 64 + c * 8) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

}  // namespace

// Feature tiles of a slab and the whole product's estimated time in us. A pair of SMs takes 0.38 us per k tile, every slab about 15 us of its own
// (two launches, first copies, last tiles, the widening's tail), the widening moves 2.5 bytes a weight at 4 TB/s. Slabs are at most 192 MB.
namespace {
struct Slabs { int tiles; double us; };
Slabs plan_slabs(const GemmParams& p, int num_sms) {
  const int tt = (p.T + kTok - 1) / kTok, nt = (p.n_rows + kFeat - 1) / kFeat, pairs = num_sms / 2;
  const long long tile_bytes = (long long)kFeat * p.K * 2;
  Slabs best{1, 1e30};
  for (int n = 1; n <= nt && (n == 1 || n * tile_bytes <= (192ll << 20)); ++n) {
    const int slabs = (nt + n - 1) / n, rest = nt - (slabs - 1) * n;
    const long long waves = (long long)(slabs - 1) * ((n * tt + pairs - 1) / pairs) + (rest * tt + pairs - 1) / pairs;
    const double us = waves * (p.K / 64) * 0.38 + slabs * 15.0 + (double)p.n_rows * p.K * 2.5 / 4e6;
    if (us < best.us) best = {n, us};
  }
  return best;
}
}  // namespace

int gemm_widen_rows(const GemmParams& p, int num_sms) { return plan_slabs(p, num_sms).tiles * kFeat; }

// Packed weights and many tokens: widening them once and running the pairs of SMs at 1.6 PFLOP/s, or widening tile by tile on the way into tensor
// memory (gemm_sm100.cu, about 1.1 PFLOP/s: 0.72 us per k tile of 128 x 384, 0.45 of 128 x 192, and 20 us around them). The first only where
// these estimates say that it wins by 5 %. Measured (us), int4: 34816 x 5120 at 8192 tokens 1939 for 2730, at 1087 tokens 520 for 383 in small
// slabs; 5120 x 17408 at 1087 tokens 400 for 187.
bool gemm_widen_takes(const GemmParams& p, int num_sms) {
  if (p.w4 == nullptr || p.wkind < 1 || p.wkind > 4 || p.out == nullptr || p.out_f32 != nullptr || (p.epi != EPI_STORE && p.epi != EPI_SILU_MUL)) return false;
  if (p.T < kWidenTokens || !gemm_pair_takes(p, num_sms)) return false;
  const long long n = (p.n_rows + 127) / 128, w1 = (n * ((p.T + 191) / 192) + num_sms - 1) / num_sms, w2 = (n * ((p.T + 383) / 384) + num_sms - 1) / num_sms;
  const double one = w1 * 0.45, two = w2 * 0.72, tile_by_tile = (p.K / 64) * (one < two ? one : two) + 20.0;
  return plan_slabs(p, num_sms).us < 0.95 * tile_by_tile;
}

// The product over slabs of widened rows; `slab` holds gemm_widen_rows x K bf16.
int gemm_widen_launch(const GemmParams& p, const void* x, int ldx, void* slab, int num_sms, cudaStream_t st) {
  const int step = gemm_widen_rows(p, num_sms);
  const bool gated = p.epi == EPI_SILU_MUL || p.epi == EPI_GELU_MUL;
  for (int row0 = 0; row0 < p.n_rows; row0 += step) {
    const int rows = p.n_rows - row0 < step ? p.n_rows - row0 : step;
    const dim3 grid((rows + 31) / 32, (p.K / 64 + 3) / 4);   // rows past the last tile do not exist: a slab's rows end with it
    auto widen = [&](auto kernel) {
      return launch_k(kernel, grid, dim3(256), 0, st, true, p.w4, p.w4_sz, reinterpret_cast<__nv_bfloat16*>(slab), row0, p.K, p.n_pad, p.group_ktiles) == cudaSuccess;
    };
    const bool ok = p.wkind == 1 ? widen(widen_kernel<1>) : p.wkind == 2 ? widen(widen_kernel<2>) : p.wkind == 3 ? widen(widen_kernel<3>) : widen(widen_kernel<4>);
    if (!ok) return -10;
    GemmParams q = p;
    q.n_rows = rows;
    q.out = p.out + (gated ? row0 / 2 : row0);
    q.N = p.N - row0 < rows ? p.N - row0 : rows;
    q.n_out = p.n_out - row0 / 2;
    if (p.bias != nullptr) q.bias = p.bias + row0;
    const int rc = gemm_pair_launch(q, x, ldx, slab, p.K, num_sms, st);
    if (rc != 0) return rc;
  }
  return 0;
}

unsigned int* gemm_pair_status_word() { return status_word_tu(); }

}  // namespace oc
