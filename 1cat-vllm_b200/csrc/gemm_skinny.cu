// out[t, n] = sum_k X[t, k] * W[n, k] for a handful of tokens and packed weights (int4, fp8, MXFP4, NVFP4 in the tile layouts of gemm_sm100.cu).
//
// What bounds it is reading the weights once. On the tcgen05 path a 4-bit tile passes through shared memory, registers and tensor memory,
// under two barriers, before a product whose 32 or 64 columns are mostly padding: about 600 cycles per 128 x 64 tile and SM where memory
// needs 185. Here a warp widens its weights in registers, in the very layout of a mma.sync operand, and multiplies from there:
//   * a unit is 64 packed bytes of each of a warp's 32 rows: 128 k of a 4-bit kind, 64 k of fp8. Lane (g, t) of the warp takes the 16 bytes of
//     quarter t of rows g, g + 8, ...: pairs of neighbouring k, which are elements a0 / a2 (a1 / a3) of eight (four) m16n8k16 steps. The order of
//     k inside a step is free as long as both operands agree, so operand B of these steps is one run of bytes of an activation row.
//   * every warp has a ring of units of its own (weights, scale words, activations) that cp.async fills: no barriers between warps, and the
//     bytes in flight take no registers.
//   * weights widen to the same bf16 numbers as in gemm_sm100.cu, so a request's results do not depend on how many others share its step by
//     more than the order of fp32 sums.
// The warps of a CTA take the units of its 32 rows in turn and meet once, for the sum over k and the epilogue.
// Packed bf16 arithmetic comes next: a scheduler takes about four cycles for one such instruction, and a 16 x 64 block of int4 has 32 of them
// (and 43 on the integer pipe, 48 % busy, issue slots 55 %). Measured on 34816 x 5120 int4 rows and 4 tokens: 46 us where the tcgen05 path takes 54 (2
// TB/s); 2048 x 1024: 8 where it takes 15.
// (reference: the decode GEMMs of csrc/sm70_turbomind; csrc/quantization/gptq_marlin)
#include "common.cuh"
#include "gemm_sm100.h"

namespace oc {
namespace {

constexpr int kStages = 3;               // units of a warp's ring
constexpr int kUnitBytes = 32 * 64;      // packed weights of a unit
constexpr int kScalePitch = 40;          // words of a k tile's scale words (32 rows), padded so that two tiles lie in different banks

__device__ __forceinline__ void cp16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp16_or_zero(uint32_t dst, const void* src, bool there) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(there ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp8(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ __nv_bfloat162 as_bf2(uint32_t v) { return *reinterpret_cast<__nv_bfloat162*>(&v); }
__device__ __forceinline__ uint32_t as_u32(__nv_bfloat162 v) { return *reinterpret_cast<uint32_t*>(&v); }
__device__ __forceinline__ uint32_t low_twice(uint32_t v) { return __byte_perm(v, 0, 0x1010); }
__device__ __forceinline__ uint32_t high_twice(uint32_t v) { return __byte_perm(v, 0, 0x3232); }

template <int WKIND> struct Kind {
  static constexpr bool kFp8 = WKIND == 2;
  static constexpr int kTiles = kFp8 ? 1 : 2;                 // 64-wide k tiles of a unit
  static constexpr int kK = 64 * kTiles;
  static constexpr int kTileBytes = kFp8 ? 8192 : 4096;
  static constexpr int kScaleWords = WKIND == 4 ? 2 : 1;      // per row and k tile
  static constexpr int kScaleBytes = (kTiles * kScalePitch * kScaleWords * 4 + 63) / 64 * 64;
  static constexpr int kXRow = kK * 2;                        // bytes of an activation row
  __host__ __device__ static constexpr int stage_bytes(int tokens) { return kUnitBytes + kScaleBytes + tokens * kXRow; }
};

// (a & b) | c in one instruction (written out, the compiler takes two where b and c are constants)
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, 0xea;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
}
// a constant that stays in a register
__device__ __forceinline__ uint32_t held(uint32_t v) {
  asm volatile("" : "+r"(v));
  return v;
}

// two neighbouring k out of a lane's 16 bytes: pair `i` of word `c` (4-bit kinds: of four, fp8: of two), as bf16 with the scale applied
template <int WKIND>
__device__ __forceinline__ uint32_t widen(uint32_t word, int i, uint32_t scale, uint32_t z, uint32_t mask, uint32_t bits) {
  if constexpr (WKIND == 1) {          // 0x4300 is 128.0, whose ulp is 1: 128 + code - (128 + zero), exactly
    const uint32_t v = and_or(word >> (4 * i), mask, bits);
    return as_u32(__hmul2(__hsub2(as_bf2(v), as_bf2(z)), as_bf2(scale)));
  } else if constexpr (WKIND == 2) {   // exponent and mantissa four places down read as value * 2^-120; the scale brings it back
    const uint32_t t = __byte_perm(word, 0, i ? 0x3424 : 0x1404);
    const uint32_t v = and_or(t, bits, (t >> 4) & mask);
    return as_u32(__hmul2(as_bf2(v), as_bf2(scale)));
  } else {                             // sign, exponent and mantissa bit in place read as value * 2^-126; the scale too
    const uint32_t q = word >> (4 * i);
    const uint32_t v = and_or(q << 12, bits, (q << 6) & mask);
    return as_u32(__hmul2(as_bf2(v), as_bf2(scale)));
  }
}

constexpr int kMaxWarps = 16;

// One CTA per 32 rows, all tokens (1 .. 8 * NB) of the call.
template <int WKIND, int NB>
__global__ void __launch_bounds__(32 * kMaxWarps) gemm_skinny_kernel(const GemmParams p, const __nv_bfloat16* x, long long ldx) {
  using Q = Kind<WKIND>;
  extern __shared__ __align__(128) uint8_t smem[];
  pdl_trigger();
  const int wk = threadIdx.x >> 5, WK = blockDim.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int nt = blockIdx.x >> 2, rt = (blockIdx.x & 3) * 32, nvalid = p.T;   // 128-row tile, first row inside it
  const int ktiles = p.K / 64, units = (ktiles + Q::kTiles - 1) / Q::kTiles, gk = p.group_ktiles;
  const uint32_t stage = (uint32_t)Q::stage_bytes(nvalid), ring = smem_u32(smem) + (uint32_t)wk * kStages * stage;

  // copies: lane -> row `lane` of the warp's 32 for the four quarters of a unit (eight lanes copy 128 neighbouring bytes). Everything a copy needs
  // is a lane's constant plus a pointer that moves on by a constant.
  const uint8_t* wsrc = p.w4 + ((size_t)nt * ktiles + wk * Q::kTiles) * Q::kTileBytes + (rt + lane) * 16;
  const size_t wstep = (size_t)WK * Q::kTiles * Q::kTileBytes;
  const uint32_t* zsrc = p.w4_sz + ((size_t)nt * 128 + rt + lane) * Q::kScaleWords;
  uint32_t wdst[4];                      // quarter q of a row lies at q ^ (row / 2 % 4): neighbouring rows in different banks
#pragma unroll
  for (int q = 0; q < 4; ++q) wdst[q] = lane * 64 + ((q ^ ((lane >> 1) & 3)) << 4);
  const uint32_t zdst = kUnitBytes + lane * (4 * Q::kScaleWords);
  auto copy_weights = [&](int u, uint32_t dst) {
    // 4-bit: quarters 0, 1 are the halves of the first tile, 2, 3 of the second (missing when the number of tiles is odd: its activations are 0)
    const bool whole = Q::kFp8 || u * 2 + 1 < ktiles;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (q < 2 || whole) cp16(dst + wdst[q], wsrc + q * 2048);
    wsrc += wstep;
#pragma unroll
    for (int i = 0; i < Q::kTiles; ++i) {
      const int kt = u * Q::kTiles + (whole ? i : 0);
      const uint32_t* z = zsrc + (size_t)(gk == 1 ? kt : (gk == 2 ? kt >> 1 : kt / gk)) * (p.n_pad * Q::kScaleWords);
      const uint32_t zd = dst + zdst + i * (kScalePitch * 4 * Q::kScaleWords);
      if (Q::kScaleWords == 2) cp8(zd, z);
      else cp4(zd, z);
    }
  };
  constexpr int XCH = Q::kXRow / 16;     // 16-byte chunks of an activation row
  constexpr int XR = 32 / XCH;           // rows per copy
  // chunk c lies at c ^ (c / 4) ^ (row % 2) (4-bit) or c ^ (row % 2) (fp8): the four quarters of two rows in different banks
  const int xc = lane % XCH, xr = lane / XCH;
  const uint32_t xdst = kUnitBytes + Q::kScaleBytes + xr * Q::kXRow + ((Q::kFp8 ? xc ^ (xr & 1) : xc ^ (xc >> 2) ^ (xr & 1)) << 4);
  const __nv_bfloat16* xsrc = x + (size_t)xr * ldx + wk * Q::kK + xc * 8;
  const size_t xstep = (size_t)WK * Q::kK, xrows = (size_t)XR * ldx;
  const int k_left = p.K - xc * 8;
  auto copy_x = [&](int u, uint32_t dst) {
    const bool there = u * Q::kK < k_left;
    const __nv_bfloat16* src = xsrc;
    int left = nvalid - xr;
#pragma unroll
    for (int r = 0; r < NB * 8; r += XR) {
      if (left > 0) cp16_or_zero(dst + xdst + r * Q::kXRow, src, there);
      left -= XR;
      src += xrows;
    }
    xsrc += xstep;
  };
#pragma unroll
  for (int i = 0; i < kStages - 1; ++i)
    if (wk + i * WK < units) copy_weights(wk + i * WK, ring + i * stage);
  pdl_wait();   // the weights are no kernel's output; activations and results are
#pragma unroll
  for (int i = 0; i < kStages - 1; ++i) {
    if (wk + i * WK < units) copy_x(wk + i * WK, ring + i * stage);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }

  float acc[2][NB][4];
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int n = 0; n < NB; ++n) acc[m][n][0] = acc[m][n][1] = acc[m][n][2] = acc[m][n][3] = 0.f;
  // reads: rows g, g + 8, g + 16, g + 24 share the swizzle of row g
  const uint32_t wrd = g * 64 + ((t ^ ((g >> 1) & 3)) << 4);
  const uint32_t zrd = kUnitBytes + (Q::kFp8 ? g * 4 : (WKIND == 4 ? ((t >> 1) * kScalePitch + g) * 8 + (t & 1) * 4 : ((t >> 1) * kScalePitch + g) * 4));
  uint32_t xrd[NB];       // columns past the tokens repeat the last one (each result column depends on its own operand column only)
#pragma unroll
  for (int n = 0; n < NB; ++n) {
    const int row = min(n * 8 + g, nvalid - 1);
    xrd[n] = kUnitBytes + Q::kScaleBytes + row * Q::kXRow + t * (Q::kXRow / 4) + ((Q::kFp8 ? row & 1 : (t ^ (row & 1)) & 3) << 4);
  }
  const uint32_t mask = held(WKIND == 1 ? 0x000f000fu : (WKIND == 2 ? 0x07f007f0u : 0x01c001c0u)), bits = held(WKIND == 1 ? 0x43004300u : 0x80008000u);
  uint32_t base = ring, fill = ring + (kStages - 1) * stage;
  const uint32_t ring_end = ring + kStages * stage;
  for (int u = wk, un = wk + (kStages - 1) * WK; u < units; u += WK, un += WK) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncwarp();         // every lane's copies of this unit have landed, and every lane is done with the stage that is refilled
    if (un < units) {
      copy_weights(un, fill);
      copy_x(un, fill);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    uint32_t b[NB][Q::kK / 8];           // this lane's run of an activation row, in pairs
#pragma unroll
    for (int n = 0; n < NB; ++n)
#pragma unroll
      for (int i = 0; i < Q::kK / 32; ++i) {
        const uint4 v = lds128((base + xrd[n]) ^ (i << 4));
        b[n][4 * i] = v.x; b[n][4 * i + 1] = v.y; b[n][4 * i + 2] = v.z; b[n][4 * i + 3] = v.w;
      }
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      uint32_t w[2][4], sw[2], sc[2], z[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint4 v = lds128(base + wrd + (m * 16 + h * 8) * 64);
        w[h][0] = v.x; w[h][1] = v.y; w[h][2] = v.z; w[h][3] = v.w;
        sw[h] = lds32(base + zrd + (m * 16 + h * 8) * (4 * Q::kScaleWords));
        // int4: scale | 128 + zero; MXFP4: the scales of the tile's two halves; NVFP4: of the lane's first and second 16 k
        sc[h] = WKIND == 3 && (t & 1) ? high_twice(sw[h]) : low_twice(sw[h]);
        z[h] = high_twice(sw[h]);
      }
#pragma unroll
      for (int st = 0; st < Q::kK / 16; ++st) {
        // two neighbouring pairs of the lane's run: operand B is then a pair of neighbouring registers too
        const int c = st >> (Q::kFp8 ? 0 : 1), i = Q::kFp8 ? 0 : (st & 1) * 2;
        const uint32_t s0 = WKIND == 4 && st >= 4 ? z[0] : sc[0], s1 = WKIND == 4 && st >= 4 ? z[1] : sc[1];
        const uint32_t a[4] = {widen<WKIND>(w[0][c], i, s0, z[0], mask, bits), widen<WKIND>(w[1][c], i, s1, z[1], mask, bits),
                               widen<WKIND>(w[0][c], i + 1, s0, z[0], mask, bits), widen<WKIND>(w[1][c], i + 1, s1, z[1], mask, bits)};
#pragma unroll
        for (int n = 0; n < NB; ++n) mma16816(acc[m][n], a, b[n][2 * st], b[n][2 * st + 1]);
      }
    }
    fill = base;
    base = base + stage == ring_end ? ring : base + stage;
  }

  // ---- sum over the warps that shared rows, then the epilogue, neighbouring threads on neighbouring output columns
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();        // the rings are done with
  float* red = reinterpret_cast<float*>(smem);
  constexpr int ROWS = 32, NP = NB * 8 + 1;
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int n = 0; n < NB; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) red[(wk * ROWS + m * 16 + g + (i >> 1) * 8) * NP + n * 8 + t * 2 + (i & 1)] = acc[m][n][i];
  __syncthreads();
  const bool gated = p.epi == EPI_SILU_MUL;      // a CTA's rows are 16 gate rows and the 16 up rows that go with them
  const int cols = gated ? ROWS / 2 : ROWS, nb = blockIdx.x * cols, lim = gated ? p.n_out : p.N;
  auto total = [&](int row, int tok) {
    float v = 0.f;
    for (int k = 0; k < WK; ++k) v += red[(k * ROWS + row) * NP + tok];
    return v;
  };
  for (int i = threadIdx.x; i < cols * nvalid; i += blockDim.x) {
    const int tok = i / cols, c = i - tok * cols;
    if (nb + c >= lim) continue;
    float v;
    if (gated) {
      const float a = total(c, tok);
      v = a / (1.f + __expf(-a)) * total(c + 16, tok);
    } else {
      v = total(c, tok) + (p.bias != nullptr ? __bfloat162float(p.bias[nb + c]) : 0.f);
    }
    p.out[(size_t)tok * p.ldo + nb + c] = __float2bfloat16(v);
  }
}

int allow(const void* kernel, int slot) {
  static bool configured_dev[kMaxDevices][8] = {};   // the limit is an attribute of (kernel, device)
  bool& configured = configured_dev[current_device_slot()][slot];
  if (!configured) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024) != cudaSuccess) return -4;
    configured = true;
  }
  return 0;
}

template <int WKIND>
int go(const GemmParams& p, const void* x, int ldx, int num_sms, cudaStream_t st) {
  using Q = Kind<WKIND>;
  const __nv_bfloat16* xb = reinterpret_cast<const __nv_bfloat16*>(x);
  const int units = (p.K / 64 + Q::kTiles - 1) / Q::kTiles;
  const int ctas = (p.n_rows + 31) / 32;
  // some sixteen warps to an SM: four to a CTA, or more where there are fewer CTAs than that takes, as long as each has a few units
  int WK = 4;
  while (WK < kMaxWarps && ctas * WK < 16 * num_sms && units >= 2 * (WK + 4) && (WK + 4) * kStages * Q::stage_bytes(p.T) <= 216 * 1024) WK += 4;
  const size_t smem = (size_t)WK * kStages * Q::stage_bytes(p.T);
  auto run = [&](auto kernel, int slot) {
    if (allow((const void*)kernel, (WKIND - 1) * 2 + slot)) return -4;
    return launch_k(kernel, dim3(ctas), dim3(32 * WK), smem, st, true, p, xb, (long long)ldx) == cudaSuccess ? 0 : -10;
  };
  return p.T <= 8 ? run(gemm_skinny_kernel<WKIND, 1>, 0) : run(gemm_skinny_kernel<WKIND, 2>, 1);
}

constexpr int kSkinnyTokens = 16;
constexpr long long kSmallWeights = 32ll << 20, kFewWeights = 24ll << 20;

}  // namespace

// Which dense products take this kernel (us here / on the tcgen05 path of gemm_sm100.cu, which splits k over clusters and starts slower).
// Up to 32 M weights, where its short start counts: 2048 x 1024 8 / 15, 4096 x 4096 int4 and MXFP4 12 / 20, fp8 14 / 20. The kinds that take more
// instructions to widen stop earlier: the fp4 kinds beyond eight tokens at 24 M (5120 x 5120 22.5 / 22, 16384 x 1536 18 / 20.5), fp8 at 24 M (5120 x
// 5120 24.5 / 23 for one token, 28 / 24 for twelve; 12288 x 2048 18.5 / 23.5). fp8 also stops
//   * where its CTAs leave three tenths of their waves' SMs idle and k is not short: 5120 x 4096, 160 CTAs, 22 / 21.5 for four tokens, 25 / 21.5 for
//     nine (4096 x 5120, 128 CTAs: 16 / 22);
//   * where long k meets few rows, a chain per warp: 1024 x 8192 20 / 19, 22 / 19 for nine tokens; 512 x 7168 18.4 / 17.4; 1536 x 7168 18 / 19 up to
//     eight tokens, 20 / 19 above; 2048 x 8192 19 / 23.
// Beyond 32 M int4 with up to eight tokens (34816 x 5120: 45 to 49 / 53; 8192 x 28672: 62 to 67 / 76), except where its CTAs leave two fifths of
// their waves' SMs idle for long: 5120 x 17408, 160 CTAs, 41 / 39 for four tokens, 43 / 39 for eight, 5120 x 25600 52.5 / 50 for one (4800 x 8192
// 23.6 / 25.8).
bool gemm_skinny_takes(const GemmParams& p, int num_sms) {
  if (p.w4 == nullptr || p.n_push != 0 || p.out == nullptr || (p.epi != EPI_STORE && p.epi != EPI_SILU_MUL) || p.T > kSkinnyTokens) return false;
  const long long weights = (long long)p.n_rows * p.K;
  const int ctas = (p.n_rows + 31) / 32, slots = (ctas + num_sms - 1) / num_sms * num_sms;
  if (p.wkind == 2)
    return weights <= kFewWeights && (p.K < 4096 || ctas <= num_sms || 10 * ctas >= 7 * slots) &&
           (p.K <= 6144 || p.n_rows >= 2048 || (p.n_rows >= 1536 && p.T <= 8));
  if (p.wkind != 1) return weights <= (p.T <= 8 ? kSmallWeights : kFewWeights);
  return weights <= kSmallWeights || (p.T <= 8 && (p.K <= 8192 || 5 * ctas >= 3 * slots));
}

// Packed weights and up to 16 tokens; operands and results as in gemm_launch.
int gemm_skinny_launch(const GemmParams& p, const void* x, int ldx, int num_sms, cudaStream_t st) {
  if (p.K % 64 || p.K <= 0 || p.group_ktiles < 1 || p.work != nullptr || p.T > kSkinnyTokens) return -1;
  if (p.T <= 0) return 0;
  int rc;
  switch (p.wkind) {
    case 1: rc = go<1>(p, x, ldx, num_sms, st); break;
    case 2: rc = go<2>(p, x, ldx, num_sms, st); break;
    case 3: rc = go<3>(p, x, ldx, num_sms, st); break;
    case 4: rc = go<4>(p, x, ldx, num_sms, st); break;
    default: return -6;
  }
  if (rc != 0) return rc;
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

}  // namespace oc
