// Paged decode attention over an fp8 (e4m3) cache, head sizes 128 and 256: the bytes go from the ring in shared memory straight into the operands
// of mma.sync, without a bf16 copy of the tile.
//
// A CTA owns the up to 16 * MB (token, query head of the group) rows of one request and KV head, and one split of its context; its four warps
// take turns of KW keys, each from a cp.async ring of its own (as in attention.cu).
//   * A byte's sign, exponent and mantissa moved into place read as value * 2^-120 in bf16, exactly (subnormals too). The factor is not
//     multiplied back element by element: queries are scaled by 2^60 when they are read and weights are 2^60 times their value, so that
//     scores and results are off by 2^-60 and meet their factors in fp32, where softmax and normalisation multiply anyway. Packed bf16
//     arithmetic (about four cycles an instruction and scheduler) is out of the loop; what is left is four integer instructions per pair.
//   * Q K^T: the order of the head dimensions inside an m16n8k16 step is free as long as both operands agree, so a lane's operand B of four steps
//     is one 16-byte chunk of a key row.
//   * P V: the eight columns of a step may be any dimensions, so lane group g takes chunk g of a value row, and column n of step j is dimension
//     16 n + j; a pair of keys is two bytes of neighbouring rows, put together by one byte permutation.
// 8 requests x 32768 keys x 8 heads of 128: those integer instructions keep the ALU pipe 62 % busy with twelve warps an SM, memory 46 %; latencies are the
// rest. Measured with the merge of the splits, against the kernel that widened tiles into shared memory (us): that case 148 / 219, 4 heads of 256 136 / 279; 64
// requests x 1152 keys 56 / 80; one request x 32000 keys 38 / 52.
// (reference: csrc/attention/paged_attention_v2.cu with fp8 caches; v1/attention/backends/flash_attn.py)
#include "common.cuh"
#include "kernels.h"

namespace oc {
namespace {

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(g) : "memory");
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
// the bytes in bits 8-15 and 24-31 of t (the others may hold anything) as two bf16, times 2^-120
__device__ __forceinline__ uint32_t place(uint32_t t, uint32_t mask, uint32_t sign) {
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, 0xea;" : "=r"(r) : "r"(t), "r"(sign), "r"((t >> 4) & mask));   // (t & sign) | rest
  return r;
}

constexpr float kTwo60 = 0x1p60f, kLog2e = 1.4426950408889634f;

template <int D, int MB> struct Cfg {
  static constexpr int KW = D * MB <= 128 ? 32 : 16;              // keys of a warp's turn
  static constexpr int ST = 2;                                    // turns in its ring
  static constexpr int kRing = 2 * KW * D;                        // bytes of a turn: keys, then values
  static constexpr bool kQRegs = D * MB <= 128;                   // queries stay in registers, else they are read from shared memory
  static constexpr int kQBytes = kQRegs ? 0 : MB * (D / 16) * 512;
  static constexpr int kPitch = D + 4;                            // floats of a row of the warps' partial results
  static constexpr int kMerge = 4 * 16 * MB * (kPitch + 2) * 4;
  static constexpr int kSmem = kQBytes + (4 * ST * kRing > kMerge ? 4 * ST * kRing : kMerge);
};

template <int D, int MB>
__global__ void __launch_bounds__(128, D * MB <= 128 ? 3 : 2) attn_decode_fp8_kernel(const AttnParams p) {
  using C = Cfg<D, MB>;
  constexpr int KW = C::KW, NK = KW / 8, HALVES = D / 128, STEPS = D / 16, ROWS = 16 * MB;
  extern __shared__ __align__(128) uint8_t smem[];
  pdl_trigger();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int G = p.Hq / p.Hkv, hkv = blockIdx.y, r = blockIdx.x;
  const int qs = p.query_start_loc[r], qlen = p.query_start_loc[r + 1] - qs, S = p.seq_lens[r];
  if (qlen <= 0 || S <= 0 || qlen > p.short_q_len) return;   // long queries belong to the prefill kernel
  const int nrows = qlen * G, ctx0 = S - qlen;
  const int nturns = (S + KW - 1) / KW;
  const int wlo = p.window > 0 ? p.window : 0x3fffffff;
  const int first = p.window > 0 ? max(0, ctx0 - p.window + 1) / KW : 0;
  int lo = first, hi = nturns;
  if (p.splits > 1) {   // whole rounds of the four warps
    const int per = (((nturns - first + 3) / 4 + p.splits - 1) / p.splits) * 4;
    lo = first + blockIdx.z * per;
    hi = min(nturns, lo + per);
  }
  const int* bt = p.block_table + (size_t)r * p.bt_stride;
  const size_t head_bytes = (size_t)p.bs * D, blk_bytes = 2 * p.Hkv * head_bytes, v_off = p.Hkv * head_bytes;
  const uint8_t* cache = reinterpret_cast<const uint8_t*>(p.kv_cache) + hkv * head_bytes;
  uint8_t* sRing = smem + C::kQBytes;
  const uint32_t ring = smem_u32(sRing) + warp * (C::ST * C::kRing);

  // a turn's keys and values: rows of D / 16 chunks, chunk c of row k at c ^ (k & 7) (low three bits). Rows past the context are left as they
  // are: any byte is a finite number, and its weight is zero.
  constexpr int CH = D / 16, RPI = 32 / CH;   // chunks of a row, rows per copy instruction
  const int lc = lane % CH, lr = lane / CH;
  auto load_turn = [&](int turn, int buf) {
    const uint32_t dst = ring + buf * C::kRing;
#pragma unroll
    for (int b = 0; b < KW / 16; ++b) {       // pages hold at least 16 keys, and turns start at multiples of 16
      const int key0 = turn * KW + b * 16;
      if (key0 >= S) break;
      const uint8_t* src = cache + (size_t)bt[key0 >> p.bs_shift] * blk_bytes + (size_t)((key0 & (p.bs - 1)) + lr) * D + lc * 16;
#pragma unroll
      for (int i = 0; i < 16; i += RPI) {
        const int k = b * 16 + i + lr;
        const uint32_t off = k * D + ((lc ^ (k & 7)) << 4);
        if (turn * KW + k < S) {
          cp_async16(dst + off, src + i * D);
          cp_async16(dst + KW * D + off, src + v_off + i * D);
        }
      }
    }
  };
#pragma unroll
  for (int i = 0; i < C::ST - 1; ++i) {
    if (lo + warp + 4 * i < hi) load_turn(lo + warp + 4 * i, i);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }

  // queries times 2^60 in operand order: step (chunk c, word w) takes dimensions 16 c + 4 w .. + 3 of the chunks of lane t
  auto q_frag = [&](int mb, int st, int ln, uint32_t (&a)[4]) {
    const int lg = ln >> 2, lt = ln & 3, hh = st >> 3, c = hh * 8 + lt * 2 + ((st >> 2) & 1), d = c * 16 + (st & 3) * 4;
    const __nv_bfloat162 up = __floats2bfloat162_rn(kTwo60, kTwo60);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int row = mb * 16 + lg + h * 8;
      uint2 v = make_uint2(0, 0);
      if (row < nrows) v = *reinterpret_cast<const uint2*>(p.q + (size_t)(qs + row / G) * p.q_st + (size_t)(hkv * G + row % G) * p.q_sh + d);
      const __nv_bfloat162 x = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&v.x), up), y = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&v.y), up);
      a[h] = *reinterpret_cast<const uint32_t*>(&x);
      a[2 + h] = *reinterpret_cast<const uint32_t*>(&y);
    }
  };
  uint32_t qreg[C::kQRegs ? STEPS : 1][4];
  if constexpr (C::kQRegs) {
#pragma unroll
    for (int st = 0; st < STEPS; ++st) q_frag(0, st, lane, qreg[st]);
  } else {
    for (int i = threadIdx.x; i < MB * STEPS * 32; i += 128) {
      uint32_t a[4];
      q_frag(i / (STEPS * 32), (i / 32) % STEPS, i & 31, a);
      *reinterpret_cast<uint4*>(smem + (size_t)i * 16) = make_uint4(a[0], a[1], a[2], a[3]);
    }
    __syncthreads();
  }

  float o[MB][D / 8][4], m[MB][2], l[MB][2];
  int pos[MB][2];
#pragma unroll
  for (int b = 0; b < MB; ++b) {
#pragma unroll
    for (int i = 0; i < D / 8; ++i) o[b][i][0] = o[b][i][1] = o[b][i][2] = o[b][i][3] = 0.f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      m[b][h] = -INFINITY;
      l[b][h] = 0.f;
      pos[b][h] = ctx0 + (b * 16 + g + h * 8) / G;   // rows past nrows are never stored
    }
  }
  const bool capped = p.softcap > 0.f;
  const float qk = p.scale * p.k_scale;
  const float sc = (capped ? qk / p.softcap : qk * kLog2e) * kTwo60, sc_post = p.softcap * kLog2e;
  uint32_t mask = 0x07f007f0u, sign = 0x80008000u;
  asm volatile("" : "+r"(mask), "+r"(sign));         // constants in registers: one instruction per combination

  int buf = 0;
  for (int turn = lo + warp; turn < hi; turn += 4, buf = buf + 1 == C::ST ? 0 : buf + 1) {
    __syncwarp();     // every lane is done with the turn that is overwritten
    if (turn + 4 * (C::ST - 1) < hi) load_turn(turn + 4 * (C::ST - 1), buf == 0 ? C::ST - 1 : buf - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group %0;" ::"n"(C::ST - 1) : "memory");
    __syncwarp();     // every lane's copies of this turn have landed
    const uint32_t kb = ring + buf * C::kRing, vb = kb + KW * D;
    const int k0 = turn * KW;

    float s[MB][NK][4];
#pragma unroll
    for (int b = 0; b < MB; ++b)
#pragma unroll
      for (int n = 0; n < NK; ++n) s[b][n][0] = s[b][n][1] = s[b][n][2] = s[b][n][3] = 0.f;
#pragma unroll
    for (int hc = 0; hc < HALVES * 2; ++hc) {        // a lane's chunks: 2 t, 2 t + 1 of every 128 dimensions
      uint32_t qa[MB][4][4];
#pragma unroll
      for (int b = 0; b < MB; ++b)
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          if constexpr (C::kQRegs) {
#pragma unroll
            for (int e = 0; e < 4; ++e) qa[b][w][e] = qreg[hc * 4 + w][e];
          } else {
            const uint4 v = lds128(smem_u32(smem) + ((b * STEPS + hc * 4 + w) * 32 + lane) * 16);
            qa[b][w][0] = v.x; qa[b][w][1] = v.y; qa[b][w][2] = v.z; qa[b][w][3] = v.w;
          }
        }
#pragma unroll
      for (int n = 0; n < NK; ++n) {
        const uint4 v = lds128(kb + (n * 8 + g) * D + (((hc >> 1) * 8 + ((t * 2 + (hc & 1)) ^ g)) << 4));
        const uint32_t w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          const uint32_t b0 = place(__byte_perm(w4[w], 0, 0x1404), mask, sign), b1 = place(__byte_perm(w4[w], 0, 0x3424), mask, sign);
#pragma unroll
          for (int b = 0; b < MB; ++b) mma_bf16(s[b][n], qa[b][w], b0, b1);
        }
      }
    }
    // ---- mask, online softmax; the sums stay per lane until the end
    const bool masked = k0 + KW - 1 > ctx0 || k0 + wlo <= ctx0 + qlen - 1;
    float alpha[MB][2];
    bool moved = false;
#pragma unroll
    for (int b = 0; b < MB; ++b)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float mx = -INFINITY;
#pragma unroll
        for (int n = 0; n < NK; ++n)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            float v = s[b][n][h * 2 + e] * sc;
            if (capped) v = tanhf(v) * sc_post;
            if (masked) {
              const int key = k0 + n * 8 + t * 2 + e;
              v = (key <= pos[b][h] && key < S && key + wlo > pos[b][h]) ? v : -INFINITY;
            }
            s[b][n][h * 2 + e] = v;
            mx = fmaxf(mx, v);
          }
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const float mn = fmaxf(m[b][h], mx), mu = (mn == -INFINITY ? 0.f : mn) - 60.f;   // weights carry 2^60
        alpha[b][h] = m[b][h] == -INFINITY ? 0.f : ex2(m[b][h] - mn);
        moved = moved || mn != m[b][h];
        m[b][h] = mn;
        float sum = 0.f;
#pragma unroll
        for (int n = 0; n < NK; ++n)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float w = ex2(s[b][n][h * 2 + e] - mu);
            s[b][n][h * 2 + e] = w;
            sum += w;
          }
        l[b][h] = (mn == -INFINITY ? 0.f : l[b][h] * alpha[b][h]) + sum;
      }
    if (__any_sync(0xffffffffu, moved)) {
#pragma unroll
      for (int b = 0; b < MB; ++b)
#pragma unroll
        for (int i = 0; i < D / 8; ++i) {
          o[b][i][0] *= alpha[b][0];
          o[b][i][1] *= alpha[b][0];
          o[b][i][2] *= alpha[b][1];
          o[b][i][3] *= alpha[b][1];
        }
    }
    // ---- O += P V, 16 keys at a time
#pragma unroll
    for (int kg = 0; kg < KW / 16; ++kg) {
      uint32_t a[MB][4];
#pragma unroll
      for (int b = 0; b < MB; ++b) {
        a[b][0] = pack_bf16(s[b][kg * 2][0], s[b][kg * 2][1]);
        a[b][1] = pack_bf16(s[b][kg * 2][2], s[b][kg * 2][3]);
        a[b][2] = pack_bf16(s[b][kg * 2 + 1][0], s[b][kg * 2 + 1][1]);
        a[b][3] = pack_bf16(s[b][kg * 2 + 1][2], s[b][kg * 2 + 1][3]);
      }
#pragma unroll
      for (int hh = 0; hh < HALVES; ++hh) {
        uint32_t v[4][4];                             // chunk g of keys 2 t, 2 t + 1, 8 + 2 t, 9 + 2 t
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int k = kg * 16 + (i >> 1) * 8 + t * 2 + (i & 1);
          const uint4 x = lds128(vb + k * D + ((hh * 8 + (g ^ (k & 7))) << 4));
          v[i][0] = x.x; v[i][1] = x.y; v[i][2] = x.z; v[i][3] = x.w;
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const uint32_t sel = ((4 + (j & 3)) << 12) | ((j & 3) << 4);
          const uint32_t b0 = place(__byte_perm(v[0][j >> 2], v[1][j >> 2], sel), mask, sign);
          const uint32_t b1 = place(__byte_perm(v[2][j >> 2], v[3][j >> 2], sel), mask, sign);
#pragma unroll
          for (int b = 0; b < MB; ++b) mma_bf16(o[b][hh * 16 + j], a[b], b0, b1);
        }
      }
    }
  }

  // ---- merge the four warps' partial results (disjoint keys), then store or hand to the merge of the splits
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float* mo = reinterpret_cast<float*>(sRing);                    // [4][ROWS][kPitch]
  float* mm = mo + 4 * ROWS * C::kPitch;                          // [4][ROWS][2]
#pragma unroll
  for (int b = 0; b < MB; ++b)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int row = b * 16 + g + h * 8;
      float sum = l[b][h];
      sum += __shfl_xor_sync(0xffffffffu, sum, 1);
      sum += __shfl_xor_sync(0xffffffffu, sum, 2);
      float* dst = mo + ((size_t)warp * ROWS + row) * C::kPitch;
#pragma unroll
      for (int hh = 0; hh < HALVES; ++hh)
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int j = 0; j < 16; j += 4) {                       // column n = 2 t + e of step j is dimension 16 n + j
            float4 x;
            x.x = o[b][hh * 16 + j][h * 2 + e] * kTwo60;
            x.y = o[b][hh * 16 + j + 1][h * 2 + e] * kTwo60;
            x.z = o[b][hh * 16 + j + 2][h * 2 + e] * kTwo60;
            x.w = o[b][hh * 16 + j + 3][h * 2 + e] * kTwo60;
            *reinterpret_cast<float4*>(dst + hh * 128 + (2 * t + e) * 16 + j) = x;
          }
      if (t == 0) {
        mm[(warp * ROWS + row) * 2] = m[b][h];
        mm[(warp * ROWS + row) * 2 + 1] = sum * (1.f / kTwo60);
      }
    }
  __syncthreads();
  for (int idx = threadIdx.x; idx < nrows * (D / 4); idx += 128) {
    const int row = idx / (D / 4), c4 = (idx % (D / 4)) * 4;
    float M = -INFINITY;
#pragma unroll
    for (int w = 0; w < 4; ++w) M = fmaxf(M, mm[(w * ROWS + row) * 2]);
    float L = 0.f, acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float mw = mm[(w * ROWS + row) * 2];
      const float f = mw == -INFINITY ? 0.f : ex2(mw - M);
      L += mm[(w * ROWS + row) * 2 + 1] * f;
      const float4 v = *reinterpret_cast<const float4*>(mo + ((size_t)w * ROWS + row) * C::kPitch + c4);
      acc[0] += v.x * f; acc[1] += v.y * f; acc[2] += v.z * f; acc[3] += v.w * f;
    }
    const int tok = row / G, gh = row % G;
    const size_t orow = (size_t)(qs + tok) * p.Hq + hkv * G + gh;
    if (p.splits > 1) {
      *reinterpret_cast<float4*>(p.ws_o + ((size_t)blockIdx.z * p.T * p.Hq + orow) * D + c4) = make_float4(acc[0], acc[1], acc[2], acc[3]);
      if (c4 == 0) {
        float* wm = p.ws_ml + ((size_t)blockIdx.z * p.T * p.Hq + orow) * 2;
        wm[0] = M;
        wm[1] = L;
      }
    } else {
      const float den = L + (p.sinks != nullptr ? ex2(p.sinks[hkv * G + gh] * kLog2e - M) : 0.f);
      const float inv = den > 0.f ? p.v_scale / den : 0.f;
      *reinterpret_cast<uint2*>(p.out + orow * D + c4) = make_uint2(pack_bf16(acc[0] * inv, acc[1] * inv), pack_bf16(acc[2] * inv, acc[3] * inv));
      if (p.lse != nullptr && c4 == 0) p.lse[orow] = (M + log2f(L)) * 0.6931471805599453f;
    }
  }
}

template <int D, int MB>
int go(const AttnParams& p, cudaStream_t st) {
  static bool configured_dev[kMaxDevices] = {};
  bool& configured = configured_dev[current_device_slot()];  // the limit is an attribute of (kernel, device)
  if (!configured) {
    if (cudaFuncSetAttribute(attn_decode_fp8_kernel<D, MB>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<D, MB>::kSmem) != cudaSuccess) return -4;
    configured = true;
  }
  return launch_k(attn_decode_fp8_kernel<D, MB>, dim3(p.R, p.Hkv, p.splits), dim3(128), (size_t)Cfg<D, MB>::kSmem, st, true, p) == cudaSuccess ? 0 : -5;
}

}  // namespace

// Decode mode over an fp8 cache (rows = short_q_len * group size <= 32 for heads of 128, <= 16 for 256); the caller merges the splits.
int attention_decode_fp8_launch(const AttnParams& p, cudaStream_t st) {
  const int rows = p.short_q_len * (p.Hq / p.Hkv);
  if (p.R == 0) return 0;
  if (p.D == 128) return rows <= 16 ? go<128, 1>(p, st) : (rows <= 32 ? go<128, 2>(p, st) : -6);
  if (p.D == 256) return rows <= 16 ? go<256, 1>(p, st) : -6;
  return -1;
}

}  // namespace oc
