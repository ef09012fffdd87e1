// Decode-size MoE expert GEMMs on NVFP4 weights: a few rows per expert (batch x top-k spread over all experts), so the
// work is streaming every touched expert's packed weights once.  The 128-row tcgen05 tile of the grouped kernel is ~6 %
// full there and pays a shared-memory round trip per converted weight; here the weights are the MMA's M operand
// (16 rows per warp), the expert's tokens the N operand (8 per `mma.sync.m16n8k16`), and FP4 -> f16 happens in
// registers on the way from global memory to the tensor core.
//
//   mode 1  a[row, j]  = silu(x[token(row)] . Wg[j]) * (x[token(row)] . Wu[j])      W13 = [E][2I][K/2], rows gathered by token
//   mode 0  y[row, n]  = a[row] . W2[n]                                              W2  = [E][H][K/2]
//
// Rows live in the expert-sorted, 128-row padded buffer built by moe_align (tile i belongs to expert tile_expert[i],
// its live rows are the leading ones with row_token >= 0), so align and combine are shared with the grouped path.
// One CTA = one tile x 64 weight rows (mode 1: 32 gate rows + the matching 32 up rows).  Per 128-wide K span a thread
// loads 16 bytes (32 weights) of each of its two rows; k is assigned to MMA slots so that those bytes are used in place:
// step s of the span takes the thread's weights 4s..4s+3, and the activation tile is staged in shared memory in the
// same order.  Block scales multiply the f16 weights (exact), the per-row global scale the fp32 result.
// Tiles of at most eight rows (most of a decode step's) stage their activations for the whole of K at once and then stream the weights
// four spans ahead without a barrier; the others stage 256 k at a time.  Bound by the weight stream: 12 tokens x 8 of 128 experts,
// 1536 x 2048 58.7 to 45 us; 2048 x 768 stays at 28 us.  The spans in flight take twice the registers (128 a thread), so that half as many
// blocks fit on an SM: steps whose tiles are mostly fuller, or whose K is too long to stage, run the kernel without that path (FEW false, 64
// registers).  The pair of products with and without it: 48 tokens x 4 of 32 experts (2048, 2048) 113 and 127 us, 100 tokens 178 and 162;
// 200 x 8 of 128 (2048, 768) 256 and 209; 64 x 2 of 16 (5120, 8192) 631 and 520.
// Reference ops replaced: moe_w4a16_grouped_gemv*.cu / w4a16_gemv*.cu (kernels/gb10/common).
#include <cuda_fp4.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "host_api.h"

namespace atlas {

constexpr int kSmThreads = 128;
constexpr int kSmTokens = 32;          // tokens per pass (four n8 tiles)
constexpr int kSmKc = 256;             // K elements staged per step (two 128-wide spans)
constexpr int kSmRow = kSmKc + 16;     // f16 per staged token row: 136 words, so 8 tokens x 4 lanes hit distinct banks
constexpr int kSmFew = 8;              // rows of a tile whose activations are staged at once
constexpr int kSmFewK = 4096;          // ... up to this K (66 KB)
constexpr int kSmAhead = 4;            // 128-wide spans of weights in flight per thread

struct SmallMoeParams {
  const __nv_bfloat16* x; long long ldx;
  const int* row_token;
  const int* tile_expert;
  const int* num_tiles;
  const uint8_t* w;        // [E][N][K/2]
  const uint8_t* sc;       // [E*N][K/16] e4m3
  const float* gs;         // [E*N]
  __nv_bfloat16* out; long long ldo;
  int K, N, I;
};

ATLAS_DEVICE uint32_t fp4x2_scaled(uint32_t byte, __half2 sc) {
  __half2_raw hr = __nv_cvt_fp4x2_to_halfraw2((__nv_fp4x2_storage_t)(byte & 0xFFu), __NV_E2M1);
  __half2 h = __hmul2(*reinterpret_cast<__half2*>(&hr), sc);
  return *reinterpret_cast<uint32_t*>(&h);
}
ATLAS_DEVICE __half2 e4m3_half2(uint32_t byte) {
  __half_raw h = __nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)(byte & 0xFFu), __NV_E4M3);
  return __half2half2(*reinterpret_cast<__half*>(&h));
}
ATLAS_DEVICE void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// one 128-wide span: the weights of two rows (w_lo, w_hi with their block scales) times the staged tokens
template <typename FB>
ATLAS_DEVICE void small_span(float (*acc)[4], int n_nt, const uint4& wlo, const uint4& whi, uint32_t slo, uint32_t shi, FB b_at) {
  const uint32_t wl_[4] = {wlo.x, wlo.y, wlo.z, wlo.w};
  const uint32_t wh_[4] = {whi.x, whi.y, whi.z, whi.w};
#pragma unroll
  for (int s = 0; s < 8; ++s) {
    const __half2 scl = e4m3_half2(slo >> (8 * (s >> 2)));
    const __half2 sch = e4m3_half2(shi >> (8 * (s >> 2)));
    const uint32_t lo16 = wl_[s >> 1] >> (16 * (s & 1));
    const uint32_t hi16 = wh_[s >> 1] >> (16 * (s & 1));
    const uint32_t a0 = fp4x2_scaled(lo16, scl), a2 = fp4x2_scaled(lo16 >> 8, scl);
    const uint32_t a1 = fp4x2_scaled(hi16, sch), a3 = fp4x2_scaled(hi16 >> 8, sch);
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      if (nt < n_nt) {
        const uint2 b = b_at(nt, s);
        mma_f16(acc[nt], a0, a1, a2, a3, b.x, b.y);
      }
    }
  }
}
// four bf16 activations as f16, kept finite
ATLAS_DEVICE uint2 small_act(uint2 raw) {
  const float2 f0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
  const float2 f1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
  const __half2 h0 = __floats2half2_rn(fminf(fmaxf(f0.x, -65504.f), 65504.f), fminf(fmaxf(f0.y, -65504.f), 65504.f));
  const __half2 h1 = __floats2half2_rn(fminf(fmaxf(f1.x, -65504.f), 65504.f), fminf(fmaxf(f1.y, -65504.f), 65504.f));
  return make_uint2(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1));
}
// place of element k (a multiple of 4) of a token row: (span, step s, lane t) order
ATLAS_DEVICE int small_place(int k) {
  const int in_span = k & 127;
  return (k & ~127) + ((in_span & 31) >> 2) * 16 + (in_span >> 5) * 4;
}

template <int MODE, bool FEW>
__global__ void __launch_bounds__(kSmThreads)
moe_small_w4_kernel(const SmallMoeParams p) {
  extern __shared__ __align__(16) __half xs[];
  chain_trigger();
  chain_wait();
  __shared__ float ex[MODE == 1 ? 2 * 32 * (kSmTokens + 1) : 1];
  __shared__ int tok_sm[128];
  __shared__ int n_live_sm;
  const int tile = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int live_tiles = *p.num_tiles;          // the three lists are read together; what tiles behind the last one say is not used
  const int e = p.tile_expert[tile];
  const int tok = p.row_token[tile * 128 + threadIdx.x];
  if (tile >= live_tiles) return;
  // live rows of the tile: the leading ones
  {
    tok_sm[threadIdx.x] = tok;
    const int cnt = __syncthreads_count(tok >= 0);
    if (threadIdx.x == 0) n_live_sm = cnt;
  }
  __syncthreads();
  const int n_live = n_live_sm;
  if (n_live == 0) return;
  // the two weight rows of this thread (g and g + 8 of the warp's 16)
  int row0;
  if (MODE == 1) row0 = (warp < 2 ? 0 : p.I) + blockIdx.x * 32 + (warp & 1) * 16;
  else           row0 = blockIdx.x * 64 + warp * 16;
  const long long wrow = (long long)e * p.N + row0 + g;
  const uint8_t* w_lo = p.w + wrow * (p.K >> 1) + 16 * t;
  const uint8_t* w_hi = w_lo + 8ll * (p.K >> 1);
  const uint8_t* s_lo = p.sc + wrow * (p.K >> 4) + 2 * t;
  const uint8_t* s_hi = s_lo + 8ll * (p.K >> 4);
  const float gs_lo = p.gs[wrow], gs_hi = p.gs[wrow + 8];
  const bool few = FEW && n_live <= kSmFew;

  for (int pass0 = 0; pass0 < n_live; pass0 += kSmTokens) {
    const int n_tok = min(kSmTokens, n_live - pass0);
    const int n_nt = (n_tok + 7) >> 3;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) { acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f; }
    auto src_of = [&](int r) {
      return MODE == 1 ? p.x + (long long)tok_sm[pass0 + r] * p.ldx : p.x + (long long)(tile * 128 + pass0 + r) * p.ldx;
    };
    if (few) {
      const int spans = p.K >> 7, row = p.K + 16;
      uint4 wl[kSmAhead], wh[kSmAhead];
      uint32_t sl[kSmAhead], sh[kSmAhead];
      auto fetch = [&](int u, int sp) {
        wl[u] = __ldg(reinterpret_cast<const uint4*>(w_lo + sp * 64));
        wh[u] = __ldg(reinterpret_cast<const uint4*>(w_hi + sp * 64));
        sl[u] = __ldg(reinterpret_cast<const unsigned short*>(s_lo + sp * 8));
        sh[u] = __ldg(reinterpret_cast<const unsigned short*>(s_hi + sp * 8));
      };
#pragma unroll
      for (int u = 0; u < kSmAhead; ++u)
        if (u < spans) fetch(u, u);
      for (int r = 0; r < n_tok; ++r) {
        const __nv_bfloat16* src = src_of(r);
#pragma unroll 4
        for (int k = threadIdx.x * 4; k < p.K; k += kSmThreads * 4)
          *reinterpret_cast<uint2*>(&xs[r * row + small_place(k)]) = small_act(*reinterpret_cast<const uint2*>(src + k));
      }
      __syncthreads();
      for (int sp0 = 0; sp0 < spans; sp0 += kSmAhead) {
#pragma unroll
        for (int u = 0; u < kSmAhead; ++u) {
          const int sp = sp0 + u;
          if (sp < spans) {
            small_span(acc, 1, wl[u], wh[u], sl[u], sh[u], [&](int, int s) {
              return g < n_tok ? *reinterpret_cast<const uint2*>(&xs[g * row + sp * 128 + s * 16 + t * 4]) : make_uint2(0u, 0u);
            });
            if (sp + kSmAhead < spans) fetch(u, sp + kSmAhead);
          }
        }
      }
    } else
    for (int k0 = 0; k0 < p.K; k0 += kSmKc) {
      // weights of this step first: their latency overlaps the activation staging below
      uint4 wl[2], wh[2];
      uint32_t sl[2], sh[2];
#pragma unroll
      for (int sp = 0; sp < 2; ++sp) {
        const int kb = (k0 >> 1) + sp * 64;
        wl[sp] = __ldg(reinterpret_cast<const uint4*>(w_lo + kb));
        wh[sp] = __ldg(reinterpret_cast<const uint4*>(w_hi + kb));
        sl[sp] = __ldg(reinterpret_cast<const unsigned short*>(s_lo + (k0 >> 4) + sp * 8));
        sh[sp] = __ldg(reinterpret_cast<const unsigned short*>(s_hi + (k0 >> 4) + sp * 8));
      }
      __syncthreads();                       // previous step's readers are done with xs
      for (int i = threadIdx.x; i < n_nt * 8 * (kSmKc / 4); i += kSmThreads) {
        const int r = i / (kSmKc / 4), q = i % (kSmKc / 4);
        uint2 packed = make_uint2(0u, 0u);
        if (r < n_tok) packed = small_act(*reinterpret_cast<const uint2*>(src_of(r) + k0 + 4 * q));
        *reinterpret_cast<uint2*>(&xs[r * kSmRow + small_place(4 * q)]) = packed;
      }
      __syncthreads();
#pragma unroll
      for (int sp = 0; sp < 2; ++sp)
        small_span(acc, n_nt, wl[sp], wh[sp], sl[sp], sh[sp], [&](int nt, int s) {
          return *reinterpret_cast<const uint2*>(&xs[(nt * 8 + g) * kSmRow + sp * 128 + s * 16 + t * 4]);
        });
    }
    // ---- epilogue: c0,c1 = (row g, tokens 2t, 2t+1), c2,c3 = (row g+8, same tokens)
    if (MODE == 0) {
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int tok = nt * 8 + 2 * t + j;
          if (tok < n_tok) {
            __nv_bfloat16* o = p.out + (long long)(tile * 128 + pass0 + tok) * p.ldo + row0 + g;
            o[0] = __float2bfloat16_rn(acc[nt][j] * gs_lo);
            o[8] = __float2bfloat16_rn(acc[nt][2 + j] * gs_hi);
          }
        }
      }
    } else {
      __syncthreads();
      const int which = warp >> 1;                 // 0 = gate, 1 = up
      const int col = (warp & 1) * 16 + g;
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int tok = nt * 8 + 2 * t + j;
          ex[(which * 32 + col) * (kSmTokens + 1) + tok] = acc[nt][j] * gs_lo;
          ex[(which * 32 + col + 8) * (kSmTokens + 1) + tok] = acc[nt][2 + j] * gs_hi;
        }
      }
      __syncthreads();
      for (int i = threadIdx.x; i < n_tok * 32; i += kSmThreads) {
        const int tok = i >> 5, c = i & 31;
        // round gate and up to bf16 first, like the unfused GEMM -> SiLU chain does
        const float gv = __bfloat162float(__float2bfloat16_rn(ex[c * (kSmTokens + 1) + tok]));
        const float uv = __bfloat162float(__float2bfloat16_rn(ex[(32 + c) * (kSmTokens + 1) + tok]));
        const float sv = gv / (1.f + __expf(-gv)) * uv;
        p.out[(long long)(tile * 128 + pass0 + tok) * p.ldo + blockIdx.x * 32 + c] = __float2bfloat16_rn(sv);
      }
    }
  }
}

}  // namespace atlas

using namespace atlas;

// mode 1: x [T, K] token rows (gathered through row_token), out [max_rows, I] = silu(gate) * up, N = 2 I rows per expert
// mode 0: x [max_rows, K] sorted rows, out [max_rows, N]
// K % 256 == 0; mode 1: I % 32 == 0; mode 0: N % 64 == 0.  max_tiles bounds the grid; CTAs past *num_tiles return.
// few: most tiles have at most eight rows.
extern "C" int atlas_moe_small_w4(int mode, const void* x, long long ldx, const int* row_token, const int* tile_expert,
                                  const int* num_tiles, int max_tiles, const void* w, const void* sc, const float* gs,
                                  void* out, long long ldo, int K, int N, int few, void* stream) {
  if (max_tiles <= 0) return 0;
  if (K % kSmKc || (ldx % 4)) return -1;
  SmallMoeParams p;
  p.x = reinterpret_cast<const __nv_bfloat16*>(x); p.ldx = ldx;
  p.row_token = row_token; p.tile_expert = tile_expert; p.num_tiles = num_tiles;
  p.w = reinterpret_cast<const uint8_t*>(w); p.sc = reinterpret_cast<const uint8_t*>(sc); p.gs = gs;
  p.out = reinterpret_cast<__nv_bfloat16*>(out); p.ldo = ldo;
  p.K = K; p.N = N; p.I = N / 2;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (N % 64) return -2;
  const bool whole = few && K <= kSmFewK;
  const int smem = max(kSmTokens * kSmRow, whole ? kSmFew * (K + 16) : 0) * (int)sizeof(__half);
  auto launch = [&](auto kern, int blocks) {
    if (ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem) != cudaSuccess) return -20;
    // The down product starts the ordinary way: blocks of an early start fill the SMs that the first product leaves first, eight to one, and a
    // small grid stays on those (2 tokens x 2 of 16 experts, 5120 x 8192: 55 us, early 100 to 190).
    launch_chain_if(mode == 1, kern, dim3(blocks, max_tiles), dim3(kSmThreads), smem, st, p);
    return cudaGetLastError() == cudaSuccess ? 0 : -20;
  };
  if (mode == 1) return whole ? launch(moe_small_w4_kernel<1, true>, p.I / 32) : launch(moe_small_w4_kernel<1, false>, p.I / 32);
  return whole ? launch(moe_small_w4_kernel<0, true>, N / 64) : launch(moe_small_w4_kernel<0, false>, N / 64);
}
