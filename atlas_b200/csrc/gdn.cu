// Gated DeltaNet kernels (Qwen3-Next linear attention), varlen over the step's sequences (the convolution in front: conv1d.cu):
//   gdn_recurrent_kernel   h_t = exp(g_t) h_{t-1} + k_t (x) ((v_t - h_{t-1}^T k_t) beta_t),  o_t = h_t^T q_t / sqrt(Dk)
//                          one CTA per (value head, sequence); thread j keeps column j of the fp32 state in registers;
//                          q/k L2-normalisation and the gates (g from A_log / dt_bias, beta = sigmoid(b)) are fused in.
//                          The same kernel serves decode (1 row), speculative verify (K rows, no commit), the
//                          write-on-accept fold (commit with a row limit) and prefill chunks, and can store
//                          mid-chunk snapshots of the state for the prefix cache.
//   gdn_prep_kernel, gdn_walk_kernel   the same for prefill steps, 64 rows at a time
// State layout: h [slots, Hv, Dk, Dv] fp32, conv window [slots, C, W-1] bf16.
// Reference ops replaced: kernels/gb10/common/{ssm_preprocess,gated_delta_rule*}.cu.
#include <climits>

#include "common.cuh"
#include "host_api.h"
#include "mma_util.cuh"

namespace atlas {

struct GdnParams {
  const __nv_bfloat16* y; long long ldy;      // conv output: [T, 2*Hk*Dk + Hv*Dv] = q | k | v
  const __nv_bfloat16* a; long long lda;      // [T, Hv]
  const __nv_bfloat16* b; long long ldb;      // [T, Hv]
  const float* A_log; const float* dt_bias;    // [Hv]
  float* h;                                    // [slots, Hv, Dk, Dv]
  __nv_bfloat16* out; long long ldo;           // [T, Hv*Dv]
  const int* query_start_loc; const int* state_slots; const unsigned char* has_state;
  const int* limit;                            // rows to process per sequence (nullptr = all)
  const int* snap_rows; const int* snap_slots; int num_snaps_per_seq;
  int B, Hk, Hv, Dv, commit;
  int row_lo, row_hi;                          // row counts of the sequences that are this launch's: [row_lo, row_hi)
  float scale;
  // chunked form: matrices and row factors of every (chunk, head) of hvn value heads from hv0 on
  float* mats; float* factors; __nv_bfloat16* rows; int hv0, hvn;
};

template <int DK>
__global__ void __launch_bounds__(256)
gdn_recurrent_kernel(const GdnParams p) {
  chain_trigger();
  chain_wait();
  const int hv = blockIdx.x, bseq = blockIdx.y;
  const int j = threadIdx.x;                   // column of the state (value dim)
  const int DV = p.Dv;
  const int hk = hv / (p.Hv / p.Hk);
  const int q0 = p.query_start_loc[bseq];
  const int qlen = p.query_start_loc[bseq + 1] - q0;
  const int n = p.limit ? min(p.limit[bseq], qlen) : qlen;
  if (n <= 0 || n >= p.row_hi) return;
  const long long slot = p.state_slots[bseq];
  float* hs = p.h + ((slot * p.Hv + hv) * (long long)DK) * DV;
  float h[DK];
  const bool live = p.has_state[bseq] != 0 && j < DV;
#pragma unroll
  for (int k = 0; k < DK; ++k) h[k] = live ? hs[(long long)k * DV + j] : 0.f;
  __shared__ float sq[DK], sk[DK];
  __shared__ float s_scal[4];                  // q norm scale, k norm scale, exp(g), beta
  const float neg_a = -__expf(p.A_log[hv]);
  const float dtb = p.dt_bias[hv];
  const int kd = p.Hk * DK;
  const int snaps = p.num_snaps_per_seq;
  for (int r = 0; r < n; ++r) {
    const long long t = q0 + r;
    const __nv_bfloat16* row = p.y + t * p.ldy;
    if (j < DK) {
      sq[j] = __bfloat162float(row[hk * DK + j]);
      sk[j] = __bfloat162float(row[kd + hk * DK + j]);
    }
    __syncthreads();
    if (j < 64) {
      // warp 0 -> q, warp 1 -> k : L2 norms
      const float* src = (j < 32) ? sq : sk;
      const int l = j & 31;
      float ss = 0.f;
      for (int k = l; k < DK; k += 32) ss += src[k] * src[k];
      ss = warp_sum(ss);
      if (l == 0) s_scal[j >> 5] = rsqrtf(ss + 1e-6f);
    } else if (j == 64) {
      const float av = __bfloat162float(p.a[t * p.lda + hv]) + dtb;
      const float sp = av > 20.f ? av : log1pf(__expf(av));
      s_scal[2] = __expf(neg_a * sp);
      s_scal[3] = 1.f / (1.f + __expf(-__bfloat162float(p.b[t * p.ldb + hv])));
    }
    __syncthreads();
    if (j < DV) {
      const float qn = s_scal[0] * p.scale, kn = s_scal[1], decay = s_scal[2], beta = s_scal[3];
      const float vt = __bfloat162float(row[2 * kd + hv * DV + j]);
      float mem = 0.f;
#pragma unroll
      for (int k = 0; k < DK; ++k) { h[k] *= decay; mem = fmaf(h[k], sk[k] * kn, mem); }
      const float delta = (vt - mem) * beta;
      float o = 0.f;
#pragma unroll
      for (int k = 0; k < DK; ++k) { h[k] = fmaf(sk[k] * kn, delta, h[k]); o = fmaf(h[k], sq[k] * qn, o); }
      p.out[t * p.ldo + hv * DV + j] = __float2bfloat16_rn(o);
      for (int s = 0; s < snaps; ++s) {
        if (p.snap_rows[bseq * snaps + s] == r + 1) {
          float* dst = p.h + (((long long)p.snap_slots[bseq * snaps + s] * p.Hv + hv) * (long long)DK) * DV;
#pragma unroll
          for (int k = 0; k < DK; ++k) dst[(long long)k * DV + j] = h[k];
        }
      }
    }
    __syncthreads();
  }
  if (p.commit && j < DV) {
#pragma unroll
    for (int k = 0; k < DK; ++k) hs[(long long)k * DV + j] = h[k];
  }
}


// ---------------------------------------------------------------------------- chunked form (prefill)
// The same recurrence evaluated 64 tokens at a time on the tensor cores (TF32 mma.sync, fp32 state and accumulation).  With k, q the
// L2-normalised rows (q scaled), G_i the running sum of the log-decays inside the chunk and h0 the state at its start:
//   (I + A) D = B,   A_ij = beta_i e^{G_i - G_j} (k_i . k_j)  (j < i),   B_i = beta_i (v_i - e^{G_i} h0^T k_i)
//   o_i = e^{G_i} h0^T q_i + sum_{j <= i} P_ij D_j,   P_ij = e^{G_i - G_j} (q_i . k_j)
//   h   = e^{G_C} h0 + sum_j e^{G_C - G_j} k_j (x) D_j
// Two kernels.  gdn_prep_kernel forms what does not depend on the state for all chunks side by side: A, P and the row factors.
// gdn_walk_kernel goes through a sequence's chunks in order: K h0, then the forward substitution on half of the warps while the others
// form Q h0, then P D and K^T D, with the state in registers.
// What bounds it: the walk is a serial chain, so everything that can leave it has left, and its operands are copied a chunk ahead.  One
// 8192-token prompt of 32 value heads: one kernel that did it all in the walk 3264 us, the two here 96 + 718 us, with the same
// operations on every value in the same order (bit for bit the same results).  A 64 x 32 slice per CTA cannot fill an M = 128
// tcgen05 tile, and the state would have to leave TMEM for every chunk.
// Decays are differences of non-positive running sums, so every exponential is <= 1.
// Reference ops replaced: gated_delta_rule_fla.cu / gated_delta_rule_chunk*.cu (WY chunk form).
//
// Order in memory: a thread of an m16n8k8 TF32 product owns k = t and t + 4 (t = lane % 4).  The raw rows are therefore kept with
// element t beside element t + 4 in every group of eight, and with row t beside row t + 4 likewise, so that one 32-bit word of an
// ldmatrix holds both.  gdn_order(p) = which element (row) of its group stands at place p.
constexpr int kGC = 64;                 // chunk length
constexpr int kGLd = 136;               // bf16 [.][128] tiles (ldmatrix: rows 4 banks apart)
constexpr int kGLdH = 132;              // fp32 [.][128] tiles, likewise
constexpr int kGLdC = 68;               // fp32 [.][64] tiles, likewise
constexpr int kGLdA = 72;               // A transposed: columns from 32 on moved by 4, so that four lanes 16 columns apart meet no bank twice
constexpr int kGFactors = 5 * kGC;      // floats per (chunk, head): 1 / |k|, scale / |q|, beta, e^G, e^{G_C - G}
constexpr int kGMats = 2 * kGC * kGC;   // floats per (chunk, head): A transposed, P
constexpr int kGRows = 128 * 128;       // bf16 per (chunk, key head): K rows, Q rows
constexpr int kGDv = 32;                // value columns per walking CTA

ATLAS_DEVICE int gdn_order(int p) { return (p >> 1) + 4 * (p & 1); }
ATLAS_DEVICE uint32_t to_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;\n" : "=r"(r) : "f"(x));
  return r;
}
ATLAS_DEVICE float round_tf32(float x) { return __uint_as_float(to_tf32(x)); }
ATLAS_DEVICE void mma_tf32(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
ATLAS_DEVICE float2 unpack_bf16x2(uint32_t v) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v)); }

// workspace index of a sequence's first chunk: no smaller than the number of chunks before it (a snapshot row adds at most one)
ATLAS_DEVICE int gdn_first_chunk(const GdnParams& p, int b) { return p.query_start_loc[b] / kGC + b * (1 + p.num_snaps_per_seq); }
// rows of the chunk that starts at row c0 of a sequence of n: a snapshot row inside ends it there
ATLAS_DEVICE int gdn_chunk_rows(const GdnParams& p, int b, int c0, int n) {
  int rows = min(kGC, n - c0);
  for (int s = 0; s < p.num_snaps_per_seq; ++s) {
    const int r = p.snap_rows[b * p.num_snaps_per_seq + s];
    if (r > c0 && r < c0 + rows) rows = r - c0;
  }
  return rows;
}

// One CTA per (chunk, key head): K K^T and Q K^T do not depend on the value head.
struct GdnPrepSmem {
  float x[128 * kGLdH];                     // K rows, Q rows (normalised, TF32)
  float g[kGC], beta[kGC];
};

__global__ void __launch_bounds__(256)
gdn_prep_kernel(const GdnParams p) {
  constexpr int DK = 128;
  extern __shared__ __align__(16) uint8_t gsm_raw[];
  GdnPrepSmem& sm = *reinterpret_cast<GdnPrepSmem*>(gsm_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t4 = lane & 3;
  const int rep = p.Hv / p.Hk;
  const int w = blockIdx.x, hk = p.hv0 / rep + blockIdx.y;
  // sequence and chunk of this workspace index: the last sequence whose first chunk is not behind it
  int bseq = -1;
  for (int b0 = 0; b0 < p.B; b0 += 32) {
    const unsigned hit = __ballot_sync(0xffffffffu, b0 + lane < p.B && gdn_first_chunk(p, b0 + lane) <= w);
    bseq += __popc(hit);
  }
  const int q0 = p.query_start_loc[bseq], n = p.query_start_loc[bseq + 1] - q0;
  if (n < p.row_lo) return;
  int c = w - gdn_first_chunk(p, bseq), c0 = -1;
  for (int base = 0; base < n;) {           // pieces between snapshot rows, each cut into chunks from its start
    int next = n;
    for (int s = 0; s < p.num_snaps_per_seq; ++s) {
      const int r = p.snap_rows[bseq * p.num_snaps_per_seq + s];
      if (r > base) next = min(next, r);
    }
    const int k = (next - base + kGC - 1) / kGC;
    if (c < k) { c0 = base + c * kGC; break; }
    c -= k;
    base = next;
  }
  if (c0 < 0) return;                       // the whole block: an index that no chunk has
  const int rows = gdn_chunk_rows(p, bseq, c0, n);
  const int kd = p.Hk * DK;
  const long long t0 = q0 + c0;
  const long long slot0 = (long long)w * p.hvn + hk * rep - p.hv0;         // of this key head's first value head
  // ---- 1. rows of k and q: raw ones in the walk's order, L2-normalised ones (q also scaled) for the products; a warp per row
  __nv_bfloat16* raw_out = p.rows + ((long long)w * gridDim.y + blockIdx.y) * kGRows;
  for (int r0 = warp * 16; r0 < warp * 16 + 16; r0 += 8) {
    uint2 raw[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int r = r0 + u, tok = r & 63;
      raw[u] = make_uint2(0u, 0u);
      if (tok < rows) raw[u] = *reinterpret_cast<const uint2*>(p.y + (t0 + tok) * p.ldy + (r < kGC ? kd : 0) + hk * DK + lane * 4);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int r = r0 + u;
      const float2 lo = unpack_bf16x2(raw[u].x), hi = unpack_bf16x2(raw[u].y);
      const float k[4] = {lo.x, lo.y, hi.x, hi.y};
      const float ks = warp_sum(k[0] * k[0] + k[1] * k[1] + k[2] * k[2] + k[3] * k[3]);
      const float norm = r < kGC ? rsqrtf(ks + 1e-6f) : rsqrtf(ks + 1e-6f) * p.scale;
      *reinterpret_cast<float4*>(sm.x + r * kGLdH + lane * 4) =
          make_float4(round_tf32(k[0] * norm), round_tf32(k[1] * norm), round_tf32(k[2] * norm), round_tf32(k[3] * norm));
      if (lane < rep) p.factors[(slot0 + lane) * kGFactors + (r < kGC ? 0 : kGC) + (r & 63)] = norm;
      // elements 0 4 1 5 from the even lane of a pair, 2 6 3 7 from the odd one; row t beside row t + 4
      const bool odd = lane & 1;
      const uint32_t other = __shfl_xor_sync(0xffffffffu, odd ? raw[u].x : raw[u].y, 1);
      const uint32_t first = odd ? other : raw[u].x, second = odd ? raw[u].y : other;
      const int place = (r & ~7) + 2 * (r & 3) + ((r >> 2) & 1);
      *reinterpret_cast<uint2*>(raw_out + place * DK + lane * 4) = make_uint2(__byte_perm(first, second, 0x5410), __byte_perm(first, second, 0x7632));
    }
  }
  __syncthreads();
  // ---- 2. K K^T (warps 0..3) and Q K^T (warps 4..7), columns up to the diagonal
  const int wr = (warp & 3) * 16, nt = 2 * ((warp & 3) + 1);          // rows of the chunk; 8-wide column tiles
  float acc[8][4];
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
#pragma unroll 2
  for (int ks = 0; ks < DK / 16; ++ks) {
    uint32_t a[2][4];
#pragma unroll
    for (int h = 0; h < 2; ++h)
      ldsm4(smem_u32(sm.x + (warp * 16 + (lane & 15)) * kGLdH + ks * 16 + h * 8 + (lane >> 4) * 4), a[h]);
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (j < nt) {
        uint32_t b[4];
        ldsm4(smem_u32(sm.x + (j * 8 + (lane & 7)) * kGLdH + ks * 16 + (lane >> 3) * 4), b);
        mma_tf32(acc[j], a[0][0], a[0][1], a[0][2], a[0][3], b[0], b[1]);
        mma_tf32(acc[j], a[1][0], a[1][1], a[1][2], a[1][3], b[2], b[3]);
      }
  }
  // ---- 3. per value head: gates and their running sum (warp 0), then A and P
  for (int hh = 0; hh < rep; ++hh) {
    const int hv = hk * rep + hh;
    __syncthreads();                        // the previous head's gates have been read
    if (warp == 0) {
      float* fac = p.factors + (slot0 + hh) * kGFactors;
      const float neg_a = -__expf(p.A_log[hv]);
      const float dtb = p.dt_bias[hv];
      float a[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int i = lane + 32 * k;
        float gi = 0.f, bi = 0.f;
        if (i < rows) {
          const long long tt = t0 + i;
          const float av = __bfloat162float(p.a[tt * p.lda + hv]) + dtb;
          const float sp = av > 20.f ? av : log1pf(__expf(av));
          gi = neg_a * sp;
          bi = 1.f / (1.f + __expf(-__bfloat162float(p.b[tt * p.ldb + hv])));
        }
        a[k] = gi;
        sm.beta[i] = bi;
        fac[2 * kGC + i] = bi;
      }
      float a0 = a[0], a1 = a[1];           // inclusive running sum of the 64 log-decays (two per lane)
      for (int o = 1; o < 32; o <<= 1) {
        const float u0 = __shfl_up_sync(0xffffffffu, a0, o), u1 = __shfl_up_sync(0xffffffffu, a1, o);
        if (lane >= o) { a0 += u0; a1 += u1; }
      }
      const float tot0 = __shfl_sync(0xffffffffu, a0, 31);
      sm.g[lane] = a0;
      sm.g[lane + 32] = a1 + tot0;
      const float gl = __shfl_sync(0xffffffffu, a1 + tot0, 31);
      fac[3 * kGC + lane] = __expf(a0); fac[3 * kGC + lane + 32] = __expf(a1 + tot0);
      fac[4 * kGC + lane] = __expf(gl - a0); fac[4 * kGC + lane + 32] = __expf(gl - a1 - tot0);
    }
    __syncthreads();
    float* A = p.mats + (slot0 + hh) * kGMats;
    float* P = A + kGC * kGC;
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (j < nt) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int i = wr + g + e * 8, m = j * 8 + 2 * t4;
          float v[2];
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const float dec = __expf(sm.g[i] - sm.g[m + q]);
            if (warp < 4) v[q] = m + q < i ? sm.beta[i] * dec * acc[j][2 * e + q] : 0.f;
            else          v[q] = m + q <= i ? round_tf32(dec * acc[j][2 * e + q]) : 0.f;
          }
          if (warp < 4) { A[m * kGC + i] = v[0]; A[(m + 1) * kGC + i] = v[1]; }
          else *reinterpret_cast<float2*>(P + i * kGC + m) = make_float2(v[0], v[1]);
        }
      }
  }
}

// One CTA per (value head, sequence, 32 value columns; the columns of the state evolve independently).  Warp w keeps rows 16 w of the
// state.  The rows of K and Q arrive as they are and are normalised, weighted and rounded in registers.
constexpr int kGLdV = kGDv + 8;
struct GdnStage {
  __nv_bfloat16 x[128 * kGLd];              // K rows, Q rows
  float a[kGC * kGLdA];                     // A transposed
  float p[kGC * kGLdC];
  __nv_bfloat16 v[kGC * kGLdV];
  float f[kGFactors];
};
struct GdnSmem {
  GdnStage stage[2];
  float h[kGDv * kGLdH];                    // state, transposed, TF32
  float b[kGDv * kGLdC];                    // B, transposed
  float d[kGDv * kGLdC];                    // D, transposed, TF32
};

__global__ void __launch_bounds__(256, 1)
gdn_walk_kernel(const GdnParams p) {
  constexpr int DK = 128, DV = 128, NT = kGDv / 8;
  extern __shared__ __align__(16) uint8_t gsm_raw[];
  GdnSmem& sm = *reinterpret_cast<GdnSmem*>(gsm_raw);
  const int hv = p.hv0 + blockIdx.x, bseq = blockIdx.y, v0 = blockIdx.z * kGDv;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t4 = lane & 3, tg = gdn_order(g);
  const int rep = p.Hv / p.Hk, kd = p.Hk * DK;
  const int q0 = p.query_start_loc[bseq];
  const int n = p.query_start_loc[bseq + 1] - q0;
  if (n < p.row_lo) return;
  const long long slot = p.state_slots[bseq];
  float* hs = p.h + ((slot * p.Hv + hv) * (long long)DK) * DV + v0;
  const int snaps = p.num_snaps_per_seq;
  const int ws = gdn_first_chunk(p, bseq);

  auto fetch = [&](GdnStage& s, int c0, int rows, int w) {
    const __nv_bfloat16* x = p.rows + ((long long)w * (p.hvn / rep) + (hv - p.hv0) / rep) * kGRows;
#pragma unroll
    for (int i = tid; i < 128 * 16; i += 256) cp_async16(smem_u32(s.x + (i >> 4) * kGLd + (i & 15) * 8), x + i * 8, true);
    for (int i = tid; i < kGC * (kGDv / 8); i += 256) {
      const int tok = i / (kGDv / 8), ch = i % (kGDv / 8);
      const __nv_bfloat16* src = p.y + (long long)(q0 + c0 + min(tok, rows - 1)) * p.ldy + 2 * kd + hv * DV + v0 + ch * 8;
      cp_async16(smem_u32(s.v + tok * kGLdV + ch * 8), src, tok < rows);
    }
    const long long item = (long long)w * p.hvn + blockIdx.x;
    const float* mats = p.mats + item * kGMats;
#pragma unroll
    for (int i = tid; i < kGC * 16; i += 256) {        // 16-wide blocks on and below the diagonal (of A and P)
      const int r = i >> 4, cc = (i & 15) * 4;
      if (cc >= (r & ~15)) cp_async16(smem_u32(s.a + r * kGLdA + cc + (cc >= 32 ? 4 : 0)), mats + r * kGC + cc, true);
      if (cc < (r | 15)) cp_async16(smem_u32(s.p + r * kGLdC + cc), mats + kGC * kGC + r * kGC + cc, true);
    }
    if (tid < kGFactors / 4) cp_async16(smem_u32(s.f + tid * 4), p.factors + item * kGFactors + tid * 4, true);
  };

  int rows = gdn_chunk_rows(p, bseq, 0, n);
  fetch(sm.stage[0], 0, rows, ws);
  cp_async_commit();
  const int n0 = warp * 16 + tg;            // state rows n0, n0 + 8; columns 8 j + 2 t4 (+ 1)
  float h[NT][4];
  {
    const bool live = p.has_state[bseq] != 0;
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float2 v = make_float2(0.f, 0.f);
        if (live) v = *reinterpret_cast<const float2*>(hs + (n0 + e * 8) * DV + j * 8 + 2 * t4);
        h[j][2 * e] = v.x; h[j][2 * e + 1] = v.y;
      }
  }
  auto put_state = [&]() {
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) sm.h[(j * 8 + 2 * t4 + (e & 1)) * kGLdH + n0 + (e >> 1) * 8] = round_tf32(h[j][e]);
  };
  put_state();

  const int wr = (warp & 3) * 16;           // this warp's rows among the chunk's 64: tokens wr + tg, + 8
  // x += (rows of K or Q, normalised) h0 for NJ column tiles from column j0 on
  auto times_state = [&](const GdnStage& s, int row0, float s0, float s1, int j0, auto& x) {
    constexpr int NJ = sizeof(x) / sizeof(x[0]);
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) x[j][e] = 0.f;
#pragma unroll
    for (int ks = 0; ks < DK / 16; ++ks) {
      uint32_t raw[4], a[2][4];
      ldsm4(smem_u32(s.x + (row0 + (lane & 15)) * kGLd + ks * 16 + (lane >> 4) * 8), raw);
#pragma unroll
      for (int q = 0; q < 4; ++q) {         // raw[q]: rows g / g + 8 (q & 1), k step q >> 1; elements t and t + 4
        const float2 f = unpack_bf16x2(raw[q]);
        const float nr = (q & 1) ? s1 : s0;
        a[q >> 1][q & 1] = to_tf32(f.x * nr); a[q >> 1][2 + (q & 1)] = to_tf32(f.y * nr);
      }
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        uint32_t b[4];
        ldsm4(smem_u32(sm.h + (j0 + j * 8 + (lane & 7)) * kGLdH + ks * 16 + (lane >> 3) * 4), b);
        mma_tf32(x[j], a[0][0], a[0][1], a[0][2], a[0][3], b[0], b[1]);
        mma_tf32(x[j], a[1][0], a[1][1], a[1][2], a[1][3], b[2], b[3]);
      }
    }
  };
  for (int c0 = 0, it = 0; c0 < n; ++it) {
    GdnStage& s = sm.stage[it & 1];
    cp_async_wait<0>();
    __syncthreads();                        // operands are here, the state is written, the other stage is free
    const int c1 = c0 + rows;
    int rows1 = 0;
    if (c1 < n) {
      rows1 = gdn_chunk_rows(p, bseq, c1, n);
      fetch(sm.stage[(it + 1) & 1], c1, rows1, ws + it + 1);
    }
    cp_async_commit();
    // ---- 1. B = beta (v - e^G (K h0)): rows 16 (w % 4), half of the columns per warp
    {
      float x[2][4];
      const int j0 = (warp >> 2) * 16;
      times_state(s, wr, s.f[wr + tg], s.f[wr + tg + 8], j0, x);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int i = wr + tg + e * 8;
        const float beta = s.f[2 * kGC + i], eg = s.f[3 * kGC + i];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int col = j0 + j * 8 + 2 * t4;
          const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(s.v + i * kGLdV + col));
          sm.b[col * kGLdC + i] = beta * (v.x - eg * x[j][2 * e]);
          sm.b[(col + 1) * kGLdC + i] = beta * (v.y - eg * x[j][2 * e + 1]);
        }
      }
    }
    __syncthreads();
    // ---- 2. warps 0..3: forward substitution (I + A) D = B, eight columns a warp, four lanes a column with 16 rows each.  The owner of
    //         block b solves it, hands its 16 values on, and the later rows take them in order.  Warps 4..7: Q h0.
    float x[NT][4];
    if (warp < 4) {
      const int col = warp * 8 + (lane >> 2), q = lane & 3;
      float d[16];
#pragma unroll
      for (int r = 0; r < 16; r += 4) {
        const float4 v = *reinterpret_cast<const float4*>(sm.b + col * kGLdC + q * 16 + r);
        d[r] = v.x; d[r + 1] = v.y; d[r + 2] = v.z; d[r + 3] = v.w;
      }
      const float* mine = s.a + q * 16 + (q >= 2 ? 4 : 0);           // this lane's rows in a row of A transposed
#pragma unroll 1
      for (int b = 0; b < 4; ++b) {
        const float* ab = mine + b * 16 * kGLdA;
        if (q == b) {
#pragma unroll
          for (int j = 0; j < 15; ++j)
#pragma unroll
            for (int r4 = (j + 1) / 4; r4 < 4; ++r4) {
              const float4 a = *reinterpret_cast<const float4*>(ab + j * kGLdA + r4 * 4);
              if (r4 * 4 > j) d[r4 * 4] = fmaf(-a.x, d[j], d[r4 * 4]);
              if (r4 * 4 + 1 > j) d[r4 * 4 + 1] = fmaf(-a.y, d[j], d[r4 * 4 + 1]);
              if (r4 * 4 + 2 > j) d[r4 * 4 + 2] = fmaf(-a.z, d[j], d[r4 * 4 + 2]);
              if (r4 * 4 + 3 > j) d[r4 * 4 + 3] = fmaf(-a.w, d[j], d[r4 * 4 + 3]);
            }
        }
        __syncwarp();
        if (b < 3) {
          float got[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) got[j] = __shfl_sync(0xffffffffu, d[j], (lane & ~3) | b);
          if (q > b) {
#pragma unroll
            for (int j = 0; j < 16; ++j)
#pragma unroll
              for (int r4 = 0; r4 < 4; ++r4) {
                const float4 a = *reinterpret_cast<const float4*>(ab + j * kGLdA + r4 * 4);
                d[r4 * 4] = fmaf(-a.x, got[j], d[r4 * 4]);
                d[r4 * 4 + 1] = fmaf(-a.y, got[j], d[r4 * 4 + 1]);
                d[r4 * 4 + 2] = fmaf(-a.z, got[j], d[r4 * 4 + 2]);
                d[r4 * 4 + 3] = fmaf(-a.w, got[j], d[r4 * 4 + 3]);
              }
          }
          __syncwarp();
        }
      }
#pragma unroll
      for (int r = 0; r < 16; r += 4)
        *reinterpret_cast<float4*>(sm.d + col * kGLdC + q * 16 + r) =
            make_float4(round_tf32(d[r]), round_tf32(d[r + 1]), round_tf32(d[r + 2]), round_tf32(d[r + 3]));
    } else {
      times_state(s, kGC + wr, s.f[kGC + wr + tg], s.f[kGC + wr + tg + 8], 0, x);
      const float e0 = s.f[3 * kGC + wr + tg], e1 = s.f[3 * kGC + wr + tg + 8];
#pragma unroll
      for (int j = 0; j < NT; ++j) { x[j][0] *= e0; x[j][1] *= e0; x[j][2] *= e1; x[j][3] *= e1; }
    }
    __syncthreads();
    // ---- 3. h = e^{G_C} h0 + K^T D;  warps 4..7 also o = e^G (Q h0) + P D
    const float gC = s.f[4 * kGC - 1];
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) h[j][e] *= gC;
#pragma unroll
    for (int ks = 0; ks < kGC / 16; ++ks) {
      uint32_t raw[4], a[2][4], b[NT][4];
#pragma unroll
      for (int j = 0; j < NT; ++j) ldsm4(smem_u32(sm.d + (j * 8 + (lane & 7)) * kGLdC + ks * 16 + (lane >> 3) * 4), b[j]);
      // K^T: rows of the operand are head dims, read transposed from [token][dim]; a thread's tokens are t and t + 4 of each eight
      ldsm4t(smem_u32(s.x + (ks * 16 + (lane >> 4) * 8 + (lane & 7)) * kGLd + warp * 16 + ((lane >> 3) & 1) * 8), raw);
#pragma unroll
      for (int st = 0; st < 2; ++st) {
        const int k0 = ks * 16 + st * 8 + t4;
        const float na = s.f[k0], nb = s.f[k0 + 4], wa = s.f[4 * kGC + k0], wb = s.f[4 * kGC + k0 + 4];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const float2 f = unpack_bf16x2(raw[2 * st + r]);
          a[st][r] = to_tf32(f.x * na * wa); a[st][2 + r] = to_tf32(f.y * nb * wb);
        }
      }
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        mma_tf32(h[j], a[0][0], a[0][1], a[0][2], a[0][3], b[j][0], b[j][1]);
        mma_tf32(h[j], a[1][0], a[1][1], a[1][2], a[1][3], b[j][2], b[j][3]);
      }
      if (warp >= 4 && ks <= (warp & 3)) {
#pragma unroll
        for (int st = 0; st < 2; ++st)
          ldsm4(smem_u32(s.p + (wr + ((lane >> 3) & 1) * 8 + gdn_order(lane & 7)) * kGLdC + ks * 16 + st * 8 + (lane >> 4) * 4), a[st]);
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          mma_tf32(x[j], a[0][0], a[0][1], a[0][2], a[0][3], b[j][0], b[j][1]);
          mma_tf32(x[j], a[1][0], a[1][1], a[1][2], a[1][3], b[j][2], b[j][3]);
        }
      }
    }
    put_state();
    if (warp >= 4) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int i = wr + tg + e * 8;
        if (i < rows) {
          __nv_bfloat16* o = p.out + (long long)(q0 + c0 + i) * p.ldo + hv * DV + v0 + 2 * t4;
#pragma unroll
          for (int j = 0; j < NT; ++j) *reinterpret_cast<__nv_bfloat162*>(o + j * 8) = __floats2bfloat162_rn(x[j][2 * e], x[j][2 * e + 1]);
        }
      }
    }
    auto keep = [&](float* dst) {
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e)
          *reinterpret_cast<float2*>(dst + (n0 + e * 8) * DV + j * 8 + 2 * t4) = make_float2(h[j][2 * e], h[j][2 * e + 1]);
    };
    for (int k = 0; k < snaps; ++k)
      if (p.snap_rows[bseq * snaps + k] == c1)
        keep(p.h + (((long long)p.snap_slots[bseq * snaps + k] * p.Hv + hv) * (long long)DK) * DV + v0);
    if (c1 >= n && p.commit) keep(hs);
    c0 = c1;
    rows = rows1;
  }
}

}  // namespace atlas

using namespace atlas;

// row_hi > 0: only sequences with fewer rows
extern "C" int atlas_gdn_recurrent(const void* y, long long ldy, const void* a, long long lda, const void* b, long long ldb,
                                   const float* A_log, const float* dt_bias, float* h, void* out, long long ldo,
                                   const int* query_start_loc, const int* state_slots, const unsigned char* has_state,
                                   const int* limit, const int* snap_rows, const int* snap_slots, int num_snaps_per_seq,
                                   int B, int Hk, int Hv, int Dk, int Dv, int commit, int row_hi, void* stream) {
  if (B <= 0) return 0;
  if (Dv > 256 || Hv % Hk) return -1;
  GdnParams p;
  p.y = reinterpret_cast<const __nv_bfloat16*>(y); p.ldy = ldy;
  p.a = reinterpret_cast<const __nv_bfloat16*>(a); p.lda = lda;
  p.b = reinterpret_cast<const __nv_bfloat16*>(b); p.ldb = ldb;
  p.A_log = A_log; p.dt_bias = dt_bias; p.h = h;
  p.out = reinterpret_cast<__nv_bfloat16*>(out); p.ldo = ldo;
  p.query_start_loc = query_start_loc; p.state_slots = state_slots; p.has_state = has_state; p.limit = limit;
  p.snap_rows = snap_rows; p.snap_slots = snap_slots; p.num_snaps_per_seq = num_snaps_per_seq;
  p.Hk = Hk; p.Hv = Hv; p.Dv = Dv; p.commit = commit; p.scale = 1.f / sqrtf((float)Dk);
  p.row_hi = row_hi > 0 ? row_hi : INT_MAX;
  dim3 grid(Hv, B);
  int threads = ((max(Dv, max(Dk, 65)) + 31) / 32) * 32;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (Dk == 128) launch_chain(gdn_recurrent_kernel<128>, grid, dim3(threads), 0, st, p);
  else if (Dk == 64) launch_chain(gdn_recurrent_kernel<64>, grid, dim3(threads), 0, st, p);
  else if (Dk == 32) launch_chain(gdn_recurrent_kernel<32>, grid, dim3(threads), 0, st, p);
  else return -2;
  return cudaGetLastError() == cudaSuccess ? 0 : -20;
}

// Chunked (64-token) evaluation of the same recurrence for prefill-sized steps of T rows: Dk = Dv = 128, whole sequences (no row
// limit); a snapshot row inside a chunk simply ends that chunk early.  Sequences of fewer than row_lo rows are left out (a chunk costs
// the same however few rows it has).  Same state layout and arguments as atlas_gdn_recurrent.
// `work`: atlas_gdn_chunked_bytes_within(limit, ...) bytes, 16-byte aligned.  Returns 1 for shapes that only the recurrence takes.
static long long gdn_items(int T, int B, int snaps) { return T / kGC + (long long)B * (1 + snaps); }

// Bytes of workspace for `heads` value heads at once (whole key heads); *heads: all of them while that stays within `limit` bytes, else as
// many as do, but at least one key head's, in several pairs of launches.
constexpr long long kGLimit = 256ll << 20;            // 11 k rows of 32 heads and 16 key heads
extern "C" long long atlas_gdn_chunked_bytes_within(long long limit, int T, int B, int snaps, int Hk, int Hv, int* heads) {
  const int rep = Hv / Hk;
  const long long per_key_head = gdn_items(T, B, snaps) * ((kGMats + kGFactors) * 4ll * rep + kGRows * 2ll);
  const long long n = max(1ll, min((long long)Hk, limit / max(per_key_head, 1ll)));
  *heads = (int)n * rep;
  return per_key_head * n;
}
extern "C" long long atlas_gdn_chunked_bytes(int T, int B, int snaps, int Hk, int Hv, int* heads) {
  return atlas_gdn_chunked_bytes_within(kGLimit, T, B, snaps, Hk, Hv, heads);
}

extern "C" int atlas_gdn_chunked_within(long long limit, const void* y, long long ldy, const void* a, long long lda, const void* b, long long ldb,
                                        const float* A_log, const float* dt_bias, float* h, void* out, long long ldo,
                                        const int* query_start_loc, const int* state_slots, const unsigned char* has_state,
                                        const int* snap_rows, const int* snap_slots, int num_snaps_per_seq, int T, int B, int Hk, int Hv,
                                        int Dk, int Dv, int commit, int row_lo, void* work, void* stream) {
  if (B <= 0) return 0;
  if (Dk != 128 || Dv != 128 || Hv % Hk || (ldy % 8) || (ldo % 2) || (reinterpret_cast<uintptr_t>(y) & 15) || Hv / Hk > 32) return 1;
  if (B > 65535) return 1;
  GdnParams p;
  p.y = reinterpret_cast<const __nv_bfloat16*>(y); p.ldy = ldy;
  p.a = reinterpret_cast<const __nv_bfloat16*>(a); p.lda = lda;
  p.b = reinterpret_cast<const __nv_bfloat16*>(b); p.ldb = ldb;
  p.A_log = A_log; p.dt_bias = dt_bias; p.h = h;
  p.out = reinterpret_cast<__nv_bfloat16*>(out); p.ldo = ldo;
  p.query_start_loc = query_start_loc; p.state_slots = state_slots; p.has_state = has_state; p.limit = nullptr;
  p.snap_rows = snap_rows; p.snap_slots = snap_slots; p.num_snaps_per_seq = num_snaps_per_seq;
  p.B = B; p.Hk = Hk; p.Hv = Hv; p.Dv = Dv; p.commit = commit; p.scale = 1.f / sqrtf((float)Dk);
  p.row_lo = max(1, row_lo);
  int heads = 1;
  atlas_gdn_chunked_bytes_within(limit, T, B, num_snaps_per_seq, Hk, Hv, &heads);
  const long long items = gdn_items(T, B, num_snaps_per_seq);
  p.mats = reinterpret_cast<float*>(work);
  p.factors = p.mats + items * heads * kGMats;
  p.rows = reinterpret_cast<__nv_bfloat16*>(p.factors + items * heads * kGFactors);
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(gdn_prep_kernel), sizeof(GdnPrepSmem)) != cudaSuccess) return -20;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(gdn_walk_kernel), sizeof(GdnSmem)) != cudaSuccess) return -20;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  for (p.hv0 = 0; p.hv0 < Hv; p.hv0 += heads) {
    p.hvn = min(heads, Hv - p.hv0);
    gdn_prep_kernel<<<dim3((unsigned)items, p.hvn / (Hv / Hk)), 256, sizeof(GdnPrepSmem), st>>>(p);
    gdn_walk_kernel<<<dim3(p.hvn, B, Dv / kGDv), 256, sizeof(GdnSmem), st>>>(p);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}
extern "C" int atlas_gdn_chunked(const void* y, long long ldy, const void* a, long long lda, const void* b, long long ldb,
                                 const float* A_log, const float* dt_bias, float* h, void* out, long long ldo,
                                 const int* query_start_loc, const int* state_slots, const unsigned char* has_state,
                                 const int* snap_rows, const int* snap_slots, int num_snaps_per_seq, int T, int B, int Hk, int Hv,
                                 int Dk, int Dv, int commit, int row_lo, void* work, void* stream) {
  return atlas_gdn_chunked_within(kGLimit, y, ldy, a, lda, b, ldb, A_log, dt_bias, h, out, ldo, query_start_loc, state_slots, has_state, snap_rows,
                                  snap_slots, num_snaps_per_seq, T, B, Hk, Hv, Dk, Dv, commit, row_lo, work, stream);
}
