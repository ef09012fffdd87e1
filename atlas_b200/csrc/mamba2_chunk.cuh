// Mamba-2 recurrence for prefill steps, 64 rows at a time on the tensor cores (P = 64 channels per head, state size N = 128, bf16
// activations).  With G_i the running sum of a head's log-decays inside the chunk and S0 the state at its start:
//   y_i = e^{G_i} S0 C_i + sum_{j <= i} e^{G_i - G_j} dt_j (C_i . B_j) x_j + D x_i
//   S   = e^{G_C} S0 + sum_j e^{G_C - G_j} dt_j x_j (x) B_j
// One CTA per (head, sequence) walks the chunks in order; warp w keeps state rows n = 16 w .. + 15 of all 64 channels in
// registers.  Rows 16 (w % 4) .. + 15 of the chunk and half of the channels are warp w's part of y: its scores C B^T stay in
// registers and are the next product's operand as they are.
//
// What bounds it: four products per chunk on mma.sync, serial over a sequence's chunks.  The row-by-row kernel reads all
// coefficients and multiplies the whole state once per row: four prompts of
// 1500 to 656 rows and 128 heads 1266 us, 500 us here.
// An M = 128 tcgen05 tile would have to take the state through TMEM and shared memory for every chunk of 64 rows.
// Precision: x, B, C are the rows as they are; fp32 operands enter as three bf16 terms (24 bits).  Running sums are kept in two floats, so that a difference of two large ones
// is as good as a small one; all exponentials are <= 1.
#pragma once
#include "linear_scan.cuh"
#include "mma_util.cuh"

namespace atlas {

constexpr int kMcRows = 64, kMcP = 64, kMcN = 128;
// Sequences with fewer rows (decode rows beside a prompt) stay with the row-by-row kernel: a chunk costs the same however few rows it
// has, about what 16 rows cost there, and fills an SM by itself.
constexpr int kMcMin = 16;
constexpr int kMcLdN = kMcN + 8, kMcLdP = kMcP + 8;

struct Mamba2Stage {
  __nv_bfloat16 c[kMcRows * kMcLdN], b[kMcRows * kMcLdN], x[kMcRows * kMcLdP];
  float g_hi[kMcRows], g_lo[kMcRows], e[kMcRows], dt[kMcRows], w[kMcRows];      // G, e^G, dt, e^{G_C - G} dt
};
struct Mamba2Smem {
  Mamba2Stage stage[2];
  __nv_bfloat16 s[3][kMcN * kMcLdP];          // state, three terms: [n][p]
  __nv_bfloat16 wx[3][kMcRows * kMcLdP];      // w_j x_j, three terms
};

__global__ void __launch_bounds__(256, 1)
mamba2_chunk_kernel(const ScanParams<__nv_bfloat16> p) {
  constexpr int NT = kMcP / 8;
  extern __shared__ __align__(16) uint8_t msm_raw[];
  Mamba2Smem& sm = *reinterpret_cast<Mamba2Smem*>(msm_raw);
  const int head = blockIdx.x, bseq = blockIdx.y;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t4 = lane & 3;
  const int q0 = p.query_start_loc[bseq];
  const int n = p.query_start_loc[bseq + 1] - q0;
  if (n < kMcMin) return;                     // the row-by-row kernel's
  const int snaps = p.num_snaps_per_seq;
  const float neg_a = -expf(p.A_log[head]), dskip = p.D[head], dtb = p.dt_bias[head];
  const __nv_bfloat16* xsrc = p.a + (long long)q0 * p.lda + head * kMcP;
  const __nv_bfloat16* bsrc = p.a + (long long)q0 * p.lda + p.H * kMcP + (head / (p.H / p.G)) * kMcN;
  const __nv_bfloat16* csrc = bsrc + p.G * kMcN;

  // rows of the chunk that starts at row c0: a snapshot row inside ends it there
  auto chunk_rows = [&](int c0) {
    int rows = min(kMcRows, n - c0);
    for (int s = 0; s < snaps; ++s) {
      const int r = p.snap_rows[bseq * snaps + s];
      if (r > c0 && r < c0 + rows) rows = r - c0;
    }
    return rows;
  };
  auto fetch = [&](Mamba2Stage& s, int c0, int rows) {
    for (int i = tid; i < kMcRows * (kMcN / 8); i += 256) {
      const int r = i / (kMcN / 8), ch = (i % (kMcN / 8)) * 8;
      const long long off = (long long)(c0 + min(r, rows - 1)) * p.lda + ch;
      cp_async16(smem_u32(s.b + r * kMcLdN + ch), bsrc + off, r < rows);
      cp_async16(smem_u32(s.c + r * kMcLdN + ch), csrc + off, r < rows);
    }
    for (int i = tid; i < kMcRows * (kMcP / 8); i += 256) {
      const int r = i / (kMcP / 8), ch = (i % (kMcP / 8)) * 8;
      cp_async16(smem_u32(s.x + r * kMcLdP + ch), xsrc + (long long)(c0 + min(r, rows - 1)) * p.lda + ch, r < rows);
    }
    cp_async_commit();
  };
  // warp 0: rows lane and lane + 32 of the chunk's step sizes; fetched a chunk ahead, turned into factors at that chunk's end
  __nv_bfloat16 raw[2];
  auto fetch_dt = [&](int c0, int rows) {
#pragma unroll
    for (int k = 0; k < 2; ++k) raw[k] = p.b[(long long)(q0 + c0 + min(lane + 32 * k, rows - 1)) * p.ldb + head];
  };
  auto factors = [&](Mamba2Stage& s, int rows) {
    float dt[2];
    double sum[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      dt[k] = lane + 32 * k < rows ? fmaxf(softplus(__bfloat162float(raw[k]) + dtb), p.dt_min) : 0.f;
      sum[k] = (double)(neg_a * dt[k]);
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double u0 = __shfl_up_sync(0xffffffffu, sum[0], o), u1 = __shfl_up_sync(0xffffffffu, sum[1], o);
      if (lane >= o) { sum[0] += u0; sum[1] += u1; }
    }
    sum[1] += __shfl_sync(0xffffffffu, sum[0], 31);
    const double last = __shfl_sync(0xffffffffu, sum[1], 31);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int i = lane + 32 * k;
      const float hi = (float)sum[k];
      s.g_hi[i] = hi;
      s.g_lo[i] = (float)(sum[k] - (double)hi);
      s.e[i] = expf((float)sum[k]);
      s.dt[i] = dt[k];
      s.w[i] = expf((float)(last - sum[k])) * dt[k];
    }
  };

  const long long slot = p.state_slots[bseq];
  float* hs = p.h + ((slot * p.H + head) * (long long)kMcP) * kMcN;
  const int n0 = warp * 16 + g;               // state rows n0, n0 + 8; columns 8 j + 2 t4 (+ 1)
  float h[NT][4];
  const bool live = p.has_state[bseq] != 0;
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) h[j][e] = live ? hs[(j * 8 + 2 * t4 + (e & 1)) * kMcN + n0 + (e >> 1) * 8] : 0.f;
  auto put_state = [&]() {
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        uint32_t t[3];
        split3_bf16x2(h[j][2 * e], h[j][2 * e + 1], t);
#pragma unroll
        for (int k = 0; k < 3; ++k) *reinterpret_cast<uint32_t*>(sm.s[k] + (n0 + e * 8) * kMcLdP + j * 8 + 2 * t4) = t[k];
      }
  };
  int rows = chunk_rows(0);
  fetch(sm.stage[0], 0, rows);
  if (warp == 0) { fetch_dt(0, rows); factors(sm.stage[0], rows); }
  put_state();

  const int wr = (warp & 3) * 16, pc = (warp >> 2) * 32;        // this warp's rows and channels of y
  const uint32_t lt = (uint32_t)((lane & 15) * kMcLdP + (lane >> 4) * 8) * 2;            // ldmatrix (transposed) lane offset
  for (int c0 = 0, it = 0; c0 < n; ++it) {
    Mamba2Stage& s = sm.stage[it & 1];
    cp_async_wait<0>();
    __syncthreads();                          // rows and factors are here, the state is written, the other stage is free
    const int c1 = c0 + rows;
    int rows1 = 0;
    if (c1 < n) {
      rows1 = chunk_rows(c1);
      fetch(sm.stage[(it + 1) & 1], c1, rows1);
      if (warp == 0) fetch_dt(c1, rows1);
    }
    // ---- w_j x_j, three terms
    for (int i = tid; i < kMcRows * kMcP / 2; i += 256) {
      const int r = i / (kMcP / 2), ch = (i % (kMcP / 2)) * 2;
      const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(s.x + r * kMcLdP + ch));
      uint32_t t[3];
      split3_bf16x2(v.x * s.w[r], v.y * s.w[r], t);
#pragma unroll
      for (int k = 0; k < 3; ++k) *reinterpret_cast<uint32_t*>(sm.wx[k] + r * kMcLdP + ch) = t[k];
    }
    // ---- C S0 and the scores C B^T share the rows of C
    float y[4][4], sc[8][4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
#pragma unroll
      for (int j = 0; j < 4; ++j) y[j][e] = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) sc[j][e] = 0.f;
    }
    const int tiles = (warp & 3) + 1;         // 16-wide column tiles of the scores up to the diagonal
#pragma unroll
    for (int ks = 0; ks < kMcN / 16; ++ks) {
      uint32_t a[4];
      ldsm4(smem_u32(s.c + (wr + (lane & 15)) * kMcLdN + ks * 16 + (lane >> 4) * 8), a);
#pragma unroll
      for (int k = 2; k >= 0; --k)            // the smallest term first
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
          uint32_t b[4];
          ldsm4t(smem_u32(sm.s[k] + ks * 16 * kMcLdP + pc + j * 8) + lt, b);
          mma16816(y[j], a, b[0], b[1]); mma16816(y[j + 1], a, b[2], b[3]);
        }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j < tiles) {
          uint32_t b[4];                      // rows 16 j .. + 15 of B
          ldsm4(smem_u32(s.b + (j * 16 + (lane >> 4) * 8 + (lane & 7)) * kMcLdN + ks * 16 + ((lane >> 3) & 1) * 8), b);
          mma16816(sc[2 * j], a, b[0], b[1]); mma16816(sc[2 * j + 1], a, b[2], b[3]);
        }
    }
    // ---- y = e^G (C S0) + (decayed scores) x + D x
    {
      const int i0 = wr + g;
      const float e0 = s.e[i0], e1 = s.e[i0 + 8];
#pragma unroll
      for (int j = 0; j < 4; ++j) { y[j][0] *= e0; y[j][1] *= e0; y[j][2] *= e1; y[j][3] *= e1; }
      const float gh[2] = {s.g_hi[i0], s.g_hi[i0 + 8]}, gl[2] = {s.g_lo[i0], s.g_lo[i0 + 8]};
#pragma unroll
      for (int ks = 0; ks < 4; ++ks)
        if (ks < tiles) {
          uint32_t a[3][4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {       // operand registers: rows g / g + 8 (q & 1), columns 16 ks + 8 (q >> 1) + 2 t4
            const int i = i0 + (q & 1) * 8, col = ks * 16 + (q >> 1) * 8 + 2 * t4;
            float m[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const float diff = (gh[q & 1] - s.g_hi[col + e]) + (gl[q & 1] - s.g_lo[col + e]);
              m[e] = col + e <= i ? expf(diff) * s.dt[col + e] * sc[2 * ks + (q >> 1)][(q & 1) * 2 + e] : 0.f;
            }
            uint32_t t[3];
            split3_bf16x2(m[0], m[1], t);
#pragma unroll
            for (int k = 0; k < 3; ++k) a[k][q] = t[k];
          }
#pragma unroll
          for (int j = 0; j < 4; j += 2) {
            uint32_t b[4];
            ldsm4t(smem_u32(s.x + ks * 16 * kMcLdP + pc + j * 8) + lt, b);
#pragma unroll
            for (int k = 2; k >= 0; --k) { mma16816(y[j], a[k], b[0], b[1]); mma16816(y[j + 1], a[k], b[2], b[3]); }
          }
        }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int i = i0 + e * 8;
        if (i < rows) {
          __nv_bfloat16* o = p.out + (long long)(q0 + c0 + i) * p.ldo + head * kMcP + pc + 2 * t4;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 xv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(s.x + i * kMcLdP + pc + j * 8 + 2 * t4));
            *reinterpret_cast<__nv_bfloat162*>(o + j * 8) = __floats2bfloat162_rn(fmaf(dskip, xv.x, y[j][2 * e]), fmaf(dskip, xv.y, y[j][2 * e + 1]));
          }
        }
      }
    }
    __syncthreads();                          // w x is written, nobody reads the state any more
    // ---- S = e^{G_C} S0 + B^T (w x)
    const float gC = s.e[kMcRows - 1];
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) h[j][e] *= gC;
#pragma unroll
    for (int ks = 0; ks < kMcRows / 16; ++ks) {
      uint32_t a[4];                          // B^T, read transposed from [row][n]
      ldsm4t(smem_u32(s.b + (ks * 16 + (lane >> 4) * 8 + (lane & 7)) * kMcLdN + warp * 16 + ((lane >> 3) & 1) * 8), a);
#pragma unroll
      for (int k = 2; k >= 0; --k)            // the smallest term first
#pragma unroll
        for (int j = 0; j < NT; j += 2) {
          uint32_t b[4];
          ldsm4t(smem_u32(sm.wx[k] + ks * 16 * kMcLdP + j * 8) + lt, b);
          mma16816(h[j], a, b[0], b[1]); mma16816(h[j + 1], a, b[2], b[3]);
        }
    }
    put_state();
    if (warp == 0 && c1 < n) factors(sm.stage[(it + 1) & 1], rows1);
    auto keep = [&](float* dst) {
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) dst[(j * 8 + 2 * t4 + (e & 1)) * kMcN + n0 + (e >> 1) * 8] = h[j][e];
    };
    for (int k = 0; k < snaps; ++k)
      if (p.snap_rows[bseq * snaps + k] == c1)
        keep(p.h + (((long long)p.snap_slots[bseq * snaps + k] * p.H + head) * (long long)kMcP) * kMcN);
    if (c1 >= n && p.commit) keep(hs);
    c0 = c1;
    rows = rows1;
  }
}

// 1: a shape that only the row-by-row kernel takes
static int mamba2_chunked(const ScanParams<__nv_bfloat16>& p, int B, cudaStream_t st) {
  if (p.P != kMcP || p.N != kMcN || p.limit || p.lda % 8 || (reinterpret_cast<uintptr_t>(p.a) & 15) || p.ldo % 2 ||
      (reinterpret_cast<uintptr_t>(p.out) & 3) || B > 65535)
    return 1;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(mamba2_chunk_kernel), sizeof(Mamba2Smem)) != cudaSuccess) return -20;
  mamba2_chunk_kernel<<<dim3(p.H, B), 256, sizeof(Mamba2Smem), st>>>(p);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

}  // namespace atlas
