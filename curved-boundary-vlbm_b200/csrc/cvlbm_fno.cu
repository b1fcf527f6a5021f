// Forward and backward kernels of the warm-start surrogate, a Fourier neural
// operator (FNO) on the solver lattice.  The spectral transforms run on the
// tensor cores through cvlbm_gemm_bf16; this file holds the CUDA-core parts.
//
// Layouts (fp32 unless stated): activations channel-major per sample,
// X[b][c][g] with g the lattice node (k fastest); spectral coefficients
// A[b][c][k] with k the retained real Fourier mode; weights W[o][i] (pointwise
// channel mixing), R[k][i][o] (per-mode channel mixing).
//
// Reductions over samples and nodes (weight gradients, the loss) go through
// fixed-size per-block partials and a second pass, so every result is
// deterministic.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "cvlbm_common.cuh"

using namespace cv;

namespace {

constexpr int kMaxC = 32;  // channel limit of the pointwise kernels

__device__ __forceinline__ float gelu_f(float z) {
  return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f));
}
__device__ __forceinline__ float gelu_grad(float z) {
  const float cdf = 0.5f * (1.0f + erff(z * 0.70710678118654752f));
  const float pdf = 0.39894228040143268f * expf(-0.5f * z * z);
  return cdf + z * pdf;
}

// Two fp32 operations in one instruction (sm_100 packed fp32); the lanes are
// rounded separately, so every sum keeps the bits of its scalar form.  The
// product is a * b + nz with nz = -0 (exact) passed to the kernel at run time: a
// packed multiply followed by a packed add would be contracted into one FMA by
// the assembler even with contraction switched off, which changes the rounding.
__device__ __forceinline__ float2 mul2(float2 a, float2 b, float nz) {
  float2 d;
  asm("{\n .reg .b64 x, y, n, z;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n"
      " mov.b64 n, {%6, %6};\n fma.rn.f32x2 z, x, y, n;\n mov.b64 {%0, %1}, z;\n}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(nz));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{\n .reg .b64 x, y, z;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n"
      " add.rn.f32x2 z, x, y;\n mov.b64 {%0, %1}, z;\n}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}

// Nodes g, g + 1 of a row of G (the second one may lie past the end); `vec`:
// rows and base allow one 8-byte access.
__device__ __forceinline__ float2 ld_pair(const float* row, int g, int G, bool vec) {
  if (vec) return *reinterpret_cast<const float2*>(row + g);
  return make_float2(row[g], g + 1 < G ? row[g + 1] : 0.0f);
}
__device__ __forceinline__ void st_pair(float* row, int g, int G, bool vec, float2 v) {
  if (vec) {
    *reinterpret_cast<float2*>(row + g) = v;
  } else {
    row[g] = v.x;
    if (g + 1 < G) row[g + 1] = v.y;
  }
}
__device__ __forceinline__ void st_pair_bf16(__nv_bfloat16* row, int g, int G, bool vec,
                                             float2 v) {
  const __nv_bfloat162 h = __halves2bfloat162(__float2bfloat16_rn(v.x), __float2bfloat16_rn(v.y));
  if (vec) {
    *reinterpret_cast<__nv_bfloat162*>(row + g) = h;
  } else {
    row[g] = h.x;
    if (g + 1 < G) row[g + 1] = h.y;
  }
}

// z[b][o][g] = bias[o] + sum_i W[o][i] x[b][i][g] (+ s[b][o][g]) in order of i;
// y = gelu(z) if act else z; yb: y rounded to bf16, the operand of the next
// spectral transform.
//
// Bound by memory: at 32 -> 32 channels and B G = 262,144 nodes it moves x, s, z, y
// and yb, 151 MB.  One thread takes two adjacent nodes (8-byte accesses, packed
// fp32 arithmetic), its 32 inputs in registers (channel counts are compile-time
// bounds; missing channels multiply zeros) and four outputs at a time; the
// weights sit in shared memory twice, side by side, so that one 16-byte read
// gives two packed operands.
template <int CI, int CO>
__global__ void __launch_bounds__(128)
    k_pointwise_fwd(int B, int G, int Cin, int Cout, const float* __restrict__ x,
                    const float* __restrict__ W, const float* __restrict__ bias,
                    const float* __restrict__ s, int act, float* __restrict__ z,
                    float* __restrict__ y, __nv_bfloat16* __restrict__ yb, int vec, float nz) {
  __shared__ float4 sW[CI][CO / 2];  // (W[o][i], W[o][i], W[o+1][i], W[o+1][i])
  __shared__ float sb[CO];
  for (int t = threadIdx.x; t < CI * CO / 2; t += blockDim.x) {
    const int i = t / (CO / 2), o = 2 * (t % (CO / 2));
    const float w0 = (i < Cin && o < Cout) ? W[o * Cin + i] : 0.0f;
    const float w1 = (i < Cin && o + 1 < Cout) ? W[(o + 1) * Cin + i] : 0.0f;
    sW[i][o / 2] = make_float4(w0, w0, w1, w1);
  }
  for (int t = threadIdx.x; t < CO; t += blockDim.x) sb[t] = t < Cout ? bias[t] : 0.0f;
  __syncthreads();
  const int half = (G + 1) / 2;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)B * half) return;
  const int b = (int)(t / half), g = 2 * (int)(t - (long long)b * half);
  float2 xi[CI];
#pragma unroll
  for (int i = 0; i < CI; ++i)
    xi[i] = i < Cin ? ld_pair(x + ((size_t)b * Cin + i) * G, g, G, vec) : make_float2(0.0f, 0.0f);
  // s of four outputs, loaded one group ahead of its use
  auto load_s = [&](int o, float2* v) {
#pragma unroll
    for (int k = 0; k < 4; ++k)
      v[k] = (s && o + k < Cout) ? ld_pair(s + ((size_t)b * Cout + o + k) * G, g, G, vec)
                                 : make_float2(0.0f, 0.0f);
  };
  float2 sv[4], sn[4];
  load_s(0, sn);
#pragma unroll 1
  for (int o = 0; o < Cout; o += 4) {
    float2 acc[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      acc[k] = make_float2(sb[o + k], sb[o + k]);
      sv[k] = sn[k];
    }
    load_s(o + 4, sn);
#pragma unroll
    for (int i = 0; i < CI; ++i) {
      const float4 w0 = sW[i][o / 2], w1 = sW[i][o / 2 + 1];
      acc[0] = add2(acc[0], mul2(make_float2(w0.x, w0.y), xi[i], nz));
      acc[1] = add2(acc[1], mul2(make_float2(w0.z, w0.w), xi[i], nz));
      acc[2] = add2(acc[2], mul2(make_float2(w1.x, w1.y), xi[i], nz));
      acc[3] = add2(acc[3], mul2(make_float2(w1.z, w1.w), xi[i], nz));
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (o + k >= Cout) break;
      const size_t row = ((size_t)b * Cout + o + k) * G;
      float2 v = s ? add2(acc[k], sv[k]) : acc[k];
      if (z) st_pair(z + row, g, G, vec, v);
      if (act) v = make_float2(gelu_f(v.x), gelu_f(v.y));
      st_pair(y + row, g, G, vec, v);
      if (yb) st_pair_bf16(yb + row, g, G, vec, v);
    }
  }
}

// dz = dy * gelu'(z)
__global__ void k_gelu_bwd(long long n, const float* __restrict__ z, const float* __restrict__ dy,
                           float* __restrict__ dz) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) dz[t] = dy[t] * gelu_grad(z[t]);
}

// Backward pass of one pointwise layer over a chunk of 128 nodes of one sample:
//   dz = dy gelu'(z) (z given) or dy;   dzb = dz rounded to bf16 (if given);
//   dx[i] (+)= sum_o W[o][i] dz[o]  in order of o (if given);
//   part[c][o*Cin+i] = sum_g dz[o][g] x[i][g], part[c][Cout*Cin+o] = sum_g dz[o][g]
// (node order).  dz itself never goes to memory: one pass reads dy, z and x and
// writes dx and dzb (151 MB at 32 channels and B G = 262,144), where separate
// GELU, bf16, dx and dW kernels moved 335 MB.  A thread owns one node for dz and
// dx; the weight gradients then take four outputs x two inputs per thread from
// the node-major tiles in shared memory (rows of 36 floats: 16-byte accesses of
// eight lanes fall into distinct banks), packed fp32 over the output pairs.
constexpr int kChunkG = 128;
template <int CI, int CO>
__global__ void __launch_bounds__(kChunkG, 5)
    k_pointwise_bwd(int B, int G, int Cin, int Cout, const float* __restrict__ dy,
                    const float* __restrict__ z, const float* __restrict__ x,
                    const float* __restrict__ W, int accumulate, float* __restrict__ dx,
                    __nv_bfloat16* __restrict__ dzb, float* __restrict__ part, float nz) {
  __shared__ __align__(16) float sW[CO][CI];
  __shared__ __align__(16) float sdz[kChunkG][CO + 4];
  __shared__ __align__(16) float sx[kChunkG][CI + 4];
  const int tid = threadIdx.x;
  for (int t = tid; t < CO * CI; t += kChunkG) {
    const int o = t / CI, i = t % CI;
    sW[o][i] = (o < Cout && i < Cin) ? W[o * Cin + i] : 0.0f;
  }
  const int chunks = (G + kChunkG - 1) / kChunkG;
  const int c = blockIdx.x, b = c / chunks, g = (c % chunks) * kChunkG + tid;
  const bool ok = g < G;
  // x goes to shared memory by itself (4-byte asynchronous copies) while dz forms
#pragma unroll
  for (int i = 0; i < CI; ++i) {
    const bool in = ok && i < Cin;
    const float* src = x + ((size_t)b * Cin + (in ? i : 0)) * G + (ok ? g : 0);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(&sx[tid][i]))),
                 "l"(src), "r"(in ? 4 : 0)
                 : "memory");
  }
  float d[CO];
  constexpr int kOC = CO < 16 ? CO : 16;  // channels whose dy and z are in flight together
#pragma unroll
  for (int o0 = 0; o0 < CO; o0 += kOC) {
    float zv[kOC];
#pragma unroll
    for (int k = 0; k < kOC; ++k) {
      const int o = o0 + k;
      const size_t at = ((size_t)b * Cout + o) * G + g;
      d[o] = (ok && o < Cout) ? dy[at] : 0.0f;
      zv[k] = (z && ok && o < Cout) ? z[at] : 0.0f;
    }
    if (z) {
#pragma unroll
      for (int k = 0; k < kOC; ++k) d[o0 + k] = d[o0 + k] * gelu_grad(zv[k]);
    }
#pragma unroll
    for (int k = 0; k < kOC; k += 4)
      *reinterpret_cast<float4*>(&sdz[tid][o0 + k]) =
          make_float4(d[o0 + k], d[o0 + k + 1], d[o0 + k + 2], d[o0 + k + 3]);
    if (dzb) {
#pragma unroll
      for (int k = 0; k < kOC; ++k) {
        const int o = o0 + k;
        if (ok && o < Cout) dzb[((size_t)b * Cout + o) * G + g] = __float2bfloat16_rn(d[o]);
      }
    }
  }
  asm volatile("cp.async.commit_group;\n cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  if (dx && ok) {
#pragma unroll 1
    for (int i = 0; i < Cin; i += 4) {
      float2 a0 = make_float2(0.0f, 0.0f), a1 = a0;
#pragma unroll
      for (int o = 0; o < CO; ++o) {
        const float4 w = *reinterpret_cast<const float4*>(&sW[o][i]);
        const float2 dd = make_float2(d[o], d[o]);
        a0 = add2(a0, mul2(make_float2(w.x, w.y), dd, nz));
        a1 = add2(a1, mul2(make_float2(w.z, w.w), dd, nz));
      }
      const float v[4] = {a0.x, a0.y, a1.x, a1.y};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (i + k < Cin) {
          const size_t at = ((size_t)b * Cin + i + k) * G + g;
          dx[at] = accumulate ? dx[at] + v[k] : v[k];
        }
      }
    }
  }
  const int nw = Cout * Cin + Cout;
  float* out = part + (size_t)c * nw;
  constexpr int kOQ = CO / 4, kIP = CI / 2;
  for (int t = tid; t < kOQ * kIP; t += kChunkG) {
    const int o = 4 * (t % kOQ), i = 2 * (t / kOQ);
    if (o >= Cout || i >= Cin) continue;
    float2 a00 = make_float2(0.0f, 0.0f), a01 = a00, a10 = a00, a11 = a00;
#pragma unroll 4
    for (int gg = 0; gg < kChunkG; ++gg) {
      const float4 e = *reinterpret_cast<const float4*>(&sdz[gg][o]);
      const float2 xv = *reinterpret_cast<const float2*>(&sx[gg][i]);
      const float2 e0 = make_float2(e.x, e.y), e1 = make_float2(e.z, e.w);
      const float2 x0 = make_float2(xv.x, xv.x), x1 = make_float2(xv.y, xv.y);
      a00 = add2(a00, mul2(e0, x0, nz));
      a01 = add2(a01, mul2(e1, x0, nz));
      a10 = add2(a10, mul2(e0, x1, nz));
      a11 = add2(a11, mul2(e1, x1, nz));
    }
    const float r0[4] = {a00.x, a00.y, a01.x, a01.y}, r1[4] = {a10.x, a10.y, a11.x, a11.y};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (o + k < Cout) {
        out[(o + k) * Cin + i] = r0[k];
        if (i + 1 < Cin) out[(o + k) * Cin + i + 1] = r1[k];
      }
    }
  }
  if (tid < Cout) {
    float acc = 0.0f;
#pragma unroll 8
    for (int gg = 0; gg < kChunkG; ++gg) acc += sdz[gg][tid];
    out[Cout * Cin + tid] = acc;
  }
}

// dW[t] (t < n_w) and db[t - n_w] = sum_c part[c][t] in chunk order.
//
// One block per 32 sums.  The chain of additions is serial by definition (chunk
// order), the loads are not: eight warps bring the next 256 partials (rows of 128
// bytes, 32 loads in flight per thread) while warp 0 adds the current 256 from
// shared memory.  2,048 partials of 1,056 sums: 132 us with one thread per sum
// loading for itself, 75 us with the loads not unrolled, 27 us with 16 in flight.
constexpr int kSumTile = 256, kSumLoaders = 8;
__global__ void __launch_bounds__(32 * (kSumLoaders + 1))
    k_sum_parts(int n_parts, int width, int n_w, const float* __restrict__ part,
                float* __restrict__ dW, float* __restrict__ db) {
  __shared__ float tile[kSumTile][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t = blockIdx.x * 32 + lane;
  constexpr int kRows = kSumTile / kSumLoaders;
  float v[kRows];
  auto load = [&](int c0) {
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const int c = c0 + (warp - 1) * kRows + r;
      v[r] = (c < n_parts && t < width) ? part[(size_t)c * width + t] : 0.0f;
    }
  };
  if (warp > 0) load(0);
  float acc = 0.0f;
  for (int c0 = 0; c0 < n_parts; c0 += kSumTile) {
    if (warp > 0) {
#pragma unroll
      for (int r = 0; r < kRows; ++r) tile[(warp - 1) * kRows + r][lane] = v[r];
    }
    __syncthreads();
    if (warp == 0) {
      const int m = n_parts - c0 < kSumTile ? n_parts - c0 : kSumTile;
      if (m == kSumTile) {
#pragma unroll 32
        for (int r = 0; r < kSumTile; ++r) acc += tile[r][lane];
      } else {
        for (int r = 0; r < m; ++r) acc += tile[r][lane];
      }
    } else if (c0 + kSumTile < n_parts) {
      load(c0 + kSumTile);
    }
    __syncthreads();
  }
  if (warp == 0 && t < width) {
    if (t < n_w)
      dW[t] = acc;
    else
      db[t - n_w] = acc;
  }
}

// Per-mode channel mixing: bh[b][o][k] = sum_i a[b][i][k] R[k][i][o] in order of
// i, written as bf16 for the inverse transform.
//
// Bound by the weights (R: 3.1 MB at 768 modes, read once) and by latency: a warp
// owns one mode with lane = output channel, so R[k] is read in 128-byte rows; the
// block's four modes of a (16-byte runs) are staged in shared memory and the
// results leave through it.  One thread per (sample, mode), each walking its own
// 4 KB of R, took 100 us.
constexpr int kMixK = 4, kMixB = 4;  // modes per block, samples per pass
__global__ void __launch_bounds__(32 * kMixK)
    k_spec_mix_fwd(int B, int C, int M, const float* __restrict__ a, const float* __restrict__ R,
                   __nv_bfloat16* __restrict__ bh) {
  __shared__ float sa[kMixB * kMaxC][kMixK + 1];
  const int k0 = blockIdx.x * kMixK, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int k = k0 + w;
  const float* Rk = R + (size_t)k * C * C;
  float r[kMaxC];
#pragma unroll
  for (int i = 0; i < kMaxC; ++i)
    r[i] = (k < M && i < C && lane < C) ? Rk[i * C + lane] : 0.0f;
  for (int b0 = 0; b0 < B; b0 += kMixB) {
    const int rows = (B - b0 < kMixB ? B - b0 : kMixB) * C;
    float ta[kMixB];
#pragma unroll
    for (int u = 0; u < kMixB; ++u) {
      const int t = threadIdx.x + u * 32 * kMixK, row = t / kMixK, kk = t % kMixK;
      ta[u] = (row < rows && k0 + kk < M) ? a[((size_t)b0 * C + row) * M + k0 + kk] : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < kMixB; ++u) {
      const int t = threadIdx.x + u * 32 * kMixK, row = t / kMixK, kk = t % kMixK;
      sa[row][kk] = ta[u];
    }
    __syncthreads();
    float acc[kMixB];
#pragma unroll
    for (int b = 0; b < kMixB; ++b) {
      acc[b] = 0.0f;
      if (b * C < rows) {
#pragma unroll
        for (int i = 0; i < kMaxC; ++i)
          if (i < C) acc[b] += sa[b * C + i][w] * r[i];
      }
    }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < kMixB; ++b)
      if (b * C < rows && lane < C) sa[b * C + lane][w] = acc[b];
    __syncthreads();
    for (int t = threadIdx.x; t < rows * kMixK; t += blockDim.x) {
      const int row = t / kMixK, kk = t % kMixK;
      if (k0 + kk < M)
        bh[((size_t)b0 * C + row) * M + k0 + kk] = __float2bfloat16_rn(sa[row][kk]);
    }
    __syncthreads();
  }
}

// Backward of the mixing: da[b][i][k] = sum_o R[k][i][o] dbh[b][o][k] in order of
// o (bf16, for the inverse transform) and dR[k][i][o] = sum_b a[b][i][k]
// dbh[b][o][k] in order of b.  The layout of k_spec_mix_fwd: a warp owns one mode,
// R[k] passes through shared memory once (rows padded to 33) because da needs
// its rows by lane, and dR[k] is summed by lane = output channel, row by row.
__global__ void __launch_bounds__(32 * kMixK)
    k_spec_mix_bwd(int B, int C, int M, const float* __restrict__ a,
                   const float* __restrict__ dbh, const float* __restrict__ R,
                   __nv_bfloat16* __restrict__ da, float* __restrict__ dR) {
  extern __shared__ float mix_sm[];
  float* sR = mix_sm;                                  // [kMixK][32][33]
  float* sa = sR + kMixK * kMaxC * (kMaxC + 1);        // [rows][kMixK + 1]
  float* sd = sa + kMixB * kMaxC * (kMixK + 1);        // [rows][kMixK + 1]
  float* so = sd + kMixB * kMaxC * (kMixK + 1);        // [rows][kMixK + 1]
  const int k0 = blockIdx.x * kMixK, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int k = k0 + w;
  const bool live = k < M && lane < C;
  float* Rw = sR + w * kMaxC * (kMaxC + 1);
  const float* Rk = R + (size_t)k * C * C;
  float dr[kMaxC];  // R[k] on its way to shared memory (all loads in flight), then dR[k]
#pragma unroll
  for (int i = 0; i < kMaxC; ++i) dr[i] = (live && i < C) ? Rk[i * C + lane] : 0.0f;
#pragma unroll
  for (int i = 0; i < kMaxC; ++i) Rw[i * (kMaxC + 1) + lane] = dr[i];
#pragma unroll
  for (int i = 0; i < kMaxC; ++i) dr[i] = 0.0f;
  for (int b0 = 0; b0 < B; b0 += kMixB) {
    const int rows = (B - b0 < kMixB ? B - b0 : kMixB) * C;
    float ta[kMixB], td[kMixB];
#pragma unroll
    for (int u = 0; u < kMixB; ++u) {
      const int t = threadIdx.x + u * 32 * kMixK, row = t / kMixK, kk = t % kMixK;
      const bool in = row < rows && k0 + kk < M;
      const size_t at = in ? ((size_t)b0 * C + row) * M + k0 + kk : 0;
      ta[u] = in ? a[at] : 0.0f;
      td[u] = in ? dbh[at] : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < kMixB; ++u) {
      const int t = threadIdx.x + u * 32 * kMixK, row = t / kMixK, kk = t % kMixK;
      sa[row * (kMixK + 1) + kk] = ta[u];
      sd[row * (kMixK + 1) + kk] = td[u];
    }
    __syncthreads();
    if (live) {
      for (int b = 0; b * C < rows; ++b) {
        float acc = 0.0f;
#pragma unroll
        for (int o = 0; o < kMaxC; ++o)
          if (o < C) acc += Rw[lane * (kMaxC + 1) + o] * sd[(b * C + o) * (kMixK + 1) + w];
        so[(b * C + lane) * (kMixK + 1) + w] = acc;
        const float e = sd[(b * C + lane) * (kMixK + 1) + w];
#pragma unroll
        for (int i = 0; i < kMaxC; ++i)
          if (i < C) dr[i] += sa[(b * C + i) * (kMixK + 1) + w] * e;
      }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < rows * kMixK; t += blockDim.x) {
      const int row = t / kMixK, kk = t % kMixK;
      if (k0 + kk < M)
        da[((size_t)b0 * C + row) * M + k0 + kk] =
            __float2bfloat16_rn(so[row * (kMixK + 1) + kk]);
    }
    __syncthreads();
  }
  if (live) {
#pragma unroll
    for (int i = 0; i < kMaxC; ++i)
      if (i < C) dR[(size_t)k * C * C + i * C + lane] = dr[i];
  }
}
constexpr size_t kMixBwdSmem =
    sizeof(float) * (kMixK * kMaxC * (kMaxC + 1) + 3 * kMixB * kMaxC * (kMixK + 1));

__global__ void k_to_bf16(long long n, const float* __restrict__ src,
                          __nv_bfloat16* __restrict__ dst) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) dst[t] = __float2bfloat16_rn(src[t]);
}

// Masked mean-squared error: loss = sum w_o mask (y - t)^2 / count,
// dy = 2 w_o mask (y - t) / count; per-block loss partials.  `mask_sum` (device,
// may be null): count = C * mask_sum, at least 1, so that the caller need not
// read the mask's sum back.  A block walks its elements in grid strides; four
// strides are loaded before the first is used (one at a time, with a 64-bit
// division each, took 38 us for 3.1 M elements).
__global__ void __launch_bounds__(256)
    k_mse(int B, int C, int G, const float* __restrict__ y, const float* __restrict__ tgt,
          const float* __restrict__ mask, const float* __restrict__ w, float inv_count,
          const float* __restrict__ mask_sum, float* __restrict__ dy, float* __restrict__ part) {
  __shared__ float red[256];
  if (mask_sum) {
    const double cnt = (double)mask_sum[0] * (double)C;
    inv_count = (float)(1.0 / (cnt > 1.0 ? cnt : 1.0));
  }
  const long long n = (long long)B * C * G, step = (long long)gridDim.x * blockDim.x;
  float acc = 0.0f;
  constexpr int kU = 4;
  for (long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x; t0 < n; t0 += kU * step) {
    float yv[kU], tv[kU], m[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const long long t = t0 + u * step;
      if (t >= n) break;
      unsigned bc;
      int g;
      if (n <= 0x7fffffffLL) {
        bc = (unsigned)t / (unsigned)G;
        g = (int)((unsigned)t - bc * (unsigned)G);
      } else {
        bc = (unsigned)(t / G);
        g = (int)(t - (long long)bc * G);
      }
      const unsigned b = bc / (unsigned)C;
      yv[u] = y[t];
      tv[u] = tgt[t];
      m[u] = mask[(size_t)b * G + g] * w[bc - b * (unsigned)C];
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const long long t = t0 + u * step;
      if (t >= n) break;
      const float e = yv[u] - tv[u];
      acc += m[u] * e * e;
      dy[t] = 2.0f * m[u] * e * inv_count;
    }
  }
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int h = 128; h > 0; h >>= 1) {
    if ((int)threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = red[0] * inv_count;
}

// Adam with bias correction (lr already includes it).
__global__ void k_adam(long long n, float* __restrict__ p, const float* __restrict__ g,
                       float* __restrict__ m, float* __restrict__ v, float lr, float b1, float b2,
                       float eps) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const float gt = g[t];
  const float mt = b1 * m[t] + (1.0f - b1) * gt;
  const float vt = b2 * v[t] + (1.0f - b2) * gt * gt;
  m[t] = mt;
  v[t] = vt;
  p[t] -= lr * mt / (sqrtf(vt) + eps);
}

// Adam over several tensors in one launch: block -> (tensor, slice) by the
// running block counts in `first` (the 16 tensors of the default network took 16
// launches, most of them a few elements long).
constexpr int kAdamTensors = 32, kAdamPerBlock = 1024;
struct AdamList {
  float* p[kAdamTensors];
  const float* g[kAdamTensors];
  float* m[kAdamTensors];
  float* v[kAdamTensors];
  long long n[kAdamTensors];
  unsigned first[kAdamTensors + 1];
  int count;
};
__global__ void __launch_bounds__(256)
    k_adam_list(const __grid_constant__ AdamList L, float lr, float b1, float b2, float eps) {
  int k = 0;
  while (k + 1 < L.count && blockIdx.x >= L.first[k + 1]) ++k;
  const long long t0 = (long long)(blockIdx.x - L.first[k]) * kAdamPerBlock + threadIdx.x;
  float* __restrict__ p = L.p[k];
  const float* __restrict__ g = L.g[k];
  float* __restrict__ m = L.m[k];
  float* __restrict__ v = L.v[k];
  const long long n = L.n[k];
#pragma unroll
  for (int u = 0; u < kAdamPerBlock / 256; ++u) {
    const long long t = t0 + u * 256;
    if (t >= n) return;
    const float gt = g[t];
    const float mt = b1 * m[t] + (1.0f - b1) * gt;
    const float vt = b2 * v[t] + (1.0f - b2) * gt * gt;
    m[t] = mt;
    v[t] = vt;
    p[t] -= lr * mt / (sqrtf(vt) + eps);
  }
}

inline unsigned nblk(long long n, int t) { return (unsigned)((n + t - 1) / t); }


bool aligned_to(const void* p, size_t n) { return (reinterpret_cast<uintptr_t>(p) & (n - 1)) == 0; }

// Forward pointwise layer; yb may be null.
int pointwise_fwd(int32_t B, int32_t G, int32_t Cin, int32_t Cout, const float* x, const float* W,
                  const float* bias, const float* s, int32_t act, float* z, float* y, void* yb,
                  cudaStream_t st) {
  // two nodes per access: even rows, 8-byte (bf16 output: 4-byte) aligned bases
  const int vec = G % 2 == 0 && aligned_to(x, 8) && aligned_to(s, 8) && aligned_to(z, 8) &&
                  aligned_to(y, 8) && aligned_to(yb, 4);
  const unsigned nb = nblk((long long)B * ((G + 1) / 2), 128);
  __nv_bfloat16* ybf = static_cast<__nv_bfloat16*>(yb);
  if (Cin <= 8)
    k_pointwise_fwd<8, kMaxC><<<nb, 128, 0, st>>>(B, G, Cin, Cout, x, W, bias, s, act, z, y, ybf, vec,
                                                      -0.0f);
  else
    k_pointwise_fwd<kMaxC, kMaxC><<<nb, 128, 0, st>>>(B, G, Cin, Cout, x, W, bias, s, act, z, y, ybf,
                                                      vec, -0.0f);
  cv::count_launches(1);
  return check_launch("cvlbm_fno_pointwise_fwd");
}

// Backward pointwise layer; z (dz = dy gelu'(z)), dx and dzb may be null.
int pointwise_bwd(int32_t B, int32_t G, int32_t Cin, int32_t Cout, const float* dy, const float* z,
                  const float* x, const float* W, float* dx, int32_t accumulate, void* dzb, float* dW,
                  float* db, float* scratch, cudaStream_t st) {
  const int chunks = (G + kChunkG - 1) / kChunkG, nparts = B * chunks;
  __nv_bfloat16* d16 = static_cast<__nv_bfloat16*>(dzb);
  if (Cin <= 8)
    k_pointwise_bwd<8, kMaxC><<<nparts, kChunkG, 0, st>>>(B, G, Cin, Cout, dy, z, x, W, accumulate, dx,
                                                          d16, scratch, -0.0f);
  else if (Cout <= 16)
    k_pointwise_bwd<kMaxC, 16><<<nparts, kChunkG, 0, st>>>(B, G, Cin, Cout, dy, z, x, W, accumulate,
                                                           dx, d16, scratch, -0.0f);
  else
    k_pointwise_bwd<kMaxC, kMaxC><<<nparts, kChunkG, 0, st>>>(B, G, Cin, Cout, dy, z, x, W, accumulate,
                                                              dx, d16, scratch, -0.0f);
  cv::count_launches(1);
  const int n_w = Cout * Cin, width = n_w + Cout;
  k_sum_parts<<<nblk(width, 32), 32 * (kSumLoaders + 1), 0, st>>>(nparts, width, n_w, scratch, dW, db);
  cv::count_launches(1);
  return check_launch("cvlbm_fno_pointwise_bwd");
}

}  // namespace

extern "C" int cvlbm_fno_pointwise_fwd(int32_t B, int32_t G, int32_t Cin, int32_t Cout,
                                       const float* x, const float* W, const float* bias,
                                       const float* s, int32_t act, float* z, float* y,
                                       void* stream) {
  if (Cin > kMaxC || Cout > kMaxC || Cin <= 0 || Cout <= 0)
    return fail(CVLBM_ERR_INVALID_ARG, "cvlbm_fno_pointwise_fwd: 1..32 channels");
  return pointwise_fwd(B, G, Cin, Cout, x, W, bias, s, act, z, y, nullptr, (cudaStream_t)stream);
}

extern "C" int cvlbm_fno_layer_fwd(int32_t B, int32_t G, int32_t Cin, int32_t Cout, const float* x,
                                   const float* W, const float* bias, const float* s, int32_t act,
                                   float* z, float* y, void* y_bf16, void* stream) {
  if (Cin > kMaxC || Cout > kMaxC || Cin <= 0 || Cout <= 0)
    return fail(CVLBM_ERR_INVALID_ARG, "cvlbm_fno_layer_fwd: 1..32 channels");
  return pointwise_fwd(B, G, Cin, Cout, x, W, bias, s, act, z, y, y_bf16, (cudaStream_t)stream);
}

extern "C" int cvlbm_fno_gelu_bwd(int64_t n, const float* z, const float* dy, float* dz,
                                  void* stream) {
  k_gelu_bwd<<<nblk(n, 256), 256, 0, (cudaStream_t)stream>>>(n, z, dy, dz);
  cv::count_launches(1);
  return check_launch("cvlbm_fno_gelu_bwd");
}

extern "C" int cvlbm_fno_pointwise_bwd(int32_t B, int32_t G, int32_t Cin, int32_t Cout,
                                       const float* dz, const float* x, const float* W,
                                       float* dx, int32_t accumulate_dx, float* dW, float* db,
                                       float* scratch, void* stream) {
  if (Cin > kMaxC || Cout > kMaxC || Cin <= 0 || Cout <= 0)
    return fail(CVLBM_ERR_INVALID_ARG, "cvlbm_fno_pointwise_bwd: 1..32 channels");
  return pointwise_bwd(B, G, Cin, Cout, dz, nullptr, x, W, dx, accumulate_dx, nullptr, dW, db, scratch,
                       (cudaStream_t)stream);
}

extern "C" int cvlbm_fno_layer_bwd(int32_t B, int32_t G, int32_t Cin, int32_t Cout, const float* dy,
                                   const float* z, const float* x, const float* W, float* dx,
                                   void* dz_bf16, float* dW, float* db, float* scratch,
                                   void* stream) {
  if (Cin > kMaxC || Cout > kMaxC || Cin <= 0 || Cout <= 0)
    return fail(CVLBM_ERR_INVALID_ARG, "cvlbm_fno_layer_bwd: 1..32 channels");
  return pointwise_bwd(B, G, Cin, Cout, dy, z, x, W, dx, 0, dz_bf16, dW, db, scratch,
                       (cudaStream_t)stream);
}

extern "C" int64_t cvlbm_fno_pointwise_scratch(int32_t B, int32_t G, int32_t Cin,
                                               int32_t Cout) {
  const long long chunks = (G + kChunkG - 1) / kChunkG;
  return ((long long)B * chunks + 1) * ((long long)Cout * Cin + Cout);
}

extern "C" int cvlbm_fno_spec_mix_fwd(int32_t B, int32_t C, int32_t M, const float* a,
                                      const float* R, void* bh_bf16, void* stream) {
  if (C > kMaxC) return fail(CVLBM_ERR_INVALID_ARG, "cvlbm_fno_spec_mix_fwd: C <= 32");
  k_spec_mix_fwd<<<nblk(M, kMixK), 32 * kMixK, 0, (cudaStream_t)stream>>>(
      B, C, M, a, R, static_cast<__nv_bfloat16*>(bh_bf16));
  cv::count_launches(1);
  return check_launch("cvlbm_fno_spec_mix_fwd");
}

extern "C" int cvlbm_fno_spec_mix_bwd(int32_t B, int32_t C, int32_t M, const float* a,
                                      const float* dbh, const float* R, void* da_bf16,
                                      float* dR, void* stream) {
  if (C > kMaxC) return fail(CVLBM_ERR_INVALID_ARG, "cvlbm_fno_spec_mix_bwd: C <= 32");
  cudaFuncSetAttribute(k_spec_mix_bwd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMixBwdSmem);
  k_spec_mix_bwd<<<nblk(M, kMixK), 32 * kMixK, kMixBwdSmem, (cudaStream_t)stream>>>(
      B, C, M, a, dbh, R, static_cast<__nv_bfloat16*>(da_bf16), dR);
  cv::count_launches(1);
  return check_launch("cvlbm_fno_spec_mix_bwd");
}

extern "C" int cvlbm_fno_to_bf16(int64_t n, const float* src, void* dst, void* stream) {
  k_to_bf16<<<nblk(n, 256), 256, 0, (cudaStream_t)stream>>>(n, src,
                                                           static_cast<__nv_bfloat16*>(dst));
  cv::count_launches(1);
  return check_launch("cvlbm_fno_to_bf16");
}

extern "C" int cvlbm_fno_mse(int32_t B, int32_t C, int32_t G, const float* y, const float* t,
                             const float* mask, const float* w, float inv_count, float* dy,
                             float* part, int32_t n_parts, void* stream) {
  k_mse<<<n_parts, 256, 0, (cudaStream_t)stream>>>(B, C, G, y, t, mask, w, inv_count, nullptr, dy,
                                                  part);
  cv::count_launches(1);
  return check_launch("cvlbm_fno_mse");
}

extern "C" int cvlbm_fno_mse_mean(int32_t B, int32_t C, int32_t G, const float* y, const float* t,
                                  const float* mask, const float* w, const float* mask_sum, float* dy,
                                  float* part, int32_t n_parts, void* stream) {
  if (!mask_sum) return fail(CVLBM_ERR_INVALID_ARG, "cvlbm_fno_mse_mean: null mask_sum");
  k_mse<<<n_parts, 256, 0, (cudaStream_t)stream>>>(B, C, G, y, t, mask, w, 1.0f, mask_sum, dy, part);
  cv::count_launches(1);
  return check_launch("cvlbm_fno_mse_mean");
}

extern "C" int cvlbm_fno_adam(int64_t n, float* p, const float* g, float* m, float* v, float lr,
                              float b1, float b2, float eps, void* stream) {
  k_adam<<<nblk(n, 256), 256, 0, (cudaStream_t)stream>>>(n, p, g, m, v, lr, b1, b2, eps);
  cv::count_launches(1);
  return check_launch("cvlbm_fno_adam");
}

extern "C" int cvlbm_fno_adam_list(int32_t count, const int64_t* n, float* const* p,
                                   const float* const* g, float* const* m, float* const* v, float lr,
                                   float b1, float b2, float eps, void* stream) {
  if (count < 0 || (count > 0 && (!n || !p || !g || !m || !v)))
    return fail(CVLBM_ERR_INVALID_ARG, "cvlbm_fno_adam_list: null table");
  for (int32_t k0 = 0; k0 < count; k0 += kAdamTensors) {
    AdamList L{};
    unsigned long long blocks = 0;
    L.count = count - k0 < kAdamTensors ? count - k0 : kAdamTensors;
    for (int k = 0; k < L.count; ++k) {
      L.p[k] = p[k0 + k];
      L.g[k] = g[k0 + k];
      L.m[k] = m[k0 + k];
      L.v[k] = v[k0 + k];
      L.n[k] = n[k0 + k];
      L.first[k] = (unsigned)blocks;
      blocks += (unsigned long long)((n[k0 + k] + kAdamPerBlock - 1) / kAdamPerBlock);
    }
    L.first[L.count] = (unsigned)blocks;
    if (blocks > 0x7fffffffULL) return fail(CVLBM_ERR_INVALID_ARG, "cvlbm_fno_adam_list: too large");
    if (blocks == 0) continue;
    k_adam_list<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(L, lr, b1, b2, eps);
    cv::count_launches(1);
  }
  return check_launch("cvlbm_fno_adam_list");
}
