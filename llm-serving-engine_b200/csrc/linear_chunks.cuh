// Linear attention with a decay per head for long portions, as matrix products over chunks of 64 tokens:
//
//   E_c = sum_j d^(n_c - 1 - j) k_j v_j^T                         (chunk c alone, n_c tokens, j from 0)
//   F_c = the state before chunk c;   F_(c+1) = d^n_c F_c + E_c
//   O   = (tril(Q K^T) * d^(i - j)) V + d^(i + 1) Q F_c           per chunk
//
// Three launches: E_c of every (chunk, head) side by side; the chain over the chunks, element by element, which leaves
// F_c where E_c was; the outputs of every (chunk, head) side by side.
//
// The products are float32 products on the tensor cores (split_mma.cuh). Relative to float64, 16 heads of 128 x 128, 2048
// tokens: 1.6e-7, where the same products on the CUDA cores had 2.2e-7 and the recurrence, token by token, 2.1e-7. Operands
// split into two tf32 numbers were built and dropped: 9e-7, and no faster.
//
// What bounds it: 2.0e9 multiply-adds are 29 us of the tensor cores at six products each (sums 11, outputs 18; 36 us of the
// CUDA cores at their peak), and around them each block waits for its rows, activates them and waits for the others:
// two blocks an SM overlap that. Rows are copied to shared memory as they lie and changed there by one copy of the
// code: through registers, with the code inlined for each operand, instructions were what a block waited for most
// (3.6 of 11 cycles an instruction), and the tensor cores gained nothing.
// Back to back at these sizes: recurrence 313 us, products on the CUDA cores 150, now 124; portions of 700 tokens 72 -> 62.
// In a model's step (with silu or rotation) the outputs take 75 us where they took 94, the sums 41 as before, the chain 19.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "split_mma.cuh"

namespace lse {
namespace lac {

constexpr int L = 64, THREADS = 256, MAX = 128;  // tokens per chunk; largest key and value size

struct Args {
  const float* proj;    // [T, stride]: q (H dk) | k (H dk) | v (H dv) | ... per row
  long long stride;
  float* out;           // [T, H dv]
  float* state;         // [slots, H, dv, dk]
  float* chunks;        // [chunks of all chunked sequences, H, dv, dk]
  const float* decay;   // [H]
  const int* cu_q;
  const int* ctx_lens;
  const int* slots;
  const float* cos;     // [positions, rot / 2] or null
  const float* sin;
  int H, dk, dv, rot, silu;
  float key_scale, query_scale;
};

struct Chunk {  // where this block's chunk lies
  int r0, t0, n, pos;      // first row of the sequence and of the chunk, tokens of the chunk, position of its first
  size_t at;               // index of the chunk in the scratch
  bool any;
};

__device__ __forceinline__ Chunk find(const Args& a, int c, int seq) {
  Chunk k;
  int base = 0;  // only sequences of more than one chunk have any
  for (int s = 0; s < seq; ++s) {
    const int m = a.cu_q[s + 1] - a.cu_q[s];
    base += m > L ? (m + L - 1) / L : 0;
  }
  k.r0 = a.cu_q[seq];
  const int n = a.cu_q[seq + 1] - k.r0;
  k.any = n > L && c * L < n;
  k.t0 = k.r0 + c * L;
  k.n = min(L, n - c * L);
  k.pos = a.ctx_lens[seq] - n + c * L;
  k.at = (size_t)(base + c);
  return k;
}

// pw[i] = d^i, i = 0 .. L, by squaring in float64
__device__ __forceinline__ void powers(float* pw, float d) {
  for (int i = threadIdx.x; i <= L; i += THREADS) {
    double r = 1., b = (double)d;
    for (int e = i; e; e >>= 1, b *= b)
      if (e & 1) r *= b;
    pw[i] = (float)r;
  }
}

__device__ __forceinline__ float act(float z, int silu) { return silu ? z / (1.f + expf(-z)) : z; }

// 64 rows of `len` columns of proj (from column `col`) are asked for, into rows `ld` apart; rows from n on are zero, and
// so is what lies behind `len` up to a multiple of 16.
__device__ __forceinline__ void ask(float* dst, int ld, const Args& a, const Chunk& k, int col, int len) {
  const int units = (len + 15) / 16 * 4, per = THREADS / units, t0 = threadIdx.x / units;
  const int i = (threadIdx.x - t0 * units) * 4;
  if (t0 < per)
#pragma unroll 1
    for (int t = t0; t < L; t += per) {
      const bool there = t < k.n && i < len;
      const float* src = a.proj + (there ? (size_t)(k.t0 + t) * a.stride + col + i : 0);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst + t * ld + i)),
                   "l"(src), "r"(there ? 16 : 0));
    }
  asm volatile("cp.async.commit_group;\n" ::);
}
__device__ __forceinline__ void arrived() {
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
}

// In place: n rows activated, their first `rot` columns rotated (pairs half a rotation apart, position t0 + row), row t
// times `scale` and, counted from the last row, pw[0], pw[1], ... Rows behind them are zero and stay so. One copy of this
// code for all operands: with the values on their way through registers and the code once per operand, a block waited
// for instructions most of its time.
static __device__ __noinline__ void transform(float* rows, int ld, int n, int len, int rot, int silu, const float* cos,
                                       const float* sin, size_t pos, float scale, const float* pw) {
  const int half = rot / 2;
  auto done = [&](float4 x) { return make_float4(act(x.x, silu), act(x.y, silu), act(x.z, silu), act(x.w, silu)); };
  auto factor = [&](int t) { return pw ? scale * pw[n - 1 - t] : scale; };
  const bool whole = half % 4 == 0;  // pairs in 16-byte pieces
  if (half > 0 && whole) {
    const int units = half / 4, per = THREADS / units, t0 = threadIdx.x / units, i = (threadIdx.x - t0 * units) * 4;
    if (t0 < per)
#pragma unroll 1
      for (int t = t0; t < n; t += per) {
        float4* pu = reinterpret_cast<float4*>(rows + t * ld + i);
        float4* pv = reinterpret_cast<float4*>(rows + t * ld + half + i);
        const float4 cs = *reinterpret_cast<const float4*>(cos + (pos + t) * half + i);
        const float4 sn = *reinterpret_cast<const float4*>(sin + (pos + t) * half + i);
        const float4 u = done(*pu), v = done(*pv);
        const float f = factor(t);
        *pu = make_float4((u.x * cs.x - v.x * sn.x) * f, (u.y * cs.y - v.y * sn.y) * f, (u.z * cs.z - v.z * sn.z) * f,
                          (u.w * cs.w - v.w * sn.w) * f);
        *pv = make_float4((v.x * cs.x + u.x * sn.x) * f, (v.y * cs.y + u.y * sn.y) * f, (v.z * cs.z + u.z * sn.z) * f,
                          (v.w * cs.w + u.w * sn.w) * f);
      }
  }
  const int first = whole ? rot : 0;  // (rot is a multiple of 8 then)
  if (first < len && (silu || pw || scale != 1.f)) {
    const int units = (len - first) / 4, per = THREADS / units, t0 = threadIdx.x / units;
    const int i = first + (threadIdx.x - t0 * units) * 4;
    if (t0 < per)
#pragma unroll 1
      for (int t = t0; t < n; t += per) {
        float4* p = reinterpret_cast<float4*>(rows + t * ld + i);
        const float4 x = done(*p);
        const float f = factor(t);
        *p = make_float4(x.x * f, x.y * f, x.z * f, x.w * f);
      }
  }
  if (half > 0 && !whole) {  // odd sizes: rotated behind the rest (the factor is in both of a pair)
    __syncthreads();
#pragma unroll 1
    for (int idx = threadIdx.x; idx < n * half; idx += THREADS) {
      const int t = idx / half, w = idx - t * half;
      float* row = rows + t * ld;
      const size_t tab = (pos + t) * half + w;
      const float cs = cos[tab], sn = sin[tab], u = row[w], v = row[w + half];
      row[w] = u * cs - v * sn;
      row[w + half] = v * cs + u * sn;
    }
  }
}
__device__ __forceinline__ void transform(float* rows, int ld, const Args& a, const Chunk& k, int len, int rot, float scale,
                                          const float* pw = nullptr) {
  transform(rows, ld, k.n, len, rot, a.silu, a.cos, a.sin, (size_t)k.pos, scale, pw);
}

// ---- E_c, [dv][dk]: a warp has 32 VH rows and 16 KH columns of it
template <int VH, int KH>
__global__ void __launch_bounds__(THREADS, 2) chunk_sums_kernel(const Args a) {
  extern __shared__ __align__(16) float smem[];
  __shared__ float pw[L + 1];
  pdl_trigger();
  const Chunk k = find(a, blockIdx.x, blockIdx.z);
  if (!k.any) {
    pdl_wait();  // no block leaves before the kernels before this one are done: the next kernel counts on it
    return;
  }
  const int h = blockIdx.y, dk = a.dk, dv = a.dv;
  constexpr int LDK = 64 * KH + 4, LDV = 64 * VH + 4;  // (columns beyond dk and dv are never stored)
  float* ks = smem;            // [64][LDK]
  float* vs = ks + L * LDK;    // [64][LDV]
  powers(pw, a.decay[h]);
  pdl_wait();
  ask(ks, LDK, a, k, (a.H + h) * dk, dk);
  ask(vs, LDV, a, k, 2 * a.H * dk + h * dv, dv);
  arrived();
  transform(ks, LDK, a, k, dk, a.rot, a.key_scale, pw);
  transform(vs, LDV, a, k, dv, 0, 1.f);
  __syncthreads();
  const int warp = threadIdx.x >> 5, g = (threadIdx.x & 31) >> 2, q = threadIdx.x & 3;
  const int r0 = (warp >> 2) * 32 * VH, c0 = (warp & 3) * 16 * KH;
  float acc[2 * VH][2 * KH][4];
#pragma unroll
  for (int i = 0; i < 2 * VH; ++i)
#pragma unroll
    for (int j = 0; j < 2 * KH; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
#pragma unroll 1
  for (int t = 0; t < L; t += 16) {
    split::B y[2 * KH];
#pragma unroll
    for (int j = 0; j < 2 * KH; ++j) split::down(y[j], ks + t * LDK + c0 + 8 * j + g, LDK, q);
#pragma unroll
    for (int i = 0; i < 2 * VH; ++i) {
      split::A x;
      split::down(x, vs + t * LDV + r0 + 16 * i + g, LDV, q);
      split::multiply_add(acc[i], x, y);
    }
  }
  float* to = a.chunks + (k.at * a.H + h) * (size_t)dv * dk;
#pragma unroll
  for (int i = 0; i < 2 * VH; ++i) {
    const bool again = split::strange(acc[i]);
#pragma unroll
    for (int j = 0; j < 2 * KH; ++j)
#pragma unroll
      for (int e = 0; e < 4; e += 2) {
        const int r = r0 + 16 * i + g + 4 * e, c = c0 + 8 * j + 2 * q;
        if (r >= dv || c >= dk) continue;
        float* x = acc[i][j] + e;
        if (again) {
          if (!split::finite(x[0])) x[0] = split::dot(vs + r, LDV, ks + c, LDK, L);
          if (!split::finite(x[1])) x[1] = split::dot(vs + r, LDV, ks + c + 1, LDK, L);
        }
        *reinterpret_cast<float2*>(to + (size_t)r * dk + c) = make_float2(x[0], x[1]);
      }
  }
}

// ---- the chain: E_c gives way to F_c; the state after the last chunk is the request's
__global__ void chain_kernel(const Args a) {
  pdl_trigger();
  const int seq = blockIdx.y;
  const Chunk k = find(a, 0, seq);
  const size_t per = (size_t)a.H * a.dv * a.dk, e = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (!k.any || e >= per) {
    pdl_wait();
    return;
  }
  const int n = a.cu_q[seq + 1] - k.r0, chunks = (n + L - 1) / L;
  const double d = (double)a.decay[e / ((size_t)a.dv * a.dk)];
  auto power = [&](int len) {
    double r = 1., b = d;
    for (int i = len; i; i >>= 1, b *= b)
      if (i & 1) r *= b;
    return (float)r;
  };
  const float whole = power(L), last = power(n - (chunks - 1) * L);
  float* st = a.state + (size_t)a.slots[seq] * per + e;
  float* mine = a.chunks + k.at * per + e;
  pdl_wait();
  float S[4] = {0.f, 0.f, 0.f, 0.f};
  if (k.pos > 0) load4<float>(st, S);
  constexpr int U = 4;  // a round's loads are all in flight before its chain
  for (int c0 = 0; c0 < chunks; c0 += U) {
    float E[U][4];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (c0 + u < chunks) load4<float>(mine + (size_t)(c0 + u) * per, E[u]);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int c = c0 + u;
      if (c < chunks) {
        store4<float>(mine + (size_t)c * per, S);
        const float f = c + 1 < chunks ? whole : last;
#pragma unroll
        for (int i = 0; i < 4; ++i) S[i] = fmaf(f, S[i], E[u][i]);
      }
    }
  }
  store4<float>(st, S);
}

// ---- outputs: a warp has 32 rows and 4 M columns of them
// Rows of q, k and F are ld_of(dk) floats apart, zeros behind dk up to a multiple of 16.
__host__ __device__ constexpr int ld_of(int dk) { return ((dk + 15) / 16 * 16) | 16; }
constexpr int LDP = L + 8;

// The sum of n values with weights: `sum`, unless it or one of the values is no number.
static __device__ __noinline__ float weighted(const float* p, const float* v, int ldv, int n, float sum) {
  bool fine = split::finite(sum);
#pragma unroll 1
  for (int t = 0; t < n; ++t) fine = fine && split::finite(v[t * ldv]);
  return fine ? sum : split::dot(p, 1, v, ldv, n);
}

template <int M>
__global__ void __launch_bounds__(THREADS, 2) chunk_outputs_kernel(const Args a) {
  extern __shared__ __align__(16) float smem[];
  __shared__ float pw[L + 1];
  pdl_trigger();
  const Chunk k = find(a, blockIdx.x, blockIdx.z);
  if (!k.any) {
    pdl_wait();
    return;
  }
  const int h = blockIdx.y, dk = a.dk, dv = a.dv, ld = ld_of(dk), tid = threadIdx.x;
  constexpr int LDV = 16 * M + 4, NT = M / 2;  // tiles of eight columns of a warp
  float* qs = smem;                            // [64][ld]; then the scores, [64][LDP]
  float* fs = qs + L * (ld > LDP ? ld : LDP);  // F [dv][ld]; then k [64][ld], v [64][LDV]
  float* ks = fs;
  float* vs = ks + L * ld;
  powers(pw, a.decay[h]);
  pdl_wait();
  const float* F = a.chunks + (k.at * a.H + h) * (size_t)dv * dk;
  {
    const int units = (dk + 15) / 16 * 4, per = THREADS / units, j0 = tid / units, i = (tid - j0 * units) * 4;
    if (j0 < per)
#pragma unroll 1
      for (int j = j0; j < dv; j += per) {
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(fs + j * ld + i);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(F + (i < dk ? (size_t)j * dk + i : 0)),
                     "r"(i < dk ? 16 : 0));
      }
  }
  ask(qs, ld, a, k, h * dk, dk);
  arrived();
  transform(qs, ld, a, k, dk, a.rot, 1.f);
  __syncthreads();
  const int warp = tid >> 5, g = (tid & 31) >> 2, q = tid & 3;
  const int r0 = (warp >> 2) * 32, c0 = (warp & 3) * 8 * NT;
  float acc[2][NT][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
  // (columns beyond dv are sums of whatever lies there, and are never stored)
#pragma unroll 1
  for (int d = 0; d < dk; d += 16) {
    split::B f[NT];
#pragma unroll
    for (int j = 0; j < NT; ++j) split::along(f[j], fs + (c0 + 8 * j + g) * ld + d, q);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      split::A x;
      split::along(x, qs + (r0 + 16 * i + g) * ld + d, ld, q);
      split::multiply_add(acc[i], x, f);
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const bool again = split::strange(acc[i]);
    const float f[2] = {pw[r0 + 16 * i + g + 1], pw[r0 + 16 * i + g + 9]};
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int r = r0 + 16 * i + g + 8 * (e >> 1), c = c0 + 8 * j + 2 * q + (e & 1);
        if (again && c < dv && !split::finite(acc[i][j][e])) acc[i][j][e] = split::dot(qs + r * ld, 1, fs + c * ld, 1, dk);
        acc[i][j][e] *= f[e >> 1];
      }
  }
  __syncthreads();  // F is used up: k and v take its place
  ask(ks, ld, a, k, (a.H + h) * dk, dk);
  ask(vs, LDV, a, k, 2 * a.H * dk + h * dv, dv);
  arrived();
  transform(ks, ld, a, k, dk, a.rot, a.key_scale);
  transform(vs, LDV, a, k, dv, 0, 1.f);
  __syncthreads();
  {
    // Scores: a warp has 16 rows and every other one of the tiles of eight columns up to their diagonal; the two warps
    // that issue from the same quarter of the SM have five tiles together.
    const int m = warp < 4 ? warp >> 1 : 3 - ((warp - 4) >> 1), odd = warp & 1;
    float s[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[j][e] = 0.f;
#pragma unroll 1
    for (int d = 0; d < dk; d += 16) {
      split::A x;
      split::along(x, qs + (16 * m + g) * ld + d, ld, q);
#pragma unroll
      for (int j = 0; j < 4; j += 2) {
        if (j > m) break;
        split::B y[2];
        split::along(y[0], ks + (16 * j + 8 * odd + g) * ld + d, q);
        if (j + 1 <= m) {
          split::along(y[1], ks + (16 * j + 16 + 8 * odd + g) * ld + d, q);
          split::multiply_add(reinterpret_cast<float(&)[2][4]>(s[j]), x, y);
        } else {
          split::multiply_add(reinterpret_cast<float(&)[1][4]>(s[j]), x, reinterpret_cast<const split::B(&)[1]>(y[0]));
        }
      }
    }
    if (split::strange(s)) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (j <= m && !split::finite(s[j][e]))
            s[j][e] = split::dot(qs + (16 * m + g + 8 * (e >> 1)) * ld, 1, ks + (16 * j + 8 * odd + 2 * q + (e & 1)) * ld, 1, dk);
    }
    __syncthreads();  // q is used up
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; e += 2)
        if (j <= m) {
          const int r = 16 * m + g + 4 * e, c = 16 * j + 8 * odd + 2 * q, back = r - c;
          *reinterpret_cast<float2*>(qs + r * LDP + c) = make_float2(back >= 0 ? s[j][e] * pw[max(back, 0)] : 0.f,
                                                                     back >= 1 ? s[j][e + 1] * pw[max(back - 1, 0)] : 0.f);
        }
  }
  __syncthreads();
  // Values, two tiles of columns at a time. Those that are no number are left out of the products (a later token's would
  // be met by a zero, and be no number all the same); sums that have one are taken again.
#pragma unroll
  for (int j0 = 0; j0 < NT; j0 += 2) {
    float part[2][2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) part[i][j][e] = 0.f;
    bool again = false;
#pragma unroll 1
    for (int t = 0; t < r0 + 32; t += 16) {
      split::B y[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float* p = vs + (t + 2 * q) * LDV + c0 + 8 * (j0 + j) + g;
        float x[4] = {p[0], p[LDV], p[8 * LDV], p[9 * LDV]};
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (!split::finite(x[e])) {
            x[e] = 0.f;
            again = again || c0 + 8 * (j0 + j) + g < dv;
          }
        y[j].set(0, x[0], x[1]), y[j].set(1, x[2], x[3]);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if (t > r0 + 16 * i) continue;
        split::A x;
        split::along_as_down(x, qs + (r0 + 16 * i + g) * LDP + t, LDP, q);
        split::multiply_add(part[i], x, y);
      }
    }
    again = __any_sync(0xffffffffu, again || split::strange(part[0]) || split::strange(part[1]));
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (again) {
            const int r = r0 + 16 * i + g + 8 * (e >> 1), c = c0 + 8 * (j0 + j) + 2 * q + (e & 1);
            if (c < dv) part[i][j][e] = weighted(qs + r * LDP, vs + c, LDV, r + 1, part[i][j][e]);
          }
          acc[i][j0 + j][e] += part[i][j][e];
        }
    __syncwarp();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int e = 0; e < 4; e += 2) {
      const int t = r0 + 16 * i + g + 4 * e;
      if (t >= k.n) continue;
      float* to = a.out + (size_t)(k.t0 + t) * ((size_t)a.H * dv) + (size_t)h * dv + c0 + 2 * q;
#pragma unroll
      for (int j = 0; j < NT; ++j)
        if (c0 + 8 * j + 2 * q < dv) {
          to[8 * j] = acc[i][j][e] * a.query_scale;
          to[8 * j + 1] = acc[i][j][e + 1] * a.query_scale;
        }
    }
}

// Rows of whole 16-byte pieces, and sizes whose tiles fit the shared memory.
inline bool serves(const Args& a) {
  auto aligned = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  return a.dk <= MAX && a.dv <= MAX && a.dk % 4 == 0 && a.dv % 4 == 0 && a.stride % 4 == 0 && aligned(a.proj) &&
         aligned(a.state) && aligned(a.chunks) && aligned(a.cos) && aligned(a.sin) && a.H <= 65535;
}

template <int VH, int KH>
inline bool launch_sums(const Args& a, dim3 grid, cudaStream_t stream) {
  constexpr int smem = L * (64 * (VH + KH) + 8) * 4;
  return allow_dynamic_smem<chunk_sums_kernel<VH, KH>, smem>() == cudaSuccess &&
         launch(chunk_sums_kernel<VH, KH>, grid, THREADS, smem, stream, a) == cudaSuccess;
}
template <int M>
inline bool launch_outputs(const Args& a, dim3 grid, cudaStream_t stream) {
  auto bytes = [](int ld, int dv) {
    const int first = dv * ld, second = L * (ld + 16 * M + 4);
    return (L * (ld > LDP ? ld : LDP) + (first > second ? first : second)) * 4;
  };
  constexpr int most = bytes(ld_of(MAX), 16 * M);
  const int smem = bytes(ld_of(a.dk), 16 * M);
  return allow_dynamic_smem<chunk_outputs_kernel<M>, most>() == cudaSuccess &&
         launch(chunk_outputs_kernel<M>, grid, THREADS, smem, stream, a) == cudaSuccess;
}

// The sequences of more than L tokens: max_chunks bounds the chunks of any.
inline int run(const Args& a, int num_seqs, int max_chunks, cudaStream_t stream) {
  const dim3 grid(max_chunks, a.H, num_seqs);
  const bool wide_v = a.dv > 64, wide_k = a.dk > 64;
  bool ok = wide_v ? (wide_k ? launch_sums<2, 2>(a, grid, stream) : launch_sums<2, 1>(a, grid, stream))
                   : (wide_k ? launch_sums<1, 2>(a, grid, stream) : launch_sums<1, 1>(a, grid, stream));
  const size_t quads = (size_t)a.H * a.dv * a.dk / 4;
  ok = ok && launch(chain_kernel, dim3((unsigned)((quads + 127) / 128), num_seqs), 128, 0, stream, a) == cudaSuccess;
  ok = ok && (wide_v ? launch_outputs<8>(a, grid, stream) : launch_outputs<4>(a, grid, stream));
  return ok ? LSE_OK : LSE_LAUNCH_FAILED;
}

}  // namespace lac
}  // namespace lse
