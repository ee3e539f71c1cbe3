// Linear attention with a decay per head for long portions, as matrix products over chunks of 64 tokens:
//
//   E_c = sum_j d^(n_c - 1 - j) k_j v_j^T                         (chunk c alone, n_c tokens, j from 0)
//   F_c = the state before chunk c;   F_(c+1) = d^n_c F_c + E_c
//   O   = (tril(Q K^T) * d^(i - j)) V + d^(i + 1) Q F_c           per chunk
//
// Three launches: E_c of every (chunk, head) side by side; the chain over the chunks, element by element, which leaves
// F_c where E_c was; the outputs of every (chunk, head) side by side.
//
// Everything is float32 on the CUDA cores. Operands split into two tf32 numbers on the tensor cores (three multiplies for
// a product) were built and dropped: relative to float64 9e-7 where this has 1.8e-7 and the recurrence, token by
// token, had 2.1e-7 (16 heads of 128 x 128, 2048 tokens), and no faster (each split is four instructions).
//
// What bounds it: the 16-byte reads of shared memory in the outputs (four passes each, 48 for 128 multiply-adds of a
// warp) and the FMA units; 1.4e9 multiply-adds at these sizes are 36 us at their peak. 269 us with the recurrence ->
// 149 us (sums 40, chain 41 from memory, outputs 106 with cold caches, overlapped). With silu, back to back, recurrence ->
// products -> products that pass over later tokens' values and do not activate rows beyond a chunk's tokens: 2048 tokens
// 313 -> 155 -> 167 us, 8192 tokens 1204 -> 631 -> 633, portions of 700 and 1300 tokens 311 -> 163 -> 146.
#pragma once

#include <type_traits>

#include "common.cuh"

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

// Sixty-four rows of `units` pieces of work each: fetch(row, piece) of up to B rows are in flight before put(row,
// piece, what it fetched) of the first.
template <int B, typename Fetch, typename Put>
__device__ __forceinline__ void for_rows(int units, Fetch fetch, Put put) {
  const int per = THREADS / units, t0 = threadIdx.x / units, u = threadIdx.x - t0 * units;
  if (t0 >= per) return;
#pragma unroll 1
  for (int t = t0; t < L; t += B * per) {
    decltype(fetch(0, 0)) x[B];
#pragma unroll
    for (int b = 0; b < B; ++b)
      if (t + b * per < L) x[b] = fetch(t + b * per, u);
#pragma unroll
    for (int b = 0; b < B; ++b)
      if (t + b * per < L) put(t + b * per, u, x[b]);
  }
}

struct Pair {
  float4 u, v, cs, sn;
};

// 64 rows of `len` columns of proj (from column `col`) into rows `ld` apart: activated, the first `rot` columns rotated
// (pairs half a rotation apart), row t times factor(t). Rows from n on are zero, and are not activated: the division of
// a zero takes the slow way (a portion of 65 tokens took longer than one of 128).
template <typename F>
__device__ __forceinline__ void stage(float* dst, int ld, const Args& a, const Chunk& k, int col, int len, int rot, F factor) {
  const int half = rot / 2;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  auto at = [&](int t, int i) {
    return t < k.n ? *reinterpret_cast<const float4*>(a.proj + (size_t)(k.t0 + t) * a.stride + col + i) : zero;
  };
  auto done = [&](float4 x, float f) {
    return make_float4(act(x.x, a.silu) * f, act(x.y, a.silu) * f, act(x.z, a.silu) * f, act(x.w, a.silu) * f);
  };
  auto store = [&](int t, int i, float4 x) { *reinterpret_cast<float4*>(dst + t * ld + i) = x; };
  const bool whole = half % 4 == 0;  // pairs in 16-byte pieces
  if (half > 0 && whole)
    for_rows<2>(half / 4,
        [&](int t, int i) {
          const size_t tab = (size_t)(k.pos + min(t, k.n - 1)) * half + 4 * i;
          return Pair{at(t, 4 * i), at(t, half + 4 * i), *reinterpret_cast<const float4*>(a.cos + tab),
                      *reinterpret_cast<const float4*>(a.sin + tab)};
        },
        [&](int t, int i, const Pair& p) {
          if (t >= k.n) {
            store(t, 4 * i, zero);
            store(t, half + 4 * i, zero);
            return;
          }
          const float4 u = done(p.u, 1.f), v = done(p.v, 1.f);
          const float f = factor(t);
          store(t, 4 * i, make_float4((u.x * p.cs.x - v.x * p.sn.x) * f, (u.y * p.cs.y - v.y * p.sn.y) * f,
                                      (u.z * p.cs.z - v.z * p.sn.z) * f, (u.w * p.cs.w - v.w * p.sn.w) * f));
          store(t, half + 4 * i, make_float4((v.x * p.cs.x + u.x * p.sn.x) * f, (v.y * p.cs.y + u.y * p.sn.y) * f,
                                             (v.z * p.cs.z + u.z * p.sn.z) * f, (v.w * p.cs.w + u.w * p.sn.w) * f));
        });
  const int first = whole ? rot : 0;  // (rot is a multiple of 8 then)
  if (first < len)
    for_rows<8>((len - first) / 4, [&](int t, int i) { return at(t, first + 4 * i); },
                [&](int t, int i, const float4& x) { store(t, first + 4 * i, t < k.n ? done(x, factor(t)) : zero); });
  if (half > 0 && !whole) {  // odd sizes: rotated in place (the factor is in both of a pair)
    __syncthreads();
    for (int idx = threadIdx.x; idx < L * half; idx += THREADS) {
      const int t = idx / half, w = idx - t * half;
      float* row = dst + t * ld;
      const size_t tab = (size_t)(k.pos + min(t, k.n - 1)) * half + w;
      const float cs = a.cos[tab], sn = a.sin[tab], u = row[w], v = row[w + half];
      row[w] = u * cs - v * sn;
      row[w + half] = v * cs + u * sn;
    }
  }
}

// ---- E_c, [dv][dk]: a thread has VH x KH tiles of 4 x 4, 64 rows and columns apart
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
  constexpr int LDK = 64 * KH, LDV = 64 * VH;  // (columns beyond dk and dv are never stored)
  float* ks = smem;            // [64][LDK]
  float* vs = ks + L * LDK;    // [64][LDV]
  powers(pw, a.decay[h]);
  __syncthreads();
  pdl_wait();
  stage(ks, LDK, a, k, (a.H + h) * dk, dk, a.rot, [&](int t) { return t < k.n ? a.key_scale * pw[k.n - 1 - t] : 0.f; });
  stage(vs, LDV, a, k, 2 * a.H * dk + h * dv, dv, 0, [](int) { return 1.f; });
  __syncthreads();
  const int tv = (threadIdx.x >> 4) * 4, tk = (threadIdx.x & 15) * 4;
  float acc[VH * 4][KH * 4];
#pragma unroll
  for (int i = 0; i < VH * 4; ++i)
#pragma unroll
    for (int j = 0; j < KH * 4; ++j) acc[i][j] = 0.f;
#pragma unroll 2
  for (int t = 0; t < L; ++t) {
    float x[VH][4], y[KH][4];
#pragma unroll
    for (int i = 0; i < VH; ++i) load4<float>(vs + t * LDV + 64 * i + tv, x[i]);
#pragma unroll
    for (int j = 0; j < KH; ++j) load4<float>(ks + t * LDK + 64 * j + tk, y[j]);
#pragma unroll
    for (int i = 0; i < VH * 4; ++i)
#pragma unroll
      for (int j = 0; j < KH * 4; ++j) acc[i][j] = fmaf(x[i / 4][i % 4], y[j / 4][j % 4], acc[i][j]);
  }
  float* to = a.chunks + (k.at * a.H + h) * (size_t)dv * dk;
#pragma unroll
  for (int i = 0; i < VH * 4; ++i) {
    const int r = 64 * (i / 4) + tv + i % 4;
    if (r >= dv) continue;
#pragma unroll
    for (int j = 0; j < KH; ++j)
      if (64 * j + tk < dk)
        *reinterpret_cast<float4*>(to + (size_t)r * dk + 64 * j + tk) =
            make_float4(acc[i][4 * j], acc[i][4 * j + 1], acc[i][4 * j + 2], acc[i][4 * j + 3]);
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

// ---- outputs: a thread has the rows ty + 16 i and the columns tx + 16 m. Rows of q, k and F are LDK = dk + 4 floats
// apart: the 16-byte reads of eight neighbouring columns then fall into different banks.
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
  const int h = blockIdx.y, dk = a.dk, dv = a.dv, ld = dk + 4, tid = threadIdx.x;
  constexpr int LDV = 16 * M, LDP = L + 4;
  float* qs = smem;             // [64][ld]; then the scores, [64][LDP]
  float* fs = qs + L * (dk > L ? ld : LDP);  // F [16 M][ld]; then k [64][ld], v [64][LDV]
  float* ks = fs;
  float* vs = ks + L * ld;
  powers(pw, a.decay[h]);
  pdl_wait();
  const float* F = a.chunks + (k.at * a.H + h) * (size_t)dv * dk;
  {
    const int units = dk / 4, per = THREADS / units, j0 = tid / units, i = (tid - j0 * units) * 4;
    if (j0 < per)
      for (int j = j0; j < dv; j += per) {
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(fs + j * ld + i);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(F + (size_t)j * dk + i));
      }
  }
  asm volatile("cp.async.commit_group;\n" ::);
  auto one = [](int) { return 1.f; };
  stage(qs, ld, a, k, h * dk, dk, a.rot, one);
  asm volatile("cp.async.wait_group 0;\n" ::);
  __syncthreads();
  const int ty = tid >> 4, tx = tid & 15;
  float acc[4][M];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int m = 0; m < M; ++m) acc[i][m] = 0.f;
  // (columns beyond dv are sums of whatever lies there, and are never stored)
  // Sums of more than 32 terms are sums of parts of 32 (and of 16 tokens below): a chain of 128 rounds more.
#pragma unroll 1
  for (int d0 = 0; d0 < dk; d0 += 32) {
    float part[4][M];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int m = 0; m < M; ++m) part[i][m] = 0.f;
    const int d1 = min(dk, d0 + 32);
#pragma unroll 1
    for (int d = d0; d < d1; d += 4) {
      float q[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) load4<float>(qs + (ty + 16 * i) * ld + d, q[i]);
#pragma unroll
      for (int m = 0; m < M; ++m) {
        float f[4];
        load4<float>(fs + (tx + 16 * m) * ld + d, f);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) part[i][m] = fmaf(q[i][e], f[e], part[i][m]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int m = 0; m < M; ++m) acc[i][m] += part[i][m];
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float f = pw[ty + 16 * i + 1];
#pragma unroll
    for (int m = 0; m < M; ++m) acc[i][m] *= f;
  }
  __syncthreads();  // F is used up: k and v take its place
  stage(ks, ld, a, k, (a.H + h) * dk, dk, a.rot, [&](int) { return a.key_scale; });
  stage(vs, LDV, a, k, 2 * a.H * dk + h * dv, dv, 0, one);
  __syncthreads();
  {
    float s[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 1
    for (int d0 = 0; d0 < dk; d0 += 32) {
      float part[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) part[i][j] = 0.f;
      const int d1 = min(dk, d0 + 32);
#pragma unroll 1
      for (int d = d0; d < d1; d += 4) {
        float kc[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) load4<float>(ks + (tx + 16 * j) * ld + d, kc[j]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float q[4];
          load4<float>(qs + (ty + 16 * i) * ld + d, q);
#pragma unroll
          for (int j = 0; j <= i; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) part[i][j] = fmaf(q[e], kc[j][e], part[i][j]);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j) s[i][j] += part[i][j];
    }
    __syncthreads();  // q is used up
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j <= i; ++j) {
        const int back = ty + 16 * i - (tx + 16 * j);
        qs[(ty + 16 * i) * LDP + tx + 16 * j] = back >= 0 ? s[i][j] * pw[max(back, 0)] : 0.f;
      }
  }
  __syncthreads();
#pragma unroll
  for (int b = 0; b < 4; ++b) {  // tokens of block b reach rows of the blocks i >= b
    float part[4][M];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int m = 0; m < M; ++m) part[i][m] = 0.f;
    // A later token's value is left out of the row's own block and not only met by a zero: it may be no number. A warp
    // has two rows of each block, so four tokens are all of them before, all of them behind, or looked at one by one.
    auto four = [&](int t, auto own) {
      float p[4][4];
#pragma unroll
      for (int i = b; i < 4; ++i) load4<float>(qs + (ty + 16 * i) * LDP + t, p[i]);
#pragma unroll
      for (int m = 0; m < M; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float v = vs[(t + e) * LDV + tx + 16 * m];
          if constexpr (own.value == 2) part[b][m] = fmaf(p[b][e], v, part[b][m]);
          if constexpr (own.value == 1) part[b][m] = fmaf(p[b][e], t + e <= ty + 16 * b ? v : 0.f, part[b][m]);
#pragma unroll
          for (int i = b + 1; i < 4; ++i) part[i][m] = fmaf(p[i][e], v, part[i][m]);
        }
    };
    const int mixed = 16 * b + (ty & ~3);  // (the same for both rows of the warp)
#pragma unroll 1
    for (int t = 16 * b; t < mixed; t += 4) four(t, std::integral_constant<int, 2>());
    four(mixed, std::integral_constant<int, 1>());
    if (b < 3)
#pragma unroll 1
      for (int t = mixed + 4; t < 16 * b + 16; t += 4) four(t, std::integral_constant<int, 0>());
#pragma unroll
    for (int i = b; i < 4; ++i)
#pragma unroll
      for (int m = 0; m < M; ++m) acc[i][m] += part[i][m];
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = ty + 16 * i;
    if (t >= k.n) continue;
    float* to = a.out + (size_t)(k.t0 + t) * ((size_t)a.H * dv) + (size_t)h * dv + tx;
#pragma unroll
    for (int m = 0; m < M; ++m)
      if (tx + 16 * m < dv) to[16 * m] = acc[i][m] * a.query_scale;
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
  constexpr int smem = L * 64 * (VH + KH) * 4;
  return allow_dynamic_smem<chunk_sums_kernel<VH, KH>, smem>() == cudaSuccess &&
         launch(chunk_sums_kernel<VH, KH>, grid, THREADS, smem, stream, a) == cudaSuccess;
}
template <int M>
inline bool launch_outputs(const Args& a, dim3 grid, cudaStream_t stream) {
  const int ld = a.dk + 4, first = 16 * M * ld, second = L * (ld + 16 * M);
  const int smem = (L * (a.dk > L ? ld : L + 4) + (first > second ? first : second)) * 4;
  constexpr int most = (L * (MAX + 4) + (16 * M > L ? 16 * M * (MAX + 4) : 0) + L * (MAX + 4 + 16 * M)) * 4;
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
