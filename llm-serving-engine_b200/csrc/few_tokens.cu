// Products of at most sixteen tokens (float32: eight) with what stands around them in a pre-norm layer, for layers that are small enough
// that a step is the chain of its launches rather than its bytes:
//
//   out[T, N]  = x + a[T, K] . w[N, K]^T           the output projections, with the residual add
//   out[T, N]  = a . w^T, act[T, I] = silu(gate) * up, [gate | up] = a . w[2 I, K]^T        a = x / rms(x) * weight
//
// Every block owns 8 features (PAIR: 8 gates and their ups) for all of K, so a product needs no sums between blocks, and it
// works out the norm of all rows for itself: 4 bytes an element that every block reads from L2 against a launch in the
// chain. A layer is five launches (q|k|v; rotation, cache write and attention; o; gate|up; down), six where a context is in
// parts, instead of eight (bfloat16) or nine (float32). What bounds each is latency: the hand-over to it, one load of
// the activations, the sum over K. The weights depend on no kernel before and are all asked for (cp.async) before the
// dependency wait; small blocks, several to an SM, so that the next launch's fit beside them. What each adds to a step of
// SmolLM2-135M sizes, us (its predecessors: norm 3.0, products 2.7 to 3.3, SiLU 2.7, attention 7 to 24; float32 products 6):
//   bfloat16, 1 token, 517 keys    q|k|v 2.3  attention 3.8  o 1.6  gate|up 2.7  down 2.5    step 736 -> 430
//   bfloat16, 16 tokens, 8100      q|k|v 2.9  attention 20.2 and merge 2.6  o 2.6  3.4  3.4  step 1305 -> 1080
//   float32, 6 tokens, 300         q|k|v 3.9  attention 3.7  o 3.4  gate|up 4.9  down 3.8    step 1275 -> 660
// (A kernel that stays for all layers, with barriers over all blocks in place of launches, was slower than the separate
// kernels: 1.7 us a barrier, and the activations that every block reads cost what the launches do.)
//
// float32 products add in the order of gemm_f32.cu (K in 32 slices, a lane per slice, eight slices to a group), so a row's
// product has the same bits whatever the batch and the kernel.
#include <climits>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace lse {
namespace few {

struct Args {
  const float* x;        // NORM: the residual stream [T, K]; else what is added to the product [T, N], or null
  const float* weight;   // of the norm, [K]
  float eps;
  const void* a;         // else the activations [T, K]
  const void* w;
  void* out;             // float32 [T, N], PAIR: [T, N] of the activations' type
  int T, N, K;
  int w_early;           // w is read before the kernels before this one are done
};

constexpr int MAX_T = 8, B_MAX_T = 16;  // tokens: float32, bfloat16

__device__ __forceinline__ void copy16(void* smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem));
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
__device__ __forceinline__ float4 ld4(const float* p) { return __ldcg(reinterpret_cast<const float4*>(p)); }

// ---------------------------------------------------------------------------------------- float32
// 8 features a block (four, on twice the SMs, read the activations twice as often: 6 tokens, 576 features of K = 1536, 3.9
// against 4.6 us in the chain), 8 warps of four slices each: lanes are (feature, slice). With PAIR a lane has a gate and its up.
constexpr int R = 8, F_WARPS = 8, F_THREADS = F_WARPS * 32, SLICES = 32, F_VECS = 8;
constexpr int F_MAX_NORM = F_VECS * 128;  // columns of a normed row

__host__ __device__ constexpr size_t f32_smem(bool norm, bool pair, int T, int K) {
  return sizeof(float) * ((size_t)R * (pair ? 2 : 1) * (K + 4) + (size_t)T * K + (norm ? K : 0) + SLICES * R * (pair ? 2 : 1) * MAX_T);
}

// NORM: the activations are the norm of x
template <bool NORM, bool PAIR>
__global__ void __launch_bounds__(F_THREADS) f32_kernel(const Args p) {
  constexpr int RL = PAIR ? 2 : 1;  // rows of a lane
  extern __shared__ __align__(16) float f32_shared[];
  const int K = p.K, T = p.T, stride = K + 4;  // 8 features' float4 of one k lie in 8 groups of banks
  float* ws = f32_shared;
  float* sums = ws + R * RL * stride;  // [SLICES][R RL][MAX_T]
  float* as = sums + SLICES * R * RL * MAX_T;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_trigger();
  if (!p.w_early) pdl_wait();
  static_assert(F_WARPS == R, "a warp a row");
#pragma unroll
  for (int r = 0; r < RL; ++r) {
    const int global = r * p.N + blockIdx.x * R + warp;
    const float* src = (const float*)p.w + (size_t)min(global, p.N * RL - 1) * K;  // (what is beyond is not stored)
    for (int c = lane * 4; c < K; c += 128) copy16(ws + (r * R + warp) * stride + c, src + c);
  }
  if constexpr (NORM) {  // a warp a row
    float* gs = as + T * K;
    for (int c = threadIdx.x * 4; c < K; c += F_THREADS * 4) copy16(gs + c, p.weight + c);
    if (p.w_early) pdl_wait();
    float4 v[F_VECS];
    float ss = 0.f;
    const bool valid = warp < T;
#pragma unroll
    for (int i = 0; i < F_VECS; ++i) {
      const int c = (i * 32 + lane) * 4;
      v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (valid && c < K) {
        v[i] = ld4(p.x + (size_t)warp * K + c);
      }
    }
#pragma unroll
    for (int i = 0; i < F_VECS; ++i) {
      ss += v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
    }
    const float rstd = rsqrtf(warp_sum(ss) / (float)K + p.eps);
    copies_done();
    __syncthreads();
#pragma unroll
    for (int i = 0; i < F_VECS; ++i) {
      const int c = (i * 32 + lane) * 4;
      if (valid && c < K) {
        const float4 g = *reinterpret_cast<const float4*>(gs + c);
        *reinterpret_cast<float4*>(as + warp * K + c) =
            make_float4(v[i].x * rstd * g.x, v[i].y * rstd * g.y, v[i].z * rstd * g.z, v[i].w * rstd * g.w);
      }
    }
  } else {
    if (p.w_early) pdl_wait();
    for (int i = threadIdx.x * 4; i < T * K; i += F_THREADS * 4) copy16(as + i, (const float*)p.a + i);
    copies_done();
  }
  // what the product is added to, by the threads that will store it
  const int my_token = threadIdx.x / R, my_j = blockIdx.x * R + threadIdx.x % R;
  const bool stores = threadIdx.x < T * R && my_j < p.N;
  const size_t out_at = (size_t)my_token * p.N + my_j;
  float residual = 0.f;
  if (!NORM && p.x && stores) residual = __ldcg(p.x + out_at);
  __syncthreads();

  const int n = lane & (R - 1), slice = warp * 4 + (lane >> 3);
  const int SL = (K + 255) / 256 * 8, lo = min(K, slice * SL), hi = min(K, lo + SL);
  float acc[RL][MAX_T];
#pragma unroll
  for (int e = 0; e < MAX_T; ++e)
#pragma unroll
    for (int r = 0; r < RL; ++r) acc[r][e] = 0.f;
  const float* wp = ws + n * stride;
#pragma unroll 2
  for (int k = lo; k < hi; k += 4) {
    float4 wv[RL];
#pragma unroll
    for (int r = 0; r < RL; ++r) wv[r] = *reinterpret_cast<const float4*>(wp + r * R * stride + k);
#pragma unroll
    for (int e = 0; e < MAX_T; ++e) {
      if (e < T) {
        const float4 av = *reinterpret_cast<const float4*>(as + e * K + k);
#pragma unroll
        for (int r = 0; r < RL; ++r) {
          acc[r][e] = fmaf(av.x, wv[r].x, acc[r][e]);
          acc[r][e] = fmaf(av.y, wv[r].y, acc[r][e]);
          acc[r][e] = fmaf(av.z, wv[r].z, acc[r][e]);
          acc[r][e] = fmaf(av.w, wv[r].w, acc[r][e]);
        }
      }
    }
  }
#pragma unroll
  for (int e = 0; e < MAX_T; ++e)
    if (e < T) {
#pragma unroll
      for (int r = 0; r < RL; ++r) sums[(slice * MAX_T + e) * (R * RL) + r * R + n] = acc[r][e];
    }
  __syncthreads();
  auto total = [&](int token, int f) {
    const float* from = sums + token * (R * RL) + f;
    float sum = 0.f;
#pragma unroll
    for (int q = 0; q < SLICES / 8; ++q) {
      float group = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) group += from[(q * 8 + i) * (MAX_T * R * RL)];
      sum += group;
    }
    return sum;
  };
  if (stores) {
    float y = total(my_token, threadIdx.x % R);
    if constexpr (PAIR) y = y / (1.f + expf(-y)) * total(my_token, threadIdx.x % R + R);
    ((float*)p.out)[out_at] = NORM ? y : residual + y;
  }
}

// ---------------------------------------------------------------------------------------- bfloat16
// 8 warps share K in chunks of 32; mma.sync m16n8k16 with the tokens as rows and 8 features as columns. Which of a chunk's
// elements meet in which multiply is free as long as both operands agree: lane t of a row takes elements 8 t .. 8 t + 7,
// one 16-byte load of either operand for two multiplies.
constexpr int B_WARPS = 8, B_THREADS = B_WARPS * 32, B_PAD = 64;  // bytes after a row: 2 rows x 64 bytes in 8 groups of banks

__host__ __device__ constexpr int b16_stride(int K) {  // bytes: an odd multiple of 64, or as K leaves it
  return K * 2 + ((K * 2) % 128 == 0 ? B_PAD : 0);
}

__device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// CH: chunks per warp, at most; TT: sets of eight tokens
template <int CH, int TT, bool NORM, bool PAIR>
__global__ void __launch_bounds__(B_THREADS) b16_kernel(const Args p) {
  extern __shared__ __align__(16) unsigned char b16_shared[];
  __shared__ float red[B_WARPS][8 * TT];
  constexpr int NTILE = PAIR ? 2 : 1;  // tiles of 8 features: gates, and their ups
  __shared__ float sums[B_WARPS][NTILE][8 * TT * 8];
  const int K = p.K, T = p.T, chunks = K / 32, stride = b16_stride(K);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  pdl_trigger();
  if (!p.w_early) pdl_wait();
#pragma unroll
  for (int r = 0; r < NTILE; ++r) {
    const int global = r * p.N + blockIdx.x * 8 + warp;
    const bf16* src = (const bf16*)p.w + (size_t)min(global, p.N * NTILE - 1) * K;  // (what is beyond is not stored)
    for (int c = lane * 8; c < K; c += 256) copy16(b16_shared + (r * 8 + warp) * stride + c * 2, src + c);
  }
  uint4 a[CH][TT];  // chunk i * 8 + warp of tokens g, then g + 8
  if constexpr (NORM) {
    float4 w[CH][2], v[CH][TT][2];
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      const int ch = i * B_WARPS + warp;
      const float* src = p.weight + ch * 32 + 8 * t;
      w[i][0] = ch < chunks ? __ldg(reinterpret_cast<const float4*>(src)) : make_float4(0.f, 0.f, 0.f, 0.f);
      w[i][1] = ch < chunks ? __ldg(reinterpret_cast<const float4*>(src) + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (p.w_early) pdl_wait();
#pragma unroll
    for (int i = 0; i < CH; ++i)
#pragma unroll
      for (int e = 0; e < TT; ++e) {
        const int ch = i * B_WARPS + warp, token = g + 8 * e;
        const float* src = p.x + (size_t)token * K + ch * 32 + 8 * t;
        const bool in = token < T && ch < chunks;
        v[i][e][0] = in ? ld4(src) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[i][e][1] = in ? ld4(src + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
    for (int e = 0; e < TT; ++e) {
      float ss = 0.f;
#pragma unroll
      for (int i = 0; i < CH; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float4 z = v[i][e][h];
          ss += z.x * z.x + z.y * z.y + z.z * z.z + z.w * z.w;
        }
      ss += __shfl_xor_sync(0xffffffffu, ss, 1);
      ss += __shfl_xor_sync(0xffffffffu, ss, 2);
      if (t == 0) red[warp][g + 8 * e] = ss;
    }
    copies_done();
    __syncthreads();
#pragma unroll
    for (int e = 0; e < TT; ++e) {
      float total = 0.f;
#pragma unroll
      for (int i = 0; i < B_WARPS; ++i) total += red[i][g + 8 * e];
      const float rstd = rsqrtf(total / (float)K + p.eps);
#pragma unroll
      for (int i = 0; i < CH; ++i) {
        const float4 z0 = v[i][e][0], z1 = v[i][e][1], w0 = w[i][0], w1 = w[i][1];
        a[i][e] = make_uint4(pack_bf16(z0.x * rstd * w0.x, z0.y * rstd * w0.y), pack_bf16(z0.z * rstd * w0.z, z0.w * rstd * w0.w),
                             pack_bf16(z1.x * rstd * w1.x, z1.y * rstd * w1.y), pack_bf16(z1.z * rstd * w1.z, z1.w * rstd * w1.w));
      }
    }
  } else {
    if (p.w_early) pdl_wait();
#pragma unroll
    for (int i = 0; i < CH; ++i)
#pragma unroll
      for (int e = 0; e < TT; ++e) {
        const int ch = i * B_WARPS + warp, token = g + 8 * e;
        const bf16* src = (const bf16*)p.a + (size_t)token * K + ch * 32 + 8 * t;
        a[i][e] = token < T && ch < chunks ? __ldcg(reinterpret_cast<const uint4*>(src)) : make_uint4(0, 0, 0, 0);
      }
    copies_done();
    __syncthreads();
  }
  // what the product is added to, by the threads that will store it
  const int my_token = threadIdx.x / 8, my_f = threadIdx.x % 8, my_j = blockIdx.x * 8 + my_f;
  const bool stores = threadIdx.x < T * 8 && my_j < p.N;
  const size_t out_at = (size_t)my_token * p.N + my_j;
  float residual = 0.f;
  if (!NORM && p.x && stores) residual = __ldcg(p.x + out_at);
  float acc[NTILE][4] = {};
#pragma unroll
  for (int i = 0; i < CH; ++i) {
    const int ch = i * B_WARPS + warp;
    if (ch < chunks) {
      const uint4 lo = a[i][0], hi = TT == 2 ? a[i][TT - 1] : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int r = 0; r < NTILE; ++r) {
        const uint4 b = *reinterpret_cast<const uint4*>(b16_shared + (r * 8 + g) * stride + ch * 64 + 16 * t);
        mma(acc[r], lo.x, hi.x, lo.y, hi.y, b.x, b.y);
        mma(acc[r], lo.z, hi.z, lo.w, hi.w, b.z, b.w);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < NTILE; ++r) {
    *reinterpret_cast<float2*>(&sums[warp][r][g * 8 + 2 * t]) = make_float2(acc[r][0], acc[r][1]);
    if constexpr (TT == 2) *reinterpret_cast<float2*>(&sums[warp][r][(g + 8) * 8 + 2 * t]) = make_float2(acc[r][2], acc[r][3]);
  }
  __syncthreads();
  auto total = [&](int r) {
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < B_WARPS; ++i) sum += sums[i][r][my_token * 8 + my_f];
    return sum;
  };
  if (stores) {
    const float y = total(0);
    if constexpr (PAIR) ((bf16*)p.out)[out_at] = __float2bfloat16(__fdividef(y, 1.f + __expf(-y)) * total(NTILE - 1));
    else ((float*)p.out)[out_at] = NORM ? y : residual + y;
  }
}

// ---------------------------------------------------------------------------------------- attention
// Rotation, cache write and attention of single tokens from the float32 rows of the fused q|k|v projection, head size
// 64. One block of 16 warps per (part of the context, key head, token): 512 keys are two tiles of 16 per warp (float32:
// four of 8), and a step of ordinary length needs no second kernel or last block for merging. Before the dependency wait
// every warp has asked (cp.async) for its first two tiles of keys and values of earlier steps; after it the chain is the
// rows from L2, the tiles, the sums of the warps.
constexpr int D = 64, A_WARPS = 16, A_THREADS = A_WARPS * 32, MAX_GROUP = 4, Q_STRIDE = 72;
constexpr int PART = D + 8;  // floats of a part's result: 64 values, maximum and sum of the exponentials, a whole sector of L2
template <typename E>
__device__ __forceinline__ float soft_exp(float v) {
  if constexpr (std::is_same<E, bf16>::value) return __expf(v);
  else return expf(v);
}

struct AttnArgs {
  const float* qkv;       // [T, (H + 2 KVH) 64]
  void* out;              // [T, H 64]
  float* parts;           // [T, H, splits, PART] if splits > 1
  void *k_pages, *v_pages;
  int H, KVH, page_tokens, page_shift, splits;
  float scale;
  const float *cos, *sin; // [positions, 32] or null
  const int *tables, *ctx_lens, *cu_q, *decode_seqs;
  int table_stride;
};

template <typename E>
constexpr int TILE = 32 / (int)sizeof(E);  // keys: 16 or 8
constexpr int KV_TILE = 2 * 32 * D;        // bytes of a tile's keys and values
constexpr int SLOTS = 2;                   // tiles on their way per warp
constexpr int ATTN_SMEM = A_WARPS * SLOTS * KV_TILE + A_WARPS * MAX_GROUP * (D + 2) * 4;

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma4(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t x) {
  uint32_t y;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}
// byte offset of 16-byte piece c of row r of a tile: the pieces of a row are permuted by the row's number
template <typename E>
__device__ __forceinline__ int place(int r, int c) { return r * (D * (int)sizeof(E)) + ((c ^ (r & 7)) << 4); }

// HEADS: query heads of a block, at most: a key head's (MAX_GROUP), or one (float32: the arithmetic of a tile goes by its heads)
template <typename E, int HEADS>
__global__ void __launch_bounds__(A_THREADS, 1) attention_kernel(const AttnArgs p) {
  constexpr bool BF16 = std::is_same<E, bf16>::value;
  constexpr int KEYS = TILE<E>, LANES = 32 / KEYS;  // of a tile; lanes that copy a row, four pieces of 16 bytes each
  extern __shared__ __align__(128) unsigned char attn_shared[];
  __shared__ __align__(16) E qs[HEADS * Q_STRIDE];
  __shared__ __align__(16) E fresh[2 * D];  // this step's key, then its value
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char* slots = attn_shared + warp * SLOTS * KV_TILE;
  float* merge = reinterpret_cast<float*>(attn_shared + A_WARPS * SLOTS * KV_TILE);  // [A_WARPS][G][D + 2]
  pdl_trigger();

  // the block's G query heads h0, h0 + 1, ... of key head kvh
  const int split = blockIdx.x, group = p.H / p.KVH, kvh = HEADS == 1 ? blockIdx.y / group : blockIdx.y;
  const int G = HEADS == 1 ? 1 : group, h0 = HEADS == 1 ? blockIdx.y : kvh * group;
  const int seq = p.decode_seqs[blockIdx.z], tok = p.cu_q[seq], ctx = p.ctx_lens[seq];
  const int all = (ctx + KEYS - 1) / KEYS, per = (all + p.splits - 1) / p.splits;  // tiles
  const int first = split * per, last = min(all, first + per);
  const int* table = p.tables + (size_t)seq * p.table_stride;
  auto row_of = [&](int key) -> size_t {
    int page, off;
    page_of(key, p.page_tokens, p.page_shift, page, off);
    return (((size_t)table[page] * p.KVH + kvh) * p.page_tokens + off) * D;
  };
  // The warp's tile number n (of the part's first + warp, + 16, ...) into its slot, as one group of copies. This step's
  // own row is not in the page yet, and rows beyond it may hold anything: they are filled in afterwards.
  const int copy_row = lane / LANES, copy_piece = (lane % LANES) * 4;
  auto ask = [&](int n) {
    const int tile = first + warp + n * A_WARPS, key = tile * KEYS + copy_row;
    if (tile < last && key < ctx - 1) {
      const size_t at = row_of(key);
      unsigned char* kt = slots + (n % SLOTS) * KV_TILE;
#pragma unroll
      for (int c = copy_piece; c < copy_piece + 4; ++c) {
        copy16(kt + place<E>(copy_row, c), (const E*)p.k_pages + at + c * (16 / sizeof(E)));
        copy16(kt + KV_TILE / 2 + place<E>(copy_row, c), (const E*)p.v_pages + at + c * (16 / sizeof(E)));
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  for (int n = 0; n < SLOTS; ++n) ask(n);

  // the queries, and in the block that ends at this step's token its key and value: one pair of dims per thread. What does
  // not depend on the projection is fetched before the wait.
  static_assert((HEADS + 2) * 32 <= A_THREADS, "");
  {
    const int i = threadIdx.x & 31, part = threadIdx.x >> 5;
    const bool mine = part < G || (part < G + 2 && last == all && first < last);
    const bool turned = p.cos && part <= G;
    const int head = part < G ? h0 + part : p.H + (part - G) * p.KVH + kvh;
    const float* src = p.qkv + (size_t)tok * (p.H + 2 * p.KVH) * D + head * D + i;
    float cv = 1.f, sv = 0.f;
    E* page = nullptr;
    if (mine && turned) {
      cv = p.cos[(size_t)(ctx - 1) * (D / 2) + i];
      sv = p.sin[(size_t)(ctx - 1) * (D / 2) + i];
    }
    if (mine && part >= G) page = (E*)(part == G ? p.k_pages : p.v_pages) + row_of(ctx - 1);
    pdl_wait();
    if (mine) {
      float x1 = __ldcg(src), x2 = __ldcg(src + D / 2);
      if (turned) {
        const float r1 = x1 * cv - x2 * sv, r2 = x2 * cv + x1 * sv;
        x1 = r1;
        x2 = r2;
      }
      const E h1 = Num<E>::from_float(x1), h2 = Num<E>::from_float(x2);
      E* dst = part < G ? qs + part * Q_STRIDE : fresh + (part - G) * D;
      dst[i] = h1;
      dst[i + D / 2] = h2;
      if (part >= G) {
        page[i] = h1;
        page[i + D / 2] = h2;
      }
    }
  }
  __syncthreads();

  float* mine = merge + warp * G * (D + 2);
  const int n_mine = last - first > warp ? (last - first - warp + A_WARPS - 1) / A_WARPS : 0;
  unsigned char *kt, *vt;
  auto tile_there = [&](int n) {  // the tile as it is to be used
    asm volatile("cp.async.wait_group %0;\n" ::"n"(SLOTS - 1) : "memory");
    kt = slots + (n % SLOTS) * KV_TILE;
    vt = kt + KV_TILE / 2;
    const int key = (first + warp + n * A_WARPS) * KEYS + copy_row;
    if (key >= ctx - 1) {
#pragma unroll
      for (int c = copy_piece; c < copy_piece + 4; ++c) {
        uint4 a = make_uint4(0, 0, 0, 0), b = a;
        if (key == ctx - 1) {
          a = *reinterpret_cast<const uint4*>(fresh + c * (16 / sizeof(E)));
          b = *reinterpret_cast<const uint4*>(fresh + D + c * (16 / sizeof(E)));
        }
        *reinterpret_cast<uint4*>(kt + place<E>(copy_row, c)) = a;
        *reinterpret_cast<uint4*>(vt + place<E>(copy_row, c)) = b;
      }
    }
    __syncwarp();
  };
  if constexpr (BF16) {
    // S^T = K Q^T and O^T = V^T P^T: 16 keys (then head dims) by 8 heads
    const int g = lane >> 2, t = lane & 3, mat = lane >> 3, r8 = lane & 7;
    float ot[4][4];
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};  // heads 2t and 2t + 1
    uint32_t qb[4][2];  // head g, dims 16 i + 2t, + 1 and + 8, + 9
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      ot[i][0] = ot[i][1] = ot[i][2] = ot[i][3] = 0.f;
      qb[i][0] = g < G ? *reinterpret_cast<const uint32_t*>(qs + g * Q_STRIDE + 16 * i + 2 * t) : 0;
      qb[i][1] = g < G ? *reinterpret_cast<const uint32_t*>(qs + g * Q_STRIDE + 16 * i + 2 * t + 8) : 0;
    }
#pragma unroll 1
    for (int n = 0; n < n_mine; ++n) {
      tile_there(n);
      const uint32_t kaddr = (uint32_t)__cvta_generic_to_shared(kt), vaddr = (uint32_t)__cvta_generic_to_shared(vt);
      float sc[4] = {0.f, 0.f, 0.f, 0.f};  // keys g, g + 8 x heads 2t, 2t + 1
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint32_t ka[4];
        ldmatrix_x4(ka, kaddr + place<E>((mat & 1) * 8 + r8, 2 * i + (mat >> 1)));
        mma4(sc, ka, qb[i][0], qb[i][1]);
      }
      uint32_t va[4][4];  // dims 16 i .. + 7 / + 8 .. + 15 (mat & 1), keys 0-7 / 8-15 (mat >> 1)
#pragma unroll
      for (int i = 0; i < 4; ++i) ldmatrix_x4_trans(va[i], vaddr + place<E>((mat >> 1) * 8 + r8, 2 * i + (mat & 1)));
      __syncwarp();
      ask(n + SLOTS);
      const int j0 = (first + warp + n * A_WARPS) * 16;
      const bool ok0 = j0 + g < ctx, ok1 = j0 + g + 8 < ctx;
      float corr[2], pr[2][2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float s0 = ok0 ? sc[e] * p.scale : -INFINITY, s1 = ok1 ? sc[2 + e] * p.scale : -INFINITY;
        float mx = fmaxf(m_run[e], fmaxf(s0, s1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
        const float m_fin = mx == -INFINITY ? 0.f : mx;
        corr[e] = __expf(m_run[e] - m_fin);
        m_run[e] = mx;
        pr[e][0] = __expf(s0 - m_fin);
        pr[e][1] = __expf(s1 - m_fin);
        l_run[e] = l_run[e] * corr[e] + pr[e][0] + pr[e][1];  // this thread's share; joined at the end
      }
      const uint32_t pb0 = movmatrix_trans(pack_bf16(pr[0][0], pr[1][0]));
      const uint32_t pb1 = movmatrix_trans(pack_bf16(pr[0][1], pr[1][1]));
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        ot[i][0] *= corr[0];
        ot[i][1] *= corr[1];
        ot[i][2] *= corr[0];
        ot[i][3] *= corr[1];
        mma4(ot[i], va[i], pb0, pb1);
      }
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float sum = l_run[e];
      sum += __shfl_xor_sync(0xffffffffu, sum, 4);
      sum += __shfl_xor_sync(0xffffffffu, sum, 8);
      sum += __shfl_xor_sync(0xffffffffu, sum, 16);
      const int head = 2 * t + e;
      if (head < G) {
        float* to = mine + head * (D + 2);
        if (g == 0) {
          to[D] = m_run[e];
          to[D + 1] = sum;
        }
        if (n_mine > 0) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            to[16 * i + g] = ot[i][e];
            to[16 * i + g + 8] = ot[i][2 + e];
          }
        }
      }
    }
  } else {
    // scores: four lanes a key, 16 dims each (the last two lanes' pieces in another order: no bank conflicts); values: two
    // dims a lane. Every lane takes part in every shuffle, whether its key is seen or not.
    float m_run[HEADS], l_run[HEADS];
    float2 o[HEADS];
#pragma unroll
    for (int h = 0; h < HEADS; ++h) {
      m_run[h] = -INFINITY;
      l_run[h] = 0.f;
      o[h] = make_float2(0.f, 0.f);
    }
    const int j = lane >> 2, quarter = lane & 3;
#pragma unroll 1
    for (int n = 0; n < n_mine; ++n) {
      tile_there(n);
      float dot[HEADS] = {};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c = quarter * 4 + (i ^ (quarter & 2));
        const float4 kv = *reinterpret_cast<const float4*>(kt + place<E>(j, c));
#pragma unroll
        for (int h = 0; h < HEADS; ++h)
          if (h < G) {
            const float4 qv = *reinterpret_cast<const float4*>(qs + h * Q_STRIDE + c * 4);
            dot[h] = fmaf(qv.x, kv.x, dot[h]);
            dot[h] = fmaf(qv.y, kv.y, dot[h]);
            dot[h] = fmaf(qv.z, kv.z, dot[h]);
            dot[h] = fmaf(qv.w, kv.w, dot[h]);
          }
      }
      const bool seen = (first + warp + n * A_WARPS) * KEYS + j < ctx;
      float pr[HEADS];
#pragma unroll
      for (int h = 0; h < HEADS; ++h)
        if (h < G) {
          dot[h] += __shfl_xor_sync(0xffffffffu, dot[h], 1);
          dot[h] += __shfl_xor_sync(0xffffffffu, dot[h], 2);
          const float sc = seen ? dot[h] * p.scale : -INFINITY;
          float mx = fmaxf(m_run[h], sc);
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
          const float base = mx == -INFINITY ? 0.f : mx, corr = expf(m_run[h] - base);
          pr[h] = expf(sc - base);
          m_run[h] = mx;
          l_run[h] = l_run[h] * corr + (quarter ? 0.f : pr[h]);
          o[h].x *= corr;
          o[h].y *= corr;
        }
#pragma unroll
      for (int c = 0; c < KEYS; ++c) {
        const float2 v = *reinterpret_cast<const float2*>(vt + place<E>(c, lane >> 1) + (lane & 1) * 8);
#pragma unroll
        for (int h = 0; h < HEADS; ++h)
          if (h < G) {
            const float w = __shfl_sync(0xffffffffu, pr[h], 4 * c);
            o[h].x = fmaf(w, v.x, o[h].x);
            o[h].y = fmaf(w, v.y, o[h].y);
          }
      }
      __syncwarp();
      ask(n + SLOTS);
    }
#pragma unroll
    for (int h = 0; h < HEADS; ++h)
      if (h < G) {
        float* to = mine + h * (D + 2);
        const float sum = warp_sum(l_run[h]);
        if (lane == 0) {
          to[D] = m_run[h];
          to[D + 1] = sum;
        }
        if (n_mine > 0) *reinterpret_cast<float2*>(to + 2 * lane) = o[h];
      }
  }
  __syncthreads();
  // the warps' sums: their weights first
  __shared__ float weight[HEADS][A_WARPS], top[HEADS], denominator[HEADS];
  if (threadIdx.x < G * A_WARPS) {
    static_assert(A_WARPS == 16, "a head's weights are worked out by half a warp");
    const unsigned half = 0xffffu << (lane & 16);
    const int h = threadIdx.x / A_WARPS, w = threadIdx.x % A_WARPS;
    const float* from = merge + (w * G + h) * (D + 2) + D;
    const float m = from[0];
    float M = m;
#pragma unroll
    for (int o = 1; o < A_WARPS; o <<= 1) M = fmaxf(M, __shfl_xor_sync(half, M, o));
    const float wt = m == -INFINITY ? 0.f : soft_exp<E>(m - M);
    float L = m == -INFINITY ? 0.f : from[1] * wt;
#pragma unroll
    for (int o = 1; o < A_WARPS; o <<= 1) L += __shfl_xor_sync(half, L, o);
    weight[h][w] = wt;
    if (w == 0) {
      top[h] = M;
      denominator[h] = L;
    }
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < G * D; idx += A_THREADS) {
    const int h = idx / D, d = idx % D;
    const float* from = merge + h * (D + 2) + d;
    float A = 0.f;
#pragma unroll
    for (int w = 0; w < A_WARPS; ++w)
      if (weight[h][w] != 0.f) A = fmaf(from[w * G * (D + 2)], weight[h][w], A);  // (a warp without keys left nothing)
    const float L = denominator[h];
    const size_t at = (size_t)tok * p.H + h0 + h;
    if (p.splits == 1) {
      ((E*)p.out)[at * D + d] = Num<E>::from_float(L > 0.f ? A / L : 0.f);
    } else {
      float* to = p.parts + (at * p.splits + split) * PART;
      to[d] = A;
      if (d == 0) {  // a whole sector of L2
        reinterpret_cast<float4*>(to + D)[0] = make_float4(top[h], L, 0.f, 0.f);
        reinterpret_cast<float4*>(to + D)[1] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
  }
}

// The parts of a context merged: a warp per (token, head), two dims a lane. (Merged by every block of the output projection
// as it reads them, without this launch: 6.5 us in the chain for 8 tokens in two parts, 11.5 for 16 in six, where the
// projection of given rows takes 2.)
constexpr int M_WARPS = 4;

template <typename E>
__global__ void __launch_bounds__(M_WARPS * 32) merge_kernel(const float* parts, E* out, int rows, int splits) {
  pdl_trigger();
  pdl_wait();
  const int row = blockIdx.x * M_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= rows) return;
  const float* from = parts + (size_t)row * splits * PART;
  float M = -INFINITY, L = 0.f;
  float2 A = make_float2(0.f, 0.f);
#pragma unroll 1
  for (int s = 0; s < splits; s += 8) {  // eight parts on their way at a time
    float2 ml[8], x[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float* f = from + min(s + k, splits - 1) * PART;
      ml[k] = __ldcg(reinterpret_cast<const float2*>(f + D));
      x[k] = __ldcg(reinterpret_cast<const float2*>(f + 2 * lane));
    }
    float top = M;
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (s + k < splits) top = fmaxf(top, ml[k].x);
    const float base = top == -INFINITY ? 0.f : top, old = soft_exp<E>(M - base);
    M = top;
    L *= old;
    A.x *= old;
    A.y *= old;
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (s + k < splits && ml[k].x != -INFINITY) {
        const float w = soft_exp<E>(ml[k].x - base);
        L = fmaf(ml[k].y, w, L);
        A.x = fmaf(x[k].x, w, A.x);
        A.y = fmaf(x[k].y, w, A.y);
      }
  }
  E* to = out + (size_t)row * D + 2 * lane;
  to[0] = Num<E>::from_float(L > 0.f ? A.x / L : 0.f);
  to[1] = Num<E>::from_float(L > 0.f ? A.y / L : 0.f);
}

// ---------------------------------------------------------------------------------------- launch
constexpr int F_MOST = 112 * 1024, B_MOST = 72 * 1024;  // shared memory of a block: at least two blocks on an SM

template <bool NORM, bool PAIR>
static int launch_f32(const Args& p, cudaStream_t stream) {
  if (allow_dynamic_smem<f32_kernel<NORM, PAIR>, F_MOST>() != cudaSuccess) return LSE_LAUNCH_FAILED;
  return lse::launch(f32_kernel<NORM, PAIR>, (p.N + R - 1) / R, F_THREADS, f32_smem(NORM, PAIR, p.T, p.K), stream, p) ==
                 cudaSuccess ? LSE_OK : LSE_LAUNCH_FAILED;
}
template <int CH, int TT, bool NORM, bool PAIR>
static int launch_b16(const Args& p, cudaStream_t stream) {
  if (allow_dynamic_smem<b16_kernel<CH, TT, NORM, PAIR>, B_MOST>() != cudaSuccess) return LSE_LAUNCH_FAILED;
  return lse::launch(b16_kernel<CH, TT, NORM, PAIR>, (p.N + 7) / 8, B_THREADS, (PAIR ? 16 : 8) * b16_stride(p.K), stream, p) ==
                 cudaSuccess ? LSE_OK : LSE_LAUNCH_FAILED;
}

static bool serves(int dtype, int T, int N, int K, bool norm, bool pair) {
  if (T < 1 || T > (dtype == LSE_F32 ? MAX_T : B_MAX_T) || N < 1 || K < 1) return false;
  if (dtype == LSE_F32) return K % 4 == 0 && (!norm || K <= F_MAX_NORM) && f32_smem(norm, pair, T, K) <= F_MOST;
  return dtype == LSE_BF16 && K % 32 == 0 && K <= (norm ? 4 : 16) * B_WARPS * 32 && (pair ? 16 : 8) * b16_stride(K) <= B_MOST;
}

template <int TT, bool NORM, bool PAIR>
static int run_b16(const Args& p, cudaStream_t stream) {
  const int ch = (p.K / 32 + B_WARPS - 1) / B_WARPS;
  if (ch <= 3) return launch_b16<3, TT, NORM, PAIR>(p, stream);
  if constexpr (NORM) return ch <= 4 ? launch_b16<4, TT, NORM, PAIR>(p, stream) : LSE_BAD_ARGUMENT;
  else return ch <= 6 ? launch_b16<6, TT, NORM, PAIR>(p, stream) : launch_b16<16, TT, NORM, PAIR>(p, stream);
}

template <bool NORM, bool PAIR>
static int run(const Args& p, int dtype, cudaStream_t stream) {
  if (dtype == LSE_F32) return launch_f32<NORM, PAIR>(p, stream);
  return p.T <= 8 ? run_b16<1, NORM, PAIR>(p, stream) : run_b16<2, NORM, PAIR>(p, stream);
}

template <typename E, int HEADS>
static int launch_attention(const AttnArgs& p, int T, cudaStream_t stream) {
  if (allow_dynamic_smem<attention_kernel<E, HEADS>, ATTN_SMEM>() != cudaSuccess) return LSE_LAUNCH_FAILED;
  const dim3 grid(p.splits, HEADS == 1 ? p.H : p.KVH, T);
  cudaError_t e = lse::launch(attention_kernel<E, HEADS>, grid, A_THREADS, ATTN_SMEM, stream, p);
  if (e == cudaSuccess && p.splits > 1)
    e = lse::launch(merge_kernel<E>, (T * p.H + M_WARPS - 1) / M_WARPS, M_WARPS * 32, 0, stream, (const float*)p.parts, (E*)p.out,
                    T * p.H, p.splits);
  return e == cudaSuccess ? LSE_OK : LSE_LAUNCH_FAILED;
}

}  // namespace few
}  // namespace lse

using namespace lse;

extern "C" int lse_few_tokens_serves(int dtype, int T, int N, int K, int norm, int pair) {
  return few::serves(dtype, T, N, K, norm != 0, pair != 0);
}

extern "C" int lse_few_tokens(const float* x, const float* norm_weight, float eps, const void* a, const void* w, void* out,
                              int dtype, int T, int N, int K, int pair, int w_early, cudaStream_t stream) {
  if (T <= 0 || N <= 0) return LSE_OK;
  const bool norm = norm_weight != nullptr;
  if (!few::serves(dtype, T, N, K, norm, pair != 0) || (norm ? !x : !a)) return LSE_BAD_ARGUMENT;
  const few::Args p{x, norm_weight, eps, a, w, out, T, N, K, w_early};
  if (norm) return pair ? few::run<true, true>(p, dtype, stream) : few::run<true, false>(p, dtype, stream);
  return pair ? LSE_BAD_ARGUMENT : few::run<false, false>(p, dtype, stream);
}

extern "C" size_t lse_few_attention_floats(int T, int H, int splits) { return (size_t)T * H * splits * few::PART; }

extern "C" int lse_few_attention(const LseFewAttention* a, cudaStream_t stream) {
  if (a->T <= 0) return LSE_OK;
  if (a->H <= 0 || a->KVH <= 0 || a->H % a->KVH || a->H / a->KVH > few::MAX_GROUP || a->splits < 1 || a->page_tokens < 1 ||
      a->H > 65535 || a->T > 65535 || !a->out || (a->splits > 1 && !a->parts))
    return LSE_BAD_ARGUMENT;
  few::AttnArgs p{a->qkv, a->out, a->parts, a->k_pages, a->v_pages, a->H, a->KVH, a->page_tokens, -1,
                  a->splits, a->scale, a->cos, a->sin, a->block_tables, a->ctx_lens, a->cu_q, a->decode_seqs, a->table_stride};
  if ((a->page_tokens & (a->page_tokens - 1)) == 0)
    for (p.page_shift = 0; (1 << p.page_shift) < a->page_tokens; ++p.page_shift) {}
  if (a->dtype == LSE_BF16) return few::launch_attention<bf16, few::MAX_GROUP>(p, a->T, stream);
  if (a->dtype != LSE_F32) return LSE_BAD_ARGUMENT;
  // A block per query head where that fits on the SMs at once: 6 tokens of 300 keys, 9 heads on 3, 7.3 us in the chain with
  // a block per key head.
  return (long long)a->splits * a->H * a->T <= 148 ? few::launch_attention<float, 1>(p, a->T, stream)
                                                   : few::launch_attention<float, few::MAX_GROUP>(p, a->T, stream);
}
