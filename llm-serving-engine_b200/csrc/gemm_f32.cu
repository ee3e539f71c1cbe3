// True float32 matrix product on the CUDA cores (no tensor-core mode, no reduced precision):
//   out[T, N] = a[T, K] . w[N, K]^T (+ bias[N])
//
// One order of additions for every shape of the batch, so that the value of a row does not depend on
// how many other rows are in the batch, on where the row sits in it, or on which kernel runs:
//   K is cut into at most 32 slices of SL = 8 ceil(K / 256) elements, and eight slices make a group;
//   a slice is summed by fused multiply-adds over ascending k from zero, a group is the sum of its
//   slices in ascending order from zero, and the result the sum of the groups in the same way, + bias.
// What is cut can be worked on side by side, which is what a step of a few rows needs: as a single
// chain of K additions per output a product of 6 rows at K = 576 .. 1536 took 66 us on average.
//
//   few rows   one block owns NB output features for all of K, a warp lane one slice: meant to be bound by
//              streaming w once; measured it is the latency of a block (load, multiply, 32 partial sums), with
//              two blocks of 110 KB per SM. 6 rows, K = 576: 49152 features 64 us (w at copy rate: 17), 3072
//              features 12 us; 576 features of K = 1536 12 us (all with 6 us of start and timing);
//   tiles      BM x BN outputs per block, TM x 4 per thread, the next K tile on its way in registers
//              while this one is multiplied: bound by the reads of shared memory (64 x 128 tiles of 8 x 4 per
//              thread: 900 rows of 49152 x 576 in 1388 us, 37 TFLOP/s; 64 x 64 of 4 x 4: 1613). Where these
//              would leave SMs idle, 32 x 32 tiles whose four groups of K are summed by four sets of threads.
#include <climits>

#include "common.cuh"
#include "kernels.h"

namespace lse {
namespace gf32 {

constexpr int SLICES = 32, GROUP = 8;

__host__ __device__ inline int slice_len(int K) { return (K + SLICES * 8 - 1) / (SLICES * 8) * 8; }

struct Args {
  const float* a;
  const float* w;
  const float* bias;
  float* out;
  int T, N, K, SL;
  int w_early;  // w is read before the kernels before this one are done
};

// ---------------------------------------------------------------------------------------- few rows
// NG warps, each NPT features of w and 8 rows of a; lane s sums slice s. A pass brings 8 elements of every
// slice of every row. A staged slice is 12 floats apart from the next: eight neighbouring lanes then read
// 16 bytes each from 8 different groups of banks.
constexpr int FEW_T = 8, CH = 8, PAD = 12, ROW = SLICES * PAD, STAGES = 3;

__device__ __forceinline__ void copy16(float* smem, const float* gmem, bool valid) {
  const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem);
  const int bytes = valid ? 16 : 0;  // the rest is filled with zeros
  asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(gmem), "r"(bytes));
}

template <int NPT, int NG>
__global__ void __launch_bounds__(32 * NG) few_rows_kernel(const Args p) {
  constexpr int NB = NPT * NG, THREADS = 32 * NG;
  extern __shared__ __align__(16) float smem[];
  pdl_trigger();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n0 = blockIdx.x * NB, t0 = blockIdx.y * FEW_T;
  const int passes = p.SL / CH;
  auto load = [&](int c, int rows, int first, const float* src, int r0, int limit) {
    float* buf = smem + (c % STAGES) * (NB + FEW_T) * ROW + first * ROW;
    for (int i = threadIdx.x; i < rows * SLICES * 2; i += THREADS) {
      const int half = i & 1, s = (i >> 1) & (SLICES - 1), r = i / (SLICES * 2);
      const int k = s * p.SL + c * CH + half * 4;
      const bool valid = k < p.K && r0 + r < limit;  // K is a multiple of 4 here
      copy16(buf + r * ROW + s * PAD + half * 4, valid ? src + (size_t)(r0 + r) * p.K + k : src, valid);
    }
  };
  // Where the caller says that w depends on no kernel still running, its first passes are asked for before the wait:
  // 24 steps of 6 rows, 30 layers, 41.7 ms against 44.1 after it (prefetching them into L2 instead: 44.0).
  if (!p.w_early) pdl_wait();
  for (int c = 0; c < STAGES - 1 && c < passes; ++c) load(c, NB, 0, p.w, n0, p.N);
  if (p.w_early) pdl_wait();
  for (int c = 0; c < STAGES - 1; ++c) {
    if (c < passes) load(c, FEW_T, NB, p.a, t0, p.T);
    asm volatile("cp.async.commit_group;\n" ::);
  }
  float acc[FEW_T][NPT];
#pragma unroll
  for (int t = 0; t < FEW_T; ++t)
#pragma unroll
    for (int j = 0; j < NPT; ++j) acc[t][j] = 0.f;
  for (int c = 0; c < passes; ++c) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2));
    __syncthreads();  // pass c is there, and everybody is done with the buffer that is filled next
    if (c + STAGES - 1 < passes) {
      load(c + STAGES - 1, NB, 0, p.w, n0, p.N);
      load(c + STAGES - 1, FEW_T, NB, p.a, t0, p.T);
    }
    asm volatile("cp.async.commit_group;\n" ::);
    const float* buf = smem + (c % STAGES) * (NB + FEW_T) * ROW + lane * PAD;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      float4 wv[NPT];
#pragma unroll
      for (int j = 0; j < NPT; ++j)
        wv[j] = *reinterpret_cast<const float4*>(buf + (warp * NPT + j) * ROW + half * 4);
#pragma unroll
      for (int t = 0; t < FEW_T; ++t) {
        const float4 av = *reinterpret_cast<const float4*>(buf + (NB + t) * ROW + half * 4);
#pragma unroll
        for (int j = 0; j < NPT; ++j) {
          acc[t][j] = fmaf(av.x, wv[j].x, acc[t][j]);
          acc[t][j] = fmaf(av.y, wv[j].y, acc[t][j]);
          acc[t][j] = fmaf(av.z, wv[j].z, acc[t][j]);
          acc[t][j] = fmaf(av.w, wv[j].w, acc[t][j]);
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
  __syncthreads();
  float* red = smem;  // [FEW_T * NB][SLICES + 1]
#pragma unroll
  for (int t = 0; t < FEW_T; ++t)
#pragma unroll
    for (int j = 0; j < NPT; ++j) red[(t * NB + warp * NPT + j) * (SLICES + 1) + lane] = acc[t][j];
  __syncthreads();
  for (int o = threadIdx.x; o < FEW_T * NB; o += THREADS) {
    const int t = t0 + o / NB, n = n0 + o % NB;
    const float* r = red + o * (SLICES + 1);
    float total = 0.f;
#pragma unroll
    for (int g = 0; g < SLICES / GROUP; ++g) {
      float sum = 0.f;
#pragma unroll
      for (int s = 0; s < GROUP; ++s) sum += r[g * GROUP + s];
      total += sum;
    }
    if (t < p.T && n < p.N) p.out[(size_t)t * p.N + n] = total + (p.bias ? p.bias[n] : 0.f);
  }
}

// ---------------------------------------------------------------------------------------- tiles
// G = 4: four sets of threads, set g sums group g of the slices. G = 1: one set sums all of K; the sum of the groups
// so far lies in shared memory, where it is touched four times in all: in registers it cost a block per SM (64 x 64
// tiles, 900 rows, 3072 x 576: 125 us; now 113, as the single chain of additions took before there were slices, 111).
constexpr int BK = 16;

template <int BM, int BN, int TM, int G, int BLOCKS>
__global__ void __launch_bounds__(G * (BM / TM) * (BN / 4), BLOCKS) tiles_kernel(const Args p, const bool vec) {
  constexpr int SET = (BM / TM) * (BN / 4);             // threads of a set
  constexpr int PA = BM * 4 / SET, PW = BN * 4 / SET;   // pieces of four k per thread and tile
  static_assert(BM * 4 % SET == 0 && BN * 4 % SET == 0, "");
  constexpr int LA = BM + 4, LW = BN + 4, TILE = BK * (LA + LW);
  extern __shared__ __align__(16) float smem[];  // the sets' tiles, two each; G == 1: then the totals
  static_assert(G == 1 || G * BM * BN <= G * 2 * TILE, "");
  pdl_trigger();
  const int set = threadIdx.x / SET, tid = threadIdx.x % SET;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int tm = (tid / (BN / 4)) * TM, tn = (tid % (BN / 4)) * 4;
  float* tiles = smem + set * 2 * TILE;
  float4* mine = reinterpret_cast<float4*>(smem + G * 2 * TILE) + tid;  // [TM][SET]
  const int per_set = SLICES / G * p.SL;                // elements of K per set, a multiple of BK
  const int k_begin = set * per_set;
  const int n_tiles = ((G == 1 ? p.K : min(p.K, per_set)) + BK - 1) / BK;  // the same for every set
  float acc[TM][4], grp[TM][4];
#pragma unroll
  for (int i = 0; i < TM; ++i) {
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = grp[i][j] = 0.f;
    if (G == 1) mine[i * SET] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  float4 av[PA], wv[PW];
  auto piece = [&](const float* src, int row, int limit, int k) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row < limit) {
      const float* q = src + (size_t)row * p.K + k;
      if (vec) {
        if (k < p.K) v = *reinterpret_cast<const float4*>(q);
      } else {
        if (k < p.K) v.x = q[0];
        if (k + 1 < p.K) v.y = q[1];
        if (k + 2 < p.K) v.z = q[2];
        if (k + 3 < p.K) v.w = q[3];
      }
    }
    return v;
  };
  auto fetch = [&](int it) {
    const int k0 = k_begin + it * BK;
#pragma unroll
    for (int i = 0; i < PA; ++i) {
      const int idx = tid + i * SET;
      av[i] = piece(p.a, m0 + idx / 4, p.T, k0 + idx % 4 * 4);
    }
#pragma unroll
    for (int i = 0; i < PW; ++i) {
      const int idx = tid + i * SET;
      wv[i] = piece(p.w, n0 + idx / 4, p.N, k0 + idx % 4 * 4);
    }
  };
  auto put = [&](int buf) {
    float* as = tiles + buf * TILE;
    float* ws = as + BK * LA;
#pragma unroll
    for (int i = 0; i < PA; ++i) {
      const int idx = tid + i * SET, r = idx / 4, k = idx % 4 * 4;
      as[k * LA + r] = av[i].x; as[(k + 1) * LA + r] = av[i].y;
      as[(k + 2) * LA + r] = av[i].z; as[(k + 3) * LA + r] = av[i].w;
    }
#pragma unroll
    for (int i = 0; i < PW; ++i) {
      const int idx = tid + i * SET, r = idx / 4, k = idx % 4 * 4;
      ws[k * LW + r] = wv[i].x; ws[(k + 1) * LW + r] = wv[i].y;
      ws[(k + 2) * LW + r] = wv[i].z; ws[(k + 3) * LW + r] = wv[i].w;
    }
  };
  auto end_of_slice = [&]() {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        grp[i][j] += acc[i][j];
        acc[i][j] = 0.f;
      }
  };
  auto end_of_group = [&]() {  // G == 1
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      float4 t = mine[i * SET];
      t.x += grp[i][0]; t.y += grp[i][1]; t.z += grp[i][2]; t.w += grp[i][3];
      mine[i * SET] = t;
#pragma unroll
      for (int j = 0; j < 4; ++j) grp[i][j] = 0.f;
    }
  };
  pdl_wait();
  fetch(0);
  put(0);
  __syncthreads();
  int left = p.SL, slices = GROUP;
  for (int it = 0; it < n_tiles; ++it) {
    if (it + 1 < n_tiles) fetch(it + 1);
    const float* as = tiles + (it & 1) * TILE + tm;
    const float* ws = tiles + (it & 1) * TILE + BK * LA + tn;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
#pragma unroll
      for (int kk = 8 * half; kk < 8 * half + 8; ++kk) {
        const float4 y = *reinterpret_cast<const float4*>(ws + kk * LW);
        const float yr[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int q = 0; q < TM / 4; ++q) {
          const float4 x = *reinterpret_cast<const float4*>(as + kk * LA + 4 * q);
          const float xr[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[4 * q + i][j] = fmaf(xr[i], yr[j], acc[4 * q + i][j]);
        }
      }
      left -= 8;
      if (left == 0) {
        left = p.SL;
        end_of_slice();
        if (--slices == 0) {
          slices = GROUP;
          if (G == 1) end_of_group();
        }
      }
    }
    if (it + 1 < n_tiles) put((it + 1) & 1);
    __syncthreads();
  }
  end_of_slice();  // what is left of the last slice (zeros after a whole one)
  if constexpr (G > 1) {  // the sets' sums meet in shared memory, in order
#pragma unroll
    for (int i = 0; i < TM; ++i)
      *reinterpret_cast<float4*>(smem + (set * BM + tm + i) * BN + tn) =
          make_float4(grp[i][0], grp[i][1], grp[i][2], grp[i][3]);
    __syncthreads();
    for (int o = threadIdx.x; o < BM * BN; o += G * SET) {
      const int m = m0 + o / BN, n = n0 + o % BN;
      float total = 0.f;
#pragma unroll
      for (int g = 0; g < G; ++g) total += smem[g * BM * BN + o];
      if (m < p.T && n < p.N) p.out[(size_t)m * p.N + n] = total + (p.bias ? p.bias[n] : 0.f);
    }
  } else {
    end_of_group();
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int m = m0 + tm + i;
      if (m >= p.T) continue;
      const float4 t = mine[i * SET];
      const float v[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int n = n0 + tn + j;
        if (n < p.N) p.out[(size_t)m * p.N + n] = v[j] + (p.bias ? p.bias[n] : 0.f);
      }
    }
  }
}

template <int NPT, int NG>
static cudaError_t launch_few(const Args& p, cudaStream_t stream) {
  constexpr int NB = NPT * NG, smem = STAGES * (NB + FEW_T) * ROW * 4;
  static_assert(FEW_T * NB * (SLICES + 1) * 4 <= smem, "");
  if (const cudaError_t e = allow_dynamic_smem<few_rows_kernel<NPT, NG>, smem>()) return e;
  const dim3 grid((p.N + NB - 1) / NB, (p.T + FEW_T - 1) / FEW_T);
  return lse::launch(few_rows_kernel<NPT, NG>, grid, 32 * NG, smem, stream, p);
}

template <int BM, int BN, int TM, int G, int BLOCKS>
static cudaError_t launch_tiles(const Args& p, bool vec, cudaStream_t stream) {
  constexpr int smem = (G * 2 * BK * (BM + BN + 8) + (G == 1 ? BM * BN : 0)) * 4;
  if (const cudaError_t e = allow_dynamic_smem<tiles_kernel<BM, BN, TM, G, BLOCKS>, smem>()) return e;
  const dim3 grid((p.N + BN - 1) / BN, (p.T + BM - 1) / BM);
  if (grid.y > 65535) return cudaErrorInvalidValue;
  return lse::launch(tiles_kernel<BM, BN, TM, G, BLOCKS>, grid, G * (BM / TM) * (BN / 4), smem, stream, p, vec);
}

}  // namespace gf32
}  // namespace lse

extern "C" int lse_gemm_f32(const float* a, const float* w, const float* bias, float* out, int T,
                            int N, int K, cudaStream_t stream, int w_early) {
  using namespace lse::gf32;
  if (T <= 0 || N <= 0) return LSE_OK;
  if (K <= 0 || (T + 63) / 64 > 65535) return LSE_BAD_ARGUMENT;
  const Args p{a, w, bias, out, T, N, K, slice_len(K), w_early};
  const bool vec = K % 4 == 0 && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
  // Blocks come to the SMs in rounds of 148, and a product takes about (a start) + (rounds) x (a block's share of an SM).
  // With the constants below (tenths of a us at K = 576; all grow with K alike, the small tiles a little less) the
  // choice was within 2.7 % of the best of the four in the mean of 316 products (N 576 to 49152, K 576 to 8192, 1 to
  // 2048 rows) and nowhere slower than a kernel of 64 x 64 tiles with one chain of additions, but for 4 % of a K that
  // is no multiple of 4. Alone with w out of L2, few rows / small / 64 x 64 / 64 x 128, us:
  //   16384 x 576   8 rows 29 / 41 / 49 / 49    32 rows 74 / 43 / 49 / 49    128 rows - / 127 / 96 / 80
  //   2048 x 2048   16 rows 22 / 41 / 104 / 139    300 rows - / 128 / 152 / 150    900 rows - / 307 / 307 / 250
  //   3072 x 576    24 rows 18 / 20 / 35 / 47    900 rows - / 164 / 113 / 121    2048 rows - / 363 / 238 / 221
  //   49152 x 576   8 rows 64 / 100 / 127 / 117    48 rows - / 186 / 131 / 119    900 rows - / 2578 / 1613 / 1388
  auto rounds = [&](int bm, int bn) {
    const long long blocks = (long long)((T + bm - 1) / bm) * ((N + bn - 1) / bn);
    return (blocks + 147) / 148;
  };
  const long long small = 100 + (K >= 1024 ? 70 : 80) * rounds(32, 32);
  const long long square = 180 + 200 * rounds(64, 64), wide = 100 + 360 * rounds(64, 128);
  const long long few = vec && T <= 32 ? 80 + 22 * rounds(FEW_T, 16) : LLONG_MAX;
  const long long tiles = square < wide ? square : wide;
  // small tiles: where no SM gets more than two blocks they may have the registers of four (123 instead of 64 a thread:
  // 6 to 11 % faster there, 6 % slower with more blocks)
  const bool airy = rounds(32, 32) <= 2;
  const cudaError_t e = few <= small && few <= tiles               ? launch_few<4, 4>(p, stream)
                        : small <= tiles && (T + 31) / 32 <= 65535 ? (airy ? launch_tiles<32, 32, 4, 4, 2>(p, vec, stream)
                                                                           : launch_tiles<32, 32, 4, 4, 4>(p, vec, stream))
                        : square <= wide                           ? launch_tiles<64, 64, 4, 1, 3>(p, vec, stream)
                                                                   : launch_tiles<64, 128, 8, 1, 2>(p, vec, stream);
  return e == cudaSuccess ? LSE_OK : LSE_LAUNCH_FAILED;
}
