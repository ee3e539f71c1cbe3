// Flash-style causal attention for portions of prompts on the 5th-generation tensor cores
// (head size 64, bfloat16, page size a power of two >= 8; everything before a row, a window or the row's chunk; soft
// caps and sinks).
//
// One block = 128 query rows of one head. Per tile of 64 keys:
//   S = Q K^T        tcgen05.mma, A = Q tile and B = K tile in shared memory (both K-major, TMA with
//                    128-byte swizzle, K tiles fetched page by page through the block table),
//                    accumulator S [128 x 64] float32 in tensor memory;
//   softmax          256 threads, two per query row: even tiles are *stream* 0, odd tiles stream 1, and each
//                    stream is a complete online softmax of its own: tcgen05.ld of its 64 scores, running
//                    maximum and sum in float32 (base-2 exponent, scale folded into the multiply-add), P
//                    rounded to bfloat16 and written back to tensor memory with tcgen05.st. The two threads of
//                    a row never talk to each other until the end;
//   O_s += P_s V     per stream s: tcgen05.mma with A = P from tensor memory and B = the V tile in shared
//                    memory (N-major: rows are keys), accumulator O_s [128 x 64] float32 in tensor memory;
//   end              O = (O_0 w_0 + O_1 w_1) / (l_0 w_0 + l_1 w_1), w_s = 2^(m_s - max m): each thread
//                    of a row writes half of the head dims.
// A stream's reference maximum moves only when a row of the warp outgrows it by 2^8; only then is
// its O rescaled in tensor memory (tcgen05.ld / st) before its next P V. Warps 0-3 are stream 0 and warps 4-7
// stream 1 (warp w owns tensor-memory lanes 32 (w mod 4) ..), warp 8 looks the pages up and its lanes issue the
// TMA copies, one lane of warp 9 issues the MMAs. Every mbarrier wait is bounded; the barriers of a cluster
// are reached by every warp of every block behind its bounded waits.
//
// What bounds it: the exp unit (16 per clock and SM) and, short of that, the latencies of a tile: wait, tcgen05.ld,
// maximum, exponentials, tcgen05.st, arrival, P V, next Q K^T. A thread therefore takes 64 scores per round, the
// two streams of a block are never in step, and two blocks share an SM. Pages of 16 tokens make eight copies per
// tile; issued by one lane they were what a tile waited for. 2040 rows behind 6144 keys, 9 heads: 123 us (one lane
// issuing, both streams on halves of one tile) -> 94 us -> 60 us with the keys shared by two blocks (exp unit alone:
// 29 us); 2048 rows behind 4096 keys, 32 heads: 166 -> 141 us (75 us); 2048 rows alone, 32 heads: 45 -> 47 us by itself,
// 37.6 -> 35.3 back to back (15 us). Short portions that just overflow the SMs lose: four of 700 rows, 15 heads (360
// blocks) 16.5 -> 18.4, eight of 300 rows, 32 heads 22.9 -> 23.3.
// 2048 rows, 32 heads, a window of 1024 with sinks: 41 us, chunks of 512: 29 us (mma.sync kernel: 125, 59).
#pragma once

#include "attention_args.h"
#include "tma_util.cuh"

namespace lse {
namespace atc {

using namespace tma;

constexpr int HD = 64;           // head size served by this kernel
constexpr int QT = 128;          // query rows per block
constexpr int KT = 64;           // keys per tile
constexpr int STAGES = 4;        // key/value tiles in flight
constexpr int SOFTMAX_WARPS = 8;  // two streams of four warps
constexpr int THREADS = (SOFTMAX_WARPS + 2) * 32;
constexpr uint32_t Q_BYTES = QT * HD * 2, KV_BYTES = KT * HD * 2;
// Tensor-memory columns: S and O of each stream. A stream's P (32 packed columns) is written over its own S once
// that is in registers; MMAs of one thread run in issue order, so the stream's next Q K^T cannot overtake the
// P V that still reads P.
constexpr uint32_t COL_S = 0, S_COLS = 64, COL_O = 128, O_COLS = 64, TMEM_COLS = 256;

__device__ __forceinline__ void umma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void umma_ts(uint32_t d, uint32_t a_tmem, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d), "r"(a_tmem), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,"
      "%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
        "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]),
        "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]),
        "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,"
      "%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]),
        "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]),
        "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]),
        "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]),
        "r"(v[31])
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
        "=r"(v[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]),
        "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]),
        "r"(v[15])
      : "memory");
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Two float32 operations in one instruction; both halves are rounded as fmaf and + round.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 x, y, z, w;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\t"
      "fma.rn.f32x2 w, x, y, z;\n\tmov.b64 {%0, %1}, w;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 x, y, w;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
      "add.rn.f32x2 w, x, y;\n\tmov.b64 {%0, %1}, w;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// This block's shared-memory address `addr` in block `rank` of the cluster.
__device__ __forceinline__ uint32_t peer_address(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void store_peer4(uint32_t addr, float a, float b, float c, float d) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ void store_peer2(uint32_t addr, float a, float b) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(a), "f"(b) : "memory");
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

struct Params {
  LseAttnArgs a;
  int page_shift;   // log2(page_tokens)
  int box_rows;     // rows per key/value TMA box: min(page_tokens, KT)
  int* error_flag;
};

// A cluster of `parts` blocks (1, 2 or 4) shares the keys of one (query tile, head); at the end every block
// merges 64 / parts head dims of all rows. Its inbox, where the key and value tiles were: [part][row][64 / parts + 4]
// sums, then [part][row] (maximum, sum).
__host__ __device__ constexpr int inbox_row(int parts) { return HD / parts + 4; }
__host__ __device__ constexpr int inbox_bytes(int parts) {
  return parts > 1 ? parts * QT * (inbox_row(parts) + 2) * 4 : 0;
}

// First key that a query at position qpos may read (window and chunk together); it never moves back.
__device__ __forceinline__ int first_local_key(const LseAttnArgs& a, int qpos) {
  const int lo = a.window > 0 ? max(0, qpos - a.window + 1) : 0;
  return a.chunk > 0 ? max(lo, qpos / a.chunk * a.chunk) : lo;
}

// CAP: the scores are scaled and soft-capped as they leave tensor memory. PARTS: blocks per (query tile, head).
// LOCAL: a window or chunks. Keys before a row's first are masked like those behind it; the first tile starts on a
// multiple of 64, and what a page that is no longer held would bring is read from the first page that is.
template <bool CAP, int PARTS, bool LOCAL>
__global__ void __launch_bounds__(THREADS, 2)
prefill_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                  const __grid_constant__ CUtensorMap map_v, const Params p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* q_tile = base;
  unsigned char* k_tiles = q_tile + Q_BYTES;
  unsigned char* v_tiles = k_tiles + STAGES * KV_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(v_tiles + STAGES * KV_BYTES);
  uint64_t* q_full = bars;                 // [1]
  uint64_t* kv_full = bars + 1;            // [STAGES]
  uint64_t* kv_empty = kv_full + STAGES;   // [STAGES]
  uint64_t* s_full = kv_empty + STAGES;    // [stream] S of the stream's next tile is in tensor memory
  uint64_t* p_full = s_full + 2;           // [stream] its P is written (and its O rescaled): 4 arrivals
  uint64_t* o_done = p_full + 2;           // [1] every P V has finished
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_done + 1);
  float* inbox = reinterpret_cast<float*>(k_tiles);
  static_assert(inbox_bytes(PARTS) <= 2 * STAGES * (int)KV_BYTES, "");
  __shared__ float pair_m[2][QT], pair_l[2][QT];  // the streams' final maxima and sums
  __shared__ volatile int failed;
  __shared__ volatile int issued;  // key/value tiles the producer has requested

  const LseAttnArgs& a = p.a;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // heads vary fastest over the grid, tiles (longest first) slowest: every head's long tiles start early
  const int seq = a.tiles[2 * blockIdx.y], q0 = a.tiles[2 * blockIdx.y + 1];
  const int head = blockIdx.x / PARTS, part = PARTS > 1 ? (int)cluster_rank() : 0;
  const int kvh = head / (a.num_heads / a.num_kv_heads);
  const int q_start = a.cu_q[seq];
  const int q_len = a.cu_q[seq + 1] - q_start;
  const int ctx = a.ctx_lens[seq];
  const int pos0 = ctx - q_len;
  const int rows_here = min(QT, q_len - q0);
  const int k_end = pos0 + q0 + rows_here;  // one past the last key any row of the tile reads
  const int k_lowest = LOCAL ? first_local_key(a, pos0 + q0) : 0;  // of the tile's first row
  const int t_lowest = k_lowest / KT, all_tiles = (k_end + KT - 1) / KT - t_lowest;
  const int t_first = t_lowest + all_tiles * part / PARTS;   // this block's tiles of keys
  const int n_tiles = t_lowest + all_tiles * (part + 1) / PARTS - t_first;

  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_q) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_k) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_v) : "memory");
    failed = 0;
    issued = 0;
    mbar_init(q_full, 1);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&kv_full[s], 1);
      mbar_init(&kv_empty[s], 1);
    }
    mbar_init(&s_full[0], 1);
    mbar_init(&s_full[1], 1);
    mbar_init(&p_full[0], 4);
    mbar_init(&p_full[1], 4);
    mbar_init(o_done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  // Dependents may become resident only now that this block holds its tensor memory: a dependent
  // that allocated columns first and then sat in its dependency wait could keep this block
  // waiting in tcgen05.alloc for ever.
  pdl_trigger();
  pdl_wait();  // queries, keys and values were written by the kernel before this one

  if (warp == SOFTMAX_WARPS) {
    // ---- TMA producer. The whole warp looks up block-table entries, one box of a key/value tile
    // per lane and 32 boxes at a time, so that the lookups of several tiles are one round trip
    // to memory; the lanes that hold a tile's rows then issue its copies themselves, keys and values.
    if (lane == 0) {
      mbar_expect_tx(q_full, Q_BYTES);
      tma_load_2d(q_tile, &map_q, q_full, head * HD, q_start + q0);
    }
    const int* table = a.block_tables + (size_t)seq * a.table_stride;
    const int last_page_idx = (k_end - 1) >> p.page_shift, first_page_idx = k_lowest >> p.page_shift;
    const int boxes = KT / p.box_rows;  // 1, 2, 4 or 8
    const int group = 32 / boxes;       // tiles looked up together
    const int t_mine = lane / boxes, b_l = lane % boxes;
    int ok = 1;
    for (int g0 = 0; g0 < n_tiles && ok; g0 += group) {
      const int t_l = g0 + t_mine;
      int row_l = 0;
      if (t_l < n_tiles) {
        const int j = (t_first + t_l) * KT + b_l * p.box_rows;
        // a box past the context re-reads the last valid page, one before the first key the first page that is
        // held: their keys are masked, and their values cleared before the multiply
        const int pi = max(min(j >> p.page_shift, last_page_idx), first_page_idx);
        const int off = (j >> p.page_shift) <= last_page_idx ? (j & (a.page_tokens - 1)) : 0;
        row_l = (table[pi] * a.num_kv_heads + kvh) * a.page_tokens + off;
      }
      const int g_end = min(g0 + group, n_tiles);
      for (int t = g0; t < g_end && ok; ++t) {
        const int s = t % STAGES;
        if (lane == 0) {
          if (failed || (t >= STAGES && !mbar_wait(&kv_empty[s], ((t / STAGES) - 1) & 1))) {
            failed = 1;
            ok = 0;
          } else {
            mbar_expect_tx(&kv_full[s], 2 * KV_BYTES);
            issued = t + 1;
          }
        }
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (ok && t_l == t) {
          tma_load_2d(k_tiles + s * KV_BYTES + b_l * p.box_rows * HD * 2, &map_k, &kv_full[s], 0, row_l);
          tma_load_2d(v_tiles + s * KV_BYTES + b_l * p.box_rows * HD * 2, &map_v, &kv_full[s], 0, row_l);
        }
        __syncwarp();
      }
    }
  } else if (warp == SOFTMAX_WARPS + 1) {
    if (lane == 0) {
      // ---- MMA issuer
      constexpr uint32_t idesc_qk = instr_desc_bf16(QT, KT, 0);   // K tile K-major
      constexpr uint32_t idesc_pv = instr_desc_bf16(QT, HD, 1);   // V tile N-major (rows are keys)
      bool ok = mbar_wait(q_full, 0);
      const uint64_t dq = smem_desc_sw128(smem_u32(q_tile));
      auto issue_qk = [&](int t) -> bool {  // S of stream t & 1 = Q K_t^T once tile t has landed
        const int s = t % STAGES;
        if (!mbar_wait(&kv_full[s], (t / STAGES) & 1)) return false;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t dk = smem_desc_sw128(smem_u32(k_tiles + s * KV_BYTES));
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk)  // 16 head dims = 32 bytes along the swizzled row
          umma_ss(tmem + COL_S + (t & 1) * S_COLS, dq + 2 * kk, dk + 2 * kk, idesc_qk, kk > 0 ? 1u : 0u);
        umma_commit(&s_full[t & 1]);
        return true;
      };
      if (ok && n_tiles > 0) ok = issue_qk(0);
      if (ok && n_tiles > 1) ok = issue_qk(1);
      for (int t = 0; t < n_tiles && ok && !failed; ++t) {
        const int s = t % STAGES, st = t & 1;
        ok = mbar_wait(&p_full[st], (t >> 1) & 1);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t dv = smem_desc_sw128(smem_u32(v_tiles + s * KV_BYTES));
#pragma unroll
        for (int kk = 0; kk < KT / 16; ++kk)  // 16 keys = 16 rows of 128 bytes = 8 packed columns of P
          umma_ts(tmem + COL_O + st * O_COLS, tmem + COL_S + st * S_COLS + 8 * kk, dv + (2048 >> 4) * kk, idesc_pv,
                  (t > 1 || kk > 0) ? 1u : 0u);
        umma_commit(&kv_empty[s]);
        if (t + 2 < n_tiles) ok = issue_qk(t + 2);
      }
      if (ok) umma_commit(o_done);
      if (!ok) failed = 2;
    }
    __syncwarp();
  } else {
    // ---- softmax: threads r and 128 + r own query row r (tensor-memory lane r), the first for even tiles
    const int st = warp >> 2, wq = warp & 3;
    const int r = wq * 32 + lane;
    const int qpos = pos0 + q0 + r;
    const bool row_valid = r < rows_here;
    const uint32_t lane_base = tmem + ((uint32_t)(wq * 32) << 16);
    const uint32_t o_col = lane_base + COL_O + st * O_COLS;
    const float sl2 = (CAP ? 1.f : a.scale) * 1.4426950408889634f;
    // cap * tanh(s / cap) by tanh(y) = 1 - 2 / (1 + 2^(2 log2(e) y)); a power below the smallest number counts as zero
    const float cap = CAP ? a.softcap : 0.f, to_exp = CAP ? a.scale * (2.8853900817779268f / a.softcap) : 0.f;
    auto softcap = [&](uint32_t s) {
      return __float_as_uint(fmaf(-2.f * cap, __fdividef(1.f, 1.f + ex2(__uint_as_float(s) * to_exp)), cap));
    };
    float m_run = -INFINITY, l_run = 0.f;
    bool ok = true;
    const uint32_t s_col = lane_base + COL_S + st * S_COLS;
    const int row_first = LOCAL ? first_local_key(a, qpos) : 0;
    const int last_first = LOCAL ? first_local_key(a, k_end - 1) : 0;  // of the tile's last row
    for (int t = st, round = 0; t < n_tiles; t += 2, ++round) {
      ok = mbar_wait(&s_full[st], round & 1);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      uint32_t sa[32], sb[32];  // the keys of the tile's first and second half
      tmem_ld32(s_col, sa);
      tmem_ld32(s_col + 32, sb);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if constexpr (CAP) {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          sa[j] = softcap(sa[j]);
          sb[j] = softcap(sb[j]);
        }
      }
      const int k0 = (t_first + t) * KT;
      if (k0 + KT - 1 > pos0 + q0 || (LOCAL && k0 < last_first)) {  // keys that reach an edge: mask per element
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          sa[j] = (k0 + j <= qpos && (!LOCAL || k0 + j >= row_first)) ? sa[j] : 0xff800000u;  // -inf
          sb[j] = (k0 + 32 + j <= qpos && (!LOCAL || k0 + 32 + j >= row_first)) ? sb[j] : 0xff800000u;
        }
      }
      // independent chains for the maximum and for the sum: a single chain of dependent
      // operations would leave the warp waiting on its own results
      float mx4[4] = {m_run, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int j = 0; j < 32; ++j)
        mx4[j & 3] = fmaxf(fmaxf(mx4[j & 3], __uint_as_float(sa[j])), __uint_as_float(sb[j]));
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      // The reference maximum of the exponent moves only when some row of the warp has outgrown
      // it by a factor 2^8: until then P may reach 256 (exact enough in bfloat16, sums are
      // float32) and O needs no rescaling, so most tiles do not touch O.
      // (-inf) - (-inf) is NaN and compares false: a row without keys asks for nothing.
      const bool grow = __any_sync(0xffffffffu, (mx - m_run) * sl2 > 8.f);
      const float m_new = grow ? mx : m_run;
      const float m_fin = (m_new == -INFINITY) ? 0.f : m_new;
      const float ms = m_fin * sl2;
      if (grow) {
        const float corr = ex2((m_run - m_fin) * sl2);  // m_run = -inf gives 0
        m_run = m_new;
        l_run *= corr;
        if (round > 0) {  // (this stream's P V of before is complete: its S came after it)
          uint32_t ov[16];
#pragma unroll 1
          for (int h = 0; h < 4; ++h) {
            tmem_ld16(o_col + 16 * h, ov);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < 16; ++j) ov[j] = __float_as_uint(__uint_as_float(ov[j]) * corr);
            tmem_st16(o_col + 16 * h, ov);
          }
        }
      }
      float2 sum2[2] = {make_float2(l_run, 0.f), make_float2(0.f, 0.f)};
      const float2 sl2x2 = make_float2(sl2, sl2), msx2 = make_float2(-ms, -ms);
      auto exponentials = [&](const uint32_t (&sv)[32], uint32_t col) {
        uint32_t pk[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float2 x = fma2(make_float2(__uint_as_float(sv[2 * j]), __uint_as_float(sv[2 * j + 1])), sl2x2, msx2);
          const float2 e = make_float2(ex2(x.x), ex2(x.y));
          sum2[j & 1] = add2(sum2[j & 1], e);
          pk[j] = pack2(e.x, e.y);  // element 2j in the low half, 2j+1 in the high half
        }
        tmem_st16(col, pk);
      };
      exponentials(sa, s_col);
      exponentials(sb, s_col + 16);
      const float2 sum = add2(sum2[0], sum2[1]);
      l_run = sum.x + sum.y;
      if (k0 + KT > k_end || (LOCAL && k0 < k_lowest)) {
        // Whole tiles are copied: values beside the keys that any row sees may be anything, NaN included, and zero
        // probabilities would not take them out. A thread of the stream clears half a row.
        const int key = k0 + (r >> 1);
        if (key >= k_end || key < k_lowest) {
          uint4* row = reinterpret_cast<uint4*>(v_tiles + (t % STAGES) * KV_BYTES + (r >> 1) * (HD * 2) + (r & 1) * HD);
#pragma unroll
          for (int e = 0; e < 4; ++e) row[e] = make_uint4(0, 0, 0, 0);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the multiply reads them through the async proxy
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[st]);
    }
    if (!ok) failed = 3;
    // ---- epilogue: the two streams of a row are merged; each of its threads writes 32 head dims
    pair_m[st][r] = m_run;
    pair_l[st][r] = l_run;
    if (ok && !failed && n_tiles > 0) {
      ok = mbar_wait(o_done, 0);
      if (!ok) failed = 4;
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("bar.sync 1, %0;" ::"n"(SOFTMAX_WARPS * 32) : "memory");  // the softmax warps only
    if (PARTS > 1) {
      // every block of the cluster gets the head dims that it merges, and every row's maximum and sum
      constexpr int DP = HD / PARTS, ROW = inbox_row(PARTS);
      const float m0 = pair_m[0][r], m1 = pair_m[1][r];
      const bool usable = ok && !failed && n_tiles > 0;
      const float mm = usable ? fmaxf(m0, m1) : -INFINITY;
      const float w0 = (!usable || m0 == -INFINITY) ? 0.f : ex2((m0 - mm) * sl2);
      const float w1 = (!usable || m1 == -INFINITY) ? 0.f : ex2((m1 - mm) * sl2);
      const float l = usable ? pair_l[0][r] * w0 + pair_l[1][r] * w1 : 0.f;
      const uint32_t here = smem_u32(inbox);
      cluster_arrive();
      cluster_wait();  // no block of the cluster reads its tiles any more
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t oa[16], ob[16];
        tmem_ld16(lane_base + COL_O + 32 * st + 16 * h, oa);
        tmem_ld16(lane_base + COL_O + O_COLS + 32 * st + 16 * h, ob);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
          float o[4];
#pragma unroll
          for (int e = 0; e < 4; ++e)
            o[e] = (w0 != 0.f ? __uint_as_float(oa[j + e]) * w0 : 0.f) + (w1 != 0.f ? __uint_as_float(ob[j + e]) * w1 : 0.f);
          const int d = 32 * st + 16 * h + j;
          store_peer4(peer_address(here + (uint32_t)(((part * QT + r) * ROW + d % DP) * 4), d / DP), o[0], o[1], o[2], o[3]);
        }
      }
      if (st == 0) {
#pragma unroll
        for (int z = 0; z < PARTS; ++z)
          store_peer2(peer_address(here + (uint32_t)((PARTS * QT * ROW + (part * QT + r) * 2) * 4), z), mm, l);
      }
    } else if (ok && !failed) {
      const float m0 = pair_m[0][r], m1 = pair_m[1][r];
      const float mm = fmaxf(m0, m1);
      const float w0 = (m0 == -INFINITY) ? 0.f : ex2((m0 - mm) * sl2);
      const float w1 = (m1 == -INFINITY) ? 0.f : ex2((m1 - mm) * sl2);
      float l = pair_l[0][r] * w0 + pair_l[1][r] * w1;
      if (a.sinks && l > 0.f) l += ex2(a.sinks[head] * 1.4426950408889634f - mm * sl2);
      const float inv = l > 0.f ? 1.f / l : 0.f;
      const float f0 = w0 * inv, f1 = w1 * inv;
      bf16* dst = (bf16*)a.out + (size_t)(q_start + q0 + r) * a.out_row_stride + (size_t)head * HD + 32 * st;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t oa[16], ob[16];
        tmem_ld16(lane_base + COL_O + 32 * st + 16 * h, oa);
        tmem_ld16(lane_base + COL_O + O_COLS + 32 * st + 16 * h, ob);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (row_valid) {
#pragma unroll
          for (int j = 0; j < 16; j += 8) {
            float o[8];
#pragma unroll
            for (int e = 0; e < 8; ++e)
              o[e] = (f0 != 0.f ? __uint_as_float(oa[j + e]) * f0 : 0.f) +
                     (f1 != 0.f ? __uint_as_float(ob[j + e]) * f1 : 0.f);  // (O of a stream without tiles was never written)
            uint4 w;
            w.x = pack2(o[0], o[1]);
            w.y = pack2(o[2], o[3]);
            w.z = pack2(o[4], o[5]);
            w.w = pack2(o[6], o[7]);
            *reinterpret_cast<uint4*>(dst + 16 * h + j) = w;
          }
        }
      }
    }
  }
  if constexpr (PARTS > 1) {
    __syncwarp();
    if (warp >= SOFTMAX_WARPS) {  // (the softmax warps did before they wrote)
      cluster_arrive();
      cluster_wait();
    }
    cluster_arrive();
    cluster_wait();
    constexpr int DP = HD / PARTS, ROW = inbox_row(PARTS), PIECES = DP / 8;
    const float sl2 = (CAP ? 1.f : a.scale) * 1.4426950408889634f;
    const float2* ml = reinterpret_cast<const float2*>(inbox + PARTS * QT * ROW);
    for (int i = threadIdx.x; i < rows_here * PIECES; i += THREADS) {
      const int r = i / PIECES, d = (i - r * PIECES) * 8;
      float top = -INFINITY;
#pragma unroll
      for (int z = 0; z < PARTS; ++z) top = fmaxf(top, ml[z * QT + r].x);
      float l = 0.f, o[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int z = 0; z < PARTS; ++z) {
        const float2 v = ml[z * QT + r];
        const float w = v.x == -INFINITY ? 0.f : ex2((v.x - top) * sl2);
        l = fmaf(v.y, w, l);
        const float4* src = reinterpret_cast<const float4*>(inbox + (z * QT + r) * ROW + d);
        const float4 x = src[0], y = src[1];
        o[0] = fmaf(x.x, w, o[0]); o[1] = fmaf(x.y, w, o[1]); o[2] = fmaf(x.z, w, o[2]); o[3] = fmaf(x.w, w, o[3]);
        o[4] = fmaf(y.x, w, o[4]); o[5] = fmaf(y.y, w, o[5]); o[6] = fmaf(y.z, w, o[6]); o[7] = fmaf(y.w, w, o[7]);
      }
      if (a.sinks && l > 0.f) l += ex2(a.sinks[head] * 1.4426950408889634f - top * sl2);
      const float inv = l > 0.f ? 1.f / l : 0.f;
      uint4 w;
      w.x = pack2(o[0] * inv, o[1] * inv);
      w.y = pack2(o[2] * inv, o[3] * inv);
      w.z = pack2(o[4] * inv, o[5] * inv);
      w.w = pack2(o[6] * inv, o[7] * inv);
      *reinterpret_cast<uint4*>((bf16*)a.out + (size_t)(q_start + q0 + r) * a.out_row_stride + (size_t)head * HD + part * DP + d) = w;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (threadIdx.x == 0 && failed != 0) {
    if (p.error_flag) atomicExch(p.error_flag, 200 + failed);
    // copies that were requested must land before the block's shared memory is given up
    mbar_wait(q_full, 0);
    for (int c = max(0, issued - STAGES); c < issued; ++c)
      if (!mbar_wait(&kv_full[c % STAGES], (c / STAGES) & 1)) break;
  }
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS)
                 : "memory");
  }
}

inline bool supported(const LseAttnArgs* a) {
  const int pt = a->page_tokens;
  return a->dtype == LSE_BF16 && pt >= 8 && (pt & (pt - 1)) == 0 &&
         (a->q_row_stride % 8) == 0 && (a->out_row_stride % 8) == 0;
}

template <bool CAP, int PARTS, bool LOCAL>
inline int launch_prefill_parts(const LseAttnArgs* a, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv,
                                const Params& p, cudaStream_t stream) {
  constexpr int smem = Q_BYTES + 2 * STAGES * KV_BYTES + (2 * STAGES + 6) * 8 + 16 + 1024;
  if (lse::allow_dynamic_smem<prefill_tc_kernel<CAP, PARTS, LOCAL>, smem>() != cudaSuccess) return LSE_LAUNCH_FAILED;
  const dim3 grid(a->num_heads * PARTS, a->num_tiles);
  return lse::launch_clusters(prefill_tc_kernel<CAP, PARTS, LOCAL>, grid, THREADS, PARTS, smem, stream, mq, mk, mv, p) == cudaSuccess
             ? LSE_OK
             : LSE_LAUNCH_FAILED;
}

// total_rows: rows of the query tensor; pool_rows: pages * kv_heads * page_tokens.
template <bool CAP, bool LOCAL>
inline int launch_prefill_form(const LseAttnArgs* a, long long total_rows, long long pool_rows,
                          int* error_flag, cudaStream_t stream) {
  CUtensorMap mq, mk, mv;
  const int box_rows = a->page_tokens < KT ? a->page_tokens : KT;
  if (!make_map_bf16(&mq, a->q, total_rows, (long long)a->num_heads * HD, a->q_row_stride, QT) ||
      !make_map_bf16(&mk, a->k_pages, pool_rows, HD, HD, box_rows) ||
      !make_map_bf16(&mv, a->v_pages, pool_rows, HD, HD, box_rows))
    return LSE_LAUNCH_FAILED;
  Params p;
  p.a = *a;
  p.box_rows = box_rows;
  p.page_shift = 0;
  while ((1 << p.page_shift) < a->page_tokens) ++p.page_shift;
  p.error_flag = error_flag;
  // Two blocks run on an SM at a time. A grid that leaves half of these places empty is as slow as its longest block,
  // so the keys of a (query tile, head) are shared by a cluster where they are enough to pay for its barriers and
  // merge. Back to back, 1 / 2 / 4 blocks each, us: 9 blocks, 40 keys 10.3 / 12.3 / 14.3 (alone), 512 keys
  // 10.1 / 9.0 / 8.8, 768 keys 12.7 / 10.4 / 9.3, 4096 keys 46 / 27 / 18; 32 blocks, 640 keys 11.0 / 11.7 / 12.3, 768 keys
  // 12.3 / 12.2 / 12.4, 1024 keys 14.8 / 13.9 / 13.2, 4096 keys 46 / 31 / 23; 64 blocks, 512 keys 10.9 / 11.8 / 13.0, 640 keys
  // 12.4 / 12.7 / 13.1 in one portion and 13.4 / 12.7 / 13.4 in four; 128 blocks, 640 keys 12.7 / 13.0 / 23 and
  // 14.1 / 13.4 / 26, 1024 keys 17.8 / 15.6 / 26, 4096 keys 56 / 36 / 46; 256 blocks, 1000 keys 23 / 29 / 51 (alone; a
  // further wave).
  const long long blocks = (long long)a->num_heads * a->num_tiles;
  long long keys = (long long)a->table_stride * a->page_tokens;
  auto at_most = [&](long long n) { keys = keys < n ? keys : n; };
  if (a->max_portion_ctx > 0) at_most(a->max_portion_ctx);
  if (a->window > 0) at_most((long long)a->window + QT);
  if (a->chunk > 0) at_most((long long)a->chunk + QT);
  int want = 1;
  if (blocks <= 18) want = keys > 512 ? 4 : 1;
  else if (blocks <= 32) want = keys >= 1024 ? 4 : keys >= 768 ? 2 : 1;
  else if (blocks <= 148) want = keys >= 640 ? 2 : 1;
  switch (want) {
    case 1: return launch_prefill_parts<CAP, 1, LOCAL>(a, mq, mk, mv, p, stream);
    case 2: return launch_prefill_parts<CAP, 2, LOCAL>(a, mq, mk, mv, p, stream);
    default: return launch_prefill_parts<CAP, 4, LOCAL>(a, mq, mk, mv, p, stream);
  }
}

inline int launch_prefill(const LseAttnArgs* a, long long total_rows, long long pool_rows,
                          int* error_flag, cudaStream_t stream) {
  const bool cap = a->softcap > 0.f;
  if (a->window > 0 || a->chunk > 0)
    return cap ? launch_prefill_form<true, true>(a, total_rows, pool_rows, error_flag, stream)
               : launch_prefill_form<false, true>(a, total_rows, pool_rows, error_flag, stream);
  return cap ? launch_prefill_form<true, false>(a, total_rows, pool_rows, error_flag, stream)
             : launch_prefill_form<false, false>(a, total_rows, pool_rows, error_flag, stream);
}

}  // namespace atc
}  // namespace lse
