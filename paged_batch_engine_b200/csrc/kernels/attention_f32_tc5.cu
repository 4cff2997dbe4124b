// Paged causal attention over float32 pages on the fifth-generation tensor cores, with float32's precision: queries, keys,
// softmax weights and values are each cut into three bfloat16 terms, x = h + m + l, which hold all of their 24 bits, and a
// product of two such factors is the six products hh, hm, mh, mm, hl, lh (what is left out is 2^-25 of it at most).
// It takes steps with a request of more than SMALL packed rows (row * group + head of the group, as in attention_simple.cu), whole;
// what it hands back is attention_simple.cu's.  Requests of at most SMALL packed rows keep that kernel's key splits.
//
// A block owns 128 packed rows of a request and key/value head and walks over tiles of 64 keys:
//  * warps 8-11 fetch a tile's keys and values from the pages, split them and lay the terms down under the 128-byte
//    swizzle that the tensor cores read (64-wide blocks; the values as they lie, MN-major), one buffer of each: a tile's
//    keys are split while the values before them are multiplied, and the other way round;
//  * warp 12 issues the products: S = Q K^T into two alternating buffers in tensor memory, the small products first, and
//    O_j = P V of one tile into two others, with P as the A operand from tensor memory;
//  * warps 0-7 are the softmax, two threads a row (32 keys and half the outputs each): weights by expf, their sums and the
//    outputs in registers.  The tensor cores cut off what does not fit a sum, so outputs are not left to them over tiles: each
//    tile's O_j is summed from zero and added with one rounding.
// The tensor pipe binds: 48 products of 128 x 64 x 16 (68 clocks each: the queries' way out of shared memory) and 24 of 128 x HD x
// 16, 4,800 clocks a tile at HD = 128; short prompts wait for the longest row tile's walk.  The split has to be free of
// branches and its loads of waits: with a test a number and a tile's pages looked up when its loads were due, a tile took
// 18,000 clocks.
// Multiply-adds (attention_simple.cu) -> this: 17 + 311 + 700 tokens, 12 heads of 128 over 2, 165 -> 46 us; 2,048 tokens, 28 heads over 4,
// 1,950 -> 255; 14 heads of 64 over 2 680 -> 82; 12 rows behind 4,000 tokens 735 -> 270; 11 rows alone 22 either way.
// Relative error against 64 bits there: 3.2e-7 -> 2.0e-7, 4.6e-7 -> 2.4e-7, 4.0e-7 -> 1.7e-7, 1.3e-6 -> 3.4e-7, 1.5e-7 -> 1.2e-7.
//
// A block that meets an element which is neither zero nor of a size from 2^-102 to 2^47 sets its flag: its rows are then made by
// attention_simple.cu's multiply-adds, launched behind (a smaller element's third term would fall under bfloat16's smallest
// normal number, and an infinity times a term or a weight that is zero is no number).
//
// Every mbarrier wait is bounded; one that runs out sets *err and the roles run to their end.
//
// Compile with -DPBE_HEAD_DIM=64 or 128.
#include <cuda_bf16.h>

#include "attention_simple.cu"
#include "float_terms.cuh"
#include "opt_in.cuh"
#include "tcgen05.cuh"

using namespace pbe::tc5;

#if !defined(PBE_HEAD_DIM) || (PBE_HEAD_DIM != 64 && PBE_HEAD_DIM != 128)
#error "PBE_HEAD_DIM must be 64 or 128"
#endif

namespace {
namespace f32_tc5 {
constexpr int TERMS = 3;
constexpr int BM = 128, BN = 64;
constexpr int SMALL = 64;                       // packed rows of a request whose long key ranges are cut into splits
constexpr int SIMPLE_ROWS = 16;                 // a row tile there
constexpr int SOFT_WARPS = 8, SPLIT_WARPS = 4, MMA_WARP = SOFT_WARPS + SPLIT_WARPS;
constexpr int NTHREADS = 32 * (MMA_WARP + 1);
constexpr int Q_BYTES = BM * HD * 2, KV_BYTES = BN * HD * 2;          // a term
constexpr int S_COL = 0, P_COL = 2 * BN, O_COL = 256, TMEM_COLS = 512;
static_assert(P_COL + TERMS * BN / 2 <= O_COL && O_COL + 2 * HD <= TMEM_COLS, "tensor memory");

struct Barriers {
  uint64_t q_full, k_full, k_empty, v_full, v_empty, s_full[2], p_full, o_ready[2];
  uint32_t tmem_base;
  int odd;
  int place[8][BN];                             // of a tile's keys in the cache, in rows of HD
  float row_max[2][2][BM];                      // by tile parity and half
};
constexpr size_t TILE_BYTES = (size_t)TERMS * (Q_BYTES + 2 * KV_BYTES);
constexpr size_t SMEM_BYTES = TILE_BYTES + sizeof(Barriers) + 1024;   // and what aligns the tiles
static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");

struct F32Extra {
  int num_tiles, R;
  int32_t* flags;                               // [places, max_splits, KV]: 1 where a block hands its rows back
};

// byte offset of element (row, col) in a [64-wide blocks][rows] bf16 tile with 128-byte swizzle
__device__ __forceinline__ uint32_t swz(int row, int col, int rows) {
  const int blk = col >> 6, cc = col & 63;
  return (uint32_t)(blk * rows * 128 + row * 128 + ((((cc >> 3) ^ (row & 7)) << 4) | ((cc & 7) << 1)));
}
__device__ __forceinline__ void tmem_st16_nowait(uint32_t taddr, const uint32_t* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
        "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
// eight consecutive numbers into the three terms' tiles at byte offset `at`
__device__ __forceinline__ void lay_down(float (&v)[8], unsigned char* tile, uint32_t at, int term_bytes, Sizes& sizes) {
#pragma unroll
  for (int i = 0; i < 8; ++i) sizes.add(v[i]);
#pragma unroll
  for (int t = 0; t < TERMS; ++t) {
    uint4 w;
    w.x = next_term(v[0], v[1]);
    w.y = next_term(v[2], v[3]);
    w.z = next_term(v[4], v[5]);
    w.w = next_term(v[6], v[7]);
    *reinterpret_cast<uint4*>(tile + t * term_bytes + at) = w;
  }
}

__device__ __forceinline__ int lowest_key(const AttnParams& p, int r) {
  return p.window > 0 ? max(0, p.seq_len[r] - p.q_len[r] - p.window + 1) : 0;
}
// blocks of a request: its row tiles, or the splits of a request of one tile
__device__ __forceinline__ int blocks_of(const AttnParams& p, int r, int G) {
  const int packed = p.q_len[r] * G;
  if (packed > SMALL) return (packed + BM - 1) / BM;
  return packed > 0 ? (p.seq_len[r] + p.split_keys - 1) / p.split_keys - lowest_key(p, r) / p.split_keys : 0;
}
// The request that block `index` of the step belongs to and its first block, by a warp (-1: there is no such block)
__device__ int2 locate(int index, const AttnParams& p, int R, int G) {
  const int lane = threadIdx.x & 31;
  int before = 0;
  for (int i0 = 0; i0 < R; i0 += 32) {
    const int n = i0 + lane < R ? blocks_of(p, i0 + lane, G) : 0;
    int t = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += up;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, index < before + t);
    if (hit) {
      const int from = __ffs(hit) - 1;
      return make_int2(i0 + from, before + __shfl_sync(0xffffffffu, t - n, from));
    }
    before += __shfl_sync(0xffffffffu, t, 31);
  }
  return make_int2(-1, before);
}

__global__ void __launch_bounds__(NTHREADS, 1) attention_f32_tc5_kernel(AttnParams p, F32Extra x, int* err) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* Qs = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);   // [TERMS][HD / 64][128][128 B]
  unsigned char* Ks = Qs + TERMS * Q_BYTES;               // [TERMS][HD / 64][64 keys][128 B]
  unsigned char* Vs = Ks + TERMS * KV_BYTES;
  Barriers& bar = *reinterpret_cast<Barriers*>(Vs + TERMS * KV_BYTES);

  pdl_wait();
  const int KV = p.num_kv_heads, H = p.num_heads, G = H / KV, P = p.page_tokens;
  const int kvh = blockIdx.x % KV;
  // the last row tiles of a request have the most keys: they come first
  const int index = x.num_tiles - 1 - (int)(blockIdx.x / KV);
  const int2 found = locate(index, p, x.R, G);
  const int r = found.x;
  if (r < 0) return;
  const int qs = p.q_start[r], nq = p.q_len[r], sl = p.seq_len[r];
  const int n_packed = nq * G;
  const bool cut = n_packed <= SMALL;
  const int nsplit = cut ? blocks_of(p, r, G) : 1, split = cut ? index - found.y : 0;
  const int tile = cut ? 0 : index - found.y, pr0 = tile * BM;
  const int rows_here = min(BM, n_packed - pr0);
  const int row_lo = pr0 / G, row_hi = (pr0 + rows_here - 1) / G;
  const int pos0 = sl - nq;
  int k_end = pos0 + row_hi + 1;
  int k_begin = p.window > 0 ? max(0, pos0 + row_lo - p.window + 1) : 0;
  if (nsplit > 1) {                                       // at absolute multiples of split_keys, none of them empty
    const int s0 = k_begin / p.split_keys + split;
    k_begin = max(k_begin, s0 * p.split_keys);
    k_end = min(k_end, (s0 + 1) * p.split_keys);
  }
  const int tile0 = (k_begin / BN) * BN;
  const int n_tiles = (k_end - tile0 + BN - 1) / BN;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    mbar_init(&bar.q_full, SOFT_WARPS);
    mbar_init(&bar.k_full, SPLIT_WARPS);
    mbar_init(&bar.k_empty, 1);
    mbar_init(&bar.v_full, SPLIT_WARPS);
    mbar_init(&bar.v_empty, 1);
    mbar_init(&bar.p_full, SOFT_WARPS);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bar.s_full[i], 1);
      mbar_init(&bar.o_ready[i], 1);
    }
    bar.odd = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&bar.tmem_base)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = bar.tmem_base;
  Sizes sizes;                                             // of what this thread has split

  if (warp < SOFT_WARPS) {
    // ---------------------------------------------------------------- softmax and outputs: half a row a thread
    const int quarter = warp & 3, half = warp >> 2;
    const int row = quarter * 32 + lane;                   // tensor-memory lane == row of the tile
    const int pr = pr0 + row;
    const bool live = pr < n_packed;
    const int qrow = live ? pr / G : 0;
    const int head = kvh * G + (live ? pr - qrow * G : 0);
    const size_t at_row = ((size_t)(qs + qrow) * H + head) * HD + half * (HD / 2);
    {
      const float* src = (const float*)p.q + at_row;
#pragma unroll 2
      for (int c = 0; c < HD / 2; c += 8) {
        float v[8];
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
        if (live) {
          a = *reinterpret_cast<const float4*>(src + c);
          b = *reinterpret_cast<const float4*>(src + c + 4);
        }
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        lay_down(v, Qs, swz(row, half * (HD / 2) + c, BM), Q_BYTES, sizes);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.q_full);
    }
    const int pos = live ? min(pos0 + qrow, k_end - 1) : -1;                 // the last key this row sees, and the first
    const int lo = max(k_begin, p.window > 0 ? pos0 + qrow - p.window + 1 : 0);
    const int pos_min = min(pos0 + row_lo, k_end - 1), lo_max = max(k_begin, p.window > 0 ? pos0 + row_hi - p.window + 1 : 0);
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const uint32_t s_addr = lane_addr + S_COL + half * (BN / 2), p_addr = lane_addr + P_COL + half * (BN / 4);
    const uint32_t o_addr = lane_addr + O_COL + half * (HD / 2);
    float m_run = -INFINITY, l_run = 0.f, alpha = 0.f;
    float acc[HD / 2];
#pragma unroll
    for (int i = 0; i < HD / 2; ++i) acc[i] = 0.f;
    auto add_outputs = [&](int j) {                        // tile j's, its weights relative to the maximum after it
#pragma unroll
      for (int c = 0; c < HD / 64; ++c) {
        float v[32];
        tmem_ld32(o_addr + (j & 1) * HD + c * 32, v);
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[c * 32 + i] = fmaf(acc[c * 32 + i], alpha, v[i]);
      }
    };
    bool ok = true;
    for (int j = 0; j < n_tiles; ++j) {
      const int ts = tile0 + j * BN + half * (BN / 2);     // this thread's first key
      ok = ok && mbar_wait(&bar.s_full[j & 1], (j >> 1) & 1, err);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      float s[BN / 2];
      tmem_ld32(s_addr + (j & 1) * BN, s);
      const bool full_tile = live && ts + BN / 2 - 1 <= pos_min && ts >= lo_max;
#pragma unroll
      for (int i = 0; i < BN / 2; ++i) s[i] *= p.scale;
      if (!full_tile) {                                    // keys lo .. pos of the row are seen
        const int from = lo - ts, to = pos - ts;
#pragma unroll
        for (int i = 0; i < BN / 2; ++i) s[i] = i < from || i > to ? -INFINITY : s[i];
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < BN / 2; ++i) mx[i & 3] = fmaxf(mx[i & 3], s[i]);
      const float mine = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      bar.row_max[j & 1][half][row] = mine;
      asm volatile("bar.sync %0, 64;" ::"r"(1 + quarter) : "memory");      // the two warps of these rows
      const float m_new = fmaxf(m_run, fmaxf(mine, bar.row_max[j & 1][half ^ 1][row]));
      const float m_use = m_new == -INFINITY ? 0.f : m_new;
      const float next_alpha = expf(m_run - m_use);        // 0 when nothing was visible before
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < BN / 2; ++i) {
        s[i] = expf(s[i] - m_use);
        sum[i & 3] += s[i];
      }
      l_run = fmaf(l_run, next_alpha, (sum[0] + sum[1]) + (sum[2] + sum[3]));
      m_run = m_new;
      uint32_t w[TERMS][BN / 4];
#pragma unroll
      for (int t = 0; t < TERMS; ++t)
#pragma unroll
        for (int i = 0; i < BN / 4; ++i) w[t][i] = next_term(s[2 * i], s[2 * i + 1]);
      // the weights before have been read once their outputs are complete
      if (j > 0) {
        ok = ok && mbar_wait(&bar.o_ready[(j - 1) & 1], ((j - 1) >> 1) & 1, err);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      }
#pragma unroll
      for (int t = 0; t < TERMS; ++t) tmem_st16_nowait(p_addr + t * (BN / 2), w[t]);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.p_full);
      if (j > 0) add_outputs(j - 1);
      alpha = next_alpha;
    }
    pdl_launch_dependents();
    ok = ok && mbar_wait(&bar.o_ready[(n_tiles - 1) & 1], ((n_tiles - 1) >> 1) & 1, err);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    add_outputs(n_tiles - 1);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    float* sums = &bar.row_max[n_tiles & 1][0][0];         // this parity's maxima have been read
    sums[half * BM + row] = l_run;
    asm volatile("bar.sync %0, 64;" ::"r"(1 + quarter) : "memory");
    const float l = sums[row] + sums[BM + row];
    const float inv = l > 0.f ? 1.0f / l : 0.f;
    if (live && nsplit > 1) {
      const size_t at = ((size_t)p.tok_split_row[qs + qrow] * H + head) * p.max_splits + split;
      float* out = p.part_o + at * HD + half * (HD / 2);
#pragma unroll
      for (int i = 0; i < HD / 2; i += 4) *reinterpret_cast<float4*>(out + i) = make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
      if (half == 0) {
        p.part_ml[at * 2] = m_run;
        p.part_ml[at * 2 + 1] = l;
      }
    } else if (live) {
      float* out = (float*)p.out + at_row;
#pragma unroll
      for (int i = 0; i < HD / 2; i += 4)
        *reinterpret_cast<float4*>(out + i) = make_float4(acc[i] * inv, acc[i + 1] * inv, acc[i + 2] * inv, acc[i + 3] * inv);
    }
  } else if (warp < MMA_WARP) {
    // ---------------------------------------------------------------- keys and values into terms
    // While a tile's piece is split, the same piece of the tile that comes next is on its way into the registers it leaves; the
    // pages' places are looked up two tiles ahead.
    constexpr int PIECES = HD / 8, ROWS = 128 / PIECES, PASSES = BN / ROWS;
    const int thread = threadIdx.x - 32 * SOFT_WARPS, first = thread / PIECES, piece = thread % PIECES;
    const int32_t* bt = p.block_table + (size_t)r * p.bt_stride;
    auto look_up = [&](int j) {                            // threads 0 .. BN - 1: a key's row in the cache, -1: there is none
      const int key = tile0 + j * BN + thread;
      if (key < k_begin || key >= k_end) return -1;
      const int page = bt[key / P];
      return page >= 0 ? (page * KV + kvh) * P + key % P : -1;
    };
    float4 v[PASSES][2];
    auto request = [&](bool keys, int j, int i) {
      const int at = max(bar.place[j & 7][i * ROWS + first], 0);
      const float4* src = reinterpret_cast<const float4*>((const float*)(keys ? p.k_cache : p.v_cache) + (size_t)at * HD + piece * 8);
      v[i][0] = src[0];
      v[i][1] = src[1];
    };
    if (thread < BN) {
      bar.place[0][thread] = look_up(0);
      bar.place[1][thread] = look_up(1);
    }
    asm volatile("bar.sync 5, 128;" ::: "memory");
#pragma unroll
    for (int i = 0; i < PASSES; ++i) request(true, 0, i);
    bool ok = true;
    // in the order in which the buffers come free: K0 V0 K1 | K2 V1 | K3 V2 | ...
    const int items = 2 * n_tiles;
    for (int it = 0; it < items; ++it) {                   // to its end also where a wait has run out: the four warps meet in it
      auto tile_of = [&](int i, bool& keys) {              // the last is a value tile
        keys = i == 0 || i == 2 || (i > 2 && (i & 1) && i != items - 1);
        return i < 2 ? 0 : i == items - 1 ? n_tiles - 1 : keys ? (i + 1) / 2 : i / 2 - 1;
      };
      bool keys, next_keys = false;
      const int j = tile_of(it, keys), next = it + 1 < items ? tile_of(it + 1, next_keys) : -1;
      const int ahead = keys && thread < BN ? look_up(j + 2) : -1;
      if (j > 0) ok = ok && mbar_wait(keys ? &bar.k_empty : &bar.v_empty, (j - 1) & 1, err);
      unsigned char* dst = keys ? Ks : Vs;
#pragma unroll
      for (int i = 0; i < PASSES; ++i) {
        const bool there = bar.place[j & 7][i * ROWS + first] >= 0;
        float w[8] = {v[i][0].x, v[i][0].y, v[i][0].z, v[i][0].w, v[i][1].x, v[i][1].y, v[i][1].z, v[i][1].w};
#pragma unroll
        for (int k = 0; k < 8; ++k) w[k] = there ? w[k] : 0.f;
        if (next >= 0) request(next_keys, next, i);
        lay_down(w, dst, swz(i * ROWS + first, piece * 8, BN), KV_BYTES, sizes);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(keys ? &bar.k_full : &bar.v_full);
      if (keys) {
        if (thread < BN) bar.place[(j + 2) & 7][thread] = ahead;
        asm volatile("bar.sync 5, 128;" ::: "memory");
      }
    }
    // the commits that release the last tiles arrive on this block's barriers: it stays until they have
    ok = ok && mbar_wait(&bar.k_empty, (n_tiles - 1) & 1, err);
    ok = ok && mbar_wait(&bar.v_empty, (n_tiles - 1) & 1, err);
  } else if (lane == 0) {
    // ---------------------------------------------------------------- products
    const uint32_t idesc_s = make_idesc(BM, BN);
    const uint32_t idesc_o = make_idesc(BM, HD) | (1u << 16);              // B as it lies: MN-major
    const uint32_t q_addr = smem_u32(Qs), k_addr = smem_u32(Ks), v_addr = smem_u32(Vs);
    bool ok = mbar_wait(&bar.q_full, 0, err);
    auto scores = [&](int j) {
      ok = ok && mbar_wait(&bar.k_full, j & 1, err);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int sum = TERMS - 1; sum >= 0; --sum)                           // the small products first
#pragma unroll
        for (int t = 0; t <= sum; ++t)
#pragma unroll
          for (int ks = 0; ks < HD / 16; ++ks) {
            const uint32_t q_off = t * Q_BYTES + (ks >> 2) * (BM * 128) + (ks & 3) * 32;
            const uint32_t k_off = (sum - t) * KV_BYTES + (ks >> 2) * (BN * 128) + (ks & 3) * 32;
            umma(tmem_base + S_COL + (j & 1) * BN, make_desc(q_addr + q_off), make_desc(k_addr + k_off), idesc_s,
                 (sum < TERMS - 1 || t > 0 || ks > 0) ? 1u : 0u);
          }
      umma_commit(&bar.k_empty);
      umma_commit(&bar.s_full[j & 1]);
    };
    scores(0);
    if (n_tiles > 1) scores(1);
    for (int j = 0; j < n_tiles && ok; ++j) {
      ok = ok && mbar_wait(&bar.v_full, j & 1, err);
      ok = ok && mbar_wait(&bar.p_full, j & 1, err);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int sum = TERMS - 1; sum >= 0; --sum)
#pragma unroll
        for (int t = 0; t <= sum; ++t)
#pragma unroll
          for (int ks = 0; ks < BN / 16; ++ks)
            umma_ts(tmem_base + O_COL + (j & 1) * HD, tmem_base + P_COL + t * (BN / 2) + ks * 8,
                    desc_mn_major(v_addr + (sum - t) * KV_BYTES + ks * 16 * 128, BN), idesc_o,
                    (sum < TERMS - 1 || t > 0 || ks > 0) ? 1u : 0u);
      umma_commit(&bar.v_empty);
      umma_commit(&bar.o_ready[j & 1]);
      if (j + 2 < n_tiles) scores(j + 2);
    }
  }
  if (!sizes.whole()) bar.odd = 1;
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (threadIdx.x == 0) x.flags[((size_t)((long long)qs * G / BM + r + tile) * p.max_splits + split) * KV + kvh] = bar.odd;
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}
}  // namespace f32_tc5
}  // namespace

// num_tiles: the row tiles of the requests of more than SMALL packed rows and the splits of the others.  flags: [T * group / BM + R + 1,
// max_splits, KV], one int for every block; attention_simple.cu then takes what is flagged.
PBE_EXPORT int pbe_attn_f32(const AttnParams* params, int num_work, int num_tiles, int R, int32_t* flags, int* err, cudaStream_t stream) {
  using namespace f32_tc5;
  if (num_tiles <= 0 || num_work <= 0) return 0;
  const AttnParams p = *params;
  if (p.num_heads % p.num_kv_heads != 0 || p.tile_rows != SIMPLE_ROWS || p.page_tokens < 1 || R < 1 || flags == nullptr ||
      p.split_keys < f32_tc5::BN || p.split_keys % f32_tc5::BN != 0 || p.max_splits < 1 || (long long)num_tiles * p.num_kv_heads > 0x7fffffffLL)
    return (int)cudaErrorInvalidValue;
  // rows that do not start on a 16-byte boundary are the multiply-adds' too
  if (((uintptr_t)p.q | (uintptr_t)p.k_cache | (uintptr_t)p.v_cache | (uintptr_t)p.out | (uintptr_t)p.part_o) & 15)
    return launch_simple(params, num_work, PBE_F32, Rest{nullptr}, stream);
  static OptIn opt_in;
  if (const cudaError_t e = opt_in(SMEM_BYTES, attention_f32_tc5_kernel)) return (int)e;
  launch_k(attention_f32_tc5_kernel, num_tiles * p.num_kv_heads, NTHREADS, SMEM_BYTES, stream, p, F32Extra{num_tiles, R, flags}, err);
  const int rc = launch_status();
  return rc != 0 ? rc : launch_simple(params, num_work, PBE_F32, Rest{flags}, stream);
}
