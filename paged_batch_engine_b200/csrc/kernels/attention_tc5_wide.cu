// Prompt attention on the fifth-generation tensor cores with softmax weights that keep 32-bit accuracy: the masked
// attention (masks, score cap, sink, turned-back outputs, gate; float32 queries) over pages, and the latent
// attention over keys and values expanded from the latents.  The plan is attention_tc5.cu's: a block owns 128 packed
// rows of one key/value head and walks over tiles of 64 keys; S = Q K^T by tcgen05.mma into two alternating buffers in
// tensor memory, one softmax thread a row, O += P V with P as the A operand from tensor memory and V as it lies (MN-major);
// warp 0 loads keys and warp 6 values by TMA (128-byte swizzle, no multicast), warp 1 issues the products, warps 2-5
// are softmax, correction and epilogue; two blocks share a multiprocessor.
//
// What differs: every weight enters O as two bfloat16 terms, hi + lo (seventeen bits), which together fill exactly the
// 64 columns its scores came from (two products a step of sixteen keys); a float32 query is two terms too
// (PBE_X_LATENT 0: another product a step, and 64 KB of shared memory, which leaves the value ring one tile: its load
// hides behind the other block's work).  The tensor pipe then has 8.4 MFLOP a tile (7.3 for the latents: 192-wide keys,
// queries of one term), 1,470 clocks at full rate.  What binds prompts is the longest row tile's walk, for a key tile one
// chain of scores, softmax and products: all row tiles run at once, and 2,048 rows take 82 us with 16 heads, 73 with 8 and 66
// with 4, 3,900 clocks for each of the last tile's 32 (latents 70 with 16 heads, 62 with 8; caches cold).
//
// PBE_X_LATENT 1: a row tile holds 128 rows of one head; keys are [K_h | kr] with K_h [keys, H * 128] and V_h [keys,
// H * 128] side by side in one matrix (the latents times the heads' maps), kr [keys, 64] shared by the heads.  The
// query's rotated part is turned as it is staged.
//
// 2,048 tokens, 16 heads of 128: masked attention (capped, turned, two key/value heads) 158 us on mma.sync, 75 here;
// latent attention with its heads' maps 775 + 228 us on the latents (mma.sync, 1,600 multiply-adds a pair and head), 63
// here and 18 for gathering and expanding.  512 rows behind 4,096 tokens: whole layers 357 -> 149 and 1,018 -> 183 us.
//
// Every mbarrier wait is bounded; one that runs out sets *err and the roles run to their end.
#include <cuda_bf16.h>

#include "attention_params.cuh"
#include "opt_in.cuh"
#include "common.cuh"
#include "masked_attention.cuh"
#include "pdl.cuh"
#include "tcgen05.cuh"

using namespace pbe;
using namespace pbe::tc5;

#ifndef PBE_X_LATENT
#error "PBE_X_LATENT must be 0 (masked attention over pages) or 1 (expanded latents)"
#endif

namespace {
typedef __nv_bfloat16 bf16;
constexpr bool LATENT = PBE_X_LATENT != 0;
constexpr int D = 128, E = 128, ROT = 64;       // key and value width; the latents' rotated part
constexpr int DK = LATENT ? D + ROT : D;        // width of a score's product
constexpr int QN = LATENT ? 1 : 2;              // terms of a query
constexpr int BM = 128, BN = 64;
constexpr int LIST_ROWS = BM / 2;               // packed rows of a tile of the masked attention's work list
constexpr int Q_BYTES = BM * DK * 2;            // one term
constexpr int K_BYTES = BN * DK * 2, V_BYTES = BN * E * 2;
constexpr int NK = 2;                           // key tiles in flight; one value tile
constexpr int NTHREADS = 224;
constexpr int TMEM_COLS = 256;
constexpr int S_COL = 0, O_COL = 128;           // S at columns 0 and 64 (then P: hi in 32 columns, lo in 32), O at 128
constexpr float LOG2E = 1.4426950408889634f;

struct Barriers {
  uint64_t k_full[NK], k_empty[NK], v_full, v_empty, s_full[2], p_full, o_ready, q_full;
  uint32_t tmem_base;
};
constexpr size_t TILE_BYTES = (size_t)QN * Q_BYTES + NK * K_BYTES + V_BYTES;
constexpr size_t SMEM_BYTES = TILE_BYTES + sizeof(Barriers) + 512;      // and what aligns the tiles
static_assert(2 * (SMEM_BYTES + 1024) <= 228 * 1024, "two blocks a multiprocessor");

struct LatentExtra {
  const bf16* q;             // [T, H * (128 + 64)]
  const int32_t* list;       // the requests whose keys are expanded, ascending; null: all of the step
  int num_tiles, R;          // their row tiles, their number
  const int32_t* positions;  // [T]
  const float* inv_freq;     // [rot_dims / 2] or null
  int rot_dims;
  float rot_scale;
  const float* sink;         // [H] or null
  const bf16* gate;          // [T, ldg] or null
  int ldg, gate_each;        // a value per output column, or one per head
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// c * tanh(s) with the argument given as e^(2 s) = 2^z (see masked_attention_mma.cu)
__device__ __forceinline__ float capped(float z, float c) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + ex2(z)));
  return fmaf(-2.0f * c, r, c);
}
// byte offset of element (row, col) in a [rows][64-wide blocks] bf16 tile with 128-byte swizzle
__device__ __forceinline__ uint32_t swz(int row, int col, int rows) {
  const int blk = col >> 6, cc = col & 63;
  return (uint32_t)(blk * rows * 128 + row * 128 + ((((cc >> 3) ^ (row & 7)) << 4) | ((cc & 7) << 1)));
}
__device__ __forceinline__ uint32_t pack2(float x, float y) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float low_of(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float high_of(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// The expanded matrix holds the keys that the rows of a list of the step's requests can see, request after request.
__device__ __forceinline__ int lowest_key(int seq_len, int q_len, int window) {
  return window > 0 ? max(0, seq_len - q_len - window + 1) : 0;
}
// By a warp, over the list's requests (null: all of the step): the request that row tile `index` belongs to (tiles: their
// rows in tiles of BM; -1: every request is passed), its first tile, and the expanded row of the first key of place `at`
// of the list (of that request if at < 0).
struct Located { int r, first_tile, key_base; };
__device__ Located locate(int index, int at, const int32_t* list, int R, const int32_t* q_len, const int32_t* seq_len, int window) {
  const int lane = threadIdx.x & 31;
  int tiles_before = 0, keys_before = 0;
  for (int i0 = 0; i0 < R; i0 += 32) {
    const int i = i0 + lane;
    const int r = i < R ? (list ? list[i] : i) : 0;
    const int n = i < R ? q_len[r] : 0;
    const int keys = i < R ? seq_len[r] - lowest_key(seq_len[r], n, window) : 0;
    const int tiles = (n + BM - 1) / BM;
    int t = tiles, k = keys;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int ut = __shfl_up_sync(0xffffffffu, t, o), uk = __shfl_up_sync(0xffffffffu, k, o);
      if (lane >= o) { t += ut; k += uk; }
    }
    const unsigned hit = __ballot_sync(0xffffffffu, at >= 0 ? i == at : (i < R && index >= 0 && index < tiles_before + t));
    if (hit) {
      const int from = __ffs(hit) - 1;
      return Located{__shfl_sync(0xffffffffu, r, from), tiles_before + __shfl_sync(0xffffffffu, t - tiles, from),
                     keys_before + __shfl_sync(0xffffffffu, k - keys, from)};
    }
    tiles_before += __shfl_sync(0xffffffffu, t, 31);
    keys_before += __shfl_sync(0xffffffffu, k, 31);
  }
  return Located{-1, tiles_before, keys_before};
}

// map_a: keys (pages), or the expanded matrix; map_b: values (pages), or the rotated parts
__global__ void __launch_bounds__(NTHREADS, 2)
attention_tc5_wide_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, AttnParams p,
                          MaskedExtra x, LatentExtra y, int* err) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  pdl_wait();
  if (base - smem_raw > 512) {                            // never: dynamic shared memory begins on such a boundary
    if (threadIdx.x == 0) atomicExch(err, 1);
    return;
  }
  unsigned char* Qs = base;                               // [QN][DK / 64][128 rows][128 B]
  unsigned char* Ks = Qs + QN * Q_BYTES;                  // [NK][DK / 64][64 keys][128 B]
  unsigned char* Vs = Ks + NK * K_BYTES;                  // [E / 64][64 keys][128 B]
  Barriers& bar = *reinterpret_cast<Barriers*>(Vs + V_BYTES);

  const int KV = p.num_kv_heads, H = p.num_heads, P = p.page_tokens;
  const int kvh = blockIdx.x % KV;
  int r, pr0, split = 0, nsplit = 1, G;
  int first_row = 0;                                      // the expanded row of the request's key 0
  if (LATENT) {
    // the last row tiles of a request have the most keys: they come first
    const int index = y.num_tiles - 1 - (int)(blockIdx.x / KV);
    const Located at = locate(index, -1, y.list, y.R, p.q_len, p.seq_len, p.window);
    r = at.r;
    if (r < 0) return;
    pr0 = (index - at.first_tile) * BM;
    first_row = at.key_base - lowest_key(p.seq_len[r], p.q_len[r], p.window);
    G = 1;
  } else {
    const int32_t* work = p.work + (size_t)(blockIdx.x / KV) * 4;
    r = work[0];
    // the list's tiles are half a block's: the block of an even tile takes the next one's rows too (a request's tiles
    // have the same key splits), that one's block is done
    if (r < 0 || (work[1] & 1)) return;
    pr0 = work[1] * LIST_ROWS;
    split = work[2];
    nsplit = work[3];
    G = H / KV;
  }
  const int qs = p.q_start[r], nq = p.q_len[r], sl = p.seq_len[r];
  const int n_packed = nq * G;
  const int rows_here = min(BM, n_packed - pr0);
  if (rows_here <= 0) return;
  const int row_lo = pr0 / G;
  const int row_hi = (pr0 + rows_here - 1) / G;
  const int pos0 = sl - nq;
  const int hi_key = pos0 + row_hi + 1;
  const int lo_key = first_visible(pos0 + row_lo, x.mask_kind, p.window);
  int k_begin = lo_key, k_end = hi_key;
  if (nsplit > 1) {
    const int lo_req = x.mask_kind ? max(0, pos0 - p.window + 1) : 0;
    const int s0 = lo_req / p.split_keys;
    k_begin = max(lo_key, (s0 + split) * p.split_keys);
    k_end = min(hi_key, (s0 + split + 1) * p.split_keys);
  }
  const int tile0 = (k_begin / BN) * BN;
  const int n_tiles = k_end > tile0 ? (k_end - tile0 + BN - 1) / BN : 0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < NK; ++i) {
      mbar_init(&bar.k_full[i], 1);
      mbar_init(&bar.k_empty[i], 1);
    }
    mbar_init(&bar.v_full, 1);
    mbar_init(&bar.v_empty, 1);
    for (int i = 0; i < 2; ++i) mbar_init(&bar.s_full[i], 1);
    mbar_init(&bar.p_full, 4);
    mbar_init(&bar.o_ready, 1);
    mbar_init(&bar.q_full, 4);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&bar.tmem_base)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = bar.tmem_base;

  // the query tile: one packed row per softmax thread, into the swizzled K-major layout
  if (warp >= 2 && warp < 6) {
    const int row = (warp - 2) * 32 + lane;
    const int pr = pr0 + row;
    const bool live = pr < n_packed;
    const int qrow = live ? pr / G : 0, hg = live ? pr - qrow * G : 0;
    if (LATENT) {
      const int t = qs + qrow;
      const bf16* src = y.q + ((size_t)t * H + kvh) * DK;
#pragma unroll
      for (int c = 0; c < D / 8; ++c)
        *reinterpret_cast<uint4*>(Qs + swz(row, c * 8, BM)) = live ? *reinterpret_cast<const uint4*>(src + c * 8) : make_uint4(0, 0, 0, 0);
      const float at = live ? (float)y.positions[t] : 0.f;
#pragma unroll
      for (int c = 0; c < ROT / 8; ++c) {
        const uint4 raw = live ? *reinterpret_cast<const uint4*>(src + D + c * 8) : make_uint4(0, 0, 0, 0);
        const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
        uint32_t o[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int pair = c * 4 + k;
          o[k] = w[k];
          if (live && 2 * pair + 1 < y.rot_dims) {        // pairs (2i, 2i + 1) of the first rot_dims values
            float sn, cs;
            sincosf(at * y.inv_freq[pair], &sn, &cs);
            sn *= y.rot_scale;
            cs *= y.rot_scale;
            const float u = low_of(w[k]), v = high_of(w[k]);
            o[k] = pack2(u * cs - v * sn, v * cs + u * sn);
          }
        }
        *reinterpret_cast<uint4*>(Qs + swz(row, D + c * 8, BM)) = make_uint4(o[0], o[1], o[2], o[3]);
      }
    } else {
      const float* src = (const float*)p.q + ((size_t)(qs + qrow) * H + kvh * G + hg) * D;
#pragma unroll 4
      for (int c = 0; c < D / 8; ++c) {
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
        if (live) {
          a = *reinterpret_cast<const float4*>(src + c * 8);
          b = *reinterpret_cast<const float4*>(src + c * 8 + 4);
        }
        const uint4 h = make_uint4(pack2(a.x, a.y), pack2(a.z, a.w), pack2(b.x, b.y), pack2(b.z, b.w));
        const uint4 l = make_uint4(pack2(a.x - low_of(h.x), a.y - high_of(h.x)), pack2(a.z - low_of(h.y), a.w - high_of(h.y)),
                                   pack2(b.x - low_of(h.z), b.y - high_of(h.z)), pack2(b.z - low_of(h.w), b.w - high_of(h.w)));
        *reinterpret_cast<uint4*>(Qs + swz(row, c * 8, BM)) = h;
        *reinterpret_cast<uint4*>(Qs + Q_BYTES + swz(row, c * 8, BM)) = l;
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // visible to the products' reads
    __syncwarp();
    if (lane == 0) mbar_arrive(&bar.q_full);
  }

  if (warp == 0 || warp == 6) {
    // ------------------------------------------------------------ TMA producers: keys (warp 0), values (warp 6)
    const bool keys = warp == 0;
    const int ring = keys ? NK : 1;
    uint64_t* full = keys ? bar.k_full : &bar.v_full;
    uint64_t* empty = keys ? bar.k_empty : &bar.v_empty;
    const int32_t* bt = LATENT ? nullptr : p.block_table + (size_t)r * p.bt_stride;
    const int last_blk = n_tiles > 0 && !LATENT ? (k_end - 1) / P : 0;
    const int box_rows = LATENT ? BN : min(P, BN);
    const int boxes = BN / box_rows;
    int go = 1;
    for (int j = 0; j < n_tiles; ++j) {
      const int st = j % ring;
      if (lane == 0) {
        go = mbar_wait(&empty[st], ((j / ring) & 1) ^ 1, err) ? 1 : 0;
        if (go) mbar_expect_tx(&full[st], keys ? K_BYTES : V_BYTES);
      }
      go = __shfl_sync(0xffffffffu, go, 0);
      if (!go) break;
      unsigned char* dst = keys ? Ks + (size_t)st * K_BYTES : Vs;
      const int ts = tile0 + j * BN;
      if (LATENT) {
        // keys that are masked may lie below the matrix' first row or behind its last: they read as zeros
        const int row = first_row + ts;
        if (lane < 2) tma_load_2d(dst + lane * BN * 128, &map_a, (keys ? 0 : H * D) + kvh * 128 + lane * 64, row, &full[st]);
        else if (lane == 2 && keys) tma_load_2d(dst + 2 * BN * 128, &map_b, 0, row, &full[st]);
      } else {
        for (int pg = lane; pg < boxes; pg += 32) {
          const int key0 = ts + pg * box_rows;
          const int blk = key0 / P;
          int page = blk <= last_blk ? bt[blk] : 0;        // beyond the range: any page, the keys are masked
          if (page < 0) page = 0;
          const int row = (page * KV + kvh) * P + (key0 - blk * P);
#pragma unroll
          for (int b = 0; b < 2; ++b)
            tma_load_2d(dst + b * BN * 128 + pg * box_rows * 128, keys ? &map_a : &map_b, b * 64, row, &full[st]);
        }
      }
      __syncwarp();
    }
    // the commits that release the last tiles arrive on this block's barriers: it stays until they have
    if (lane == 0) {
      bool ok = go != 0;
      for (int j = n_tiles > ring ? n_tiles - ring : 0; j < n_tiles && ok; ++j)
        ok = mbar_wait(&empty[j % ring], (j / ring) & 1, err);
    }
  } else if (warp == 1) {
    if (lane == 0 && n_tiles > 0) {
      // ------------------------------------------------------------ MMA issuer
      const uint32_t idesc_s = make_idesc(BM, BN);
      const uint32_t idesc_o = make_idesc(BM, E) | (1u << 16);             // B as it lies: MN-major
      const uint32_t q_addr = smem_u32(Qs);
      bool ok = true;
      auto issue_qk = [&](int j) {
        const int st = j & 1, kst = j % NK;
        ok = ok && mbar_wait(&bar.k_full[kst], (j / NK) & 1, err);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t k_addr = smem_u32(Ks + (size_t)kst * K_BYTES);
#pragma unroll
        for (int term = 0; term < QN; ++term)
#pragma unroll
          for (int ks = 0; ks < DK / 16; ++ks) {
            const uint32_t q_off = term * Q_BYTES + (ks >> 2) * (BM * 128) + (ks & 3) * 32;
            const uint32_t k_off = (ks >> 2) * (BN * 128) + (ks & 3) * 32;
            umma(tmem_base + S_COL + st * BN, make_desc(q_addr + q_off), make_desc(k_addr + k_off), idesc_s,
                 (term > 0 || ks > 0) ? 1u : 0u);
          }
        umma_commit(&bar.k_empty[kst]);                       // the key tile is free once its scores exist
        umma_commit(&bar.s_full[st]);
      };
      ok = ok && mbar_wait(&bar.q_full, 0, err);              // the query tile is in shared memory
      issue_qk(0);
      if (n_tiles > 1) issue_qk(1);
      for (int j = 0; j < n_tiles && ok; ++j) {
        const int st = j & 1;
        ok = ok && mbar_wait(&bar.v_full, j & 1, err);
        ok = ok && mbar_wait(&bar.p_full, j & 1, err);        // P_j written, O rescaled
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t v_addr = smem_u32(Vs);
#pragma unroll
        for (int term = 0; term < 2; ++term)
#pragma unroll
          for (int ks = 0; ks < BN / 16; ++ks)
            umma_ts(tmem_base + O_COL, tmem_base + S_COL + st * BN + term * 32 + ks * 8, desc_mn_major(v_addr + ks * 16 * 128, BN),
                    idesc_o, (j > 0 || term > 0 || ks > 0) ? 1u : 0u);
        umma_commit(&bar.v_empty);
        umma_commit(&bar.o_ready);
        if (j + 2 < n_tiles) issue_qk(j + 2);                 // over P_j's columns: the tensor pipe runs them in order
      }
    }
  } else {
    // ---------------------------------------------------------------- softmax, correction, epilogue
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;                   // TMEM lane == row of the tile
    const int pr = pr0 + row;
    const bool row_valid = pr < n_packed;
    const int qrow = row_valid ? pr / G : 0;
    const int head = kvh * G + (row_valid ? pr - qrow * G : 0);
    const int tok = qs + qrow;
    const int pos = row_valid ? pos0 + qrow : -1;
    const int lo = row_valid ? max(k_begin, first_visible(pos, x.mask_kind, p.window)) : 0;
    const int hi = min(pos, k_end - 1);                    // the last key this row sees
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const bool cap = x.softcap > 0.f;
    const float cap_scale = cap ? p.scale * (2.0f * LOG2E / x.softcap) : 0.f;
    const float mul = cap ? LOG2E : p.scale * LOG2E;       // what is held as scores, in units of log2
    // tiles whose every key is visible to every row of the block need no mask
    const int pos_min = pos0 + row_lo;
    const int lo_max = first_visible(pos0 + row_hi, x.mask_kind, p.window);
    float m_run = -INFINITY, l_run = 0.f;
    bool ok = true;
    for (int j = 0; j < n_tiles; ++j) {
      const int st = j & 1;
      const int ts = tile0 + j * BN;
      ok = ok && mbar_wait(&bar.s_full[st], (j >> 1) & 1, err);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      float s[BN];
#pragma unroll
      for (int c = 0; c < BN / 32; ++c) tmem_ld32_nowait(lane_addr + S_COL + st * BN + c * 32, &s[c * 32]);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (cap) {
#pragma unroll
        for (int i = 0; i < BN; ++i) s[i] = capped(s[i] * cap_scale, x.softcap);
      }
      const bool full_tile = ts >= k_begin && ts + BN <= k_end && ts + BN - 1 <= pos_min && ts >= lo_max;
      if (!full_tile) {
#pragma unroll
        for (int i = 0; i < BN; ++i) s[i] = ts + i >= lo && ts + i <= hi ? s[i] : -INFINITY;
      }
      float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
#pragma unroll
      for (int i = 0; i < BN; i += 4) {
        mx0 = fmaxf(mx0, s[i]);
        mx1 = fmaxf(mx1, s[i + 1]);
        mx2 = fmaxf(mx2, s[i + 2]);
        mx3 = fmaxf(mx3, s[i + 3]);
      }
      // the running maximum moves only when it has grown by more than 2^8: until then the old one keeps every
      // exponential within 256, and O needs no rescale
      float m_new = fmaxf(m_run, fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3)));
      if (m_run != -INFINITY && (m_new - m_run) * mul <= 8.0f) m_new = m_run;
      const float m_use = m_new == -INFINITY ? 0.f : m_new;
      const float alpha = ex2((m_run - m_use) * mul);      // 0 when nothing was visible before
      const float neg = -m_use * mul;
      float sum0 = 0.f, sum1 = 0.f, sum2 = 0.f, sum3 = 0.f;
      uint32_t w[BN / 2];
#pragma unroll
      for (int i = 0; i < BN; i += 4) {
        s[i] = ex2(fmaf(s[i], mul, neg));
        s[i + 1] = ex2(fmaf(s[i + 1], mul, neg));
        s[i + 2] = ex2(fmaf(s[i + 2], mul, neg));
        s[i + 3] = ex2(fmaf(s[i + 3], mul, neg));
        sum0 += s[i];
        sum1 += s[i + 1];
        sum2 += s[i + 2];
        sum3 += s[i + 3];
        w[i / 2] = pack2(s[i], s[i + 1]);
        w[i / 2 + 1] = pack2(s[i + 2], s[i + 3]);
      }
      l_run = l_run * alpha + ((sum0 + sum1) + (sum2 + sum3));
      // P over the scores it came from: the roundings, then what they left
      tmem_st32_nowait(lane_addr + S_COL + st * BN, &w[0]);
#pragma unroll
      for (int i = 0; i < BN / 2; ++i) w[i] = pack2(s[2 * i] - low_of(w[i]), s[2 * i + 1] - high_of(w[i]));
      tmem_st32_nowait(lane_addr + S_COL + st * BN + 32, &w[0]);
      // the previous tile's P V must be complete before O is rescaled
      if (j > 0) {
        ok = ok && mbar_wait(&bar.o_ready, (j - 1) & 1, err);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (__any_sync(0xffffffffu, m_new > m_run)) {      // rescale the rows of this warp
#pragma unroll 1
          for (int c = 0; c < E / 32; ++c) {
            float v[32];
            tmem_ld32(lane_addr + O_COL + c * 32, v);
            uint32_t u[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) u[i] = __float_as_uint(v[i] * alpha);
            tmem_st32_nowait(lane_addr + O_COL + c * 32, u);
          }
        }
      }
      m_run = m_new;
      // values of keys outside the range are zeroed (P is 0 there, but what lies there may be no number)
      if (ts < k_begin || ts + BN > k_end) {
        ok = ok && mbar_wait(&bar.v_full, j & 1, err);     // the tile has landed
        const int key = ts + row;                          // thread `row` owns key row `row` of the tile
        if (row < BN && (key < k_begin || key >= k_end)) {
#pragma unroll
          for (int b = 0; b < E / 64; ++b)
#pragma unroll
            for (int c = 0; c < 8; ++c)
              *reinterpret_cast<uint4*>(Vs + b * BN * 128 + row * 128 + c * 16) = make_uint4(0, 0, 0, 0);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.p_full);
    }
    pdl_launch_dependents();
    if (n_tiles > 0) {
      ok = ok && mbar_wait(&bar.o_ready, (n_tiles - 1) & 1, err);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    float m_nat = m_run == -INFINITY ? -INFINITY : m_run * (mul * 0.6931471805599453f);
    float l = l_run, rescale = 1.f;
    const float* sink = LATENT ? y.sink : x.sink;
    if (nsplit <= 1 && (LATENT ? sink != nullptr : x.has_sink != 0)) add_sink(m_nat, l, rescale, sink ? sink[head] : 0.f);
    const float inv = l > 0.f ? rescale / l : 0.f;
    const bf16* gate = nullptr;
    float head_gate = 1.f;
    if (row_valid && nsplit <= 1) {
      if (LATENT) {
        if (y.gate && y.gate_each) gate = y.gate + (size_t)tok * y.ldg + head * E;
        else if (y.gate) head_gate = sigmoidf_(__bfloat162float(y.gate[(size_t)tok * y.ldg + head]));
      } else if (x.gate) {
        gate = (const bf16*)x.gate + (size_t)tok * x.ldg + head * E;
      }
    }
    const bool gate16 = ((uintptr_t)gate & 15) == 0;
    // half the columns at a time, each with its partner half way across the head (turned outputs pair them)
#pragma unroll 1
    for (int c = 0; c < E / 64; ++c) {
      float v[2][32];
      __syncwarp();                                        // rows beyond the request left the turn before early
      if (n_tiles > 0) {                                   // block-uniform: every lane takes part in the loads
        tmem_ld32_nowait(lane_addr + O_COL + c * 32, v[0]);
        tmem_ld32_nowait(lane_addr + O_COL + E / 2 + c * 32, v[1]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) v[0][i] = v[1][i] = 0.f;
      }
      if (!row_valid) continue;
      if (nsplit <= 1) {
        if (!LATENT && x.turn) {
          const float2* cs = x.turn + (size_t)tok * (E / 2) + c * 32;
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float4 c2 = *reinterpret_cast<const float4*>(cs + i);
            turn_back(v[0][i], v[1][i], make_float2(c2.x, c2.y));
            turn_back(v[0][i + 1], v[1][i + 1], make_float2(c2.z, c2.w));
          }
        }
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int e0 = half * (E / 2) + c * 32;
          bf16* dst = (bf16*)p.out + ((size_t)tok * H + head) * E + e0;
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            float o[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) o[k] = v[half][i + k] * inv * head_gate;
            if (gate) {
              float g[8];
              if (gate16) {
                const uint4 raw = *reinterpret_cast<const uint4*>(gate + e0 + i);
                g[0] = low_of(raw.x); g[1] = high_of(raw.x); g[2] = low_of(raw.y); g[3] = high_of(raw.y);
                g[4] = low_of(raw.z); g[5] = high_of(raw.z); g[6] = low_of(raw.w); g[7] = high_of(raw.w);
              } else {
#pragma unroll
                for (int k = 0; k < 8; ++k) g[k] = __bfloat162float(gate[e0 + i + k]);
              }
#pragma unroll
              for (int k = 0; k < 8; ++k) o[k] *= sigmoidf_(g[k]);
            }
            *reinterpret_cast<uint4*>(dst + i) = make_uint4(pack2(o[0], o[1]), pack2(o[2], o[3]), pack2(o[4], o[5]), pack2(o[6], o[7]));
          }
        }
      } else {
        const size_t at = ((size_t)p.tok_split_row[tok] * H + head) * p.max_splits + split;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          float* dst = p.part_o + at * E + half * (E / 2) + c * 32;
#pragma unroll
          for (int i = 0; i < 32; i += 4)
            *reinterpret_cast<float4*>(dst + i) = make_float4(v[half][i], v[half][i + 1], v[half][i + 2], v[half][i + 3]);
        }
        if (c == 0) {
          p.part_ml[at * 2] = m_nat;
          p.part_ml[at * 2 + 1] = l_run;
        }
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// [rows, columns] row-major bfloat16 with rows `ld` elements apart, boxes of box_rows x 64, zeros outside
int map_rows(CUtensorMap* map, const void* at, long long rows, int columns, long long ld, int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return (int)cudaErrorNotSupported;
  cuuint64_t dims[2] = {(cuuint64_t)columns, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  const CUresult rc = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(at), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return rc == CUDA_SUCCESS ? 0 : (int)cudaErrorInvalidValue;
}

int launch_wide(const CUtensorMap& a, const CUtensorMap& b, const AttnParams& p, const MaskedExtra& x, const LatentExtra& y,
                long long blocks, int* err, cudaStream_t stream) {
  if (blocks > 0x7fffffffLL) return (int)cudaErrorInvalidValue;
  static OptIn opt_in;
  if (const cudaError_t e = opt_in(SMEM_BYTES, attention_tc5_wide_kernel)) return (int)e;
  launch_k(attention_tc5_wide_kernel, (int)blocks, NTHREADS, SMEM_BYTES, stream, a, b, p, x, y, err);
  return launch_status();
}
}  // namespace

#if !PBE_X_LATENT
// The masked attention over a work list of 64-row tiles (all its tiles); the caller merges key splits.
PBE_EXPORT int pbe_masked_attention_tc5(const AttnParams* params, int mask_kind, int has_sink, const float* sink,
                                        float softcap, const float2* turn, const void* gate, int ldg, int num_work, int* err,
                                        cudaStream_t stream) {
  if (num_work <= 0) return 0;
  AttnParams p = *params;
  const int P = p.page_tokens;
  if (p.num_heads % p.num_kv_heads != 0 || p.tile_rows != LIST_ROWS || p.split_keys % BN != 0 || P < 8 || P % 8 != 0 ||
      (BN % P != 0 && P % BN != 0) || mask_kind < 0 || mask_kind > 2 || (mask_kind != 0 && p.window < 1) || !(p.scale > 0.f))
    return (int)cudaErrorInvalidValue;
  if (((uintptr_t)p.q | (uintptr_t)turn | (uintptr_t)p.k_cache | (uintptr_t)p.v_cache | (uintptr_t)p.part_o | (uintptr_t)p.out) & 15)
    return (int)cudaErrorMisalignedAddress;
  CUtensorMap map_k, map_v;
  const long long rows = (long long)p.num_pages * p.num_kv_heads * P;
  const int box_rows = P < BN ? P : BN;
  int rc = map_rows(&map_k, p.k_cache, rows, D, D, box_rows);
  if (rc == 0) rc = map_rows(&map_v, p.v_cache, rows, E, E, box_rows);
  if (rc != 0) return rc;
  MaskedExtra x{nullptr, 0, mask_kind, has_sink, sink, softcap, turn, gate, ldg, D, E};
  return launch_wide(map_k, map_v, p, x, LatentExtra{}, (long long)num_work * p.num_kv_heads, err, stream);
}
#else
// The latent attention over expanded keys and values: kv [keys, 2 * H * 128] (K of all heads, then V of all heads),
// kr [keys, 64]; rows in tiles of 128 of one request.  Only the list's requests' rows of out are written.
PBE_EXPORT int pbe_latent_attention_tc5(const void* q, const void* kv, const void* kr, void* out, long long num_keys,
                                        int num_tiles, const int32_t* list, int R, const int32_t* q_start, const int32_t* q_len,
                                        const int32_t* seq_len, const int32_t* positions, const float* inv_freq, int rot_dims, float rot_scale,
                                        const float* sink, const void* gate, int ldg, int gate_each, int H, int window,
                                        float scale, int* err, cudaStream_t stream) {
  if (num_tiles <= 0) return 0;
  if (H < 1 || num_keys < 1 || num_keys > 0x7fffffffLL || R < 1 || !(scale > 0.f) || (rot_dims > 0 && inv_freq == nullptr) || rot_dims > ROT)
    return (int)cudaErrorInvalidValue;
  if (((uintptr_t)q | (uintptr_t)kv | (uintptr_t)kr | (uintptr_t)out) & 15) return (int)cudaErrorMisalignedAddress;
  CUtensorMap map_kv, map_kr;
  int rc = map_rows(&map_kv, kv, num_keys, 2 * H * D, 2LL * H * D, BN);
  if (rc == 0) rc = map_rows(&map_kr, kr, num_keys, ROT, ROT, BN);
  if (rc != 0) return rc;
  AttnParams p = {};
  p.out = out;
  p.q_start = q_start;
  p.q_len = q_len;
  p.seq_len = seq_len;
  p.num_heads = p.num_kv_heads = H;
  p.page_tokens = BN;
  p.window = window;
  p.scale = scale;
  MaskedExtra x = {};
  x.mask_kind = window > 0 ? 1 : 0;
  LatentExtra y{(const bf16*)q, list, num_tiles, R, positions, inv_freq, rot_dims, rot_scale, sink,
                (const bf16*)gate, ldg, gate_each};
  return launch_wide(map_kv, map_kr, p, x, y, (long long)num_tiles * H, err, stream);
}

// The latents and rotated parts of the keys that the list's requests' rows can see, gathered from the pages, request after
// request: c [keys, rank], kr [keys, 64].  grid.y: the place in the list; a warp a key, 16-byte pieces.
namespace {
__global__ void __launch_bounds__(256) gather_latents_kernel(const bf16* pages, const int32_t* block_table, int bt_stride,
                                                             int page_tokens, int rank, const int32_t* q_len,
                                                             const int32_t* seq_len, const int32_t* list, int R, int window,
                                                             bf16* c, bf16* kr) {
  pdl_launch_dependents();
  pdl_wait();
  const int r = list ? list[blockIdx.y] : (int)blockIdx.y, lane = threadIdx.x & 31;
  const int low = lowest_key(seq_len[r], q_len[r], window);
  const int key = low + blockIdx.x * 8 + (threadIdx.x >> 5);
  if (key >= seq_len[r]) return;
  const size_t row = (size_t)(locate(-1, (int)blockIdx.y, list, R, q_len, seq_len, window).key_base + key - low);
  const int page = block_table[(size_t)r * bt_stride + key / page_tokens];
  const int width = rank + ROT;
  const bf16* src = pages + ((size_t)max(page, 0) * page_tokens + key % page_tokens) * width;
  for (int i = lane * 8; i < width; i += 256) {
    const uint4 v = page >= 0 ? *reinterpret_cast<const uint4*>(src + i) : make_uint4(0, 0, 0, 0);
    if (i < rank) *reinterpret_cast<uint4*>(c + row * rank + i) = v;
    else *reinterpret_cast<uint4*>(kr + row * ROT + (i - rank)) = v;
  }
}
}  // namespace

PBE_EXPORT int pbe_gather_latents(const void* pages, const int32_t* block_table, int bt_stride, int page_tokens, int rank,
                                  const int32_t* q_len, const int32_t* seq_len, const int32_t* list, int R, int window,
                                  int most_keys, void* c, void* kr, cudaStream_t stream) {
  if (R <= 0 || most_keys <= 0) return 0;
  if (rank % 8 || (((uintptr_t)pages | (uintptr_t)c | (uintptr_t)kr) & 15) || R > 65535) return (int)cudaErrorInvalidValue;
  launch_k(gather_latents_kernel, dim3((most_keys + 7) / 8, R), 256, 0, stream, (const bf16*)pages, block_table, bt_stride,
           page_tokens, rank, q_len, seq_len, list, R, window, (bf16*)c, (bf16*)kr);
  return launch_status();
}
#endif
