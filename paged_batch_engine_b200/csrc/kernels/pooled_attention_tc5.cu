// Window and pooled-block attention with mixed heads (pooled_attention_mma.cu: the same rows, keys and mixture) on the fifth-
// generation tensor cores, for heads of 128 x 128 in bfloat16.
//
// With P_g head g's probabilities and V_c a key/value head's values, head h's output is the sum over g of M_hg (P_g V_c(h)): the
// mixture is taken behind the values, of U_gc = P_g V_c in float32, so that neither normalised probabilities of all heads nor
// the heads' probabilities side by side are needed before any value is weighted.  That costs a product with the values
// of every key/value head, G times as many as without a mixture, which the tensor cores have room for, and U's way through memory.
//
// Two kernels:
//  * A block takes 128 rows of a request, one head and one or two key/value heads (whose V share the scores and the softmax), and
//    walks over tiles of 64 keys, pooled blocks first: S = Q K^T by tcgen05.mma into tensor memory, the weights as three bfloat16
//    terms (24 bits; queries, keys and values are bfloat16 and exact) back to one of two buffers in tensor memory as the A
//    operand, O = P V per key/value head.  Sixteen warps are softmax and outputs, four threads a row: sixteen keys and a quarter of
//    the outputs each, which stay in registers: the tensor cores cut off what does not fit a sum, so a tile's products are summed
//    from zero, the small terms first, and added with one rounding.  Left to the tensor cores for two, four or all tiles they
//    are 3.2e-7, 5.3e-7 or 1.7e-6 off 64 bits where this is 2.0e-7 and mma.sync's mixture 2.3e-7.  Warp 16 issues
//    the products, warp 17 the TMA copies (128-byte swizzle, no multicast), three key tiles and two value tiles in flight.
//    A row's outputs leave through shared memory: 16 bytes of 32 rows at a time took 7 to 11 us a block.
//  * The mixture: a block a row, a thread four columns of a key/value head, U read once.
// What bounds the first is the softmax warps' chain, 4,500 clocks a key tile, of which reads of tensor memory, 350 clocks each
// beside the products, are 1,900 (the products are 2,048); 96 registers a thread leave room for sixteen columns at a time.
// 2,048 tokens, sixteen heads over four key/value heads, window 1,024, blocks of 64: 291 us on mma.sync, 151 here and
// some 20 for the mixture (a layer 352 -> 229); over two key/value heads a layer 330 -> 166, 8,192 tokens over four 1,378 -> 965.
//
// A value that is not finite reaches, as a product with a weight of zero, rows of its tile that do not see it.  Blocks that find one in
// a tile which not all of their rows see whole set a flag; the rows of flagged tiles are made by pooled_attention_mma.cu, launched behind.
//
// Every mbarrier wait is bounded; one that runs out sets *err and the block runs to its end.
#define PBE_PM_D 128
#define PBE_PM_E 128
#include "pooled_attention_mma.cu"
#include "float_terms.cuh"
#include "opt_in.cuh"
#include "tcgen05.cuh"

using namespace pbe::tc5;

namespace {
namespace pooled_tc5 {
constexpr int ROWS = 128, BN = 64, WIDTH = 128;
constexpr int SOFT_WARPS = 16, MMA_WARP = 16, TMA_WARP = 17, NTHREADS = 32 * 18, SOFT_THREADS = 32 * SOFT_WARPS;
constexpr int Q_BYTES = ROWS * WIDTH * 2, K_BYTES = BN * WIDTH * 2;     // a value tile of one key/value head is as large
constexpr int NK = 3, NV = 2;
constexpr int S_COL = 0, P_COL = BN, P_COLS = TERMS * BN / 2, O_COL = 256, TMEM_COLS = 512;     // two buffers of weights
static_assert(P_COL + 2 * P_COLS <= O_COL, "tensor memory");
constexpr int U_STRIDE = 4;                      // floats between the rows of outputs in shared memory, past a row: eight rows in different banks

struct Barriers {
  uint64_t k_full[NK], k_empty[NK], v_full[NV], v_empty[NV], s_full, s_empty, p_full, o_ready;
  uint32_t tmem_base;
  int odd;
  float row_max[2][4][ROWS];                     // by tile parity and part
};
template <int NKV>
constexpr size_t smem_bytes() { return Q_BYTES + NK * K_BYTES + NV * NKV * K_BYTES + sizeof(Barriers) + 1024; }

struct TcParams {
  PmParams m;
  float* U;                 // [rows of the launch, H, G, WIDTH]
  int first_tile, num_tiles, first_row;
  int32_t* flags;           // [tiles, H * (G / NKV)]
  int* err;
};

__device__ __forceinline__ void tmem_st8_nowait(uint32_t taddr, const uint32_t (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
__device__ __forceinline__ unsigned long long pair_of(float x, float y) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
  return d;
}
__device__ __forceinline__ float2 floats_of(unsigned long long p) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(p));
  return f;
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// byte offset of the 16-byte piece `piece` of a row in a [64-wide blocks][rows] bf16 tile with 128-byte swizzle
__device__ __forceinline__ uint32_t swz(int row, int piece, int rows) {
  return (uint32_t)((piece >> 3) * rows * 128 + row * 128 + (((piece & 7) ^ (row & 7)) << 4));
}

template <int NKV>
__global__ void __launch_bounds__(NTHREADS, 1)
pooled_attention_tc5_kernel(const __grid_constant__ CUtensorMap map_kt, const __grid_constant__ CUtensorMap map_vt,
                            const __grid_constant__ CUtensorMap map_kp, const __grid_constant__ CUtensorMap map_vp, TcParams x) {
  constexpr int COLS = NKV * WIDTH / 4;                    // of the outputs, a thread
  const PmParams& p = x.m;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned char* Qs = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* Ks = Qs + Q_BYTES;                        // [NK][2][64 keys][128 B]
  unsigned char* Vs = Ks + NK * K_BYTES;                   // [NV][NKV][2][64 keys][128 B]
  Barriers& bar = *reinterpret_cast<Barriers*>(Vs + NV * NKV * K_BYTES);
  pdl_wait();

  const int H = p.H, G = p.G, PT = p.page_tokens, groups = G / NKV;
  // the last row tiles see the most keys: they come first
  const int tile = x.first_tile + x.num_tiles - 1 - (int)blockIdx.x / (H * groups), sub = (int)blockIdx.x % (H * groups);
  const int head = sub / groups, kv0 = sub % groups * NKV, own_kv = head / (H / G);
  const int r = p.tiles[tile * 3], row0 = p.tiles[tile * 3 + 1], rows = p.tiles[tile * 3 + 2];
  const int pos0 = p.seq_len[r] - p.q_len[r] + (row0 - p.q_start[r]), pos_last = pos0 + rows - 1;
  const int W = p.window, PL = p.pool;
  auto blocks_seen = [&](int pos) { return PL > 0 && pos - W + 1 > 0 ? (pos - W + 1) / PL : 0; };
  const int nb_max = blocks_seen(pos_last), nb_min = blocks_seen(pos0);
  const int tok_lo = max(0, pos0 - W + 1), tok0 = tok_lo / BN * BN;
  const int pool_tiles = (nb_max + BN - 1) / BN, n_tiles = pool_tiles + (pos_last - tok0) / BN + 1;
  const int32_t* bt_tok = p.bt_tok + (size_t)r * p.bt_tok_stride;
  const int32_t* bt_pool = p.bt_pool ? p.bt_pool + (size_t)r * p.bt_pool_stride : nullptr;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (int i = 0; i < NK; ++i) {
      mbar_init(&bar.k_full[i], 1);
      mbar_init(&bar.k_empty[i], 1);
    }
    for (int i = 0; i < NV; ++i) {
      mbar_init(&bar.v_full[i], 1);
      mbar_init(&bar.v_empty[i], 1);
    }
    mbar_init(&bar.s_full, 1);
    mbar_init(&bar.s_empty, SOFT_WARPS);
    mbar_init(&bar.p_full, SOFT_WARPS);
    mbar_init(&bar.o_ready, 1);
    bar.odd = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&bar.tmem_base)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  for (int i = tid; i < ROWS * (WIDTH / 8); i += NTHREADS) {
    const int row = i / (WIDTH / 8), piece = i % (WIDTH / 8);
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (row < rows) v = *reinterpret_cast<const uint4*>(p.q + ((size_t)(row0 + row) * H + head) * WIDTH + piece * 8);
    *reinterpret_cast<uint4*>(Qs + swz(row, piece, ROWS)) = v;
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = bar.tmem_base;

  auto v_tile = [&](int j, int kv) { return Vs + ((j % NV) * NKV + kv) * K_BYTES; };
  bool ok = true;

  if (warp == TMA_WARP) {
    // ---------------------------------------------------------------- keys and values, in boxes of a page or less, one a lane
    const int box = min(PT, BN), boxes = BN / box;
    auto place_of = [&](int j) {                           // the row of the pages, of this lane's box of tile j
      if (j >= n_tiles || lane >= boxes) return 0;
      const bool pooled = j < pool_tiles;
      const int key = (pooled ? j * BN : tok0 + (j - pool_tiles) * BN) + lane * box;
      // beyond the range any page does: its keys are masked, its values zeroed
      const int page = pooled ? (key < nb_max ? bt_pool[key / PT] : 0) : (key <= pos_last ? bt_tok[key / PT] : 0);
      return max(page, 0) * G * PT + key % PT;
    };
    auto copy = [&](int j, int place, bool keys) {
      const int ring = keys ? NK : NV, st = j % ring;
      int go = 1;
      if (lane == 0) {
        go = mbar_wait(keys ? &bar.k_empty[st] : &bar.v_empty[st], ((j / ring) & 1) ^ 1, x.err) ? 1 : 0;
        if (go) mbar_expect_tx(keys ? &bar.k_full[st] : &bar.v_full[st], keys ? K_BYTES : NKV * K_BYTES);
      }
      ok = ok && __shfl_sync(0xffffffffu, go, 0);
      if (ok && lane < boxes) {
        const bool pooled = j < pool_tiles;
#pragma unroll
        for (int kv = 0; kv < (keys ? 1 : NKV); ++kv)
#pragma unroll
          for (int b = 0; b < 2; ++b)
            tma_load_2d((keys ? Ks + st * K_BYTES : v_tile(j, kv)) + b * BN * 128 + lane * box * 128,
                        keys ? (pooled ? &map_kp : &map_kt) : (pooled ? &map_vp : &map_vt), b * 64,
                        place + (keys ? own_kv : kv0 + kv) * PT, keys ? &bar.k_full[st] : &bar.v_full[st]);
      }
      __syncwarp();
    };
    // the values of tile j behind the keys of tile j + 1; the pages are looked up two tiles ahead
    int now = place_of(0), next = place_of(1);
    copy(0, now, true);
    for (int j = 0; j < n_tiles && ok; ++j) {
      const int ahead = place_of(j + 2);
      if (j + 1 < n_tiles) copy(j + 1, next, true);
      copy(j, now, false);
      now = next;
      next = ahead;
    }
    // the commits that release the last tiles arrive on this block's barriers: it stays until they have
    if (lane == 0) {
      for (int j = max(0, n_tiles - NK); j < n_tiles && ok; ++j) ok = mbar_wait(&bar.k_empty[j % NK], (j / NK) & 1, x.err);
      for (int j = max(0, n_tiles - NV); j < n_tiles && ok; ++j) ok = mbar_wait(&bar.v_empty[j % NV], (j / NV) & 1, x.err);
    }
  } else if (warp == MMA_WARP) {
    // ---------------------------------------------------------------- products
    if (lane == 0) {
      const uint32_t idesc_s = make_idesc(ROWS, BN), idesc_o = make_idesc(ROWS, WIDTH) | (1u << 16);     // B as it lies: MN-major
      auto scores = [&](int j) {
        if (j >= n_tiles) return;
        ok = ok && mbar_wait(&bar.k_full[j % NK], (j / NK) & 1, x.err) && mbar_wait(&bar.s_empty, (j & 1) ^ 1, x.err);
        if (!ok) return;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t q_addr = smem_u32(Qs), k_addr = smem_u32(Ks + (j % NK) * K_BYTES);
#pragma unroll
        for (int ks = 0; ks < WIDTH / 16; ++ks)
          umma(tmem_base + S_COL, make_desc(q_addr + (ks >> 2) * (ROWS * 128) + (ks & 3) * 32),
               make_desc(k_addr + (ks >> 2) * (BN * 128) + (ks & 3) * 32), idesc_s, ks > 0 ? 1u : 0u);
        umma_commit(&bar.k_empty[j % NK]);
        umma_commit(&bar.s_full);
      };
      scores(0);
      for (int j = 0; j < n_tiles && ok; ++j) {
        scores(j + 1);
        ok = ok && mbar_wait(&bar.v_full[j % NV], (j / NV) & 1, x.err) && mbar_wait(&bar.p_full, j & 1, x.err);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int kv = 0; kv < NKV; ++kv) {
          const uint32_t v_addr = smem_u32(v_tile(j, kv));
#pragma unroll
          for (int t = TERMS - 1; t >= 0; --t)             // the small terms first
#pragma unroll
            for (int ks = 0; ks < BN / 16; ++ks)
              umma_ts(tmem_base + O_COL + kv * WIDTH, tmem_base + P_COL + (j & 1) * P_COLS + t * (BN / 2) + ks * 8, desc_mn_major(v_addr + ks * 16 * 128, BN),
                      idesc_o, t < TERMS - 1 || ks > 0 ? 1u : 0u);
        }
        umma_commit(&bar.v_empty[j % NV]);
        umma_commit(&bar.o_ready);
      }
    }
  } else {
    // ---------------------------------------------------------------- softmax and outputs
    const int quarter = warp & 3, part = warp >> 2;
    const int row = quarter * 32 + lane;                     // tensor-memory lane == row of the tile
    const bool live = row < rows;
    const int pos = live ? pos0 + row : -1;
    const int my_blocks = live ? blocks_seen(pos) : 0;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    float m_run = -INFINITY, l_run = 0.f, alpha = 0.f;
    unsigned long long acc[COLS / 2];                      // pairs of columns
#pragma unroll
    for (int i = 0; i < COLS / 2; ++i) acc[i] = 0ull;
    auto add_outputs = [&]() {                               // of the tile before
      const unsigned long long by = pair_of(alpha, alpha);
#pragma unroll
      for (int c = 0; c < COLS / 16; ++c) {
        float v[16];
        tmem_ld16(lane_addr + O_COL + part * COLS + c * 16, v);
#pragma unroll
        for (int i = 0; i < 16; i += 2)
          asm("fma.rn.f32x2 %0, %0, %1, %2;" : "+l"(acc[(c * 16 + i) / 2]) : "l"(by), "l"(pair_of(v[i], v[i + 1])));
      }
    };
#pragma unroll 1
    for (int j = 0; j < n_tiles; ++j) {
      const bool pooled = j < pool_tiles;
      const int first = pooled ? j * BN : tok0 + (j - pool_tiles) * BN;
      ok = ok && mbar_wait(&bar.s_full, j & 1, x.err);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      float s[16];
      tmem_ld16(lane_addr + S_COL + part * 16, s);
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.s_empty);
      // does every row of the tile see every key of it?
      const bool whole = rows == ROWS && (pooled ? first + BN <= nb_min : first + BN - 1 <= pos0 && first > pos_last - W);
      if (!whole) {
        const int from = (pooled ? 0 : max(0, pos - W + 1)) - (first + part * 16), to = (pooled ? my_blocks - 1 : pos) - (first + part * 16);
#pragma unroll
        for (int i = 0; i < 16; ++i) s[i] = i < from || i > to ? -INFINITY : s[i];
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < 16; ++i) mx[i & 3] = fmaxf(mx[i & 3], s[i]);
      float(&row_max)[4][ROWS] = bar.row_max[j & 1];
      row_max[part][row] = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * p.scale_log2;
      asm volatile("bar.sync %0, 128;" ::"r"(1 + quarter) : "memory");       // the four warps of these rows
      const float m_new = fmaxf(m_run, fmaxf(fmaxf(row_max[0][row], row_max[1][row]), fmaxf(row_max[2][row], row_max[3][row])));
      const float m_use = m_new == -INFINITY ? 0.f : m_new;
      const float next_alpha = ex2(m_run - m_use);         // 0 when nothing was visible before
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        s[i] = ex2(fmaf(s[i], p.scale_log2, -m_use));
        sum[i & 3] += s[i];
      }
      l_run = fmaf(l_run, next_alpha, (sum[0] + sum[1]) + (sum[2] + sum[3]));
      m_run = m_new;
      if (!whole) {                                          // values of keys out of the range are zeroed, odd ones reported
        ok = ok && mbar_wait(&bar.v_full[j % NV], (j / NV) & 1, x.err);
        const int lo = pooled ? 0 : tok_lo - first, hi = (pooled ? nb_max - 1 : pos_last) - first;
        uint32_t largest = 0;                              // exponents of all ones are the largest
        for (int i = tid; i < NKV * BN * (WIDTH / 8); i += SOFT_THREADS) {
          const int key = i / (WIDTH / 8) % BN;
          uint4* at = reinterpret_cast<uint4*>(v_tile(j, i / (BN * (WIDTH / 8))) + swz(key, i % (WIDTH / 8), BN));
          if (key < lo || key > hi) {
            *at = make_uint4(0u, 0u, 0u, 0u);
          } else {
            if (head > 0) continue;                        // all heads have the same values
            const uint4 raw = *at;
            largest = __vmaxu2(__vmaxu2(largest, raw.x & 0x7fff7fffu), raw.y & 0x7fff7fffu);
            largest = __vmaxu2(__vmaxu2(largest, raw.z & 0x7fff7fffu), raw.w & 0x7fff7fffu);
          }
        }
        if ((largest & 0xffffu) >= 0x7f80u || (largest >> 16) >= 0x7f80u) bar.odd = 1;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      }
      // the weights of two tiles before have been read: their outputs were waited for
#pragma unroll
      for (int k = 0; k < TERMS; ++k) {
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) w[i] = next_term(s[2 * i], s[2 * i + 1]);
        tmem_st8_nowait(lane_addr + P_COL + (j & 1) * P_COLS + k * (BN / 2) + part * 8, w);
      }
      if (j > 0) {
        ok = ok && mbar_wait(&bar.o_ready, (j - 1) & 1, x.err);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        add_outputs();
      }
      alpha = next_alpha;
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.p_full);
    }
    pdl_launch_dependents();
    ok = ok && mbar_wait(&bar.o_ready, (n_tiles - 1) & 1, x.err);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    add_outputs();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    float(&sums)[4][ROWS] = bar.row_max[n_tiles & 1];        // this parity's maxima have been read
    sums[part][row] = l_run;
    asm volatile("bar.sync %0, 128;" ::"r"(1 + quarter) : "memory");
    const float l = (sums[0][row] + sums[1][row]) + (sums[2][row] + sums[3][row]);
    float inv = l > 0.f ? 1.0f / l : 0.f;
    if (l != l) inv = l;                                     // not a number: the row's result is none
    // through shared memory, whose tiles have been read, so that a row's outputs leave together
    constexpr int STRIDE = NKV * WIDTH + U_STRIDE;
    static_assert(sizeof(float) * ROWS * STRIDE <= Q_BYTES + NK * K_BYTES + NV * NKV * K_BYTES, "shared memory");
    float* rows_out = reinterpret_cast<float*>(Qs);
#pragma unroll
    for (int i = 0; i < COLS; i += 4) {
      const float2 a = floats_of(acc[i / 2]), b = floats_of(acc[i / 2 + 1]);
      *reinterpret_cast<float4*>(rows_out + row * STRIDE + part * COLS + i) = make_float4(a.x * inv, a.y * inv, b.x * inv, b.y * inv);
    }
    asm volatile("bar.sync 5, %0;" ::"n"(SOFT_THREADS) : "memory");
    for (int i = tid; i < rows * (NKV * WIDTH / 4); i += SOFT_THREADS) {
      const int at = i / (NKV * WIDTH / 4), col = i % (NKV * WIDTH / 4) * 4;
      *reinterpret_cast<float4*>(x.U + (((size_t)(row0 + at - x.first_row) * H + head) * G + kv0) * WIDTH + col) =
          *reinterpret_cast<const float4*>(rows_out + at * STRIDE + col);
    }
  }
  __syncthreads();
  if (tid == 0) x.flags[(size_t)tile * H * groups + sub] = bar.odd;
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// out[t, h] = sum over g of talk[h, g] U[t, g, h's key/value head]; a block a row, a thread four columns of a key/value head
__global__ void __launch_bounds__(256) mix_heads_kernel(const float* U, const float* talk, bf16* out, int first_row, int H, int G) {
  extern __shared__ float M[];                             // [H, H]
  pdl_launch_dependents();
  pdl_wait();
  for (int i = threadIdx.x; i < H * H; i += blockDim.x) M[i] = talk[i];
  __syncthreads();
  const int per = H / G;
  const float4* row = reinterpret_cast<const float4*>(U + (size_t)blockIdx.x * H * G * WIDTH);
  for (int i = threadIdx.x; i < G * (WIDTH / 4); i += blockDim.x) {
    const int kv = i / (WIDTH / 4), col = i % (WIDTH / 4);
    for (int h0 = kv * per; h0 < (kv + 1) * per; h0 += 4) {
      float4 o[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) o[k] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
      for (int g = 0; g < H; ++g) {
        const float4 u = row[g * G * (WIDTH / 4) + i];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float m = h0 + k < (kv + 1) * per ? M[(h0 + k) * H + g] : 0.f;
          o[k].x = fmaf(m, u.x, o[k].x);
          o[k].y = fmaf(m, u.y, o[k].y);
          o[k].z = fmaf(m, u.z, o[k].z);
          o[k].w = fmaf(m, u.w, o[k].w);
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (h0 + k < (kv + 1) * per) {
          const __nv_bfloat162 a = __floats2bfloat162_rn(o[k].x, o[k].y), b = __floats2bfloat162_rn(o[k].z, o[k].w);
          *reinterpret_cast<uint2*>(out + ((size_t)(first_row + blockIdx.x) * H + h0 + k) * WIDTH + col * 4) =
              make_uint2(*reinterpret_cast<const unsigned*>(&a), *reinterpret_cast<const unsigned*>(&b));
        }
    }
  }
}

int map_pages(CUtensorMap* map, const void* at, long long rows, int page_tokens) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return (int)cudaErrorNotSupported;
  cuuint64_t dims[2] = {(cuuint64_t)WIDTH, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)WIDTH * 2};
  cuuint32_t box[2] = {64, (cuuint32_t)(page_tokens < BN ? page_tokens : BN)};
  cuuint32_t estr[2] = {1, 1};
  const CUresult rc = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(at), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return rc == CUDA_SUCCESS ? 0 : (int)cudaErrorInvalidValue;
}

template <int NKV>
int launch_tc5(const CUtensorMap (&maps)[4], const TcParams& x, cudaStream_t stream) {
  static OptIn opt_in;
  if (const cudaError_t e = opt_in(smem_bytes<NKV>(), pooled_attention_tc5_kernel<NKV>)) return (int)e;
  launch_k(pooled_attention_tc5_kernel<NKV>, x.num_tiles * x.m.H * (x.m.G / NKV), NTHREADS, smem_bytes<NKV>(), stream, maps[0], maps[1],
           maps[2], maps[3], x);
  return launch_status();
}
}  // namespace pooled_tc5
}  // namespace

// Key/value heads a block takes (0: not this kernel): heads of 128 x 128 in at most sixteen heads, pages that divide a key tile of 64
// or are a multiple of it.
PBE_EXPORT int pbe_pooled_attention_tc5_kv(int H, int G, int page_tokens) {
  if (pbe_pooled_attention_mma_keys(H, G) == 0 || page_tokens < 8 || page_tokens % 8 ||
      (pooled_tc5::BN % page_tokens && page_tokens % pooled_tc5::BN))
    return 0;
  return G % 2 == 0 ? 2 : 1;
}

// tiles: [n, 3] request, first batch row, rows (at most 128), in the order of the rows; row_of: [n + 1] (on the host) the tiles' first batch rows and the
// step's rows.  U: float32 [most_rows, H, G, 128] (128 rows at least): as many goes as the rows take.  flags: [n, H, G / pbe_pooled_attention_tc5_kv].
PBE_EXPORT int pbe_pooled_attention_tc5(const void* q, const void* k_tok, const void* v_tok, const void* k_pool, const void* v_pool,
                                        void* out, const float* talk, const int32_t* tiles, int n_tiles, const int32_t* row_of,
                                        const int32_t* q_start, const int32_t* q_len, const int32_t* seq_len, const int32_t* bt_tok,
                                        int bt_tok_stride, const int32_t* bt_pool, int bt_pool_stride, int H, int G, int page_tokens,
                                        int tok_pages, int pool_pages, int window, int pool, float scale, float* U, int most_rows,
                                        int32_t* flags, int* err, cudaStream_t stream) {
  using namespace pooled_tc5;
  if (n_tiles <= 0) return 0;
  const uintptr_t at = (uintptr_t)q | (uintptr_t)k_tok | (uintptr_t)v_tok | (uintptr_t)k_pool | (uintptr_t)v_pool | (uintptr_t)out | (uintptr_t)U;
  const int nkv = pbe_pooled_attention_tc5_kv(H, G, page_tokens);
  if (nkv == 0 || talk == nullptr || !(scale > 0.f) || (at & 15) || window < 1 || most_rows < ROWS || (pool > 0 && (!k_pool || !v_pool || !bt_pool)))
    return (int)cudaErrorInvalidValue;
  CUtensorMap maps[4];
  int rc = map_pages(&maps[0], k_tok, (long long)tok_pages * G * page_tokens, page_tokens);
  if (rc == 0) rc = map_pages(&maps[1], v_tok, (long long)tok_pages * G * page_tokens, page_tokens);
  if (rc == 0) rc = map_pages(&maps[2], pool > 0 ? k_pool : k_tok, (long long)(pool > 0 ? pool_pages : tok_pages) * G * page_tokens, page_tokens);
  if (rc == 0) rc = map_pages(&maps[3], pool > 0 ? v_pool : v_tok, (long long)(pool > 0 ? pool_pages : tok_pages) * G * page_tokens, page_tokens);
  if (rc != 0) return rc;
  PmParams m{(const bf16*)q, (const bf16*)k_tok, (const bf16*)v_tok, (const bf16*)k_pool, (const bf16*)v_pool, (bf16*)out,
             talk, tiles, q_start, q_len, seq_len, bt_tok, bt_pool, bt_tok_stride, bt_pool_stride, H, G, page_tokens,
             window, pool, scale * 1.4426950408889634f};
  for (int t0 = 0; t0 < n_tiles && rc == 0;) {
    int t1 = t0 + 1;
    while (t1 < n_tiles && row_of[t1 + 1] - row_of[t0] <= most_rows) ++t1;
    const TcParams x{m, U, t0, t1 - t0, row_of[t0], flags, err};
    rc = nkv == 2 ? launch_tc5<2>(maps, x, stream) : launch_tc5<1>(maps, x, stream);
    if (rc == 0) {
      launch_k(mix_heads_kernel, row_of[t1] - row_of[t0], 128, H * H * sizeof(float), stream, (const float*)U, talk, (bf16*)out, row_of[t0], H, G);
      rc = launch_status();
    }
    t0 = t1;
  }
  if (rc != 0) return rc;
  m.flags = flags;
  m.flags_a_tile = H * (G / nkv);
  return pbe_pooled_attention_mma_keys(H, G) == 32 ? launch_pm<32>(m, n_tiles * (ROWS / BM), stream) : launch_pm<16>(m, n_tiles * (ROWS / BM), stream);
}
