// Softmax attention over a window of tokens and pooled blocks of older ones, with the heads' probabilities mixed by
// a matrix after the softmax, for prompt portions in bfloat16: the products of pooled_attention.cu on the tensor cores
// (mma.sync m16n8k16, bfloat16 operands, float32 sums).
//
// A block takes sixteen rows of a request and all heads, a warp a head.  Pass 1 walks the key tiles and keeps every
// (row, head)'s running maximum and sum in registers.  Pass 2 walks them again: the probabilities, normalised, go to
// shared memory as three bfloat16 terms, which hold their 24 bits (queries, keys and values are bfloat16 and exact),
// every warp mixes the heads of one row, W = M P, as a product over the sixteen heads (M as three terms too: the six
// products that count), and head h's warp adds a tile's W V, three products summed from zero, to its 16 x E outputs,
// which stay in registers (the tensor cores cut off what does not fit a sum, so the outputs are not left to them).  Scores are computed twice because the mixture needs normalised probabilities of all heads
// before any value is weighted; keeping the heads' values apart until the end would take G times the value products.
//
// What bounds it: the shared-memory pipe (every head's warp reads its key/value head's tile: 3 x 8 KB a warp and
// tile) and three block barriers a tile with one block a multiprocessor (202 KB).  A key tile travels while the
// tile before it is mixed, a value tile while its scores are made, so one buffer of each is enough.
// A 2,048-token prompt, sixteen heads of 128 over four key/value heads, window 1,024, blocks of 64: 4,336 us in
// float32 multiply-adds, 292 us here.  Two terms took 243; where the mixture nearly cancels they were further off 64 bits
// than the multiply-adds (5e-4 of the bfloat16 result's own rounding), three are as close to seven digits.
#include "common.cuh"
#include "mma_sync.cuh"
#include "pdl.cuh"

using namespace pbe;
using namespace pbe::mma_sync;

#if !defined(PBE_PM_D) || !defined(PBE_PM_E)
#error "PBE_PM_D (key width) and PBE_PM_E (value width) must be defined"
#endif

namespace {
constexpr int D = PBE_PM_D, E = PBE_PM_E;
static_assert(D % 16 == 0 && E % 16 == 0 && D <= 128 && E <= 128, "head widths are multiples of 16 up to 128");
constexpr int BM = 16, HEADS = 16;         // rows of a block, most heads
constexpr int KSTR = D + 8, VSTR = E + 8;  // padded rows: eight neighbouring ones start in different banks

struct PmParams {
  const bf16* q;            // [T, H * D]
  const bf16* k_tok;        // [page][G][page_tokens][D]
  const bf16* v_tok;
  const bf16* k_pool;
  const bf16* v_pool;
  bf16* out;                // [T, H * E]
  const float* talk;        // [H, H] or null
  const int32_t* tiles;     // [n, 3]: request, first batch row, rows
  const int32_t* q_start;
  const int32_t* q_len;
  const int32_t* seq_len;
  const int32_t* bt_tok;
  const int32_t* bt_pool;
  int bt_tok_stride, bt_pool_stride;
  int H, G, page_tokens, window, pool;
  float scale_log2;         // scale * log2(e): scores in units of the exponential's base
  // when not null: tiles are of 128 rows, another kernel's but for those with a flag set ([n, flags_a_tile])
  const int32_t* flags = nullptr;
  int flags_a_tile = 0;
};

// The probabilities' buffer: [head][row][key], rows and heads padded so that eight rows of a head and eight heads of
// a row both start in different banks
template <int BN> __host__ __device__ constexpr int p_row() { return BN + 8; }
template <int BN> __host__ __device__ constexpr int p_head() { return BM * p_row<BN>() + 8; }
template <int BN> __host__ __device__ constexpr size_t pm_smem(int H, int G) {
  return 2 * ((size_t)H * BM * KSTR + (size_t)G * BN * (2 * (KSTR > VSTR ? KSTR : VSTR)) + TERMS * (size_t)HEADS * p_head<BN>());
}

template <int N>
struct Width { static constexpr int value = N; };
using KeyWidth = Width<D>;
using ValueWidth = Width<E>;

template <int BN>
__global__ void __launch_bounds__(32 * HEADS, 1) pooled_attention_mma_kernel(PmParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int ring[4][BN];
  constexpr int TILE = KSTR > VSTR ? KSTR : VSTR;
  constexpr int PR = p_row<BN>(), PH = p_head<BN>();
  const int H = p.H, G = p.G, PT = p.page_tokens;
  bf16* Qs = reinterpret_cast<bf16*>(smem_raw);            // [H][BM][KSTR]
  bf16* const buf0 = Qs + H * BM * KSTR;                   // [G][BN][KSTR]
  bf16* const buf1 = buf0 + G * BN * TILE;                 // [G][BN][VSTR]; pass 1: the other key buffer
  bf16* Ps = buf1 + G * BN * TILE;                         // [TERMS][HEADS] of PH
  const int tid = threadIdx.x, NT = blockDim.x, warp = tid >> 5, lane = tid & 31;
  const int g8 = lane >> 2, q2 = (lane & 3) * 2;
  const int lrow = (lane & 7) + ((lane >> 3) & 1) * 8, lcol = (lane >> 4) * 8;     // ldmatrix: A operands, and B transposed
  const int krow = (lane & 7) + (lane >> 4) * 8, kcol = ((lane >> 3) & 1) * 8;     // B operands as they lie
  pdl_launch_dependents();
  pdl_wait();
  const int32_t* tile = p.tiles + (size_t)(p.flags ? blockIdx.x / 8 : blockIdx.x) * 3;
  const int r = tile[0], skip = p.flags ? (int)blockIdx.x % 8 * BM : 0, row0 = tile[1] + skip, rows = p.flags ? min(BM, tile[2] - skip) : tile[2];
  if (p.flags) {
    int set = 0;
    for (int i = threadIdx.x; i < p.flags_a_tile; i += blockDim.x) set |= p.flags[(size_t)(blockIdx.x / 8) * p.flags_a_tile + i];
    if (!__syncthreads_or(set) || rows <= 0) return;
  }
  const int pos0 = p.seq_len[r] - p.q_len[r] + (row0 - p.q_start[r]);     // position of the tile's first row
  const int pos_last = pos0 + rows - 1;
  const int W = p.window, PL = p.pool;
  // pooled blocks the last row sees, tokens from the first row's window on
  const int nb_max = (PL > 0 && pos_last - W + 1 > 0) ? (pos_last - W + 1) / PL : 0;
  const int tok_lo = max(0, pos0 - W + 1);
  const int pool_tiles = (nb_max + BN - 1) / BN;
  const int tiles = pool_tiles + (pos_last - tok_lo + BN) / BN;
  const int32_t* bt_tok = p.bt_tok + (size_t)r * p.bt_tok_stride;
  const int32_t* bt_pool = p.bt_pool ? p.bt_pool + (size_t)r * p.bt_pool_stride : nullptr;

  // Where tile kt's key `key` lies in the pages, in rows of a key/value head (-1: there is no such key).  The page is
  // looked up two tiles ahead and kept in a ring, so that a tile's copies do not wait for it.
  auto look_up = [&](int kt, int key) {
    const bool pooled = kt < pool_tiles;
    const int idx = (pooled ? kt * BN : tok_lo + (kt - pool_tiles) * BN) + key;
    if (kt >= tiles || idx >= (pooled ? nb_max : pos_last + 1)) return -1;
    const int page = pooled ? bt_pool[idx / PT] : bt_tok[idx / PT];
    return page >= 0 ? page * G * PT + idx % PT : -1;
  };
  auto start_ring = [&]() {
    for (int i = tid; i < 2 * BN; i += NT) ring[i / BN][i % BN] = look_up(i / BN, i % BN);
  };
  // a tile's keys or values of all key/value heads; keys that do not exist become zeros
  auto load = [&](int kt, bf16* dst, const bf16* tok, const bf16* pool, auto width) {
    constexpr int WD = decltype(width)::value, PIECES = WD / 8, STR = WD + 8;
    const bf16* src = kt < pool_tiles ? pool : tok;
    for (int i = tid; i < BN * PIECES; i += NT) {
      const int key = i / PIECES, piece = i - key * PIECES;
      const int at = ring[kt & 3][key];
      const bool live = at >= 0;
      const bf16* s = src + (live ? (size_t)at * WD + piece * 8 : 0);
      for (int g = 0; g < G; ++g)
        cp16(dst + (g * BN + key) * STR + piece * 8, s + (live ? (size_t)g * PT * WD : 0), live);
    }
  };

  start_ring();
  __syncthreads();
  load(0, buf0, p.k_tok, p.k_pool, KeyWidth());
  cp_commit();
  for (int i = tid; i < H * BM * (D / 8); i += NT) {
    const int piece = i % (D / 8), rh = i / (D / 8);
    const int row = rh % BM, h = rh / BM;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (row < rows) v = *reinterpret_cast<const uint4*>(p.q + (size_t)(row0 + row) * H * D + h * D + piece * 8);
    *reinterpret_cast<uint4*>(Qs + (h * BM + row) * KSTR + piece * 8) = v;
  }
  // heads that do not exist take part in the mixture as zeros
  for (int i = tid; i < (HEADS - H) * PH; i += NT)
#pragma unroll
    for (int t = 0; t < TERMS; ++t) Ps[(t * HEADS + H) * PH + i] = __float2bfloat16_rn(0.f);
  unsigned mix[TERMS][4] = {};                             // M as the A operand
  if (p.talk) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int h = g8 + (i & 1) * 8, g = q2 + (i >> 1) * 8;
      const float x = h < H && g < H ? p.talk[h * H + g] : 0.f, y = h < H && g + 1 < H ? p.talk[h * H + g + 1] : 0.f;
      unsigned terms[TERMS];
      split3(x, y, terms);
#pragma unroll
      for (int t = 0; t < TERMS; ++t) mix[t][i] = terms[t];
    }
  }
  const bf16* Qh = Qs + warp * BM * KSTR;
  const int kv = warp / (H / G);                           // this warp's head is its number
  // scores of the warp's head against a tile, in units of log2; -inf where a row does not see a key
  float s[BN / 8][4];
  auto score = [&](int kt, const bf16* keys, auto query) {
#pragma unroll
    for (int j = 0; j < BN / 8; ++j) s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
    const bf16* Kh = keys + kv * BN * KSTR;
#pragma unroll
    for (int kk = 0; kk < D; kk += 16) {
      unsigned a[4];
      query(a, kk);
#pragma unroll
      for (int j = 0; j < BN / 16; ++j) {
        unsigned b[4];
        ldm4(b, Kh + (j * 16 + krow) * KSTR + kk + kcol);
        mma(s[2 * j], a, b[0], b[1]);
        mma(s[2 * j + 1], a, b[2], b[3]);
      }
    }
    const bool pooled = kt < pool_tiles;
    const int first = pooled ? kt * BN : tok_lo + (kt - pool_tiles) * BN;
    // does every row see every key of the tile?
    const bool whole = rows == BM && (pooled ? first + BN <= nb_max && (first + BN - 1) * PL + PL - 1 <= pos0 - W
                                             : first + BN - 1 <= pos0 && first > pos_last - W);
#pragma unroll
    for (int j = 0; j < BN / 8; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float x = s[j][c] * p.scale_log2;
        if (!whole) {
          const int row = g8 + (c >> 1) * 8, idx = first + j * 8 + q2 + (c & 1), pos = pos0 + row;
          const bool see = row < rows && (pooled ? idx < nb_max && idx * PL + PL - 1 <= pos - W : idx <= pos && idx > pos - W);
          if (!see) x = -INFINITY;
        }
        s[j][c] = x;
      }
  };

  // ---- pass 1: every (row, head)'s maximum and sum; a thread keeps those of its own columns
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
  {
  __syncthreads();                                         // the queries are in shared memory
  unsigned qf[D / 16][4];
#pragma unroll
  for (int kk = 0; kk < D; kk += 16) ldm4(qf[kk / 16], Qh + lrow * KSTR + kk + lcol);
#pragma unroll 1
  for (int kt = 0; kt < tiles; ++kt) {
    cp_wait<0>();
    __syncthreads();                                       // tile kt has landed, tile kt - 1's buffer is free
    if (kt + 1 < tiles) load(kt + 1, (kt & 1) ? buf0 : buf1, p.k_tok, p.k_pool, KeyWidth());
    cp_commit();
    const int ahead = tid < BN ? look_up(kt + 2, tid) : 0;
    score(kt, (kt & 1) ? buf1 : buf0, [&](unsigned (&a)[4], int kk) {
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = qf[kk / 16][i];
    });
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      float top = m[hh];
#pragma unroll
      for (int j = 0; j < BN / 8; ++j) top = fmaxf(top, fmaxf(s[j][2 * hh], s[j][2 * hh + 1]));
      if (top != -INFINITY) {
        float sum = l[hh] * exp2f(m[hh] - top);
#pragma unroll
        for (int j = 0; j < BN / 8; ++j) sum += exp2f(s[j][2 * hh] - top) + exp2f(s[j][2 * hh + 1] - top);
        l[hh] = sum;
        m[hh] = top;
      }
    }
    if (tid < BN) ring[(kt + 2) & 3][tid] = ahead;
  }
  }
  __syncthreads();
  start_ring();
  __syncthreads();
  load(0, buf0, p.k_tok, p.k_pool, KeyWidth());
  cp_commit();
  load(0, buf1, p.v_tok, p.v_pool, ValueWidth());
  cp_commit();
  float inv[2];
#pragma unroll
  for (int hh = 0; hh < 2; ++hh) {
    float top = fmaxf(m[hh], __shfl_xor_sync(0xffffffffu, m[hh], 1));
    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
    float sum = m[hh] == -INFINITY ? 0.f : l[hh] * exp2f(m[hh] - top);
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    inv[hh] = sum > 0.f ? 1.0f / sum : 0.f;
    if (sum != sum) inv[hh] = sum;                         // not a number: the row's result is none
    m[hh] = top == -INFINITY ? 0.f : top;                  // a row beyond the tile's: all its scores are -inf
  }

  // ---- pass 2: probabilities, mixture, values
  float o[E / 8][4];
#pragma unroll
  for (int j = 0; j < E / 8; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
  cp_wait<1>();
  __syncthreads();
#pragma unroll 1
  for (int kt = 0; kt < tiles; ++kt) {
    // the keys of tile kt have landed, its values are on their way
    const int ahead = tid < BN ? look_up(kt + 2, tid) : 0;
    score(kt, buf0, [&](unsigned (&a)[4], int kk) { ldm4(a, Qh + lrow * KSTR + kk + lcol); });
#pragma unroll
    for (int j = 0; j < BN / 8; ++j)
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        unsigned terms[TERMS];
        split3(exp2f(s[j][2 * hh] - m[hh]) * inv[hh], exp2f(s[j][2 * hh + 1] - m[hh]) * inv[hh], terms);
        const int at = warp * PH + (g8 + hh * 8) * PR + j * 8 + q2;
#pragma unroll
        for (int t = 0; t < TERMS; ++t) *reinterpret_cast<unsigned*>(Ps + t * HEADS * PH + at) = terms[t];
      }
    if (tid < BN) ring[(kt + 2) & 3][tid] = ahead;
    __syncthreads();                                       // all heads' probabilities; the key buffer is free
    if (kt + 1 < tiles) load(kt + 1, buf0, p.k_tok, p.k_pool, KeyWidth());
    cp_commit();
    if (p.talk) {
      for (int row = warp; row < BM; row += NT / 32) {     // in place: nobody else touches this row now
        unsigned b[BN / 16][TERMS][4];
#pragma unroll
        for (int j = 0; j < BN / 16; ++j)                  // B operands: k the heads, n sixteen keys
#pragma unroll
          for (int t = 0; t < TERMS; ++t) ldm4t(b[j][t], Ps + (t * HEADS + lrow) * PH + row * PR + j * 16 + lcol);
        __syncwarp();
#pragma unroll
        for (int j = 0; j < BN / 8; ++j) {
          float w[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int sum = TERMS - 1; sum >= 0; --sum)       // the small products first
#pragma unroll
            for (int t = 0; t <= sum; ++t) mma(w, mix[t], b[j / 2][sum - t][(j & 1) * 2], b[j / 2][sum - t][(j & 1) * 2 + 1]);
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            unsigned terms[TERMS];
            split3(w[2 * hh], w[2 * hh + 1], terms);
            const int at = (g8 + hh * 8) * PH + row * PR + j * 8 + q2;
#pragma unroll
            for (int t = 0; t < TERMS; ++t) *reinterpret_cast<unsigned*>(Ps + t * HEADS * PH + at) = terms[t];
          }
        }
      }
    }
    cp_wait<1>();
    __syncthreads();                                       // mixed; the values of tile kt have landed
    const bf16* Vh = buf1 + kv * BN * VSTR;
    unsigned a[BN / 16][TERMS][4];
#pragma unroll
    for (int kk = 0; kk < BN / 16; ++kk)
#pragma unroll
      for (int t = 0; t < TERMS; ++t) ldm4(a[kk][t], Ps + (t * HEADS + warp) * PH + lrow * PR + kk * 16 + lcol);
#pragma unroll
    for (int j = 0; j < E / 16; ++j) {
      float y[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
      for (int kk = 0; kk < BN / 16; ++kk) {
        unsigned b[4];
        ldm4t(b, Vh + (kk * 16 + lrow) * VSTR + j * 16 + lcol);
#pragma unroll
        for (int t = TERMS - 1; t >= 0; --t) {
          mma(y[0], a[kk][t], b[0], b[1]);
          mma(y[1], a[kk][t], b[2], b[3]);
        }
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        o[2 * j][c] += y[0][c];
        o[2 * j + 1][c] += y[1][c];
      }
    }
    cp_wait<0>();
    __syncthreads();                                       // the keys of the next tile; the value buffer is free
    if (kt + 1 < tiles) load(kt + 1, buf1, p.v_tok, p.v_pool, ValueWidth());
    cp_commit();
  }
  cp_wait<0>();
#pragma unroll
  for (int hh = 0; hh < 2; ++hh) {
    const int row = g8 + hh * 8;
    if (row >= rows) continue;
    bf16* dst = p.out + (size_t)(row0 + row) * H * E + warp * E + q2;
#pragma unroll
    for (int j = 0; j < E / 8; ++j)
      *reinterpret_cast<__nv_bfloat162*>(dst + j * 8) = __floats2bfloat162_rn(o[j][2 * hh], o[j][2 * hh + 1]);
  }
}

constexpr size_t MOST_SMEM = 226 * 1024;       // and the ring of page places

template <int BN>
int launch_pm(const PmParams& p, int n_tiles, cudaStream_t stream) {
  const size_t smem = pm_smem<BN>(p.H, p.G);
  cudaFuncSetAttribute(pooled_attention_mma_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  launch_k(pooled_attention_mma_kernel<BN>, n_tiles, 32 * p.H, smem, stream, p);
  return launch_status();
}
}  // namespace

// Keys of a tile for that many heads and key/value heads (0: not this kernel).
PBE_EXPORT int pbe_pooled_attention_mma_keys(int H, int G) {
  if (H < 1 || H > HEADS || G < 1 || H % G) return 0;
  return pm_smem<32>(H, G) <= MOST_SMEM ? 32 : pm_smem<16>(H, G) <= MOST_SMEM ? 16 : 0;
}

PBE_EXPORT int pbe_pooled_attention_mma(const void* q, const void* k_tok, const void* v_tok, const void* k_pool,
                                        const void* v_pool, void* out, const float* talk, const int32_t* tiles,
                                        int n_tiles, const int32_t* q_start, const int32_t* q_len,
                                        const int32_t* seq_len, const int32_t* bt_tok, int bt_tok_stride,
                                        const int32_t* bt_pool, int bt_pool_stride, int H, int G, int page_tokens,
                                        int window, int pool, float scale, cudaStream_t stream) {
  if (n_tiles <= 0) return 0;
  const uintptr_t at = (uintptr_t)q | (uintptr_t)k_tok | (uintptr_t)v_tok | (uintptr_t)k_pool | (uintptr_t)v_pool | (uintptr_t)out;
  const int keys = pbe_pooled_attention_mma_keys(H, G);
  if (keys == 0 || (at & 15) || page_tokens < 1 || window < 1 || (pool > 0 && (!k_pool || !v_pool || !bt_pool)))
    return (int)cudaErrorInvalidValue;
  PmParams p{(const bf16*)q, (const bf16*)k_tok, (const bf16*)v_tok, (const bf16*)k_pool, (const bf16*)v_pool, (bf16*)out,
             talk, tiles, q_start, q_len, seq_len, bt_tok, bt_pool, bt_tok_stride, bt_pool_stride, H, G, page_tokens,
             window, pool, scale * 1.4426950408889634f};
  return keys == 32 ? launch_pm<32>(p, n_tiles, stream) : launch_pm<16>(p, n_tiles, stream);
}
