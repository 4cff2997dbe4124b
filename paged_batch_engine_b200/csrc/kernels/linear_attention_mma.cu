// The recurrence of linear_attention.cu over prompt portions in bfloat16 on the tensor cores (mma.sync m16n8k16,
// bfloat16 operands, float32 sums):
//   S_t = a_{t,h} S_{t-1} + k_t (s_{t,h} v_t)^T,   o_t = S_t^T q_t + skip_h v_t        (S: [D, E] float32)
// in chunks of 64 tokens.  With c_i the sum of log2 a from the chunk's start to token i, S the state at its start:
//   o_i = 2^c_i S^T q_i + sum_{j<=i} (q_i . k_j) 2^(c_i - c_j) s_j v_j + skip v_i
//   S  <- 2^c_last S + sum_j k_j (2^(c_last - c_j) s_j v_j)^T
// q, k and v are bfloat16 and exact in the products; what is float32 (the state as it is read, the weights of the
// second sum, the weighted k of the third) enters them as three bfloat16 terms, which hold all of its 24 bits, and the
// state itself stays in float32: products are summed from zero, four or twelve of them, and added with one rounding.  Sums of
// logarithms and their differences are taken in double (a decay of zero counts as 2^-400), so a weight keeps float32's
// accuracy however strong the decays before it are.
//
// A product multiplies the zero weight of a later token with that token's values too, so values that are not finite would
// reach back to the tokens before theirs: a chunk that has some takes the products of a row tile with its own tokens one
// by one.
//
// One block per (work item or request, head), four warps: a warp makes sixteen rows of o and keeps D / 4 rows of the
// state in registers; o's weights pass from score accumulators to operands in registers.  Two blocks a multiprocessor
// (99 KB at 128 x 64) fill each other's barriers and copies.  Work items cut long portions as in
// linear_attention.cu: a pass without outputs leaves each item's own contribution and decay product.
// 2,048 tokens, 64 heads of 128 x 64 over 8 groups (both passes): 144 us against 823 of the recurrence token by token.  Two
// terms a factor, the weighted v in shared memory, took 104, but outputs and state were 10 to 30 times further off 64 bits
// than the recurrence's (1 to 3e-7); now they are 0.6 to 1.2 times.
#include "common.cuh"
#include "opt_in.cuh"
#include "mma_sync.cuh"
#include "pdl.cuh"

using namespace pbe;
using namespace pbe::mma_sync;

namespace {
constexpr int L = 64;                     // tokens of a chunk
constexpr int THREADS = 128;
constexpr int RUN = 4;                    // products a sum is left to the tensor cores for, which cut off what does not fit it
constexpr double LOG2_ZERO = -400.0;      // of a decay that has underflowed: 2^-400 is 0 in float32

struct SsdParams {
  const bf16* q;            // element (row 0, head 0, 0) inside the projection
  const bf16* k;
  const bf16* v;
  int ld;
  float* out;               // [T, H * E]; null: the items' own contributions only
  float* state;             // [slots, H, D, E]
  const float* decay;       // [H] or null
  const int32_t* q_start;
  const int32_t* q_len;
  const int32_t* slots;
  const int32_t* items;     // [n, 4] or null, as in linear_attention.cu
  float* scratch;
  int H;
  float k_scale;
  const float* tok_decay;   // [T, H] or null
  const float* tok_scale;   // [T, H] or null
  const float* skip;        // [H] or null
  int kq_share;
  float* chunk_decay;       // [entries, H] or null
};

template <int D, int E>
constexpr size_t ssd_smem() {
  return 2 * (2 * (size_t)L * (D + 8) + (size_t)L * (E + 8) + TERMS * (size_t)D * (E + 8));
}

template <int D, int E>
__global__ void __launch_bounds__(THREADS, 2) linear_attention_mma_kernel(SsdParams p) {
  constexpr int QSTR = D + 8, VSTR = E + 8;            // padded rows: eight neighbouring ones start in different banks
  constexpr int MT = D / 64;                           // sixteen-row tiles of the state a warp keeps
  static_assert(D % 64 == 0 && E % 16 == 0, "tiles");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  bf16* Qs = reinterpret_cast<bf16*>(smem_raw);        // [L][QSTR]
  bf16* Ks = Qs + L * QSTR;
  bf16* Vs = Ks + L * QSTR;                            // [L][VSTR]
  bf16* Ss = Vs + L * VSTR;                            // [TERMS][D][VSTR] the terms of the state at the chunk's start
  __shared__ float cs_hi[L], cs_lo[L];                 // the sums of logarithms, as two floats
  __shared__ float factor[L], into[L], from[L];        // s_j; its weight in the new state; 2^c_i
  __shared__ double half_total, total;
  __shared__ float keep_all;                           // 2^total

  const int h = blockIdx.y;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g8 = lane >> 2, q2 = (lane & 3) * 2;
  const int lrow = (lane & 7) + ((lane >> 3) & 1) * 8, lcol = (lane >> 4) * 8;
  const int krow = (lane & 7) + (lane >> 4) * 8, kcol = ((lane >> 3) & 1) * 8;
  int n, t0, src, dst;
  if (p.items) {
    const int32_t* it = p.items + (size_t)blockIdx.x * 4;
    t0 = it[0]; n = it[1]; src = it[2]; dst = it[3];
  } else {
    n = p.q_len[blockIdx.x];
    t0 = p.q_start[blockIdx.x];
    src = dst = n > 0 ? p.slots[blockIdx.x] : -1;
  }
  if (n <= 0) return;
  auto place = [&](int at) -> float* {
    if (at == -1) return nullptr;
    return (at >= 0 ? p.state + (size_t)at * p.H * (D * E) : p.scratch + (size_t)(-(at + 2)) * p.H * (D * E)) +
           (size_t)h * (D * E);
  };
  const float* st_in = place(src);
  float S[MT][E / 8][4];                               // rows warp * D / 4 + 16 m + g8 (+ 8), columns 8 j + q2 (+ 1)
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int j = 0; j < E / 8; ++j)
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        float2 x = make_float2(0.f, 0.f);
        if (st_in) x = *reinterpret_cast<const float2*>(st_in + (size_t)(warp * (D / 4) + m * 16 + g8 + hh * 8) * E + j * 8 + q2);
        S[m][j][2 * hh] = x.x;
        S[m][j][2 * hh + 1] = x.y;
      }
  const bool outputs = p.out != nullptr;
  const float skip = p.skip ? p.skip[h] : 0.f;
  const float lam = p.decay ? p.decay[h] : 1.f;
  const bf16* qp = p.q + (size_t)(h / p.kq_share) * D;
  const bf16* kp = p.k + (size_t)(h / p.kq_share) * D;
  const bf16* vp = p.v + (size_t)h * E;
  double log_all = 0.0;                                // of the whole item's decays

#pragma unroll 1
  for (int c0 = 0; c0 < n; c0 += L) {
    const int left = min(L, n - c0);
    __syncthreads();                                   // the chunk before is computed
    for (int i = tid; i < L * (D / 8); i += THREADS) {
      const int row = i / (D / 8), piece = (i - row * (D / 8)) * 8;
      const bool live = row < left;
      const size_t at = live ? (size_t)(t0 + c0 + row) * p.ld + piece : 0;
      if (outputs) cp16(Qs + row * QSTR + piece, qp + at, live);
      cp16(Ks + row * QSTR + piece, kp + at, live);
    }
    for (int i = tid; i < L * (E / 8); i += THREADS) {
      const int row = i / (E / 8), piece = (i - row * (E / 8)) * 8;
      const bool live = row < left;
      cp16(Vs + row * VSTR + piece, vp + (live ? (size_t)(t0 + c0 + row) * p.ld + piece : 0), live);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    double c = 0.0;                                    // thread i < L: the sum of logarithms up to token i
    if (tid < L) {
      float s = 0.f;
      if (tid < left) {
        const size_t th = (size_t)(t0 + c0 + tid) * p.H + h;
        const float a = p.tok_decay ? p.tok_decay[th] : lam;
        s = (p.tok_scale ? p.tok_scale[th] : 1.f) * p.k_scale;
        c = a == 0.f ? LOG2_ZERO : log2((double)a);
        c = c < LOG2_ZERO ? LOG2_ZERO : c;
      }
      factor[tid] = s;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double up = __shfl_up_sync(0xffffffffu, c, o);
        if (lane >= o) c += up;
      }
      if (tid == 31) half_total = c;
    }
    if (outputs) {
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int j = 0; j < E / 8; ++j)
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            unsigned t[TERMS];
            split3(S[m][j][2 * hh], S[m][j][2 * hh + 1], t);
            const int at = (warp * (D / 4) + m * 16 + g8 + hh * 8) * VSTR + j * 8 + q2;
#pragma unroll
            for (int i = 0; i < TERMS; ++i) *reinterpret_cast<unsigned*>(Ss + i * D * VSTR + at) = t[i];
          }
    }
    __syncthreads();
    if (tid < L) {
      if (tid >= 32) c += half_total;
      if (tid == L - 1) {
        total = c;
        keep_all = (float)exp2(c);
      }
      cs_hi[tid] = (float)c;
      cs_lo[tid] = (float)(c - (double)(float)c);
      from[tid] = (float)exp2(c);
    }
    __syncthreads();
    if (tid < L) into[tid] = factor[tid] * (float)exp2(total - c);
    const float keep = keep_all;
    log_all += total;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    bool odd = false;                                  // values that are not finite, among those this thread fetched
    for (int i = tid; i < L * (E / 8); i += THREADS) {
      const int row = i / (E / 8);
      const uint4 raw = *reinterpret_cast<const uint4*>(Vs + row * VSTR + (i - row * (E / 8)) * 8);
      const unsigned x[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) odd = odd || (x[k] & 0x7f80u) == 0x7f80u || (x[k] & 0x7f800000u) == 0x7f800000u;
    }
    odd = __syncthreads_or(odd) != 0;
    if (outputs && warp * 16 < left) {
      const int r0 = warp * 16 + g8;                   // this thread's rows: r0 and r0 + 8
      auto queries = [&](unsigned (&q)[RUN][4], int k0) {
#pragma unroll
        for (int k = 0; k < RUN; ++k) ldm4(q[k], Qs + (warp * 16 + lrow) * QSTR + (k0 + k) * 16 + lcol);
      };
      float o[E / 8][4];
#pragma unroll
      for (int j = 0; j < E / 8; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
#pragma unroll 1
      for (int i = TERMS - 1; i >= 0; --i)             // the small terms' sums first
#pragma unroll 1
        for (int k0 = 0; k0 < D / 16; k0 += RUN) {
          unsigned q[RUN][4];
          queries(q, k0);
#pragma unroll
          for (int j = 0; j < E / 16; ++j) {
            float y[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
            for (int k = 0; k < RUN; ++k) {
              unsigned b[4];
              ldm4t(b, Ss + i * D * VSTR + ((k0 + k) * 16 + lrow) * VSTR + j * 16 + lcol);
              mma(y[0], q[k], b[0], b[1]);
              mma(y[1], q[k], b[2], b[3]);
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              o[2 * j][c] += y[0][c];
              o[2 * j + 1][c] += y[1][c];
            }
          }
        }
      const float f0 = from[r0], f1 = from[r0 + 8];
#pragma unroll
      for (int j = 0; j < E / 8; ++j) {
        o[j][0] *= f0; o[j][1] *= f0;
        o[j][2] *= f1; o[j][3] *= f1;
      }
      const float hi0 = cs_hi[r0], lo0 = cs_lo[r0], hi1 = cs_hi[r0 + 8], lo1 = cs_lo[r0 + 8];
#pragma unroll 1
      for (int jt = 0; jt <= warp; ++jt) {             // sixteen tokens j at a time, up to the rows' own
        float g[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int k0 = 0; k0 < D / 16; k0 += RUN) {
          unsigned q[RUN][4];
          queries(q, k0);
          float y[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
          for (int k = 0; k < RUN; ++k) {
            unsigned b[4];
            ldm4(b, Ks + (jt * 16 + krow) * QSTR + (k0 + k) * 16 + kcol);
            mma(y[0], q[k], b[0], b[1]);
            mma(y[1], q[k], b[2], b[3]);
          }
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            g[0][c] += y[0][c];
            g[1][c] += y[1][c];
          }
        }
        unsigned w[TERMS][4];
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const int j = jt * 16 + t * 8 + q2;
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const float chi = cs_hi[j + x], clo = cs_lo[j + x], s = factor[j + x];
            g[t][x] = j + x <= r0 ? g[t][x] * (s * exp2f((hi0 - chi) + (lo0 - clo))) : 0.f;
            g[t][2 + x] = j + x <= r0 + 8 ? g[t][2 + x] * (s * exp2f((hi1 - chi) + (lo1 - clo))) : 0.f;
          }
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            unsigned terms[TERMS];
            split3(g[t][2 * hh], g[t][2 * hh + 1], terms);
#pragma unroll
            for (int i = 0; i < TERMS; ++i) w[i][2 * t + hh] = terms[i];
          }
        }
        if (odd && jt == warp) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {               // token j's weights lie in the quad's lane (j % 8) / 2
            const int from_lane = (lane & ~3) | ((j & 7) >> 1);
            const float w0 = __shfl_sync(0xffffffffu, g[j >> 3][j & 1], from_lane);
            const float w1 = __shfl_sync(0xffffffffu, g[j >> 3][2 + (j & 1)], from_lane);
#pragma unroll
            for (int c = 0; c < E / 8; ++c) {
              const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(Vs + (jt * 16 + j) * VSTR + c * 8 + q2));
              if (j <= g8) {
                o[c][0] = fmaf(w0, x.x, o[c][0]);
                o[c][1] = fmaf(w0, x.y, o[c][1]);
              }
              if (j <= g8 + 8) {
                o[c][2] = fmaf(w1, x.x, o[c][2]);
                o[c][3] = fmaf(w1, x.y, o[c][3]);
              }
            }
          }
          break;
        }
#pragma unroll
        for (int j = 0; j < E / 16; ++j) {
          unsigned b[4];
          ldm4t(b, Vs + (jt * 16 + lrow) * VSTR + j * 16 + lcol);
          float y[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
          for (int i = TERMS - 1; i >= 0; --i) {
            mma(y[0], w[i], b[0], b[1]);
            mma(y[1], w[i], b[2], b[3]);
          }
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            o[2 * j][c] += y[0][c];
            o[2 * j + 1][c] += y[1][c];
          }
        }
      }
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        const int row = r0 + hh * 8;
        if (row >= left) continue;
        float* y = p.out + (size_t)(t0 + c0 + row) * p.H * E + (size_t)h * E + q2;
#pragma unroll
        for (int j = 0; j < E / 8; ++j) {
          const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(Vs + row * VSTR + j * 8 + q2));
          *reinterpret_cast<float2*>(y + j * 8) = make_float2(fmaf(skip, x.x, o[j][2 * hh]), fmaf(skip, x.y, o[j][2 * hh + 1]));
        }
      }
    }
    if (c0 + L >= n && dst == -1) break;               // nothing is passed on: an item in the middle of a portion, its outputs made
    // the chunk's writes: k times its weight in the new state, split in registers, times v
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      unsigned a[L / 16][TERMS][4];
#pragma unroll
      for (int kk = 0; kk < L / 16; ++kk) {
        if (kk * 16 >= left) break;                    // tokens that do not exist weigh nothing
        unsigned x[4];
        ldm4t(x, Ks + (kk * 16 + krow) * QSTR + warp * (D / 4) + m * 16 + kcol);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int t = kk * 16 + (c >> 1) * 8 + q2;         // the tokens of this register's pair
          unsigned terms[TERMS];
          split3(__uint_as_float(x[c] << 16) * into[t], __uint_as_float(x[c] & 0xffff0000u) * into[t + 1], terms);
#pragma unroll
          for (int i = 0; i < TERMS; ++i) a[kk][i][c] = terms[i];
        }
      }
#pragma unroll
      for (int j = 0; j < E / 16; ++j) {
        float y[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int kk = 0; kk < L / 16; ++kk) {
          if (kk * 16 >= left) break;
          unsigned b[4];
          ldm4t(b, Vs + (kk * 16 + lrow) * VSTR + j * 16 + lcol);
#pragma unroll
          for (int i = TERMS - 1; i >= 0; --i) {
            mma(y[0], a[kk][i], b[0], b[1]);
            mma(y[1], a[kk][i], b[2], b[3]);
          }
        }
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
          for (int c = 0; c < 4; ++c) S[m][2 * j + t][c] = fmaf(keep, S[m][2 * j + t][c], y[t][c]);
      }
    }
  }
  float* st = place(dst);
  if (st) {
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int j = 0; j < E / 8; ++j)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh)
          *reinterpret_cast<float2*>(st + (size_t)(warp * (D / 4) + m * 16 + g8 + hh * 8) * E + j * 8 + q2) =
              make_float2(S[m][j][2 * hh], S[m][j][2 * hh + 1]);
  }
  if (p.chunk_decay && dst <= -2 && tid == 0) p.chunk_decay[(size_t)(-(dst + 2)) * p.H + h] = exp2f((float)log_all);
}

template <int D, int E>
int launch_ssd(const SsdParams& p, int R, cudaStream_t stream) {
  const int smem = (int)ssd_smem<D, E>();
  static OptIn opt_in;
  if (const cudaError_t e = opt_in(smem, linear_attention_mma_kernel<D, E>)) return (int)e;
  // without the programmatic dependency: few long-running blocks, which would else be placed several to a
  // multiprocessor while the kernel before still fills the others
  linear_attention_mma_kernel<D, E><<<dim3(R, p.H), THREADS, smem, stream>>>(p);
  return launch_status();
}
}  // namespace

PBE_EXPORT int pbe_linear_attention_mma(const void* q, const void* k, const void* v, int ld, float* out, float* state,
                                        const float* decay, const int32_t* q_start, const int32_t* q_len,
                                        const int32_t* slots, const int32_t* items, float* scratch, int R, int H, int D,
                                        int E, float k_scale, const float* tok_decay, const float* tok_scale,
                                        const float* skip, int kq_share, float* chunk_decay, cudaStream_t stream) {
  if (R <= 0) return 0;
  if (kq_share < 1 || H % kq_share || ld % 8 || (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)state) & 15) || H > 65535)
    return (int)cudaErrorInvalidValue;
  SsdParams p{(const bf16*)q, (const bf16*)k, (const bf16*)v, ld, out, state, decay, q_start, q_len, slots, items, scratch,
              H, k_scale, tok_decay, tok_scale, skip, kq_share, chunk_decay};
  if (D == 128 && E == 64) return launch_ssd<128, 64>(p, R, stream);
  if (D == 64 && E == 64) return launch_ssd<64, 64>(p, R, stream);
  if (D == 64 && E == 128) return launch_ssd<64, 128>(p, R, stream);
  return (int)cudaErrorInvalidValue;
}
