// Residual streams and the norms around them.
//
// stream_norm: the residual is S parallel streams r_0..r_{S-1} per row (S = 1: the usual
// single stream).  One launch (a) folds the pending output y of the sublayer before into the
// streams, r'_j = sum_s M[s, j] r_s + beta_j y (M = 1, beta = 1 with one stream: the plain
// residual add), (b) collapses them, a = sum_j alpha_j r'_j, and (c) normalises a:
// LayerNorm ((a - mean) / sqrt(mean((a - mean)^2) + eps) * g + b, the variance from the
// deviations, two passes over the row in shared memory) or RMSNorm (a / sqrt(mean(a^2) + eps)
// * g).  With a row index the rows are gathered and the streams are left alone (the final
// norm on the wanted rows).  Streams, sums and statistics are float32.
//
// branch_rms_mean: the mean of up to four branches, each divided by its root mean square
// over the row and multiplied by a gain of its own.
//
// gated_rms: o / rms(o) (over the whole row or over each head's slice), times an optional
// gain, times sigmoid(g) or silu(g) of a gate that lies in a wider matrix; or, gate first, the
// gated values o * act(g) divided by their own root mean square, times the gain.
#include "common.cuh"
#include "opt_in.cuh"
#include "pdl.cuh"

using namespace pbe;

namespace {
constexpr int MAX_STREAMS = 8;

struct StreamNormParams {
  float* streams;          // [T, S, W]
  const void* y;           // [T, W] pending sublayer output, or null
  const float* mix;        // [S, S] indexed [from, to]
  const float* beta;       // [S]
  const float* alpha;      // [S]
  const float* gain;       // [W]
  const float* bias;       // [W] or null
  void* out;               // [n, W]
  const int32_t* rows;     // [n] or null
  int S, W;
  float eps;
  int rms;                 // 1: RMSNorm, 0: LayerNorm
};

template <typename TY, typename TO>
__global__ void stream_norm_kernel(StreamNormParams p) {
  __shared__ float red[33];
  __shared__ float coef[MAX_STREAMS * MAX_STREAMS + 2 * MAX_STREAMS];
  extern __shared__ __align__(16) float row[];       // W floats: the collapsed row
  pdl_launch_dependents();
  const int S = p.S, W = p.W;
  float* mix = coef;
  float* beta = coef + MAX_STREAMS * MAX_STREAMS;
  float* alpha = beta + MAX_STREAMS;
  for (int i = threadIdx.x; i < S * S; i += blockDim.x) mix[i] = p.mix[i];
  for (int i = threadIdx.x; i < S; i += blockDim.x) {
    beta[i] = p.beta[i];
    alpha[i] = p.alpha[i];
  }
  pdl_wait();
  __syncthreads();
  const int r = blockIdx.x;
  const int src = p.rows ? p.rows[r] : r;
  float* res = p.streams + (size_t)src * S * W;
  const TY* y = p.y ? (const TY*)p.y + (size_t)src * W : nullptr;
  const bool write_back = p.rows == nullptr && y != nullptr;
  float sum = 0.f;
  for (int c = threadIdx.x; c < W; c += blockDim.x) {
    float x[MAX_STREAMS], z[MAX_STREAMS];
#pragma unroll
    for (int s = 0; s < MAX_STREAMS; ++s) x[s] = s < S ? res[(size_t)s * W + c] : 0.f;
    float a = 0.f;
    if (y) {
      const float yc = to_float(y[c]);
#pragma unroll
      for (int j = 0; j < MAX_STREAMS; ++j) {
        if (j < S) {
          float v = 0.f;
          for (int s = 0; s < S; ++s) v = fmaf(mix[s * S + j], x[s], v);
          z[j] = fmaf(beta[j], yc, v);
          if (write_back) res[(size_t)j * W + c] = z[j];
        }
      }
#pragma unroll
      for (int j = 0; j < MAX_STREAMS; ++j)
        if (j < S) a = fmaf(alpha[j], z[j], a);
    } else {
#pragma unroll
      for (int j = 0; j < MAX_STREAMS; ++j)
        if (j < S) a = fmaf(alpha[j], x[j], a);
    }
    row[c] = a;
    sum += p.rms ? a * a : a;
  }
  const float total = block_sum(sum, red);
  TO* o = (TO*)p.out + (size_t)r * W;
  if (p.rms) {
    const float scale = rsqrtf(total / (float)W + p.eps);
    for (int c = threadIdx.x; c < W; c += blockDim.x) o[c] = from_float<TO>((p.gain[c] * row[c]) * scale);
    return;
  }
  const float mean = total / (float)W;
  float sq = 0.f;
  for (int c = threadIdx.x; c < W; c += blockDim.x) {
    const float d = row[c] - mean;
    sq += d * d;
  }
  const float var = block_sum(sq, red) / (float)W;
  const float scale = 1.0f / sqrtf(var + p.eps);
  for (int c = threadIdx.x; c < W; c += blockDim.x) {
    float v = (row[c] - mean) * scale * p.gain[c];
    if (p.bias) v += p.bias[c];
    o[c] = from_float<TO>(v);
  }
}

struct BranchParams {
  const void* x[4];        // each [T, W]
  const float* gain[4];    // each [W]
  void* out;               // [T, W]
  int n, W;
  float eps;
};

template <typename T>
__global__ void branch_rms_mean_kernel(BranchParams p) {
  __shared__ float red[33];
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x, W = p.W;
  float scale[4];
  for (int b = 0; b < p.n; ++b) {
    const T* x = (const T*)p.x[b] + (size_t)t * W;
    float ss = 0.f;
    for (int c = threadIdx.x; c < W; c += blockDim.x) {
      const float v = to_float(x[c]);
      ss += v * v;
    }
    scale[b] = rsqrtf(block_sum(ss, red) / (float)W + p.eps);
  }
  const float inv_n = 1.0f / (float)p.n;
  T* o = (T*)p.out + (size_t)t * W;
  for (int c = threadIdx.x; c < W; c += blockDim.x) {
    float a = 0.f;
    for (int b = 0; b < p.n; ++b)
      a += to_float(((const T*)p.x[b])[(size_t)t * W + c]) * scale[b] * p.gain[b][c];
    o[c] = from_float<T>(a * inv_n);
  }
}

struct GatedRmsParams {
  const float* o;          // [T, H * E]
  const void* gate;        // first gate element of row 0; row stride ld_gate elements
  const float* gain;       // [H * E] or null
  void* out;               // [T, H * E]
  int ld_gate, H, E;
  float eps;
  int per_head;            // 1: each head's E values have a root mean square of their own
  int gate_act;            // 0: sigmoid, 1: silu
  int gate_f32;            // 1: the gate is float32 whatever the output is
  int gate_first;          // 1: the gate multiplies o before the root mean square is taken (of the gated values)
};

template <typename T>
__global__ void gated_rms_kernel(GatedRmsParams p) {
  __shared__ float red[33];
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x, H = p.H, E = p.E, N = H * E;
  const float* o = p.o + (size_t)t * N;
  const T* g = (const T*)p.gate + (size_t)t * p.ld_gate;
  const float* gf = (const float*)p.gate + (size_t)t * p.ld_gate;
  T* out = (T*)p.out + (size_t)t * N;
  auto gate_of = [&](int c) {
    const float gv = p.gate_f32 ? gf[c] : to_float(g[c]);
    const float sg = 1.0f / (1.0f + expf(-gv));
    return p.gate_act ? gv * sg : sg;
  };
  // what the root mean square is taken of: o itself, or (gate_first) o times its gate
  auto value = [&](int c) { return p.gate_first ? o[c] * gate_of(c) : o[c]; };
  auto finish = [&](int c, float scale) {
    float v = value(c) * scale;
    if (p.gain) v *= p.gain[c];
    out[c] = from_float<T>(p.gate_first ? v : v * gate_of(c));
  };
  if (p.per_head) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int h = warp; h < H; h += nw) {
      float ss = 0.f;
      for (int e = lane; e < E; e += 32) {
        const float v = value(h * E + e);
        ss += v * v;
      }
      const float scale = rsqrtf(warp_sum(ss) / (float)E + p.eps);
      for (int e = lane; e < E; e += 32) finish(h * E + e, scale);
    }
    return;
  }
  float ss = 0.f;
  for (int c = threadIdx.x; c < N; c += blockDim.x) {
    const float v = value(c);
    ss += v * v;
  }
  const float scale = rsqrtf(block_sum(ss, red) / (float)N + p.eps);
  for (int c = threadIdx.x; c < N; c += blockDim.x) finish(c, scale);
}

// The same over each head, heads of whole groups of four values: a warp a head of a row, four neighbouring values a
// lane and access, everything of a head requested at once and kept in registers between the sum and the result (the
// kernel above reads every value and makes every gate twice, 4 bytes an access: 2,048 rows of 4,096 in eight parts
// 45 -> 16 us).
constexpr int GR_WARPS = 8;

__device__ __forceinline__ float4 load_four(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load_four(const __nv_bfloat16* p) {
  const uint2 w = *reinterpret_cast<const uint2*>(p);
  return make_float4(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u), __uint_as_float(w.y << 16),
                     __uint_as_float(w.y & 0xffff0000u));
}
__device__ __forceinline__ void store_four(float* p, const float (&v)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void store_four(__nv_bfloat16* p, const float (&v)[4]) {
  const __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
  *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const unsigned*>(&a), *reinterpret_cast<const unsigned*>(&b));
}

template <typename T, typename TG, int QUADS>       // groups of four a lane holds at most
__global__ void __launch_bounds__(32 * GR_WARPS) gated_rms_heads_kernel(GatedRmsParams p, int rows) {
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const long long rh = (long long)blockIdx.x * GR_WARPS + (threadIdx.x >> 5);
  if (rh >= (long long)rows * p.H) return;
  const int t = (int)(rh / p.H), h = (int)(rh - (long long)t * p.H), E = p.E;
  const float* o = p.o + (size_t)rh * E;
  const TG* g = (const TG*)p.gate + (size_t)t * p.ld_gate + (size_t)h * E;
  const float* gain = p.gain ? p.gain + (size_t)h * E : nullptr;
  float v[QUADS][4], gate[QUADS][4];
#pragma unroll
  for (int i = 0; i < QUADS; ++i) {
    const int e = (i * 32 + lane) * 4;
    const float4 x = e < E ? load_four(o + e) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 y = e < E ? load_four(g + e) : make_float4(0.f, 0.f, 0.f, 0.f);
    v[i][0] = x.x; v[i][1] = x.y; v[i][2] = x.z; v[i][3] = x.w;
    gate[i][0] = y.x; gate[i][1] = y.y; gate[i][2] = y.z; gate[i][3] = y.w;
  }
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < QUADS; ++i)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float gv = gate[i][k];
      const float sg = 1.0f / (1.0f + expf(-gv));
      gate[i][k] = p.gate_act ? gv * sg : sg;
      if (p.gate_first) v[i][k] *= gate[i][k];
      ss += v[i][k] * v[i][k];
    }
  const float scale = rsqrtf(warp_sum(ss) / (float)E + p.eps);
  T* out = (T*)p.out + (size_t)rh * E;
#pragma unroll
  for (int i = 0; i < QUADS; ++i) {
    const int e = (i * 32 + lane) * 4;
    if (e >= E) break;
    const float4 w = gain ? load_four(gain + e) : make_float4(1.f, 1.f, 1.f, 1.f);
    const float ws[4] = {w.x, w.y, w.z, w.w};
    float y[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      y[k] = v[i][k] * scale * ws[k];
      if (!p.gate_first) y[k] *= gate[i][k];
    }
    store_four(out + e, y);
  }
}

template <typename T, typename TG>
void launch_gated_heads(const GatedRmsParams& p, int rows, cudaStream_t stream) {
  const long long warps = (long long)rows * p.H;
  const int blocks = (int)((warps + GR_WARPS - 1) / GR_WARPS);
  if (p.E <= 128) launch_k(gated_rms_heads_kernel<T, TG, 1>, blocks, 32 * GR_WARPS, 0, stream, p, rows);
  else if (p.E <= 256) launch_k(gated_rms_heads_kernel<T, TG, 2>, blocks, 32 * GR_WARPS, 0, stream, p, rows);
  else launch_k(gated_rms_heads_kernel<T, TG, 4>, blocks, 32 * GR_WARPS, 0, stream, p, rows);
}
}  // namespace

PBE_EXPORT int pbe_stream_norm(float* streams, const void* y, int y_dtype, const float* mix, const float* beta,
                               const float* alpha, const float* gain, const float* bias, void* out, int out_dtype,
                               const int32_t* rows, int n, int S, int W, float eps, int rms, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (S < 1 || S > MAX_STREAMS) return (int)cudaErrorInvalidValue;
  StreamNormParams p{streams, y, mix, beta, alpha, gain, bias, out, rows, S, W, eps, rms};
  const int threads = W >= 2048 ? 512 : (W >= 512 ? 256 : 128);
  const size_t smem = sizeof(float) * (size_t)W;
  cudaError_t e;
#define PBE_SN(TY, TO)                                                                                  \
  do {                                                                                                  \
    static OptIn opt_in;                                                                                \
    if (smem > 48 * 1024) opt_in(smem, stream_norm_kernel<TY, TO>);                                     \
    e = launch_k(stream_norm_kernel<TY, TO>, n, threads, smem, stream, p);                              \
  } while (0)
  const bool yb = y != nullptr && y_dtype == PBE_BF16;
  if (out_dtype == PBE_F32) {
    if (yb) PBE_SN(__nv_bfloat16, float); else PBE_SN(float, float);
  } else {
    if (yb) PBE_SN(__nv_bfloat16, __nv_bfloat16); else PBE_SN(float, __nv_bfloat16);
  }
#undef PBE_SN
  (void)e;
  return launch_status();
}

PBE_EXPORT int pbe_branch_rms_mean(const void* const* x, const float* const* gain, int n, void* out, int dtype,
                                   int T, int W, float eps, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (n < 1 || n > 4) return (int)cudaErrorInvalidValue;
  BranchParams p{};
  for (int b = 0; b < n; ++b) {
    p.x[b] = x[b];
    p.gain[b] = gain[b];
  }
  p.out = out; p.n = n; p.W = W; p.eps = eps;
  const int threads = W >= 512 ? 256 : 128;
  if (dtype == PBE_F32) launch_k(branch_rms_mean_kernel<float>, T, threads, 0, stream, p);
  else launch_k(branch_rms_mean_kernel<__nv_bfloat16>, T, threads, 0, stream, p);
  return launch_status();
}

PBE_EXPORT int pbe_gated_rms(const float* o, const void* gate, int gate_dtype, int ld_gate, const float* gain, void* out, int dtype,
                             int T, int H, int E, float eps, int per_head, int gate_act, int gate_first,
                             cudaStream_t stream) {
  if (T <= 0) return 0;
  GatedRmsParams p{o, gate, gain, out, ld_gate, H, E, eps, per_head, gate_act, gate_dtype == PBE_F32 ? 1 : 0, gate_first};
  // heads of up to 512 values in groups of four that lie on the boundaries of such a group's access
  const uintptr_t at = (uintptr_t)o | (uintptr_t)gain | (dtype == PBE_F32 ? (uintptr_t)out : (uintptr_t)out << 1) |
                       (p.gate_f32 ? (uintptr_t)gate : (uintptr_t)gate << 1);
  if (per_head && E % 4 == 0 && E <= 512 && ld_gate % 4 == 0 && (at & 15) == 0 && (long long)T * H < (1LL << 33)) {
    if (dtype == PBE_F32) launch_gated_heads<float, float>(p, T, stream);
    else if (p.gate_f32) launch_gated_heads<__nv_bfloat16, float>(p, T, stream);
    else launch_gated_heads<__nv_bfloat16, __nv_bfloat16>(p, T, stream);
    return launch_status();
  }
  const int threads = H * E >= 512 ? 256 : 128;
  if (dtype == PBE_F32) launch_k(gated_rms_kernel<float>, T, threads, 0, stream, p);
  else launch_k(gated_rms_kernel<__nv_bfloat16>, T, threads, 0, stream, p);
  return launch_status();
}
