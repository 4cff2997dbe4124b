// A feed-forward made of many small gated experts of which each token uses a few.
//
// route: from float32 router logits [T, E]: scores s = softmax over all experts, or (score_kind 1)
// sigmoid of each logit; the choice is made on c = s + correction (a learned vector, optional);
// experts form `groups` equal groups of neighbours, a group's rank is its largest c or (group_rank
// 2) the sum of its two largest, and only experts of the `keep` best groups can be chosen (groups =
// 1: no restriction; a barred expert is out whatever its c, which may be negative); the `top`
// allowed experts with the largest c are chosen (ties: the lower index); their weights are their
// scores s, without the correction, over the sum of the chosen scores (+ 1e-20) unless they are taken
// as they are, times `scale`.  One warp per token.
//
// expert_rows: for few rows (decoded tokens).  Per (token, chosen expert) pair the expert's gate
// and up rows are streamed against the token's input (blocks of 32 hidden units, a warp per unit,
// the lanes along the input in 16-byte loads), h = silu(g) * u goes to scratch memory in float32;
// a second launch streams the down rows against it (blocks of 32 output columns) and writes the
// weighted result to the pair's own slot, [T, top, W]; combine adds a token's slots in order, so
// a token's result never depends on what else is in the step.
//
// Experts without a gate (act 2: h = relu(W_up x)^2) have up rows only.  A router's weight may multiply an
// expert's input instead of its output (weight_in): expert_rows then scales the up product, which is the
// same, and the gather scales the rows.  What is added for every token (a shared expert) may carry a factor
// sigmoid(z_t), z one float32 number per token.
//
// For many rows the host side sorts the rows by expert (pair_rows / scatter below) and runs one
// matrix product per expert over its rows.
#include "common.cuh"
#include "opt_in.cuh"
#include "pdl.cuh"

using namespace pbe;

namespace {
constexpr int MAX_PER_LANE = 16;       // experts a lane holds: up to 512 experts
constexpr int MAX_TOP = 32;

struct RouteParams {
  const float* logits;       // [T, ld]
  int ld;
  int32_t* chosen;           // [T, top]
  float* weights;            // [T, top]
  int T, E, top, groups, keep;
  float scale;
  int score_kind;            // 0: softmax over the experts, 1: sigmoid
  const float* correction;   // [E] or null: added to the scores for the choice only
  int group_rank;            // 1: a group's largest choice score, 2: the sum of its two largest
  int normalize;             // 1: the weights are divided by the chosen scores' sum
};

// the lane-distributed argmax of v (lane l holds experts l, l + 32, ...); ties go to the lower index
__device__ __forceinline__ void warp_argmax(float& best, int& at) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ob = __shfl_xor_sync(0xffffffffu, best, o);
    const int oa = __shfl_xor_sync(0xffffffffu, at, o);
    if (ob > best || (ob == best && oa < at)) { best = ob; at = oa; }
  }
}

// A warp a token; PER_LANE: experts a lane holds at most (one for up to 32 experts: every pass over a lane's experts is
// then one compare; 2,048 tokens, 32 experts in four groups 17.2 us with sixteen for all sizes, 6.2 now).
template <int PER_LANE>
__global__ void route_kernel(RouteParams p) {
  pdl_launch_dependents();
  pdl_wait();
  const int warps = blockDim.x >> 5;
  const int t = blockIdx.x * warps + (threadIdx.x >> 5);
  if (t >= p.T) return;
  const int lane = threadIdx.x & 31, E = p.E;
  const float* z = p.logits + (size_t)t * p.ld;
  float s[PER_LANE];     // the scores
  float c[PER_LANE];     // the choice scores
  if (p.score_kind == 1) {
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
      const int e = lane + 32 * i;
      const float v = e < E ? 1.0f / (1.0f + expf(-z[e])) : 0.f;
      s[i] = v >= 0.f ? v : 0.f;          // not a number (a padding row nobody wrote): counts as 0
    }
  } else {
    float m = -INFINITY;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
      const int e = lane + 32 * i;
      s[i] = e < E ? z[e] : -INFINITY;
      m = fmaxf(m, s[i]);
    }
    m = warp_max(m);
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
      const int e = lane + 32 * i;
      s[i] = e < E ? expf(s[i] - m) : 0.f;
      sum += s[i];
    }
    sum = warp_sum(sum);
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
      // a row of logits that are not numbers (a padding row of a captured step, whose input nobody
      // wrote) still chooses experts that exist: its scores count as 0 and the lowest indices win
      const float v = s[i] / sum;
      s[i] = v >= 0.f ? v : 0.f;
    }
  }
#pragma unroll
  for (int i = 0; i < PER_LANE; ++i) {
    const int e = lane + 32 * i;
    c[i] = s[i] + ((p.correction && e < E) ? p.correction[e] : 0.f);
    // plain sigmoid scores rank like their logits, which stay apart where the scores round to one or zero
    if (p.score_kind == 1 && !p.correction && p.groups == 1 && e < E) c[i] = z[e] == z[e] ? z[e] : -INFINITY;
  }
  // allowed[i]: may expert lane + 32 i still be chosen
  bool allowed[PER_LANE];
#pragma unroll
  for (int i = 0; i < PER_LANE; ++i) allowed[i] = lane + 32 * i < E;
  if (p.groups > 1 && p.keep < p.groups) {
    const int per = E / p.groups;
    // rank of group g: in lane g % 32, slot g / 32 (groups <= 64)
    float rank[2] = {-INFINITY, -INFINITY};
    for (int g = 0; g < p.groups; ++g) {
      float best = -INFINITY;
      int at = 0x7fffffff;
#pragma unroll
      for (int i = 0; i < PER_LANE; ++i) {
        const int e = lane + 32 * i;
        if (e < E && e / per == g && (c[i] > best || (c[i] == best && e < at))) { best = c[i]; at = e; }
      }
      warp_argmax(best, at);
      float value = best;
      if (p.group_rank == 2 && per > 1) {
        float second = -INFINITY;
        int at2 = 0x7fffffff;
#pragma unroll
        for (int i = 0; i < PER_LANE; ++i) {
          const int e = lane + 32 * i;
          if (e < E && e / per == g && e != at && (c[i] > second || (c[i] == second && e < at2))) {
            second = c[i];
            at2 = e;
          }
        }
        warp_argmax(second, at2);
        value = best + second;
      }
      if (lane == (g & 31)) rank[g >> 5] = value;
    }
    unsigned long long kept_lo = 0ull;          // bit g: group g is kept
    for (int round = 0; round < p.keep; ++round) {
      float best = -INFINITY;
      int at = 0x7fffffff;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int g = lane + 32 * j;
        if (g < p.groups && !((kept_lo >> g) & 1ull) && (rank[j] > best || (rank[j] == best && g < at))) {
          best = rank[j];
          at = g;
        }
      }
      warp_argmax(best, at);
      if (at >= p.groups) {                     // nothing compares (ranks that are not numbers): the lowest group left
        at = 0;
        while ((kept_lo >> at) & 1ull) ++at;
      }
      kept_lo |= 1ull << at;
    }
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
      const int e = lane + 32 * i;
      allowed[i] = e < E && ((kept_lo >> (e / per)) & 1ull);
    }
  }
  float picked_s = 0.f;              // lane k keeps the k-th choice
  int picked_e = 0;
  float total = 0.f;
  for (int k = 0; k < p.top; ++k) {
    float best = -INFINITY, best_s = 0.f;
    int at = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
      const int e = lane + 32 * i;
      if (allowed[i] && (at == 0x7fffffff || c[i] > best || (c[i] == best && e < at))) { best = c[i]; at = e; best_s = s[i]; }
    }
    {   // the warp's best: the larger choice score, ties (and lanes with nothing) to the lower index
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oa = __shfl_xor_sync(0xffffffffu, at, o);
        const float os = __shfl_xor_sync(0xffffffffu, best_s, o);
        const bool take = oa != 0x7fffffff && (at == 0x7fffffff || ob > best || (ob == best && oa < at));
        if (take) { best = ob; at = oa; best_s = os; }
      }
    }
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i)
      if (lane + 32 * i == at) allowed[i] = false;
    if (lane == k) { picked_s = best_s; picked_e = at; }
    total += best_s;
  }
  if (lane < p.top) {
    const float inv = p.normalize ? p.scale / (total + 1e-20f) : p.scale;
    p.chosen[(size_t)t * p.top + lane] = picked_e;
    p.weights[(size_t)t * p.top + lane] = picked_s * inv;
  }
}

// ------------------------------------------------------------------------------------------------
struct ExpertRowsParams {
  const void* x;             // [T, W]
  const void* w_gate;        // expert e's [F, W] at element e * gu_stride
  const void* w_up;          // the same (gate and up may lie in one [E, 2F, W] tensor)
  long long gu_stride;
  const void* w_down;        // [E, W, F]
  const int32_t* chosen;     // [T, top]
  const float* weights;      // [T, top]
  float* hidden;             // [T * top, F] scratch: silu(gate) * up of every pair
  float* part;               // [T, top, W]
  int T, W, F, top;
  int act;                   // 0: silu(g) * u; 1: g <- min(g, limit), u <- clamp(u, +-limit), g sigmoid(alpha g) (u + 1);
                             // 2: relu(u)^2, no gate
  float limit, alpha;
  int weight_in;             // 1: the weight multiplies the expert's input
};

// dot product of a weight row with a float32 vector in shared memory, the lanes along the row;
// 16-byte loads of the weights where the row allows them (n a multiple of 8 bfloat16 / 4 float)
__device__ __forceinline__ float dot_row(const float* __restrict__ w, const float* __restrict__ x, int n, int lane) {
  float a = 0.f;
  if ((n & 3) == 0 && (((uintptr_t)w) & 15) == 0) {
    for (int i = lane * 4; i < n; i += 128) {
      const float4 v = *reinterpret_cast<const float4*>(w + i);
      a = fmaf(v.x, x[i], a); a = fmaf(v.y, x[i + 1], a); a = fmaf(v.z, x[i + 2], a); a = fmaf(v.w, x[i + 3], a);
    }
  } else {
    for (int i = lane; i < n; i += 32) a = fmaf(w[i], x[i], a);
  }
  return warp_sum(a);
}
__device__ __forceinline__ float dot_row(const __nv_bfloat16* __restrict__ w, const float* __restrict__ x, int n,
                                         int lane) {
  float a = 0.f;
  if ((n & 7) == 0 && (((uintptr_t)w) & 15) == 0) {
    for (int i = lane * 8; i < n; i += 256) {
      const uint4 raw = *reinterpret_cast<const uint4*>(w + i);
      const unsigned u[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u[j]));
        a = fmaf(f.x, x[i + 2 * j], a);
        a = fmaf(f.y, x[i + 2 * j + 1], a);
      }
    }
  } else {
    for (int i = lane; i < n; i += 32) a = fmaf(to_float(w[i]), x[i], a);
  }
  return warp_sum(a);
}

constexpr int ER_WARPS = 8;
constexpr int ER_UNITS = 32;      // hidden units (first kernel) or output columns (second) a block takes

// block (pair, slice of the hidden units): h = silu(W_gate x) * (W_up x) for its units
template <typename T>
__global__ void __launch_bounds__(ER_WARPS * 32) expert_hidden_kernel(ExpertRowsParams p) {
  extern __shared__ __align__(16) float xs[];        // [W]
  pdl_launch_dependents();
  pdl_wait();
  const int pair = blockIdx.x;
  const int t = pair / p.top;
  const int e = p.chosen[pair];
  const T* x = (const T*)p.x + (size_t)t * p.W;
  for (int i = threadIdx.x; i < p.W; i += blockDim.x) xs[i] = to_float(x[i]);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const T* wg = (const T*)p.w_gate + (size_t)e * p.gu_stride;
  const T* wu = (const T*)p.w_up + (size_t)e * p.gu_stride;
  const int f_end = min(p.F, (blockIdx.y + 1) * ER_UNITS);
  const float scale_in = p.weight_in ? p.weights[pair] : 1.0f;
  for (int f = blockIdx.y * ER_UNITS + warp; f < f_end; f += ER_WARPS) {
    const float g = p.act == 2 ? 0.f : dot_row(wg + (size_t)f * p.W, xs, p.W, lane) * scale_in;
    const float u = dot_row(wu + (size_t)f * p.W, xs, p.W, lane) * scale_in;
    if (lane == 0) {
      float h;
      if (p.act == 2) {
        const float ur = fmaxf(u, 0.f);
        h = ur * ur;
      } else if (p.act == 1) {
        const float gc = fminf(g, p.limit), uc = fminf(fmaxf(u, -p.limit), p.limit);
        h = (gc / (1.0f + expf(-p.alpha * gc))) * (uc + 1.0f);
      } else {
        h = (g / (1.0f + expf(-g))) * u;
      }
      p.hidden[(size_t)pair * p.F + f] = h;
    }
  }
}

// block (pair, slice of the output columns): weight * W_down h for its columns
template <typename T>
__global__ void __launch_bounds__(ER_WARPS * 32) expert_down_kernel(ExpertRowsParams p) {
  extern __shared__ __align__(16) float hs[];        // [F]
  pdl_launch_dependents();
  pdl_wait();
  const int pair = blockIdx.x;
  const int e = p.chosen[pair];
  const float weight = p.weight_in ? 1.0f : p.weights[pair];
  for (int i = threadIdx.x; i < p.F; i += blockDim.x) hs[i] = p.hidden[(size_t)pair * p.F + i];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const T* wd = (const T*)p.w_down + (size_t)e * p.W * p.F;
  float* out = p.part + (size_t)pair * p.W;
  const int c_end = min(p.W, (blockIdx.y + 1) * ER_UNITS);
  for (int c = blockIdx.y * ER_UNITS + warp; c < c_end; c += ER_WARPS) {
    const float y = dot_row(wd + (size_t)c * p.F, hs, p.F, lane);
    if (lane == 0) out[c] = weight * y;
  }
}

// `addend` (optional, [T, W]): what every token gets besides its experts (a shared expert's output), times
// sigmoid(gate[t * ld_gate]) when there is a gate
__device__ __forceinline__ float addend_factor(const float* gate, int ld_gate, size_t t) {
  return gate ? 1.0f / (1.0f + expf(-gate[t * ld_gate])) : 1.0f;
}

template <typename T>
__global__ void combine_kernel(const float* part, const T* addend,
                               const float* gate, int ld_gate, T* out, int top, int W,
                               size_t total) {
  pdl_launch_dependents();
  pdl_wait();
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const size_t t = i / W;
    const int c = (int)(i - t * W);
    float a = 0.f;
    for (int k = 0; k < top; ++k) a += part[(t * top + k) * W + c];
    if (addend) a = fmaf(addend_factor(gate, ld_gate, t), to_float(addend[i]), a);
    out[i] = from_float<T>(a);
  }
}

// ------------------------------------------------------------------------------------------------
// Rows sorted by expert: pair (t, k) gets a place in the run of its expert.  counts[e] first
// (count_kernel), then the runs' starts on the host or by a scan, then place_kernel hands the
// places out in (t, k) order inside every expert's run: a single block walks the pairs of an
// expert in order, so the order inside a run is the tokens' own and nothing depends on timing.
// Block e reads all pairs, a thread PLACE_PER neighbouring ones: each counts its own, one scan over the block turns
// the counts into places.  8,192 pairs, 32 experts: 21.9 us with a pair a thread and three barriers for every 256
// pairs, about 6 now.
// (No __restrict__ on what a kernel before wrote: these kernels are resident before that one has ended, and loads that
// may be taken for read-only are not ordered behind the wait.)
constexpr int PLACE_THREADS = 512, PLACE_PER = 16;

__global__ void __launch_bounds__(PLACE_THREADS) place_kernel(const int32_t* chosen, int pairs, int E,
                                                              int32_t* counts, int32_t* place) {
  __shared__ int warp_tot[PLACE_THREADS / 32];
  const int e = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  pdl_launch_dependents();
  pdl_wait();
  const bool aligned = ((uintptr_t)chosen & 15) == 0;      // then every sixteenth pair lies on a 16-byte boundary
  int base = 0;
  for (long long first = 0; first < pairs; first += PLACE_THREADS * PLACE_PER) {
    const long long i0 = first + (long long)threadIdx.x * PLACE_PER;
    unsigned mine = 0;                       // bit j: pair i0 + j chose this block's expert
    if (aligned && i0 + PLACE_PER <= pairs) {
#pragma unroll
      for (int j = 0; j < PLACE_PER; j += 4) {
        const int4 c = *reinterpret_cast<const int4*>(chosen + i0 + j);
        mine |= (unsigned)(c.x == e) << j | (unsigned)(c.y == e) << (j + 1) | (unsigned)(c.z == e) << (j + 2) |
                (unsigned)(c.w == e) << (j + 3);
      }
    } else {
#pragma unroll
      for (int j = 0; j < PLACE_PER; ++j)
        if (i0 + j < pairs) mine |= (unsigned)(chosen[i0 + j] == e) << j;
    }
    int upto = __popc(mine);                 // inclusive scan: of the warp, then of the block
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += n;
    }
    if (lane == 31) warp_tot[warp] = upto;
    __syncthreads();
    int at = base + upto - __popc(mine);
#pragma unroll
    for (int w = 0; w < PLACE_THREADS / 32; ++w) {
      if (w < warp) at += warp_tot[w];
      base += warp_tot[w];
    }
    for (unsigned left = mine; left; left &= left - 1) place[i0 + __ffs(left) - 1] = at++;
    __syncthreads();                         // warp_tot is written again
  }
  if (threadIdx.x == 0) counts[e] = base;
}

// gathered[start[e] + place] = x[t] for every pair; and the way back, weighted.  VEC values a thread and access
// (eight bfloat16 or four floats where the rows lie on 16-byte boundaries): the sum of 8,192 rows of 2,048 bfloat16
// values into 2,048 took 23.7 us with a value a thread, 9 now.  A block takes a token, all of its experts: on the way out
// its row is read once (2,048 rows to four experts each: 11.5 us with a block a pair, 7.9 now).
template <typename T, int VEC>
struct __align__(sizeof(T) * VEC) RowPiece {
  T v[VEC];
};

template <typename T, int VEC>
__global__ void gather_rows_kernel(const T* x, const int32_t* chosen,
                                   const int32_t* place, const int32_t* start,
                                   const float* weights, T* gathered, int top, int W) {
  using P = RowPiece<T, VEC>;
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x;
  const P* src = reinterpret_cast<const P*>(x + (size_t)t * W);
  for (int i = threadIdx.x; i < W / VEC; i += blockDim.x) {
    const P p = src[i];
#pragma unroll 4
    for (int k = 0; k < top; ++k) {
      const int pair = t * top + k;
      P o = p;
      if (weights) {
        const float f = weights[pair];
#pragma unroll
        for (int j = 0; j < VEC; ++j) o.v[j] = from_float<T>(f * to_float(p.v[j]));
      }
      reinterpret_cast<P*>(gathered + (size_t)(start[chosen[pair]] + place[pair]) * W)[i] = o;
    }
  }
}

template <typename T, int VEC>
__global__ void scatter_rows_kernel(const T* y, const int32_t* chosen,
                                    const int32_t* place, const int32_t* start,
                                    const float* weights, const T* addend,
                                    const float* gate, int ld_gate, T* out, int top, int W) {
  using P = RowPiece<T, VEC>;
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x;
  const float factor = addend_factor(gate, ld_gate, t);
  for (int i = threadIdx.x; i < W / VEC; i += blockDim.x) {
    float a[VEC];
#pragma unroll
    for (int j = 0; j < VEC; ++j) a[j] = 0.f;
#pragma unroll 4
    for (int k = 0; k < top; ++k) {
      const int pair = t * top + k;
      const float f = weights ? weights[pair] : 1.0f;
      const P p = reinterpret_cast<const P*>(y + (size_t)(start[chosen[pair]] + place[pair]) * W)[i];
#pragma unroll
      for (int j = 0; j < VEC; ++j) a[j] += f * to_float(p.v[j]);
    }
    if (addend) {
      const P p = reinterpret_cast<const P*>(addend + (size_t)t * W)[i];
#pragma unroll
      for (int j = 0; j < VEC; ++j) a[j] = fmaf(factor, to_float(p.v[j]), a[j]);
    }
    P o;
#pragma unroll
    for (int j = 0; j < VEC; ++j) o.v[j] = from_float<T>(a[j]);
    reinterpret_cast<P*>(out + (size_t)t * W)[i] = o;
  }
}

inline bool on_16_bytes(const void* p) { return ((uintptr_t)p & 15) == 0; }

template <typename T>
void gather_rows(const void* x, const int32_t* chosen, const int32_t* place, const int32_t* start, const float* weights,
                 void* gathered, int T_, int top, int W, cudaStream_t stream) {
  constexpr int VEC = 16 / (int)sizeof(T);
  const int threads = W / VEC > 128 ? 256 : 128;
  if (W % VEC == 0 && on_16_bytes(x) && on_16_bytes(gathered))
    launch_k(gather_rows_kernel<T, VEC>, T_, threads, 0, stream, (const T*)x, chosen, place, start, weights, (T*)gathered, top, W);
  else
    launch_k(gather_rows_kernel<T, 1>, T_, threads, 0, stream, (const T*)x, chosen, place, start, weights, (T*)gathered, top, W);
}

template <typename T>
void scatter_rows(const void* y, const int32_t* chosen, const int32_t* place, const int32_t* start, const float* weights,
                  const void* addend, const float* gate, int ld_gate, void* out, int T_, int top, int W, cudaStream_t stream) {
  constexpr int VEC = 16 / (int)sizeof(T);
  const int threads = W / VEC > 128 ? 256 : 128;
  if (W % VEC == 0 && on_16_bytes(y) && on_16_bytes(out) && on_16_bytes(addend))
    launch_k(scatter_rows_kernel<T, VEC>, T_, threads, 0, stream, (const T*)y, chosen, place, start, weights, (const T*)addend,
             gate, ld_gate, (T*)out, top, W);
  else
    launch_k(scatter_rows_kernel<T, 1>, T_, threads, 0, stream, (const T*)y, chosen, place, start, weights, (const T*)addend,
             gate, ld_gate, (T*)out, top, W);
}
}  // namespace

PBE_EXPORT int pbe_route(const float* logits, int ld, int32_t* chosen, float* weights, int T, int E, int top, int groups,
                         int keep, float scale, int score_kind, const float* correction, int group_rank,
                         int normalize, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (E < 1 || E > 32 * MAX_PER_LANE || top < 1 || top > MAX_TOP || top > E || groups < 1 || groups > 64 ||
      E % groups != 0 || keep < 1 || keep > groups || top > keep * (E / groups) || score_kind < 0 || score_kind > 1 ||
      group_rank < 1 || group_rank > 2)
    return (int)cudaErrorInvalidValue;
  RouteParams p{logits, ld, chosen, weights, T, E, top, groups, keep, scale, score_kind, correction, group_rank, normalize};
  const dim3 grid((T + 3) / 4);
  if (E <= 32) launch_k(route_kernel<1>, grid, 128, 0, stream, p);
  else if (E <= 64) launch_k(route_kernel<2>, grid, 128, 0, stream, p);
  else if (E <= 128) launch_k(route_kernel<4>, grid, 128, 0, stream, p);
  else launch_k(route_kernel<MAX_PER_LANE>, grid, 128, 0, stream, p);
  return launch_status();
}

PBE_EXPORT int pbe_expert_rows(const void* x, const void* w_gate, const void* w_up, long long gu_stride,
                               const void* w_down, const int32_t* chosen, const float* weights, float* hidden,
                               float* part, void* out, int dtype, int T, int W, int F, int top, int act, float limit,
                               float alpha, const void* addend, const float* addend_gate, int ld_gate, int weight_in,
                               cudaStream_t stream) {
  if (T <= 0) return 0;
  ExpertRowsParams p{x, w_gate, w_up, gu_stride, w_down, chosen, weights, hidden, part, T, W, F, top, act, limit, alpha, weight_in};
  const size_t smem1 = sizeof(float) * (size_t)W, smem2 = sizeof(float) * (size_t)F;
  if (smem1 > 200 * 1024 || smem2 > 200 * 1024) return (int)cudaErrorInvalidValue;
  dim3 grid1(T * top, (F + ER_UNITS - 1) / ER_UNITS), grid2(T * top, (W + ER_UNITS - 1) / ER_UNITS);
#define PBE_ER(TT)                                                                                             \
  do {                                                                                                         \
    static OptIn opt_in;                                                                                       \
    if (smem1 > 48 * 1024 || smem2 > 48 * 1024) opt_in(200 * 1024, expert_hidden_kernel<TT>, expert_down_kernel<TT>);\
    launch_k(expert_hidden_kernel<TT>, grid1, ER_WARPS * 32, smem1, stream, p);                                \
    launch_k(expert_down_kernel<TT>, grid2, ER_WARPS * 32, smem2, stream, p);                                  \
  } while (0)
  if (dtype == PBE_F32) PBE_ER(float); else PBE_ER(__nv_bfloat16);
#undef PBE_ER
  int e = launch_status();
  if (e != 0) return e;
  const size_t total = (size_t)T * W;
  size_t blocks = (total + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  if (dtype == PBE_F32)
    launch_k(combine_kernel<float>, (int)blocks, 256, 0, stream, (const float*)part, (const float*)addend, addend_gate,
             ld_gate, (float*)out, top, W, total);
  else
    launch_k(combine_kernel<__nv_bfloat16>, (int)blocks, 256, 0, stream, (const float*)part,
             (const __nv_bfloat16*)addend, addend_gate, ld_gate, (__nv_bfloat16*)out, top, W, total);
  return launch_status();
}

PBE_EXPORT int pbe_expert_places(const int32_t* chosen, int pairs, int E, int32_t* counts, int32_t* place,
                                 cudaStream_t stream) {
  if (pairs <= 0) return 0;
  launch_k(place_kernel, E, PLACE_THREADS, 0, stream, chosen, pairs, E, counts, place);
  return launch_status();
}

PBE_EXPORT int pbe_expert_gather(const void* x, const int32_t* chosen, const int32_t* place, const int32_t* start,
                                 const float* weights, void* gathered, int dtype, int T, int top, int W,
                                 cudaStream_t stream) {
  if (T <= 0) return 0;
  if (dtype == PBE_F32) gather_rows<float>(x, chosen, place, start, weights, gathered, T, top, W, stream);
  else gather_rows<__nv_bfloat16>(x, chosen, place, start, weights, gathered, T, top, W, stream);
  return launch_status();
}

PBE_EXPORT int pbe_expert_scatter(const void* y, const int32_t* chosen, const int32_t* place, const int32_t* start,
                                  const float* weights, void* out, int dtype, int T, int top, int W,
                                  const void* addend, const float* addend_gate, int ld_gate, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (dtype == PBE_F32) scatter_rows<float>(y, chosen, place, start, weights, addend, addend_gate, ld_gate, out, T, top, W, stream);
  else scatter_rows<__nv_bfloat16>(y, chosen, place, start, weights, addend, addend_gate, ld_gate, out, T, top, W, stream);
  return launch_status();
}
