// The float32 product Y[M, N] = X[M, K] * W[N, K]^T (+ bias[N]) of many rows on the fifth-generation tensor cores, with
// float32's precision: every operand is cut into three bfloat16 terms, x = h + m + l, |m| <= 2^-8 |x| and |l| <= 2^-17 |x|,
// which hold all of its 24 bits, and the six products hh, hm, mh, mm, hl, lh are added; ml and lm, which are left out, are
// 2^-25 of a product each at most, together as large as the rounding of the multiply-add that they stand for.
//
// The tensor cores add in float32 but cut off what does not fit instead of rounding it, so a sum is not left to them
// for long: after every 64 k the accumulator in tensor memory starts anew, the small products are issued before hh, and the
// epilogue's warps add its contents to the tile's running sums in registers, with a rounding add each; after 1,792 k at most the
// running sums are added to the output.  Against 64 bits, relative root mean square error of sgemm.cu's multiply-adds -> this: normal
// numbers 4.1e-7 -> 1.2e-7 (K = 1,536) and 1.3e-7 (8,960), positive ones 2.1e-7 -> 1.1e-7 and 1.1e-7 -> 1.0e-7; a float32 model's
// logits after 1,028 prompt tokens 2.8e-6 -> 2.5e-6.  Where single products outweigh all others (factors spread over e^3) both
// are at the last bit: 0.5-1.5e-7 and 0.7-1.4e-7.
//
// Two kernels a product:
//  * split3: X's three terms as bfloat16 matrices one below the other, rows padded with zeros to 64 k.
//  * the product, of tiles of 128 rows of W by up to 192 rows of X, as many X tiles as there have to be and of one size (a multiple
//    of 16: 1,028 rows are six tiles of 176, where tiles of 128 rows of X leave four rows to a tile of their own).  W comes as it
//    is: warp 14 fetches 128 rows x 64 k by TMA, warps 0-3 cut them into terms, a row a thread, and write these to tensor memory,
//    where the MMAs take A from (terms written out by a kernel of their own took 47 us of 345 for 1,028 x 17,920 x 1,536, and are
//    6 bytes an element to fetch instead of 4).  Warp 12 fetches X's terms, two sets of three; warp 13 issues the MMAs in
//    the order l h, h l, m m, m h, h m, h h; warps 4-11 hold the running sums, a row of W and half of the tile's rows of X a
//    thread, and write them out, 32 neighbouring columns of Y a warp.  Two accumulators alternate, and two of W's terms h; l and
//    m are written while the products that do not need them run.  Persistent blocks walk over tiles, or over parts of K of
//    tiles where there are too few (a small kernel adds the parts in order).
// Either kernel also tells whether an element is other than zero or of a size from SMALLEST to LARGEST: such a product is left to
// sgemm.cu, whose kernel is launched behind and looks at the flag.  A smaller one's third term would fall under bfloat16's
// smallest normal number, larger ones' products could overflow with either sign where their sum does not, and an infinity
// times a term that is zero would be no number.
//
// What bounds it is the tensor pipe, 2,112 clocks a K block of 176 rows (2,340 measured), and, where a wave of blocks ends, the
// outputs' way to memory (350 clocks a K block on average).  The split has to be free of branches: with a test a number it took
// 4,700 clocks a K block and bound everything.  A pair of blocks with cta_group::2 (half of X's rows a block) was slower, 305 us
// against 258: the hand-over of W's terms then crosses blocks.
// Terms of both operands written out and tiles of 128 x 256 -> this, all launches: 1,028 rows 1,536 -> 17,920 345 -> 254 us,
// 8,960 -> 1,536 224 -> 166; 2,048 rows 1,536 -> 17,920 547 -> 480 (235 TFLOP/s of float32, 1.4 PFLOP/s of bfloat16 products);
// 65 rows 1,536 -> 17,920 102 -> 57, 1,024 -> 1,024 37 -> 31.  Multiply-adds: 1,028 rows 1,190 and 652 us, 2,048 rows 2,278.
//
// Every wait on an mbarrier is bounded; one that runs out sets *err and the block goes on to its end.
#include <cuda_bf16.h>

#include "common.cuh"
#include "float_terms.cuh"
#include "opt_in.cuh"
#include "tcgen05.cuh"

using namespace pbe;
using namespace pbe::tc5;

namespace {
typedef __nv_bfloat16 bf16;
constexpr int BM = 128, BK = 64, UMMA_K = 16, TERMS = 3;
constexpr int SLICE = 28;                         // K blocks whose sums are added in one chain, at most
constexpr int MAX_BN = 192;                       // rows of X a tile has at most
constexpr int SPLIT_WARPS = 4, EPI_WARPS = 8, X_WARP = 12, MMA_WARP = 13, W_WARP = 14, NTHREADS = 32 * 15;

// ------------------------------------------------------------------ the terms
// planes [TERMS][rows][Kp]; a thread takes eight k of a row
__global__ void __launch_bounds__(256) split3_kernel(const float* x, bf16* planes, int rows, int K, int Kp, int vec, int* flag) {
  const int pieces = Kp / 8;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)rows * pieces) return;
  const int row = (int)(idx / pieces), k = (int)(idx - (long long)row * pieces) * 8;
  const float* src = x + (size_t)row * K + k;
  float v[8];
  if (vec && k + 8 <= K) {
    const float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = k + i < K ? src[i] : 0.f;
  }
  Sizes sizes;
  unsigned out[TERMS][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float a = v[2 * i], b = v[2 * i + 1];
    sizes.add(a);
    sizes.add(b);
#pragma unroll
    for (int t = 0; t < TERMS; ++t) {
      const __nv_bfloat162 p = __floats2bfloat162_rn(a, b);
      out[t][i] = *reinterpret_cast<const unsigned*>(&p);
      a -= __low2float(p);                          // exact: what the term leaves has fewer bits than x
      b -= __high2float(p);
    }
  }
  if (!sizes.whole()) *flag = 1;
#pragma unroll
  for (int t = 0; t < TERMS; ++t)
    *reinterpret_cast<uint4*>(planes + ((size_t)t * rows + row) * Kp + k) = make_uint4(out[t][0], out[t][1], out[t][2], out[t][3]);
}

// ------------------------------------------------------------------ the product
struct ProductParams {
  const float* bias;       // [N] or null
  float* Y;                // [parts, M, ldy]
  int M, N, Kp, ldy;
  int bn;                  // rows of X a tile, a multiple of 16 up to MAX_BN
  int parts, part_blocks;  // of K, and K blocks a part
  int* flag;               // set when an element of W is not whole in its terms
  int* err;
};

constexpr int XB = MAX_BN * BK * 2, WB = BM * BK * 4;            // a slot of X's terms, a stage of W
constexpr int X_SLOTS = 2 * TERMS, W_STAGES = 2;
constexpr int PRODUCT_SMEM = X_SLOTS * XB + W_STAGES * WB + 1024;
constexpr int A_COL = 2 * MAX_BN, TMEM_COLS = 512;               // the accumulators, then W's terms: l, m, h and the next h
static_assert(A_COL + 4 * (BK / 2) <= TMEM_COLS && PRODUCT_SMEM <= 226 * 1024, "tensor and shared memory");
__device__ __forceinline__ int slot_l() { return 0; }
__device__ __forceinline__ int slot_m() { return 1; }
__device__ __forceinline__ int slot_h(int block) { return 2 + (block & 1); }

// acc_full, a K block's end, also gives back what it read: W's term h and X's terms, of which there are two sets
struct ProductBarriers {
  uint64_t w_full[W_STAGES], w_empty[W_STAGES], a_lh_full, a_m_full, l_empty, m_empty, x_full[2], acc_full[2], acc_empty[2];
  uint32_t tmem_base;
};

__global__ void __launch_bounds__(NTHREADS, 1)
sgemm_tc5_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, ProductParams p) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* Ws = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);   // [stage][32 k][128 rows][128 B]
  unsigned char* Xs = Ws + W_STAGES * WB;                                                                  // [slot][bn rows][128 B]
  __shared__ ProductBarriers bar;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kblocks = p.Kp / BK, bn = p.bn;
  const int mtiles = (p.M + bn - 1) / bn, num_tiles = mtiles * ((p.N + BM - 1) / BM), items = num_tiles * p.parts;
  auto first_block = [&](int t) { return t / num_tiles * p.part_blocks; };
  auto last_block = [&](int t) { return min(first_block(t) + p.part_blocks, kblocks); };

  if (threadIdx.x == 0) {
    for (int i = 0; i < W_STAGES; ++i) {
      mbar_init(&bar.w_full[i], 1);
      mbar_init(&bar.w_empty[i], SPLIT_WARPS);
    }
    mbar_init(&bar.a_lh_full, SPLIT_WARPS);
    mbar_init(&bar.a_m_full, SPLIT_WARPS);
    mbar_init(&bar.l_empty, 1);
    mbar_init(&bar.m_empty, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bar.x_full[i], 1);
      mbar_init(&bar.acc_full[i], 1);
      mbar_init(&bar.acc_empty[i], EPI_WARPS);
    }
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

  if (warp < SPLIT_WARPS) {
    // -------------------------------------------------------------- W into terms: a row (tensor-memory lane) a thread
    const int row = warp * 32 + lane;
    const uint32_t a_addr = tmem_base + ((uint32_t)(warp * 32) << 16) + A_COL;
    int b = 0;                                        // K blocks so far
    bool ok = true;
    Sizes sizes;
    for (int t = blockIdx.x; t < items && ok; t += gridDim.x)
      for (int kb = first_block(t); kb < last_block(t); ++kb, ++b) {
        const int st = b % W_STAGES;
        ok = mbar_wait_warp(&bar.w_full[st], (b / W_STAGES) & 1, p.err);
        if (!ok) break;
        uint32_t w[TERMS][BK / 2];
#pragma unroll
        for (int c = 0; c < BK / 4; ++c) {
          const unsigned char* at = Ws + st * WB + (c >> 3) * (BM * 128) + row * 128 + (((c & 7) ^ (row & 7)) << 4);
          float4 v = *reinterpret_cast<const float4*>(at);
          sizes.add(v.x);
          sizes.add(v.y);
          sizes.add(v.z);
          sizes.add(v.w);
#pragma unroll
          for (int i = 0; i < TERMS; ++i) {
            w[i][2 * c] = next_term(v.x, v.y);
            w[i][2 * c + 1] = next_term(v.z, v.w);
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar.w_empty[st]);
        const int h = slot_h(b);
        // the term h of two blocks before is given back with that block's accumulator
        ok = mbar_wait_warp(&bar.l_empty, (b & 1) ^ 1, p.err) && mbar_wait_warp(&bar.acc_full[b & 1], ((b >> 1) & 1) ^ 1, p.err);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        tmem_st32_nowait(a_addr + slot_l() * (BK / 2), w[2]);
        tmem_st32_nowait(a_addr + h * (BK / 2), w[0]);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar.a_lh_full);
        ok = mbar_wait_warp(&bar.m_empty, (b & 1) ^ 1, p.err);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        tmem_st32_nowait(a_addr + slot_m() * (BK / 2), w[1]);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar.a_m_full);
      }
    if (!sizes.whole()) *p.flag = 1;
    // the commits that release the last terms arrive on this block's barriers: it stays until they have
    if (ok && b > 0) mbar_wait(&bar.l_empty, (b - 1) & 1, p.err) && mbar_wait(&bar.m_empty, (b - 1) & 1, p.err);
  } else if (warp < SPLIT_WARPS + EPI_WARPS) {
    // -------------------------------------------------------------- running sums: a row of W, half the tile's rows of X a thread
    const int quarter = warp & 3, half = (warp - SPLIT_WARPS) >> 2;
    constexpr int CHUNKS = MAX_BN / 32;
    const int chunks = bn / 16, mine = half ? chunks / 2 : (chunks + 1) / 2, c0 = half ? (chunks + 1) / 2 : 0;
    const uint32_t addr0 = tmem_base + ((uint32_t)(quarter * 32) << 16) + c0 * 16;
    int it = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < items && ok; t += gridDim.x) {
      const int tile = t % num_tiles, part = t / num_tiles;
      const int n = (tile / mtiles) * BM + quarter * 32 + lane, m0 = (tile % mtiles) * bn + c0 * 16;
      const int begin = first_block(t), end = last_block(t);
      const int rows = n < p.N ? min(p.M - m0, mine * 16) : 0;
      const int slices = (end - begin + SLICE - 1) / SLICE, slice = (end - begin + slices - 1) / slices;
      for (int k0 = begin; k0 < end && ok; k0 += slice) {
        float acc[CHUNKS * 16];
#pragma unroll
        for (int i = 0; i < CHUNKS * 16; ++i) acc[i] = 0.f;
        const int k1 = min(k0 + slice, end);
        for (int kb = k0; kb < k1; ++kb, ++it) {
          const int buf = it & 1;
          ok = mbar_wait_warp(&bar.acc_full[buf], (it >> 1) & 1, p.err);
          if (!ok) break;                             // flagged; the roles run to their end
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
          for (int c = 0; c < CHUNKS; ++c) {
            if (c < mine) {
              float v[16];
              tmem_ld16(addr0 + buf * MAX_BN + c * 16, v);
#pragma unroll
              for (int i = 0; i < 16; ++i) acc[c * 16 + i] += v[i];
            }
          }
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(&bar.acc_empty[buf]);
        }
        if (!ok) break;
        // the slices before lie in Y, written by this thread; 32 neighbouring columns a warp and row
        float* y = p.Y + ((size_t)part * p.M + m0) * p.ldy + n;
        const bool first = k0 == begin;
        const float bias = k1 == end && p.bias && n < p.N ? p.bias[n] : 0.f;
        const bool add = k1 == end && p.bias != nullptr;
#pragma unroll
        for (int i = 0; i < CHUNKS * 16; i += 8) {
          if (i >= rows) continue;
          float before[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) before[k] = !first && i + k < rows ? y[(size_t)k * p.ldy] : 0.f;
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            if (i + k < rows) {
              float v = first ? acc[i + k] : before[k] + acc[i + k];
              if (add) v += bias;
              *y = v;
            }
            y += p.ldy;
          }
          asm volatile("" ::: "memory");              // eight loads ahead, not ninety-six
        }
      }
    }
  } else if (warp == X_WARP) {
    if (lane == 0) {
      // ------------------------------------------------------------ TMA: X's terms
      int b = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < items && ok; t += gridDim.x) {
        const int m0 = (t % num_tiles % mtiles) * bn;
        for (int kb = first_block(t); kb < last_block(t); ++kb, ++b) {
          ok = mbar_wait(&bar.acc_full[b & 1], ((b >> 1) & 1) ^ 1, p.err);       // the block two before
          if (!ok) break;
          mbar_expect_tx(&bar.x_full[b & 1], TERMS * bn * BK * 2);
          // rows behind X's last belong to its next term (or are zeros): they reach no output that is written
          for (int term = 0; term < TERMS; ++term)
            tma_load_2d(Xs + ((b & 1) * TERMS + term) * XB, &map_x, kb * BK, term * p.M + m0, &bar.x_full[b & 1]);
        }
      }
    }
  } else if (warp == W_WARP) {
    if (lane == 0) {
      // ------------------------------------------------------------ TMA: W as it is
      int b = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < items && ok; t += gridDim.x) {
        const int n0 = (t % num_tiles / mtiles) * BM;
        for (int kb = first_block(t); kb < last_block(t); ++kb, ++b) {
          const int st = b % W_STAGES;
          ok = mbar_wait(&bar.w_empty[st], ((b / W_STAGES) & 1) ^ 1, p.err);
          if (!ok) break;
          mbar_expect_tx(&bar.w_full[st], WB);
          tma_load_2d(Ws + st * WB, &map_w, kb * BK, n0, &bar.w_full[st]);
          tma_load_2d(Ws + st * WB + WB / 2, &map_w, kb * BK + BK / 2, n0, &bar.w_full[st]);
        }
      }
    }
  } else if (lane == 0) {
    // -------------------------------------------------------------- MMA issuer: an accumulator a K block
    const uint32_t idesc = make_idesc(BM, bn);
    const uint64_t x_desc = make_desc(smem_u32(Xs));
    int b = 0;
    bool ok = true;
    // what block b's first products need; called before the last ones of the block before are issued, which run meanwhile
    auto ready = [&](int b) {
      return mbar_wait(&bar.acc_empty[b & 1], ((b >> 1) & 1) ^ 1, p.err) && mbar_wait(&bar.x_full[b & 1], (b >> 1) & 1, p.err) &&
             mbar_wait(&bar.a_lh_full, b & 1, p.err);
    };
    int left = 0;                                     // K blocks this thread block has in all
    for (int t = blockIdx.x; t < items; t += gridDim.x) left += last_block(t) - first_block(t);
    if (left > 0) ok = ready(0);
    for (; b < left && ok; ++b) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t tmem_d = tmem_base + (b & 1) * MAX_BN, tmem_a = tmem_base + A_COL;
      const uint64_t xb = x_desc + (uint64_t)(((b & 1) * TERMS * XB) >> 4);
      auto product = [&](int a_slot, int x_term, bool fresh) {
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k)
          umma_ts(tmem_d, tmem_a + a_slot * (BK / 2) + k * (UMMA_K / 2), xb + (uint64_t)((x_term * XB + k * UMMA_K * 2) >> 4), idesc,
                  fresh && k == 0 ? 0u : 1u);
      };
      const int h = slot_h(b);
      product(slot_l(), 0, true);
      product(h, 2, false);
      umma_commit(&bar.l_empty);
      ok = mbar_wait(&bar.a_m_full, b & 1, p.err);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      product(slot_m(), 1, false);
      product(slot_m(), 0, false);
      umma_commit(&bar.m_empty);
      product(h, 1, false);
      if (b + 1 < left) ok = ready(b + 1);
      product(h, 0, false);
      umma_commit(&bar.acc_full[b & 1]);              // the accumulator, its h terms and X's terms
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// A matrix whose rows the TMA unit cannot take (not of a multiple of 16 bytes, or misaligned), rows padded with zeros to 64 k
__global__ void __launch_bounds__(256) pad_rows_kernel(const float* w, float* out, long long rows, int K, int Kp) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows * Kp) return;
  const long long row = i / Kp;
  const int k = (int)(i - row * Kp);
  out[i] = k < K ? w[row * K + k] : 0.f;
}

// Y = the parts of K, in order, + bias
__global__ void __launch_bounds__(256) add_parts_kernel(const float* parts, int num_parts, const float* bias, float* Y, int M, int N,
                                                        int ldy) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)M * N) return;
  const int row = (int)(idx / N), n = (int)(idx - (long long)row * N);
  float v = parts[idx];
  for (int i = 1; i < num_parts; ++i) v += parts[(size_t)i * M * N + idx];
  Y[(size_t)row * ldy + n] = bias ? v + bias[n] : v;
}

int multiprocessors() {
  static int n = 0;
  if (n == 0) {
    int dev = 0, got = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&got, cudaDevAttrMultiProcessorCount, dev);
    n = got > 0 ? got : 148;
  }
  return n;
}

// [rows, K] row-major float32, rows ld elements apart, boxes of BM rows x 32, 128-byte swizzle, zeros outside
int make_map_f32(CUtensorMap* map, const float* base, int rows, int K, int ld) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return (int)cudaErrorNotSupported;
  cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
  cuuint32_t box[2] = {32, (cuuint32_t)BM};
  cuuint32_t estr[2] = {1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : (int)cudaErrorInvalidValue;
}

int launch_product(const CUtensorMap& map_w, const CUtensorMap& map_x, const ProductParams& p, cudaStream_t stream) {
  static OptIn opt_in;
  if (const cudaError_t e = opt_in(PRODUCT_SMEM, sgemm_tc5_kernel)) return (int)e;
  const long long tiles = (long long)((p.M + p.bn - 1) / p.bn) * ((p.N + BM - 1) / BM) * p.parts;
  const int blocks = (int)(tiles < multiprocessors() ? tiles : multiprocessors());
  sgemm_tc5_kernel<<<blocks, NTHREADS, PRODUCT_SMEM, stream>>>(map_w, map_x, p);
  return launch_status();
}

int split3(const float* x, bf16* planes, int rows, int K, int Kp, int* flag, cudaStream_t stream) {
  const long long threads = (long long)rows * (Kp / 8);
  const int vec = K % 4 == 0 && ((uintptr_t)x & 15) == 0;
  split3_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, stream>>>(x, planes, rows, K, Kp, vec, flag);
  return launch_status();
}

int padded(int K) { return (K + BK - 1) / BK * BK; }

// Rows of W that are padded and multiplied at a time, where they have to be: all, unless they would take more than 256 MB.
int columns_at_a_time(int N, int Kp) {
  const long long most = (256LL << 20) / ((long long)Kp * 4) / BM * BM;
  return most < BM ? (N < BM ? N : BM) : (int)(N < most ? N : most);
}

// Rows of X whose terms are made at a time: all, unless they would take more than 256 MB, else groups of one size, about.
int rows_at_a_time(int M, int Kp) {
  const long long most = (256LL << 20) / ((long long)TERMS * Kp * 2) / 16 * 16;
  if (M <= most || M <= 16) return M;
  const long long groups = most < 16 ? (M + 15) / 16 : (M + most - 1) / most;
  return (int)(((M + groups - 1) / groups + 15) / 16 * 16);
}

// How M x N outputs over K are cut: the rows of X a tile has and the parts of K that take least by this count (microseconds, as
// measured: a K block of a tile, its start and end, the parts' way through memory).
struct Plan {
  int bn, parts, part_blocks;
  float us;
};

Plan plan_of(int M, int N, int Kp) {
  const int kblocks = Kp / BK, sms = multiprocessors();
  Plan best{0, 1, kblocks, 0.f};
  const int fewest = (M + MAX_BN - 1) / MAX_BN;
  int before = 0;
  for (int mtiles = fewest; mtiles < fewest + 4; ++mtiles) {
    const int bn = ((M + mtiles - 1) / mtiles + 15) / 16 * 16;
    if (bn == before) continue;
    before = bn;
    const long long tiles = (long long)((M + bn - 1) / bn) * ((N + BM - 1) / BM);
    const float block_us = 1.1f + bn * 0.0025f;
    for (int parts = 1; parts <= 8; ++parts) {
      const int per = (kblocks + parts - 1) / parts;
      const long long bytes = (long long)parts * M * N * 4;
      if (parts > 1 && (per < 8 || (long long)per * (parts - 1) >= kblocks || bytes > (128LL << 20))) continue;
      const long long waves = (tiles * parts + sms - 1) / sms;
      const float us = (float)waves * (float)per * block_us + 4.f + (parts > 1 ? 4.f + (float)bytes * 2.f / 4e6f : 0.f);
      if (best.bn == 0 || us < best.us) best = Plan{bn, parts, per, us};
    }
  }
  return best;
}

long long aligned256(long long bytes) { return (bytes + 255) / 256 * 256; }
long long part_bytes(const Plan& plan, int M, int N) { return plan.parts > 1 ? aligned256((long long)plan.parts * M * N * 4) : 0; }
bool takes_rows(int K) { return K % 4 == 0; }              // can the TMA unit take W's rows where they lie?
}  // namespace

namespace {
long long scratch_bytes(int M, int N, int K, bool pad) {
  const int Kp = padded(K), columns = pad ? columns_at_a_time(N, Kp) : N, rows = rows_at_a_time(M, Kp);
  long long parts = 0;
  for (const int m : {rows, M % rows})                   // the groups' sizes
    for (const int n : {columns, N % columns})
      if (m > 0 && n > 0) {
        const long long bytes = part_bytes(plan_of(m, n, Kp), m, n);
        if (bytes > parts) parts = bytes;
      }
  return 256 + aligned256((long long)rows * TERMS * Kp * 2) + (pad ? aligned256((long long)columns * Kp * 4) : 0) + parts;
}
}  // namespace

// Bytes of scratch memory, 256-byte aligned, that pbe_sgemm_tc5 needs: the flag, X's terms, W's padded rows where the TMA unit
// cannot take them where they lie, the parts' sums; at most 256 + 256 + 128 MB whatever M and N are (K up to 500,000, where 128 rows
// of W and 80 rows' terms take 256 MB).  _padded: for a W that does not start on a 16-byte boundary.
PBE_EXPORT long long pbe_sgemm_tc5_scratch(int M, int N, int K) { return scratch_bytes(M, N, K, !takes_rows(K)); }
PBE_EXPORT long long pbe_sgemm_tc5_scratch_padded(int M, int N, int K) { return scratch_bytes(M, N, K, true); }

// X [M, K], W [N, K], Y [M, N], float32, contiguous.  Afterwards the first int of scratch says whether an element was not
// finite, too large or too small: Y is then to be made by pbe_sgemm_nt_if.
// err: device int, set to 1 if a bounded wait ran out (the result is then invalid).
PBE_EXPORT int pbe_sgemm_tc5(const float* X, const float* W, const float* bias, float* Y, int M, int N, int K, void* scratch,
                             int* err, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || scratch == nullptr || ((uintptr_t)scratch & 255)) return (int)cudaErrorInvalidValue;
  if ((long long)M * TERMS > 0x7fffffffLL - 512 || N > 0x7fffffff - 512 || K > 0x7fffffff - BK) return (int)cudaErrorInvalidValue;
  const bool pad = !takes_rows(K) || ((uintptr_t)W & 15);
  const int Kp = padded(K), columns = pad ? columns_at_a_time(N, Kp) : N, rows = rows_at_a_time(M, Kp);
  int* flag = (int*)scratch;
  bf16* xt = (bf16*)((char*)scratch + 256);
  float* wp = (float*)((char*)xt + aligned256((long long)rows * TERMS * Kp * 2));
  float* sums = (float*)((char*)wp + (pad ? aligned256((long long)columns * Kp * 4) : 0));
  const cudaError_t e = cudaMemsetAsync(flag, 0, sizeof(int), stream);
  if (e != cudaSuccess) return (int)e;
  int rc = 0;
  CUtensorMap map_x, map_w;
  for (int m0 = 0; m0 < M && rc == 0; m0 += rows) {
    const int m = M - m0 < rows ? M - m0 : rows;
    rc = split3(X + (size_t)m0 * K, xt, m, K, Kp, flag, stream);
    for (int n0 = 0; n0 < N && rc == 0; n0 += columns) {
      const int n = N - n0 < columns ? N - n0 : columns;
      const float* w = W + (size_t)n0 * K;
      if (pad) {
        if (m0 == 0 || columns < N) {
          pad_rows_kernel<<<(unsigned)(((long long)n * Kp + 255) / 256), 256, 0, stream>>>(w, wp, n, K, Kp);
          rc = launch_status();
        }
        w = wp;
      }
      const Plan plan = plan_of(m, n, Kp);
      if (rc == 0) rc = make_map(&map_x, xt, m * TERMS, Kp, plan.bn);
      if (rc == 0) rc = pad ? make_map_f32(&map_w, w, n, Kp, Kp) : make_map_f32(&map_w, w, n, K, K);
      if (rc != 0) break;
      const bool parts = plan.parts > 1;
      float* out = Y + (size_t)m0 * N + n0;
      const float* b = bias ? bias + n0 : nullptr;
      const ProductParams p{parts ? nullptr : b, parts ? sums : out, m, n, Kp, parts ? n : N, plan.bn, plan.parts, plan.part_blocks,
                            flag, err};
      rc = launch_product(map_w, map_x, p, stream);
      if (rc == 0 && parts) {
        add_parts_kernel<<<(unsigned)(((long long)m * n + 255) / 256), 256, 0, stream>>>(sums, plan.parts, b, out, m, n, N);
        rc = launch_status();
      }
    }
  }
  return rc;
}
