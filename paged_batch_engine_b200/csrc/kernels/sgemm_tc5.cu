// The float32 product Y[M, N] = X[M, K] * W[N, K]^T (+ bias[N]) of many rows on the fifth-generation tensor cores, with
// float32's precision: every operand is cut into three bfloat16 terms, x = h + m + l, |m| <= 2^-8 |x| and |l| <= 2^-17 |x|,
// which hold all of its 24 bits, and the six products hh, hm, mh, mm, hl, lh are added; ml and lm, which are left out, are
// 2^-25 of a product each at most, together as large as the rounding of the multiply-add that they stand for.
//
// The tensor cores add in float32 but cut off what does not fit instead of rounding it, so a sum is not left to them
// for long: after every 64 k the accumulator in tensor memory starts anew, the small products are issued before hh, and the epilogue's warps add its contents to the tile's running sums in registers, with a rounding
// add each; after 2,048 k the running sums are added to the output.  Against 64 bits, relative root mean square error of
// sgemm.cu's multiply-adds -> this: normal numbers 4.1e-7 -> 1.2e-7 (K = 1,536) and 1.4e-7 (8,960, 19,200), positive ones
// 2.1e-7 -> 1.1e-7 and 1.1e-7 -> 1.0e-7; a float32 model's logits after 1,028 prompt tokens 2.8e-6 -> 2.5e-6.  Where single
// products outweigh all others (factors spread over e^3) both are at the last bit: 0.5-1.5e-7 and 0.7-1.4e-7.
//
// Two kernels a product:
//  * split3: an operand's three terms as bfloat16 matrices one below the other, rows padded with zeros to 64 k; bound by
//    memory (4 bytes in, 6 out).  It also tells whether an element is other than zero or of a size from SMALLEST to
//    LARGEST: such a product is left to sgemm.cu, whose kernel is launched behind and looks at the flag.  A smaller one's
//    third term would fall under bfloat16's smallest normal number, larger ones' products could overflow with either sign
//    where their sum does not, and an infinity times a term that is zero would be no number.
//  * the product: persistent blocks walk over tiles of 128 x BN, or over parts of K of such tiles where there are too few
//    (a small kernel adds the parts in order); warp 0 is the TMA producer, warp 1 issues the MMAs (128 x BN x 16), warps
//    2-9 hold the running sums, half a tile row a thread, and write them out.  Two accumulators alternate.  What bounds
//    it is the tensor pipe, six products of the bfloat16 rate.  A slot of the ring holds one term of A and of W, 64 k
//    wide (boxes 32 k wide, a stage with all terms a slot, were bound by the TMA unit, two cycles a row of 64 bytes:
//    1,028 x 17,920 x 1,536 395 us); the terms come in the order l, h, m, so that a slot is free again after 8, 20 and 24
//    of a block's 24 MMAs and each load has the time of a dozen MMAs or more.
// Multiply-adds -> this, all launches: 1,028 rows 1,536 -> 17,920 1,190 -> 342 us, 8,960 -> 1,536 652 -> 223; 2,048 rows
// 1,536 -> 17,920 2,278 -> 543 (208 TFLOP/s of float32, 1.25 PFLOP/s of bfloat16 products; a tile's operands out of L2 are
// the next bound: 24 blocks of one wave take 1.6 us each, of eight waves 2.4); 65 rows 1,024 -> 1,024 66 -> 39.
//
// Every wait on an mbarrier is bounded; one that runs out sets *err and the block goes on to its end.
#include <cuda_bf16.h>

#include "common.cuh"
#include "tcgen05.cuh"

using namespace pbe;
using namespace pbe::tc5;

namespace {
typedef __nv_bfloat16 bf16;
constexpr int BM = 128, BK = 64, UMMA_K = 16, TERMS = 3;
constexpr int SLICE = 2048 / BK;                  // K blocks whose sums are added in one chain
constexpr int EPI_WARPS = 8, NTHREADS = 64 + 32 * EPI_WARPS;
constexpr float SMALLEST = 0x1p-102f;              // its last bit, 2^-125, is a bfloat16 number
constexpr float LARGEST = 0x1p47f;                 // a sum of 2^31 products of two such numbers stays below 2^127

// ------------------------------------------------------------------ the terms
__device__ __forceinline__ bool whole_in_terms(float x) { return x == 0.f || (fabsf(x) >= SMALLEST && fabsf(x) <= LARGEST); }

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
  bool plain = true;
  unsigned out[TERMS][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float a = v[2 * i], b = v[2 * i + 1];
    plain = plain && whole_in_terms(a) && whole_in_terms(b);
#pragma unroll
    for (int t = 0; t < TERMS; ++t) {
      const __nv_bfloat162 p = __floats2bfloat162_rn(a, b);
      out[t][i] = *reinterpret_cast<const unsigned*>(&p);
      a -= __low2float(p);                          // exact: what the term leaves has fewer bits than x
      b -= __high2float(p);
    }
  }
  if (!plain) *flag = 1;
#pragma unroll
  for (int t = 0; t < TERMS; ++t)
    *reinterpret_cast<uint4*>(planes + ((size_t)t * rows + row) * Kp + k) = make_uint4(out[t][0], out[t][1], out[t][2], out[t][3]);
}

// ------------------------------------------------------------------ the product
struct ProductParams {
  const float* bias;       // [N] or null
  float* Y;                // [parts, M, ldy]
  int M, N, Kp, ldy, aligned;
  int parts, part_blocks;  // of K, and K blocks a part
  int* err;
};

template <int BN> __host__ __device__ constexpr int slot_bytes() { return (BM + BN) * BK * 2; }
template <int BN> __host__ __device__ constexpr int num_slots() { return BN == 256 ? 4 : 6; }

template <int BN>
__global__ void __launch_bounds__(NTHREADS, 1)
sgemm_tc5_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, ProductParams p) {
  constexpr int SLOTS = num_slots<BN>(), A_BYTES = BM * BK * 2, SLOT_BYTES = slot_bytes<BN>();
  constexpr int TMEM_COLS = 2 * BN, HALF = BN / 2;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* slots = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full_bar[SLOTS];
  __shared__ __align__(8) uint64_t empty_bar[SLOTS];
  __shared__ __align__(8) uint64_t acc_full[2];
  __shared__ __align__(8) uint64_t acc_empty[2];
  __shared__ uint32_t tmem_base_smem;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kblocks = p.Kp / BK;
  const int mtiles = (p.M + BM - 1) / BM, num_tiles = mtiles * ((p.N + BN - 1) / BN), items = num_tiles * p.parts;

  if (threadIdx.x == 0) {
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], EPI_WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&tmem_base_smem)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = tmem_base_smem;

  if (warp == 0) {
    if (lane == 0) {
      // ------------------------------------------------------------ TMA producer
      int it = 0;                                   // slots filled
      bool ok = true;
      for (int t = blockIdx.x; t < items && ok; t += gridDim.x) {
        const int tile = t % num_tiles, k0 = t / num_tiles * p.part_blocks, k1 = min(k0 + p.part_blocks, kblocks);
        const int m0 = (tile % mtiles) * BM, n0 = (tile / mtiles) * BN;
        for (int kb = k0; kb < k1 && ok; ++kb) {
#pragma unroll
          for (int i = 0; i < TERMS; ++i, ++it) {
            const int term = i == 0 ? 2 : i - 1;    // l, h, m
            const int s = it % SLOTS;
            ok = mbar_wait(&empty_bar[s], ((it / SLOTS) & 1) ^ 1, p.err);
            if (!ok) break;
            unsigned char* a = slots + (size_t)s * SLOT_BYTES;
            mbar_expect_tx(&full_bar[s], SLOT_BYTES);
            // rows behind an operand's last belong to its next term (or are zeros): they reach no output that is written
            tma_load_2d(a + A_BYTES, &map_w, kb * BK, term * p.N + n0, &full_bar[s]);
            tma_load_2d(a, &map_a, kb * BK, term * p.M + m0, &full_bar[s]);
          }
        }
      }
      // the commits that release the last slots arrive on this block's barriers: it stays until they have
      for (int q = it > SLOTS ? it - SLOTS : 0; q < it && ok; ++q)
        ok = mbar_wait(&empty_bar[q % SLOTS], (q / SLOTS) & 1, p.err);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // ------------------------------------------------------------ MMA issuer: an accumulator a K block
      const uint32_t idesc = make_idesc(BM, BN);
      int it = 0, blocks = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < items && ok; t += gridDim.x) {
        const int k0 = t / num_tiles * p.part_blocks, k1 = min(k0 + p.part_blocks, kblocks);
        for (int kb = k0; kb < k1; ++kb, ++blocks, it += TERMS) {
          const int buf = blocks & 1, sl = it % SLOTS, sh = (it + 1) % SLOTS, sm = (it + 2) % SLOTS;
          ok = mbar_wait(&acc_empty[buf], ((blocks >> 1) & 1) ^ 1, p.err) &&
               mbar_wait(&full_bar[sl], (it / SLOTS) & 1, p.err) &&
               mbar_wait(&full_bar[sh], ((it + 1) / SLOTS) & 1, p.err);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t tmem_d = tmem_base + buf * BN, base = smem_u32(slots);
          const uint32_t l = base + sl * SLOT_BYTES, h = base + sh * SLOT_BYTES, m = base + sm * SLOT_BYTES;
          auto product = [&](uint32_t a, uint32_t b, bool fresh) {
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k)
              umma(tmem_d, make_desc(a + k * UMMA_K * 2), make_desc(b + A_BYTES + k * UMMA_K * 2), idesc, fresh && k == 0 ? 0u : 1u);
          };
          product(l, h, true);
          product(h, l, false);
          umma_commit(&empty_bar[sl]);
          ok = mbar_wait(&full_bar[sm], ((it + 2) / SLOTS) & 1, p.err);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          product(m, m, false);
          product(m, h, false);
          product(h, m, false);
          umma_commit(&empty_bar[sm]);
          product(h, h, false);
          umma_commit(&empty_bar[sh]);
          umma_commit(&acc_full[buf]);
        }
      }
    }
  } else {
    // -------------------------------------------------------------- running sums, warps 2..9
    const int quarter = warp & 3;                   // the tensor-memory lanes this warp may read
    const int half = (warp - 2) >> 2;               // of the tile's columns
    int it = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < items && ok; t += gridDim.x) {
      const int tile = t % num_tiles, part = t / num_tiles;
      const int row = (tile % mtiles) * BM + quarter * 32 + lane, n0 = (tile / mtiles) * BN + half * HALF;
      const int begin = part * p.part_blocks, end = min(begin + p.part_blocks, kblocks);
      float* y = p.Y + ((size_t)part * p.M + row) * p.ldy + n0;
      for (int k0 = begin; k0 < end && ok; k0 += SLICE) {
        float acc[HALF];
#pragma unroll
        for (int i = 0; i < HALF; ++i) acc[i] = 0.f;
        const int k1 = min(k0 + SLICE, end);
        for (int kb = k0; kb < k1; ++kb, ++it) {
          const int buf = it & 1;
          ok = mbar_wait(&acc_full[buf], (it >> 1) & 1, p.err);
          if (!ok) break;                             // flagged; the roles run to their end
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t addr = tmem_base + ((uint32_t)(quarter * 32) << 16) + buf * BN + half * HALF;
#pragma unroll
          for (int c = 0; c < HALF / 32; ++c) {
            float v[32];
            tmem_ld32(addr + c * 32, v);
#pragma unroll
            for (int i = 0; i < 32; ++i) acc[c * 32 + i] += v[i];
          }
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(&acc_empty[buf]);
        }
        if (!ok || row >= p.M) continue;
        // the slices before lie in Y, written by this thread
        const bool first = k0 == begin, last = k1 == end;
#pragma unroll
        for (int i = 0; i < HALF; i += 4) {
          if (n0 + i >= p.N) break;
          if (p.aligned && n0 + i + 4 <= p.N) {
            float4* at = reinterpret_cast<float4*>(y + i);
            float4 v = make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
            if (!first) {
              const float4 u = *at;
              v = make_float4(u.x + v.x, u.y + v.y, u.z + v.z, u.w + v.w);
            }
            if (last && p.bias) {
              v.x += p.bias[n0 + i];
              v.y += p.bias[n0 + i + 1];
              v.z += p.bias[n0 + i + 2];
              v.w += p.bias[n0 + i + 3];
            }
            *at = v;
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              if (n0 + i + j >= p.N) break;
              float v = first ? acc[i + j] : y[i + j] + acc[i + j];
              if (last && p.bias) v += p.bias[n0 + i + j];
              y[i + j] = v;
            }
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
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

template <int BN>
int launch_product(const CUtensorMap& map_a, const CUtensorMap& map_w, const ProductParams& p, cudaStream_t stream) {
  const int smem = num_slots<BN>() * slot_bytes<BN>() + 1024;
  const cudaError_t e = cudaFuncSetAttribute(sgemm_tc5_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  const long long tiles = (long long)((p.M + BM - 1) / BM) * ((p.N + BN - 1) / BN) * p.parts;
  const int blocks = (int)(tiles < multiprocessors() ? tiles : multiprocessors());
  sgemm_tc5_kernel<BN><<<blocks, NTHREADS, smem, stream>>>(map_a, map_w, p);
  return launch_status();
}

int split3(const float* x, bf16* planes, int rows, int K, int Kp, int* flag, cudaStream_t stream) {
  const long long threads = (long long)rows * (Kp / 8);
  const int vec = K % 4 == 0 && ((uintptr_t)x & 15) == 0;
  split3_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, stream>>>(x, planes, rows, K, Kp, vec, flag);
  return launch_status();
}

int padded(int K) { return (K + BK - 1) / BK * BK; }

// Columns of W whose terms are made and multiplied at a time: all, unless the terms would take more than 256 MB (the
// 1.5B model's gate and up matrix takes 165, a vocabulary of 152 thousand 1,400).
int columns_at_a_time(int N, int Kp) {
  const long long most = (256LL << 20) / ((long long)TERMS * Kp * 2) / 256 * 256;
  return most < 256 ? (N < 256 ? N : 256) : (int)(N < most ? N : most);
}

// Rows of X whose terms are made at a time: all, unless they would take more than 256 MB, else groups of whole tiles and about
// one size (2,304 rows and more for K up to 18,944, so that making W's terms once more for each costs a tenth at most).
int rows_at_a_time(int M, int Kp) {
  const long long most = (256LL << 20) / ((long long)TERMS * Kp * 2) / BM * BM;
  if (M <= most || M <= BM) return M;
  const long long groups = most < BM ? (M + BM - 1) / BM : (M + most - 1) / most;
  return (int)(((M + groups - 1) / groups + BM - 1) / BM * BM);
}

// How M x N outputs over K are cut: the tiles' columns and the parts of K that take least by this count (microseconds, as
// measured: a K block of a tile, its start and end, the parts' way through memory).
struct Plan {
  int bn, parts, part_blocks;
  float us;
};

Plan plan_of(int M, int N, int Kp) {
  const int kblocks = Kp / BK, sms = multiprocessors();
  Plan best{0, 1, kblocks, 0.f};
  for (int bn = 256; bn >= 128; bn -= 128) {
    const long long tiles = (long long)((M + BM - 1) / BM) * ((N + bn - 1) / bn);
    for (int parts = 1; parts <= 8; ++parts) {
      const int per = (kblocks + parts - 1) / parts;
      const long long bytes = (long long)parts * M * N * 4;
      if (parts > 1 && (per < 8 || (long long)per * (parts - 1) >= kblocks || bytes > (128LL << 20))) continue;
      const long long waves = (tiles * parts + sms - 1) / sms;
      const float us = (float)waves * ((float)per * (bn == 256 ? 1.9f : 1.0f) + 4.f) + (parts > 1 ? 4.f + (float)bytes * 2.f / 4e6f : 0.f);
      if (best.bn == 0 || us < best.us) best = Plan{bn, parts, per, us};
    }
  }
  return best;
}

long long aligned256(long long bytes) { return (bytes + 255) / 256 * 256; }
long long part_bytes(const Plan& plan, int M, int N) { return plan.parts > 1 ? aligned256((long long)plan.parts * M * N * 4) : 0; }
}  // namespace

// Rows of M that pbe_sgemm_tc5 should be given: without those behind the last whole tile of 128, where a tile row of
// their own would cost more than pbe_sgemm_nt's streaming of the weights for up to sixteen rows.
PBE_EXPORT int pbe_sgemm_tc5_rows(int M, int N, int K) {
  const int rest = M % BM, Kp = padded(K);
  if (M <= BM || rest < 1 || rest > 16) return M;
  const float stream_us = 8.f + (float)N * (float)K * 4.f / 4.5e6f;
  return plan_of(M - rest, N, Kp).us + stream_us < plan_of(M, N, Kp).us ? M - rest : M;
}

// Bytes of scratch memory, 256-byte aligned, that pbe_sgemm_tc5 needs: the flag, X's terms, W's terms, the parts' sums; at
// most 256 + 256 + 128 MB whatever M and N are (K up to 174,762, where 256 rows' or columns' terms take 256 MB).
PBE_EXPORT long long pbe_sgemm_tc5_scratch(int M, int N, int K) {
  const int Kp = padded(K), columns = columns_at_a_time(N, Kp), rows = rows_at_a_time(M, Kp);
  long long parts = 0;
  for (const int m : {rows, M % rows})                   // the groups' sizes
    for (const int n : {columns, N % columns})
      if (m > 0 && n > 0) {
        const long long bytes = part_bytes(plan_of(m, n, Kp), m, n);
        if (bytes > parts) parts = bytes;
      }
  return 256 + aligned256((long long)rows * TERMS * Kp * 2) + aligned256((long long)columns * TERMS * Kp * 2) + parts;
}

// X [M, K], W [N, K], Y [M, N], float32, contiguous.  Afterwards the first int of scratch says whether an element was not
// finite, too large or too small: Y is then to be made by pbe_sgemm_nt_if.
// err: device int, set to 1 if a bounded wait ran out (the result is then invalid).
PBE_EXPORT int pbe_sgemm_tc5(const float* X, const float* W, const float* bias, float* Y, int M, int N, int K, void* scratch,
                             int* err, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || scratch == nullptr || ((uintptr_t)scratch & 255)) return (int)cudaErrorInvalidValue;
  if ((long long)M * TERMS > 0x7fffffffLL - 512 || (long long)N * TERMS > 0x7fffffffLL - 512 || K > 0x7fffffff - BK)
    return (int)cudaErrorInvalidValue;
  const int Kp = padded(K), columns = columns_at_a_time(N, Kp), rows = rows_at_a_time(M, Kp);
  int* flag = (int*)scratch;
  bf16* xt = (bf16*)((char*)scratch + 256);
  bf16* wt = (bf16*)((char*)xt + aligned256((long long)rows * TERMS * Kp * 2));
  float* sums = (float*)((char*)wt + aligned256((long long)columns * TERMS * Kp * 2));
  const cudaError_t e = cudaMemsetAsync(flag, 0, sizeof(int), stream);
  if (e != cudaSuccess) return (int)e;
  int rc = 0;
  CUtensorMap map_a, map_w;
  for (int m0 = 0; m0 < M && rc == 0; m0 += rows) {
    const int m = M - m0 < rows ? M - m0 : rows;
    rc = split3(X + (size_t)m0 * K, xt, m, K, Kp, flag, stream);
    if (rc == 0) rc = make_map(&map_a, xt, m * TERMS, Kp, BM);
    for (int n0 = 0; n0 < N && rc == 0; n0 += columns) {
      const int n = N - n0 < columns ? N - n0 : columns;
      if (m0 == 0 || columns < N) rc = split3(W + (size_t)n0 * K, wt, n, K, Kp, flag, stream);
      const Plan plan = plan_of(m, n, Kp);
      if (rc == 0) rc = make_map(&map_w, wt, n * TERMS, Kp, plan.bn);
      if (rc != 0) break;
      const bool parts = plan.parts > 1;
      float* out = Y + (size_t)m0 * N + n0;
      float* y = parts ? sums : out;
      const int ldy = parts ? n : N;
      const float* b = bias ? bias + n0 : nullptr;
      const ProductParams p{parts ? nullptr : b, y, m, n, Kp, ldy, (ldy % 4 == 0 && ((uintptr_t)y & 15) == 0) ? 1 : 0,
                            plan.parts, plan.part_blocks, err};
      rc = plan.bn == 128 ? launch_product<128>(map_a, map_w, p, stream) : launch_product<256>(map_a, map_w, p, stream);
      if (rc == 0 && parts) {
        add_parts_kernel<<<(unsigned)(((long long)m * n + 255) / 256), 256, 0, stream>>>(sums, plan.parts, b, out, m, n, N);
        rc = launch_status();
      }
    }
  }
  return rc;
}
