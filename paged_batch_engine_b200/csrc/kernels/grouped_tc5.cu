// The experts' products on the fifth-generation tensor cores: rows sorted by expert, every expert's run
// padded to whole tiles of 128 rows, out[row] = W_g a[row] for the rows of every tile (group g), in one launch
// for all experts.  tcgen05.mma of 128 x 256 x 16, operands staged by TMA (128-byte swizzle, no multicast), the
// float32 accumulator in tensor memory, read back with tcgen05.ld for the epilogue.
//
// What bounds it: with hundreds of rows an expert, the tensor pipe and the tiles' way from L2 into shared memory
// (48 KB for 4.2 MFLOP); with a few rows an expert, reading every chosen expert's weights once.  A persistent block a
// multiprocessor walks over the tiles; the tiles of one column block of all experts are neighbours in that order,
// so the two or three row tiles of an expert read its weight tile at the same time (L2), and a wave touches every
// expert.  Warp 0 is the TMA producer (four stages of A 128 x 64 and W 256 x 64), warp 1 issues the MMAs, warps
// 2-5 are the epilogue; two accumulators alternate, so a tile's epilogue overlaps the next tile's products.
//
// Epilogues: none, relu squared, and gates (W_g = [gate rows; up rows]: a tile takes 128 of each, a thread holds
// the gate and the up value of an output, so the activation costs no pass over memory and sees float32 sums).
//
// 2,048 rows, 4 of 32 experts, 2,048 -> 2 x 1,408 -> 2,048: 113 + 65 us, 0.80 PFLOP/s without the padding rows;
// the mma.sync products of grouped_gemm.cu and the activation's own pass took 826 + 95.  16 rows (weights read once,
// 4.9 TB/s): the whole feed-forward 319 -> 135 us; 100 rows 325 -> 141, 512 rows 391 -> 147.
//
// Every wait on an mbarrier is bounded; one that runs out sets *err and the block goes on to its end.
#include <cuda_bf16.h>

#include "common.cuh"
#include "pdl.cuh"
#include "tcgen05.cuh"

using namespace pbe;
using namespace pbe::tc5;

namespace {
typedef __nv_bfloat16 bf16;
constexpr int BM = 128, BN = 256, BK = 64, UMMA_K = 16, STAGES = 4;
constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int NTHREADS = 192, TMEM_COLS = 512;

enum Epilogue { PLAIN = 0, RELU2 = 1, SILU_GLU = 2, CAPPED_GLU = 3 };

struct GroupedParams {
  bf16* out;
  int N;               // rows of a group's matrix
  int N_out;           // columns of the output (N, or N / 2 with a gate)
  int K;
  const int32_t* tiles;   // [max_tiles, 3]: group (-1: idle, behind all live ones), first row, rows; null: one group, all rows
  int rows;
  int max_tiles;
  float limit, alpha;     // of the capped gate
  int* err;
};

// 32 consecutive outputs of one row; whole 16-byte pieces where the row lies on them
__device__ __forceinline__ void store_row32(bf16* dst, const float (&v)[32], int valid, bool aligned) {
  if (valid >= 32 && aligned) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      unsigned w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        __nv_bfloat162 h = __floats2bfloat162_rn(v[i * 8 + 2 * j], v[i * 8 + 2 * j + 1]);
        w[j] = *reinterpret_cast<unsigned*>(&h);
      }
      reinterpret_cast<uint4*>(dst)[i] = make_uint4(w[0], w[1], w[2], w[3]);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (i < valid) dst[i] = __float2bfloat16_rn(v[i]);
  }
}

template <int EPI>
__global__ void __launch_bounds__(NTHREADS, 1)
grouped_tc5_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, GroupedParams p) {
  constexpr bool GLU = EPI == SILU_GLU || EPI == CAPPED_GLU;
  constexpr int COLS = GLU ? 128 : BN;          // output columns of a tile
  extern __shared__ unsigned char smem_raw[];
  unsigned char* stages = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full_bar[STAGES];
  __shared__ __align__(8) uint64_t empty_bar[STAGES];
  __shared__ __align__(8) uint64_t acc_full[2];
  __shared__ __align__(8) uint64_t acc_empty[2];
  __shared__ uint32_t tmem_base_smem;
  __shared__ int live_smem;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kblocks = (p.K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    live_smem = 0;
#pragma unroll
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 4);          // one arrival per epilogue warp
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {   // tensor memory: all 512 columns, allocated and later freed by this warp
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&tmem_base_smem)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  __syncthreads();
  pdl_wait();          // the tile list and the rows come from the kernels before
  // the live tiles stand at the front of the list
  for (int i = threadIdx.x; i < p.max_tiles; i += NTHREADS)
    if (p.tiles == nullptr || p.tiles[3 * i] >= 0) atomicAdd(&live_smem, 1);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = tmem_base_smem;
  const int live = live_smem;
  const int num_tiles = live * ((p.N_out + COLS - 1) / COLS);

  if (warp == 0) {
    if (lane == 0) {
      // ------------------------------------------------------------ TMA producer
      int it = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
        const int32_t* tile = p.tiles ? p.tiles + 3 * (t % live) : nullptr;
        const int n0 = (t / live) * COLS;
        const int m0 = tile ? tile[1] : (t % live) * BM;
        const int wrow0 = (tile ? tile[0] * p.N : 0) + n0;
        const int wrow1 = wrow0 + (GLU ? p.N_out : 128);
        for (int kb = 0; kb < kblocks; ++kb, ++it) {
          const int s = it % STAGES;
          ok = mbar_wait(&empty_bar[s], ((it / STAGES) & 1) ^ 1, p.err);
          if (!ok) break;
          unsigned char* a = stages + (size_t)s * STAGE_BYTES;
          unsigned char* b = a + A_BYTES;
          mbar_expect_tx(&full_bar[s], STAGE_BYTES);
          tma_load_2d(b, &map_w, kb * BK, wrow0, &full_bar[s]);
          tma_load_2d(b + 128 * BK * 2, &map_w, kb * BK, wrow1, &full_bar[s]);
          tma_load_2d(a, &map_a, kb * BK, m0, &full_bar[s]);
        }
      }
      // the commits that release the last stages arrive on this block's barriers: it stays until they have
      for (int q = it > STAGES ? it - STAGES : 0; q < it && ok; ++q)
        ok = mbar_wait(&empty_bar[q % STAGES], (q / STAGES) & 1, p.err);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // ------------------------------------------------------------ MMA issuer
      const uint32_t idesc = make_idesc(BM, BN);
      int it = 0, j = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x, ++j) {
        const int buf = j & 1;
        ok = mbar_wait(&acc_empty[buf], ((j >> 1) & 1) ^ 1, p.err);   // the epilogue has drained this accumulator
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tmem_d = tmem_base + buf * BN;
        for (int kb = 0; kb < kblocks && ok; ++kb, ++it) {
          const int s = it % STAGES;
          ok = mbar_wait(&full_bar[s], (it / STAGES) & 1, p.err);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a_addr = smem_u32(stages + (size_t)s * STAGE_BYTES);
          const uint32_t b_addr = a_addr + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            umma(tmem_d, make_desc(a_addr + k * UMMA_K * 2), make_desc(b_addr + k * UMMA_K * 2), idesc,
                 (kb > 0 || k > 0) ? 1u : 0u);
          umma_commit(&empty_bar[s]);      // the stage is free once these MMAs have read it
        }
        umma_commit(&acc_full[buf]);       // this tile's accumulator is complete
      }
    }
  } else {
    // -------------------------------------------------------------- epilogue warps 2..5
    const int quarter = warp & 3;          // the TMEM lanes this warp may read
    const bool aligned = (p.N_out % 8) == 0;
    int j = 0;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x, ++j) {
      const int32_t* tile = p.tiles ? p.tiles + 3 * (t % live) : nullptr;
      const int n0 = (t / live) * COLS;
      const int m0 = tile ? tile[1] : (t % live) * BM;
      const int rows = tile ? tile[2] : min(BM, p.rows - m0);
      const int buf = j & 1;
      const int r = quarter * 32 + lane;
      const bool row_live = r < rows;
      bf16* yrow = p.out + (size_t)(m0 + r) * p.N_out;
      if (!mbar_wait(&acc_full[buf], (j >> 1) & 1, p.err)) break;      // flagged; the roles run to their end
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16) + buf * BN;
      // rows beyond the tile's are padding: a warp without a live row reads nothing back
      if (quarter * 32 < rows) {
#pragma unroll 1
        for (int c = 0; c < COLS / 32; ++c) {
          const int col = n0 + c * 32;
          if (col >= p.N_out) break;
          float v[32];
          tmem_ld32(lane_addr + c * 32, v);
          if (GLU) {
            float u[32];
            tmem_ld32(lane_addr + 128 + c * 32, u);
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              if (EPI == CAPPED_GLU) {
                const float g = fminf(v[i], p.limit);
                const float x = fminf(fmaxf(u[i], -p.limit), p.limit);
                v[i] = (g * __fdividef(1.0f, 1.0f + __expf(-p.alpha * g))) * (x + 1.0f);
              } else {
                v[i] = (v[i] * __fdividef(1.0f, 1.0f + __expf(-v[i]))) * u[i];
              }
            }
          } else if (EPI == RELU2) {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = fmaxf(v[i], 0.f) * fmaxf(v[i], 0.f);
          }
          if (row_live) store_row32(yrow + col, v, p.N_out - col, aligned);
        }
      }
      // this warp has read its quarter of the accumulator: hand it back to the MMA warp
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
    }
    pdl_launch_dependents();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

template <int EPI>
void launch_grouped(const CUtensorMap& map_a, const CUtensorMap& map_w, const GroupedParams& p, cudaStream_t stream) {
  const size_t smem = (size_t)STAGES * STAGE_BYTES + 1024;
  cudaFuncSetAttribute(grouped_tc5_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  static int num_sms = 0;
  if (num_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (num_sms <= 0) num_sms = 148;
  }
  const int cols = (EPI == SILU_GLU || EPI == CAPPED_GLU) ? 128 : BN;
  const long long most = (long long)p.max_tiles * ((p.N_out + cols - 1) / cols);
  launch_k(grouped_tc5_kernel<EPI>, (int)(most < num_sms ? most : num_sms), NTHREADS, smem, stream, map_a, map_w, p);
}
}  // namespace

// a [rows, K], w [groups, N, K], out [rows, N or N / 2], all bfloat16; tiles as the kernel's (null: all rows are group
// 0's); epilogue as enumerated.
// err: device int, set to 1 if a bounded wait ran out (the result is then invalid).
PBE_EXPORT int pbe_grouped_tc5(const void* a, const void* w, void* out, int rows, int K, int N, int groups,
                               const int32_t* tiles, int max_tiles, int epilogue, float limit, float alpha, int* err,
                               cudaStream_t stream) {
  if (rows <= 0 || N <= 0 || groups <= 0 || (tiles && max_tiles <= 0)) return 0;
  if (K <= 0 || (K & 7) || ((uintptr_t)a & 15) || ((uintptr_t)w & 15) || ((uintptr_t)out & 15))
    return (int)cudaErrorInvalidValue;
  const bool glu = epilogue == SILU_GLU || epilogue == CAPPED_GLU;
  if (epilogue < PLAIN || epilogue > CAPPED_GLU || (glu && (N & 1)) || (long long)groups * N > 0x7fffffffLL - 512)
    return (int)cudaErrorInvalidValue;
  CUtensorMap map_a, map_w;
  int rc = make_map(&map_a, a, rows, K);
  if (rc == 0) rc = make_map(&map_w, w, groups * N, K);
  if (rc != 0) return rc;
  GroupedParams p{(bf16*)out, N, glu ? N / 2 : N, K, tiles, rows, tiles ? max_tiles : (rows + BM - 1) / BM, limit, alpha, err};
  switch (epilogue) {
    case RELU2: launch_grouped<RELU2>(map_a, map_w, p, stream); break;
    case SILU_GLU: launch_grouped<SILU_GLU>(map_a, map_w, p, stream); break;
    case CAPPED_GLU: launch_grouped<CAPPED_GLU>(map_a, map_w, p, stream); break;
    default: launch_grouped<PLAIN>(map_a, map_w, p, stream); break;
  }
  return launch_status();
}
