// The experts' products on the fifth-generation tensor cores: rows sorted by expert, cut into tiles of up to 256
// rows of one expert (any height, any first row), out[row] = W_g a[row] for the rows of every tile (group g), in one
// launch for all experts.  A cluster of two blocks works on a tile: tcgen05.mma with cta_group::2, the MATRIX as the A
// operand (256 of its rows, 128 in each block) and the tile's rows as the B operand (N = their number rounded up to
// sixteen, half of them in each block), operands staged by TMA (128-byte swizzle, no multicast), the float32
// accumulator, output columns by rows, in tensor memory.
//
// What bounds it: with a few rows an expert, reading every chosen expert's matrices once (DRAM); with hundreds, that and
// the tiles' way from L2 into shared memory.  Hence
//   - the operands' places: rows are padded to sixteen instead of 128, and an expert's 264 rows are tiles of 144 and
//     120, which a block stages in 16 KB of matrix and 9 KB of rows for 256 columns, not three tiles in 48 KB each;
//   - the pair: a block stages its half of the matrix tile and its half of the rows;
//   - the order: all column blocks of eight row tiles before the next eight, so that these rows stay in L2 while the
//     matrices stream past; with the column blocks of all experts one after another the rows were fetched again and
//     again (525 MB for 402).  The matrices give their place in L2 up first.
// A persistent pair of blocks walks over the tiles.  Warp 0 is the TMA producer, warp 1 of the leader issues the MMAs,
// warps 2-5 are the epilogue; two accumulators alternate, so a tile's epilogue overlaps the next tile's products.  Three
// stages of 128 k: between two stages the issuer waits, fences and commits while the tensor pipe runs dry, some 200
// clocks whatever the tile's height, so stages of 64 k (six) cost a tenth (matrices in L2, 256-row tiles: 77.8 -> 69.0 us,
// 1.21 -> 1.37 PFLOP/s).  Results leave through shared memory: stores of two bytes along the accumulator's lanes took ten
// microseconds a tile.
//
// Epilogues: none, relu squared, and gates (W_g = [gate rows; up rows]: a block takes 64 of each, and the threads of an
// output's gate and up sums swap halves of their rows, so the activation costs no pass over memory and sees float32 sums).
//
// 2,048 rows, 4 of 32 experts, 2,048 -> 2 x 1,408 -> 2,048 (matrices from DRAM): 130 + 73 -> 111 + 63 us; 4,096 rows
// 204 + 106 -> 162 + 90, 16 rows 83 + 46 -> 68 + 36 (one block a tile of 128 rows x 256 columns before; the mma.sync
// products of grouped_gemm.cu and the activation's own pass took 826 + 95 at 2,048 rows).
//
// Every wait on an mbarrier is bounded; one that runs out sets *err and the block goes on to its end.
#include <cuda_bf16.h>

#include "common.cuh"
#include "opt_in.cuh"
#include "pdl.cuh"
#include "tcgen05.cuh"

using namespace pbe;
using namespace pbe::tc5;

namespace {
typedef __nv_bfloat16 bf16;
constexpr int BAND = 8;                  // row tiles that all column blocks are made for before the next ones
constexpr int BM = 128, MAX_ROWS = 256, BK = 64, UMMA_K = 16, STAGES = 3, IN_STAGE = 2;
constexpr int A_BYTES = BM * BK * 2, B_BYTES = MAX_ROWS / 2 * BK * 2, BLOCK_BYTES = A_BYTES + B_BYTES;
constexpr int STAGE_BYTES = IN_STAGE * BLOCK_BYTES;        // a stage is two blocks of 64 k
constexpr int BOUNCE_BYTES = 2 * 32 * (128 + 8) * 2;         // results of 32 rows on their way out, twice (gated ones
static_assert(BOUNCE_BYTES >= 2 * 32 * (64 + 8) * 2 + 16 * 128 * 4, "");      // are half, and the swap beside them)
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

// tma_load_2d_pair for what is read once or by neighbours at the same time: L2 gives it up first
__device__ __forceinline__ void tma_load_2d_pair_once(void* smem_dst, const CUtensorMap* map, int x, int y, uint32_t bar_cluster_addr) {
  uint64_t policy;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3}], [%4], %5;"
      ::"r"(smem_u32(smem_dst)), "l"(map), "r"(x), "r"(y), "r"(bar_cluster_addr), "l"(policy) : "memory");
}

// The matrices in boxes of 128 rows (64 for gated ones), the rows in boxes of 8, 16, 32, 64 and 128.
struct Maps {
  CUtensorMap w;
  CUtensorMap x[5];
};

struct Tile {
  int group, m0, rows, n0;
};
__device__ __forceinline__ Tile tile_at(const GroupedParams& p, int t, int live, int cols) {
  Tile o;
  const int across = (p.N_out + cols - 1) / cols;
  const int first = t / (BAND * across) * BAND, left = t - first * across;
  const int in_band = min(BAND, live - first);
  const int i = first + left % in_band;
  o.n0 = left / in_band * cols;
  if (p.tiles) {
    o.group = p.tiles[3 * i];
    o.m0 = p.tiles[3 * i + 1];
    o.rows = min(p.tiles[3 * i + 2], MAX_ROWS);
  } else {                                    // all rows are one group's: tiles of one height
    const int height = (p.rows + 16 * live - 1) / (16 * live) * 16;
    o.group = 0;
    o.m0 = i * height;
    o.rows = min(height, p.rows - o.m0);
  }
  return o;
}
__device__ __forceinline__ int padded_rows(int rows) { return (rows + 15) & ~15; }

template <int EPI>
__global__ void __launch_bounds__(NTHREADS, 1)
grouped_tc5_kernel(const __grid_constant__ Maps maps, GroupedParams p) {
  constexpr bool GLU = EPI == SILU_GLU || EPI == CAPPED_GLU;
  constexpr int COLS = GLU ? 128 : 256;         // output columns of a pair's tile
  constexpr int OWN = COLS / 2;                 // and of a block's part
  constexpr int LD = OWN + 8;                   // columns of a row in shared memory: no bank conflicts either way
  extern __shared__ unsigned char smem_raw[];
  unsigned char* stages = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full_bar[STAGES];       // used in the leader
  __shared__ __align__(8) uint64_t empty_bar[STAGES];
  __shared__ __align__(8) uint64_t acc_full[2];
  __shared__ __align__(8) uint64_t acc_empty[2];           // used in the leader: eight arrivals
  __shared__ uint32_t tmem_base_smem;
  __shared__ int live_smem;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_rank();
  const bool leader = rank == 0;
  const int kblocks = (p.K + BK - 1) / BK;
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;

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
      mbar_init(&acc_empty[b], 8);          // one arrival per epilogue warp of either block
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {   // tensor memory: all 512 columns in both blocks, by the same warp of each
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&tmem_base_smem)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  __syncthreads();
  pdl_wait();          // the tile list and the rows come from the kernels before
  // the live tiles stand at the front of the list
  for (int i = threadIdx.x; i < p.max_tiles; i += NTHREADS)
    if (p.tiles == nullptr || p.tiles[3 * i] >= 0) atomicAdd(&live_smem, 1);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_all();                          // the other block's barriers exist from here on
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = tmem_base_smem;
  const int live = live_smem;
  const int num_tiles = live * ((p.N_out + COLS - 1) / COLS);

  if (warp == 0) {
    // -------------------------------------------------------------- TMA producer (one in each block)
    // A copy a lane.  The block's 128 matrix rows: one box, or, gated, 64 gate rows and their 64 up rows.  Its half of
    // the tile's rows: the boxes of 8 to 128 rows that make it up, the largest first.
    const bool for_w = lane < (GLU ? 2 : 1);
    const int piece = lane - 8;                // box of 8 << piece rows
    int it = 0;
    bool ok = true;
    for (int t = pair; t < num_tiles && ok; t += num_pairs) {
      const Tile tile = tile_at(p, t, live, COLS);
      const int half = padded_rows(tile.rows) / 2;
      const bool for_x = piece >= 0 && piece < 5 && ((half >> 3) & (1 << piece));
      const int before = for_x ? half >> (4 + piece) << (4 + piece) : 0;     // the larger boxes' rows
      const CUtensorMap* map = for_w ? &maps.w : &maps.x[for_x ? piece : 0];
      const int y = for_x ? tile.m0 + rank * half + before
                    : GLU ? tile.group * p.N + tile.n0 + rank * 64 + lane * p.N_out
                          : tile.group * p.N + tile.n0 + rank * 128;
      const int to = for_x ? A_BYTES + before * BK * 2 : lane * 64 * BK * 2;
      const uint32_t bytes = 2 * (A_BYTES + half * BK * 2);                  // both blocks' copies
      for (int kb = 0; kb < kblocks; kb += IN_STAGE, ++it) {
        const int s = it % STAGES, blocks = min(IN_STAGE, kblocks - kb);
        ok = mbar_wait_warp(&empty_bar[s], ((it / STAGES) & 1) ^ 1, p.err);
        if (!ok) break;
        if (leader && lane == 0) mbar_expect_tx(&full_bar[s], blocks * bytes);
        __syncwarp();
        unsigned char* dst = stages + (size_t)s * STAGE_BYTES + to;
        const uint32_t bar = map_to_rank(&full_bar[s], 0);
        for (int h = 0; h < blocks; ++h) {
          if (for_w) tma_load_2d_pair_once(dst + h * BLOCK_BYTES, map, (kb + h) * BK, y, bar);
          else if (for_x) tma_load_2d_pair(dst + h * BLOCK_BYTES, map, (kb + h) * BK, y, bar);
        }
      }
    }
    // The commits that release the last stages arrive on both blocks' barriers: neither leaves before they have.
    for (int q = it > STAGES ? it - STAGES : 0; q < it && ok; ++q)
      ok = mbar_wait(&empty_bar[q % STAGES], (q / STAGES) & 1, p.err);
  } else if (warp == 1) {
    if (leader && lane == 0) {
      // ------------------------------------------------------------ MMA issuer (the leader's, for the pair)
      int it = 0, j = 0;
      bool ok = true;
      for (int t = pair; t < num_tiles && ok; t += num_pairs, ++j) {
        const uint32_t idesc = make_idesc(256, padded_rows(tile_at(p, t, live, COLS).rows));
        const int buf = j & 1;
        ok = mbar_wait(&acc_empty[buf], ((j >> 1) & 1) ^ 1, p.err);   // the epilogues have drained this accumulator
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tmem_d = tmem_base + buf * MAX_ROWS;
        for (int kb = 0; kb < kblocks && ok; kb += IN_STAGE, ++it) {
          const int s = it % STAGES;
          ok = mbar_wait(&full_bar[s], (it / STAGES) & 1, p.err);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const int blocks = min(IN_STAGE, kblocks - kb);
          for (int h = 0; h < blocks; ++h) {
            const uint32_t a_addr = smem_u32(stages + (size_t)s * STAGE_BYTES + h * BLOCK_BYTES);
            const uint32_t b_addr = a_addr + A_BYTES;
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k)
              umma_pair(tmem_d, make_desc(a_addr + k * UMMA_K * 2), make_desc(b_addr + k * UMMA_K * 2), idesc,
                        (kb > 0 || h > 0 || k > 0) ? 1u : 0u);
          }
          umma_commit_pair(&empty_bar[s]);   // the stage is free in both blocks once these MMAs have read it
        }
        umma_commit_pair(&acc_full[buf]);    // the accumulator is complete in both blocks
      }
      // the other block's epilogue warps arrive on this block's acc_empty: all of it is in before this block leaves
      for (int q = j > 2 ? j - 2 : 0; q < j && ok; ++q) ok = mbar_wait(&acc_empty[q & 1], (q >> 1) & 1, p.err);
    }
  } else {
    // -------------------------------------------------------------- epilogue warps 2..5 of each block
    // A thread holds one matrix row, that is one output column, of 32 rows at a time (gated: the threads of an output's
    // gate and up sums swap sixteen each and take half of the rows).  The results go through shared memory and leave it
    // as whole pieces of rows.
    const int quarter = warp & 3;          // the TMEM lanes this warp may read
    const int thread = quarter * 32 + lane;
    const bool up = thread >= 64;
    const bool aligned = (p.N_out & 7) == 0;
    const uint32_t leader_acc_empty[2] = {map_to_rank(&acc_empty[0], 0), map_to_rank(&acc_empty[1], 0)};
    bf16* const bounce = reinterpret_cast<bf16*>(stages + (size_t)STAGES * STAGE_BYTES);
    float* const swap = reinterpret_cast<float*>(bounce + 2 * 32 * LD);
    bool ok = true;
    int j = 0, turn = 0;
    for (int t = pair; t < num_tiles; t += num_pairs, ++j) {
      const Tile tile = tile_at(p, t, live, COLS);
      const int buf = j & 1;
      const int col0 = tile.n0 + rank * OWN;
      ok = ok && mbar_wait(&acc_full[buf], (j >> 1) & 1, p.err);      // flagged; all roles run to their end
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16) + buf * MAX_ROWS;
#pragma unroll 1
      for (int c = 0; c < tile.rows; c += 32, turn ^= 1) {
        float v[32];
        tmem_ld32(lane_addr + c, v);
        bf16* const mine = bounce + turn * 32 * LD;
        if (GLU) {
#pragma unroll
          for (int i = 0; i < 16; ++i) swap[i * 128 + thread] = up ? v[i] : v[16 + i];
          asm volatile("bar.sync 1, 128;" ::: "memory");
          float other[16];                 // all of them before the first store: the compiler would not move them across
#pragma unroll
          for (int i = 0; i < 16; ++i) other[i] = swap[i * 128 + (thread ^ 64)];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float g = up ? other[i] : v[i], x = up ? v[16 + i] : other[i], r;
            if (EPI == CAPPED_GLU) {
              g = fminf(g, p.limit);
              x = fminf(fmaxf(x, -p.limit), p.limit);
              r = (g * __fdividef(1.0f, 1.0f + __expf(-p.alpha * g))) * (x + 1.0f);
            } else {
              r = (g * __fdividef(1.0f, 1.0f + __expf(-g))) * x;
            }
            mine[(up ? 16 + i : i) * LD + (thread & 63)] = __float2bfloat16_rn(r);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            mine[i * LD + quarter * 32 + lane] = __float2bfloat16_rn(EPI == RELU2 ? fmaxf(v[i], 0.f) * fmaxf(v[i], 0.f) : v[i]);
        }
        // the pieces before last were read before the last barrier: one a piece is enough
        asm volatile("bar.sync 1, 128;" ::: "memory");
        bf16* const y = p.out + (size_t)(tile.m0 + c) * p.N_out + col0;
        const int rows = min(32, tile.rows - c), cols = p.N_out - col0;
        if (aligned) {
          const int x = thread % (OWN / 8) * 8;
#pragma unroll
          for (int i = 0; i < OWN / 32; ++i) {
            const int r = thread / (OWN / 8) + i * (1024 / OWN);
            if (r < rows && x < cols) *reinterpret_cast<uint4*>(y + (size_t)r * p.N_out + x) = *reinterpret_cast<const uint4*>(mine + r * LD + x);
          }
        } else {
          for (int i = thread; i < rows * OWN; i += 128)
            if (i % OWN < cols) y[(size_t)(i / OWN) * p.N_out + i % OWN] = mine[i / OWN * LD + i % OWN];
        }
      }
      // this warp has read its part of the accumulator: hand it back to the leader's MMA warp
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(leader_acc_empty[buf]);
    }
    pdl_launch_dependents();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_all();                          // nothing of this block is signalled or read from here on
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

template <int EPI>
int launch_grouped(const Maps& maps, const GroupedParams& p, cudaStream_t stream) {
  const size_t smem = (size_t)STAGES * STAGE_BYTES + BOUNCE_BYTES + 1024;
  static OptIn opt_in;
  if (const cudaError_t e = opt_in(smem, grouped_tc5_kernel<EPI>)) return (int)e;
  static int num_sms = 0;
  if (num_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (num_sms <= 0) num_sms = 148;
  }
  const int cols = (EPI == SILU_GLU || EPI == CAPPED_GLU) ? 128 : 256;
  const long long most = (long long)p.max_tiles * ((p.N_out + cols - 1) / cols);
  const int pairs = (int)(most < num_sms / 2 ? most : num_sms / 2);
  launch_k_cluster(grouped_tc5_kernel<EPI>, 2 * pairs, NTHREADS, smem, stream, 2, maps, p);
  return launch_status();
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
  Maps maps;
  int rc = make_map(&maps.w, w, groups * N, K, glu ? BM / 2 : BM);
  for (int i = 0; i < 5 && rc == 0; ++i) rc = make_map(&maps.x[i], a, rows, K, 8 << i);
  if (rc != 0) return rc;
  GroupedParams p{(bf16*)out, N, glu ? N / 2 : N, K, tiles, rows, tiles ? max_tiles : (rows + MAX_ROWS - 1) / MAX_ROWS, limit, alpha, err};
  switch (epilogue) {
    case RELU2: return launch_grouped<RELU2>(maps, p, stream);
    case SILU_GLU: return launch_grouped<SILU_GLU>(maps, p, stream);
    case CAPPED_GLU: return launch_grouped<CAPPED_GLU>(maps, p, stream);
    default: return launch_grouped<PLAIN>(maps, p, stream);
  }
}
