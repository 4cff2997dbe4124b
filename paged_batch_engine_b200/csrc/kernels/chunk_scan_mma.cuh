// The scan over chunks of sixteen tokens (chunk_scan.cuh: the same records, the same recurrence) on the tensor cores,
// for bfloat16 runs: mma.sync m16n8k16, a float32 factor as three bfloat16 terms h + m + l, which hold its 24 bits, a
// product of two such factors as six (h h, h m, m h, m m, h l, l h; what is left out is 2^-24 of it at most), float32 sums.
// The tensor cores cut off what does not fit a sum instead of rounding it, so the state is not left to them: what a chunk
// writes is summed from zero and added to the state with one rounding.
//
// A block takes 64 columns of a head's state (32 or 16 where two or four warps share sixteen columns, see launch): warps 0-3
// compute, sixteen columns each, whose [16, D] piece of S^T (or their share of its key channels) stays in float32
// accumulators and turns into an operand in registers; the other warps fetch the next chunk's record and values, split
// them and lay them down in the other of two buffers, one barrier a chunk.  Per chunk a computing warp has
//   [W | QG]: S^T (as it lies) times the records' vectors, two tiles of eight tokens each; with corrected writes a quarter of the
//   key channels at a time, summed from zero, the quarters q added as (q0 + q1) + (q2 + q3) by one warp or, through shared
//   memory, by those that share columns: a request has the same bits whatever its neighbours let the blocks be cut into;
//   u = U - S^T W;   o = S^T QG + u MQ;   S^T <- decays S^T + u KD.
// What binds the scan of chunk_scan.cuh is the shared-memory pipe (every half warp reads the whole record for its
// two or four columns); here sixteen columns share each fragment, and the 300 products of a chunk and computing warp bind.
// Delta rule, 1,100 + 37 + 911 tokens, 16 heads of 128 x 128: 264 -> 157 us (the longest request's 69 chunks, 2.3 us each), with
// two warps to sixteen columns 114;
// time mixing, 2,048 tokens in segments, both passes: 118 -> 91 us.  Two terms a factor took 91 and 77, but read-outs and
// state were 5e-6 off 64 bits on given inputs; the multiply-adds are 0.5e-7 to 5e-7 off and this 0.6 to 1.4 times that.
#pragma once
#include "chunk_scan.cuh"
#include "opt_in.cuh"
#include "mma_sync.cuh"

namespace pbe {
namespace scan_mma {

using namespace mma_sync;

constexpr int USTR = 64 + 4;             // floats a row of U: four rows apart start in different banks
constexpr int MSTR = CH + 8;             // elements a row of MQ
template <int DS>
__host__ __device__ constexpr int block_cols() { return 64 / DS; }
template <int DS>
__host__ __device__ constexpr int fetch_threads() { return DS > 1 ? 256 : 128; }

template <int DP>
__host__ __device__ constexpr int row_elems() { return DP + 8; }
// one buffer: QG, KD and W as terms [CH][DP + 8], MQ as terms [CH][MSTR], the decays [DP], U [CH][USTR]
template <int DP, bool CORRECT>
__host__ __device__ constexpr int buffer_bytes() {
  return 2 * TERMS * ((CORRECT ? 3 : 2) * CH * row_elems<DP>() + CH * MSTR) + 4 * (DP + CH * USTR);
}

// two tiles of eight columns of C as the A operand of sixteen steps of k
__device__ __forceinline__ void as_operand(const float (&c0)[4], const float (&c1)[4], unsigned (&a)[TERMS][4]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    unsigned t[TERMS];
    split3(k < 2 ? c0[2 * k] : c1[2 * k - 4], k < 2 ? c0[2 * k + 1] : c1[2 * k - 3], t);
#pragma unroll
    for (int i = 0; i < TERMS; ++i) a[i][k] = t[i];
  }
}
// The products of terms x of A and y of B that count, x + y < 3: the small ones are added apart from h h, so that they are
// not cut off against it.  B: sixteen k times sixteen columns, its terms `apart` elements from one another.
template <bool TRANSPOSED, bool A_EXACT = false>
__device__ __forceinline__ void products(float (&big)[2][4], float (&small)[2][4], const unsigned (&a)[TERMS][4], const bf16* at,
                                         int apart) {
#pragma unroll
  for (int y = TERMS - 1; y >= 0; --y) {
    unsigned b[4];
    if (TRANSPOSED) ldm4t(b, at + y * apart);
    else ldm4(b, at + y * apart);
#pragma unroll
    for (int x = (A_EXACT ? 0 : TERMS - 1 - y); x >= 0; --x) {
      mma(x + y == 0 ? big[0] : small[0], a[x], b[0], b[1]);
      mma(x + y == 0 ? big[1] : small[1], a[x], b[2], b[3]);
    }
  }
}

// DS: computing warps that share sixteen columns, DP / DS of their key channels each
template <int DP, bool CORRECT, bool OWN, typename TU, int DS>
__global__ void __launch_bounds__(128 + fetch_threads<DS>(), CORRECT ? 1 : 2) scan_chunks_mma_kernel(ChunkScanParams<TU> p) {
  static_assert(DS == 1 || ((DS == 2 || DS == 4) && CORRECT), "warps of sixteen columns");
  static_assert(!(CORRECT && OWN), "what a segment adds of its own is made of given rows: it fetches no W");
  constexpr int COLS = block_cols<DS>();
  constexpr int DW = DP / DS;                            // key channels of a warp
  constexpr int STR = row_elems<DP>();
  constexpr int MATS = CORRECT ? 3 : 2;                  // QG, KD, W
  constexpr int REC = record_floats(DP, CORRECT);
  constexpr int BYTES = buffer_bytes<DP, CORRECT>();
  constexpr int FT = fetch_threads<DS>();
  // what is fetched of a record: all of it, or KD and the decays behind it where nothing is read out
  constexpr int FROM = OWN ? rec_kd(DP) : 0, TO = OWN ? rec_mq(DP) : REC;
  constexpr int PER = ((TO - FROM) / 4 + FT - 1) / FT;   // float4s of a record a fetching thread takes
  constexpr int UPER = CH * COLS / FT;
  constexpr bool U_EXACT = sizeof(TU) == 2 && !CORRECT;  // u is a bfloat16 number: its other terms are zero
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int QUARTERS = CORRECT ? 4 / DS : 1;         // a warp's parts of the products with the state (one: left to the tensor cores)
  __shared__ float shares[DS > 1 ? 4 : 1][16][33];       // their sums, by warp
  pdl_launch_dependents();
  pdl_wait();
  const int h = blockIdx.y;
  const int tid = threadIdx.x;
  int r = blockIdx.x, t0, n, src, dst;
  if (p.items) {
    const int32_t* it = p.items + (size_t)blockIdx.x * 4;
    t0 = it[0]; n = it[1]; src = it[2]; dst = it[3];
    r = p.request_of_row[t0];
  } else {
    n = p.q_len[r];
    t0 = p.q_start[r];
    src = dst = n > 0 ? p.slots[r] : -1;
  }
  if (n <= 0) return;
  const int D = p.D, E = p.E, H = p.H;
  const int e0 = blockIdx.z * COLS;
  const int nc = (n + CH - 1) / CH;
  const int q0 = p.q_start[r];
  const float* rec0 = p.records + ((size_t)(first_record(q0, r) + (t0 - q0) / CH) * H + h) * REC;
  auto matrix = [&](int buf, int which, int term) {
    return reinterpret_cast<bf16*>(smem_raw + buf * BYTES) + (which * TERMS + term) * CH * STR;
  };
  auto mixed = [&](int buf, int term) { return reinterpret_cast<bf16*>(smem_raw + buf * BYTES) + MATS * TERMS * CH * STR + term * CH * MSTR; };
  auto decays = [&](int buf) { return reinterpret_cast<float*>(smem_raw + buf * BYTES + 2 * TERMS * (MATS * CH * STR + CH * MSTR)); };
  auto values = [&](int buf) { return decays(buf) + DP; };

  if (tid >= 128) {
    // ---------------------------------------------------------------- fetch and split
    const int ft = tid - 128;
    float4 raw[PER];
    float u[UPER];
    auto request = [&](int c) {
      const float4* from = reinterpret_cast<const float4*>(rec0 + (size_t)c * H * REC);
#pragma unroll
      for (int i = 0; i < PER; ++i)
        raw[i] = ft + i * FT < (TO - FROM) / 4 ? from[FROM / 4 + ft + i * FT] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < UPER; ++i) {
        const int x = ft + i * FT, t = c * CH + x / COLS, e = e0 + x % COLS;
        u[i] = t < n && e < E ? to_float(p.u[(size_t)(t0 + t) * p.ld_u + h * E + e]) : 0.f;
      }
    };
    auto lay_down = [&](int buf) {
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int x = FROM + (ft + i * FT) * 4;
        if (x >= TO) break;
        unsigned t0[TERMS], t1[TERMS];
        split3(raw[i].x, raw[i].y, t0);
        split3(raw[i].z, raw[i].w, t1);
        if (x < rec_decay(DP) || (CORRECT && x >= rec_w(DP))) {
          const int y = x < rec_decay(DP) ? x : x - rec_w(DP) + 2 * CH * DP;       // QG, KD, W in a row
          const int which = y / (CH * DP), row = (y / DP) % CH, at = row * STR + y % DP;
#pragma unroll
          for (int t = 0; t < TERMS; ++t) *reinterpret_cast<uint2*>(matrix(buf, which, t) + at) = make_uint2(t0[t], t1[t]);
        } else if (x < rec_mq(DP)) {
          *reinterpret_cast<float4*>(decays(buf) + x - rec_decay(DP)) = raw[i];
        } else {
          const int y = x - rec_mq(DP), at = (y / CH) * MSTR + y % CH;
#pragma unroll
          for (int t = 0; t < TERMS; ++t) *reinterpret_cast<uint2*>(mixed(buf, t) + at) = make_uint2(t0[t], t1[t]);
        }
      }
#pragma unroll
      for (int i = 0; i < UPER; ++i) {
        const int x = ft + i * FT;
        values(buf)[(x / COLS) * USTR + x % COLS] = u[i];
      }
    };
    request(0);
    lay_down(0);
    if (nc > 1) request(1);
    __syncthreads();
    for (int c = 0; c < nc; ++c) {       // while chunk c is computed
      if (c + 1 < nc) lay_down((c + 1) & 1);
      if (c + 2 < nc) request(c + 2);
      __syncthreads();
    }
    return;
  }

  // ------------------------------------------------------------------ compute
  const int warp = tid >> 5, lane = tid & 31;
  const int g8 = lane >> 2, q2 = (lane & 3) * 2;
  const int lrow = (lane & 7) + ((lane >> 3) & 1) * 8, lcol = (lane >> 4) * 8;
  const int krow = (lane & 7) + (lane >> 4) * 8, kcol = ((lane >> 3) & 1) * 8;
  const int group = warp / DS, d0 = warp % DS * DW;      // of sixteen columns; this warp's first key channel
  const int col = e0 + group * 16 + g8;                  // this thread's columns: col and col + 8
  auto place = [&](int v) -> float* {
    if (v == -1) return nullptr;
    return (v >= 0 ? p.state + ((size_t)v * H + h) * E * D : p.scratch + ((size_t)(-(v + 2)) * H + h) * E * D);
  };
  const float* st_in = place(src);
  float S[DW / 8][4];                                    // S^T: columns g8 (+ 8), key channels d0 + 8 j + q2 (+ 1)
#pragma unroll
  for (int j = 0; j < DW / 8; ++j)
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      float2 x = make_float2(0.f, 0.f);
      if (st_in && col + hh * 8 < E && d0 + j * 8 + q2 < D)
        x = *reinterpret_cast<const float2*>(st_in + (size_t)(col + hh * 8) * D + d0 + j * 8 + q2);
      S[j][2 * hh] = x.x;
      S[j][2 * hh + 1] = x.y;
    }
  float product[OWN ? DP / 8 : 1][2];                    // of the decays of this thread's key channels
#pragma unroll
  for (int j = 0; j < (OWN ? DP / 8 : 1); ++j) product[j][0] = product[j][1] = 1.f;
  __syncthreads();
#pragma unroll 1
  for (int c = 0; c < nc; ++c) {
    const int buf = c & 1;
    // S^T times the records' vectors
    float w[2][4], q[2][4], wc[2][4], qc[2][4], sums[16], pair[16];
#pragma unroll
    for (int part = 0; part < QUARTERS; ++part) {
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int k = 0; k < 4; ++k) w[t][k] = q[t][k] = wc[t][k] = qc[t][k] = 0.f;
      if (CORRECT || !OWN) {
#pragma unroll
        for (int kk = part * (DW / 16 / QUARTERS); kk < (part + 1) * (DW / 16 / QUARTERS); ++kk) {
          unsigned a[TERMS][4];
          as_operand(S[2 * kk], S[2 * kk + 1], a);
          const int at = krow * STR + d0 + kk * 16 + kcol;
          if (CORRECT) products<false>(w, wc, a, matrix(buf, 2, 0) + at, CH * STR);
          if (!OWN) products<false>(q, qc, a, matrix(buf, 0, 0) + at, CH * STR);
        }
      }
      if constexpr (CORRECT) {
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const float of = k < 8 ? w[k >> 2][k & 3] + wc[k >> 2][k & 3] : q[k / 4 - 2][k & 3] + qc[k / 4 - 2][k & 3];
          pair[k] = part & 1 ? pair[k] + of : of;
          if (part & 1 || QUARTERS == 1) sums[k] = part > 1 ? sums[k] + pair[k] : pair[k];
        }
      }
    }
    if constexpr (DS > 1) {                              // (the block's barrier parts two chunks' uses)
#pragma unroll
      for (int k = 0; k < 16; ++k) shares[warp][k][lane] = sums[k];
      asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(32 * DS) : "memory");
      const auto of = &shares[group * DS];
#pragma unroll
      for (int k = 0; k < 16; ++k)
        sums[k] = DS == 2 ? of[0][k][lane] + of[1][k][lane] : (of[0][k][lane] + of[1][k][lane]) + (of[DS - 2][k][lane] + of[DS - 1][k][lane]);
    }
    if constexpr (CORRECT) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        w[k >> 2][k & 3] = sums[k];
        q[k >> 2][k & 3] = sums[8 + k];
        wc[k >> 2][k & 3] = qc[k >> 2][k & 3] = 0.f;
      }
    }
    // u: token 8 t + q2 (+ 1) of columns g8 (+ 8)
    const float* U = values(buf) + group * 16 + g8;
    float u[2][4];
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int k = 0; k < 4; ++k) u[t][k] = U[(t * 8 + q2 + (k & 1)) * USTR + (k >> 1) * 8] - (w[t][k] + wc[t][k]);
    unsigned ua[TERMS][4];
    as_operand(u[0], u[1], ua);
    if (!OWN && (DS == 1 || d0 == 0)) products<true, U_EXACT>(q, qc, ua, mixed(buf, 0) + lrow * MSTR + lcol, CH * MSTR);
    const float* decay = decays(buf) + d0 + q2;
#pragma unroll
    for (int j = 0; j < DW / 16; ++j) {
      float y[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}}, yc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
      products<true, U_EXACT>(y, yc, ua, matrix(buf, 1, 0) + lrow * STR + d0 + j * 16 + lcol, CH * STR);
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const float2 f = *reinterpret_cast<const float2*>(decay + (2 * j + t) * 8);
        if (OWN) {
          product[2 * j + t][0] *= f.x;
          product[2 * j + t][1] *= f.y;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) S[2 * j + t][k] = fmaf(k & 1 ? f.y : f.x, S[2 * j + t][k], y[t][k] + yc[t][k]);
      }
    }
    if (!OWN && (DS == 1 || d0 == 0)) {
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int token = c * CH + t * 8 + q2 + (k & 1), e = col + (k >> 1) * 8;
          if (token < n && e < E) p.out[((size_t)(t0 + token) * H + h) * E + e] = q[t][k] + qc[t][k];
        }
    }
    __syncthreads();       // this chunk's buffer is free, the next chunk's is laid down
  }
  float* st_out = place(dst);
  if (OWN && dst <= -2 && blockIdx.z == 0 && warp == 0 && g8 == 0) {
    float* out = p.own_decay + ((size_t)(-(dst + 2)) * H + h) * D;
#pragma unroll
    for (int j = 0; j < DP / 8; ++j)
      if (j * 8 + q2 < D) *reinterpret_cast<float2*>(out + j * 8 + q2) = make_float2(product[j][0], product[j][1]);
  }
  if (!st_out || (dst >= 0 && !p.write_state)) return;
#pragma unroll
  for (int j = 0; j < DW / 8; ++j)
#pragma unroll
    for (int hh = 0; hh < 2; ++hh)
      if (col + hh * 8 < E && d0 + j * 8 + q2 < D)
        *reinterpret_cast<float2*>(st_out + (size_t)(col + hh * 8) * D + d0 + j * 8 + q2) = make_float2(S[j][2 * hh], S[j][2 * hh + 1]);
}

template <int DP, bool CORRECT, bool OWN, typename TU, int DS>
int launch_of(const ChunkScanParams<TU>& p, int items, cudaStream_t stream) {
  // warps that share columns: one block a multiprocessor, so that blocks behind the first wave find the ones that short requests leave
  constexpr int smem = 2 * buffer_bytes<DP, CORRECT>() > 120 * 1024 || DS == 1 ? 2 * buffer_bytes<DP, CORRECT>() : 120 * 1024;
  auto kernel = scan_chunks_mma_kernel<DP, CORRECT, OWN, TU, DS>;
  static OptIn opt_in;
  if (const cudaError_t e = opt_in(smem, kernel)) return (int)e;
  launch_spread(kernel, dim3(items, p.H, (p.E + block_cols<DS>() - 1) / block_cols<DS>()), 128 + fetch_threads<DS>(), smem, stream, p);
  return launch_status();
}

// Heads of an even number of key channels in records of DP of them (64 or 128).
template <int DP, bool CORRECT, bool OWN, typename TU>
int launch(const ChunkScanParams<TU>& p, int items, cudaStream_t stream, int busy = 0) {
  // Corrected writes walk a request's chunks one after the other: two or four warps share sixteen columns where the blocks, as many
  // times more then, still find a multiprocessor each (`busy` requests of about the longest one's rows; 0: not known).
  // A layer of 16 heads of 128, one warp -> two: 1,100 + 37 + 911 tokens 359 -> 312 us; with blocks for more than every
  // multiprocessor 359 -> 397.  2,048 tokens, one -> two -> four: 488 -> 391 -> 361.
  if constexpr (CORRECT && !OWN) {
    static int sms = 0;
    if (sms == 0) {
      int dev = 0, got = 0;
      cudaGetDevice(&dev);
      cudaDeviceGetAttribute(&got, cudaDevAttrMultiProcessorCount, dev);
      sms = got > 0 ? got : 148;
    }
    if (busy > 0 && (long long)busy * p.H * ((p.E + 15) / 16) <= sms) return launch_of<DP, CORRECT, OWN, TU, 4>(p, items, stream);
    if (busy > 0 && (long long)busy * p.H * ((p.E + 31) / 32) <= sms) return launch_of<DP, CORRECT, OWN, TU, 2>(p, items, stream);
  }
  return launch_of<DP, CORRECT, OWN, TU, 1>(p, items, stream);
}
}  // namespace scan_mma
}  // namespace pbe
