// The scan over chunks of sixteen tokens (chunk_scan.cuh: the same records, the same recurrence) on the tensor cores,
// for bfloat16 runs: mma.sync m16n8k16, a float32 factor as two bfloat16 terms, a product of two such factors as three
// (hi hi + hi lo + lo hi, what is left out is 2^-16 of it), float32 sums.
//
// A block takes 64 columns of a head's state: warps 0-3 compute, sixteen columns each, whose [16, D] piece of S^T stays in
// float32 accumulators and turns into an operand in registers; warps 4-7 fetch the next chunk's record and values,
// split them and lay them down in the other of two buffers, one barrier a chunk.  Per chunk a computing warp has
//   [W | QG]: S^T (as it lies) times the records' vectors, two tiles of eight tokens each;
//   u = U - S^T W;   o = S^T QG + u MQ;   S^T <- decays S^T + u KD.
// What binds the scan of chunk_scan.cuh is the shared-memory pipe (every half warp reads the whole record for its
// two or four columns); here sixteen columns share each fragment.  Delta rule, 1,100 + 37 + 911 tokens, 16 heads of
// 128 x 128: 264 -> 91 us (the longest request's 69 chunks, 1.3 us each); time mixing, 2,048 tokens in segments, both
// passes: 118 -> 77 us.  Against 64 bits on given inputs the read-outs are 5e-6 off (1e-7 in float32 multiply-adds);
// the layers, whose inputs are bfloat16, 0.004 either way.
#pragma once
#include <cuda_bf16.h>

#include "chunk_scan.cuh"

namespace pbe {
namespace scan_mma {

typedef __nv_bfloat16 bf16;
constexpr int COLS = 64;                 // columns of a block
constexpr int USTR = COLS + 4;           // floats a row of U: four rows apart start in different banks
constexpr int MSTR = CH + 8;             // elements a row of MQ

template <int DP>
__host__ __device__ constexpr int row_elems() { return DP + 8; }
// one buffer: QG, KD and W as hi and lo [CH][DP + 8], MQ as hi and lo [CH][MSTR], the decays [DP], U [CH][USTR]
template <int DP, bool CORRECT>
__host__ __device__ constexpr int buffer_bytes() {
  return 2 * 2 * ((CORRECT ? 3 : 2) * CH * row_elems<DP>() + CH * MSTR) + 4 * (DP + CH * USTR);
}

__device__ __forceinline__ unsigned at_smem(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldm4(unsigned (&r)[4], const bf16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at_smem(p)) : "memory");
}
__device__ __forceinline__ void ldm4t(unsigned (&r)[4], const bf16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at_smem(p)) : "memory");
}
__device__ __forceinline__ void mma(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void split2(float x, float y, unsigned& hi, unsigned& lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
  hi = *reinterpret_cast<const unsigned*>(&h);
  const __nv_bfloat162 l = __floats2bfloat162_rn(x - __uint_as_float(hi << 16), y - __uint_as_float(hi & 0xffff0000u));
  lo = *reinterpret_cast<const unsigned*>(&l);
}
// two tiles of eight columns of C as the A operand of sixteen steps of k
__device__ __forceinline__ void as_operand(const float (&c0)[4], const float (&c1)[4], unsigned (&hi)[4], unsigned (&lo)[4]) {
  split2(c0[0], c0[1], hi[0], lo[0]);
  split2(c0[2], c0[3], hi[1], lo[1]);
  split2(c1[0], c1[1], hi[2], lo[2]);
  split2(c1[2], c1[3], hi[3], lo[3]);
}

template <int DP, bool CORRECT, bool OWN, typename TU>
__global__ void __launch_bounds__(256, CORRECT ? 1 : 2) scan_chunks_mma_kernel(ChunkScanParams<TU> p) {
  constexpr int STR = row_elems<DP>();
  constexpr int MATS = CORRECT ? 3 : 2;                  // QG, KD, W
  constexpr int REC = record_floats(DP, CORRECT);
  constexpr int BYTES = buffer_bytes<DP, CORRECT>();
  constexpr int PER = (REC / 4 + 127) / 128;             // float4s of a record a fetching thread takes
  constexpr int UPER = CH * COLS / 128;
  constexpr bool U_EXACT = sizeof(TU) == 2 && !CORRECT;  // u is a bfloat16 number: its second term is zero
  extern __shared__ __align__(16) unsigned char smem_raw[];
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
    return reinterpret_cast<bf16*>(smem_raw + buf * BYTES) + (which * 2 + term) * CH * STR;
  };
  auto mixed = [&](int buf, int term) { return reinterpret_cast<bf16*>(smem_raw + buf * BYTES) + MATS * 2 * CH * STR + term * CH * MSTR; };
  auto decays = [&](int buf) { return reinterpret_cast<float*>(smem_raw + buf * BYTES + 2 * 2 * (MATS * CH * STR + CH * MSTR)); };
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
        raw[i] = ft + i * 128 < REC / 4 ? from[ft + i * 128] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < UPER; ++i) {
        const int x = ft + i * 128, t = c * CH + x / COLS, e = e0 + x % COLS;
        u[i] = t < n && e < E ? to_float(p.u[(size_t)(t0 + t) * p.ld_u + h * E + e]) : 0.f;
      }
    };
    auto lay_down = [&](int buf) {
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int x = (ft + i * 128) * 4;
        if (x >= REC) break;
        uint2 hi, lo;
        split2(raw[i].x, raw[i].y, hi.x, lo.x);
        split2(raw[i].z, raw[i].w, hi.y, lo.y);
        if (x < rec_decay(DP) || (CORRECT && x >= rec_w(DP))) {
          const int y = x < rec_decay(DP) ? x : x - rec_w(DP) + 2 * CH * DP;       // QG, KD, W in a row
          const int which = y / (CH * DP), row = (y / DP) % CH, at = row * STR + y % DP;
          *reinterpret_cast<uint2*>(matrix(buf, which, 0) + at) = hi;
          *reinterpret_cast<uint2*>(matrix(buf, which, 1) + at) = lo;
        } else if (x < rec_mq(DP)) {
          *reinterpret_cast<float4*>(decays(buf) + x - rec_decay(DP)) = raw[i];
        } else {
          const int y = x - rec_mq(DP), at = (y / CH) * MSTR + y % CH;
          *reinterpret_cast<uint2*>(mixed(buf, 0) + at) = hi;
          *reinterpret_cast<uint2*>(mixed(buf, 1) + at) = lo;
        }
      }
#pragma unroll
      for (int i = 0; i < UPER; ++i) {
        const int x = ft + i * 128;
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
  const int col = e0 + warp * 16 + g8;                   // this thread's columns: col and col + 8
  auto place = [&](int v) -> float* {
    if (v == -1) return nullptr;
    return (v >= 0 ? p.state + ((size_t)v * H + h) * E * D : p.scratch + ((size_t)(-(v + 2)) * H + h) * E * D);
  };
  const float* st_in = place(src);
  float S[DP / 8][4];                                    // S^T: columns g8 (+ 8), key channels 8 j + q2 (+ 1)
#pragma unroll
  for (int j = 0; j < DP / 8; ++j)
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      float2 x = make_float2(0.f, 0.f);
      if (st_in && col + hh * 8 < E && j * 8 + q2 < D)
        x = *reinterpret_cast<const float2*>(st_in + (size_t)(col + hh * 8) * D + j * 8 + q2);
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
    // S^T times the records' vectors; sums of the leading products and of the corrections apart, so that fewer wait
    // for one another
    float w[2][4], q[2][4], wc[2][4], qc[2][4];
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int k = 0; k < 4; ++k) w[t][k] = q[t][k] = wc[t][k] = qc[t][k] = 0.f;
    if (CORRECT || !OWN) {
#pragma unroll
      for (int kk = 0; kk < DP / 16; ++kk) {
        unsigned hi[4], lo[4], b[4], d[4];
        as_operand(S[2 * kk], S[2 * kk + 1], hi, lo);
        if (CORRECT) {
          ldm4(b, matrix(buf, 2, 0) + krow * STR + kk * 16 + kcol);
          ldm4(d, matrix(buf, 2, 1) + krow * STR + kk * 16 + kcol);
          mma(w[0], hi, b[0], b[1]);
          mma(w[1], hi, b[2], b[3]);
          mma(wc[0], hi, d[0], d[1]);
          mma(wc[1], hi, d[2], d[3]);
          mma(wc[0], lo, b[0], b[1]);
          mma(wc[1], lo, b[2], b[3]);
        }
        if (!OWN) {
          ldm4(b, matrix(buf, 0, 0) + krow * STR + kk * 16 + kcol);
          ldm4(d, matrix(buf, 0, 1) + krow * STR + kk * 16 + kcol);
          mma(q[0], hi, b[0], b[1]);
          mma(q[1], hi, b[2], b[3]);
          mma(qc[0], hi, d[0], d[1]);
          mma(qc[1], hi, d[2], d[3]);
          mma(qc[0], lo, b[0], b[1]);
          mma(qc[1], lo, b[2], b[3]);
        }
      }
    }
    // u: token 8 t + q2 (+ 1) of columns g8 (+ 8)
    const float* U = values(buf) + warp * 16 + g8;
    float u[2][4];
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int k = 0; k < 4; ++k) u[t][k] = U[(t * 8 + q2 + (k & 1)) * USTR + (k >> 1) * 8] - (w[t][k] + wc[t][k]);
    unsigned uh[4], ul[4];
    as_operand(u[0], u[1], uh, ul);
    if (!OWN) {
      unsigned b[4], d[4];
      ldm4t(b, mixed(buf, 0) + lrow * MSTR + lcol);
      ldm4t(d, mixed(buf, 1) + lrow * MSTR + lcol);
      mma(q[0], uh, b[0], b[1]);
      mma(q[1], uh, b[2], b[3]);
      mma(qc[0], uh, d[0], d[1]);
      mma(qc[1], uh, d[2], d[3]);
      if (!U_EXACT) {
        mma(qc[0], ul, b[0], b[1]);
        mma(qc[1], ul, b[2], b[3]);
      }
    }
    const float* decay = decays(buf) + q2;
#pragma unroll
    for (int j = 0; j < DP / 8; ++j) {
      const float2 f = *reinterpret_cast<const float2*>(decay + j * 8);
      if (OWN) {
        product[j][0] *= f.x;
        product[j][1] *= f.y;
      }
      S[j][0] *= f.x;
      S[j][1] *= f.y;
      S[j][2] *= f.x;
      S[j][3] *= f.y;
    }
#pragma unroll
    for (int j = 0; j < DP / 16; ++j) {
      unsigned b[4], d[4];
      ldm4t(b, matrix(buf, 1, 0) + lrow * STR + j * 16 + lcol);
      ldm4t(d, matrix(buf, 1, 1) + lrow * STR + j * 16 + lcol);
      mma(S[2 * j], uh, b[0], b[1]);
      mma(S[2 * j + 1], uh, b[2], b[3]);
      mma(S[2 * j], uh, d[0], d[1]);
      mma(S[2 * j + 1], uh, d[2], d[3]);
      if (!U_EXACT) {
        mma(S[2 * j], ul, b[0], b[1]);
        mma(S[2 * j + 1], ul, b[2], b[3]);
      }
    }
    if (!OWN) {
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
  for (int j = 0; j < DP / 8; ++j)
#pragma unroll
    for (int hh = 0; hh < 2; ++hh)
      if (col + hh * 8 < E && j * 8 + q2 < D)
        *reinterpret_cast<float2*>(st_out + (size_t)(col + hh * 8) * D + j * 8 + q2) = make_float2(S[j][2 * hh], S[j][2 * hh + 1]);
}

// Heads of an even number of key channels in records of DP of them (64 or 128).
template <int DP, bool CORRECT, bool OWN, typename TU>
int launch(const ChunkScanParams<TU>& p, int items, cudaStream_t stream) {
  constexpr int smem = 2 * buffer_bytes<DP, CORRECT>();
  auto kernel = scan_chunks_mma_kernel<DP, CORRECT, OWN, TU>;
  static bool opted = false;
  if (!opted) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    opted = true;
  }
  launch_spread(kernel, dim3(items, p.H, (p.E + COLS - 1) / COLS), 256, smem, stream, p);
  return launch_status();
}
}  // namespace scan_mma
}  // namespace pbe
