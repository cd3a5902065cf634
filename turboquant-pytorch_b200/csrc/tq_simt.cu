// FP32 CUDA-core kernels: the exact-arithmetic path of every entry point.
//
// All rotation work goes through one register-tiled FP32 contraction
// (tile_gemm) whose k-loop is a sequential fma chain per output, i.e. ordinary
// fp32 dot products.  A tile is 64 vectors; the CTA keeps the tile in shared
// memory across the chained stages of a kernel (normalise -> rotate ->
// quantise -> rotate back -> residual -> project), so intermediates never
// touch HBM.  These kernels serve fp32 inputs, head_dims other than 128 and
// every API surface that is not throughput critical; the 16-bit, head_dim-128
// quantise / dequantise traffic goes to the tensor-core kernels in tq_umma.cu.

#include <atomic>

#include "tq_common.cuh"
#include "tq_internal.h"
#include "tq_pdl.cuh"

namespace tq {

constexpr int TM = 64;    // vectors per tile of the large form (RI = 4)
constexpr int KC = 16;    // k rows of B staged per step
constexpr int NT = 256;   // threads per CTA
constexpr int BPAD = 4;
// Stages of the ring that B travels through, for 64 * nj columns.  A fifth leaves room for one CTA fewer per SM.
__host__ __device__ constexpr int b_stages(int nj) { return nj <= 2 ? 4 : 3; }

enum { B_KN = 0, B_NK = 1 };

// A thread's place in the 16 x 16 grid over a tile; a warp is 4 rows of it by 8 columns.
__device__ __forceinline__ int tile_tx() { return (threadIdx.x & 7) | ((threadIdx.x >> 2) & 8); }
__device__ __forceinline__ int tile_ty() { return ((threadIdx.x >> 3) & 3) | ((threadIdx.x >> 4) & 12); }

__host__ __device__ inline int lda_for(int K) { return round_up(K, KC) + 4; }
__host__ __device__ inline int ldb_for(int N) { return round_up(N, 64) + BPAD; }
// floats of shared memory for the ring of a contraction with 64 * nj columns
__host__ __device__ inline int b_ring_floats(int nj) { return b_stages(nj) * KC * (64 * nj + BPAD); }

__device__ __forceinline__ void cp_async4(float* dst, const float* src, bool ok) {
  const int bytes = ok ? 4 : 0;                          // 0: the word is filled with zero, nothing is read
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool ok) {
  const int bytes = ok ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}

// One k-chunk of B (rows k0 .. k0 + KC) into its ring stage, as one group of asynchronous copies.  A chunk
// past the end of B commits an empty group, so that groups and chunks keep step.
template <int NJ, int BL>
__device__ __forceinline__ void b_stage(int k0, int K, const float* __restrict__ Bg, int64_t ldg, int N, float* ring) {
  constexpr int npad = 64 * NJ;
  constexpr int ldb = npad + BPAD;
  float* Bs = ring + (k0 / KC) % b_stages(NJ) * (KC * ldb);
  if (k0 < round_up(K, KC)) {
    if (BL == B_KN && (N & 3) == 0 && (ldg & 3) == 0 && ((uintptr_t)Bg & 15u) == 0) {
      for (int e = threadIdx.x; e < KC * (npad / 4); e += NT) {
        const int kk = e / (npad / 4), n = 4 * (e - kk * (npad / 4));
        const int k = k0 + kk;
        const bool ok = k < K && n < N;
        cp_async16(Bs + kk * ldb + n, ok ? Bg + (int64_t)k * ldg + n : Bg, ok);
      }
    } else {
      for (int e = threadIdx.x; e < KC * npad; e += NT) {
        const int kk = BL == B_KN ? e / npad : e % KC, n = BL == B_KN ? e % npad : e / KC;
        const int k = k0 + kk;
        const bool ok = k < K && n < N;
        const float* src = BL == B_KN ? Bg + (int64_t)k * ldg + n : Bg + (int64_t)n * ldg + k;
        cp_async4(Bs + kk * ldb + n, ok ? src : Bg, ok);
      }
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// The first chunks of B: issued before whatever the kernel does ahead of the contraction, so that their
// latency runs beside it.  The previous contraction's readers must be past their last barrier.
template <int NJ, int BL>
__device__ __forceinline__ void b_begin(int K, const float* __restrict__ Bg, int64_t ldg, int N, float* ring) {
#pragma unroll
  for (int c = 0; c < b_stages(NJ) - 1; ++c) b_stage<NJ, BL>(c * KC, K, Bg, ldg, N, ring);
}

// acc[ri][4*j+c] += sum_k As[(ty*RI+ri)*lda + k] * B[k][tx*4 + 64*j + c]
// B is global, fp32, either [K][N] row-major with row stride ldg (B_KN) or
// [N][K] row-major with row stride ldg (B_NK).  Columns >= N and rows >= K read
// as zero.  As must hold zeros in columns [K, round_up(K,16)).  b_begin() with the same B comes first.
//
// B goes through a ring of chunks of 16 rows by asynchronous copies: one barrier per chunk, and a chunk's L2
// latency passes under those before it (staged through registers with two barriers, each chunk cost that latency:
// 40 us for 4096 vectors of head_dim 128 on 64 SMs).  Every output is one chain of fused multiply-adds in
// ascending k, whatever RI is.
//
// What bounds it is what the shared-memory loads return: 128 bytes a clock into the registers, broadcast or not, that is
// RI + 4 NJ floats a thread and k (80 clocks of a 32 x 128 tile's k, 96 of a 64 x 128 tile's) against RI x 4 NJ / 128 lanes of
// multiply-adds (32 and 64).  So with one tile per SM the small tile is faster, with two the large one.  With RI = 2 the
// operands of the next four k are loaded while the last four are multiplied; two columns share one packed multiply-add
// (fma.rn.f32x2: the same IEEE result in each half).
__device__ __forceinline__ void fma2_acc(float& c0, float& c1, float a, float b0, float b1) {
  unsigned long long av, bv, cv;
  asm("mov.b64 %0, {%1, %1};" : "=l"(av) : "f"(a));
  asm("mov.b64 %0, {%1, %2};" : "=l"(bv) : "f"(b0), "f"(b1));
  asm("mov.b64 %0, {%1, %2};" : "=l"(cv) : "f"(c0), "f"(c1));
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(cv) : "l"(av), "l"(bv), "l"(cv));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(c0), "=f"(c1) : "l"(cv));
}
// volatile: the compiler otherwise moves the loads back to their uses
__device__ __forceinline__ float4 lds4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
template <int RI, int NJ, int BL>
__device__ __forceinline__ void tile_gemm(const float* As, int lda, int K, const float* __restrict__ Bg, int64_t ldg,
                                          int N, float* ring, float (&acc)[RI][4 * NJ]) {
  const int tx = tile_tx(), ty = tile_ty();
  constexpr int ldb = 64 * NJ + BPAD;
  const int kpad = round_up(K, KC);
  const uint32_t Ar = (uint32_t)__cvta_generic_to_shared(As + ty * RI * lda);
  for (int k0 = 0; k0 < kpad; k0 += KC) {
    asm volatile("cp.async.wait_group %0;" ::"n"(b_stages(NJ) - 2) : "memory");
    __syncthreads();                            // chunk k0 is there for everyone; the stage of chunk k0 - KC is free
    b_stage<NJ, BL>(k0 + (b_stages(NJ) - 1) * KC, K, Bg, ldg, N, ring);
    const uint32_t Bs = (uint32_t)__cvta_generic_to_shared(ring + (k0 / KC) % b_stages(NJ) * (KC * ldb) + tx * 4);
    constexpr int BUF = RI <= 2 ? 2 : 1;        // the large tile has no registers for a second set
    float4 a[BUF][RI], b[BUF][4][NJ];
    auto load = [&](int g) {
#pragma unroll
      for (int ri = 0; ri < RI; ++ri) a[g % BUF][ri] = lds4(Ar + 4u * (uint32_t)(ri * lda + k0 + 4 * g));
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int j = 0; j < NJ; ++j) b[g % BUF][u][j] = lds4(Bs + 4u * (uint32_t)((4 * g + u) * ldb + 64 * j));
    };
    if (BUF == 2) load(0);
#pragma unroll
    for (int g = 0; g < KC / 4; ++g) {
      if (BUF == 1) load(g);
      else if (g + 1 < KC / 4) load(g + 1);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
#pragma unroll
        for (int ri = 0; ri < RI; ++ri) {
          const float4 af = a[g % BUF][ri];
          const float av = (u == 0) ? af.x : (u == 1) ? af.y : (u == 2) ? af.z : af.w;
#pragma unroll
          for (int j = 0; j < NJ; ++j) {
            const float4 bf = b[g % BUF][u][j];
            fma2_acc(acc[ri][4 * j + 0], acc[ri][4 * j + 1], av, bf.x, bf.y);
            fma2_acc(acc[ri][4 * j + 2], acc[ri][4 * j + 3], av, bf.z, bf.w);
          }
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");     // only empty groups are left
}

template <int RI, int NJ>
__device__ __forceinline__ void zero_acc(float (&acc)[RI][4 * NJ]) {
#pragma unroll
  for (int ri = 0; ri < RI; ++ri)
#pragma unroll
    for (int c = 0; c < 4 * NJ; ++c) acc[ri][c] = 0.f;
}

// registers -> Cs[r*ldc + n] for n < ncols (a multiple of 4, at most ldc); caller syncs around it
template <int RI, int NJ>
__device__ __forceinline__ void acc_to_smem(const float (&acc)[RI][4 * NJ], float* Cs, int ldc, int ncols) {
  const int tx = tile_tx(), ty = tile_ty();
#pragma unroll
  for (int ri = 0; ri < RI; ++ri)
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int col = tx * 4 + 64 * j;
      if (col < ncols)
        *reinterpret_cast<float4*>(Cs + (ty * RI + ri) * ldc + col) =
            make_float4(acc[ri][4 * j], acc[ri][4 * j + 1], acc[ri][4 * j + 2], acc[ri][4 * j + 3]);
    }
}

// Load a tile of vectors as fp32 into Xs (zero padded to kpad columns, zero rows
// past n_total); per-row L2 norms into nrm[] when wanted, and As = x / (norm + 1e-8) of the warp's own rows.
// A warp loads up to four of its rows at a time, so that sixteen of a lane's loads are in flight.
template <int XDT, int RI>
__device__ __forceinline__ void load_tile_rows(const void* x, int64_t row0, int64_t n_total, int D, int64_t H, int64_t S,
                                               int64_t sb, int64_t sh, int64_t ss, float* Xs, int ld, float* nrm,
                                               float* As = nullptr) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kpad = round_up(D, KC);
  constexpr int R = RI == 1 ? 2 : 4;
#pragma unroll
  for (int r0 = warp; r0 < 16 * RI; r0 += R * (NT / 32)) {
    float ssq[R];
    int64_t off[R];
#pragma unroll
    for (int h = 0; h < R; ++h) {
      ssq[h] = 0.f;
      const int64_t n = row0 + r0 + h * (NT / 32);
      off[h] = n < n_total ? vec_offset(n, H, S, sb, sh, ss) : -1;
    }
    for (int k0 = 0; k0 < kpad; k0 += 128) {
      float v[R][4];
#pragma unroll
      for (int h = 0; h < R; ++h)
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int k = k0 + 32 * u + lane;
          v[h][u] = (off[h] >= 0 && k < D) ? load_elem<XDT>(x, off[h] + k) : 0.f;
        }
#pragma unroll
      for (int h = 0; h < R; ++h)
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int k = k0 + 32 * u + lane;
          if (k < kpad) {
            Xs[(r0 + h * (NT / 32)) * ld + k] = v[h][u];
            ssq[h] = fmaf(v[h][u], v[h][u], ssq[h]);
          }
        }
    }
    if (nrm != nullptr) {
#pragma unroll
      for (int h = 0; h < R; ++h) ssq[h] = __fsqrt_rn(warp_sum(ssq[h]));
#pragma unroll
      for (int h = 0; h < R; ++h)
        if (lane == 0) nrm[r0 + h * (NT / 32)] = ssq[h];
    }
    if (As != nullptr) {                          // each lane its own columns
      for (int k0 = lane; k0 < kpad; k0 += 128) {
#pragma unroll
        for (int h = 0; h < R; ++h)
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int at = (r0 + h * (NT / 32)) * ld + k0 + 32 * u;
            if (k0 + 32 * u < kpad) As[at] = nrm != nullptr ? __fdiv_rn(Xs[at], ssq[h] + 1e-8f) : Xs[at];
          }
      }
    }
  }
}

__device__ __forceinline__ void load_codebook(const float* cb, float* cent_s, float* thr_s) {
  for (int i = threadIdx.x; i < 256; i += NT) {
    cent_s[i] = __ldg(cb + kCentroidOff + i);
    thr_s[i] = __ldg(cb + kThresholdOff + i);
  }
}

// quantize_scalar for U values side by side: a search is `bits` dependent look-ups, so several in step hide one another
// (with 16-byte stores in k_dequantize: first-generation cache of 8192 keys and values 111 -> 106 us a pass, fp32 round trip of
// 4096 vectors 26.7 -> 24.6 us).
template <int U>
__device__ __forceinline__ void quantize_many(const float (&y)[U], const float* thr, int bits, int (&q)[U]) {
#pragma unroll
  for (int u = 0; u < U; ++u) q[u] = 0;
  for (int half = 1 << (bits - 1); half > 0; half >>= 1) {
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (y[u] > thr[q[u] + half - 1]) q[u] += half;
  }
}

// Packed bytes of one row, NB bytes per lane and step.
template <int IPB, int NB>
__device__ __forceinline__ void emit_packed_row(const float* row, int D, int bits, const float* thr_s, uint8_t* o, int lane) {
  const int G = (D + IPB - 1) / IPB;
  for (int g0 = lane; g0 < G; g0 += 32 * NB) {
    float y[IPB * NB];
    int q[IPB * NB];
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int i = 0; i < IPB; ++i) {
        const int c = (g0 + 32 * b) * IPB + i;
        y[b * IPB + i] = c < D ? row[c] : -INFINITY;          // past the end: index 0
      }
    quantize_many<IPB * NB>(y, thr_s, bits, q);
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      unsigned byte = 0;
#pragma unroll
      for (int i = 0; i < IPB; ++i) byte |= (unsigned)q[b * IPB + i] << (bits * (IPB - 1 - i));
      if (g0 + 32 * b < G) o[g0 + 32 * b] = (uint8_t)byte;
    }
  }
}

// Quantise the row Cs[r][0..D) and write it in the requested layout.
__device__ __forceinline__ void emit_indices_row(const float* row, int D, int bits, int mode, const float* thr_s,
                                                 void* out, int64_t n, int lane) {
  if (mode == TQ_IDX_PACKED) {
    const int ipb = 8 / bits;
    uint8_t* o = reinterpret_cast<uint8_t*>(out) + n * (int64_t)((D + ipb - 1) / ipb);
    if (ipb == 1) emit_packed_row<1, 4>(row, D, bits, thr_s, o, lane);
    else if (ipb == 2) emit_packed_row<2, 2>(row, D, bits, thr_s, o, lane);
    else if (ipb == 4) emit_packed_row<4, 1>(row, D, bits, thr_s, o, lane);
    else emit_packed_row<8, 1>(row, D, bits, thr_s, o, lane);
    return;
  }
  for (int c0 = lane; c0 < D; c0 += 128) {
    float y[4];
    int q[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) y[u] = c0 + 32 * u < D ? row[c0 + 32 * u] : 0.f;
    quantize_many<4>(y, thr_s, bits, q);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int c = c0 + 32 * u;
      if (c >= D) continue;
      if (mode == TQ_IDX_U8) reinterpret_cast<uint8_t*>(out)[n * (int64_t)D + c] = (uint8_t)q[u];
      else reinterpret_cast<int64_t*>(out)[n * (int64_t)D + c] = (int64_t)q[u];
    }
  }
}

// The same for the rows warp + 8 i of a tile, four at a time where there are as many: a search is `bits` dependent look-ups,
// which the other rows' hide.
template <int R, int IPB, int NB>
__device__ __forceinline__ void emit_packed_rows(const float* Cs, int ldc, int D, int bits, const float* thr_s, uint8_t* out, int64_t row0,
                                                 int64_t n_total, int r0, int lane) {
  const int G = (D + IPB - 1) / IPB;
  for (int g0 = lane; g0 < G; g0 += 32 * NB) {
    float y[R * IPB * NB];
    int q[R * IPB * NB];
#pragma unroll
    for (int h = 0; h < R; ++h)
#pragma unroll
      for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int i = 0; i < IPB; ++i) {
          const int c = (g0 + 32 * b) * IPB + i;
          y[(h * NB + b) * IPB + i] = c < D ? Cs[(r0 + 8 * h) * ldc + c] : -INFINITY;      // past the end: index 0
        }
    quantize_many<R * IPB * NB>(y, thr_s, bits, q);
#pragma unroll
    for (int h = 0; h < R; ++h)
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        unsigned byte = 0;
#pragma unroll
        for (int i = 0; i < IPB; ++i) byte |= (unsigned)q[(h * NB + b) * IPB + i] << (bits * (IPB - 1 - i));
        const int64_t n = row0 + r0 + 8 * h;
        if (g0 + 32 * b < G && n < n_total) out[n * G + g0 + 32 * b] = (uint8_t)byte;
      }
  }
}
template <int RI>
__device__ __forceinline__ void emit_indices_tile(const float* Cs, int ldc, int D, int bits, int mode, const float* thr_s, void* out,
                                                  int64_t row0, int64_t n_total) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int R = RI == 1 ? 2 : 4;
#pragma unroll 1
  for (int r0 = warp; r0 < 16 * RI; r0 += 8 * R) {
    if (mode == TQ_IDX_PACKED) {
      const int ipb = 8 / bits;
      uint8_t* o = reinterpret_cast<uint8_t*>(out);
      if (ipb == 1) emit_packed_rows<R, 1, 4>(Cs, ldc, D, bits, thr_s, o, row0, n_total, r0, lane);
      else if (ipb == 2) emit_packed_rows<R, 2, 2>(Cs, ldc, D, bits, thr_s, o, row0, n_total, r0, lane);
      else if (ipb == 4) emit_packed_rows<R, 4, 1>(Cs, ldc, D, bits, thr_s, o, row0, n_total, r0, lane);
      else emit_packed_rows<R, 8, 1>(Cs, ldc, D, bits, thr_s, o, row0, n_total, r0, lane);
      continue;
    }
    for (int c0 = lane; c0 < D; c0 += 128) {
      float y[4 * R];
      int q[4 * R];
#pragma unroll
      for (int h = 0; h < R; ++h)
#pragma unroll
        for (int u = 0; u < 4; ++u) y[4 * h + u] = c0 + 32 * u < D ? Cs[(r0 + 8 * h) * ldc + c0 + 32 * u] : 0.f;
      quantize_many<4 * R>(y, thr_s, bits, q);
#pragma unroll
      for (int h = 0; h < R; ++h) {
        const int64_t n = row0 + r0 + 8 * h;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int c = c0 + 32 * u;
          if (c >= D || n >= n_total) continue;
          if (mode == TQ_IDX_U8) reinterpret_cast<uint8_t*>(out)[n * (int64_t)D + c] = (uint8_t)q[4 * h + u];
          else reinterpret_cast<int64_t*>(out)[n * (int64_t)D + c] = (int64_t)q[4 * h + u];
        }
      }
    }
  }
}

__device__ __forceinline__ int fetch_index(const void* idx, int mode, int64_t n, int c, int D, int bits) {
  if (mode == TQ_IDX_PACKED) {
    const int ipb = 8 / bits;
    const int G = (D + ipb - 1) / ipb;
    unsigned byte = reinterpret_cast<const uint8_t*>(idx)[n * (int64_t)G + c / ipb];
    return (int)((byte >> (bits * (ipb - 1 - c % ipb))) & ((1u << bits) - 1u));
  } else if (mode == TQ_IDX_U8) {
    return (int)reinterpret_cast<const uint8_t*>(idx)[n * (int64_t)D + c];
  }
  return (int)(reinterpret_cast<const int64_t*>(idx)[n * (int64_t)D + c] & 255);
}

// ---------------------------------------------------------------------------
// K0: rotated values -> indices
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(NT) k_quantize_rotated(const float* __restrict__ y, int64_t n, int D, int bits,
                                                        const float* __restrict__ cb, int mode, void* out) {
  __shared__ float thr_s[256];
  for (int i = threadIdx.x; i < 256; i += NT) thr_s[i] = __ldg(cb + kThresholdOff + i);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t wstride = (int64_t)gridDim.x * (NT / 32);
  for (int64_t r = (int64_t)blockIdx.x * (NT / 32) + warp; r < n; r += wstride)
    emit_indices_row(y + r * D, D, bits, mode, thr_s, out, r, lane);
}

// ---------------------------------------------------------------------------
// K1: norm + rotate + quantise + pack
// ---------------------------------------------------------------------------
template <int XDT, int NJ, int RI>
__global__ void __launch_bounds__(NT) k_quantize(TqQuantizeJob job) {
  constexpr int TM = 16 * RI;                   // vectors per tile
  extern __shared__ __align__(16) float smem[];
  const int D = job.D;
  const int lda = lda_for(D);
  float* As = smem;
  float* Bs = As + TM * lda;
  float* cent_s = Bs + b_ring_floats(NJ);
  float* thr_s = cent_s + 256;
  float* nrm = thr_s + 256;
  load_codebook(job.codebook, cent_s, thr_s);
  const int64_t n_total = job.B * job.H * job.S;
  const int64_t tiles = (n_total + TM - 1) / TM;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kpad = round_up(D, KC);
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int64_t row0 = tile * TM;
    __syncthreads();
    b_begin<NJ, B_KN>(D, job.rotation_t, D, D, Bs);
    load_tile_rows<XDT, RI>(job.x, row0, n_total, D, job.H, job.S, job.stride_b, job.stride_h, job.stride_s, As, lda,
                        job.normalize ? nrm : nullptr, job.normalize ? As : nullptr);
    if (job.normalize) {
      __syncwarp();                               // a warp's rows are warp + 8 i
      const int r = warp + 8 * lane;
      if (r < TM && row0 + r < n_total) job.norms_out[row0 + r] = __half_as_ushort(__float2half_rn(nrm[r]));
    }
    float acc[RI][4 * NJ];
    zero_acc<RI, NJ>(acc);
    tile_gemm<RI, NJ, B_KN>(As, lda, D, job.rotation_t, D, D, Bs, acc);
    __syncthreads();
    acc_to_smem<RI, NJ>(acc, As, lda, kpad);
    __syncthreads();
    emit_indices_tile<RI>(As, lda, D, job.bits, job.idx_mode, thr_s, job.idx_out, row0, n_total);
  }
}

// ---------------------------------------------------------------------------
// K2: unpack + lookup + inverse rotation + rescale
// ---------------------------------------------------------------------------
template <int ODT, int NJ, int RI>
__global__ void __launch_bounds__(NT) k_dequantize(TqDequantizeJob job) {
  constexpr int TM = 16 * RI;                   // vectors per tile
  extern __shared__ __align__(16) float smem[];
  const int D = job.D;
  const int lda = lda_for(D);
  float* As = smem;
  float* Bs = As + TM * lda;
  float* cent_s = Bs + b_ring_floats(NJ);
  float* thr_s = cent_s + 256;
  load_codebook(job.codebook, cent_s, thr_s);
  const int64_t n_total = job.B * job.H * job.S;
  const int64_t tiles = (n_total + TM - 1) / TM;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tx = tile_tx(), ty = tile_ty();
  const int kpad = round_up(D, KC);
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int64_t row0 = tile * TM;
    __syncthreads();
    b_begin<NJ, B_KN>(D, job.rotation, D, D, Bs);
#pragma unroll 4
    for (int r = warp; r < TM; r += NT / 32) {
      int64_t n = row0 + r;
#pragma unroll 4
      for (int c = lane; c < kpad; c += 32) {
        float v = 0.f;
        if (n < n_total && c < D) v = cent_s[fetch_index(job.idx, job.idx_mode, n, c, D, job.bits)];
        As[r * lda + c] = v;
      }
    }
    float acc[RI][4 * NJ];
    zero_acc<RI, NJ>(acc);
    tile_gemm<RI, NJ, B_KN>(As, lda, D, job.rotation, D, D, Bs, acc);
#pragma unroll
    for (int ri = 0; ri < RI; ++ri) {
      int64_t n = row0 + ty * RI + ri;
      if (n >= n_total) continue;
      float nv = (job.norms != nullptr) ? __half2float(__ushort_as_half(job.norms[n])) : 1.f;
      int64_t off = vec_offset(n, job.H, job.S, job.ostride_b, job.ostride_h, job.ostride_s);
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int col = tx * 4 + 64 * j;
        float v[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) v[c] = (job.norms != nullptr) ? acc[ri][4 * j + c] * nv : acc[ri][4 * j + c];
        if (ODT == TQ_F32 && col + 4 <= D && ((uintptr_t)(reinterpret_cast<float*>(job.out) + off + col) & 15u) == 0) {
          *reinterpret_cast<float4*>(reinterpret_cast<float*>(job.out) + off + col) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
          for (int c = 0; c < 4; ++c)
            if (col + c < D) store_elem<ODT>(job.out, off + col + c, v[c]);
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// generic projection out = x @ m
// ---------------------------------------------------------------------------
template <int XDT, int NJ>
__global__ void __launch_bounds__(NT) k_project(const void* x, int64_t n_total, int K, const float* m, int N,
                                                float* out) {
  extern __shared__ __align__(16) float smem[];
  const int lda = lda_for(K);
  float* As = smem;
  float* Bs = As + TM * lda;
  const int64_t tiles = (n_total + TM - 1) / TM;
  const int tx = tile_tx(), ty = tile_ty();
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int64_t row0 = tile * TM;
    __syncthreads();
    b_begin<NJ, B_KN>(K, m, N, N, Bs);
    load_tile_rows<XDT, 4>(x, row0, n_total, K, 1, n_total, 0, 0, K, As, lda, nullptr);
    float acc[4][4 * NJ];
    zero_acc<4, NJ>(acc);
    tile_gemm<4, NJ, B_KN>(As, lda, K, m, N, N, Bs, acc);
#pragma unroll
    for (int ri = 0; ri < 4; ++ri) {
      int64_t n = row0 + ty * 4 + ri;
      if (n >= n_total) continue;
#pragma unroll
      for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          int col = tx * 4 + 64 * j + c;
          if (col < N) out[n * N + col] = acc[ri][4 * j + c];
        }
    }
  }
}

// ---------------------------------------------------------------------------
// K3: logits from packed keys.  One thread per key, RQ query rows at a time.
// qrot: (B, Hq, Sq, D) rotated queries.  stats: per (row, key block) {max, sum}.
// ---------------------------------------------------------------------------
constexpr int RQ = 4;
constexpr int SCORE_KEYS_PER_BLOCK = 1024;

__global__ void __launch_bounds__(NT) k_score_packed(TqScoreJob job, const float* __restrict__ qrot, float* stats,
                                                    int nblk) {
  __shared__ float cent_s[256];
  __shared__ __align__(16) float qs[TQ_MAX_DIM * RQ];
  __shared__ float red[NT / 32][RQ];
  const int D = job.D, bits = job.bits;
  const int ipb = 8 / bits;
  const int G = (D + ipb - 1) / ipb;
  const unsigned mask = (1u << bits) - 1u;
  for (int i = threadIdx.x; i < 256; i += NT) cent_s[i] = __ldg(job.codebook + kCentroidOff + i);
  const int blk = blockIdx.x % nblk;
  const int64_t bh = blockIdx.x / nblk;           // b * Hkv + hkv
  const int64_t b = bh / job.Hkv, hkv = bh % job.Hkv;
  const int rep = (int)(job.Hq / job.Hkv);
  const int R = rep * (int)job.Sq;               // query rows that read this KV head
  const int64_t s_begin = (int64_t)blk * SCORE_KEYS_PER_BLOCK;
  const int64_t s_end = min(s_begin + SCORE_KEYS_PER_BLOCK, job.Sk);
  const uint8_t* keys = job.idx_bytes + bh * job.Sk * G;
  const uint16_t* norms = job.norms + bh * job.Sk;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int r0 = 0; r0 < R; r0 += RQ) {
    __syncthreads();
    // stage RQ rotated query rows as qs[j][rq]
    for (int e = threadIdx.x; e < D * RQ; e += NT) {
      int j = e / RQ, rq = e % RQ;
      int r = r0 + rq;
      float v = 0.f;
      if (r < R) {
        int64_t hq = hkv * rep + r / job.Sq, sq = r % job.Sq;
        v = qrot[((b * job.Hq + hq) * job.Sq + sq) * D + j];
      }
      qs[e] = v;
    }
    __syncthreads();
    float run_max[RQ], run_sum[RQ];
#pragma unroll
    for (int rq = 0; rq < RQ; ++rq) { run_max[rq] = -INFINITY; run_sum[rq] = 0.f; }
    for (int64_t s0 = s_begin; s0 < s_end; s0 += NT) {
      int64_t s = s0 + threadIdx.x;
      float acc[RQ] = {0.f, 0.f, 0.f, 0.f};
      if (s < s_end) {
        const uint8_t* row = keys + s * G;
        for (int g = 0; g < G; ++g) {
          unsigned byte = row[g];
          for (int i = 0; i < ipb; ++i) {
            int j = g * ipb + i;
            if (j < D) {
              float c = cent_s[(byte >> (bits * (ipb - 1 - i))) & mask];
              float4 qv = *reinterpret_cast<const float4*>(qs + j * RQ);
              acc[0] = fmaf(qv.x, c, acc[0]);
              acc[1] = fmaf(qv.y, c, acc[1]);
              acc[2] = fmaf(qv.z, c, acc[2]);
              acc[3] = fmaf(qv.w, c, acc[3]);
            }
          }
        }
        float nv = __half2float(__ushort_as_half(norms[s]));
#pragma unroll
        for (int rq = 0; rq < RQ; ++rq) {
          int r = r0 + rq;
          if (r < R) {
            float l = acc[rq] * nv * job.scale;
            int64_t hq = hkv * rep + r / job.Sq, sq = r % job.Sq;
            job.logits[((b * job.Hq + hq) * job.Sq + sq) * job.Sk + s] = l;
            acc[rq] = l;
          }
        }
      }
      if (stats != nullptr) {
        // online (max, sum exp) per row over this thread's keys
#pragma unroll
        for (int rq = 0; rq < RQ; ++rq) {
          if (s < s_end && r0 + rq < R) {
            float l = acc[rq];
            float m = fmaxf(run_max[rq], l);
            if (m == -INFINITY) {
              run_sum[rq] += 0.f;
            } else {
              run_sum[rq] = run_sum[rq] * __expf(run_max[rq] - m) + __expf(l - m);
            }
            run_max[rq] = m;
          }
        }
      }
    }
    if (stats != nullptr) {
#pragma unroll
      for (int rq = 0; rq < RQ; ++rq) {
        float m = warp_max(run_max[rq]);
        float sc = (run_max[rq] == -INFINITY) ? 0.f : run_sum[rq] * __expf(run_max[rq] - m);
        float sm = warp_sum(sc);
        if (lane == 0) { red[warp][rq] = m; }
        __syncthreads();
        float bm = -INFINITY;
        for (int w = 0; w < NT / 32; ++w) bm = fmaxf(bm, red[w][rq]);
        __syncthreads();
        float contrib = (m == -INFINITY) ? 0.f : sm * __expf(m - bm);
        if (lane == 0) red[warp][rq] = contrib;
        __syncthreads();
        if (threadIdx.x == 0 && r0 + rq < R) {
          float tot = 0.f;
          for (int w = 0; w < NT / 32; ++w) tot += red[w][rq];
          int r = r0 + rq;
          int64_t hq = hkv * rep + r / job.Sq, sq = r % job.Sq;
          int64_t grow = (b * job.Hq + hq) * job.Sq + sq;
          stats[(grow * nblk + blk) * 2 + 0] = bm;
          stats[(grow * nblk + blk) * 2 + 1] = tot;
        }
        __syncthreads();
      }
    }
  }
}

// y = x @ m for up to a few thousand rows (queries): one block per RPB rows, one thread per
// output coordinate, the same sequential-k fma order as the tiled contraction.  A matrix
// element is loaded once and used for all RPB rows of the block.
template <int XDT, int RPB>
__device__ __forceinline__ void project_rows(const void* x, int64_t n, int K, const float* __restrict__ m, int N, float* out) {
  __shared__ float xs[RPB][TQ_MAX_DIM];
  const int64_t row0 = (int64_t)blockIdx.x * RPB;
#pragma unroll
  for (int r = 0; r < RPB; ++r)
    for (int k = threadIdx.x; k < K; k += blockDim.x) xs[r][k] = row0 + r < n ? load_elem<XDT>(x, (row0 + r) * K + k) : 0.f;
  __syncthreads();
  for (int col = threadIdx.x; col < N; col += blockDim.x) {
    float acc[RPB];
#pragma unroll
    for (int r = 0; r < RPB; ++r) acc[r] = 0.f;
    int k = 0;
    constexpr int kBatch = RPB == 1 ? 64 : 16;   // independent loads in flight before the ordered fma chains
    for (; k + kBatch <= K; k += kBatch) {
      float mv[kBatch];
#pragma unroll
      for (int u = 0; u < kBatch; ++u) mv[u] = __ldg(m + (int64_t)(k + u) * N + col);
#pragma unroll
      for (int u = 0; u < kBatch; ++u)
#pragma unroll
        for (int r = 0; r < RPB; ++r) acc[r] = fmaf(xs[r][k + u], mv[u], acc[r]);
    }
    for (; k < K; ++k) {
      const float mv = __ldg(m + (int64_t)k * N + col);
#pragma unroll
      for (int r = 0; r < RPB; ++r) acc[r] = fmaf(xs[r][k], mv, acc[r]);
    }
#pragma unroll
    for (int r = 0; r < RPB; ++r)
      if (row0 + r < n) out[(row0 + r) * N + col] = acc[r];
  }
}

// `followed`: a kernel launched with launch_after() comes next in the call (see tq_pdl.cuh)
template <int XDT, int RPB>
__global__ void k_project_rows(const void* x, int64_t n, int K, const float* __restrict__ m, int N, float* out, bool followed) {
  if (followed) pdl_trigger();
  project_rows<XDT, RPB>(x, n, K, m, N, out);
}
// the same rows by two matrices: blockIdx.y picks one
template <int XDT>
__global__ void k_project_rows_two(const void* x, int64_t n, int D, const float* m0, const float* m1, float* out0, float* out1) {
  pdl_trigger();
  project_rows<XDT, 1>(x, n, D, blockIdx.y ? m1 : m0, D, blockIdx.y ? out1 : out0);
}

// head_dim 128 specialisation: a thread owns whole keys (two at a time, 64 keys per warp and
// round), so no partial sums cross lanes.  The packed row is read in 16-byte pieces; for every
// coordinate the centroid comes from a shared look-up (byte offsets prepared a word at a
// time, so the load is [register + constant]) and the four rotated query values of that
// coordinate come from one broadcast 16-byte shared load, used for both keys.  Lane L holds
// the logits of keys L and L + 32 of the round, so logits leave as 128-byte rows and the
// softmax partials are per lane.
__device__ __forceinline__ float lds_f32(uint32_t addr) {
  float v;
  asm("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}

// Shared-memory addresses of the centroids of the CPW coordinates packed in one 32-bit word,
// in coordinate order.  `base` is the shared address of the table, aligned to 1024 bytes, so
// it can be merged into the byte offsets (index * 4) by the same permute / logic instruction
// that isolates them: no separate address addition per look-up.
template <int BITS>
__device__ __forceinline__ void word_offsets(uint32_t x, uint32_t base, uint32_t (&off)[4 * (8 / BITS)]) {
  constexpr int IPB = 8 / BITS;
  constexpr int CPW = 4 * IPB;
  constexpr uint32_t MASK = (1u << BITS) - 1u;
  if constexpr (BITS == 4) {
    const uint32_t even = (x >> 2) & 0x3C3C3C3Cu, odd = (x << 2) & 0x3C3C3C3Cu;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      off[2 * k] = __byte_perm(even, base, 0x7650u | k);       // byte k of `even` under bytes 1..3 of base
      off[2 * k + 1] = __byte_perm(odd, base, 0x7650u | k);
    }
  } else if constexpr (BITS == 2) {
    const uint32_t f0 = (x >> 4) & 0x0C0C0C0Cu, f1 = (x >> 2) & 0x0C0C0C0Cu, f2 = x & 0x0C0C0C0Cu, f3 = (x << 2) & 0x0C0C0C0Cu;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      off[4 * k] = __byte_perm(f0, base, 0x7650u | k);
      off[4 * k + 1] = __byte_perm(f1, base, 0x7650u | k);
      off[4 * k + 2] = __byte_perm(f2, base, 0x7650u | k);
      off[4 * k + 3] = __byte_perm(f3, base, 0x7650u | k);
    }
  } else {
#pragma unroll
    for (int u = 0; u < CPW; ++u) {
      const int byte = u / IPB;
      const int sh = 8 * byte + BITS * (IPB - 1 - (u % IPB));
      off[u] = (sh >= 2 ? ((x >> (sh - 2)) & (MASK << 2)) : ((x << (2 - sh)) & (MASK << 2))) | base;
    }
  }
}

template <int BITS>
__global__ void __launch_bounds__(NT) k_score_packed_d128(TqScoreJob job, const float* __restrict__ qrot, float* stats,
                                                         int nblk) {
  constexpr int D = 128;
  constexpr int IPB = 8 / BITS;
  constexpr int G = D / IPB;                     // packed bytes per key: 16, 32, 64 or 128
  constexpr int PIECES = G / 16;                 // 16-byte pieces per key
  constexpr int CPW = 4 * IPB;                   // coordinates per 32-bit word
  __shared__ __align__(1024) float cent_s[256];
  __shared__ float4 q_s[D];
  __shared__ float red[NT / 32][RQ];
  for (int i = threadIdx.x; i < 256; i += NT) cent_s[i] = __ldg(job.codebook + kCentroidOff + i);
  const uint32_t cent_base = (uint32_t)__cvta_generic_to_shared(cent_s);
  const int blk = blockIdx.x % nblk;
  const int64_t bh = blockIdx.x / nblk;
  const int64_t b = bh / job.Hkv, hkv = bh % job.Hkv;
  const int rep = (int)(job.Hq / job.Hkv);
  const int R = rep * (int)job.Sq;
  const int64_t s_begin = (int64_t)blk * SCORE_KEYS_PER_BLOCK;
  const int64_t s_end = min(s_begin + SCORE_KEYS_PER_BLOCK, job.Sk);
  const uint8_t* keys = job.idx_bytes + bh * job.Sk * G;
  const uint16_t* norms = job.norms + bh * job.Sk;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int r0 = 0; r0 < R; r0 += RQ) {
    int64_t out_row[RQ];
#pragma unroll
    for (int rq = 0; rq < RQ; ++rq) {
      const int r = r0 + rq;
      int64_t grow = 0;
      if (r < R) {
        const int64_t hq = hkv * rep + r / job.Sq, sq = r % job.Sq;
        grow = (b * job.Hq + hq) * job.Sq + sq;
      }
      out_row[rq] = grow;
    }
    __syncthreads();                             // the previous group's readers of q_s are done
#pragma unroll
    for (int rq = 0; rq < RQ; ++rq)
      for (int e = threadIdx.x; e < D; e += NT)
        reinterpret_cast<float*>(q_s)[e * RQ + rq] = (r0 + rq < R) ? __ldg(qrot + out_row[rq] * D + e) : 0.f;
    __syncthreads();
    float run_max[RQ], run_sum[RQ];
#pragma unroll
    for (int rq = 0; rq < RQ; ++rq) { run_max[rq] = -INFINITY; run_sum[rq] = 0.f; }
    for (int64_t kb = s_begin + warp * 64; kb < s_end; kb += (NT / 32) * 64) {
      const int64_t key_a = kb + lane, key_b = kb + 32 + lane;
      const bool ok_a = key_a < s_end, ok_b = key_b < s_end;
      const uint4* src_a = reinterpret_cast<const uint4*>(keys + (ok_a ? key_a : s_begin) * G);
      const uint4* src_b = reinterpret_cast<const uint4*>(keys + (ok_b ? key_b : s_begin) * G);
      float acc_a[RQ] = {0.f, 0.f, 0.f, 0.f}, acc_b[RQ] = {0.f, 0.f, 0.f, 0.f};
      uint4 cur_a = __ldg(src_a), cur_b = __ldg(src_b);
#pragma unroll 1
      for (int pc = 0; pc < PIECES; ++pc) {
        uint4 nxt_a = cur_a, nxt_b = cur_b;
        if (pc + 1 < PIECES) { nxt_a = __ldg(src_a + pc + 1); nxt_b = __ldg(src_b + pc + 1); }
        const float4* qp = q_s + pc * 4 * CPW;
        const uint32_t wa[4] = {cur_a.x, cur_a.y, cur_a.z, cur_a.w};
        const uint32_t wb[4] = {cur_b.x, cur_b.y, cur_b.z, cur_b.w};
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          uint32_t oa[CPW], ob[CPW];
          word_offsets<BITS>(wa[w], cent_base, oa);
          word_offsets<BITS>(wb[w], cent_base, ob);
#pragma unroll
          for (int u = 0; u < CPW; ++u) {
            const float4 q = qp[w * CPW + u];
            const float ca = lds_f32(oa[u]), cb = lds_f32(ob[u]);
            acc_a[0] = fmaf(q.x, ca, acc_a[0]); acc_a[1] = fmaf(q.y, ca, acc_a[1]);
            acc_a[2] = fmaf(q.z, ca, acc_a[2]); acc_a[3] = fmaf(q.w, ca, acc_a[3]);
            acc_b[0] = fmaf(q.x, cb, acc_b[0]); acc_b[1] = fmaf(q.y, cb, acc_b[1]);
            acc_b[2] = fmaf(q.z, cb, acc_b[2]); acc_b[3] = fmaf(q.w, cb, acc_b[3]);
          }
        }
        cur_a = nxt_a; cur_b = nxt_b;
      }
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int64_t key = half ? key_b : key_a;
        if (half ? ok_b : ok_a) {
          const float nv = __half2float(__ushort_as_half(norms[key]));
#pragma unroll
          for (int rq = 0; rq < RQ; ++rq) {
            if (r0 + rq < R) {
              const float l = (half ? acc_b[rq] : acc_a[rq]) * nv * job.scale;
              job.logits[out_row[rq] * job.Sk + key] = l;
              if (stats != nullptr) {
                const float m = fmaxf(run_max[rq], l);
                if (m != -INFINITY) run_sum[rq] = run_sum[rq] * __expf(run_max[rq] - m) + __expf(l - m);
                run_max[rq] = m;
              }
            }
          }
        }
      }
    }
    if (stats != nullptr) {
#pragma unroll
      for (int rq = 0; rq < RQ; ++rq) {
        const float m = warp_max(run_max[rq]);
        const float sc = (run_max[rq] == -INFINITY) ? 0.f : run_sum[rq] * __expf(run_max[rq] - m);
        const float sm = warp_sum(sc);
        if (lane == 0) red[warp][rq] = m;
        __syncthreads();
        float bm = -INFINITY;
        for (int w = 0; w < NT / 32; ++w) bm = fmaxf(bm, red[w][rq]);
        __syncthreads();
        const float contrib = (m == -INFINITY) ? 0.f : sm * __expf(m - bm);
        if (lane == 0) red[warp][rq] = contrib;
        __syncthreads();
        if (threadIdx.x == 0 && r0 + rq < R) {
          float tot = 0.f;
          for (int w = 0; w < NT / 32; ++w) tot += red[w][rq];
          stats[(out_row[rq] * nblk + blk) * 2 + 0] = bm;
          stats[(out_row[rq] * nblk + blk) * 2 + 1] = tot;
        }
        __syncthreads();
      }
    }
  }
}

// probs = exp(l - M) / Z with (M, Z) folded from the per-block partials.
__global__ void __launch_bounds__(NT) k_softmax_finish(const float* logits, const float* stats, int nblk, int64_t Sk, float* probs) {
  __shared__ float sh_m, sh_z;
  pdl_wait();
  const int64_t row = blockIdx.x;
  if (threadIdx.x < 32) {
    float m = -INFINITY;
    for (int i = threadIdx.x; i < nblk; i += 32) m = fmaxf(m, stats[(row * nblk + i) * 2]);
    m = warp_max(m);
    float z = 0.f;
    for (int i = threadIdx.x; i < nblk; i += 32) {
      float pm = stats[(row * nblk + i) * 2];
      if (pm != -INFINITY) z += stats[(row * nblk + i) * 2 + 1] * __expf(pm - m);
    }
    z = warp_sum(z);
    if (threadIdx.x == 0) { sh_m = m; sh_z = z; }
  }
  __syncthreads();
  const float m = sh_m, inv = 1.f / sh_z;
  const int64_t per = ((Sk + gridDim.y - 1) / gridDim.y + 3) / 4 * 4;
  const int64_t lo = blockIdx.y * per, hi = min(lo + per, Sk);
  const float* src = logits + row * Sk;
  float* dst = probs + row * Sk;
  if ((Sk & 3) == 0 && (((uintptr_t)src | (uintptr_t)dst) & 15u) == 0) {     // 16-byte rows: four logits per access
    for (int64_t s = lo + 4 * (int64_t)threadIdx.x; s < hi; s += 4 * NT) {
      const float4 l = *reinterpret_cast<const float4*>(src + s);
      float4 p;
      p.x = __expf(l.x - m) * inv; p.y = __expf(l.y - m) * inv; p.z = __expf(l.z - m) * inv; p.w = __expf(l.w - m) * inv;
      *reinterpret_cast<float4*>(dst + s) = p;
    }
  } else {
    for (int64_t s = lo + threadIdx.x; s < hi; s += NT) dst[s] = __expf(src[s] - m) * inv;
  }
}

// ---------------------------------------------------------------------------
// K4: MSE stage + QJL signs on one resident tile
// ---------------------------------------------------------------------------
template <int XDT, int NJ, int NJM, int RI>
__global__ void __launch_bounds__(NT) k_qjl_compress(TqQjlCompressJob job) {
  constexpr int TM = 16 * RI;                   // vectors per tile
  extern __shared__ __align__(16) float smem[];
  const int D = job.D, M = job.M;
  const int lda = lda_for(D);
  constexpr int NJB = (NJ > NJM) ? NJ : NJM;
  float* Xs = smem;
  float* As = Xs + TM * lda;
  float* Bs = As + TM * lda;
  float* cent_s = Bs + b_ring_floats(NJB);
  float* thr_s = cent_s + 256;
  float* nrm = thr_s + 256;
  load_codebook(job.codebook, cent_s, thr_s);
  const int64_t n_total = job.B * job.H * job.S;
  const int64_t tiles = (n_total + TM - 1) / TM;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tx = tile_tx(), ty = tile_ty();
  const int kpad = round_up(D, KC);
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int64_t row0 = tile * TM;
    __syncthreads();
    b_begin<NJ, B_KN>(D, job.rotation_t, D, D, Bs);
    load_tile_rows<XDT, RI>(job.x, row0, n_total, D, job.H, job.S, job.stride_b, job.stride_h, job.stride_s, Xs, lda,
                        job.normalize ? nrm : nullptr, As);
    {
      float acc[RI][4 * NJ];
      zero_acc<RI, NJ>(acc);
      tile_gemm<RI, NJ, B_KN>(As, lda, D, job.rotation_t, D, D, Bs, acc);
      __syncthreads();
      b_begin<NJ, B_KN>(D, job.rotation, D, D, Bs);
      acc_to_smem<RI, NJ>(acc, As, lda, kpad);
    }
    __syncthreads();
    // quantise in place: As <- centroid of the nearest level
#pragma unroll 1
    for (int r = warp; r < TM; r += 4 * (NT / 32)) {
      for (int c0 = lane; c0 < kpad; c0 += 128) {
        float y[16];
        int q[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) y[u] = c0 + 32 * (u & 3) < D ? As[(r + 8 * (u >> 2)) * lda + c0 + 32 * (u & 3)] : 0.f;
        quantize_many<16>(y, thr_s, job.bits, q);
#pragma unroll
        for (int u = 0; u < 16; ++u) {
          const int c = c0 + 32 * (u & 3), rr = r + 8 * (u >> 2);
          const int64_t n = row0 + rr;
          if (c < D && job.idx_out != nullptr && n < n_total) {
            if (job.idx_mode == TQ_IDX_I64) reinterpret_cast<int64_t*>(job.idx_out)[n * D + c] = q[u];
            else if (job.idx_mode == TQ_IDX_U8) reinterpret_cast<uint8_t*>(job.idx_out)[n * D + c] = (uint8_t)q[u];
          }
          if (c < kpad) As[rr * lda + c] = c < D ? cent_s[q[u]] : 0.f;
        }
      }
    }
    {
      float acc[RI][4 * NJ];
      zero_acc<RI, NJ>(acc);
      tile_gemm<RI, NJ, B_KN>(As, lda, D, job.rotation, D, D, Bs, acc);
      __syncthreads();
      b_begin<NJM, B_KN>(D, job.qjl_t, M, M, Bs);
      // k_mse (fp32) -> optional fp16 output; residual = x - k_mse back into As
#pragma unroll
      for (int ri = 0; ri < RI; ++ri) {
        int r = ty * RI + ri;
        int64_t n = row0 + r;
        float nv = job.normalize ? nrm[r] : 1.f;
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            int col = tx * 4 + 64 * j + c;
            if (col < kpad) {
              float km = job.normalize ? acc[ri][4 * j + c] * nv : acc[ri][4 * j + c];
              if (col >= D) km = 0.f;
              if (job.k_mse_out != nullptr && n < n_total && col < D)
                job.k_mse_out[n * D + col] = __half_as_ushort(__float2half_rn(km));
              As[r * lda + col] = (col < D) ? Xs[r * lda + col] - km : 0.f;
            }
          }
      }
    }
    __syncthreads();
    for (int r = warp; r < TM; r += NT / 32) {
      float ssq = 0.f;
      for (int k = lane; k < D; k += 32) ssq = fmaf(As[r * lda + k], As[r * lda + k], ssq);
      ssq = warp_sum(ssq);
      int64_t n = row0 + r;
      if (lane == 0 && n < n_total) {
        float rn = __fsqrt_rn(ssq);
        if (job.rnorm_dtype == TQ_F16) reinterpret_cast<uint16_t*>(job.rnorm_out)[n] = __half_as_ushort(__float2half_rn(rn));
        else reinterpret_cast<float*>(job.rnorm_out)[n] = rn;
        if (job.vec_norms_out != nullptr && job.normalize) job.vec_norms_out[n] = nrm[r];
      }
    }
    {
      float acc[RI][4 * NJM];
      zero_acc<RI, NJM>(acc);
      tile_gemm<RI, NJM, B_KN>(As, lda, D, job.qjl_t, M, M, Bs, acc);
#pragma unroll
      for (int ri = 0; ri < RI; ++ri) {
        int64_t n = row0 + ty * RI + ri;
        if (n >= n_total) continue;
#pragma unroll
        for (int j = 0; j < NJM; ++j)
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            int col = tx * 4 + 64 * j + c;
            if (col < M) {
              float p = acc[ri][4 * j + c];
              if (job.signs_dtype == 0) {
                reinterpret_cast<int8_t*>(job.signs_out)[n * M + col] = (p >= 0.f) ? (int8_t)1 : (int8_t)-1;
              } else {
                float sg = (p > 0.f) ? 1.f : (p < 0.f) ? -1.f : (p == 0.f) ? 1.f : p;
                reinterpret_cast<float*>(job.signs_out)[n * M + col] = sg;
              }
            }
          }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// K5: scores = Q k_mse^T + sqrt(pi/2)/m * (Q S^T) signs^T * ||r||
// Tile rows are keys; columns are queries (chunks of up to 256).
// ---------------------------------------------------------------------------
template <int QDT, int NJ>
__global__ void __launch_bounds__(NT) k_qjl_scores(TqQjlScoreJob job, const float* __restrict__ qproj, float corr) {
  extern __shared__ __align__(16) float smem[];
  const int D = job.D;
  const int lda = lda_for(D);
  float* As = smem;
  float* Bs = As + TM * lda;
  float* Cs = Bs + b_ring_floats(NJ);   // [64*NJ][TM+1]
  const int ldc = TM + 1;
  const int64_t key_tiles = (job.Sk + TM - 1) / TM;
  const int64_t total = job.BH * key_tiles;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tx = tile_tx(), ty = tile_ty();
  const int kpad = round_up(D, KC);
  for (int64_t t = blockIdx.x; t < total; t += gridDim.x) {
    const int64_t bh = t / key_tiles;
    const int64_t s0 = (t % key_tiles) * TM;
    const uint16_t* km = job.k_mse + (bh * job.Sk) * D;
    const int8_t* sg = job.signs + (bh * job.Sk) * D;
    for (int q0 = 0; q0 < job.Sq; q0 += 64 * NJ) {
      const int nq = (int)min((int64_t)(64 * NJ), job.Sq - q0);
      float acc1[4][4 * NJ], acc2[4][4 * NJ];
      zero_acc<4, NJ>(acc1);
      zero_acc<4, NJ>(acc2);
      __syncthreads();
      for (int r = warp; r < TM; r += NT / 32) {
        int64_t s = s0 + r;
        for (int k = lane; k < kpad; k += 32)
          As[r * lda + k] = (s < job.Sk && k < D) ? __half2float(__ushort_as_half(km[s * D + k])) : 0.f;
      }
      // queries as B in [N][K] layout, converted to fp32 on the fly for 16-bit q
      // (16-bit queries were upcast into the workspace behind qproj by the host wrapper)
      const float* qf = QDT == TQ_F32 ? reinterpret_cast<const float*>(job.q) + (bh * job.Sq + q0) * D
                                      : qproj + (job.BH * job.Sq + bh * job.Sq + q0) * D;
      b_begin<NJ, B_NK>(D, qf, D, nq, Bs);
      tile_gemm<4, NJ, B_NK>(As, lda, D, qf, D, nq, Bs, acc1);
      __syncthreads();
      for (int r = warp; r < TM; r += NT / 32) {
        int64_t s = s0 + r;
        for (int k = lane; k < kpad; k += 32) As[r * lda + k] = (s < job.Sk && k < D) ? (float)sg[s * D + k] : 0.f;
      }
      b_begin<NJ, B_NK>(D, qproj + (bh * job.Sq + q0) * D, D, nq, Bs);
      tile_gemm<4, NJ, B_NK>(As, lda, D, qproj + (bh * job.Sq + q0) * D, D, nq, Bs, acc2);
      __syncthreads();
#pragma unroll
      for (int ri = 0; ri < 4; ++ri) {
        int r = ty * 4 + ri;
        int64_t s = s0 + r;
        float rn = (s < job.Sk) ? __half2float(__ushort_as_half(job.rnorm[bh * job.Sk + s])) : 0.f;
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            int col = tx * 4 + 64 * j + c;
            float t2 = (corr * acc2[ri][4 * j + c]) * rn;
            Cs[col * ldc + r] = acc1[ri][4 * j + c] + t2;
          }
      }
      __syncthreads();
      for (int col = warp; col < nq; col += NT / 32) {
        float* o = job.scores + (bh * job.Sq + q0 + col) * job.Sk + s0;
        for (int r = lane; r < TM; r += 32)
          if (s0 + r < job.Sk) o[r] = Cs[col * ldc + r];
      }
    }
  }
}

// Query operand of the tensor-core score kernel (tq_qjl_umma.cu), head_dim a multiple of 64: per unit (head, block of
// 16 or 64 queries) the rows [Q | corr * Q S^T] as fp16 pieces hi + lo, laid out [chunk of 64 columns][piece][row][64], rows of
// 128 bytes with 16-byte chunk c at c ^ (row & 7); rows past Sq are zero.  A CTA takes 16 or 32 rows and 64 columns: the
// projection (one sequential chain per output, as tq_project), then the query's own columns and the projected ones.
// 1024 queries of head_dim 256 took 27 us as projection, upcast and image kernels (the projection read the whole matrix
// for every four rows).
template <int QDT, int RI>
__global__ void __launch_bounds__(NT) k_qjl_query_operand(const void* q, int D, int64_t Sq, int n_qblocks, int per_unit,
                                                         const float* __restrict__ qjl_t, float corr, uint8_t* __restrict__ images) {
  constexpr int ROWS = 16 * RI;
  pdl_trigger();
  extern __shared__ __align__(16) float smem[];
  const int lda = lda_for(D);
  float* As = smem;
  float* Bs = As + ROWS * lda;
  const int chunks = D / 64;
  const int groups = per_unit / ROWS;
  const int cb = blockIdx.x % chunks, group = (blockIdx.x / chunks) % groups, unit = blockIdx.x / (groups * chunks);
  const int64_t bh = unit / n_qblocks;
  const int64_t q0 = (int64_t)(unit % n_qblocks) * per_unit + group * ROWS;       // first query of this CTA, of head bh
  b_begin<1, B_KN>(D, qjl_t + cb * 64, D, 64, Bs);
  // rows past the end of this head read as zero, so the row limit is the head's own end
  load_tile_rows<QDT, RI>(q, bh * Sq + q0, (bh + 1) * Sq, D, 1, (bh + 1) * Sq, 0, 0, D, As, lda, nullptr);
  float acc[RI][4];
  zero_acc<RI, 1>(acc);
  tile_gemm<RI, 1, B_KN>(As, lda, D, qjl_t + cb * 64, D, 64, Bs, acc);
  const int tx = tile_tx(), ty = tile_ty();
  const size_t piece = (size_t)per_unit * 64;                              // elements of one piece of a chunk
  uint16_t* img = reinterpret_cast<uint16_t*>(images) + (size_t)unit * 2 * chunks * 2 * piece;
#pragma unroll
  for (int ri = 0; ri < RI; ++ri) {
    const int r = ty * RI + ri, n = group * ROWS + r;
#pragma unroll
    for (int part = 0; part < 2; ++part) {                                 // the query's columns, then the projected ones
      uint16_t hi[4], lo[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float v = part == 0 ? As[r * lda + cb * 64 + 4 * tx + c] : corr * acc[ri][c];
        const __half h = __float2half_rn(v);
        hi[c] = __half_as_ushort(h);
        lo[c] = __half_as_ushort(__float2half_rn(v - __half2float(h)));
      }
      const size_t off = (size_t)(part * chunks + cb) * 2 * piece + (size_t)n * 64 + (size_t)((((4 * tx) >> 3) ^ (n & 7)) * 8 + ((4 * tx) & 7));
      *reinterpret_cast<uint2*>(img + off) = make_uint2(hi[0] | ((uint32_t)hi[1] << 16), hi[2] | ((uint32_t)hi[3] << 16));
      *reinterpret_cast<uint2*>(img + piece + off) = make_uint2(lo[0] | ((uint32_t)lo[1] << 16), lo[2] | ((uint32_t)lo[3] << 16));
    }
  }
}

// upcast a 16-bit tensor to fp32
template <int XDT>
__global__ void k_upcast(const void* x, int64_t n, float* out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = load_elem<XDT>(x, i);
}

// out[n] = <y_n, xhat_n> + (rnorm_n * corr) * <sy_n, signs_n>
__global__ void __launch_bounds__(NT) k_prod_inner(const float* __restrict__ y, int64_t ny, const float* __restrict__ xhat,
                                                  const float* __restrict__ sy, const float* __restrict__ signs,
                                                  const float* __restrict__ rnorm, int64_t n, int D, int M, float corr,
                                                  float* out) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t wstride = (int64_t)gridDim.x * (NT / 32);
  for (int64_t r = (int64_t)blockIdx.x * (NT / 32) + warp; r < n; r += wstride) {
    const int64_t yr = (ny == 1) ? 0 : r;
    float t1 = 0.f, ip = 0.f;
    for (int k = lane; k < D; k += 32) t1 = fmaf(y[yr * D + k], xhat[r * D + k], t1);
    for (int k = lane; k < M; k += 32) ip = fmaf(sy[yr * M + k], signs[r * M + k], ip);
    t1 = warp_sum(t1);
    ip = warp_sum(ip);
    if (lane == 0) out[r] = t1 + (rnorm[r] * corr) * ip;
  }
}

// One query against every vector: <y, c[idx] Pi> = <y Pi^T, c[idx]>, so the query is rotated once instead of every
// vector being rotated back.  k_query_rotate computes yr = y Pi^T and sy = y S^T.
__global__ void __launch_bounds__(NT) k_query_rotate(const float* __restrict__ y, int D, int M, const float* __restrict__ rotation,
                                                    const float* __restrict__ qjl_t, float* yr, float* sy) {
  __shared__ float ys[TQ_MAX_DIM];
  __shared__ float part[NT / 32][33];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int k = threadIdx.x; k < D; k += NT) ys[k] = y[k];
  __syncthreads();
  const int row_blocks = (D + 7) / 8;
  if ((int)blockIdx.x < row_blocks) {                 // a warp per row of Pi
    const int j = blockIdx.x * 8 + warp;
    float t = 0.f;
    if (j < D)
      for (int k = lane; k < D; k += 32) t = fmaf(ys[k], __ldg(rotation + (int64_t)j * D + k), t);
    t = warp_sum(t);
    if (lane == 0 && j < D) yr[j] = t;
  } else {                                            // 32 columns of S^T, its rows split over the warps
    const int m = ((int)blockIdx.x - row_blocks) * 32 + lane;
    float t = 0.f;
    if (m < M)
#pragma unroll 8
      for (int k = warp; k < D; k += NT / 32) t = fmaf(ys[k], __ldg(qjl_t + (int64_t)k * M + m), t);
    part[warp][lane] = t;
    __syncthreads();
    if (warp == 0 && m < M) {
      float a = 0.f;
#pragma unroll
      for (int w = 0; w < NT / 32; ++w) a += part[w][lane];
      sy[m] = a;
    }
  }
}

// out[n] = <yr, c[idx_n]> + (rnorm_n * corr) * <sy, signs_n>: a warp per vector, bound by reading the 8-byte indices and
// 4-byte signs once.  8192 vectors of head_dim 128: 52 us as dequantise, projection and row products, 8 us so.
__global__ void __launch_bounds__(NT) k_prod_inner_one(const int64_t* __restrict__ idx, const float* __restrict__ signs,
                                                      const float* __restrict__ rnorm, int64_t n, int D, int M,
                                                      const float* __restrict__ cb, const float* __restrict__ yr,
                                                      const float* __restrict__ sy, float corr, float* out) {
  __shared__ float cent_s[256];
  __shared__ float yr_s[TQ_MAX_DIM], sy_s[TQ_MAX_DIM];
  for (int i = threadIdx.x; i < 256; i += NT) {
    cent_s[i] = __ldg(cb + kCentroidOff + i);
    if (i < D) yr_s[i] = yr[i];
    if (i < M) sy_s[i] = sy[i];
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t wstride = (int64_t)gridDim.x * (NT / 32);
  for (int64_t r = (int64_t)blockIdx.x * (NT / 32) + warp; r < n; r += wstride) {
    float t1 = 0.f, ip = 0.f;
#pragma unroll 4
    for (int k = lane; k < D; k += 32) t1 = fmaf(yr_s[k], cent_s[(int)(__ldg(idx + r * D + k) & 255)], t1);
#pragma unroll 4
    for (int k = lane; k < M; k += 32) ip = fmaf(sy_s[k], __ldg(signs + r * M + k), ip);
    t1 = warp_sum(t1);
    ip = warp_sum(ip);
    if (lane == 0) out[r] = t1 + (rnorm[r] * corr) * ip;
  }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
static thread_local int g_last_cuda_error = 0;
static std::atomic<long long> g_launches{0};
int last_cuda_error() { return g_last_cuda_error; }
long long launch_count() { return g_launches.load(); }
void note_cuda_error(int e) { g_last_cuda_error = e; }
int refused(cudaError_t e) {
  g_last_cuda_error = (int)e;
  cudaGetLastError();                            // it is this call's error: the next launch must not find it
  return TQ_ELAUNCH;
}

int check_launch() {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { g_last_cuda_error = (int)e; return TQ_ELAUNCH; }
  g_launches.fetch_add(1);
  return TQ_OK;
}

static int sm_count() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 148;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
  return n;
}

static int grid_for(int64_t tiles, int per_sm) {
  int64_t cap = (int64_t)sm_count() * per_sm;
  return (int)(tiles < cap ? (tiles > 0 ? tiles : 1) : cap);
}

template <typename K>
static int set_smem(K kernel, size_t bytes) {
  if (bytes > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return refused(e);
  }
  return TQ_OK;
}

static inline int nj_for(int n) { return (n + 63) / 64; }

// Vectors per tile: 64 (RI = 4) where an SM would get two tiles of 32 (RI = 2), which load more from shared memory per multiply-add
// (see tile_gemm).  One contraction of head_dim 128: 12 300 clocks for one tile of 32 on an SM, 20 000 for two, 15 700 for one of 64.
// Head_dim 128 in fp32: 4096 vectors quantised in 16.6 -> 14.4 us, 8192 in 22.7 -> 18.6 (32-vector tiles before), 16384 in 41 -> 27
// and 100 000 in 160 -> 130 (operands of 64-vector tiles loaded four k at a time, two columns an instruction).
static inline bool small_tiles(int64_t n) { return n <= (int64_t)(TM / 2) * sm_count(); }

#define TQ_DISPATCH_NJ(nj, ...)                              \
  switch (nj) {                                              \
    case 1: { constexpr int NJ_ = 1; __VA_ARGS__; } break;   \
    case 2: { constexpr int NJ_ = 2; __VA_ARGS__; } break;   \
    case 3: { constexpr int NJ_ = 3; __VA_ARGS__; } break;   \
    default: { constexpr int NJ_ = 4; __VA_ARGS__; } break;  \
  }

#define TQ_DISPATCH_DT(dt, ...)                                         \
  switch (dt) {                                                         \
    case TQ_F32: { constexpr int DT_ = TQ_F32; __VA_ARGS__; } break;    \
    case TQ_F16: { constexpr int DT_ = TQ_F16; __VA_ARGS__; } break;    \
    default: { constexpr int DT_ = TQ_BF16; __VA_ARGS__; } break;       \
  }

int simt_quantize_rotated(const float* y, int64_t n, int D, int bits, const float* cb, int mode, void* out,
                          cudaStream_t st) {
  if (n == 0) return TQ_OK;
  int grid = grid_for((n + NT / 32 - 1) / (NT / 32), 8);
  k_quantize_rotated<<<grid, NT, 0, st>>>(y, n, D, bits, cb, mode, out);
  return check_launch();
}

int simt_quantize(const TqQuantizeJob& job, cudaStream_t st) {
  const int64_t n = job.B * job.H * job.S;
  if (n == 0) return TQ_OK;
  const int nj = nj_for(job.D);
  const bool small = small_tiles(n);
  const int tm = small ? TM / 2 : TM;
  const size_t smem = sizeof(float) * (tm * lda_for(job.D) + b_ring_floats(nj) + 512 + tm);
  const int grid = grid_for((n + tm - 1) / tm, 2);
  int rc = TQ_OK;
  TQ_DISPATCH_DT(job.x_dtype, TQ_DISPATCH_NJ(nj, {
    auto kern = small ? k_quantize<DT_, NJ_, 2> : k_quantize<DT_, NJ_, 4>;
    rc = set_smem(kern, smem);
    if (rc == TQ_OK) kern<<<grid, NT, smem, st>>>(job);
  }));
  return rc != TQ_OK ? rc : check_launch();
}

int simt_dequantize(const TqDequantizeJob& job, cudaStream_t st) {
  const int64_t n = job.B * job.H * job.S;
  if (n == 0) return TQ_OK;
  const int nj = nj_for(job.D);
  const bool small = small_tiles(n);
  const int tm = small ? TM / 2 : TM;
  const size_t smem = sizeof(float) * (tm * lda_for(job.D) + b_ring_floats(nj) + 512);
  const int grid = grid_for((n + tm - 1) / tm, 2);
  int rc = TQ_OK;
  TQ_DISPATCH_DT(job.out_dtype, TQ_DISPATCH_NJ(nj, {
    auto kern = small ? k_dequantize<DT_, NJ_, 2> : k_dequantize<DT_, NJ_, 4>;
    rc = set_smem(kern, smem);
    if (rc == TQ_OK) kern<<<grid, NT, smem, st>>>(job);
  }));
  return rc != TQ_OK ? rc : check_launch();
}

int simt_project(const void* x, int x_dtype, int64_t n, int K, const float* m, int N, float* out, cudaStream_t st, bool followed) {
  if (n == 0) return TQ_OK;
  if (n <= 8192) {         // few rows: a 64-row tile kernel would run on a handful of SMs
    const int threads = N <= 128 ? 128 : 256;
    if (n <= 512) {
      TQ_DISPATCH_DT(x_dtype, (k_project_rows<DT_, 1><<<(unsigned)n, threads, 0, st>>>(x, n, K, m, N, out, followed)));
    } else {
      TQ_DISPATCH_DT(x_dtype, (k_project_rows<DT_, 4><<<(unsigned)((n + 3) / 4), threads, 0, st>>>(x, n, K, m, N, out, followed)));
    }
    return check_launch();
  }
  const int nj = nj_for(N);
  const size_t smem = sizeof(float) * (TM * lda_for(K) + b_ring_floats(nj));
  const int grid = grid_for((n + TM - 1) / TM, 2);
  int rc = TQ_OK;
  TQ_DISPATCH_DT(x_dtype, TQ_DISPATCH_NJ(nj, {
    auto kern = k_project<DT_, NJ_>;
    rc = set_smem(kern, smem);
    if (rc == TQ_OK) kern<<<grid, NT, smem, st>>>(x, n, K, m, N, out);
  }));
  return rc != TQ_OK ? rc : check_launch();
}

// Two projections of the same rows (head_dim square matrices) in one launch, or in two where the rows are many; a kernel
// launched with launch_after() follows.
int simt_project_two(const void* x, int x_dtype, int64_t n, int D, const float* m0, const float* m1, float* out0, float* out1,
                     cudaStream_t st) {
  if (n == 0) return TQ_OK;
  if (n <= 512) {
    const int threads = D <= 128 ? 128 : 256;
    TQ_DISPATCH_DT(x_dtype, (k_project_rows_two<DT_><<<dim3((unsigned)n, 2), threads, 0, st>>>(x, n, D, m0, m1, out0, out1)));
    return check_launch();
  }
  const int rc = simt_project(x, x_dtype, n, D, m0, D, out0, st);
  return rc != TQ_OK ? rc : simt_project(x, x_dtype, n, D, m1, D, out1, st, true);
}

size_t simt_score_workspace(int64_t B, int64_t Hq, int64_t Sq, int64_t Sk, int D) {
  const int64_t rows = B * Hq * Sq;
  const int64_t nblk = (Sk + SCORE_KEYS_PER_BLOCK - 1) / SCORE_KEYS_PER_BLOCK;
  size_t q = (size_t)rows * D * sizeof(float);
  q = (q + 255) / 256 * 256;
  return q + (size_t)rows * (nblk > 0 ? nblk : 1) * 2 * sizeof(float);
}

// Room for the partials of blocks of 128 keys, with which a short call fills the chip, up to a megabyte; never less than
// simt_score_workspace(), which every caller brings.
size_t score_workspace_wanted(int64_t B, int64_t Hq, int64_t Sq, int64_t Sk, int D) {
  const size_t least = simt_score_workspace(B, Hq, Sq, Sk, D);
  if (D != 128) return least;
  const int64_t rows = B * Hq * Sq;
  const size_t q = ((size_t)rows * D * sizeof(float) + 255) / 256 * 256;
  const size_t part = (size_t)rows * 2 * sizeof(float);
  size_t blocks = (size_t)((Sk + 127) / 128);
  if (blocks * part > ((size_t)1 << 20)) blocks = part > 0 ? ((size_t)1 << 20) / part : 0;
  const size_t want = q + blocks * part;
  return want > least && want <= TQ_SCORE_NOALLOC_SCRATCH_BYTES ? want : least;
}

int simt_score_packed(const TqScoreJob& job, cudaStream_t st) {
  const int64_t rows = job.B * job.Hq * job.Sq;
  if (rows == 0 || job.Sk == 0) return TQ_OK;
  // the tensor-core kernel takes its block size as a parameter, with as many blocks as the scratch has room for
  const bool use_mma = mma_score_eligible(job);
  float* qrot = reinterpret_cast<float*>(job.workspace);
  const size_t qbytes = ((size_t)rows * job.D * sizeof(float) + 255) / 256 * 256;
  float* stats = reinterpret_cast<float*>(reinterpret_cast<char*>(job.workspace) + qbytes);
  const int64_t most = (int64_t)((job.workspace_bytes - qbytes) / ((size_t)rows * 2 * sizeof(float)));
  const int kpb = use_mma ? mma_score_keys_per_block(job, most) : SCORE_KEYS_PER_BLOCK;
  const int nblk = (int)((job.Sk + kpb - 1) / kpb);
  int rc = simt_project(job.q, job.q_dtype, rows, job.D, job.rotation_t, job.D, qrot, st, use_mma);
  if (rc != TQ_OK) return rc;
  const int64_t blocks = job.B * job.Hkv * nblk;
  float* st_ptr = job.probs != nullptr ? stats : nullptr;
  if (use_mma) {
    rc = mma_score_packed(job, qrot, st_ptr, nblk, kpb, st);
    if (rc != TQ_OK) return rc;
  } else if (job.D == 128 && ((uintptr_t)job.idx_bytes & 15u) == 0) {
    switch (job.bits) {
      case 1: k_score_packed_d128<1><<<(unsigned)blocks, NT, 0, st>>>(job, qrot, st_ptr, nblk); break;
      case 2: k_score_packed_d128<2><<<(unsigned)blocks, NT, 0, st>>>(job, qrot, st_ptr, nblk); break;
      case 3: k_score_packed_d128<3><<<(unsigned)blocks, NT, 0, st>>>(job, qrot, st_ptr, nblk); break;
      case 4: k_score_packed_d128<4><<<(unsigned)blocks, NT, 0, st>>>(job, qrot, st_ptr, nblk); break;
      case 5: k_score_packed_d128<5><<<(unsigned)blocks, NT, 0, st>>>(job, qrot, st_ptr, nblk); break;
      case 6: k_score_packed_d128<6><<<(unsigned)blocks, NT, 0, st>>>(job, qrot, st_ptr, nblk); break;
      case 7: k_score_packed_d128<7><<<(unsigned)blocks, NT, 0, st>>>(job, qrot, st_ptr, nblk); break;
      default: k_score_packed_d128<8><<<(unsigned)blocks, NT, 0, st>>>(job, qrot, st_ptr, nblk); break;
    }
  } else {
    k_score_packed<<<(unsigned)blocks, NT, 0, st>>>(job, qrot, st_ptr, nblk);
  }
  if (!use_mma) rc = check_launch();
  if (rc != TQ_OK || job.probs == nullptr) return rc;
  int chunks = (int)((job.Sk + 4095) / 4096);
  dim3 grid((unsigned)rows, (unsigned)chunks);
  if (use_mma) launch_after(k_softmax_finish, grid, dim3(NT), 0, st, job.logits, stats, nblk, job.Sk, job.probs);
  else k_softmax_finish<<<grid, NT, 0, st>>>(job.logits, stats, nblk, job.Sk, job.probs);
  return check_launch();
}

int simt_qjl_compress(const TqQjlCompressJob& job, cudaStream_t st) {
  const int64_t n = job.B * job.H * job.S;
  if (n == 0) return TQ_OK;
  const int nj = nj_for(job.D), njm = nj_for(job.M);
  const int njb = nj > njm ? nj : njm;
  const bool small = small_tiles(n);
  const int tm = small ? TM / 2 : TM;
  const size_t smem = sizeof(float) * (2 * tm * lda_for(job.D) + b_ring_floats(njb) + 512 + tm);
  const int grid = grid_for((n + tm - 1) / tm, small ? 2 : 1);
  int rc = TQ_OK;
  // the projection width shares the head_dim's tile class unless it is wider
  TQ_DISPATCH_DT(job.x_dtype, TQ_DISPATCH_NJ(njb, {
    auto kern = small ? k_qjl_compress<DT_, NJ_, NJ_, 2> : k_qjl_compress<DT_, NJ_, NJ_, 4>;
    rc = set_smem(kern, smem);
    if (rc == TQ_OK) kern<<<grid, NT, smem, st>>>(job);
  }));
  return rc != TQ_OK ? rc : check_launch();
}

size_t simt_qjl_scores_workspace(int64_t BH, int64_t Sq, int D) {
  return (size_t)2 * BH * Sq * D * sizeof(float);   // projected queries + room for upcast queries
}

int simt_qjl_query_operand(const TqQjlScoreJob& job, void* images, int per_unit, cudaStream_t st) {
  const int n_qblocks = (int)((job.Sq + per_unit - 1) / per_unit);
  const int rows = per_unit == 16 ? 16 : 32;
  const int64_t blocks = job.BH * n_qblocks * (per_unit / rows) * (job.D / 64);
  const size_t smem = sizeof(float) * (rows * lda_for(job.D) + b_ring_floats(1));
  const float corr = (float)(1.2533141373155001 / (double)job.D);   // sqrt(pi/2) / m with m = D
  int rc = TQ_OK;
  TQ_DISPATCH_DT(job.q_dtype, {
    auto kern = rows == 16 ? k_qjl_query_operand<DT_, 1> : k_qjl_query_operand<DT_, 2>;
    rc = set_smem(kern, smem);
    if (rc == TQ_OK) kern<<<(unsigned)blocks, NT, smem, st>>>(job.q, job.D, job.Sq, n_qblocks, per_unit, job.qjl_t, corr, reinterpret_cast<uint8_t*>(images));
  });
  return rc != TQ_OK ? rc : check_launch();
}

int simt_qjl_queries(const TqQjlScoreJob& job, const float** qf_out, const float** qproj_out, cudaStream_t st) {
  float* qproj = reinterpret_cast<float*>(job.workspace);
  const int64_t nq = job.BH * job.Sq;
  int rc = simt_project(job.q, job.q_dtype, nq, job.D, job.qjl_t, job.D, qproj, st);
  if (rc != TQ_OK) return rc;
  const float* qf = reinterpret_cast<const float*>(job.q);
  if (job.q_dtype != TQ_F32) {
    float* up = qproj + nq * job.D;
    int g = grid_for((nq * job.D + 255) / 256, 8);
    if (job.q_dtype == TQ_F16) k_upcast<TQ_F16><<<g, 256, 0, st>>>(job.q, nq * job.D, up);
    else k_upcast<TQ_BF16><<<g, 256, 0, st>>>(job.q, nq * job.D, up);
    rc = check_launch();
    if (rc != TQ_OK) return rc;
    qf = up;
  }
  *qf_out = qf;
  *qproj_out = qproj;
  return TQ_OK;
}

int simt_qjl_scores(const TqQjlScoreJob& job, cudaStream_t st) {
  if (job.BH == 0 || job.Sq == 0 || job.Sk == 0) return TQ_OK;
  const float* qf_unused = nullptr;
  const float* qproj_c = nullptr;
  int rc = simt_qjl_queries(job, &qf_unused, &qproj_c, st);
  if (rc != TQ_OK) return rc;
  const float* qproj = qproj_c;
  const int nj = nj_for((int)(job.Sq < 256 ? job.Sq : 256));
  const size_t smem = sizeof(float) * (TM * lda_for(job.D) + b_ring_floats(nj) + 64 * nj * (TM + 1));
  const int64_t tiles = job.BH * ((job.Sk + TM - 1) / TM);
  const int grid = grid_for(tiles, 1);
  const float corr = (float)(1.2533141373155001 / (double)job.D);   // sqrt(pi/2) / m with m = D
  if (job.q_dtype == TQ_F32) {
    TQ_DISPATCH_NJ(nj, {
      auto kern = k_qjl_scores<TQ_F32, NJ_>;
      rc = set_smem(kern, smem);
      if (rc == TQ_OK) kern<<<grid, NT, smem, st>>>(job, qproj, corr);
    });
  } else {
    TQ_DISPATCH_NJ(nj, {
      auto kern = k_qjl_scores<TQ_F16, NJ_>;
      rc = set_smem(kern, smem);
      if (rc == TQ_OK) kern<<<grid, NT, smem, st>>>(job, qproj, corr);
    });
  }
  return rc != TQ_OK ? rc : check_launch();
}

int simt_prod_inner_product(const float* y, int64_t ny, const int64_t* idx, const float* signs, const float* rnorm,
                            int64_t n, int D, int M, const float* rotation, const float* codebook, const float* qjl_t,
                            float* out, void* workspace, cudaStream_t st) {
  if (n == 0) return TQ_OK;
  const float corr = (float)(1.2533141373155001 / (double)M);
  if (ny == 1) {
    float *yr = reinterpret_cast<float*>(workspace), *sy = yr + 256;
    k_query_rotate<<<(unsigned)((D + 7) / 8 + (M + 31) / 32), NT, 0, st>>>(y, D, M, rotation, qjl_t, yr, sy);
    int rc = check_launch();
    if (rc != TQ_OK) return rc;
    const int grid = grid_for((n + NT / 32 - 1) / (NT / 32), 8);
    k_prod_inner_one<<<grid, NT, 0, st>>>(idx, signs, rnorm, n, D, M, codebook, yr, sy, corr, out);
    return check_launch();
  }
  float* xhat = reinterpret_cast<float*>(workspace);
  float* sy = xhat + n * 256;
  TqDequantizeJob dj{};
  dj.idx = idx; dj.norms = nullptr; dj.idx_mode = TQ_IDX_I64; dj.D = D; dj.bits = 8; dj.out_dtype = TQ_F32;
  dj.B = 1; dj.H = 1; dj.S = n; dj.out = xhat; dj.ostride_b = 0; dj.ostride_h = 0; dj.ostride_s = D;
  dj.rotation = rotation; dj.codebook = codebook;
  int rc = simt_dequantize(dj, st);
  if (rc != TQ_OK) return rc;
  rc = simt_project(y, TQ_F32, ny, D, qjl_t, M, sy, st);
  if (rc != TQ_OK) return rc;
  int grid = grid_for((n + NT / 32 - 1) / (NT / 32), 8);
  k_prod_inner<<<grid, NT, 0, st>>>(y, ny, xhat, sy, signs, rnorm, n, D, M, corr, out);
  return check_launch();
}

}  // namespace tq
