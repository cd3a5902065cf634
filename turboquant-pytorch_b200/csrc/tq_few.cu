// Quantise / dequantise for few vectors, many jobs: one token of every layer of a model that is generating, first of
// all.  Head_dim 64 or 128, fp32 arithmetic, the same chain of operations per value as the FP32 kernels in tq_simt.cu.
//
// What bounds such a call is not throughput: 32 layers x K and V x 8 heads are 512 vectors under 64 matrices.  The
// tensor-core kernels give each of them a tile of 128 rows (21 us to quantise, 16 us to rebuild; 10 and 10 here) and a tensor
// map that the host encodes anew on every call, because the token's address moves.  Here a CTA takes 16 vectors and 64 output
// columns of one job, fetches its half of the matrix (32 KB) with asynchronous copies while it reads the vectors, and
// everything a launch needs travels as plain pointers.

#include <cstddef>
#include <cstring>

#include "tq_common.cuh"
#include "tq_internal.h"

namespace tq {

namespace {

constexpr int kFewRows = 16;       // vectors per CTA
constexpr int kFewCols = 64;       // output columns per CTA
constexpr int kFewThreads = 256;   // thread = (row, 4 columns)
constexpr int kFewMaxJobs = 96;
constexpr int kFewSmall = 8;       // jobs of the launch form with the small parameter block

struct FewQuantJob {
  const void* x;
  const float* matrix;             // Pi^T
  const float* codebook;
  void* idx_out;
  uint16_t* norms_out;
  int64_t sb, sh, ss;
  int64_t n;                       // vectors
  int32_t H, S;
  int32_t bits, normalize, idx_mode, begin;     // begin: first CTA
};
struct FewDeqJob {
  const void* idx;
  const uint16_t* norms;
  const float* matrix;             // Pi
  const float* codebook;
  void* out;
  int64_t sb, sh, ss;
  int64_t n;
  int32_t H, S;
  int32_t bits, idx_mode, wide, begin;          // wide: rows of 16-bit outputs start on 8-byte boundaries, of fp32 on 16
};
template <typename Job, int J>
struct FewBatch {
  int32_t n_jobs, pad_;
  Job jobs[J];
};
static_assert(sizeof(FewBatch<FewQuantJob, kFewMaxJobs>) < 16384 && sizeof(FewBatch<FewDeqJob, kFewMaxJobs>) < 16384, "parameter space");

__device__ __forceinline__ void few_cp16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// the job this CTA belongs to
template <typename Job, int J>
__device__ __forceinline__ int few_find(const FewBatch<Job, J>& p) {
  int lo = 0, hi = p.n_jobs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if ((int)blockIdx.x >= p.jobs[mid].begin) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// rows of `matrix` (D x D), columns [col0, col0 + 64), into Bs[D][64]
template <int D>
__device__ __forceinline__ void few_load_matrix(const float* matrix, int col0, float* Bs) {
#pragma unroll
  for (int e = threadIdx.x; e < D * (kFewCols / 4); e += kFewThreads) {
    const int k = e / (kFewCols / 4), c = 4 * (e % (kFewCols / 4));
    few_cp16(Bs + k * kFewCols + c, matrix + k * D + col0 + c);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// acc[c] = sum_k As[row][k] * Bs[k][4 tx + c]: one chain in ascending k per output
template <int D>
__device__ __forceinline__ void few_gemm(const float* a_row, const float* Bs, int tx, float (&acc)[4]) {
  acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
#pragma unroll 8
  for (int k = 0; k < D; k += 4) {
    const float4 a = *reinterpret_cast<const float4*>(a_row + k);
    const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float4 b = *reinterpret_cast<const float4*>(Bs + (k + u) * kFewCols + 4 * tx);
      acc[0] = fmaf(av[u], b.x, acc[0]);
      acc[1] = fmaf(av[u], b.y, acc[1]);
      acc[2] = fmaf(av[u], b.z, acc[2]);
      acc[3] = fmaf(av[u], b.w, acc[3]);
    }
  }
}

template <int XDT, int D, int J>
__global__ void __launch_bounds__(kFewThreads) k_few_quantize(const __grid_constant__ FewBatch<FewQuantJob, J> p) {
  constexpr int kHalves = D / kFewCols, LDA = D + 4;
  __shared__ __align__(16) float Bs[D * kFewCols];
  __shared__ __align__(16) float As[kFewRows * LDA];
  __shared__ float thr_s[256];
  const FewQuantJob& job = p.jobs[few_find(p)];
  const int local = (int)blockIdx.x - job.begin;
  const int half = local % kHalves;
  const int64_t row0 = (int64_t)(local / kHalves) * kFewRows;
  few_load_matrix<D>(job.matrix, half * kFewCols, Bs);
  thr_s[threadIdx.x] = __ldg(job.codebook + kThresholdOff + threadIdx.x);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // a warp's two vectors: both loads first, then norm and scale as the FP32 kernels take them
  float v[2][D / 32];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int64_t n = row0 + warp + 8 * h;
    const int64_t off = n < job.n ? vec_offset(n, job.H, job.S, job.sb, job.sh, job.ss) : 0;
#pragma unroll
    for (int u = 0; u < D / 32; ++u) v[h][u] = n < job.n ? load_elem<XDT>(job.x, off + 32 * u + lane) : 0.f;
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int r = warp + 8 * h;
    float den = 1.f;
    if (job.normalize) {
      float ssq = 0.f;
#pragma unroll
      for (int u = 0; u < D / 32; ++u) ssq = fmaf(v[h][u], v[h][u], ssq);
      const float norm = __fsqrt_rn(warp_sum(ssq));
      if (lane == 0 && half == 0 && row0 + r < job.n) job.norms_out[row0 + r] = __half_as_ushort(__float2half_rn(norm));
      den = norm + 1e-8f;
    }
#pragma unroll
    for (int u = 0; u < D / 32; ++u) As[r * LDA + 32 * u + lane] = job.normalize ? __fdiv_rn(v[h][u], den) : v[h][u];
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float acc[4];
  few_gemm<D>(As + ty * LDA, Bs, tx, acc);
  __syncthreads();                                  // everyone has read its vectors: As takes the rotated values
  *reinterpret_cast<float4*>(As + ty * LDA + 4 * tx) = make_float4(acc[0], acc[1], acc[2], acc[3]);
  __syncthreads();
  const int bits = job.bits, levels = 1 << bits;
  if (job.idx_mode == TQ_IDX_PACKED) {              // 64 coordinates are whole bytes for every width
    const int ipb = 8 / bits, g = kFewCols / ipb, G = D / ipb;
    for (int e = threadIdx.x; e < kFewRows * g; e += kFewThreads) {
      const int r = e / g, b = e - r * g;
      if (row0 + r >= job.n) continue;
      unsigned byte = 0;
      for (int i = 0; i < ipb; ++i)
        byte |= (unsigned)quantize_scalar(As[r * LDA + b * ipb + i], thr_s, levels) << (bits * (ipb - 1 - i));
      reinterpret_cast<uint8_t*>(job.idx_out)[(row0 + r) * G + half * g + b] = (uint8_t)byte;
    }
  } else {
    for (int e = threadIdx.x; e < kFewRows * kFewCols; e += kFewThreads) {
      const int r = e / kFewCols, c = e % kFewCols;
      if (row0 + r >= job.n) continue;
      const int q = quantize_scalar(As[r * LDA + c], thr_s, levels);
      const int64_t at = (row0 + r) * D + half * kFewCols + c;
      if (job.idx_mode == TQ_IDX_U8) reinterpret_cast<uint8_t*>(job.idx_out)[at] = (uint8_t)q;
      else reinterpret_cast<int64_t*>(job.idx_out)[at] = q;
    }
  }
}

template <int ODT, int D, int J>
__global__ void __launch_bounds__(kFewThreads) k_few_dequantize(const __grid_constant__ FewBatch<FewDeqJob, J> p) {
  constexpr int kHalves = D / kFewCols, LDA = D + 4;
  __shared__ __align__(16) float Bs[D * kFewCols];
  __shared__ __align__(16) float As[kFewRows * LDA];
  __shared__ float cent_s[256];
  const FewDeqJob& job = p.jobs[few_find(p)];
  const int local = (int)blockIdx.x - job.begin;
  const int half = local % kHalves;
  const int64_t row0 = (int64_t)(local / kHalves) * kFewRows;
  few_load_matrix<D>(job.matrix, half * kFewCols, Bs);
  cent_s[threadIdx.x] = __ldg(job.codebook + kCentroidOff + threadIdx.x);
  // this thread's coordinates of the 16 vectors: all index loads first, then the look-ups
  const int bits = job.bits, ipb = 8 / bits, G = D / ipb;
  constexpr int kPer = kFewRows * D / kFewThreads;
  int q[kPer];
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const int e = threadIdx.x + u * kFewThreads, r = e / D, c = e % D;
    const int64_t n = row0 + r;
    q[u] = -1;
    if (n < job.n) {
      if (job.idx_mode == TQ_IDX_PACKED) {
        const unsigned byte = __ldg(reinterpret_cast<const uint8_t*>(job.idx) + n * G + c / ipb);
        q[u] = (int)((byte >> (bits * (ipb - 1 - c % ipb))) & ((1u << bits) - 1u));
      } else if (job.idx_mode == TQ_IDX_U8) {
        q[u] = (int)__ldg(reinterpret_cast<const uint8_t*>(job.idx) + n * D + c);
      } else {
        q[u] = (int)(__ldg(reinterpret_cast<const int64_t*>(job.idx) + n * D + c) & 255);
      }
    }
  }
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int64_t n = row0 + ty;
  const float nv = job.norms != nullptr && n < job.n ? __half2float(__ushort_as_half(__ldg(job.norms + n))) : 1.f;
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const int e = threadIdx.x + u * kFewThreads, r = e / D, c = e % D;
    As[r * LDA + c] = q[u] >= 0 ? cent_s[q[u]] : 0.f;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float acc[4];
  few_gemm<D>(As + ty * LDA, Bs, tx, acc);
  if (n >= job.n) return;
  if (job.norms != nullptr) { acc[0] *= nv; acc[1] *= nv; acc[2] *= nv; acc[3] *= nv; }
  const int64_t off = vec_offset(n, job.H, job.S, job.sb, job.sh, job.ss) + half * kFewCols + 4 * tx;
  if (!job.wide) {
#pragma unroll
    for (int c = 0; c < 4; ++c) store_elem<ODT>(job.out, off + c, acc[c]);
  } else if constexpr (ODT == TQ_F32) {
    *reinterpret_cast<float4*>(reinterpret_cast<float*>(job.out) + off) = make_float4(acc[0], acc[1], acc[2], acc[3]);
  } else if constexpr (ODT == TQ_F16) {
    const __half2 a = __floats2half2_rn(acc[0], acc[1]), b = __floats2half2_rn(acc[2], acc[3]);
    *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(job.out) + off) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
  } else {
    const __nv_bfloat162 a = __floats2bfloat162_rn(acc[0], acc[1]), b = __floats2bfloat162_rn(acc[2], acc[3]);
    *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(job.out) + off) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
  }
}

// A job of `n` vectors in slabs of S is mostly padding in tiles of `rows` when at most an eighth of them is filled.
bool mostly_padding(int64_t slabs, int64_t S, int D) {
  const int64_t rows = 16384 / D;                   // vectors per tile of the tensor-core kernels
  return 8 * S <= rows * ((S + rows - 1) / rows) && slabs > 0;
}

// Most vectors of one call that come here from the tensor-core kernels: 512 CTAs of 16 vectors and 64 columns at head_dim
// 128, 256 at 64, all resident at four per SM (592).
constexpr int64_t kFewVectors = 4096;
// Whether `n` vectors of `jobs` jobs, which take `tiles` tiles on the tensor cores, run faster here.  Time per call with new buffers,
// host included (bf16, 4 bits, quantise), head_dim 128: 9 us here up to about 1200 vectors, a CTA per SM, then 5 + 2.7 n / 1000;
// over there 5 + 8 tiles / 1000, at least 9.7 + 0.2 jobs (a tensor map and a rotation image each).  One job of 2000 slabs of 2
// tokens 17 here against 25 us there, 512 of 4 12.4 each, 256 of 8 12.4 against 10.2, 128 of 16 12.4 against 9.9; 8 jobs of 32
// slabs of 8 12.4 against 10.7, of 16 17.6 against 11.0; 64 jobs of 8 slabs of 1 14 against 21, of 8 18.7 against 21.  At head_dim 64
// this kernel reads half as much matrix and is the faster one throughout (4000 vectors in slabs of 8: 8.9 against 12.5; in slabs
// of 16 9 against 10).
bool few_faster(int D, int64_t n, int64_t tiles, int jobs) {
  return n <= kFewVectors && (D == 64 || n <= 3 * tiles || n <= 1216 + 64 * jobs);
}
// The same for calls that would run on the FP32 kernels, whose tiles of 32 vectors reuse the matrix more.  Quantise into
// int64 indices, here against there: head_dim 128, 1024 vectors 8.2 against 16.4 us, 2048 10.3 against 16.4, 4096 16.4 each (rebuilt
// 16.4 against 14.4), 8192 24.6 against 20.5; head_dim 64, 4096 vectors 8.3 against 8.8, 8192 10.4 against 11.0.
constexpr int64_t few_fp32(int D) { return D == 64 ? 8192 : 2048; }

template <int D, typename Batch, typename Few, typename K0, typename K1>
int launch_few(const Batch& b, int blocks, K0 small, K1 large, cudaStream_t st) {
  if (b.n_jobs <= kFewSmall) {
    static_assert(offsetof(Few, jobs) == offsetof(Batch, jobs), "a prefix");
    small<<<blocks, kFewThreads, 0, st>>>(reinterpret_cast<const Few&>(b));
  } else {
    large<<<blocks, kFewThreads, 0, st>>>(b);
  }
  return check_launch();
}

}  // namespace

// ---------------------------------------------------------------- dispatch
// True when a whole call runs here: jobs of one dtype and head_dim whose matrices start on 16 bytes.  Where any job could run
// on the tensor cores: each such job is mostly padding in their tiles and the call is faster here (a job that would take a
// launch of the FP32 kernels of its own counts a tile for each vector); where none could: at most few_fp32() vectors.  A call
// with other jobs among them stays in one launch over there.  The order of the jobs does not matter.
template <typename Job, typename Dtype, typename Matrix, typename Tensor>
static bool few_eligible(const Job* jobs, int n_jobs, Dtype dtype, Matrix matrix, Tensor on_tensor_cores) {
  if (force_simt()) return false;
  int64_t vectors = 0, tiles = 0;
  bool tensor = false;
  for (int k = 0; k < n_jobs; ++k) {
    const Job& j = jobs[k];
    if ((j.D != 64 && j.D != 128) || dtype(j) != dtype(jobs[0]) || j.D != jobs[0].D || ((uintptr_t)matrix(j) & 15u)) return false;
    if (j.B <= 0 || j.H <= 0 || j.S <= 0 || j.H > 65535 || j.S > 65535) return false;
    const int64_t n = j.B * j.H * j.S;
    vectors += n;
    if (vectors > kFewVectors && vectors > few_fp32(j.D)) return false;
    if (on_tensor_cores(j)) {
      if (!mostly_padding(j.B * j.H, j.S, j.D)) return false;
      tensor = true;
      const int64_t rows = 16384 / j.D;
      tiles += j.B * j.H * ((j.S + rows - 1) / rows);
    } else {
      tiles += n;
    }
  }
  if (n_jobs == 0) return false;
  return tensor ? few_faster(jobs[0].D, vectors, tiles, n_jobs) : vectors <= few_fp32(jobs[0].D);
}

bool few_quantize_eligible(const TqQuantizeJob* jobs, int n_jobs) {
  return few_eligible(jobs, n_jobs, [](const TqQuantizeJob& j) { return j.x_dtype; },
                      [](const TqQuantizeJob& j) { return j.rotation_t; }, umma_quantize_eligible);
}

int few_quantize(const TqQuantizeJob* jobs, int n_jobs, cudaStream_t st) {
  for (; n_jobs > kFewMaxJobs; jobs += kFewMaxJobs, n_jobs -= kFewMaxJobs) {
    const int rc = few_quantize(jobs, kFewMaxJobs, st);
    if (rc != TQ_OK) return rc;
  }
  FewBatch<FewQuantJob, kFewMaxJobs> b;
  b.n_jobs = n_jobs;
  const int D = jobs[0].D, dt = jobs[0].x_dtype;
  int blocks = 0;
  for (int i = 0; i < n_jobs; ++i) {
    const TqQuantizeJob& j = jobs[i];
    FewQuantJob& u = b.jobs[i];
    u.x = j.x; u.matrix = j.rotation_t; u.codebook = j.codebook; u.idx_out = j.idx_out; u.norms_out = j.norms_out;
    u.sb = j.stride_b; u.sh = j.stride_h; u.ss = j.stride_s;
    u.n = j.B * j.H * j.S; u.H = (int32_t)j.H; u.S = (int32_t)j.S;
    u.bits = j.bits; u.normalize = j.normalize; u.idx_mode = j.idx_mode; u.begin = blocks;
    blocks += (int)((u.n + kFewRows - 1) / kFewRows) * (D / kFewCols);
  }
  using Few = FewBatch<FewQuantJob, kFewSmall>;
#define TQ_FEW(DT, DD) launch_few<DD, FewBatch<FewQuantJob, kFewMaxJobs>, Few>(b, blocks, k_few_quantize<DT, DD, kFewSmall>, k_few_quantize<DT, DD, kFewMaxJobs>, st)
  if (D == 128) return dt == TQ_F32 ? TQ_FEW(TQ_F32, 128) : dt == TQ_F16 ? TQ_FEW(TQ_F16, 128) : TQ_FEW(TQ_BF16, 128);
  return dt == TQ_F32 ? TQ_FEW(TQ_F32, 64) : dt == TQ_F16 ? TQ_FEW(TQ_F16, 64) : TQ_FEW(TQ_BF16, 64);
#undef TQ_FEW
}

bool few_dequantize_eligible(const TqDequantizeJob* jobs, int n_jobs) {
  return few_eligible(jobs, n_jobs, [](const TqDequantizeJob& j) { return j.out_dtype; },
                      [](const TqDequantizeJob& j) { return j.rotation; }, umma_dequantize_eligible);
}

int few_dequantize(const TqDequantizeJob* jobs, int n_jobs, cudaStream_t st) {
  for (; n_jobs > kFewMaxJobs; jobs += kFewMaxJobs, n_jobs -= kFewMaxJobs) {
    const int rc = few_dequantize(jobs, kFewMaxJobs, st);
    if (rc != TQ_OK) return rc;
  }
  FewBatch<FewDeqJob, kFewMaxJobs> b;
  b.n_jobs = n_jobs;
  const int D = jobs[0].D, dt = jobs[0].out_dtype;
  int blocks = 0;
  for (int i = 0; i < n_jobs; ++i) {
    const TqDequantizeJob& j = jobs[i];
    FewDeqJob& u = b.jobs[i];
    u.idx = j.idx; u.norms = j.norms; u.matrix = j.rotation; u.codebook = j.codebook; u.out = j.out;
    u.sb = j.ostride_b; u.sh = j.ostride_h; u.ss = j.ostride_s;
    u.n = j.B * j.H * j.S; u.H = (int32_t)j.H; u.S = (int32_t)j.S;
    u.bits = j.bits; u.idx_mode = j.idx_mode; u.begin = blocks;
    // a thread stores four values: 16 bytes of fp32, 8 of a 16-bit type
    const uintptr_t align = dt == TQ_F32 ? 15u : 7u;
    u.wide = ((uintptr_t)j.out & align) == 0 && (j.B == 1 || j.ostride_b % 4 == 0) && (j.H == 1 || j.ostride_h % 4 == 0) &&
             (j.S == 1 || j.ostride_s % 4 == 0);
    blocks += (int)((u.n + kFewRows - 1) / kFewRows) * (D / kFewCols);
  }
  using Few = FewBatch<FewDeqJob, kFewSmall>;
#define TQ_FEW(DT, DD) launch_few<DD, FewBatch<FewDeqJob, kFewMaxJobs>, Few>(b, blocks, k_few_dequantize<DT, DD, kFewSmall>, k_few_dequantize<DT, DD, kFewMaxJobs>, st)
  if (D == 128) return dt == TQ_F32 ? TQ_FEW(TQ_F32, 128) : dt == TQ_F16 ? TQ_FEW(TQ_F16, 128) : TQ_FEW(TQ_BF16, 128);
  return dt == TQ_F32 ? TQ_FEW(TQ_F32, 64) : dt == TQ_F16 ? TQ_FEW(TQ_F16, 64) : TQ_FEW(TQ_BF16, 64);
#undef TQ_FEW
}

}  // namespace tq
