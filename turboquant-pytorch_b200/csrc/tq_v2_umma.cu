// Tensor-core (tcgen05 / TMEM / TMA) path for the MSE + QJL compress stage (K4), fp16 vectors,
// head_dim 128 or 256.  The reference's three chained D x D contractions
// (turboquant/compressors.py:83-120) run as three stages of one persistent kernel, each with its own
// epilogue; operands that are fp32 in the reference are carried as fp16 pieces
// hi + lo (lo reaches into fp16 subnormals), so products match an fp32 matmul to ~2^-21:
//
//   stage 1  y = x Pi^T            A = x (exact fp16), B = Pi hi/lo.  Epilogue: ||y|| = ||x||, scale,
//                                  nearest centroid by exact thresholds, one index byte per coordinate -> scratch
//   stage 2  k = (c Pi) ||x||      A = centroid pieces, which expander warps write into the operand ring from the
//                                  index bytes, B = Pi^T hi/lo (hi.hi + lo.hi + hi.lo).  Epilogue:
//                                  k_mse (fp16 out), residual r = x - k, ||r|| (out), residual pieces -> scratch
//   stage 3  p = r S^T             A = residual pieces, B = S hi/lo.  Epilogue: signs (int8 out)
//
// A CTA per SM walks its 128-vector tiles two at a time: stage 1 of both, stage 2 of both, stage 3 of both.  A stage of one tile
// needs nothing but the stage before of the same tile, so while one tile is in its epilogue the other is on the tensor
// core, whatever their stages, and the scratch between the stages is the two tiles' own (it stays in L2: as three launches
// over all vectors, stages 2 and 3 moved 866 MB through DRAM for 262144 vectors of head_dim 256, of which 540 MB were
// residual pieces written and read again, and each stage waited for its own bottleneck: nearest centroids in stage 1,
// memory in 2, the operand images in 3.  That call takes 399 -> 322 us where it runs on and on, under the power cap, and 290 in a
// short burst; 445 000 clocks, of which the tensor core's own are 228 000.  What bounds it then is the shared-memory data path: an
// MMA of N = 256 reads 12 KB in its 129 clocks and B arrives at 64 bytes a clock, which leaves the epilogues little).
//
// Warps: 0 the A side's TMA loads (128 rows x 64 columns, 128-byte swizzle) and the index bytes; 1 issues tcgen05.mma M=128 N=D
// K=16 into one accumulator per tile; four epilogue warpgroups; two expander warps.  Warp 0 also issues the
// bulk copies of B chunks (pre-swizzled image in global memory, L2-resident) through a ring of their own.  Every mbarrier wait is bounded; on expiry the CTA raises an abort flag, records a
// status word and leaves through the normal exit.

#include <cuda.h>
#include <cuda_fp16.h>

#include <atomic>
#include <cstdlib>

#include "tq_common.cuh"
#include "tq_internal.h"
#include "tq_pdl.cuh"

namespace tq {

namespace {

#include "tq_tc_ptx.cuh"

constexpr int kRowsT = 128;                    // vectors per tile (MMA M)
constexpr uint32_t kChunk = 128 * 128;         // 128 rows x 64 fp16 = 16 KB (an A chunk or a B chunk)
constexpr int kNB = 3;                         // B ring stages
constexpr int kNA = 3;                         // A ring slots
constexpr uint32_t kRawChunk = 128 * 64;       // index bytes of a k-chunk: 128 rows x 64
constexpr int kExpandThreads = 64;             // stage 2: two expander warps, thread = two rows

template <int D>
struct VCfg {
  static constexpr int KC = D / 64;            // k chunks
  static constexpr int NBLK = D / 128;         // blocks of 128 output columns
  // A: slots of one k-chunk (both pieces), released as soon as its MMAs are done, so
  // that the B ring can hold stages of ALL output columns: one MMA of N = D per k-step instead of one per block of
  // 128 columns, which reads the A operand once (M = 128 takes 65 clocks at N = 128 and 129 at N = 256)
  static constexpr uint32_t kBStage = NBLK * kChunk;                     // one k-chunk of B for all D output columns
  static constexpr uint32_t kOffA = 0;                                   // [slot][piece] chunks
  static constexpr uint32_t kOffB = kOffA + 2u * kNA * kChunk;           // ring
  static constexpr uint32_t kOffRaw = kOffB + kNB * kBStage;             // stage 2: index bytes of two k-chunks
  static constexpr uint32_t kOffTab = kOffRaw + 2u * kRawChunk;          // thresholds, centroid piece pairs, cell table, partial sums, norms
  static constexpr uint32_t kOffBar = kOffTab + 9216;
  // Epilogue: four warpgroups, one per 64 columns of a tile: all four on every tile at head_dim 256, two on each of the two
  // tiles in flight at head_dim 128.
  static constexpr int kWgs = D / 64;                                    // warpgroups of a tile
  static constexpr int kEpiThreads = 512;
  static constexpr int kExpandBegin = 64 + kEpiThreads;
  static constexpr int kThreads = kExpandBegin + kExpandThreads;
  static constexpr uint32_t kUsedBytes = kOffBar + 256;
  static constexpr uint32_t kSmemBytes = kUsedBytes + 1024;
  static constexpr uint32_t kImageBytes = 2u * KC * NBLK * kChunk;       // [piece][kc][nb] chunks of one operand
  static constexpr int kTmemCols = 2 * NBLK * 128;                       // two tiles in flight
};
static_assert(VCfg<256>::kSmemBytes <= 232448 && VCfg<128>::kSmemBytes <= 232448, "shared memory budget");

struct V2Args {
  CUtensorMap x_map;         // fp16 (D, n), box 64 x 128, 128-byte swizzle
  CUtensorMap idx_map;       // index bytes: rows of D bytes, 2 D bytes apart, at the head of the rows of p_hi
  CUtensorMap hi_map;        // the residual's pieces
  CUtensorMap lo_map;
  const uint8_t* images;     // three operand images [piece][kc][nb][128 rows x 128 bytes swizzled]
  const float* codebook;
  const uint16_t* x;         // the vectors (n, D) fp16
  uint16_t* p_hi;            // scratch rows (D): after stage 1 the first D bytes of a row are the vector's index bytes, after
                             // stage 2 (which reads a tile's bytes before it writes the tile's rows) the residual's pieces
  uint16_t* p_lo;
  float* vec_norms_out;      // optional, ||x||
  uint8_t* idx_u8_out;       // stage 1: optional, one index per byte (n, D)
  uint8_t* idx_packed_out;   // stage 1: optional, bit-packed rows (n, G), first index in the high bits
  uint8_t* sign_bits_out;    // stage 3: optional, one bit per sign (n, D / 8), coordinate j in bit 7 - j % 8, set for +1
  uint16_t* k_mse_out;       // stage 2: optional
  uint16_t* rnorm_out;       // stage 2, fp16 bits
  int8_t* signs_out;         // stage 3
  int32_t* status;
  int64_t n;
  int32_t tiles;
  int32_t bits;
};

__device__ int g_v2_status;    // 0 = ok; otherwise (code << 16) | block

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}

// Operand image of a D x D matrix B (rows = output columns n, columns = contraction index k):
// value hi + lo in fp16, [piece][kc][nb][row n % 128][64 columns], rows of 128 bytes, 16-byte
// chunk c at c ^ (row & 7).  B[n][k] = src[n * ld_n + k * ld_k].
// blockIdx.y = the operand: Pi (B[n][k] = Pi[n][k]), Pi^T (Pi[k][n]) and S (qjl_t[k][n]), one image after the other; three
// launches of a microsecond's work cost 9 us a call.
template <int D>
__global__ void k_v2_operand_image(const float* __restrict__ rotation, const float* __restrict__ qjl_t, int64_t M,
                                  uint8_t* __restrict__ images) {
  pdl_trigger();
  constexpr int KC = VCfg<D>::KC, NBLK = VCfg<D>::NBLK;
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= D * D) return;
  const float* src = blockIdx.y == 2 ? qjl_t : rotation;
  const int64_t ld_n = blockIdx.y == 0 ? D : 1, ld_k = blockIdx.y == 0 ? 1 : blockIdx.y == 1 ? D : M;
  uint8_t* image = images + (size_t)blockIdx.y * VCfg<D>::kImageBytes;
  const int n = e / D, k = e % D;
  // operand row (= accumulator column) n holds output column 16 t + 2 r + j of its 64, where n = 8 r + 2 t + j: the
  // epilogues' TMEM loads give thread t of a quad the accumulator columns 8 r + 2 t + {0, 1}, which are then 16 in a row
  const int col = (n & ~63) + 16 * ((n >> 1) & 3) + 2 * ((n >> 3) & 7) + (n & 1);
  const float v = __ldg(src + (int64_t)col * ld_n + (int64_t)k * ld_k);
  const __half hi = __float2half_rn(v);
  const __half lo = __float2half_rn(v - __half2float(hi));
  const int kc = k / 64, nb = n / 128, rr = n % 128, c = (k % 64) / 8, w = k % 8;
  const size_t off = ((size_t)kc * NBLK + nb) * (kChunk / 2) + (size_t)rr * 64 + (size_t)((c ^ (rr & 7)) * 8 + w);
  uint16_t* img = reinterpret_cast<uint16_t*>(image);
  img[off] = __half_as_ushort(hi);
  img[(size_t)KC * NBLK * (kChunk / 2) + off] = __half_as_ushort(lo);
}

// The 32 bytes of one vector's row that an epilogue step produces or reads.  A warp's access touches 32 rows, that is 32
// lines, whatever its width, and the load/store unit takes them one at a time: that was the whole cost of stages 1
// and 2 (eight 16-byte accesses per step are 33 000 of the 36 000 clocks that stage 2 took per tile), so a row's 32
// bytes go as one access (262144 vectors of head_dim 256: stages 183 + 264 + 87 us before, 154 + 195 + 81 us so).  `wide`
// is false where a caller's buffer starts on an odd multiple of 16 bytes.
__device__ __forceinline__ void store_row32(void* dst, const uint32_t (&v)[8], bool wide) {
  if (wide) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
                 "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
  } else {
    uint4* d = reinterpret_cast<uint4*>(dst);
    d[0] = make_uint4(v[0], v[1], v[2], v[3]);
    d[1] = make_uint4(v[4], v[5], v[6], v[7]);
  }
}
__device__ __forceinline__ void load_row32(const void* src, uint32_t (&v)[8], bool wide) {
  if (wide) {
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]),
                 "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "l"(src));
  } else {
    const uint4* s = reinterpret_cast<const uint4*>(src);
    const uint4 a = __ldg(s), b = __ldg(s + 1);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  }
}

// 16 rows x 64 accumulator columns of this warp's lanes: registers 4 r + {0, 1} are row lane / 4, columns 8 r + 2 (lane % 4) +
// {0, 1}, registers 4 r + {2, 3} the same of row lane / 4 + 8
__device__ __forceinline__ void tmem_ld_quads(uint32_t taddr, uint32_t (&r)[32]) {
  __syncwarp();
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x8.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                 "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]),
                 "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]),
                 "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
               :
               : "memory");
}

// Quantiser of a row's 16 accumulator columns: four index bytes a word.  The search shortcut of a codebook with at most 31
// thresholds (see tq_umma.cu: a candidate from a cubic, its threshold from a lane, one saturating compare), or any codebook.
struct V2Quantiser {
  float s, c1, c2, c3, thr_lane_h;      // shortcut; threshold[lane] * 2^40
  float t0, t1, t2;                     // the first three thresholds * 2^40
  float s_inv, h_inv;                   // per vector: s / (norm + 1e-8) and 2^40 / (norm + 1e-8)
};
// Row hh of the two whose 16 columns each a thread holds: a[4 j + 2 hh + {0, 1}] are columns 2 j, 2 j + 1.  COUNT: up to three thresholds
// (1- and 2-bit codes) are all compared, from registers; a shuffle per coordinate takes as much of the shared-memory data
// path as the tensor core's operands leave.
template <bool COUNT, bool LINEAR>
__device__ __forceinline__ void index_bytes_fast(const uint32_t (&a)[32], int hh, const V2Quantiser& q, uint32_t (&ib)[4]) {
  constexpr uint32_t kMagic = 0x4B000000u;     // bits of 2^23, which ride along with every index
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    uint32_t acc = 0u - (kMagic + (kMagic << 8) + (kMagic << 16) + (kMagic << 24));
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const float r = __uint_as_float(a[4 * (2 * w + (b >> 1)) + 2 * hh + (b & 1)]);
      float t, pf, u;
      if constexpr (COUNT) {
        float p1, p2;
        asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(pf) : "f"(r), "f"(q.h_inv), "f"(-q.t0));
        asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(p1) : "f"(r), "f"(q.h_inv), "f"(-q.t1));
        asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(p2) : "f"(r), "f"(q.h_inv), "f"(-q.t2));
        u = p1 + (p2 + 8388608.0f);
      } else {
        asm("fma.rn.sat.f32 %0, %1, %2, 0f3F000000;" : "=f"(t) : "f"(r), "f"(q.s_inv));
        if constexpr (LINEAR) u = fmaf(q.c1, t, 8388608.0f);
        else u = fmaf(fmaf(fmaf(q.c3, t, q.c2), t, q.c1), t, 8388608.0f);
        const float thr_h = __shfl_sync(0xffffffffu, q.thr_lane_h, __float_as_int(u));
        asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(pf) : "f"(r), "f"(q.h_inv), "f"(-thr_h));
      }
      acc = __float_as_uint(u + pf) * (1u << (8 * b)) + acc;
    }
    ib[w] = acc;
  }
}
// Out of line, its arguments by value: cold, and nothing of it weighs on the path that runs.
__device__ __noinline__ uint4 index_bytes_any(uint4 v0, uint4 v1, uint4 v2, uint4 v3, float inv, const float* codebook, const float* thr,
                                              const uint8_t* cells, int bits) {
  const int mode = (int)__ldg(codebook + 512);
  const float s = __ldg(codebook + 513), c1 = __ldg(codebook + 514), c2 = __ldg(codebook + 515), c3 = __ldg(codebook + 516);
  const uint32_t v[16] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w, v2.x, v2.y, v2.z, v2.w, v3.x, v3.y, v3.z, v3.w};
  uint32_t ib[4] = {0u, 0u, 0u, 0u};
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const float y = __uint_as_float(v[e]) * inv;
    int idx;
    if (mode != 0) {
      // candidate e0 with index in {e0, e0 + 1} (verified on the host for every y), then one exact compare
      float t;
      asm("fma.rn.sat.f32 %0, %1, %2, 0f3F000000;" : "=f"(t) : "f"(y), "f"(s));
      int e0;
      if (mode == 1) e0 = __float_as_int(fmaf(fmaf(fmaf(c3, t, c2), t, c1), t, 8388608.0f)) & 0xFF;
      else e0 = cells[__float_as_int(fmaf(t, 1024.0f, 8388608.0f)) & 0x7FF];
      idx = e0 + (y > thr[e0] ? 1 : 0);
    } else {
      int lo = 0, hi = (1 << bits) - 1;
      for (int step = 0; step < bits; ++step) {
        const int mid = (lo + hi) >> 1;
        if (y > thr[mid]) lo = mid + 1; else hi = mid;
      }
      idx = lo;
    }
    ib[e >> 2] |= (uint32_t)idx << (8 * (e & 3));
  }
  return make_uint4(ib[0], ib[1], ib[2], ib[3]);
}

// 16 index bytes as 16 / ipb bytes of a packed row
__device__ __forceinline__ void store_packed16(uint8_t* dst, const uint32_t (&ib)[4], int bits) {
  const int ipb = 8 / bits;
  if (ipb == 1) {
    *reinterpret_cast<uint4*>(dst) = make_uint4(ib[0], ib[1], ib[2], ib[3]);
  } else if (ipb == 2) {           // 3- and 4-bit codes: byte k = idx[2k] << bits | idx[2k+1]
    uint32_t o[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t a = ib[2 * h], b = ib[2 * h + 1];
      const uint32_t b0 = (((a >> 0) & 0xFFu) << bits) | ((a >> 8) & 0xFFu), b1 = (((a >> 16) & 0xFFu) << bits) | (a >> 24);
      const uint32_t b2 = (((b >> 0) & 0xFFu) << bits) | ((b >> 8) & 0xFFu), b3 = (((b >> 16) & 0xFFu) << bits) | (b >> 24);
      o[h] = b0 | (b1 << 8) | (b2 << 16) | (b3 << 24);
    }
    *reinterpret_cast<uint2*>(dst) = make_uint2(o[0], o[1]);
  } else if (ipb == 4) {           // 2-bit codes
    uint32_t o = 0u;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t a = ib[k];
      o |= ((((a >> 0) & 3u) << 6) | (((a >> 8) & 3u) << 4) | (((a >> 16) & 3u) << 2) | ((a >> 24) & 3u)) << (8 * k);
    }
    *reinterpret_cast<uint32_t*>(dst) = o;
  } else {                          // 1-bit codes
    uint32_t o = 0u;
#pragma unroll
    for (int e = 0; e < 16; ++e) o |= ((ib[e >> 2] >> (8 * (e & 3))) & 1u) << (8 * (e >> 3) + 7 - (e & 7));
    *reinterpret_cast<uint16_t*>(dst) = (uint16_t)o;
  }
}

// Stage 2's operand from index bytes.  Up to 2 bits the fp16 pieces of all centroids fit two registers each and a byte permute picks
// those of two coordinates at once, with 2 idx and 2 idx + 1 as its selectors; with 3 bits the low and the high bytes of a
// piece fit two registers each, and two permutes pair what they pick.  A look-up in shared memory per coordinate, two warps
// of them, took 2400 clocks per 64 coordinates of a tile where the MMAs take 1550.
//   pool, up to 2 bits: {hi01, hi23, lo01, lo23};  3 bits: low bytes of hi (2), high bytes of hi (2), the same of lo
__device__ __forceinline__ void piece_pool(const uint32_t* lut, int bits, uint32_t (&pool)[8]) {
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    if (bits <= 2) {
      pool[j] = __byte_perm(lut[2 * j], lut[2 * j + 1], 0x5410);
      pool[2 + j] = __byte_perm(lut[2 * j], lut[2 * j + 1], 0x7632);
    } else {
#pragma unroll
      for (int byte = 0; byte < 4; ++byte) {
        uint32_t w = 0u;
#pragma unroll
        for (int k = 0; k < 4; ++k) w |= ((lut[4 * j + k] >> (8 * byte)) & 0xFFu) << (8 * k);
        pool[2 * byte + j] = w;
      }
    }
  }
}
// 4 index bytes -> operand words of the high and of the low pieces
template <int BITS>
__device__ __forceinline__ void pieces_of_four(uint32_t w, const uint32_t (&pool)[8], uint32_t lut, uint32_t* hi, uint32_t* lo) {
  if constexpr (BITS == 2) {
    const uint32_t sel = w * 0x22u + 0x10101010u;
    hi[0] = __byte_perm(pool[0], pool[1], sel & 0xFFFFu);
    lo[0] = __byte_perm(pool[2], pool[3], sel & 0xFFFFu);
    hi[1] = __byte_perm(pool[0], pool[1], sel >> 16);
    lo[1] = __byte_perm(pool[2], pool[3], sel >> 16);
  } else if constexpr (BITS == 3) {
    uint32_t sel = (w | (w >> 4)) & 0x00FF00FFu;
    sel = (sel | (sel >> 8)) & 0x7777u;
    const uint32_t h0 = __byte_perm(pool[0], pool[1], sel), h1 = __byte_perm(pool[2], pool[3], sel);
    const uint32_t l0 = __byte_perm(pool[4], pool[5], sel), l1 = __byte_perm(pool[6], pool[7], sel);
    hi[0] = __byte_perm(h0, h1, 0x5140); hi[1] = __byte_perm(h0, h1, 0x7362);
    lo[0] = __byte_perm(l0, l1, 0x5140); lo[1] = __byte_perm(l0, l1, 0x7362);
  } else {
    uint32_t e[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t off = u == 0 ? ((w << 2) & 0x3FCu) : ((w >> (8 * u - 2)) & 0x3FCu);
      asm volatile("ld.shared.b32 %0, [%1];" : "=r"(e[u]) : "r"(lut + off));
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      hi[j] = __byte_perm(e[2 * j], e[2 * j + 1], 0x5410);
      lo[j] = __byte_perm(e[2 * j], e[2 * j + 1], 0x7632);
    }
  }
}
template <int BITS>
__device__ __forceinline__ void expand_chunk(uint32_t raw, uint32_t dst0, int et, const uint32_t (&pool)[8], uint32_t lut) {
#pragma unroll 1
  for (int row = et; row < kRowsT; row += kExpandThreads) {
    const uint32_t r1 = (uint32_t)(row >> 1) & 1u, r2 = (uint32_t)(row >> 2) & 1u;
    const uint32_t g = ((r2 ^ r1) << 1) | r2;
    const uint32_t src = raw + (uint32_t)row * 64u, dst = dst0 + (uint32_t)row * 128u;
    uint4 x[4];
#pragma unroll
    for (uint32_t c = 0; c < 4; ++c) x[c] = ld_shared_v4(src + (c ^ g) * 16u);
#pragma unroll
    for (uint32_t c = 0; c < 4; ++c) {
      const uint32_t xw[4] = {x[c].x, x[c].y, x[c].z, x[c].w};
#pragma unroll
      for (uint32_t h = 0; h < 2; ++h) {                  // 8 coordinates: one 16-byte operand chunk per piece
        uint32_t hi[4], lo[4];
        pieces_of_four<BITS>(xw[2 * h], pool, lut, hi, lo);
        pieces_of_four<BITS>(xw[2 * h + 1], pool, lut, hi + 2, lo + 2);
        const uint32_t at = dst + (((2u * (c ^ g) + h) ^ (uint32_t)(row & 7)) << 4);
        st_shared_v4(at, hi[0], hi[1], hi[2], hi[3]);
        st_shared_v4(at + kChunk, lo[0], lo[1], lo[2], lo[3]);
      }
    }
  }
}

// two fused multiply-adds in one instruction (sm_100): the same IEEE results per half as fmaf
__device__ __forceinline__ unsigned long long square2(uint32_t lo, uint32_t hi, unsigned long long sum) {
  unsigned long long v, d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(lo), "r"(hi));
  asm("fma.rn.f32x2 %0, %1, %1, %2;" : "=l"(d) : "l"(v), "l"(sum));
  return d;
}

// The CTA's walk: item (stage, tile), the tiles in pairs, a pair's stages one after the other, tile slot 0 before slot 1.  Every
// role goes through the same items.
struct Walk {
  int n_local, i0 = 0, stage = 1, slot = 0;
  __device__ __forceinline__ explicit Walk(int n) : n_local(n) {}
  __device__ __forceinline__ bool done() const { return i0 >= n_local; }
  __device__ __forceinline__ int tile() const { return i0 + slot; }
  __device__ __forceinline__ int use() const { return (i0 >> 1) * 3 + stage - 1; }     // the slot's items before this one
  __device__ __forceinline__ void next() {
    if (slot == 0 && i0 + 1 < n_local) { slot = 1; return; }
    slot = 0;
    if (++stage > 3) { stage = 1; i0 += 2; }
  }
};
template <typename F>
__device__ __forceinline__ bool walk_items(int n_local, F&& f) {      // f(tile, slot, stage, use) returns false to leave
#pragma unroll 1
  for (Walk w(n_local); !w.done(); w.next())
    if (!f(w.tile(), w.slot, w.stage, w.use())) return false;
  return true;
}

// STAGE: the last stage that the launch runs; only the whole walk is launched.
template <int D, int STAGE = 3>
__global__ void __launch_bounds__(VCfg<D>::kThreads, 1) k_umma_v2_stage(const __grid_constant__ V2Args p) {
  // The wait comes before the TMEM allocation: a dependent that held TMEM while its predecessor still had to allocate some
  // on the same SM would wait for good.  For the same reason the last kernel of the call does not let a dependent start: what
  // follows it is not this library's, and may allocate TMEM before it waits.
  if constexpr (STAGE != 3) pdl_trigger();
  pdl_wait();
  using C = VCfg<D>;
  constexpr int KC = C::KC, NBLK = C::NBLK;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gbase = smem_raw + (base - smem_u32(smem_raw));
  {
    uint32_t dyn_bytes;
    asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn_bytes));
    if (base - smem_u32(smem_raw) + C::kUsedBytes > dyn_bytes) {     // the layout does not fit: report, do nothing
      if (threadIdx.x == 0 && p.status != nullptr) atomicCAS(p.status, 0, (9 << 16) | (int)blockIdx.x);
      return;
    }
  }
  const uint32_t a_smem = base + C::kOffA;      // slot s: its high (or only) piece, then its low piece
  const uint32_t b_smem = base + C::kOffB;
  const uint32_t raw_smem = base + C::kOffRaw;
  float* thr_s = reinterpret_cast<float*>(gbase + C::kOffTab);
  uint32_t* lut_s = reinterpret_cast<uint32_t*>(gbase + C::kOffTab + 1024);
  uint8_t* cells_s = gbase + C::kOffTab + 2048;                        // 1028 bytes
  float* part_s = reinterpret_cast<float*>(gbase + C::kOffTab + 4096); // [slot 2][warpgroup 4][row 128] partial sums of the norms
  float* norm_s = reinterpret_cast<float*>(gbase + C::kOffTab + 8192); // [slot 2][row 128] vector norms, stage 1 -> 2
  const uint32_t bar_afull = base + C::kOffBar;             // [kNA] TMA or expanders -> MMA (all pieces of a k-chunk)
  const uint32_t bar_aempty = bar_afull + 8 * kNA;          // [kNA] MMA commit -> producer, expanders
  const uint32_t bar_bfull = bar_aempty + 8 * kNA;          // [kNB] bulk copy -> MMA
  const uint32_t bar_bempty = bar_bfull + 8 * kNB;          // [kNB] MMA commit -> B producer
  const uint32_t bar_tfull = bar_bempty + 8 * kNB;          // [2] MMA commit -> epilogue
  const uint32_t bar_tempty = bar_tfull + 16;               // [2] epilogue (a warp each) -> MMA
  const uint32_t bar_ready = bar_tempty + 16;               // [2] epilogue (a warp each): the scratch of the next stage is written
  const uint32_t bar_rfull = bar_ready + 16;                // [2] stage 2: TMA -> expanders (index bytes)
  const uint32_t bar_rempty = bar_rfull + 16;               // [2] stage 2: expanders -> producer
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gbase + C::kOffBar + 216);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gbase + C::kOffBar + 224);
  static_assert(16 * (kNA + kNB) + 80 <= 216, "barriers");

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int total = p.tiles;
  const int t0 = (int)((int64_t)total * blockIdx.x / gridDim.x);
  const int t1 = (int)((int64_t)total * (blockIdx.x + 1) / gridDim.x);
  const int n_local = t1 - t0;
  auto failed = [&](int code) {
    *abort_flag = 1;
    if (p.status != nullptr) atomicCAS(p.status, 0, (code << 16) | (int)blockIdx.x);
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < kNA; ++i) { mbar_init(bar_afull + 8 * i, 1); mbar_init(bar_aempty + 8 * i, 1); }
    for (int i = 0; i < kNB; ++i) { mbar_init(bar_bfull + 8 * i, 1); mbar_init(bar_bempty + 8 * i, 1); }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar_tfull + 8 * i, 1);
      mbar_init(bar_tempty + 8 * i, 4 * C::kWgs);
      mbar_init(bar_ready + 8 * i, 4 * C::kWgs);
      mbar_init(bar_rfull + 8 * i, 1);
      mbar_init(bar_rempty + 8 * i, 1);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x >= 64 && threadIdx.x < 64 + 256) {
    const int e = threadIdx.x - 64;
    thr_s[e] = __ldg(p.codebook + kThresholdOff + e);
    const float c = __ldg(p.codebook + kCentroidOff + e);
    const __half h = __float2half_rn(c);
    const __half l = __float2half_rn(c - __half2float(h));
    lut_s[e] = (uint32_t)__half_as_ushort(h) | ((uint32_t)__half_as_ushort(l) << 16);
    for (int w = e; w < 257; w += 256) reinterpret_cast<uint32_t*>(cells_s)[w] = __float_as_uint(__ldg(p.codebook + 528 + w));
  }
  if (warp == 1) tmem_alloc(smem_u32((const void*)tmem_slot), C::kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------ producer.  The A side and B have a position each and
    // whichever has room goes on: B's chunks of a stage are there when its A is, which may have to wait for an epilogue.
    if (lane == 0) {
      int ac = 0, kc = 0;                                   // A: running chunk counter (slot ac % kNA, use ac / kNA), chunk of the item
      int rc = 0;                                           // running count of index chunks
      int loads = 0;                                        // bit s: the last use of A slot s was a load of ours
      int bc = 0, kp = 0;                                   // B: running chunk counter, chunk and piece of the item
      bool ready = false;                                   // what the stage before wrote is there
      Walk wa(n_local), wb(n_local);
      long long start = 0;
      bool ok = true;
      for (uint32_t idle = 0; !wa.done() || !wb.done();) {
        bool moved = false;
        if (!wb.done() && mbar_try_wait(bar_bempty + 8 * (bc % kNB), (uint32_t)(((bc / kNB) & 1) ^ 1))) {
          const int s = bc % kNB;
          mbar_arrive_expect_tx(bar_bfull + 8 * s, C::kBStage);
          bulk_load(b_smem + s * C::kBStage, p.images + (size_t)(wb.stage - 1) * C::kImageBytes + (size_t)((kp & 1) * KC + (kp >> 1)) * C::kBStage,
                    C::kBStage, bar_bfull + 8 * s);
          ++bc;
          if (++kp == 2 * KC) { kp = 0; wb.next(); }
          moved = true;
        }
        if (!wa.done()) {
          if (!ready) {
            ready = wa.stage == 1 || mbar_try_wait(bar_ready + 8 * wa.slot, (uint32_t)(wa.stage & 1));
          }
          const bool raw = wa.stage == 2;                   // the operand itself is written by the expanders
          if (ready && (raw ? mbar_try_wait(bar_rempty + 8 * (rc & 1), (uint32_t)(((rc >> 1) & 1) ^ 1))
                            : mbar_try_wait(bar_aempty + 8 * (ac % kNA), (uint32_t)(((ac / kNA) & 1) ^ 1)))) {
            // the scratch rows are those of the CTA's first two tiles
            const int row0 = wa.stage == 1 ? (t0 + wa.tile()) * kRowsT : (t0 + wa.slot) * kRowsT;
            const int as = ac % kNA;
            if (raw) {
              mbar_arrive_expect_tx(bar_rfull + 8 * (rc & 1), kRawChunk);
              tma_load_2d(raw_smem + (rc & 1) * kRawChunk, &p.idx_map, kc * 64, row0, bar_rfull + 8 * (rc & 1));
              ++rc;
              loads &= ~(1 << as);
            } else {
              const uint32_t dst = a_smem + 2u * as * kChunk;
              mbar_arrive_expect_tx(bar_afull + 8 * as, wa.stage == 1 ? kChunk : 2 * kChunk);
              tma_load_2d(dst, wa.stage == 1 ? &p.x_map : &p.hi_map, kc * 64, row0, bar_afull + 8 * as);
              if (wa.stage == 3) tma_load_2d(dst + kChunk, &p.lo_map, kc * 64, row0, bar_afull + 8 * as);
              loads |= 1 << as;
            }
            ++ac;
            if (++kc == KC) { kc = 0; ready = false; wa.next(); }
            moved = true;
          }
        }
        if (moved) { idle = 0; start = 0; continue; }
        if ((++idle & 255u) == 0u) {                        // bounded, as mbar_wait
          const long long now = clock64();
          if (start == 0) start = now;
          if (*abort_flag || now - start > kWaitLimitCycles) { ok = false; break; }
        }
      }
      if (!ok) failed(1);
      // none of this CTA's own copies may still be in flight when it exits
      for (int k = 0; k < kNA && k < ac; ++k) {
        const int j = ac - 1 - k;
        if (loads & (1 << (j % kNA))) mbar_wait(bar_afull + 8 * (j % kNA), (uint32_t)((j / kNA) & 1), abort_flag);
      }
      for (int k = 0; k < 2 && k < rc; ++k) {
        const int j = rc - 1 - k;
        mbar_wait(bar_rfull + 8 * (j & 1), (uint32_t)((j >> 1) & 1), abort_flag);
      }
      for (int k = 0; k < kNB && k < bc; ++k) {
        const int j = bc - 1 - k;
        mbar_wait(bar_bfull + 8 * (j % kNB), (uint32_t)((j / kNB) & 1), abort_flag);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (converged warp, one elected lane issues)
    int ac = 0, bc = 0;
    // M = 128, N = D (all output columns in one instruction: rows 128.. of the B stage are the second block), fp16
    const uint32_t idesc = idesc_f16(false, (uint32_t)D);
    const bool ok = walk_items(n_local, [&](int i, int slot, int stage, int use) {
      bool go = mbar_wait(bar_tempty + 8 * slot, (uint32_t)((use & 1) ^ 1), abort_flag);
      if (!__all_sync(0xffffffffu, go)) return false;
      const uint32_t d_tmem = tmem_base + (uint32_t)(slot * NBLK * 128);
#pragma unroll 1
      for (int kc = 0; kc < KC; ++kc, ++ac) {
        const int as = ac % kNA;
        go = mbar_wait(bar_afull + 8 * as, (uint32_t)((ac / kNA) & 1), abort_flag);
        if (!__all_sync(0xffffffffu, go)) return false;
        const uint64_t a_hi = smem_desc_sw128(a_smem + 2u * as * kChunk);
        const uint64_t a_lo = smem_desc_sw128(a_smem + 2u * as * kChunk + kChunk);
#pragma unroll 1
        for (int pb = 0; pb < 2; ++pb, ++bc) {
          const int s = bc % kNB;
          go = mbar_wait(bar_bfull + 8 * s, (uint32_t)((bc / kNB) & 1), abort_flag);
          if (!__all_sync(0xffffffffu, go)) return false;
          tc_fence_after();
          const uint64_t b_desc = smem_desc_sw128(b_smem + s * C::kBStage);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_f16(d_tmem, a_hi + (uint64_t)(k * 2), b_desc + (uint64_t)(k * 2), idesc, (kc | k | pb) != 0 ? 1u : 0u);
            if (pb == 0 && stage != 1) {
#pragma unroll
              for (int k = 0; k < 4; ++k) umma_f16(d_tmem, a_lo + (uint64_t)(k * 2), b_desc + (uint64_t)(k * 2), idesc, 1u);
            }
            umma_commit(bar_bempty + 8 * s);                // the ring stage is free once these MMAs are done
            if (pb == 1) {
              umma_commit(bar_aempty + 8 * as);             // last use of this k-chunk of A
              if (kc == KC - 1) umma_commit(bar_tfull + 8 * slot);
            }
          }
          __syncwarp();
        }
      }
      return true;
    });
    if (!ok && lane == 0) failed(2);
  } else if (threadIdx.x >= C::kExpandBegin) {
    // ------------------------------------------------------------ expanders (stage 2): index bytes of a k-chunk -> centroid
    // pieces hi and lo in operand layout, thread = two rows.  The thread walks its four 16-byte pieces in an order XOR-ed with
    // `g`, a linear map of the row's bits 1 and 2 for which the map and its sum with the identity are both one-to-one:
    // the eight rows of a quarter warp then read eight different bank groups of the raw chunk and write eight different
    // ones of the operand.
    const uint32_t lut = smem_u32(lut_s);
    const int et = threadIdx.x - C::kExpandBegin;
    uint32_t pool[8];
    piece_pool(lut_s, p.bits, pool);
    int ac = 0, rc = 0;
    const bool ok = walk_items(n_local, [&](int i, int slot, int stage, int use) {
      if (stage != 2) { ac += KC; return true; }
      for (int kc = 0; kc < KC; ++kc, ++ac, ++rc) {
        const int as = ac % kNA, rs = rc & 1;
        bool go = mbar_wait(bar_rfull + 8 * rs, (uint32_t)((rc >> 1) & 1), abort_flag) &&
                  mbar_wait(bar_aempty + 8 * as, (uint32_t)(((ac / kNA) & 1) ^ 1), abort_flag);
        go = bar_red_and(5, kExpandThreads, go);            // leave together: the two warps meet at a barrier below
        if (!go) return false;
        const uint32_t raw = raw_smem + rs * kRawChunk, dst = a_smem + 2u * as * kChunk;
        if (p.bits <= 2) expand_chunk<2>(raw, dst, et, pool, lut);
        else if (p.bits == 3) expand_chunk<3>(raw, dst, et, pool, lut);
        else expand_chunk<8>(raw, dst, et, pool, lut);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // operand writes -> visible to the tensor core
        asm volatile("bar.sync 6, %0;" ::"n"(kExpandThreads) : "memory");
        if (et == 0) {
          mbar_arrive(bar_afull + 8 * as);
          mbar_arrive(bar_rempty + 8 * rs);
        }
      }
      return true;
    });
    if (!ok && lane == 0) failed(4);
  } else {
    // ------------------------------------------------------------ epilogue: a warpgroup per 64 columns of a tile, thread = vector.
    // What bounds a tile is the chain of its stages (contraction, epilogue, the way through the scratch), so
    // as many warps as there are share one epilogue: with a warpgroup per 128 columns and two of the four for each tile,
    // stage 2's took 15 400 clocks of the 24 500 between its contraction's start and the next one's.
    constexpr int kWgs = C::kWgs;
    const int ew = warp - 2;
    const int wgi = ew >> 2;
    const int group = wgi / kWgs, part = wgi % kWgs;
    const int quarter = warp & 3;                 // TMEM lanes this warp may touch: 32*quarter ..
    const int rloc = quarter * 32 + lane;
    const int col0 = part * 64;
    V2Quantiser q;
    q.s = __ldg(p.codebook + 513);
    q.c1 = __ldg(p.codebook + 514);
    q.c2 = __ldg(p.codebook + 515);
    q.c3 = __ldg(p.codebook + 516);
    q.thr_lane_h = thr_s[lane] * 1099511627776.0f;
    q.t0 = thr_s[0] * 1099511627776.0f;
    q.t1 = thr_s[1] * 1099511627776.0f;
    q.t2 = thr_s[2] * 1099511627776.0f;
    const bool fast = (int)__ldg(p.codebook + 512) == 1 && p.bits <= 5;             // up to 31 thresholds: one per lane
    const bool linear = __ldg(p.codebook + 518) == 1.0f;
    const bool x_wide = ((uintptr_t)p.x & 31u) == 0, k_wide = ((uintptr_t)p.k_mse_out & 31u) == 0;
    const bool ok = walk_items(n_local, [&](int i, int slot, int stage, int use) {
      if (kWgs == 2 && slot != group) return true;
      const uint32_t tacc = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(slot * NBLK * 128 + col0);
      const int64_t row = (int64_t)(t0 + i) * kRowsT + rloc;
      const int64_t srow = (int64_t)(t0 + slot) * kRowsT + rloc;      // its row of the scratch
      const bool valid = row < p.n;
      // stage 2: a quad of lanes holds 64 columns of a row, 16 each, so that its accesses to x, k_mse and the pieces are whole
      // 128-byte lines (see below).  The first coordinates are in flight while the tile's contraction runs.
      const int quad = lane & 3, r8 = lane >> 2;
      const int64_t qrow = (int64_t)(t0 + i) * kRowsT + quarter * 32 + r8;        // rows qrow + {0, 8, 16, 24}
      uint32_t xn[2][8];
      auto x_load = [&](int step) {                 // step = (16 rows rg, 8 rows hh)
        const int64_t r = qrow + 8 * step;
        load_row32(p.x + (r < p.n ? r : 0) * D + col0 + 16 * quad, xn[step & 1], x_wide);
      };
      if (stage == 2) { x_load(0); x_load(1); }
      // The exit decision is made uniform before anything collective, over all the warps that meet at named barriers below, so
      // that nobody waits at a barrier for a warp that left (the TMEM loads are collective over a warp).
      const bool go = bar_red_and(3 + group, 128 * kWgs, mbar_wait(bar_tfull + 8 * slot, (uint32_t)(use & 1), abort_flag));
      if (!go) return false;
      tc_fence_after();
      float* parts = part_s + slot * 4 * 128;
      if (stage == 1) {
#pragma unroll 1
        for (int rg = 0; rg < 2; ++rg) {
          uint32_t a[32];
          tmem_ld_quads(tacc + ((uint32_t)(rg * 16) << 16), a);
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            unsigned long long ssq2 = 0ull, ssq3 = 0ull;
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
              ssq2 = square2(a[4 * j + 2 * hh], a[4 * j + 2 * hh + 1], ssq2);
              ssq3 = square2(a[4 * j + 4 + 2 * hh], a[4 * j + 4 + 2 * hh + 1], ssq3);
            }
            float sq = (__uint_as_float((uint32_t)ssq2) + __uint_as_float((uint32_t)(ssq2 >> 32))) +
                       (__uint_as_float((uint32_t)ssq3) + __uint_as_float((uint32_t)(ssq3 >> 32)));
            sq += __shfl_xor_sync(0xffffffffu, sq, 1);          // the quad's four parts of the row
            sq += __shfl_xor_sync(0xffffffffu, sq, 2);
            if (quad == 0) parts[part * 128 + quarter * 32 + r8 + 16 * rg + 8 * hh] = sq;
          }
        }
        asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(128 * kWgs) : "memory");
        float ssq = 0.f;                           // lane = row
#pragma unroll
        for (int w = 0; w < kWgs; ++w) ssq += parts[w * 128 + rloc];
        const float norm = __fsqrt_rn(ssq);
        const float inv = __fdiv_rn(1.0f, norm + 1e-8f);
        if (part == 0) {
          norm_s[slot * 128 + rloc] = norm;
          if (valid && p.vec_norms_out != nullptr) p.vec_norms_out[row] = norm;
        }
#pragma unroll 1
        for (int rg = 0; rg < 2; ++rg) {
          uint32_t a[32];
          tmem_ld_quads(tacc + ((uint32_t)(rg * 16) << 16), a);
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            const int step = 2 * rg + hh;
            const int64_t r = qrow + 8 * step;
            const float inv_r = __shfl_sync(0xffffffffu, inv, r8 + 8 * step);
            q.s_inv = q.s * inv_r;
            q.h_inv = 1099511627776.0f * inv_r;    // 2^40: exact scaling
            uint32_t ib[4];
            if (fast && p.bits <= 2) index_bytes_fast<true, false>(a, hh, q, ib);
            else if (fast && linear) index_bytes_fast<false, true>(a, hh, q, ib);
            else if (fast) index_bytes_fast<false, false>(a, hh, q, ib);
            else {
              auto four = [&](int j) { return make_uint4(a[4 * j + 2 * hh], a[4 * j + 2 * hh + 1], a[4 * j + 4 + 2 * hh], a[4 * j + 5 + 2 * hh]); };
              const uint4 o = index_bytes_any(four(0), four(2), four(4), four(6), inv_r, p.codebook, thr_s, cells_s, p.bits);
              ib[0] = o.x; ib[1] = o.y; ib[2] = o.z; ib[3] = o.w;
            }
            if (r < p.n) {
              const int col = col0 + 16 * quad;
              const uint4 bytes = make_uint4(ib[0], ib[1], ib[2], ib[3]);
              *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(p.p_hi + (srow - lane + r8 + 8 * step) * D) + col) = bytes;
              if (p.idx_u8_out != nullptr) *reinterpret_cast<uint4*>(p.idx_u8_out + r * D + col) = bytes;
              if (p.idx_packed_out != nullptr)
                store_packed16(p.idx_packed_out + r * (int64_t)(D / (8 / p.bits)) + col / (8 / p.bits), ib, p.bits);
            }
          }
        }
      } else if (stage == 2) {
        // Rows x 32 bytes per access cost the load/store unit a slot per row (see store_row32), and the operand traffic of the
        // MMAs and the expanders runs through the same data path: thread = row took 199 us here for 262144 vectors of head_dim
        // 256 in a launch of its own, of which 16 400 of 26 600 clocks per tile were such slots.  tcgen05.ld.16x256b spreads a
        // row over a quad of lanes instead: thread (r8, quad) gets rows r8 and r8 + 8 of 16, 16 columns each, and a warp's
        // access is 8 lines: 133 us.
        float nv4[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) nv4[u] = norm_s[slot * 128 + quarter * 32 + r8 + 8 * u];
#pragma unroll
        for (int rg = 0; rg < 2; ++rg) {            // 16 rows
          uint32_t a[32];
          tmem_ld_quads(tacc + ((uint32_t)(rg * 16) << 16), a);
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {          // row r8 or r8 + 8 of them
            const int step = 2 * rg + hh;
            const int64_t r = qrow + 8 * step;
            const int64_t col = col0 + 16 * quad;
            const int64_t sat = (srow - lane + r8 + 8 * step) * D + col;        // the scratch row of r
            uint32_t xw[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) xw[j] = xn[hh][j];
            if (step + 2 < 4) x_load(step + 2);
            float sq = 0.f;
            if (r < p.n) {
              const float nv = nv4[step];
              uint32_t kq[8], rh[8], rl[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const float k0 = __uint_as_float(a[4 * j + 2 * hh]) * nv, k1 = __uint_as_float(a[4 * j + 2 * hh + 1]) * nv;
                const __half2 xh = *reinterpret_cast<const __half2*>(&xw[j]);
                const float r0 = __low2float(xh) - k0, r1 = __high2float(xh) - k1;
                sq = fmaf(r0, r0, sq);
                sq = fmaf(r1, r1, sq);
                const __half2 kh = __floats2half2_rn(k0, k1);
                kq[j] = *reinterpret_cast<const uint32_t*>(&kh);
                const __half2 h2 = __floats2half2_rn(r0, r1);
                rh[j] = *reinterpret_cast<const uint32_t*>(&h2);
                const __half2 l2 = __floats2half2_rn(r0 - __low2float(h2), r1 - __high2float(h2));
                rl[j] = *reinterpret_cast<const uint32_t*>(&l2);
              }
              store_row32(p.p_hi + sat, rh, true);
              store_row32(p.p_lo + sat, rl, true);
              if (p.k_mse_out != nullptr) store_row32(p.k_mse_out + r * D + col, kq, k_wide);
            }
            sq += __shfl_xor_sync(0xffffffffu, sq, 1);          // the quad's four parts of the row
            sq += __shfl_xor_sync(0xffffffffu, sq, 2);
            if (quad == 0) parts[part * 128 + quarter * 32 + r8 + 8 * step] = sq;
          }
        }
        asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(128 * kWgs) : "memory");
        if (part == 0 && valid) {
          float ssq = 0.f;
#pragma unroll
          for (int w = 0; w < kWgs; ++w) ssq += parts[w * 128 + rloc];
          p.rnorm_out[row] = __half_as_ushort(__float2half_rn(__fsqrt_rn(ssq)));
        }
        // the parts are written again after the barrier that opens the tile's next stage
      } else {
#pragma unroll 1
        for (int rg = 0; rg < 2; ++rg) {
          uint32_t a[32];
          tmem_ld_quads(tacc + ((uint32_t)(rg * 16) << 16), a);
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            const int64_t r = qrow + 16 * rg + 8 * hh;
            const int col = col0 + 16 * quad;
            if (r < p.n && p.signs_out != nullptr) {
              uint32_t sw[4];
#pragma unroll
              for (int w = 0; w < 4; ++w) {
                uint32_t x = 0u;
#pragma unroll
                for (int b = 0; b < 4; ++b)
                  x |= (__uint_as_float(a[4 * (2 * w + (b >> 1)) + 2 * hh + (b & 1)]) >= 0.f ? 0x01u : 0xFFu) << (8 * b);
                sw[w] = x;
              }
              *reinterpret_cast<uint4*>(p.signs_out + r * D + col) = make_uint4(sw[0], sw[1], sw[2], sw[3]);
            }
            if (r < p.n && p.sign_bits_out != nullptr) {
              uint32_t o = 0u;
#pragma unroll
              for (int e = 0; e < 16; ++e)
                o |= (__uint_as_float(a[4 * (e >> 1) + 2 * hh + (e & 1)]) >= 0.f ? 1u : 0u) << (8 * (e >> 3) + 7 - (e & 7));
              *reinterpret_cast<uint16_t*>(p.sign_bits_out + r * (D / 8) + col / 8) = (uint16_t)o;
            }
          }
        }
      }
      tc_fence_before();
      if (stage < 3) asm volatile("fence.proxy.async.global;" ::: "memory");   // the scratch is read by the copy engine
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(bar_tempty + 8 * slot);
        if (stage < 3) mbar_arrive(bar_ready + 8 * slot);
      }
      return true;
    });
    if (!ok && lane == 0) failed(3);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
}

int encode_rows(TensorMapEncodeFn enc, CUtensorMap* map, const void* ptr, int64_t n, int D) {
  cuuint64_t dims[2] = {(cuuint64_t)D, (cuuint64_t)n};
  cuuint64_t strides[1] = {(cuuint64_t)D * 2};
  cuuint32_t box[2] = {64, (cuuint32_t)kRowsT};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { note_cuda_error(100000 + (int)r); return TQ_ELAUNCH; }
  return TQ_OK;
}

// index bytes: n rows of D bytes, 2 D bytes apart
int encode_index_rows(TensorMapEncodeFn enc, CUtensorMap* map, const void* ptr, int64_t n, int D) {
  cuuint64_t dims[2] = {(cuuint64_t)D, (cuuint64_t)n};
  cuuint64_t strides[1] = {(cuuint64_t)D * 2};
  cuuint32_t box[2] = {64, (cuuint32_t)kRowsT};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { note_cuda_error(100000 + (int)r); return TQ_ELAUNCH; }
  return TQ_OK;
}

template <int D>
int run(const TqQjlCompressJob& job, cudaStream_t st) {
  TensorMapEncodeFn enc = tensor_map_encoder();
  if (enc == nullptr) return TQ_ELAUNCH;
  const int64_t n = job.B * job.H * job.S;
  const int64_t tiles = (n + kRowsT - 1) / kRowsT;
  if (tiles >= ((int64_t)1 << 30)) return TQ_ETOOBIG;
  // workspace: three operand images, then the two piece arrays
  uint8_t* ws = reinterpret_cast<uint8_t*>(((uintptr_t)job.workspace + 1023u) & ~(uintptr_t)1023u);
  const size_t img = VCfg<D>::kImageBytes;
  const size_t piece = ((size_t)n * D * 2 + 1023) / 1024 * 1024;
  V2Args p;
  p.images = ws;
  p.p_hi = reinterpret_cast<uint16_t*>(ws + 3 * img);
  p.p_lo = reinterpret_cast<uint16_t*>(ws + 3 * img + piece);
  void* status_ptr = nullptr;
  cudaGetSymbolAddress(&status_ptr, g_v2_status);
  p.status = reinterpret_cast<int32_t*>(status_ptr);
  p.codebook = job.codebook;
  p.x = reinterpret_cast<const uint16_t*>(job.x);
  p.vec_norms_out = job.vec_norms_out;
  p.idx_u8_out = job.idx_mode == TQ_IDX_PACKED ? nullptr : reinterpret_cast<uint8_t*>(job.idx_out);
  p.idx_packed_out = job.idx_mode == TQ_IDX_PACKED ? reinterpret_cast<uint8_t*>(job.idx_out) : nullptr;
  p.k_mse_out = job.k_mse_out;
  p.rnorm_out = reinterpret_cast<uint16_t*>(job.rnorm_out);
  p.signs_out = job.signs_dtype == 2 ? nullptr : reinterpret_cast<int8_t*>(job.signs_out);
  p.sign_bits_out = job.signs_dtype == 2 ? reinterpret_cast<uint8_t*>(job.signs_out) : nullptr;
  p.n = n;
  p.tiles = (int32_t)tiles;
  p.bits = job.bits;
  int rc;
  if ((rc = encode_rows(enc, &p.x_map, job.x, n, D)) != TQ_OK) return rc;
  if ((rc = encode_index_rows(enc, &p.idx_map, p.p_hi, n, D)) != TQ_OK) return rc;
  if ((rc = encode_rows(enc, &p.hi_map, p.p_hi, n, D)) != TQ_OK) return rc;
  if ((rc = encode_rows(enc, &p.lo_map, p.p_lo, n, D)) != TQ_OK) return rc;
  const cudaError_t e = cudaFuncSetAttribute(k_umma_v2_stage<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)VCfg<D>::kSmemBytes);
  if (e != cudaSuccess) return refused(e);        // before the first launch, which lets a dependent start
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int grid = (int)(tiles < sms ? tiles : sms);
  k_v2_operand_image<D><<<dim3((D * D + 255) / 256, 3), 256, 0, st>>>(job.rotation, job.qjl_t, job.M, ws);
  if ((rc = check_launch()) != TQ_OK) return rc;
  launch_after(k_umma_v2_stage<D>, dim3(grid), dim3(VCfg<D>::kThreads), VCfg<D>::kSmemBytes, st, p);
  return check_launch();
}

}  // namespace

size_t umma_v2_compress_workspace(int64_t n, int D) {
  if (D != 128 && D != 256) return 0;
  const size_t img = D == 256 ? VCfg<256>::kImageBytes : VCfg<128>::kImageBytes;
  const size_t piece = ((size_t)n * D * 2 + 1023) / 1024 * 1024;
  return 1024 + 3 * img + 2 * piece + (size_t)n * sizeof(float) + 1024;
}

bool umma_v2_compress_eligible(const TqQjlCompressJob& job) {
  if (force_simt()) return false;
  if (job.D != 128 && job.D != 256) return false;
  if (job.x_dtype != TQ_F16 || job.normalize != 1 || (job.signs_dtype != 0 && job.signs_dtype != 2) || job.rnorm_dtype != TQ_F16)
    return false;
  if (job.M != job.D || (job.idx_out != nullptr && job.idx_mode != TQ_IDX_U8 && job.idx_mode != TQ_IDX_PACKED)) return false;
  if (job.bits < 1 || job.bits > 8) return false;
  const int64_t n = job.B * job.H * job.S;
  if (n <= 0) return false;
  // rows must be contiguous: (B, H, S, D) without gaps
  if (job.S > 1 && job.stride_s != job.D) return false;
  if (job.H > 1 && job.stride_h != job.S * job.D) return false;
  if (job.B > 1 && job.stride_b != job.H * job.S * job.D) return false;
  if (((uintptr_t)job.x & 15u) || ((uintptr_t)job.k_mse_out & 15u) || ((uintptr_t)job.signs_out & 15u) ||
      ((uintptr_t)job.idx_out & 15u))
    return false;
  if (job.workspace == nullptr || job.workspace_bytes < umma_v2_compress_workspace(n, job.D)) return false;
  return true;
}

int umma_v2_compress(const TqQjlCompressJob& job, cudaStream_t st) {
  return job.D == 256 ? run<256>(job, st) : run<128>(job, st);
}

int umma_v2_device_status() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_v2_status, sizeof(int)) != cudaSuccess) return -1;
  return v;
}

}  // namespace tq
