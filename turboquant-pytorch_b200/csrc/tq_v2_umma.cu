// Tensor-core (tcgen05 / TMEM / TMA) path for the MSE + QJL compress stage (K4), fp16 vectors,
// head_dim 128 or 256.  The reference's three chained D x D contractions
// (turboquant/compressors.py:83-120) run as three launches of one contraction kernel with a
// different epilogue each; operands that are fp32 in the reference are carried as fp16 pieces
// hi + lo (lo reaches into fp16 subnormals), so products match an fp32 matmul to ~2^-21:
//
//   stage 1  y = x Pi^T            A = x (exact fp16), B = Pi hi/lo.  Epilogue: ||y|| = ||x||, scale,
//                                  nearest centroid by exact thresholds, one index byte per coordinate -> scratch
//   stage 2  k = (c Pi) ||x||      A = centroid pieces, which expander warps write into the operand ring from the
//                                  index bytes, B = Pi^T hi/lo (hi.hi + lo.hi + hi.lo).  Epilogue:
//                                  k_mse (fp16 out), residual r = x - k, ||r|| (out), residual pieces -> scratch
//   stage 3  p = r S^T             A = residual pieces, B = S hi/lo.  Epilogue: signs (int8 out)
//
// A persistent CTA per SM walks 128-vector tiles.  warp 0: TMA loads of the tile's A chunks
// (128 rows x 64 columns, 128-byte swizzle, one slot per k-chunk and piece) and bulk copies of
// B chunks (128 output columns x 64 k, 16 KB, pre-swizzled image in global memory, L2-resident)
// through a ring; warp 1: tcgen05.mma M=128 N=128 K=16 into one 128-column accumulator per
// block of 128 output columns; the other warps: per tile in flight (two) one epilogue warpgroup
// per block of 128 columns, thread = vector.  Every mbarrier wait is bounded; on expiry the CTA raises an abort flag, records a
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
constexpr int kNB = 4;                         // B ring stages
constexpr uint32_t kRawChunk = 128 * 64;       // index bytes of a k-chunk: 128 rows x 64
constexpr int kExpandThreads = 64;             // stage 2: two expander warps, thread = two rows

template <int D>
struct VCfg {
  static constexpr int KC = D / 64;            // k chunks
  static constexpr int NBLK = D / 128;         // blocks of 128 output columns
  // A: two k-chunk slots per piece (chunk kc lands in slot kc & 1 and is released as soon as its MMAs are done), so
  // that the B ring can hold stages of ALL output columns: one MMA of N = D per k-step instead of one per block of
  // 128 columns, which reads the A operand once (M = 128 takes 65 clocks at N = 128 and 129 at N = 256)
  static constexpr int kASlots = 2;
  static constexpr uint32_t kBStage = NBLK * kChunk;                     // one k-chunk of B for all D output columns
  static constexpr uint32_t kOffA = 0;                                   // [piece 2][slot 2] chunks
  static constexpr uint32_t kOffB = kOffA + 2u * kASlots * kChunk;       // ring
  static constexpr uint32_t kOffRaw = kOffB + kNB * kBStage;             // stage 2: index bytes of two k-chunks
  static constexpr uint32_t kOffTab = kOffRaw + 2u * kRawChunk;          // thresholds, centroid piece pairs, cell table, partial sums
  static constexpr uint32_t kOffBar = kOffTab + 6144;
  static constexpr int kThreads = 64 + 2 * NBLK * 128;                   // two tiles in flight, one warpgroup per 128 columns
  static constexpr int threads(int stage) { return kThreads + (stage == 2 ? kExpandThreads : 0); }
  static constexpr uint32_t kUsedBytes = kOffBar + 256;
  static constexpr uint32_t kSmemBytes = kUsedBytes + 1024;
  static constexpr uint32_t kImageBytes = 2u * KC * NBLK * kChunk;       // [piece][kc][nb] chunks of one operand
  static constexpr int kTmemCols = 2 * NBLK * 128;                       // two tiles in flight
};
static_assert(VCfg<256>::kSmemBytes <= 232448 && VCfg<128>::kSmemBytes <= 232448, "shared memory budget");

struct V2Stage {
  CUtensorMap a_hi_map;      // fp16 (D, n), box 64 x 128, 128-byte swizzle
  CUtensorMap a_lo_map;      // second piece of A (stages 2 and 3)
  const uint8_t* b_image;    // [piece][kc][nb][128 rows x 128 bytes swizzled]
  const float* codebook;     // stage 1
  const uint16_t* x;         // stage 2: the original vectors (n, D) fp16
  uint16_t* p_hi;            // scratch (n, D): after stage 1 (156 -> 124 us for the call below with one byte per coordinate
                             // instead of four of centroid pieces) the first D bytes of a row are the vector's index bytes, after
                             // stage 2 (which reads a tile's bytes before it writes the tile's rows) the residual's pieces
  uint16_t* p_lo;
  float* norms;              // scratch (n): ||x||
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

__device__ int g_v2_status;    // 0 = ok; otherwise (stage << 20) | (code << 16) | block

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
  // operand row (= accumulator column) n of Pi^T holds output column 16 t + 2 r + j of its 64, where n = 8 r + 2 t + j: the
  // stage's TMEM loads give thread t of a quad the accumulator columns 8 r + 2 t + {0, 1}, which are then 16 in a row
  const int col = blockIdx.y == 1 ? (n & ~63) + 16 * ((n >> 1) & 3) + 2 * ((n >> 3) & 7) + (n & 1) : n;
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

template <int D, int STAGE>
__global__ void __launch_bounds__(VCfg<D>::kThreads + (STAGE == 2 ? kExpandThreads : 0), 1) k_umma_v2_stage(const __grid_constant__ V2Stage p) {
  // The wait comes before the TMEM allocation: a dependent that held TMEM while its predecessor still had to allocate some
  // on the same SM would wait for good.  For the same reason the last stage does not let a dependent start: what follows it
  // is not this library's, and may allocate TMEM before it waits.
  if constexpr (STAGE != 3) pdl_trigger();
  pdl_wait();
  using C = VCfg<D>;
  constexpr int KC = C::KC, NBLK = C::NBLK;
  constexpr int PA = STAGE == 1 ? 1 : 2;       // pieces of A
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gbase = smem_raw + (base - smem_u32(smem_raw));
  {
    uint32_t dyn_bytes;
    asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn_bytes));
    if (base - smem_u32(smem_raw) + C::kUsedBytes > dyn_bytes) {     // the layout does not fit: report, do nothing
      if (threadIdx.x == 0 && p.status != nullptr) atomicCAS(p.status, 0, (STAGE << 20) | (9 << 16) | (int)blockIdx.x);
      return;
    }
  }
  const uint32_t a_smem = base + C::kOffA;
  const uint32_t b_smem = base + C::kOffB;
  float* thr_s = reinterpret_cast<float*>(gbase + C::kOffTab);
  uint32_t* lut_s = reinterpret_cast<uint32_t*>(gbase + C::kOffTab + 1024);
  uint8_t* cells_s = gbase + C::kOffTab + 2048;                        // 1028 bytes
  float* part_s = reinterpret_cast<float*>(gbase + C::kOffTab + 4096); // [slot 2][block 2][row 128] partial sums of the residual norms
  const uint32_t bar0 = base + C::kOffBar;
  const uint32_t bar_afull = bar0;                          // [kASlots] TMA -> MMA (all pieces of a k-chunk)
  const uint32_t bar_aempty = bar_afull + 8 * 4;            // [kASlots] MMA commit -> producer
  const uint32_t bar_bfull = bar_aempty + 8 * 4;            // [kNB] bulk copy -> MMA
  const uint32_t bar_bempty = bar_bfull + 8 * kNB;          // [kNB] MMA commit -> producer
  const uint32_t bar_tfull = bar_bempty + 8 * kNB;          // [2] MMA commit -> epilogue
  const uint32_t bar_tempty = bar_tfull + 16;               // [2] epilogue (4 arrivals) -> MMA
  const uint32_t bar_rfull = bar_tempty + 16;               // [2] stage 2: TMA -> expanders (index bytes)
  const uint32_t bar_rempty = bar_rfull + 16;               // [2] stage 2: expanders -> producer
  const uint32_t raw_smem = base + C::kOffRaw;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gbase + C::kOffBar + 200);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gbase + C::kOffBar + 208);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int total = p.tiles;
  const int t0 = (int)((int64_t)total * blockIdx.x / gridDim.x);
  const int t1 = (int)((int64_t)total * (blockIdx.x + 1) / gridDim.x);
  const int n_local = t1 - t0;

  if (threadIdx.x == 0) {
    for (int i = 0; i < C::kASlots; ++i) { mbar_init(bar_afull + 8 * i, STAGE == 2 ? kExpandThreads : 1); mbar_init(bar_aempty + 8 * i, 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(bar_rfull + 8 * i, 1); mbar_init(bar_rempty + 8 * i, kExpandThreads); }
    for (int i = 0; i < kNB; ++i) { mbar_init(bar_bfull + 8 * i, 1); mbar_init(bar_bempty + 8 * i, 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(bar_tfull + 8 * i, 1); mbar_init(bar_tempty + 8 * i, 4 * NBLK); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if constexpr (STAGE != 3) {
    if (threadIdx.x >= 64 && threadIdx.x < 64 + 256) {
      const int e = threadIdx.x - 64;
      thr_s[e] = __ldg(p.codebook + kThresholdOff + e);
      const float c = __ldg(p.codebook + kCentroidOff + e);
      const __half h = __float2half_rn(c);
      const __half l = __float2half_rn(c - __half2float(h));
      lut_s[e] = (uint32_t)__half_as_ushort(h) | ((uint32_t)__half_as_ushort(l) << 16);
      for (int w = e; w < 257; w += 256) reinterpret_cast<uint32_t*>(cells_s)[w] = __float_as_uint(__ldg(p.codebook + 528 + w));
    }
  }
  if (warp == 1) tmem_alloc(smem_u32((const void*)tmem_slot), C::kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      bool ok = true;
      int bc = 0;                                           // running B chunk counter
      int ac = 0;                                           // running A chunk counter: slot ac & 1, use ac / 2
      for (int i = 0; i < n_local && ok; ++i) {
        const int row0 = (t0 + i) * kRowsT;
        for (int kc = 0; kc < KC && ok; ++kc, ++ac) {
          const int as = ac % C::kASlots;
          if constexpr (STAGE == 2) {                       // the operand itself is written by the expanders
            ok = mbar_wait(bar_rempty + 8 * as, (uint32_t)(((ac / C::kASlots) & 1) ^ 1), abort_flag);
            if (!ok) break;
            mbar_arrive_expect_tx(bar_rfull + 8 * as, kRawChunk);
            tma_load_2d(raw_smem + as * kRawChunk, &p.a_hi_map, kc * 64, row0, bar_rfull + 8 * as);
          } else {
            ok = mbar_wait(bar_aempty + 8 * as, (uint32_t)(((ac / C::kASlots) & 1) ^ 1), abort_flag);
            if (!ok) break;
            mbar_arrive_expect_tx(bar_afull + 8 * as, PA * kChunk);
            tma_load_2d(a_smem + as * kChunk, &p.a_hi_map, kc * 64, row0, bar_afull + 8 * as);
            if constexpr (PA == 2) tma_load_2d(a_smem + (C::kASlots + as) * kChunk, &p.a_lo_map, kc * 64, row0, bar_afull + 8 * as);
          }
          for (int pb = 0; pb < 2; ++pb) {
            const int s = bc % kNB;
            ok = mbar_wait(bar_bempty + 8 * s, (uint32_t)(((bc / kNB) & 1) ^ 1), abort_flag);
            if (!ok) break;
            mbar_arrive_expect_tx(bar_bfull + 8 * s, C::kBStage);
            bulk_load(b_smem + s * C::kBStage, p.b_image + (size_t)(pb * KC + kc) * C::kBStage, C::kBStage, bar_bfull + 8 * s);
            ++bc;
          }
        }
      }
      if (!ok) {
        *abort_flag = 1;
        if (p.status != nullptr) atomicCAS(p.status, 0, (STAGE << 20) | (1 << 16) | (int)blockIdx.x);
      }
      // none of this CTA's own copies may still be in flight when it exits
      for (int k = 0; k < C::kASlots && k < ac; ++k) {
        const int j = ac - 1 - k;
        mbar_wait((STAGE == 2 ? bar_rfull : bar_afull) + 8 * (j % C::kASlots), (uint32_t)((j / C::kASlots) & 1), abort_flag);
      }
      for (int k = 0; k < kNB && k < bc; ++k) {
        const int j = bc - 1 - k;
        mbar_wait(bar_bfull + 8 * (j % kNB), (uint32_t)((j / kNB) & 1), abort_flag);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (converged warp, one elected lane issues)
    bool ok = true;
    int bc = 0;
    // M = 128, N = D (all output columns in one instruction: rows 128.. of the B stage are the second block), fp16
    const uint32_t idesc = (idesc_f16(false) & ~(0x3Fu << 17)) | ((uint32_t)(D >> 3) << 17);
    int ac = 0;
    for (int i = 0; i < n_local && ok; ++i) {
      const int slot = i & 1;
      ok = mbar_wait(bar_tempty + 8 * slot, (uint32_t)(((i >> 1) & 1) ^ 1), abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
#pragma unroll 1
      for (int kc = 0; kc < KC && ok; ++kc, ++ac) {
        const int as = ac % C::kASlots;
        ok = mbar_wait(bar_afull + 8 * as, (uint32_t)((ac / C::kASlots) & 1), abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        const uint64_t a_hi = smem_desc_sw128(a_smem + as * kChunk);
        const uint64_t a_lo = smem_desc_sw128(a_smem + (C::kASlots + as) * kChunk);
        {
          const uint32_t d_tmem = tmem_base + (uint32_t)(slot * NBLK * 128);
#pragma unroll 1
          for (int pb = 0; pb < 2; ++pb) {
            const int s = bc % kNB;
            ok = mbar_wait(bar_bfull + 8 * s, (uint32_t)((bc / kNB) & 1), abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const uint64_t b_desc = smem_desc_sw128(b_smem + s * C::kBStage);
            if (elect_one()) {
              if (pb == 0) {
#pragma unroll
                for (int k = 0; k < 4; ++k) umma_f16(d_tmem, a_hi + (uint64_t)(k * 2), b_desc + (uint64_t)(k * 2), idesc, (kc | k) != 0 ? 1u : 0u);
                if constexpr (PA == 2) {
#pragma unroll
                  for (int k = 0; k < 4; ++k) umma_f16(d_tmem, a_lo + (uint64_t)(k * 2), b_desc + (uint64_t)(k * 2), idesc, 1u);
                }
              } else {
#pragma unroll
                for (int k = 0; k < 4; ++k) umma_f16(d_tmem, a_hi + (uint64_t)(k * 2), b_desc + (uint64_t)(k * 2), idesc, 1u);
              }
              umma_commit(bar_bempty + 8 * s);              // the ring stage is free once these MMAs are done
              if (pb == 1) {
                umma_commit(bar_aempty + 8 * as);           // last use of this k-chunk of A
                if (kc == KC - 1) umma_commit(bar_tfull + 8 * slot);
              }
            }
            __syncwarp();
            ++bc;
          }
        }
      }
    }
    if (!ok && lane == 0) {
      *abort_flag = 1;
      if (p.status != nullptr) atomicCAS(p.status, 0, (STAGE << 20) | (2 << 16) | (int)blockIdx.x);
    }
  } else if (STAGE == 2 && warp >= C::kThreads / 32) {
    // ------------------------------------------------------------ expanders (stage 2): index bytes of a k-chunk -> centroid
    // pieces hi and lo in operand layout, thread = two rows.  The thread walks its four 16-byte pieces in an order XOR-ed with
    // `g`, a linear map of the row's bits 1 and 2 for which the map and its sum with the identity are both one-to-one:
    // the eight rows of a quarter warp then read eight different bank groups of the raw chunk and write eight different
    // ones of the operand.
    const uint32_t lut = smem_u32(lut_s);
    bool ok = true;
    int ac = 0;
    for (int i = 0; i < n_local && ok; ++i) {
      for (int kc = 0; kc < KC && ok; ++kc, ++ac) {
        const int as = ac % C::kASlots;
        const uint32_t parity = (uint32_t)((ac / C::kASlots) & 1);
        ok = mbar_wait(bar_rfull + 8 * as, parity, abort_flag) && mbar_wait(bar_aempty + 8 * as, parity ^ 1u, abort_flag);
        if (!ok) break;
#pragma unroll 1
        for (int row = threadIdx.x - C::kThreads; row < kRowsT; row += kExpandThreads) {
        const uint32_t r1 = (uint32_t)(row >> 1) & 1u, r2 = (uint32_t)(row >> 2) & 1u;
        const uint32_t g = ((r2 ^ r1) << 1) | r2;
        const uint32_t src = raw_smem + as * kRawChunk + (uint32_t)row * 64u;
        const uint32_t dst = a_smem + as * kChunk + (uint32_t)row * 128u;
#pragma unroll
        for (uint32_t c = 0; c < 4; ++c) {
          const uint32_t cc = c ^ g;
          const uint4 x = ld_shared_v4(src + cc * 16u);
          const uint32_t xw[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
          for (uint32_t h = 0; h < 2; ++h) {                // 8 coordinates: one 16-byte operand chunk per piece
            uint32_t e[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              const uint32_t w = xw[2 * h + (u >> 2)];
              const int sh = 8 * (u & 3);
              const uint32_t off = sh == 0 ? ((w << 2) & 0x3FCu) : ((w >> (sh - 2)) & 0x3FCu);
              asm volatile("ld.shared.b32 %0, [%1];" : "=r"(e[u]) : "r"(lut + off));
            }
            const uint32_t at = dst + (((2u * cc + h) ^ (uint32_t)(row & 7)) << 4);
            st_shared_v4(at, __byte_perm(e[0], e[1], 0x5410), __byte_perm(e[2], e[3], 0x5410), __byte_perm(e[4], e[5], 0x5410),
                         __byte_perm(e[6], e[7], 0x5410));
            st_shared_v4(at + C::kASlots * kChunk, __byte_perm(e[0], e[1], 0x7632), __byte_perm(e[2], e[3], 0x7632),
                         __byte_perm(e[4], e[5], 0x7632), __byte_perm(e[6], e[7], 0x7632));
          }
        }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // operand writes -> visible to the tensor core
        mbar_arrive(bar_afull + 8 * as);
        mbar_arrive(bar_rempty + 8 * as);
      }
    }
    if (!ok) {
      *abort_flag = 1;
      if (p.status != nullptr) atomicCAS(p.status, 0, (STAGE << 20) | (4 << 16) | (int)blockIdx.x);
    }
  } else {
    // ------------------------------------------------------------ epilogue: per tile in flight one warpgroup per block
    // of 128 output columns, thread = vector
    const int ew = warp - 2;
    const int wgi = ew >> 2;
    const int slot = wgi / NBLK, blk = wgi % NBLK;
    const int quarter = warp & 3;                 // TMEM lanes this warp may touch: 32*quarter ..
    const int rloc = quarter * 32 + lane;
    bool ok = true;
    // search shortcut of the codebook (stage 1): 1 = polynomial, 2 = cell table, 0 = binary search
    int mode = 0;
    float sc_s = 0.f, sc_c1 = 0.f, sc_c2 = 0.f, sc_c3 = 0.f;
    if constexpr (STAGE == 1) {
      mode = (int)__ldg(p.codebook + 512);
      sc_s = __ldg(p.codebook + 513);
      sc_c1 = __ldg(p.codebook + 514);
      sc_c2 = __ldg(p.codebook + 515);
      sc_c3 = __ldg(p.codebook + 516);
    }
    for (int i = slot; i < n_local && ok; i += 2) {
      const int64_t row = (int64_t)(t0 + i) * kRowsT + rloc;
      const bool valid = row < p.n;
      // stage 2: a quad of lanes holds 64 columns of a row, 16 each, so that its accesses to x, k_mse and the pieces are whole
      // 128-byte lines (see below).  The norms and the first coordinates are in flight while the tile's contraction runs.
      const int quad = lane & 3, r8 = lane >> 2;
      const int64_t qrow = (int64_t)(t0 + i) * kRowsT + quarter * 32 + r8;        // rows qrow + {0, 8, 16, 24}
      const bool x_wide = ((uintptr_t)p.x & 31u) == 0;
      uint32_t xn[8];
      float nv4[4];
      if constexpr (STAGE == 2) {
#pragma unroll
        for (int u = 0; u < 4; ++u) nv4[u] = qrow + 8 * u < p.n ? p.norms[qrow + 8 * u] : 0.f;
        load_row32(p.x + (qrow < p.n ? qrow : 0) * D + blk * 128 + 16 * quad, xn, x_wide);
      }
      // The exit decision is made uniform before anything collective: per warp (the TMEM loads are
      // warp-collective) and, where the two warpgroups of a tile later meet at a named barrier (stage 2,
      // head_dim 256), over those 256 threads, so that nobody waits at that barrier for a warp that left.
      ok = __all_sync(0xffffffffu, mbar_wait(bar_tfull + 8 * slot, (uint32_t)((i >> 1) & 1), abort_flag));
      if constexpr (STAGE == 2 && NBLK == 2) ok = bar_red_and(3 + slot, 256, ok);
      if (!ok) break;
      tc_fence_after();
      const uint32_t tile_acc = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(slot * NBLK * 128);
      const uint32_t tacc = tile_acc + (uint32_t)(blk * 128);     // this warpgroup's block of columns
      const int col0 = blk * 128;
      uint32_t v[16];
      if constexpr (STAGE == 1) {
        float ssq = 0.f;                         // the norm needs every column: both warpgroups sweep the whole row
        uint32_t v2[16];                         // two buffers: a TMEM load is in flight behind the arithmetic
        tmem_issue16(tile_acc, v);
#pragma unroll 1
        for (int c = 0; c < D / 16; c += 2) {
          tmem_wait16(v);
          tmem_issue16(tile_acc + (c + 1) * 16, v2);
#pragma unroll
          for (int e = 0; e < 16; ++e) ssq = fmaf(__uint_as_float(v[e]), __uint_as_float(v[e]), ssq);
          tmem_wait16(v2);
          tmem_issue16(c + 2 < D / 16 ? tile_acc + (c + 2) * 16 : tacc, v);      // after the last step: step 0 of the sweep below
#pragma unroll
          for (int e = 0; e < 16; ++e) ssq = fmaf(__uint_as_float(v2[e]), __uint_as_float(v2[e]), ssq);
        }
        const float norm = __fsqrt_rn(ssq);
        const float inv = __fdiv_rn(1.0f, norm + 1e-8f);
        if (valid && blk == 0) p.norms[row] = norm;
        const int bits = p.bits;
        uint32_t ib0[4] = {0u, 0u, 0u, 0u};       // index bytes of the even step
#pragma unroll 1
        for (int c = 0; c < 8; ++c) {
          tmem_wait16(v);
          uint32_t ib[4] = {0u, 0u, 0u, 0u};
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const float y = __uint_as_float(v[e]) * inv;
            int idx;
            if (mode != 0) {
              // candidate e0 with index in {e0, e0 + 1} (verified on the host for every y), then one exact compare
              float t;
              asm("fma.rn.sat.f32 %0, %1, %2, 0f3F000000;" : "=f"(t) : "f"(y), "f"(sc_s));
              int e0;
              if (mode == 1) {
                float q = fmaf(sc_c3, t, sc_c2);
                q = fmaf(q, t, sc_c1);
                e0 = __float_as_int(fmaf(q, t, 8388608.0f)) & 0xFF;
              } else {
                e0 = cells_s[__float_as_int(fmaf(t, 1024.0f, 8388608.0f)) & 0x7FF];
              }
              idx = e0 + (y > thr_s[e0] ? 1 : 0);
            } else {
              int lo = 0, hi = (1 << bits) - 1;
              for (int step = 0; step < bits; ++step) {
                const int mid = (lo + hi) >> 1;
                if (y > thr_s[mid]) lo = mid + 1; else hi = mid;
              }
              idx = lo;
            }
            ib[e >> 2] |= (uint32_t)idx << (8 * (e & 3));
          }
          if (c + 1 < 8) tmem_issue16(tacc + (c + 1) * 16, v);
          if (valid && p.idx_u8_out != nullptr)
            *reinterpret_cast<uint4*>(p.idx_u8_out + row * D + col0 + c * 16) = make_uint4(ib[0], ib[1], ib[2], ib[3]);
          if (valid && p.idx_packed_out != nullptr) {
            // the 16 indices of this step as 16 / ipb packed bytes of the row
            const int ipb = 8 / bits;
            uint8_t* dst = p.idx_packed_out + row * (int64_t)(D / ipb) + (col0 + c * 16) / ipb;
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
          if ((c & 1) == 0) {                     // two steps leave as one access
#pragma unroll
            for (int j = 0; j < 4; ++j) ib0[j] = ib[j];
          } else if (valid) {
            const uint32_t both[8] = {ib0[0], ib0[1], ib0[2], ib0[3], ib[0], ib[1], ib[2], ib[3]};
            store_row32(reinterpret_cast<uint8_t*>(p.p_hi + row * D) + col0 + (c - 1) * 16, both, true);
          }
        }
      } else if constexpr (STAGE == 2) {
        // Rows x 32 bytes per access cost the load/store unit a slot per row (see store_row32), and the operand traffic of the
        // MMAs and the expanders runs through the same data path: thread = row took 199 us here for the call above, of
        // which 16 400 of 26 600 clocks per tile were such slots.  tcgen05.ld.16x256b spreads a row over a quad of lanes
        // instead: thread (r8, quad) gets rows r8 and r8 + 8 of 16, 16 columns each, and a warp's access is 8 lines: 133 us.
        const bool k_wide = ((uintptr_t)p.k_mse_out & 31u) == 0;
#pragma unroll
        for (int rg = 0; rg < 2; ++rg) {            // 16 rows
          float sq[2] = {0.f, 0.f};
#pragma unroll
          for (int cg = 0; cg < 2; ++cg) {          // 64 columns
            uint32_t a[32];
            tmem_ld_quads(tacc + ((uint32_t)(rg * 16) << 16) + (uint32_t)(cg * 64), a);
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
              const int64_t r = qrow + 16 * rg + 8 * hh;
              const int64_t at = r * D + col0 + 64 * cg + 16 * quad;
              uint32_t xw[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) xw[j] = xn[j];
              const int nxt = 4 * rg + 2 * cg + hh + 1;                // the next (rg, cg, hh)
              if (nxt < 8) {
                const int64_t rn = qrow + 16 * (nxt >> 2) + 8 * (nxt & 1);
                load_row32(p.x + (rn < p.n ? rn : 0) * D + col0 + 64 * ((nxt >> 1) & 1) + 16 * quad, xn, x_wide);
              }
              if (r < p.n) {
                const float nv = nv4[2 * rg + hh];
                uint32_t kq[8], rh[8], rl[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                  const float k0 = __uint_as_float(a[4 * j + 2 * hh]) * nv, k1 = __uint_as_float(a[4 * j + 2 * hh + 1]) * nv;
                  const __half2 xh = *reinterpret_cast<const __half2*>(&xw[j]);
                  const float r0 = __low2float(xh) - k0, r1 = __high2float(xh) - k1;
                  sq[hh] = fmaf(r0, r0, sq[hh]);
                  sq[hh] = fmaf(r1, r1, sq[hh]);
                  const __half2 kh = __floats2half2_rn(k0, k1);
                  kq[j] = *reinterpret_cast<const uint32_t*>(&kh);
                  const __half2 h2 = __floats2half2_rn(r0, r1);
                  rh[j] = *reinterpret_cast<const uint32_t*>(&h2);
                  const __half2 l2 = __floats2half2_rn(r0 - __low2float(h2), r1 - __high2float(h2));
                  rl[j] = *reinterpret_cast<const uint32_t*>(&l2);
                }
                if (p.k_mse_out != nullptr) store_row32(p.k_mse_out + at, kq, k_wide);
                store_row32(p.p_hi + at, rh, true);
                store_row32(p.p_lo + at, rl, true);
              }
            }
          }
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {          // the quad's four parts of a row
            sq[hh] += __shfl_xor_sync(0xffffffffu, sq[hh], 1);
            sq[hh] += __shfl_xor_sync(0xffffffffu, sq[hh], 2);
            const int64_t r = qrow + 16 * rg + 8 * hh;
            if constexpr (NBLK == 2) {
              // the residual norm spans both blocks: each warpgroup leaves its part
              if (quad == 0) part_s[(slot * 2 + blk) * 128 + quarter * 32 + r8 + 16 * rg + 8 * hh] = sq[hh];
            } else {
              if (quad == 0 && r < p.n) p.rnorm_out[r] = __half_as_ushort(__float2half_rn(__fsqrt_rn(sq[hh])));
            }
          }
        }
        if constexpr (NBLK == 2) {
          asm volatile("bar.sync %0, 256;" ::"r"(1 + slot) : "memory");
          if (blk == 0 && valid)
            p.rnorm_out[row] = __half_as_ushort(__float2half_rn(__fsqrt_rn(part_s[slot * 2 * 128 + rloc] + part_s[(slot * 2 + 1) * 128 + rloc])));
          asm volatile("bar.sync %0, 256;" ::"r"(1 + slot) : "memory");     // part_s is reused by the next tile
        }
      } else {
        const bool s_wide = ((uintptr_t)p.signs_out & 31u) == 0;
#pragma unroll 1
        for (int c = 0; c < 8; c += 2) {
          uint32_t v2[16];
          tmem_issue16(tacc + c * 16, v);
          tmem_issue16(tacc + (c + 1) * 16, v2);
          tmem_wait16(v);
          tmem_wait16(v2);
          if (valid && p.signs_out != nullptr) {
            uint32_t sw[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              uint32_t x = 0u;
#pragma unroll
              for (int b = 0; b < 4; ++b) {
                const uint32_t s8 = __uint_as_float(j < 4 ? v[4 * j + b] : v2[4 * (j - 4) + b]) >= 0.f ? 0x01u : 0xFFu;
                x |= s8 << (8 * b);
              }
              sw[j] = x;
            }
            store_row32(p.signs_out + row * D + col0 + c * 16, sw, s_wide);
          }
          if (valid && p.sign_bits_out != nullptr) {
            uint32_t o = 0u;
#pragma unroll
            for (int e = 0; e < 32; ++e)
              o |= (__uint_as_float(e < 16 ? v[e] : v2[e - 16]) >= 0.f ? 1u : 0u) << (8 * (e >> 3) + 7 - (e & 7));
            *reinterpret_cast<uint32_t*>(p.sign_bits_out + row * (D / 8) + (col0 + c * 16) / 8) = o;
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_tempty + 8 * slot);
    }
    if (!ok && lane == 0) {
      *abort_flag = 1;
      if (p.status != nullptr) atomicCAS(p.status, 0, (STAGE << 20) | (3 << 16) | (int)blockIdx.x);
    }
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

template <int D, int STAGE>
int launch_stage(const V2Stage& p, int grid, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(k_umma_v2_stage<D, STAGE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)VCfg<D>::kSmemBytes);
  if (e != cudaSuccess) return refused(e);
  launch_after(k_umma_v2_stage<D, STAGE>, dim3(grid), dim3(VCfg<D>::threads(STAGE)), VCfg<D>::kSmemBytes, st, p);
  return check_launch();
}

template <int D>
int run(const TqQjlCompressJob& job, cudaStream_t st) {
  TensorMapEncodeFn enc = tensor_map_encoder();
  if (enc == nullptr) return TQ_ELAUNCH;
  const int64_t n = job.B * job.H * job.S;
  const int64_t tiles = (n + kRowsT - 1) / kRowsT;
  if (tiles >= ((int64_t)1 << 30)) return TQ_ETOOBIG;
  // workspace: three operand images, then the two piece arrays, then the norms
  uint8_t* ws = reinterpret_cast<uint8_t*>(((uintptr_t)job.workspace + 1023u) & ~(uintptr_t)1023u);
  const size_t img = VCfg<D>::kImageBytes;
  uint8_t* img1 = ws;
  uint8_t* img2 = ws + img;
  uint8_t* img3 = ws + 2 * img;
  const size_t piece = ((size_t)n * D * 2 + 1023) / 1024 * 1024;
  uint16_t* p_hi = reinterpret_cast<uint16_t*>(ws + 3 * img);
  uint16_t* p_lo = reinterpret_cast<uint16_t*>(ws + 3 * img + piece);
  float* norms = reinterpret_cast<float*>(ws + 3 * img + 2 * piece);
  const int ib = (D * D + 255) / 256;
  k_v2_operand_image<D><<<dim3(ib, 3), 256, 0, st>>>(job.rotation, job.qjl_t, job.M, img1);
  int rc = check_launch();
  if (rc != TQ_OK) return rc;
  static thread_local V2Stage p;
  void* status_ptr = nullptr;
  cudaGetSymbolAddress(&status_ptr, g_v2_status);
  p.status = reinterpret_cast<int32_t*>(status_ptr);
  p.codebook = job.codebook;
  p.x = reinterpret_cast<const uint16_t*>(job.x);
  p.p_hi = p_hi;
  p.p_lo = p_lo;
  p.norms = job.vec_norms_out != nullptr ? job.vec_norms_out : norms;
  p.idx_u8_out = job.idx_mode == TQ_IDX_PACKED ? nullptr : reinterpret_cast<uint8_t*>(job.idx_out);
  p.idx_packed_out = job.idx_mode == TQ_IDX_PACKED ? reinterpret_cast<uint8_t*>(job.idx_out) : nullptr;
  p.k_mse_out = job.k_mse_out;
  p.rnorm_out = reinterpret_cast<uint16_t*>(job.rnorm_out);
  p.signs_out = job.signs_dtype == 2 ? nullptr : reinterpret_cast<int8_t*>(job.signs_out);
  p.sign_bits_out = job.signs_dtype == 2 ? reinterpret_cast<uint8_t*>(job.signs_out) : nullptr;
  p.n = n;
  p.tiles = (int32_t)tiles;
  p.bits = job.bits;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int grid = (int)(tiles < sms ? tiles : sms);
  // stage 1: A = x
  if ((rc = encode_rows(enc, &p.a_hi_map, job.x, n, D)) != TQ_OK) return rc;
  p.a_lo_map = p.a_hi_map;
  p.b_image = img1;
  if ((rc = launch_stage<D, 1>(p, grid, st)) != TQ_OK) return rc;
  // stage 2: A from the index bytes at the head of the rows of p_hi
  if ((rc = encode_index_rows(enc, &p.a_hi_map, p_hi, n, D)) != TQ_OK) return rc;
  p.b_image = img2;
  if ((rc = launch_stage<D, 2>(p, grid, st)) != TQ_OK) return rc;
  // stage 3: A = the piece arrays
  if ((rc = encode_rows(enc, &p.a_hi_map, p_hi, n, D)) != TQ_OK) return rc;
  if ((rc = encode_rows(enc, &p.a_lo_map, p_lo, n, D)) != TQ_OK) return rc;
  p.b_image = img3;
  return launch_stage<D, 3>(p, grid, st);
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
