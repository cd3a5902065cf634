// Attention straight from packed keys (and packed values) on the tensor cores, head_dim 128.
//
// Logits  l[g][s] = scale * norm_s * sum_j (q_g Pi^T)_j * c[idx_sj]  are a contraction over the 128
// coordinates.  The FP32 kernel (tq_simt.cu) spends ~1 400 instructions per key on it; here the
// multiply-adds run as mma.sync.m16n8k16 (fp16 inputs, fp32 accumulate) and only the centroid look-ups
// stay on the CUDA cores:
//   * M = 16 rows = 8 keys x the fp16 pieces hi and lo of their centroids (key gid's pieces are rows gid and gid + 8, which
//     the same lanes hold), K = 16 coordinates per instruction (8 k-steps per key), N = 8 columns = up to 4 query rows (the
//     query heads that share the KV head x query tokens) as fp16 pieces: columns 0..3 hold q_hi, columns 4..7 q_lo;
//   * the key operand is assembled IN REGISTERS: thread (gid = lane / 4, t = lane % 4) reads quarter t of
//     the packed rows of its keys (one 4..32-byte load each) and looks up the centroids each
//     k-step needs in a shared table.  A dot product does not care in which
//     order its terms are visited, so the coordinates are assigned to k-steps in the order that makes a
//     thread's operand elements come from its own contiguous bytes: k-step ks, thread t covers coordinates
//     32 t + 4 ks + 0..3 (the query operand uses the same order);
//   * a look-up of one packed byte returns the high pieces of two neighbouring coordinates in one word and their low pieces in the
//     next: two operand registers in a row (rows gid and gid + 8), as the instruction wants them.  With the pieces of ONE
//     coordinate as the neighbouring k of a register, and 16 keys as the rows, the registers of an operand came from two
//     look-ups each and took a move per coordinate (80 of the 311 instructions per 16 keys);
//   * rows gid and gid + 8 of column g add up to (c_hi + c_lo).q_hi, of column g + 4 to (c_hi + c_lo).q_lo; their sum is the
//     fp32-accurate logit (all four cross terms), one shuffle away.
// The softmax partials per block of keys and the finishing pass are those of the FP32 path.

#include <atomic>
#include <cfloat>
#include <type_traits>

#include "tq_common.cuh"
#include "tq_internal.h"
#include "tq_pdl.cuh"

namespace tq {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kRows = 4;                       // query rows per pass (columns g and g + 4 of the accumulator)
constexpr int kDimA = 128;

__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                          uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t pack_half2(float x, float y) {
  __half2 h = __floats2half2_rn(x, y);
  return *reinterpret_cast<uint32_t*>(&h);
}

// fp16 pieces of two floats: hi = rn(x), lo = rn(x - hi)
__device__ __forceinline__ void split2(float x, float y, uint32_t& hi, uint32_t& lo) {
  const __half hx = __float2half_rn(x), hy = __float2half_rn(y);
  hi = (uint32_t)__half_as_ushort(hx) | ((uint32_t)__half_as_ushort(hy) << 16);
  lo = pack_half2(x - __half2float(hx), y - __half2float(hy));
}

template <int BITS>
struct Packed {
  static constexpr int IPB = 8 / BITS;
  static constexpr int G = kDimA / IPB;        // packed bytes per key
  static constexpr int CB = G / 4;             // bytes per thread: a quarter row = 32 coordinates
  static constexpr int CW = CB / 4;            // 32-bit words per thread: 1, 2, 4 or 8
};

// the quarter row `t` of one key
template <int BITS>
__device__ __forceinline__ void load_quarter(const uint8_t* row, int t, uint32_t (&w)[Packed<BITS>::CW]) {
  constexpr int CW = Packed<BITS>::CW;
  const uint8_t* p = row + t * Packed<BITS>::CB;
  if constexpr (CW == 1) {
    w[0] = __ldg(reinterpret_cast<const uint32_t*>(p));
  } else if constexpr (CW == 2) {
    const uint2 v = __ldg(reinterpret_cast<const uint2*>(p));
    w[0] = v.x; w[1] = v.y;
  } else {
#pragma unroll
    for (int k = 0; k < CW / 4; ++k) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(p) + k);
      w[4 * k] = v.x; w[4 * k + 1] = v.y; w[4 * k + 2] = v.z; w[4 * k + 3] = v.w;
    }
  }
}

// Table of a packed BYTE: row v (128 bytes) holds what a byte of value v stands for, once per lane that reads in the same
// shared-memory wavefront: 32 copies of one coordinate (5 to 8 bits), 16 of two (3 and 4 bits), 8 of four (2 bits), 4 of
// eight (1 bit).  A look-up is then one load of 4, 8 or 16 bytes that never meets another lane's in a bank, and its address a
// shift, a mask and the lane's own offset.  With one 4-byte entry per coordinate, stored once, a coordinate cost a byte permute
// and a load of its own, and 64 or more entries collided in the banks (131072 keys x 8 heads, four query rows, with projection
// and softmax: 4 bits 59 -> 49 us, 8 bits 86 -> 56 us).
// PAIRS: the words of a row are {hi0 | hi1 << 16, lo0 | lo1 << 16} for every two coordinates; otherwise, and for codes of one
// coordinate a byte, hi | lo << 16 for each.
template <int BITS>
struct ByteTable {
  static constexpr int IPB = Packed<BITS>::IPB;
  static constexpr int kEntries = 1 << (BITS * IPB);       // 3 bits: 64, the fields that a byte can hold
  static constexpr uint32_t kEntryBytes = 4 * IPB;
  static constexpr uint32_t kLanes = 128 / kEntryBytes;    // copies
  static constexpr uint32_t kBytes = 128 * kEntries;
  static constexpr uint32_t kMask = (uint32_t)(kEntries - 1) << 7;
  __device__ __forceinline__ static uint32_t lane_offset(int lane) { return ((uint32_t)lane % kLanes) * kEntryBytes; }
};

// all threads of the CTA, kThreads >= kEntries; the caller synchronises
template <int BITS, bool PAIRS>
__device__ __forceinline__ void build_table(uint8_t* table, const float* codebook) {
  using T = ByteTable<BITS>;
  const int v = threadIdx.x;
  if (v >= T::kEntries) return;
  uint32_t e[T::IPB];
#pragma unroll
  for (int p = 0; p < T::IPB; ++p) {                       // field p, the first index in the high bits
    const float c = __ldg(codebook + kCentroidOff + ((v >> (BITS * (T::IPB - 1 - p))) & ((1 << BITS) - 1)));
    const __half h = __float2half_rn(c);
    e[p] = (uint32_t)__half_as_ushort(h) | ((uint32_t)__half_as_ushort(__float2half_rn(c - __half2float(h))) << 16);
  }
  if constexpr (PAIRS && T::IPB > 1) {
#pragma unroll
    for (int p = 0; p < T::IPB; p += 2) {
      const uint32_t hi = __byte_perm(e[p], e[p + 1], 0x5410), lo = __byte_perm(e[p], e[p + 1], 0x7632);
      e[p] = hi; e[p + 1] = lo;
    }
  }
  uint4* row = reinterpret_cast<uint4*>(table + 128 * v);
#pragma unroll
  for (int k = 0; k < 8; ++k) {                            // rotated: the stores of a warp spread over the banks
    const int j = (k + v) & 7;
    if constexpr (T::IPB == 8) row[j] = (j & 1) ? make_uint4(e[4], e[5], e[6], e[7]) : make_uint4(e[0], e[1], e[2], e[3]);
    else row[j] = make_uint4(e[0], e[1 % T::IPB], e[2 % T::IPB], e[3 % T::IPB]);
  }
}

// table words of the thread's local coordinates 4 ks .. 4 ks + 3, whose packed bytes are consecutive in w; `lane_off` from
// ByteTable::lane_offset
template <int BITS, int W>
__device__ __forceinline__ void entries4(const uint32_t (&w)[W], int ks, const uint8_t* table, uint32_t lane_off, uint32_t (&e)[4]) {
  using T = ByteTable<BITS>;
  auto row = [&](int byte) -> const uint8_t* {
    const int sh = 8 * (byte & 3) - 7;
    const uint32_t x = w[byte >> 2];
    return table + (((sh < 0 ? x << 7 : x >> (sh < 0 ? 0 : sh)) & T::kMask) | lane_off);
  };
  if constexpr (T::IPB == 1) {
#pragma unroll
    for (int p = 0; p < 4; ++p) e[p] = *reinterpret_cast<const uint32_t*>(row(4 * ks + p));
  } else if constexpr (T::IPB == 2) {
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const uint2 v = *reinterpret_cast<const uint2*>(row(2 * ks + p));
      e[2 * p] = v.x; e[2 * p + 1] = v.y;
    }
  } else {
    const uint4 v = *reinterpret_cast<const uint4*>(row(T::IPB == 4 ? ks : ks >> 1) + (T::IPB == 8 ? 16 * (ks & 1) : 0));
    e[0] = v.x; e[1] = v.y; e[2] = v.z; e[3] = v.w;
  }
}

// operand of one key, k-step ks, from a table of PAIRS: high pieces of coordinates 4 ks, 4 ks + 1 (row gid), their low pieces
// (row gid + 8), and the same of 4 ks + 2, 4 ks + 3
template <int BITS, int W>
__device__ __forceinline__ void key_operand(const uint32_t (&w)[W], int ks, const uint8_t* table, uint32_t lane_off, uint32_t (&a)[4]) {
  entries4<BITS>(w, ks, table, lane_off, a);
  if constexpr (ByteTable<BITS>::IPB == 1) {
#pragma unroll
    for (int p = 0; p < 4; p += 2) {
      const uint32_t hi = __byte_perm(a[p], a[p + 1], 0x5410), lo = __byte_perm(a[p], a[p + 1], 0x7632);
      a[p] = hi; a[p + 1] = lo;
    }
  }
}

// exp for arguments <= 0: below 2^-126 the result is zero
__device__ __forceinline__ float exp_neg(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x * 1.4426950408889634f));
  return y;
}

// (max, sum of exp) running pair
__device__ __forceinline__ void stat_merge(float& m, float& s, float m2, float s2) {
  const float nm = fmaxf(m, m2);
  if (nm != -INFINITY) s = (m == -INFINITY ? 0.f : s * __expf(m - nm)) + (m2 == -INFINITY ? 0.f : s2 * __expf(m2 - nm));
  m = nm;
}

// Codes of one coordinate a byte (5 to 8 bits) with four query rows: the words of a byte table already are operand registers if
// the two neighbouring k of a register are the pieces of ONE coordinate, the rows are 16 keys and the query value stands in
// both places of the other operand.  Pairing the high and the low pieces of two look-ups takes a byte permute per coordinate
// more: 131072 8-bit keys x 8 heads 56 us against 66.  With eight query rows the permutes serve twice the products and the
// widened query values would not fit the registers (65536 6-bit keys x 8 heads, 16 query rows: 90 against 81).
template <int BITS> constexpr bool kCoordWords = BITS >= 5;

// Query operand of one pass of four rows: column n = lane / 4 of the 8-column operand is row r0 + (n & 3) of the rotated
// queries, as its high piece (n < 4) or low piece (n >= 4); thread t holds coordinates 32 t + 4 ks + 0..3, two a register
// (N = 2 registers a k-step) or each in both halves of its own (N = 4).
template <int N>
__device__ __forceinline__ void query_fragments(const float* qrot, int64_t row, bool row_ok, int lane, uint32_t (&bq)[8][N]) {
  const int t = lane & 3;
  const bool low = (lane >> 2) >= 4;
#pragma unroll
  for (int ks = 0; ks < 8; ++ks) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row_ok) v = *reinterpret_cast<const float4*>(qrot + row * kDimA + 32 * t + 4 * ks);
    uint32_t hi[2], lo[2];
    split2(v.x, v.y, hi[0], lo[0]);
    split2(v.z, v.w, hi[1], lo[1]);
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const uint32_t two = low ? lo[p] : hi[p];
      if constexpr (N == 2) {
        bq[ks][p] = two;
      } else {
        bq[ks][2 * p] = __byte_perm(two, 0u, 0x1010);
        bq[ks][2 * p + 1] = __byte_perm(two, 0u, 0x3232);
      }
    }
  }
}

// The same for eight query rows per pass: column n is row r0 + n, high pieces in bh, low pieces in bl.
__device__ __forceinline__ void query_fragments8(const float* qrot, int64_t row, bool row_ok, int lane,
                                                 uint32_t (&bh)[8][2], uint32_t (&bl)[8][2]) {
  const int t = lane & 3;
#pragma unroll
  for (int ks = 0; ks < 8; ++ks) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row_ok) v = *reinterpret_cast<const float4*>(qrot + row * kDimA + 32 * t + 4 * ks);
    split2(v.x, v.y, bh[ks][0], bl[ks][0]);
    split2(v.z, v.w, bh[ks][1], bl[ks][1]);
  }
}
// 16 keys x 8 query rows: c[0..1] = key gid, c[2..3] = key gid + 8, rows 2t, 2t + 1
template <int BITS>
__device__ __forceinline__ void score_block8(const uint32_t (&w0)[Packed<BITS>::CW], const uint32_t (&w1)[Packed<BITS>::CW],
                                             const uint32_t (&bh)[8][2], const uint32_t (&bl)[8][2], const uint8_t* table,
                                             uint32_t lane_off, float (&c)[4]) {
  // the high and the low query pieces in accumulators of their own: the tensor core truncates its sums at their size
  float x[2][4] = {}, y[2][4] = {};
#pragma unroll
  for (int ks = 0; ks < 8; ++ks) {
    uint32_t e[4], f[4];
    key_operand<BITS>(w0, ks, table, lane_off, e);
    key_operand<BITS>(w1, ks, table, lane_off, f);
    mma_16816(x[0], e[0], e[1], e[2], e[3], bh[ks][0], bh[ks][1]);
    mma_16816(y[0], f[0], f[1], f[2], f[3], bh[ks][0], bh[ks][1]);
    mma_16816(x[1], e[0], e[1], e[2], e[3], bl[ks][0], bl[ks][1]);
    mma_16816(y[1], f[0], f[1], f[2], f[3], bl[ks][0], bl[ks][1]);
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    c[j] = x[0][j] + ((x[0][j + 2] + x[1][j]) + x[1][j + 2]);
    c[j + 2] = y[0][j] + ((y[0][j + 2] + y[1][j]) + y[1][j + 2]);
  }
}

// 16 keys x 4 query rows, before the low query pieces (columns g + 4, two lanes away) are added: c[0..1] = key gid,
// c[2..3] = key gid + 8, columns 2t, 2t + 1.  Neighbouring MMAs go to different accumulators and do not wait for one another.
template <int BITS, int N>
__device__ __forceinline__ void score_block(const uint32_t (&w0)[Packed<BITS>::CW], const uint32_t (&w1)[Packed<BITS>::CW],
                                            const uint32_t (&bq)[8][N], const uint8_t* table, uint32_t lane_off, float (&c)[4]) {
  if constexpr (N == 2) {
    // per key one accumulator for each half of the coordinates
    float x[2][4] = {}, y[2][4] = {};
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      uint32_t e[4], f[4];
      key_operand<BITS>(w0, ks, table, lane_off, e);
      key_operand<BITS>(w1, ks, table, lane_off, f);
      mma_16816(x[ks & 1], e[0], e[1], e[2], e[3], bq[ks][0], bq[ks][1]);
      mma_16816(y[ks & 1], f[0], f[1], f[2], f[3], bq[ks][0], bq[ks][1]);
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      c[j] = (x[0][j] + x[1][j]) + (x[0][j + 2] + x[1][j + 2]);
      c[j + 2] = (y[0][j] + y[1][j]) + (y[0][j + 2] + y[1][j + 2]);
    }
  } else {
    float x[4] = {}, y[4] = {};
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      uint32_t e[4], f[4];
      entries4<BITS>(w0, ks, table, lane_off, e);
      entries4<BITS>(w1, ks, table, lane_off, f);
      mma_16816(x, e[0], f[0], e[1], f[1], bq[ks][0], bq[ks][1]);
      mma_16816(y, e[2], f[2], e[3], f[3], bq[ks][2], bq[ks][3]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) c[j] = x[j] + y[j];
  }
}

// grid: B * Hkv * nblk CTAs, each over keys_per_block keys of one KV head; stats as in the FP32 path:
// stats[(row * nblk + blk) * 2 + {0, 1}] = (max, sum of exp(l - max)) of the block's keys.
// Two CTAs per SM: three (80 registers) 49 us against 45 for the call below.
// 8 KV heads x 131072 4-bit keys, 32 query heads: the call, with projection and softmax, 59 us with a table entry per
// coordinate and three waves of blocks, 45 us as it is (kernel 48 -> 36 under ncu: 386 -> 245 instructions per 16 keys, issued
// 0.55 of the time).  8 KV heads x 65536 keys with 8 query rows per KV head: 42 -> 35 us.
//
// ROWS: query rows per pass over the keys.  With eight a lane finishes keys gid and gid + 8 for rows 2t, 2t + 1 and the
// look-ups of a key serve twice the rows; four rows put their low pieces into the other four columns instead.
template <int BITS, int ROWS>
__global__ void __launch_bounds__(kThreads, 2) k_score_mma(TqScoreJob job, const float* qrot, float* stats, int nblk,
                                                        int keys_per_block) {
  if (stats != nullptr) pdl_trigger();           // the softmax pass follows
  constexpr int G = Packed<BITS>::G;
  constexpr int CW = Packed<BITS>::CW;
  __shared__ __align__(128) uint8_t table[ByteTable<BITS>::kBytes];
  constexpr bool kEight = ROWS == 8;
  __shared__ float red_m[kWarps][ROWS], red_s[kWarps][ROWS];
  build_table<BITS, true>(table, job.codebook);
  const int blk = blockIdx.x % nblk;
  const int64_t bh = blockIdx.x / nblk;
  const int64_t b = bh / job.Hkv, hkv = bh % job.Hkv;
  const int rep = (int)(job.Hq / job.Hkv);
  const int R = rep * (int)job.Sq;
  const int64_t s_begin = (int64_t)blk * keys_per_block;
  const int n_keys = (int)min((int64_t)keys_per_block, job.Sk - s_begin);      // of this CTA; keys below count from s_begin
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gid = lane >> 2, t = lane & 3;
  const uint32_t lane_off = ByteTable<BITS>::lane_offset(lane);
  const int my = gid + (!kEight && t >= 2 ? 8 : 0);     // the (first) key of a block whose logits this lane finishes
  const uint8_t* keys = job.idx_bytes + (bh * job.Sk + s_begin) * G + t * Packed<BITS>::CB;
  const uint16_t* norms = job.norms + bh * job.Sk + s_begin;
  __syncthreads();
  auto global_row = [&](int r) -> int64_t {
    const int64_t hq = hkv * rep + r / job.Sq, sq = r % job.Sq;
    return (b * job.Hq + hq) * job.Sq + sq;
  };
  pdl_wait();                                    // the rotated queries come from the launch before
  for (int r0 = 0; r0 < R; r0 += ROWS) {
    uint32_t bq[8][kCoordWords<BITS> ? 4 : 2], bh[8][2], bl[8][2];        // four or eight rows: the others stay unused
    if constexpr (kEight) {
      const int r = r0 + gid;
      query_fragments8(qrot, r < R ? global_row(r) : 0, r < R, lane, bh, bl);
    } else {
      const int r = r0 + (gid & 3);
      query_fragments(qrot, r < R ? global_row(r) : 0, r < R, lane, bq);
    }
    // four rows: after the shuffle below this lane finishes ONE key (gid for t < 2, gid + 8 otherwise) and the
    // two query rows r0 + 2 (t & 1) + {0, 1}
    const int ra = r0 + 2 * (kEight ? t : t & 1);
    const bool ok_a = ra < R, ok_b = ra + 1 < R;
    float* out_a = job.logits + (ok_a ? global_row(ra) : 0) * job.Sk + s_begin;
    float* out_b = job.logits + (ok_b ? global_row(ra + 1) : 0) * job.Sk + s_begin;
    // running (max, sum of exp(l - max)) of the two rows over this lane's keys.  The maximum starts at the lowest finite
    // value, so that logits of -inf add exp(-inf) = 0; it moves about ln(n) times in n keys.
    float m_a = -FLT_MAX, s_a = 0.f, m_b = -FLT_MAX, s_b = 0.f;
    // the packed quarter rows and the norm of the NEXT block of 16 keys are in flight while this one is scored
    uint32_t w0[CW], w1[CW], n0[CW], n1[CW];
    uint32_t nv_bits = 0, nn_bits = 0;          // norm of key `my`; eight rows: that of the key 8 further in the high half
    auto fetch = [&](int kb, uint32_t (&a0)[CW], uint32_t (&a1)[CW], uint32_t& nb) {
      load_quarter<BITS>(keys + (int64_t)min(kb + gid, n_keys - 1) * G, 0, a0);
      load_quarter<BITS>(keys + (int64_t)min(kb + 8 + gid, n_keys - 1) * G, 0, a1);
      nb = __ldg(norms + min(kb + my, n_keys - 1));
      if constexpr (kEight) nb |= (uint32_t)__ldg(norms + min(kb + my + 8, n_keys - 1)) << 16;
    };
    auto finish_key = [&](int key, float ca, float cb, uint32_t nb) {
      if (key < n_keys) {
        const float nv = __half2float(__ushort_as_half((uint16_t)nb)) * job.scale;
        const float la = ca * nv, lb = cb * nv;
        if (ok_a) out_a[key] = la;
        if (ok_b) out_b[key] = lb;
        if (la > m_a) { s_a *= exp_neg(m_a - la); m_a = la; }
        if (lb > m_b) { s_b *= exp_neg(m_b - lb); m_b = lb; }
        s_a += exp_neg(la - m_a);
        s_b += exp_neg(lb - m_b);
      }
    };
    auto score = [&](const uint32_t (&a0)[CW], const uint32_t (&a1)[CW], int kb, uint32_t nb) {
      float c[4];
      if constexpr (kEight) {
        score_block8<BITS>(a0, a1, bh, bl, table, lane_off, c);
        finish_key(kb + my, c[0], c[1], nb & 0xFFFFu);
        finish_key(kb + my + 8, c[2], c[3], nb >> 16);
      } else {
        score_block<BITS>(a0, a1, bq, table, lane_off, c);
        // lane t ^ 2 holds the other query piece of the same rows and finishes the other key: each sends what the other needs
        const float xa = __shfl_xor_sync(0xffffffffu, t < 2 ? c[2] : c[0], 2), xb = __shfl_xor_sync(0xffffffffu, t < 2 ? c[3] : c[1], 2);
        finish_key(kb + my, (t < 2 ? c[0] : c[2]) + xa, (t < 2 ? c[1] : c[3]) + xb, nb);
      }
    };
    int kb = warp * 16;
    if (kb < n_keys) fetch(kb, w0, w1, nv_bits);
    for (; kb < n_keys; kb += 2 * kWarps * 16) {              // two blocks a round: the buffers swap without copies
      const int k1 = kb + kWarps * 16, k2 = k1 + kWarps * 16;
      if (k1 < n_keys) fetch(k1, n0, n1, nn_bits);
      score(w0, w1, kb, nv_bits);
      if (k1 < n_keys) {
        if (k2 < n_keys) fetch(k2, w0, w1, nv_bits);
        score(n0, n1, k1, nn_bits);
      }
    }
    if (stats != nullptr) {
      // lanes that share t (four rows: t & 1) share the two rows: fold over the other lane bits, then over the warps
#pragma unroll
      for (int o = kEight ? 4 : 2; o <= 16; o <<= 1) {
        const float m2 = __shfl_xor_sync(0xffffffffu, m_a, o), s2 = __shfl_xor_sync(0xffffffffu, s_a, o);
        stat_merge(m_a, s_a, m2, s2);
        const float m3 = __shfl_xor_sync(0xffffffffu, m_b, o), s3 = __shfl_xor_sync(0xffffffffu, s_b, o);
        stat_merge(m_b, s_b, m3, s3);
      }
      if (lane < ROWS / 2) {
        red_m[warp][2 * lane] = m_a; red_s[warp][2 * lane] = s_a;
        red_m[warp][2 * lane + 1] = m_b; red_s[warp][2 * lane + 1] = s_b;
      }
      __syncthreads();
      if (threadIdx.x < ROWS && r0 + (int)threadIdx.x < R) {
        float m = -INFINITY, s = 0.f;
        for (int wv = 0; wv < kWarps; ++wv) stat_merge(m, s, red_m[wv][threadIdx.x], red_s[wv][threadIdx.x]);
        const int64_t orow = global_row(r0 + threadIdx.x);
        stats[(orow * nblk + blk) * 2 + 0] = m;
        stats[(orow * nblk + blk) * 2 + 1] = s;
      }
      __syncthreads();
    }
  }
}

// ---------------------------------------------------------------------------------------------------
// Decode attention on packed keys AND packed values:  out = softmax(scale * q k_hat^T) v_hat  without
// reconstructing either.  With v_hat_s = norm_s * (c_v[idx_s] Pi_v), the weighted sum is taken in the
// rotated domain,  acc[g][j] = sum_s p[g][s] * norm_v[s] * c_v[idx_v[s][j]],  and Pi_v is applied once at the
// end (k_decode_finish).  Per block of 16 keys a warp
//   1. scores the keys as above (score_block), applies norm and scale;
//   2. keeps a running maximum and sum per query row (online softmax) and rescales its accumulators when
//      the maximum moves;
//   3. forms P' = exp(l - max) * norm_v as fp16 pieces, columns [P'_hi rows 0..3 | P'_lo rows 0..3], and
//      turns the accumulator-layout block (16 keys x 8 columns) into the B operand of the next product with
//      two 8x8 transposes (movmatrix);
//   4. accumulates  acc^T (16 coordinates x 8 columns) += V^T (16 coordinates x 16 keys) P'  for 8 blocks of
//      coordinates, value pieces hi and lo: thread (gid, t) assembles the value operand for keys
//      2t, 2t+1, 2t+8, 2t+9 and its own 16 coordinates 16 gid .. 16 gid + 15 from the packed value rows.
// Each CTA covers keys_per_block keys of one (batch, KV head) and writes one partial (max, sum, acc) per
// query row; k_decode_finish merges the partials, the 16-bit window tokens and applies Pi_v.

template <int BITS>
struct PackedV {
  static constexpr int IPB = 8 / BITS;
  static constexpr int G = kDimA / IPB;         // packed bytes per value row
  static constexpr int CB = G / 8;              // bytes per thread and key: an eighth of a row = 16 coordinates
  static constexpr int CW = CB >= 4 ? CB / 4 : 1;
};

// the eighth `e` of one packed value row (16 coordinates): 2 (1-bit), 4, 8 or 16 bytes
template <int BITS>
__device__ __forceinline__ void load_eighth(const uint8_t* row, int e, uint32_t (&w)[PackedV<BITS>::CW]) {
  constexpr int CB = PackedV<BITS>::CB;
  const uint8_t* p = row + e * CB;
  if constexpr (CB == 2) {
    w[0] = __ldg(reinterpret_cast<const uint16_t*>(p));
  } else if constexpr (CB == 4) {
    w[0] = __ldg(reinterpret_cast<const uint32_t*>(p));
  } else if constexpr (CB == 8) {
    const uint2 v = __ldg(reinterpret_cast<const uint2*>(p));
    w[0] = v.x; w[1] = v.y;
  } else {
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
    w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
  }
}

__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t x) {
  uint32_t y;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}

struct DecodeParams {
  const float* qrot;          // (rows, 128) rotated queries
  const uint8_t* k_idx; const uint16_t* k_norms;
  const uint8_t* v_idx; const uint16_t* v_norms;
  const float* k_codebook; const float* v_codebook;
  float* part;                // [rows][nblk][130]: max, sum, acc[128] (rotated domain, coordinates in natural order)
  int64_t B, Hq, Sq, Hkv, Sk;
  float scale;
  int nblk, keys_per_block;
};
constexpr int kPartStride = 130;

template <int KBITS, int VBITS>
__global__ void __launch_bounds__(kThreads, 2) k_decode_attn(DecodeParams P) {
  pdl_trigger();
  constexpr int GK = Packed<KBITS>::G, KW = Packed<KBITS>::CW;
  constexpr int GV = PackedV<VBITS>::G, VW = PackedV<VBITS>::CW;
  extern __shared__ __align__(128) uint8_t tables[];
  uint8_t* table_k = tables;
  uint8_t* table_v = tables + ByteTable<KBITS>::kBytes;
  __shared__ float sm_m[kWarps][kRows], sm_l[kWarps][kRows];
  __shared__ float sm_acc[kWarps][kRows][kDimA];          // 16 KB
  build_table<KBITS, true>(table_k, P.k_codebook);
  build_table<VBITS, false>(table_v, P.v_codebook);
  const int blk = blockIdx.x % P.nblk;
  const int64_t bh = blockIdx.x / P.nblk;
  const int64_t b = bh / P.Hkv, hkv = bh % P.Hkv;
  const int rep = (int)(P.Hq / P.Hkv);
  const int R = rep * (int)P.Sq;
  // this CTA's keys count from s_begin; a lane's own parts of the rows
  const int64_t s_begin = (int64_t)blk * P.keys_per_block;
  const int n_keys = (int)min((int64_t)P.keys_per_block, P.Sk - s_begin);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gid = lane >> 2, t = lane & 3;
  const uint8_t* keys = P.k_idx + (bh * P.Sk + s_begin) * GK + t * Packed<KBITS>::CB;
  const uint8_t* vals = P.v_idx + (bh * P.Sk + s_begin) * GV + gid * PackedV<VBITS>::CB;
  const uint16_t* k_norms = P.k_norms + bh * P.Sk + s_begin;
  const uint16_t* v_norms = P.v_norms + bh * P.Sk + s_begin;
  const uint32_t off_k = ByteTable<KBITS>::lane_offset(lane), off_v = ByteTable<VBITS>::lane_offset(lane);
  __syncthreads();
  auto global_row = [&](int r) -> int64_t {
    const int64_t hq = hkv * rep + r / P.Sq, sq = r % P.Sq;
    return (b * P.Hq + hq) * P.Sq + sq;
  };
  pdl_wait();                                    // the rotated queries come from the launch before
  for (int r0 = 0; r0 < R; r0 += kRows) {
    uint32_t bq[8][2];
    {
      const int r = r0 + (gid & 3);
      query_fragments(P.qrot, r < R ? global_row(r) : 0, r < R, lane, bq);
    }
    // this lane's two query rows: r0 + 2 (t & 1) + {0, 1}; lanes t and t ^ 2 hold the same rows, the first as
    // the high pieces of P' (columns 0..3), the second as the low pieces (columns 4..7)
    float run_m[2] = {-INFINITY, -INFINITY}, run_l[2] = {0.f, 0.f};
    float acc[8][4];
#pragma unroll
    for (int mb = 0; mb < 8; ++mb) acc[mb][0] = acc[mb][1] = acc[mb][2] = acc[mb][3] = 0.f;
    // Two blocks of 16 keys a round where their rows fit the registers: one maximum, one rescaling and two independent
    // chains of look-ups and products.  The next round's lines are fetched into L1 meanwhile; keeping them in registers took
    // the room of the second block, and K6/V4 and wider spilled (131072 tokens x 8 heads, with projection and finish: K4/V2
    // 84 -> 70 us, K4/V4 90 -> 79, K8/V8 153 -> 104; two blocks with 4-bit values spill: 83).
    constexpr int NB = 4 * KW + 8 * VW <= 24 ? 2 : 1;
    uint32_t w0[NB][KW], w1[NB][KW], vw[NB][4][VW];
    uint32_t kn_bits[NB], vn_bits[NB];            // norms of keys gid (low half) and gid + 8 (high half)
    for (int kb = warp * 16 * NB; kb < n_keys; kb += kWarps * 16 * NB) {
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        const int k0 = kb + 16 * nb;
        const int c_lo = k0 + gid < n_keys ? k0 + gid : 0, c_hi = k0 + 8 + gid < n_keys ? k0 + 8 + gid : 0;
        load_quarter<KBITS>(keys + (uint32_t)(c_lo * GK), 0, w0[nb]);
        load_quarter<KBITS>(keys + (uint32_t)(c_hi * GK), 0, w1[nb]);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int key = k0 + 2 * t + (q & 1) + 8 * (q >> 1);           // keys 2t, 2t+1, 2t+8, 2t+9
          load_eighth<VBITS>(vals + (uint32_t)((key < n_keys ? key : 0) * GV), 0, vw[nb][q]);
        }
        kn_bits[nb] = (uint32_t)__ldg(k_norms + c_lo) | ((uint32_t)__ldg(k_norms + c_hi) << 16);
        vn_bits[nb] = (uint32_t)__ldg(v_norms + c_lo) | ((uint32_t)__ldg(v_norms + c_hi) << 16);
      }
      {
        const int row = kb + kWarps * 16 * NB + (lane & (16 * NB - 1));
        if (row < n_keys) {
          if (NB == 2 || lane < 16) asm volatile("prefetch.global.L1 [%0];" ::"l"(keys - t * Packed<KBITS>::CB + (uint32_t)(row * GK)));
          if (NB == 2 || lane >= 16) asm volatile("prefetch.global.L1 [%0];" ::"l"(vals - gid * PackedV<VBITS>::CB + (uint32_t)(row * GV)));
          if (lane < 2) asm volatile("prefetch.global.L1 [%0];" ::"l"((lane ? v_norms : k_norms) + row));
        }
      }
      float l[NB][4];
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        float c[4];
        score_block<KBITS>(w0[nb], w1[nb], bq, table_k, off_k, c);
#pragma unroll
        for (int j = 0; j < 4; ++j) c[j] += __shfl_xor_sync(0xffffffffu, c[j], 2);       // lanes t and t ^ 2 both hold the full sums
        // logits of keys gid (c[0], c[1]) and gid + 8 (c[2], c[3]) for this lane's two rows
        const bool in_lo = kb + 16 * nb + gid < n_keys, in_hi = kb + 16 * nb + 8 + gid < n_keys;
        const float nk_lo = __half2float(__ushort_as_half((uint16_t)(kn_bits[nb] & 0xFFFFu))) * P.scale;
        const float nk_hi = __half2float(__ushort_as_half((uint16_t)(kn_bits[nb] >> 16))) * P.scale;
        l[nb][0] = in_lo ? c[0] * nk_lo : -INFINITY; l[nb][1] = in_lo ? c[1] * nk_lo : -INFINITY;
        l[nb][2] = in_hi ? c[2] * nk_hi : -INFINITY; l[nb][3] = in_hi ? c[3] * nk_hi : -INFINITY;
      }
      // maximum per row over the round's keys (lanes that differ in gid)
      float bm[2] = {fmaxf(l[0][0], l[0][2]), fmaxf(l[0][1], l[0][3])};
#pragma unroll
      for (int nb = 1; nb < NB; ++nb) {
        bm[0] = fmaxf(bm[0], fmaxf(l[nb][0], l[nb][2]));
        bm[1] = fmaxf(bm[1], fmaxf(l[nb][1], l[nb][3]));
      }
#pragma unroll
      for (int o = 4; o <= 16; o <<= 1) {
        bm[0] = fmaxf(bm[0], __shfl_xor_sync(0xffffffffu, bm[0], o));
        bm[1] = fmaxf(bm[1], __shfl_xor_sync(0xffffffffu, bm[1], o));
      }
      float alpha[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float nm = fmaxf(run_m[j], bm[j]);              // the round holds at least one valid key: finite
        alpha[j] = run_m[j] == -INFINITY ? 0.f : exp_neg(run_m[j] - nm);
        run_m[j] = nm;
        run_l[j] *= alpha[j];
      }
      // rescale the accumulators when a maximum moved (columns 2t, 2t+1 are this lane's two rows in both halves)
      if (__any_sync(0xffffffffu, alpha[0] != 1.f || alpha[1] != 1.f)) {
#pragma unroll
        for (int mb = 0; mb < 8; ++mb) {
          acc[mb][0] *= alpha[0]; acc[mb][1] *= alpha[1]; acc[mb][2] *= alpha[0]; acc[mb][3] *= alpha[1];
        }
      }
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        float p[4];
        p[0] = exp_neg(l[nb][0] - run_m[0]); p[1] = exp_neg(l[nb][1] - run_m[1]);
        p[2] = exp_neg(l[nb][2] - run_m[0]); p[3] = exp_neg(l[nb][3] - run_m[1]);
        // row sums: every (row, key) pair is counted by exactly one of the lanes t and t ^ 2
        run_l[0] += t < 2 ? p[0] : p[2];
        run_l[1] += t < 2 ? p[1] : p[3];
        // P' = p * norm_v as fp16 pieces; this lane contributes the high (t < 2) or low (t >= 2) piece
        const float nv_lo = __half2float(__ushort_as_half((uint16_t)(vn_bits[nb] & 0xFFFFu)));
        const float nv_hi = __half2float(__ushort_as_half((uint16_t)(vn_bits[nb] >> 16)));
        uint32_t x0, x1;
        {
          uint32_t h, lo2;
          split2(p[0] * nv_lo, p[1] * nv_lo, h, lo2);
          x0 = t < 2 ? h : lo2;
          split2(p[2] * nv_hi, p[3] * nv_hi, h, lo2);
          x1 = t < 2 ? h : lo2;
        }
        const uint32_t pb0 = movmatrix_trans(x0);               // keys 2t, 2t+1  x column gid
        const uint32_t pb1 = movmatrix_trans(x1);               // keys 2t+8, 2t+9 x column gid
        const uint32_t p0 = __byte_perm(pb0, 0u, 0x1010), p1 = __byte_perm(pb0, 0u, 0x3232);     // each value in both halves
        const uint32_t p2 = __byte_perm(pb1, 0u, 0x1010), p3 = __byte_perm(pb1, 0u, 0x3232);
        // acc^T += V^T P' for 8 blocks of 16 coordinates; this thread's rows are coordinates 16 gid + 2 mb + {0, 1}
#pragma unroll
        for (int m2 = 0; m2 < 4; ++m2) {
          uint32_t e[4][4];
#pragma unroll
          for (int q = 0; q < 4; ++q) entries4<VBITS>(vw[nb][q], m2, table_v, off_v, e[q]);
          // an entry is the operand's two neighbouring k, the pieces of one value; rows gid, gid + 8 are the two coordinates,
          // the k pairs t, t + 4 the keys 2t, 2t + 1 (first MMA) and 2t + 8, 2t + 9 (second)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            mma_16816(acc[2 * m2 + h], e[0][2 * h], e[0][2 * h + 1], e[1][2 * h], e[1][2 * h + 1], p0, p1);
            mma_16816(acc[2 * m2 + h], e[2][2 * h], e[2][2 * h + 1], e[3][2 * h], e[3][2 * h + 1], p2, p3);
          }
        }
      }
    }
    // ---- fold the warp: sums over the lanes that share (t & 1), pieces hi + lo two lanes apart
#pragma unroll
    for (int o = 2; o <= 16; o <<= 1) {
      run_l[0] += __shfl_xor_sync(0xffffffffu, run_l[0], o);
      run_l[1] += __shfl_xor_sync(0xffffffffu, run_l[1], o);
    }
#pragma unroll
    for (int mb = 0; mb < 8; ++mb)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[mb][j] += __shfl_xor_sync(0xffffffffu, acc[mb][j], 2);
    // run_m is already uniform over gid (every block maximum was); lanes t < 2 publish rows 2t, 2t + 1
    if (lane < 2) {
      sm_m[warp][2 * lane] = run_m[0]; sm_m[warp][2 * lane + 1] = run_m[1];
      sm_l[warp][2 * lane] = run_l[0]; sm_l[warp][2 * lane + 1] = run_l[1];
    }
    if (t < 2) {
#pragma unroll
      for (int mb = 0; mb < 8; ++mb) {
        // acc[mb][0..1]: coordinate 16 gid + 2 mb, rows 2t, 2t+1;  acc[mb][2..3]: coordinate 16 gid + 2 mb + 1
        sm_acc[warp][2 * t][16 * gid + 2 * mb] = acc[mb][0];
        sm_acc[warp][2 * t + 1][16 * gid + 2 * mb] = acc[mb][1];
        sm_acc[warp][2 * t][16 * gid + 2 * mb + 1] = acc[mb][2];
        sm_acc[warp][2 * t + 1][16 * gid + 2 * mb + 1] = acc[mb][3];
      }
    }
    __syncthreads();
    // ---- fold the CTA's warps and write the partial of this block of keys
    for (int idx = threadIdx.x; idx < kRows * kDimA; idx += kThreads) {
      const int rr = idx / kDimA, j = idx % kDimA;
      if (r0 + rr >= R) continue;
      float m = -INFINITY;
      for (int wv = 0; wv < kWarps; ++wv) m = fmaxf(m, sm_m[wv][rr]);
      float a = 0.f, lsum = 0.f;
      for (int wv = 0; wv < kWarps; ++wv) {
        const float wm = sm_m[wv][rr];
        if (wm != -INFINITY) {
          const float f = __expf(wm - m);
          a += sm_acc[wv][rr][j] * f;
          lsum += sm_l[wv][rr] * f;
        }
      }
      float* dst = P.part + (global_row(r0 + rr) * P.nblk + blk) * kPartStride;
      dst[2 + j] = a;
      if (j == 0) { dst[0] = m; dst[1] = lsum; }
    }
    __syncthreads();
  }
}

// One CTA per query row: merge the partials of the packed tokens, add the 16-bit window tokens (their logits use
// the UNROTATED query), normalise, and rotate back:  out = (acc / L) Pi_v + sum_w p_w v_w / L.
// Nothing here is large (a few hundred KB for all rows); what it costs is the number of memory latencies in a row.
// So every phase spreads its loads over all 16 warps, a few independent 16-byte loads per thread, and the rows of
// Pi_v are fetched before the first barrier.
// 32 query rows, 16 partials and 128 window tokens each: 59 us as one warp per 32 tokens and a loop over rows of Pi_v, 9 us so.
struct FinishParams {
  const void* q; int q_dtype;
  const float* part; int nblk;
  const float* v_rotation;    // Pi_v (128 x 128, row-major): out = acc @ Pi_v
  const void* k_window; const void* v_window; int window_dtype;
  int64_t W, ws_b, ws_h, ws_s;
  int64_t B, Hq, Sq, Hkv, Sk;
  float scale;
  float* out;
};
constexpr int kFinWarps = 16;
constexpr int kFinThreads = 32 * kFinWarps;

// N consecutive elements as fp32; VEC: the address is a multiple of 16 bytes (of 8 for four 16-bit elements)
template <int DT, int N, bool VEC>
__device__ __forceinline__ void load_run(const void* p, int64_t off, float (&v)[N]) {
  if constexpr (!VEC) {
#pragma unroll
    for (int e = 0; e < N; ++e) v[e] = load_elem<DT>(p, off + e);
  } else if constexpr (DT == TQ_F32) {
#pragma unroll
    for (int e = 0; e < N; e += 4) {
      const float4 f = __ldg(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p) + off + e));
      v[e] = f.x; v[e + 1] = f.y; v[e + 2] = f.z; v[e + 3] = f.w;
    }
  } else {
    uint32_t w[N / 2];
    const uint16_t* src = reinterpret_cast<const uint16_t*>(p) + off;
    if constexpr (N == 4) {
      const uint2 u = __ldg(reinterpret_cast<const uint2*>(src));
      w[0] = u.x; w[1] = u.y;
    } else {
#pragma unroll
      for (int e = 0; e < N / 8; ++e) {
        const uint4 u = __ldg(reinterpret_cast<const uint4*>(src) + e);
        w[4 * e] = u.x; w[4 * e + 1] = u.y; w[4 * e + 2] = u.z; w[4 * e + 3] = u.w;
      }
    }
#pragma unroll
    for (int e = 0; e < N / 2; ++e) {
      if constexpr (DT == TQ_F16) {
        const __half2 h = *reinterpret_cast<const __half2*>(&w[e]);
        v[2 * e] = __low2float(h); v[2 * e + 1] = __high2float(h);
      } else {
        v[2 * e] = __uint_as_float(w[e] << 16); v[2 * e + 1] = __uint_as_float(w[e] & 0xFFFF0000u);
      }
    }
  }
}

template <int QDT, int WDT, bool VEC>
__global__ void __launch_bounds__(kFinThreads) k_decode_finish(FinishParams F) {
  __shared__ float sh_q[kDimA], sh_acc[kDimA], sh_m[kFinWarps], sh_l[kFinWarps];
  __shared__ __align__(16) float sh_part[kFinWarps][kDimA];
  extern __shared__ float sh_w[];                 // window logits, then probabilities: W floats
  const int64_t row = blockIdx.x;
  const int64_t hq = (row / F.Sq) % F.Hq, b = row / (F.Sq * F.Hq);
  const int64_t hkv = hq / (F.Hq / F.Hkv);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // rows 8 warp .. 8 warp + 7 of Pi_v, columns 4 lane .. 4 lane + 3
  constexpr int kRot = kDimA / kFinWarps;
  float rot[kRot][4];
#pragma unroll
  for (int u = 0; u < kRot; ++u)
    load_run<TQ_F32, 4, VEC>(F.v_rotation, (int64_t)(kRot * warp + u) * kDimA + 4 * lane, rot[u]);
  if (tid < kDimA) sh_q[tid] = load_elem<QDT>(F.q, row * kDimA + tid);
  __syncthreads();
  // window logits: eight lanes per token, 16 coordinates each
  const int64_t wbase = b * F.ws_b + hkv * F.ws_h;
  float m = -INFINITY;
  const int sub = tid & 7;
#pragma unroll 2
  for (int64_t w0 = 0; w0 < F.W; w0 += kFinThreads / 8) {
    const int64_t w = w0 + (tid >> 3);
    float d = 0.f;
    if (w < F.W) {
      float kv[16];
      load_run<WDT, 16, VEC>(F.k_window, wbase + w * F.ws_s + 16 * sub, kv);
#pragma unroll
      for (int e = 0; e < 16; ++e) d = fmaf(sh_q[16 * sub + e], kv[e], d);
    }
    d += __shfl_xor_sync(0xffffffffu, d, 4);
    d += __shfl_xor_sync(0xffffffffu, d, 2);
    d += __shfl_xor_sync(0xffffffffu, d, 1);
    d *= F.scale;
    if (w < F.W) {
      if (sub == 0) sh_w[w] = d;
      m = fmaxf(m, d);
    }
  }
  // global maximum over the partials (of the launch before) and the window
  pdl_wait();
  const float* parts = F.part + row * F.nblk * kPartStride;
  if (F.Sk > 0)
    for (int i = tid; i < F.nblk; i += kFinThreads) m = fmaxf(m, parts[(int64_t)i * kPartStride]);
  m = warp_max(m);
  if (lane == 0) sh_m[warp] = m;
  __syncthreads();
  m = sh_m[0];
#pragma unroll
  for (int u = 1; u < kFinWarps; ++u) m = fmaxf(m, sh_m[u]);
  // window probabilities, and the rotated-domain sums of this warp's partials (lane = four coordinates)
  float lsum = 0.f;
  for (int64_t w = tid; w < F.W; w += kFinThreads) {
    const float pw = __expf(sh_w[w] - m);
    sh_w[w] = pw;
    lsum += pw;
  }
  lsum = warp_sum(lsum);                          // of the warp's window tokens, the same in every lane
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  if (F.Sk > 0) {
    constexpr int kBatch = 4;                     // partials in flight per warp
    for (int i0 = warp; i0 < F.nblk; i0 += kBatch * kFinWarps) {
      float2 ms[kBatch], lo[kBatch], hi[kBatch];
#pragma unroll
      for (int u = 0; u < kBatch; ++u) {
        const int i = i0 + u * kFinWarps;
        const float2* pp = reinterpret_cast<const float2*>(parts + (int64_t)(i < F.nblk ? i : i0) * kPartStride);
        ms[u] = pp[0];
        if (i >= F.nblk) ms[u].x = -INFINITY;
        lo[u] = pp[1 + 2 * lane];
        hi[u] = pp[2 + 2 * lane];
      }
#pragma unroll
      for (int u = 0; u < kBatch; ++u) {
        if (ms[u].x != -INFINITY) {
          const float f = __expf(ms[u].x - m);
          acc[0] += lo[u].x * f; acc[1] += lo[u].y * f; acc[2] += hi[u].x * f; acc[3] += hi[u].y * f;
          lsum += ms[u].y * f;
        }
      }
    }
  }
  *reinterpret_cast<float4*>(&sh_part[warp][4 * lane]) = make_float4(acc[0], acc[1], acc[2], acc[3]);
  if (lane == 0) sh_l[warp] = lsum;
  __syncthreads();
  if (tid < kDimA) {
    float a = 0.f;
#pragma unroll
    for (int u = 0; u < kFinWarps; ++u) a += sh_part[u][tid];
    sh_acc[tid] = a;
  }
  // this warp's window tokens while the sums settle: o += p_w v_w
  float o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
  for (int64_t w = warp; w < F.W; w += kFinWarps) {
    float vv[4];
    load_run<WDT, 4, VEC>(F.v_window, wbase + w * F.ws_s + 4 * lane, vv);
    const float pw = sh_w[w];
#pragma unroll
    for (int e = 0; e < 4; ++e) o[e] = fmaf(pw, vv[e], o[e]);
  }
  __syncthreads();
  // o += acc @ Pi_v over this warp's eight rows of Pi_v
#pragma unroll
  for (int u = 0; u < kRot; ++u) {
    const float a = sh_acc[kRot * warp + u];
#pragma unroll
    for (int e = 0; e < 4; ++e) o[e] = fmaf(a, rot[u][e], o[e]);
  }
  *reinterpret_cast<float4*>(&sh_part[warp][4 * lane]) = make_float4(o[0], o[1], o[2], o[3]);
  __syncthreads();
  if (tid < kDimA) {
    float sum = 0.f, total = 0.f;
#pragma unroll
    for (int u = 0; u < kFinWarps; ++u) { sum += sh_part[u][tid]; total += sh_l[u]; }
    F.out[row * kDimA + tid] = sum / total;
  }
}

}  // namespace

size_t decode_attention_workspace(int64_t B, int64_t Hq, int64_t Sq, int64_t Sk, int keys_per_block) {
  const int64_t rows = B * Hq * Sq;
  const int64_t nblk = Sk > 0 ? (Sk + keys_per_block - 1) / keys_per_block : 1;
  size_t q = ((size_t)rows * kDimA * sizeof(float) + 255) / 256 * 256;
  return q + (size_t)rows * nblk * kPartStride * sizeof(float);
}

template <int KB, int VB>
static int launch_decode_kv(const DecodeParams& P, unsigned blocks, cudaStream_t st) {
  constexpr int smem = (int)(ByteTable<KB>::kBytes + ByteTable<VB>::kBytes);
  const cudaError_t e = cudaFuncSetAttribute(k_decode_attn<KB, VB>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return refused(e);
  launch_after(k_decode_attn<KB, VB>, dim3(blocks), dim3(kThreads), (size_t)smem, st, P);
  return check_launch();
}

template <int KB>
static int launch_decode_v(const DecodeParams& P, int vbits, unsigned blocks, cudaStream_t st) {
  switch (vbits) {
    case 1: return launch_decode_kv<KB, 1>(P, blocks, st);
    case 2: return launch_decode_kv<KB, 2>(P, blocks, st);
    case 3: return launch_decode_kv<KB, 3>(P, blocks, st);
    case 4: return launch_decode_kv<KB, 4>(P, blocks, st);
    case 5: return launch_decode_kv<KB, 5>(P, blocks, st);
    case 6: return launch_decode_kv<KB, 6>(P, blocks, st);
    case 7: return launch_decode_kv<KB, 7>(P, blocks, st);
    default: return launch_decode_kv<KB, 8>(P, blocks, st);
  }
}

static int device_sm_count() {
  static std::atomic<int> cached[64] = {};
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 148;
  if (dev >= 0 && dev < 64 && (n = cached[dev].load()) > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
  if (dev >= 0 && dev < 64) cached[dev].store(n);
  return n;
}

// Blocks of keys per (batch, KV head): fewer keys per CTA fill the chip sooner, and every CTA pays a fixed cost
// (tables, query pieces, first loads, folding its warps) worth about kFixedKeys keys of its loop.  The count with the
// smallest  waves x (keys per CTA + kFixedKeys)  is taken, at most `most` (what the scratch holds) and never blocks
// of fewer than min_keys keys.
// Decode attention, 8 KV heads x 32640 tokens, K4/V2: 36 us as 128 CTAs of 2048 keys with one CTA per SM, 30 us as 296 CTAs with
// two.
constexpr int kDecodeMinKeys = 256;               // two rounds of the CTA's eight warps
constexpr int kScoreMinKeys = 128;                // one
static int key_blocks(int64_t units, int64_t Sk, int min_keys, int64_t most, int slots) {
  constexpr int64_t kFixedKeys = 256;
  int64_t cap = (Sk + min_keys - 1) / min_keys;
  if (cap > most) cap = most;
  if (cap > 1024) cap = 1024;
  int64_t best = 1, best_cost = -1;
  for (int64_t nblk = 1; nblk <= cap; ++nblk) {
    const int64_t kpb = ((Sk + nblk - 1) / nblk + 15) / 16 * 16;
    const int64_t cost = ((units * nblk + slots - 1) / slots) * (kpb + kFixedKeys);
    if (best_cost < 0 || cost < best_cost) { best = nblk; best_cost = cost; }
  }
  return (int)best;
}

// Scratch the entry point asks for: room for the blocks of one full wave (two CTAs per SM) at one unit, as long as
// the partials stay within 16 MB; never less than decode_attention_workspace(), which every caller brings.
size_t decode_attention_workspace_wanted(int64_t B, int64_t Hq, int64_t Sq, int64_t Sk) {
  const size_t least = decode_attention_workspace(B, Hq, Sq, Sk, 2048);
  const int64_t rows = B * Hq * Sq;
  if (rows <= 0 || Sk <= 0) return least;
  int64_t nblk = (Sk + kDecodeMinKeys - 1) / kDecodeMinKeys;
  if (nblk > 320) nblk = 320;
  const int64_t fit = ((int64_t)16 << 20) / (rows * kPartStride * (int64_t)sizeof(float));
  if (nblk > fit) nblk = fit;
  const size_t q = ((size_t)rows * kDimA * sizeof(float) + 255) / 256 * 256;
  const size_t want = q + (size_t)rows * (nblk > 0 ? nblk : 1) * kPartStride * sizeof(float);
  return want > least ? want : least;
}

int decode_attention(const TqDecodeAttnJob& job, cudaStream_t st) {
  const int64_t rows = job.B * job.Hq * job.Sq;
  int nblk = 1, kKeysPerBlock = 16;
  if (job.Sk > 0) {
    const size_t q = ((size_t)rows * kDimA * sizeof(float) + 255) / 256 * 256;
    const int64_t most = (int64_t)((job.workspace_bytes - q) / ((size_t)rows * kPartStride * sizeof(float)));
    nblk = key_blocks(job.B * job.Hkv, job.Sk, kDecodeMinKeys, most, 2 * device_sm_count());
    kKeysPerBlock = (int)(((job.Sk + nblk - 1) / nblk + 15) / 16 * 16);
    nblk = (int)((job.Sk + kKeysPerBlock - 1) / kKeysPerBlock);
  }
  float* qrot = reinterpret_cast<float*>(job.workspace);
  const size_t qbytes = ((size_t)rows * kDimA * sizeof(float) + 255) / 256 * 256;
  float* part = reinterpret_cast<float*>(reinterpret_cast<char*>(job.workspace) + qbytes);
  FinishParams F;
  F.q = job.q; F.q_dtype = job.q_dtype;
  F.part = part; F.nblk = nblk;
  F.v_rotation = job.v_rotation;
  F.k_window = job.k_window; F.v_window = job.v_window; F.window_dtype = job.window_dtype;
  F.W = job.k_window != nullptr ? job.W : 0;
  F.ws_b = job.wstride_b; F.ws_h = job.wstride_h; F.ws_s = job.wstride_s;
  F.B = job.B; F.Hq = job.Hq; F.Sq = job.Sq; F.Hkv = job.Hkv; F.Sk = job.Sk;
  F.scale = job.scale;
  F.out = job.out;
  const size_t smem = (size_t)(F.W > 0 ? F.W : 1) * sizeof(float);
  const int wdt = F.W > 0 ? job.window_dtype : TQ_F16;
  // 16-byte loads where every row of the windows and of Pi_v starts on such a boundary
  const int64_t per16 = wdt == TQ_F32 ? 4 : 8;
  const bool vec = (((uintptr_t)F.k_window | (uintptr_t)F.v_window | (uintptr_t)F.v_rotation) & 15u) == 0 &&
                   (F.ws_b % per16 == 0 && F.ws_h % per16 == 0 && F.ws_s % per16 == 0);
  void (*finish)(FinishParams) = nullptr;
#define TQ_FIN(QD, WD) finish = vec ? k_decode_finish<QD, WD, true> : k_decode_finish<QD, WD, false>
  if (job.q_dtype == TQ_F32) { if (wdt == TQ_F16) TQ_FIN(TQ_F32, TQ_F16); else if (wdt == TQ_BF16) TQ_FIN(TQ_F32, TQ_BF16); else TQ_FIN(TQ_F32, TQ_F32); }
  else if (job.q_dtype == TQ_F16) { if (wdt == TQ_F16) TQ_FIN(TQ_F16, TQ_F16); else if (wdt == TQ_BF16) TQ_FIN(TQ_F16, TQ_BF16); else TQ_FIN(TQ_F16, TQ_F32); }
  else { if (wdt == TQ_F16) TQ_FIN(TQ_BF16, TQ_F16); else if (wdt == TQ_BF16) TQ_FIN(TQ_BF16, TQ_BF16); else TQ_FIN(TQ_BF16, TQ_F32); }
#undef TQ_FIN
  if (smem > 36 * 1024) {                          // with its 10 KB of static shared memory past the default limit
    const cudaError_t e = cudaFuncSetAttribute(finish, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return refused(e);       // before the first launch: the attention kernel counts on this one
  }
  int rc = TQ_OK;
  if (job.Sk > 0) {
    rc = simt_project(job.q, job.q_dtype, rows, kDimA, job.k_rotation_t, kDimA, qrot, st, true);
    if (rc != TQ_OK) return rc;
    DecodeParams P;
    P.qrot = qrot;
    P.k_idx = job.k_idx; P.k_norms = job.k_norms; P.v_idx = job.v_idx; P.v_norms = job.v_norms;
    P.k_codebook = job.k_codebook; P.v_codebook = job.v_codebook;
    P.part = part;
    P.B = job.B; P.Hq = job.Hq; P.Sq = job.Sq; P.Hkv = job.Hkv; P.Sk = job.Sk;
    P.scale = job.scale;
    P.nblk = nblk; P.keys_per_block = kKeysPerBlock;
    const unsigned blocks = (unsigned)(job.B * job.Hkv * nblk);
    switch (job.key_bits) {
      case 1: rc = launch_decode_v<1>(P, job.value_bits, blocks, st); break;
      case 2: rc = launch_decode_v<2>(P, job.value_bits, blocks, st); break;
      case 3: rc = launch_decode_v<3>(P, job.value_bits, blocks, st); break;
      case 4: rc = launch_decode_v<4>(P, job.value_bits, blocks, st); break;
      case 5: rc = launch_decode_v<5>(P, job.value_bits, blocks, st); break;
      case 6: rc = launch_decode_v<6>(P, job.value_bits, blocks, st); break;
      case 7: rc = launch_decode_v<7>(P, job.value_bits, blocks, st); break;
      default: rc = launch_decode_v<8>(P, job.value_bits, blocks, st); break;
    }
    if (rc != TQ_OK) return rc;
  }
  if (job.Sk > 0) launch_after(finish, dim3((unsigned)rows), dim3(kFinThreads), smem, st, F);
  else finish<<<(unsigned)rows, kFinThreads, smem, st>>>(F);
  return check_launch();
}

bool mma_score_eligible(const TqScoreJob& job) {
  if (force_simt()) return false;
  return job.D == kDimA && (((uintptr_t)job.idx_bytes) & 15u) == 0 && (((uintptr_t)job.norms) & 1u) == 0;
}

// Keys per CTA of the call below, `most` blocks at most.  131072 4-bit keys x 8 heads with four query rows: 888 CTAs of 1184 keys (three
// waves) 59 us a call, one wave of 296 45 us (with the byte tables).  Blocks of 1024 keys and more, as it was, left a short call on few SMs.
int mma_score_keys_per_block(const TqScoreJob& job, int64_t most) {
  const int nblk = key_blocks(job.B * job.Hkv, job.Sk, kScoreMinKeys, most, 2 * device_sm_count());      // two CTAs per SM
  return (int)(((job.Sk + nblk - 1) / nblk + 15) / 16 * 16);
}

// logits (and the per-block softmax partials when stats != NULL) for a job whose queries are already rotated
int mma_score_packed(const TqScoreJob& job, const float* qrot, float* stats, int nblk, int keys_per_block, cudaStream_t st) {
  const int64_t blocks = job.B * job.Hkv * nblk;
  const bool eight = job.Hq / job.Hkv * job.Sq > 4;      // more than four query rows per KV head: one pass serves eight
  auto go = [&](auto bits) {
    constexpr int BITS = decltype(bits)::value;
    if (eight) launch_after(k_score_mma<BITS, 8>, dim3((unsigned)blocks), dim3(kThreads), 0, st, job, qrot, stats, nblk, keys_per_block);
    else launch_after(k_score_mma<BITS, 4>, dim3((unsigned)blocks), dim3(kThreads), 0, st, job, qrot, stats, nblk, keys_per_block);
  };
  switch (job.bits) {
    case 1: go(std::integral_constant<int, 1>{}); break;
    case 2: go(std::integral_constant<int, 2>{}); break;
    case 3: go(std::integral_constant<int, 3>{}); break;
    case 4: go(std::integral_constant<int, 4>{}); break;
    case 5: go(std::integral_constant<int, 5>{}); break;
    case 6: go(std::integral_constant<int, 6>{}); break;
    case 7: go(std::integral_constant<int, 7>{}); break;
    default: go(std::integral_constant<int, 8>{}); break;
  }
  return check_launch();
}

}  // namespace tq
