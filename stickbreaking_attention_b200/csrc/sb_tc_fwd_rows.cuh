// The forward's row arithmetic, shared by the forward kernels: one query row per thread, scores read from tensor
// memory in chunks of 16 columns, P written back to tensor memory as the A operand of O += P V.
#pragma once

#include "sb_tc_common.cuh"

namespace sb {

namespace fwd256 {
constexpr int kBN = 64;                       // keys per sub-tile
constexpr int kPBytes = kBM * kBN * 2;        // a 128 x 64 16-bit tile (the staging unit of the O epilogue)
// P, the 16-bit A operand of O += P V, goes to the second MMA through tensor memory: the row threads write their
// packed row into columns 32..63 of the very S slot they have just read (key k of the step in column 32 + k / 2;
// the chunks are read last column first, so every column written has been read before), and the MMA takes its A
// operand from there.  The next S MMA into that slot is issued by the same thread after this P V MMA, and MMAs of
// one thread execute in order.
constexpr uint32_t kPCol = 32;
}  // namespace fwd256

using fwd256::kPCol;

// A row's sum of log2(1 + e) over the keys of the earlier sub-tiles, as an unevaluated pair of floats: exact for as long as
// the sum's terms span less than 48 bits, and a few FMA-pipe operations on the way to the next sub-tile's start value where
// fp64 takes a conversion, an addition and a conversion back.
struct LogSum {
  float hi = 0.f, lo = 0.f;
  __device__ __forceinline__ void add(float x) {   // Knuth's two-sum
    const float s = hi + x, b = s - hi;
    lo += (hi - (s - b)) + (x - b);
    hi = s;
  }
  __device__ __forceinline__ float stick() const { return ex2(-(hi + lo)); }   // product of (1 - beta) over those keys
  __device__ __forceinline__ double value() const { return (double)hi + (double)lo; }
};

// One row, 16 consecutive key columns of a 64-key sub-tile, last column first.  key0: index inside the sequence of
// the chunk's first column; row: index of this query row.
//   x = z log2(e), clamped at 30;  e = 2^x;  t = 1 + e;  1 - beta = 1 / t;  beta = e / t
//   p_j = beta_j * (product of (1 - beta) over the allowed keys after j) = e_j * (product of 1 / t over j and after)
// R carries that product over everything after the current column.  Four columns share one reciprocal and one
// logarithm of t0 t1 t2 t3; the four inclusive products follow from R, that reciprocal and partial products with
// five multiplications, and beta itself is never formed.
// The log-space sums are added up in the order the backward uses -- the groups of a chunk from the last to the first, the
// chunks of a sub-tile from the first to the last, which is the way it walks: the two agree bit for bit, so that
// the backward may start at any sub-tile from the fp64 sum of the sub-tiles after it (see `tile_start`).
template <bool kFp16, bool kMasked>
__device__ __forceinline__ void fwd256_row_chunk(const uint32_t (&v)[16], int c0, int key0, int row, int ac,
                                                 float scale2, float &R, float &logsum, uint32_t tmem_p) {
  float pr[16];
  logsum = 0.f;
  const float2 sc = make_float2(scale2, scale2), one = make_float2(1.f, 1.f);
#pragma unroll
  for (int g = 3; g >= 0; --g) {   // four columns at a time, last group first; independent work in packed pairs
    const float2 x01 = mul2(make_float2(__uint_as_float(v[4 * g]), __uint_as_float(v[4 * g + 1])), sc);
    const float2 x23 = mul2(make_float2(__uint_as_float(v[4 * g + 2]), __uint_as_float(v[4 * g + 3])), sc);
    float2 e01 = make_float2(ex2(fminf(x01.x, 30.f)), ex2(fminf(x01.y, 30.f)));
    float2 e23 = make_float2(ex2(fminf(x23.x, 30.f)), ex2(fminf(x23.y, 30.f)));
    float2 t01 = add2(e01, one), t23 = add2(e23, one);
    if (kMasked) {
      const int key = key0 + 4 * g, lim = row + ac;
      if (!(key < lim)) { e01.x = 0.f; t01.x = 1.f; }
      if (!(key + 1 < lim)) { e01.y = 0.f; t01.y = 1.f; }
      if (!(key + 2 < lim)) { e23.x = 0.f; t23.x = 1.f; }
      if (!(key + 3 < lim)) { e23.y = 0.f; t23.y = 1.f; }
    }
    const float p01 = t01.x * t01.y, p23 = t23.x * t23.y;
    const float prod = p01 * p23;
    const float rp = rcp(prod);
    logsum += lg2(prod);
    const float rb = R * (rp * p01);          // R / (t2 t3): inclusive product at column 2
    const float r3 = rb * t23.x;              // R / t3
    R *= rp;                                  // R / (t0 t1 t2 t3): at column 0, and the carry into the next group
    const float r1 = R * t01.x;               // R / (t1 t2 t3)
    const float2 q01 = mul2(e01, make_float2(R, r1));
    const float2 q23 = mul2(e23, make_float2(rb, r3));
    pr[4 * g] = q01.x;
    pr[4 * g + 1] = q01.y;
    pr[4 * g + 2] = q23.x;
    pr[4 * g + 3] = q23.y;
  }
  uint32_t w[8];   // 16 keys = 8 packed columns of this row's lane
  pack_row_chunk16<kFp16>(pr, w);
  tmem_st8(tmem_p + (c0 >> 1), w);
}

// P of 32 key columns (from column c0 of the sub-tile on) set to zero without looking at the scores.
__device__ __forceinline__ void fwd256_zero_pair(int c0, uint32_t tmem_p) {
  const uint32_t z[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
  tmem_st8(tmem_p + (c0 >> 1), z);
  tmem_st8(tmem_p + (c0 >> 1) + 8, z);
}

__device__ __forceinline__ void fwd256_zero_row(uint32_t tmem_p) {
  fwd256_zero_pair(0, tmem_p);
  fwd256_zero_pair(32, tmem_p);
}

// One row of a 64-key sub-tile whose P is known to be exactly zero: only the log-space sum is formed, with the same
// operations in the same order as fwd256_row_chunk, so that it is the same number bit for bit.
__device__ __forceinline__ void fwd256_logsum_chunk(const uint32_t (&v)[16], float scale2, float &logsum) {
  const float2 sc = make_float2(scale2, scale2), one = make_float2(1.f, 1.f);
  logsum = 0.f;
#pragma unroll
  for (int g = 3; g >= 0; --g) {
    const float2 x01 = mul2(make_float2(__uint_as_float(v[4 * g]), __uint_as_float(v[4 * g + 1])), sc);
    const float2 x23 = mul2(make_float2(__uint_as_float(v[4 * g + 2]), __uint_as_float(v[4 * g + 3])), sc);
    const float2 e01 = make_float2(ex2(fminf(x01.x, 30.f)), ex2(fminf(x01.y, 30.f)));
    const float2 e23 = make_float2(ex2(fminf(x23.x, 30.f)), ex2(fminf(x23.y, 30.f)));
    const float2 t01 = add2(e01, one), t23 = add2(e23, one);
    const float p01 = t01.x * t01.y, p23 = t23.x * t23.y;
    logsum += lg2(p01 * p23);
  }
}
// (The chunk of columns 48..63 has been requested into va.)
__device__ __forceinline__ void fwd256_logsum_pass(uint32_t ts, float scale2, float &logsum, uint32_t tmem_p, uint32_t (&va)[16]) {
  uint32_t vb[16];
  float l3 = 0.f, l2 = 0.f;   // the chunks of the upper pair
#pragma unroll 1
  for (int pair = 1; pair >= 0; --pair) {
    float la, lb;
    tmem_wait_ld_regs(va);
    tmem_ld16(ts + pair * 32, vb);
    fwd256_logsum_chunk(va, scale2, la);
    tmem_wait_ld_regs(vb);
    if (pair == 1) tmem_ld16(ts + 16, va);
    fwd256_logsum_chunk(vb, scale2, lb);
    logsum = ((lb + la) + l2) + l3;
    l3 = la;
    l2 = lb;
  }
  // P is written last: its columns alias scores that have all been read by now
  fwd256_zero_row(tmem_p);
}

// One row of a 64-key sub-tile.  In a masked sub-tile the columns from (last row of this warp) + ac on are masked for
// every row of the warp (its 32 rows are consecutive and 32-aligned): such 32-column halves are not computed at all,
// their P is zero and R and logsum stay as they are -- 6 of the 16 (warp, half) pairs of a diagonal 128 x 128 tile.
// An unmasked sub-tile whose P is exactly zero for all rows of the warp that exist (their product has underflowed) only
// sums its logs (skip_zero).  drop_zero: it does nothing instead and returns true, log_rem is to cover the keys up to here.
template <bool kFp16, bool kMasked>
__device__ __forceinline__ bool fwd256_row_pass(uint32_t ts, int key0, int row, int ac, float scale2, const LogSum &sum,
                                                float &logsum, uint32_t tmem_p, bool exists, bool skip_zero = false, bool drop_zero = false) {
  float R;
  uint32_t va[16], vb[16];
  int hi = 1;   // last 32-column half with an allowed key
  if (kMasked) {
    const int span = (row | 31) + ac - key0;   // the warp's rows may attend to columns [0, span) of this sub-tile
    hi = span > 32 ? 1 : (span > 0 ? 0 : -1);
    if (hi < 1) fwd256_zero_pair(32, tmem_p);
    if (hi < 0) {
      fwd256_zero_pair(0, tmem_p);
      return false;
    }
    tmem_ld16(ts + hi * 32 + 16, va);
    R = sum.stick();
  } else {
    tmem_ld16(ts + 48, va);
    R = sum.stick();   // (under the load's latency; the registers it fills must not cross a branch)
    const bool zero = skip_zero && __all_sync(0xffffffffu, !exists || R == 0.f);
    tmem_wait_ld_regs(va);
    if (zero) {
      // The product over the keys after this sub-tile has underflowed to exactly 0 for all rows of the warp: every p of
      // the sub-tile is e * 0 = 0 (e is finite: its exponent is clamped).
      if (drop_zero) return true;
      fwd256_logsum_pass(ts, scale2, logsum, tmem_p, va);
      return false;
    }
  }
  float l3 = 0.f, l2 = 0.f;   // log sums of the upper pair of chunks
#pragma unroll 1
  for (int pair = hi; pair >= 0; --pair) {
    float la, lb;
    tmem_wait_ld_regs(va);
    tmem_ld16(ts + pair * 32, vb);
    fwd256_row_chunk<kFp16, kMasked>(va, pair * 32 + 16, key0 + pair * 32 + 16, row, ac, scale2, R, la, tmem_p);
    tmem_wait_ld_regs(vb);
    if (pair == 1) tmem_ld16(ts + 16, va);
    fwd256_row_chunk<kFp16, kMasked>(vb, pair * 32, key0 + pair * 32, row, ac, scale2, R, lb, tmem_p);
    logsum = ((lb + la) + l2) + l3;
    l3 = la;
    l2 = lb;
  }
  return false;
}

// ---- stopping early ------------------------------------------------------------------------------------------------
// A row warp is through once the product R has underflowed to exactly 0 for all its rows: no earlier key can add anything
// to O or rem.  From then on it only writes zeros for P, its log sum stays what it is, and the key it got to is recorded
// for the backward.  Each of a query tile's four warps publishes the step it was through at; from the step on in which all
// four are, the tile's MMA issuer leaves P V out (P is zero), and it stops before the next step that it has not issued the
// scores of yet and tells the rows with the word that accompanies every step's scores.  Where exactly it stops depends on
// timing, what is stored does not: not even where a value of V behind the last warp's stop is not finite (0 times it would
// be NaN).  Rows that never finish pay nothing: the vote is the one the row pass takes anyway to skip its arithmetic, and the
// issuer's look is a 16-byte read.  It looks between the rows' word that P is there and P V (from the third step on: a tile's
// first row has no keys in its own tile and loses at most 30 bits per key), and for the stop once P V is out: with that look
// ahead of the wait for P the forward of 8 x 2048 x 16 heads N(0, 1) takes 82.5 us instead of 79.2.
constexpr int kStepStop = -1;
// No stop with fewer than three sub-tiles to go: what is left costs about as much as stopping and restarting the stream.
__device__ __forceinline__ bool may_stop_before(int sub_tile) { return sub_tile >= 2; }
struct alignas(16) EarlyStop {                // shared memory, one per query tile
  int through[4];                             // per row warp: the last step it was through at (counted over all items), plus one
  int word[2];                                // per S slot: K/V stage of the step, or kStepStop (read where it can matter)
  int stopped;                                // item + 1: the tile wants no more keys of this item
};
__device__ __forceinline__ void publish_through(volatile EarlyStop &e, int warp, int step) { e.through[warp] = step + 1; }
// Whether all four warps were through by step `u` of the item whose steps count from `first` on.
__device__ __forceinline__ bool all_through(const volatile EarlyStop &e, int first, int u) {
  uint32_t a, b, c, d;
  asm volatile("ld.volatile.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(a), "=r"(b), "=r"(c), "=r"(d)
               : "r"(smem_u32(const_cast<const int *>(&e.through[0])))
               : "memory");
  const uint32_t t = (uint32_t)first + 1u;   // entries of earlier items are smaller and wrap around
  return max(max(a - t, b - t), max(c - t, d - t)) <= (uint32_t)u;
}

}  // namespace sb
