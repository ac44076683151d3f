// Tensor-core backward kernels for bf16 / fp16 tensors (reference counterpart: _backward_one_row,
// sb_varlen_bwd.py:297-481, which accumulates dK/dV across blocks under a global spin lock).
//
// Two kernels per call, no atomics, no locks, fixed summation order:
//   dq kernel (tc_bwd_dq3_kernel)   query-stationary, 128 query rows per block.  Walks the keys 0 -> diagonal in
//               64-key sub-tiles; per step S = Q K^T and dP = dO V^T go to TMEM, one thread per query row recomputes
//               A and dz = G - beta * C with the log-space suffix sum (a pair of floats across tiles, started from
//               the saved fp64 log_rem) and the prefix sum C of G carried in registers, writes dz to TMEM in 16 bits, and
//               dQ += dz K accumulates in TMEM.  It leaves for the second kernel either its A and dz tiles
//               (stored-tiles mode) or, every 32 keys, the two carried values R1 and S2 (small-workspace mode).
//   dK/dV kernel  key-stationary, one 128-key tile per block, query tiles diagonal -> end.
//               tc_bwd_dkv5_kernel: dK += dz^T Q and dV += A^T dO as plain GEMMs over the stored tiles.
//               tc_bwd_dkv4_kernel: repeats the row pass of each tile from the recorded R1/S2 first.
// Head sizes below 128 run the same code: TMA zero-fills the columns past head_dim.  All waits are bounded.
#include "sb_tc_common.cuh"

namespace sb {

// One row, 16 consecutive key columns.  s: raw q.k accumulators, dp: <dO_i, v_j>.
//   x = z log2(e), clamped at 30;  e = 2^x;  t = 1 + e;  1 - beta = 1 / t;  beta = e / t
//   A_j = beta_j * W_j,  W_j = product of (1 - beta) over the allowed keys after j up to the diagonal
//       = e_j * (product of 1 / t over j and the allowed keys after it)
//   G = A (dP - dR);  C = gpre + inclusive prefix of G;  dz = G - beta C
// Three sweeps over the 16 columns, all in registers: (1) e, beta and, per group of four columns, one reciprocal
// and one logarithm of t0 t1 t2 t3, which gives the log-space sum through the end of the chunk; (2) last group to
// first: the product is seeded with 2^(r1 + that sum) -- the largest value it takes in the chunk, so it only
// underflows where A rounds to zero anyway -- shrinks by the group's reciprocal per group, and the four inclusive
// products inside a group come from partial reciprocals sweep 1 already has; (3) first group to last: the prefix
// sum of G, carried per group, and dz.  About 1.6 transcendentals per score (ex2, rcp / 4, lg2 / 4, ex2 / 16).
// kMasked tiles (the diagonal one, or one with rows past the sequence end) zero what is not allowed.
// The chunk is kept to 16 columns so that the unrolled code of all variants stays inside the instruction cache.
// mc0: key index of the first column inside the 128-key tile (for the diagonal mask).
// kSkip (unmasked chunks only): where the product of (1 - beta) at the END of the chunk -- its largest value in
// the chunk -- has underflowed to exactly 0 and the prefix of G is still exactly 0, for all 32 rows of the warp, every
// A, G and dz of the chunk is exactly 0 (e, the reciprocals and dP - dR are finite): the log-space sum is formed with the same
// operations as otherwise, and sweep 3 (in the recomputing dK/dV kernel sweep 2 as well) is left out.
// Packed pairs (two fp32 per instruction) are used where a pair sits in adjacent registers anyway -- accumulator columns and
// what is computed column by column from them.  Products across columns stay scalar: pairing their operands up costs as many
// register moves as the packed instruction saves.
struct BwdExp {                    // what follows from a chunk's scores alone
  float2 e01[4], e23[4];           // e
  float2 be01[4], be23[4];         // beta
  float rpg[4], i23[4], ri1[4], ri3[4];   // per group: 1 / t0 t1 t2 t3, 1 / t2 t3, 1 / t1, 1 / t3
  float log;                       // log2 of the product of t, added up like the forward's (see fwd256_row_chunk): the two agree bit for bit
};

// Sweep 1.
template <bool kMasked>
__device__ __forceinline__ void bwd_chunk_exp(const uint32_t (&s)[16], int mc0, int limit, float scale2, BwdExp &c) {
  const float2 sc = make_float2(scale2, scale2), one = make_float2(1.f, 1.f);
  c.log = 0.f;
#pragma unroll
  for (int g = 3; g >= 0; --g) {
    const float2 x01 = mul2(make_float2(__uint_as_float(s[4 * g]), __uint_as_float(s[4 * g + 1])), sc);
    const float2 x23 = mul2(make_float2(__uint_as_float(s[4 * g + 2]), __uint_as_float(s[4 * g + 3])), sc);
    float2 e01 = make_float2(ex2(fminf(x01.x, 30.f)), ex2(fminf(x01.y, 30.f)));
    float2 e23 = make_float2(ex2(fminf(x23.x, 30.f)), ex2(fminf(x23.y, 30.f)));
    float2 t01 = add2(e01, one), t23 = add2(e23, one);
    if (kMasked) {
      const int col = mc0 + 4 * g;
      if (!(col < limit)) { e01.x = 0.f; t01.x = 1.f; }
      if (!(col + 1 < limit)) { e01.y = 0.f; t01.y = 1.f; }
      if (!(col + 2 < limit)) { e23.x = 0.f; t23.x = 1.f; }
      if (!(col + 3 < limit)) { e23.y = 0.f; t23.y = 1.f; }
    }
    const float p01 = t01.x * t01.y, p23 = t23.x * t23.y, prod = p01 * p23;
    c.log += lg2(prod);
    const float rp = rcp(prod);
    const float i01 = rp * p23;                 // 1 / t0 t1
    c.i23[g] = rp * p01;                        // 1 / t2 t3
    const float2 ri01 = make_float2(i01 * t01.y, i01 * t01.x);
    const float2 ri23 = make_float2(c.i23[g] * t23.y, c.i23[g] * t23.x);
    c.e01[g] = e01;
    c.e23[g] = e23;
    c.be01[g] = mul2(e01, ri01);
    c.be23[g] = mul2(e23, ri23);
    c.rpg[g] = rp;
    c.ri1[g] = ri01.y;
    c.ri3[g] = ri23.y;
  }
}

// Sweep 2.  wend: the product of (1 - beta) over everything after the chunk.  pa: A.
__device__ __forceinline__ void bwd_chunk_products(const BwdExp &c, float wend, float (&pa)[16]) {
#pragma unroll
  for (int g = 3; g >= 0; --g) {
    const float2 w23 = make_float2(wend * c.i23[g], wend * c.ri3[g]);   // inclusive products at columns 2, 3
    wend *= c.rpg[g];                                                    // at column 0 = after the previous group
    const float2 w01 = make_float2(wend, w23.x * c.ri1[g]);
    const float2 a01 = mul2(c.e01[g], w01);
    const float2 a23 = mul2(c.e23[g], w23);
    pa[4 * g] = a01.x;
    pa[4 * g + 1] = a01.y;
    pa[4 * g + 2] = a23.x;
    pa[4 * g + 3] = a23.y;
  }
}

// Sweep 3.  On entry `gs` is the sum of G between gpre and the chunk; pz: dz.
template <bool kMasked>
__device__ __forceinline__ void bwd_chunk_dz(const BwdExp &c, const uint32_t (&dp)[16], int mc0, int limit, float gpre, float dr, float &gs,
                                             float (&pa)[16], float (&pz)[16]) {
  const float2 ndr = make_float2(-dr, -dr);
  float cb = gpre + gs, csum = 0.f;   // C before the group; the chunk's own sum of G
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    float2 g01 = mul2(make_float2(pa[4 * g], pa[4 * g + 1]),
                      add2(make_float2(__uint_as_float(dp[4 * g]), __uint_as_float(dp[4 * g + 1])), ndr));
    float2 g23 = mul2(make_float2(pa[4 * g + 2], pa[4 * g + 3]),
                      add2(make_float2(__uint_as_float(dp[4 * g + 2]), __uint_as_float(dp[4 * g + 3])), ndr));
    if (kMasked) {   // rows past the sequence end carry arbitrary values: select, do not rely on 0 * x
      const int col = mc0 + 4 * g;
      if (!(col < limit)) { g01.x = 0.f; pa[4 * g] = 0.f; }
      if (!(col + 1 < limit)) { g01.y = 0.f; pa[4 * g + 1] = 0.f; }
      if (!(col + 2 < limit)) { g23.x = 0.f; pa[4 * g + 2] = 0.f; }
      if (!(col + 3 < limit)) { g23.y = 0.f; pa[4 * g + 3] = 0.f; }
    }
    const float t1 = g01.x + g01.y, t23 = g23.x + g23.y;
    const float tg = t1 + t23;
    const float c0v = cb + g01.x, c1v = cb + t1;
    const float c2v = c1v + g23.x;
    cb += tg;
    csum += tg;
    pz[4 * g] = fmaf(-c.be01[g].x, c0v, g01.x);
    pz[4 * g + 1] = fmaf(-c.be01[g].y, c1v, g01.y);
    pz[4 * g + 2] = fmaf(-c.be23[g].x, c2v, g23.x);
    pz[4 * g + 3] = fmaf(-c.be23[g].y, cb, g23.y);
    if (kMasked) {
#pragma unroll
      for (int i = 0; i < 4; ++i) pz[4 * g + i] = limit >= 0 ? pz[4 * g + i] : 0.f;
    }
  }
  gs += csum;
}

// columns (tile-local key indices) below the limit are allowed: one compare per column, no branches
__device__ __forceinline__ int chunk_limit(bool row_valid, bool diag, int r, int ac) {
  return !row_valid ? -1 : (diag ? r + ac : 0x7fffffff);
}

// All three sweeps.  kSkip: see above.
template <bool kMasked, bool kSkip>
__device__ __forceinline__ void bwd_chunk(const uint32_t (&s)[16], const uint32_t (&dp)[16], int mc0, int limit, float scale2, float r1,
                                          float gpre, float dr, float &gs, float &logsum, float (&pa)[16], float (&pz)[16], bool may_skip) {
  BwdExp c;
  bwd_chunk_exp<kMasked>(s, mc0, limit, scale2, c);
  logsum += c.log;
  const float wend = ex2(r1 + logsum);
  if (kSkip && may_skip && __all_sync(0xffffffffu, wend == 0.f && gpre + gs == 0.f)) {
#pragma unroll
    for (int i = 0; i < 16; ++i) pa[i] = pz[i] = 0.f;
    return;
  }
  bwd_chunk_products(c, wend, pa);
  bwd_chunk_dz<kMasked>(c, dp, mc0, limit, gpre, dr, gs, pa, pz);
}

// What is recorded as R1 (a log2) where a row has not started: the product is 0, and so is all that follows from it.
constexpr float kNothingLeft = -1e6f;

namespace dq3 {
enum { bQ = 0, bG, bKFull, bKEmpty = bKFull + 3, bVFull = bKEmpty + 3, bVEmpty = bVFull + 2, bSFull = bVEmpty + 2, bDpFull, bDqFull, bSEmpty,
       bDpEmpty, bZFull, bNum = bZFull + 2 };
}  // namespace dq3
// One row of a 64-key sub-tile of the dq kernel, 16 columns at a time.  The loop's body is one chunk, about 330 instructions:
// straight code over more of them is fetched more slowly than it is issued.  The next chunk's scores are requested as soon as
// this one's are in use, dP under the products that do not need it; the S slot is handed back with a chunk and a half to go.
// dz goes to tensor memory (key k of the sub-tile in column tz + k / 2, two per column), at 128 columns over the dP columns
// that have been read by then.
// mc0: key index of the sub-tile's first column inside its 128-key tile (for the diagonal mask).  Returns false if a wait gave up.
// out: stored-tiles mode: this row's 64 values of A in the workspace, those of dz `off` elements further; otherwise this row's
// record of R1 at the sub-tile's first key, S2 `off` floats further, both again kBM floats further for the key 32 columns on.
template <bool kFp16, bool kMasked, bool kStored, bool kSkip>
__device__ __forceinline__ bool strip_row_pass(uint32_t ts, uint32_t tp, uint32_t tz, int u, int mc0, int limit, float scale2, float r1,
                                              float gpre, float dr, float &gs, float &logsum, uint32_t bars, void *out, long long off) {
  uint32_t s[16], d[16];
  bool ok = true;
  tmem_ld16(ts, s);
#pragma unroll 1
  for (int c0 = 0; c0 < 64; c0 += 16) {
    if (!kStored && c0 == 32) {   // the carried values after 32 of the 64 columns
      float *rec = reinterpret_cast<float *>(out) + kBM;
      rec[0] = r1 + logsum;
      rec[off] = gpre + gs;
    }
    BwdExp x;
    float pa[16], pz[16];
    tmem_wait_ld_regs(s);
    bwd_chunk_exp<kMasked>(s, mc0 + c0, limit, scale2, x);
    if (c0 == 0) {
      ok = mbar_wait(bars + 8u * dq3::bDpFull, u & 1);
      tc_fence_after();
    }
    tmem_ld16(ts + min(c0 + 16, 48), s);   // (the last time: not used)
    tmem_ld16(tp + c0, d);
    logsum += x.log;
    const float wend = ex2(r1 + logsum);
    const bool zero = kSkip && __all_sync(0xffffffffu, wend == 0.f && gpre + gs == 0.f);
    bwd_chunk_products(x, wend, pa);   // (not left out where `zero`: no branch while a tcgen05.ld is under way)
    tmem_wait_ld_regs(s, d);
    if (c0 >= 32) {   // the last columns of S (32: the chunk to come has them), then of dP are in registers
      tc_fence_before();
      __syncwarp();
      if ((threadIdx.x & 31) == 0) mbar_arrive(bars + 8u * (c0 == 32 ? dq3::bSEmpty : dq3::bDpEmpty));
    }
    if (zero) {   // (A is zero as it is: e is finite)
#pragma unroll
      for (int i = 0; i < 16; ++i) pz[i] = 0.f;
    } else {
      bwd_chunk_dz<kMasked>(x, d, mc0 + c0, limit, gpre, dr, gs, pa, pz);
    }
    uint32_t w[8];
    pack_row_chunk16<kFp16>(pz, w);
    tmem_st8(tz + (c0 >> 1), w);
    if constexpr (kStored) {
      unsigned short *row = reinterpret_cast<unsigned short *>(out) + c0;
      store_packed_global16(row + off, w);
      pack_row_chunk16<kFp16>(pa, w);
      store_packed_global16(row, w);
    }
  }
  return ok;
}

// The same for a sub-tile before the first key of the warp's rows: dz (and the stored A) are zeros, the scores are not read.
template <bool kStored>
__device__ __forceinline__ bool zero_strip_row(uint32_t tz, int u, uint32_t bars, void *out, long long off) {
  const uint32_t z[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
  const bool ok = mbar_wait(bars + 8u * dq3::bDpFull, u & 1);   // (every phase is followed; and dz may lie over dP)
  tc_fence_after();
#pragma unroll
  for (int c = 0; c < 64; c += 16) {
    tmem_st8(tz + (c >> 1), z);
    if constexpr (kStored) {
      unsigned short *row = reinterpret_cast<unsigned short *>(out) + c;
      store_packed_global16(row, z);
      store_packed_global16(row + off, z);
    }
  }
  if constexpr (!kStored) {
    float *rec = reinterpret_cast<float *>(out) + kBM;
    rec[0] = kNothingLeft;
    rec[off] = 0.f;
  }
  __syncwarp();
  if ((threadIdx.x & 31) == 0) {
    mbar_arrive(bars + 8u * dq3::bSEmpty);
    mbar_arrive(bars + 8u * dq3::bDpEmpty);
  }
  return ok;
}

// =======================================================================================================
// dq kernel: 128 query rows per CTA, two CTAs per SM
// =======================================================================================================
// A block owns one 128-row query tile and walks the 64-key K/V sub-tiles from the first key its rows reach to its diagonal.
// Per sub-tile: S = Q K^T and dP = dO V^T (128 x 64), the row pass (which, where the tiles are not stored, records R1/S2
// every 32 keys), then dQ += dz K with dz read from tensor memory.
//   warps 0-3  rows, one thread per query row;  warp 4  TMA;  warp 5  MMA issue;  warps 6, 7 fill their warpgroup up
// Two blocks share an SM -- half of its tensor memory, of its registers and, to the byte, of its shared memory each --, so
// that nothing ties the two tiles of an SM together: one's loads, first scores and epilogue run under the other's row passes.
// What bounds it: the MMAs (an instruction of 64 keys takes as long as one of 128, ~64 clk: 2500 clk per step of both tiles)
// and the row arithmetic (~2900), which overlap only in part, because S and dP fill what tensor memory dQ leaves and have a
// single slot each.  A block of 256 rows, its two tiles sharing the K/V stream and dz in shared memory, took (us, then now)
// 178 / 141 on 8 sequences of 2048 tokens x 16 heads N(0, 1), whose tiles visit two key tiles; 630 / 573 on 48 heads x 4096;
// 377 / 338 at 64 columns; 165 / 128 on 131072 tokens without the stored tiles.  One tile per SM with 128 keys per step needs
// half of the MMA time, but its lone row warp per scheduler makes less of the issue slots than two do: 145 / 622.
// TMEM columns: S 0, dP 64, dQ 128.  At 128 columns dz lies over the first half of dP, which the next dP MMA therefore
// overwrites behind this step's dQ; at 64 columns it has two tiles of its own (192, 224), so that the next S and dP both go
// ahead of dQ (dP of step t + 2 is issued behind dQ of step t: who has seen the one may overwrite what the other read).
namespace dq3 {
constexpr int kThreads = 256;
constexpr int kBN = 64;
constexpr int kKvBox = kBN * 64 * 2;           // 64 keys x 64 columns
constexpr uint32_t kCols = 256;
constexpr uint32_t tcS = 0, tcP = 64, tcDQ = 128;
template <int D>                               // head size rounded up to 64 or 128
struct Cfg {
  static constexpr int kBoxes = D / 64;
  static constexpr int kTileBytes = kBoxes * kBoxBytes;   // Q or dO tile
  static constexpr int kKvTile = kBoxes * kKvBox;         // K or V sub-tile
  static constexpr int kKStages = D == 64 ? 3 : 2;        // K is read twice, by S and a pass later by dQ, V once
  static constexpr int kVStages = D == 64 ? 2 : 1;
  static constexpr bool kOwnDz = D == 64;                 // dz has columns of its own: the next dP need not wait for dQ
  static constexpr uint32_t tcZ = kOwnDz ? 192 : tcP, kZToggle = kOwnDz ? 32 : 0;
  static constexpr int kSmem = 2 * kTileBytes + (kKStages + kVStages) * kKvTile + 1024;
  static_assert(2 * (kSmem + 1024) <= 233472, "two blocks per SM");
};
// What the rows need again after their loop, kept out of their registers meanwhile.
struct Shared {
  Ctl ctl;
  int first;     // the sub-tile in stage 0
  int h, hh, len, idx;
  long long tok0, boff;
};
static_assert(bNum * 8 + sizeof(Shared) <= 1024, "barriers and control words");
}  // namespace dq3

// d_rem + <d_out, v> of one row (g, v: its d_out and v), rounded like a caller's d_rem.  (Not inlined, and by value: see
// fill_rows.)
template <bool kFp16, typename T>
__device__ __noinline__ float fused_drem_row(const T *g, const T *v, int head_dim, float d_rem) {
  float s = 0.f;
#pragma unroll 2
  for (int x = 0; x < head_dim; x += 8) {
    float gx[8], vx[8], part = 0.f;
    load_row8<kFp16>(g + x, gx);
    load_row8<kFp16>(v + x, vx);
#pragma unroll
    for (int i = 0; i < 8; ++i) part = fmaf(gx[i], vx[i], part);
    s += part;
  }
  return to_f32<T>(from_f32<T>(s + d_rem));
}

template <int D, bool kFp16, bool kStored>
__global__ void __launch_bounds__(dq3::kThreads, 2)
tc_bwd_dq3_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                  const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_g,
                  const __grid_constant__ CUtensorMap tm_dq, const KParams p) {
  enter_kernel<false>();
  using namespace dq3;
  using C = Cfg<D>;
  constexpr int kTileBytes = C::kTileBytes, kKvTile = C::kKvTile, kKStages = C::kKStages, kVStages = C::kVStages, kBoxes = C::kBoxes;
  extern __shared__ __align__(1024) uint8_t smem_tiles[];   // (no byte is left to align it here)
  if (gated(p)) return;
  if (threadIdx.x == 0) trace_block(p, 0);
  const uint32_t sQ = smem_u32(smem_tiles);
  const uint32_t sG = sQ + kTileBytes;
  const uint32_t sK = sG + kTileBytes;
  const uint32_t sV = sK + kKStages * kKvTile;
  const uint32_t sBar = sV + kVStages * kKvTile;
  // the item table lies where the second K sub-tile goes, which is not asked for before the block's barrier
  static_assert(sizeof(SmallTable) <= kKvTile, "item table in a K stage");
  SmallTable &tb = *reinterpret_cast<SmallTable *>(smem_tiles + 2 * kTileBytes + kKvTile);
  bool refused;
  const long long covered = open_table(p, tb, refused);
  if (covered < p.tokens) fill_rows<typename std::conditional<kFp16, __half, __nv_bfloat16>::type>(p.dq, fill_job(p, covered, refused, blockIdx.x, gridDim.x));
  TileCoord c;
  int hh;
  if (refused || !decode_block(p, tb, true, c, hh)) return;
  const int I = c.idx;
  Shared *sh = reinterpret_cast<Shared *>(smem_tiles + (sBar - sQ) + bNum * 8);
  Ctl *ctl = &sh->ctl;
  volatile int *abort_flag = &ctl->abort;
  auto bar = [&](int i) { return sBar + 8u * i; };

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = p.head0 + hh;
  const int n_sub = (c.len + kBN - 1) / kBN;
  const int end = min(2 * I + 2, n_sub);       // sub-tiles 0 .. 2 I + 1 reach the tile's diagonal
  // the sub-tile the tile starts at (an even number: whole key tiles): earlier keys have weight exactly 0
  const int first = tile_first_key(p, c, h, I, kBM) / kBM * 2;
  const int n_steps = end - first;
  int tr_cur = 0;   // cursor of this thread's event-log lane (diagnostics)

  auto load_k = [&](int t) {
    const int st = t % kKStages;
    mbar_arrive_expect_tx(bar(bKFull + st), kKvTile);
    for (int kb = 0; kb < kBoxes; ++kb)
      tma_load_4d(sK + st * kKvTile + kb * kKvBox, &tm_k, bar(bKFull + st), kb * 64, (int)c.tok0 + (first + t) * kBN, h, (int)c.boff);
  };
  auto load_v = [&](int t) {
    const int st = t % kVStages;
    mbar_arrive_expect_tx(bar(bVFull + st), kKvTile);
    for (int kb = 0; kb < kBoxes; ++kb)
      tma_load_4d(sV + st * kKvTile + kb * kKvBox, &tm_v, bar(bVFull + st), kb * 64, (int)c.tok0 + (first + t) * kBN, h, (int)c.boff);
  };
  if (warp == 4 && lane == 0) {   // the first loads are on their way while the rest of the block gets ready
    for (int i = 0; i < bNum; ++i) mbar_init(bar(i), i >= bSEmpty ? 4 : 1);
    ctl->abort = 0;
    sh->first = first; sh->h = h; sh->hh = hh; sh->len = c.len; sh->idx = I;
    sh->tok0 = c.tok0; sh->boff = c.boff;
    fence_barrier_init();
    const int qrow = (int)c.tok0 + I * kBM;
    mbar_arrive_expect_tx(bar(bQ), kTileBytes);
    for (int kb = 0; kb < kBoxes; ++kb) tma_load_4d(sQ + kb * kBoxBytes, &tm_q, bar(bQ), kb * 64, qrow, h, (int)c.boff);
    load_k(0);
    mbar_arrive_expect_tx(bar(bG), kTileBytes);
    for (int kb = 0; kb < kBoxes; ++kb) tma_load_4d(sG + kb * kBoxBytes, &tm_g, bar(bG), kb * 64, qrow, h, (int)c.boff);
    load_v(0);
  }
  if (warp == 5) {
    tmem_alloc(smem_u32(&ctl->tmem_base), kCols);
    tmem_relinquish();
  }
  fence_proxy_async_smem();   // the item table's bytes are TMA's from here on
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = ctl->tmem_base;

  // The row warps take over registers the other warpgroup does not need (128 x 192 + 128 x 64 of the launch's 256 x 128).
  if (warp >= 4) {
  reg_dec<64>();
  if (warp == 4) {
    if (lane == 0) {
      for (int t = 1; t < n_steps; ++t) {
        if (t >= kKStages && !wait_or_abort(bar(bKEmpty + t % kKStages), ((t / kKStages) - 1) & 1, abort_flag, p, 510)) break;
        if (*abort_flag) break;
        load_k(t);
        if (t >= kVStages && !wait_or_abort(bar(bVEmpty + t % kVStages), ((t / kVStages) - 1) & 1, abort_flag, p, 511)) break;
        if (*abort_flag) break;
        load_v(t);
      }
    }
  } else if (warp == 5) {
    // ------------------------------------------------ MMA issuer
    if (lane == 0) {
      constexpr uint32_t idesc_s = idesc_f16(kBM, kBN, kFp16, false, false);
      constexpr uint32_t idesc_dq = idesc_f16(kBM, D, kFp16, false, true);
      bool ok = true;
      auto issue_s = [&](int t) {   // S = Q K^T
        const int st = t % kKStages;
        ok = ok && wait_or_abort(bar(bKFull + st), (t / kKStages) & 1, abort_flag, p, 521);
        if (!ok) return;
        tc_fence_after();
        mma_kmajor_kmajor<D, kBoxBytes, kKvBox>(tmem + tcS, sQ, sK + st * kKvTile, idesc_s, false);
        mma_commit(bar(bSFull));
      };
      auto issue_dp = [&](int t) {   // dP = dO V^T
        const int st = t % kVStages;
        ok = ok && wait_or_abort(bar(bVFull + st), (t / kVStages) & 1, abort_flag, p, 523);
        if (!ok) return;
        tc_fence_after();
        mma_kmajor_kmajor<D, kBoxBytes, kKvBox>(tmem + tcP, sG, sV + st * kKvTile, idesc_s, false);
        mma_commit(bar(bDpFull));
        mma_commit(bar(bVEmpty + st));
      };
      ok = wait_or_abort(bar(bQ), 0, abort_flag, p, 520);
      issue_s(0);
      ok = ok && wait_or_abort(bar(bG), 0, abort_flag, p, 524);
      issue_dp(0);
      for (int t = 0; ok && t < n_steps; ++t) {
        // the rows of step t have read their S (they are still computing): the next scores go first ...
        if (t + 1 < n_steps) {
          ok = wait_or_abort(bar(bSEmpty), t & 1, abort_flag, p, 526);
          trace_event(p, 1, tr_cur, 2, t + 1);
          issue_s(t + 1);
          if (C::kOwnDz) {
            ok = ok && wait_or_abort(bar(bDpEmpty), t & 1, abort_flag, p, 527);
            issue_dp(t + 1);
          }
          trace_event(p, 1, tr_cur, 3, t + 1);
        }
        // ... then, once its dz is written, this step's dQ += dz K (K sub-tile: 64 keys x (2 x 64) columns, MN-major)
        ok = ok && wait_or_abort(bar(bZFull + (t & 1)), (t >> 1) & 1, abort_flag, p, 522);
        if (!ok) break;
        trace_event(p, 1, tr_cur, 6, t);
        tc_fence_after();
        mma_tmem_mnmajor<kBN, kKvBox>(tmem + tcDQ, tmem + C::tcZ + (t & 1) * C::kZToggle, sK + (t % kKStages) * kKvTile, idesc_dq, t > 0);
        mma_commit(bar(bKEmpty + t % kKStages));
        // ... and, where dz lay over it, the next dP
        if (!C::kOwnDz && t + 1 < n_steps) issue_dp(t + 1);
        trace_event(p, 1, tr_cur, 7, t);
      }
      if (ok) mma_commit(bar(bDqFull));
    }
  }
  } else {
    reg_inc<192>();
    // ------------------------------------------------ rows: one thread per query row
    using T = typename std::conditional<kFp16, __half, __nv_bfloat16>::type;
    const int r = threadIdx.x;
    const uint32_t lane_off = (uint32_t)(warp * 32) << 16;
    const float scale2 = p.scale * kLog2e;
    const volatile Shared &item = *sh;
    const int row0 = I * kBM;
    const bool valid = row0 + r < c.len;
    const long long idx = (c.boff * p.heads + h) * p.tokens + c.tok0 + row0 + r;
    // sum of log2(1 - beta) over the keys from the current sub-tile on, as an unevaluated pair (see LogSum in the forward)
    float r1 = 0.f, r1_lo = 0.f, dr = 0.f, gpre = 0.f;
    if (valid) {
      const double total = p.log_rem[idx];
      r1 = (float)total;
      r1_lo = (float)(total - (double)r1);
      // out = o + rem * v: its gradient reaches rem through <d_out, v>.  (Formed here, the row of either comes from L2 while the
      // SM's other block works; a kernel of its own took 21 us for 16 heads x 16384 x 64.)
      if (p.d_rem != nullptr) dr = load_drem<T>(p, idx);
      if (p.drem_in_dq) {
        const long long tok = c.tok0 + row0 + r;
        dr = fused_drem_row<kFp16, T>(reinterpret_cast<const T *>(p.d_o.ptr) + c.boff * p.d_o.sb + (long long)h * p.d_o.sh + tok * p.d_o.st,
                                      reinterpret_cast<const T *>(p.v.ptr) + c.boff * p.v.sb + (long long)h * p.v.sh + tok * p.v.st, p.head_dim, dr);
      }
    }
    const uint32_t tS = tmem + tcS + lane_off, tP = tmem + tcP + lane_off, tZ = tmem + C::tcZ + lane_off;
    // this row's part of the workspace for sub-tile 0: A, or the boundary records [pair (I, J)][quarter of the key tile][row]
    const long long pair00 = kStored && p.pair_slot != nullptr
                                 ? p.pair_slot[(long long)h * p.tiles_cap + tile_id(p, c, I)]
                                 : (long long)(kStored ? 2 * hh : hh) * p.pairs_cap + c.pair0 + (long long)I * (I + 1) / 2;
    char *out = kStored ? reinterpret_cast<char *>(p.az + (pair00 * kBM + r) * kBM) : reinterpret_cast<char *>(p.bnd_r1 + pair00 * (4 * kBM) + r);
    const int u_diag = 2 * I, u_tail = c.len / kBN;   // a sub-tile with rows past the sequence is number u_tail
    // this warp's rows start at sub-tile u_warp (never, if they are past the sequence): before it, A and dz are zeros
    const int u_warp = row0 + (r & ~31) < c.len ? first_key(p, c, h, row0 + (r & ~31)) / kBN : 0x7fffffff;
    // Where the forward has said where each warp's rows start, hardly a chunk of zeros is left, and the test for them costs
    // every chunk a tenth of its instructions.
    const bool skip = p.tile_start == nullptr && !p.dense;
    // stored tiles: elements from A to dz; records: floats from R1 to S2
    const long long off = kStored ? p.pairs_cap * (kBM * kBM) : p.bnd_s2 - p.bnd_r1;
    bool ok = true;
    // One step: `pass` does the rows of sub-tile u, `dst` is its part of this row's workspace.  Zeros up to the warp's first
    // key, then full sub-tiles, then the diagonal: three loops, because what the kinds of step need would otherwise be kept in
    // registers for one another (see the forward's row loop).
    // u: 64-key sub-tile inside the sequence; the first one is even, so that phases follow from u alone
    int u = first;
    auto step = [&](auto pass, auto tail) {
      ok = wait_or_abort(bar(bSFull), u & 1, abort_flag, p, 530);
      if (!ok) return;
      if (r == 0) trace_event(p, 2, tr_cur, 4, u);
      tc_fence_after();
      void *dst = kStored ? out + ((long long)(u >> 1) * (kBM * kBM) + (u & 1) * kBN) * 2 : out + (long long)u * (2 * kBM * sizeof(float));
      if (!pass(dst)) {   // a bounded wait inside the pass gave up
        *abort_flag = 1;
        if (p.status != nullptr) { p.status[0] = SB_DEV_WAIT_TIMEOUT; p.status[1] = 531; }
        ok = false;
      }
      // the sequence ends inside this sub-tile: its dz columns behind the end are exact zeros, the K rows there are
      // not this sequence's (see zero_tile_rows) and are cleared before this step's dz K MMA is released
      if (decltype(tail)::value && u == u_tail) {
        zero_tile_rows(smem_tiles + (sK - sQ) + ((u - item.first) % kKStages) * kKvTile, item.len - u * kBN, kBN, kBoxes, kKvBox, r, kBM);
        fence_proxy_async_smem();
      }
      tmem_wait_st();
      tc_fence_before();          // this step's TMEM reads and its writes of dz are done before the slots are handed back
      __syncwarp();
      if (r == 0) trace_event(p, 2, tr_cur, 5, u);
      // (two barriers in turn: a warp whose dz is zeros may get to the next step's before another has got to this one's)
      if (lane == 0) mbar_arrive(bar(bZFull + (u & 1)));
    };
    auto record = [&](void *dst, float r1f) {
      if constexpr (!kStored) {
        reinterpret_cast<float *>(dst)[0] = r1f;
        reinterpret_cast<float *>(dst)[off] = gpre;
      }
    };
    auto carry = [&](float logsum, float gs) {   // r1 += logsum, gpre += gs
      const float sum = r1 + logsum, b = sum - r1;
      r1_lo += (r1 - (sum - b)) + (logsum - b);
      r1 = sum;
      gpre += gs;
    };
    using std::false_type; using std::true_type;
    for (; u < min(u_warp, end) && ok; ++u)
      step([&](void *dst) {
        record(dst, kNothingLeft);
        return zero_strip_row<kStored>(tZ + (u & 1) * C::kZToggle, u, sBar, dst, off);
      }, true_type());
    // rows past the sequence end must be zero in the stored tiles (the dK/dV GEMMs sum over all 128 query rows): the warp that
    // holds the end masks throughout
    const int u_full = kStored && row0 + (r | 31) >= c.len ? 0 : min(u_diag, end);
    if (!skip) {
      for (; u < u_full && ok; ++u)
        step([&](void *dst) {
          const float r1f = r1 + r1_lo;
          float gs = 0.f, logsum = 0.f;
          record(dst, r1f);
          const bool good = strip_row_pass<kFp16, false, kStored, false>(tS, tP, tZ + (u & 1) * C::kZToggle, u, 0, 0, scale2, r1f, gpre, dr, gs, logsum, sBar, dst, off);
          carry(logsum, gs);
          return good;
        }, false_type());
    } else {
      for (; u < u_full && ok; ++u)
        step([&](void *dst) {
          const float r1f = r1 + r1_lo;
          float gs = 0.f, logsum = 0.f;
          record(dst, r1f);
          const bool good = strip_row_pass<kFp16, false, kStored, true>(tS, tP, tZ + (u & 1) * C::kZToggle, u, 0, 0, scale2, r1f, gpre, dr, gs, logsum, sBar, dst, off);
          carry(logsum, gs);
          return good;
        }, false_type());
    }
    for (; u < end && ok; ++u)
      step([&](void *dst) {
        const bool on_diag = u >= u_diag;
        const float r1f = r1 + r1_lo;
        float gs = 0.f, logsum = 0.f;
        record(dst, r1f);
        const bool good = strip_row_pass<kFp16, true, kStored, false>(tS, tP, tZ + (u & 1) * C::kZToggle, u, on_diag ? (u - u_diag) * kBN : 0,
                                                                      chunk_limit(valid || !kStored, on_diag, r, p.attend_current), scale2, r1f,
                                                                      gpre, dr, gs, logsum, sBar, dst, off);
        carry(logsum, gs);
        return good;
      }, true_type());
    if (ok) ok = wait_or_abort(bar(bDqFull), 0, abort_flag, p, 532);
    if (ok) {
      tc_fence_after();
      const uint32_t t_acc = tmem + tcDQ + lane_off;
      const long long tok0 = item.tok0, boff = item.boff;
      const int hd = item.h, tile_row0 = item.idx * kBM;
      if (tile_row0 + kBM <= item.len) {
        // full tile: through Q's memory (every MMA is done), one TMA store per warp and 64 columns -- full lines instead of
        // 16 bytes per thread and row
        stage_acc_rows<D, kFp16>(t_acc, smem_tiles, r, p.scale);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          const int trow = (int)tok0 + tile_row0 + warp * 32;
          tma_store_4d(&tm_dq, sQ + warp * 32 * 128, 0, trow, hd, (int)boff);
          if (D > 64 && p.head_dim > 64) tma_store_4d(&tm_dq, sQ + kBoxBytes + warp * 32 * 128, 64, trow, hd, (int)boff);
          tma_store_commit();
          tma_store_wait_all();
        }
      } else {
        // the sequence ends inside the tile: row by row, rows past the end are left alone
        T *grow = reinterpret_cast<T *>(p.dq.ptr) + boff * p.dq.sb + (long long)hd * p.dq.sh + (tok0 + tile_row0 + r) * p.dq.st;
        store_acc_rows<D, kFp16, T>(t_acc, grow, tile_row0 + r < item.len, p.head_dim, p.scale);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0) trace_block(p, 2);
  if (warp == 5) tmem_dealloc(tmem, kCols);
}

// =======================================================================================================
// dkv kernel for head sizes 72..128, pipelined: one CTA per 128-key tile, all eight row warps on one query tile
// =======================================================================================================
// The key tile is handled as two 64-key strips (h = 0, 1) that share every Q/dO tile: a step is one query tile
// against one strip, and the two steps of a query tile use the same Q/dO stage, so Q/dO are loaded once per
// 128 keys.  Within a step, warps 0-3 own key columns 0..31 of the strip and warps 4-7 columns 32..63 for the same
// 128 query rows; each group restarts from its own R1/S2 record (the dq kernel records them every 32 keys), so the
// groups are independent.  S/dP are double-buffered in TMEM and the Q/dO tiles sit in a two-stage ring: the S/dP
// MMAs of step g+1 (issuer warp 9) and the dK^T/dV^T MMAs of step g-1 (issuer warp 10) run while the rows of
// step g are processed.  The A/dz tiles are single-buffered; the rows wait for the previous step's dK^T/dV^T MMAs
// only before their first store, i.e. after a quarter of the step's arithmetic.
// TMEM columns: S[slot] at 128 slot, dP[slot] at 128 slot + 64, dK^T[h] at 256 + 128 h, dV^T[h] at 320 + 128 h.
namespace dkv4 {
constexpr int kThreads = 352;
constexpr int kBN = 64;
constexpr int kTileBytes = kBM * 128 * 2;      // Q, dO, K or V tile: two 128 x 64 boxes
constexpr int kStripOffset = kBN * 128;        // byte offset of strip 1 inside a box (64 rows of 128 bytes)
constexpr int kAzBytes = kBM * kBN * 2;        // A or dz tile, 128 rows x 64 keys
constexpr int kSmem = 1024 + 2 * kTileBytes + 4 * kTileBytes + 2 * kAzBytes + 512 + kListBits / 8;
static_assert(kSmem <= 232448, "shared memory per block");
enum { bKV = 0, bQgFull = 1, bQgEmpty = 3, bSpFull = 5, bSpEmpty = 7, bAzFull = 9, bAzEmpty = 10, bOutFull = 11, bStaged = 12,
       bDrained = 14, bNum = 16 };
}  // namespace dkv4

template <bool kFp16>
__global__ void __launch_bounds__(dkv4::kThreads, 1)
tc_bwd_dkv4_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                   const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_g,
                   const __grid_constant__ CUtensorMap tm_dk, const __grid_constant__ CUtensorMap tm_dv, const KParams p) {
  enter_kernel<false>();
  using namespace dkv4;
  constexpr int D = 128;
  extern __shared__ uint8_t smem_raw[];
  if (gated(p)) return;
  if (threadIdx.x == 0) trace_block(p, 0);
  SmallTable &tb = *reinterpret_cast<SmallTable *>(smem_raw);   // never used: the launch sees to that, there is no room for it
  bool refused;
  const long long covered = open_table(p, tb, refused);
  if (covered < p.tokens) {
    using T = typename std::conditional<kFp16, __half, __nv_bfloat16>::type;
    fill_rows<T>(p.dk, fill_job(p, covered, refused, blockIdx.x, gridDim.x));
    fill_rows<T>(p.dv, fill_job(p, covered, refused, blockIdx.x, gridDim.x));
  }
  TileCoord c;
  int hh_blk;
  if (refused || !decode_block(p, tb, false, c, hh_blk)) return;
  const int J = c.idx;                         // the 128-key tile
  const int n_halves = J * kBM + kBN < c.len ? 2 : 1;   // the sequence may end inside the first strip

  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t *gbase = smem_raw + (base - raw);
  const uint32_t sK = base;
  const uint32_t sV = sK + kTileBytes;
  const uint32_t sQ = sV + kTileBytes;               // stage b: Q at sQ + b * 2 * kTileBytes, dO right behind it
  const uint32_t sAZ = sQ + 4 * kTileBytes;          // A, then dz
  const uint32_t sBar = sAZ + 2 * kAzBytes;
  Ctl *ctl = reinterpret_cast<Ctl *>(gbase + (sBar - base) + bNum * 8);
  volatile int *abort_flag = &ctl->abort;
  auto bar = [&](int i) { return sBar + 8u * i; };

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int hh = hh_blk, h = p.head0 + hh;
  // step g: the (g / n_halves)-th query tile that reaches this key tile, strip g % n_halves
  QueryList list{p, c, h, J, kBM, c.n_tiles - J, reinterpret_cast<uint32_t *>(gbase + (sBar - base) + 512)};
  const int hshift = n_halves - 1;
  list.build();
  int tr_cur = 0;   // cursor of this thread's event-log lane (diagnostics)

  if (threadIdx.x == 0) {
    mbar_init(bar(bKV), 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar(bQgFull + b), 1);
      mbar_init(bar(bQgEmpty + b), 1);
      mbar_init(bar(bSpFull + b), 1);
      mbar_init(bar(bSpEmpty + b), 8);
    }
    mbar_init(bar(bAzFull), 8);
    mbar_init(bar(bAzEmpty), 1);
    mbar_init(bar(bOutFull), 1);
    for (int b = 0; b < 2; ++b) { mbar_init(bar(bStaged + b), 4); mbar_init(bar(bDrained + b), 1); }
    ctl->abort = 0;
    fence_barrier_init();
  }
  if (warp == 9) {
    tmem_alloc(smem_u32(&ctl->tmem_base), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = ctl->tmem_base;

  if (warp == 8) {
    if (lane == 0) {
      prefetch_tensormap(&tm_q); prefetch_tensormap(&tm_k); prefetch_tensormap(&tm_v); prefetch_tensormap(&tm_g);
      const int krow = (int)c.tok0 + J * kBM;
      mbar_arrive_expect_tx(bar(bKV), 2 * kTileBytes);
      for (int kb = 0; kb < 2; ++kb) {
        tma_load_4d(sK + kb * kBoxBytes, &tm_k, bar(bKV), kb * 64, krow, h, (int)c.boff);
        tma_load_4d(sV + kb * kBoxBytes, &tm_v, bar(bKV), kb * 64, krow, h, (int)c.boff);
      }
      for (int u = 0, off = 0; off < list.n; ++u, off = list.next(off + 1)) {
        const int b = u & 1;
        if (u >= 2 && !wait_or_abort(bar(bQgEmpty + b), ((u >> 1) - 1) & 1, abort_flag, p, 610)) break;
        if (*abort_flag) break;
        const int qrow = (int)c.tok0 + (J + off) * kBM;
        const uint32_t dst = sQ + b * 2 * kTileBytes;
        trace_event(p, 0, tr_cur, 1, u);
        mbar_arrive_expect_tx(bar(bQgFull + b), 2 * kTileBytes);
        for (int kb = 0; kb < 2; ++kb) {
          tma_load_4d(dst + kb * kBoxBytes, &tm_q, bar(bQgFull + b), kb * 64, qrow, h, (int)c.boff);
          tma_load_4d(dst + kTileBytes + kb * kBoxBytes, &tm_g, bar(bQgFull + b), kb * 64, qrow, h, (int)c.boff);
        }
      }
    }
  } else if (warp == 9) {
    // ------------------------------------------------ issuer of S = Q K^T and dP = dO V^T (128 x 64)
    if (lane == 0) {
      constexpr uint32_t idesc_s = idesc_f16(kBM, kBN, kFp16, false, false);
      bool ok = wait_or_abort(bar(bKV), 0, abort_flag, p, 620);
      for (int g = 0, off = 0; ok && off < list.n; off = (g & hshift) == hshift ? list.next(off + 1) : off, ++g) {
        const int u = g >> hshift, hf = g & hshift, b = u & 1, slot = g & 1;
        ok = wait_or_abort(bar(bQgFull + b), (u >> 1) & 1, abort_flag, p, 621);
        // the rows of step g-2 have read this S/dP slot
        if (ok && g >= 2) ok = wait_or_abort(bar(bSpEmpty + slot), ((g >> 1) - 1) & 1, abort_flag, p, 622);
        if (!ok) break;
        trace_event(p, 1, tr_cur, 2, g);
        tc_fence_after();
        const uint32_t qaddr = sQ + b * 2 * kTileBytes;
        mma_kmajor_kmajor<D>(tmem + slot * 128, qaddr, sK + hf * kStripOffset, idesc_s, false);
        mma_kmajor_kmajor<D>(tmem + slot * 128 + 64, qaddr + kTileBytes, sV + hf * kStripOffset, idesc_s, false);
        mma_commit(bar(bSpFull + slot));
        trace_event(p, 1, tr_cur, 3, g);
      }
    }
  } else if (warp == 10) {
    // ------------------------------------------------ issuer of dK^T += Q^T dz and dV^T += dO^T A (128 x 64)
    if (lane == 0) {
      constexpr uint32_t idesc_t = idesc_f16(kBM, kBN, kFp16, true, true);
      const uint64_t a0 = smem_desc_sw128(sAZ, 16, 1024), z0 = smem_desc_sw128(sAZ + kAzBytes, 16, 1024);
      bool ok = true;
      for (int g = 0, off = 0; ok && off < list.n; off = (g & hshift) == hshift ? list.next(off + 1) : off, ++g) {
        const int u = g >> hshift, hf = g & hshift, b = u & 1;
        ok = wait_or_abort(bar(bAzFull), g & 1, abort_flag, p, 623);
        if (!ok) break;
        trace_event(p, 4, tr_cur, 6, g);
        tc_fence_after();
        const uint32_t qaddr = sQ + b * 2 * kTileBytes;
        const uint64_t q0 = smem_desc_sw128(qaddr, kBoxBytes, 1024), g0 = smem_desc_sw128(qaddr + kTileBytes, kBoxBytes, 1024);
        const uint32_t t_dk = tmem + 256 + hf * 128, t_dv = t_dk + 64;
#pragma unroll
        for (int ks = 0; ks < kBM / 16; ++ks)
          mma_f16_ss(t_dk, q0 + (uint64_t)(ks * 128), z0 + (uint64_t)(ks * 128), idesc_t, u > 0 || ks > 0);
#pragma unroll
        for (int ks = 0; ks < kBM / 16; ++ks)
          mma_f16_ss(t_dv, g0 + (uint64_t)(ks * 128), a0 + (uint64_t)(ks * 128), idesc_t, u > 0 || ks > 0);
        mma_commit(bar(bAzEmpty));
        if (hf == hshift) mma_commit(bar(bQgEmpty + b));   // the tile's last strip: its Q/dO stage is free
        trace_event(p, 4, tr_cur, 7, g);
      }
      if (ok) mma_commit(bar(bOutFull));
    }
  } else {
    // ------------------------------------------------ rows: warps 0-3 columns 0..31, warps 4-7 columns 32..63
    using T = typename std::conditional<kFp16, __half, __nv_bfloat16>::type;
    const int w = warp >> 2;
    const int r = threadIdx.x & 127;
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    const float scale2 = p.scale * kLog2e;
    bool ok = true;
    // the per-row start values of a step come from global memory: they are fetched one step ahead
    // (the gradient of rem stays a raw 16-bit value until the step that uses it, so that nothing in this step depends
    // on the load)
    auto fetch = [&](int I, int hf, float &r1f, float &gpre, unsigned short &dr_raw) {
      const int quarter = 2 * hf + w;   // which 32-key quarter of the 128-key tile
      const int gi = I * kBM + r;
      const long long slot = (((long long)hh * p.pairs_cap + c.pair0 + (long long)I * (I + 1) / 2 + J) * 4 + quarter) * kBM + r;
      r1f = p.bnd_r1[slot];
      gpre = p.bnd_s2[slot];
      const long long row = (c.boff * p.heads + h) * p.tokens + c.tok0 + min(gi, c.len - 1);
      dr_raw = reinterpret_cast<const unsigned short *>(p.d_rem)[row];
    };
    uint8_t *gA = gbase + (sAZ - base);
    uint8_t *gZ = gA + kAzBytes;
    float nr1, ngpre;
    unsigned short ndr;
    fetch(J, 0, nr1, ngpre, ndr);
    int off = 0, off_next = 0;   // this step's and the next step's query tile
    for (int g = 0; off < list.n && ok; ++g, off = off_next) {
      const int u = g >> hshift, hf = g & hshift, slot = g & 1;
      const int I = J + off;
      off_next = hf == hshift ? list.next(off + 1) : off;
      const int quarter = 2 * hf + w;
      const bool valid = I * kBM + r < c.len;
      const float r1f = nr1, gpre = ngpre;
      const float dr = valid ? to_f32<T>(*reinterpret_cast<const T *>(&ndr)) : 0.f;
      if (off_next < list.n) fetch(J + off_next, (g + 1) & hshift, nr1, ngpre, ndr);
      ok = wait_or_abort(bar(bSpFull + slot), (g >> 1) & 1, abort_flag, p, 630);
      if (!ok) break;
      if (threadIdx.x == 0 && g == 0) trace_block(p, 1);
      if (r == 0) trace_event(p, 2 + w, tr_cur, 4 + 16 * w, g);
      tc_fence_after();
      const uint32_t tS = tmem + slot * 128 + w * 32 + lane_off, tP = tS + 64;
      float gs = 0.f, logsum = 0.f;
      const bool diag = (u == 0);
      const bool masked = diag || (I == c.n_tiles - 1 && (c.len & (kBM - 1)) != 0);
      // On the diagonal tile the quarters after this warp's last row are masked for all of its 32 rows, and a warp whose
      // rows all lie past the sequence end has nothing allowed anywhere: A and dz are zero, the scores are not read.
      const bool skip = (diag && quarter * 32 >= (r | 31) + p.attend_current) || I * kBM + (r & ~31) >= c.len;
      if (!skip) {
        uint32_t s0[16], d0[16], s1[16], d1[16];
        tmem_ld16(tS, s0);
        tmem_ld16(tP, d0);
        tmem_wait_ld_regs(s0, d0);
        tmem_ld16(tS + 16, s1);
        tmem_ld16(tP + 16, d1);
        const int limit = chunk_limit(valid, diag, r, p.attend_current);
        {
          float pa[16], pz[16];
          if (masked) bwd_chunk<true, false>(s0, d0, quarter * 32, limit, scale2, r1f, gpre, dr, gs, logsum, pa, pz, false);
          else bwd_chunk<false, true>(s0, d0, 0, limit, scale2, r1f, gpre, dr, gs, logsum, pa, pz, !p.dense);
          // the A/dz tiles are still being read by the previous step's MMAs
          if (g >= 1) {
            ok = wait_or_abort(bar(bAzEmpty), (g - 1) & 1, abort_flag, p, 631);
            tc_fence_after();
          }
          store_row_chunk16<kFp16>(gA, r, w * 32, pa);
          store_row_chunk16<kFp16>(gZ, r, w * 32, pz);
        }
        tmem_wait_ld_regs(s1, d1);
        tc_fence_before();          // this step's TMEM reads are done: the S/dP slot is handed back
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(bSpEmpty + slot));
        {
          float pa[16], pz[16];
          if (masked) bwd_chunk<true, false>(s1, d1, quarter * 32 + 16, limit, scale2, r1f, gpre, dr, gs, logsum, pa, pz, false);
          else bwd_chunk<false, true>(s1, d1, 0, limit, scale2, r1f, gpre, dr, gs, logsum, pa, pz, !p.dense);
          store_row_chunk16<kFp16>(gA, r, w * 32 + 16, pa);
          store_row_chunk16<kFp16>(gZ, r, w * 32 + 16, pz);
        }
      } else {
        if (g >= 1) {
          ok = wait_or_abort(bar(bAzEmpty), (g - 1) & 1, abort_flag, p, 631);
          tc_fence_after();
        }
        const uint32_t zero[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          store_packed_chunk16(gA, r, w * 32 + 16 * q, zero);
          store_packed_chunk16(gZ, r, w * 32 + 16 * q, zero);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(bSpEmpty + slot));
      }
      // the sequence ends inside this query tile: the A and dz rows behind the end are exact zeros, the Q and dO rows
      // there are not this sequence's (see zero_tile_rows) and are cleared before this step's MMAs are released
      if (c.len - I * kBM < kBM)
        zero_tile_rows(gbase + (sQ - base) + (u & 1) * 2 * kTileBytes, c.len - I * kBM, kBM, 4, kBoxBytes, threadIdx.x, 2 * kBM);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(bAzFull));
      if (r == 0) trace_event(p, 2 + w, tr_cur, 5 + 16 * w, g);
    }
    // ---- epilogue: dK^T (warps 0-3) and dV^T (warps 4-7), lanes = head dimension, columns = keys.  A full strip is
    // transposed into this warpgroup's buffer (A for dK, dz for dV: all their MMAs are done) and leaves by TMA;
    // a strip the sequence ends in is written element by element.
    if (ok) ok = wait_or_abort(bar(bOutFull), 0, abort_flag, p, 632);
    if (ok) {
      tc_fence_after();
      const TensorRef &out = w == 0 ? p.dk : p.dv;
      const CUtensorMap *omap = w == 0 ? &tm_dk : &tm_dv;
      const float mul = w == 0 ? p.scale : 1.f;
      uint8_t *stage = w == 0 ? gA : gZ;
      const uint32_t stage_addr = sAZ + w * kAzBytes;
      T *obase = reinterpret_cast<T *>(out.ptr) + c.boff * out.sb + (long long)h * out.sh + (c.tok0 + J * kBM) * out.st + r;
      int round = 0;
#pragma unroll 1
      for (int hf = 0; hf < n_halves && ok; ++hf) {
        // the same for all row warps; columns at and beyond head_dim lie outside the tensor map and are not written
        const bool full = J * kBM + hf * kBN + kBN <= c.len;
#pragma unroll 1
        for (int ch = 0; ch < 4; ++ch) {
          uint32_t va[16];
          tmem_ld16(tmem + 256 + hf * 128 + w * 64 + ch * 16 + lane_off, va);
          tmem_wait_ld();
          if (full) {
            // element (key, r) of a [64 keys x 128] tile: two 64-column blocks, 128-byte swizzle
            const uint32_t col_off = (r >> 6) * (kBN * 128) + (r & 7) * 2;
#pragma unroll
            for (int k = 0; k < 16; ++k) {
              const int key = ch * 16 + k;
              const uint32_t off = col_off + (key >> 3) * 1024 + (key & 7) * 128 + ((((r & 63) >> 3) ^ (key & 7)) << 4);
              *reinterpret_cast<T *>(stage + off) = from_f32<T>(__uint_as_float(va[k]) * mul);
            }
          } else if (r < p.head_dim) {
#pragma unroll
            for (int k = 0; k < 16; ++k) {
              const int key = J * kBM + hf * kBN + ch * 16 + k;
              if (key < c.len) obase[(long long)(hf * kBN + ch * 16 + k) * out.st] = from_f32<T>(__uint_as_float(va[k]) * mul);
            }
          }
        }
        if (full) {
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(bStaged + w));
          if (r == 0 && (ok = wait_or_abort(bar(bStaged + w), round & 1, abort_flag, p, 633))) {
            const int krow = (int)c.tok0 + J * kBM + hf * kBN;
            tma_store_4d(omap, stage_addr, 0, krow, h, (int)c.boff);
            if (p.head_dim > 64) tma_store_4d(omap, stage_addr + kBN * 128, 64, krow, h, (int)c.boff);
            tma_store_commit();
            tma_store_wait_read();
            mbar_arrive(bar(bDrained + w));
          }
          // the buffer is rewritten for the next strip
          if (ok && hf + 1 < n_halves) ok = wait_or_abort(bar(bDrained + w), round & 1, abort_flag, p, 634);
          ++round;
        }
      }
      if (r == 0) tma_store_wait_all();
    }
  }

  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0) trace_block(p, 2);
  if (warp == 9) tmem_dealloc(tmem, kTmemCols);
}

// =======================================================================================================
// dK/dV from stored tiles (head sizes 72..128): two GEMMs per 128-key tile, no row passes
// =======================================================================================================
// In stored-tiles mode the dq kernel leaves the 16-bit A and dz tiles of every (query tile, key tile) pair in the
// workspace.  This kernel owns one 128-key tile and walks its query tiles diagonal -> end, 32 query rows per stage:
//   dK[keys x d] += dz^T Q,   dV[keys x d] += A^T dO      (M = 128 keys, N = 128 columns, K = 32 query rows)
// with all four operands read row-major as "MN-major" tiles (rows = query rows = the contraction).  Accumulators sit
// in TMEM with lanes = keys, so the epilogue writes plain rows.  Fixed summation order, no atomics.
//   warp 4    TMA producer: per stage A, dz (from the workspace), Q, dO -- 32 KiB, three stages
//   warp 5    MMA issuer
//   warps 0-3 epilogue: dK, dV rows -> shared memory -> TMA stores
// The kernel is bound by reading the stored tiles (64 KiB per 128x128 pair) from HBM.  A block has a fixed cost of
// several microseconds (first loads, and at the end accumulators -> shared memory -> TMA stores) next to ~17 stages
// on average, so the stages are kept small enough for TWO blocks per SM (100 KB of shared memory, 256 TMEM columns
// each): one block's prologue and epilogue run under the other's stages.
namespace dkv5 {
constexpr int kThreads = 192;
constexpr int kStages = 3;
constexpr int kRows = 32;                    // query rows per stage
constexpr int kSub = kBM / kRows;            // stages per query tile
constexpr int kBox = kRows * 64 * 2;         // kRows rows x 64 columns, 16-bit
constexpr int kStageBytes = 8 * kBox;        // A, dz, Q, dO: two 64-column blocks each; also one 128 x 128 output tile
constexpr int kSmem = 1024 + kStages * kStageBytes + 512 + kListBits / 8 + (int)sizeof(SmallTable);
constexpr uint32_t kCols = 256;              // dK 0..127, dV 128..255
enum { bFull = 0, bEmpty = 3, bOut = 6, bClean = 7, bLanded = 8, bNum = 9 };
}  // namespace dkv5

template <bool kFp16>
__global__ void __launch_bounds__(dkv5::kThreads, 2)
tc_bwd_dkv5_kernel(const __grid_constant__ CUtensorMap tm_az, const __grid_constant__ CUtensorMap tm_q,
                   const __grid_constant__ CUtensorMap tm_g, const __grid_constant__ CUtensorMap tm_dk,
                   const __grid_constant__ CUtensorMap tm_dv, const KParams p) {
  enter_kernel<false>();
  using namespace dkv5;
  constexpr int D = 128;
  extern __shared__ uint8_t smem_raw[];
  if (gated(p)) return;
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t *gbase = smem_raw + (base - raw);
  const uint32_t sBar = base + kStages * kStageBytes;
  SmallTable &tb = *reinterpret_cast<SmallTable *>(gbase + (sBar - base) + 512 + kListBits / 8);
  bool refused;
  const long long covered = open_table(p, tb, refused);
  if (covered < p.tokens) {
    using T = typename std::conditional<kFp16, __half, __nv_bfloat16>::type;
    fill_rows<T>(p.dk, fill_job(p, covered, refused, blockIdx.x, gridDim.x));
    fill_rows<T>(p.dv, fill_job(p, covered, refused, blockIdx.x, gridDim.x));
  }
  TileCoord c;
  int hh;
  if (refused || !decode_block(p, tb, false, c, hh)) return;
  const int h = p.head0 + hh;
  const int J = c.idx;                        // the 128-key tile
  // The sequence may end inside the last query tile.  The A and dz rows behind the end are zeros in the workspace; the
  // Q and dO rows there are not this sequence's (see zero_tile_rows).  Stages that hold such rows are cleaned: the
  // issuer tells the epilogue warps, idle until the end, that such a stage has landed (bLanded; a barrier of its own,
  // because a parity wait on bFull only works for a waiter that follows every phase), they clear the rows and hand
  // the stage back through bClean.
  const int last_rows = c.len - (c.n_tiles - 1) * kBM;          // 1 .. 128 rows of the last query tile exist
  const int clean_from = last_rows / kRows;                     // first such stage of the last query tile

  Ctl *ctl = reinterpret_cast<Ctl *>(gbase + (sBar - base) + bNum * 8);
  volatile int *abort_flag = &ctl->abort;
  volatile int *clean_stage = reinterpret_cast<volatile int *>(ctl + 1);
  auto bar = [&](int i) { return sBar + 8u * i; };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the query tiles that reach this key tile, kSub stages each
  const int last = c.n_tiles - J - 1;
  QueryList list{p, c, h, J, kBM, p.pair_span == nullptr ? last + 1 : min(last, p.pair_span[h]) + 1,
                 reinterpret_cast<uint32_t *>(gbase + (sBar - base) + 512)};
  list.build();

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(bar(bFull + s), 1); mbar_init(bar(bEmpty + s), 1); }
    mbar_init(bar(bOut), 1);
    mbar_init(bar(bClean), 4);
    mbar_init(bar(bLanded), 1);
    ctl->abort = 0;
    fence_barrier_init();
  }
  if (warp == 5) {
    tmem_alloc(smem_u32(&ctl->tmem_base), kCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = ctl->tmem_base;

  if (warp == 4) {
    if (lane == 0) {
      prefetch_tensormap(&tm_az); prefetch_tensormap(&tm_q); prefetch_tensormap(&tm_g);
      for (int t = 0, off = 0; off < list.n; ++t, off = t % kSub == 0 ? list.next(off + 1) : off) {
        const int st = t % kStages;
        if (t >= kStages && !wait_or_abort(bar(bEmpty + st), ((t / kStages) - 1) & 1, abort_flag, p, 640)) break;
        if (*abort_flag) break;
        const int I = J + off, hq = t % kSub;
        const bool packed = p.pair_slot != nullptr;
        const long long pair = (packed ? (long long)p.pair_slot[(long long)h * p.tiles_cap + tile_id(p, c, I)] : c.pair0 + (long long)I * (I + 1) / 2) + J;
        const int az_head = packed ? 0 : hh;
        const int az_row = (int)(pair * kBM) + hq * kRows;
        const int qrow = (int)c.tok0 + I * kBM + hq * kRows;
        const uint32_t dst = base + st * kStageBytes;
        mbar_arrive_expect_tx(bar(bFull + st), kStageBytes);
        for (int kb = 0; kb < 2; ++kb) {
          tma_load_4d(dst + (0 + kb) * kBox, &tm_az, bar(bFull + st), kb * 64, az_row, 0, az_head);   // A
          tma_load_4d(dst + (2 + kb) * kBox, &tm_az, bar(bFull + st), kb * 64, az_row, 1, az_head);   // dz
          tma_load_4d(dst + (4 + kb) * kBox, &tm_q, bar(bFull + st), kb * 64, qrow, h, (int)c.boff);
          tma_load_4d(dst + (6 + kb) * kBox, &tm_g, bar(bFull + st), kb * 64, qrow, h, (int)c.boff);
        }
      }
    }
  } else if (warp == 5) {
    if (lane == 0) {
      // all operands MN-major: rows = query rows (the contraction), two 64-column blocks kBox apart
      constexpr uint32_t idesc = idesc_f16(kBM, D, kFp16, true, true);
      bool ok = true;
      int cleaned = 0;
      for (int t = 0, off = 0; ok && off < list.n; ++t, off = t % kSub == 0 ? list.next(off + 1) : off) {
        const int st = t % kStages;
        ok = wait_or_abort(bar(bFull + st), (t / kStages) & 1, abort_flag, p, 641);
        if (ok && off == last && t % kSub >= clean_from) {
          *clean_stage = st;
          mbar_arrive(bar(bLanded));
          ok = wait_or_abort(bar(bClean), cleaned++ & 1, abort_flag, p, 643);
        }
        if (!ok) break;
        tc_fence_after();
        const uint32_t a = base + st * kStageBytes;
        const uint64_t dA = smem_desc_sw128(a, kBox, 1024), dZ = smem_desc_sw128(a + 2 * kBox, kBox, 1024);
        const uint64_t dQ = smem_desc_sw128(a + 4 * kBox, kBox, 1024), dG = smem_desc_sw128(a + 6 * kBox, kBox, 1024);
#pragma unroll
        for (int ks = 0; ks < kRows / 16; ++ks)   // 16 query rows = 2048 bytes per step
          mma_f16_ss(tmem, dZ + (uint64_t)(ks * 128), dQ + (uint64_t)(ks * 128), idesc, t > 0 || ks > 0);
#pragma unroll
        for (int ks = 0; ks < kRows / 16; ++ks)
          mma_f16_ss(tmem + 128, dA + (uint64_t)(ks * 128), dG + (uint64_t)(ks * 128), idesc, t > 0 || ks > 0);
        mma_commit(bar(bEmpty + st));
      }
      if (ok) mma_commit(bar(bOut));
    }
  } else {
    // ------------------------------------------------ epilogue: one thread per key row
    using T = typename std::conditional<kFp16, __half, __nv_bfloat16>::type;
    const int r = threadIdx.x;
    const uint32_t lane_off = (uint32_t)(warp * 32) << 16;
    bool ok = true;
    const bool last_listed = last < list.n && list.next(last) == last;
    for (int hq = clean_from; ok && last_listed && hq < kSub; ++hq) {
      ok = wait_or_abort(bar(bLanded), (hq - clean_from) & 1, abort_flag, p, 644);
      if (!ok) break;
      const int st = *clean_stage;
      int keep = last_rows - hq * kRows;   // rows of this stage that belong to the sequence
      keep = keep < 0 ? 0 : keep;
      zero_tile_rows(gbase + st * kStageBytes + 4 * kBox, keep, kRows, 4, kBox, r, kBM);   // Q and dO: boxes 4..7 of the stage
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(bClean));
    }
    if (ok && wait_or_abort(bar(bOut), 0, abort_flag, p, 642)) {
      tc_fence_after();
      const int key = J * kBM + r;
      const bool valid = key < c.len;
      // out = o + rem * v was requested: dV gains rem * d_out on its own row (rem = 2^log_rem)
      const T *grow = nullptr;
      float rem_f = 0.f;
      if (p.fuse_rem_v && valid) {
        grow = reinterpret_cast<const T *>(p.d_o.ptr) + c.boff * p.d_o.sb + (long long)h * p.d_o.sh + (c.tok0 + key) * p.d_o.st;
        rem_f = exp2f((float)p.log_rem[(c.boff * p.heads + h) * p.tokens + c.tok0 + key]);
      }
      if (J * kBM + kBM <= c.len) {
        // full tile: through the first two stages' memory (all MMAs are done), one TMA store per warp and half
#pragma unroll 1
        for (int which = 0; which < 2; ++which) {
          uint8_t *stage = gbase + which * kStageBytes;                // [128 x 128] as two blocks of 128-byte rows
          stage_acc_rows<D, kFp16>(tmem + which * 128 + lane_off, stage, r, which == 0 ? p.scale : 1.f,
                                   which == 1 ? grow : nullptr, rem_f, p.head_dim);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            const uint32_t src = base + which * kStageBytes + warp * 32 * 128;
            const int trow = (int)c.tok0 + J * kBM + warp * 32;
            const CUtensorMap *omap = which == 0 ? &tm_dk : &tm_dv;
            tma_store_4d(omap, src, 0, trow, h, (int)c.boff);
            if (p.head_dim > 64) tma_store_4d(omap, src + kBoxBytes, 64, trow, h, (int)c.boff);
            tma_store_commit();
          }
        }
        if (lane == 0) tma_store_wait_all();
      } else {
        // the sequence ends inside the tile: row by row, rows past the end are left alone
        T *krow = reinterpret_cast<T *>(p.dk.ptr) + c.boff * p.dk.sb + (long long)h * p.dk.sh + (c.tok0 + key) * p.dk.st;
        T *vrow = reinterpret_cast<T *>(p.dv.ptr) + c.boff * p.dv.sb + (long long)h * p.dv.sh + (c.tok0 + key) * p.dv.st;
        store_acc_rows<D, kFp16, T>(tmem + lane_off, krow, valid, p.head_dim, p.scale);
        store_acc_rows<D, kFp16, T>(tmem + 128 + lane_off, vrow, valid, p.head_dim, 1.f, grow, rem_f);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 5) tmem_dealloc(tmem, kCols);
}

// -------------------------------------------------------------------------------------------------------
template <bool kFp16>
static cudaError_t launch_bwd_t(const KParams &p, int dtype, cudaStream_t s) {
  CUtensorMap mq, mk, mv, mg;
  cudaError_t e;
  if ((e = make_tile_map(&mq, p.q, p, dtype)) != cudaSuccess) return e;
  if ((e = make_tile_map(&mk, p.k, p, dtype)) != cudaSuccess) return e;
  if ((e = make_tile_map(&mv, p.v, p, dtype)) != cudaSuccess) return e;
  if ((e = make_tile_map(&mg, p.d_o, p, dtype)) != cudaSuccess) return e;
  const dim3 grid((unsigned)item_blocks(p));
  if (!p.skip_dq) {
    const bool narrow = p.head_dim <= 64;
    auto kernel = p.az != nullptr ? (narrow ? tc_bwd_dq3_kernel<64, kFp16, true> : tc_bwd_dq3_kernel<128, kFp16, true>)
                                  : (narrow ? tc_bwd_dq3_kernel<64, kFp16, false> : tc_bwd_dq3_kernel<128, kFp16, false>);
    const int smem = narrow ? dq3::Cfg<64>::kSmem : dq3::Cfg<128>::kSmem;
    if ((e = allow_dynamic_smem(reinterpret_cast<const void *>(kernel), smem)) != cudaSuccess) return e;
    CUtensorMap mk64, mv64, mdq;   // 64-row boxes: the kernel streams 64-key sub-tiles; dQ leaves 32 rows per warp
    if ((e = make_tile_map(&mk64, p.k, p, dtype, 64)) != cudaSuccess) return e;
    if ((e = make_tile_map(&mv64, p.v, p, dtype, 64)) != cudaSuccess) return e;
    if ((e = make_tile_map(&mdq, p.dq, p, dtype, 32)) != cudaSuccess) return e;
    if ((e = launch_kernel(kernel, grid, dq3::kThreads, smem, s, mq, mk64, mv64, mg, mdq, p)) != cudaSuccess) return e;
  }
  if (!p.skip_dkv && p.az != nullptr) {
    auto kernel = tc_bwd_dkv5_kernel<kFp16>;
    e = allow_dynamic_smem(reinterpret_cast<const void *>(kernel), dkv5::kSmem);
    if (e != cudaSuccess) return e;
    CUtensorMap maz, mq64, mg64, mdk, mdv;
    if ((e = make_az_map(&maz, p, dtype, dkv5::kRows)) != cudaSuccess) return e;
    if ((e = make_tile_map(&mq64, p.q, p, dtype, dkv5::kRows)) != cudaSuccess) return e;
    if ((e = make_tile_map(&mg64, p.d_o, p, dtype, dkv5::kRows)) != cudaSuccess) return e;
    if ((e = make_tile_map(&mdk, p.dk, p, dtype, 32)) != cudaSuccess) return e;   // stores: 32 rows per warp
    if ((e = make_tile_map(&mdv, p.dv, p, dtype, 32)) != cudaSuccess) return e;
    if ((e = launch_kernel(kernel, grid, dkv5::kThreads, dkv5::kSmem, s, maz, mq64, mg64, mdk, mdv, p)) != cudaSuccess) return e;
  } else if (!p.skip_dkv) {
    auto kernel = tc_bwd_dkv4_kernel<kFp16>;
    e = allow_dynamic_smem(reinterpret_cast<const void *>(kernel), dkv4::kSmem);
    if (e != cudaSuccess) return e;
    CUtensorMap mdk, mdv;   // stores: one 64-key strip at a time
    if ((e = make_tile_map(&mdk, p.dk, p, dtype, 64)) != cudaSuccess) return e;
    if ((e = make_tile_map(&mdv, p.dv, p, dtype, 64)) != cudaSuccess) return e;
    if ((e = launch_kernel(kernel, grid, dkv4::kThreads, dkv4::kSmem, s, mq, mk, mv, mg, mdk, mdv, p)) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// TMA fills the columns past head_dim with zeros, so every head size up to 128 runs the 64- or 128-column kernels.
cudaError_t launch_tc_bwd(const KParams &p, int dtype, cudaStream_t s, int *launches) {
  *launches += (p.skip_dq ? 0 : 1) + (p.skip_dkv ? 0 : 1);
  return dtype == SB_DTYPE_F16 ? launch_bwd_t<true>(p, dtype, s) : launch_bwd_t<false>(p, dtype, s);
}

}  // namespace sb
