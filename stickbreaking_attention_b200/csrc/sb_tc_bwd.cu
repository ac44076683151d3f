// Tensor-core backward kernels for bf16 / fp16 tensors (reference counterpart: _backward_one_row,
// sb_varlen_bwd.py:297-481, which accumulates dK/dV across blocks under a global spin lock).
//
// Two kernels per call, no atomics, no locks, fixed summation order:
//   dq kernel (tc_bwd_dq2_kernel)   query-stationary, 256 query rows per block.  Walks the keys 0 -> diagonal in
//               64-key sub-tiles; per step S = Q K^T and dP = dO V^T go to TMEM, one thread per query row recomputes
//               A and dz = G - beta * C with the log-space suffix sum (a pair of floats across tiles, started from
//               the saved fp64 log_rem) and the prefix sum C of G carried in registers, writes dz as a 16-bit tile, and
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
// A, G and dz of the chunk is exactly 0 (e, the reciprocals and dP - dR are finite): only the log-space sum is formed,
// with the same operations as otherwise, and the rest is not computed.
// Packed pairs (two fp32 per instruction) are used where a pair sits in adjacent registers anyway -- accumulator columns and
// what is computed column by column from them.  Products across columns stay scalar: pairing their operands up costs as many
// register moves as the packed instruction saves.
struct BwdChunk {
  float2 be01[4], be23[4];   // beta
  float pa[16];              // A
  bool zero;                 // the chunk is known to be zero for all rows of the warp
};

// Sweeps 1 and 2, which do not need dP; `between` runs where the fewest registers are in use and half of sweep 2 is left.
template <bool kMasked, bool kSkip, class Between>
__device__ __forceinline__ void bwd_chunk_weights(const uint32_t (&s)[16], int mc0, int limit, float scale2, float r1, float g_before,
                                                  float &logsum, BwdChunk &c, Between between, bool may_skip = true) {
  float chunk_log = 0.f;   // summed per chunk, like the forward's (see fwd256_row_chunk): the two agree bit for bit
  const float2 sc = make_float2(scale2, scale2), one = make_float2(1.f, 1.f);
  float2 e01[4], e23[4], t01[4], t23[4];
#pragma unroll
  for (int g = 3; g >= 0; --g) {
    const float2 x01 = mul2(make_float2(__uint_as_float(s[4 * g]), __uint_as_float(s[4 * g + 1])), sc);
    const float2 x23 = mul2(make_float2(__uint_as_float(s[4 * g + 2]), __uint_as_float(s[4 * g + 3])), sc);
    e01[g] = make_float2(ex2(fminf(x01.x, 30.f)), ex2(fminf(x01.y, 30.f)));
    e23[g] = make_float2(ex2(fminf(x23.x, 30.f)), ex2(fminf(x23.y, 30.f)));
    t01[g] = add2(e01[g], one);
    t23[g] = add2(e23[g], one);
    if (kMasked) {
      const int col = mc0 + 4 * g;
      if (!(col < limit)) { e01[g].x = 0.f; t01[g].x = 1.f; }
      if (!(col + 1 < limit)) { e01[g].y = 0.f; t01[g].y = 1.f; }
      if (!(col + 2 < limit)) { e23[g].x = 0.f; t23[g].x = 1.f; }
      if (!(col + 3 < limit)) { e23[g].y = 0.f; t23[g].y = 1.f; }
    }
    chunk_log += lg2((t01[g].x * t01[g].y) * (t23[g].x * t23[g].y));
  }
  logsum += chunk_log;
  c.zero = kSkip && may_skip && __all_sync(0xffffffffu, ex2(r1 + logsum) == 0.f && g_before == 0.f);
  if (c.zero) {
#pragma unroll
    for (int i = 0; i < 16; ++i) c.pa[i] = 0.f;
    between();
    return;
  }
  float rpg[4], i23[4], ri1[4], ri3[4];
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    const float p01 = t01[g].x * t01[g].y, p23 = t23[g].x * t23[g].y;
    const float rp = rcp(p01 * p23);
    const float i01 = rp * p23;                 // 1 / t0 t1
    i23[g] = rp * p01;                          // 1 / t2 t3
    const float2 ri01 = make_float2(i01 * t01[g].y, i01 * t01[g].x);
    const float2 ri23 = make_float2(i23[g] * t23[g].y, i23[g] * t23[g].x);
    c.be01[g] = mul2(e01[g], ri01);
    c.be23[g] = mul2(e23[g], ri23);
    rpg[g] = rp;
    ri1[g] = ri01.y;
    ri3[g] = ri23.y;
  }
  between();
  float wend = ex2(r1 + logsum);   // product of (1 - beta) over everything after the chunk
#pragma unroll
  for (int g = 3; g >= 0; --g) {
    const float2 w23 = make_float2(wend * i23[g], wend * ri3[g]);   // inclusive products at columns 2, 3
    wend *= rpg[g];                                                  // at column 0 = after the previous group
    const float2 w01 = make_float2(wend, w23.x * ri1[g]);
    const float2 a01 = mul2(e01[g], w01);
    const float2 a23 = mul2(e23[g], w23);
    c.pa[4 * g] = a01.x;
    c.pa[4 * g + 1] = a01.y;
    c.pa[4 * g + 2] = a23.x;
    c.pa[4 * g + 3] = a23.y;
  }
}

// Sweep 3.  On entry `gs` is the pass's sum of G before the chunk; pz: dz.
template <bool kMasked, bool kSkip>
__device__ __forceinline__ void bwd_chunk_dz(const uint32_t (&dp)[16], int mc0, int limit, float gpre, float dr, float &gs, BwdChunk &c,
                                             float (&pz)[16]) {
  if (kSkip && c.zero) {
#pragma unroll
    for (int i = 0; i < 16; ++i) pz[i] = 0.f;
    return;
  }
  const float2 ndr = make_float2(-dr, -dr);
  float cb = gpre + gs, csum = 0.f;   // C before the group; the chunk's own sum of G
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    float2 g01 = mul2(make_float2(c.pa[4 * g], c.pa[4 * g + 1]),
                      add2(make_float2(__uint_as_float(dp[4 * g]), __uint_as_float(dp[4 * g + 1])), ndr));
    float2 g23 = mul2(make_float2(c.pa[4 * g + 2], c.pa[4 * g + 3]),
                      add2(make_float2(__uint_as_float(dp[4 * g + 2]), __uint_as_float(dp[4 * g + 3])), ndr));
    if (kMasked) {   // rows past the sequence end carry arbitrary values: select, do not rely on 0 * x
      const int col = mc0 + 4 * g;
      if (!(col < limit)) { g01.x = 0.f; c.pa[4 * g] = 0.f; }
      if (!(col + 1 < limit)) { g01.y = 0.f; c.pa[4 * g + 1] = 0.f; }
      if (!(col + 2 < limit)) { g23.x = 0.f; c.pa[4 * g + 2] = 0.f; }
      if (!(col + 3 < limit)) { g23.y = 0.f; c.pa[4 * g + 3] = 0.f; }
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

// All three sweeps, A and dz written to the 16-bit tiles; c0 addresses the output tiles.
template <bool kFp16, bool kMasked, bool kSkip>
__device__ __forceinline__ void bwd_row_chunk(const uint32_t (&s)[16], const uint32_t (&dp)[16], int c0, int mc0, int r, int limit,
                                              float scale2, float r1, float gpre, float dr, float &gs, float &logsum, uint8_t *tile_a,
                                              uint8_t *tile_z, bool may_skip = true) {
  BwdChunk c;
  float pz[16];
  bwd_chunk_weights<kMasked, kSkip>(s, mc0, limit, scale2, r1, gpre + gs, logsum, c, [] {}, may_skip);
  bwd_chunk_dz<kMasked, kSkip>(dp, mc0, limit, gpre, dr, gs, c, pz);
  store_row_chunk16<kFp16>(tile_a, r, c0, c.pa);
  store_row_chunk16<kFp16>(tile_z, r, c0, pz);
}

// One row of a 64-key sub-tile of the dq kernel: four 16-column chunks.  What a pair of chunks still needs is requested
// together in the first one's sweep 2, the second chunk's dP into the registers of the first one's scores, so that 48
// registers do for everything in flight, and the last S and dP columns are in registers after two thirds of the pass:
// bSpEmpty is signalled then (one arrival per warp), and the next sub-tile's scores are computed under the rest.  dP is not
// waited for before half of the first chunk is done.
// mc0: key index of the sub-tile's first column inside its 128-key tile (for the diagonal mask).  The dz tile of the
// sub-tile before is waited for before the first store to it (in a tile's first sub-tile, an even one, that is the phase
// before the barrier's first: no wait).  Returns false if a wait gave up.
namespace dq2 {
constexpr int kMaxStages = 4;
enum { bQG = 0, bKvFull = 1, bKvEmpty = bKvFull + kMaxStages, bSFull = bKvEmpty + kMaxStages, bDpFull = bSFull + 2, bZFull = bDpFull + 2,
       bZEmpty = bZFull + 2, bFirst = bZEmpty + 2, bSpEmpty = bFirst + 1, bDqFull = bSpEmpty + 2, bNum = bDqFull + 2 };
}  // namespace dq2
// `bars`: the dq kernel's barriers, offset by the tile's number.  out: stored-tiles mode: this row's 64 values of A in the
// workspace; otherwise this row's record of R1 at the sub-tile's first key (S2 is `s2_off` floats further, both again kBM
// floats further for the key 32 columns on).
template <bool kFp16, bool kMasked, bool kStored, bool kSkip>
__device__ __forceinline__ bool strip_row_pass(uint32_t ts, uint32_t tp, int r, int u, int mc0, int limit, float scale2, float r1, float gpre,
                                              float dr, float &gs, float &logsum, uint8_t *tile_z, uint32_t bars, void *out,
                                              long long s2_off) {
  uint32_t s0[16], s1[16], d[16];
  bool ok = true;
  auto store = [&](int c0, const BwdChunk &c, const float (&pz)[16]) {
    uint32_t wz[8];
    pack_row_chunk16<kFp16>(pz, wz);
    store_packed_chunk16(tile_z, r, c0, wz);
    if constexpr (kStored) {
      uint32_t wa[8];
      pack_row_chunk16<kFp16>(c.pa, wa);
      store_packed_global16(reinterpret_cast<unsigned short *>(out) + c0, wa);
    }
  };
  tmem_ld16(ts, s0);
#pragma unroll 1
  for (int pair = 0; pair < 2; ++pair) {
    const int c0 = pair * 32;
    tmem_wait_ld_regs(s0);
    {
      BwdChunk c;
      bwd_chunk_weights<kMasked, kSkip>(s0, mc0 + c0, limit, scale2, r1, gpre + gs, logsum, c, [&] {
        if (pair == 0) {
          ok = mbar_wait(bars + 8u * dq2::bDpFull, u & 1);
          tc_fence_after();
        }
        tmem_ld16(tp + c0, d);
        tmem_ld16(ts + c0 + 16, s1);
        tmem_ld16(tp + c0 + 16, s0);
      });
      tmem_wait_ld_regs(d, s0);
      asm volatile("" : "+r"(s1[0]), "+r"(s1[1]), "+r"(s1[2]), "+r"(s1[3]), "+r"(s1[4]), "+r"(s1[5]), "+r"(s1[6]), "+r"(s1[7]), "+r"(s1[8]),
                   "+r"(s1[9]), "+r"(s1[10]), "+r"(s1[11]), "+r"(s1[12]), "+r"(s1[13]), "+r"(s1[14]), "+r"(s1[15])::"memory");
      if (pair == 0) {
        ok = mbar_wait(bars + 8u * dq2::bZEmpty, (u + 1) & 1) && ok;   // the previous sub-tile's dz has been read
        tc_fence_after();
      } else {               // the last columns are in registers: the S / dP slots can be overwritten
        tc_fence_before();
        __syncwarp();
        if ((threadIdx.x & 31) == 0) mbar_arrive(bars + 8u * dq2::bSpEmpty);
      }
      float pz[16];
      bwd_chunk_dz<kMasked, kSkip>(d, mc0 + c0, limit, gpre, dr, gs, c, pz);
      store(c0, c, pz);
    }
    {
      BwdChunk c;
      float pz[16];
      bwd_chunk_weights<kMasked, kSkip>(s1, mc0 + c0 + 16, limit, scale2, r1, gpre + gs, logsum, c, [] {});
      bwd_chunk_dz<kMasked, kSkip>(s0, mc0 + c0 + 16, limit, gpre, dr, gs, c, pz);
      store(c0 + 16, c, pz);
    }
    if (pair == 0) {
      tmem_ld16(ts + 32, s0);
      if constexpr (!kStored) {   // the carried values after 32 of the 64 columns
        float *rec = reinterpret_cast<float *>(out) + kBM;
        rec[0] = r1 + logsum;
        rec[s2_off] = gpre + gs;
      }
    }
  }
  return ok;
}

// What is recorded as R1 (a log2) where a row has not started: the product is 0, and so is all that follows from it.
constexpr float kNothingLeft = -1e6f;

// The same for a sub-tile before the first key of the warp's rows: dz (and the stored A) are zeros, the scores are not read.
template <bool kStored>
__device__ __forceinline__ bool zero_strip_row(uint8_t *tile_z, int r, int u, uint32_t bars, void *out, long long s2_off) {
  const uint32_t z[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
  const bool ok = mbar_wait(bars + 8u * dq2::bDpFull, u & 1) && mbar_wait(bars + 8u * dq2::bZEmpty, (u + 1) & 1);   // (every phase is followed)
#pragma unroll
  for (int c = 0; c < 64; c += 16) {
    store_packed_chunk16(tile_z, r, c, z);
    if constexpr (kStored) store_packed_global16(reinterpret_cast<unsigned short *>(out) + c, z);
  }
  if constexpr (!kStored) {
    float *rec = reinterpret_cast<float *>(out) + kBM;
    rec[0] = kNothingLeft;
    rec[s2_off] = 0.f;
  }
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(bars + 8u * dq2::bSpEmpty);
  return ok;
}

// =======================================================================================================
// dq kernel: 256 query rows per CTA
// =======================================================================================================
// Two adjacent 128-row query tiles (a, b) share one stream of 64-key K/V sub-tiles, walked from the first key their rows
// reach to tile b's diagonal.  Each tile has its own row-owning warpgroup (warps 0-3 / 4-7), MMA issuer (warps 9 / 10),
// S/dP slots and dQ accumulator in TMEM and dz tile in shared memory.  Per sub-tile and tile: S = Q K^T and
// dP = dO V^T (128 x 64), the row pass (which also records R1/S2 at the sub-tile's first key, i.e. at keys 0 and 64
// of every 128-key tile), then dQ += dz K.
// TMEM columns: S_a 0, dP_a 64, S_b 128, dP_b 192, dQ_a 256, dQ_b 384.
// What bounds it: the row arithmetic (~2700 clk per sub-tile of both tiles in isolation, ~4200 here) and the MMAs'
// shared-memory operand traffic (~80 clk per 128 x 64 x 16 instruction, ~3300 clk at 128 columns), so the two have to
// overlap although S and dP fill all the tensor memory there is and cannot be double-buffered: rows start on S alone, dP
// has until the middle of the first chunk, and both slots are handed back after two thirds of the pass (see strip_row_pass).
namespace dq2 {
constexpr int kThreads = 384;   // three warpgroups (one warp idles)
constexpr int kBN = 64;
constexpr int kKvBox = kBN * 64 * 2;           // 64 keys x 64 columns
constexpr int kZBytes = kBM * kBN * 2;         // dz tile: 128 rows x 64 keys
template <int D>                               // head size rounded up to 64 or 128
struct Cfg {
  static constexpr int kBoxes = D / 64;
  static constexpr int kTileBytes = kBoxes * kBoxBytes;   // Q or dO tile
  static constexpr int kKvTile = kBoxes * kKvBox;         // K or V sub-tile
  static constexpr int kStageBytes = 2 * kKvTile;
  static constexpr int kStages = D == 64 ? 4 : 2;         // what shared memory holds
  static constexpr int kSmem = 1024 + 4 * kTileBytes + kStages * kStageBytes + 2 * kZBytes + 512 + (int)sizeof(SmallTable);
  static_assert(kSmem <= 232448, "shared memory per block");
};
// What the rows need again after their loop, kept out of their registers meanwhile.
struct Shared {
  Ctl ctl;
  int first;     // the sub-tile in stage 0
  int h, hh, len, idx;
  long long tok0, boff, pair0;
};
static_assert(bNum * 8 + sizeof(Shared) <= 512, "barriers and control words");
}  // namespace dq2

template <int D, bool kFp16, bool kStored>
__global__ void __launch_bounds__(dq2::kThreads, 1)
tc_bwd_dq2_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                  const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_g,
                  const __grid_constant__ CUtensorMap tm_dq, const __grid_constant__ CUtensorMap tm_az, const KParams p) {
  using namespace dq2;
  using C = Cfg<D>;
  constexpr int kTileBytes = C::kTileBytes, kKvTile = C::kKvTile, kStageBytes = C::kStageBytes, kStages = C::kStages, kBoxes = C::kBoxes;
  extern __shared__ uint8_t smem_raw[];
  if (threadIdx.x == 0) trace_block(p, 0);
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t *gbase = smem_raw + (base - raw);
  const uint32_t sQ = base;                     // tile w: Q at sQ + w * 2 * kTileBytes, dO right behind it
  const uint32_t sKV = sQ + 4 * kTileBytes;     // stage: K sub-tile then V sub-tile
  const uint32_t sZ = sKV + kStages * kStageBytes;
  const uint32_t sBar = sZ + 2 * kZBytes;
  SmallTable &tb = *reinterpret_cast<SmallTable *>(gbase + (sBar - base) + 512);
  bool refused;
  const long long covered = open_table(p, 2, tb, refused);
  if (covered < p.tokens) fill_rows<typename std::conditional<kFp16, __half, __nv_bfloat16>::type>(p.dq, fill_job(p, covered, refused, blockIdx.x, gridDim.x));
  TileCoord c;
  int hh_blk;
  if (refused || !decode_block(p, tb, 2, true, c, hh_blk)) return;   // c.idx: the even tile of the pair (idx, idx + 1)
  const int Ia = c.idx;
  const bool b_active = Ia + 1 < c.n_tiles;
  Shared *sh = reinterpret_cast<Shared *>(gbase + (sBar - base) + bNum * 8);
  Ctl *ctl = &sh->ctl;
  volatile int *abort_flag = &ctl->abort;
  auto bar = [&](int i) { return sBar + 8u * i; };

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int hh = hh_blk, h = p.head0 + hh;
  const int n_sub = (c.len + kBN - 1) / kBN;
  const int steps_a = min(2 * Ia + 2, n_sub);            // sub-tiles 0 .. 2 Ia + 1 reach tile a's diagonal
  const int steps_b = b_active ? min(2 * Ia + 4, n_sub) : 0;
  const int n_steps = b_active ? steps_b : steps_a;
  const int issuers = b_active ? 2 : 1;
  // the sub-tiles each tile starts at (even numbers: whole key tiles), and the block's: earlier keys have weight exactly 0
  const int first_a = tile_first_key(p, c, p.head0 + hh_blk, Ia, kBM) / kBM * 2;
  const int first_b = b_active ? tile_first_key(p, c, p.head0 + hh_blk, Ia + 1, kBM) / kBM * 2 : first_a;
  const int first = min(first_a, first_b);
  int tr_cur = 0;   // cursor of this thread's event-log lane (diagnostics)

  if (threadIdx.x == 0) {
    mbar_init(bar(bQG), 1);
    mbar_init(bar(bFirst), 1);
    for (int s = 0; s < kStages; ++s) { mbar_init(bar(bKvFull + s), 1); mbar_init(bar(bKvEmpty + s), issuers); }
    for (int w = 0; w < 2; ++w) {
      mbar_init(bar(bSFull + w), 1);
      mbar_init(bar(bDpFull + w), 1);
      mbar_init(bar(bZFull + w), 4);
      mbar_init(bar(bZEmpty + w), kStored ? 2 : 1);   // the dQ MMAs have read the dz tile, and it has left for the workspace
      mbar_init(bar(bSpEmpty + w), 4);
    }
    mbar_init(bar(bDqFull), 1);
    mbar_init(bar(bDqFull + 1), 1);
    ctl->abort = 0;
    sh->first = first; sh->h = h; sh->hh = hh; sh->len = c.len; sh->idx = Ia;
    sh->tok0 = c.tok0; sh->boff = c.boff; sh->pair0 = c.pair0;
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

  // The row warps take over registers the other warpgroup does not need (8 x 32 x 216 + 4 x 32 x 64 of the launch's
  // 12 x 32 x 168): at 168 they spill.
  if (warp >= 8) {
  reg_dec<64>();
  if (warp == 8) {
    if (lane == 0) {
      prefetch_tensormap(&tm_q); prefetch_tensormap(&tm_k); prefetch_tensormap(&tm_v); prefetch_tensormap(&tm_g);
      const int qrow = (int)c.tok0 + Ia * kBM;
      mbar_arrive_expect_tx(bar(bQG), 4 * kTileBytes);
      for (int w = 0; w < 2; ++w)
        for (int kb = 0; kb < kBoxes; ++kb) {
          tma_load_4d(sQ + w * 2 * kTileBytes + kb * kBoxBytes, &tm_q, bar(bQG), kb * 64, qrow + w * kBM, h, (int)c.boff);
          tma_load_4d(sQ + w * 2 * kTileBytes + kTileBytes + kb * kBoxBytes, &tm_g, bar(bQG), kb * 64, qrow + w * kBM, h, (int)c.boff);
        }
      for (int t = 0; t < n_steps - first; ++t) {
        const int st = t % kStages;
        if (t >= kStages && !wait_or_abort(bar(bKvEmpty + st), ((t / kStages) - 1) & 1, abort_flag, p, 510)) break;
        if (*abort_flag) break;
        const int krow = (int)c.tok0 + (first + t) * kBN;
        const uint32_t dst = sKV + st * kStageBytes;
        mbar_arrive_expect_tx(bar(bKvFull + st), kStageBytes);
        for (int kb = 0; kb < kBoxes; ++kb) {
          tma_load_4d(dst + kb * kKvBox, &tm_k, bar(bKvFull + st), kb * 64, krow, h, (int)c.boff);
          tma_load_4d(dst + kKvTile + kb * kKvBox, &tm_v, bar(bKvFull + st), kb * 64, krow, h, (int)c.boff);
        }
      }
    }
  } else if (warp == 9 || warp == 10) {
    // ------------------------------------------------ MMA issuers, one per tile
    const int w = warp - 9;
    if (lane == 0 && w < issuers) {
      constexpr uint32_t idesc_s = idesc_f16(kBM, kBN, kFp16, false, false);
      constexpr uint32_t idesc_dq = idesc_f16(kBM, D, kFp16, false, true);
      const uint32_t qaddr = sQ + w * 2 * kTileBytes, gaddr = qaddr + kTileBytes, zaddr = sZ + w * kZBytes;
      const uint32_t tS = tmem + w * 128, tP = tS + 64, tDQ = tmem + 256 + w * 128;
      // this tile takes part in stages t_first .. t_end - 1 of the block's n_stages; u counts from its first one
      const int n_stages = n_steps - first;
      const int t_first = (w == 0 ? first_a : first_b) - first, t_end = (w == 0 ? steps_a : steps_b) - first;
      const int my_steps = t_end - t_first;
      const int z_row = (int)((c.pair0 + (long long)(Ia + w) * (Ia + w + 1) / 2) * kBM);   // of the stored dz tiles
      auto issue_sp = [&](int u) {
        const uint32_t kaddr = sKV + ((t_first + u) % kStages) * kStageBytes;
        mma_kmajor_kmajor<D, kBoxBytes, kKvBox>(tS, qaddr, kaddr, idesc_s, false);            // S = Q K^T
        mma_commit(bar(bSFull + w));
        mma_kmajor_kmajor<D, kBoxBytes, kKvBox>(tP, gaddr, kaddr + kKvTile, idesc_s, false);  // dP = dO V^T
        mma_commit(bar(bDpFull + w));
      };
      bool ok = true;
      // stages the tile does not read are released on its behalf once they have arrived
      auto release = [&](int t, int t_stop) {
        for (; ok && t < t_stop; ++t) {
          ok = wait_or_abort(bar(bKvFull + t % kStages), (t / kStages) & 1, abort_flag, p, 524);
          if (ok) mbar_arrive(bar(bKvEmpty + t % kStages));
        }
      };
      release(0, t_first);
      ok = ok && wait_or_abort(bar(bQG), 0, abort_flag, p, 520) &&
           wait_or_abort(bar(bKvFull + t_first % kStages), (t_first / kStages) & 1, abort_flag, p, 521);
      // if both tiles start at the same stage, tile b starts once tile a's first scores are done, so that one tile's MMAs fall into the other's row pass
      // (bFirst completes exactly once: this waiter does not follow the phases of tile a's own barriers)
      if (ok && w == 1 && first_a == first_b) ok = wait_or_abort(bar(bFirst), 0, abort_flag, p, 525);
      if (ok) {
        tc_fence_after();
        issue_sp(0);
        if (w == 0) mma_commit(bar(bFirst));
      }
      for (int u = 0; ok && u < my_steps; ++u) {
        // the rows of step u have read their S/dP (they are still computing): the next scores go first ...
        if (u + 1 < my_steps) {
          ok = wait_or_abort(bar(bSpEmpty + w), u & 1, abort_flag, p, 526) &&
               wait_or_abort(bar(bKvFull + (t_first + u + 1) % kStages), ((t_first + u + 1) / kStages) & 1, abort_flag, p, 523);
          if (!ok) break;
          trace_event(p, 1 + 3 * w, tr_cur, 2 + 16 * w, u + 1);
          tc_fence_after();
          issue_sp(u + 1);
          trace_event(p, 1 + 3 * w, tr_cur, 3 + 16 * w, u + 1);
        }
        // ... then, once its dz tile is written, this step's dQ
        ok = wait_or_abort(bar(bZFull + w), u & 1, abort_flag, p, 522);
        if (!ok) break;
        trace_event(p, 1 + 3 * w, tr_cur, 6 + 16 * w, u);
        tc_fence_after();
        // dQ += dz K: dz [128 x 64] K-major, K sub-tile [64 keys x (2 x 64) columns] MN-major
        mma_kmajor_mnmajor<kBN, kKvBox>(tDQ, zaddr, sKV + ((t_first + u) % kStages) * kStageBytes, idesc_dq, u > 0);
        mma_commit(bar(bZEmpty + w));
        mma_commit(bar(bKvEmpty + (t_first + u) % kStages));
        if constexpr (kStored) {
          // The dz tile also leaves for the workspace.  (Issued by the row warps, 32 rows each, these stores held every one of
          // them up for ~900 clk a step; this thread has nothing to do before two thirds of the next pass.)
          const int ub = u + (w == 0 ? first_a : first_b);   // sub-tile inside the sequence
          tma_store_4d(&tm_az, zaddr, (ub & 1) * kBN, z_row + (ub >> 1) * kBM, 1, hh);
          tma_store_commit();
          tma_store_wait_read();
          mbar_arrive(bar(bZEmpty + w));
        }
      }
      if (ok) mma_commit(bar(bDqFull + w));   // this tile's dQ is complete: its rows store it while the other tile goes on
      release(t_end, n_stages);   // tile a does not read the last sub-tiles
      if constexpr (kStored) tma_store_wait_all();
    }
  }
  } else {
    reg_inc<216>();
    // ------------------------------------------------ rows: warpgroup w owns query tile Ia + w
    using T = typename std::conditional<kFp16, __half, __nv_bfloat16>::type;
    const int w = warp >> 2;
    const int r = threadIdx.x & 127;
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    const float scale2 = p.scale * kLog2e;
    const volatile Shared &item = *sh;
    const int I = Ia + w, row0 = I * kBM;
    const int my_steps = w == 0 ? steps_a : steps_b;
    const bool valid = row0 + r < c.len;
    const long long idx = (c.boff * p.heads + h) * p.tokens + c.tok0 + row0 + r;
    // sum of log2(1 - beta) over the keys from the current sub-tile on, as an unevaluated pair (see LogSum in the forward)
    float r1 = 0.f, r1_lo = 0.f, dr = 0.f, gpre = 0.f;
    if (valid && my_steps > 0) {
      const double total = p.log_rem[idx];
      r1 = (float)total;
      r1_lo = (float)(total - (double)r1);
      dr = load_drem<T>(p, idx);
    }
    uint8_t *gZ = gbase + (sZ - base) + w * kZBytes;
    const uint32_t tS = tmem + w * 128 + lane_off, tP = tS + 64;
    const uint32_t bars = sBar + 8u * w;
    // this row's part of the workspace for sub-tile 0: A, or the boundary records [pair (I, J)][quarter of the key tile][row]
    const long long pair00 = (long long)(kStored ? 2 * hh : hh) * p.pairs_cap + c.pair0 + (long long)I * (I + 1) / 2;
    char *out = kStored ? reinterpret_cast<char *>(p.az + (pair00 * kBM + r) * kBM) : reinterpret_cast<char *>(p.bnd_r1 + pair00 * (4 * kBM) + r);
    const int u_diag = 2 * I, u_tail = c.len / kBN;   // a sub-tile with rows past the sequence is number u_tail
    // this warp's rows start at sub-tile u_warp (never, if they are past the sequence): before it, A and dz are zeros
    const int u_warp = row0 + (r & ~31) < c.len ? first_key(p, c, h, row0 + (r & ~31)) / kBN : 0x7fffffff;
    // Where the forward has said where each warp's rows start, hardly a chunk of zeros is left, and the test for them costs
    // every chunk a tenth of its instructions.
    const bool skip = p.tile_start == nullptr && !p.dense;
    const long long s2_off = kStored ? 0 : p.bnd_s2 - p.bnd_r1;
    bool ok = true;
    // One step: `pass` does the rows of sub-tile u, `dst` is its part of this row's workspace.  Zeros up to the warp's first
    // key, then full sub-tiles, then the diagonal: three loops, because what the kinds of step need would otherwise be kept in
    // registers for one another (see the forward's row loop).
    // u: 64-key sub-tile inside the sequence; the first one is even, so that phases follow from u alone
    int u = w == 0 ? first_a : first_b;
    auto step = [&](auto pass, auto tail) {
      ok = wait_or_abort(bars + 8u * bSFull, u & 1, abort_flag, p, 530);
      if (!ok) return;
      if (r == 0) trace_event(p, 2 + w, tr_cur, 4 + 16 * w, u);
      tc_fence_after();
      void *dst = kStored ? out + ((long long)(u >> 1) * (kBM * kBM) + (u & 1) * kBN) * 2 : out + (long long)u * (2 * kBM * sizeof(float));
      if (!pass(dst)) {   // a bounded wait inside the pass gave up
        *abort_flag = 1;
        if (p.status != nullptr) { p.status[0] = SB_DEV_WAIT_TIMEOUT; p.status[1] = 531; }
        ok = false;
      }
      // the sequence ends inside this sub-tile: its dz columns behind the end are exact zeros, the K rows there are
      // not this sequence's (see zero_tile_rows) and are cleared before this step's dz K MMA is released
      if (decltype(tail)::value && u == u_tail)
        zero_tile_rows(gbase + (sKV - base) + ((u - item.first) % kStages) * kStageBytes, item.len - u * kBN, kBN, kBoxes, kKvBox, r, kBM);
      tc_fence_before();          // this step's TMEM reads are done before the slots are handed back
      fence_proxy_async_smem();
      __syncwarp();
      if (r == 0) trace_event(p, 2 + w, tr_cur, 5 + 16 * w, u);
      if (lane == 0) mbar_arrive(bars + 8u * bZFull);
    };
    auto record = [&](void *dst, float r1f) {
      if constexpr (!kStored) {
        reinterpret_cast<float *>(dst)[0] = r1f;
        reinterpret_cast<float *>(dst)[s2_off] = gpre;
      }
    };
    auto carry = [&](float logsum, float gs) {   // r1 += logsum, gpre += gs
      const float sum = r1 + logsum, b = sum - r1;
      r1_lo += (r1 - (sum - b)) + (logsum - b);
      r1 = sum;
      gpre += gs;
    };
    using std::false_type; using std::true_type;
    for (; u < min(u_warp, my_steps) && ok; ++u)
      step([&](void *dst) {
        record(dst, kNothingLeft);
        return zero_strip_row<kStored>(gZ, r, u, bars, dst, s2_off);
      }, true_type());
    // rows past the sequence end must be zero in the stored tiles (the dK/dV GEMMs sum over all 128 query rows): the warp that
    // holds the end masks throughout
    const int u_full = kStored && row0 + (r | 31) >= c.len ? 0 : min(u_diag, my_steps);
    if (!skip) {
      for (; u < u_full && ok; ++u)
        step([&](void *dst) {
          const float r1f = r1 + r1_lo;
          float gs = 0.f, logsum = 0.f;
          record(dst, r1f);
          const bool good = strip_row_pass<kFp16, false, kStored, false>(tS, tP, r, u, 0, 0, scale2, r1f, gpre, dr, gs, logsum, gZ, bars, dst, s2_off);
          carry(logsum, gs);
          return good;
        }, false_type());
    } else {
      for (; u < u_full && ok; ++u)
        step([&](void *dst) {
          const float r1f = r1 + r1_lo;
          float gs = 0.f, logsum = 0.f;
          record(dst, r1f);
          const bool good = strip_row_pass<kFp16, false, kStored, true>(tS, tP, r, u, 0, 0, scale2, r1f, gpre, dr, gs, logsum, gZ, bars, dst, s2_off);
          carry(logsum, gs);
          return good;
        }, false_type());
    }
    for (; u < my_steps && ok; ++u)
      step([&](void *dst) {
        const bool on_diag = u >= u_diag;
        const float r1f = r1 + r1_lo;
        float gs = 0.f, logsum = 0.f;
        record(dst, r1f);
        const bool good = strip_row_pass<kFp16, true, kStored, false>(tS, tP, r, u, on_diag ? (u - u_diag) * kBN : 0,
                                                                      chunk_limit(valid || !kStored, on_diag, r, p.attend_current), scale2, r1f,
                                                                      gpre, dr, gs, logsum, gZ, bars, dst, s2_off);
        carry(logsum, gs);
        return good;
      }, true_type());
    // the dz buffer is reused by the epilogue: its last tile has been read (in stored-tiles mode by the store as well)
    if (ok && my_steps > 0) ok = wait_or_abort(bars + 8u * bZEmpty, (my_steps - 1) & 1, abort_flag, p, 533);
    if (ok && my_steps > 0) ok = wait_or_abort(bar(bDqFull + w), 0, abort_flag, p, 532);
    if (ok && my_steps > 0) {
      tc_fence_after();
      const uint32_t t_acc = tmem + 256 + w * 128 + lane_off;
      const long long tok0 = item.tok0, boff = item.boff;
      const int hd = item.h, tile_row0 = (item.idx + w) * kBM;
      if (tile_row0 + kBM <= item.len) {
        // full tile: two 64-column halves through this tile's dz buffer (its last dQ MMA is done), one TMA store per
        // warp and half -- full lines instead of 16 bytes per thread and row
        const uint32_t src = sZ + w * kZBytes + (warp & 3) * 32 * 128;
        const int trow = (int)tok0 + tile_row0 + (warp & 3) * 32;
#pragma unroll 1
        for (int half = 0; half < (D > 64 && p.head_dim > 64 ? 2 : 1); ++half) {   // columns past head_dim do not exist
#pragma unroll 1
          for (int ch = 0; ch < 2; ++ch) {
            uint32_t v[32];
            tmem_ld32(t_acc + half * 64 + ch * 32, v);
            tmem_wait_ld();
            float x[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) x[i] = __uint_as_float(v[i]) * p.scale;
            store_row_chunk<kFp16>(gZ, r, ch * 32, x);
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_4d(&tm_dq, src, half * 64, trow, hd, (int)boff);
            tma_store_commit();
            tma_store_wait_read();   // the buffer is rewritten by the next half
          }
          __syncwarp();
        }
        if (lane == 0) tma_store_wait_all();
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
  if (warp == 9) tmem_dealloc(tmem, kTmemCols);
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
  using namespace dkv4;
  constexpr int D = 128;
  extern __shared__ uint8_t smem_raw[];
  if (threadIdx.x == 0) trace_block(p, 0);
  SmallTable &tb = *reinterpret_cast<SmallTable *>(smem_raw);   // never used: the launch sees to that, there is no room for it
  bool refused;
  const long long covered = open_table(p, 1, tb, refused);
  if (covered < p.tokens) {
    using T = typename std::conditional<kFp16, __half, __nv_bfloat16>::type;
    fill_rows<T>(p.dk, fill_job(p, covered, refused, blockIdx.x, gridDim.x));
    fill_rows<T>(p.dv, fill_job(p, covered, refused, blockIdx.x, gridDim.x));
  }
  TileCoord c;
  int hh_blk;
  if (refused || !decode_block(p, tb, 1, false, c, hh_blk)) return;
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
          BwdChunk k;
          float pz[16];
          if (masked) {
            bwd_chunk_weights<true, false>(s0, quarter * 32, limit, scale2, r1f, gpre, logsum, k, [] {});
            bwd_chunk_dz<true, false>(d0, quarter * 32, limit, gpre, dr, gs, k, pz);
          } else {
            bwd_chunk_weights<false, true>(s0, 0, limit, scale2, r1f, gpre, logsum, k, [] {}, !p.dense);
            bwd_chunk_dz<false, true>(d0, 0, limit, gpre, dr, gs, k, pz);
          }
          // the A/dz tiles are still being read by the previous step's MMAs
          if (g >= 1) {
            ok = wait_or_abort(bar(bAzEmpty), (g - 1) & 1, abort_flag, p, 631);
            tc_fence_after();
          }
          store_row_chunk16<kFp16>(gA, r, w * 32, k.pa);
          store_row_chunk16<kFp16>(gZ, r, w * 32, pz);
        }
        tmem_wait_ld_regs(s1, d1);
        tc_fence_before();          // this step's TMEM reads are done: the S/dP slot is handed back
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(bSpEmpty + slot));
        if (masked)
          bwd_row_chunk<kFp16, true, false>(s1, d1, w * 32 + 16, quarter * 32 + 16, r, limit, scale2, r1f, gpre, dr, gs, logsum, gA, gZ);
        else
          bwd_row_chunk<kFp16, false, true>(s1, d1, w * 32 + 16, 0, r, limit, scale2, r1f, gpre, dr, gs, logsum, gA, gZ, !p.dense);
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
  using namespace dkv5;
  constexpr int D = 128;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t *gbase = smem_raw + (base - raw);
  const uint32_t sBar = base + kStages * kStageBytes;
  SmallTable &tb = *reinterpret_cast<SmallTable *>(gbase + (sBar - base) + 512 + kListBits / 8);
  bool refused;
  const long long covered = open_table(p, 1, tb, refused);
  if (covered < p.tokens) {
    using T = typename std::conditional<kFp16, __half, __nv_bfloat16>::type;
    fill_rows<T>(p.dk, fill_job(p, covered, refused, blockIdx.x, gridDim.x));
    fill_rows<T>(p.dv, fill_job(p, covered, refused, blockIdx.x, gridDim.x));
  }
  TileCoord c;
  int hh;
  if (refused || !decode_block(p, tb, 1, false, c, hh)) return;
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
  QueryList list{p, c, h, J, kBM, c.n_tiles - J, reinterpret_cast<uint32_t *>(gbase + (sBar - base) + 512)};
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
        const long long pair = c.pair0 + (long long)I * (I + 1) / 2 + J;
        const int az_row = (int)(pair * kBM) + hq * kRows;
        const int qrow = (int)c.tok0 + I * kBM + hq * kRows;
        const uint32_t dst = base + st * kStageBytes;
        mbar_arrive_expect_tx(bar(bFull + st), kStageBytes);
        for (int kb = 0; kb < 2; ++kb) {
          tma_load_4d(dst + (0 + kb) * kBox, &tm_az, bar(bFull + st), kb * 64, az_row, 0, hh);   // A
          tma_load_4d(dst + (2 + kb) * kBox, &tm_az, bar(bFull + st), kb * 64, az_row, 1, hh);   // dz
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
        if (ok && off == list.n - 1 && t % kSub >= clean_from) {
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
    const bool last_listed = list.next(list.n - 1) < list.n;
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
  const dim3 grid((unsigned)item_blocks(p, 1)), grid_pairs((unsigned)item_blocks(p, 2));
  if (!p.skip_dq) {
    const bool narrow = p.head_dim <= 64;
    auto kernel = p.az != nullptr ? (narrow ? tc_bwd_dq2_kernel<64, kFp16, true> : tc_bwd_dq2_kernel<128, kFp16, true>)
                                  : (narrow ? tc_bwd_dq2_kernel<64, kFp16, false> : tc_bwd_dq2_kernel<128, kFp16, false>);
    const int smem = narrow ? dq2::Cfg<64>::kSmem : dq2::Cfg<128>::kSmem;
    if ((e = allow_dynamic_smem(reinterpret_cast<const void *>(kernel), smem)) != cudaSuccess) return e;
    CUtensorMap mk64, mv64;   // 64-row boxes: the kernel streams 64-key sub-tiles
    if ((e = make_tile_map(&mk64, p.k, p, dtype, 64)) != cudaSuccess) return e;
    if ((e = make_tile_map(&mv64, p.v, p, dtype, 64)) != cudaSuccess) return e;
    CUtensorMap mdq, maz128;   // stores: dQ 32 rows per warp, dz one tile at a time
    if ((e = make_tile_map(&mdq, p.dq, p, dtype, 32)) != cudaSuccess) return e;
    if (p.az != nullptr) { if ((e = make_az_map(&maz128, p, dtype, kBM)) != cudaSuccess) return e; }
    else maz128 = mdq;         // not used
    kernel<<<grid_pairs, dq2::kThreads, smem, s>>>(mq, mk64, mv64, mg, mdq, maz128, p);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
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
    kernel<<<grid, dkv5::kThreads, dkv5::kSmem, s>>>(maz, mq64, mg64, mdk, mdv, p);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  } else if (!p.skip_dkv) {
    auto kernel = tc_bwd_dkv4_kernel<kFp16>;
    e = allow_dynamic_smem(reinterpret_cast<const void *>(kernel), dkv4::kSmem);
    if (e != cudaSuccess) return e;
    CUtensorMap mdk, mdv;   // stores: one 64-key strip at a time
    if ((e = make_tile_map(&mdk, p.dk, p, dtype, 64)) != cudaSuccess) return e;
    if ((e = make_tile_map(&mdv, p.dv, p, dtype, 64)) != cudaSuccess) return e;
    kernel<<<grid, dkv4::kThreads, dkv4::kSmem, s>>>(mq, mk, mv, mg, mdk, mdv, p);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// TMA fills the columns past head_dim with zeros, so every head size up to 128 runs the 64- or 128-column kernels.
cudaError_t launch_tc_bwd(const KParams &p, int dtype, cudaStream_t s, int *launches) {
  *launches += (p.skip_dq ? 0 : 1) + (p.skip_dkv ? 0 : 1);
  return dtype == SB_DTYPE_F16 ? launch_bwd_t<true>(p, dtype, s) : launch_bwd_t<false>(p, dtype, s);
}

}  // namespace sb
