// Shared host/device definitions of the stick-breaking attention kernels (sm_100a).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

#include "../../include/sb_b200.h"

namespace sb {

constexpr float kLog2e = 1.4426950408889634f;
constexpr double kLog2eD = 1.4426950408889634074;
constexpr double kLn2D = 0.69314718055994530942;

struct TensorRef {
  char *ptr;
  long long sb, sh, st;  // element strides of batch, head, token
};

// Everything a kernel needs; passed by value.
struct KParams {
  TensorRef q, k, v, o, d_o, dq, dk, dv;
  char *rem;
  const char *d_rem;
  double *log_rem;
  const void *cu;      // sequence end offsets, or nullptr for a fixed-length batch
  int cu64;
  int batch, heads, head_dim, num_seq;
  long long tokens;
  int attend_current;
  float scale;         // logit scale (natural units)
  int head0, head_cnt; // heads [head0, head0 + head_cnt) are processed by this launch
  int tile;            // rows per query tile == keys per key tile of the launch
  int tiles_cap;       // upper bound on the number of query tiles over all sequences
  int n_max;           // upper bound on tiles per sequence
  int max_seqlen;
  int check_leading_zero;  // the element before cu[0] must be 0
  int skip_dq, skip_dkv;   // timing aids: leave one of the two backward kernels out
  int dense;               // measuring aid: do the per-score arithmetic even where it is known to give exact zeros
  int small_table;         // packed batches: every block builds the item table itself (see SmallTable)
  const int2 *order;       // packed batches: work items by descending weight, see decode_item
  int order_span;          // entries of one sequence that stay neighbours in order (>= 1)
  int trace_mode;          // diagnostics builds: bit 1 = log every block's SM, start, first row work and end time
  int dbg;                 // experiments only (SbParams.reserved): 0 = normal arithmetic
  unsigned long long *trace;  // experiments only: event log of block (0,0) in the workspace tail, or nullptr
  // workspace views
  int *hdr;            // [0] cu_seqlens refused, [1] end of the last sequence, [2] entries of order
  unsigned *item_counter;  // hdr[4]: items the workers of a persistent kernel have drawn, or null: fixed assignment
  long long *pair_prefix;  // [num_seq] exclusive prefix of n(n+1)/2 (varlen)
  float *bnd_r1;       // [head_cnt][pairs_cap][tile]  suffix sums of log(1-beta) at tile starts
  float *bnd_s2;       // [head_cnt][pairs_cap][tile]  prefix sums of G before each key tile
  unsigned short *az;  // stored-tiles mode: [head_cnt][pairs_cap][A, dz][128 query rows][128 keys], 16-bit; else null
                       // (CUDA-core kernels: fp32, [head_cnt][pairs_cap][32 query rows][32 A, 32 dz])
  long long pairs_cap;
  // Stored-tiles mode where the tiles of all pairs would not fit, but those that the saved tile starts leave may (see
  // launch_pair_slots): the slots of a query tile's visited pairs follow one another, slot = pair_slot[head][tile_id] + key
  // tile, and `az` holds pairs_cap of them for all heads together.  Null otherwise.
  int *pair_slot;      // [heads][tiles_cap]
  int *pair_span;      // [heads] the most key tiles before its own that a query tile of the head visits
  const int *gate;     // kernels of a launch whose gate_want is not *gate do nothing (null: no gate)
  int gate_want;
  float *attn;         // forward, CUDA-core kernels only: [batch][heads][tokens][attn_cols] attention weights, or null
  long long attn_cols;
  int *tile_start;     // [batch * heads][tile_start_stride]: first key a group of 32 query rows reaches (see first_key), or null
  long long tile_start_stride;
  int fuse_rem_v;      // forward writes o + rem * v; backward folds the two extra gradient terms in
  char *d_rem_fused;   // backward with fuse_rem_v: [batch][heads][tokens] d_rem + <d_out, v> in the tensors' dtype,
                       // written by the first kernel of the call; `d_rem` then points here for the other kernels
  int drem_in_dq;      // ... or formed by the tensor-core dQ kernel, where no other kernel reads it (d_rem may be null then)
  int *status;
};

// One (sequence, query-or-key tile) work item.
struct TileCoord {
  int seq;         // sequence (varlen) or batch element (fixed)
  int idx;         // tile index inside the sequence
  int n_tiles;     // tiles of this sequence
  int len;         // sequence length
  long long tok0;  // first token of the sequence on the tokens axis
  long long boff;  // batch element (fixed) else 0
  long long pair0; // first (query tile, key tile) pair slot of this sequence
};

__device__ __forceinline__ long long load_cu(const KParams &p, int i) {
  return p.cu64 ? reinterpret_cast<const long long *>(p.cu)[i]
                : (long long)reinterpret_cast<const int *>(p.cu)[i];
}

template <typename T> __device__ __forceinline__ float to_f32(T x);
template <> __device__ __forceinline__ float to_f32<float>(float x) { return x; }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }
template <> __device__ __forceinline__ float to_f32<__half>(__half x) { return __half2float(x); }

template <typename T> __device__ __forceinline__ T from_f32(float x);
template <> __device__ __forceinline__ float from_f32<float>(float x) { return x; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }
template <> __device__ __forceinline__ __half from_f32<__half>(float x) { return __float2half_rn(x); }

// Where the group of 32 query rows from row0 on (a multiple of 32, inside the sequence) stopped: keys before this one have
// weight exactly 0 for all of them, and log_rem of these rows covers the keys from it on.  One entry per 32 tokens: a
// sequence's first two groups always reach its first key and have none, the later groups of all packed sequences start at
// least 32 tokens apart.
__device__ __forceinline__ int *tile_start_entry(const KParams &p, const TileCoord &c, int h, int row0) {
  return p.tile_start + (c.boff * p.heads + h) * p.tile_start_stride + ((c.tok0 + row0) >> 5);
}
__device__ __forceinline__ int first_key(const KParams &p, const TileCoord &c, int h, int row0) {
  return p.tile_start == nullptr || row0 < 64 ? 0 : *tile_start_entry(p, c, h, row0);
}
// ... and where query tile I of `tile` rows did.
__device__ __forceinline__ int tile_first_key(const KParams &p, const TileCoord &c, int h, int I, int tile) {
  int first = first_key(p, c, h, I * tile);
  for (int row0 = I * tile + 32; row0 < min((I + 1) * tile, c.len); row0 += 32) first = min(first, first_key(p, c, h, row0));
  return first;
}

// A number for query tile I that no other tile of the call has, below tiles_cap: the tiles of a packed sequence begin at least
// one after where the sequence before them ends.
__device__ __forceinline__ int tile_id(const KParams &p, const TileCoord &c, int I) {
  return (p.cu == nullptr ? c.seq * c.n_tiles : (int)(c.tok0 / p.tile) + c.seq) + I;
}
__device__ __forceinline__ bool gated(const KParams &p) { return p.gate != nullptr && *p.gate != p.gate_want; }

// The query tiles I = J + off that reach key tile J (the others stopped before it), as a bit per tile in shared memory for
// the first kListBits of them; later ones are looked up.  Tile J itself always does.
constexpr int kListBits = 8192;
struct QueryList {
  const KParams &p;
  const TileCoord &c;
  int h, J, tile, n;      // n: query tiles J .. n_tiles - 1, or the first of them if none behind those reaches J
  uint32_t *bits;         // [kListBits / 32]
  __device__ __forceinline__ bool reaches(int off) const { return tile_first_key(p, c, h, J + off, tile) < (J + 1) * tile; }
  // by all threads of the block, before a barrier; one global read per query tile, all in flight together
  __device__ __forceinline__ void build() {
    const int lim = min(n, kListBits), lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    for (int b = (threadIdx.x >> 5) * 32; b < lim; b += warps * 32) {
      const uint32_t w = __ballot_sync(0xffffffffu, b + lane < n && reaches(b + lane));
      if (lane == 0) bits[b >> 5] = w;
    }
  }
  // first listed tile at or after `off`, n if there is none
  __device__ __forceinline__ int next(int off) const {
    while (off < n) {
      if (off >= kListBits) {
        if (reaches(off)) return off;
        ++off;
        continue;
      }
      const uint32_t w = bits[off >> 5] >> (off & 31);
      if (w != 0) return off + __ffs(w) - 1;
      off = (off | 31) + 1;
    }
    return n;
  }
};

// ---- which work items there are ---------------------------------------------------------------------------------------
// Work items (query or key tiles) are ordered by weight across ALL sequences: the tile with the most key (or query) tiles
// to visit comes first, so that the blocks that run longest start earliest and the last blocks of a launch are the short
// ones.  An entry is (sequence, k), k = tile index counted so that larger means heavier.  For a fixed-length batch the order is
// arithmetic.  For a packed batch it is a table, either written by a kernel that runs first (p.order, p.pair_prefix, p.hdr),
// or, for small calls (p.small_table), built by every block for itself in shared memory: a launch and its hand-over cost more
// than the microsecond this takes.
constexpr int kSmallSeqs = 128, kSmallItems = 256;
struct SmallTable {                       // 1.5 KB: what the kernels' shared memory has left
  uint32_t pair0[kSmallSeqs];             // first (query tile, key tile) pair of each sequence; while building: its entries
  uint32_t order[kSmallItems];            // sequence << 16 | entry
};

__device__ __forceinline__ bool seq_valid(const KParams &p, long long start, long long end) {
  return start >= 0 && end >= start && end <= p.tokens && end - start <= p.max_seqlen;
}

// By all threads of the block (at least kSmallSeqs of them); contains barriers.  Returns whether cu_seqlens was refused.
__device__ __forceinline__ bool build_small_table(const KParams &p, SmallTable &tb) {
  const int t = threadIdx.x, span = p.order_span;
  bool bad = false;
  uint32_t n = 0;
  if (t < p.num_seq) {
    const long long start = t == 0 ? 0 : load_cu(p, t - 1), end = load_cu(p, t);
    bad = !seq_valid(p, start, end);
    n = bad ? 0 : (uint32_t)((end - start + p.tile - 1) / p.tile);
    tb.pair0[t] = n;
    if (bad && p.status != nullptr && blockIdx.x == 0) { p.status[0] = SB_DEV_BAD_CU_SEQLENS; p.status[1] = t; }
  }
  if (t == 0 && p.check_leading_zero && load_cu(p, -1) != 0) {
    bad = true;
    if (p.status != nullptr && blockIdx.x == 0) { p.status[0] = SB_DEV_BAD_CU_SEQLENS; p.status[1] = -1; }
  }
  if (__syncthreads_or(bad)) return true;
  // Position of entry e of sequence s: the entries of heavier classes (a class is `span` consecutive entries), then those
  // of the same class in the sequences before, then the heavier ones of its own.
  for (int i = t; i < kSmallItems; i += blockDim.x) tb.order[i] = 0xffffffffu;
  __syncthreads();
  // One pass to find the thread's entry and one to place it: placing the entries while walking the sequences would let a
  // warp run the inner loop once per sequence that its threads hold (8 heads, 16000 tokens in sequences of 32 to 1000: 77 us, now 55).
  for (int i = t; i < kSmallItems; i += blockDim.x) {
    int s = 0, e = i, m = 0;
    for (; s < p.num_seq; ++s) {
      m = (int)tb.pair0[s];
      if (e < m) break;
      e -= m;
    }
    if (s == p.num_seq) break;
    const int lo = e / span * span, hi = lo + span;
    int pos = min(hi, m) - 1 - e;
    for (int q = 0; q < p.num_seq; ++q) {
      const int mq = (int)tb.pair0[q];
      pos += max(mq - hi, 0);
      if (q < s) pos += min(max(mq - lo, 0), span);
    }
    tb.order[pos] = (uint32_t)s << 16 | (uint32_t)e;
  }
  uint32_t before = 0;
  if (t < p.num_seq)
    for (int q = 0; q < t; ++q) before += tb.pair0[q] * (tb.pair0[q] + 1) / 2;
  __syncthreads();
  if (t < p.num_seq) tb.pair0[t] = before;
  __syncthreads();
  return false;
}

// `reverse`: the heavy tiles are the late ones (a query tile sees all earlier keys); otherwise the early ones (a key tile
// is seen by all later queries).
__device__ __forceinline__ bool decode_item(const KParams &p, const SmallTable &tb, int item, bool reverse, TileCoord &c) {
  int s, k;
  if (p.cu == nullptr) {
    const int n = (int)((p.tokens + p.tile - 1) / p.tile);
    if (item >= n * p.batch) return false;
    const int j = item / p.batch;
    s = item - j * p.batch;
    k = n - 1 - j;
    c.n_tiles = n;
    c.len = (int)p.tokens;
    c.tok0 = 0;
    c.boff = s;
    c.pair0 = (long long)s * ((long long)n * (n + 1) / 2);
  } else {
    if (p.small_table) {
      if (item >= kSmallItems) return false;
      const uint32_t e = tb.order[item];
      if (e == 0xffffffffu) return false;
      s = (int)(e >> 16);
      k = (int)(e & 0xffffu);
      c.pair0 = tb.pair0[s];
    } else {
      if (item >= p.hdr[2]) return false;
      const int2 e = p.order[item];
      s = e.x;
      k = e.y;
      c.pair0 = p.pair_prefix[s];
    }
    c.tok0 = s == 0 ? 0 : load_cu(p, s - 1);
    c.len = (int)(load_cu(p, s) - c.tok0);
    c.n_tiles = (c.len + p.tile - 1) / p.tile;
    c.boff = 0;
  }
  c.seq = s;
  c.idx = reverse ? k : c.n_tiles - 1 - k;
  return true;
}
// One-dimensional grids: block = item * head_cnt + head, so that equal-weight items of all heads are neighbours.
__device__ __forceinline__ bool decode_block(const KParams &p, const SmallTable &tb, bool reverse, TileCoord &c, int &hh) {
  const int item = blockIdx.x / p.head_cnt;
  hh = blockIdx.x - item * p.head_cnt;
  return decode_item(p, tb, item, reverse, c);
}

// ---- rows no sequence covers --------------------------------------------------------------------------------------------
// Rows past the end of the last packed sequence get zeros.  When cu_seqlens was refused nothing is computed and every row
// of the outputs is filled with NaN instead, so that a caller who does not look at the status word cannot mistake
// uninitialised memory for results.  Both are done by whichever kernel writes the tensor, each block taking its share.
// (By value and not inlined: a reference would have every kernel copy its parameters to local memory on entry.)
struct FillJob {
  long long tokens, first;   // rows [first, tokens) of heads [head0, head0 + head_cnt)
  int head0, head_cnt, head_dim, block, blocks;
  float value;
};
__device__ __forceinline__ FillJob fill_job(const KParams &p, long long first, bool refused, int block, int blocks) {
  return FillJob{p.tokens, first, p.head0, p.head_cnt, p.head_dim, block, blocks, refused ? __int_as_float(0x7fc00000) : 0.f};
}
template <typename T>
__device__ __noinline__ void fill_rows(TensorRef out, FillJob f) {
  const long long rows = f.tokens - f.first, all = rows * f.head_cnt;
  for (long long i = f.block; i < all; i += f.blocks) {
    const long long h = i / rows, row = f.first + (i - h * rows);
    T *o = reinterpret_cast<T *>(out.ptr) + (f.head0 + h) * out.sh + row * out.st;
    for (int x = threadIdx.x; x < f.head_dim; x += blockDim.x) o[x] = from_f32<T>(f.value);
  }
}
template <typename T>
__device__ __noinline__ void fill_row_state(T *rem, double *log_rem, FillJob f) {
  const long long rows = f.tokens - f.first, all = rows * f.head_cnt;
  for (long long i = (long long)f.block * blockDim.x + threadIdx.x; i < all; i += (long long)f.blocks * blockDim.x) {
    const long long h = i / rows, idx = (f.head0 + h) * f.tokens + f.first + (i - h * rows);
    rem[idx] = from_f32<T>(f.value);
    log_rem[idx] = (double)f.value;
  }
}
template <typename T>
__device__ __forceinline__ void fill_forward_rows(const KParams &p, long long first, bool refused, int block, int blocks) {
  const FillJob f = fill_job(p, first, refused, block, blocks);
  fill_rows<T>(p.o, f);
  fill_row_state<T>(reinterpret_cast<T *>(p.rem), p.log_rem, f);
}
// A kernel's first step: its item table (by all threads; contains barriers for a small packed batch).  Returns the end of
// the last sequence; `refused`: cu_seqlens was, nothing is to be computed and no row counts as covered.
__device__ __forceinline__ long long open_table(const KParams &p, SmallTable &tb, bool &refused) {
  refused = false;
  if (p.cu == nullptr) return p.tokens;
  if (!p.small_table) {
    const int4 h = *reinterpret_cast<const int4 *>(p.hdr);
    refused = h.x != 0;
    return h.y;
  }
  refused = build_small_table(p, tb);
  return refused ? 0 : load_cu(p, p.num_seq - 1);
}

// Blocks to launch for such a grid (an upper bound for packed batches: surplus blocks leave at once).
inline long long item_blocks(const KParams &p) {
  const long long items = p.cu == nullptr ? (p.tokens + p.tile - 1) / p.tile * p.batch : p.tiles_cap;
  return items * p.head_cnt;
}

// Upstream gradient of rem for row `idx` of the (batch, heads, tokens) array.
template <typename T>
__device__ __forceinline__ float load_drem(const KParams &p, long long idx) {
  return to_f32<T>(reinterpret_cast<const T *>(p.d_rem)[idx]);
}

// Kernels follow one another without a gap: each is launched before the one ahead of it has ended (programmatic dependent
// launch) and, as its first step, waits for that; nothing is read or written, no tensor memory taken, before.  kLetGo: the
// next kernel's blocks may take their places as soon as all of this one's have theirs.  That hides a launch's way to the GPU
// (one 200-token forward after the other: 11.7 us without any of this, 9.6) and is right for kernels of few blocks ahead of a
// kernel of many.  Where this kernel's blocks are many or long, the next one's would sit in the places that its SMs have free
// and be spread unevenly over them: kernels that let go / do not, 16 heads x 8 x 2048, d 64: 847 / 826 us forward + backward,
// 2 heads x 131072: 384 / 376; CUDA cores, 7 heads x 500 x 50: 134 / 92 (98 without any of this).
template <bool kLetGo = true>
__device__ __forceinline__ void enter_kernel() {
  if (kLetGo) asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <typename... Params, typename... Args>
inline cudaError_t launch_kernel(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t s, Args &&...args) {
  cudaLaunchAttribute early = {};
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &early;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// Host-side launch helpers implemented in the .cu files; all return cudaError_t of the launch.
cudaError_t launch_fused_drem(const KParams &p, int dtype, cudaStream_t s);   // fills d_rem_fused (all heads)
cudaError_t launch_fused_dv(const KParams &p, int dtype, cudaStream_t s);     // dv += rem * d_out (all heads)
cudaError_t launch_prep(const KParams &p, cudaStream_t s, int *launches);   // the sequence table, where the call needs one
cudaError_t launch_pair_slots(const KParams &p, cudaStream_t s);   // fills pair_slot, pair_span and the gate
cudaError_t launch_simt_fwd(const KParams &p, int dtype, cudaStream_t s, int *launches);
cudaError_t launch_simt_bwd(const KParams &p, int dtype, cudaStream_t s, int *launches);
cudaError_t launch_tc_fwd(const KParams &p, int dtype, cudaStream_t s, int *launches);
cudaError_t launch_tc_bwd(const KParams &p, int dtype, cudaStream_t s, int *launches);
bool tc_supported(int dtype, int head_dim, bool backward);
int tc_tile(int head_dim, bool backward, int max_seqlen);   // rows per work item of the tensor-core kernels
cudaError_t launch_tc_fwd256(const KParams &p, int dtype, cudaStream_t s);
cudaError_t launch_tc_fwd128(const KParams &p, int dtype, cudaStream_t s);
cudaError_t sm_count(int *out);              // SMs of the current device (cached)
cudaError_t allow_dynamic_smem(const void *kernel, int bytes);   // MaxDynamicSharedMemorySize, once per kernel and device

constexpr size_t kTraceBytes = 8 * 1024 * 16;   // workspace tail reserved for the event log

// Event log of block (0,0): each logging thread owns a lane of 1024 entries [tag << 32 | step][SM clock]
// and keeps its own cursor, so that logging costs two stores and no round trip.
#ifdef SB_TRACE
__device__ __forceinline__ void trace_event(const KParams &p, int lane_id, int &cursor, unsigned tag, unsigned step) {
  if (p.trace == nullptr || (p.trace_mode & 2) || blockIdx.x != 0 || blockIdx.y != 0 || cursor >= 1023) return;
  const unsigned long long t = (unsigned long long)clock64();   // SM clock: all logging threads share one SM
  unsigned long long *slot = p.trace + ((size_t)lane_id * 1024 + cursor) * 2;
  slot[0] = ((unsigned long long)tag << 32) | step;
  slot[1] = t;
  ++cursor;
}
// Block schedule log: [linear block id][3] = (globaltimer ns << 10 | SM id) at entry, first row work and exit.
__device__ __forceinline__ void trace_block(const KParams &p, int which) {
  if (p.trace == nullptr || !(p.trace_mode & 2)) return;
  const unsigned lin = blockIdx.y * gridDim.x + blockIdx.x;
  if (lin >= 5400) return;
  unsigned long long t;
  unsigned smid;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
  p.trace[lin * 3 + which] = (t << 10) | smid;
}
#else   // the event log is compiled in only for diagnostic builds (nvcc -DSB_TRACE)
__device__ __forceinline__ void trace_block(const KParams &, int) {}
__device__ __forceinline__ void trace_event(const KParams &, int, int &, unsigned, unsigned) {}
#endif

constexpr int kSimtTile = 32;
constexpr int kTcTile = 128;

}  // namespace sb
