// CUDA-core (fp32 FMA) kernels: the exact path for fp32 tensors and for head sizes the tensor-core
// kernels do not take.  Also holds the sequence-table builder and the elementwise kernels of the fused form.
#include "sb_common.cuh"
#include "sb_ptx.cuh"

namespace sb {

// ------------------------------------------------------------------------------------------------
// Sequence table of the larger packed batches: the first (query tile, key tile) pair of every sequence, and the work items
// by descending weight (see decode_item).
// ------------------------------------------------------------------------------------------------
// The order is a counting sort over classes of `order_span` consecutive tiles, the heaviest class first.  The tiles of one
// sequence inside a class stay neighbours (they read the same keys or queries at about the same time and share them through
// L2); the order of the sequences inside a class is whatever the shared-memory atomics give, which does not matter.
// One block: what bounds it is latency, so every phase is a few steps of 1024 threads.  Sequences of few classes are taken
// one per thread, with one atomic per warp and class; long ones one per warp.  One 131072-token sequence: 8.3 us (one thread
// per sequence and serial prefix sums before: 82 us); 1024 sequences of up to 512 tokens: 9.4 us (16.3).
constexpr int kMaxClasses = 8192;
constexpr int kPrepThreads = 1024;

// Exclusive prefix sum over the block's threads; `total` is the sum over all of them.
template <typename V>
__device__ __forceinline__ V block_exclusive_scan(V x, V *s_warp, V &total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  V incl = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const V up = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += up;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    V w = lane < kPrepThreads / 32 ? s_warp[lane] : V(0);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const V up = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += up;
    }
    s_warp[lane] = w;
  }
  __syncthreads();
  total = s_warp[kPrepThreads / 32 - 1];
  const V before = (warp > 0 ? s_warp[warp - 1] : V(0)) + incl - x;
  __syncthreads();
  return before;
}

__device__ __forceinline__ int seq_tiles(const KParams &p, int s) {
  const long long start = s == 0 ? 0 : load_cu(p, s - 1), end = load_cu(p, s);
  return (int)((end - start + p.tile - 1) / p.tile);
}

__device__ void build_order(const KParams &p, int2 *out, int *s_cls, int *s_warp) {
  const int t = threadIdx.x, lane = t & 31;
  const int span = p.order_span;                         // entries of one sequence that stay neighbours
  const int c_max = (p.n_max + span - 1) / span;         // classes
  if (c_max > kMaxClasses) {   // sequences beyond millions of tokens: sequence by sequence, serially
    if (t == 0) {
      int pos = 0;
      for (int s = 0; s < p.num_seq; ++s)
        for (int j = seq_tiles(p, s) - 1; j >= 0; --j) out[pos++] = make_int2(s, j);
      p.hdr[2] = pos;
    }
    __syncthreads();
    return;
  }
  const bool wide = c_max > 8;   // a warp per sequence, a lane per class; otherwise a thread per sequence
  for (int j = t; j < c_max; j += kPrepThreads) s_cls[j] = 0;
  __syncthreads();
  // one sweep counts the entries of every class, a second one writes them
  auto sweep = [&](bool write) {
    const int step = wide ? kPrepThreads / 32 : kPrepThreads;
    for (int s0 = 0; s0 < p.num_seq; s0 += step) {
      const int s = s0 + (wide ? t >> 5 : t);
      const int m = s < p.num_seq ? seq_tiles(p, s) : 0;
      if (wide) {
        for (int cl = lane; cl * span < m; cl += 32) {
          const int n = min(span, m - cl * span), pos = atomicAdd(&s_cls[cl], n);
          if (write)
            for (int i = 0; i < n; ++i) out[pos + i] = make_int2(s, cl * span + n - 1 - i);   // heaviest first
        }
      } else {
        for (int cl = 0; cl < c_max; ++cl) {   // the same class in all lanes: one atomic per warp
          const int n = min(span, max(m - cl * span, 0));
          int incl = n;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
          }
          const int sum = __shfl_sync(0xffffffffu, incl, 31);
          if (sum == 0) break;
          int base = 0;
          if (lane == 0) base = atomicAdd(&s_cls[cl], sum);
          const int pos = __shfl_sync(0xffffffffu, base, 0) + incl - n;
          if (write)
            for (int i = 0; i < n; ++i) out[pos + i] = make_int2(s, cl * span + n - 1 - i);
        }
      }
    }
  };
  sweep(false);
  __syncthreads();
  // -> first position of every class, the heaviest class first
  int base = 0;
  for (int j0 = 0; j0 < c_max; j0 += kPrepThreads) {
    const int cl = c_max - 1 - (j0 + t);
    const int n = cl >= 0 ? s_cls[cl] : 0;
    int total;
    const int before = block_exclusive_scan(n, s_warp, total);
    if (cl >= 0) s_cls[cl] = base + before;
    base += total;
  }
  if (t == 0) p.hdr[2] = base;
  __syncthreads();
  sweep(true);
  __syncthreads();
}

__global__ void __launch_bounds__(kPrepThreads) prep_kernel(KParams p) {
  enter_kernel();
  __shared__ int s_cls[kMaxClasses];
  __shared__ long long s_warp[32];
  const int t = threadIdx.x;
  const int per = (p.num_seq + kPrepThreads - 1) / kPrepThreads;
  const int s0 = min(p.num_seq, t * per), s1 = min(p.num_seq, s0 + per);
  long long tiles = 0, pairs = 0;
  int bad = -2;
  if (t == 0 && p.check_leading_zero && load_cu(p, -1) != 0) bad = -1;
  for (int s = s0; s < s1; ++s) {
    const long long start = s == 0 ? 0 : load_cu(p, s - 1), end = load_cu(p, s);
    if (!seq_valid(p, start, end)) { if (bad == -2) bad = s; continue; }
    const long long n = (end - start + p.tile - 1) / p.tile;
    tiles += n;
    pairs += n * (n + 1) / 2;
  }
  long long all_tiles, all_pairs;
  block_exclusive_scan(tiles, s_warp, all_tiles);
  long long before = block_exclusive_scan(pairs, s_warp, all_pairs);
  // (more than the workspace holds cannot happen for valid cu_seqlens)
  const bool refused = __syncthreads_or(bad != -2) || all_tiles > p.tiles_cap || all_pairs > p.pairs_cap;
  if (bad != -2 && p.status != nullptr) { p.status[0] = SB_DEV_BAD_CU_SEQLENS; p.status[1] = bad; }
  if (t == 0) {
    p.hdr[0] = refused ? 1 : 0;
    p.hdr[4] = 0;
    p.hdr[1] = refused ? 0 : (int)load_cu(p, p.num_seq - 1);
  }
  if (refused) return;   // no kernel will look at the table
  for (int s = s0; s < s1; ++s) {
    p.pair_prefix[s] = before;
    const long long n = seq_tiles(p, s);
    before += n * (n + 1) / 2;
  }
  build_order(p, const_cast<int2 *>(p.order), s_cls, reinterpret_cast<int *>(s_warp));
}

#ifdef SB_TRACE
__global__ void clear_trace_kernel(unsigned long long *trace) {
  for (int i = threadIdx.x; i < (int)(kTraceBytes / 8); i += blockDim.x) trace[i] = 0;
}
#endif

cudaError_t launch_prep(const KParams &p, cudaStream_t s, int *launches) {
#ifdef SB_TRACE
  if (p.trace != nullptr) clear_trace_kernel<<<1, 32, 0, s>>>(p.trace);
#endif
  if (p.cu == nullptr || p.small_table) return cudaSuccess;
  *launches += 1;
  return launch_kernel(prep_kernel, dim3(1), kPrepThreads, 0, s, p);
}

// Where the stored tiles go if there is room for the visited pairs only: the slots are given out query tile by query tile, and
// whether they suffice is known before the first kernel that would need them -- *gate says so, and the launches for either
// case are made, one of which then does nothing.  One block: latency (two dependent reads per 1024 tiles and heads).
__global__ void __launch_bounds__(kPrepThreads) pair_slots_kernel(KParams p, int *gate) {
  enter_kernel();
  __shared__ int s_warp[32];
  __shared__ SmallTable tb;   // (not used: such calls have a table in memory)
  const int t = threadIdx.x;
  bool refused;
  open_table(p, tb, refused);
  if (refused) {              // the kernels of one of the two launches fill the outputs
    if (t == 0) *gate = 1;
    return;
  }
  for (int h = t; h < p.heads; h += kPrepThreads) p.pair_span[h] = 0;
  __syncthreads();
  const long long items = (p.cu == nullptr ? (p.tokens + p.tile - 1) / p.tile * p.batch : (long long)p.hdr[2]) * p.heads;
  long long base = 0;
  for (long long i0 = 0; i0 < items; i0 += kPrepThreads) {
    const long long i = i0 + t;
    TileCoord c;
    int n = 0, h = 0, first = 0;
    if (i < items && decode_item(p, tb, (int)(i / p.heads), true, c)) {
      h = (int)(i % p.heads);
      first = tile_first_key(p, c, h, c.idx, p.tile) / p.tile;
      n = c.idx + 1 - first;
      atomicMax(&p.pair_span[h], c.idx - first);
    }
    int total;
    const int before = block_exclusive_scan(n, s_warp, total);
    // (slots beyond the room there is are never used)
    if (n > 0) p.pair_slot[(long long)h * p.tiles_cap + tile_id(p, c, c.idx)] = (int)min(base + before, (long long)0x3fffffff) - first;
    base += total;
  }
  if (t == 0) *gate = base <= p.pairs_cap;
}

cudaError_t launch_pair_slots(const KParams &p, cudaStream_t s) {
  return launch_kernel(pair_slots_kernel, dim3(1), kPrepThreads, 0, s, p, const_cast<int *>(p.gate));
}

// Backward with out = o + rem * v: the upstream gradient of rem gains <d_out, v> per row, and dv gains rem * d_out
// (rem = 2^log_rem, from the saved fp64 value) on the rows that belong to a sequence.  Two elementwise kernels over
// the (batch, heads, tokens) rows: grid (token blocks, heads, batch); `group` consecutive lanes share a row, each
// lane holding `kVec` consecutive elements (16 bytes when the rows allow it, else one element).
template <typename T, int kVec>
struct alignas(16) RowVec {
  T e[kVec];
};
template <typename T, int kVec>
__device__ __forceinline__ RowVec<T, kVec> load_vec(const T *src) {
  RowVec<T, kVec> r;
  if (kVec == 1) r.e[0] = *src;
  else *reinterpret_cast<uint4 *>(&r) = *reinterpret_cast<const uint4 *>(src);
  return r;
}

template <typename T, int kVec>
__global__ void __launch_bounds__(256) fused_drem_kernel(KParams p, int group) {
  enter_kernel();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rows_per_warp = 32 / group;
  const long long tok = ((long long)blockIdx.x * 8 + warp) * rows_per_warp + lane / group;
  const int x0 = (lane % group) * kVec;
  const long long h = blockIdx.y, b = blockIdx.z;
  float s = 0.f;
  if (tok < p.tokens) {
    const T *g = reinterpret_cast<const T *>(p.d_o.ptr) + b * p.d_o.sb + h * p.d_o.sh + tok * p.d_o.st;
    const T *v = reinterpret_cast<const T *>(p.v.ptr) + b * p.v.sb + h * p.v.sh + tok * p.v.st;
    for (int x = x0; x < p.head_dim; x += group * kVec) {
      const RowVec<T, kVec> gv = load_vec<T, kVec>(g + x), vv = load_vec<T, kVec>(v + x);
#pragma unroll
      for (int i = 0; i < kVec; ++i) s = fmaf(to_f32<T>(gv.e[i]), to_f32<T>(vv.e[i]), s);
    }
  }
  for (int o = group >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (tok < p.tokens && x0 == 0) {
    const long long row = (b * p.heads + h) * p.tokens + tok;
    reinterpret_cast<T *>(p.d_rem_fused)[row] =
        from_f32<T>(s + (p.d_rem != nullptr ? to_f32<T>(reinterpret_cast<const T *>(p.d_rem)[row]) : 0.f));
  }
}

template <typename T, int kVec>
__global__ void __launch_bounds__(256) fused_dv_kernel(KParams p, int group) {
  enter_kernel();
  if (gated(p)) return;
  if (p.cu != nullptr && p.hdr[0]) return;   // (a small call's table never comes with this kernel)
  const long long covered = p.cu != nullptr ? (long long)p.hdr[1] : p.tokens;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rows_per_warp = 32 / group;
  const long long tok = ((long long)blockIdx.x * 8 + warp) * rows_per_warp + lane / group;
  if (tok >= covered) return;
  const int x0 = (lane % group) * kVec;
  const long long h = blockIdx.y, b = blockIdx.z;
  const T *g = reinterpret_cast<const T *>(p.d_o.ptr) + b * p.d_o.sb + h * p.d_o.sh + tok * p.d_o.st;
  T *dv = reinterpret_cast<T *>(p.dv.ptr) + b * p.dv.sb + h * p.dv.sh + tok * p.dv.st;
  const float rem = exp2f((float)p.log_rem[(b * p.heads + h) * p.tokens + tok]);
  for (int x = x0; x < p.head_dim; x += group * kVec) {
    const RowVec<T, kVec> gv = load_vec<T, kVec>(g + x);
    RowVec<T, kVec> dvv = load_vec<T, kVec>(dv + x);
#pragma unroll
    for (int i = 0; i < kVec; ++i) dvv.e[i] = from_f32<T>(fmaf(rem, to_f32<T>(gv.e[i]), to_f32<T>(dvv.e[i])));
    if (kVec == 1) dv[x] = dvv.e[0];
    else *reinterpret_cast<uint4 *>(dv + x) = *reinterpret_cast<const uint4 *>(&dvv);
  }
}

// 16-byte accesses need rows that start on 16-byte boundaries and hold a whole number of them.
static bool rows_vectorizable(const TensorRef &t, int head_dim, int esize) {
  const long long m = 16 / esize;
  return reinterpret_cast<uintptr_t>(t.ptr) % 16 == 0 && head_dim % m == 0 && t.sb % m == 0 && t.sh % m == 0 && t.st % m == 0;
}

template <typename T, bool kDv>
static cudaError_t launch_fused_t(const KParams &p, cudaStream_t s) {
  constexpr int kVec = 16 / (int)sizeof(T);
  const bool vec = rows_vectorizable(p.d_o, p.head_dim, sizeof(T)) &&
                   rows_vectorizable(kDv ? p.dv : p.v, p.head_dim, sizeof(T));
  const int per_lane = vec ? kVec : 1;
  int group = 1;
  while (group < 32 && group * per_lane < p.head_dim) group <<= 1;
  const long long rows_per_block = 8 * (32 / group);
  const dim3 grid((unsigned)((p.tokens + rows_per_block - 1) / rows_per_block), p.heads, p.batch);
  auto kernel = kDv ? (vec ? fused_dv_kernel<T, kVec> : fused_dv_kernel<T, 1>) : (vec ? fused_drem_kernel<T, kVec> : fused_drem_kernel<T, 1>);
  return launch_kernel(kernel, grid, 256, 0, s, p, group);
}

cudaError_t launch_fused_drem(const KParams &p, int dtype, cudaStream_t s) {
  if (dtype == SB_DTYPE_F32) return launch_fused_t<float, false>(p, s);
  if (dtype == SB_DTYPE_BF16) return launch_fused_t<__nv_bfloat16, false>(p, s);
  return launch_fused_t<__half, false>(p, s);
}

cudaError_t launch_fused_dv(const KParams &p, int dtype, cudaStream_t s) {
  if (dtype == SB_DTYPE_F32) return launch_fused_t<float, true>(p, s);
  if (dtype == SB_DTYPE_BF16) return launch_fused_t<__nv_bfloat16, true>(p, s);
  return launch_fused_t<__half, true>(p, s);
}

// ------------------------------------------------------------------------------------------------
// CUDA-core kernels: fp32 arithmetic throughout, for fp32 tensors and head sizes the tensor-core kernels do not take.
// ------------------------------------------------------------------------------------------------
// What bounds them: latency at three blocks per SM, next to no single unit (one group per block, 2 x 8 heads x 1024 x 64 fp32:
// shared-memory and L1 pipe 59 to 66 % busy, FMA pipe 43 to 47 %, issue slots 41 to 46 %), and the tail of 512 blocks of unequal
// length (a quarter of the SMs' time).  The products' operands come from shared memory: a block is one or two groups of 128
// threads; a product of scores gives each thread a 4 x 4 patch, so that eight 16-byte shared loads feed 64 FMAs, and of an
// accumulator each thread has four rows and a sixteenth of its group's columns.  Per group a step is 32 query rows x 64 keys
// (forward, dQ) or 64 query rows x 32 keys (dK/dV): small enough for three or four blocks of one group per SM at head size 64,
// and for a few heads of a few hundred tokens to spread over the GPU.  The scans over the keys of a row are shared by four
// (dK/dV: two) lanes per 64 (32) keys, 16 keys each.  Next operands are requested while the other product of the step runs:
// cp.async for fp32, registers for 16-bit tensors (which are widened on their way to shared memory).
// Measured, forward + backward: 2 x 8 heads x 1024 tokens, head size 64, fp32: 408 us; one thread per row scanning
// serially and one shared load per FMA before: 2290 us.
// Two groups give the bits of one: what a sequence's results are does not depend on what else is in the launch.  So the groups
// share an accumulator's columns, and a step of 128 keys carries its sums and stops like two of 64.  With half of the keys each
// and a sum over the groups at the end, a shared load fed twice the FMAs (7 heads x 500 x 64, fp32: 118 us instead of 124).
constexpr int kT = kSimtTile;      // 32 rows or keys per tile
template <int DP> constexpr int kLd = DP + 4;   // row stride of an operand tile: 16-byte rows, four banks apart
constexpr int kLdH = kT + 4;       // row stride of a score tile with 32 columns
// A block is G groups of 128 threads, and a step is 64 keys (or query rows) per group (see simt_run for which is taken).
template <int G> constexpr int kThreads = 128 * G;
template <int G> constexpr int kStep = 2 * kT * G;
template <int G> constexpr int kLdS = kStep<G> + 4;            // row stride of a score tile with kStep columns
template <int DP, int G> constexpr int kBlocks = DP == 64 ? (G == 1 ? 3 : 2) : 1;   // blocks per SM the register allocation leaves room for

__device__ __forceinline__ void cp_async16(float *dst, const void *src, bool take) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(take ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async4(float *dst, const void *src, bool take) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(take ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// A tile of ROWS rows of one tensor on its way into shared memory: issue() requests it, land() makes it visible to the
// issuing thread's next barrier.  Rows outside [0, end) become zeros; columns past head_dim are zeroed once by clear().
template <typename T, int DP, int ROWS, int G>
struct TileLoad {
  static constexpr int kWords = ROWS * DP / 2 / kThreads<G>;   // 16-bit tensors: two elements per register
  uint32_t w[sizeof(T) == 4 ? 1 : kWords];

  __device__ __forceinline__ static const T *row_ptr(const TensorRef &t, const TileCoord &c, int h) {
    return reinterpret_cast<const T *>(t.ptr) + c.boff * t.sb + (long long)h * t.sh + c.tok0 * t.st;
  }
  __device__ __forceinline__ void issue(float *dst, const TensorRef &t, const TileCoord &c, int h, int row0, int d, bool wide) {
    issue(dst, t, c, h, row0, d, wide, c.len);
  }
  __device__ __forceinline__ void issue(float *dst, const TensorRef &t, const TileCoord &c, int h, int row0, int d, bool wide, int end) {
    const T *base = row_ptr(t, c, h);
    if constexpr (sizeof(T) == 4) {
      if (wide) {   // rows of whole 16-byte chunks
#pragma unroll 4
        for (int e = threadIdx.x; e < ROWS * (DP / 4); e += kThreads<G>) {
          const int r = e / (DP / 4), x = (e % (DP / 4)) * 4, row = row0 + r;
          const bool take = row >= 0 && row < end;
          if (x < d) cp_async16(dst + r * kLd<DP> + x, base + (take ? row * t.st + x : 0), take);
        }
      } else {
#pragma unroll 4
        for (int e = threadIdx.x; e < ROWS * DP; e += kThreads<G>) {
          const int r = e / DP, x = e % DP, row = row0 + r;
          const bool take = row >= 0 && row < end;
          if (x < d) cp_async4(dst + r * kLd<DP> + x, base + (take ? row * t.st + x : 0), take);
        }
      }
    } else {
      const unsigned short *b16 = reinterpret_cast<const unsigned short *>(base);
#pragma unroll
      for (int i = 0; i < kWords; ++i) {
        const int e = threadIdx.x + i * kThreads<G>;
        const int r = e / (DP / 2), x = (e % (DP / 2)) * 2, row = row0 + r;
        w[i] = 0u;
        if (row >= 0 && row < end && x < d) {
          const unsigned short *src = b16 + row * t.st + x;
          if (wide) w[i] = *reinterpret_cast<const uint32_t *>(src);   // even head size, 4-byte aligned rows
          else w[i] = (uint32_t)src[0] | (x + 1 < d ? (uint32_t)src[1] << 16 : 0u);
        }
      }
    }
  }
  __device__ __forceinline__ void land(float *dst) {
    if constexpr (sizeof(T) == 4) {
      cp_async_wait();
    } else {
#pragma unroll
      for (int i = 0; i < kWords; ++i) {
        const int e = threadIdx.x + i * kThreads<G>;
        const int r = e / (DP / 2), x = (e % (DP / 2)) * 2;
        const unsigned short lo = (unsigned short)(w[i] & 0xffffu), hi = (unsigned short)(w[i] >> 16);
        *reinterpret_cast<float2 *>(dst + r * kLd<DP> + x) =
            make_float2(to_f32<T>(*reinterpret_cast<const T *>(&lo)), to_f32<T>(*reinterpret_cast<const T *>(&hi)));
      }
    }
  }
};
template <int DP, int ROWS, int G>
__device__ __forceinline__ void clear_tile(float *dst, int d) {   // columns past head_dim stay zero from here on
  if (d == DP) return;
  for (int e = threadIdx.x; e < ROWS * DP; e += kThreads<G>) dst[(e / DP) * kLd<DP> + e % DP] = 0.f;
}

// S[m][n] = mul * <A_m, B_n>, M x N with 16 results per thread: thread (ty, tx) owns rows ty + i * (M / 4), columns tx + j * (N / 4).
template <int DP, int M, int N>
__device__ __forceinline__ void tile_dot(float *S, const float *A, const float *B, float mul) {
  constexpr int kTx = N / 4, kTy = M / 4, kLdO = N + 4;
  const int tx = threadIdx.x % kTx, ty = threadIdx.x / kTx;
  float2 acc[4][4] = {};   // even and odd columns: both operands are adjacent pairs, one instruction for two products
  const float *a = A + ty * kLd<DP>, *b = B + tx * kLd<DP>;
#pragma unroll 4
  for (int x = 0; x < DP; x += 4) {
    float4 av[4], bv[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) av[i] = *reinterpret_cast<const float4 *>(a + i * kTy * kLd<DP> + x);
#pragma unroll
    for (int j = 0; j < 4; ++j) bv[j] = *reinterpret_cast<const float4 *>(b + j * kTx * kLd<DP> + x);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[i][j] = ptx::fma2(make_float2(av[i].x, av[i].y), make_float2(bv[j].x, bv[j].y), acc[i][j]);
        acc[i][j] = ptx::fma2(make_float2(av[i].z, av[i].w), make_float2(bv[j].z, bv[j].w), acc[i][j]);
      }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) S[(ty + i * kTy) * kLdO + tx + j * kTx] = (acc[i][j].x + acc[i][j].y) * mul;
}

// A thread's part of a 32-row accumulator: rows 4 ty .. + 3 and, of the group's DP / G columns, kWide next to each other at
// column(u) for every u < kChunks.  Each element is one thread's, who adds its terms up in the order of the keys (query
// rows) as they are walked: one group or two, the sum has the same bits.
template <int DP, int G>
struct Patch {
  static constexpr int kCols = DP / 16 / G, kWide = kCols < 4 ? kCols : 4, kChunks = kCols / kWide;
  float x[4][kCols] = {};
  __device__ __forceinline__ static int row() { return threadIdx.x / 16 % 8 * 4; }
  __device__ __forceinline__ static int column(int u) { return threadIdx.x / 128 * (DP / G) + threadIdx.x % 16 * kWide + 16 * kWide * u; }
  // x[i][..] += s[i] * b[column(u) ..], b: a row of the operand from column(0) on
  __device__ __forceinline__ void add_scaled(const float (&s)[4], const float *b) {
#pragma unroll
    for (int u = 0; u < kChunks; ++u) {
      float2 bv[kWide / 2];
      if constexpr (kWide == 4) {
        const float4 f = *reinterpret_cast<const float4 *>(b + 16 * kWide * u);
        bv[0] = make_float2(f.x, f.y);
        bv[1] = make_float2(f.z, f.w);
      } else {
        bv[0] = *reinterpret_cast<const float2 *>(b + 16 * kWide * u);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int w = 0; w < kWide; w += 2) {   // two columns at a time
          float *a = &x[i][kWide * u + w];
          const float2 r = ptx::fma2(make_float2(s[i], s[i]), bv[w / 2], make_float2(a[0], a[1]));
          a[0] = r.x;
          a[1] = r.y;
        }
    }
  }
};

// acc (32 rows x DP) += P (32 x 64) B (64 x DP): 64 of the step's keys, from key `first` on.  (A trip count that is known only
// as it runs costs the 16-bit kernels, short of registers at 128 columns, a tenth: dQ + dK/dV of 20 bf16 heads x 640 x 100,
// one group, 455 us instead of 409.)
template <int DP, int G>
__device__ __forceinline__ void tile_pv(Patch<DP, G> &acc, const float *P, const float *B, int first) {
  const float *pp = P + acc.row() * kLdS<G> + first, *b = B + first * kLd<DP> + acc.column(0);
#pragma unroll 2
  for (int k = 0; k < 64; k += 4) {
    float4 pv[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) pv[i] = *reinterpret_cast<const float4 *>(pp + i * kLdS<G> + k);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      float sv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) sv[i] = kk == 0 ? pv[i].x : kk == 1 ? pv[i].y : kk == 2 ? pv[i].z : pv[i].w;
      acc.add_scaled(sv, b + (k + kk) * kLd<DP>);
    }
  }
}
// acc (32 keys x DP) += P^T B with P (64 x 32 keys), B (64 x DP): 64 of the step's query rows, from row `first` on
template <int DP, int G>
__device__ __forceinline__ void tile_ptb(Patch<DP, G> &acc, const float *P, const float *B, int first) {
  const float *pp = P + first * kLdH + acc.row(), *b = B + first * kLd<DP> + acc.column(0);
#pragma unroll 4
  for (int k = 0; k < 64; ++k) {
    const float4 pv = *reinterpret_cast<const float4 *>(pp + k * kLdH);
    const float sv[4] = {pv.x, pv.y, pv.z, pv.w};
    acc.add_scaled(sv, b + k * kLd<DP>);
  }
}

// One lane's 16 keys of a row: beta and 1 - beta per key, and the sum of softplus(z) over the allowed ones.
//   u = e^-|z|, t = 1 + u in (1, 2]:  beta = (z > 0 ? 1 : u) / t,  1 - beta = (z > 0 ? u : 1) / t,
//   softplus(z) = max(z, 0) + log t;  16 factors t share one logarithm.  What the roundings of 1 + u and of the product
//   dropped is carried along (`rest`, exact to first order) and comes back as rest / prod, so that the sum is as good as
//   16 log1p.  (Without the product's part a head whose scores lie around -12 loses the factors near 1 altogether: log_rem
//   off by 7e-5 instead of 2e-8.)
// Keys [key0, key0 + 16) below `limit` are allowed, negative ones never.
__device__ __forceinline__ float stick_segment(float (&z)[16], int key0, int limit, float (&beta)[16], float (&keep)[16]) {
  float lin = 0.f, prod = 1.f, rest = 0.f;   // the product of the exact factors is prod + rest
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const bool on = key0 + j >= 0 && key0 + j < limit;
    const float u = expf(-fabsf(z[j])), t = 1.f + u, rt = __frcp_rn(t);
    const bool pos = z[j] > 0.f;
    beta[j] = on ? (pos ? rt : u * rt) : 0.f;
    keep[j] = on ? (pos ? u * rt : rt) : 1.f;
    lin += on && pos ? z[j] : 0.f;
    const float factor = on ? t : 1.f, dropped = on ? u - (t - 1.f) : 0.f, next = prod * factor;
    rest = fmaf(rest, factor, fmaf(prod, dropped, fmaf(prod, factor, -next)));
    prod = next;
  }
  return lin + (logf(prod) + rest * __frcp_rn(prod));
}
__device__ __forceinline__ void load16(float (&x)[16], const float *src) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 f = *reinterpret_cast<const float4 *>(src + 4 * i);
    x[4 * i] = f.x; x[4 * i + 1] = f.y; x[4 * i + 2] = f.z; x[4 * i + 3] = f.w;
  }
}
__device__ __forceinline__ void store16(float *dst, const float (&x)[16]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) *reinterpret_cast<float4 *>(dst + 4 * i) = make_float4(x[4 * i], x[4 * i + 1], x[4 * i + 2], x[4 * i + 3]);
}

// Forward: one block per (sequence, 32-row query tile, head), keys walked from the diagonal back to the sequence start in
// steps of 64 per group; every row carries sum softplus(z) over the keys already visited, in fp64 (reference: _forward_one_row,
// sb_varlen_fwd.py:81-215).
template <typename T, int DP, int G>
__global__ void __launch_bounds__(kThreads<G>, kBlocks<DP, G>) simt_fwd_kernel(const __grid_constant__ KParams p, bool wide) {
  enter_kernel<false>();
  extern __shared__ float4 smem4[];
  __shared__ SmallTable tb;
  bool refused;
  const long long covered = open_table(p, tb, refused);
  const int block = blockIdx.y * gridDim.x + blockIdx.x, blocks = gridDim.x * gridDim.y;
  if (covered < p.tokens) fill_forward_rows<T>(p, covered, refused, block, blocks);
  TileCoord c;
  if (refused || !decode_item(p, tb, blockIdx.x, true, c)) return;
  const int d = p.head_dim, h = p.head0 + blockIdx.y, t = threadIdx.x;
  float *Qs = reinterpret_cast<float *>(smem4), *Ks = Qs + kT * kLd<DP>, *Vs = Ks + kStep<G> * kLd<DP>, *Ss = Vs + kStep<G> * kLd<DP>;
  const int row0 = c.idx * kT, ac = p.attend_current;
  constexpr int kLanes = 4 * G;
  const int r = t / kLanes, seg = t % kLanes, gi = row0 + r;   // the row this thread scans, and which 16 of the step's keys
  const int limit = gi < c.len ? gi + ac : 0;

  clear_tile<DP, kT, G>(Qs, d);
  clear_tile<DP, kStep<G>, G>(Ks, d);
  clear_tile<DP, kStep<G>, G>(Vs, d);
  if (d != DP) __syncthreads();
  TileLoad<T, DP, kT, G> lq;
  TileLoad<T, DP, kStep<G>, G> lk, lv;
  int key0 = row0 + kT - kStep<G>;          // first key of the step (negative: keys before the sequence, masked)
  lq.issue(Qs, p.q, c, h, row0, d, wide);
  lk.issue(Ks, p.k, c, h, key0, d, wide);
  lq.land(Qs);
  lk.land(Ks);
  __syncthreads();
  Patch<DP, G> acc;
  double run = 0.0;                         // sum of softplus(z) over the keys visited
  const bool may_stop = p.tile_start != nullptr && !p.dense;
  int reached = 0;                          // first key visited
  for (; key0 > -kStep<G>; key0 -= kStep<G>) {
    lv.issue(Vs, p.v, c, h, key0, d, wide);
    tile_dot<DP, kT, kStep<G>>(Ss, Qs, Ks, p.scale);
    lv.land(Vs);
    __syncthreads();
    bool more = key0 > 0;
    if (more) lk.issue(Ks, p.k, c, h, key0 - kStep<G>, d, wide);
    double mid = 0.0;                       // two groups: `run` after the later 64 keys of the step
    {
      float z[16], beta[16], keep[16];
      float *srow = Ss + r * kLdS<G> + seg * 16;
      load16(z, srow);
      const float sp = stick_segment(z, key0 + seg * 16, limit, beta, keep);
      float prod = 1.f;
#pragma unroll
      for (int j = 0; j < 16; ++j) prod *= keep[j];
      // product over the lanes with later keys of the same 64, then down the lane's own keys
      const float p1 = __shfl_down_sync(0xffffffffu, prod, 1, 4), p2 = __shfl_down_sync(0xffffffffu, prod, 2, 4),
                  p3 = __shfl_down_sync(0xffffffffu, prod, 3, 4);
      // (in fp64: the backward subtracts its own sums from log_rem, and what an fp32 sum over the lanes rounds off is seen there)
      double sum = (double)sp;
      sum += __shfl_xor_sync(0xffffffffu, sum, 1);
      sum += __shfl_xor_sync(0xffffffffu, sum, 2);
      double from = run;                    // ... over the keys after this lane's 64
      if (G == 2) {
        const double other = __shfl_xor_sync(0xffffffffu, sum, 4);
        mid = run + (seg >= 4 ? sum : other);
        if (seg < 4) from = mid;
        run = mid + (seg >= 4 ? other : sum);
      } else {
        run += sum;
      }
      float R = expf(-(float)from);
      if ((seg & 3) < 3) R *= p1;
      if ((seg & 3) < 2) R *= p2;
      if ((seg & 3) < 1) R *= p3;
#pragma unroll
      for (int j = 15; j >= 0; --j) {
        z[j] = beta[j] * R;
        R *= keep[j];
      }
      store16(srow, z);
    }
    // Once every row's product has underflowed to 0, no earlier key has any weight.  With two groups a step is two of one
    // group's: the tile stops where one group's would.
    int from_key = 0;                       // the first key of the step that is visited, counted from key0
    if (may_stop && G == 2 && !__syncthreads_or(gi < c.len && expf(-(float)mid) != 0.f) && key0 + 64 > 0) {
      more = false;
      reached = key0 + 64;
      run = mid;
      from_key = 64;
    } else if (may_stop) {
      if (!__syncthreads_or(gi < c.len && expf(-(float)run) != 0.f) && more) {
        more = false;
        reached = key0;
      }
    } else {
      __syncthreads();
    }
    if (p.attn != nullptr) {   // debugging aid: the attention weights of this step, keys indexed inside the sequence
      for (int e = t; e < kT * kStep<G>; e += kThreads<G>) {
        const int ri = row0 + e / kStep<G>, gj = key0 + e % kStep<G>;
        if (ri < c.len && gj >= 0 && e % kStep<G> >= from_key && gj < c.len && gj < p.attn_cols)
          p.attn[((c.boff * p.heads + h) * p.tokens + c.tok0 + ri) * p.attn_cols + gj] = Ss[(e / kStep<G>) * kLdS<G> + e % kStep<G>];
      }
    }
    if (G == 2) tile_pv(acc, Ss, Vs, 64);   // the later keys first
    if (G == 1 || (from_key == 0 && key0 + 64 > 0)) tile_pv(acc, Ss, Vs, 0);
    if (!more) break;
    lk.land(Ks);
    __syncthreads();
  }
  if constexpr (sizeof(T) == 4) cp_async_wait();   // keys requested before the stop was known
  __syncthreads();
  if (p.tile_start != nullptr && t == 0 && row0 >= 64) *tile_start_entry(p, c, h, row0) = reached;

  const float rem = expf(-(float)run);
  if (seg == 0 && gi < c.len) {
    const long long idx = (c.boff * p.heads + h) * p.tokens + c.tok0 + gi;
    reinterpret_cast<T *>(p.rem)[idx] = from_f32<T>(rem);
    p.log_rem[idx] = -run * kLog2eD;
  }
  if (p.fuse_rem_v) {   // out = o + rem * v: the row owners publish rem through the free score tile
    if (seg == 0) Ss[r] = rem;
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = row0 + acc.row() + i;
    if (row >= c.len) continue;
    T *o = reinterpret_cast<T *>(p.o.ptr) + c.boff * p.o.sb + (long long)h * p.o.sh + (c.tok0 + row) * p.o.st;
    const T *v = reinterpret_cast<const T *>(p.v.ptr) + c.boff * p.v.sb + (long long)h * p.v.sh + (c.tok0 + row) * p.v.st;
#pragma unroll
    for (int u = 0; u < acc.kChunks; ++u)
#pragma unroll
      for (int x = 0; x < acc.kWide; ++x) {
        const int col = acc.column(u) + x;
        const float sum = acc.x[i][acc.kWide * u + x];
        if (col < d) o[col] = from_f32<T>(p.fuse_rem_v ? fmaf(Ss[acc.row() + i], to_f32<T>(v[col]), sum) : sum);
      }
  }
}

// The backward of one lane's 16 keys: z, dP in; dz, A out.  LANES lanes share a row's keys of a step, or, with G == 2, of
// either half of it; the second half goes on where the first one ends, as the next step of one group would.
// r1: minus the sum of softplus over the allowed keys from the step's first key on; gpre: sum of G over the keys before it;
// on return the same for the next step.  r1_seg / g_seg: both at this lane's first key.
template <int LANES, int G>
__device__ __forceinline__ void bwd_segment(float (&z)[16], float (&dp)[16], int key0, int limit, double &r1, float &gpre, float dr,
                                            double &r1_seg, float &g_seg) {
  const int lane = threadIdx.x & (LANES - 1);
  const bool second = G == 2 && (threadIdx.x & LANES);
  float beta[16], keep[16];
  const float own = stick_segment(z, key0, limit, beta, keep);
  double incl = own;                       // through this lane's last key
#pragma unroll
  for (int o = 1; o < LANES; o <<= 1) {
    const double up = __shfl_up_sync(0xffffffffu, incl, o, LANES);
    if (lane >= o) incl += up;
  }
  const double sp = __shfl_sync(0xffffffffu, incl, LANES - 1, LANES);
  const double sp_other = G == 2 ? __shfl_xor_sync(0xffffffffu, sp, LANES) : 0.0;
  if (second) r1 += sp_other;
  r1_seg = r1 + (incl - (double)own);
  float W = expf((float)(r1 + incl));      // product of (1 - beta) over the keys after this lane's
  r1 += sp;
  if (G == 2 && !second) r1 += sp_other;
  float loc = 0.f;
#pragma unroll
  for (int j = 15; j >= 0; --j) {
    const float a = beta[j] * W;
    W *= keep[j];
    z[j] = a;
    dp[j] = a != 0.f ? a * (dp[j] - dr) : 0.f;   // a row or key outside the sequence carries nothing over
  }
#pragma unroll
  for (int j = 0; j < 16; ++j) loc += dp[j];
  float gi = loc;
#pragma unroll
  for (int o = 1; o < LANES; o <<= 1) {
    const float up = __shfl_up_sync(0xffffffffu, gi, o, LANES);
    if (lane >= o) gi += up;
  }
  const float gs = __shfl_sync(0xffffffffu, gi, LANES - 1, LANES);
  const float gs_other = G == 2 ? __shfl_xor_sync(0xffffffffu, gs, LANES) : 0.f;
  const float before = __shfl_up_sync(0xffffffffu, gi, 1, LANES);
  if (second) gpre += gs_other;
  g_seg = gpre + (lane > 0 ? before : 0.f);
  float C = g_seg;
  gpre += gs;
  if (G == 2 && !second) gpre += gs_other;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const float g = dp[j];
    C += g;
    dp[j] = z[j];                          // A
    z[j] = fmaf(-beta[j], C, g);           // dz
  }
}

// dQ: query-stationary, keys from the sequence start to the diagonal (reference: _backward_one_row,
// sb_varlen_bwd.py:297-481, which adds dK/dV under a spin lock instead).  Leaves A and dz of every (query tile, key tile)
// pair in the workspace (p.az), or, where those would not fit the scratch budget, the carried R1 and S2 per pair and row.
template <typename T, int DP, int G>
__global__ void __launch_bounds__(kThreads<G>, kBlocks<DP, G>) simt_bwd_dq_kernel(const __grid_constant__ KParams p, bool wide) {
  enter_kernel<false>();
  extern __shared__ float4 smem4[];
  __shared__ SmallTable tb;
  bool refused;
  const long long covered = open_table(p, tb, refused);
  const int block = blockIdx.y * gridDim.x + blockIdx.x, blocks = gridDim.x * gridDim.y;
  if (covered < p.tokens) fill_rows<T>(p.dq, fill_job(p, covered, refused, block, blocks));
  TileCoord c;
  if (refused || !decode_item(p, tb, blockIdx.x, true, c)) return;
  const int d = p.head_dim, hh = blockIdx.y, h = p.head0 + hh, t = threadIdx.x;
  float *Qs = reinterpret_cast<float *>(smem4), *Gs = Qs + kT * kLd<DP>, *Ks = Gs + kT * kLd<DP>, *Vs = Ks + kStep<G> * kLd<DP>;
  // the scores, later dz, and dP; with two groups dP follows the scores into the one tile, so that two blocks fit an SM
  float *Zs = Vs + kStep<G> * kLd<DP>, *Ps = G == 1 ? Zs + kT * kLdS<G> : Zs;
  const int I = c.idx, row0 = I * kT;
  constexpr int kLanes = 4 * G;
  const int r = t / kLanes, seg = t % kLanes, gi = row0 + r;
  const int limit = gi < c.len ? gi + p.attend_current : 0;

  clear_tile<DP, kT, G>(Qs, d);
  clear_tile<DP, kT, G>(Gs, d);
  clear_tile<DP, kStep<G>, G>(Ks, d);
  clear_tile<DP, kStep<G>, G>(Vs, d);
  if (d != DP) __syncthreads();
  TileLoad<T, DP, kT, G> lq, lg;
  TileLoad<T, DP, kStep<G>, G> lk, lv;
  lq.issue(Qs, p.q, c, h, row0, d, wide);
  lg.issue(Gs, p.d_o, c, h, row0, d, wide);
  const int key_first = first_key(p, c, h, row0);
  // The last step runs past the tile.  dz is 0 there, and so is K to be: whatever later tokens hold, it is none of these rows'.
  const int key_end = min(c.len, row0 + kT);
  lk.issue(Ks, p.k, c, h, key_first, d, wide, key_end);
  lq.land(Qs);
  lg.land(Gs);
  lk.land(Ks);
  double r1 = 0.0;
  float gpre = 0.f, dr = 0.f;
  if (gi < c.len) {
    const long long idx = (c.boff * p.heads + h) * p.tokens + c.tok0 + gi;
    r1 = p.log_rem[idx] * kLn2D;
    dr = load_drem<T>(p, idx);
  }
  __syncthreads();
  Patch<DP, G> acc;
  const long long pair0 = (long long)hh * p.pairs_cap + c.pair0 + (long long)I * (I + 1) / 2;
  for (int key0 = key_first; key0 <= row0; key0 += kStep<G>) {
    lv.issue(Vs, p.v, c, h, key0, d, wide);
    tile_dot<DP, kT, kStep<G>>(Zs, Qs, Ks, p.scale);
    lv.land(Vs);
    __syncthreads();
    float z[16], dp[16];
    float *zrow = Zs + r * kLdS<G> + seg * 16;
    if (G > 1) {
      load16(z, zrow);
      __syncthreads();
    }
    tile_dot<DP, kT, kStep<G>>(Ps, Gs, Vs, 1.f);
    __syncthreads();
    // V is done with: the next K goes into its buffer while this step goes on, and the next V into this K's
    const bool more = key0 + kStep<G> <= row0;
    if (more) lk.issue(Vs, p.k, c, h, key0 + kStep<G>, d, wide, key_end);
    {
      if (G == 1) load16(z, zrow);
      load16(dp, Ps + r * kLdS<G> + seg * 16);
      double r1_seg;
      float g_seg;
      bwd_segment<4, G>(z, dp, key0 + seg * 16, limit, r1, gpre, dr, r1_seg, g_seg);
      store16(zrow, z);
      const int J = key0 / kT + (seg >> 1);
      if (J <= I) {
        if (p.az != nullptr) {
          float *az = reinterpret_cast<float *>(p.az) + ((pair0 + J) * kT + r) * (2 * kT) + (seg & 1) * 16;   // row: A, then dz
          store16(az, dp);
          store16(az + kT, z);
        } else if ((seg & 1) == 0) {
          p.bnd_r1[(pair0 + J) * kT + r] = (float)r1_seg;
          p.bnd_s2[(pair0 + J) * kT + r] = g_seg;
        }
      }
    }
    __syncthreads();
    tile_pv(acc, Zs, Ks, 0);
    if (G == 2 && key0 + 64 <= row0) tile_pv(acc, Zs, Ks, 64);
    if (more) lk.land(Vs);
    __syncthreads();
    float *tmp = Ks;
    Ks = Vs;
    Vs = tmp;
  }

#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = row0 + acc.row() + i;
    if (row >= c.len) continue;
    T *o = reinterpret_cast<T *>(p.dq.ptr) + c.boff * p.dq.sb + (long long)h * p.dq.sh + (c.tok0 + row) * p.dq.st;
#pragma unroll
    for (int u = 0; u < acc.kChunks; ++u)
#pragma unroll
      for (int x = 0; x < acc.kWide; ++x) {
        const int col = acc.column(u) + x;
        if (col < d) o[col] = from_f32<T>(acc.x[i][acc.kWide * u + x] * p.scale);
      }
  }
}

// dK, dV: key-stationary, one block per 32-key tile, query tiles diagonal -> end two per group at a time; accumulators in registers,
// fixed summation order, no atomics.  kStored: A and dz come from the workspace; otherwise they are computed again.
template <typename T, int DP, int G, bool kStored>
__global__ void __launch_bounds__(kThreads<G>, kBlocks<DP, G>) simt_bwd_dkv_kernel(const __grid_constant__ KParams p, bool wide) {
  enter_kernel<false>();
  extern __shared__ float4 smem4[];
  __shared__ SmallTable tb;
  bool refused;
  const long long covered = open_table(p, tb, refused);
  const int block = blockIdx.y * gridDim.x + blockIdx.x, blocks = gridDim.x * gridDim.y;
  if (covered < p.tokens) {
    fill_rows<T>(p.dk, fill_job(p, covered, refused, block, blocks));
    fill_rows<T>(p.dv, fill_job(p, covered, refused, block, blocks));
  }
  TileCoord c;
  if (refused || !decode_item(p, tb, blockIdx.x, false, c)) return;
  const int d = p.head_dim, hh = blockIdx.y, h = p.head0 + hh, t = threadIdx.x;
  float *Qs = reinterpret_cast<float *>(smem4), *Gs = Qs + kStep<G> * kLd<DP>, *Zs = Gs + kStep<G> * kLd<DP>, *Ps = Zs + kStep<G> * kLdH;
  float *Ks = Ps + kStep<G> * kLdH, *Vs = Ks + kT * kLd<DP>;   // recomputation only
  const int J = c.idx;
  __shared__ uint32_t list_bits[kListBits / 32];
  QueryList list{p, c, h, J, kT, c.n_tiles - J, list_bits};
  list.build();

  constexpr int kTiles = 2 * G;   // query tiles per step
  clear_tile<DP, kStep<G>, G>(Qs, d);
  clear_tile<DP, kStep<G>, G>(Gs, d);
  TileLoad<T, DP, kT, G> lq[kTiles], lg[kTiles];
  if constexpr (!kStored) {
    clear_tile<DP, kT, G>(Ks, d);
    clear_tile<DP, kT, G>(Vs, d);
    if (d != DP) __syncthreads();
    TileLoad<T, DP, kT, G> lk, lv;
    lk.issue(Ks, p.k, c, h, J * kT, d, wide);
    lv.issue(Vs, p.v, c, h, J * kT, d, wide);
    lk.land(Ks);
    lv.land(Vs);
  }
  __syncthreads();
  Patch<DP, G> dk, dv;
  // The next query tiles that reach this key tile (n_tiles where there are no more: rows past the sequence, zeros).
  int off = 0, I[kTiles];
  auto advance = [&](int from) {
    off = list.next(from);
    int o = off;
#pragma unroll
    for (int i = 0; i < kTiles; ++i) {
      I[i] = J + o;
      o = list.next(o + 1);
    }
  };
  advance(0);
  auto load_rows = [&](TileLoad<T, DP, kT, G> (&l)[kTiles], float *dst, const TensorRef &x) {
#pragma unroll
    for (int i = 0; i < kTiles; ++i) l[i].issue(dst + i * kT * kLd<DP>, x, c, h, I[i] * kT, d, wide);
  };
  auto land_rows = [&](TileLoad<T, DP, kT, G> (&l)[kTiles], float *dst) {
#pragma unroll
    for (int i = 0; i < kTiles; ++i) l[i].land(dst + i * kT * kLd<DP>);
  };
  if constexpr (kStored) {
    auto load_stored = [&](float *dst, int part) {   // the query rows of A (part 0) or dz (part 1): 8 float4 per row
#pragma unroll
      for (int i = 0; i < kStep<G> * 8 / kThreads<G>; ++i) {
        const int e = t + i * kThreads<G>, row = e >> 3, x = (e & 7) * 4;
        const int Ir = I[i * kThreads<G> / (8 * kT)];
        const bool take = Ir < c.n_tiles;
        const long long pair = (long long)hh * p.pairs_cap + c.pair0 + (long long)Ir * (Ir + 1) / 2 + J;
        const float *src = reinterpret_cast<const float *>(p.az) + (take ? (pair * kT + (row & 31)) * (2 * kT) + part * kT + x : 0);
        cp_async16(dst + row * kLdH + x, src, take);
      }
    };
    // the operands of either product arrive while the other one runs
    load_rows(lq, Qs, p.q);
    load_stored(Zs, 1);
    while (off < list.n) {
      land_rows(lq, Qs);
      cp_async_wait();
      __syncthreads();
      load_rows(lg, Gs, p.d_o);
      load_stored(Ps, 0);
      const bool wider = G == 2 && I[2 * (G - 1)] < c.n_tiles;   // there is a third tile
      tile_ptb(dk, Zs, Qs, 0);
      if (wider) tile_ptb(dk, Zs, Qs, 64);
      land_rows(lg, Gs);
      cp_async_wait();
      __syncthreads();
      advance(I[kTiles - 1] - J + 1);
      if (off < list.n) {
        load_rows(lq, Qs, p.q);
        load_stored(Zs, 1);
      }
      tile_ptb(dv, Ps, Gs, 0);
      if (wider) tile_ptb(dv, Ps, Gs, 64);
    }
  } else {
    static_assert(kStored || G == 1, "64 query rows per step, the 32 keys of a row shared by two lanes");
    for (; off < list.n; advance(I[kTiles - 1] - J + 1)) {
      load_rows(lq, Qs, p.q);
      load_rows(lg, Gs, p.d_o);
      land_rows(lq, Qs);
      land_rows(lg, Gs);
      __syncthreads();
      tile_dot<DP, kStep<G>, kT>(Zs, Qs, Ks, p.scale);
      tile_dot<DP, kStep<G>, kT>(Ps, Gs, Vs, 1.f);
      __syncthreads();
      const int row = t >> 1, seg = t & 1, Ir = row < kT ? I[0] : I[1], gi = Ir * kT + (row & 31);
      double r1 = 0.0;
      float gpre = 0.f, dr = 0.f;
      if (gi < c.len) {
        const long long slot = ((long long)hh * p.pairs_cap + c.pair0 + (long long)Ir * (Ir + 1) / 2 + J) * kT + (row & 31);
        r1 = p.bnd_r1[slot];
        gpre = p.bnd_s2[slot];
        dr = load_drem<T>(p, (c.boff * p.heads + h) * p.tokens + c.tok0 + gi);
      }
      float z[16], dp[16];
      load16(z, Zs + row * kLdH + seg * 16);
      load16(dp, Ps + row * kLdH + seg * 16);
      double r1_seg;
      float g_seg;
      bwd_segment<2, 1>(z, dp, J * kT + seg * 16, gi < c.len ? gi + p.attend_current : 0, r1, gpre, dr, r1_seg, g_seg);
      store16(Zs + row * kLdH + seg * 16, z);
      store16(Ps + row * kLdH + seg * 16, dp);
      __syncthreads();
      tile_ptb(dk, Zs, Qs, 0);
      tile_ptb(dv, Ps, Gs, 0);
      __syncthreads();
    }
  }

#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int key = J * kT + dk.row() + i;
    if (key >= c.len) continue;
    T *ok = reinterpret_cast<T *>(p.dk.ptr) + c.boff * p.dk.sb + (long long)h * p.dk.sh + (c.tok0 + key) * p.dk.st;
    T *ov = reinterpret_cast<T *>(p.dv.ptr) + c.boff * p.dv.sb + (long long)h * p.dv.sh + (c.tok0 + key) * p.dv.st;
    // out = o + rem * v was requested: dV gains rem * d_out on its own row (rem = 2^log_rem)
    const T *g = reinterpret_cast<const T *>(p.d_o.ptr) + c.boff * p.d_o.sb + (long long)h * p.d_o.sh + (c.tok0 + key) * p.d_o.st;
    const float rem = p.fuse_rem_v ? exp2f((float)p.log_rem[(c.boff * p.heads + h) * p.tokens + c.tok0 + key]) : 0.f;
#pragma unroll
    for (int u = 0; u < dk.kChunks; ++u)
#pragma unroll
      for (int x = 0; x < dk.kWide; ++x) {
        const int col = dk.column(u) + x;
        const float sum = dv.x[i][dv.kWide * u + x];
        if (col < d) {
          ok[col] = from_f32<T>(dk.x[i][dk.kWide * u + x] * p.scale);
          ov[col] = from_f32<T>(p.fuse_rem_v ? fmaf(rem, to_f32<T>(g[col]), sum) : sum);
        }
      }
  }
}

template <int G, typename K>
static cudaError_t launch_one(K kernel, const KParams &p, size_t floats, bool wide, cudaStream_t s) {
  const size_t smem = floats * sizeof(float);
  cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void *>(kernel), (int)smem);
  if (e != cudaSuccess) return e;
  dim3 grid(p.tiles_cap, p.head_cnt);
  return launch_kernel(kernel, dim3(grid), kThreads<G>, smem, s, p, wide);
}

// Whether rows can be fetched in the loader's wide unit: 16 bytes of fp32, 4 bytes (two elements) of 16-bit tensors.
template <typename T>
static bool wide_rows(const TensorRef &t, int head_dim) {
  const long long m = sizeof(T) == 4 ? 4 : 2;
  return t.ptr == nullptr || (reinterpret_cast<uintptr_t>(t.ptr) % (m * sizeof(T)) == 0 && head_dim % m == 0 && t.sb % m == 0 &&
                              t.sh % m == 0 && t.st % m == 0);
}

template <typename T, int DP, int G>
static cudaError_t simt_run(const KParams &p, bool backward, cudaStream_t s) {
  const bool wide = wide_rows<T>(p.q, p.head_dim) && wide_rows<T>(p.k, p.head_dim) && wide_rows<T>(p.v, p.head_dim) &&
                    (!backward || wide_rows<T>(p.d_o, p.head_dim));
  constexpr size_t kRow = kT * kLd<DP>;
  if (!backward) return launch_one<G>(simt_fwd_kernel<T, DP, G>, p, (1 + 4 * G) * kRow + kT * kLdS<G>, wide, s);
  cudaError_t e = cudaSuccess;
  if (!p.skip_dq) e = launch_one<G>(simt_bwd_dq_kernel<T, DP, G>, p, (2 + 4 * G) * kRow + (G == 1 ? 2 : 1) * kT * kLdS<G>, wide, s);
  if (e != cudaSuccess || p.skip_dkv) return e;
  if (p.az != nullptr) return launch_one<G>(simt_bwd_dkv_kernel<T, DP, G, true>, p, 4 * G * kRow + 2 * kStep<G> * kLdH, wide, s);
  return launch_one<1>(simt_bwd_dkv_kernel<T, DP, 1, false>, p, 6 * kRow + 2 * kStep<1> * kLdH, wide, s);
}
// Two groups per block are taken where one would leave the SMs with few warps and the longest sequence is worth their steps of
// 128 keys.  Forward + backward, one group / two (us; fp32, 64 columns unless said otherwise):
// * up to 64 tokens a tile is one step either way, at least half of the wider one masked: 8 heads x 4 x 64 tokens 33.6 / 38.9,
//   200 x 12 tokens 44.5 / 54.8, at 100 columns 74.5 / 105;
// * up to one block per SM: 80 tokens 47 / 41, 250 tokens 79.8 / 70.3, 500 tokens 143 / 124, 100 columns 184 / 135 (768 tokens:
//   365 / 271);
// * up to two, 64 columns: two steps of 64 in one are what is gained, half of the last step of an odd number of them is lost:
//   192 tokens take 75 / 85, 320 118 / 126, 448 160 / 167, but 256 96 / 95, 384 138 / 135, 512 169 / 162, 1024 202 / 191;
// * up to two, 128 columns: one group's operands leave room for a second block, two groups' do not.  fp32, 100 columns, up to 1.5
//   blocks per SM: 256 tokens 152 / 147, 448 tokens 245 / 227, but 192 tokens 127 / 137; up to two: 256 tokens 183 / 195, 448
//   tokens 290 / 307, 512 tokens 332 / 324.  16-bit tensors, which are widened on their way, gain from 256 tokens on (151 / 108
//   to 211 / 201); 192 tokens 146 / 142, with two blocks per SM 170 / 184; 96 tokens 101 / 105, with two 120 / 113;
// * beyond that one group makes better use of the SM: 512 blocks 413 / 482.
// 256 columns: two groups' operands do not fit.
template <typename T, int DP>
static bool two_groups(const KParams &p, int sms) {
  long long tiles = p.tiles_cap, longest = p.max_seqlen;
  if (p.cu != nullptr) {
    if ((long long)p.num_seq * p.n_max < tiles) tiles = (long long)p.num_seq * p.n_max;
    // a bound that says nothing was most likely not given: four times the mean length instead
    if (p.num_seq > 1 && longest >= p.tokens) longest = 4 * p.tokens / p.num_seq;
  }
  const long long blocks = tiles * p.head_cnt, steps = (longest + 63) / 64;
  if (steps <= 1 || blocks > 2 * sms) return false;
  if (blocks <= sms || steps >= 8) return true;
  if (DP == 64) return steps % 2 == 0;
  const bool few = 2 * blocks <= 3 * sms;
  return sizeof(T) == 2 ? steps > 3 || (steps == 3) == few : steps > 3 && few;
}
template <typename T, int DP>
static cudaError_t simt_run_g(const KParams &p, bool backward, cudaStream_t s) {
  if constexpr (DP <= 128) {
    int sms = 0;
    const cudaError_t e = sm_count(&sms);
    if (e != cudaSuccess) return e;
    if (two_groups<T, DP>(p, sms)) return simt_run<T, DP, 2>(p, backward, s);
  }
  return simt_run<T, DP, 1>(p, backward, s);
}
template <typename T>
static cudaError_t simt_run_t(const KParams &p, bool backward, cudaStream_t s) {
  if (p.head_dim <= 64) return simt_run_g<T, 64>(p, backward, s);
  if (p.head_dim <= 128) return simt_run_g<T, 128>(p, backward, s);
  return simt_run_g<T, 256>(p, backward, s);
}
static cudaError_t simt_dispatch(const KParams &p, int dtype, bool backward, cudaStream_t s) {
  if (dtype == SB_DTYPE_F32) return simt_run_t<float>(p, backward, s);
  if (dtype == SB_DTYPE_BF16) return simt_run_t<__nv_bfloat16>(p, backward, s);
  return simt_run_t<__half>(p, backward, s);
}

cudaError_t launch_simt_fwd(const KParams &p, int dtype, cudaStream_t s, int *launches) {
  *launches += 1;
  return simt_dispatch(p, dtype, false, s);
}

cudaError_t launch_simt_bwd(const KParams &p, int dtype, cudaStream_t s, int *launches) {
  *launches += (p.skip_dq ? 0 : 1) + (p.skip_dkv ? 0 : 1);
  return simt_dispatch(p, dtype, true, s);
}

}  // namespace sb
