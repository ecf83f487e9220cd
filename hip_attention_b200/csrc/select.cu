// Chunk-list bookkeeping between scan stages: initial list, top-k selection + split into the next
// stage's chunks, and the final conversion to sorted unique block indices.
//
// One CTA owns one (batch, query block) row.  The chunks a stage keeps are wanted in order of their left bound, and the list
// already is in that order, so nothing has to be sorted: the K-th best score is found by bisecting the score image (two bits
// per step, sixteen counts of the row held in registers), and the chunks above it, with as many of those equal to it as are
// still wanted (lower position first), are compacted in place.  (Two to three bitonic sorts in shared memory before: a
// hundred block-wide barriers.  Rows of 508 / 1024 chunks: 13 to 15 us for a selection and 22 us for the final conversion
// then, 6 to 9 and 8 us now, bound by the sixteen dependent counts.)  A list that is not in order, which only a caller's own stage
// cache can be, is sorted after the compaction.
#include <type_traits>

#include "common.cuh"
#include "host_kernels.h"

namespace hipattn {
namespace {

constexpr int kMaxKeep = 2048;   // entries the final conversion holds

__host__ __device__ inline int next_pow2(int x) {
  int p = 1;
  while (p < x) p <<= 1;
  return p;
}

template <typename K>
__device__ void bitonic_sort(K* a, int N) {
  for (int k = 2; k <= N; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = threadIdx.x; i < (N >> 1); i += blockDim.x) {
        const int l = ((i & ~(j - 1)) << 1) | (i & (j - 1));
        const int r = l | j;
        const bool up = (l & k) == 0;
        const K x = a[l], y = a[r];
        if ((x > y) == up) {
          a[l] = y;
          a[r] = x;
        }
      }
      __syncthreads();
    }
  }
}

// The `keep` best entries of a row of n scores (higher score first, lower position first among equals): item i of a thread is
// position warp * 32 * IPT + i * 32 + lane, so positions ascend with (warp, i, lane).
template <int THREADS, int IPT>
struct TopK {
  static constexpr int W = THREADS / 32;
  struct Shared {
    uint2 counts[2][W];
    int ties[W], taken[W];
  };
  uint32_t chosen;   // bit i: item i is one of the best
  int rank0;         // entries chosen at positions before this warp's first

  __device__ __forceinline__ static int position(int i) { return ((threadIdx.x >> 5) * IPT + i) * 32 + (threadIdx.x & 31); }

  __device__ void run(const int32_t* __restrict__ score, int n, int keep, Shared& sh) {
    static_assert(IPT <= 32, "one bit per item");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t key[IPT];
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
      const int c = position(i);
      key[i] = c < n ? (uint32_t)__ldg(score + c) ^ 0x80000000u : 0u;   // (no score encodes to the smallest integer)
    }
    // threshold: the largest t with at least `keep` entries >= t
    uint32_t t = 0;
    int above = n;            // entries >= t
    if (keep < n) {
#pragma unroll 1
      for (int step = 0; step < 16; ++step) {
        const int sft = 30 - 2 * step;
        const uint32_t t1 = t | (1u << sft), t2 = t | (2u << sft), t3 = t | (3u << sft);
        uint32_t c12 = 0, c3 = 0;
#pragma unroll
        for (int i = 0; i < IPT; ++i) {
          c12 += (key[i] >= t1 ? 1u : 0u) + (key[i] >= t2 ? 0x10000u : 0u);
          c3 += key[i] >= t3 ? 1u : 0u;
        }
        c12 = __reduce_add_sync(0xffffffffu, c12);
        c3 = __reduce_add_sync(0xffffffffu, c3);
        if (lane == 0) sh.counts[step & 1][warp] = make_uint2(c12, c3);
        __syncthreads();
        const uint2 v = lane < W ? sh.counts[step & 1][lane] : make_uint2(0u, 0u);
        c12 = __reduce_add_sync(0xffffffffu, v.x);
        c3 = __reduce_add_sync(0xffffffffu, v.y);
        const int n1 = (int)(c12 & 0xffffu), n2 = (int)(c12 >> 16), n3 = (int)c3;
        if (n3 >= keep) { t = t3; above = n3; }
        else if (n2 >= keep) { t = t2; above = n2; }
        else if (n1 >= keep) { t = t1; above = n1; }
        if (above == keep) break;
      }
    }
    // entries above the threshold, and the first of those equal to it (none has to be left out when the count is exact)
    const bool exact = above == keep;
    uint32_t eq = 0;
    chosen = 0;
    int more = 0, ties = 0;
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
      const bool in = position(i) < n;
      if (in && (key[i] > t || (exact && key[i] == t))) { chosen |= 1u << i; ++more; }
      else if (in && key[i] == t) { eq |= 1u << i; ++ties; }
    }
    more = __reduce_add_sync(0xffffffffu, more);
    ties = __reduce_add_sync(0xffffffffu, ties);
    if (lane == 0) { sh.taken[warp] = more; sh.ties[warp] = ties; }
    __syncthreads();
    int before_ties = 0, total = 0;
    rank0 = 0;
    for (int w = 0; w < W; ++w) {
      total += sh.taken[w];
      if (w < warp) { rank0 += sh.taken[w]; before_ties += sh.ties[w]; }
    }
    const int want = keep - total;        // ties still to take, over the whole row
    rank0 += min(before_ties, want);
    if (!exact) {
#pragma unroll
      for (int i = 0; i < IPT; ++i) {
        const uint32_t b = __ballot_sync(0xffffffffu, eq >> i & 1u);
        if ((eq >> i & 1u) && before_ties + __popc(b & ((1u << lane) - 1u)) < want) chosen |= 1u << i;
        before_ties += __popc(b);
      }
    }
  }
  // calls f(rank, position) for every chosen entry of this thread, ranks ascending with the position
  template <typename F>
  __device__ __forceinline__ void each(F f) const {
    const int lane = threadIdx.x & 31;
    int r = rank0;
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
      const uint32_t b = __ballot_sync(0xffffffffu, chosen >> i & 1u);
      if (chosen >> i & 1u) f(r + __popc(b & ((1u << lane) - 1u)), position(i));
      r += __popc(b);
    }
  }
};

// Whether a[0 .. n) ascends; the answer is the same in every thread.
__device__ __forceinline__ bool ascending(const uint32_t* a, int n) {
  bool bad = false;
  for (int j = threadIdx.x + 1; j < n; j += blockDim.x) bad |= a[j] < a[j - 1];
  return !__syncthreads_or(bad);
}
__device__ __forceinline__ void sort_padded(uint32_t* a, int n, int n_pad) {
  for (int j = n + threadIdx.x; j < n_pad; j += blockDim.x) a[j] = 0xffffffffu;
  __syncthreads();
  bitonic_sort(a, n_pad);
}

template <int THREADS, int IPT>
__global__ void __launch_bounds__(THREADS)
    select_stage_kernel(const int32_t* __restrict__ score_max, const int32_t* __restrict__ left, int n, int k_keep, int k_pad, int sink,
                        int c_prev, int c_next, int32_t* __restrict__ next_left, int32_t* __restrict__ next_right,
                        int32_t* __restrict__ next_score_max, int64_t* __restrict__ next_left64, int64_t* __restrict__ next_right64) {
  extern __shared__ __align__(16) uint32_t kept[];   // [k_pad] left bounds of the kept chunks, on the previous chunk grid
  __shared__ typename TopK<THREADS, IPT>::Shared sh;
  const int64_t row = blockIdx.x;
  TopK<THREADS, IPT> top;
  top.run(score_max + row * n, n, k_keep, sh);
  top.each([&](int r, int c) {
    const int l = __ldg(left + row * n + c);
    kept[r] = (uint32_t)((l - sink) / c_prev * c_prev + sink);  // l >= sink
  });
  __syncthreads();
  if (!ascending(kept, k_keep)) sort_padded(kept, k_keep, k_pad);

  const int s = c_prev / c_next;
  const int64_t out_n = (int64_t)k_keep * s;
  const int32_t init = encode_score(HIPATTN_SCORE_INIT);
  for (int64_t o = threadIdx.x; o < out_n; o += THREADS) {
    const int j = (int)o / s, i = (int)o - j * s;
    const int la = (int)kept[j];
    const int ra = la + c_prev;
    // attention_extend.py:2133-2165: chunk sizes and offsets go through fp32
    const float w = fmaxf(__fdiv_rn((float)(ra - la), (float)s), 0.f);
    const int nl = la + (int)floorf(__fmul_rn((float)i, w)), nr = ra - (int)floorf(__fmul_rn((float)(s - 1 - i), w));
    next_left[row * out_n + o] = nl;
    next_right[row * out_n + o] = nr;
    if (next_left64) next_left64[row * out_n + o] = nl;
    if (next_right64) next_right64[row * out_n + o] = nr;
    next_score_max[row * out_n + o] = init;
  }
}

template <int THREADS, int IPT>
__global__ void __launch_bounds__(THREADS)
    finalize_kernel(const int32_t* __restrict__ score_max, const int32_t* __restrict__ left_heads, int64_t left_row_stride,
                    int64_t left_head_stride, const int64_t* __restrict__ pos, int64_t pos_stride_b, int64_t pos_stride_t,
                    int BDST, int H, int n, int K, int K_pad, int c_last, int block_size_q,
                    int64_t* __restrict__ indices, int64_t* __restrict__ ks, int32_t* __restrict__ ks_start_end) {
  __shared__ typename TopK<THREADS, IPT>::Shared sh;
  __shared__ uint32_t cand[kMaxKeep], uniq[kMaxKeep];
  __shared__ int s_warp[THREADS / 32], s_count;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t row = blockIdx.x;
  const int b = (int)(row / BDST), d = (int)(row % BDST);
  const long long limit = pos[(int64_t)b * pos_stride_b + (int64_t)d * block_size_q * pos_stride_t] + block_size_q;
  TopK<THREADS, IPT> top;
  top.run(score_max + row * n, n, K, sh);

  const int n_heads_distinct = left_head_stride == 0 ? 1 : H;
  for (int hh = 0; hh < n_heads_distinct; ++hh) {
    const int32_t* lh = left_heads + row * left_row_stride + (int64_t)hh * left_head_stride;
    top.each([&](int r, int c) { cand[r] = (uint32_t)(__ldg(lh + c) / c_last * c_last); });
    if (threadIdx.x == 0) s_count = 0;
    __syncthreads();
    if (!ascending(cand, K)) sort_padded(cand, K, K_pad);
    // duplicates (compared with the previous entry, wrapping around) become padding behind the others
    int base = 0;
    for (int j0 = 0; j0 < K; j0 += THREADS) {
      const int j = j0 + threadIdx.x;
      const bool own = j < K && cand[j] != cand[j > 0 ? j - 1 : K - 1];
      const uint32_t m = __ballot_sync(0xffffffffu, own);
      if (lane == 0) s_warp[warp] = __popc(m);
      __syncthreads();
      int at = base;
      for (int w = 0; w < THREADS / 32; ++w) {
        if (w < warp) at += s_warp[w];
        base += s_warp[w];
      }
      if (own) uniq[at + __popc(m & ((1u << lane) - 1u))] = cand[j];
      __syncthreads();
    }
    int local = 0;
    for (int j = threadIdx.x; j < K; j += THREADS) {
      const long long v64 = j < base ? (long long)uniq[j] : INT64_MAX;
      local += v64 < limit ? 1 : 0;
      if (n_heads_distinct == 1) {
        for (int h = 0; h < H; ++h) indices[(((int64_t)b * H + h) * BDST + d) * K + j] = v64;
      } else {
        indices[(((int64_t)b * H + hh) * BDST + d) * K + j] = v64;
      }
    }
    local = __reduce_add_sync(0xffffffffu, local);
    if (lane == 0) atomicAdd(&s_count, local);
    __syncthreads();
    const int c = s_count;
    for (int h = (n_heads_distinct == 1 ? 0 : hh) + threadIdx.x; h < (n_heads_distinct == 1 ? H : hh + 1); h += THREADS) {
      const int64_t o = ((int64_t)b * H + h) * BDST + d;
      ks[o] = c;
      ks_start_end[o * 2] = 0;
      ks_start_end[o * 2 + 1] = c;
    }
    __syncthreads();
  }
}

// calls f(threads, items per thread) as integral constants: rows of up to 1024 chunks keep four items in each of 256 threads
template <typename F>
int by_row_length(int n, F f) {
  if (n <= 1024) return f(std::integral_constant<int, 256>{}, std::integral_constant<int, 4>{});
  if (n <= 4096) return f(std::integral_constant<int, 512>{}, std::integral_constant<int, 8>{});
  return f(std::integral_constant<int, 512>{}, std::integral_constant<int, 32>{});
}

__global__ void decode_scores_kernel(const int32_t* codes, float* scores, int64_t count) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x)
    scores[i] = decode_score(codes[i]);
}
__global__ void widen_kernel(const int32_t* src, int64_t* dst, int64_t count) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x)
    dst[i] = src[i];
}

inline unsigned grid_for(int64_t total, int threads) {
  int64_t g = (total + threads - 1) / threads;
  return (unsigned)(g < 1 ? 1 : (g > 148 * 16 ? 148 * 16 : g));
}

}  // namespace
}  // namespace hipattn

using namespace hipattn;

extern "C" int hipattn_init_chunks(int32_t* left, int32_t* right, int32_t* score_max, int64_t rows, int32_t n,
                                   int32_t sink, int32_t chunk, int32_t T, int32_t scan_window, void* stream) {
  HIPATTN_REQUIRE(rows >= 0 && n >= 0 && chunk > 0 && sink >= 0, HIPATTN_ERR_INVALID, "init_chunks: bad sizes");
  if (rows * n == 0) return HIPATTN_OK;
  HIPATTN_REQUIRE(left && right && score_max, HIPATTN_ERR_INVALID, "init_chunks: null output");
  BeginCall c{};
  c.left = left; c.right = right; c.score_max = score_max;
  c.rows = rows; c.n = n;
  c.sink = sink; c.chunk = chunk; c.T = T; c.scan_window = scan_window;
  return begin_call(c, (cudaStream_t)stream);
}

int hipattn::select_stage(const int32_t* score_max, const int32_t* left, int64_t rows, int32_t n, int32_t k_keep, int32_t sink,
                          int32_t c_prev, int32_t c_next, int32_t* next_left, int32_t* next_right, int32_t* next_score_max,
                          int64_t* next_left64, int64_t* next_right64, cudaStream_t stream) {
  HIPATTN_REQUIRE(score_max && left && next_left && next_right && next_score_max, HIPATTN_ERR_INVALID,
                  "select_stage: null pointer");
  HIPATTN_REQUIRE(rows > 0 && n > 0 && k_keep > 0 && k_keep <= n, HIPATTN_ERR_INVALID,
                  "select_stage: need 0 < k_keep (%d) <= n (%d)", k_keep, n);
  HIPATTN_REQUIRE(n <= HIPATTN_MAX_CHUNKS, HIPATTN_ERR_UNSUPPORTED, "select_stage: %d chunks per row exceed %d", n,
                  HIPATTN_MAX_CHUNKS);
  HIPATTN_REQUIRE(c_next > 0 && c_prev % c_next == 0, HIPATTN_ERR_INVALID,
                  "select_stage: chunk size %d is not a multiple of %d", c_prev, c_next);
  const int k_pad = next_pow2(k_keep < 2 ? 2 : k_keep);
  const size_t smem = (size_t)k_pad * sizeof(uint32_t);
  return by_row_length(n, [&](auto threads, auto items) -> int {
    auto kern = select_stage_kernel<decltype(threads)::value, decltype(items)::value>;
    if (smem > 40 * 1024) HIPATTN_CUDA_OK(allow_smem((const void*)kern, smem));
    kern<<<(unsigned)rows, decltype(threads)::value, smem, stream>>>(score_max, left, n, k_keep, k_pad, sink, c_prev, c_next, next_left, next_right,
                                                                    next_score_max, next_left64, next_right64);
    return check_launch("select_stage_kernel");
  });
}

extern "C" int hipattn_select_stage(const int32_t* score_max, const int32_t* left, int64_t rows, int32_t n, int32_t k_keep,
                                    int32_t sink, int32_t c_prev, int32_t c_next, int32_t* next_left,
                                    int32_t* next_right, int32_t* next_score_max, void* stream) {
  return select_stage(score_max, left, rows, n, k_keep, sink, c_prev, c_next, next_left, next_right, next_score_max, nullptr, nullptr,
                      (cudaStream_t)stream);
}

extern "C" int hipattn_finalize_indices(const int32_t* score_max, const int32_t* left_heads, int64_t left_row_stride,
                                        int64_t left_head_stride, const int64_t* pos, int64_t pos_stride_b,
                                        int64_t pos_stride_t, int32_t B, int32_t BDST, int32_t H, int32_t n, int32_t K,
                                        int32_t c_last, int32_t block_size_q, int64_t* indices, int64_t* ks,
                                        int32_t* ks_start_end, void* stream) {
  HIPATTN_REQUIRE(score_max && left_heads && pos && indices && ks && ks_start_end, HIPATTN_ERR_INVALID,
                  "finalize_indices: null pointer");
  HIPATTN_REQUIRE(B > 0 && BDST > 0 && H > 0 && n > 0 && K > 0 && K <= n && c_last > 0, HIPATTN_ERR_INVALID,
                  "finalize_indices: need 0 < K (%d) <= n (%d)", K, n);
  HIPATTN_REQUIRE(n <= HIPATTN_MAX_CHUNKS, HIPATTN_ERR_UNSUPPORTED, "finalize_indices: %d chunks per row exceed %d", n,
                  HIPATTN_MAX_CHUNKS);
  const int K_pad = next_pow2(K < 2 ? 2 : K);
  HIPATTN_REQUIRE(K_pad <= kMaxKeep, HIPATTN_ERR_UNSUPPORTED, "finalize_indices: K = %d exceeds %d", K, kMaxKeep);
  return by_row_length(n, [&](auto threads, auto items) -> int {
    finalize_kernel<decltype(threads)::value, decltype(items)::value><<<(unsigned)(B * BDST), decltype(threads)::value, 0, (cudaStream_t)stream>>>(
        score_max, left_heads, left_row_stride, left_head_stride, pos, pos_stride_b, pos_stride_t, BDST, H, n, K, K_pad, c_last,
        block_size_q, indices, ks, ks_start_end);
    return check_launch("finalize_kernel");
  });
}

extern "C" int hipattn_decode_scores(const int32_t* codes, float* scores, int64_t count, void* stream) {
  if (count <= 0) return HIPATTN_OK;
  HIPATTN_REQUIRE(codes && scores, HIPATTN_ERR_INVALID, "decode_scores: null pointer");
  decode_scores_kernel<<<grid_for(count, 256), 256, 0, (cudaStream_t)stream>>>(codes, scores, count);
  return check_launch("decode_scores_kernel");
}

extern "C" int hipattn_widen_i32(const int32_t* src, int64_t* dst, int64_t count, void* stream) {
  if (count <= 0) return HIPATTN_OK;
  HIPATTN_REQUIRE(src && dst, HIPATTN_ERR_INVALID, "widen_i32: null pointer");
  widen_kernel<<<grid_for(count, 256), 256, 0, (cudaStream_t)stream>>>(src, dst, count);
  return check_launch("widen_kernel");
}
