// Block-sparse attention, prefill, 16-bit types, head dim 64 or 128: warp-specialised tcgen05 / TMEM kernel.
//
// One CTA (8 warps: four softmax, one MMA issuer, three copy warps) owns 128 query rows -- two heads
// of a KV group x 64 rows, or one head x 128 rows -- and walks the key list [sink | selected blocks | window] in tiles of 64 keys.  Two CTAs
// are resident per SM, so one CTA's softmax overlaps the other's tensor-core work.
//
//   S = Q K^T   tcgen05.mma (M 128, N 64, K 16) x 8, operands in shared memory (128-byte-swizzled
//               canonical layouts, K-major), accumulator double buffered in TMEM
//   softmax     thread t owns row t = TMEM lane t: tcgen05.ld of its 64 logits, admission rule,
//               base-2 online softmax with a lazily updated maximum, P written back to TMEM
//   O += P V    tcgen05.mma (M 128, N head dim, K 16) x 4, A operand = P in TMEM, V staged row-major
//               (MN-major operand)
//
// K / V rows are gathered with 16-byte cp.async through the page table directly into the swizzled
// operand layouts.  O stays in TMEM for the whole key list: the running maximum used for the
// exponentials is only raised (and O rescaled in TMEM) when the true maximum has grown by more than
// 2^13 (fp16) / 2^24 (bf16), which keeps P within the element type's range and makes rescaling rare.
// Every wait on an mbarrier is bounded; a wait that runs out sets HIPATTN_STATUS_TIMEOUT and the CTA
// leaves through the normal exit (TMEM freed), so a fault in the pipeline cannot hang the device.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "bsa_common.cuh"
#include "tcgen05_common.cuh"
#include "rope.cuh"

namespace hipattn {
namespace {

constexpr int TK5 = 64;            // keys per tile
constexpr float kLog2e = 1.4426950408889634f;
// log2 of the growth of a row's maximum that triggers a rescale of O: P = 2^(s - m) stays below 2^13 in fp16 (largest
// finite value 2^16) and 2^24 in bf16; O and the row sums are fp32.  A reference maximum that lags the true one costs no
// accuracy because the row sums are taken from the rounded P (see the softmax loop): with sums of the unrounded values
// the largest output error against an fp32 recompute grew from 0.019 (threshold 2^8) to 0.025 (2^24) on the 128k
// prefill workload; with rounded sums it is 0.012 at every threshold, the figure of the exact-maximum kernel.
template <int DT> constexpr float kRescaleThreshold = DT == HIPATTN_BF16 ? 24.f : 13.f;

// 2^x on the special-function unit alone (ex2.approx: about 2 ulp, flushes denormal results, 2^-inf = 0).
// The probabilities are rounded to 8 or 11 significant bits right after, so the exact exp2f sequence
// (range split + rescale around the same instruction) buys nothing here and costs three more instructions
// per logit in the longest loop of the kernel.
__device__ __forceinline__ float exp2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}

// the two 16-bit elements of a packed pair as floats (exact)
template <int DT>
__device__ __forceinline__ float pair_lo(uint32_t w) {
  if (DT == HIPATTN_BF16) return __uint_as_float(w << 16);
  return __half2float(__ushort_as_half((unsigned short)(w & 0xffffu)));
}
template <int DT>
__device__ __forceinline__ float pair_hi(uint32_t w) {
  if (DT == HIPATTN_BF16) return __uint_as_float(w & 0xffff0000u);
  return __half2float(__ushort_as_half((unsigned short)(w >> 16)));
}

// maximum of three values in one instruction
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;\n" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// Record of a tile for the softmax warps (ring of eight: the copy warps run at most three tiles ahead of the softmax
// warps, so a slot is rewritten long after its readers have left it) ...
// 256 zero bytes in device memory: the row address of a key that no query admits, so that the copy loops carry neither
// a predicate nor a source size
__device__ __align__(256) unsigned char g_zero_row[256];

struct MetaS {
  int tpos[TK5];
  unsigned char twin[TK5];
  int far_ok[2];
  int win_ok[2];
  int rpos[TK5];          // in-kernel RoPE: table position the key is rotated to (-1: no key)
};
// ... and for the copy warps (ring of four)
struct Meta5 {
  const char* kptr[TK5];   // address of the K / V row (the zero row when the entry has none)
  const char* vptr[TK5];
  long long start[TK5];   // warp-specialised kernel: block starts of the tile's selected entries, fetched a tile ahead
};

// In-kernel RoPE on an operand tile of two 128-byte-swizzled K-blocks ([2][rows][128 B], head dim 128): row r is rotated
// to table position pos(r) (negative: left alone).  Thread `tid` of `nthreads` takes piece tid & 7 of rows (tid >> 3) +
// i * nthreads / 8; the table pieces of up to ITEMS rows are requested together (fetch), so that their latency is paid
// once and can overlap with whatever the caller waits for before it rotates (apply).  The caller synchronises the threads
// around apply and fences towards the tensor cores afterwards.
template <int DT, int ITEMS>
struct RopeTile {
  uint4 c[ITEMS], s[ITEMS];
  uint32_t live;
  template <typename PosFn>
  __device__ __forceinline__ void fetch(const hipattn_bsa_params_t& p, int row0, int rows, int tid, int nthreads, PosFn pos) {
    live = 0;
    const int pc = tid & 7;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const int r = row0 + (tid >> 3) + i * (nthreads >> 3);
      const int t = r < rows ? pos(r) : -1;
      if (t >= 0) {
        live |= 1u << i;
        c[i] = rope_table_raw(p.rope_cos, p.rope_stride, p.rope_rows, t, pc);
        s[i] = rope_table_raw(p.rope_sin, p.rope_stride, p.rope_rows, t, pc);
      }
    }
  }
  __device__ __forceinline__ void apply(unsigned char* tile, int kblock_bytes, int row0, int tid, int nthreads) {
    const int pc = tid & 7;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      if (!(live >> i & 1)) continue;
      const int r = row0 + (tid >> 3) + i * (nthreads >> 3);
      uint4* plo = reinterpret_cast<uint4*>(tile + sw128(r, pc));
      uint4* phi = reinterpret_cast<uint4*>(tile + kblock_bytes + sw128(r, pc));
      uint4 lo = *plo, hi = *phi;
      rope_rotate_packed<DT>(lo, hi, c[i], s[i]);
      *plo = lo;
      *phi = hi;
    }
  }
};


// ---------------------------------------------------------------------------------------------------
// Roles (8 warps): warps 0-3 run the softmax (thread = query row = TMEM lane), warp 4 issues the MMAs, warps 5 and 7
// resolve the tile records and gather the K rows, warp 6 gathers the V rows.
//   TMEM: S buffers at columns [0, 64) and [64, 128) (S(it) in buffer it & 1), O at [128, 256).
//   P(it) is written back over the first 32 columns of S(it)'s buffer as packed 16-bit pairs and is
//   the A operand of O += P V straight from TMEM, so no shared memory is needed for P.
//   S runs two tiles ahead of the softmax: once P(it) is written and V(it) / K(it + 2) are in place the issuer launches
//   PV(it) and S(it + 2), so the tensor pipe computes S(it + 1) / S(it + 2) while the softmax of tile it / it + 1 runs.
//   K and V tiles are double buffered.
// The roles meet on mbarriers only; every mbarrier wait is bounded.
// ---------------------------------------------------------------------------------------------------
__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}\n"
      ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u));
}

// KV8 = K and V rows are e5m2 bytes: the copy warps load them into registers, widen them (exactly) and store the 16-bit
// operand tiles themselves.  P then goes to TMEM as two 16-bit terms (value rounded, and what the rounding left), each
// multiplied with V, so that an fp8 cache keeps softmax weights of at least 16 significant bits: the general kernel, which
// served it before, multiplies fp32 weights.  (2 x 3001 queries, RoPE: 12.2 ms there, 1.43 ms here; output 5e-5 apart.)
// Head dim 64: the same roles with half the MMAs and copies per tile; 2 x 2999 queries of 16 heads 0.44 ms with mma.sync,
// 0.27 here.  Its weights go in two terms as well: with one, and the lagging maximum, no weight of a row is exact, while
// mma.sync has the row's largest at exactly 1 (error against 64 bits before the output is rounded, fp16: 5.7e-5 with
// mma.sync, 9.5e-5 with one term, 6e-6 with two).
// SPLIT = the grid may cut key lists into ranges (p.n_splits); the variant without is 2 % faster on grids that need none.
template <int DT, int D, bool ROPE, bool KV8, bool SPLIT>
__global__ void __launch_bounds__(256, 2) bsa_tcgen05_ws_kernel(const hipattn_bsa_params_t p, int BQ, int n_sub) {
  using T = typename Elem<DT>::type;
  constexpr int NT = 256;
  static_assert(D == 128 || (D == 64 && !ROPE), "in-kernel RoPE pairs the two 128-byte halves of a 256-byte row");
  constexpr bool TWO = KV8 || D == 64;        // softmax weights in two 16-bit terms
  constexpr int KB = D / 64;                  // 128-byte blocks per row
  constexpr int PIECES = D / 8;               // 16-byte pieces per row
  constexpr int Q_BYTES = KB * 128 * 128;
  constexpr int KT_BYTES = KB * TK5 * 128;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  unsigned char* smem = smem_raw + ((1024u - (raw & 1023u)) & 1023u);
  unsigned char* sQ = smem;                   // also the output staging area
  unsigned char* sK = sQ + Q_BYTES;           // 2 buffers
  unsigned char* sV = sK + 2 * KT_BYTES;      // 2 buffers
  Meta5* meta = reinterpret_cast<Meta5*>(sV + 2 * KT_BYTES);  // 4 entries
  MetaS* metas = reinterpret_cast<MetaS*>(meta + 4);            // 8 entries
  // S buffer 0 / 1 ready, PV of an even tile done (tensor-core commits, one arrival each); P buffer 0 / 1 written (128
  // softmax threads);
  // K buffer 0 / 1 filled (64 key-copy threads), V buffer 0 / 1 filled (32 value-copy threads); PV of an odd
  // tile done.  PV completions alternate between two barriers because a waiter may look for PV(t - 1) after PV(t) has
  // completed: with one barrier its phase bit would have wrapped by then.
  __shared__ __align__(8) unsigned long long s_mbar[12];
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  __shared__ int s_rowpos[128];
  __shared__ int s_mm[4];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int Gq = p.H / p.HKV;
  const int NH = 128 / BQ;
  const int NBLK = cdiv(p.TQ, p.block_size_q);
  const int hslots = p.H / NH;
  int64_t bid = blockIdx.x;
  int split = 0;
  if constexpr (SPLIT) { split = (int)(bid % p.n_splits); bid /= p.n_splits; }
  const int sub = (int)(bid % n_sub); bid /= n_sub;
  const int d = (int)(bid % NBLK); bid /= NBLK;
  const int hs = (int)(bid % hslots); bid /= hslots;
  const int b = (int)bid;
  const int h0 = hs * NH;
  const int hkv = h0 / Gq;
  const int blk_t0 = d * p.block_size_q;
  const int blk_rows = min(p.block_size_q, p.TQ - blk_t0);
  const int row_t0 = blk_t0 + sub * BQ;
  const int rows_here = max(0, min(BQ, blk_rows - sub * BQ));
  const uint32_t mbar_s0 = smem_u32(&s_mbar[0]);
  // barrier and phase bit of "PV(t) has completed"
  auto mbar_o = [&](int t) { return smem_u32(&s_mbar[(t & 1) ? 9 : 2]); };
  auto phase_o = [](int t) { return (uint32_t)((t >> 1) & 1); };
  const uint32_t mbar_p0 = smem_u32(&s_mbar[3]), mbar_k0 = smem_u32(&s_mbar[5]), mbar_v0 = smem_u32(&s_mbar[7]);
  // in-kernel RoPE: K buffer 0 / 1 has landed, not yet rotated (64 key-copy threads); the softmax warps rotate it between
  // two of their tiles - they wait for S there anyway - and report the buffer ready (128 arrivals instead of 64)
  const uint32_t mbar_kraw0 = smem_u32(&s_mbar[10]);
  // rotates rows 32-63 of K(tile) in place; called by the 128 softmax threads (rows 0-31 are rotated by the key-copy
  // warps before they report the tile as landed: those warps idle for about as long as that takes)
  auto rotate_k_tile = [&](int tile) {
    RopeTile<DT, 2> rk;
    rk.fetch(p, 32, TK5, tid, 128, [&](int r) { return metas[tile & 7].rpos[r]; });
    mbar_wait(mbar_kraw0 + 8 * (tile & 1), (tile >> 1) & 1, &s_abort, p.status);
    rk.apply(sK + (tile & 1) * KT_BYTES, TK5 * 128, 32, tid, 128);
    fence_async_smem();
    mbar_arrive(mbar_k0 + 8 * (tile & 1));
  };

  if (tid == 0) {
    for (int i = 0; i < 3; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(mbar_s0 + 8 * i));
    for (int i = 3; i < 5; ++i) mbar_init(mbar_s0 + 8 * i, 128);
    for (int i = 5; i < 7; ++i) mbar_init(mbar_s0 + 8 * i, ROPE ? 128 : 64);
    for (int i = 10; i < 12; ++i) mbar_init(mbar_s0 + 8 * i, 64);
    for (int i = 7; i < 9; ++i) mbar_init(mbar_s0 + 8 * i, 32);
    mbar_init(mbar_s0 + 8 * 9, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    s_abort = 0;
  }
  if (tid < 4) s_mm[tid] = (tid & 1) ? -1 : 0x7fffffff;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s_tmem)), "r"(256u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;
  {
    int lo = 0x7fffffff, hi = -1;
    for (int i = tid; i < blk_rows; i += NT) {
      const long long x = p.pos[(int64_t)b * p.pos_stride_b + (int64_t)(blk_t0 + i) * p.pos_stride_t];
      const int v = (int)(x > 0x7ffffff0LL ? 0x7ffffff0LL : (x < 0 ? 0 : x));
      lo = min(lo, v); hi = max(hi, v);
    }
    if (hi >= 0) { atomicMin(&s_mm[0], lo); atomicMax(&s_mm[1], hi); }
  }
  if (tid < 128) {
    const int i = tid % BQ;
    int pv = -0x40000000;
    if (i < rows_here) {
      const long long x = p.pos[(int64_t)b * p.pos_stride_b + (int64_t)(row_t0 + i) * p.pos_stride_t];
      pv = (int)(x > 0x7ffffff0LL ? 0x7ffffff0LL : (x < 0 ? 0 : x));
      atomicMin(&s_mm[2], pv);
      atomicMax(&s_mm[3], pv);
    }
    s_rowpos[tid] = pv;
  }
  // the query tile: one batch of asynchronous 16-byte copies per thread (rows beyond the block are zero-filled), so that
  // the tile costs one trip to memory instead of one per loop iteration
  for (int i = tid; i < 128 * PIECES; i += NT) {
    const int r = i >> (D == 128 ? 4 : 3), pc = i & (PIECES - 1);
    const bool live = (r % BQ) < rows_here;
    const T* qp = reinterpret_cast<const T*>(p.q) + (int64_t)b * p.q_stride_b + (int64_t)(row_t0 + (live ? r % BQ : 0)) * p.q_stride_t +
                  (int64_t)(h0 + r / BQ) * p.q_stride_h + pc * 8;
    cp_async16_zfill(smem_u32(sQ) + (pc >> 3) * (128 * 128) + sw128(r, pc & 7), qp, live);
  }
  cp_async_commit();
  cp_async_wait<0>();
  if constexpr (ROPE) {   // in-kernel RoPE: every query row at its own position (attention_extend_bsa.py:797-856)
    __syncthreads();
    RopeTile<DT, 4> rq;   // 128 rows x 8 pieces over 256 threads: 32 rows per pass
    rq.fetch(p, 0, 128, tid, NT, [&](int r) { return s_rowpos[r]; });
    rq.apply(sQ, 128 * 128, 0, tid, NT);
  }
  fence_async_smem();
  __syncthreads();
  const int pmin = s_mm[0], pmax = s_mm[1];
  const int rmin = s_mm[2], rmax = s_mm[3];
  KeyList kl = make_key_list(p, b, h0, d, pmin, pmax);
  if (lists_ascend(p)) trim_selected(kl, rmax, p.window);
  // the tiles of this CTA's key range (all of them unless the caller asked for key splits)
  const int all_tiles = cdiv(kl.total, TK5);
  const int per_split = SPLIT ? cdiv(all_tiles, p.n_splits) : all_tiles;
  const int tile0 = SPLIT ? split * per_split : 0;
  const int n_tiles = SPLIT ? max(0, min(per_split, all_tiles - tile0)) : all_tiles;
  constexpr int EB = KV8 ? 1 : 2;   // bytes of a K / V element
  constexpr int FMT = DT == HIPATTN_BF16 ? 1 : 0;
  const uint32_t idesc_s = make_idesc(FMT, 128, TK5, 0);
  const uint32_t idesc_o = make_idesc(FMT, 128, D, 1);
  const uint32_t tmem_o = tmem + 128;

  const char* kbase = (const char*)(p.k.cache ? p.k.cache : p.k.dense);
  const char* vbase = (const char*)(p.v.cache ? p.v.cache : p.v.dense);
  const bool dense_kv = p.k.cache == nullptr && p.v.cache == nullptr;
  // paged K and V that share block table, sequence lengths and page size (what a serving pool hands over)
  const bool paged_fast = p.k.cache != nullptr && p.v.cache != nullptr && p.k.block_table == p.v.block_table &&
                          p.k.table_stride_b == p.v.table_stride_b && p.k.table_width == p.v.table_width &&
                          p.k.table_is_i64 == p.v.table_is_i64 && p.k.cache_seq_lens == p.v.cache_seq_lens &&
                          p.k.seq_lens_is_i64 == p.v.seq_lens_is_i64 && p.k.page_size == p.v.page_size && p.k.page_size > 0;
  const int page_shift = (paged_fast && (p.k.page_size & (p.k.page_size - 1)) == 0) ? 31 - __clz(p.k.page_size) : -1;
  long long seq_len = 0;
  if (paged_fast)
    seq_len = p.k.seq_lens_is_i64 ? ((const int64_t*)p.k.cache_seq_lens)[b] : (long long)((const int32_t*)p.k.cache_seq_lens)[b];
  const long long k_base_off = ((long long)b * p.k.stride_b + (long long)hkv * p.k.stride_h) * EB, k_step = p.k.stride_t * EB;
  const long long v_base_off = ((long long)b * p.v.stride_b + (long long)hkv * p.v.stride_h) * EB, v_step = p.v.stride_t * EB;
  // requests the block start of entry e of `tile` (if it is a selected entry) into the tile's record; the copy joins
  // the calling thread's next commit group and must be consumed by the same thread
  auto prefetch_start = [&](int tile, int e) {
    if (tile >= n_tiles) return;
    const int blk = selected_block_of(kl, (tile0 + tile) * TK5 + e);
    if (blk >= 0)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(smem_u32(&meta[tile & 3].start[e])), "l"(kl.idx + blk));
  };
  // position, addresses and admission summary of entry e of `tile`; all 32 lanes of a warp call it with e = 32 h + lane
  auto make_meta = [&](int tile, int e, bool prefetched) {
    Meta5& m = meta[tile & 3];
    MetaS& ms = metas[tile & 7];
    bool w;
    const int j = (tile0 + tile) * TK5 + e;
    const int t = prefetched ? key_position_at(kl, j, m.start[e], &w) : key_position(kl, j, &w);
    ms.tpos[e] = t;
    ms.twin[e] = (t >= 0 && w) ? 1 : 0;
    long long ko = -1, vo = -1;
    if (t >= 0) {
      if (dense_kv) {   // dense tensors: one multiply-add per tensor on top of the CTA's own base
        ko = k_base_off + (long long)t * k_step;
        vo = v_base_off + (long long)t * v_step;
      } else if (paged_fast) {
        // paged K and V behind one block table: one look-up in 32-bit arithmetic (token_row's rules: a position beyond
        // the sequence or the table reads page 0; a page id outside the pool is reported and reads page 0)
        const int pi = page_shift >= 0 ? (t >> page_shift) : (t / p.k.page_size);
        const int off = t - pi * p.k.page_size;
        long long page = 0;
        if (t < seq_len && pi < p.k.table_width) {
          const int64_t o = (int64_t)b * p.k.table_stride_b + pi;
          page = p.k.table_is_i64 ? ((const int64_t*)p.k.block_table)[o] : (long long)((const int32_t*)p.k.block_table)[o];
          if (page < 0 || page >= p.k.n_pages || page >= p.v.n_pages) {
            atomicOr(p.status, HIPATTN_STATUS_PAGE_RANGE);
            page = 0;
          }
        }
        ko = (page * p.k.stride_page + (long long)off * p.k.stride_off + (long long)hkv * p.k.stride_ch) * EB;
        vo = (page * p.v.stride_page + (long long)off * p.v.stride_off + (long long)hkv * p.v.stride_ch) * EB;
      } else {
        ko = token_row(p.k, b, t, hkv, 2, p.status) - kbase;
        vo = token_row(p.v, b, t, hkv, 2, p.status) - vbase;
      }
    }
    m.kptr[e] = ko >= 0 ? kbase + ko : reinterpret_cast<const char*>(g_zero_row);
    m.vptr[e] = vo >= 0 ? vbase + vo : reinterpret_cast<const char*>(g_zero_row);
    if (ROPE) ms.rpos[e] = t >= 0 ? rope_key_position(kl, j, t) : -1;
    const bool far_ok = t >= 0 && !w && t <= rmin - p.window;
    const bool win_ok = t >= 0 && w && t > rmax - p.window && t <= rmin;
    const int f = __all_sync(0xffffffffu, far_ok), g = __all_sync(0xffffffffu, win_ok);
    if (lane == 0) {
      ms.far_ok[e >> 5] = f;
      ms.win_ok[e >> 5] = g;
    }
  };

  if (warp >= 5) {
    // ================================ producers: addresses + gathers ================================
    // Warps 5 and 7 (64 threads) resolve the records of the tiles and copy the K tiles (and rotate them under in-kernel
    // RoPE); warp 6 copies the V tiles.  With four softmax warps and four helper warps every scheduler of the
    // multiprocessor carries one of each per CTA.
    const bool k_role = warp != 6;
    const int ptid = warp == 5 ? lane : (warp == 7 ? 32 + lane : lane);   // 0..63 in the K group, 0..31 in the V warp
    // K group: thread ptid copies piece ptid % PIECES of rows ptid / PIECES + i * 64 / PIECES;
    // V warp:  the same with 32 threads, in batches of at most sixteen rows
    constexpr int KSTEP = 64 / PIECES, KN = TK5 / KSTEP;        // rows apart, rows per thread (K group)
    constexpr int VN = TK5 * PIECES / 32, VB = VN > 16 ? 2 : 1; // rows per thread and batches (V warp)
    constexpr int VSTEP = VB * 32 / PIECES, NB = VN / VB;       // rows apart within a batch, rows per batch
    static_assert(KN <= 16 && NB <= 16, "a batch of copies is at most sixteen rows");
    const int g_pc = ptid & (PIECES - 1), g_r0 = ptid >> (D == 128 ? 4 : 3);
    // All row addresses of a batch are read first and the copies follow without a branch between them.
    auto gather_rows = [&](const char* const* rowp, unsigned char* dst, int row0, auto step, auto count) {
      constexpr int S = decltype(step)::value, N = decltype(count)::value;
      const uint32_t d0 = smem_u32(dst) + (g_pc >> 3) * (TK5 * 128);
      const char* o[N];
#pragma unroll
      for (int i = 0; i < N; ++i) o[i] = rowp[row0 + S * i];
#pragma unroll
      for (int i = 0; i < N; ++i)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d0 + sw128(row0 + S * i, g_pc & 7)), "l"(o[i] + g_pc * 16));
    };
    using KStep = std::integral_constant<int, KSTEP>;
    using KCount = std::integral_constant<int, KN>;
    using VStep = std::integral_constant<int, VSTEP>;
    using VCount = std::integral_constant<int, NB>;
    // fp8 rows: eight bytes become one 16-byte piece.  The loads of a batch are all in flight before the first is used,
    // and they are issued before the wait for the tile's buffer (load_rows8 / store_rows8).
    auto load_rows8 = [&](const char* const* rowp, int row0, auto step, auto count, uint2* w) {
      constexpr int S = decltype(step)::value, N = decltype(count)::value;
#pragma unroll
      for (int i = 0; i < N; ++i) w[i] = __ldg(reinterpret_cast<const uint2*>(rowp[row0 + S * i] + g_pc * 8));
    };
    auto store_rows8 = [&](const uint2* w, unsigned char* dst, int row0, auto step, auto count) {
      constexpr int S = decltype(step)::value, N = decltype(count)::value;
      const uint32_t d0 = smem_u32(dst) + (g_pc >> 3) * (TK5 * 128);
#pragma unroll
      for (int i = 0; i < N; ++i) sts128(d0 + sw128(row0 + S * i, g_pc & 7), widen_fp8_e5m2<DT>(w[i]));
    };
    // K(tile) / V(tile) into its buffer once wait() says the buffer is free
    auto gather_k = [&](int tile, auto wait) {
      unsigned char* dst = sK + (tile & 1) * KT_BYTES;
      if constexpr (KV8) {
        uint2 w[KN];
        load_rows8(meta[tile & 3].kptr, g_r0, KStep{}, KCount{}, w);
        wait();
        store_rows8(w, dst, g_r0, KStep{}, KCount{});
      } else {
        wait();
        gather_rows(meta[tile & 3].kptr, dst, g_r0, KStep{}, KCount{});
      }
    };
    auto gather_v = [&](int tile, auto wait) {
      unsigned char* dst = sV + (tile & 1) * KT_BYTES;
      if constexpr (KV8) {
        uint2 w[VB][NB];
#pragma unroll
        for (int i = 0; i < VB; ++i) load_rows8(meta[tile & 3].vptr, g_r0 + i * (32 / PIECES), VStep{}, VCount{}, w[i]);
        wait();
#pragma unroll
        for (int i = 0; i < VB; ++i) store_rows8(w[i], dst, g_r0 + i * (32 / PIECES), VStep{}, VCount{});
      } else {
        wait();
#pragma unroll
        for (int i = 0; i < VB; ++i) gather_rows(meta[tile & 3].vptr, dst, g_r0 + i * (32 / PIECES), VStep{}, VCount{});
      }
    };
    auto no_wait = [] {};
    // all 96 producer threads; returns the OR of the arguments
    auto producer_sync_or = [&](bool v) -> bool {
      uint32_t r;
      asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.or.pred p, 1, 96, q;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
                   : "=r"(r) : "r"((uint32_t)v) : "memory");
      return r != 0;
    };
    // in-kernel RoPE: rows 0-31 of a key tile, by the 64 key-copy threads once all their copies have landed
    auto rotate_k_front = [&](int tile) {
      RopeTile<DT, 4> rk;
      rk.fetch(p, 0, 32, ptid, 64, [&](int r) { return metas[tile & 7].rpos[r]; });
      cp_async_wait<0>();
      asm volatile("bar.sync 2, 64;\n" ::: "memory");
      rk.apply(sK + (tile & 1) * KT_BYTES, TK5 * 128, 0, ptid, 64);
    };
    if (k_role) {
      for (int t = 0; t < 3 && t < n_tiles; ++t) make_meta(t, ptid, false);
    }
    producer_sync_or(false);
    if (k_role) {
      for (int t = 0; t < 2 && t < n_tiles; ++t) gather_k(t, no_wait);
      prefetch_start(3, ptid);
      cp_async_commit();
      cp_async_wait<0>();
      if constexpr (ROPE) {
        for (int t = 0; t < 2 && t < n_tiles; ++t) rotate_k_front(t);
      }
      fence_async_smem();
      for (int t = 0; t < 2 && t < n_tiles; ++t) mbar_arrive((ROPE ? mbar_kraw0 : mbar_k0) + 8 * t);
    } else {
      if (n_tiles > 0) gather_v(0, no_wait);
      cp_async_commit();
    }
    __syncthreads();  // B0: Q is in place
    for (int it = 0; it < n_tiles; ++it) {
      if (k_role) {
        // K(it + 2) goes where K(it) was: wait until S(it) has been computed
        if (it + 2 < n_tiles) {
          if constexpr (KV8) gather_k(it + 2, [&] { mbar_wait(mbar_s0 + 8 * (it & 1), (it >> 1) & 1, &s_abort, p.status); });
          else {
            mbar_wait(mbar_s0 + 8 * (it & 1), (it >> 1) & 1, &s_abort, p.status);
            gather_rows(meta[(it + 2) & 3].kptr, sK + ((it + 2) & 1) * KT_BYTES, g_r0, KStep{}, KCount{});
          }
        }
        prefetch_start(it + 4, ptid);   // block start of this thread's entry of tile it + 4, used one tile from now
        cp_async_commit();
        // the record of tile it + 3 (its block start arrived with the copies of the previous round)
        if (it + 3 < n_tiles) make_meta(it + 3, ptid, true);
        if (ROPE && it + 2 < n_tiles) rotate_k_front(it + 2);
        cp_async_wait<0>();   // K(it + 2) has landed
        fence_async_smem();
        // K(it + 2) is in place (under in-kernel RoPE: has landed, for the softmax warps to rotate)
        if (it + 2 < n_tiles) mbar_arrive((ROPE ? mbar_kraw0 : mbar_k0) + 8 * (it & 1));
      } else {
        // V(it), requested one round ago, is reported before anything else is waited for: PV(it) needs it as soon as
        // P(it) is written
        cp_async_wait<0>();
        fence_async_smem();
        mbar_arrive(mbar_v0 + 8 * (it & 1));   // V(it) is in place
        // V(it + 1) goes where V(it - 1) was: wait until PV(it - 1) has completed
        if (it + 1 < n_tiles) {
          if constexpr (KV8) gather_v(it + 1, [&] { if (it >= 1) mbar_wait(mbar_o(it - 1), phase_o(it - 1), &s_abort, p.status); });
          else {
            if (it >= 1) mbar_wait(mbar_o(it - 1), phase_o(it - 1), &s_abort, p.status);
            gather_v(it + 1, no_wait);
          }
        }
        cp_async_commit();
      }
      // the records of tile it + 3 are complete before the next round's copies read them; all copy threads leave together
      if (producer_sync_or(s_abort != 0)) break;
    }
    cp_async_wait<0>();
  } else if (warp == 4) {
    // ================================ MMA issuer ================================
    const uint64_t dk = make_desc(0, 16, 1024);
    const uint64_t dv = make_desc(0, TK5 * 128, 1024);
    const uint32_t q_lo = smem_u32(sQ) >> 4, k_lo = smem_u32(sK) >> 4, v_lo = smem_u32(sV) >> 4;
    auto issue_s = [&](int tile) {
      const uint32_t kb = k_lo + (tile & 1) * (KT_BYTES >> 4);
      const uint32_t ts = tmem + (tile & 1) * 64;
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) {
        const uint32_t off = (kk >> 2) * ((128 * 128) >> 4) + (kk & 3) * 2;
        const uint32_t offk = (kk >> 2) * ((TK5 * 128) >> 4) + (kk & 3) * 2;
        umma(ts, dk | (uint64_t)((q_lo + off) & 0x3fffu), dk | (uint64_t)((kb + offk) & 0x3fffu), idesc_s, kk > 0);
      }
      umma_commit(mbar_s0 + 8 * (tile & 1));
    };
    __syncthreads();  // B0
    if (lane == 0) {
      for (int t = 0; t < 2 && t < n_tiles; ++t) {
        if (!mbar_wait(mbar_k0 + 8 * t, 0, &s_abort, p.status)) break;   // K(t) is in place
        tc_fence_after();
        issue_s(t);
      }
    }
    if (lane == 0) {
      // The roles meet on mbarriers only: the softmax warps run ahead to S(it + 1) as soon as P(it) is written, and the
      // copies of K(it + 2) have that whole tile to land.
      for (int it = 0; it < n_tiles; ++it) {
        const uint32_t ph = (it >> 1) & 1;
        if (!mbar_wait(mbar_p0 + 8 * (it & 1), ph, &s_abort, p.status)) break;   // P(it) is in TMEM
        if (!mbar_wait(mbar_v0 + 8 * (it & 1), ph, &s_abort, p.status)) break;   // V(it) has landed
        tc_fence_after();
        const uint32_t tp = tmem + (it & 1) * 64;                        // P(it): 32 columns of packed pairs
        const uint32_t vb = v_lo + (it & 1) * (KT_BYTES >> 4);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          umma_ts(tmem_o, tp + kk * 8, dv | (uint64_t)((vb + kk * 128) & 0x3fffu), idesc_o, (it > 0 || kk > 0) ? 1u : 0u);
        if (TWO) {   // the weights' second terms
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) umma_ts(tmem_o, tp + 32 + kk * 8, dv | (uint64_t)((vb + kk * 128) & 0x3fffu), idesc_o, 1u);
        }
        umma_commit(mbar_o(it));
        if (it + 2 < n_tiles) {
          if (!mbar_wait(mbar_k0 + 8 * (it & 1), ((it + 2) >> 1) & 1, &s_abort, p.status)) break;   // K(it + 2) is in place
          tc_fence_after();
          issue_s(it + 2);
        }
      }
    }
    __syncwarp();
  } else {
    // ================================ softmax: thread = row = TMEM lane ================================
    const uint32_t lane_base = (uint32_t)(warp * 32) << 16;
    const int prow = s_rowpos[tid];
    const float cap = p.logit_softcap;
    float m_ref = -INFINITY, l_run = 0.f;
    __syncthreads();  // B0
    if (ROPE) {
      for (int t = 0; t < 2 && t < n_tiles; ++t) rotate_k_tile(t);
    }
    for (int it = 0; it < n_tiles; ++it) {
      const MetaS& mt = metas[it & 7];
      const uint32_t ts = tmem + (it & 1) * 64 + lane_base;
      mbar_wait(mbar_s0 + 8 * (it & 1), (it >> 1) & 1, &s_abort, p.status);
      __syncwarp();
      tc_fence_after();
      float s[TK5];
      tmem_ld64(ts, s);   // one instruction: the two halves' latencies overlap
      const bool full = (mt.far_ok[0] && mt.far_ok[1]) || (mt.win_ok[0] && mt.win_ok[1]);
      // CTA-uniform slow paths, each behind its own branch (in one loop the compiler evaluates the soft-cap's tanh for
      // every element, wanted or not)
      if (cap > 0.f) {
#pragma unroll
        for (int j = 0; j < TK5; ++j) s[j] = tanhf(s[j] / cap) * cap;
      }
      if (!full) {   // per-element admission
#pragma unroll
        for (int j = 0; j < TK5; ++j)
          if (!admits(prow, mt.tpos[j], mt.twin[j] != 0, p.window)) s[j] = -INFINITY;
      }
      // row maximum with the three-input maximum: four chains of eight instructions instead of sixteen
      float mx4[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
      for (int j = 4; j + 7 < TK5; j += 8) {
        mx4[0] = max3(mx4[0], s[j], s[j + 4]);
        mx4[1] = max3(mx4[1], s[j + 1], s[j + 5]);
        mx4[2] = max3(mx4[2], s[j + 2], s[j + 6]);
        mx4[3] = max3(mx4[3], s[j + 3], s[j + 7]);
      }
#pragma unroll
      for (int j = TK5 - 4; j < TK5; ++j) mx4[j & 3] = fmaxf(mx4[j & 3], s[j]);
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * kLog2e;
      const bool need = mx > m_ref + kRescaleThreshold<DT> || (m_ref == -INFINITY && mx > -INFINITY);
      if (__any_sync(0xffffffffu, need)) {   // warp-uniform: tcgen05.ld / st are warp-collective
        const float alpha = !need ? 1.f : (m_ref == -INFINITY ? 0.f : exp2f(m_ref - mx));
        if (it > 0) {
          mbar_wait(mbar_o(it - 1), phase_o(it - 1), &s_abort, p.status);   // O is stable once PV(it - 1) is done
          __syncwarp();
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < D; c += 32) {
            float o[32];
            tmem_ld32(tmem_o + lane_base + c, o);
#pragma unroll
            for (int j = 0; j < 32; ++j) o[j] *= alpha;
            tmem_st32<false>(tmem_o + lane_base + c, o);   // the four stores are waited for together
          }
          tmem_wait_st();
        }
        if (need) {
          l_run *= alpha;
          m_ref = mx;
        }
      }
      const float base = m_ref > -INFINITY ? m_ref : 0.f;
      // the scaling and the row sum run two values per instruction
      const unsigned long long scale2 = f32x2(kLog2e, kLog2e), nbase2 = f32x2(-base, -base);
      unsigned long long sum2[4] = {0ull, 0ull, 0ull, 0ull};
      float pk[32], pk2[TWO ? 32 : 1];
#pragma unroll
      for (int j = 0; j < TK5; j += 2) {
        float x0, x1;
        f32x2_split(fma_f32x2(f32x2(s[j], s[j + 1]), scale2, nbase2), x0, x1);
        const float e0 = exp2_approx(x0), e1 = exp2_approx(x1);
        const uint32_t w = pack2<DT>(e0, e1);
        pk[j >> 1] = __uint_as_float(w);
        if constexpr (TWO) {
          pk2[j >> 1] = __uint_as_float(pack2<DT>(e0 - pair_lo<DT>(w), e1 - pair_hi<DT>(w)));
          sum2[(j >> 1) & 3] = add_f32x2(sum2[(j >> 1) & 3], f32x2(e0, e1));
          continue;
        }
        // the row sum takes the ROUNDED weights, the ones P V is computed with: numerator and denominator then carry the
        // same rounding of a row's largest terms and it cancels in O / l
        sum2[(j >> 1) & 3] = add_f32x2(sum2[(j >> 1) & 3], f32x2(pair_lo<DT>(w), pair_hi<DT>(w)));
      }
      {
        float a0, a1, b0, b1;
        f32x2_split(add_f32x2(add_f32x2(sum2[0], sum2[1]), add_f32x2(sum2[2], sum2[3])), a0, a1);
        (void)b0; (void)b1;
        l_run += a0 + a1;
      }
      if constexpr (TWO) tmem_st32<false>(ts + 32, pk2);   // ... and the second terms over the other half
      tmem_st32(ts, pk);        // P(it) over the first half of S(it)
      tc_fence_before();
      if (__any_sync(0xffffffffu, s_abort != 0)) break;   // warp-uniform: the TMEM accesses are warp-collective
      mbar_arrive(mbar_p0 + 8 * (it & 1));
      if (ROPE && it + 2 < n_tiles) rotate_k_tile(it + 2);   // K(it + 2) landed while this tile was worked on
    }
    // ---- epilogue for this thread's row ----
    bool ok = n_tiles > 0;
    if (ok) {
      ok = mbar_wait(mbar_o(n_tiles - 1), phase_o(n_tiles - 1), &s_abort, p.status);
      __syncwarp();
      tc_fence_after();
    }
    const bool warp_ok = __all_sync(0xffffffffu, ok);
    const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
#pragma unroll 1
    for (int c = 0; c < D; c += 32) {
      float o[32];
      if (warp_ok) {
        tmem_ld32(tmem_o + lane_base + c, o);
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) o[j] = 0.f;
      }
      if (SPLIT && p.n_splits > 1) {   // a normalised fp32 partial row per key range, merged by merge_kernel
        if ((tid % BQ) < rows_here) {
          float* po = p.part_o + ((((int64_t)b * p.TQ + row_t0 + tid % BQ) * p.H + h0 + tid / BQ) * p.n_splits + split) * D + c;
#pragma unroll
          for (int j = 0; j < 32; j += 4)
            *reinterpret_cast<float4*>(po + j) = make_float4(o[j] * inv, o[j + 1] * inv, o[j + 2] * inv, o[j + 3] * inv);
        }
        continue;
      }
#pragma unroll
      for (int j = 0; j < 32; j += 8) {
        uint4 w;
        w.x = pack2<DT>(o[j] * inv, o[j + 1] * inv); w.y = pack2<DT>(o[j + 2] * inv, o[j + 3] * inv);
        w.z = pack2<DT>(o[j + 4] * inv, o[j + 5] * inv); w.w = pack2<DT>(o[j + 6] * inv, o[j + 7] * inv);
        const int pc = (c + j) >> 3;
        *reinterpret_cast<uint4*>(sQ + (pc >> 3) * (128 * 128) + sw128(tid, pc & 7)) = w;
      }
    }
    if (SPLIT && p.n_splits > 1 && (tid % BQ) < rows_here)
      p.part_lse[(((int64_t)b * p.TQ + row_t0 + tid % BQ) * p.H + h0 + tid / BQ) * p.n_splits + split] =
          l_run > 0.f ? m_ref + log2f(l_run) : -INFINITY;
    if ((!SPLIT || p.n_splits == 1) && p.lse_out && (tid % BQ) < rows_here)
      p.lse_out[((int64_t)b * p.TQ + row_t0 + tid % BQ) * p.H + h0 + tid / BQ] = l_run > 0.f ? m_ref + log2f(l_run) : -INFINITY;
    tc_fence_before();
  }
  __syncthreads();  // all roles: output rows staged, every TMEM access finished
  for (int i = tid; i < 128 * PIECES && (!SPLIT || p.n_splits == 1); i += NT) {
    const int r = i >> (D == 128 ? 4 : 3), pc = i & (PIECES - 1);
    if ((r % BQ) < rows_here) {
      T* op = reinterpret_cast<T*>(p.out) + (int64_t)b * p.o_stride_b + (int64_t)(row_t0 + r % BQ) * p.o_stride_t +
              (int64_t)(h0 + r / BQ) * p.o_stride_h + pc * 8;
      *reinterpret_cast<uint4*>(op) = *reinterpret_cast<const uint4*>(sQ + (pc >> 3) * (128 * 128) + sw128(r, pc & 7));
    }
  }
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(256u) : "memory");
  }
}

template <int DT, int D, bool ROPE, bool KV8, bool SPLIT>
int launch5_ws(const hipattn_bsa_params_t& p, int BQ, int n_sub, cudaStream_t stream) {
  const size_t smem = 1024 + (D / 64) * (128 * 128 + 4 * TK5 * 128) + 4 * sizeof(Meta5) + 8 * sizeof(MetaS);
  const int NH = 128 / BQ;
  const int NBLK = cdiv(p.TQ, p.block_size_q);
  const int64_t grid = (int64_t)p.B * (p.H / NH) * NBLK * n_sub * p.n_splits;
  HIPATTN_REQUIRE(grid > 0 && grid < 0x7fffffffLL, HIPATTN_ERR_INVALID, "attention grid of %lld blocks", (long long)grid);
  auto kern = bsa_tcgen05_ws_kernel<DT, D, ROPE, KV8, SPLIT>;
  HIPATTN_CUDA_OK(allow_smem((const void*)kern, smem));
  kern<<<(unsigned)grid, 256, smem, stream>>>(p, BQ, n_sub);
  return check_launch("bsa_tcgen05_ws_kernel");
}

// One CTA waits on an mbarrier that nothing ever arrives on, through the same bounded wait the
// attention kernel uses, and then leaves normally: exercises the time-out path without any fault.
__global__ void bounded_wait_probe_kernel(uint32_t* status) {
  __shared__ __align__(8) unsigned long long bar;
  __shared__ int abort_flag;
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&bar)));
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    abort_flag = 0;
  }
  __syncthreads();
  mbar_wait(smem_u32(&bar), 0, &abort_flag, status);
  __syncthreads();
}

}  // namespace

int bounded_wait_probe(uint32_t* status, cudaStream_t stream) {
  bounded_wait_probe_kernel<<<1, 64, 0, stream>>>(status);
  return check_launch("bounded_wait_probe_kernel");
}

// Rows per CTA and CTAs per attention block, or false: 16-bit prefill with head dim 64 or 128 and attention blocks of 64 rows
// (two heads of a KV group that share their key list per CTA) or a multiple of 128 rows.
static bool tcgen05_shape(const hipattn_bsa_params_t& p, int* BQ, int* n_sub) {
  if (p.dtype == HIPATTN_F32 || (p.D != 128 && (p.D != 64 || p.rope_cos)) || p.TQ < 64) return false;
  if (p.k.fp8_e5m2 != p.v.fp8_e5m2) return false;
  if (p.out && (((uintptr_t)p.out % 16) || (p.o_stride_b % 8) || (p.o_stride_t % 8) || (p.o_stride_h % 8))) return false;
  const int Gq = p.H / p.HKV;
  if (p.block_size_q == 64 && p.heads_share_mask && (Gq % 2) == 0) { *BQ = 64; *n_sub = 1; return true; }
  if (p.block_size_q % 128 == 0) { *BQ = 128; *n_sub = p.block_size_q / 128; return true; }
  return false;
}

// CTAs of the kernel without key splits, and how many the GPU holds at once (0: another kernel takes the call)
int64_t bsa_tcgen05_ctas(const hipattn_bsa_params_t& p, int* resident, int* tile_keys) {
  int BQ, n_sub;
  if (!tcgen05_shape(p, &BQ, &n_sub)) return 0;
  *resident = 148 * 2;
  *tile_keys = TK5;
  return (int64_t)p.B * (p.H / (128 / BQ)) * cdiv(p.TQ, p.block_size_q) * n_sub;
}

template <int DT>
static int launch5(const hipattn_bsa_params_t& p, int BQ, int n_sub, cudaStream_t stream) {
  const bool split = p.n_splits > 1;
  if (p.D == 64) {
    if (p.k.fp8_e5m2) return launch5_ws<DT, 64, false, true, true>(p, BQ, n_sub, stream);
    return split ? launch5_ws<DT, 64, false, false, true>(p, BQ, n_sub, stream) : launch5_ws<DT, 64, false, false, false>(p, BQ, n_sub, stream);
  }
  if (p.k.fp8_e5m2)
    return p.rope_cos ? launch5_ws<DT, 128, true, true, true>(p, BQ, n_sub, stream) : launch5_ws<DT, 128, false, true, true>(p, BQ, n_sub, stream);
  if (p.rope_cos) return launch5_ws<DT, 128, true, false, true>(p, BQ, n_sub, stream);
  return split ? launch5_ws<DT, 128, false, false, true>(p, BQ, n_sub, stream) : launch5_ws<DT, 128, false, false, false>(p, BQ, n_sub, stream);
}

int bsa_tcgen05(const hipattn_bsa_params_t& p, cudaStream_t stream, bool* handled) {
  *handled = false;
  int BQ, n_sub;
  if (!tcgen05_shape(p, &BQ, &n_sub)) return HIPATTN_OK;
  *handled = true;
  return p.dtype == HIPATTN_BF16 ? launch5<HIPATTN_BF16>(p, BQ, n_sub, stream) : launch5<HIPATTN_F16>(p, BQ, n_sub, stream);
}

}  // namespace hipattn
