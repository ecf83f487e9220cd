// Scan stage of the mask estimator for 16-bit prefill, few pooled rows: the keys of a tile stay, the query blocks that selected them
// pass by.
//
// The stages after the first look at the sub-chunks of what each query block kept.  With few pooled rows (16 per head,
// 64 for the four heads of a KV head) the rows that the halving search asks for are more bytes than the queries: 9 rows a
// head and chunk of 32, 72 KB per kept chunk of 256 tokens and query block, against 16 KB of pooled queries.  So the lists
// are turned round: a CTA takes 256 consecutive tokens of a KV head, keeps them in shared memory as the A operand, and streams
// the pooled queries of the blocks that kept this chunk through a ring as the B operand, 256 rows a stage.  Everything
// after the product is as in scan_query_tiles.cu: row maxima per group (one head of one query block), bounds, and the halving
// search replayed on them (scan_tiles.cuh).
//
// pool_queries_kernel writes the pooled queries in operand layout, list_queries_kernel the blocks that kept a chunk.
//
// Bound: as scan_query_tiles.cu, the chain from an accumulator's MMAs to its release.  128k prefill, second stage (chunk
// 32, 4 heads x 16 rows): 3146 us by rounds, which were bound by their gathers (10.7 TB/s from L2), 1862 here (1740 on
// another board) and 74 for the pooled queries and the lists; ragged fp16 prefill 179 -> 97 us and less than 20.
#include "host_kernels.h"
#include "scan_tiles.cuh"

namespace hipattn {
namespace {

constexpr int kFirstSearchWarp = 4, kSearchSets = 3, kSearchWarps = 4 * kSearchSets;
constexpr int kThreads = (kFirstSearchWarp + kSearchWarps) * 32;
constexpr int kRows = 16, kChunk = 32;   // pooled rows of a head, tokens of a chunk
constexpr int kTile = 256;               // tokens of a CTA

// A launch takes a slice of the query blocks, nd of them from d0 on, of nb sequences from b0 on.
struct KeyTiles {
  unsigned char* pooled;         // [nb, HKV, nd][rows / 8][D / 64][8 rows][128 B], swizzled; rows = heads of a KV head x pooled rows
  float* q_max;                  // [nb, H, nd] largest |pooled query|
  int32_t* last;                 // [nb, nd] chunks that begin beyond this position are not active
  int2* entries;                 // [nb, n_grid, nd]: query block of the slice, position of the chunk in its list of kept ones
  int32_t* counts;               // [nb, n_grid]
  int b0, nb, d0, nd;
  int n_grid, sink, c_prev;      // chunks of the stage before: grid of c_prev tokens from `sink`
};

// ---- pooled queries of a (batch, KV head, query block), rows beyond the last one repeat the first ----
// (All query rows of a piece are requested before the first is added up: one after the other 150 us for the 268 MB of the 128k
// prefill, 61 here.)
template <int DT, int D>
__global__ void __launch_bounds__(256) pool_queries_kernel(const hipattn_scan_params_t p, const KeyTiles kt) {
  using T = typename Elem<DT>::type;
  constexpr int PIECES = D / 8, KB = D / 64, BATCH = 4;
  const int Gq = p.H / p.HKV;
  int64_t bid = blockIdx.x;
  const int d = (int)(bid % kt.nd); bid /= kt.nd;
  const int hkv = (int)(bid % p.HKV), bl = (int)(bid / p.HKV), b = kt.b0 + bl;
  const int t0 = (kt.d0 + d) * p.block_size_q, Rv = min(kRows, (p.TQ - t0 + p.stride_q - 1) / p.stride_q);
  __shared__ int s_max[16];
  if (threadIdx.x < 16) s_max[threadIdx.x] = 0;
  __syncthreads();
  unsigned char* dst = kt.pooled + (((int64_t)bl * p.HKV + hkv) * kt.nd + d) * Gq * kRows * D * 2;
  for (int i = threadIdx.x; i < Gq * kRows * PIECES; i += 256) {
    const int pc = i % PIECES, rr = i / PIECES, hh = rr / kRows, r = rr % kRows;
    const int t = t0 + (r < Rv ? r : 0) * p.stride_q;
    const T* src = reinterpret_cast<const T*>(p.q) + (int64_t)b * p.q_stride_b + (int64_t)(hkv * Gq + hh) * p.q_stride_h + pc * 8;
    float sum[8], v[8], cnt = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) sum[e] = 0.f;
    for (int o0 = 0; o0 < p.stride_q; o0 += BATCH) {   // (sums in row order, as pooled_query_piece has them)
      uint4 raw[BATCH];
#pragma unroll
      for (int u = 0; u < BATCH; ++u)
        if (o0 + u < p.stride_q && t + o0 + u < p.TQ) raw[u] = __ldg(reinterpret_cast<const uint4*>(src + (int64_t)(t + o0 + u) * p.q_stride_t));
#pragma unroll
      for (int u = 0; u < BATCH; ++u)
        if (o0 + u < p.stride_q && t + o0 + u < p.TQ) {
          widen_piece<DT>(raw[u], v);
#pragma unroll
          for (int e = 0; e < 8; ++e) sum[e] = __fadd_rn(sum[e], v[e]);
          cnt += 1.f;
        }
    }
    mean_and_scale<DT>(sum, cnt, p.q_scale, v);
    *reinterpret_cast<uint4*>(dst + (rr >> 3) * (KB * 1024) + (pc >> 3) * 1024 + sw128(rr & 7, pc & 7)) =
        make_uint4(pack2<DT>(v[0], v[1]), pack2<DT>(v[2], v[3]), pack2<DT>(v[4], v[5]), pack2<DT>(v[6], v[7]));
    float m = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) m = fmaxf(m, fabsf(v[e]));
    // (the pieces of a warp belong to one head: 32 divides a head's kRows * PIECES; non-negative floats order as ints)
    const int top = __reduce_max_sync(0xffffffffu, __float_as_int(m));
    if ((threadIdx.x & 31) == 0) atomicMax(&s_max[hh], top);
  }
  if (threadIdx.x < 32 && hkv == 0) {
    const int m = block_min_position(p, b, t0, Rv, threadIdx.x);
    if (threadIdx.x == 0) kt.last[bl * kt.nd + d] = max(m - p.scan_window, 0);
  }
  __syncthreads();
  if (threadIdx.x < Gq) kt.q_max[((int64_t)bl * p.H + hkv * Gq + threadIdx.x) * kt.nd + d] = __int_as_float(s_max[threadIdx.x]);
}

// ---- the query blocks whose list holds a chunk of the grid, and where; blocks it is not active for are left out ----
__global__ void __launch_bounds__(256) list_queries_kernel(const int32_t* __restrict__ left, int n, int per, int BDST, const KeyTiles kt) {
  const int g = blockIdx.x % kt.n_grid, bl = blockIdx.x / kt.n_grid;
  const int want = kt.sink + g * kt.c_prev, kept = n / per, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __shared__ int s_warp[8];
  int2* out = kt.entries + ((int64_t)bl * kt.n_grid + g) * kt.nd;
  int total = 0;
  for (int d0 = 0; d0 < kt.nd; d0 += 256) {
    const int d = d0 + threadIdx.x;
    int lo = 0;
    bool in = false;
    if (d < kt.nd && want <= __ldg(kt.last + bl * kt.nd + d)) {
      const int32_t* row = left + ((int64_t)(kt.b0 + bl) * BDST + kt.d0 + d) * n;   // the kept chunks ascend; each is `per` entries
      int hi = kept;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(row + (int64_t)mid * per) < want) lo = mid + 1; else hi = mid;
      }
      in = lo < kept && __ldg(row + (int64_t)lo * per) == want;
    }
    const unsigned m = __ballot_sync(0xffffffffu, in);
    if (lane == 0) s_warp[warp] = __popc(m);
    __syncthreads();
    int before = total, all = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      if (w < warp) before += s_warp[w];
      all += s_warp[w];
    }
    if (in) out[before + __popc(m & ((1u << lane) - 1u))] = make_int2(d, lo);
    total += all;
    __syncthreads();
  }
  if (threadIdx.x == 0) kt.counts[bl * kt.n_grid + g] = total;
}

// ---- per-head results of chunks that no list holds: not active, so as they came ----
__global__ void __launch_bounds__(256) untouched_heads_kernel(const hipattn_scan_params_t p, int64_t total) {
  const int64_t per_row = (int64_t)p.H * p.n_chunks;
  for (int64_t i = blockIdx.x * 256LL + threadIdx.x; i < total; i += gridDim.x * 256LL) {
    const int64_t c = i / per_row * p.n_chunks + i % p.n_chunks;
    p.left_out[i] = p.left[c];
    p.right_out[i] = p.right[c];
    p.score_out[i] = HIPATTN_SCORE_INIT;
  }
}

// CHECKED: per-head results, statistics, and in check mode every score by both definitions.
template <int DT, int D, bool CHECKED, bool PATIENT>
__global__ void __launch_bounds__(kThreads, 1) scan_key_tiles_kernel(const hipattn_scan_params_t p, const KeyTiles t) {
  constexpr int ROWB = D * 2, PIECES = ROWB / 16, KB = D / 64;
  constexpr int R = kRows, CHUNK = kChunk, COLS = 256, NG = COLS / R;   // columns of a stage, groups (query block, head)
  constexpr int A_BLOCK = 128 * 128, A_TILE = KB * A_BLOCK;             // two tiles of 128 keys, an accumulator's rows each
  constexpr int Q_STAGE = COLS * ROWB, STAGES = 2;
  constexpr int TAB_WORDS = NG * kTabStride;

  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ unsigned long long s_full[STAGES], s_empty[STAGES], s_accf[kSearchSets][2], s_acce[2];
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  unsigned char* sA = smem;                                // [tile][KB][128 keys][128 B], swizzled
  unsigned char* sQ = sA + 2 * A_TILE;                     // [stage][COLS / 8][KB][8 rows][128 B], swizzled
  uint32_t* tabs = reinterpret_cast<uint32_t*>(sQ + STAGES * Q_STAGE);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int Gq = p.H / p.HKV, BDST = cdiv(p.TQ, p.block_size_q), EB = NG / Gq;   // entries of a stage
  const int parts = t.c_prev / kTile;
  int64_t bid = blockIdx.x;
  const int part = (int)(bid % parts); bid /= parts;
  const int gi = (int)(bid % t.n_grid); bid /= t.n_grid;
  const int hkv = (int)(bid % p.HKV), bl = (int)(bid / p.HKV), b = t.b0 + bl;
  const int count = __ldg(t.counts + bl * t.n_grid + gi);
  if (count == 0) return;
  const int base = t.sink + gi * t.c_prev + part * kTile;   // the CTA's first token
  const int2* entries = t.entries + ((int64_t)bl * t.n_grid + gi) * t.nd;
  const int stages_total = cdiv(count, EB);
  const int64_t bh = (int64_t)b * p.HKV + hkv, slice = (int64_t)bl * p.HKV + hkv;
  const int entry_bytes = Gq * R * ROWB;
  const char* kbase = reinterpret_cast<const char*>(p.k_scaled) + bh * p.T * ROWB;

  if (tid == 0) {
    for (int i = 0; i < STAGES; ++i) { mbar_init(smem_u32(&s_full[i]), 1); mbar_init(smem_u32(&s_empty[i]), 2); }
    for (int i = 0; i < 2 * kSearchSets; ++i) mbar_init(smem_u32(&s_accf[i >> 1][i & 1]), 1);
    for (int i = 0; i < 2; ++i) mbar_init(smem_u32(&s_acce[i]), 4);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    s_abort = 0;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s_tmem)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  // ---- the keys: 256 rows, 16 bytes a thread and turn; tokens beyond the keys are the last one ----
  for (int i = tid; i < kTile * PIECES; i += kThreads) {
    const int rr = i / PIECES, pc = i % PIECES, tk = min(base + rr, p.T - 1);
    cp_async16(sA + (rr >> 7) * A_TILE + (pc >> 3) * A_BLOCK + sw128(rr & 127, pc & 7), kbase + (int64_t)tk * ROWB + pc * 16);
  }
  cp_async_commit();
  cp_async_wait<0>();
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;

  if (warp == 0) {
    // ---- pooled queries: one bulk copy per entry ----
    if (lane == 0) {
      const unsigned char* src = t.pooled + slice * t.nd * entry_bytes;
      int slot = 0, use = 0, next = __ldg(&entries[0].x), k = 0;
      for (int e = 0; k < stages_total; ++k) {
        if (use > 0 && !mbar_wait_quick<PATIENT>(smem_u32(&s_empty[slot]), (use - 1) & 1, &s_abort, p.status)) break;
        const int ne = min(EB, count - k * EB);
        const uint32_t bar = smem_u32(&s_full[slot]), dst = smem_u32(sQ) + slot * Q_STAGE;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(ne * entry_bytes) : "memory");
        for (int i = 0; i < ne; ++i, ++e) {
          const int d = next;
          if (e + 1 < count) next = __ldg(&entries[e + 1].x);
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                       ::"r"(dst + i * entry_bytes), "l"(src + (int64_t)d * entry_bytes), "r"(entry_bytes), "r"(bar) : "memory");
        }
        if (++slot == STAGES) { slot = 0; ++use; }
      }
      for (int i = max(0, k - STAGES); i < k; ++i) mbar_drain(smem_u32(&s_full[i % STAGES]), (i / STAGES) & 1);
    }
    __syncwarp();
  } else if (warp == 2 || warp == 3) {
    // ---- MMAs: a thread for each key tile and accumulator ----
    const int acc = warp - 2;
    if (lane == 0) {
      const uint64_t da0 = make_desc(smem_u32(sA) + acc * A_TILE, 16, 1024), db0 = make_desc(smem_u32(sQ), 16, KB * 1024);
      int slot = 0, use = 0, set = acc, k = 0, last = 0;
      for (; k < stages_total; ++k) {
        if (!mbar_wait_quick<PATIENT>(smem_u32(&s_full[slot]), use & 1, &s_abort, p.status)) break;
        if (k > 0 && !mbar_wait_quick<PATIENT>(smem_u32(&s_acce[acc]), (k - 1) & 1, &s_abort, p.status)) break;
        tc_fence_after();
        const uint32_t idesc = make_idesc(DT == HIPATTN_BF16 ? 1 : 0, 128, min(EB, count - k * EB) * Gq * R, 0);
        const uint64_t db = db0 + (uint64_t)((slot * Q_STAGE) >> 4);
#pragma unroll
        for (int q = 0; q < D / 16; ++q)
          umma(tmem + acc * COLS, da0 + (uint64_t)(((q >> 2) * A_BLOCK + (q & 3) * 32) >> 4), db + (uint64_t)(((q >> 2) * 1024 + (q & 3) * 32) >> 4), idesc,
               q > 0 ? 1u : 0u);
        umma_commit(smem_u32(&s_empty[slot]));
        umma_commit(smem_u32(&s_accf[set][acc]));   // (last: waited for before the role ends)
        last = set;
        set += 2;
        if (set >= kSearchSets) set -= kSearchSets;
        if (++slot == STAGES) { slot = 0; ++use; }
      }
      // (every third accumulator of a thread is a set's)
      if (k > 0) mbar_drain(smem_u32(&s_accf[last][acc]), ((k - 1) / kSearchSets) & 1);
    }
    __syncwarp();
  } else if (warp >= kFirstSearchWarp) {
    // ---- searches: the sets take the accumulators in turn; a warp reads its quarter of the TMEM lanes ----
    const int set = (warp - kFirstSearchWarp) >> 2, quarter = warp & 3;
    uint32_t* tab = tabs + (warp - kFirstSearchWarp) * TAB_WORDS;
    const uint32_t my_tmem = tmem + ((uint32_t)(quarter * 32) << 16);
    const int per = t.c_prev / CHUNK, n = p.n_chunks;
    const int64_t row0 = (int64_t)b * BDST + t.d0;   // row of the slice's first block
    const bool counting = p.access_counter != nullptr;
    int32_t* counter = counting ? p.access_counter + (int64_t)b * p.access_stride_b + (int64_t)hkv * p.access_stride_h : nullptr;
    // this lane's key of each tile: magnitudes and the slot of the access counter
    const int tk0 = min(base + quarter * 32 + lane, p.T - 1), tk1 = min(base + 128 + quarter * 32 + lane, p.T - 1);
    const float abs0 = __ldg(p.key_abs + bh * p.T + tk0), abs1 = __ldg(p.key_abs + bh * p.T + tk1);
    const int64_t mark0 = counting ? access_index(p.k, b, tk0) : (int64_t)-1, mark1 = counting ? access_index(p.k, b, tk1) : (int64_t)-1;
    // this lane's task: group g (entry g / Gq of the stage, head g % Gq) of the warp's chunk; the upper half of the warp has none
    const int g = lane % NG, eg = g / Gq;
    const float* q_max = t.q_max + ((int64_t)bl * p.H + hkv * Gq + g % Gq) * t.nd;
    const bool walker = lane < NG;
    // What a round needs from memory is requested ahead: a lane's entry two rounds, what hangs on it one.
    struct Next {
      int d, pt, code;
      float q_max;
    };
    auto entry_of = [&](int u) {
      const int e = (u >> 1) * EB + eg;
      return e < count ? __ldg(entries + e) : make_int2(-1, 0);
    };
    auto chunk_of = [&](int u, int j) { return j * per + (part * kTile + (u & 1) * 128 + quarter * 32) / CHUNK; };
    auto details = [&](int u, int2 e) {
      Next x{e.x, 0, 0, 0.f};
      if (e.x >= 0) {
        x.pt = __ldg(t.last + bl * t.nd + e.x);
        x.q_max = __ldg(q_max + e.x);
        x.code = __ldcg(p.score_max + (row0 + e.x) * n + chunk_of(u, e.y));
      }
      return x;
    };
    int2 ent = entry_of(set), ent2 = entry_of(set + kSearchSets);
    Next nx = details(set, ent);
    const bool per_head = CHECKED && p.left_out != nullptr;
    unsigned st_keys = 0, st_fb = 0, st_wrong = 0;
    float st_ratio = 0.f;
    uint32_t phase = 0;
    bool ok = true;
    for (int u = set; u < stages_total * 2 && ok; u += kSearchSets) {
      const int acc = u & 1, j = ent.y;   // (accumulator = key tile)
      const Next cur = nx;
      ent = ent2;
      nx = details(u + kSearchSets, ent);
      ent2 = entry_of(u + 2 * kSearchSets);
      const int ng = min(EB, count - (u >> 1) * EB) * Gq;
      const int l = base + acc * 128 + quarter * 32;   // the warp's chunk: CHUNK tokens from here
      const bool valid = walker && cur.d >= 0;
      ok = __all_sync(0xffffffffu, mbar_wait_quick<PATIENT>(smem_u32(&s_accf[set][acc]), phase >> acc & 1, &s_abort, p.status));
      if (!ok) break;
      phase ^= 1u << acc;
      tc_fence_after();
      float x[NG];
      group_maxima<R, NG>(my_tmem + acc * COLS, ng, x);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&s_acce[acc]));
      // the rounded score lies between round(x - e) and round(x + e)
      const float unit = kEps * cur.q_max * 1.01f, s_abs = acc ? abs1 : abs0;
#pragma unroll
      for (int i = 0; i < NG; ++i) {
        const float e_ = __shfl_sync(0xffffffffu, unit, i) * s_abs;
        tab[i * kTabStride + lane] = pack2<DT>(x[i] - e_, x[i] + e_);
      }
      __syncwarp();
      // strict score of a token for the group of lane `owner`
      const int d_mine = cur.d;
      auto strict_of = [&](int tk, int owner) -> float {
        // one pooled row per lane, from the operand's copy in memory (its stage may hold other queries by now)
        const int d = __shfl_sync(0xffffffffu, d_mine, owner), rr = owner % NG % Gq * R + lane % R;
        const uint4* kp = reinterpret_cast<const uint4*>(kbase + (int64_t)tk * ROWB);
        const unsigned char* qp = t.pooled + (slice * t.nd + d) * (int64_t)entry_bytes + (rr >> 3) * (KB * 1024);
        float a = 0.f;
#pragma unroll 1
        for (int p0 = 0; p0 < PIECES; p0 += 8) {
          uint4 kw[8], qw[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            kw[e] = __ldg(kp + p0 + e);
            qw[e] = __ldg(reinterpret_cast<const uint4*>(qp + (p0 >> 3) * 1024 + sw128(rr & 7, e)));
          }
#pragma unroll
          for (int e = 0; e < 8; ++e) a = strict_piece<DT>(qw[e], kw[e], a);
        }
        float top = fmaxf(a, -INFINITY);   // (a score that is not a number is the lowest)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
        return top;
      };
      if constexpr (CHECKED) {
#pragma unroll 1
        for (int i = 0; i < ng; ++i) {
          uint32_t* w = tab + i * kTabStride + lane;
          ++st_keys;
          if (lo_f32<DT>(*w) != hi_f32<DT>(*w)) ++st_fb;
          if (p.mode != HIPATTN_SCAN_CHECK) continue;
          const float e_ = __shfl_sync(0xffffffffu, unit, i) * s_abs;
#pragma unroll 1
          for (int o = 0; o < 32; ++o) {
            const float raw = strict_of(min(l + o, p.T - 1), i), ex = Elem<DT>::round(raw);
            if (lane == o) {
              if (lo_f32<DT>(*w) == hi_f32<DT>(*w) && hi_f32<DT>(*w) != ex) ++st_wrong;
              if (e_ > 0.f) st_ratio = fmaxf(st_ratio, fabsf(x[i] - raw) / e_);
              *w = pack2<DT>(ex, ex);
            }
          }
        }
        __syncwarp();
      }
      const int64_t row = row0 + cur.d;
      const int c = chunk_of(u, j);
      const float so_far = decode_score(cur.code);
      uint32_t seen = 0;
      int off = 0;
      float slo, shi, best;
      bool closed = search_whole<DT, CHUNK>(tab + g * kTabStride, off, slo, shi, seen);
      const bool plain = __all_sync(0xffffffffu, !valid || (l + CHUNK - 1 <= cur.pt && l + CHUNK <= p.T));
      if (!valid) { slo = shi = HIPATTN_SCORE_INIT; seen = 0; }
      best = fmaxf(slo, so_far);
      for (int o = 1; o < Gq; o <<= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, o));
      // a score that may raise the chunk's best has to be certain
      closed |= !valid;
      const bool compared = plain && !per_head && __all_sync(0xffffffffu, closed);
      if (!compared || __any_sync(0xffffffffu, shi > slo && shi > best)) {
        ChunkTask task;
        task.valid = valid;
        task.l = l;
        task.r = l + CHUNK;
        task.pt = cur.pt;
        task.first = l;
        task.row0 = 0;
        task.known = so_far;
        task.tab = tab + g * kTabStride;
        task.slo = compared ? slo : HIPATTN_SCORE_INIT;
        task.shi = compared ? shi : HIPATTN_SCORE_INIT;
        search_chunks<DT, CHUNK>(task, p.T, Gq, compared, per_head, strict_of, [](int) {});
        if (task.valid && task.out_of_range) atomicOr(p.status, HIPATTN_STATUS_TOKEN_RANGE);
        if (per_head && valid) {
          const int64_t o = (row * p.H + hkv * Gq + g % Gq) * n + c;
          p.left_out[o] = task.l;
          p.right_out[o] = task.r;
          p.score_out[o] = task.score;
        }
        seen = compared ? seen : (valid ? task.seen : 0);
        best = fmaxf(task.score, so_far);
        for (int o = 1; o < Gq; o <<= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, o));
      }
      if (valid && g % Gq == 0 && best > so_far) atomicMax(p.score_max + row * n + c, encode_score(best));
      if (counting) {
        seen = __reduce_or_sync(0xffffffffu, seen);
        const int64_t m = acc ? mark1 : mark0;
        if ((seen >> lane & 1) && m >= 0 && m < p.access_n) counter[m] = 1;
      }
      __syncwarp();   // the table is written anew
    }
    if (CHECKED && p.stats) add_stats(p.stats, st_keys, st_fb, st_wrong, st_ratio);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512u) : "memory");
  }
}

template <int DT, int D>
int run(const hipattn_scan_params_t& p, const KeyTiles& t, cudaStream_t stream) {
  pool_queries_kernel<DT, D><<<(unsigned)(t.nb * p.HKV * t.nd), 256, 0, stream>>>(p, t);
  int rc = check_launch("pool_queries_kernel");
  if (rc) return rc;
  list_queries_kernel<<<(unsigned)(t.nb * t.n_grid), 256, 0, stream>>>(p.left, p.n_chunks, t.c_prev / kChunk, cdiv(p.TQ, p.block_size_q), t);
  rc = check_launch("list_queries_kernel");
  if (rc) return rc;
  const size_t smem = 1024 + (size_t)kTile * D * 2 + 2 * (size_t)256 * D * 2 + (size_t)kSearchWarps * (256 / kRows) * kTabStride * 4;
  const int64_t grid = (int64_t)t.nb * p.HKV * t.n_grid * (t.c_prev / kTile);
  HIPATTN_REQUIRE(grid > 0 && grid < 0x7fffffffLL, HIPATTN_ERR_INVALID, "scan grid of %lld blocks", (long long)grid);
  auto kern = p.left_out || p.stats || p.mode == HIPATTN_SCAN_CHECK ? scan_key_tiles_kernel<DT, D, true, true> : scan_key_tiles_kernel<DT, D, false, true>;
  if constexpr (DT == HIPATTN_BF16 && D == 128)
    if (without_patience()) kern = scan_key_tiles_kernel<DT, D, false, false>;
  HIPATTN_CUDA_OK(allow_smem((const void*)kern, smem));
  kern<<<(unsigned)grid, kThreads, smem, stream>>>(p, t);
  return check_launch("scan_key_tiles_kernel");
}

// Scratch of a launch, and how a call is cut so that no launch needs more than kMaxScratch (a single query block may): whole
// sequences as long as one fits, else query blocks of one sequence in equal parts.  The lists alone are 8 bytes a grid chunk and
// query block, which grows with the square of the length (a million tokens on themselves: 2.1 GB of pooled queries of 32 heads, 0.5 GB
// of lists).  A launch of that size fetches each key once for hundreds of query blocks.
constexpr int64_t kMaxScratch = 128ll << 20;
struct Slices {
  int n_grid, nb, nd;   // chunks of the grid, most sequences and query blocks of a launch
  int64_t pooled, q_max, last, entries, counts;   // bytes
  int64_t bytes() const { return pooled + q_max + last + entries + counts; }
};
Slices plan_slices(const hipattn_scan_params_t& p, int sink, int c_prev) {
  const int BDST = cdiv(p.TQ, p.block_size_q);
  auto align16 = [](int64_t x) { return (x + 15) / 16 * 16; };
  Slices s;
  s.n_grid = cdiv(p.T - sink, c_prev);
  auto size = [&](int nb, int nd) {
    s.nb = nb;
    s.nd = nd;
    const int64_t blocks = (int64_t)nb * nd;
    s.pooled = blocks * p.H * kRows * p.D * 2;
    s.q_max = align16(blocks * p.H * 4);
    s.last = align16(blocks * 4);
    s.entries = align16(blocks * s.n_grid * 8);
    s.counts = align16((int64_t)nb * s.n_grid * 4);
    return s.bytes();
  };
  const int64_t one = size(1, BDST);
  if (one <= kMaxScratch) size((int)min((int64_t)p.B, kMaxScratch / one), BDST);
  else size(1, cdiv(BDST, (int)min((int64_t)BDST, (one + kMaxScratch - 1) / kMaxScratch)));
  return s;
}

// Whether the keys are worth keeping.  A CTA's keys, operands and start cost 5 us, its list runs as one chain, and CTAs are few where
// heads and chunks are; the rounds pay per (query block, head) instead.  In units of 14 ns, what the rounds lose on a
// list entry of 16 groups (head, block): they take `listed` of them and a fifth per block and head, the key tiles 50 per
// entry of the longest list, that of a chunk which every block keeps, and 400 per CTA of a multiprocessor.  Entries are counted for
// queries that are the last TQ of T, without the blocks that a chunk is not active for.  On 1235 random calls (1 to 16 heads a KV
// head, 1 to 16 KV heads, 200 to 16384 queries of 1400 to 100000 tokens, 8 to 128 kept chunks) the stage took 379 ms by rounds, 247.4 by
// the better of the two, 248.2 by this rule, 24 calls slower than by rounds by more than 3 %, 1.5 times at most (65 -> 97 us: three
// chunks of 2595 tokens).  A threshold of 64 groups a chunk, whatever its blocks and CTAs, had 253.2, 208 calls and 3.8 times at
// most (16 heads of one KV head and 2309 tokens: 16 us by rounds, 59 here, on nine CTAs).
bool worth_turning(const hipattn_scan_params_t& p, int sink, int c_prev) {
  const int G = p.H / p.HKV, BDST = cdiv(p.TQ, p.block_size_q), kept = p.n_chunks / (c_prev / kChunk);
  int64_t listed = 0, longest = 0, chunks = 0;
  for (int d = 0; d < BDST; ++d) {
    const int64_t reach = (int64_t)p.T - p.TQ + (int64_t)d * p.block_size_q - p.scan_window - sink;
    if (reach < 0) continue;
    chunks = reach / c_prev + 1;
    listed += min((int64_t)kept, chunks);
    ++longest;
  }
  const double pairs = (double)p.B * p.HKV * (c_prev / kTile), entries = G / 16.0;
  return pairs * listed * entries + p.B * (double)p.H * BDST / 5 > 50 * longest * entries + 400 * fmax(1.0, pairs * chunks / 148);
}

}  // namespace

// Bytes of scratch that scan_key_tiles needs for this call, 0 where it does not take it: chunks of 32 cut from chunks of whole key
// tiles, 16 pooled rows a head, no in-kernel RoPE, all of the per-head results or none.  With 32 pooled rows the tiles
// took 0.99 to 1.4 of the rounds' time, "relative" 0.92 to 1.6.
int64_t scan_key_tiles_scratch(const hipattn_scan_params_t& p, int sink, int c_prev) {
  const int R = p.block_size_q / p.stride_q, G = p.H / p.HKV, BDST = cdiv(p.TQ, p.block_size_q);
  const bool heads = p.left_out && p.right_out && p.score_out;
  if (p.mode == HIPATTN_SCAN_STRICT || p.dtype == HIPATTN_F32 || (p.D != 64 && p.D != 128) || p.key_abs == nullptr || p.k_scaled == nullptr) return 0;
  if (p.rope_mode != HIPATTN_ROPE_NONE || (!heads && (p.left_out || p.right_out || p.score_out))) return 0;
  if (R != kRows || (G & (G - 1)) != 0 || G > 16 || p.TQ <= p.stride_q) return 0;
  if (p.chunk_size != kChunk || c_prev % kTile != 0 || p.n_chunks % (c_prev / kChunk) != 0 || p.T <= sink) return 0;
  if ((int64_t)p.B * p.T * p.HKV >= 0x7fffffffLL || (int64_t)p.B * p.HKV * BDST >= 0x7fffffffLL) return 0;
  const ScanChoice choice = scan_choice();
  if (choice == SCAN_BY_MMA || choice == SCAN_BY_ROUNDS || (choice != SCAN_BY_TILES && !worth_turning(p, sink, c_prev))) return 0;
  return plan_slices(p, sink, c_prev).bytes();
}

// The scan stage on a list that select_stage has made from chunks of c_prev tokens (kept chunks on the grid from `sink`, ascending,
// each cut into whole chunks of p.chunk_size); scratch: 16-byte aligned, used by one launch after the other.
int scan_key_tiles(const hipattn_scan_params_t& p, int sink, int c_prev, void* scratch, cudaStream_t stream) {
  const Slices s = plan_slices(p, sink, c_prev);
  KeyTiles t;
  unsigned char* at = (unsigned char*)scratch;
  auto take = [&](int64_t bytes) {
    unsigned char* x = at;
    at += bytes;
    return x;
  };
  t.pooled = take(s.pooled);
  t.q_max = (float*)take(s.q_max);
  t.last = (int32_t*)take(s.last);
  t.entries = (int2*)take(s.entries);
  t.counts = (int32_t*)take(s.counts);
  t.n_grid = s.n_grid;
  t.sink = sink;
  t.c_prev = c_prev;
  const int BDST = cdiv(p.TQ, p.block_size_q);
  if (p.left_out) {
    const int64_t total = (int64_t)p.B * BDST * p.H * p.n_chunks;
    untouched_heads_kernel<<<(unsigned)min((total + 255) / 256, (int64_t)148 * 16), 256, 0, stream>>>(p, total);
    const int rc = check_launch("untouched_heads_kernel");
    if (rc) return rc;
  }
  for (t.b0 = 0; t.b0 < p.B; t.b0 += s.nb) {
    t.nb = min(s.nb, p.B - t.b0);
    for (t.d0 = 0; t.d0 < BDST; t.d0 += s.nd) {
      t.nd = min(s.nd, BDST - t.d0);
      int rc;
      if (p.dtype == HIPATTN_BF16) rc = p.D == 128 ? run<HIPATTN_BF16, 128>(p, t, stream) : run<HIPATTN_BF16, 64>(p, t, stream);
      else rc = p.D == 128 ? run<HIPATTN_F16, 128>(p, t, stream) : run<HIPATTN_F16, 64>(p, t, stream);
      if (rc) return rc;
    }
  }
  return HIPATTN_OK;
}

}  // namespace hipattn
