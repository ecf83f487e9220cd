// Scan stage of the mask estimator for 16-bit prefill, small chunks: every token of every active chunk is fetched ONCE for
// several query heads of a KV head, scored on tcgen05, and the halving search is replayed on the scores (scan_tiles.cuh).
//
// The kernel that goes by rounds (scan_stage_tcgen05.cu) fetches the rows that each head's rounds ask for: 5 rows a head
// for a chunk of 8, 20 for the four heads of a KV head, and every round is a dependent chain of copy, MMA, read, decision.
// Here a chunk costs its 8 rows, nothing depends on anything, and the work streams: the pooled queries of up to 256
// (head, row) pairs stay in shared memory as the B operand, key tiles of 128 tokens pass through a ring as the A operand,
// D = K Q^T lands in one of two 256-column TMEM accumulators.
//
// Roles: warps 0 and 1 copy key rows (16-byte cp.async into the 128-byte-swizzled operand layout), warps 2 and 3 issue the MMAs,
// three sets of four warps take the accumulators in turn: row maxima per head, bounds, searches.
//
// Bound: the chain of an accumulator, MMAs 1024 to 1200 cycles (head dim 128, 256 columns), commit 530, row maxima 1000,
// release 200: two accumulators hold 512 columns, all of TMEM, so a tile takes 1500 where its MMAs alone would take 1024.
// Shared memory is the reason why the links are long: the MMAs read 96 of its 128 bytes a cycle (half accumulators of 128
// columns all 128, and were slower) and the loads of everyone else queue behind them.  128k prefill, third stage
// (chunk 8, 4 heads x 64 rows): 2750 us by rounds, 1985 here (1820 on another board); 131072 queries of 64 heads (8 x 128 rows): 28.8
// -> 23.6 ms.  On the way, on the board of the 1820: two sets 2190, one MMA thread 2080, strict scores that read shared memory
// piece by piece 2030.
#include "scan_tiles.cuh"

namespace hipattn {
namespace {

constexpr int kCopyWarps = 2, kFirstSearchWarp = 4, kSearchSets = 3, kSearchWarps = 4 * kSearchSets;
constexpr int kTileThreads = (kFirstSearchWarp + kSearchWarps) * 32;
constexpr int kTileChunk = 8;          // tokens of a chunk
constexpr int kTileSlack = 1024;       // padding in front of the operand tiles
constexpr size_t kTileSmem = 227 * 1024 - 512;   // dynamic shared memory beside the kernel's own variables

struct QueryTiles {
  int passes;        // column passes per key tile: the pooled queries of passes * NG heads stay in shared memory
  int head_groups;   // CTAs of a (batch, KV head, query block) that share out its heads
  int stages;        // key tiles in the ring
  int split;         // CTAs that share out the key tiles
  int check;
};

template <int DT, int D, int R, bool PATIENT>
__global__ void __launch_bounds__(kTileThreads, 1) scan_query_tiles_kernel(const hipattn_scan_params_t p, const QueryTiles cfg) {
  constexpr int ROWB = D * 2, PIECES = ROWB / 16, KB = D / 64;
  constexpr int COLS = 256, NG = COLS / R;                 // columns and heads of a pass
  constexpr int A_BLOCK = 128 * 128;                       // one 64-element K-block of 128 key rows
  constexpr int A_STAGE = KB * A_BLOCK;
  constexpr int Q_BLOCK = COLS * 128, Q_PASS = KB * Q_BLOCK;
  constexpr int CHUNK = kTileChunk, CPT = 128 / CHUNK, CPW = 32 / CHUNK;   // chunks of a tile, of a warp's 32 rows
  constexpr int TAB_WORDS = NG * kTabStride;

  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ unsigned long long s_full[4], s_empty[4], s_accf[kSearchSets][2], s_acce[2];
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort, s_pmin, s_active, s_qmax[16];
  __shared__ float s_eps[32];   // by head: error radius per unit of key magnitude
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  unsigned char* sQ = smem;                                // [pass][KB][COLS rows][128 B], swizzled
  unsigned char* sA = sQ + cfg.passes * Q_PASS;            // [stage][KB][128 keys][128 B], swizzled
  uint32_t* tabs = reinterpret_cast<uint32_t*>(sA + cfg.stages * A_STAGE);   // [warp][NG][kTabStride]
  float* raws = reinterpret_cast<float*>(tabs + kSearchWarps * TAB_WORDS);   // check mode: the approximate products

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int Gq = p.H / p.HKV, BDST = cdiv(p.TQ, p.block_size_q);
  int64_t bid = blockIdx.x;
  const int part = (int)(bid % cfg.split); bid /= cfg.split;
  const int hg = (int)(bid % cfg.head_groups); bid /= cfg.head_groups;
  const int d = (int)(bid % BDST); bid /= BDST;
  const int hkv = (int)(bid % p.HKV); bid /= p.HKV;
  const int b = (int)bid;
  const int head0 = hkv * Gq + hg * cfg.passes * NG;
  const int heads = min(cfg.passes * NG, Gq - hg * cfg.passes * NG);
  const int passes = cdiv(heads, NG);
  const int t0 = d * p.block_size_q;
  const int Rv = min(R, (p.TQ - t0 + p.stride_q - 1) / p.stride_q);   // >= 1: a query block begins inside the queries
  const int n = p.n_chunks;
  const int64_t row = (int64_t)b * BDST + d;
  const int32_t* gl = p.left + row * n;
  const int32_t* gr = p.right + row * n;

  if (tid == 0) {
    for (int i = 0; i < 4; ++i) { mbar_init(smem_u32(&s_full[i]), 1); mbar_init(smem_u32(&s_empty[i]), passes); }
    for (int i = 0; i < 2 * kSearchSets; ++i) mbar_init(smem_u32(&s_accf[i >> 1][i & 1]), 1);
    for (int i = 0; i < 2; ++i) mbar_init(smem_u32(&s_acce[i]), 4);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    s_abort = 0;
    s_active = 0;
  }
  if (tid < 16) s_qmax[tid] = 0;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s_tmem)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  } else if (warp == 1) {
    const int m = block_min_position(p, b, t0, Rv, lane);
    if (lane == 0) s_pmin = m;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;
  const int pt = max(s_pmin - p.scan_window, 0);

  // ---- the pooled queries as the B operand; rows beyond the last pooled row repeat row 0, which leaves every maximum as it is ----
  {
    auto store = [&](int hh, int r, int pc, const float* v) {
      uint4 w;
      w.x = pack2<DT>(v[0], v[1]); w.y = pack2<DT>(v[2], v[3]); w.z = pack2<DT>(v[4], v[5]); w.w = pack2<DT>(v[6], v[7]);
      const int c = (hh % NG) * R + r;
      *reinterpret_cast<uint4*>(sQ + (hh / NG) * Q_PASS + (pc >> 3) * Q_BLOCK + sw128(c, pc & 7)) = w;
      float m = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) m = fmaxf(m, fabsf(v[e]));
      // the pieces of a warp belong to one head: 32 divides a head's R * PIECES pieces
      const int top = __reduce_max_sync(0xffffffffu, __float_as_int(m));   // (non-negative floats order as ints)
      if (lane == 0) atomicMax(&s_qmax[hh], top);
    };
    const int total = heads * R * PIECES;
    if (p.stride_q == 1 && p.rope_mode == HIPATTN_ROPE_NONE) {
      // one query row per pooled row: four loads of a thread in flight
      using T = typename Elem<DT>::type;
      const T* qb = reinterpret_cast<const T*>(p.q) + (int64_t)b * p.q_stride_b + (int64_t)t0 * p.q_stride_t;
      for (int i0 = warp * 32; i0 < total; i0 += 4 * kTileThreads) {
        uint4 raw[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int i = i0 + u * kTileThreads + lane, hh = i / (R * PIECES), r = i / PIECES % R, pc = i % PIECES;
          if (i < total) raw[u] = *reinterpret_cast<const uint4*>(qb + (int64_t)(head0 + hh) * p.q_stride_h + (int64_t)(r < Rv ? r : 0) * p.q_stride_t + pc * 8);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int i = i0 + u * kTileThreads + lane, hh = i / (R * PIECES), r = i / PIECES % R, pc = i % PIECES;
          if (i < total) {
            float v[8], sum[8];
            widen_piece<DT>(raw[u], v);
#pragma unroll
            for (int e = 0; e < 8; ++e) sum[e] = __fadd_rn(0.f, v[e]);
            mean_and_scale<DT>(sum, 1.f, p.q_scale, v);
            store(hh, r, pc, v);
          }
        }
      }
    } else {
      for (int i = tid; i < total; i += kTileThreads) {
        const int hh = i / (R * PIECES), r = i / PIECES % R, pc = i % PIECES;
        float v[8];
        pooled_query_piece<DT>(p, b, head0 + hh, t0 + (r < Rv ? r : 0) * p.stride_q, pc, v);
        store(hh, r, pc, v);
      }
    }
    // one past the last chunk that is active; per-head results are wanted for all of them
    int last = 0;
    if (p.left_out || p.right_out || p.score_out) last = n;
    else
      for (int i = tid; i < n; i += kTileThreads) {
        const int l = __ldg(gl + i);
        if (l < __ldg(gr + i) && l <= pt && l >= 0) last = i + 1;
      }
    last = __reduce_max_sync(0xffffffffu, last);
    if (lane == 0 && last > 0) atomicMax(&s_active, last);
    fence_async_smem();
  }
  __syncthreads();
  if (tid < 32) s_eps[tid] = tid < 16 ? kEps * __int_as_float(s_qmax[tid]) * 1.01f : 0.f;
  __syncthreads();
  const int tiles = cdiv(s_active, CPT);
  const int mine = part < tiles ? cdiv(tiles - part, cfg.split) : 0;   // tiles part, part + split, ...

  if (warp < kCopyWarps) {
    // ---- copies: the two warps take the tiles in turn, 8 lanes per row ----
    const char* kbase = reinterpret_cast<const char*>(p.k_scaled) + ((int64_t)b * p.HKV + hkv) * p.T * ROWB + (lane & 7) * 16;
    const uint32_t sA_u32 = smem_u32(sA) + ((lane >> 3) << 7);
    auto bound = [&](int it) {
      const int c = (part + it * cfg.split) * CPT + lane;
      return lane < CPT && it < mine && c < n ? __ldg(gl + c) : 0;
    };
    int next = bound(warp), slot = warp, use = 0, tail = -1;   // (at least two slots); tail: slot whose copies have not been reported
    bool ok = true;
    auto report = [&]() {
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&s_full[tail]));
      tail = -1;
    };
    for (int it = warp; it < mine; it += kCopyWarps) {
      // (a chunk near the end of the keys: the last CHUNK tokens, among them the one its candidates are clamped to)
      const int first = max(0, min(next, p.T - CHUNK));
      next = bound(it + kCopyWarps);
      if (use > 0 && !__all_sync(0xffffffffu, mbar_test(smem_u32(&s_empty[slot]), (use - 1) & 1))) {
        // no room yet: what is on its way is reported before the wait, not behind it
        if (tail >= 0) {
          cp_async_wait<0>();
          report();
        }
        ok = __all_sync(0xffffffffu, mbar_wait_quick<PATIENT>(smem_u32(&s_empty[slot]), (use - 1) & 1, &s_abort, p.status));
        if (!ok) break;
      }
      const uint32_t dst = sA_u32 + slot * A_STAGE;
#pragma unroll
      for (int r0 = 0; r0 < 128; r0 += 4) {
        const int j = r0 + (lane >> 3);
        const int tk = __shfl_sync(0xffffffffu, first, j / CHUNK) + j % CHUNK;
        const char* gp = kbase + (int64_t)tk * ROWB;
        const uint32_t sp = dst + r0 * 128 + (((lane & 7) ^ (j & 7)) << 4);
#pragma unroll
        for (int kb = 0; kb < KB; ++kb) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sp + kb * A_BLOCK), "l"(gp + kb * 128));
      }
      cp_async_commit();
      if (it < kCopyWarps) {   // the first tile is waited for at once: nothing else can begin
        cp_async_wait<0>();
        tail = slot;
        report();
      } else {
        if (tail >= 0) {
          cp_async_wait<1>();
          report();
        }
        tail = slot;
      }
      slot += kCopyWarps;
      while (slot >= cfg.stages) { slot -= cfg.stages; ++use; }
    }
    cp_async_wait<0>();
    if (ok && tail >= 0) report();
  } else if (warp < kFirstSearchWarp) {
    // ---- MMAs: two threads take the accumulators in turn, so that one waits for its operands while the other's MMAs run ----
    const int acc = warp - kCopyWarps;
    if (lane == 0) {
      const uint64_t da0 = make_desc(smem_u32(sA), 16, 1024), db0 = make_desc(smem_u32(sQ), 16, 1024);
      int it = 0, j = 0, slot = 0, use = 0, set = acc;
      auto advance = [&]() {
        if (++j == passes) {
          j = 0;
          ++it;
          if (++slot == cfg.stages) { slot = 0; ++use; }
        }
      };
      if (acc) advance();
      int k = 0, last = 0;
      for (; it < mine; ++k) {
        if (!mbar_wait_quick<PATIENT>(smem_u32(&s_full[slot]), use & 1, &s_abort, p.status)) break;
        if (k > 0 && !mbar_wait_quick<PATIENT>(smem_u32(&s_acce[acc]), (k - 1) & 1, &s_abort, p.status)) break;
        tc_fence_after();
        const uint32_t idesc = make_idesc(DT == HIPATTN_BF16 ? 1 : 0, 128, min(NG, heads - j * NG) * R, 0);
        const uint64_t da = da0 + (uint64_t)((slot * A_STAGE) >> 4), db = db0 + (uint64_t)((j * Q_PASS) >> 4);
#pragma unroll
        for (int q = 0; q < D / 16; ++q)
          umma(tmem + acc * COLS, da + (uint64_t)(((q >> 2) * A_BLOCK + (q & 3) * 32) >> 4),
               db + (uint64_t)(((q >> 2) * Q_BLOCK + (q & 3) * 32) >> 4), idesc, q > 0 ? 1u : 0u);
        umma_commit(smem_u32(&s_empty[slot]));
        umma_commit(smem_u32(&s_accf[set][acc]));   // (last: waited for before the role ends)
        last = set;
        set += 2;
        if (set >= kSearchSets) set -= kSearchSets;
        advance();
        advance();
      }
      // (every third accumulator of a thread is a set's)
      if (k > 0) mbar_drain(smem_u32(&s_accf[last][acc]), ((k - 1) / kSearchSets) & 1);
    }
    __syncwarp();
  } else if (warp >= kFirstSearchWarp) {
    // ---- searches: the sets take the accumulators in turn; a warp reads its quarter of the TMEM lanes ----
    const int set = (warp - kFirstSearchWarp) >> 2, quarter = warp & 3;
    uint32_t* tab = tabs + (warp - kFirstSearchWarp) * TAB_WORDS;
    float* rawx = raws + (warp - kFirstSearchWarp) * NG * 32;
    const uint32_t my_tmem = tmem + ((uint32_t)(quarter * 32) << 16);
    const uint32_t sQ_u32 = smem_u32(sQ);
    const char* kbase = reinterpret_cast<const char*>(p.k_scaled) + ((int64_t)b * p.HKV + hkv) * p.T * ROWB;
    const float* abs_base = p.key_abs + ((int64_t)b * p.HKV + hkv) * p.T;
    int32_t* score_row = p.score_max + row * n;
    const bool per_head = p.left_out || p.right_out || p.score_out, counting = p.access_counter != nullptr;
    unsigned st_keys = 0, st_fb = 0, st_wrong = 0;
    float st_ratio = 0.f;
    bool ok = true;
    // (tile, pass) of an accumulator
    struct Cursor {
      int it, j, passes;
      __device__ __forceinline__ void skip(int k) {
        j += k;
        while (j >= passes) { j -= passes; ++it; }
      }
    };
    // What a round needs from memory is requested ahead: the bounds of a lane's chunk two rounds, the magnitude of its key one.
    // With them comes the chunk's score so far: others may raise it meanwhile, nobody lowers it.
    struct Bounds {
      int l, r, known;
    };
    auto bounds_of = [&](const Cursor& k) {
      Bounds x{0, 0, 0};
      const int c = (part + k.it * cfg.split) * CPT + quarter * CPW + lane / CHUNK;
      if (k.it < mine && c < n) { x.l = __ldg(gl + c); x.r = __ldg(gr + c); x.known = __ldcg(score_row + c); }
      return x;
    };
    auto token_of = [&](const Bounds& x) { return max(0, min(x.l, p.T - CHUNK)) + lane % CHUNK; };
    auto magnitude = [&](const Bounds& x) { return x.l < x.r && x.l <= pt && x.l >= 0 ? __ldg(abs_base + token_of(x)) : 0.f; };
    Cursor cur{0, 0, passes}, ahead{0, 0, passes};
    cur.skip(set);
    ahead.skip(set);
    Bounds b1 = bounds_of(ahead), b2;
    ahead.skip(kSearchSets);
    b2 = bounds_of(ahead);
    float abs1 = magnitude(b1);
    auto slot_of = [&](const Bounds& x) {
      return counting && x.l < x.r && x.l <= pt && x.l >= 0 ? access_index(p.k, b, token_of(x)) : (int64_t)-1;
    };
    int64_t slot1 = slot_of(b1);
    int32_t* counter = p.access_counter + (int64_t)b * p.access_stride_b + (int64_t)hkv * p.access_stride_h;
    // (a barrier per set and accumulator: its phases come from one thread and are all waited for by one set, in order)
    uint32_t phase = 0;
    for (int u = set; cur.it < mine && ok; cur.skip(kSearchSets), u += kSearchSets) {
      const int acc = u & 1;
      const int it = cur.it, j = cur.j, ng = min(NG, heads - j * NG);
      const int c0 = (part + it * cfg.split) * CPT + quarter * CPW, cl = c0 + lane / CHUNK;    // the warp's first chunk, the lane's
      const int l = b1.l, r = b1.r, known = b1.known, token = token_of(b1), first = token - lane % CHUNK;
      const bool act = l < r && l <= pt && l >= 0;
      const float s_abs = abs1;
      const int64_t mark = slot1;
      b1 = b2;
      abs1 = magnitude(b1);
      slot1 = slot_of(b1);
      ahead.skip(kSearchSets);
      b2 = bounds_of(ahead);
      float eps[NG];   // radius per unit of key magnitude
#pragma unroll
      for (int g = 0; g < NG; ++g) eps[g] = s_eps[j * NG + g];
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
#pragma unroll
      for (int g = 0; g < NG; ++g)
        if (g < ng) {
          const float e_ = eps[g] * s_abs;
          const uint32_t w = pack2<DT>(x[g] - e_, x[g] + e_);
          tab[g * kTabStride + lane] = w;
          if (p.stats && act) {
            ++st_keys;
            if (lo_f32<DT>(w) != hi_f32<DT>(w)) ++st_fb;
          }
          if (cfg.check) rawx[g * 32 + lane] = x[g];
        }
      __syncwarp();
      // strict score of a token for head g of this pass: one pooled row per lane, the key's pieces the same in every lane
      auto strict_of = [&](int tk, int g) -> float {
        // (While MMAs run they take most of the shared memory's bandwidth and a load from it takes hundreds of cycles: the pieces
        // are read four at a time.  One by one a score took 7600 cycles.)
        const uint4* kp = reinterpret_cast<const uint4*>(kbase + tk * (int64_t)ROWB);
        constexpr int RL = R > 32 ? R / 32 : 1;   // rows, and independent chains, of a lane
        constexpr int BATCH = RL > 2 ? 2 : 4;
        float a[RL];
#pragma unroll
        for (int i = 0; i < RL; ++i) a[i] = 0.f;
#pragma unroll 1
        for (int p0 = 0; p0 < PIECES; p0 += BATCH) {
          uint4 kw[BATCH], qw[BATCH][RL];
#pragma unroll
          for (int e = 0; e < BATCH; ++e) {
            kw[e] = __ldg(kp + p0 + e);
#pragma unroll
            for (int i = 0; i < RL; ++i)
              qw[e][i] = lds128(sQ_u32 + j * Q_PASS + ((p0 + e) >> 3) * Q_BLOCK + sw128(g * R + (R < 32 ? (lane & (R - 1)) : i * 32 + lane), (p0 + e) & 7));
          }
#pragma unroll
          for (int e = 0; e < BATCH; ++e)
#pragma unroll
            for (int i = 0; i < RL; ++i) a[i] = strict_piece<DT>(qw[e][i], kw[e], a[i]);
        }
        float best = -INFINITY;
#pragma unroll
        for (int i = 0; i < RL; ++i) best = fmaxf(best, a[i]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, o));
        return best;
      };
      if (cfg.check) {   // every score by both definitions
        for (int g = 0; g < ng; ++g) {
          for (unsigned m = __ballot_sync(0xffffffffu, act); m; m &= m - 1) {
            const int o = __ffs(m) - 1;
            const float raw = strict_of(__shfl_sync(0xffffffffu, token, o), g);
            if (lane == o) {
              uint32_t* w = tab + g * kTabStride + lane;
              const float e_ = s_eps[j * NG + g] * s_abs, ex = Elem<DT>::round(raw);
              if (lo_f32<DT>(*w) == hi_f32<DT>(*w) && hi_f32<DT>(*w) != ex) ++st_wrong;
              if (e_ > 0.f) st_ratio = fmaxf(st_ratio, fabsf(rawx[g * 32 + lane] - raw) / e_);
              *w = pack2<DT>(ex, ex);
            }
          }
        }
        __syncwarp();
      }
      uint32_t seen = 0;
      // (at most 32 tasks: their bounds and results stay in registers between the two forms of the search)
      constexpr bool ONE = CPW * NG <= 32;
      float slo = HIPATTN_SCORE_INIT, shi = HIPATTN_SCORE_INIT;
      uint32_t asked = 0;
      bool compared = false;   // every comparison is settled, some scores are not
      bool settled = !per_head && __all_sync(0xffffffffu, cl >= n || (l >= 0 && r - l == CHUNK && l + CHUNK - 1 <= pt && l + CHUNK <= p.T));
      if (settled) {
        for (int w0 = 0; w0 < CPW * NG; w0 += 32) {
          const int g = (w0 + lane) % NG, cw = (w0 + lane) / NG, cc = cw < CPW ? cw : 0;
          const bool valid = cw < CPW && g < ng && c0 + cc < n;
          const int code = __shfl_sync(0xffffffffu, known, cc * CHUNK);
          const float so_far = decode_score(code);
          int off = cc * CHUNK;
          asked = 0;
          bool closed = search_whole<DT, CHUNK>(tab + g * kTabStride, off, slo, shi, asked);
          if (!valid) slo = shi = HIPATTN_SCORE_INIT;
          else seen |= asked;
          float best = fmaxf(slo, so_far);
#pragma unroll
          for (int o = 1; o < NG; o <<= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, o));
          // a score that may raise the chunk's best has to be certain
          closed |= !valid;
          if (!__all_sync(0xffffffffu, closed && !(shi > slo && shi > best))) {
            compared = ONE && __all_sync(0xffffffffu, closed);
            settled = false;
            break;
          }
          if (valid && g == 0 && best > so_far) atomicMax(score_row + c0 + cc, encode_score(best));
        }
      }
      if (!settled) {
        seen = compared ? seen : 0;
        for (int w0 = 0; w0 < CPW * NG; w0 += 32) {
          const int g = (w0 + lane) % NG, cw = (w0 + lane) / NG, cc = cw < CPW ? cw : 0;
          ChunkTask t;
          t.l = __shfl_sync(0xffffffffu, l, cc * CHUNK);
          t.r = __shfl_sync(0xffffffffu, r, cc * CHUNK);
          t.first = __shfl_sync(0xffffffffu, first, cc * CHUNK);
          t.row0 = cc * CHUNK;
          t.known = decode_score(__shfl_sync(0xffffffffu, known, cc * CHUNK));
          t.valid = cw < CPW && g < ng && c0 + cc < n;
          t.pt = pt;
          t.tab = tab + g * kTabStride;
          t.slo = compared ? slo : HIPATTN_SCORE_INIT;
          t.shi = compared ? shi : HIPATTN_SCORE_INIT;
          search_chunks<DT, CHUNK>(t, p.T, NG, compared, p.score_out != nullptr,
              [&](int tk, int owner) { return strict_of(tk, (w0 + owner) % NG); },
              [&](int tk) { if (counting) mark_access(p.access_counter, p.access_stride_b, p.access_stride_h, p.access_n, p.k, b, hkv, tk); });
          const int h = head0 + j * NG + g, c = c0 + cc;
          if (t.valid) {
            const int64_t o = (row * p.H + h) * n + c;
            if (p.left_out) p.left_out[o] = t.l;
            if (p.right_out) p.right_out[o] = t.r;
            if (p.score_out) p.score_out[o] = t.score;
            if (t.out_of_range) atomicOr(p.status, HIPATTN_STATUS_TOKEN_RANGE);
            seen |= t.seen;
          }
          float best = t.score;
#pragma unroll
          for (int o = 1; o < NG; o <<= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, o));
          if (t.valid && g == 0 && best > t.known) atomicMax(score_row + c, encode_score(best));
        }
      }
      if (counting) {
        seen = __reduce_or_sync(0xffffffffu, seen);
        if ((seen >> lane & 1) && mark >= 0 && mark < p.access_n) counter[mark] = 1;
      }
      __syncwarp();   // the table is written anew
    }
    if (p.stats) add_stats(p.stats, st_keys, st_fb, st_wrong, st_ratio);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// Heads of a KV head that a CTA takes: all of them as long as two key tiles fit beside their pooled queries, so that the keys
// are fetched once.
struct TilePlan {
  int passes, head_groups;
  size_t fixed, stage;   // bytes of shared memory without key tiles, of a key tile
};
TilePlan plan_tiles(const hipattn_scan_params_t& p) {
  const int R = p.block_size_q / p.stride_q, NG = 256 / R, Gq = p.H / p.HKV;
  const size_t q_pass = (size_t)256 * p.D * 2, tab = (size_t)kSearchWarps * NG * (kTabStride * 4 + (p.mode == HIPATTN_SCAN_CHECK ? 128 : 0));
  TilePlan t;
  t.stage = (size_t)128 * p.D * 2;
  t.passes = min(cdiv(Gq, NG), 16 / NG);
  while (t.passes > 1 && kTileSlack + t.passes * q_pass + 2 * t.stage + tab > kTileSmem) --t.passes;
  t.head_groups = cdiv(Gq, t.passes * NG);
  t.fixed = kTileSlack + t.passes * q_pass + tab;
  return t;
}

template <int DT, int D, int R>
int launch(const hipattn_scan_params_t& p, cudaStream_t stream) {
  const TilePlan plan = plan_tiles(p);
  QueryTiles cfg;
  cfg.check = p.mode == HIPATTN_SCAN_CHECK ? 1 : 0;
  cfg.passes = plan.passes;
  cfg.head_groups = plan.head_groups;
  // (an even number of slots: with one pass a tile, a slot's phases are then all waited for by one of the two MMA threads)
  cfg.stages = plan.fixed + 4 * plan.stage <= kTileSmem ? 4 : 2;
  const size_t smem = plan.fixed + cfg.stages * plan.stage;
  const int64_t units = (int64_t)p.B * p.HKV * cdiv(p.TQ, p.block_size_q) * cfg.head_groups;
  cfg.split = scan_ctas_per_unit(units * 8, cdiv(p.n_chunks, 128 / kTileChunk));   // (one CTA a multiprocessor, a wave of them)
  const int64_t grid = units * cfg.split;
  HIPATTN_REQUIRE(grid > 0 && grid < 0x7fffffffLL, HIPATTN_ERR_INVALID, "scan grid of %lld blocks", (long long)grid);
  auto kern = scan_query_tiles_kernel<DT, D, R, true>;
  if constexpr (DT == HIPATTN_BF16 && D == 128 && R == 64)
    if (without_patience()) kern = scan_query_tiles_kernel<DT, D, R, false>;
  HIPATTN_CUDA_OK(allow_smem((const void*)kern, smem));
  kern<<<(unsigned)grid, kTileThreads, smem, stream>>>(p, cfg);
  return check_launch("scan_query_tiles_kernel");
}

template <int DT, int D>
int dispatch_rows(const hipattn_scan_params_t& p, cudaStream_t stream) {
  switch (p.block_size_q / p.stride_q) {
    case 16: return launch<DT, D, 16>(p, stream);
    case 32: return launch<DT, D, 32>(p, stream);
    case 64: return launch<DT, D, 64>(p, stream);
    default: return launch<DT, D, 128>(p, stream);
  }
}

}  // namespace

// Called for what the tcgen05 scan takes (prepared keys, 16-bit prefill, head dim 64 / 128).  Chunks of 8 without in-kernel RoPE, 16
// to 128 pooled rows a head, where the heads of a KV head fill half of an accumulator's columns or more: times against the rounds,
// by heads x rows, 4096 queries of 65536 tokens: 4 x 64 0.69, 4 x 32 0.74, 4 x 128 0.83, 8 x 16 0.70, 8 x 128 0.84, 2 x 128 0.80,
// but 4 x 16 1.11, 2 x 64 0.93 (head dim 64: 1.05), 1 x 128 1.05.  Chunks of 16 would take 0.78 (8 x 32) to 1.25 of the rounds'
// time, of 32 1.14 to 1.8; "relative", whose every key has two scores, 0.78 (8 x 32) to 1.2.  With fewer than 32 units the
// rounds, whose CTAs are smaller, spread better: 16 units 1.09 to 1.16, 32 units 0.89 to 0.98.
//
// A CTA puts 64 to 128 KB of pooled queries in place before its first tile, so its list has to be worth that: three steps (a key
// tile against 256 columns), seven per 64 query rows where a pooled row is the mean of several, and ten steps per multiprocessor in
// all.  On 1330 random calls (2 to 16 heads a KV head, 1 to 16 KV heads, 200 to 16384 queries of 1400 to 100000 tokens, 32 to 1024
// chunks) the stage took 414 ms by rounds, 306.0 by the better of the two, 307.5 by this rule, with 52 calls slower than by rounds by
// more than 3 %, 1.32 times at most; with the units alone 310.7, 337 calls and 2.4 times at most (8 x 32 rows, 64 chunks, 48 units:
// 15 us by rounds, 35 here).
int scan_query_tiles(const hipattn_scan_params_t& p, cudaStream_t stream, bool* handled) {
  *handled = false;
  const int R = p.block_size_q / p.stride_q, G = p.H / p.HKV;
  if (p.rope_mode != HIPATTN_ROPE_NONE || (R != 16 && R != 32 && R != 64 && R != 128)) return HIPATTN_OK;
  if (p.chunk_size != kTileChunk || p.T < kTileChunk || G < 2 || G * R < 128) return HIPATTN_OK;
  const ScanChoice choice = scan_choice();
  if (choice == SCAN_BY_ROUNDS) return HIPATTN_OK;
  if (choice != SCAN_BY_TILES) {
    if (G < 4 && G * R < 192) return HIPATTN_OK;
    const int64_t blocks = (int64_t)p.B * p.HKV * cdiv(p.TQ, p.block_size_q), ctas = plan_tiles(p).head_groups;
    const int64_t steps = (int64_t)cdiv(p.n_chunks, 128 / kTileChunk) * cdiv(G, 256 / R);   // of a query block and KV head
    if (blocks * ctas < 32 || blocks * steps < 10 * 148) return HIPATTN_OK;
    if (p.stride_q == 1 ? steps < ctas * 3 : steps * 64 < ctas * 7 * p.block_size_q) return HIPATTN_OK;
  }
  *handled = true;
  if (p.dtype == HIPATTN_BF16) return p.D == 128 ? dispatch_rows<HIPATTN_BF16, 128>(p, stream) : dispatch_rows<HIPATTN_BF16, 64>(p, stream);
  return p.D == 128 ? dispatch_rows<HIPATTN_F16, 128>(p, stream) : dispatch_rows<HIPATTN_F16, 64>(p, stream);
}

}  // namespace hipattn
