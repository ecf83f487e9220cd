// Search of whole chunks on score bounds: the part that the tensor-core scans which score every token of a chunk share
// (scan_query_tiles.cu, scan_key_tiles.cu).
//
// A warp holds the scores of 32 consecutive rows of a key tile (TMEM lanes) against some groups of pooled queries (a group = the
// pooled rows of one head and query block), as bounds lo <= rounded score <= hi packed in one word per (group, row) in
// shared memory.  One lane per (chunk, group) replays the halving search of the reference (attention_extend.py:413-1249) on
// the bounds; where they leave a comparison open, or the chunk's best score uncertain, the lane asks for the strict score of
// one key and the whole warp computes it, so that bounds and scores are those of the strict kernel.
#pragma once
#include <cstdlib>
#include <cstring>

#include "scan_common.cuh"
#include "tcgen05_common.cuh"

namespace hipattn {

constexpr int kTabStride = 33;   // words of a group: 32 rows, the odd stride spreads the banks

// largest of three
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;\n" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// At the end of a role: waits, with a limit of its own, for what the role issued last, so that a CTA leaves nothing in flight however
// its other roles ended (a role that has issued all it had may be gone before another one's wait runs out).
static __device__ __noinline__ void mbar_drain(uint32_t mbar, uint32_t parity) {
  const long long t0 = clock64();
  uint32_t done = 0;
  while (!done && clock64() - t0 < kWaitCycles)
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
                 : "=r"(done) : "r"(mbar), "r"(parity) : "memory");
}

// Row maxima of a thread's accumulator columns: NG groups of R columns from column `taddr`, 64 columns per TMEM load.  Groups at
// `ng` and beyond are skipped in steps of whole loads.
template <int R, int NG>
__device__ __forceinline__ void group_maxima(uint32_t taddr, int ng, float* x) {
  constexpr int PER = R >= 64 ? 1 : 64 / R;        // groups per load
  constexpr int LOADS = R > 64 ? R / 64 : 1;       // loads per group
  constexpr int COLS = R > 64 ? 64 : R;
#pragma unroll
  for (int g0 = 0; g0 < NG; g0 += PER) {
    if (g0 >= ng) break;
#pragma unroll
    for (int l = 0; l < LOADS; ++l) {
      float v[64];
      tmem_ld64(taddr + g0 * R + l * 64, v);
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const float* w = v + i * COLS;
        float m[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) m[k] = fmaxf(w[2 * k], w[2 * k + 1]);
#pragma unroll
        for (int k = 8; k < COLS; k += 8)
#pragma unroll
          for (int e = 0; e < 4; ++e) m[e] = max3(m[e], w[k + 2 * e], w[k + 2 * e + 1]);
        const float y = fmaxf(max3(m[0], m[1], m[2]), m[3]);
        x[g0 + i] = l == 0 ? y : fmaxf(x[g0 + i], y);
      }
    }
  }
}

// The strict definition's sum over the eight elements of a piece: fused multiply-adds in ascending order.
template <int DT>
__device__ __forceinline__ float strict_piece(const uint4& q, const uint4& k, float a) {
  a = fmaf(lo_f32<DT>(q.x), lo_f32<DT>(k.x), a);
  a = fmaf(hi_f32<DT>(q.x), hi_f32<DT>(k.x), a);
  a = fmaf(lo_f32<DT>(q.y), lo_f32<DT>(k.y), a);
  a = fmaf(hi_f32<DT>(q.y), hi_f32<DT>(k.y), a);
  a = fmaf(lo_f32<DT>(q.z), lo_f32<DT>(k.z), a);
  a = fmaf(hi_f32<DT>(q.z), hi_f32<DT>(k.z), a);
  a = fmaf(lo_f32<DT>(q.w), lo_f32<DT>(k.w), a);
  return fmaf(hi_f32<DT>(q.w), hi_f32<DT>(k.w), a);
}

// Adds what a thread counted to the statistics words.
__device__ __forceinline__ void add_stats(uint64_t* stats, unsigned keys, unsigned fallback, unsigned wrong, float ratio) {
  unsigned long long* st = reinterpret_cast<unsigned long long*>(stats);
  if (keys) atomicAdd(st + ST_KEYS, (unsigned long long)keys);
  if (fallback) atomicAdd(st + ST_FALLBACK, (unsigned long long)fallback);
  if (wrong) atomicAdd(st + ST_WRONG, (unsigned long long)wrong);
  atomicMax(reinterpret_cast<unsigned int*>(st + ST_RATIO_BITS), __float_as_uint(ratio));
}

// An mbarrier's phase: tried a few times, and waited for out of line.  The roles of these kernels go through long straight code, each
// warp its own, so that instructions come from beyond the first-level caches and cost five to six cycles apiece: the way through a
// barrier that is ready is kept short.
__device__ __forceinline__ bool mbar_try(uint32_t mbar, uint32_t parity) {
  uint32_t done;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
               : "=r"(done) : "r"(mbar), "r"(parity) : "memory");
  return done != 0;
}
// (without waiting: try_wait suspends the thread for a while)
__device__ __forceinline__ bool mbar_test(uint32_t mbar, uint32_t parity) {
  uint32_t done;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
               : "=r"(done) : "r"(mbar), "r"(parity) : "memory");
  return done != 0;
}
// PATIENT: as always.  Otherwise a barrier that is not ready counts as a wait that ran out.
template <bool PATIENT>
static __device__ __noinline__ bool mbar_wait_slow(uint32_t mbar, uint32_t parity, volatile int* abort_flag, uint32_t* status) {
  if (PATIENT) return mbar_wait(mbar, parity, abort_flag, status);
  if (mbar_test(mbar, parity)) return true;
  *abort_flag = 1;
  atomicOr(status, HIPATTN_STATUS_TIMEOUT);
  return false;
}
template <bool PATIENT>
__device__ __forceinline__ bool mbar_wait_quick(uint32_t mbar, uint32_t parity, volatile int* abort_flag, uint32_t* status) {
  if (PATIENT) {
#pragma unroll 1
    for (int i = 0; i < 64; ++i)
      if (mbar_try(mbar, parity)) return true;
  }
  return mbar_wait_slow<PATIENT>(mbar, parity, abort_flag, status);
}
// HIPATTN_SCAN_KERNEL, for comparisons: the prefill scans on mma.sync, by rounds, or on whole tiles wherever these can be had, whether
// they are the faster ones or not.
enum ScanChoice { SCAN_BY_RULE, SCAN_BY_MMA, SCAN_BY_ROUNDS, SCAN_BY_TILES };
inline ScanChoice scan_choice() {
  const char* v = getenv("HIPATTN_SCAN_KERNEL");
  if (!v) return SCAN_BY_RULE;
  return strcmp(v, "mma") == 0 ? SCAN_BY_MMA : strcmp(v, "rounds") == 0 ? SCAN_BY_ROUNDS : strcmp(v, "tiles") == 0 ? SCAN_BY_TILES : SCAN_BY_RULE;
}
// HIPATTN_SCAN_WAIT=none: the instantiation without patience, with which a test takes a kernel's ways out of a wait that has run
// out.  (bf16, head dim 128 and four heads of 64 rows only.  An instantiation and not an argument: how often to try, read from
// the launch's parameters at every wait, cost the query tiles 1.7 %.)
inline bool without_patience() {
  const char* v = getenv("HIPATTN_SCAN_WAIT");
  return v && strcmp(v, "none") == 0;
}

// The search of a lane's chunk where every chunk of the warp is whole and active to its last token, as all of a step's chunks but
// the last few are: rounds without conditions.  Returns false where a comparison is open; slo / shi: bounds of the best
// winner.  off: the first row on entry, the row that is left on return.
template <int DT, int CHUNK>
__device__ __forceinline__ bool search_whole(const uint32_t* tab, int& off, float& slo, float& shi, uint32_t& seen) {
  bool open = false;
  slo = shi = HIPATTN_SCORE_INIT;
#pragma unroll
  for (int s = CHUNK; s >= 2; s >>= 1) {
    const int il = off + s / 4, ir = off + s / 2 + s / 4;
    seen |= 1u << il | 1u << ir;
    const uint32_t bl = tab[il], br = tab[ir];
    const float llo = lo_f32<DT>(bl), lhi = hi_f32<DT>(bl), rlo = lo_f32<DT>(br), rhi = hi_f32<DT>(br);
    const bool win = llo > rhi;
    open |= !win && !(lhi <= rlo);
    const float whi = win ? lhi : rhi;
    slo = fmaxf(slo, win ? llo : rlo);
    shi = fmaxf(shi, whi == whi ? whi : INFINITY);   // (bounds that are not numbers bound nothing)
    if (!win) off += s / 2;
  }
  return !open;
}

// A lane's search of one chunk for one group; the lanes of one chunk and query block are `width` neighbours (a power of two).
struct ChunkTask {
  bool valid;            // the lane has a task
  int l, r;              // the chunk's bounds; the search narrows them
  int pt;                // chunks that begin beyond pt are not active
  int first;             // token of the chunk's first row in the table
  int row0;              // that row
  float known;           // a score that the chunk has for certain (of any head)
  uint32_t* tab;         // bounds of this group
  float score;           // result: the chunk's score
  float slo, shi;        // bounds of the best winner, where the comparisons are settled already
  uint32_t seen;         // result: rows that the rounds ask for
  bool out_of_range;     // result: a round asked for a token beyond the keys
};

// Runs the searches of a warp, whatever its chunks are like.  strict(token, owner) is called by the whole warp with uniform
// arguments and returns the strict score, before rounding, of a token for the group of lane `owner`; mark(token) records a token
// outside the table's rows (of a chunk longer than CHUNK, which only a caller's own list can hold).
//
// The winners' scores enter only through their maximum over the heads, so a score that is not certain is made so only where its
// upper bound exceeds every certain one of its chunk, those of other CTAs' heads included (`every`: a chunk's score is wanted
// for each head).  A strict score costs a warp more than the whole search, and the slowest of the four warps of an accumulator
// sets the pace.
template <int DT, int CHUNK, typename Strict, typename Mark>
__device__ __forceinline__ void search_chunks(ChunkTask& t, int T, int width, bool settled, bool every, Strict strict, Mark mark) {
  const int lane = threadIdx.x & 31;
  const int l0 = t.l, r0 = t.r;
  float slo = t.slo, shi = t.shi;
  t.seen = 0;
  t.out_of_range = false;
  // Two walks: the first settles the comparisons (`settled`: they are), the second the scores of the lanes that may raise their
  // chunk's best.
#pragma unroll 1
  for (int pass = settled ? 1 : 0; pass < 2; ++pass) {
    bool live = t.valid;
    float floor = 0.f;
    if (pass == 1) {
      floor = slo;
      if (!every) {
        floor = fmaxf(floor, t.known);
        for (int o = 1; o < width; o <<= 1) floor = fmaxf(floor, __shfl_xor_sync(0xffffffffu, floor, o));
      }
      live = t.valid && shi > slo && shi > floor;
      if (!__any_sync(0xffffffffu, live)) break;
    }
    const bool mine = live;
    const bool big = r0 - l0 > CHUNK;
    int wl = l0, wr = r0, tl = 0, tr = 0;
    bool loaded = false, first = true;
    float llo = 0.f, lhi = 0.f, rlo = 0.f, rhi = 0.f, nlo = HIPATTN_SCORE_INIT, nhi = HIPATTN_SCORE_INIT;
    for (;;) {
      int need = -1;   // side of the key whose strict score is wanted
      while (live) {
        const int mid = (wl + wr) >> 1;
        if (!loaded) {
          if (!(wl < wr && wl <= t.pt && wl >= 0 && (first || wr - wl > 1))) {
            live = false;
            break;
          }
          first = false;
          tl = (wl + mid) >> 1;
          tr = (mid + wr) >> 1;
          t.out_of_range |= tr >= T;
          if (big) {
            llo = rlo = -INFINITY;
            lhi = rhi = INFINITY;
            mark(min(tl, T - 1));
            mark(min(tr, T - 1));
          } else {
            // (tokens beyond the keys are the last one, whose row a chunk that begins beyond them holds throughout)
            const int il = t.row0 + max(0, min(tl, T - 1) - t.first), ir = t.row0 + max(0, min(tr, T - 1) - t.first);
            t.seen |= 1u << il | 1u << ir;
            const uint32_t bl = t.tab[il], br = t.tab[ir];
            llo = lo_f32<DT>(bl); lhi = hi_f32<DT>(bl);
            rlo = lo_f32<DT>(br); rhi = hi_f32<DT>(br);
          }
          loaded = true;
        }
        const bool same = tl == tr;   // a key does not beat itself
        const bool win = llo > rhi && !same;
        const float wlo = win ? llo : rlo, whi = win ? lhi : rhi;
        if (!win && !(lhi <= rlo) && !same) {   // open: the left key's score first, where it is not certain
          need = llo == lhi ? 1 : 0;
          break;
        }
        if (pass == 1 && wlo != whi && !(whi <= fmaxf(nlo, floor))) {
          need = win ? 0 : 1;
          break;
        }
        if (win) wr = mid; else wl = mid;
        nlo = fmaxf(nlo, wlo);
        nhi = fmaxf(nhi, whi == whi ? whi : INFINITY);
        loaded = false;
      }
      unsigned todo = __ballot_sync(0xffffffffu, need >= 0);
      if (!todo) break;
      while (todo) {
        const int owner = __ffs(todo) - 1;
        todo &= todo - 1;
        const int side = __shfl_sync(0xffffffffu, need, owner);
        const int tk = min(__shfl_sync(0xffffffffu, need == 0 ? tl : tr, owner), T - 1);
        const float raw = strict(tk, owner);
        if (lane == owner) {
          const float ex = Elem<DT>::round(raw);
          if (side == 0) llo = lhi = ex; else rlo = rhi = ex;
          if (!big) t.tab[t.row0 + max(0, tk - t.first)] = pack2<DT>(ex, ex);
        }
      }
    }
    if (mine) {
      slo = nlo;
      shi = nhi;
      t.l = wl;
      t.r = wr;
    }
  }
  t.score = slo;
}

}  // namespace hipattn
