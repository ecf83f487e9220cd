// Scan stage of the mask estimator for decode (one pooled query row per head), small chunks, 16-bit types: every token
// of every active chunk is fetched ONCE for up to eight query heads of a KV head, scored on the tensor cores, and the
// halving search of the reference (attention_extend.py:413-1249) is replayed on the scores.
//
// As in scan_chunks_strict.cu the whole chunk is cheaper to fetch than the rows the heads' rounds would ask for.  That
// kernel spends its time on the dot products, though: 32 fused multiply-adds and twelve shared-memory wavefronts per
// 16-byte piece of a row, 3.6 TB/s of rows.  Here the products of a pass (64 rows x 8 heads) are 32 mma.sync, and, as in the
// prefill scans, a score is used only where it is certain: the rounded score of a key equals the strict one when x - e and
// x + e round alike, e = kEps * max|q'| * sum_d |k'_d|.  The search works on the bounds round(x - e), round(x + e): the
// scores that are not certain (2 % of them in bf16, 12 % in fp16) seldom decide anything.  Where they do, the pass's uncertain
// scores are listed and one lane each scores them by the strict definition (sequential fp32 FMA over the head dimension),
// up to 32 at a time.  Bounds and scores are those of the strict kernel.  (Every uncertain score by the strict
// definition: 0.56 ms on the case below.)
//
// In-kernel RoPE: "streaming" rotates a row to its chunk's index, "relative" scores every row twice, rotated to table
// position 0 for the left and 1 for the right candidate.  Rotation and key scale run on the packed operand registers (a
// row's elements d and d + D / 2 sit in the same lane).  fp8 rows are widened in registers.
//
// Mapping: a warp takes 64 consecutive rows = 64 / chunk whole chunks per pass, sixteen rows at a time; the rows are the A
// operand, the heads' queries the B operand.  A row goes straight from global memory to operand registers: the order of a
// contraction is free, so lane j of a row's four lanes takes the sixteen-byte pieces 4 i + j and the queries' fragments are
// laid out alike.  Nothing is staged, so registers alone bound the resident warps, and the next sixteen rows are in
// flight while these are multiplied.  (Staged through shared memory, 24 warps of 32 rows or 12 of 64: 0.66 ms on the case
// below; the 192 KB of staging bound the warps, and one warp's search and strict scores left its share of them idle.)
//
// Bound: HBM (random 256-byte rows).  32 sequences of 131072 tokens, chunk 32 / 8, bf16: 0.59 / 0.16 ms with the strict
// kernel, 0.45 / 0.12 ms here (4.8 / 4.4 TB/s); "relative", 12 sequences of 20-40 thousand tokens: 0.55 / 0.35 ms by rounds, 0.33 / 0.11 here.
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "mma_common.cuh"
#include "scan_common.cuh"

namespace hipattn {

int strict_chunk_heads(const hipattn_scan_params_t& p);

namespace {

constexpr int kPass = 64;        // rows of a warp's pass
constexpr int kTabStride = 65;   // floats per head of the score table (64 rows; the odd stride spreads the banks)
constexpr int kQPad = 4;         // floats behind each query row: heads start in different banks

__device__ __align__(256) unsigned char g_zero_key[256];   // the row of a token that is not scored

__device__ __forceinline__ uint4 load_row16(const char* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint2 load_row8(const char* p) {
  uint2 v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];\n" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}

// MODE: HIPATTN_ROPE_NONE / _RELATIVE / _STREAMING; F8: e5m2 rows
template <int DT, int D, int MODE, bool F8>
__global__ void __launch_bounds__(128, MODE == HIPATTN_ROPE_NONE || F8 ? 4 : 3)
    scan_chunks_mma_kernel(const hipattn_scan_params_t p, int c_log2, int HB, int n_split, int passes_total, int check, int nan_loses) {
  constexpr int PIECES = D / 8, QS = D + kQPad, NL = D / 32;   // pieces of a row; pieces per lane
  constexpr int NV = MODE == HIPATTN_ROPE_RELATIVE ? 2 : 1;    // scores per row and head
  using Raw = typename std::conditional<F8, uint2, uint4>::type;
  extern __shared__ __align__(16) unsigned char smem[];
  float* q32 = reinterpret_cast<float*>(smem);                                      // [HB][QS] pooled, scaled queries
  uint4* trig = reinterpret_cast<uint4*>(q32 + HB * QS);                            // relative: [2 positions][cos, sin][D / 16 pieces]
  float2* tabs = reinterpret_cast<float2*>(trig + (NV == 2 ? D / 4 : 0));           // [4 warps][NV][HB][kTabStride] bounds of the rounded scores
  __shared__ unsigned short s_list[4][32];
  __shared__ unsigned long long s_src[4][2][kPass];
  __shared__ int s_pmin;
  __shared__ float s_qmax[8];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int Gq = p.H / p.HKV;
  const int BDST = cdiv(p.TQ, p.block_size_q);
  const int n_hb = cdiv(Gq, HB);
  int64_t bid = blockIdx.x;
  const int split = (int)(bid % n_split); bid /= n_split;
  const int hb = (int)(bid % n_hb); bid /= n_hb;
  const int d = (int)(bid % BDST); bid /= BDST;
  const int hkv = (int)(bid % p.HKV); bid /= p.HKV;
  const int b = (int)bid;
  const int h0 = hkv * Gq + hb * HB;
  const int heads = min(HB, Gq - hb * HB);
  const int t0 = d * p.block_size_q;
  if (t0 >= p.TQ) return;

  if (threadIdx.x < 8) s_qmax[threadIdx.x] = 0.f;
  __syncthreads();
  for (int i = threadIdx.x; i < HB * PIECES; i += 128) {
    const int hh = i / PIECES, pc = i % PIECES;
    float v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = 0.f;
    if (hh < heads) pooled_query_piece<DT>(p, b, h0 + hh, t0, pc, v);
    float m = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      q32[hh * QS + pc * 8 + e] = v[e];
      m = fmaxf(m, fabsf(v[e]));
    }
    atomicMax(reinterpret_cast<int*>(&s_qmax[hh]), __float_as_int(m));   // non-negative floats order as ints
  }
  if (MODE == HIPATTN_ROPE_RELATIVE) {
    for (int i = threadIdx.x; i < D / 4; i += 128)
      trig[i] = rope_table_raw((i / (D / 16)) & 1 ? p.rope_sin : p.rope_cos, p.rope_stride, p.rope_rows, i / (D / 8), i % (D / 16));
  }
  if (warp == 0) {
    const int m = block_min_position(p, b, t0, 1, lane);
    if (lane == 0) s_pmin = m;
  }
  __syncthreads();
  const int pt = max(s_pmin - p.scan_window, 0);
  const int C = 1 << c_log2;
  const int cpp_log2 = 6 - c_log2;                  // chunks per pass = kPass / C
  const int n = p.n_chunks;
  const int64_t row = (int64_t)b * BDST + d;
  const int32_t* gl = p.left + row * n;
  const int32_t* gr = p.right + row * n;
  const int bc_log2 = 31 - __clz(p.block_chunk);
  float2* wtab = tabs + warp * NV * HB * kTabStride;
  // queries as the B operand: column lane / 4 = head; the k index of lane j's registers follows the rows' loads:
  // load i holds elements 32 i + 8 j .. + 7, its words 0 / 1 feed product 2 i, words 2 / 3 product 2 i + 1
  uint32_t qb[2 * NL][2];
#pragma unroll
  for (int ks = 0; ks < 2 * NL; ++ks)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float* s = q32 + (lane >> 2) * QS + (ks >> 1) * 32 + (lane & 3) * 8 + (ks & 1) * 4 + i * 2;
      qb[ks][i] = (lane >> 2) < HB ? pack2<DT>(s[0], s[1]) : 0u;   // exact: the queries are numbers of the element type
    }
  const uint32_t kscale2 = pack_scalar2<DT>(p.k_scale);
  // this lane's columns of a product: heads (lane % 4) * 2 and + 1
  const int col = (lane & 3) * 2;
  // (1.05: the magnitudes are summed in packed 16-bit arithmetic, at most 16 terms each)
  const float eps0 = kEps * 1.05f * s_qmax[col], eps1 = kEps * 1.05f * s_qmax[col + 1];
  const int check_tab = 4 * NV * HB * kTabStride;   // check mode: tables of the raw products and their radii follow
  int cur_group = -1, cur_gmax = 0;
  unsigned long long st_keys = 0, st_fb = 0, st_wrong = 0;
  float st_ratio = 0.f;

  // Address of this KV head's row of token t (token_row's rules, the call's constants taken out of the loop; positions that
  // read page 0 and page ids that are out of range included).
  const int eb = F8 ? 1 : 2;
  const bool paged = p.k.cache != nullptr;
  const char* hbase = paged ? (const char*)p.k.cache + (int64_t)hkv * p.k.stride_ch * eb
                            : (const char*)p.k.dense + ((int64_t)b * p.k.stride_b + (int64_t)hkv * p.k.stride_h) * eb;
  const int64_t step_b = (paged ? p.k.stride_off : p.k.stride_t) * eb, page_b = p.k.stride_page * eb;
  const int page_size = p.k.page_size;
  const int page_shift = paged && (page_size & (page_size - 1)) == 0 ? 31 - __clz(page_size) : -1;
  int64_t seq_len = 0;
  if (paged) seq_len = p.k.seq_lens_is_i64 ? ((const int64_t*)p.k.cache_seq_lens)[b] : (int64_t)((const int32_t*)p.k.cache_seq_lens)[b];
  const int reach = (int)max((int64_t)0, min(seq_len, (int64_t)p.k.table_width * page_size));   // tokens the table maps
  // (*mark: the slot of the access counter, the position of a dense key or the page as the table has it)
  auto row_of = [&](int t, int* mark) -> const char* {
    *mark = t;
    if (!paged) return hbase + (int64_t)t * step_b;
    const int pi = page_shift >= 0 ? (t >> page_shift) : (t / page_size);
    int64_t page = 0;
    *mark = 0;
    if (t < reach) {
      const int64_t o = (int64_t)b * p.k.table_stride_b + pi;
      page = p.k.table_is_i64 ? __ldg((const long long*)p.k.block_table + o) : (int64_t)__ldg((const int*)p.k.block_table + o);
      *mark = page < 0 || page > 0x7fffffff ? -1 : (int)page;
      if (page < 0 || page >= p.k.n_pages) {
        atomicOr(p.status, HIPATTN_STATUS_PAGE_RANGE);
        page = 0;
      }
    }
    return hbase + page * page_b + (int64_t)(t - pi * page_size) * step_b;
  };

  // What a pass needs before its rows can be requested: the chunk bounds and the row addresses of this lane's two tokens
  // (rows lane and lane + 32 of the pass; two dependent global reads: the bounds, then the page table), resolved one pass
  // ahead.  A row that is not needed reads the zero row.
  struct PassInput {
    int l[2], rt[2];
    const char* src[2];
    int mark[2];
    bool any;
  };
  auto resolve_pass = [&](int ps) {
    PassInput in{{0, 0}, {0, 0}, {(const char*)g_zero_key, (const char*)g_zero_key}, {-1, -1}, false};
    if (ps >= passes_total) return in;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int c = (ps << cpp_log2) + ((lane + 32 * i) >> c_log2);
      if (c < n) { in.l[i] = __ldg(gl + c); in.rt[i] = __ldg(gr + c); }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int l = in.l[i], rt = in.rt[i];
      if (rt - l > C) atomicOr(p.status, HIPATTN_STATUS_CHUNK_SIZE);
      int tk = l + (lane & (C - 1));
      if (l <= pt && l >= 0 && tk < rt) {
        if (!paged && tk >= p.T) {
          atomicOr(p.status, HIPATTN_STATUS_TOKEN_RANGE);
          tk = p.T - 1;
        }
        in.src[i] = row_of(tk, &in.mark[i]);
        in.any = true;
      }
    }
    return in;
  };

  using P = typename Pair16<DT>::type;
  auto as_p = [](uint32_t w) { return *reinterpret_cast<const P*>(&w); };
  auto as_u = [](P w) { return *reinterpret_cast<const uint32_t*>(&w); };
  auto load_raw = [](const char* row, int piece) -> Raw {
    if constexpr (F8) return load_row8(row + piece * 8);
    else return load_row16(row + piece * 16);
  };
  auto widen = [](const Raw& r) -> uint4 {
    if constexpr (F8) return widen_fp8_e5m2<DT>(r);
    else return r;
  };
  // strict score of a row for head hh: sequential fp32 dot product of round(rotated k * k_scale)
  auto strict_score = [&](const char* row, int hh, int c, int side) -> float {
    const float* qr = q32 + hh * QS;
    float acc = 0.f;
    auto add = [&](const uint4& w, int pc) {
      const float4 qa = *reinterpret_cast<const float4*>(qr + pc * 8), qc = *reinterpret_cast<const float4*>(qr + pc * 8 + 4);
      const float qv[8] = {qa.x, qa.y, qa.z, qa.w, qc.x, qc.y, qc.z, qc.w};
      const uint32_t wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t m = mul2<DT>(wv[i], kscale2);
        acc = fmaf(qv[2 * i], lo_f32<DT>(m), acc);
        acc = fmaf(qv[2 * i + 1], hi_f32<DT>(m), acc);
      }
    };
    if constexpr (MODE == HIPATTN_ROPE_NONE) {
#pragma unroll 1
      for (int p0 = 0; p0 < PIECES; p0 += 8) {
        Raw r[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) r[i] = load_raw(row, p0 + i);
#pragma unroll
        for (int i = 0; i < 8; ++i) add(widen(r[i]), p0 + i);
      }
    } else {
      constexpr int HALF = PIECES / 2;
      const int pos = MODE == HIPATTN_ROPE_RELATIVE ? side : c;
      // (the sum runs over the first half of the row, then the second: the pairs are rotated twice, which costs less than
      // keeping the rotated second half)
#pragma unroll 1
      for (int p0 = 0; p0 < PIECES; p0 += 4) {
        Raw r[4], rr[4];
        const int x0 = p0 < HALF ? p0 + HALF : p0 - HALF;
#pragma unroll
        for (int i = 0; i < 4; ++i) { r[i] = load_raw(row, p0 + i); rr[i] = load_raw(row, x0 + i); }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int tp = (p0 + i) % HALF;
          uint4 tc, ts;
          if (MODE == HIPATTN_ROPE_RELATIVE) {
            tc = trig[(pos * 2) * (D / 16) + tp];
            ts = trig[(pos * 2 + 1) * (D / 16) + tp];
          } else {
            tc = rope_table_raw(p.rope_cos, p.rope_stride, p.rope_rows, pos, tp);
            ts = rope_table_raw(p.rope_sin, p.rope_stride, p.rope_rows, pos, tp);
          }
          uint4 lo = p0 < HALF ? widen(r[i]) : widen(rr[i]), hi = p0 < HALF ? widen(rr[i]) : widen(r[i]);
          rope_rotate_packed<DT>(lo, hi, tc, ts);
          add(p0 < HALF ? lo : hi, p0 + i);
        }
      }
    }
    return acc;
  };

  // sixteen rows of a pass as operand registers: pieces 4 i + lane % 4 of rows 16 mt + lane / 4 and + 8
  struct Rows {
    Raw lo[NL], hi[NL];
  };
  auto load_rows = [&](Rows& r, int buf, int mt) {
    const char* a = (const char*)s_src[warp][buf][mt * 16 + (lane >> 2)];
    const char* c = (const char*)s_src[warp][buf][mt * 16 + (lane >> 2) + 8];
#pragma unroll
    for (int i = 0; i < NL; ++i) {
      r.lo[i] = load_raw(a, 4 * i + (lane & 3));
      r.hi[i] = load_raw(c, 4 * i + (lane & 3));
    }
  };

  const int ps_step = n_split * 4;
  // The pass at hand and the one behind it: addresses are written to shared memory a pass ahead, and the first sixteen
  // rows of the next pass are requested before this pass's last ones are multiplied.
  PassInput next_in = resolve_pass(split * 4 + warp);
  auto publish = [&](const PassInput& in, int buf) {
    s_src[warp][buf][lane] = (unsigned long long)in.src[0];
    s_src[warp][buf][lane + 32] = (unsigned long long)in.src[1];
    __syncwarp();
  };
  publish(next_in, 0);
  int buf = 0;
  Rows rows[2];
  load_rows(rows[0], 0, 0);
  for (int ps = split * 4 + warp; ps < passes_total; ps += ps_step, buf ^= 1) {
    const PassInput in = next_in;
    const int c_first = ps << cpp_log2;
    next_in = resolve_pass(ps + ps_step);
    publish(next_in, buf ^ 1);
    // halving rounds: from the largest chunk of the reference group of block_chunk chunks (all chunks of a
    // pass lie in one group: a pass holds at most 16 chunks, a group at least 16, both powers of two)
    const int group = c_first >> bc_log2;
    if (group != cur_group) {
      int m = 0;
      const int gbase = group << bc_log2;
      for (int i = lane; i < p.block_chunk; i += 32) {
        const int cc = gbase + i;
        if (cc < n) m = max(m, __ldg(gr + cc) - __ldg(gl + cc));
      }
      cur_gmax = __reduce_max_sync(0xffffffffu, m);
      cur_group = group;
    }
    const int rounds = cur_gmax >= 1 ? 32 - __clz(cur_gmax) : 0;
    const bool any_valid = __any_sync(0xffffffffu, in.any);
    uint32_t unsure = 0;
    if (!any_valid) {
      load_rows(rows[0], buf ^ 1, 0);
    } else {
      // ---- scores of 64 rows x HB heads, 16 rows at a time; bit (mt * NV + v) * 4 + i of `unsure`: this lane's
      // accumulator i of that product is not certain ----
#pragma unroll 1
      for (int m2 = 0; m2 < kPass / 16; m2 += 2)
#pragma unroll
      for (int mi = 0; mi < 2; ++mi) {
        const int mt = m2 + mi;
        if (mt + 1 < kPass / 16) load_rows(rows[mi ^ 1], buf, mt + 1);
        else load_rows(rows[mi ^ 1], buf ^ 1, 0);
        const Rows& cur = rows[mi];
        float x[NV][4], s[NV][4];
        P mag[NV][2];
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          mag[v][0] = mag[v][1] = as_p(0u);
#pragma unroll
          for (int i = 0; i < 4; ++i) x[v][i] = 0.f;
        }
        // one load of both rows: scale, magnitudes, two products
        auto product = [&](int v, const uint4& rl, const uint4& rh, int i) {
          uint32_t a[4], w[4];
          a[0] = mul2<DT>(rl.x, kscale2); a[2] = mul2<DT>(rl.y, kscale2); w[0] = mul2<DT>(rl.z, kscale2); w[2] = mul2<DT>(rl.w, kscale2);
          a[1] = mul2<DT>(rh.x, kscale2); a[3] = mul2<DT>(rh.y, kscale2); w[1] = mul2<DT>(rh.z, kscale2); w[3] = mul2<DT>(rh.w, kscale2);
          mma16816<DT>(x[v], a, qb[2 * i][0], qb[2 * i][1]);
          mma16816<DT>(x[v], w, qb[2 * i + 1][0], qb[2 * i + 1][1]);
          mag[v][0] = __hadd2(__hadd2(mag[v][0], __habs2(as_p(a[0]))), __habs2(as_p(a[2])));
          mag[v][1] = __hadd2(__hadd2(mag[v][1], __habs2(as_p(a[1]))), __habs2(as_p(a[3])));
          mag[v][0] = __hadd2(__hadd2(mag[v][0], __habs2(as_p(w[0]))), __habs2(as_p(w[2])));
          mag[v][1] = __hadd2(__hadd2(mag[v][1], __habs2(as_p(w[1]))), __habs2(as_p(w[3])));
        };
        if constexpr (MODE == HIPATTN_ROPE_NONE) {
#pragma unroll
          for (int i = 0; i < NL; ++i) product(0, widen(cur.lo[i]), widen(cur.hi[i]), i);
        } else {
          const int cr0 = c_first + ((mt * 16 + (lane >> 2)) >> c_log2), cr1 = c_first + ((mt * 16 + (lane >> 2) + 8) >> c_log2);
#pragma unroll
          for (int i = 0; i < NL / 2; ++i) {
            const int tp = 4 * i + (lane & 3);
#pragma unroll
            for (int v = 0; v < NV; ++v) {
              uint4 l0 = widen(cur.lo[i]), l1 = widen(cur.lo[i + NL / 2]), u0 = widen(cur.hi[i]), u1 = widen(cur.hi[i + NL / 2]);
              if (MODE == HIPATTN_ROPE_RELATIVE) {
                const uint4 tc = trig[(v * 2) * (D / 16) + tp], ts = trig[(v * 2 + 1) * (D / 16) + tp];
                rope_rotate_packed<DT>(l0, l1, tc, ts);
                rope_rotate_packed<DT>(u0, u1, tc, ts);
              } else {
                rope_rotate_packed<DT>(l0, l1, rope_table_raw(p.rope_cos, p.rope_stride, p.rope_rows, cr0, tp),
                                       rope_table_raw(p.rope_sin, p.rope_stride, p.rope_rows, cr0, tp));
                rope_rotate_packed<DT>(u0, u1, rope_table_raw(p.rope_cos, p.rope_stride, p.rope_rows, cr1, tp),
                                       rope_table_raw(p.rope_sin, p.rope_stride, p.rope_rows, cr1, tp));
              }
              product(v, l0, u0, i);
              product(v, l1, u1, i + NL / 2);
            }
          }
        }
#pragma unroll
        for (int v = 0; v < NV; ++v)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const uint32_t w = as_u(mag[v][i]);
            float m = lo_f32<DT>(w) + hi_f32<DT>(w);
            m += __shfl_xor_sync(0xffffffffu, m, 1);
            m += __shfl_xor_sync(0xffffffffu, m, 2);
            s[v][2 * i] = m;
          }
        const int r = mt * 16 + (lane >> 2);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          float2* t = wtab + (v * HB + col) * kTabStride + r;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float e = ((i & 1) ? eps1 : eps0) * s[v][i & 2];
            const float lo = Elem<DT>::round(x[v][i] - e), hi = Elem<DT>::round(x[v][i] + e);
            const int at = (i & 1) * kTabStride + (i >> 1) * 8;
            if (col + (i & 1) < HB) t[at] = make_float2(lo, hi);
            if (lo != hi) unsure |= 1u << ((mt * NV + v) * 4 + i);
            if (check && col + (i & 1) < heads) {   // every score by both definitions, compared below
              t[check_tab + at] = make_float2(x[v][i], e);
              unsure |= 1u << ((mt * NV + v) * 4 + i);
            }
          }
        }
      }
      __syncwarp();
    }
    // One lane per (chunk, head) replays the search on the bounds.  Where they leave a comparison or a chunk's best score
    // open (a few passes in a hundred), the pass's uncertain scores are computed by the strict definition and the search
    // runs again.  Chunks that are not active report their unchanged bounds.
    bool exact = check || p.score_out != nullptr;
    for (;;) {
      if (exact) {
        // ---- the uncertain scores by the strict definition, one per lane ----
        // (A column beyond the heads has neither a table nor a query row.  Its bounds differ where a key's product or magnitude
        // is not finite - 0 * inf is not a number -, so it is taken off the list here: bit 0 of an accumulator's number is its
        // column.)
        unsure &= (col < heads ? 0x55555555u : 0u) | (col + 1 < heads ? 0xaaaaaaaau : 0u);
        while (__any_sync(0xffffffffu, unsure != 0)) {
          const int mine = __popc(unsure);
          int at = mine;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, at, o);
            if (lane >= o) at += y;
          }
          const int total = min(32, __shfl_sync(0xffffffffu, at, 31));
          at -= mine;
          while (unsure && at < 32) {
            const int bit = __ffs(unsure) - 1;
            unsure &= unsure - 1;
            const int i = bit & 3, v = (bit >> 2) % NV, mt = (bit >> 2) / NV;
            s_list[warp][at++] = (unsigned short)((v << 9) | ((col + (i & 1)) << 6) | (mt * 16 + (lane >> 2) + (i >> 1) * 8));
          }
          __syncwarp();
          if (lane < total) {
            const int code = s_list[warp][lane], r = code & 63, hh = (code >> 6) & 7, v = code >> 9;
            float2* t = wtab + (v * HB + hh) * kTabStride + r;
            const float raw = strict_score((const char*)s_src[warp][buf][r], hh, c_first + (r >> c_log2), v);
            float ex = Elem<DT>::round(raw);
            if (nan_loses) ex = fmaxf(ex, -INFINITY);
            if (check) {
              const float xv = t[check_tab].x, e = t[check_tab].y;
              ++st_keys;
              if (t->x != t->y) ++st_fb;
              else if (t->x != ex) ++st_wrong;
              if (e > 0.f) st_ratio = fmaxf(st_ratio, fabsf(xv - raw) / e);
            }
            *t = make_float2(ex, ex);
          }
          __syncwarp();
        }
        __syncwarp();
      }
      bool open = false;
      uint32_t seen0 = 0, seen1 = 0;   // rows the reference's rounds would have loaded
      const int hb_log2 = 31 - __clz(HB);
      for (int w0 = 0; w0 < (HB << cpp_log2); w0 += 32) {
        const int wi = w0 + lane;
        const int hh = wi & (HB - 1), cw = wi >> hb_log2;
        const int c = c_first + cw;
        const int rbase = (cw << c_log2) & (kPass - 1);
        const int la = __shfl_sync(0xffffffffu, in.l[0], rbase & 31), lb = __shfl_sync(0xffffffffu, in.l[1], rbase & 31);
        const int ra = __shfl_sync(0xffffffffu, in.rt[0], rbase & 31), rb = __shfl_sync(0xffffffffu, in.rt[1], rbase & 31);
        const int l = rbase < 32 ? la : lb, rt = rbase < 32 ? ra : rb;
        const bool walker = hh < heads && cw < (1 << cpp_log2) && c < n;
        float slo = HIPATTN_SCORE_INIT, shi = HIPATTN_SCORE_INIT;
        bool mine_open = false;
        int wl = l, wr = rt;
        if (walker) {
          const float2* t0_ = wtab + hh * kTabStride + rbase;
          const float2* t1_ = t0_ + (NV - 1) * HB * kTabStride;
          for (int it = 0; it < rounds; ++it) {
            if (!(wl < wr && wl <= pt && wl >= 0)) break;
            const int mid = (wl + wr) >> 1, tl = (wl + mid) >> 1, tr = (mid + wr) >> 1;
            const int ol = min(tl - l, C - 1), orr = min(tr - l, C - 1);
            if (p.access_counter) {
              const unsigned long long m = (1ull << (rbase + ol)) | (1ull << (rbase + orr));
              seen0 |= (uint32_t)m;
              seen1 |= (uint32_t)(m >> 32);
            }
            const float2 sl = t0_[ol], sr = t1_[orr];
            const bool win = sl.x > sr.y;
            // (a key does not beat itself; bounds that are not numbers leave its score open all the same)
            if (!exact && !win && !(sl.y <= sr.x) && (NV == 2 || ol != orr || !(sl.x <= sl.y))) {
              mine_open = true;
              break;
            }
            if (win) wr = mid; else wl = mid;
            slo = fmaxf(slo, win ? sl.x : sr.x);
            shi = fmaxf(shi, win ? sl.y : sr.y);
          }
          if (!mine_open) {
            const int64_t o = (row * p.H + h0 + hh) * n + c;
            if (p.left_out) p.left_out[o] = wl;
            if (p.right_out) p.right_out[o] = wr;
            if (p.score_out) p.score_out[o] = slo;
          }
        }
        for (int o = 1; o < HB; o <<= 1) {
          slo = fmaxf(slo, __shfl_xor_sync(0xffffffffu, slo, o));
          shi = fmaxf(shi, __shfl_xor_sync(0xffffffffu, shi, o));
          mine_open |= (bool)__shfl_xor_sync(0xffffffffu, (int)mine_open, o);
        }
        mine_open |= slo != shi;
        open |= mine_open;
        if (!mine_open && walker && hh == 0 && slo > HIPATTN_SCORE_INIT) atomicMax(p.score_max + row * n + c, encode_score(slo));
      }
      if (!exact && __any_sync(0xffffffffu, open)) {
        exact = true;
        continue;
      }
      if (p.access_counter) {
        seen0 = __reduce_or_sync(0xffffffffu, seen0);
        seen1 = __reduce_or_sync(0xffffffffu, seen1);
        int32_t* ctr = p.access_counter + (int64_t)b * p.access_stride_b + (int64_t)hkv * p.access_stride_h;
        if ((seen0 >> lane & 1) && in.mark[0] >= 0 && in.mark[0] < p.access_n) ctr[in.mark[0]] = 1;
        if ((seen1 >> lane & 1) && in.mark[1] >= 0 && in.mark[1] < p.access_n) ctr[in.mark[1]] = 1;
      }
      break;
    }
    __syncwarp();
  }
  if (p.stats) {
    unsigned long long* st = reinterpret_cast<unsigned long long*>(p.stats);
    if (st_keys) atomicAdd(st + ST_KEYS, st_keys);
    if (st_fb) atomicAdd(st + ST_FALLBACK, st_fb);
    if (st_wrong) atomicAdd(st + ST_WRONG, st_wrong);
    atomicMax(reinterpret_cast<unsigned int*>(p.stats + ST_RATIO_BITS), __float_as_uint(st_ratio));
  }
}

template <int DT, int D, int MODE, bool F8>
int launch(const hipattn_scan_params_t& p, int c_log2, int HB, cudaStream_t stream) {
  constexpr int NV = MODE == HIPATTN_ROPE_RELATIVE ? 2 : 1;
  const size_t smem = (size_t)HB * (D + kQPad) * 4 + (NV == 2 ? D * 4 : 0) + (size_t)4 * NV * HB * kTabStride * 8 * (p.mode == HIPATTN_SCAN_CHECK ? 2 : 1);
  const int BDST = cdiv(p.TQ, p.block_size_q);
  const int n_hb = cdiv(p.H / p.HKV, HB);
  const int passes_total = cdiv(p.n_chunks, kPass >> c_log2);
  const int64_t units = (int64_t)p.B * p.HKV * BDST * n_hb;
  // enough CTAs to fill the GPU three times over, never more than there are passes for four warps each
  int64_t want = (148 * 4 * 3 + units - 1) / units;
  const int64_t most = cdiv(passes_total, 4);
  int n_split = (int)(want < 1 ? 1 : (want > most ? most : want));
  if (n_split < 1) n_split = 1;
  const int64_t grid = units * n_split;
  HIPATTN_REQUIRE(grid > 0 && grid < 0x7fffffffLL, HIPATTN_ERR_INVALID, "scan grid of %lld blocks", (long long)grid);
  auto kern = scan_chunks_mma_kernel<DT, D, MODE, F8>;
  HIPATTN_CUDA_OK(allow_smem((const void*)kern, smem));
  // A score that is not a number: the whole-chunk strict kernel compares it as it is, the kernel that goes by rounds takes it
  // for the lowest.  Masks are those of the strict mode, whichever of the two that takes.
  const bool nan_loses = strict_chunk_heads(p) == 0;
  kern<<<(unsigned)grid, 128, smem, stream>>>(p, c_log2, HB, n_split, passes_total, p.mode == HIPATTN_SCAN_CHECK ? 1 : 0, nan_loses ? 1 : 0);
  return check_launch("scan_chunks_mma_kernel");
}

template <int DT, int D, bool F8>
int dispatch_mode(const hipattn_scan_params_t& p, int c_log2, int HB, cudaStream_t stream) {
  switch (p.rope_mode) {
    case HIPATTN_ROPE_RELATIVE: return launch<DT, D, HIPATTN_ROPE_RELATIVE, F8>(p, c_log2, HB, stream);
    case HIPATTN_ROPE_STREAMING: return launch<DT, D, HIPATTN_ROPE_STREAMING, F8>(p, c_log2, HB, stream);
    default: return launch<DT, D, HIPATTN_ROPE_NONE, F8>(p, c_log2, HB, stream);
  }
}

template <int DT>
int dispatch_dim(const hipattn_scan_params_t& p, int c_log2, int HB, cudaStream_t stream) {
  if (p.k.fp8_e5m2) return p.D == 128 ? dispatch_mode<DT, 128, true>(p, c_log2, HB, stream) : dispatch_mode<DT, 64, true>(p, c_log2, HB, stream);
  return p.D == 128 ? dispatch_mode<DT, 128, false>(p, c_log2, HB, stream) : dispatch_mode<DT, 64, false>(p, c_log2, HB, stream);
}

}  // namespace

// 16-bit decode (a single pooled query row), head dim 64 or 128, whose chunk size is a known power of two between 4 and 32
// and no larger than the number of rows the rounds of the heads sharing the chunk would fetch: with more, the rounds
// move fewer bytes.  HIPATTN_SCAN_MODE=strict and HIPATTN_DECODE_SCAN=rounds | strict keep the other kernels.
int scan_chunks_mma(const hipattn_scan_params_t& p, cudaStream_t stream, bool* handled) {
  *handled = false;
  const int R = p.block_size_q / p.stride_q;
  if (p.mode == HIPATTN_SCAN_STRICT || p.dtype == HIPATTN_F32 || min(R, cdiv(p.TQ, p.stride_q)) > 1 || (p.D != 64 && p.D != 128)) return HIPATTN_OK;
  const int C = p.chunk_size;
  if (C < 4 || C > 32 || (C & (C - 1)) != 0) return HIPATTN_OK;
  const char* v = getenv("HIPATTN_DECODE_SCAN");
  if (v && (strcmp(v, "rounds") == 0 || strcmp(v, "strict") == 0)) return HIPATTN_OK;
  int c_log2 = 0;
  while ((1 << c_log2) < C) ++c_log2;
  const int Gq = p.H / p.HKV;
  int HB = 1;
  while (HB < 8 && HB < Gq) HB <<= 1;
  if (C > min(HB, Gq) * 2 * (c_log2 + 1)) return HIPATTN_OK;
  *handled = true;
  return p.dtype == HIPATTN_F16 ? dispatch_dim<HIPATTN_F16>(p, c_log2, HB, stream) : dispatch_dim<HIPATTN_BF16>(p, c_log2, HB, stream);
}

}  // namespace hipattn
