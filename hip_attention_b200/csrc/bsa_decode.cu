// Block-sparse attention, decode (one query row per sequence): two kernels, both bound by memory.
//
// bsa_decode_mma_kernel (16-bit and fp8 rows of head dim 64 or 128, up to eight query heads per KV head; described where it
// begins) is the one that decode calls run on.  bsa_decode_kernel takes the rest: fp32, and 16-bit rows of head dim 256.
//
// bsa_decode_kernel: one CTA owns (batch, KV head, key range).  The G query heads of the KV group share every K / V row
// that is fetched.  A warp walks its part of the key list 32 keys at a time:
//   lanes resolve 32 list entries to positions, admission and row addresses (page-table lookups);
//   K rows are read with 16-byte loads, LPR lanes per row (a 256-byte row = 16 lanes), several rows
//   in flight per lane; partial dot products are reduced inside the LPR-lane group;
//   the 32 x G logits are soft-maxed as one group (base 2, running maximum per head);
//   V rows are read the same way and accumulated with the probabilities.
// Warps are merged through shared memory; the CTA writes either the final rows (one range) or a
// normalised partial output with its base-2 log-sum-exp (several ranges, merged by merge_kernel).
#include "bsa_common.cuh"
#include "mma_common.cuh"
#include "rope.cuh"
#include <type_traits>

namespace hipattn {
namespace {

constexpr int kWarps = 8;
constexpr float kLog2e = 1.4426950408889634f;

template <int DT>
__device__ __forceinline__ void widen16(const uint4& w, float* out);
template <>
__device__ __forceinline__ void widen16<HIPATTN_F32>(const uint4& w, float* out) {
  out[0] = __uint_as_float(w.x); out[1] = __uint_as_float(w.y); out[2] = __uint_as_float(w.z); out[3] = __uint_as_float(w.w);
}
template <>
__device__ __forceinline__ void widen16<HIPATTN_BF16>(const uint4& w, float* out) {
  const uint32_t v[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    out[2 * i] = __uint_as_float(v[i] << 16);
    out[2 * i + 1] = __uint_as_float(v[i] & 0xffff0000u);
  }
}
template <>
__device__ __forceinline__ void widen16<HIPATTN_F16>(const uint4& w, float* out) {
  const uint32_t v[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&v[i]));
    out[2 * i] = f.x;
    out[2 * i + 1] = f.y;
  }
}

__device__ __forceinline__ uint4 ldg_nc16(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// LPR = lanes per K / V row (row bytes / 16), G = query heads per KV head
template <int DT, int LPR, int G>
__global__ void __launch_bounds__(kWarps * 32, 1) bsa_decode_kernel(const hipattn_bsa_params_t p) {
  using T = typename Elem<DT>::type;
  constexpr int VEC = 16 / Elem<DT>::bytes;
  constexpr int D = LPR * VEC;
  constexpr int TPP = 32 / LPR;                      // keys per pass (one 16-byte load per lane)
  constexpr int PBMAX = G > 4 ? 8 : 16;              // bounds the rows a lane keeps in flight (registers)
  constexpr int PB = LPR < PBMAX ? LPR : PBMAX;      // passes per group
  constexpr int GK = PB * TPP;                       // keys per group (<= 32)

  __shared__ unsigned long long s_kptr[kWarps][2][32];
  __shared__ unsigned long long s_vptr[kWarps][2][32];
  extern __shared__ __align__(16) float s_merge[];  // [kWarps][G][D + 2]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane / LPR, piece = lane % LPR;  // key within a pass, 16-byte piece of the row
  int64_t bid = blockIdx.x;
  const int split = (int)(bid % p.n_splits); bid /= p.n_splits;
  const int hkv = (int)(bid % p.HKV); bid /= p.HKV;
  const int b = (int)bid;
  const int h0 = hkv * G;

  const long long px = p.pos[(int64_t)b * p.pos_stride_b];
  const int pq = (int)(px > 0x7ffffff0LL ? 0x7ffffff0LL : (px < 0 ? 0 : px));
  const KeyList kl = make_key_list(p, b, h0, 0, pq, pq);
  const int per = cdiv(cdiv(kl.total, p.n_splits), GK) * GK;
  const int j_begin = split * per, j_end = min(kl.total, j_begin + per);

  // this lane's slice of the G query rows
  float q[G][VEC];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const T* qp = reinterpret_cast<const T*>(p.q) + (int64_t)b * p.q_stride_b + (int64_t)(h0 + g) * p.q_stride_h + piece * VEC;
    widen16<DT>(*reinterpret_cast<const uint4*>(qp), q[g]);
  }
  float m_run[G], l_run[G], acc[G][VEC];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    m_run[g] = -INFINITY;
    l_run[g] = 0.f;
#pragma unroll
    for (int e = 0; e < VEC; ++e) acc[g][e] = 0.f;
  }
  const float cap = p.logit_softcap;

  // resolve the list entries of one group to row addresses (0 = not admitted)
  auto resolve = [&](int j0, int buf) {
    unsigned long long ka = 0, va = 0;
    const int j = j0 + lane;
    if (lane < GK && j < j_end) {
      bool w = false;
      const int t = key_position(kl, j, &w);
      if (admits(pq, t, w, p.window)) {
        ka = (unsigned long long)token_row(p.k, b, t, hkv, Elem<DT>::bytes, p.status);
        va = (unsigned long long)token_row(p.v, b, t, hkv, Elem<DT>::bytes, p.status);
      }
    }
    s_kptr[warp][buf][lane] = ka;
    s_vptr[warp][buf][lane] = va;
  };
  auto load_rows = [&](const unsigned long long* ptrs, uint4* regs) {
#pragma unroll
    for (int i = 0; i < PB; ++i) {
      const unsigned long long a = ptrs[i * TPP + sub];
      regs[i] = a != 0ull ? ldg_nc16((const char*)a + piece * 16) : make_uint4(0, 0, 0, 0);
    }
  };

  // software pipeline over groups: K rows of group i + 1 and V rows of group i are in flight while
  // group i is soft-maxed; addresses are resolved one group ahead
  const int stride = kWarps * GK;
  int j0 = j_begin + warp * GK;
  uint4 kw[PB], vw[PB];
  int buf = 0;
  if (j0 < j_end) {
    resolve(j0, 0);
    __syncwarp();
    load_rows(s_kptr[warp][0], kw);
  }
  for (; j0 < j_end; j0 += stride, buf ^= 1) {
    const bool more = j0 + stride < j_end;
    if (more) resolve(j0 + stride, buf ^ 1);
    load_rows(s_vptr[warp][buf], vw);
    // ---- logits: the key of pass r, slot sub ends up in lane sub * LPR + r ----
    float s[G];
#pragma unroll
    for (int g = 0; g < G; ++g) s[g] = -INFINITY;
#pragma unroll
    for (int i = 0; i < PB; ++i) {
      float kv[VEC];
      widen16<DT>(kw[i], kv);
      float part[G];
#pragma unroll
      for (int g = 0; g < G; ++g) {
        float a = 0.f;
#pragma unroll
        for (int e = 0; e < VEC; ++e) a = fmaf(q[g][e], kv[e], a);
        part[g] = a;
      }
#pragma unroll
      for (int o = LPR >> 1; o > 0; o >>= 1) {
#pragma unroll
        for (int g = 0; g < G; ++g) part[g] += __shfl_xor_sync(0xffffffffu, part[g], o);
      }
      if (piece == i && s_kptr[warp][buf][i * TPP + sub] != 0ull) {
#pragma unroll
        for (int g = 0; g < G; ++g) {
          float x = part[g];
          if (cap > 0.f) x = tanhf(x / cap) * cap;
          s[g] = x * kLog2e;
        }
      }
    }
    __syncwarp();
    if (more) load_rows(s_kptr[warp][buf ^ 1], kw);
    // ---- group softmax ----
    float pr[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
      float mx = s[g];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      const float m_new = fmaxf(m_run[g], mx);
      float alpha = 1.f;
      pr[g] = 0.f;
      if (m_new > -INFINITY) {
        alpha = exp2f(m_run[g] - m_new);
        pr[g] = exp2f(s[g] - m_new);
      }
      float sum = pr[g];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      l_run[g] = l_run[g] * alpha + sum;
      m_run[g] = m_new;
#pragma unroll
      for (int e = 0; e < VEC; ++e) acc[g][e] *= alpha;
    }
    // ---- O += P V ----
#pragma unroll
    for (int i = 0; i < PB; ++i) {
      float vv[VEC];
      widen16<DT>(vw[i], vv);
      const int keeper = sub * LPR + i;
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float pg = __shfl_sync(0xffffffffu, pr[g], keeper);
#pragma unroll
        for (int e = 0; e < VEC; ++e) acc[g][e] = fmaf(pg, vv[e], acc[g][e]);
      }
    }
  }

  // ---- combine the TPP key slots of a warp (same maxima), then the warps ----
#pragma unroll
  for (int o = LPR; o < 32; o <<= 1) {
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
      for (int e = 0; e < VEC; ++e) acc[g][e] += __shfl_xor_sync(0xffffffffu, acc[g][e], o);
  }
  constexpr int MS = D + 2;
  if (sub == 0) {
#pragma unroll
    for (int g = 0; g < G; ++g) {
      float* dst = s_merge + ((size_t)warp * G + g) * MS;
#pragma unroll
      for (int e = 0; e < VEC; ++e) dst[piece * VEC + e] = acc[g][e];
      if (piece == 0) { dst[D] = m_run[g]; dst[D + 1] = l_run[g]; }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < G * D; i += kWarps * 32) {
    const int g = i / D, e = i % D;
    float M = -INFINITY;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) M = fmaxf(M, s_merge[((size_t)w * G + g) * MS + D]);
    float num = 0.f, den = 0.f;
    if (M > -INFINITY) {
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        const float* src = s_merge + ((size_t)w * G + g) * MS;
        const float f = exp2f(src[D] - M);
        num += f * src[e];
        den += f * src[D + 1];
      }
    }
    const float val = den > 0.f ? num / den : 0.f;
    const float lse = den > 0.f ? M + log2f(den) : -INFINITY;
    const int hh = h0 + g;
    if (p.n_splits > 1) {
      const int64_t o = ((int64_t)b * p.H + hh) * p.n_splits + split;
      p.part_o[o * D + e] = val;
      if (e == 0) p.part_lse[o] = lse;
    } else {
      reinterpret_cast<T*>(p.out)[(int64_t)b * p.o_stride_b + (int64_t)hh * p.o_stride_h + e] = Elem<DT>::from_f32(val);
      if (e == 0 && p.lse_out) p.lse_out[(int64_t)b * p.H + hh] = lse;
    }
  }
}

// ---------------------------------------------------------------------------------------------------
// 16-bit types: tensor-core variant.  The G heads of the KV group are the rows of a 16-row MMA tile.  Every warp walks its
// own part of the key list, sixteen keys at a time, and keeps its own running maximum, sum and output; nothing is shared
// before the end, so the loop has no block-wide barrier.
//
// K and V rows go from global memory straight into operand registers.  S = Q K^T: the order of a contraction is free, so
// lane j of a key's four lanes loads the sixteen-byte pieces 4 i + j and the queries' fragments are laid out alike.
// O += P V: a register of the B operand pairs two keys of one column, so lane (g, j) loads eight consecutive columns
// 8 g .. of keys 2 j, 2 j + 1, 2 j + 8, 2 j + 9, pairs the keys with byte permutes, and column t of its load becomes
// column g of product t: the output's columns come out permuted and are put right when they are stored.
//
// Key ranges of one (sequence, KV head) are the CTAs of a cluster: their partial results meet in distributed shared memory,
// so a small batch fills the GPU without a second launch.  (A caller may also ask for ranges with partial outputs of
// their own, n_splits.)
//
// In-kernel RoPE: the key's pieces i and i + D / 64 hold elements d and d + D / 2, rotated in registers; the table pieces
// travel with the rows.  fp8 rows are widened in registers.
//
// TWO = the softmax weights go in two 16-bit terms, the rounded weight and what the rounding left.  A single term is exact for
// the largest weight of each warp's keys only, so its error grows as fewer warps share a list.  fp8 rows: always (the general
// kernel, which served them before, kept the weights in fp32).  RoPE: always (12 sequences, bf16, error against 64 bits before
// the output is rounded: 1.4e-4 with the sixteen warps to a list of the kernel before, 1.8e-4 with the eight here, below 2e-5
// with two terms, which cost nothing beside the rotation).  Else: in clusters of two, whose twelve warps replace the twelve to
// sixteen of the kernel before (12 sequences, bf16: 1.5e-4 then, 1.9e-4 with one term, 1e-6 with two, 49.4 -> 53.0 us a cached
// call).  A single CTA has six warps and more where there were four, larger clusters have as many warps as there were: one term
// (32 sequences: 2.5e-4 then, 2.4e-4 here; two terms would cost 6 % of a full batch).
//
// Bound: HBM.  32 sequences, 3328 keys each (436 MB): 0.115 ms with a three-stage shared-memory ring and a barrier per
// 64 keys (3.8 TB/s), 0.080 ms here (5.4 TB/s).  One sequence: 10.8 + 4.7 us (attention, merge), 12.9 us here.  RoPE, 12 sequences:
// 0.121 ms, 0.061 here.  fp8 with RoPE, 5 sequences: 0.254 ms (general kernel), 0.045 here.
// ---------------------------------------------------------------------------------------------------
// Warps per CTA, two CTAs per multiprocessor: six (168 registers), so that 256 CTAs of a full batch are resident at once;
// four with RoPE on 16-bit rows, whose table pieces take the registers of the difference (six would spill: 76 us for 61).
template <bool ROPE, bool F8> constexpr int kDecodeWarps = ROPE && !F8 ? 4 : 6;
constexpr int kMaxCluster = 16;   // CTAs of a cluster (beyond eight: allowed per kernel; one sequence 13.8 us with eight, 12.9 with sixteen)

__device__ __align__(256) unsigned char g_zero_kv[256];   // the row of a key that is not admitted

__device__ __forceinline__ uint2 ldg_nc8(const void* p) {
  uint2 v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];\n" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// address of the same shared-memory location in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ float ld_cluster(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

template <int DT, int D, bool ROPE, bool F8, bool TWO>
__global__ void __launch_bounds__(kDecodeWarps<ROPE, F8> * 32, 2) bsa_decode_mma_kernel(const hipattn_bsa_params_t p, int cluster) {
  using T = typename Elem<DT>::type;
  constexpr int NL = D / 32;        // pieces of a K row per lane
  constexpr int NB = D / 64;        // 64-column blocks
  constexpr int MS = D + 2;
  constexpr int EB = F8 ? 1 : 2;
  constexpr int kDW = kDecodeWarps<ROPE, F8>;
  using Raw = typename std::conditional<F8, uint2, uint4>::type;
  extern __shared__ __align__(16) float s_merge[];   // [kDW][G][MS], then the CTA's own result [G][MS]
  __shared__ unsigned long long s_ptr[kDW][2][32][2];  // K / V row of the 32 keys of a group, double buffered
  __shared__ int s_rpos[ROPE ? kDW : 1][2][32];
  __shared__ __align__(16) uint4 s_q[8][D / 8];      // query rows (rotated under RoPE)

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, jq = lane & 3;
  const int G = p.H / p.HKV;
  int64_t bid = blockIdx.x;
  const int rank = (int)(bid % cluster); bid /= cluster;
  const int split = (int)(bid % p.n_splits); bid /= p.n_splits;
  const int hkv = (int)(bid % p.HKV); bid /= p.HKV;
  const int b = (int)bid;
  const int h0 = hkv * G;

  const long long px = p.pos[(int64_t)b * p.pos_stride_b];
  const int pq = (int)(px > 0x7ffffff0LL ? 0x7ffffff0LL : (px < 0 ? 0 : px));
  const KeyList kl = make_key_list(p, b, h0, 0, pq, pq);
  // this warp's keys: the list is cut into n_splits ranges, a range over the warps of the cluster
  const int per_split = cdiv(cdiv(kl.total, p.n_splits), 16) * 16;
  const int s_begin = split * per_split, s_end = min(kl.total, s_begin + per_split);
  const int per = cdiv(cdiv(max(0, s_end - s_begin), cluster * kDW), 16) * 16;
  const int j_begin = s_begin + (rank * kDW + warp) * per, j_end = min(s_end, j_begin + per);

  // row addresses, with the call's constants taken out of the loop (token_row's rules)
  const bool paged = p.k.cache != nullptr && p.v.cache != nullptr && p.k.block_table == p.v.block_table &&
                     p.k.table_stride_b == p.v.table_stride_b && p.k.table_width == p.v.table_width && p.k.table_is_i64 == p.v.table_is_i64 &&
                     p.k.cache_seq_lens == p.v.cache_seq_lens && p.k.seq_lens_is_i64 == p.v.seq_lens_is_i64 && p.k.page_size == p.v.page_size;
  const bool dense = p.k.cache == nullptr && p.v.cache == nullptr;
  const char* kb = paged ? (const char*)p.k.cache + (int64_t)hkv * p.k.stride_ch * EB
                         : (const char*)p.k.dense + ((int64_t)b * p.k.stride_b + (int64_t)hkv * p.k.stride_h) * EB;
  const char* vb = paged ? (const char*)p.v.cache + (int64_t)hkv * p.v.stride_ch * EB
                         : (const char*)p.v.dense + ((int64_t)b * p.v.stride_b + (int64_t)hkv * p.v.stride_h) * EB;
  const int page_size = p.k.page_size;
  const int page_shift = paged && (page_size & (page_size - 1)) == 0 ? 31 - __clz(page_size) : -1;
  int64_t seq_len = 0;
  if (paged) seq_len = p.k.seq_lens_is_i64 ? ((const int64_t*)p.k.cache_seq_lens)[b] : (int64_t)((const int32_t*)p.k.cache_seq_lens)[b];
  const int reach = paged ? (int)max((int64_t)0, min(seq_len, (int64_t)p.k.table_width * page_size)) : 0;

  // The 32 keys of a group are resolved one per lane in three steps, one group apart, so that no step waits for memory:
  // the block start of a selected entry, the page of its token, the addresses.
  long long start = 0;      // step 1: of the group after next
  auto fetch_start = [&](int j0) {
    const int j = j0 + lane;
    const int blk = j < j_end ? selected_block_of(kl, j) : -1;
    start = blk >= 0 ? __ldg(reinterpret_cast<const long long*>(kl.idx) + blk) : 0;
  };
  int tok = -1, rp = -1;    // step 2: of the next group
  long long page = 0;
  auto fetch_page = [&](int j0) {
    const int j = j0 + lane;
    tok = -1;
    rp = -1;
    if (j < j_end) {
      bool w = false;
      const int t = key_position_at(kl, j, start, &w);
      if (admits(pq, t, w, p.window)) {
        tok = t;
        if (ROPE) rp = rope_key_position(kl, j, t);
        page = 0;
        if (paged && t < reach) {
          const int64_t o = (int64_t)b * p.k.table_stride_b + (page_shift >= 0 ? (t >> page_shift) : (t / page_size));
          page = p.k.table_is_i64 ? __ldg((const long long*)p.k.block_table + o) : (long long)__ldg((const int*)p.k.block_table + o);
        }
      }
    }
  };
  auto publish = [&](int buf) -> uint32_t {   // step 3; returns which keys are admitted
    const char *ka = (const char*)g_zero_kv, *va = (const char*)g_zero_kv;
    if (tok >= 0) {
      if (dense) {
        ka = kb + (int64_t)tok * p.k.stride_t * EB;
        va = vb + (int64_t)tok * p.v.stride_t * EB;
      } else if (paged) {
        if (page < 0 || page >= p.k.n_pages || page >= p.v.n_pages) {
          atomicOr(p.status, HIPATTN_STATUS_PAGE_RANGE);
          page = 0;
        }
        const int off = tok - (page_shift >= 0 ? ((tok >> page_shift) << page_shift) : (tok / page_size) * page_size);
        ka = kb + (page * p.k.stride_page + (int64_t)off * p.k.stride_off) * EB;
        va = vb + (page * p.v.stride_page + (int64_t)off * p.v.stride_off) * EB;
      } else {
        ka = token_row(p.k, b, tok, hkv, 2, p.status);
        va = token_row(p.v, b, tok, hkv, 2, p.status);
      }
    }
    s_ptr[warp][buf][lane][0] = (unsigned long long)ka;
    s_ptr[warp][buf][lane][1] = (unsigned long long)va;
    if (ROPE) s_rpos[warp][buf][lane] = max(rp, 0);
    const uint32_t m = __ballot_sync(0xffffffffu, tok >= 0);
    __syncwarp();
    return m;
  };
  auto load_raw = [](const char* row, int piece) -> Raw {
    if constexpr (F8) return ldg_nc8(row + piece * 8);
    else return ldg_nc16(row + piece * 16);
  };
  auto widen = [](const Raw& r) -> uint4 {
    if constexpr (F8) return widen_fp8_e5m2<DT>(r);
    else return r;
  };

  // group 0 on its way while the queries are prepared
  fetch_start(j_begin);
  fetch_page(j_begin);
  fetch_start(j_begin + 32);
  uint32_t live = publish(0);

  for (int i = tid; i < 8 * (D / 8); i += kDW * 32) {
    const int r = i / (D / 8), pc = i % (D / 8);
    uint4 v = make_uint4(0, 0, 0, 0);
    if (r < G) v = *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.q) + (int64_t)b * p.q_stride_b + (int64_t)(h0 + r) * p.q_stride_h + pc * 8);
    s_q[r][pc] = v;
  }
  __syncthreads();
  if (ROPE) {   // the query rows at the query's position (attention_decode_bsa.py:174-215)
    for (int i = tid; i < G * (D / 16); i += kDW * 32) {
      const int r = i / (D / 16), pc = i % (D / 16);
      uint4 lo = s_q[r][pc], hi = s_q[r][pc + D / 16];
      rope_rotate_packed<DT>(lo, hi, rope_table_raw(p.rope_cos, p.rope_stride, p.rope_rows, pq, pc),
                             rope_table_raw(p.rope_sin, p.rope_stride, p.rope_rows, pq, pc));
      s_q[r][pc] = lo;
      s_q[r][pc + D / 16] = hi;
    }
    __syncthreads();
  }

  float o[NB * 8][2];
#pragma unroll
  for (int i = 0; i < NB * 8; ++i) o[i][0] = o[i][1] = 0.f;
  float m_run = -INFINITY, l_run = 0.f;
  const float cap = p.logit_softcap;

  // sixteen keys: K pieces of keys g and g + 8, V columns of keys 2 j, 2 j + 1, 2 j + 8, 2 j + 9
  Raw kr[2][NL];
  uint4 tc[ROPE ? 2 : 1][ROPE ? NL / 2 : 1], ts[ROPE ? 2 : 1][ROPE ? NL / 2 : 1];
  auto load_k = [&](int buf, int half) {
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      const char* row = (const char*)s_ptr[warp][buf][half * 16 + nt * 8 + g][0];
#pragma unroll
      for (int i = 0; i < NL; ++i) kr[nt][i] = load_raw(row, 4 * i + jq);
      if constexpr (ROPE) {
        const int t = s_rpos[warp][buf][half * 16 + nt * 8 + g];
#pragma unroll
        for (int i = 0; i < NL / 2; ++i) {
          tc[nt][i] = rope_table_raw(p.rope_cos, p.rope_stride, p.rope_rows, t, 4 * i + jq);
          ts[nt][i] = rope_table_raw(p.rope_sin, p.rope_stride, p.rope_rows, t, 4 * i + jq);
        }
      }
    }
  };
  int buf = 0;
  if (j_begin < j_end) load_k(0, 0);
  for (int j0 = j_begin; j0 < j_end; j0 += 32, buf ^= 1) {
    fetch_page(j0 + 32);     // (its block starts arrived with the group before)
    fetch_start(j0 + 64);
    uint32_t next_live = 0;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      if (half == 1 && j0 + 16 >= j_end) break;
      Raw vr[4][NB];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const char* row = (const char*)s_ptr[warp][buf][half * 16 + 2 * jq + (i & 1) + (i >> 1) * 8][1];
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) vr[i][nb] = load_raw(row, nb * 8 + g);
      }
      // ---- S = Q K^T (rows lane / 4 < G; rows 8..15 are padding) ----
      float s[2][4];
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        s[nt][0] = s[nt][1] = s[nt][2] = s[nt][3] = 0.f;
        uint4 w[NL];
#pragma unroll
        for (int i = 0; i < NL; ++i) w[i] = widen(kr[nt][i]);
        if constexpr (ROPE) {
#pragma unroll
          for (int i = 0; i < NL / 2; ++i) rope_rotate_packed<DT>(w[i], w[i + NL / 2], tc[nt][i], ts[nt][i]);
        }
#pragma unroll
        for (int i = 0; i < NL; ++i) {
          const uint4 q = s_q[g][4 * i + jq];
          const uint32_t a0[4] = {q.x, 0u, q.y, 0u}, a1[4] = {q.z, 0u, q.w, 0u};
          mma16816<DT>(s[nt], a0, w[i].x, w[i].y);
          mma16816<DT>(s[nt], a1, w[i].z, w[i].w);
        }
      }
      // the next keys' rows travel while these are soft-maxed
      if (half == 0) {
        if (j0 + 16 < j_end) load_k(buf, 1);
      }
      if (half == 1 || j0 + 16 >= j_end) {
        next_live = publish(buf ^ 1);
        if (j0 + 32 < j_end) load_k(buf ^ 1, 0);
      }
      // ---- admission + online softmax ----
      if (cap > 0.f) {   // soft-cap behind its own uniform branch: inside the loop the tanh is evaluated under a predicate
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int e = 0; e < 2; ++e) s[nt][e] = tanhf(s[nt][e] / cap) * cap;
      }
      float mx = -INFINITY;
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const bool in = live >> (half * 16 + nt * 8 + jq * 2 + e) & 1u;
          s[nt][e] = in ? s[nt][e] * kLog2e : -INFINITY;
          mx = fmaxf(mx, s[nt][e]);
        }
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      const float m_new = fmaxf(m_run, mx);
      const float base = m_new > -INFINITY ? m_new : 0.f;
      const float alpha = exp2f(m_run - base);
      float sum = 0.f;
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        s[nt][0] = exp2f(s[nt][0] - base);
        s[nt][1] = exp2f(s[nt][1] - base);
        sum += s[nt][0] + s[nt][1];
      }
      l_run = l_run * alpha + sum;     // (this lane's keys; the four lanes of a row are added up at the end)
      m_run = m_new;
      if (__any_sync(0xffffffffu, alpha != 1.f)) {
#pragma unroll
        for (int i = 0; i < NB * 8; ++i) { o[i][0] *= alpha; o[i][1] *= alpha; }
      }
      // ---- O += P V ----
      uint32_t pa[4] = {pack2<DT>(s[0][0], s[0][1]), 0u, pack2<DT>(s[1][0], s[1][1]), 0u};
      uint32_t pl[4] = {0u, 0u, 0u, 0u};
      if constexpr (TWO) {   // what the rounding of the weights left
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          const float r0 = s[nt][0] - Elem<DT>::round(s[nt][0]), r1 = s[nt][1] - Elem<DT>::round(s[nt][1]);
          pl[nt * 2] = pack2<DT>(r0, r1);
        }
      }
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        uint4 w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = widen(vr[i][nb]);
        const uint32_t v0[4] = {w[0].x, w[0].y, w[0].z, w[0].w}, v1[4] = {w[1].x, w[1].y, w[1].z, w[1].w};
        const uint32_t v8[4] = {w[2].x, w[2].y, w[2].z, w[2].w}, v9[4] = {w[3].x, w[3].y, w[3].z, w[3].w};
#pragma unroll
        for (int t = 0; t < 8; ++t) {
          const uint32_t sel = (t & 1) ? 0x7632u : 0x5410u;
          const uint32_t b0 = __byte_perm(v0[t >> 1], v1[t >> 1], sel), b1 = __byte_perm(v8[t >> 1], v9[t >> 1], sel);
          float c[4] = {o[nb * 8 + t][0], o[nb * 8 + t][1], 0.f, 0.f};
          mma16816<DT>(c, pa, b0, b1);
          if constexpr (TWO) mma16816<DT>(c, pl, b0, b1);
          o[nb * 8 + t][0] = c[0];
          o[nb * 8 + t][1] = c[1];
        }
      }
    }
    live = next_live;
  }
  l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
  l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);

  // ---- merge the warps, then the CTAs of the cluster ----
  if (g < G) {
    float* dst = s_merge + ((size_t)warp * G + g) * MS;
#pragma unroll
    for (int i = 0; i < NB * 8; ++i) {   // column c of product t of block nb is column nb * 64 + 8 c + t
      const int c0 = (i >> 3) * 64 + (i & 7) + 16 * jq;
      dst[c0] = o[i][0];
      dst[c0 + 8] = o[i][1];
    }
    if (jq == 0) { dst[D] = m_run; dst[D + 1] = l_run; }
  }
  __syncthreads();
  float* s_cta = s_merge + (size_t)kDW * G * MS;
  auto finish = [&](int i, float M, float num, float den) {
    const int hh = h0 + i / D, e = i % D;
    const float val = den > 0.f ? num / den : 0.f;
    const float lse = den > 0.f ? M + log2f(den) : -INFINITY;
    if (p.n_splits > 1) {
      const int64_t oo = ((int64_t)b * p.H + hh) * p.n_splits + split;
      p.part_o[oo * D + e] = val;
      if (e == 0) p.part_lse[oo] = lse;
    } else {
      reinterpret_cast<T*>(p.out)[(int64_t)b * p.o_stride_b + (int64_t)hh * p.o_stride_h + e] = Elem<DT>::from_f32(val);
      if (e == 0 && p.lse_out) p.lse_out[(int64_t)b * p.H + hh] = lse;
    }
  };
  for (int i = tid; i < G * D; i += kDW * 32) {
    const int h = i / D, e = i % D;
    float M = -INFINITY;
#pragma unroll
    for (int w = 0; w < kDW; ++w) M = fmaxf(M, s_merge[((size_t)w * G + h) * MS + D]);
    float num = 0.f, den = 0.f;
    if (M > -INFINITY) {
#pragma unroll
      for (int w = 0; w < kDW; ++w) {
        const float* src = s_merge + ((size_t)w * G + h) * MS;
        const float f = exp2f(src[D] - M);
        num += f * src[e];
        den += f * src[D + 1];
      }
    }
    if (cluster == 1) {
      finish(i, M, num, den);
    } else {
      s_cta[h * MS + e] = num;
      if (e == 0) { s_cta[h * MS + D] = M; s_cta[h * MS + D + 1] = den; }
    }
  }
  if (cluster > 1) {
    cluster_sync();
    const uint32_t own = (uint32_t)__cvta_generic_to_shared(s_cta);
    for (int i = tid + rank * kDW * 32; i < G * D; i += cluster * kDW * 32) {
      const int h = i / D, e = i % D;
      float M = -INFINITY, num = 0.f, den = 0.f;
      for (int r = 0; r < cluster; ++r) {
        const uint32_t a = map_rank(own + (uint32_t)(h * MS) * 4, r);
        const float m = ld_cluster(a + D * 4), x = ld_cluster(a + e * 4), l = ld_cluster(a + (D + 1) * 4);
        if (m > -INFINITY) {
          const float m2 = fmaxf(M, m), fo = exp2f(M - m2), fn = exp2f(m - m2);
          num = num * fo + x * fn;
          den = den * fo + l * fn;
          M = m2;
        }
      }
      finish(i, M, num, den);
    }
    cluster_sync();   // no CTA leaves while another reads its shared memory
  }
  // Launched beside the kernel before it: that one has ended, and its writes are visible, before this one ends, so that what follows
  // on the stream finds both (nothing to wait for otherwise).
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
}

template <int DT, int D, bool ROPE, bool F8>
int launch_mma(const hipattn_bsa_params_t& p, cudaStream_t stream, bool beside) {
  constexpr int kDW = kDecodeWarps<ROPE, F8>;
  const int G = p.H / p.HKV;
  const size_t smem = sizeof(float) * (size_t)(kDW + 1) * G * (D + 2);
  const int64_t units = (int64_t)p.B * p.HKV * p.n_splits;
  // CTAs per unit: as many as put two on every multiprocessor, as long as every warp has at least sixteen keys and the device
  // holds the clusters of all units at once (a multiprocessor group has room for a whole number of them).  Sizes between the
  // powers of two count: with 4 for the 40 units of five sequences, where 7 fit, 24 warps shared a list instead of 42, and
  // the error of their single-term weights was 1.2 to 1.3 times as large.
  const int64_t keys = (p.sink < p.T ? p.sink : p.T) + (int64_t)p.K * p.block_size_k + (p.window < p.T ? p.window : p.T);
  auto kern = bsa_decode_mma_kernel<DT, D, ROPE, F8, F8 || ROPE>;
  HIPATTN_CUDA_OK(allow_smem((const void*)kern, smem));
  int64_t most = 148 * 2 / units;
  if (most > keys / p.n_splits / (kDW * 16)) most = keys / p.n_splits / (kDW * 16);
  int cluster = most < 1 ? 1 : (most > kMaxCluster ? kMaxCluster : (int)most);
  while (cluster > 1 && resident_clusters((const void*)kern, cluster, kDW * 32, smem) < units) --cluster;
  if constexpr (!F8 && !ROPE) {
    if (cluster == 2) {   // (see TWO)
      kern = bsa_decode_mma_kernel<DT, D, ROPE, F8, true>;
      HIPATTN_CUDA_OK(allow_smem((const void*)kern, smem));
    }
  }
  const int64_t grid = units * cluster;
  HIPATTN_REQUIRE(grid > 0 && grid < 0x7fffffffLL, HIPATTN_ERR_INVALID, "decode grid of %lld blocks", (long long)grid);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(kDW * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)cluster;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  // Beside the copies of the cached mask, which the launch before makes for the caller and the attention does not read: a cached call
  // of one sequence 18.5 -> 16.0 us, of 32 sequences 86.3 -> 84.8.
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = beside ? 2 : 1;
  HIPATTN_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, p, cluster));
  return check_launch("bsa_decode_mma_kernel");
}

template <int DT, int D>
int dispatch_mma(const hipattn_bsa_params_t& p, cudaStream_t stream, bool beside) {
  if (p.k.fp8_e5m2) return p.rope_cos ? launch_mma<DT, D, true, true>(p, stream, beside) : launch_mma<DT, D, false, true>(p, stream, beside);
  return p.rope_cos ? launch_mma<DT, D, true, false>(p, stream, beside) : launch_mma<DT, D, false, false>(p, stream, beside);
}

template <int DT, int LPR, int G>
int launch(const hipattn_bsa_params_t& p, cudaStream_t stream) {
  constexpr int D = LPR * (16 / Elem<DT>::bytes);
  const size_t smem = sizeof(float) * (size_t)kWarps * G * (D + 2);
  const int64_t grid = (int64_t)p.B * p.HKV * p.n_splits;
  HIPATTN_REQUIRE(grid > 0 && grid < 0x7fffffffLL, HIPATTN_ERR_INVALID, "decode grid of %lld blocks", (long long)grid);
  auto kern = bsa_decode_kernel<DT, LPR, G>;
  HIPATTN_CUDA_OK(allow_smem((const void*)kern, smem));
  kern<<<(unsigned)grid, kWarps * 32, smem, stream>>>(p);
  return check_launch("bsa_decode_kernel");
}

template <int DT, int LPR>
int dispatch_group(const hipattn_bsa_params_t& p, cudaStream_t stream, bool* handled) {
  *handled = true;
  switch (p.H / p.HKV) {
    case 1: return launch<DT, LPR, 1>(p, stream);
    case 2: return launch<DT, LPR, 2>(p, stream);
    case 4: return launch<DT, LPR, 4>(p, stream);
    case 8: return launch<DT, LPR, 8>(p, stream);
    default: *handled = false; return HIPATTN_OK;
  }
}

// rows of 128, 256 or 512 bytes; 16-bit rows of head dim 64 and 128 are the tensor-core kernel's
template <int DT>
int dispatch_row(const hipattn_bsa_params_t& p, cudaStream_t stream, bool* handled) {
  const int lpr = p.D * Elem<DT>::bytes / 16;
  if constexpr (DT == HIPATTN_F32) {
    if (lpr == 8) return dispatch_group<DT, 8>(p, stream, handled);
    if (lpr == 16) return dispatch_group<DT, 16>(p, stream, handled);
  }
  return lpr == 32 ? dispatch_group<DT, 32>(p, stream, handled) : HIPATTN_OK;
}

}  // namespace

// 16-bit types with at most eight query heads per KV head and head dim 64 or 128: the tensor-core kernel
bool decode_on_tensor_cores(const hipattn_bsa_params_t& p) {
  return p.TQ == 1 && p.dtype != HIPATTN_F32 && p.H / p.HKV <= 8 && (p.D == 64 || p.D == 128) && p.k.fp8_e5m2 == p.v.fp8_e5m2;
}

// Decode shapes: one query row; what the tensor-core kernel does not take, with 1 / 2 / 4 / 8 query heads per KV head and K / V
// rows of 128, 256 or 512 bytes.
int bsa_decode(const hipattn_bsa_params_t& p, cudaStream_t stream, bool* handled, bool beside) {
  *handled = false;
  if (decode_on_tensor_cores(p)) {
    *handled = true;
    if (p.dtype == HIPATTN_BF16) return p.D == 128 ? dispatch_mma<HIPATTN_BF16, 128>(p, stream, beside) : dispatch_mma<HIPATTN_BF16, 64>(p, stream, beside);
    return p.D == 128 ? dispatch_mma<HIPATTN_F16, 128>(p, stream, beside) : dispatch_mma<HIPATTN_F16, 64>(p, stream, beside);
  }
  // an fp8 cache and in-kernel RoPE: only the tensor-core kernel above; the rest is the general kernel's
  if (p.TQ != 1 || p.k.fp8_e5m2 || p.v.fp8_e5m2 || p.rope_cos) return HIPATTN_OK;
  switch (p.dtype) {
    case HIPATTN_F32: return dispatch_row<HIPATTN_F32>(p, stream, handled);
    case HIPATTN_F16: return dispatch_row<HIPATTN_F16>(p, stream, handled);
    case HIPATTN_BF16: return dispatch_row<HIPATTN_BF16>(p, stream, handled);
    default: return HIPATTN_OK;
  }
}

}  // namespace hipattn
