// Block-sparse attention, prefill, fp32 (head dims 64 and 128): fp32 arithmetic in register tiles on the CUDA cores.
//
// A CTA of 128 threads owns 64 query rows of one head and walks its key list in tiles of 64 keys; a thread owns 8 rows x 4
// keys of S = Q K^T and 8 rows x D / 16 columns of O += P V, so that a float4 read from shared memory feeds 16 to 32
// multiply-adds and the FMA pipes, not the reads, set the pace (the general kernel's tile of 2 x 4 is bound by the reads).
// Both products use the two-wide fma: S over pairs of head-dim elements, O over pairs of rows.
// K and V have one buffer each: while S is computed the tile's V arrives, while O is updated the next tile's K does.  That
// keeps the CTA at 113 KB for D 128: two on an SM, each hiding the copies and the softmax of the other. (D 64 would fit three
// times, but not its registers: 228 us with spills, 222 with two.)
// The rows of P belong to one half-warp from the softmax to the second product: no CTA barrier between them.
// 8 heads x 4096 queries, up to 895 keys a row, D 64: 412 us with the general kernel, 222 us here; its multiply-adds alone take 104.
#include "bsa_common.cuh"

namespace hipattn {
namespace {

constexpr int kRows = 64, kKeys = 64, kThr = 128;
constexpr float kLog2e = 1.4426950408889634f;
constexpr int kNoPos = -0x40000000;   // position of a row beyond the tile: admits nothing

template <int D>
constexpr int fp32_smem_bytes() { return (kRows * D + 2 * kKeys * D + kKeys * kRows) * 4; }

template <int D>
__global__ void __launch_bounds__(kThr, 2) bsa_fp32_kernel(const hipattn_bsa_params_t p, int n_sub) {
  constexpr int PC = D / 4;      // 16-byte pieces of a row
  constexpr int RPI = 32 / PC;   // rows a warp copies per instruction: 2 or 1
  constexpr int NQ = D / 64;     // float4 columns of O per thread
  extern __shared__ __align__(16) float sm[];
  float* Qs = sm;                // [64][D], piece ^ (row / 8 & 1)
  float* Ks = Qs + kRows * D;    // [64][D], piece ^ (key & 7)
  float* Vs = Ks + kKeys * D;    // [64][D]
  float* Ps = Vs + kKeys * D;    // [key][64 rows], row quad ^ (key & 7)
  __shared__ int s_tpos[2][kKeys], s_all[2][4], s_rowpos[kRows], s_mm[4];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, tx = lane & 15, ty = tid >> 4;
  const int NBLK = cdiv(p.TQ, p.block_size_q);
  int64_t bid = blockIdx.x;
  const int split = (int)(bid % p.n_splits); bid /= p.n_splits;
  const int sub = (int)(bid % n_sub); bid /= n_sub;
  const int h = (int)(bid % p.H); bid /= p.H;
  const int b = (int)(bid % p.B); bid /= p.B;
  const int d = NBLK - 1 - (int)bid;       // under a causal mask the last blocks have the longest lists: they start first
  const int hkv = h / (p.H / p.HKV);
  const int blk_t0 = d * p.block_size_q;
  const int blk_rows = min(p.block_size_q, p.TQ - blk_t0);
  const int n_rows = min(kRows, blk_rows - sub * kRows);
  if (n_rows <= 0) return;

  // smallest / largest position of the attention block and of the tile's rows
  if (tid < 4) s_mm[tid] = tid & 1 ? -1 : 0x7fffffff;
  __syncthreads();
  for (int i = tid; i < blk_rows; i += kThr) {
    const long long x = p.pos[(int64_t)b * p.pos_stride_b + (int64_t)(blk_t0 + i) * p.pos_stride_t];
    const int v = (int)(x > 0x7ffffff0LL ? 0x7ffffff0LL : (x < 0 ? 0 : x));
    atomicMin(&s_mm[0], v);
    atomicMax(&s_mm[1], v);
    const int r = i - sub * kRows;
    if (r >= 0 && r < kRows) {
      s_rowpos[r] = v;
      atomicMin(&s_mm[2], v);
      atomicMax(&s_mm[3], v);
    }
  }
  for (int r = n_rows + tid; r < kRows; r += kThr) s_rowpos[r] = kNoPos;
  for (int i = tid; i < kRows * PC; i += kThr) {
    const int r = i / PC, pc = i % PC;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < n_rows)
      v = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.q) + (int64_t)b * p.q_stride_b +
                                           (int64_t)(blk_t0 + sub * kRows + r) * p.q_stride_t + (int64_t)h * p.q_stride_h + pc * 4);
    *reinterpret_cast<float4*>(Qs + r * D + (pc ^ ((r >> 3) & 1)) * 4) = v;
  }
  __syncthreads();
  const int rmin = s_mm[2], rmax = s_mm[3];
  KeyList kl = make_key_list(p, b, h, d, s_mm[0], s_mm[1]);
  if (lists_ascend(p)) trim_selected(kl, rmax, p.window);
  const int far_end = kl.n_sink + kl.n_sel;   // entries from here on are the window's
  const int per = cdiv(cdiv(kl.total, p.n_splits), kKeys) * kKeys;
  const int j_begin = split * per, j_end = min(kl.total, j_begin + per);

  // A warp copies keys 16 * warp .. + 15 of a tile: lane l < 16 holds the address of the K row of key l, lane l + 16 that of
  // its V row, null when no row of the tile can admit the key.
  const char* row_ptr = nullptr;
  auto find_rows = [&](int j0, int buf) {
    const int kk = warp * 16 + tx, j = j0 + kk;
    bool w = false;
    const int t = j < j_end ? key_position(kl, j, &w) : -1;
    row_ptr = t < 0 ? nullptr : token_row(lane < 16 ? p.k : p.v, b, t, hkv, 4, p.status);
    const bool all = t >= 0 && (w ? t > rmax - p.window && t <= rmin : t <= rmin - p.window);
    if (lane < 16) s_tpos[buf][kk] = t;
    const bool warp_all = __all_sync(0xffffffffu, all);
    if (lane == 0) s_all[buf][warp] = warp_all;
  };
  auto copy_rows = [&](float* dst, int first_lane, bool swizzle) {
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(dst + warp * 16 * D);
#pragma unroll
    for (int i = 0; i < 16 / RPI; ++i) {
      const int r = i * RPI + lane / PC, pc = lane % PC;
      const char* src = reinterpret_cast<const char*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(row_ptr), first_lane + r));
      cp_async16_zfill(base + (r * D + (swizzle ? pc ^ (r & 7) : pc) * 4) * 4, src ? src + pc * 16 : reinterpret_cast<const char*>(p.q), src != nullptr);
    }
    cp_async_commit();
  };

  float m_run[8], l_run[8];
  unsigned long long acc[4][NQ * 4];   // pairs of rows x columns
#pragma unroll
  for (int r = 0; r < 8; ++r) { m_run[r] = -INFINITY; l_run[r] = 0.f; }
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < NQ * 4; ++c) acc[r][c] = 0ull;
  const float cap = p.logit_softcap;
  const float* q_even = Qs + ty * 8 * D + (ty & 1) * 4;   // piece e of a row lies at e ^ (ty & 1)
  const float* q_odd = Qs + ty * 8 * D - (ty & 1) * 4;

  int buf = 0;
  if (j_begin < j_end) {
    find_rows(j_begin, 0);
    copy_rows(Ks, 0, true);
  }
  for (int j0 = j_begin; j0 < j_end; j0 += kKeys, buf ^= 1) {
    cp_async_wait<0>();
    __syncthreads();              // K has arrived, V has been consumed
    copy_rows(Vs, 16, false);
    unsigned long long s2[8][4];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) s2[r][c] = 0ull;
#pragma unroll 4
    for (int e = 0; e < PC; ++e) {
      ulonglong2 kv[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) kv[c] = *reinterpret_cast<const ulonglong2*>(Ks + (tx + 16 * c) * D + (e ^ (tx & 7)) * 4);
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const ulonglong2 qv = *reinterpret_cast<const ulonglong2*>((e & 1 ? q_odd : q_even) + r * D + e * 4);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          s2[r][c] = fma_f32x2(qv.x, kv[c].x, s2[r][c]);
          s2[r][c] = fma_f32x2(qv.y, kv[c].y, s2[r][c]);
        }
      }
    }
    // mask and online softmax (base 2); the row sums stay per thread until the end
    const bool all = (s_all[buf][0] & s_all[buf][1] & s_all[buf][2] & s_all[buf][3]) != 0;
    float s[8][4];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float lo, hi;
        f32x2_split(s2[r][c], lo, hi);
        s[r][c] = lo + hi;
        if (cap > 0.f) s[r][c] = tanhf(s[r][c] / cap) * cap;
        s[r][c] *= kLog2e;
      }
    if (!all) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int t = s_tpos[buf][tx + 16 * c];
        const bool w = j0 + tx + 16 * c >= far_end;
#pragma unroll
        for (int r = 0; r < 8; ++r)
          if (!admits(s_rowpos[ty * 8 + r], t, w, p.window)) s[r][c] = -INFINITY;
      }
    }
    float alpha[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      float mx = fmaxf(fmaxf(s[r][0], s[r][1]), fmaxf(s[r][2], s[r][3]));
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      const float m_new = fmaxf(m_run[r], mx), base = m_new > -INFINITY ? m_new : 0.f;
      alpha[r] = exp2f(m_run[r] - base);
      m_run[r] = m_new;
#pragma unroll
      for (int c = 0; c < 4; ++c) s[r][c] = exp2f(s[r][c] - base);
      l_run[r] = l_run[r] * alpha[r] + ((s[r][0] + s[r][1]) + (s[r][2] + s[r][3]));
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const unsigned long long a2 = f32x2(alpha[2 * r], alpha[2 * r + 1]);
#pragma unroll
      for (int c = 0; c < NQ * 4; ++c) acc[r][c] = mul_f32x2(acc[r][c], a2);
    }
    __syncwarp();                 // the half-warp has read its rows of the previous P
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      float* pk = Ps + (tx + 16 * c) * kRows;
      *reinterpret_cast<float4*>(pk + ((2 * ty) ^ (tx & 7)) * 4) = make_float4(s[0][c], s[1][c], s[2][c], s[3][c]);
      *reinterpret_cast<float4*>(pk + ((2 * ty + 1) ^ (tx & 7)) * 4) = make_float4(s[4][c], s[5][c], s[6][c], s[7][c]);
    }
    if (j0 + kKeys < j_end) find_rows(j0 + kKeys, buf ^ 1);
    cp_async_wait<0>();
    __syncthreads();              // V has arrived, K has been consumed
    if (j0 + kKeys < j_end) copy_rows(Ks, 0, true);
#pragma unroll 8
    for (int k = 0; k < kKeys; ++k) {
      const ulonglong2 pa = *reinterpret_cast<const ulonglong2*>(Ps + k * kRows + ((2 * ty) ^ (k & 7)) * 4);
      const ulonglong2 pb = *reinterpret_cast<const ulonglong2*>(Ps + k * kRows + ((2 * ty + 1) ^ (k & 7)) * 4);
#pragma unroll
      for (int n = 0; n < NQ; ++n) {
        const float4 v = *reinterpret_cast<const float4*>(Vs + k * D + (tx + 16 * n) * 4);
        const unsigned long long v2[4] = {f32x2(v.x, v.x), f32x2(v.y, v.y), f32x2(v.z, v.z), f32x2(v.w, v.w)};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          acc[0][n * 4 + c] = fma_f32x2(pa.x, v2[c], acc[0][n * 4 + c]);
          acc[1][n * 4 + c] = fma_f32x2(pa.y, v2[c], acc[1][n * 4 + c]);
          acc[2][n * 4 + c] = fma_f32x2(pb.x, v2[c], acc[2][n * 4 + c]);
          acc[3][n * 4 + c] = fma_f32x2(pb.y, v2[c], acc[3][n * 4 + c]);
        }
      }
    }
  }

#pragma unroll
  for (int r = 0; r < 8; ++r) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], o);
    const int row = ty * 8 + r;
    if (row >= n_rows) continue;
    const int ti = blk_t0 + sub * kRows + row;
    const float inv = l_run[r] > 0.f ? 1.f / l_run[r] : 0.f;
    const float lse = l_run[r] > 0.f ? m_run[r] + log2f(l_run[r]) : -INFINITY;
    const int64_t o_row = ((int64_t)b * p.TQ + ti) * p.H + h;
    float* op;
    if (p.n_splits > 1) {
      op = p.part_o + (o_row * p.n_splits + split) * D;
      if (tx == 0) p.part_lse[o_row * p.n_splits + split] = lse;
    } else {
      op = reinterpret_cast<float*>(p.out) + (int64_t)b * p.o_stride_b + (int64_t)ti * p.o_stride_t + (int64_t)h * p.o_stride_h;
      if (p.lse_out && tx == 0) p.lse_out[o_row] = lse;
    }
#pragma unroll
    for (int c = 0; c < NQ * 4; ++c) {
      float lo, hi;
      f32x2_split(acc[r >> 1][c], lo, hi);
      op[(tx + 16 * (c >> 2)) * 4 + (c & 3)] = (r & 1 ? hi : lo) * inv;
    }
  }
}

template <int D>
int launch(const hipattn_bsa_params_t& p, cudaStream_t stream) {
  const int n_sub = cdiv(p.block_size_q, kRows);
  const int64_t grid = (int64_t)p.B * p.H * cdiv(p.TQ, p.block_size_q) * n_sub * p.n_splits;
  HIPATTN_REQUIRE(grid > 0 && grid < 0x7fffffffLL, HIPATTN_ERR_INVALID, "attention grid of %lld blocks", (long long)grid);
  auto kern = bsa_fp32_kernel<D>;
  HIPATTN_CUDA_OK(allow_smem((const void*)kern, fp32_smem_bytes<D>()));
  kern<<<(unsigned)grid, kThr, fp32_smem_bytes<D>(), stream>>>(p, n_sub);
  return check_launch("bsa_fp32_kernel");
}

}  // namespace

// Takes fp32 blocks of more than 16 rows (below, most of a 64-row tile would be padding) without in-kernel RoPE.
int bsa_fp32(const hipattn_bsa_params_t& p, cudaStream_t stream, bool* handled) {
  *handled = p.dtype == HIPATTN_F32 && (p.D == 64 || p.D == 128) && (p.TQ < p.block_size_q ? p.TQ : p.block_size_q) > 16 && !p.rope_cos;
  if (!*handled) return HIPATTN_OK;
  return p.D == 64 ? launch<64>(p, stream) : launch<128>(p, stream);
}

}  // namespace hipattn
