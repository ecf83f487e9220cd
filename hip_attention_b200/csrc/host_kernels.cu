// Small kernels of the host path: what a call writes before its first scan stage, and copies of several tensors in one launch.
#include "common.cuh"
#include "host_kernels.h"

namespace hipattn {
namespace {

// The initial chunk list (attention_extend.py:2027-2046), the query positions of a call that gave none (the last TQ of T)
// and the constants its stage caches show: one launch where they were five.
__global__ void begin_call_kernel(const BeginCall c) {
  const int32_t init = encode_score(HIPATTN_SCORE_INIT);
  const int64_t step = (int64_t)gridDim.x * blockDim.x, first = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t total = c.rows * c.n;
  for (int64_t i = first; i < total; i += step) {
    if (c.left) {
      const int l = c.sink + (int)(i % c.n) * c.chunk;
      c.left[i] = l;
      c.right[i] = min(l + c.chunk, c.T - c.scan_window);
    }
    c.score_max[i] = init;
  }
  for (int64_t i = first; i < c.n_pos; i += step) c.pos[i] = c.pos0 + i;
  for (int64_t i = first; i < c.n_const; i += step) c.consts[i] = HIPATTN_SCORE_INIT;
}

__device__ __forceinline__ int clamp_position(int64_t x) { return (int)(x < 0 ? 0 : (x > 0x3fffffff ? 0x3fffffff : x)); }

__global__ void last_positions_kernel(const QueryPositions q, int32_t* last_pos) {
  __shared__ int s_max;
  if (threadIdx.x == 0) s_max = 0;
  __syncthreads();
  int m = 0;
  if (q.q_pos == nullptr) m = clamp_position(q.pos0 + q.TQ - 1);
  else
    for (int i = threadIdx.x; i < q.TQ; i += blockDim.x) m = max(m, clamp_position(q.q_pos[blockIdx.x * q.stride_b + i * q.stride_t]));
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) atomicMax(&s_max, m);
  __syncthreads();
  if (threadIdx.x == 0) last_pos[blockIdx.x] = s_max;
}

// Four elements per thread and step.  A call touches table rows up to its largest position, and only the first half of the
// columns (the tables repeat): a server's 131072-row tables cost 38 us when they were converted whole on every call.
template <int DT>
__global__ void __launch_bounds__(256) convert_rope_tables_kernel(const RopeTables t) {
  __shared__ int s_max;
  if (threadIdx.x == 0) s_max = t.floor;
  __syncthreads();
  int m = t.floor;
  if (t.last_pos) {
    for (int i = threadIdx.x; i < t.q.B; i += 256) m = max(m, t.last_pos[i]);
  } else if (t.q.q_pos == nullptr) {
    m = max(m, clamp_position(t.q.pos0 + t.q.TQ - 1));
  } else {
    for (int i = threadIdx.x; i < t.q.B * t.q.TQ; i += 256) m = max(m, clamp_position(t.q.q_pos[i / t.q.TQ * t.q.stride_b + i % t.q.TQ * t.q.stride_t]));
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) atomicMax(&s_max, m);
  __syncthreads();
  const int rows = min(t.rows, s_max + 1), q4 = t.cols / 4;
  const int64_t total = (int64_t)rows * q4, side = (int64_t)t.rows * t.cols;
  for (int64_t i = blockIdx.x * 256LL + threadIdx.x; i < total; i += gridDim.x * 256LL) {
    const int r = (int)(i / q4), c = (int)(i - (int64_t)r * q4) * 4;
#pragma unroll
    for (int sd = 0; sd < 2; ++sd) {
      const float4 v = __ldg(reinterpret_cast<const float4*>((sd ? t.sin : t.cos) + r * t.row_stride + c));
      uint16_t* dst = reinterpret_cast<uint16_t*>(t.dst) + sd * side + (int64_t)r * t.cols + c;
      *reinterpret_cast<uint2*>(dst) = make_uint2(pack2<DT>(v.x, v.y), pack2<DT>(v.z, v.w));
    }
  }
}

template <typename E>
__global__ void __launch_bounds__(256) gather_table_kernel(const E* __restrict__ table, int64_t table_rows, int64_t row_stride, uint32_t* status,
                                                           const void* rows, int rows_i64, const void* lens, int lens_i64, int width,
                                                           E* __restrict__ dst) {
  const int i = blockIdx.y;
  int64_t row = rows_i64 ? ((const int64_t*)rows)[i] : (int64_t)((const int32_t*)rows)[i];
  if (row < 0 || row >= table_rows) {
    if (threadIdx.x == 0) atomicOr(status, HIPATTN_STATUS_PAGE_RANGE);
    row = 0;
  }
  int n = width;
  if (lens) {
    const int64_t l = lens_i64 ? ((const int64_t*)lens)[i] : (int64_t)((const int32_t*)lens)[i];
    n = (int)min((int64_t)width, max(l, (int64_t)0));
  }
  const E* src = table + row * row_stride;
  E* out = dst + (int64_t)i * width;
  constexpr int V = 16 / sizeof(E);
  const bool vec = ((uintptr_t)src % 16) == 0 && ((uintptr_t)out % 16) == 0;
  const int nv = vec ? n / V : 0, first = blockIdx.x * 256 + threadIdx.x, step = gridDim.x * 256;
  for (int j = first; j < nv; j += step) reinterpret_cast<uint4*>(out)[j] = __ldg(reinterpret_cast<const uint4*>(src) + j);
  for (int j = nv * V + first; j < n; j += step) out[j] = src[j];
}

__global__ void __launch_bounds__(128) check_order_kernel(const int64_t* __restrict__ indices, int64_t stride_n, int64_t stride_d,
                                                          const int64_t* __restrict__ ks, int64_t ks_stride_n, int64_t ks_stride_d, int64_t rows,
                                                          int BDST, int K, int32_t* out_of_order) {
  for (int64_t row = blockIdx.x; row < rows; row += gridDim.x) {
    const int64_t n = row / BDST, d = row % BDST;
    const int64_t* idx = indices + n * stride_n + d * stride_d;
    const int64_t have = ks[n * ks_stride_n + d * ks_stride_d];
    const int count = (int)(have < 0 ? 0 : (have > K ? K : have));
    bool bad = false;
    for (int j = threadIdx.x + 1; j < count; j += 128) bad |= idx[j] < idx[j - 1];
    if (bad) *out_of_order = 1;
  }
}

__device__ __forceinline__ int64_t load_int(const CopySeg& s, int64_t at) {
  switch (s.src_type) {
    case COPY_I64: return ((const int64_t*)s.src)[at];
    case COPY_I32: return ((const int32_t*)s.src)[at];
    case COPY_U32: return (int64_t)((const uint32_t*)s.src)[at];
    default: return 0;   // COPY_ZERO
  }
}
__device__ __forceinline__ float load_float(const CopySeg& s, int64_t at) {
  switch (s.src_type) {
    case COPY_F32: return ((const float*)s.src)[at];
    case COPY_BF16: return __bfloat162float(((const __nv_bfloat16*)s.src)[at]);
    default: return 0.f;   // COPY_ZERO
  }
}

// EARLY: a kernel behind this one that was launched for it (hipattn::bsa_attention, beside) may begin at once.
template <bool EARLY>
__global__ void multi_copy_kernel(const CopyList list) {
  if (EARLY) asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  const CopySeg& s = list.seg[blockIdx.y];
  const int64_t total = s.n0 * s.n1 * s.n2;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    int64_t so, dof;
    if (s.plain) {
      so = dof = i;
    } else {
      const int64_t i2 = i % s.n2, r = i / s.n2, i1 = r % s.n1, i0 = r / s.n1;
      so = i0 * s.src_s[0] + i1 * s.src_s[1] + i2 * s.src_s[2];
      dof = i0 * s.dst_s[0] + i1 * s.dst_s[1] + i2 * s.dst_s[2];
    }
    switch (s.dst_type) {
      case COPY_I64: ((int64_t*)s.dst)[dof] = load_int(s, so); break;
      case COPY_I32: case COPY_U32: ((uint32_t*)s.dst)[dof] = (uint32_t)load_int(s, so); break;
      case COPY_F32: ((float*)s.dst)[dof] = load_float(s, so); break;
      case COPY_BF16: ((__nv_bfloat16*)s.dst)[dof] = __float2bfloat16_rn(load_float(s, so)); break;
    }
  }
}

}  // namespace

int begin_call(const BeginCall& c, cudaStream_t stream) {
  int64_t work = c.rows * c.n;
  if (c.n_pos > work) work = c.n_pos;
  if (c.n_const > work) work = c.n_const;
  if (work <= 0) return HIPATTN_OK;
  int64_t grid = (work + 255) / 256;
  if (grid > 148 * 8) grid = 148 * 8;
  begin_call_kernel<<<(unsigned)grid, 256, 0, stream>>>(c);
  return check_launch("begin_call_kernel");
}

int last_positions(const QueryPositions& q, int32_t* last_pos, cudaStream_t stream) {
  last_positions_kernel<<<(unsigned)q.B, q.TQ > 256 ? 1024 : 256, 0, stream>>>(q, last_pos);
  return check_launch("last_positions_kernel");
}

int convert_rope_tables(const RopeTables& t, cudaStream_t stream) {
  int64_t grid = ((int64_t)t.rows * (t.cols / 4) + 1023) / 1024;
  if (grid > 148 * 8) grid = 148 * 8;
  if (grid < 1) grid = 1;
  if (t.dtype == HIPATTN_BF16) convert_rope_tables_kernel<HIPATTN_BF16><<<(unsigned)grid, 256, 0, stream>>>(t);
  else convert_rope_tables_kernel<HIPATTN_F16><<<(unsigned)grid, 256, 0, stream>>>(t);
  return check_launch("convert_rope_tables_kernel");
}

int gather_table(const void* table, int64_t table_rows, int64_t row_stride, uint32_t* status, int entry_bytes, const void* rows, int rows_i64,
                 const void* lens, int lens_i64, int n, int width, void* dst, cudaStream_t stream) {
  if (n <= 0 || width <= 0) return HIPATTN_OK;
  int64_t gx = ((int64_t)width * entry_bytes / 16 + 255) / 256;
  const int64_t most = (148 * 8 + n - 1) / n;
  if (gx > most) gx = most;
  if (gx < 1) gx = 1;
  HIPATTN_REQUIRE(n <= 65535, HIPATTN_ERR_INVALID, "gather_table: %d rows", n);
  const dim3 grid((unsigned)gx, (unsigned)n);
  if (entry_bytes == 8)
    gather_table_kernel<int64_t><<<grid, 256, 0, stream>>>((const int64_t*)table, table_rows, row_stride, status, rows, rows_i64, lens, lens_i64, width,
                                                           (int64_t*)dst);
  else
    gather_table_kernel<int32_t><<<grid, 256, 0, stream>>>((const int32_t*)table, table_rows, row_stride, status, rows, rows_i64, lens, lens_i64, width,
                                                           (int32_t*)dst);
  return check_launch("gather_table_kernel");
}

int check_order(const int64_t* indices, int64_t stride_n, int64_t stride_d, const int64_t* ks, int64_t ks_stride_n, int64_t ks_stride_d, int N, int BDST,
                int K, int32_t* out_of_order, cudaStream_t stream) {
  const int64_t rows = (int64_t)N * BDST;
  if (rows <= 0 || K <= 1) return HIPATTN_OK;
  check_order_kernel<<<(unsigned)(rows > 148 * 16 ? 148 * 16 : rows), 128, 0, stream>>>(indices, stride_n, stride_d, ks, ks_stride_n, ks_stride_d, rows, BDST,
                                                                                        K, out_of_order);
  return check_launch("check_order_kernel");
}

int zero_memory(void* ptr, int64_t bytes, cudaStream_t stream) {
  HIPATTN_CUDA_OK(cudaMemsetAsync(ptr, 0, (size_t)bytes, stream));
  return HIPATTN_OK;
}

int multi_copy(const CopyList& list, cudaStream_t stream, bool early) {
  int64_t most = 0;
  for (int i = 0; i < list.count; ++i) {
    const CopySeg& s = list.seg[i];
    const bool to_float = s.dst_type == COPY_F32 || s.dst_type == COPY_BF16, from_float = s.src_type == COPY_F32 || s.src_type == COPY_BF16;
    HIPATTN_REQUIRE(s.dst && s.dst_type >= 0 && s.dst_type < COPY_ZERO &&
                        (s.src_type == COPY_ZERO || (s.src && s.src_type >= 0 && s.src_type < COPY_ZERO && from_float == to_float)),
                    HIPATTN_ERR_INVALID, "multi_copy: segment %d: type %d to type %d", i, s.src_type, s.dst_type);
    const int64_t t = list.seg[i].n0 * list.seg[i].n1 * list.seg[i].n2;
    if (t > most) most = t;
  }
  if (most <= 0) return HIPATTN_OK;
  int64_t grid = (most + 1023) / 1024;
  if (grid > 148 * 4) grid = 148 * 4;
  auto kern = early ? multi_copy_kernel<true> : multi_copy_kernel<false>;
  kern<<<dim3((unsigned)grid, (unsigned)list.count), 256, 0, stream>>>(list);
  return check_launch("multi_copy_kernel");
}

}  // namespace hipattn
