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

__device__ __forceinline__ int64_t load_int(const CopySeg& s, int64_t at) {
  switch (s.src_type) {
    case COPY_I64: return ((const int64_t*)s.src)[at];
    case COPY_I32: return ((const int32_t*)s.src)[at];
    case COPY_U32: return (int64_t)((const uint32_t*)s.src)[at];
    default: return 0;   // COPY_ZERO
  }
}

__global__ void multi_copy_kernel(const CopyList list) {
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
      case COPY_F32:
        ((float*)s.dst)[dof] = s.src_type == COPY_F32 ? ((const float*)s.src)[so] : __bfloat162float(((const __nv_bfloat16*)s.src)[so]);
        break;
      case COPY_BF16:
        ((__nv_bfloat16*)s.dst)[dof] = s.src_type == COPY_F32 ? __float2bfloat16_rn(((const float*)s.src)[so]) : ((const __nv_bfloat16*)s.src)[so];
        break;
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

int zero_memory(void* ptr, int64_t bytes, cudaStream_t stream) {
  HIPATTN_CUDA_OK(cudaMemsetAsync(ptr, 0, (size_t)bytes, stream));
  return HIPATTN_OK;
}

int multi_copy(const CopyList& list, cudaStream_t stream) {
  int64_t most = 0;
  for (int i = 0; i < list.count; ++i) {
    const int64_t t = list.seg[i].n0 * list.seg[i].n1 * list.seg[i].n2;
    if (t > most) most = t;
  }
  if (most <= 0) return HIPATTN_OK;
  int64_t grid = (most + 1023) / 1024;
  if (grid > 148 * 4) grid = 148 * 4;
  multi_copy_kernel<<<dim3((unsigned)grid, (unsigned)list.count), 256, 0, stream>>>(list);
  return check_launch("multi_copy_kernel");
}

}  // namespace hipattn
