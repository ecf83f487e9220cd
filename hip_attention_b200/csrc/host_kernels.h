// Functions of libhipattn_sm100.so that only the package's own host path calls (host.cpp).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace hipattn {

struct BeginCall {
  int32_t* left;        // [rows, n] or null: only the scores are set (an estimator restart)
  int32_t* right;
  int32_t* score_max;   // [rows, n]
  int64_t rows, n;
  int sink, chunk, T, scan_window;
  int64_t* pos;         // [n_pos]: pos0, pos0 + 1, ...
  int64_t n_pos, pos0;
  float* consts;        // [n_const]: HIPATTN_SCORE_INIT
  int64_t n_const;
};
int begin_call(const BeginCall& c, cudaStream_t stream);

// Element types of multi_copy; integers go to integers (narrowing keeps the low bits), floats to floats.
enum { COPY_I64 = 0, COPY_I32 = 1, COPY_U32 = 2, COPY_F32 = 3, COPY_BF16 = 4, COPY_ZERO = 5 };
struct CopySeg {
  const void* src;
  void* dst;
  int64_t n0, n1, n2;
  int64_t src_s[3], dst_s[3];   // strides in elements
  int src_type, dst_type;
  int plain;                    // both sides contiguous
};
constexpr int kMaxCopies = 24;
struct CopyList {
  CopySeg seg[kMaxCopies];
  int count;
};
int multi_copy(const CopyList& list, cudaStream_t stream);

int zero_memory(void* ptr, int64_t bytes, cudaStream_t stream);

// hipattn_select_stage that also writes the next stage's bounds as int64 (either pointer may be null)
int select_stage(const int32_t* score_max, const int32_t* left, int64_t rows, int32_t n, int32_t k_keep, int32_t sink, int32_t c_prev,
                 int32_t c_next, int32_t* next_left, int32_t* next_right, int32_t* next_score_max, int64_t* next_left64,
                 int64_t* next_right64, cudaStream_t stream);

}  // namespace hipattn
