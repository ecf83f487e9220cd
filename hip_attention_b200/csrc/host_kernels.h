// Functions of libhipattn_sm100.so that only the package's own host path calls (host.cpp).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/hipattn.h"

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
int multi_copy(const CopyList& list, cudaStream_t stream, bool early = false);

// hipattn_bsa_attention; beside: the launch before this one on the stream is a multi_copy with `early` whose outputs the attention does
// not read, and the two may run side by side (decode on the tensor cores; other kernels wait for the copies as usual).
int bsa_attention(const hipattn_bsa_params_t* p, cudaStream_t stream, bool beside);

// Largest query position of every batch element, clamped to [0, 2^30): q_pos [B, TQ], or pos0 + TQ - 1 when q_pos is null.
struct QueryPositions {
  const int64_t* q_pos;
  int64_t stride_b, stride_t, pos0;
  int B, TQ;
};
int last_positions(const QueryPositions& q, int32_t* last_pos, cudaStream_t stream);

// The rows of two fp32 cos / sin tables that a call can touch, converted to the 16-bit element type: rows up to the larger of
// `floor` and the largest query position; dst [2][rows][cols].
struct RopeTables {
  const float *cos, *sin;
  int64_t row_stride;
  int rows, cols, dtype, floor;
  QueryPositions q;         // few positions: read by every block
  const int32_t* last_pos;  // [q.B] when given: read instead of the positions
  void* dst;
};
int convert_rope_tables(const RopeTables& t, cudaStream_t stream);

// rows[i] of table [table_rows, width] -> dst [n, width], only the first lens[i] entries of a row when lens is given; a row
// outside the table reads row 0 and sets HIPATTN_STATUS_PAGE_RANGE
int gather_table(const void* table, int64_t table_rows, int64_t row_stride, uint32_t* status, int entry_bytes, const void* rows, int rows_i64,
                 const void* lens, int lens_i64, int n, int width, void* dst, cudaStream_t stream);

// hipattn_scan_prepare_keys[_rope] for live tokens only: those at most `reach` behind last_pos[b]
int scan_prepare_keys(const hipattn_tokens_t& k, int dtype, int D, int B, int T, int HKV, float k_scale, float* key_abs, void* k_scaled,
                      uint32_t* status, cudaStream_t stream, const void* rope_cos, const void* rope_sin, int64_t rope_stride, int rope_rows,
                      int rope_position, const int32_t* last_pos, int reach);
int validate_tokens(const hipattn_tokens_t& t, int elem_bytes, int D, const char* name);
// hipattn_merge_partials into rows of `rows_per_group`, the groups group_stride apart
int merge_partials(const float* part_o, const float* part_lse, int64_t rows, int n_parts, int D, int dtype, void* out, int64_t out_stride,
                   float* lse_out, int64_t rows_per_group, int64_t group_stride, cudaStream_t stream);
// Log-sum-exp merge of shard outputs in the element type: outs [parts, rows, D], lses [parts, rows] base-2 -> out [rows, D]
int merge_shards(const void* outs, const float* lses, int64_t rows, int parts, int D, int dtype, void* out, cudaStream_t stream);
// Sets *out_of_order (zeroed by the caller) where the first ks[n][d] of the K entries of a row of indices [N, BDST, K] do not ascend.
int check_order(const int64_t* indices, int64_t stride_n, int64_t stride_d, const int64_t* ks, int64_t ks_stride_n, int64_t ks_stride_d, int N, int BDST,
                int K, int32_t* out_of_order, cudaStream_t stream);
int zero_memory(void* ptr, int64_t bytes, cudaStream_t stream);

// hipattn_select_stage that also writes the next stage's bounds as int64 (either pointer may be null)
int select_stage(const int32_t* score_max, const int32_t* left, int64_t rows, int32_t n, int32_t k_keep, int32_t sink, int32_t c_prev,
                 int32_t c_next, int32_t* next_left, int32_t* next_right, int32_t* next_score_max, int64_t* next_left64,
                 int64_t* next_right64, cudaStream_t stream);

// The scan stage for a list that select_stage has made, from whole chunks of c_prev tokens on the grid from `sink`, each at most once in
// a row (few pooled rows, see scan_key_tiles.cu).  scratch: device memory of scan_key_tiles_scratch bytes, at most 128 MB
// or what one query block needs; 0 bytes where the stage is hipattn_scan_stage's.
int64_t scan_key_tiles_scratch(const hipattn_scan_params_t& p, int sink, int c_prev);
int scan_key_tiles(const hipattn_scan_params_t& p, int sink, int c_prev, void* scratch, cudaStream_t stream);

}  // namespace hipattn
