// C ABI of the row compaction in front of a wide output layer's backward (see sparse_rows.cu).
#pragma once
#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

// dy [rows, cols] and x [rows, x_cols], 16-bit, rows ld / x_ld elements apart (multiples of 8, 16-byte aligned bases).  A row
// counts unless every element of dy's is +0 and every element of x's is finite.  ctl[0]: how many rows count; ctl[1]: whether
// they are to be gathered (some, and with a row of zeros behind them no more than `room`).  live: a byte per row; idx: `room`
// row numbers in order; pos: for each row its place among them, or -1.  `room` is a multiple of 64.
int rb_rows_plan(const void* dy, long long ld, const void* x, long long x_ld, int rows, int cols, int x_cols, int room,
                 uint8_t* live, int32_t* idx, int32_t* pos, int32_t* ctl, int dtype, void* stream);
// The rows that count, in order, to dy_out [room, cols] and x_out [room, x_cols], with rows of zeros behind them up to the next
// multiple of 64 (one at least); as many rows of dx32 [room, x_cols], and one more, are cleared (null: none)
int rb_rows_gather(const void* dy, long long ld, const void* x, long long x_ld, int cols, int x_cols, const int32_t* idx,
                   const int32_t* ctl, void* dy_out, void* x_out, float* dx32, void* stream);
// dx [rows, x_cols] (16-bit): each row's place in dx32, or the row behind the last for those that were left out.  _parts: the
// sum of ctl[2] rows, ctl[3] rows apart, in that order (RB_GEMM_ROWS_M)
int rb_rows_scatter_parts(const float* dx32, void* dx, int rows, int x_cols, const int32_t* pos, const int32_t* ctl, int dtype,
                          void* stream);
int rb_rows_scatter(const float* dx32, void* dx, int rows, int x_cols, const int32_t* pos, const int32_t* ctl, int dtype,
                    void* stream);

#ifdef __cplusplus
}
#endif
