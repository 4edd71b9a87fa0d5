// Host-side helpers shared by the .cu files (defined in gemm.cu).
#pragma once
#include <cuda.h>
#include <stdint.h>
namespace aeris {
// 2-D bf16 map with 128-byte swizzle: `inner` contiguous elements, `rows` rows of pitch `ld` elements.
int make_tmap_2d_bf16(CUtensorMap* out, const void* base, uint64_t inner, uint64_t rows, uint64_t ld,
                      uint32_t box_inner, uint32_t box_rows);
// The same with the 64-byte swizzle, for boxes of 32 columns.
int make_tmap_2d_sw64_bf16(CUtensorMap* out, const void* base, uint64_t inner, uint64_t rows, uint64_t ld,
                           uint32_t box_inner, uint32_t box_rows);
// Heads of window-major token rows, 128-byte swizzle: dims {d, heads, tokens, windows} of a [windows * tokens, ld] tensor
// whose first head starts at `base`; box {64, 1, box_rows, 1}. Channels past d, tokens past the window's end: zeros.
int make_tmap_heads_bf16(CUtensorMap* out, const void* base, int d, int heads, int tokens, int windows, uint64_t ld,
                         uint32_t box_rows);
// The same dims with box {32, 1, box_rows, 1} and the 64-byte swizzle: for tiled stores of 32 columns.
int make_tmap_heads32_bf16(CUtensorMap* out, const void* base, int d, int heads, int tokens, int windows, uint64_t ld,
                           uint32_t box_rows);
int num_sms();
// Slices of an accumulating product's reduction over `kb_total` blocks of 64: see gemm.cu.
int choose_k_splits(int tiles, int kb_total, int units, int most, int want);
// aeris_gemm_bf16 (api.h) with gate rows of pitch `ld_gate`.
int gemm_one_cta(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc, int a_mn, int b_mn,
                 int epi, const void* resid, int ldr, const float* gate, int rows_per_gate, int ld_gate, void* aux,
                 int ld_aux, int swiglu_f, int k_splits, int bn, int* status, void* stream);
}  // namespace aeris
