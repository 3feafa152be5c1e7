// Tensor maps over bf16 matrices for copies into 128-byte-swizzled shared memory (boxes 64 entries wide); made in dense_tc.cu.
#pragma once
#include <cuda.h>

namespace b2 {

// [nb][rows][cols], rows `ld` and batch entries `bs` entries apart; boxes of 64 x box_rows. Entries past the end are read as zeros.
bool bf16_rows_map(CUtensorMap* m, const void* base, long cols, long rows, long ld, long nb, long bs, int box_rows);
// the same as [nb][cols / 64][rows][64] (cols a multiple of 64): boxes of `slices` 64-entry slices of box_rows rows; coordinates
// (0, row, slice, entry)
bool bf16_slices_map(CUtensorMap* m, const void* base, long cols, long rows, long ld, long nb, long bs, int box_rows, int slices);
// [nb][parts][rows][cols]: parts are rows * ld entries apart; boxes of 64 x box_rows of all parts; coordinates (column, row, 0, entry)
bool bf16_parts_map(CUtensorMap* m, const void* base, long cols, long rows, long ld, long nb, long bs, int parts, int box_rows);
// [rows][heads][cols]: boxes of 64 columns of box_heads heads, box_rows rows; coordinates (column, head, row)
bool bf16_heads_map(CUtensorMap* m, const void* base, long cols, long heads, long rows, int box_heads, int box_rows);

}  // namespace b2
