// Order of the V-build's rows over symmetric Cholesky vectors.
//
// Rows (i, j) and (j, i) of symmetric vectors are the same sums, so only the
// 8 x 8 blocks (I <= J) of the n x n rows are cut and multiplied, in the order
// J (J + 1) / 2 + I, and a result is written to both places (an entry of its
// own would have the same bits).  Whether the vectors are symmetric is seen on
// the device (*asym == 0); otherwise the rows are the n^2 as they come.
// Blocks of 8 keep the mirrored writes at whole 32-byte sectors (16 bytes of
// bf16) and cost n = 61 2304 rows of 3721, n = 200 20800 of 40000.
#pragma once

namespace afq {

struct SymRows {
    const int* asym;  // null: rows as they come
    int n, r0;        // orbitals; first row of this chunk (rows as they come: added to their place)
};
__host__ __device__ __forceinline__ int sym_total(int n) { return ((n + 7) / 8) * ((n + 7) / 8 + 1) * 32; }
__device__ __forceinline__ bool sym_on(const SymRows& y) { return y.asym && *y.asym == 0; }
// rows of the chunk, of `rows` as they come
__device__ __forceinline__ int sym_rows(const SymRows& y, bool on, int rows) {
    return on ? max(0, min(rows, sym_total(y.n) - y.r0)) : rows;
}
// block b is (I, J)
__device__ __forceinline__ void sym_block(int b, int& I, int& J) {
    J = (int)((sqrtf(8.f * b + 1.f) - 1.f) * 0.5f);
    if (J * (J + 1) / 2 > b) --J;
    if ((J + 1) * (J + 2) / 2 <= b) ++J;
    I = b - J * (J + 1) / 2;
}
// entry (i, j) of row r; false: a block's part past n
__device__ __forceinline__ bool sym_at(const SymRows& y, int r, int& i, int& j) {
    int I, J;
    sym_block((r + y.r0) >> 6, I, J);
    i = 8 * I + ((r >> 3) & 7);  // r0 is a multiple of 64
    j = 8 * J + (r & 7);
    return i < y.n && j < y.n;
}

}  // namespace afq
