// bsa_pair64.cuh -- the product chunks of the FP64 pair form (bsa_pair64.cu) and their tensor-core
// contraction (bsa_pair64_tc.cu).
#pragma once
#include <cuda_runtime.h>

#include "bsa_common.cuh"

namespace bsa {
namespace p64 {

constexpr int kTM = 128, kTN = 32;  // product tile: rows (x, a, b) by columns (y, j)

// A chunk of products sum_k Q[k][a] A(x)[k][b] A(y)[k][j], Q of qn and A of an columns (nm and nm;
// nm and 1 for the diagonal-only spectra): rows r = (x - x0) qn an + a an + b of the first rows x in
// [x0, x1), in tiles of kTM; row tile mt holds the column tiles ct0[mt] .. ct0[mt] + nct[mt] of
// c = y an + j, row-major from base[mt].
struct RowTile {
    int ct0, nct;
    long long base;   // first element in E
    long long item0;  // product tiles before this row tile
};

struct Chunk {
    int x0, x1, qn, an, K, hi, ntiles;
    long long items;
    const RowTile *rt;
    double *E;
    __host__ __device__ int rx() const { return qn * an; }  // rows of one x
};

// Row tile of a product tile.
__device__ __forceinline__ int tile_row(const Chunk &c, long long item) {
    int lo = 0, up = c.ntiles - 1;
    while (lo < up) {
        const int mid = (lo + up + 1) >> 1;
        if (c.rt[mid].item0 <= item) lo = mid; else up = mid - 1;
    }
    return lo;
}

// Tensor-core products.  tc_col_bytes / tc_row_bytes: scratch of the column operand (nr rows of the A
// table) and of the row operand of nrows product rows.  tc_prep_cols once per analysis, then
// tc_products per chunk.  err receives a nonzero code if a pipeline wait ran out of its budget.
size_t tc_col_bytes(int nr, int an, int K);
size_t tc_row_bytes(long long nrows, int K);
cudaError_t tc_prep_cols(cudaStream_t st, int nr, int an, int K, const double *A, void *cols);
cudaError_t tc_products(cudaStream_t st, const Chunk &c, int nr, const double *A, const double *Q, void *cols,
                        void *rows, int *err);

}  // namespace p64
}  // namespace bsa
