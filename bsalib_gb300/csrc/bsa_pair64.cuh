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
    int rpad;         // rows of one x in the row operand (rx, or whole tiles in a pair list)
    const int *xmap;  // pair list: A row of x (x0 = 0); null: x itself
    int test_skip1 = 0;  // tile pass + 1 whose ready signal block 0 omits (bsa_gpu_setWaitTestFP64)
    __host__ __device__ int rx() const { return qn * an; }  // rows of one x
};

// A list of products instead (point sets, bsa_list64.cu): the columns of an A row come in np blocks
// of bw (a multiple of 8, at most 32), kSlots(bw) blocks to a product tile.  Item i multiplies row tile
// items[i].x with the blocks blk[items[i].y] .. (items[i].z of them); product pair[e] of entry e goes
// to E[pair][a nm + b][j].
struct PairList {
    const int4 *items;
    const int *blk, *pair;
    int np, bw, tiles_x;  // row tiles of one x
};
__host__ __device__ inline int blocks_of(int nm) { return (nm + kTN - 1) / kTN; }
__host__ __device__ inline int block_width(int nm) { return ((nm + blocks_of(nm) - 1) / blocks_of(nm) + 7) / 8 * 8; }

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
// table) and of the row operand of nrows product rows in items tiles.  tc_prep_cols once per analysis, then
// tc_products per chunk.  err receives a nonzero code if a pipeline wait ran out of its budget.
size_t tc_col_bytes(int nr, int an, int K);
size_t tc_row_bytes(long long nrows, int K, long long items);
cudaError_t tc_prep_cols(cudaStream_t st, int nr, int an, int K, const double *A, void *cols);
cudaError_t tc_products(cudaStream_t st, const Chunk &c, int nr, const double *A, const double *Q, void *cols,
                        void *rows, int *err);

// The same for a pair list: column blocks of nr A rows, then the products of c.x1 rows (c.items items).
size_t tc_block_bytes(int nr, int nm, int K);
cudaError_t tc_prep_blocks(cudaStream_t st, int nr, int nm, int K, const double *A, void *cols);
cudaError_t tc_list_products(cudaStream_t st, const Chunk &c, const PairList &l, int nr, const double *A, const double *Q,
                             void *cols, void *rows, int *err);

}  // namespace p64
}  // namespace bsa
