// Sparse direct factorization of J = K - diag(FP): the plan (host) and its
// device driver.  K couples an unknown to its 14 mesh neighbours only, so a
// nested-dissection order leaves L with a few per cent of the dense matrix's
// entries and splits the elimination into independent subtrees.
#pragma once

#include <cstdint>
#include <vector>

namespace mp {

constexpr int ND_TILE = 64;   // unknowns of a tile column; tiles are ND_TILE x ND_TILE
constexpr int ND_LEAF = 128;  // a part this small is not cut further

// Position of entry (r, c) in a stored tile.  A tile is a sequence of 8 x 8
// blocks, block column by block column; a block's 64 values are laid out as
// the FP64 tensor-core operand reads them (mma.sync m8n8k4: lane 4r + c%4 holds
// row r, column c), the two 4-column halves side by side, so a warp's operand
// load is 512 consecutive bytes and the first k columns of a tile are one
// contiguous run.
#ifdef __CUDACC__
__host__ __device__
#endif
inline int nd_at(int r, int c) {
    return (c >> 3) * 512 + (r >> 3) * 64 + ((r & 7) * 4 + (c & 3)) * 2 + ((c >> 2) & 1);
}

// One product of a task: tile a (rows) times tile b (columns), summed over the
// columns of tile column col.
struct NdItem {
    int32_t a, b;    // tile ids; b < 0: one of the kinds below
    int32_t col;     // the tile column summed over
    int32_t kblocks; // ceil(width of col / 8)
};
constexpr int ND_DIAG_ONLY = -1;  // diagonal task: only the product of a with itself
constexpr int ND_INV = -2;        // a is the inverse of a diagonal block: the task's tile is finished with it
constexpr int ND_BEGIN = -3;      // no operands: a task's first item
constexpr int ND_ADD = -4;        // a holds a partial sum of the task's (row, col) products
constexpr int ND_ADDX = -5;       // a holds a partial sum of a diagonal task's (col, pred) products

// A task forms tile (row, col).  A diagonal task (row == col) also forms the
// tile (col, pred) of one earlier column first, when pred >= 0.  A partial
// task only sums some of another task's products, into scratch tiles (ids from
// NdPlan::ntile on; tile: the (row, col) sum, xtile: the (col, pred) sum).
struct NdTask {
    int32_t row, col, pred;
    int32_t tile, xtile;      // the tile formed; (col, pred)'s tile
    int32_t item0, item1;     // its products, in order
    int32_t ent0, ent1;       // K's entries of `tile`
    int32_t xent0, xent1;     // K's entries of `xtile`
    int16_t partial;
    int16_t rblocks, cblocks, pblocks;  // 8-row blocks in use: of row, col and pred
    int32_t pad[3];
};
static_assert(sizeof(NdTask) == 64, "NdTask layout");

// A task's products whose columns are more than ND_NEAR ranks above its own
// are ready long before the rest: from ND_SPLIT_FROM of them on they go to
// partial tasks of about ND_SPLIT products each, so that the task itself, once
// its last operands come, has few products left.
constexpr int ND_NEAR = 2, ND_SPLIT_FROM = 6, ND_SPLIT = 8;

struct NdPlan {
    int n = 0, ncol = 0, ntile = 0;
    int nscratch = 0;                // scratch tiles of partial sums
    int chain = 0;                   // tile columns on the longest elimination chain
    long long products = 0;          // 64^3 products
    std::vector<int32_t> perm;       // [ncol][64] unknown of a tile column's row, -1: padding
    std::vector<int32_t> width;      // [ncol]
    std::vector<int32_t> tile_ptr;   // [ncol + 1] column's tiles: the diagonal one, then rows ascending
    std::vector<int32_t> tile_row, tile_col;  // [ntile]
    std::vector<int32_t> row_ptr, row_tile;   // tiles left of the diagonal by row, columns ascending
    std::vector<NdTask> task;
    std::vector<NdItem> item;
    std::vector<int32_t> ent_src;    // slot of K's value
    std::vector<uint16_t> ent_at;    // nd_at position in the tile
};

// The plan of the symmetric pattern (ptr, col; diagonal included), using the
// unknowns' positions [n][3] where they differ.  slot(k) of CSR entry k is
// given by `slot`.  Returns false when a tile graph would exceed max_products
// 64^3 products (the pattern has no good order: the dense path is the better one).
bool nd_build_plan(int n, const std::vector<long long> &ptr, const std::vector<int> &col,
                   const std::vector<long long> &slot, const std::vector<double> &pos, long long max_products,
                   NdPlan &plan);

}  // namespace mp
