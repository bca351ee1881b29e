// Tensor-core scoring of wide windows (dense.cu): declarations.
#pragma once
#include "hfx_internal.h"
#include "batched.h"

namespace hfx {

// A block is one from this many pairs per candidate of its union on (dense.cu).
constexpr int32_t kDenseMinPairs = 32;
constexpr int kDenseSpectra = 128;  // spectra per block: the rows of one MMA
constexpr int kDenseQueue = 16;     // queued candidates per spectrum

// A run of up to 128 spectra of one class, neighbours in the planned order.
struct DenseBlock {
    uint32_t pos0, count;  // members: perm[pos0 .. pos0 + count)
    uint32_t lo, hi;       // union of their candidate windows
    int32_t maxlen, charges;
    uint32_t chunk;        // candidates per work item
    uint32_t tile;         // index of its operand tile
    uint32_t ladder;       // prefixes of its longest candidate (k_dense_ladders)
};

struct DenseWs {
    DenseBlock *blocks;    // [cap_blocks]
    uint32_t *item_off;    // [cap_blocks + 1]: first work item of each block (blocks that are not dense have none)
    uint32_t *tile_block;  // [cap_blocks]: block of each operand tile
    uint32_t *n_tiles;     // [1]
    uint32_t *total_items; // [1]
    uint32_t *counter;     // [1] work-stealing cursor
    unsigned long long *best;  // [nspec][32] each spectrum's best candidates so far, descending: score order << 32 | ~position
    unsigned long long *left;  // [items][128][kDenseQueue] candidates an item did not merge into it (0: none)
    uint32_t *lock;        // [nspec] of that list
    unsigned long long *kth;  // [nspec] its K-th entry (0: none yet)
    const uint32_t *hold;  // failure test: not 0: the first spectrum's lock starts held by nobody
    int32_t cap_blocks;
};

// Blocks of nspec spectra (every class may end in a partial one).
constexpr int32_t dense_blocks(int32_t nspec) { return nspec / kDenseSpectra + 13; }
// 128-bin chunks of a row, and the bytes of one operand tile.
constexpr int64_t dense_chunks(int64_t stride) { return (stride + 127) / 128; }
constexpr size_t dense_tile_bytes(int64_t stride, int pieces) {
    return (size_t)dense_chunks(stride) * pieces * kDenseSpectra * 128;
}

}  // namespace hfx

// 8-bit pieces a row value is split into for a row precision (0 FP32, 1 BF16, 2 FP16).
int hfx_dense_pieces(int elem_kind);
// Marks the blocks whose windows overlap enough (their groups get no work
// items of their own) and cuts them into items; between k_groups and the scan
// of the groups' items.
int hfx_dense_plan(const hfx::SpecMeta *meta, int32_t nspec, const uint32_t *wb, const uint32_t *we, int32_t G,
                   const uint32_t *bucket_end, const hfx::BatchedWs &ws, uint32_t *nchunks, const hfx::DenseWs &dw,
                   cudaStream_t st);
int hfx_dense_pack(const float *rows, int64_t stride, const hfx::BatchedWs &ws, const hfx::DenseWs &dw,
                   uint32_t cap_tiles, int pieces, uint8_t *tiles, uint32_t *err, cudaStream_t st);
int hfx_dense_score(const uint16_t *lists, uint64_t list_total, const uint32_t *lstart, uint64_t total10,
                    const uint16_t *list_len, uint32_t num_pep, const uint8_t *tiles, uint32_t cap_tiles,
                    int64_t stride, int pieces, const uint32_t *wb, const uint32_t *we, const hfx::BatchedWs &ws,
                    const hfx::DenseWs &dw, int32_t K, unsigned long long *stats, uint32_t *err, cudaStream_t st);
// FP32 searches, after the rescoring: of each spectrum of a dense block, whether
// its out_s[topn] certainly hold its best candidates (dense.cu).  open_meta: meta
// with a status other than 0 for every spectrum that needs nothing more;
// *n_open: how many do.
int hfx_dense_prove(const hfx::DevDB &db, const hfx::SpecMeta *meta, const hfx::BatchedWs &ws, const hfx::DenseWs &dw,
                    const uint32_t *wb, const uint32_t *we, const float *rows, int64_t stride, const float *kept_s,
                    const uint64_t *kept_k, int32_t nspec, int32_t topn, const float *out_s, const uint64_t *out_k,
                    hfx::SpecMeta *open_meta, uint32_t *n_open, cudaStream_t st);
// Their results from a plan of the open spectra alone into the search's outputs.
int hfx_dense_close(const hfx::SpecMeta *open_meta, const float *in_s, const uint64_t *in_k, int32_t nspec,
                    int32_t topn, const uint32_t *idx_sorted, float *out_s, uint64_t *out_k, uint32_t *out_pep,
                    cudaStream_t st);
