// Records of the tiled upper-triangle layout shared by the build (build_h.cu) and tiles.cu.
#pragma once
#include <cstdint>

namespace risq {

// Cursor of a bin whose tile is too sparse to stage: its pairs go to the panel's leftovers.
constexpr unsigned long long LEFT_BIN = 1ull << 63;

// One non-empty bin (block of 2^kb rows x window) of a dense tile.
struct TileBlock {
    int64_t bin;       // its fill cursor
    int64_t el;        // first element of its candidates, over the handle's panels
    int64_t group;     // first group of 32 slots, in its chunk's arrays
    int64_t vec;       // first pair of elements
    int32_t n_groups;
    int32_t len;       // stored pairs
    int32_t row;       // first row
    int32_t chunk;
    float row_bound;   // largest row / column sum of |H| in the bin
    float col_bound;
};

// A sigma work unit: the row blocks [lo, hi) (at most 32) of a tile, or, with tile < 0, the
// leftovers [lo, hi) of a panel (FP64 values: the leftovers of its rows [lo, hi)).
struct SigmaUnit {
    int32_t tile, panel, lo, hi, chunk;
};

// The element arrays of one chunk of panels.
struct TileChunk {
    int64_t* grp_off = nullptr;   // first pair of elements of each group
    uint32_t* slots = nullptr;    // 32 per group: row in panel | elements << 16
    uint16_t* col = nullptr;      // column in window
    void* val = nullptr;          // FP64 or FP32 values
    float* lo = nullptr;          // FP32 remainders (MIXED)
};

// What a panel holds, by candidates: pairs in dense tiles and left over, dense tiles,
// their non-empty bins, and about the pairs of elements and groups those need.
struct PanelCount {
    long long dense, left, tiles, blocks, vecs, groups;
};

// First element, tile and bin record of a panel.
struct PanelBase {
    long long el, tile, block;
};

// Where the build's search and fill passes put what they find for the tiled layout.
struct TileOut {
    int rb = 0, cb = 0, kb = 0;
    const int64_t* bin_off = nullptr;        // first bin of each block of rows
    uint32_t* hist = nullptr;                // search: candidates per bin
    unsigned long long* cur = nullptr;       // fill: next element of every bin
    unsigned long long* left_cur = nullptr;  // fill: next leftover of every panel
    long long el0 = 0;                       // first element of the chunk being filled
    long long cap = 0, left_cap = 0;         // elements its arrays and the leftovers' hold
    uint32_t* code = nullptr;                // fill: row in panel << cb | column in window
    uint32_t* lcol = nullptr;                // leftovers: column, row in panel, values
    uint16_t* lrow = nullptr;
    float* l32 = nullptr;
    float* llo = nullptr;
};

}  // namespace risq
