// Host side of the matrix form of the indexer (tile_index.cuh): the digit
// lists of a pattern set as the columns of a 64-square weight matrix, in the
// fragment order of the tensor-core instruction that multiplies positions by
// it.
#pragma once
#include <cstdint>
#include <vector>

#include "patterns.h"

namespace cas {

// Digit lists of at most this many squares fit the matrix form: the largest
// weight, 3^10 = 59049, is two bytes.
constexpr int kTileSquares = 11;
constexpr int kTileLists = 8;        // digit lists (matrix columns) of one tile
constexpr int kTileWords = 2 * 128;  // 32-bit words of one tile: 64 squares x 8 lists, low and high bytes
constexpr int kChunkTiles = 32;      // most tiles of one chunk (32 KB of shared memory)

// The slots of one pattern that are computed together, from one tile (two for
// kDiagPair).  kDirect, kTable: list j of the tile is slot j.  kPair: lists
// 2j and 2j+1 are slot j's halves.  kDiagPair: a pair tile, then a tile whose
// list 2j is slot j's diagonal.
struct IndexUnit {
    uint8_t kind;
    uint8_t slots;       // slots of the unit (1..8)
    uint8_t high[2];     // the tile has weights above 255
    uint16_t tile0;      // first tile, counted from the chunk's first
    uint32_t slot0;      // first slot (in the row)
    uint32_t offset;     // column offset of the pattern
    uint32_t half_size, diag_size, table_offset;
    uint32_t pad;
};
static_assert(sizeof(IndexUnit) == 32, "IndexUnit layout");

struct TileSet {
    bool usable = false;             // every list fits
    std::vector<IndexUnit> units;
    std::vector<int32_t> chunk_unit; // first unit of each chunk, and the end
    std::vector<int32_t> chunk_tile; // first tile of each chunk, and the end
    std::vector<uint32_t> tiles;     // kTileWords words each
    int chunks() const { return static_cast<int>(chunk_unit.size()) - 1; }
};

// One tile from up to kTileLists digit lists (null: a list of zeros).
// Returns whether any weight is above 255.
bool append_tile(const uint8_t* const (&sq)[kTileLists], const int (&n)[kTileLists], std::vector<uint32_t>& tiles);

// The units of a pattern set (usable = false when a list is too long).
TileSet build_tiles(const PatternSet& ps);

}  // namespace cas
