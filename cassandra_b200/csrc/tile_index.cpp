// The digit lists of a pattern set as tensor-core operands (tile_index.h).
#include "tile_index.h"

namespace cas {

bool append_tile(const uint8_t* const (&sq)[kTileLists], const int (&n)[kTileLists], std::vector<uint32_t>& tiles)
{
    uint32_t weight[64][kTileLists] = {};
    bool high = false;
    for (int l = 0; l < kTileLists; l++) {
        uint32_t w = 1;
        for (int i = 0; i < (sq[l] ? n[l] : 0); i++, w *= 3) {
            weight[sq[l][i]][l] += w;
            high = high || w > 255;
        }
    }
    // B fragments of the 64 x 8 matrix, low bytes then high bytes, per part
    // one 16-byte word a lane (two k-steps of two registers).  Byte b of
    // register r of step s is square 2t + s + 8b + 32r, t the lane in its
    // quad: the order in which a position's bit words give the A fragments
    // with one shift and one mask per register.
    const size_t base = tiles.size();
    tiles.resize(base + kTileWords);
    for (int part = 0; part < 2; part++)
        for (int lane = 0; lane < 32; lane++)
            for (int s = 0; s < 2; s++)
                for (int r = 0; r < 2; r++) {
                    const int t = lane & 3, l = lane >> 2;
                    uint32_t word = 0;
                    for (int b = 0; b < 4; b++)
                        word |= ((weight[2 * t + s + 8 * b + 32 * r][l] >> (8 * part)) & 255u) << (8 * b);
                    tiles[base + part * 128 + lane * 4 + s * 2 + r] = word;
                }
    return high;
}

TileSet build_tiles(const PatternSet& ps)
{
    TileSet ts;
    for (const Instance& in : ps.instances)
        if (in.n0 > kTileSquares || in.n1 > kTileSquares || in.n2 > kTileSquares) return ts;
    ts.chunk_unit = {0};
    ts.chunk_tile = {0};
    int tiles = 0;  // of all chunks so far
    size_t s0 = 0;
    for (size_t p = 0; p < ps.indexers.size(); p++) {
        const int slots = ps.indexers[p].order;
        if (slots > kTileLists || s0 + slots > ps.instances.size()) return ts;
        const Instance& in = ps.instances[s0];
        const bool pair = in.kind == kPair || in.kind == kDiagPair;
        if (pair && slots > kTileLists / 2) return ts;
        const int need = in.kind == kDiagPair ? 2 : 1;
        if (tiles + need - ts.chunk_tile.back() > kChunkTiles) {
            ts.chunk_unit.push_back(static_cast<int32_t>(ts.units.size()));
            ts.chunk_tile.push_back(tiles);
        }
        IndexUnit u{};
        u.kind = in.kind;
        u.slots = static_cast<uint8_t>(slots);
        u.tile0 = static_cast<uint16_t>(tiles - ts.chunk_tile.back());
        u.slot0 = static_cast<uint32_t>(s0);
        u.offset = in.offset;
        u.half_size = in.half_size;
        u.diag_size = in.diag_size;
        u.table_offset = in.table_offset;
        const uint8_t* sq[kTileLists] = {};
        const uint8_t* dg[kTileLists] = {};
        int n[kTileLists] = {}, nd[kTileLists] = {};
        for (int j = 0; j < slots; j++) {
            const Instance& ij = ps.instances[s0 + j];
            if (pair) {
                sq[2 * j] = ij.sq[0], n[2 * j] = ij.n0;
                sq[2 * j + 1] = ij.sq[1], n[2 * j + 1] = ij.n1;
                dg[2 * j] = ij.sq[2], nd[2 * j] = ij.n2;
            } else {
                sq[j] = ij.sq[0], n[j] = ij.n0;
            }
        }
        u.high[0] = append_tile(sq, n, ts.tiles);
        if (need == 2) u.high[1] = append_tile(dg, nd, ts.tiles);
        tiles += need;
        s0 += slots;
        ts.units.push_back(u);
    }
    ts.chunk_unit.push_back(static_cast<int32_t>(ts.units.size()));
    ts.chunk_tile.push_back(tiles);
    ts.usable = true;
    return ts;
}

}  // namespace cas
