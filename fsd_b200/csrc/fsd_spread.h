// Which spreading kernel runs, on what tile, and the columns particles are
// binned by (host code; mobility.cu).
#pragma once

#include <math.h>

#include <algorithm>

#include "fsd_internal.h"

namespace fsd {

// Binning columns: one per (x, y) up to 160 nodes along z, else as many pieces of
// equal length at most that.  A warp ranks a column's members against one another
// and counts them once per 32 nodes, so its work grows with the square of the
// length: with whole columns of 1563 nodes and 78 members (16 x 16 x 1563,
// N = 20000) a wave-space product takes 464 us, with pieces 382.
inline int bin_pieces(int Nz) { return (Nz + 159) / 160; }
inline int bin_piece_nodes(int Nz) { return (Nz + bin_pieces(Nz) - 1) / bin_pieces(Nz); }
inline size_t bin_columns(const GridParams& g) { return (size_t)g.Nx * g.Ny * bin_pieces(g.Nz); }

enum { kSpreadBlocks = 0, kSpreadRows = 1, kSpreadFour = 2 };  // TuneChoice::spread_rows

struct SpreadChoice {
    int TX, TY, TZ;
    int form;
    bool local;  // node-particle separations are tile-relative
};

// Node-particle separations stay below (T + P) cells per axis, plus the
// tilt's x shift; below half the box they are their own minimum image.
inline bool spread_local(const GridParams& g, float xy, int TX, int TY, int TZ) {
    const float tilt = 1.0f + fabsf(xy);
    return (TX + g.P) * tilt < 0.5f * g.Nx && (TY + g.P) * tilt < 0.5f * g.Ny && (TZ + g.P) * tilt < 0.5f * g.Nz;
}

inline int spread_tiles(const GridParams& g, int TX, int TY, int TZ) {
    return ((g.Nx + TX - 1) / TX) * ((g.Ny + TY - 1) / TY) * ((g.Nz + TZ - 1) / TZ);
}

inline SpreadChoice spread_choice(const GridParams& g, float xy, const TuneChoice& tune) {
    SpreadChoice c;
    bool four = false, rows = false;
    // A tuned choice was timed at some tilt, maybe another handle's: four nodes
    // per lane are taken from it only while separations are tile-relative.
    if (tune.set && tune.TX > 0 &&
        (tune.spread_rows != kSpreadFour || spread_local(g, xy, tune.TX, tune.TY, tune.TZ))) {
        c.TX = tune.TX;
        c.TY = tune.TY;
        c.TZ = tune.TZ;
        four = tune.spread_rows == kSpreadFour;
        rows = tune.spread_rows == kSpreadRows;
    } else {
        // Four nodes per lane on 8 x 8 x 8 tiles when separations are
        // tile-relative and the tiles, four warps each, fill the chip four
        // times over (with fewer warps in flight each tile's serial walk over
        // its particles shows: 34 us against 17.8 with one node per lane at
        // N = 8000, phi = 0.45; 47 against 52 at N = 32768, 72^3).  Else one node per
        // lane on smaller tiles, which stage each particle more often but are
        // more, and keep separations tile-relative in a smaller box.
        const int shapes[4][5] = {{8, 8, 8, 4, 4 * 148}, {4, 8, 8, 1, 2 * 148}, {4, 4, 8, 1, 2 * 148}, {4, 4, 4, 1, 0}};
        for (int k = 0; k < 4; ++k) {
            c.TX = std::min(shapes[k][0], g.Nx - g.P + 1);
            c.TY = std::min(shapes[k][1], g.Ny - g.P + 1);
            c.TZ = std::min(shapes[k][2], g.Nz - g.P + 1);
            four = shapes[k][3] == 4;
            if (k < 3 && c.TX == shapes[k][0] && c.TY == shapes[k][1] && c.TZ == shapes[k][2] &&
                spread_tiles(g, c.TX, c.TY, c.TZ) >= shapes[k][4] && spread_local(g, xy, c.TX, c.TY, c.TZ))
                break;
        }
    }
    rows = rows || !(c.TX % 2 == 0 && c.TY % 4 == 0 && c.TZ % 4 == 0);
    c.form = four ? kSpreadFour : rows ? kSpreadRows : kSpreadBlocks;
    c.local = spread_local(g, xy, c.TX, c.TY, c.TZ);
    return c;
}

}  // namespace fsd
