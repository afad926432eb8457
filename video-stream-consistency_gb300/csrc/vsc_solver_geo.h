// Geometry of the blend solver's solves in planes: the tiles of a round, what each
// reads and waits for, and where the frame's edges lie in it.  Plain integer
// arithmetic for the kernels, the launch code and tests on the host.
#pragma once

#ifdef __CUDACC__
#define VSC_HD __host__ __device__ __forceinline__
#else
#define VSC_HD inline
#endif

namespace vsc {

enum SolverForm { kSolverExact = 0, kSolverFma = 1 };

#ifndef VSC_SOLVER_T
#define VSC_SOLVER_T 8
#endif
constexpr int kTbT = VSC_SOLVER_T;        // steps of a round (its ring's width); longer ones are multiples of half
constexpr int kPlW = 128;                 // tile width (a warp: 32 lanes x 4 columns)

// How a solve in planes runs: its form (bit 0) and whether its rounds are 16
// steps with a 16-pixel ring (bit 1) or 12 with 12 (bit 2) instead of 8.
constexpr int kPlLong = 2, kPlMid = 4;

// A form's tile: kPlanes input planes, kWarps warps of kRPT rows each, and the
// registers of the compute and the control warps.
template <int kForm>
struct PlG;
template <>
struct PlG<kSolverFma> {  // O, U, nK, Cs
    static constexpr int kPlanes = 4, kWarps = 8, kRPT = 9;
    static constexpr int kComputeRegs = 216, kControlRegs = 72;
};
// The exact form's step needs three constants of a pixel, consWt, lap P and A:
// 160 registers of state for 4 x 8 blocks, a tile of 128 x 64 (interior 112 x
// 48, 66 %).
template <>
struct PlG<kSolverExact> {  // O, U, consWt, lap P, A
    static constexpr int kPlanes = 5, kWarps = 8, kRPT = 8;
    static constexpr int kComputeRegs = 224, kControlRegs = 56;
};

constexpr int pl_round_steps(int cfg) { return cfg & kPlLong ? 2 * kTbT : cfg & kPlMid ? 3 * kTbT / 2 : kTbT; }

template <int kCfg>
struct PlGeo : PlG<kCfg & 1> {
    using B = PlG<kCfg & 1>;
    using B::kPlanes;
    using B::kRPT;
    using B::kWarps;
    static constexpr bool kFma = (kCfg & 1) == kSolverFma;
    static constexpr int kT = pl_round_steps(kCfg);            // steps a round, the ring's width: 8, 12, 16
    static constexpr int kIW = kPlW - 2 * kT;            // interior columns: 112, 104, 96
    static constexpr int kRows = kRPT * kWarps;          // 72 (FMA), 64 (exact)
    static constexpr int kIRows = kRows - 2 * kT;        // interior rows: 56, 48, 40 (FMA), 48, 40, 32 (exact)
    static constexpr int kStage = kRows * kPlW;          // floats of one input tile
    static constexpr int kStageBytes = kStage * static_cast<int>(sizeof(float));
    static constexpr int kSlots = (kWarps + 2) * 2 * kPlW;  // edge-row slots of one buffer
    static constexpr int kOut = kIRows * kIW;            // floats of one interior tile
    static constexpr int kSmem =
        kPlanes * kStageBytes + (2 * kSlots + 2 * kOut) * static_cast<int>(sizeof(float)) + 128;
    static_assert(kSmem <= 232448, "dynamic shared memory per CTA");
    static_assert((kPlanes * kStageBytes) % 128 == 0 && (2 * kSlots * 4) % 128 == 0 && (kOut * 4) % 128 == 0,
        "TMA sources and destinations on the 128-byte grid");
    static_assert(kT <= kIW && kT <= kIRows, "a tile reads only its 3 x 3 neighbours' interiors");
    static_assert((kIW * 4) % 16 == 0 && (kT * 4) % 16 == 0, "TMA x coordinates must be 16-byte aligned");
    // rows of the tile that the frame's rows 0 (tiles at oy = -kT) and h - 2, h - 1
    // (tiles that end on the frame's last row) sit in, as warp and row
    static constexpr int kTopWarp = kT / kRPT, kTopRow = kT % kRPT;
    static constexpr int kBot2Warp = (kRows - kT - 2) / kRPT, kBot2Row = (kRows - kT - 2) % kRPT;
    static constexpr int kBot1Warp = (kRows - kT - 1) / kRPT, kBot1Row = (kRows - kT - 1) % kRPT;
};

template <int kCfg>
VSC_HD int pl_tiles_x(int w)
{
    return (w + PlGeo<kCfg>::kIW - 1) / PlGeo<kCfg>::kIW;
}
template <int kCfg>
VSC_HD int pl_tiles(int w, int h)
{
    return 3 * pl_tiles_x<kCfg>(w) * ((h + PlGeo<kCfg>::kIRows - 1) / PlGeo<kCfg>::kIRows);
}

// The moved bottom row of tiles reads two rows of tiles up.
template <int kCfg>
VSC_HD bool pl_deep(int h, int ty_n)
{
    using G = PlGeo<kCfg>;
    return G::kT > kTbT && ty_n >= 3 && h - (ty_n - 1) * G::kIRows < G::kT;
}

// Tile `local` of a solve of h rows: channel, place among the channel's per_plane =
// tx_n x ty_n tiles, and its origin (ring included).
struct PlTileAt {
    int c, tx, ty, ty_n, ox, oy;
};

template <int kCfg>
VSC_HD PlTileAt pl_tile(int h, int tx_n, int per_plane, int local)
{
    using G = PlGeo<kCfg>;
    PlTileAt t;
    t.c = local / per_plane;
    const int r = local - t.c * per_plane;
    t.tx = r % tx_n;
    t.ty = r / tx_n;
    const int ty_n = t.ty_n = per_plane / tx_n;
    t.ox = t.tx * G::kIW - G::kT;
    t.oy = t.ty * G::kIRows - G::kT;
    // The bottom row of tiles is moved up until its interior ends on the
    // frame's last row (rows h - 2 and h - 1 then sit in fixed rows of fixed
    // warps, where a step tests them without per-row tests), when its top ring
    // still lies in the row of tiles above (the 3 x 3 dependency holds) or, in
    // longer rounds, whose 16-pixel ring reaches further than 40 % of the frames'
    // last rows of tiles (12 pixels: 27 %), in the two rows above (pl_watched_tile
    // has two rows up and down there).  Its interior then overlaps those rows':
    // both compute the shared rows from the same inputs with the same arithmetic
    // and store the same bits.
    if (t.ty == ty_n - 1 && t.ty > 0 && (h - t.ty * G::kIRows >= G::kT || pl_deep<kCfg>(h, ty_n)))
        t.oy = h - G::kRows + G::kT;
    return t;
}

// Watched tile i of kPlWatched, as an index among its channel's tiles, or -1: a
// tile's round k waits for round k - 1 of its 3 x 3 neighbourhood (itself included)
// and, where the bottom row of tiles reads two rows up, of the tiles it reads there,
// whose writers wait for it in turn.
constexpr int kPlWatched = 12;

template <int kCfg>
VSC_HD int pl_watched_tile(int h, int tx_n, const PlTileAt& t, int i)
{
    const int ty_n = t.ty_n;
    if (i >= (PlGeo<kCfg>::kT > kTbT ? kPlWatched : 9))
        return -1;
    const int x = t.tx + i % 3 - 1;
    int y = t.ty + i / 3 - 1;
    if (i >= 9)
        y = !pl_deep<kCfg>(h, ty_n) ? -1 : t.ty == ty_n - 1 ? ty_n - 3 : t.ty == ty_n - 3 ? ty_n - 1 : -1;
    return x >= 0 && x < tx_n && y >= 0 && y < ty_n ? y * tx_n + x : -1;
}

// Neighbour tests of the planar step.  kernel_consist_out reads a neighbour as
// +0 unless it lies in [0, w - 2] x [0, h - 2] (left: gx - 1 >= 0, right:
// gx + 1 < w - 1, up: gy - 1 >= 0, down: gy + 1 < h - 1), so the only pixels of
// the frame with a neighbour read as +0 are column 0 (left), columns w - 2 and
// w - 1 (right), row 0 (up) and rows h - 2 and h - 1 (down); every other read
// of a pixel inside the frame is of a pixel inside the frame.  Pixels outside
// the frame (the ring of a border tile) are computed too, but no pixel inside
// the frame reads them unmasked, so their values never reach the output.
//   kPlAll:   an interior tile, no test.
//   kPlLanes: a border tile of a frame whose width, like the tile origins, is
//             a multiple of 4: column 0 is then column j = 0 of the thread
//             with gx0 = 0 and columns w - 2, w - 1 are j = 2, 3 of the thread
//             with gx0 = w - 4 (three selects a row); row 0 of a tile at
//             oy = -kT and rows h - 2, h - 1 of one at oy = h - kRows + kT are fixed
//             rows of fixed warps (kTopRow ..: a select of a row's up or down
//             neighbours in every warp, true only in that one).  A tile
//             holding row 0, h - 2 or h - 1 elsewhere (frames of few rows)
//             takes kPlEvery.
//   kPlCols:  the same for any other width: columns w - 2 and w - 1 may be any
//             column of a thread (five selects a row).
//   kPlEvery: rows 0, h - 2 and h - 1 anywhere, too (a select of every row's up
//             and down neighbours).
enum { kPlAll, kPlLanes, kPlCols, kPlEvery };

// What a step needs to know of its thread's place.  zl / zr: it holds column 0 /
// columns w - 4 .. w - 1; zt / zb2 / zb1 (kPlLanes, kPlCols): its row kTopRow /
// kBot2Row / kBot1Row is the frame's row 0 / h - 2 / h - 1.
struct PlPlace {
    int xlim;      // its first column that is column w - 2 or beyond
    int top, bot;  // kPlEvery: its row that is row 0, its first one that is row h - 2 or beyond
    bool zl, zr, zt, zb2, zb1;
};

// The planar step's test mode for a tile at (ox, oy) of a w x h frame.
template <int kCfg>
VSC_HD int pl_mode(int ox, int oy, int w, int h)
{
    using G = PlGeo<kCfg>;
    constexpr int kRows = G::kRows;
    if (ox >= 1 && oy >= 1 && ox + kPlW - 1 <= w - 3 && oy + kRows - 1 <= h - 3)
        return kPlAll;
    const bool row0 = oy <= 0 && oy + kRows - 1 >= 0;
    const bool last2 = oy <= h - 1 && oy + kRows - 1 >= h - 2;
    if ((!row0 || oy == -G::kT) && (!last2 || oy == h - kRows + G::kT))  // ox is a multiple of 4
        return (w & 3) == 0 ? kPlLanes : kPlCols;
    return kPlEvery;
}

// Whether some row of tiles of a solve takes kPlEvery.
template <int kCfg>
VSC_HD bool pl_row_tests(int w, int h)
{
    const int tx_n = pl_tiles_x<kCfg>(w), per_plane = pl_tiles<kCfg>(w, h) / 3;
    for (int first = 0; first < per_plane; first += tx_n) {
        const PlTileAt t = pl_tile<kCfg>(h, tx_n, per_plane, first);
        if (pl_mode<kCfg>(t.ox, t.oy, w, h) == kPlEvery)
            return true;
    }
    return false;
}

// A thread's place in a tile at (ox, oy).
template <int kCfg>
VSC_HD PlPlace pl_place(int ox, int oy, int w, int h, int lane, int warp)
{
    using G = PlGeo<kCfg>;
    const int gx0 = ox + 4 * lane, gy0 = oy + G::kRPT * warp;
    PlPlace t;
    t.xlim = w - 2 - gx0;
    t.top = -gy0;
    t.bot = h - 2 - gy0;
    t.zl = gx0 == 0;
    t.zr = gx0 == w - 4;
    t.zt = oy == -G::kT && warp == G::kTopWarp;
    t.zb2 = oy == h - G::kRows + G::kT && warp == G::kBot2Warp;
    t.zb1 = oy == h - G::kRows + G::kT && warp == G::kBot1Warp;
    return t;
}

}  // namespace vsc
