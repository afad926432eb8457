"""The solve kernel's tiles for both forms and its rounds of 8, 12 and 16 steps:
the library's own geometry (csrc/vsc_solver_geo.h), compiled on the host and
checked for every height up to several rows of tiles and widths of every kind.

What the kernel relies on: interiors cover the frame; a row or column that a
tile reads is written by a tile that it waits for; a tile that writes a region
again waits for every tile that read it; tiles with a region in common wait for
each other; and a step's neighbour tests mask exactly the neighbours that the
reference reads as zero."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "video-stream-consistency_gb300" / "csrc"

PROGRAM = r"""
#include "vsc_solver_geo.h"
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <vector>
using namespace vsc;
#define CHECK(c) do { if (!(c)) { std::printf("cfg %d %dx%d tile %d %d: %s\n", kCfg, w, h, a.tx, a.ty, #c); std::exit(1); } } while (0)

struct Span { int lo, hi; bool meets(Span o) const { return std::max(lo, o.lo) < std::min(hi, o.hi); } };

template <int kCfg> void frame(int w, int h)
{
    using G = PlGeo<kCfg>;
    const int tx_n = pl_tiles_x<kCfg>(w), per = pl_tiles<kCfg>(w, h) / 3, ty_n = per / tx_n;
    std::vector<PlTileAt> t(per);
    std::vector<Span> rx(per), ry(per), wx(per), wy(per);  // read and written, inside the frame
    for (int i = 0; i < per; ++i) {
        PlTileAt& a = t[i] = pl_tile<kCfg>(h, tx_n, per, i);
        CHECK(a.c == 0 && a.tx == i % tx_n && a.ty == i / tx_n && a.ty_n == ty_n);
        const PlTileAt c2 = pl_tile<kCfg>(h, tx_n, per, 2 * per + i);
        CHECK(c2.c == 2 && c2.ox == a.ox && c2.oy == a.oy);
        CHECK(a.ox % 4 == 0 && (a.ox + G::kT) % 4 == 0);  // TMA's x coordinates, in floats
        CHECK(a.ox + G::kT >= 0 && a.oy + G::kT >= 0);    // no store at a negative coordinate
        rx[i] = {std::max(0, a.ox), std::min(w, a.ox + kPlW)};
        ry[i] = {std::max(0, a.oy), std::min(h, a.oy + G::kRows)};
        wx[i] = {a.ox + G::kT, std::min(w, a.ox + G::kT + G::kIW)};
        wy[i] = {a.oy + G::kT, std::min(h, a.oy + G::kT + G::kIRows)};
        CHECK(wx[i].lo < wx[i].hi && wy[i].lo < wy[i].hi);
    }
    std::vector<std::vector<char>> waits(per, std::vector<char>(per, 0));
    for (int i = 0; i < per; ++i) {
        const PlTileAt& a = t[i];
        for (int k = 0; k < 32; ++k) {  // the loading warp's lanes
            const int f = pl_watched_tile<kCfg>(h, tx_n, a, k);
            CHECK(f < per && (k < kPlWatched || f < 0));
            if (f >= 0)
                waits[i][f] = 1;
        }
        CHECK(waits[i][i]);
    }
    for (int i = 0; i < per; ++i) {
        const PlTileAt& a = t[i];
        for (int y = ry[i].lo; y < ry[i].hi; ++y) {  // rows and columns of a tile's neighbours factor
            bool ok = false;
            for (int f = 0; f < per && !ok; ++f)
                ok = waits[i][f] && t[f].tx == a.tx && wy[f].lo <= y && y < wy[f].hi;
            CHECK(ok);
        }
        for (int x = rx[i].lo; x < rx[i].hi; ++x) {
            bool ok = false;
            for (int f = 0; f < per && !ok; ++f)
                ok = waits[i][f] && t[f].ty == a.ty && wx[f].lo <= x && x < wx[f].hi;
            CHECK(ok);
        }
        for (int f = 0; f < per; ++f) {
            if (rx[i].meets(wx[f]) && ry[i].meets(wy[f]))
                CHECK(waits[f][i]);  // f writes what i read
            if (f != i && wx[i].meets(wx[f]) && wy[i].meets(wy[f]))
                CHECK(waits[i][f] && waits[f][i]);
        }
        // the masks of every thread
        const int mode = pl_mode<kCfg>(a.ox, a.oy, w, h);
        const bool lanes = mode == kPlLanes, cols = mode == kPlCols || mode == kPlEvery, fixed = lanes || mode == kPlCols;
        if (lanes)
            CHECK(w % 4 == 0);
        for (int warp = 0; warp < G::kWarps; ++warp)
            for (int lane = 0; lane < 32; ++lane) {
                const PlPlace p = pl_place<kCfg>(a.ox, a.oy, w, h, lane, warp);
                for (int r = 0; r < G::kRPT; ++r) {
                    const int y = a.oy + G::kRPT * warp + r;
                    if (y < 0 || y >= h)
                        continue;
                    const bool up = (fixed && r == G::kTopRow && p.zt) || (mode == kPlEvery && r == p.top);
                    const bool down = (fixed && ((r == G::kBot2Row && p.zb2) || (r == G::kBot1Row && p.zb1))) ||
                                      (mode == kPlEvery && r >= p.bot);
                    CHECK(up == (y == 0) && down == (y >= h - 2));
                }
                for (int j = 0; j < 4; ++j) {
                    const int x = a.ox + 4 * lane + j;
                    if (x < 0 || x >= w)
                        continue;
                    const bool left = mode != kPlAll && j == 0 && p.zl;
                    const bool right = lanes ? j >= 2 && p.zr : cols && j >= p.xlim;
                    CHECK(left == (x == 0) && right == (x >= w - 2));
                }
            }
    }
    PlTileAt a{};
    for (int y = 0; y < h; ++y) {
        bool ok = false;
        for (int i = 0; i < per && !ok; ++i)
            ok = wy[i].lo <= y && y < wy[i].hi;
        CHECK(ok);
    }
    for (int x = 0; x < w; ++x) {
        bool ok = false;
        for (int i = 0; i < tx_n && !ok; ++i)
            ok = wx[i].lo <= x && x < wx[i].hi;
        CHECK(ok);
    }
}

template <int kCfg> void all()
{
    for (int h = 1; h <= 330; ++h)
        for (int w : {1, 2, 3, 4, 5, 96, 97, 104, 105, 112, 113, 114, 115, 128, 224, 225, 226, 241, 340})
            frame<kCfg>(w, h);
    for (int h : {719, 720, 1079, 1080, 1081, 2160})
        frame<kCfg>(1920 + h % 4, h);
}
int main()
{
    all<PLACEHOLDER>();
    std::puts("ok");
}
"""


@pytest.mark.parametrize("cfg", ["kSolverExact", "kSolverExact | kPlMid", "kSolverExact | kPlLong", "kSolverFma",
                                 "kSolverFma | kPlMid", "kSolverFma | kPlLong"])
def test_tiles_waits_and_masks(tmp_path, cfg):
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM.replace("PLACEHOLDER", cfg))
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
