"""The index arithmetic of the tile form (csrc/solver_common.h set_tile_axis, csrc/sweep_tile.cuh pack_place),
called on the host: tiles cover each cell once, scanned units keep to one segment, and a packed
thread never lies outside the stretch it stands for."""
import ctypes as C

import numpy as np
import pytest

import armon_gb300 as A
from test_tile_gpu import patches, same, solve

TILE = ("len", "width", "lines", "segs", "groups", "scan", "big", "units")


def tile_axis(n, nlines, rows, halo, slots, y_lines, tail, scan=True):
    out = (C.c_int32 * 8)()
    A.lib().armon_selftest_tile_axis(n, nlines, int(rows), halo, 152, slots, y_lines, tail, int(scan), out)
    return dict(zip(TILE, out))


def tile_pack(cells, halo):
    place = np.zeros((256, 3), np.int32)
    a = np.array(cells, np.int32)
    take = A.lib().armon_selftest_tile_pack(a.ctypes.data_as(C.c_void_p), len(cells), halo,
                                            place.ctypes.data_as(C.c_void_p))
    return take, place


@pytest.mark.parametrize("halo", [2, 3, 4])
@pytest.mark.parametrize("count", [1, 20, 31, 32, 33, 128])
def test_packed_threads_stay_in_their_stretches(halo, count):
    # stretches of one to eight cells (a segment's last cells, and whole chunks), alone and mixed
    rng = np.random.default_rng(100 * halo + count)
    for cells in [[c] * count for c in range(1, 9)] + [rng.integers(1, 9, count).tolist() for _ in range(20)]:
        take, place = tile_pack(cells, halo)
        want = [(k, q) for k, c in enumerate(cells[:take]) for q in range(c + 2 * halo)]
        assert len(want) <= 256 and take == min(32, count) or len(want) + cells[take] + 2 * halo > 256
        assert place[:len(want), 2].all() and not place[len(want):, 2].any()
        assert [tuple(p[:2]) for p in place[:len(want)]] == want


@pytest.mark.parametrize("tail", [4, 8, 16])
@pytest.mark.parametrize("halo", [2, 3, 4])
@pytest.mark.parametrize("y_lines", [2, 4, 8])
def test_tiles_cover_each_cell_once_and_fit_the_block(halo, y_lines, tail):
    sizes = (1, 5, 17, 31, 32, 100, 119, 120, 121, 240, 247, 248, 249, 300, 757, 1000)
    for n in sizes:
        for nlines in (1, 2, 7, 33, 700):
            for rows in (True, False):
                for slots in (1, 40, 608):
                    g = tile_axis(n, nlines, rows, halo, slots, y_lines, tail)
                    assert g["width"] == g["len"] + 2 * halo and g["lines"] * g["width"] <= 256 and g["len"] < 256
                    if rows:
                        assert g["len"] <= 248        # 31 chunks of eight
                    # every segment holds a cell, the last one's included; tiles past the lines are empty
                    assert (g["segs"] - 1) * g["len"] < n <= g["segs"] * g["len"]
                    assert (g["groups"] * g["lines"] >= nlines) and g["lines"] <= nlines
                    tiles = g["segs"] * g["groups"]
                    assert not tile_axis(n, nlines, rows, halo, slots, y_lines, tail, scan=False)["scan"]
                    assert g["units"] == g["big"] + tiles - 8 * g["big"] and 0 <= 8 * g["big"] <= tiles
                    if g["scan"]:
                        assert n >= 32 and tiles >= 3 * slots
                        if rows:
                            assert g["lines"] == 1
                        else:
                            # a unit lies in one segment, and its columns' chunks in the block's threads
                            assert g["groups"] % 8 == 0 and 8 * g["lines"] * -(-g["width"] // 8) <= 256
                        # the list holds what a scan can add (runs two idle chunks apart) and what packing
                        # leaves: 512 stretches
                        chunks = -(-g["len"] // 8)
                        assert 8 * g["lines"] * -(-chunks // 3) + 32 <= 512


# scanned domains whose last segment along Y (FP32: eight columns a tile, FP64: two) or X is shorter than a
# stretch of eight threads: reach 2 (Godunov, euler) with up to three cells, reach 3 with one
SHORT = [
    ("Godunov", "euler", 32, 6011, 757, 1, 1), ("Godunov", "euler", 32, 6211, 731, 1, 3),
    ("GAD", "euler", 32, 7011, 651, 1, 1), ("Godunov", "euler_2nd", 32, 6711, 677, 1, 1),
    ("Godunov", "euler", 64, 48, 15007, 1, 3), ("GAD", "euler", 64, 48, 14763, 1, 1),
    ("Godunov", "euler", 64, 60763, 16, 0, 3), ("Godunov", "euler", 32, 60763, 80, 0, 3),
]


@pytest.mark.parametrize("scheme,projection,precision,nx,ny,axis,last", SHORT)
def test_short_last_segments_are_what_the_solves_below_scan(scheme, projection, precision, nx, ny, axis, last):
    halo = 2 + (scheme == "GAD") + (projection == "euler_2nd")
    n, lines = (ny, nx) if axis else (nx, ny)
    g = tile_axis(n, lines, axis == 0, halo, 152 * (3 if precision == 64 else 4), 2 if precision == 64 else 8,
                  8 if precision == 64 else 4)
    assert A.lib().armon_selftest_scan_default(nx, ny, precision)
    assert g["scan"] and n - (g["segs"] - 1) * g["len"] == last


@pytest.mark.gpu
@pytest.mark.parametrize("scheme,projection,precision,nx,ny,axis,last", SHORT)
def test_short_last_segments_give_the_computed_bits(scheme, projection, precision, nx, ny, axis, last):
    # fronts and moving patches against the high wall, so that its short stretches are listed and packed
    case = A.Case(test="Sod_circ", scheme=scheme, projection=projection, limiter="Minmod", nghost=5, stencil=5, nx=nx, ny=ny,
                  cfl=0.5, max_cycles=8, max_time=1e9)
    state = patches(case, 11 + ny, 60)
    ref = solve(case, state, precision=precision, reuse=-1)
    same(solve(case, state, precision=precision), ref, "scan")
    same(solve(case, state, precision=precision, split_pass=-1, reuse=-1, seg_len=100), ref, "march")
