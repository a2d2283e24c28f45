"""Scanned units of the tile form (csrc/sweep_tile.cuh) where a window leaves the mirrored band or holds no
ordinary numbers: the same bits as with every position computed and as the marches."""
import numpy as np
import pytest

import armon_gb300 as A
from test_tile_gpu import FIELDS, OPTIONS, patches, same, solve

pytestmark = pytest.mark.gpu

# the smallest sizes with odd sides that a lone domain is scanned at (FP32 ones from 4.5 million cells on)
SCANNED = {64: (811, 803), 32: (2411, 2003)}


@pytest.mark.parametrize("longest", [24, 300])
@pytest.mark.parametrize("kw", OPTIONS, ids=lambda k: f"{k['scheme']}-{k['projection']}-{k['splitting']}")
def test_scanned_fp32_regions_give_the_computed_bits(kw, longest):
    nx, ny = SCANNED[32]
    case = A.Case(test="Sod_circ", nx=nx, ny=ny, stencil=kw["nghost"], cfl=0.5, max_cycles=6, max_time=1e9, **kw)
    state = patches(case, 7 * longest, longest)
    ref = solve(case, state, precision=32, reuse=-1)
    same(solve(case, state, precision=32), ref, "scan")
    same(solve(case, state, precision=32, split_pass=-1, reuse=-1, seg_len=100), ref, "march")
    same(solve(case, state, precision=32, materialize_eos=0), ref, "p, c, g stored by the passes")


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("longest", [24, 300])
@pytest.mark.parametrize("kw", OPTIONS, ids=lambda k: f"{k['scheme']}-{k['projection']}-{k['splitting']}")
def test_a_mirrored_band_narrower_than_the_stencil(kw, longest, precision):
    # the default band is one cell short of the stencil's reach except for GAD + second order, and here also
    # two short: positions past it read ghosts that no pass writes, and walls are never kept
    for stencil in (-1, 1):
        nx, ny = SCANNED[precision]
        case = A.Case(test="Sod_circ", nx=nx, ny=ny, cfl=0.5, max_cycles=6, max_time=1e9, stencil=stencil, **kw)
        state = patches(case, 5 * longest, longest)
        ref = solve(case, state, precision=precision, reuse=-1)
        same(solve(case, state, precision=precision), ref, "scan")
        same(solve(case, state, precision=precision, split_pass=-1, reuse=-1, seg_len=100), ref, "march")


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("kw", OPTIONS, ids=lambda k: f"{k['scheme']}-{k['projection']}-{k['splitting']}")
def test_patches_without_ordinary_numbers(kw, value, precision):
    # a density that is NaN or infinite has a NaN sound speed, which dt_CFL leaves out, so the loop goes on
    nx, ny = SCANNED[precision]
    case = A.Case(test="Sod_circ", nx=nx, ny=ny, stencil=kw["nghost"], cfl=0.5, max_cycles=5, max_time=1e9, **kw)
    state = patches(case, 77, 200)
    moving = state["umat"] != 0
    rows = np.arange(moving.size) // A.make_params(case).row_length
    state["rho"][moving & (rows % 500 < 250)] = value
    out = []
    for o in (dict(reuse=-1), dict(), dict(split_pass=-1, reuse=-1, seg_len=100)):
        end, f = solve(case, state, precision=precision, **o)
        assert np.isnan(f["rho"]).any() and np.isfinite(f["rho"]).any()
        # one NaN for all: two NaNs' payloads do not matter
        out.append((end, {k: np.where(np.isnan(a), np.nan, a) for k, a in f.items()}))
    same(out[1], out[0], "scan")
    same(out[2], out[0], "march")


def bands(case, seed, axis):
    """States that change from line to line and hold along lines of the given axis, with breaks: a band of
    lines keeps its states for a stretch of 3 to 400 positions, then takes others.  Ghosts included."""
    rng = np.random.default_rng(seed)
    p = A.make_params(case)
    shape = (p.col_length, p.row_length)
    f = {k: np.empty(shape) for k in ("rho", "umat", "vmat", "pr")}
    n, m = (shape[0], shape[1]) if axis == 1 else (shape[1], shape[0])     # along the axis, across
    line = 0
    while line < m:
        wide = int(rng.integers(1, 40))
        at = 0
        while at < n:
            long = int(rng.integers(3, 400))
            k = min(wide, m - line)
            for name, lo, hi in (("rho", 0.5, 1.5), ("umat", -0.2, 0.2), ("vmat", -0.2, 0.2), ("pr", 0.5, 1.5)):
                v = np.full(k, rng.uniform(lo, hi)) if rng.random() < 0.3 else rng.uniform(lo, hi, k)
                if axis == 1:
                    f[name][at:at + long, line:line + k] = v[None, :]
                else:
                    f[name][line:line + k, at:at + long] = v[:, None]
            at += long
        line += wide
    # a region at rest, so that the passes keep states and scan
    f["rho"][: shape[0] // 3], f["pr"][: shape[0] // 3], f["umat"][: shape[0] // 3], f["vmat"][: shape[0] // 3] = 1.0, 1.0, 0.0, 0.0
    E = f["pr"] / (0.4 * f["rho"]) + 0.5 * (f["umat"] ** 2 + f["vmat"] ** 2)
    return {"rho": f["rho"].ravel(), "umat": f["umat"].ravel(), "vmat": f["vmat"].ravel(), "Emat": E.ravel()}


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("kw", OPTIONS, ids=lambda k: f"{k['scheme']}-{k['projection']}-{k['splitting']}")
def test_runs_of_many_states(kw, axis, precision):
    # runs of states that are not kept, computed at one position each, ends and breaks at any chunk
    nx, ny = SCANNED[precision]
    case = A.Case(test="Sod_circ", nx=nx, ny=ny, stencil=kw["nghost"], cfl=0.4, max_cycles=4, max_time=1e9, **kw)
    state = bands(case, 100 + axis, axis)
    ref = solve(case, state, precision=precision, reuse=-1)
    same(solve(case, state, precision=precision), ref, "runs")
    same(solve(case, state, precision=precision, split_pass=-1, reuse=-1, seg_len=100), ref, "march")
    same(solve(case, state, precision=precision, materialize_eos=0), ref, "p, c, g stored by the passes")


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("test", ["Sod", "Sod_y"])
def test_planar_fronts_match_the_computed_bits(test, precision):
    # a planar front: the lines along it hold one state each, from wall to wall
    nx, ny = SCANNED[precision]
    case = A.Case(test=test, scheme="GAD", projection="euler_2nd", nghost=5, nx=nx, ny=ny, cfl=0.6, max_cycles=50, max_time=1e9)
    ref = solve(case, precision=precision, reuse=-1)
    same(solve(case, precision=precision), ref, "runs")
    with A.Batch(precision=precision) as b:
        i = b.add(A.make_params(case))
        j = b.add(A.make_params(A.Case(**{**case.__dict__, "nx": 128, "ny": 150})))
        assert b.run() == 0
        p, _ = b.state(i)
        assert b.state(j)[0].cycle == 50
        got = ((p.cycle, p.time, p.next_cycle_dt), {k: A.real_cells(b.params[i], b.download(i, k)) for k in FIELDS})
        same(got, ref, "batch")
