"""Scanned units of the tile form (csrc/sweep_tile.cuh) where a window leaves the mirrored band or holds no
ordinary numbers: the same bits as with every position computed and as the marches."""
import numpy as np
import pytest

import armon_gb300 as A
from test_tile_gpu import OPTIONS, patches, same, solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("longest", [24, 300])
@pytest.mark.parametrize("kw", OPTIONS, ids=lambda k: f"{k['scheme']}-{k['projection']}-{k['splitting']}")
def test_a_mirrored_band_narrower_than_the_stencil(kw, longest, precision):
    # the default band is one cell short of the stencil's reach except for GAD + second order, and here also
    # two short: positions past it read ghosts that no pass writes, and walls are never kept
    for stencil in (-1, 1):
        case = A.Case(test="Sod_circ", nx=811, ny=803, cfl=0.5, max_cycles=7, max_time=1e9, stencil=stencil, **kw)
        state = patches(case, 5 * longest, longest)
        ref = solve(case, state, precision=precision, reuse=-1)
        same(solve(case, state, precision=precision), ref, "scan")
        same(solve(case, state, precision=precision, split_pass=-1, reuse=-1, seg_len=100), ref, "march")


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("kw", OPTIONS, ids=lambda k: f"{k['scheme']}-{k['projection']}-{k['splitting']}")
def test_patches_without_ordinary_numbers(kw, value, precision):
    # a density that is NaN or infinite has a NaN sound speed, which dt_CFL leaves out, so the loop goes on
    case = A.Case(test="Sod_circ", nx=811, ny=803, stencil=kw["nghost"], cfl=0.5, max_cycles=5, max_time=1e9, **kw)
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
