"""The marches' own measurements, which run when options select marches without fixing their segments: a
solver's tiling (both pass forms) and a batch's wave count.  Results never depend on them."""
import numpy as np
import pytest

import armon_gb300 as A

pytestmark = pytest.mark.gpu

FIELDS = ("rho", "umat", "vmat", "Emat", "pmat")


def fields(s):
    return {k: A.real_cells(s.params, s.download(k)) for k in FIELDS}


def same(a, b):
    for k in FIELDS:
        assert np.array_equal(a[k].view(np.int64), b[k].view(np.int64)), k


@pytest.mark.parametrize("precision", [64, 32])
def test_marches_measure_their_tiling_and_keep_the_results(precision):
    case = A.Case(test="Sod_circ", scheme="GAD", projection="euler_2nd", nghost=5, nx=1024, ny=1056, cfl=0.6,
                  max_cycles=120, max_time=1e9, test_option=0.04)
    A.tiling_cache_clear()
    with A.Solver(case, precision=precision, block_lines=128) as s:
        s.init_test()
        assert s.tuning()
        s.run()
        p, status = s.state()
        assert status == 0 and p.cycle == 120 and not s.tuning()
        # segments for one form in FP32 and two in FP64: more candidates than the tile form's two
        assert s.measurement_cycles() > 8 and s.measurement_cycles() % 2 == 0
        got, end = fields(s), (p.time, p.next_cycle_dt)
        chosen = s.tiling()
    with A.Solver(case, precision=precision, block_lines=128) as s:
        s.init_test()
        assert not s.tuning() and s.tiling() == chosen       # the cached choice
    with A.Solver(case, precision=precision) as s:           # the tile form measures for itself
        s.init_test()
        assert s.tuning()
        s.run()
        q, _ = s.state()
        assert s.measurement_cycles() == 8
        assert (q.time, q.next_cycle_dt) == end
        same(fields(s), got)
    A.tiling_cache_clear()


@pytest.mark.parametrize("split_pass", [1, -1])
@pytest.mark.parametrize("precision", [64, 32])
def test_march_batches_choose_their_waves_and_keep_the_results(precision, split_pass):
    case = A.Case(test="Sod_circ", scheme="GAD", projection="euler_2nd", nghost=5, nx=1024, ny=1100, cfl=0.6,
                  max_cycles=200, max_time=1e9, test_option=0.04)
    cases = [case, A.Case(**{**case.__dict__, "nx": 960}), A.Case(**{**case.__dict__, "ny": 96})]
    seen, out = [], []
    for kw in (dict(split_pass=split_pass), dict()):
        with A.Batch(precision=precision, cycles_per_graph=4, **kw) as b:
            ids = [b.add(A.make_params(c)) for c in cases]
            for _ in range(8):
                b.run(cycle_limit=4)
                if kw:
                    seen.append(b.schedule()[0])
            out.append([{k: A.real_cells(b.params[i], b.download(i, k)) for k in FIELDS} for i in ids])
            assert all(b.state(i)[0].cycle == 32 for i in ids)
    # one candidate a graph batch, then the fastest of them
    assert seen[:5] == [2, 4, 8, 16, 64] and seen[5] == seen[6] == seen[7] and seen[5] in seen[:5]
    for a, c in zip(*out):
        same(a, c)


@pytest.mark.parametrize("precision", [64, 32])
def test_a_measured_choice_belongs_to_what_the_loop_starts_from(precision):
    # one test problem's choice is not another's, nor that of a state that the caller uploads, for a new solver
    # as for the same one
    kw = dict(scheme="GAD", projection="euler_2nd", nghost=5, nx=1024, ny=1056, cfl=0.6, max_cycles=40, max_time=1e9)
    sod, sedov = (A.Case(test=t, **kw) for t in ("Sod", "Sedov"))
    A.tiling_cache_clear()
    with A.Solver(sod, precision=precision) as s:
        s.init_test()
        assert s.tuning()
        s.run()
        assert s.measurement_cycles() > 0
        s.init_test()
        assert not s.tuning()
        state = {k: s.download(k) for k in ("rho", "umat", "vmat", "Emat")}
        for k, a in state.items():
            s.upload(k, a)
        s.begin_loop()
        assert s.tuning()
        s.run()
        own = fields(s)
        s.init_test()
        assert not s.tuning()
        s.run()
        same(fields(s), own)
    with A.Solver(sedov, precision=precision) as s:
        s.init_test()
        assert s.tuning()
        s.run(cycle_limit=21)             # a candidate is in use
        s.init_test()
        s.run()
        again = fields(s)
    with A.Solver(sedov, precision=precision, reuse=-1) as s:
        s.init_test()
        s.run()
        same(fields(s), again)
    A.tiling_cache_clear()


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("test", ["Sod", "Sod_y", "Sod_circ", "Sedov"])
@pytest.mark.parametrize("shape", [(1024, 1056), (2400, 1900), (700, 6600)])
def test_candidates_of_every_form_keep_the_results(shape, test, precision):
    # tiles scanned and computed, and marches for planar fronts, one after another on the cycles of one solve
    nx, ny = shape
    case = A.Case(test=test, scheme="GAD", projection="euler_2nd", nghost=5, nx=nx, ny=ny, cfl=0.5, max_cycles=40,
                  max_time=1e9)
    A.tiling_cache_clear()
    out = []
    for kw in (dict(), dict(), dict(reuse=-1), dict(split_pass=-1, seg_len=64)):
        with A.Solver(case, precision=precision, **kw) as s:
            s.init_test()
            s.run()
            p, status = s.state()
            assert status == 0 and p.cycle == 40 and not s.tuning()
            assert kw or len(out) or s.measurement_cycles() == (16 if test in ("Sod", "Sod_y") else 8)
            out.append((fields(s), (p.time, p.current_cycle_dt, p.next_cycle_dt)))
    for got, end in out[1:]:
        assert end == out[0][1]
        same(got, out[0][0])
    A.tiling_cache_clear()
