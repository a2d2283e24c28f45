"""Batches and servers in the tile form (csrc/batch.cu): what their launches share is set up on their own
stream."""
import numpy as np
import pytest

import armon_gb300 as A
from test_batch_gpu import small_domains, solo

pytestmark = pytest.mark.gpu

FIELDS = ("rho", "umat", "vmat", "Emat", "pmat")


def busy_default_stream(torch):
    """Some tens of milliseconds of ordinary work queued on the default stream."""
    t = torch.ones(1 << 28, device="cuda")
    for _ in range(100):
        t.mul_(1.0)
    return t


@pytest.mark.parametrize("precision", [64, 32])
def test_batch_created_while_the_default_stream_is_busy(precision):
    torch = pytest.importorskip("torch")
    specs = small_domains(6, seed=17)
    refs = [solo(s, precision=precision) for s in specs]
    states = [s.initial_state() for s in specs]
    busy = busy_default_stream(torch)
    with A.Batch(precision=precision, cycles_per_graph=4) as b:
        ids = [b.add(s.params(), st) for s, st in zip(specs, states)]
        assert b.run() == 0
        for i, (ps, _, ref) in zip(ids, refs):
            pb, st = b.state(i)
            assert st == 0 and (pb.cycle, pb.time, pb.next_cycle_dt) == (ps.cycle, ps.time, ps.next_cycle_dt)
            for k in FIELDS:
                got = A.real_cells(b.params[i], b.download(i, k))
                assert np.array_equal(got.view(np.int64), ref[k].view(np.int64)), k
    torch.cuda.synchronize()
    del busy


def test_server_created_while_the_default_stream_is_busy():
    torch = pytest.importorskip("torch")
    specs = small_domains(6, seed=19)
    refs = [solo(s, precision=64 if k % 2 else 32) for k, s in enumerate(specs)]
    busy = busy_default_stream(torch)
    with A.Server() as srv:
        ids = [srv.submit(s.params(), 64 if k % 2 else 32, s.sod_interface()) for k, s in enumerate(specs)]
        done = set()
        while len(done) < len(ids):
            srv.step()
            while (r := srv.next_done()) is not None:
                done.add(r)
        for i, (ps, _, ref) in zip(ids, refs):
            assert (srv.info(i).cycle, srv.info(i).time) == (ps.cycle, ps.time)
            for k in FIELDS:
                got = A.real_cells(srv.params[i], srv.download(i, k))
                assert np.array_equal(got.view(np.int64), ref[k].view(np.int64)), k
    torch.cuda.synchronize()
    del busy


@pytest.mark.parametrize("precision", [64, 32])
def test_a_table_that_cannot_be_built_is_not_run(precision):
    # one cell per thread needs more partial slots than a 512 x 512 domain holds: refused at every call, and
    # the batch goes on as before once the segments are automatic again
    big = A.Case(test="Sod_circ", scheme="GAD", projection="euler_2nd", nghost=5, nx=512, ny=512, cfl=0.6, max_cycles=20,
                 max_time=1e9)
    small = A.Case(**{**big.__dict__, "nx": 48, "ny": 64})
    with A.Batch(precision=precision, cycles_per_graph=4) as b:
        ids = [b.add(A.make_params(c)) for c in (big, small)]
        b.run(cycle_limit=6)
        b.set_seg_len(ids[0], 1)
        for _ in range(2):
            with pytest.raises(A.ArmonError) as e:
                b.run(cycle_limit=4)
            assert e.value.code == A.ERR_STATE
        b.set_seg_len(ids[0], 0)
        assert b.run() == 0
        for i, c in zip(ids, (big, small)):
            with A.Solver(c, precision=precision) as s:
                s.init_test()
                s.run()
                p, q = b.state(i)[0], s.state()[0]
                assert (p.cycle, p.time, p.next_cycle_dt) == (q.cycle, q.time, q.next_cycle_dt)
                for k in FIELDS:
                    got, ref = A.real_cells(b.params[i], b.download(i, k)), A.real_cells(s.params, s.download(k))
                    assert np.array_equal(got.view(np.int64), ref.view(np.int64)), k


def test_the_marches_candidates_are_not_timed_on_tile_passes():
    # marches (one domain fixes its segments) start to time their schedule; tile passes end that
    case = A.Case(test="Sod_circ", scheme="GAD", projection="euler_2nd", nghost=5, nx=1024, ny=1100, cfl=0.6, max_cycles=200,
                  max_time=1e9)
    with A.Batch(cycles_per_graph=4) as b:
        ids = [b.add(A.make_params(c)) for c in (case, case, A.Case(**{**case.__dict__, "nx": 64}))]
        b.run(cycle_limit=4)
        untuned = b.schedule()[0]
        b.set_seg_len(ids[2], 64)
        b.run(cycle_limit=4)
        assert b.schedule()[0] != untuned          # the first candidate
        b.set_seg_len(ids[2], 0)
        for _ in range(7):
            b.run(cycle_limit=4)
            assert b.schedule()[0] == untuned
        assert all(b.state(i)[0].cycle == 36 for i in ids)
        got = [A.real_cells(b.params[i], b.download(i, "rho")) for i in ids[:2]]
        assert np.array_equal(got[0], got[1])


@pytest.mark.parametrize("precision", [64, 32])
def test_many_small_domains_and_a_large_one_match_solo(precision):
    # more domains than the launch has blocks, most of them dealt out, one that all blocks join in the end, and
    # a few that end before the others; every distinct size is compared
    def case(nx, ny, cycles):
        return A.Case(test="Sod_circ", scheme="GAD", projection="euler_2nd", nghost=5, nx=nx, ny=ny, cfl=0.6,
                      max_cycles=cycles, max_time=1e9)

    kinds = [case(16, 16, 12), case(17, 40, 9), case(33, 16, 12), case(90, 21, 12), case(700, 650, 12)]
    order = [k % 4 for k in range(1300)]
    order[801] = 4
    refs = []
    for c in kinds:
        with A.Solver(c, precision=precision) as s:
            s.init_test()
            s.run()
            p, _ = s.state()
            refs.append(((p.cycle, p.time, p.next_cycle_dt), {k: A.real_cells(s.params, s.download(k)) for k in FIELDS}))
    with A.Batch(precision=precision, cycles_per_graph=4) as b:
        ids = [b.add(A.make_params(kinds[k])) for k in order]
        assert b.run() == 0
        for n, (i, k) in enumerate(zip(ids, order)):
            p, st = b.state(i)
            assert st == 0 and (p.cycle, p.time, p.next_cycle_dt) == refs[k][0], n
            for f in FIELDS if n % 20 < 4 or k == 4 else ("rho",):
                got = A.real_cells(b.params[i], b.download(i, f))
                assert np.array_equal(got.view(np.int64), refs[k][1][f].view(np.int64)), (n, f)


@pytest.mark.parametrize("precision", [64, 32])
def test_planar_domains_run_in_marches_while_they_are_many(precision):
    # 40 planar domains, most of which end early: marches until fewer than 2^19 cells are left, tiles after
    # that and whenever a front that is not planar is among them
    def case(test, cycles):
        return A.Case(test=test, scheme="GAD", projection="euler_2nd", nghost=5, nx=128, ny=144, cfl=0.6, max_cycles=cycles,
                      max_time=1e9)

    kinds = [case("Sod", 8), case("Sod_y", 8), case("Sod", 20), case("Sod_circ", 12)]
    refs = []
    for c in kinds:
        with A.Solver(c, precision=precision) as s:
            s.init_test()
            s.run()
            p, _ = s.state()
            refs.append(((p.cycle, p.time, p.next_cycle_dt), {k: A.real_cells(s.params, s.download(k)) for k in FIELDS}))
    per_cycle = {True: 2, False: 5 if precision == 64 else 3}     # launches: tiles; marches and their block order
    for circular in (False, True):
        with A.Batch(precision=precision, cycles_per_graph=4) as b:
            order = [0, 1] * 17 + [2] * 6 + [3] * circular
            ids = [b.add(A.make_params(kinds[k])) for k in order]
            b.run(cycle_limit=4)
            for tiles in (circular, True):
                before = b.kernel_launches
                b.run(cycle_limit=4)
                # (a new table of marches starts from index order: one launch more)
                assert 0 <= b.kernel_launches - before - 4 * per_cycle[tiles] <= 1
            assert b.run() == 0
            for i, k in zip(ids, order):
                p, st = b.state(i)
                assert st == 0 and (p.cycle, p.time, p.next_cycle_dt) == refs[k][0]
                for f in FIELDS:
                    got = A.real_cells(b.params[i], b.download(i, f))
                    assert np.array_equal(got.view(np.int64), refs[k][1][f].view(np.int64)), (k, f)


def test_interfaces_along_an_axis_count_as_planar():
    def launches(shape, nx, ny):
        c = A.Case(test="Sod", scheme="GAD", projection="euler_2nd", nghost=5, nx=256, ny=256, cfl=0.6, max_cycles=8, max_time=1e9)
        sod = A.SodInterface(shape=shape, cx=0.5, cy=0.5, nx=nx, ny=ny, offset=0.0, r2=0.04, rho_high=1.0, p_high=1.0,
                             rho_low=0.125, p_low=0.1)
        with A.Batch(cycles_per_graph=4) as b:
            ids = [b.add_sod(c, sod) for _ in range(8)]
            b.run(cycle_limit=4)
            before = b.kernel_launches
            b.run(cycle_limit=4)
            n = b.kernel_launches - before
            return n, [b.download(i, "rho") for i in ids]

    for nx, ny in ((1.0, 0.0), (0.0, 1.0)):
        n, rho = launches(0, nx, ny)
        assert n == 4 * 5 and all(np.array_equal(rho[0], r) for r in rho)
    for shape, nx, ny in ((0, 0.6, 0.8), (1, 0.0, 0.0)):
        n, rho = launches(shape, nx, ny)
        assert n == 4 * 2 and all(np.array_equal(rho[0], r) for r in rho)
