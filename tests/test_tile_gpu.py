"""The tile form of the axis pass (csrc/sweep_tile.cuh), which default solvers and batches run: the same
bits as the marches (which fixed segments select) and as the oracle, at the edges of its tiles, with
units scanned for uniform regions and without, next to walls, and in batches of uneven domains."""
import ctypes as C

import numpy as np
import pytest

import armon_gb300 as A
import oracle_lib as O

FIELDS = ("rho", "umat", "vmat", "Emat", "pmat", "cmat")


# ---- tile geometry, restated on the CPU ----

def tile_axis(n, nlines, rows, halo, sms, slots, y_lines):
    want = 1 if rows else max(1, min(y_lines, nlines))
    longest = max(1, min(248, 256 - 2 * halo) if rows else 256 // want // 8 * 8 - 2 * halo)
    segs = -(-n // longest)
    length = -(-n // segs)
    segs = -(-n // length)
    width = length + 2 * halo
    fit = max(1, 256 // width)
    spread = max(1, nlines * segs // sms)
    lines = max(1, min(fit if rows else min(fit, want), nlines, spread))
    groups = -(-nlines // lines)
    scan = (lines == 1 if rows else lines * 8 <= 64 and -(-width // 8) * 8 * lines <= 256) and 32 <= n < 1 << 23 \
        and segs * groups >= 3 * slots
    if not rows and scan:
        groups = -(-groups // 8) * 8
    tiles = segs * groups
    big = max(0, (tiles - 4 * slots) // 8)
    return dict(len=length, width=width, segs=segs, lines=lines, groups=groups, scan=scan, big=big,
                units=big + tiles - 8 * big)


@pytest.mark.parametrize("halo", [2, 3, 4])
@pytest.mark.parametrize("y_lines", [2, 4, 8])
def test_tiles_cover_each_cell_once_and_stay_in_the_ghosts(halo, y_lines):
    sizes = (1, 5, 17, 31, 32, 100, 119, 120, 121, 239, 240, 241, 247, 248, 249, 256, 300, 497, 1000)
    for n in sizes:
        for nlines in (1, 2, 7, 33, 700):
            for rows in (True, False):
                for slots in (1, 456):
                    g = tile_axis(n, nlines, rows, halo, 152, slots, y_lines)
                    assert g["lines"] * g["width"] <= 256
                    if rows:
                        assert g["len"] <= 248        # 31 chunks of eight, a bit per position in 8 words
                    owned = np.zeros((nlines, n), int)
                    seen = 0
                    for u in range(g["units"]):
                        t0 = 8 * u if u < g["big"] else 8 * g["big"] + u - g["big"]
                        nk = 8 if u < g["big"] else 1
                        segs = set()
                        for t in range(t0, t0 + nk):
                            seen += 1
                            grp, seg = divmod(t, g["segs"]) if rows else divmod(t, g["groups"])[::-1]
                            segs.add(seg)
                            a0 = seg * g["len"]
                            b0 = min(n, a0 + g["len"])
                            assert b0 > a0 and a0 - halo >= -halo and b0 + halo <= n + halo
                            for line in range(grp * g["lines"], min(nlines, (grp + 1) * g["lines"])):
                                owned[line, a0:b0] += 1
                        if g["scan"] and not rows:
                            assert len(segs) == 1     # a scanned unit of columns lies in one segment
                            cols = nk * g["lines"]
                            assert -(-g["width"] // 8) * cols <= 256
                    assert seen == g["segs"] * g["groups"] and (owned == 1).all()


# ---- states with uniform regions ----

def patches(case, seed, longest):
    """Rectangles of three states, two at rest, of sides 1 .. longest, on all cells, ghosts included."""
    rng = np.random.default_rng(seed)
    p = A.make_params(case)

    def labels(n):
        out, lab = [], 0
        while len(out) < n:
            lab += int(rng.integers(1, 3))
            out += [lab] * int(rng.integers(1, longest))
        return np.array(out[:n])

    idx = (labels(p.row_length)[None, :] + labels(p.col_length)[:, None]) % 3
    rho, pr = np.array([1.0, 0.125, 0.7]), np.array([1.0, 0.1, 0.8])
    u, v = np.array([0.0, 0.0, 0.2]), np.array([0.0, -0.0, -0.1])
    E = pr / (0.4 * rho) + 0.5 * (u * u + v * v)
    return {k: a[idx].ravel() for k, a in dict(rho=rho, umat=u, vmat=v, Emat=E).items()}


def solve(case, state=None, **kw):
    with A.Solver(case, **kw) as s:
        s.init_test()
        if state is not None:
            for k, a in state.items():
                s.upload(k, a)
            s.begin_loop()
        s.run()
        p, st = s.state()
        assert st == 0
        return (p.cycle, p.time, p.next_cycle_dt), {k: A.real_cells(s.params, s.download(k)) for k in FIELDS}


def same(a, b, what):
    assert a[0] == b[0], what
    for k in FIELDS:
        t = np.uint64 if a[1][k].dtype == np.float64 else np.uint32
        assert np.array_equal(np.ascontiguousarray(a[1][k]).view(t), np.ascontiguousarray(b[1][k]).view(t)), (what, k)


OPTIONS = [
    dict(scheme="GAD", projection="euler_2nd", limiter="Minmod", splitting="Sequential", nghost=5),
    dict(scheme="GAD", projection="euler", limiter="Superbee", splitting="SequentialSym", nghost=3),
    dict(scheme="Godunov", projection="euler_2nd", limiter="None", splitting="Strang", nghost=4),
    dict(scheme="Godunov", projection="euler", limiter="Minmod", splitting="Sequential", nghost=2),
]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("kw", OPTIONS, ids=lambda k: f"{k['scheme']}-{k['projection']}-{k['splitting']}")
def test_tiles_give_the_marches_bits_at_tile_edges(kw, precision):
    # widths and heights at, below and above a tile's limits, single lines' worth of remainders
    for nx, ny in ((241, 121), (248, 120), (249, 119), (17, 497), (500, 16), (64, 73)):
        case = A.Case(test="Sod_circ", nx=nx, ny=ny, stencil=kw["nghost"], cfl=0.5, max_cycles=7, max_time=1e9, **kw)
        same(solve(case, precision=precision), solve(case, precision=precision, split_pass=-1, seg_len=64), (nx, ny))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("longest", [24, 300])
@pytest.mark.parametrize("kw", OPTIONS, ids=lambda k: f"{k['scheme']}-{k['projection']}-{k['splitting']}")
def test_scanned_uniform_regions_give_the_computed_bits(kw, longest, precision):
    # large enough for the units to be scanned (three tiles a resident block); patches shorter than a
    # window and longer than a tile, against every position computed and against the marches
    case = A.Case(test="Sod_circ", nx=811, ny=803, stencil=kw["nghost"], cfl=0.5, max_cycles=9, max_time=1e9, **kw)
    state = patches(case, 7 * longest, longest)
    ref = solve(case, state, precision=precision, reuse=-1)
    same(solve(case, state, precision=precision), ref, "scan")
    same(solve(case, state, precision=precision, split_pass=-1, reuse=-1, seg_len=100), ref, "march")
    same(solve(case, state, precision=precision, materialize_eos=0), ref, "p, c, g stored by the passes")


@pytest.mark.gpu
def test_scanned_regions_match_the_oracle():
    case = A.Case(test="Sod_circ", scheme="GAD", projection="euler_2nd", nghost=5, nx=811, ny=803, cfl=0.5, max_cycles=12,
                  max_time=1e9)
    state = patches(case, 3, 200)
    L = O.lib()
    p = O.make_params(O.Case(**case.__dict__))
    st = O.OracleState(p)
    L.o_init_test_p(C.byref(p), C.byref(st.data), 0)
    for k, a in state.items():
        st[k][:] = a
    status = C.c_int()
    L.o_time_loop(C.byref(p), C.byref(st.data), C.byref(status))
    assert status.value == 0
    same(solve(case, state), ((p.cycle, p.time, p.next_cycle_dt), {k: O.real_cells(p, st[k]) for k in FIELDS}), "oracle")


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [64, 32])
def test_batch_of_uneven_domains_matches_solo(precision):
    # one domain large enough to be scanned, small ones that blocks join when theirs are done, and a
    # change to marches and back while p, c, g are not in memory
    def case(nx, ny, cycles):
        return A.Case(test="Sod_circ", scheme="GAD", projection="euler_2nd", nghost=5, nx=nx, ny=ny, cfl=0.6,
                      max_cycles=cycles, max_time=1e9)

    cases = [case(900, 1100, 14), case(64, 64, 25), case(333, 41, 9), case(16, 700, 18), case(130, 257, 14)]
    states = [patches(c, k, 150) for k, c in enumerate(cases)]
    with A.Batch(precision=precision, cycles_per_graph=4) as b:
        ids = [b.add(A.make_params(c), s) for c, s in zip(cases, states)]
        b.run(cycle_limit=6)
        b.set_seg_len(ids[0], 40)
        b.run(cycle_limit=4)
        b.set_seg_len(ids[0], 0)
        assert b.run() == 0
        for i, c, s in zip(ids, cases, states):
            p, st = b.state(i)
            assert st == 0
            got = ((p.cycle, p.time, p.next_cycle_dt), {k: A.real_cells(b.params[i], b.download(i, k)) for k in FIELDS})
            same(got, solve(c, s, precision=precision, split_pass=-1, reuse=-1, seg_len=64), (c.nx, c.ny))
