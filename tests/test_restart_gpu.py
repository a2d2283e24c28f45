"""A solver whose loop is started again while its state is in the second buffer set."""
import numpy as np
import pytest

import armon_gb300 as A

pytestmark = pytest.mark.gpu

FIELDS = ("rho", "umat", "vmat", "Emat", "pmat", "cmat")


@pytest.mark.parametrize("kw", [dict(), dict(split_pass=1, seg_len=24), dict(precision=32)], ids=["tiles", "marches", "fp32"])
@pytest.mark.parametrize("splitting", ["Strang", "X_only", "Sequential"])
def test_init_test_after_enqueued_cycles(splitting, kw):
    # an odd number of passes (three or one a cycle) leaves the state in the other set
    case = A.Case(test="Sod_circ", scheme="GAD", projection="euler_2nd", nghost=5, nx=64, ny=48, cfl=0.6, max_cycles=7,
                  max_time=1e9, splitting=splitting)
    out = []
    for cycles in (0, 1, 2):
        with A.Solver(case, **kw) as s:
            s.init_test()
            if cycles:
                s.enqueue_cycles(cycles)
                s.init_test()
            s.run()
            p, status = s.state()
            assert status == 0
            out.append(((p.cycle, p.time, p.next_cycle_dt), {k: s.download(k) for k in FIELDS}))
    for end, f in out[1:]:
        assert end == out[0][0]
        for k in FIELDS:
            assert np.array_equal(f[k].view(np.int64), out[0][1][k].view(np.int64)), k
