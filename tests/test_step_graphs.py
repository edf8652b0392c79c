"""The captured form of the steps, which every flow of more than 64 steps runs, against the same
kernels launched one by one: bitwise, for every set of kernels, with defect-corrected members whose
refreshes fall on different steps."""
import os
import subprocess
import sys

import numpy as np
import pytest

from tests._profile import trace, traced
from tests.test_march import inputs, params_for

pytestmark = pytest.mark.gpu

SMALL, LARGE = (23, 13, 45), (57, 58, 57)   # rho: the fused FP32 kernels up to 56^3 sites, separate walks beyond


def _engine(eng, members, periods):
    ids = []
    for k, (name, precision, dims) in enumerate(members):
        _, p_i, p_f = params_for(name, dims)
        F, V = inputs(int(p_i[5]), dims, seed=30 + k)
        ids.append(eng.add(name, (p_i, p_f), F, V, precision=precision))
        if periods[k] is not None:
            eng.set_defect_period(ids[-1], periods[k])
    return ids


def _state(eng, ids):
    out = []
    for i in ids:
        s = eng.stats(i)
        out.append(((s.energy, s.baryon, s.err, s.gabs, s.kinetic, s.arrested, s.step),) + eng.read(i))
    return out


def _same(a, b):
    for x, y in zip(a, b):
        assert x[0] == y[0]
        assert np.array_equal(x[1], y[1]) and np.array_equal(x[2], y[2])


@pytest.mark.parametrize("name,dims", [("nuclear", SMALL), ("omega", SMALL), ("coulomb", SMALL), ("berger", SMALL),
                                       ("lightly_bound", SMALL), ("rho", SMALL), ("rho", LARGE)])
@pytest.mark.parametrize("precision", ["fp64", "fp32", "fp32d"])
def test_captured_steps_equal_launched_ones(name, precision, dims):
    from skyrmion_solver_b200.engine import Engine
    n = 90 if dims == SMALL else 70
    out = []
    for captured in (True, False):
        with Engine(0) as eng:
            ids = _engine(eng, [(name, precision, dims)], [None])
            if captured:
                eng.step(n)          # more than 64 steps at once: captured from the first
            else:
                eng.time_stages(n)   # one kernel after the other
            out.append(_state(eng, ids))
    _same(*out)


def test_captured_steps_with_refreshes_out_of_phase():
    """Three defect-corrected members (periods 16, 5 and 3: more patterns of refreshes than an engine
    keeps), an FP64 one and one that is paused for a while; in calls of different lengths."""
    from skyrmion_solver_b200.engine import Engine
    members = [("omega", "fp32d", SMALL), ("rho", "fp32d", (20, 17, 33)), ("nuclear", "fp32d", (24, 20, 28)),
               ("coulomb", "fp64", (16, 21, 30)), ("berger", "fp32", (19, 18, 31))]
    out = []
    for captured in (True, False):
        with Engine(0) as eng:
            ids = _engine(eng, members, [None, 5, 3, None, None])
            run = eng.step if captured else eng.time_stages
            run(67)
            eng.set_active(ids[0], False)
            run(9)
            eng.set_active(ids[0], True)
            for n in (13, 1, 40):
                run(n)
            out.append(_state(eng, ids))
    _same(*out)


def _refresh_kernels():
    from skyrmion_solver_b200.engine import Engine

    def run():
        with Engine(0) as eng:
            _engine(eng, [("omega", "fp32d", SMALL)], [None])
            for due in (0, 1, 0, 1):     # steps 1-8, 9-16, ..
                names = [e["name"] for e in trace(lambda: eng.step(8)) if "grid" in e.get("args", {})]
                assert sum("k_grad_stage" in k for k in names) >= 8
                assert sum("k_defect" in k for k in names) == due
    traced(run)


def test_only_steps_with_a_refresh_run_its_kernel():
    """A step without a defect refresh launches no refresh kernel (and does not order stage 1 after
    stage 4 for its sake).  In a process of its own, where the profiler has not been used before."""
    r = subprocess.run([sys.executable, "-c", "from tests import test_step_graphs as t; t._refresh_kernels()"],
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))), capture_output=True, text=True,
                       timeout=300)
    if "Skipped" in r.stderr:
        pytest.skip("torch's profiler records no device events here")
    assert r.returncode == 0, r.stderr[-2000:]
