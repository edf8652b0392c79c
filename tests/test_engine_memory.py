"""Device memory of the engine's instances: driver allocations of an admission and a removal, and
the accounting of the bytes they take."""
import numpy as np
import pytest

from tests._profile import trace, traced
from tests.test_march import inputs, params_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32d"])
def test_a_request_takes_and_frees_one_block_of_memory(precision):
    """Admission and removal beside a resident of the same group, from a field on the device: one
    cudaMalloc and one cudaFree.  (The group's descriptor and tile lists grow by more than they
    need, so the request finds room in them.)"""
    import torch
    from skyrmion_solver_b200.engine import Engine
    th, p_i, p_f = params_for("nuclear", (24, 20, 28))
    F = torch.from_numpy(inputs(4, (24, 20, 28))[0]).cuda()

    def run():
        with Engine(0) as eng:
            eng.add("nuclear", (p_i, p_f), F, None, precision=precision)
            before = eng.bytes
            got = []
            calls = [e["name"] for e in trace(
                lambda: got.append(eng.add("nuclear", (p_i, p_f), F, None, precision=precision)))]
            assert calls.count("cudaMalloc") == 1
            taken = eng.bytes - before
            calls = [e["name"] for e in trace(lambda: eng.remove(got[0]))]
            assert calls.count("cudaFree") == 1
            assert eng.bytes == before and taken > 0
    traced(run)


def test_bytes_follow_a_retiled_instance():
    """A change of the x-chunk replaces the partials: the bytes change with their sizes, do not
    drift over several changes, and all are given back."""
    from skyrmion_solver_b200.engine import Engine
    th, p_i, p_f = params_for("omega", (24, 20, 28))
    F, V = inputs(5, (24, 20, 28))
    with Engine(0) as eng:
        i = eng.add("omega", (p_i, p_f), F, V, precision="fp32")
        seen = []
        for xc in (4, 24, 4, 24):
            eng.retile(i, xc)
            seen.append(eng.bytes)
        assert seen[0] == seen[2] > seen[1] == seen[3]
        eng.step(2)
        assert np.isfinite(eng.stats(i).energy)
        eng.remove(i)
        assert eng.bytes == 0
