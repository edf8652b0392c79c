"""The host's estimate of an instance's device memory."""
from skyrmion_solver_b200 import engine, serving

def test_memory_estimate_of_small_rho_lattices():
    """The curls of rho's FP32 energy walks are counted where those walks run (above 56^3 sites)."""
    for f in (serving.instance_bytes, engine.instance_bytes):
        small, large = 48 ** 3, 60 ** 3
        assert f(13, small, "fp32") - 7 * 4 * 13 * small < 8192 * 48 + small // 2
        assert f(13, large, "fp32") - 7 * 4 * 13 * large >= 72 * large
    assert serving.stored_sites([10, 11, 13]) == 10 * 11 * 16 and serving.stored_sites([10, 11, 12]) == 10 * 11 * 12
