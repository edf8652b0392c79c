"""The autotuner's use of an engine, against a fake that counts what it is asked to time (no GPU)."""
import numpy as np

from skyrmion_solver_b200 import autotune, engine


class _Fake:
    """An engine whose step takes a time that depends on staging and chunk, and on how often it was
    asked: two timings of the same kernels differ by noise."""
    made = []

    def __init__(self, device=0):
        self.timed = []
        self.now = {}
        self.calls = 0
        _Fake.made.append(self)

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        pass

    def add(self, theory, params, field, velocity, precision):
        self.now = {"st": (True, False), "xc": 7}
        return 1

    def remove(self, iid):
        pass

    def staging(self, iid):
        return self.now["st"]

    def set_staging(self, iid, tma, pair=False):
        self.now["st"] = (bool(tma), bool(pair))

    def retile(self, iid, xc):
        self.now["xc"] = xc or 7

    def xc(self, iid):
        return self.now["xc"]

    def time_stages(self, n):
        self.calls += 1
        if n > 2:
            self.timed.append(self.now["st"] + (self.now["xc"],))
        return {"stage1": (1.0 if self.now["st"][0] else 2.0) + 0.01 * abs(self.now["xc"] - 8) - 1e-4 * self.calls}


def test_the_pair_flag_is_not_timed_again(monkeypatch, tmp_path):
    """Both flags of a TMA staging run the same kernels: they are timed once, and where the times are
    the same the flag stays off."""
    monkeypatch.setattr(engine, "Engine", _Fake)
    monkeypatch.setattr(autotune, "_device_name", lambda d: "fake")
    p_i = np.array([40, 24, 36, 2, 3, 5, 40 * 24 * 36, 5 * 40 * 24 * 36, 1, 1, 1, 4], np.int32)
    p_f = np.array([0, 0, 0, 0.2, 0.2, 0.2, 0.008, 0.02, 1, 1], float)
    res = autotune.tune("omega", p_i, p_f, "fp32c", cache=autotune.TuneCache(str(tmp_path / "t.json")), steps=4)
    timed = _Fake.made[-1].timed
    assert not any(k[1] for k in timed) and timed
    keys = {tuple(int(v) for v in k.split(",")) for k in res["timings"]}
    assert {k[:2] for k in keys} == {(1, 0), (1, 1), (0, 0)}
    assert all(res["timings"]["1,0,%d" % k[2]] == res["timings"]["1,1,%d" % k[2]] for k in keys if k[:2] == (1, 1))
    assert (res["tma"], res["pair"]) == (1, 0)

