"""The autotuner's records, with the measurement replaced by one whose later
candidates always come out faster."""
import numpy as np
import pytest
import torch

from aapm_lowdosectimagerecon_competition_b200 import serve


class _Plan:
    def __init__(self, *a, **k):
        pass

    def proj(self, angs, vol, out=None):
        return vol

    def back(self, angs, prj, out=None, mode=None):
        return out

    def close(self):
        pass


@pytest.fixture
def lib(monkeypatch):
    ms = iter(np.linspace(100.0, 1.0, 200))

    class Event:
        def __init__(self, **k):
            pass

        def record(self):
            pass

        def elapsed_time(self, other):
            return float(next(ms))

    monkeypatch.setattr(serve, "Plan", _Plan)
    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda *a: None)
    lib = serve.load()
    yield lib
    for zb in (10, 16):
        lib.ddfan_tune_set_zl(zb, 0)
        lib.ddfan_tune_set_nz(zb, 0)


@pytest.mark.parametrize("sat", ["hilo", "direct"])
def test_modes_without_tables_record_no_width(lib, sat):
    width = {zb: lib.ddfan_tune_get_zl(zb) for zb in (10, 16)}
    t = serve.TileTuner(sat=sat)
    for zb in (10, 16):
        zl, nz = t.tune(N=8, Z=4 * zb, P=4, device=torch.device("cpu"), reps=1)
        assert zl == width[zb] and lib.ddfan_tune_get_zl(zb) == width[zb]
        assert nz == (lib.ddfan_tune_get_nz(zb) if sat == "direct" else 0)


def test_table_modes_record_the_fastest_width(lib):
    t = serve.TileTuner(sat="fp32")
    assert t.tune(N=8, Z=40, P=4, device=torch.device("cpu"), reps=1) == [1, 0]
    assert lib.ddfan_tune_get_zl(10) == 1
