"""Device-byte estimates: never below what a plan or solver allocates, and the
serving engine's admission figure for each kind of request."""
from types import SimpleNamespace

import numpy as np
import pytest

from aapm_lowdosectimagerecon_competition_b200 import configs, dd2, serve
from aapm_lowdosectimagerecon_competition_b200._lib import SAT_MODES, load


def _table_floor(N, Z, P, U):
    """Two image tables and a sinogram table of 48-byte hi/lo cells of 4 slices."""
    ZB = (Z + 3) // 4
    return 48 * ZB * (2 * N * N + P * (U + 1))


@pytest.mark.parametrize("N,Z,P,U", [(64, 1, 30, 72), (256, 16, 30, 736), (512, 128, 96, 736)])
def test_hilo_estimates_hold_the_tables(N, Z, P, U):
    lib, m = load(), SAT_MODES
    assert lib.ddfan_plan_estimate_bytes(N, N, U, Z, P, m["hilo"]) >= _table_floor(N, Z, P, U)
    assert lib.ddfan_ossart_estimate_bytes(N, N, U, Z, 8 * P, 8, m["hilo"]) >= _table_floor(N, Z, P, U)
    for sat in ("fp32", "hilo", "fp64", "direct"):
        assert lib.ddfan_plan_estimate_bytes(0, N, U, Z, P, m[sat]) == 0
        assert lib.ddfan_ossart_estimate_bytes(N, N, U, Z, 7, 8, m[sat]) == 0


def test_engine_admits_by_the_mode_a_request_runs_in():
    s = configs.scaled(configs.c2(SLN=9), XN=64, DNU=72, PN=48)
    s.numOfOS = 4
    est = lambda sat: float(load().ddfan_ossart_estimate_bytes(64, 64, 72, 9, 48, 4, SAT_MODES[sat]))
    assert est("direct") < est("hilo")
    per_slice = configs.scaled(configs.c2(SLN=9), XN=64, DNU=72, PN=48)
    per_slice.numOfOS = 4
    h = s.hangs() + 0.1 * np.arange(9, dtype=np.float32)
    per_slice.hangs = lambda: h
    engine = lambda sat: SimpleNamespace(sat=sat)
    got = lambda sat, mask, scan=s: serve.Engine.estimate(engine(sat), SimpleNamespace(scan=scan, mask=mask))
    disk = s.circular_mask()
    assert got("hilo", disk) == got("hilo", None) == est("direct")
    assert got("hilo", 2 * disk) == est("hilo")
    assert got("hilo", disk, per_slice) == est("hilo")
    assert got("direct", disk) == est("direct") and got("fp64", disk) == est("fp64")


@pytest.mark.gpu
@pytest.mark.parametrize("sat", ["fp32", "hilo", "fp64", "direct"])
@pytest.mark.parametrize("scale", [None, 1, 2])
@pytest.mark.parametrize("Z", [1, 6, 33])
def test_estimates_cover_what_is_allocated(Z, scale, sat):
    from aapm_lowdosectimagerecon_competition_b200 import device
    s = configs.scaled(configs.c2(SLN=Z), XN=96, DNU=120, PN=60)
    x0, y0, xds, yds = dd2.fan_geometry(s.sid, s.sdd, s.DNU, s.detCellWidth, s.detCntIdx)
    mask = None if scale is None else (scale * s.circular_mask()).astype(np.uint8)
    lib = load()
    plan = device.Plan(x0, y0, s.DNU, xds, yds, s.detCntIdx, 96, 96, Z, 60, s.dx, mask=mask, sat=sat)
    assert plan.device_bytes <= lib.ddfan_plan_estimate_bytes(96, 96, s.DNU, Z, 60, SAT_MODES[sat])
    plan.close()
    sv = device.OSSART(x0, y0, s.DNU, xds, yds, s.detCntIdx, s.hangs(), 96, 96, Z, s.dx, mask=mask, numOfOS=4, sat=sat)
    assert sv.device_bytes <= lib.ddfan_ossart_estimate_bytes(96, 96, s.DNU, Z, 60, 4, SAT_MODES[sat])
    sv.close()
