"""Infinite and NaN sinogram values in the backprojectors without tables: they
reach the voxels whose footprints hold them, in the slices that hold them, and
no others."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (side, slices, views, channels, masked): one slice, one vector, several, and
# launches of many and few warps
CASES = [(40, 1, 24, 72, True), (40, 4, 24, 72, False), (41, 8, 40, 60, True), (40, 24, 24, 72, True),
         (96, 40, 150, 96, False), (160, 9, 6, 900, True)]


@pytest.mark.parametrize("N,Z,PN,U,masked", CASES)
@pytest.mark.parametrize("back", ["adj", "ref"])
@pytest.mark.parametrize("sat", ["direct", "hilo"])
def test_nonfinite_channels_stay_in_their_footprints(N, Z, PN, U, masked, back, sat):
    import torch
    from aapm_lowdosectimagerecon_competition_b200 import configs, dd2, device
    from oracle import oracle as O
    s = configs.scaled(configs.c2(SLN=Z), XN=N, DNU=U, PN=PN)
    x0, y0, xds, yds = dd2.fan_geometry(s.sid, s.sdd, U, s.detCellWidth, s.detCntIdx)
    rng = np.random.default_rng(N + Z)
    prj = (rng.random((PN, U, Z)) - 0.3).astype(np.float32)
    mask = (rng.random((N, N)) < 0.8).astype(np.uint8) if masked else None
    # (view, channel, slice, value), one of them on the last channel
    bad = [(1, U // 2, 0, np.inf), (PN - 1, U // 3, Z - 1, np.nan), (PN // 2, U - 1, Z // 2, -np.inf)]
    clean, hit = prj.copy(), np.zeros_like(prj)
    for v, u, z, x in bad:
        prj[v, u, z], clean[v, u, z], hit[v, u, z] = x, 0.0, 1.0
    angs = torch.from_numpy(s.angles()).cuda()
    plan = device.Plan(x0, y0, U, xds, yds, s.detCntIdx, N, N, Z, PN, s.dx, mask=mask, sat=sat)
    got = plan.back(angs, torch.from_numpy(prj).cuda(), mode=back).cpu().numpy()
    ref = plan.back(angs, torch.from_numpy(clean).cuda(), mode=back).cpu().numpy()
    plan.close()
    h = np.repeat(s.angles()[:, None], Z, 1)
    part = np.abs(O.back(x0, y0, U, xds, yds, s.detCntIdx, 0, 0, h, PN, N, N, Z, hit, s.dx, mask,
                         mode=O.ADJ if back == "adj" else O.REF))
    outside, inside = part < 1e-9, part > 1e-4
    assert inside.any() and not np.isfinite(got[inside]).any()
    assert np.isfinite(got[outside]).all()
    assert np.abs(got - ref)[outside].max() <= 1e-5 * np.abs(ref).max()
    if masked:
        assert not got[mask == 0].any()
