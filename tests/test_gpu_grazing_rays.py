"""Rays that only graze the masked image: their row sums, one or two small parts
of cells, divide the residual, so they must be right relative to themselves.

A part is a whole number of 2^-32 cells from boundary positions rounded twice
(the line's constant and the sum, 2^-33 each): off by at most 2^-31 cells for a
part between two boundaries, times at most 3.5 (ray weight 1.42 over a footprint
of 0.4 cells) in at most four parts of a short row: 6.5e-9 pixels.  On top come
the roundings of its float factors, eight of 2^-24: 4.8e-7 of the row sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scan(configs, N, P, U, Z):
    s = configs.c2(SLN=Z)
    s.XN = s.YN = N
    s.dx = np.float32(0.7 * 512.0 / N)
    s.DNU, s.PN = U, P
    s.detCellWidth, s.detCntIdx = np.float32(1.2858 * 736.0 / U), np.float32((U + 1) / 2)
    return s


# slices: the kernels of one slice, of up to 4 and of more than 8
@pytest.mark.parametrize("Z,sat", [(1, "direct"), (4, "direct"), (24, "direct"), (24, "hilo")])
@pytest.mark.parametrize("N,P,U", [(423, 883, 522), (241, 377, 544), (179, 432, 856)])
def test_short_row_sums(N, P, U, Z, sat):
    import torch
    from aapm_lowdosectimagerecon_competition_b200 import configs, dd2, device
    from oracle import oracle as O
    s = _scan(configs, N, P, U, Z)
    x0, y0, xds, yds = dd2.fan_geometry(s.sid, s.sdd, U, s.detCellWidth, s.detCntIdx)
    a, mask = s.angles(), s.circular_mask()
    plan = device.Plan(x0, y0, U, xds, yds, s.detCntIdx, N, N, Z, P, s.dx, mask=mask, sat=sat)
    got = plan.proj(torch.from_numpy(a).cuda(), torch.ones((N, N, Z), device="cuda")).cpu().numpy().astype(np.float64)
    plan.close()
    exp = O.proj(x0, y0, U, xds, yds, 0, 0, a[:, None], P, N, N, 1, np.ones((N, N, 1), np.float32), s.dx, mask)
    short = (exp[:, :, 0] > 0) & (exp[:, :, 0] < 0.01)
    assert short.any()
    err = np.abs(got - exp)[short]
    assert (err <= 5e-7 * exp[short] + 6.5e-9).all(), float((err / exp[short]).max())


@pytest.mark.parametrize("N,P,U,subsets,Z,sat", [(241, 1508, 544, 5, 1, "direct"), (423, 883, 522, 8, 4, "direct"),
                                                 (241, 1508, 544, 5, 9, "hilo")])
def test_solves_with_grazing_rays(N, P, U, subsets, Z, sat):
    """One iteration against the FP64 oracle.  Solves without such a ray are
    0.8 to 1.5e-7 off; the bound is twice the largest."""
    import torch
    from aapm_lowdosectimagerecon_competition_b200 import configs, dd2, device
    from oracle import oracle as O
    s = _scan(configs, N, P, U, Z)
    x0, y0, xds, yds = dd2.fan_geometry(s.sid, s.sdd, U, s.detCellWidth, s.detCntIdx)
    mask = s.circular_mask()
    y = O.proj(x0, y0, U, xds, yds, 0, 0, s.hangs(), P, N, N, Z, configs.phantom(s), s.dx, mask)
    y = np.ascontiguousarray(configs.poisson_log(y, 1.5e5, seed=5), np.float32)
    sv = device.OSSART(x0, y0, U, xds, yds, s.detCntIdx, s.hangs(), N, N, Z, s.dx, mask=mask, numOfOS=subsets, useFISTA=1,
                       nonneg=1, sat=sat, back="ref")
    sv.set_sinogram(torch.from_numpy(y).cuda())
    sv.set_image(torch.zeros((N, N, Z), device="cuda"))
    sv.iterate(1)
    got = sv.image().cpu().numpy()
    sv.close()
    exp = O.ossart(x0, y0, U, xds, yds, s.detCntIdx, 0, 0, s.hangs(), P, N, N, Z, y, np.zeros((N, N, Z), np.float32), s.dx, mask,
                   1, subsets, 1, 1, O.REF)
    assert np.linalg.norm((got - exp).ravel()) < 3e-7 * np.linalg.norm(exp.ravel())


@pytest.mark.parametrize("N,P,U,back", [(200, 1000, 800, "adj"), (241, 754, 544, "adj"), (241, 754, 544, "ref")])
def test_per_slice_solves_with_grazing_rays(N, P, U, back):
    """The same with an angle list per slice (the slice-major kernels), whose row
    sums come from slice 0's list, so the rays of other slices are divided by
    sums that are not theirs and the image at the disk's edge is large.  The
    kernels' own FP32 positions leave 1.6 to 3.6e-7 at eight sizes; with row sums
    from tables it was up to 9e-7."""
    import torch
    from aapm_lowdosectimagerecon_competition_b200 import configs, dd2, device
    from oracle import oracle as O
    Z = 6
    s = _scan(configs, N, P, U, Z)
    x0, y0, xds, yds = dd2.fan_geometry(s.sid, s.sdd, U, s.detCellWidth, s.detCntIdx)
    mask = s.circular_mask()
    h = np.stack([(s.angles() + np.float32(0.37 * z)).astype(np.float32) for z in range(Z)], 1)
    y = O.proj(x0, y0, U, xds, yds, 0, 0, h, P, N, N, Z, configs.phantom(s), s.dx, mask)
    y = np.ascontiguousarray(configs.poisson_log(y, 1.5e5, seed=5), np.float32)
    sv = device.OSSART(x0, y0, U, xds, yds, s.detCntIdx, h, N, N, Z, s.dx, mask=mask, numOfOS=5, useFISTA=1, nonneg=1, back=back)
    sv.set_sinogram(torch.from_numpy(y).cuda())
    sv.set_image(torch.zeros((N, N, Z), device="cuda"))
    sv.iterate(1)
    got = sv.image().cpu().numpy()
    sv.close()
    exp = O.ossart(x0, y0, U, xds, yds, s.detCntIdx, 0, 0, h, P, N, N, Z, y, np.zeros((N, N, Z), np.float32), s.dx, mask, 1, 5,
                   1, 1, O.REF if back == "ref" else O.ADJ)
    assert np.linalg.norm((got - exp).ravel()) < 4e-7 * np.linalg.norm(exp.ravel())
