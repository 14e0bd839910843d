"""The direct-mode kernels at the edges of their launch shapes, against the
FP64 oracle: slice counts that fill, leave over or split the vectors and
z-tiles (1 to 260 slices), channel counts around a warp's and a CTA's, footprints
of no cell to many cells, rays that all cross or mostly miss the image, and
launches small and large enough to split and not to split a ray's lines.
The bound is the direct mode's (2e-6 relative L2: FP32 products of FP64
weights rounded to FP32, summed in short chunks)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (XN, YN, slices, views, channels, off-centre, masked)
CASES = [
    (40, 40, 1, 24, 72, False, False),     # one slice, few warps: lines split
    (33, 27, 3, 17, 41, True, True),       # ragged, off centre
    (24, 24, 8, 30, 48, False, False),     # one 8-slice vector
    (24, 30, 12, 30, 48, False, True),     # three 4-slice vectors
    (30, 24, 40, 12, 49, True, False),     # five vectors: idle lanes in a warp
    (20, 20, 88, 12, 31, False, False),    # eleven vectors: two z-tiles
    (16, 18, 260, 9, 33, False, True),     # more vectors than a warp has lanes
    (64, 64, 16, 20, 12, False, False),    # 5 pixels a channel: wide footprints
    (12, 12, 16, 20, 240, False, False),   # 20 channels a pixel: narrow footprints, wide voxels
    (48, 40, 24, 700, 64, False, True),    # enough warps that lines are not split
    (3, 5, 9, 7, 2, False, False),         # fewer pixels and channels than any tile
    (160, 150, 9, 6, 900, True, True),     # windows of more values than a record holds
    (161, 160, 2, 6, 900, False, False),   # the same for one vector of slices
]


@pytest.mark.parametrize("XN,YN,Z,PN,U,off,masked", CASES)
@pytest.mark.parametrize("sat", ["direct", "hilo"])
def test_direct_shapes_match_oracle(XN, YN, Z, PN, U, off, masked, sat):
    import torch
    from aapm_lowdosectimagerecon_competition_b200 import configs, dd2, device
    from oracle import oracle as O
    assert torch.cuda.is_available()
    s = configs.scaled(configs.c2(SLN=Z), XN=XN, DNU=U, PN=PN)
    x0, y0, xds, yds = dd2.fan_geometry(s.sid, s.sdd, U, s.detCellWidth, s.detCntIdx)
    cx, cy = (np.float32(2.5 * s.dx), np.float32(-1.5 * s.dx)) if off else (np.float32(0), np.float32(0))
    rng = np.random.default_rng(XN + 7 * Z + PN)
    vol = (rng.random((YN, XN, Z)) * 0.04).astype(np.float32)
    prj = (rng.random((PN, U, Z)) - 0.3).astype(np.float32)
    mask = (rng.random((YN, XN)) < 0.9).astype(np.uint8) if masked else None
    a = s.angles()
    h = np.repeat(a[:, None], Z, 1)
    plan = device.Plan(x0, y0, U, xds, yds, s.detCntIdx, XN, YN, Z, PN, s.dx, mask=mask, imgXCenter=cx, imgYCenter=cy, sat=sat)
    angs = torch.from_numpy(a).cuda()
    rel = lambda g, e: float(np.linalg.norm((g - e).ravel()) / max(np.linalg.norm(e.ravel()), 1e-30))
    got = plan.proj(angs, torch.from_numpy(vol).cuda()).cpu().numpy()
    exp = O.proj(x0, y0, U, xds, yds, cx, cy, h, PN, XN, YN, Z, vol, s.dx, mask)
    assert rel(got, exp) < 2e-6
    for back, mode in (("adj", O.ADJ), ("ref", O.REF)):
        gb = plan.back(angs, torch.from_numpy(prj).cuda(), mode=back).cpu().numpy()
        eb = O.back(x0, y0, U, xds, yds, s.detCntIdx, cx, cy, h, PN, XN, YN, Z, prj, s.dx, mask, mode=mode)
        assert rel(gb, eb) < 2e-6, back
    plan.close()


@pytest.mark.parametrize("sat", ["hilo", "fp64"])
def test_mask_bytes_above_one_scale_the_image(sat):
    """A mask byte multiplies its voxel (MultiSlicesProjGPU.cu:202-209), also
    in the hi/lo mode, whose direct kernels take 0/1 masks only: a plan with
    other bytes keeps its tables, a solver its weights from them."""
    import torch
    from aapm_lowdosectimagerecon_competition_b200 import configs, dd2, device
    from oracle import oracle as O
    s = configs.scaled(configs.c2(SLN=9), XN=32, DNU=48, PN=24)
    s.numOfOS = 4
    x0, y0, xds, yds = dd2.fan_geometry(s.sid, s.sdd, s.DNU, s.detCellWidth, s.detCntIdx)
    rng = np.random.default_rng(3)
    vol = (rng.random((32, 32, 9)) * 0.04).astype(np.float32)
    mask = rng.integers(0, 3, (32, 32)).astype(np.uint8)
    rel = lambda g, e: float(np.linalg.norm((g - e).ravel()) / np.linalg.norm(e.ravel()))
    plan = device.Plan(x0, y0, s.DNU, xds, yds, s.detCntIdx, 32, 32, 9, s.PN, s.dx, mask=mask, sat=sat)
    y = plan.proj(torch.from_numpy(s.angles()).cuda(), torch.from_numpy(vol).cuda()).cpu().numpy()
    assert rel(y, O.proj(x0, y0, s.DNU, xds, yds, 0, 0, s.hangs(), s.PN, 32, 32, 9, vol, s.dx, mask)) < 2e-6
    plan.close()
    init = np.zeros_like(vol)
    xg = dd2.OSSART_AAPM(y, s.hangs(), init, s.conf(), 2, s.numOfOS, mask, 1, 1, sat=sat, back="ref")
    xo = O.ossart(x0, y0, s.DNU, xds, yds, s.detCntIdx, 0, 0, s.hangs(), s.PN, 32, 32, 9, y, init, s.dx, mask, 2,
                  s.numOfOS, 1, 1, O.REF)
    assert rel(xg, xo) < 1e-5


# (XN, YN, slices, views, channels, image centre in mm); with up to 4 slices the
# launch groups of equal lists run instead
REF_ROWS = [
    (40, 40, 7, 24, 72, 0.0),    # a warp's and a row group's remainders
    (33, 27, 6, 17, 41, 3.0),
    (3, 5, 5, 7, 12, 0.0),
    (12, 13, 6, 30, 48, 0.0),    # 30 mm pixels: angle steps beyond the series
    (64, 65, 5, 12, 900, 300.0),  # rays far off the fan, beyond 45 degrees
    (160, 9, 5, 12, 60, 0.0),
]


@pytest.mark.parametrize("XN,YN,Z,PN,U,cx", REF_ROWS)
@pytest.mark.parametrize("sat", ["hilo", "fp64"])
def test_per_slice_ref_backprojection_matches_oracle(XN, YN, Z, PN, U, cx, sat):
    """The slice-major REF backprojector (per-slice angle lists) at the edges
    of its row groups and of its angle steps, within the compensated modes'
    2e-6 of the FP64 oracle."""
    from aapm_lowdosectimagerecon_competition_b200 import configs, dd2
    from oracle import oracle as O
    s = configs.scaled(configs.c2(SLN=Z), XN=XN, DNU=U, PN=PN)
    x0, y0, xds, yds = dd2.fan_geometry(s.sid, s.sdd, U, s.detCellWidth, s.detCntIdx)
    a = s.angles()
    h = np.stack([(a + 0.37 * z).astype(np.float32) for z in range(Z)], 1)
    prj = np.random.default_rng(XN + PN).random((PN, U, Z)).astype(np.float32)
    args = (x0, y0, U, xds, yds, s.detCntIdx, np.float32(cx), np.float32(0), h, PN, XN, YN, Z, prj, s.dx)
    got, exp = dd2.MultiSlicesBackGPU(*args, sat=sat, back="ref"), O.back(*args, mode=O.REF)
    assert np.linalg.norm((got - exp).ravel()) < 2e-6 * np.linalg.norm(exp.ravel())


# runs of slices with one angle list each; few enough that the calls stay
# grouped (z-tiles of 8 or 32 slices against 1.45, 2.7 and 4.4 times the slices)
GROUPS = [(96, (31, 96)), (96, (3, 61, 96)), (26, (13, 26)), (8, (5, 8)), (7, (2, 7))]


@pytest.mark.parametrize("Z,ends", GROUPS)
@pytest.mark.parametrize("sat", ["direct", "hilo"])
def test_slice_groups_stage_their_own_slices(Z, ends, sat):
    """Calls whose slices fall into runs with different angle lists stage each
    run's vectors of slices only; runs that share a vector, begin or end inside
    one, and few slices, against the oracle.  A second call on other inputs
    meets what the first left in the staging buffers."""
    import torch
    from aapm_lowdosectimagerecon_competition_b200 import configs, dd2, device
    from oracle import oracle as O
    XN, YN, PN, U = 30, 26, 11, 40
    s = configs.scaled(configs.c2(SLN=Z), XN=XN, DNU=U, PN=PN)
    x0, y0, xds, yds = dd2.fan_geometry(s.sid, s.sdd, U, s.detCellWidth, s.detCntIdx)
    a = s.angles()
    h = np.stack([(a + 0.21 * sum(z >= e for e in ends)).astype(np.float32) for z in range(Z)], 1)
    mask = np.ones((YN, XN), np.uint8)
    mask[:, :2] = 0
    plan = device.Plan(x0, y0, U, xds, yds, s.detCntIdx, XN, YN, Z, PN, s.dx, mask=mask, sat=sat)
    hd = torch.from_numpy(np.ascontiguousarray(h)).cuda()
    rel = lambda g, e: float(np.linalg.norm((g - e).ravel()) / np.linalg.norm(e.ravel()))
    for seed in (1, 2):
        rng = np.random.default_rng(seed)
        vol = (rng.random((YN, XN, Z)) * 0.04).astype(np.float32)
        prj = (rng.random((PN, U, Z)) - 0.3).astype(np.float32)
        got = plan.proj(hd, torch.from_numpy(vol).cuda()).cpu().numpy()
        assert rel(got, O.proj(x0, y0, U, xds, yds, 0, 0, h, PN, XN, YN, Z, vol, s.dx, mask)) < 2e-6
        for back, mode in (("adj", O.ADJ), ("ref", O.REF)):
            gb = plan.back(hd, torch.from_numpy(prj).cuda(), mode=back).cpu().numpy()
            eb = O.back(x0, y0, U, xds, yds, s.detCntIdx, 0, 0, h, PN, XN, YN, Z, prj, s.dx, mask, mode=mode)
            assert rel(gb, eb) < 2e-6, back
    plan.close()


@pytest.mark.parametrize("offset", [0, 4, 1])
def test_image_alignment(offset):
    """An image 16 but not 32 bytes aligned is read in vectors of 4 slices
    instead of 8, one that is neither is staged first; 16 and 72 slices (one
    z-tile and two), against the oracle."""
    import torch
    from aapm_lowdosectimagerecon_competition_b200 import configs, dd2, device
    from oracle import oracle as O
    for Z in (16, 72):
        XN, YN, PN, U = 30, 26, 13, 40
        s = configs.scaled(configs.c2(SLN=Z), XN=XN, DNU=U, PN=PN)
        x0, y0, xds, yds = dd2.fan_geometry(s.sid, s.sdd, U, s.detCellWidth, s.detCntIdx)
        vol = (np.random.default_rng(Z).random((YN, XN, Z)) * 0.04).astype(np.float32)
        buf = torch.zeros(vol.size + 8, device="cuda")
        img = buf[offset:offset + vol.size].view(YN, XN, Z)
        img.copy_(torch.from_numpy(vol))
        assert img.data_ptr() % 32 == 4 * offset
        plan = device.Plan(x0, y0, U, xds, yds, s.detCntIdx, XN, YN, Z, PN, s.dx, sat="direct")
        got = plan.proj(torch.from_numpy(s.angles()).cuda(), img).cpu().numpy()
        plan.close()
        exp = O.proj(x0, y0, U, xds, yds, 0, 0, s.hangs(), PN, XN, YN, Z, vol, s.dx)
        assert np.linalg.norm((got - exp).ravel()) < 2e-6 * np.linalg.norm(exp.ravel())


# one z-tile of 16 vectors, and two of 8 for an image that L2 does not hold
@pytest.mark.parametrize("N,PN,U", [(96, 9, 64), (512, 5, 48)])
def test_many_slices_in_one_tile_or_two(N, PN, U):
    import torch
    from aapm_lowdosectimagerecon_competition_b200 import configs, dd2, device
    from oracle import oracle as O
    Z = 128
    s = configs.scaled(configs.c2(SLN=Z), XN=N, DNU=U, PN=PN)
    x0, y0, xds, yds = dd2.fan_geometry(s.sid, s.sdd, U, s.detCellWidth, s.detCntIdx)
    vol = (np.random.default_rng(N).random((N, N, Z), dtype=np.float32) * np.float32(0.04))
    plan = device.Plan(x0, y0, U, xds, yds, s.detCntIdx, N, N, Z, PN, s.dx, sat="direct")
    got = plan.proj(torch.from_numpy(s.angles()).cuda(), torch.from_numpy(vol).cuda()).cpu().numpy()
    plan.close()
    exp = O.proj(x0, y0, U, xds, yds, 0, 0, s.hangs(), PN, N, N, Z, vol, s.dx)
    assert np.linalg.norm((got - exp).ravel()) < 2e-6 * np.linalg.norm(exp.ravel())
