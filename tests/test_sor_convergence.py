"""The SOR's convergence checks in the register kernels (rgbd-flow_b200/csrc/sor_regs.cuh, level_bands.cuh): the
iteration they stop at, the change they report and the flow are the tile SOR's, bit for bit."""
import numpy as np
import pytest

import rgbdflow as rf
from test_resident_tiles import pair


def solve(ctx, W, H, seed, **over):
    p = pair(W, H, seed)
    prm = rf.benchmark_params(W, **over)
    prm.min_width = max(2, W // 3)
    cam = rf.CameraParams.make(W, H, p["cam"].f, p["cam"].cx, p["cam"].cy)
    flow, st = ctx.scene_flow_two_frames(cam, p["bgr1"], p["depth1"], p["bgr2"], p["depth2"], prm)
    return flow, st.summary(), np.array(st.sor_maxdiff)


def assert_same(a, b):
    assert a[1] == b[1]
    np.testing.assert_array_equal(a[2], b[2])
    np.testing.assert_array_equal(a[0], b[0])


@pytest.mark.gpu
@pytest.mark.parametrize("tol", [1e-2, 3e-3, 1e-3, 3e-4, 1e-4])
@pytest.mark.parametrize("W,H", [(117, 93), (64, 48)])
def test_unclamped_step_stops_at_the_tile_sors_check(ctx, monkeypatch, W, H, tol):
    """An unbounded step, several iterations between exchanges, checks that a level passes inside its schedule: a
    check is of its own iteration's change, not of the largest since the exchange before."""
    over = dict(max_flow_step=float("inf"), n_outer=3, n_sor=200, sor_check_period=5, sor_tol=tol)
    monkeypatch.setenv("RGBDFLOW_RESIDENT_K", "5")
    regs = solve(ctx, W, H, 5, **over)
    monkeypatch.setenv("RGBDFLOW_SOR_LEVEL", "0")
    tile = solve(ctx, W, H, 5, **over)
    assert any(0 < n < 200 for level in tile[1] for n in level[3])
    assert_same(regs, tile)


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,omega,step,n_sor", [
    (117, 93, 1.9, float("inf"), 100), (117, 93, 1.9, 3e38, 100), (64, 48, 1.9, float("inf"), 400), (64, 48, 1.9, 3e38, 100),
    (200, 150, 1.9, 3e38, 400), (200, 150, 4.0, float("inf"), 100), (200, 150, 4.0, 1e37, 100)])
def test_unknowns_that_overflow_do_so_as_the_tile_sors(ctx, monkeypatch, W, H, omega, step, n_sor):
    """A relaxation that diverges until unknowns are infinite or NaN, on levels that end inside a tile and at a
    tile's last column: nothing outside the image takes part."""
    over = dict(max_flow_step=step, omega=omega, n_outer=2, n_sor=n_sor, sor_tol=0.0)
    monkeypatch.setenv("RGBDFLOW_RESIDENT_K", "5")
    regs = solve(ctx, W, H, 5, **over)
    monkeypatch.setenv("RGBDFLOW_SOR_LEVEL", "0")
    tile = solve(ctx, W, H, 5, **over)
    assert np.nanmax(np.abs(tile[0])) > 1e30
    assert_same(regs, tile)
