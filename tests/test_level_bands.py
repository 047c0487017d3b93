"""The levels that are solved in one launch (k_level_bands, rgbd-flow_b200/csrc/level_bands.cuh): its row bands
and the rule for its CTAs on the CPU, and on a GPU the flow against the tile SOR's launches at the sizes where
a band can go wrong.
"""
import os
import shutil
import subprocess

import numpy as np
import pytest

import rgbdflow as rf
from test_resident_tiles import pair

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc to compile the pipeline header")
def test_level_bands_cover_the_level(tmp_path):
    exe = str(tmp_path / "level_bands_check")
    subprocess.run(["nvcc", "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "-o", exe,
                    os.path.join(HERE, "cpp", "level_bands_check.cu")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.splitlines()[-1].startswith("ok level bands")


def args(W, H, seed, **over):
    p = pair(W, H, seed)
    prm = rf.benchmark_params(W, **over)
    prm.min_width = max(2, W // 3)
    cam = rf.CameraParams.make(W, H, p["cam"].f, p["cam"].cx, p["cam"].cy)
    return cam, p["bgr1"], p["depth1"], p["bgr2"], p["depth2"], prm


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,over", [
    (20, 15, {}), (33, 31, dict(n_inner=2)), (32, 33, dict(n_sor=27)), (75, 56, dict(n_sor=55)), (101, 75, dict(n_inner=3, n_sor=25)),
    (160, 120, {}), (159, 119, dict(fixed_schedule=1, n_outer=2)), (24, 400, {}), (400, 24, dict(n_inner=2)), (64, 48, dict(n_sor=0)),
    (90, 70, dict(max_flow_step=float("inf"), n_outer=3)), (90, 70, dict(storage=rf.STORE_FP16)),
    (90, 70, dict(regularization=rf.REG_HPB, n_outer=3))], ids=str)
def test_level_bands_agree_with_tile_sor_bitwise(ctx, monkeypatch, W, H, over):
    a = args(W, H, W + H, **over)
    bands, st_bands = ctx.scene_flow_two_frames(*a)
    monkeypatch.setenv("RGBDFLOW_SOR_LEVEL", "0")
    tile, st_tile = ctx.scene_flow_two_frames(*a)
    assert st_tile.summary() == st_bands.summary()
    np.testing.assert_array_equal(tile, bands)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 8, 17, 40])
def test_level_bands_of_a_ragged_batch(ctx, monkeypatch, n):
    """More items, fewer CTAs each (down to one, and back to the launches of their own): each pair's solve alone."""
    sizes = [(48, 36), (37, 41), (40, 30), (33, 20)]
    prm = rf.benchmark_params(48, n_outer=3)
    prm.min_width = 15
    pairs = []
    for i in range(n):
        W, H = sizes[i % len(sizes)]
        cam, b1, d1, b2, d2, _ = args(W, H, 10 + i)
        pairs.append(dict(W=W, H=H, cam=cam, bgr1=b1, depth1=d1, bgr2=b2, depth2=d2))
    batch = ctx.scene_flow_batch(pairs, prm, stats=False)
    monkeypatch.setenv("RGBDFLOW_SOR_LEVEL", "0")
    for q, b in list(zip(pairs, batch))[:9]:
        np.testing.assert_array_equal(ctx.scene_flow_two_frames(q["cam"], q["bgr1"], q["depth1"], q["bgr2"], q["depth2"], prm,
                                                                stats=False), b)


@pytest.mark.gpu
def test_no_outer_iterations_launch_nothing(ctx, monkeypatch):
    a = args(160, 120, 7, n_outer=0)
    bands = ctx.scene_flow_two_frames(*a, stats=False)
    launches = ctx.last_launch_count()
    monkeypatch.setenv("RGBDFLOW_SOR_LEVEL", "0")
    np.testing.assert_array_equal(ctx.scene_flow_two_frames(*a, stats=False), bands)
    assert ctx.last_launch_count() == launches


@pytest.mark.gpu
def test_profile_counts_the_linearisation_of_its_own_launches(ctx):
    """320x240 is linearised by k_linearize, the levels below it inside k_level_bands, in the SOR's time."""
    a = args(320, 240, 7)
    a[-1].min_width = 20
    ctx.profile(1)
    _, st = ctx.scene_flow_two_frames(*a)
    kst = ctx.profile_read()
    ctx.profile(0)
    assert kst["linearize"][2] == 320 * 240 * 128.0 * st.outer_iters[0]
