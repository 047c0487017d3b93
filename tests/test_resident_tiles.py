"""The tiles of the register-resident SOR (rgbd-flow_b200/csrc/sor_regs.cuh) and the rule for the iterations
between its exchanges (resident_k in pipeline.cuh), checked on the CPU, and on a GPU the flow against the
tile SOR at the sizes where the tiling can go wrong.

tests/cpp/resident_tiles_check.cu walks every tile of levels at the edges of the tiling for every K: each
pixel is owned by one tile, owned pixels are 2 K pixels inside their region, and every other pixel of a
region is one that a neighbouring tile sends.  No kernel is launched there.
"""
import os
import shutil
import subprocess

import numpy as np
import pytest

import rgbdflow as rf
import synthetic as syn

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc to compile the pipeline header")
def test_resident_tiles_cover_the_level(tmp_path):
    exe = str(tmp_path / "resident_tiles_check")
    subprocess.run(["nvcc", "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "-o", exe,
                    os.path.join(HERE, "cpp", "resident_tiles_check.cu")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.splitlines()[-1].startswith("ok resident tiles")


def pair(W, H, seed):
    return syn.make_pair(W=W, H=H, f=0.8 * W, cx=(W - 1) / 2, cy=(H - 1) / 2, n_patches=2, hole_frac=0.04, seed=seed)


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,K,n_inner,n_sor", [
    (64, 48, 0, 1, 30), (65, 48, 0, 2, 30), (64, 49, 5, 1, 27), (109, 77, 5, 1, 30), (117, 93, 1, 2, 55), (160, 120, 2, 1, 0),
    (160, 120, 3, 1, 4), (40, 130, 4, 1, 30), (331, 243, 0, 1, 60)])
def test_register_sor_agrees_with_tile_sor_bitwise(ctx, monkeypatch, W, H, K, n_inner, n_sor):
    """Levels at the edges of the register kernels' tiling, K iterations between exchanges (0: the rule's),
    iteration counts that end with, before and after a convergence check: the tile SOR's flow and executed
    schedule, bit for bit."""
    p = pair(W, H, W + H)
    prm = rf.benchmark_params(W, n_inner=n_inner, n_sor=n_sor)
    prm.min_width = max(2, W // 3)
    cam = rf.CameraParams.make(W, H, p["cam"].f, p["cam"].cx, p["cam"].cy)
    args = (cam, p["bgr1"], p["depth1"], p["bgr2"], p["depth2"], prm)
    monkeypatch.setenv("RGBDFLOW_RESIDENT_K", str(K))
    regs, st_regs = ctx.scene_flow_two_frames(*args)
    monkeypatch.setenv("RGBDFLOW_SOR_LEVEL", "0")
    tile, st_tile = ctx.scene_flow_two_frames(*args)
    assert st_tile.summary() == st_regs.summary()
    np.testing.assert_array_equal(tile, regs)


@pytest.mark.gpu
@pytest.mark.parametrize("step", [float("inf"), 1e-3])
def test_register_sor_keeps_pixels_outside_the_image_still(ctx, monkeypatch, step):
    """An unbounded step (no clamp: unknowns may overflow) and a tight one, on a level that ends inside a tile."""
    p = pair(101, 67, 5)
    prm = rf.benchmark_params(101, max_flow_step=step, n_outer=3)
    prm.min_width = 40
    cam = rf.CameraParams.make(101, 67, p["cam"].f, p["cam"].cx, p["cam"].cy)
    args = (cam, p["bgr1"], p["depth1"], p["bgr2"], p["depth2"], prm)
    regs = ctx.scene_flow_two_frames(*args, stats=False)
    monkeypatch.setenv("RGBDFLOW_SOR_LEVEL", "0")
    np.testing.assert_array_equal(ctx.scene_flow_two_frames(*args, stats=False), regs)


@pytest.mark.gpu
def test_register_sor_batch_larger_than_the_device(ctx, monkeypatch):
    """Ragged pairs that together need several times the device's CTAs: each equals its solve alone."""
    sizes = [(320, 240), (200, 150), (320, 240), (90, 70), (640, 480), (501, 377), (320, 240), (160, 120)]
    pairs, prm = [], rf.benchmark_params(640, n_outer=4)
    for i, (W, H) in enumerate(sizes):
        p = pair(W, H, 70 + i)
        pairs.append(dict(W=W, H=H, cam=rf.CameraParams.make(W, H, p["cam"].f, p["cam"].cx, p["cam"].cy), bgr1=p["bgr1"],
                          depth1=p["depth1"], bgr2=p["bgr2"], depth2=p["depth2"]))
    batch = ctx.scene_flow_batch(pairs, prm, stats=False)
    monkeypatch.setenv("RGBDFLOW_SOR_LEVEL", "0")
    for q, b in zip(pairs, batch):
        np.testing.assert_array_equal(ctx.scene_flow_two_frames(q["cam"], q["bgr1"], q["depth1"], q["bgr2"], q["depth2"], prm,
                                                                stats=False), b)


@pytest.mark.gpu
@pytest.mark.parametrize("W,H", [(608, 456), (200, 152)])
def test_listing_names_the_exchanges_that_run(ctx, W, H):
    """The iterations between exchanges at which the level's tiles fit the device, not the most there may be."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    p = pair(W, H, 1)
    prm = rf.benchmark_params(W, n_outer=1)
    prm.min_width = W
    cam = rf.CameraParams.make(W, H, p["cam"].f, p["cam"].cx, p["cam"].cy)
    ctx.scene_flow_two_frames(cam, p["bgr1"], p["depth1"], p["bgr2"], p["depth2"], prm, stats=False)
    tiles = lambda K: -(-(W - 4 * K) // (64 - 4 * K)) * -(-(H - 4 * K) // (48 - 4 * K))  # noqa: E731
    K = max(k for k in range(1, 6) if tiles(k) <= sms)
    assert "f%dx%d*1, registers, exchange every %d;" % (W, H, K) in rf.autotune_describe(0)
