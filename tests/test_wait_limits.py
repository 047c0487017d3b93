"""Waits between thread blocks that run out: the call that waited reports it, and the context stays usable.

RGBDFLOW_WAIT_POLLS=0 makes every such wait of the SOR give up at once.  Nothing hangs and no access leaves its
buffers: the blocks go on with what they have, or return.
"""
import os
import shutil
import subprocess

import numpy as np
import pytest

import rgbdflow as rf
from test_resident_tiles import pair

HERE = os.path.dirname(os.path.abspath(__file__))
TIMEOUT = -5  # RGBDFLOW_ERR_TIMEOUT


@pytest.mark.gpu
@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc to compile the probe")
def test_a_wait_lost_by_any_thread_is_reported(tmp_path):
    exe = str(tmp_path / "lost_wait_check")
    subprocess.run(["nvcc", "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "-o", exe,
                    os.path.join(HERE, "cpp", "lost_wait_check.cu")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc to compile the pipeline header")
def test_resident_waits_outlast_the_items_queued_before(tmp_path):
    exe = str(tmp_path / "resident_waits_check")
    subprocess.run(["nvcc", "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "-o", exe,
                    os.path.join(HERE, "cpp", "resident_waits_check.cu")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def solve(ctx, W=160, H=120):
    p = pair(W, H, 3)
    cam = rf.CameraParams.make(W, H, p["cam"].f, p["cam"].cx, p["cam"].cy)
    return ctx.scene_flow_two_frames(cam, p["bgr1"], p["depth1"], p["bgr2"], p["depth2"], rf.benchmark_params(W), stats=False)


def assert_reported_once(ctx, monkeypatch):
    before = solve(ctx)
    monkeypatch.setenv("RGBDFLOW_WAIT_POLLS", "0")
    with pytest.raises(rf.RgbdFlowError) as e:
        solve(ctx)
    assert e.value.code == TIMEOUT
    monkeypatch.delenv("RGBDFLOW_WAIT_POLLS")
    ctx.synchronize()
    np.testing.assert_array_equal(solve(ctx), before)


@pytest.mark.gpu
def test_level_bands_report_lost_waits(ctx, monkeypatch):
    assert_reported_once(ctx, monkeypatch)


@pytest.mark.gpu
@pytest.mark.parametrize("K", [1, 5])
def test_resident_sor_reports_lost_waits(ctx, monkeypatch, K):
    monkeypatch.setenv("RGBDFLOW_RESIDENT_K", str(K))
    assert_reported_once(ctx, monkeypatch)


@pytest.mark.gpu
def test_served_batches_report_lost_waits(ctx, monkeypatch):
    """A server captures its streams' batches ahead of their first launch: those carry the status too."""
    monkeypatch.setenv("RGBDFLOW_WAIT_POLLS", "0")
    W, H = 160, 120
    frames = [pair(W, H, 90 + k) for k in range(4)]
    cam = rf.CameraParams.make(W, H, frames[0]["cam"].f, frames[0]["cam"].cx, frames[0]["cam"].cy)
    srv = rf.Server(ctx, rf.benchmark_params(W), max_streams=2, max_batch=2, warm_start=False)
    status = []
    try:
        for k, f in enumerate(frames):
            srv.submit(0, k, cam, f["bgr1"], f["depth1"])
            while srv.pending():
                status += [r[5] for r in srv.step(wait=True)]
    finally:
        srv.close()
    assert status == [TIMEOUT] * 3


@pytest.mark.gpu
@pytest.mark.parametrize("K", ["0", "2"])
def test_a_lost_wait_of_the_allocation_free_solve_is_in_its_flow(monkeypatch, K):
    import torch
    W, H = 160, 120
    p = pair(W, H, 3)
    dev = {k: torch.from_numpy(np.ascontiguousarray(p[k])).cuda() for k in ("bgr1", "depth1", "bgr2", "depth2")}
    q = dict(dev, W=W, H=H, cam=rf.CameraParams.make(W, H, p["cam"].f, p["cam"].cx, p["cam"].cy),
             out=torch.zeros((H, W, 3), dtype=torch.float32, device="cuda"))
    st = torch.cuda.Stream()

    def flow():
        rf.scene_flow_noalloc(q, rf.benchmark_params(W), stream=st)
        st.synchronize()
        return q["out"].cpu().numpy()

    monkeypatch.setenv("RGBDFLOW_RESIDENT_K", K)  # 0: level bands and the rule's exchanges
    before = flow()
    assert np.isfinite(before).all()
    monkeypatch.setenv("RGBDFLOW_WAIT_POLLS", "0")
    assert np.isnan(flow()).all()
    monkeypatch.delenv("RGBDFLOW_WAIT_POLLS")
    np.testing.assert_array_equal(flow(), before)


@pytest.mark.gpu
@pytest.mark.parametrize("n_inner", [1, 2])
def test_2d_sor_reports_lost_waits(ctx, monkeypatch, n_inner):
    """Several bands and groups of sweeps, so that tasks wait for others' values; later solves run as before."""
    p = pair(64, 80, 3)
    prm = rf.flow2d_params(n_outer=2, n_inner=n_inner, n_sor=40)
    before = ctx.optical_flow_2d(p["bgr1"], p["bgr2"], prm)
    monkeypatch.setenv("RGBDFLOW_WAIT_POLLS", "0")
    with pytest.raises(rf.RgbdFlowError) as e:
        ctx.optical_flow_2d(p["bgr1"], p["bgr2"], prm)
    assert e.value.code == TIMEOUT
    monkeypatch.delenv("RGBDFLOW_WAIT_POLLS")
    np.testing.assert_array_equal(ctx.optical_flow_2d(p["bgr1"], p["bgr2"], prm), before)


@pytest.mark.gpu
@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc to compile the probe")
def test_level_bands_waits_take_a_second(tmp_path):
    exe = str(tmp_path / "wait_time_check")
    subprocess.run(["nvcc", "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "-o", exe,
                    os.path.join(HERE, "cpp", "wait_time_check.cu")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
