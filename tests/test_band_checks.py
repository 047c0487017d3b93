"""The convergence checks of k_level_bands at short check periods: their order between a cluster's CTAs on the
CPU, and on a GPU the flow and the executed schedule against the tile SOR's."""
import os
import shutil
import subprocess

import pytest

import rgbdflow as rf
from test_sor_convergence import assert_same, solve

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc to compile the kernel's header")
def test_check_arrays_are_not_written_while_they_are_read(tmp_path):
    exe = str(tmp_path / "band_checks_check")
    subprocess.run(["nvcc", "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "-o", exe,
                    os.path.join(HERE, "cpp", "band_checks_check.cu")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.splitlines()[-1].startswith("ok band checks")


@pytest.mark.gpu
@pytest.mark.parametrize("period", [1, 2, 3, 8])
@pytest.mark.parametrize("W,H,over", [(80, 60, {}), (160, 120, {}), (24, 400, {}), (33, 31, dict(n_inner=2)),
                                      (20, 15, dict(storage=rf.STORE_FP16))], ids=str)
def test_level_bands_check_at_short_periods(ctx, monkeypatch, W, H, over, period):
    over = dict(dict(n_outer=4, n_sor=60, sor_check_period=period, sor_tol=1e-4), **over)
    bands = solve(ctx, W, H, W + H, **over)
    monkeypatch.setenv("RGBDFLOW_SOR_LEVEL", "0")
    tile = solve(ctx, W, H, W + H, **over)
    assert_same(bands, tile)
