"""The device 2-D optical flow (rgbdflow_optical_flow_2d, the reference demo's flow type 1) on a
B200: it keeps the reference's FP64 arithmetic, operation order and lexicographic SOR order (as
overlapping anti-diagonal sweeps), so its flow equals the reference's bit for bit (as floats,
the reference's cv::Vec2f result):
  * the golden vectors the reference made (tests/golden/ref_flow2d_golden.npz);
  * the pinned oracle on a scene where a red-black SOR order would move the flow by 1.2 px;
  * the number of sweeps in flight does not change the result."""
import importlib.util
import os

import numpy as np
import pytest

import oracle_binding as ob
import rgbdflow as rf
import synthetic as syn

pytestmark = pytest.mark.gpu

GOLDEN_DIR = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")


def _params(tag):
    spec = importlib.util.spec_from_file_location("make_flow2d_golden", os.path.join(GOLDEN_DIR, "make_flow2d_golden.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    q = m.PARAMS[tag]
    return rf.flow2d_params(alpha=q["alpha"], pyramid_ratio=q["ratio"], min_width=q["min_width"], n_outer=q["n_outer"],
                            n_inner=q["n_inner"], n_sor=q["n_sor"])


@pytest.mark.parametrize("tag", ["shift", "patch"])
def test_equals_reference_golden(ctx, tag):
    g = np.load(os.path.join(GOLDEN_DIR, "ref_flow2d_golden.npz"))
    flow = ctx.optical_flow_2d(g[tag + "_bgr1"], g[tag + "_bgr2"], _params(tag))
    expect = np.stack([g[tag + "_u"], g[tag + "_v"]], -1).astype(np.float32)
    np.testing.assert_array_equal(flow, expect)


def test_equals_oracle_on_a_fragile_scene(ctx):
    p = syn.make_config_pair("160x120", seed=1)
    flow = ctx.optical_flow_2d(p["bgr1"], p["bgr2"])
    u, v = ob.optical_flow_2d(p["bgr1"], p["bgr2"])
    np.testing.assert_array_equal(flow, np.stack([u, v], -1).astype(np.float32))


def test_sweeps_in_flight_do_not_change_the_flow(ctx):
    g = np.load(os.path.join(GOLDEN_DIR, "ref_flow2d_golden.npz"))
    a = ctx.optical_flow_2d(g["patch_bgr1"], g["patch_bgr2"], _params("patch"))
    for ring in (2, 16):
        p = _params("patch")
        p.sor_ring = ring
        np.testing.assert_array_equal(ctx.optical_flow_2d(g["patch_bgr1"], g["patch_bgr2"], p), a)


def test_bad_parameters_are_status_codes(ctx):
    b = np.zeros((24, 32, 3), np.uint8)
    for over in (dict(min_width=0), dict(pyramid_ratio=0.0), dict(alpha=-1.0), dict(n_sor=0), dict(sor_ring=17)):
        with pytest.raises(rf.RgbdFlowError) as e:
            ctx.optical_flow_2d(b, b, rf.flow2d_params(**over))
        assert e.value.code == -1


@pytest.mark.parametrize("tag", ["shift", "patch"])
def test_cluster_sor_equals_reference_golden(ctx, monkeypatch, tag):
    """Every level's SOR over a cluster of CTAs with 32 sweeps in flight (the path of the larger
    levels): the same flow as the reference's, bit for bit."""
    monkeypatch.setenv("RGBDFLOW_FLOW2D_CLUSTER_MIN_PX", "1")
    g = np.load(os.path.join(GOLDEN_DIR, "ref_flow2d_golden.npz"))
    flow = ctx.optical_flow_2d(g[tag + "_bgr1"], g[tag + "_bgr2"], _params(tag))
    expect = np.stack([g[tag + "_u"], g[tag + "_v"]], -1).astype(np.float32)
    np.testing.assert_array_equal(flow, expect)


def test_cluster_sor_equals_single_cta_on_a_config_pair(ctx, monkeypatch):
    p = syn.make_config_pair("320x240", seed=2)
    monkeypatch.setenv("RGBDFLOW_FLOW2D_CLUSTER_MIN_PX", "1000000000")
    a = ctx.optical_flow_2d(p["bgr1"], p["bgr2"])
    monkeypatch.setenv("RGBDFLOW_FLOW2D_CLUSTER_MIN_PX", "1")
    b = ctx.optical_flow_2d(p["bgr1"], p["bgr2"])
    np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("w, h, n_sor, over", [
    (37, 29, 1, {}), (33, 32, 7, {}), (31, 33, 8, {}), (65, 70, 9, {}), (3, 97, 21, dict(min_width=3)),
    (100, 5, 40, dict(min_width=60)), (2, 2, 5, dict(min_width=2)),
    (37, 29, 100, dict(sor_ring=2)),    # work space for one group of sweeps a launch
    (40, 40, 400, dict(alpha=0.5)),
], ids=str)
def test_sor_pipeline_equals_oracle_at_its_edges(ctx, w, h, n_sor, over):
    """Widths and heights around a band's 32 rows, sweep counts around a group's 8, several launches a solve:
    the arithmetic and its order are the oracle's, so the flow is equal."""
    rng = np.random.default_rng(w * 1000 + h)
    b1 = rng.integers(0, 256, (h, w, 3), dtype=np.uint8)
    b2 = np.clip(np.roll(b1, 1, axis=1).astype(int) + rng.integers(-3, 4, b1.shape), 0, 255).astype(np.uint8)
    q = dict(dict(min_width=20, n_outer=2, n_inner=2), **over)
    flow = ctx.optical_flow_2d(b1, b2, rf.flow2d_params(n_sor=n_sor, **q))
    q.pop("sor_ring", None)
    u, v = ob.optical_flow_2d(b1, b2, n_sor=n_sor, **q)
    np.testing.assert_array_equal(flow, np.stack([u, v], -1).astype(np.float32))


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_sor_pipeline_stops_at_the_first_converged_sweep(ctx, seed):
    """Frames that are equal (the first sweep converges) in all but a faint patch, whose sweeps converge inside a
    group: the increments are that sweep's."""
    rng = np.random.default_rng(seed)
    b1 = np.full((48, 60, 3), 90, np.uint8)
    b2 = b1.copy()
    b1[10 * seed:10 * seed + 6, 20:30] += rng.integers(0, 3, (6, 10, 3), dtype=np.uint8)
    for n_sor in (3, 400):
        flow = ctx.optical_flow_2d(b1, b2, rf.flow2d_params(n_sor=n_sor, n_outer=2))
        u, v = ob.optical_flow_2d(b1, b2, n_sor=n_sor, n_outer=2)
        np.testing.assert_array_equal(flow, np.stack([u, v], -1).astype(np.float32))
