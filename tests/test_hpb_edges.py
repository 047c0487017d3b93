"""The HPB weights at sizes around the 32-row bands and 32-pixel steps of its integral images, against the oracle
with the tolerances of tests/test_hpb_gpu.py (weights within 1e-6 on 99.5 % of the pixels, mean difference 1e-3)."""
import numpy as np
import pytest

import oracle_binding as ob
import rgbdflow as rf
from test_hpb_gpu import hpb_params
from test_resident_tiles import pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(33, 31), (64, 32), (65, 97), (31, 33), (96, 40), (200, 17)])
def test_hpb_weights_match_oracle_at_odd_sizes(ctx, W, H):
    p = pair(W, H, 3 * W + H)
    prm = hpb_params(W, n_outer=1)
    prm.min_width = W
    cam = rf.CameraParams.make(W, H, p["cam"].f, p["cam"].cx, p["cam"].cy)
    ctx.scene_flow_two_frames(cam, p["bgr1"], p["depth1"], p["bgr2"], p["depth2"], prm)
    img = np.stack([ctx.debug_plane(0, 0, rf.PLANE_PYRAMID, c) for c in range(3)], -1)
    hpb = ob.heuristic_pb(img, ctx.debug_plane(0, 0, rf.PLANE_HPB_DEPTH)).astype(np.float64)
    for c in range(2):
        o = 1 - hpb[..., c] * .99
        o[(slice(None), W - 1) if c == 0 else (H - 1, slice(None))] = 0
        diff = np.abs(ctx.debug_plane(0, 0, rf.PLANE_REG, c) - o.astype(np.float32))
        assert np.mean(diff <= 1e-6) >= 0.995 and diff.mean() <= 1e-3
