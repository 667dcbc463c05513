"""Rays at the edges of what the fast set-up takes (directions and starts in a plain range,
moving along every axis) and beyond them: axis-aligned and scaled cameras, starts outside
the world, on cell faces, tiny, huge or no number.  Every kernel gives the oracle's frame,
step counts included."""
import numpy as np
import pytest

import vrt
from helpers import assert_same_frame, gpu_render, make_world

pytestmark = pytest.mark.gpu

W, H = 45, 38
POSITIONS = {
    "inside": (20.3, 33.6, 19.7), "on faces": (20.0, 33.0, 19.0), "negative": (-4.5, 20.25, -3.75),
    "beyond": (60.5, 30.5, 71.25), "tiny": (1e-30, 30.5, 2e-19), "zero": (0.0, 30.5, 0.0), "huge": (5e6, 20.5, 20.5),
    "not a number": (float("nan"), 30.5, 20.5), "infinite": (20.5, float("inf"), 20.5),
}
MATRICES = ("turned", "identity", "back", "doubled", "small", "vanishing", "zero", "not a number")


def matrix_of(name):
    turned = vrt.rotate_matrix(0.5, 0.7)
    return {"turned": turned, "identity": vrt.rotate_matrix(0.0, 0.0), "back": vrt.rotate_matrix(0.4, 3.6),
            "doubled": [2.5 * v for v in turned], "small": [1e-6 * v for v in turned],
            "vanishing": [1e-20 * v for v in turned], "zero": [0.0] * 16,
            "not a number": [float("nan")] + turned[1:]}[name]


@pytest.mark.parametrize("matrix", MATRICES)
@pytest.mark.parametrize("jumps", [False, True])
def test_rays_beside_the_plain_range(cuda, oracle, matrix, jumps):
    rng = np.random.default_rng(11)
    words = np.where(rng.random(W * H * W) < 0.02, 0x01000000 | rng.integers(0, 1 << 24, W * H * W), -1).astype(np.int32)
    words.reshape(W, H, W)[:, :4, :] = 0x01808080
    w = make_world(words, W, H)
    if jumps:
        w.fix_depth_field()
        words = w.download(words)
    kernels = [vrt.KERNEL_WORD, vrt.KERNEL_MASK_PIXEL] + ([] if jumps else [vrt.KERNEL_BITMASK])
    for name, pos in POSITIONS.items():
        u = vrt.default_uniforms()
        u.camPos[:] = pos
        u.rotateMatrix[:] = matrix_of(matrix)
        u.lightPos[:] = [22.5, 22.0, 90.0] if name == "inside" else [20.0, 120.0, 3.0]
        u.localLights[0][:] = [20.5, 20.5, 20.5, 0.6]
        u.localLightDist = 25.0
        u.maxSteps = 97
        u.aspectRatio = 1.0
        o = oracle.render(words, W, H, u, 21, 21)
        for k in kernels:
            assert_same_frame(o, gpu_render(w, u, 21, 21, kernel=k))
            f = gpu_render(w, u, 21, 21, kernel=k, debug=False)
            assert np.array_equal(f["rgba"], o["rgba"]), (name, k)
