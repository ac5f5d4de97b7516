"""The denoiser's tiles (csrc/image.cu) at sizes and steps where they can go wrong: images smaller than a tile or a
step, ragged edges, short and long histories side by side, background, steps past the image. Equal to the oracle (NaN where it has one)."""
import numpy as np
import pytest

import oracle.binding as ob
import restir_b200 as rb
from restir_b200.abi import RestirParams


def inputs(w, h, seed):
    rng = np.random.default_rng(seed)
    n = w * h
    color = rng.lognormal(-1.0, 1.0, (n, 4)).astype(np.float16)
    lum = color[:, :3].astype(np.float32) @ np.array([0.2126, 0.7152, 0.0722], np.float32)
    moments = np.stack([lum, lum * lum * 1.3, rng.integers(1, 9, n), np.zeros(n)], 1).astype(np.float16)
    receiver = np.zeros((n, 4), np.float32)
    receiver[:, :3] = rng.normal(0.0, 0.02, (n, 3)) + np.stack([np.arange(n) % w, np.arange(n) // w, np.zeros(n)], 1) * 0.01
    normal = np.zeros((n, 4), np.float32)
    normal[:, :3] = [0.0, 0.1, -1.0] + rng.normal(0.0, 0.03, (n, 3))
    normal[rng.random(n) < 0.1] = 0.0
    if n > 4:
        color[n // 2, 1], receiver[n // 3, 2] = np.nan, np.inf
    return color, moments, receiver, normal


@pytest.mark.gpu
@pytest.mark.parametrize("size", [(1, 1), (3, 2), (15, 7), (16, 8), (17, 9), (33, 70), (129, 65)])
def test_tiles(size):
    import torch
    w, h = size
    arrays = inputs(w, h, seed=w)
    params = RestirParams()
    params.gi_width, params.gi_height, params.scene_scale = w, h, 1.3
    device = [torch.from_numpy(a).cuda() for a in arrays]
    color, moments, receiver, normal = (d.data_ptr() for d in device)
    want = np.zeros((w * h, 4), np.float16)
    got = torch.zeros((w * h, 4), dtype=torch.float16, device="cuda")
    ob.load().oracle_svgf_variance(params, *(a.ctypes.data for a in arrays), want.ctypes.data)
    rb.check(rb.load().restir_svgf_variance(params, color, moments, receiver, normal, got.data_ptr(), None), "variance")
    torch.cuda.synchronize()
    np.testing.assert_array_equal(got.cpu().numpy(), want)
    for step in (1, 2, 3, 8, 16, 64, 1 << 30):
        filtered = np.zeros_like(want)
        out = torch.zeros_like(got)
        ob.load().oracle_svgf_atrous(params, step, want.ctypes.data, arrays[2].ctypes.data, arrays[3].ctypes.data,
                                     filtered.ctypes.data)
        rb.check(rb.load().restir_svgf_atrous(params, step, got.data_ptr(), receiver, normal, out.data_ptr(), None), "atrous")
        torch.cuda.synchronize()
        np.testing.assert_array_equal(out.cpu().numpy(), filtered, err_msg=str(step))


@pytest.mark.gpu
@pytest.mark.parametrize("size", [(320, 180), (641, 359)])
def test_taps_from_the_image(size):
    """Steps on both sides of the line between tiles and taps read from the image (as many blocks as are in flight at
    once, tiles mostly empty), up to the image's size."""
    import torch
    w, h = size
    color, moments, receiver, normal = inputs(w, h, seed=h)
    params = RestirParams()
    params.gi_width, params.gi_height, params.scene_scale = w, h, 0.7
    source, positions, normals = (torch.from_numpy(a).cuda() for a in (color, receiver, normal))
    for step in (16, 32, 33, 47, 48, 100, w - 1, w, w + 1):
        want = np.zeros_like(color)
        out = torch.zeros_like(source)
        ob.load().oracle_svgf_atrous(params, step, color.ctypes.data, receiver.ctypes.data, normal.ctypes.data, want.ctypes.data)
        rb.check(rb.load().restir_svgf_atrous(params, step, source.data_ptr(), positions.data_ptr(), normals.data_ptr(),
                                              out.data_ptr(), None), "atrous")
        torch.cuda.synchronize()
        np.testing.assert_array_equal(out.cpu().numpy(), want, err_msg=str(step))
