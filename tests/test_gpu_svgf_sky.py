"""Blocks without a surface, which the staged a-trous passes neither prepare nor filter: frames of sky alone, of
sky with a single surface pixel (at a corner, inside, at the ragged edge) and with a band of surfaces give the
direct loads' frames bit for bit in every staging."""
import numpy as np
import pytest

from test_gpu_svgf_tiles import _frames, _run, torch  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (33, 9), (161, 131)])
@pytest.mark.parametrize("kind", ["sky", "corner", "inside", "edge", "band"])
def test_sky_blocks_are_bit_identical(torch, w, h, kind):  # noqa: F811
    cams, frames = _frames(torch, w, h, 3)
    keep = torch.zeros((h, w), dtype=torch.bool, device="cuda")
    if kind == "band":
        keep[h // 3:h // 2 + 1] = True
    elif kind != "sky":
        y, x = dict(corner=(0, 0), inside=(h // 2, w // 2), edge=(h - 1, w - 1))[kind]
        keep[y, x] = True
    for f in frames:
        mat = f["position"][..., 3]
        mat.copy_(torch.where(keep, mat.clamp(min=0), torch.full_like(mat, -1)))
    torch.cuda.synchronize()
    want = _run(torch, 0, cams, frames, w, h, 5)
    for mode in (None, 1, 2, 3):
        for a, b in zip(_run(torch, mode, cams, frames, w, h, 5), want):
            assert np.array_equal(a, b), mode
