"""The denoiser's staged passes (TMA tiles, rows, the variance estimate's tile) against direct global loads on
drawn G-buffers: every staging gives the same frames bit for bit, over a few frames with history, at sizes
of one pixel, one row, tile edges and remainders, for every number of passes up to one past the staged ones;
and the allocation-free denoise, whose passes are all staged by rows, gives a session's first frame."""
import numpy as np
import pytest

from photon_b200 import abi, native, workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device for torch")
    return torch


def _frames(torch, w, h, n):
    """Random surfaces in a few materials, with misses, seen by a camera that moves a little."""
    gen = torch.Generator(device="cuda").manual_seed(w * 1000 + h)
    r = lambda *s: torch.rand(s, generator=gen, device="cuda")  # noqa: E731
    cams = [workloads.look_at((0.02 * k, 0.0, -3.0), (0, 0, 0), 50.0, w / h) for k in range(n)]
    mat = torch.floor(r(h, w, 1) * 1.3 + 0.8 * (torch.arange(w, device="cuda") > w // 2)[None, :, None]) - (r(h, w, 1) < 0.1).float() * 3
    mat = torch.where(mat < 0, -1.0, mat)
    x = torch.linspace(-1.2, 1.2, w, device="cuda")[None, :, None].expand(h, w, 1)
    y = torch.linspace(1.0, -1.0, h, device="cuda")[:, None, None].expand(h, w, 1)
    out = []
    for k in range(n):
        nrm = torch.cat([r(h, w, 2) * 0.4 - 0.2, -torch.ones((h, w, 1), device="cuda")], -1)
        nrm = nrm / nrm.norm(dim=-1, keepdim=True)
        one = torch.ones((h, w, 1), device="cuda")
        out.append({"color": torch.cat([r(h, w, 3) * 3, one], -1).contiguous(), "albedo": torch.cat([r(h, w, 3), one], -1).contiguous(),
                    "normal_depth": torch.cat([nrm, 3 + 0.1 * r(h, w, 1)], -1).contiguous(),
                    "position": torch.cat([x, y, 0.1 * r(h, w, 1), mat], -1).contiguous(),
                    "emission": torch.cat([r(h, w, 3) * 0.1, one], -1).contiguous()})
    return cams, out


def _run(torch, mode, cams, frames, w, h, passes):
    s = native.Svgf(w, h)
    if mode is not None:
        s.set_tma(mode)
    got = []
    for k, f in enumerate(frames):
        out = torch.zeros((h, w, 4), device="cuda")
        s.run(*(f[n].data_ptr() for n in ("color", "albedo", "normal_depth", "position", "emission")), cams[max(k - 1, 0)],
              abi.svgf_settings(atrous_iterations=passes), out.data_ptr())
        torch.cuda.synchronize()
        got.append(out.cpu().numpy().view(np.uint32))
    s.close()
    return got


@pytest.mark.parametrize("w,h", [(1, 1), (33, 1), (1, 70), (32, 8), (49, 17), (161, 131), (701, 577)])
@pytest.mark.parametrize("passes", [0, 1, 4, 5, 6])
def test_stagings_are_bit_identical(torch, w, h, passes):
    cams, frames = _frames(torch, w, h, 5)
    torch.cuda.synchronize()
    want = _run(torch, 0, cams, frames, w, h, passes)
    for mode in (None, 1, 2, 3):
        for a, b in zip(_run(torch, mode, cams, frames, w, h, passes), want):
            assert np.array_equal(a, b), mode
    out = torch.zeros((h, w, 4), device="cuda")
    f = frames[0]
    native.svgf_run_noalloc(w, h, *(f[n].data_ptr() for n in ("color", "albedo", "normal_depth", "position", "emission")),
                            abi.svgf_settings(atrous_iterations=passes), out.data_ptr())
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want[0])
