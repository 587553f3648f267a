"""The denoiser keeps subnormal radiance: a frame of one tiny colour comes back as that colour, in every staging of
the a-trous passes. A sum of n products is off by at most n halves of the spacing of subnormals (2^-149), the
normalisation by one more: 50 taps of the variance estimate and five passes of 25 by less than 100 spacings."""
import pytest

from photon_b200 import abi, native, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [None, 0, 1, 3, "noalloc"])
@pytest.mark.parametrize("w,h", [(97, 61), (701, 577)])
def test_a_subnormal_frame_survives(mode, w, h):
    torch = pytest.importorskip("torch")
    tiny = 1e-40
    full = lambda *v: torch.tensor(v, device="cuda", dtype=torch.float32).expand(h, w, 4).contiguous()  # noqa: E731
    f = [full(tiny, 2 * tiny, 3 * tiny, 1), full(1, 1, 1, 1), full(0, 0, -1, 3), full(0, 0, 0, 2), full(0, 0, 0, 1)]
    out = torch.zeros((h, w, 4), device="cuda")
    torch.cuda.synchronize()
    st = abi.svgf_settings(atrous_iterations=5)
    if mode == "noalloc":
        native.svgf_run_noalloc(w, h, *(t.data_ptr() for t in f), st, out.data_ptr())
    else:
        s = native.Svgf(w, h)
        if mode is not None:
            s.set_tma(mode)
        s.run(*(t.data_ptr() for t in f), workloads.look_at((0, 0, -3), (0, 0, 0), 50.0, w / h), st, out.data_ptr())
    torch.cuda.synchronize()
    got = out.cpu().double()[..., :3]  # (on the host: device arithmetic of another library may flush)
    want = f[0].cpu().double()[..., :3]
    assert float((got - want).abs().max()) <= 100 * 2.0 ** -149
