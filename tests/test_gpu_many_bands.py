"""262400 bands with per-band frequencies in mixed precision with the 8-band tile:
within the per-term kernels' limit of 65535 band tiles, past what a grid
dimension of the series would hold.  The sums equal those of the two halves of
the bands, norm-wise to 1e-10 (float-float sums, 2^-44 a term)."""
import pytest

from gppsigma import build, capi

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_more_bands_than_the_series_holds():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    build.build()
    from gppsigma import ops
    lib = capi.load()
    nb, nc, ng, nw = 262400, 512, 16, 3
    g = torch.Generator(device="cuda").manual_seed(2)

    def z(rows, re, im):
        out = torch.empty((rows, nc), dtype=torch.complex128, device="cuda")
        v = torch.view_as_real(out)
        v[..., 0].uniform_(*re, generator=g)
        v[..., 1].uniform_(*im, generator=g)
        return out

    def of(a, b, t):
        return ops.DeviceInputs(b - a, 0, nc, ng, nw, t["aqsm"][a:b], t["aqsn"][a:b], t["ieps"], t["wt"],
                                t["vcoul"], t["igp"], None, t["wx"][a:b], nw)

    t = {"aqsm": z(nb, (-0.5, 0.5), (-0.5, 0.5)), "aqsn": z(nb, (-0.5, 0.5), (-0.5, 0.5)),
         "ieps": z(ng, (-0.5, 0.5), (-0.5, 0.5)), "wt": z(ng, (0.5, 2.0), (-0.05, 0.05)),
         "vcoul": torch.rand(nc, dtype=torch.float64, device="cuda", generator=g) + 0.1,
         "igp": torch.arange(0, 32 * ng, 32, dtype=torch.int32, device="cuda")}
    e = 20.0 * torch.rand((nb, 1), dtype=torch.float64, device="cuda", generator=g)
    t["wx"] = (10.0 + torch.arange(1, nw + 1, dtype=torch.float64, device="cuda")[None, :] - e).contiguous()
    capi.check(lib.gpp_set_variant(nw, 8), "gpp_set_variant")
    try:
        whole = ops.sigma(of(0, nb, t), "mixed", acht_n1=True)
        ops.wait()
        a, b = (ops.sigma(of(*r, t), "mixed", acht_n1=True) for r in ((0, nb // 2), (nb // 2, nb)))
        ops.wait()
    finally:
        capi.check(lib.gpp_set_variant(nw, -1), "gpp_set_variant")
    want, n1 = a.achtemp + b.achtemp, torch.cat([a.acht_n1_loc, b.acht_n1_loc])
    assert (whole.achtemp - want).abs().max() <= 1e-10 * want.abs().max()
    assert (whole.acht_n1_loc - n1).abs().max() <= 1e-10 * n1.abs().max()
