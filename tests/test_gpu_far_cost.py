"""The series is not taken where it loses: at small sizes where its planes, its
grids that do not fill the SMs and few frequencies a band make it dearer than
the per-term kernels, and where wtilde leaves no box, a call takes at most 1.1
times what it takes with the series' scratch refused (gpp_selftest_scratch_limit,
which leaves the per-term kernels).  The two times are taken in turn, the best of
several calls each; on GB300 the first two were 1.33 and 1.13 of it when the
cost of a term was its cost in large calls."""
import numpy as np
import pytest

from gppsigma import build, capi, workload as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

CASES = [  # precision, nb, ncouls, ngpown, nw, spread
    ("mixed", 330, 25601, 73, 2, False),
    ("fp64", 200, 25601, 33, 1, False),
    ("fp64", 420, 7937, 17, 3, True),
    ("mixed", 512, 8192, 100, 3, True),
]


@pytest.mark.parametrize("precision,nb,nc,ng,nw,spread", CASES)
def test_no_slower_than_per_term(precision, nb, nc, ng, nw, spread):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    build.build()
    from gppsigma import ops
    lib = capi.load()
    inp = W.make_inputs(W.Shape(nb, 0, nc, ng, nw), 6)
    if spread:
        rng = np.random.default_rng(1)
        inp.wtilde_array[:] = rng.uniform(-12, 16, (ng, nc)) + 1j * rng.uniform(-1, 1, (ng, nc))
    d = ops.DeviceInputs.from_host(inp)
    out = ops.sigma(d, precision)

    def ms(limit):
        capi.check(lib.gpp_selftest_scratch_limit(limit), "limit")
        try:
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            ops.sigma(d, precision, out=out)
            a.record()
            for _ in range(5):
                ops.sigma(d, precision, out=out)
            b.record()
            b.synchronize()
            return a.elapsed_time(b) / 5
        finally:
            capi.check(lib.gpp_selftest_scratch_limit(0), "limit")

    times = [(ms(0), ms(400 << 20)) for _ in range(6)][1:]
    ops.wait()
    assert min(t[0] for t in times) <= 1.1 * min(t[1] for t in times), times
