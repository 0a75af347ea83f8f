"""One wx row, FP64, no per-band output: the occupied bands in the frequency
pass of the band sum (gemm_occupied_kernel), against the oracle and against the
separate kernels that a call with the per-band output takes, over wtilde of six
decades with values in every branch of the solver: odd row counts, one to
several parts of the columns, frequency chunks with a remainder, the most
occupied bands the pass takes and one more."""
import numpy as np
import pytest

from gppsigma import build, capi
from gppsigma import workload as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

CASES = [  # nv, unoccupied bands, ncouls, ngpown, nw, semantics
    (1, 32, 40, 1, 1, "complex_seq"),
    (2, 40, 1023, 5, 2, "complex_seq"),
    (2, 33, 2049, 4, 3, "kerseq"),
    (5, 35, 3100, 7, 4, "complex_seq"),
    (3, 64, 500, 3, 5, "complex_seq"),
    (64, 32, 300, 3, 3, "complex_seq"),
    (65, 32, 300, 3, 3, "complex_seq"),
    (2, 32, 1200, 9, 13, "kerseq"),
]


@pytest.fixture(scope="module", autouse=True)
def _lib():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    build.build()
    capi.load()


def _inputs(nv, un, nc, ng, nw, seed):
    inp = W.make_inputs(W.Shape(nv + un, nv, nc, ng, nw), seed)
    rng = np.random.default_rng(seed)
    size = 10.0 ** rng.uniform(-3, 3, (ng, nc)) * rng.choice([-1.0, 1.0], (ng, nc))
    inp.wtilde_array[:] = size + 1j * (0.05 * size * rng.uniform(-1, 1, (ng, nc)))
    wx = rng.choice([-30.0, -2.5, -1.0, -0.4, 0.3, 0.999, 1.0, 1.7, 5.0, 200.0], (1, nw))
    inp.wx_array = wx + (np.abs(wx) != 1.0) * rng.uniform(-0.05, 0.05, (1, nw))
    near = rng.uniform(size=(ng, nc)) < 0.2
    pick = inp.wx_array.ravel()[rng.integers(0, nw, (ng, nc))]
    off = rng.uniform(-0.3, 0.3, (ng, nc)) * rng.choice([1.0, 1e-4], (ng, nc))
    inp.wtilde_array[near] = (pick + off + 0.01j)[near]
    return inp


# Sums of signed terms: 1e-12 of the largest output covers n 2^-53 for the
# terms here with the solver's few roundings each.
@pytest.mark.parametrize("nv,un,nc,ng,nw,semantics", CASES)
def test_occupied_bands_in_the_band_sum(nv, un, nc, ng, nw, semantics):
    import oracle_py
    from gppsigma import ops
    inp = _inputs(nv, un, nc, ng, nw, 17 * nc + nw)
    want = oracle_py.run(inp, semantics, nthreads=4)
    d = ops.DeviceInputs.from_host(inp)
    assert d.wx_stride == 0
    r = ops.sigma(d, "fp64", semantics)
    again = ops.sigma(d, "fp64", semantics)
    apart = ops.sigma(d, "fp64", semantics, acht_n1=True) if nw >= 3 else r
    ops.wait()
    for key in ("achtemp", "asxtemp"):
        got, w = getattr(r, key).cpu().numpy(), want[key]
        scale = np.max(np.abs(w))
        assert np.max(np.abs(got - w)) <= 1e-12 * scale, (key, got, w)
        assert np.max(np.abs(getattr(apart, key).cpu().numpy() - w)) <= 1e-12 * scale
        assert torch.equal(getattr(r, key), getattr(again, key))
