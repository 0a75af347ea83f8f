"""Occupied bands at the edges of the solver's branches, against the oracle:
every frequency-chunk remainder, ragged column counts, one and several bands
(alone and in pairs), wtilde over six decades and both signs, frequencies at,
below and above 1 in magnitude (where the kernels change how they form the
branch-A sum) and of both signs (with and without the cutoff), and wtilde
that are infinite or NaN, which neither branch takes.

Norm-wise tolerances: each term is formed with a few roundings, and terms of
one output are summed in float64 (1e-12) or float-float (1e-8), as in the
other suites."""
import numpy as np
import pytest

from gppsigma import build, capi, workload as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

CASES = [  # nv, ncouls, ngpown, nw, one wx row, semantics
    (1, 1, 1, 1, False, "complex_seq"),
    (1, 127, 3, 2, False, "complex_seq"),
    (2, 128, 4, 3, True, "complex_seq"),
    (3, 129, 5, 3, True, "kerseq"),
    (3, 300, 7, 4, False, "complex_seq"),
    (2, 515, 6, 5, True, "complex_seq"),
    (4, 261, 3, 6, False, "kerseq"),
    (5, 700, 2, 7, True, "complex_seq"),
    (2, 640, 9, 9, False, "complex_seq"),
    (3, 385, 4, 13, True, "kerseq"),
]


@pytest.fixture(scope="module", autouse=True)
def _lib():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    build.build()
    capi.load()


def _inputs(nv, nc, ng, nw, one_row, seed):
    inp = W.make_inputs(W.Shape(nv, nv, nc, ng, nw), seed)
    rng = np.random.default_rng(seed)
    size = 10.0 ** rng.uniform(-3, 3, (ng, nc)) * rng.choice([-1.0, 1.0], (ng, nc))
    inp.wtilde_array[:] = size + 1j * (0.05 * size * rng.uniform(-1, 1, (ng, nc)))
    rows = 1 if one_row else nv
    wx = rng.choice([-30.0, -2.5, -1.0, -0.4, 0.3, 0.999, 1.0, 1.7, 5.0, 200.0], (rows, nw))
    inp.wx_array = wx + (np.abs(wx) != 1.0) * rng.uniform(-0.05, 0.05, (rows, nw))
    # Some wtilde close to a frequency (branch B and the pole).
    near = rng.uniform(size=(ng, nc)) < 0.2
    pick = inp.wx_array.ravel()[rng.integers(0, rows * nw, (ng, nc))]
    off = rng.uniform(-0.3, 0.3, (ng, nc)) * rng.choice([1.0, 1e-4], (ng, nc))
    inp.wtilde_array[near] = (pick + off + 0.01j)[near]
    if nc > 100:
        inp.wtilde_array[0, 5] = complex(np.inf, 0.0)
        inp.wtilde_array[ng - 1, 77] = complex(1.0, np.nan)
    return inp


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-8)])
@pytest.mark.parametrize("nv,nc,ng,nw,one_row,semantics", CASES)
def test_occupied_branches(nv, nc, ng, nw, one_row, semantics, precision, tol):
    import oracle_py
    from gppsigma import ops
    inp = _inputs(nv, nc, ng, nw, one_row, 31 * nc + nw)
    with np.errstate(all="ignore"):
        want = oracle_py.run(inp, semantics, nthreads=4)
    d = ops.DeviceInputs.from_host(inp)
    r = ops.sigma(d, precision, semantics)
    ops.wait()
    for key in ("achtemp", "asxtemp"):
        got, w = getattr(r, key).cpu().numpy(), want[key]
        assert np.all(np.isfinite(w))
        scale = np.max(np.abs(w))
        assert np.max(np.abs(got - w)) <= tol * scale, (key, got, w)


@pytest.mark.parametrize("nv,ng", [(2, 304), (3, 400), (2, 60)])
def test_band_pairs_give_the_per_band_bits_at_both_grid_sizes(nv, ng, monkeypatch):
    """Pairs of occupied bands (enough blocks for the SMs) and one band per
    block (fewer): the same bits as with pairs switched off."""
    from gppsigma import ops
    d = ops.DeviceInputs.from_host(_inputs(nv, 421, ng, 3, True, 11 * ng))
    a = ops.sigma(d, "fp64")
    ops.wait()
    monkeypatch.setenv("GPP_FLAG_MULTI", "0")
    b = ops.sigma(d, "fp64")
    ops.wait()
    assert torch.equal(a.asxtemp, b.asxtemp) and torch.equal(a.achtemp, b.achtemp)
