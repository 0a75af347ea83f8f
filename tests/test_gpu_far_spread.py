"""The series of gpp_far.cu takes a band only where fixed point holds its terms:

* aqsn large just where I_eps is small, over 10^3, 10^6 and 10^9 within every
  chunk: all bands are summed term by term, with the bits of the per-term entry
  point (a fixed point relative to each factor's largest value would be off by
  3e-14, 3e-11 and 3e-8);
* a tenth of the bands like that: theirs are as accurate as per-term sums (to
  2^-48 of the sum of the terms' magnitudes in FP64, 2^-40 in mixed precision,
  against long double), the others still take the series;
* uniform and Gaussian data and factors that fall together over decades keep
  the series (other bits than the per-term sums)."""
import numpy as np
import pytest

from gppsigma import build, capi, workload as W
from test_gpu_far_range import per_term

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SHAPE = {"fp64": (64, 2, 5003, 17, 32, 0.25), "mixed": (64, 2, 20003, 40, 32, 0.25)}


@pytest.fixture(scope="module", autouse=True)
def _lib():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    build.build()
    capi.load()


def _state(precision):
    nb, nv, nc, ng, nw, dw = SHAPE[precision]
    return W.make_inputs(W.Shape(nb, nv, nc, ng, nw, dw=dw), 21)


def _oppose(inp, ratio, bands):
    """One column in 50: aqsn up by `ratio` in these bands, I_eps down by it."""
    at = np.arange(7, inp.shape.ncouls, 50)
    inp.I_eps_array[:, at] /= ratio
    for n in bands:
        inp.aqsntemp[n, at] *= ratio


def _run(inp, precision):
    from gppsigma import ops
    d = ops.DeviceInputs.from_host(inp)
    lib = capi.load()
    lib.gpp_reset_launch_count()
    r = ops.sigma(d, precision, acht_n1=True)
    ops.wait()
    assert lib.gpp_launch_count() > 20
    return d, r


@pytest.mark.parametrize("ratio", [1e3, 1e6, 1e9])
def test_opposed_ranges_are_summed_term_by_term(ratio):
    inp = _state("fp64")
    _oppose(inp, ratio, range(inp.shape.number_bands))
    d, r = _run(inp, "fp64")
    ach, asx = per_term(d)
    assert np.array_equal(r.achtemp.cpu().numpy(), ach) and np.array_equal(r.asxtemp.cpu().numpy(), asx)


@pytest.mark.parametrize("precision,bits", [("fp64", 48), ("mixed", 40)])
@pytest.mark.parametrize("ratio", [1e3, 1e6, 1e9])
def test_opposed_bands_are_as_accurate_as_per_term(precision, bits, ratio):
    inp = _state(precision)
    bands = list(range(5, 64, 10))
    _oppose(inp, ratio, bands)
    d, r = _run(inp, precision)
    got = r.acht_n1_loc.cpu().numpy()
    ld = np.clongdouble
    wt, ie = inp.wtilde_array.astype(ld), inp.I_eps_array.astype(ld)
    igp = np.minimum(inp.inv_igp_index, inp.shape.ncouls - 1)
    for n in bands + [6, 40]:
        f = wt * ie / (inp.wx_array[n, 2] - wt) * inp.aqsntemp[n][None, :].astype(ld)
        c = 0.5 * inp.vcoul[igp] * np.conj(inp.aqsmtemp[n, igp])
        want, size = np.sum(c * f.sum(axis=1)), np.sum(np.abs(c) * np.abs(f).sum(axis=1))
        assert abs(got[n] - want) <= 2.0 ** -bits * size, n
    if precision == "fp64":
        assert not np.array_equal(r.achtemp.cpu().numpy(), per_term(d)[0])  # the others' series


@pytest.mark.parametrize("kind", ["uniform", "gaussian", "decades"])
def test_ordinary_data_keeps_the_series(kind):
    inp = _state("fp64")
    rng = np.random.default_rng(5)
    if kind == "gaussian":
        for name in ("aqsntemp", "I_eps_array"):
            a = getattr(inp, name)
            a[:] = rng.normal(size=a.shape) + 1j * rng.normal(size=a.shape)
    elif kind == "decades":
        fall = np.exp(-18.0 * np.arange(inp.shape.ncouls) / inp.shape.ncouls)
        inp.aqsntemp *= fall
        inp.I_eps_array *= fall
    d, r = _run(inp, "fp64")
    ach, _ = per_term(d)
    got = r.achtemp.cpu().numpy()
    assert not np.array_equal(got, ach)
    assert np.max(np.abs(got - ach)) <= 1e-12 * np.max(np.abs(ach))
