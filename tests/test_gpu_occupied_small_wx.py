"""Occupied bands at frequencies of zero, far below float's range, and far above
it (only the reference's driver clamps |wx| below 1e-6; the entry points take
what they are given): with every |wtilde| below 0.5 such a frequency is all
branch B, ssx = -Q / (2 (wx + wtilde)), sch = 0, and with a large one the
branches mix.  Against the oracle, through the kernels of one wx row (the band
sum's frequency pass, and the occupied tiles beside it) and of per-band wx, both
precisions and semantics.  Norm-wise tolerances of the suites."""
import numpy as np
import pytest

from gppsigma import build, capi, workload as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

WX = [0.0, -0.0, 1e-90, -1e-90, 1e-30, -1e-13, 0.3, -1e-6, 1e16, -3e15]


@pytest.fixture(scope="module", autouse=True)
def _lib():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    build.build()
    capi.load()


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-8)])
@pytest.mark.parametrize("semantics", ["complex_seq", "kerseq"])
@pytest.mark.parametrize("one_row,acht_n1", [(True, False), (True, True), (False, True)])
def test_branch_b_at_any_frequency(precision, tol, semantics, one_row, acht_n1):
    import oracle_py
    from gppsigma import ops
    inp = W.make_inputs(W.Shape(40, 5, 300, 13, len(WX)), 9)
    rng = np.random.default_rng(1)
    size = inp.wtilde_array.shape
    inp.wtilde_array[:] = rng.uniform(0.05, 0.45, size) * np.exp(1j * rng.uniform(-0.1, 0.1, size))
    if one_row:
        inp.wx_array = np.array([WX])
    else:
        inp.wx_array[:5] = WX
    with np.errstate(all="ignore"):
        want = oracle_py.run(inp, semantics, nthreads=4)
    d = ops.DeviceInputs.from_host(inp)
    r = ops.sigma(d, precision, semantics, acht_n1=acht_n1)
    ops.wait()
    got = r.asxtemp.cpu().numpy()
    assert np.all(np.isfinite(want["asxtemp"])) and np.all(np.abs(want["asxtemp"][:8]) > 0)
    for w in range(len(WX)):  # the frequencies' sums differ by decades
        assert abs(got[w] - want["asxtemp"][w]) <= tol * max(abs(want["asxtemp"][w]), 1e-300), WX[w]
    if not one_row:  # sch: the unoccupied bands' frequencies are ordinary
        ach = r.achtemp.cpu().numpy()
        assert np.max(np.abs(ach - want["achtemp"])) <= tol * np.max(np.abs(want["achtemp"]))


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-8)])
@pytest.mark.parametrize("one_row", [True, False])
def test_branch_a_far_past_the_range_of_float(precision, tol, one_row):
    """wx of 1e-20 with |wtilde| above 0.5 (branch A): ssx is 1e40 times Omega2, past
    float's range; wx of 1e17, where it is 1e-34 of it."""
    import oracle_py
    from gppsigma import ops
    wx = [1e-20, -1e-20, 2.0, 1e17]
    inp = W.make_inputs(W.Shape(40, 3, 300, 13, len(wx)), 3)
    if one_row:
        inp.wx_array = np.array([wx])
    else:
        inp.wx_array[:3] = wx
    want = oracle_py.run(inp, "kerseq", nthreads=4)
    r = ops.sigma(ops.DeviceInputs.from_host(inp), precision, "kerseq")
    ops.wait()
    got = r.asxtemp.cpu().numpy()
    assert np.all(np.isfinite(want["asxtemp"])) and abs(want["asxtemp"][0]) > 1e38
    for w in range(len(wx)):
        assert abs(got[w] - want["asxtemp"][w]) <= tol * abs(want["asxtemp"][w]), wx[w]
