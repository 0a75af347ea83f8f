"""One wx row of 300000 frequencies, FP64 and mixed: within the grid limits of the
chunks of 8 the band sum takes, past those of the occupied bands' 3 or 4, which
run in several launches' worth then.  Against the oracle, norm-wise."""
import numpy as np
import pytest

from gppsigma import build, capi, workload as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-8)])
def test_more_frequency_chunks_than_a_grid_dimension(precision, tol):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    build.build()
    import oracle_py
    from gppsigma import ops
    inp = W.make_inputs(W.Shape(34, 2, 16, 2, 300000, dw=1e-4), 4)
    inp.wx_array = inp.wx_array[:1].copy()
    want = oracle_py.run(inp, "complex_seq", nthreads=8)
    r = ops.sigma(ops.DeviceInputs.from_host(inp), precision)
    ops.wait()
    for key in ("achtemp", "asxtemp"):
        got, w = getattr(r, key).cpu().numpy(), want[key]
        assert np.max(np.abs(got - w)) <= tol * np.max(np.abs(w)), key
