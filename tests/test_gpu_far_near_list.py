"""The near list of the series (gpp_far.cu): its making takes time in
proportion to the (band, frequency) pairs, also where a band has long runs of
near frequencies; and runs that start and end at every place of a warp's 32
frequencies, single near pairs and bands without any give the per-term sums.

Timing: 30000 frequencies a band in runs of up to 22000 near ones; the call
may not take longer than the per-term kernels take for the same state (one row
less, which the series does not serve, times 16 / 15)."""
import ctypes as C

import numpy as np
import pytest

from gppsigma import build, capi, workload as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _lib():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    build.build()
    capi.load()


def _ms(ng):
    from gppsigma import ops
    d = ops.DeviceInputs.from_host(W.make_inputs(W.Shape(34, 0, 1024, ng, 30000, dw=1e-4), 3))
    ops.sigma(d, "fp64")
    best = 1e9
    for _ in range(3):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        ops.sigma(d, "fp64")
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b))
    ops.wait()
    return best


def test_time_is_linear_in_the_run_length():
    assert _ms(16) <= _ms(15) * 16 / 15


@pytest.mark.parametrize("nw", [31, 32, 33, 64, 67])
def test_runs_at_every_place(nw):
    import oracle_py
    from gppsigma import ops
    inp = W.make_inputs(W.Shape(64, 1, 4099, 17, nw, dw=0.25), nw)
    rng = np.random.default_rng(nw)
    # Far everywhere, then near runs: [start, start + length) of each band.
    inp.wx_array[:] = np.where(rng.uniform(size=inp.wx_array.shape) < 0.5, -6.0, 9.0) \
        + rng.uniform(-1, 1, inp.wx_array.shape)
    for n in range(64):
        start, length = n % nw, [0, 1, 2, 3, 4, 7, 30, 35][(n // 8 + n) % 8]
        inp.wx_array[n, start:start + length] = rng.uniform(0.6, 1.9, inp.wx_array[n, start:start + length].shape)
    want = oracle_py.run(inp, "complex_seq", nthreads=8)
    d = ops.DeviceInputs.from_host(inp)
    lib = capi.load()
    lib.gpp_reset_launch_count()
    r = ops.sigma(d, "fp64", acht_n1=True)
    ops.wait()
    assert lib.gpp_launch_count() > 20
    for key in ("achtemp", "asxtemp", "acht_n1_loc"):
        got, w = getattr(r, key).cpu().numpy(), want[key]
        assert np.max(np.abs(got - w)) <= 1e-12 * np.max(np.abs(w)), key
