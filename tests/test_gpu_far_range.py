"""The FP64 series (gpp_far.cu) at the ends of FP64's range: I_eps of 1e-309
(every product wtilde I_eps subnormal) against aqsn of 1e20, and I_eps of 1e300
against aqsn of 1e-200, give what the per-term kernels of the allocation-free
entry point give, to 1e-11 of the largest: the subnormal products have 48 bits
or more, the same in both, and what the two sums do with them is FP64's."""
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


def per_term(d, semantics="complex_seq"):
    """achtemp and asxtemp of the per-term FP64 kernels."""
    from gppsigma import ops
    lib = capi.load()
    ach, asx = (torch.empty(d.nw, dtype=torch.complex128, device="cuda") for _ in range(2))
    o = capi.GppOutputs()
    o.achtemp, o.asxtemp = ach.data_ptr(), asx.data_ptr()
    p = ops.problem_struct(d, "fp64", semantics, 1.0)
    capi.check(lib.gpp_sigma_static_scratch(C.byref(p), C.byref(o),
                                            torch.cuda.current_stream().cuda_stream), "static")
    torch.cuda.synchronize()
    return ach.cpu().numpy(), asx.cpu().numpy()


@pytest.mark.parametrize("ieps,aqsn", [(1e-309, 1e20), (1e300, 1e-200)])
def test_chunks_at_the_ends_of_the_range(ieps, aqsn):
    from gppsigma import ops
    inp = W.make_inputs(W.Shape(64, 0, 5003, 17, 32, dw=0.25), 11)
    inp.I_eps_array *= ieps
    inp.aqsntemp *= aqsn
    d = ops.DeviceInputs.from_host(inp)
    lib = capi.load()
    lib.gpp_reset_launch_count()
    r = ops.sigma(d, "fp64")
    ops.wait()
    assert lib.gpp_launch_count() > 20
    want, _ = per_term(d)
    got = r.achtemp.cpu().numpy()
    assert np.all(want != 0) and not np.array_equal(got, want)  # the series ran
    assert np.max(np.abs(got / aqsn - want / aqsn)) <= 1e-11 * np.max(np.abs(want / aqsn))
