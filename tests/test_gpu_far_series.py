"""Unoccupied bands with per-band frequencies through the series of
gpp_far.cu, at the smallest sizes that take it, against the oracle: ragged
rows, columns and chunks, one to many frequencies per band, frequencies on
both sides of and inside the plasmon band, strays outside it (next to
frequencies, far beyond them, with a large imaginary part), wtilde spread over
everything (no box pays: the per-term kernel runs, with its bits), columns
over many decades, a NaN; the same bits through gpp_sigma, the host path, a
batch and a captured graph.

Norm-wise tolerances, as in the other suites: FP64 1e-12, mixed 1e-8 vs the
oracle."""
import ctypes as C

import numpy as np
import pytest

from gppsigma import build, capi, workload as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SHAPES = [  # nb, nv, ncouls, ngpown, nw, dw
    (64, 2, 5003, 17, 32, 0.25),   # several chunks, a ragged last one; odd rows
    (130, 3, 12289, 23, 8, 0.5),   # 127 unoccupied: one short of a row tile
    (420, 0, 7937, 17, 3, 1.0),    # several row tiles
    (200, 8, 25601, 33, 1, 1.0),   # one frequency per band
]


@pytest.fixture(scope="module", autouse=True)
def _lib():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    build.build()
    capi.load()


def _inputs(shape, kind):
    nb, nv, nc, ng, nw, dw = shape
    inp = W.make_inputs(W.Shape(nb, nv, nc, ng, nw, dw=dw), 7 * nc + nw)
    rng = np.random.default_rng(nc)
    wt = inp.wtilde_array
    if kind == "strays":
        at = rng.uniform(size=wt.shape) < 0.015
        pick = inp.wx_array.ravel()[rng.integers(0, inp.wx_array.size, wt.shape)]
        off = rng.choice([1e-4, 0.3], wt.shape) * rng.uniform(-1, 1, wt.shape)
        wt[at] = (pick + off + 1e-5j)[at]
        wt[0, :3] = [300.0, 1.0 + 40.0j, -1e9]
    elif kind == "spread":
        wt[:] = rng.uniform(-12, 16, wt.shape) + 1j * rng.uniform(-1, 1, wt.shape)
    elif kind == "decades":
        fall = np.exp(-18.0 * np.arange(nc) / nc)
        inp.aqsntemp *= fall
        inp.I_eps_array *= fall
    return inp


def _run(inp, precision, **kw):
    from gppsigma import ops
    lib = capi.load()
    d = ops.DeviceInputs.from_host(inp)
    lib.gpp_reset_launch_count()
    r = ops.sigma(d, precision, acht_n1=inp.shape.nw >= 3, **kw)
    ops.wait()
    return d, r, lib.gpp_launch_count()


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-8)])
@pytest.mark.parametrize("kind", ["band", "strays", "spread", "decades"])
@pytest.mark.parametrize("shape", SHAPES)
def test_series_against_the_oracle(shape, kind, precision, tol):
    import oracle_py
    inp = _inputs(shape, kind)
    want = oracle_py.run(inp, "complex_seq", nthreads=8)
    d, r, launches = _run(inp, precision)
    if precision == "fp64":
        assert launches > 20  # the series' passes were launched
    keys = ["achtemp", "asxtemp"] + (["acht_n1_loc"] if inp.shape.nw >= 3 else [])
    for key in keys:
        got, w = getattr(r, key).cpu().numpy(), want[key]
        assert np.max(np.abs(got - w)) <= tol * max(np.max(np.abs(w)), 1e-300), key
    if kind == "spread" and precision == "fp64":
        # No box pays: the per-term kernel's own bits (it never takes the series
        # in the allocation-free entry point).
        lib = capi.load()
        from gppsigma import ops
        ach, asx = torch.empty_like(r.achtemp), torch.empty_like(r.asxtemp)
        o = capi.GppOutputs()
        o.achtemp, o.asxtemp = ach.data_ptr(), asx.data_ptr()
        p = ops.problem_struct(d, "fp64", "complex_seq", 1.0)
        capi.check(lib.gpp_sigma_static_scratch(C.byref(p), C.byref(o),
                                                torch.cuda.current_stream().cuda_stream), "static")
        torch.cuda.synchronize()
        assert torch.equal(ach, r.achtemp) and torch.equal(asx, r.asxtemp)


def test_nan_reaches_every_frequency_as_in_the_per_term_kernel():
    inp = _inputs(SHAPES[0], "band")
    inp.wtilde_array[3, 100] = complex(np.nan, 0.0)
    _, r, _ = _run(inp, "fp64")
    assert np.all(np.isnan(r.achtemp.cpu().numpy()))
    inp = _inputs(SHAPES[0], "band")
    inp.aqsntemp[40, 17] = complex(np.inf, 0.0)
    _, r, _ = _run(inp, "fp64")
    n1 = r.acht_n1_loc.cpu().numpy()
    assert not np.isfinite(n1[40]) and np.isfinite(np.delete(n1, 40)).all()


@pytest.mark.parametrize("shape,precision", [(SHAPES[0], "fp64"), ((64, 2, 20003, 40, 32, 0.25), "mixed")])
def test_same_bits_through_every_entry_point(shape, precision):
    from gppsigma import ops
    inp = _inputs(shape, "strays")
    d, r, launches = _run(inp, precision)
    assert launches > 20
    lib = capi.load()
    arrays = {k: getattr(inp, k) for k in ("aqsmtemp", "aqsntemp", "I_eps_array", "wtilde_array",
                                           "vcoul", "inv_igp_index", "indinv", "wx_array")}
    with ops.HostContext() as ctx:
        h = ctx.sigma(arrays, inp.shape, precision, acht_n1=True)
    assert np.array_equal(h["achtemp"], r.achtemp.cpu().numpy())
    assert np.array_equal(h["acht_n1_loc"], r.acht_n1_loc.cpu().numpy())
    # A batch with a small state beside it, replayed from its graph.
    small = ops.DeviceInputs.from_host(W.make_inputs(W.Shape(12, 2, 300, 9, shape[4]), 5))
    problems, outs = (capi.GppProblem * 2)(), (capi.GppOutputs * 2)()
    keep = []
    for k, x in enumerate((small, d)):
        problems[k] = ops.problem_struct(x, precision, "complex_seq", 1.0)
        t = [torch.zeros(n, dtype=torch.complex128, device="cuda")
             for n in (x.nw, x.nw, x.number_bands)]
        keep.append(t)
        outs[k].achtemp, outs[k].asxtemp, outs[k].acht_n1_loc = (v.data_ptr() for v in t)
    handle = C.c_void_p()
    capi.check(lib.gpp_batch_create(C.byref(handle), problems, outs, 2), "gpp_batch_create")
    alone = ops.sigma(small, precision, acht_n1=True)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(2):
        for t in keep:
            for v in t:
                v.zero_()
        torch.cuda.synchronize()
        capi.check(lib.gpp_batch_run(handle, stream.cuda_stream), "gpp_batch_run")
        stream.synchronize()
        for t, want in zip(keep, (alone, r)):
            assert torch.equal(t[0], want.achtemp) and torch.equal(t[1], want.asxtemp)
            assert torch.equal(t[2], want.acht_n1_loc)
    lib.gpp_batch_destroy(handle)
    # A captured call.
    out = ops.SigmaResult(*(torch.zeros_like(v) for v in (r.achtemp, r.asxtemp, r.acht_n1_loc)), None)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops.sigma(d, precision, acht_n1=True, out=out)
    for _ in range(2):
        out.achtemp.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out.achtemp, r.achtemp) and torch.equal(out.acht_n1_loc, r.acht_n1_loc)
