"""A batch plan holds the scratch of its states that take the series
(gpp_batched.cu): runs leave no allocations in their graph, also with another
tile variant set since the plan was made; where the scratch cannot be had (the
library's own self-test: an allocation of that size answers out of memory), the
plan is made all the same and sums every state term by term, and so does
gpp_sigma, to the rounding of the two."""
import ctypes as C

import numpy as np
import pytest

from gppsigma import build, capi, workload as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

RESERVED = 2  # cuda.h, CU_GRAPH_MEM_ATTR_RESERVED_MEM_CURRENT


@pytest.fixture(scope="module", autouse=True)
def _lib():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    build.build()
    capi.load()


def _graph_memory():
    torch.cuda.synchronize()
    cu = C.CDLL("libcuda.so.1")
    assert cu.cuInit(0) == 0
    v = C.c_uint64()
    assert cu.cuDeviceGetGraphMemAttribute(torch.cuda.current_device(), RESERVED, C.byref(v)) == 0
    return v.value


class _Plan:
    def __init__(self, inputs, precision):
        from gppsigma import ops
        n = len(inputs)
        self.keep = [ops.DeviceInputs.from_host(i) for i in inputs]
        self.outs = []
        problems, outs = (capi.GppProblem * n)(), (capi.GppOutputs * n)()
        for k, d in enumerate(self.keep):
            problems[k] = ops.problem_struct(d, precision, "complex_seq", 1.0)
            o = [torch.empty(m, dtype=torch.complex128, device="cuda") for m in (d.nw, d.nw, d.number_bands)]
            outs[k].achtemp, outs[k].asxtemp, outs[k].acht_n1_loc = (t.data_ptr() for t in o)
            self.outs.append(o)
        self.lib, self.handle = capi.load(), C.c_void_p()
        torch.cuda.synchronize()
        capi.check(self.lib.gpp_batch_create(C.byref(self.handle), problems, outs, n), "gpp_batch_create")

    def run(self, stream):
        capi.check(self.lib.gpp_batch_run(self.handle, stream.cuda_stream), "gpp_batch_run")
        stream.synchronize()
        return [[t.cpu().numpy() for t in o] for o in self.outs]

    def close(self):
        self.lib.gpp_batch_destroy(self.handle)


def _inputs():
    return [W.make_inputs(W.Shape(64, 2, 5003, 17, 32, dw=0.25), 3),  # takes the series in FP64
            W.make_inputs(W.Shape(12, 2, 300, 9, 32), 5)]


def _close(a, b, tol):
    return all(np.max(np.abs(x - y)) <= tol * np.max(np.abs(y)) for p, q in zip(a, b) for x, y in zip(p, q))


def test_runs_allocate_nothing():
    before = _graph_memory()
    plan, stream = _Plan(_inputs(), "fp64"), torch.cuda.Stream()
    first = plan.run(stream)
    again = plan.run(stream)
    assert _graph_memory() == before
    assert all(np.array_equal(x, y) for p, q in zip(first, again) for x, y in zip(p, q))
    plan.close()


def test_a_larger_tile_layout_after_the_plan_was_made():
    """More tiles than the plan's scratch was made for (the variants of 8 bands
    a tile leave half as many partial sums as those of 4)."""
    lib = capi.load()
    inputs = [W.make_inputs(W.Shape(64, 2, 20003, 40, 32, dw=0.25), 3)]
    stream = torch.cuda.Stream()
    names = [lib.gpp_variant_name(v).decode() for v in range(lib.gpp_variant_count())]
    try:
        capi.check(lib.gpp_set_variant(32, 8), "gpp_set_variant")
        plan = _Plan(inputs, "mixed")
        want = plan.run(stream)
        plan.close()
        plan = _Plan(inputs, "mixed")
        capi.check(lib.gpp_set_variant(32, 0), names[0])
        got = plan.run(stream)
        plan.close()
    finally:
        capi.check(lib.gpp_set_variant(32, -1), "gpp_set_variant")
    assert _close(got, want, 1e-12)


def test_no_room_for_the_series():
    from gppsigma import ops
    lib = capi.load()
    inputs, stream = _inputs(), torch.cuda.Stream()
    plan = _Plan(inputs, "fp64")
    want = plan.run(stream)
    plan.close()
    capi.check(lib.gpp_selftest_scratch_limit(64 << 20), "limit")
    try:
        plan = _Plan(inputs, "fp64")
        got = plan.run(stream)
        plan.close()
        d = ops.DeviceInputs.from_host(inputs[0])
        lib.gpp_reset_launch_count()
        r = ops.sigma(d, "fp64", acht_n1=True)
        ops.wait()
        assert lib.gpp_launch_count() < 10  # term by term
        alone = [r.achtemp.cpu().numpy(), r.asxtemp.cpu().numpy(), r.acht_n1_loc.cpu().numpy()]
    finally:
        capi.check(lib.gpp_selftest_scratch_limit(0), "limit")
    assert not np.array_equal(got[0][0], want[0][0])
    assert _close(got, want, 1e-12) and _close([alone], want[:1], 1e-12)
    assert all(np.array_equal(x, y) for x, y in zip(got[0], alone))


def test_no_room_inside_a_capture():
    """The same inside a caller's capture, where the allocation is only a node of
    the graph: the captured call sums term by term."""
    from gppsigma import ops
    lib = capi.load()
    d = ops.DeviceInputs.from_host(_inputs()[0])
    out = ops.sigma(d, "fp64")
    ops.wait()
    want = out.achtemp.cpu().numpy()
    capi.check(lib.gpp_selftest_scratch_limit(64 << 20), "limit")
    try:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            ops.sigma(d, "fp64", out=out)
    finally:
        capi.check(lib.gpp_selftest_scratch_limit(0), "limit")
    for _ in range(2):
        out.achtemp.zero_()
        graph.replay()
        torch.cuda.synchronize()
        got = out.achtemp.cpu().numpy()
        assert not np.array_equal(got, want)
        assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))


def test_planes_and_scratch_share_their_memory():
    """A plan's split planes and the scratch of its states that take the series
    are one region, used one after the other: a plan of two such states and a
    small one, run several times, gives every state the bits it has alone."""
    from gppsigma import ops
    inputs = [W.make_inputs(W.Shape(64, 2, 20003, 40, 32, dw=0.25), 3),
              W.make_inputs(W.Shape(40, 2, 3000, 30, 32), 5),
              W.make_inputs(W.Shape(66, 1, 19001, 42, 32, dw=0.25), 4)]
    plan, stream = _Plan(inputs, "mixed"), torch.cuda.Stream()
    runs = [plan.run(stream) for _ in range(3)]
    plan.close()
    for k, inp in enumerate(inputs):
        r = ops.sigma(ops.DeviceInputs.from_host(inp), "mixed", acht_n1=True)
        ops.wait()
        want = [r.achtemp.cpu().numpy(), r.asxtemp.cpu().numpy(), r.acht_n1_loc.cpu().numpy()]
        for got in runs:
            assert all(np.array_equal(x, y) for x, y in zip(got[k], want))
