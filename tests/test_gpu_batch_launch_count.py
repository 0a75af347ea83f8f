"""gpp_launch_count over a batch: a run replayed from its graph counts what the
same run counts on the default stream, where it is not captured, and that is
at least what the state that takes the series counts alone; a capture counts
nothing of its own."""
import pytest

from gppsigma import build, capi, workload as W
from test_gpu_batch_scratch import _Plan, _inputs

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _lib():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    build.build()
    capi.load()


class _Legacy:
    cuda_stream = 0

    @staticmethod
    def synchronize():
        torch.cuda.synchronize()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_replays_count_what_uncaptured_runs_count(precision):
    from gppsigma import ops
    lib = capi.load()
    inputs = _inputs()

    def count(run):
        lib.gpp_reset_launch_count()
        run()
        return lib.gpp_launch_count()

    plan, stream = _Plan(inputs, precision), torch.cuda.Stream()
    first, replay = count(lambda: plan.run(stream)), count(lambda: plan.run(stream))
    legacy = count(lambda: plan.run(_Legacy))
    plan.close()
    d = ops.DeviceInputs.from_host(inputs[0])
    alone = count(lambda: ops.sigma(d, precision, acht_n1=True))
    torch.cuda.synchronize()
    assert first == replay == legacy
    if precision == "fp64":
        assert alone > 20 and replay > alone
