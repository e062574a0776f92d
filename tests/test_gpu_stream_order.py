"""Device bounds that the caller's stream is still filling: propagation comes after
what the stream holds, on the default stream (handle 0) as on any other."""
import numpy as np
import pytest

import gdp
import gdpgen

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("sync", [gdp.CPU_LOOP, gdp.GPU_LOOP, gdp.MEGAKERNEL])
@pytest.mark.parametrize("side", [False, True])
def test_bounds_still_being_written(sync, side):
    mip = gdpgen.random_mip(0, seed=24)
    with gdp.Context(mip, sync_type=sync) as ctx:
        rlb, rub, rst = ctx.propagate()
        assert rst["rounds"] > 2
        stream = torch.cuda.Stream() if side else torch.cuda.default_stream()
        lb0, ub0 = torch.tensor(mip.lb, device="cuda"), torch.tensor(mip.ub, device="cuda")
        lb, ub = torch.tensor(rlb, device="cuda"), torch.tensor(rub, device="cuda")  # a fixpoint: one round
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            torch.cuda._sleep(20_000_000)  # about 10 ms
            lb.copy_(lb0)
            ub.copy_(ub0)
            assert (stream.cuda_stream == 0) == (not side)
            st = ctx.propagate_device(lb.data_ptr(), ub.data_ptr(), stream.cuda_stream)
        torch.cuda.synchronize()
        assert st["rounds"] == rst["rounds"]
        assert np.array_equal(lb.cpu().numpy(), rlb) and np.array_equal(ub.cpu().numpy(), rub)


def test_while_a_stream_is_captured():
    """A capture in progress neither fails the call nor is ended by it."""
    mip = gdpgen.random_mip(0, seed=24)
    with gdp.Context(mip) as ctx:
        rlb, rub, rst = ctx.propagate()
        lb, ub = torch.tensor(mip.lb, device="cuda"), torch.tensor(mip.ub, device="cuda")
        a = torch.zeros(8, device="cuda")
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, capture_error_mode="relaxed"):
            a += 1
            st = ctx.propagate_device(lb.data_ptr(), ub.data_ptr(), 0)
        graph.replay()
        torch.cuda.synchronize()
        assert st["rounds"] == rst["rounds"] and a.tolist() == [1.0] * 8
        assert np.array_equal(lb.cpu().numpy(), rlb) and np.array_equal(ub.cpu().numpy(), rub)
