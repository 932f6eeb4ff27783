"""learnGradient of small plain fp32 networks at the edges of its tiles and widths, and clears of a few bytes."""
import numpy as np
import pytest

from oracle import oracle
from slang_b200 import config as C

from mlp_testlib import layer_rel_errs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def device():
    from slang_b200.api import Device
    d = Device(0)
    yield d
    d.destroy()


@pytest.mark.parametrize("order", [C.SUM_NEURAL, C.SUM_BIAS_FIRST_FUSED], ids=["neural", "fused"])
@pytest.mark.parametrize("count", [1, 31, 32, 33, 4096, 148 * 4 * 32 + 1, 148 * 4 * 32 * 2 + 31])
@pytest.mark.parametrize("dims", [[1, 1], [2, 16, 16, 16, 1], [3, 32, 31, 5], [32, 32, 32, 32, 32, 32, 32, 32, 32], [17, 6, 18]],
                         ids=lambda d: "-".join(map(str, d)))
def test_small_fp32_networks(device, dims, count, order):
    """Against the oracle.  Samples are summed 32 at a time, then by CTA, then in any order: some sqrt(count) roundings of 2^-24
    of sums that cancel by as much, well below 1e-5 of the largest element of a tensor; a ReLU at the rounding of zero would move
    one sample's share, but both sides add the products of a sample in the same order."""
    from slang_b200.api import Trainer
    cfg = C.make_config(dims, C.F32, C.ACT_RELU, input_dtype=C.F32, target_dtype=C.F32, sum_order=order)
    rng = np.random.default_rng(sum(dims) + count)
    x = rng.uniform(-1, 1, (count, dims[0])).astype(np.float32)
    t = rng.uniform(-1, 1, (count, dims[-1])).astype(np.float32)
    p0 = C.init_params(cfg, seed=3, scheme="kaiming")
    tr = Trainer(device, cfg, p0)
    xb, tb = device.create_buffer(x.nbytes, x), device.create_buffer(t.nbytes, t)
    tr.learn_gradient(xb.address, tb.address, count)
    grads = np.zeros(tr.total, dtype=np.float32)
    ref = oracle.learn_gradient(cfg, p0, grads, x, t, count, n_threads=8).view(np.float32)
    assert max(layer_rel_errs(cfg, tr.read_grads(), grads)) < 1e-5
    largest, total = tr.read_loss()
    assert abs(largest - ref[0]) <= 1e-6 * ref[0] and abs(total - ref[1]) <= 1e-5 * ref[1]


@pytest.mark.parametrize("offset,size", [(0, 8), (4, 4), (1, 3), (8, 64), (3, 61), (16, 65), (5, 1024), (5, 0)])
def test_clears_touch_their_range_only(device, offset, size):
    b = device.create_buffer(8192, np.full(8192, 0xa5, dtype=np.uint8))
    b.clear(offset, size)
    want = np.full(8192, 0xa5, dtype=np.uint8)
    want[offset:offset + size] = 0
    assert np.array_equal(b.read(np.uint8), want)


def test_clears_of_wrapped_memory_stay_memsets(device):
    """A small clear is a kernel where the library owns the memory.  Memory that was wrapped may be anywhere (another device's, or an address that
    only a memset refuses), so no kernel writes there: read from what a capture records, without running it."""
    from cuda.bindings import runtime as rt
    from slang_b200.api import Device

    def ok(result):
        assert result[0] == rt.cudaError_t.cudaSuccess, result[0]
        return result[1] if len(result) == 2 else result[1:]

    stream = ok(rt.cudaStreamCreate())
    d = Device(0, int(stream))
    owned = d.create_buffer(64)
    kinds = []
    for b in (owned, d.wrap_buffer(owned.address, 64)):
        ok(rt.cudaStreamBeginCapture(stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal))
        b.clear(0, 8)
        graph = ok(rt.cudaStreamEndCapture(stream))
        nodes, n = ok(rt.cudaGraphGetNodes(graph, 4))
        assert n == 1
        kinds.append(ok(rt.cudaGraphNodeGetType(nodes[0])))
        rt.cudaGraphDestroy(graph)
    assert kinds == [rt.cudaGraphNodeType.cudaGraphNodeTypeKernel, rt.cudaGraphNodeType.cudaGraphNodeTypeMemset]
    d.destroy()
    rt.cudaStreamDestroy(stream)
