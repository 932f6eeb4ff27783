"""Edges of the kernels' own tiling: samples around a warp's block, a group's unit and a tile; widths around the padded
widths, the fragment layouts (up to 8, up to 16, beyond) and the output tiles; Adam segments around the four-element launch."""
import numpy as np
import pytest

from oracle import oracle
from slang_b200 import config as C

from mlp_testlib import rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def device():
    from slang_b200.api import Device
    d = Device(0)
    yield d
    d.destroy()


@pytest.mark.parametrize("count", [1, 15, 16, 17, 79, 80, 81, 20001])
@pytest.mark.parametrize("dims", [[1, 17, 1], [8, 32, 32, 8], [9, 33, 16], [16, 31, 9], [17, 64, 64, 64, 64], [3, 64, 65, 5]],
                         ids=lambda d: "-".join(map(str, d)))
def test_training_and_forward_at_tile_edges(device, dims, count):
    """Gradients, loss and outputs of the fastest kernels against the oracle (fp16, ReLU)."""
    from slang_b200.api import Trainer
    cfg = C.make_config(dims, C.F16, C.ACT_RELU, input_dtype=C.F32, target_dtype=C.F32, adam_master=1)
    rng = np.random.default_rng(sum(dims) + count)
    x = rng.uniform(-1, 1, (count, dims[0])).astype(np.float32)
    t = rng.uniform(-1, 1, (count, dims[-1])).astype(np.float32)
    p0 = C.init_params(cfg, seed=3, scheme="xavier")
    tr = Trainer(device, cfg, p0)
    xb, tb = device.create_buffer(x.nbytes, x), device.create_buffer(t.nbytes, t)
    yb = device.create_buffer(4 * count * dims[-1])
    tr.learn_gradient(xb.address, tb.address, count)
    grads = np.zeros(tr.total, dtype=np.float32)
    oracle.learn_gradient(cfg, p0, grads, x, t, count, n_threads=8)
    assert rel_err(tr.read_grads(), grads) < 1e-2
    tr.forward(xb.address, yb.address, count)
    want = oracle.forward(cfg, p0, x, count)
    got = yb.read(np.float32).reshape(count, dims[-1])
    assert rel_err(got, np.asarray(want).reshape(got.shape)) < 1e-2


@pytest.mark.parametrize("count", [148 * 8 * 1024 - 1, 148 * 8 * 1024, 148 * 8 * 1024 + 1023])
def test_adam_over_large_segments_is_bit_exact(device, count):
    """Four elements a thread, and parameters that no gradient has reached."""
    from slang_b200.api import AdjustParamsParams
    cfg = C.make_config([1, 1], C.F32, lr=1e-2)
    rng = np.random.default_rng(5)
    p = rng.uniform(-1, 1, count).astype(np.float32)
    st = np.zeros(count, dtype=C.ADAM_STATE_DTYPE)
    st["master"] = p
    pb, sb, gb = device.create_buffer(p.nbytes, p), device.create_buffer(st.nbytes, st), device.create_buffer(p.nbytes)
    k = device.kernel("adjustParameters", cfg)
    for _ in range(2):
        g = np.where(rng.random(count) < 0.3, rng.normal(size=count), 0.0).astype(np.float32)
        g[:3] = [np.nan, np.inf, -0.0]
        gb.write(g)
        k.dispatch(AdjustParamsParams(sb.address, pb.address, gb.address, count), (count + 255) // 256)
        oracle.adjust_parameters(cfg, st, p, g)
    assert np.array_equal(pb.read(np.float32).view(np.uint32), p.view(np.uint32))
    got = sb.read(np.uint8).view(C.ADAM_STATE_DTYPE)
    assert all(np.array_equal(got[f], st[f]) for f in ("mean", "variance", "iteration"))
    assert not gb.read(np.float32).any()


@pytest.mark.parametrize("train", [[64, 64, 64, 64], [8, 24, 24, 4]], ids=["tensor-memory", "registers"])
@pytest.mark.parametrize("width", [16, 64, 128])
def test_inference_and_training_steps_back_to_back(device, width, train):
    """A forward pass and a training step of another network, each launched to overlap the one before: what they compute
    is what they compute with a wait in between."""
    from slang_b200.api import Trainer
    fcfg = C.make_config([width] * 5, C.F16, C.ACT_RELU, input_dtype=C.F16, target_dtype=C.F32)
    tcfg = C.make_config(train, C.F16, C.ACT_RELU, input_dtype=C.F32, target_dtype=C.F32, adam_master=1)
    count = 40000
    rng = np.random.default_rng(width)
    fx = device.create_buffer(2 * count * width, C.to_storage(rng.uniform(-1, 1, (count, width)), C.F16))
    fy = device.create_buffer(4 * count * width)
    x = device.create_buffer(4 * count * train[0], rng.uniform(-1, 1, (count, train[0])).astype(np.float32))
    t = device.create_buffer(4 * count * train[-1], rng.uniform(-1, 1, (count, train[-1])).astype(np.float32))
    ftr = Trainer(device, fcfg, C.init_params(fcfg, seed=1, scheme="kaiming"))
    ttr = Trainer(device, tcfg, C.init_params(tcfg, seed=2, scheme="kaiming"))
    results = []
    for wait in (True, False):
        ttr.grads.clear()
        for _ in range(20):
            for call in (lambda: ftr.forward(fx.address, fy.address, count),
                         lambda: ttr.learn_gradient(x.address, t.address, count, clear_loss=False)):
                call()
                if wait:
                    device.wait()
        results.append((ttr.read_grads(), fy.read(np.uint32).copy()))
        fy.clear()
    assert rel_err(results[1][0], results[0][0]) < 1e-5   # fp32 sums of the CTAs in another order
    assert np.array_equal(results[0][1], results[1][1])
