"""Edges of the kernels' own tiling: samples around a warp's block, a group's unit and a tile; widths around the padded
widths, the fragment layouts (up to 8, up to 16, beyond) and the output tiles; Adam segments around the four-element launch."""
import numpy as np
import pytest

from oracle import oracle
from slang_b200 import config as C

from mlp_testlib import layer_rel_errs, rel_err

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
    _against_the_oracle(device, C.make_config(dims, C.F16, C.ACT_RELU, input_dtype=C.F32, target_dtype=C.F32, adam_master=1), count, 1e-2)


@pytest.mark.parametrize("count", [1, 33, 81, 6001])
@pytest.mark.parametrize("dtype,act", [(C.F16, C.ACT_LEAKY_RELU), (C.F16, C.ACT_GELU_TANH), (C.F16, C.ACT_TANH), (C.BF16, C.ACT_RELU),
                                       (C.BF16, C.ACT_GELU_TANH)], ids=["f16-leaky", "f16-gelu", "f16-any", "bf16-relu", "bf16-gelu"])
@pytest.mark.parametrize("dims", [[8, 32, 32, 8], [17, 64, 64, 64, 64], [5, 40, 2]], ids=lambda d: "-".join(map(str, d)))
def test_other_builds_at_tile_edges(device, dims, dtype, act, count):
    """The builds of the same kernels for the other formats and activations.  In bf16 a sum that rounds the other way is
    2^-8 of its value, and a few of them meet in a gradient."""
    cfg = C.make_config(dims, dtype, act, input_dtype=C.F32, target_dtype=C.F32, adam_master=1)
    _against_the_oracle(device, cfg, count, 2e-2 if dtype == C.BF16 else 1e-2)


def _against_the_oracle(device, cfg, count, bar):
    from slang_b200.api import Trainer
    dims = cfg.layer_dims
    rng = np.random.default_rng(sum(dims) + count)
    x = rng.uniform(-1, 1, (count, dims[0])).astype(np.float32)
    t = rng.uniform(-1, 1, (count, dims[-1])).astype(np.float32)
    p0 = C.init_params(cfg, seed=3, scheme="xavier")
    tr = Trainer(device, cfg, p0)
    xb, tb = device.create_buffer(x.nbytes, x), device.create_buffer(t.nbytes, t)
    yb = device.create_buffer(4 * count * dims[-1])
    tr.learn_gradient(xb.address, tb.address, count)
    grads = np.zeros(tr.total, dtype=np.float32)
    ref = oracle.learn_gradient(cfg, p0, grads, x, t, count, n_threads=8).view(np.float32)
    assert max(layer_rel_errs(cfg, tr.read_grads(), grads)) < bar
    largest, total = tr.read_loss()
    assert abs(largest - ref[0]) <= bar * ref[0] and abs(total - ref[1]) <= bar * ref[1]
    tr.forward(xb.address, yb.address, count)
    want = oracle.forward(cfg, p0, x, count)
    got = yb.read(np.float32).reshape(count, dims[-1])
    assert rel_err(got, np.asarray(want).reshape(got.shape)) < bar


@pytest.mark.parametrize("dtype,master,count", [(C.F32, 0, 148 * 8 * 1024 - 1), (C.F32, 0, 148 * 8 * 1024), (C.F32, 0, 148 * 8 * 1024 + 1023),
                                                (C.F32, 1, 148 * 8 * 1024 + 1023), (C.F16, 1, 148 * 8 * 1024 + 1), (C.BF16, 0, 148 * 8 * 1024 + 1)])
def test_adam_over_large_segments_is_bit_exact(device, dtype, master, count):
    """Four elements a thread, with and without a master copy, and parameters that no gradient has reached."""
    from slang_b200.api import AdjustParamsParams
    cfg = C.make_config([1, 1], dtype, lr=1e-2, adam_master=master)
    rng = np.random.default_rng(5)
    p = C.to_storage(rng.uniform(-1, 1, count).astype(np.float32), dtype)
    st = np.zeros(count, dtype=C.ADAM_STATE_DTYPE)
    st["master"] = C.from_storage(p, dtype)
    pb, sb, gb = device.create_buffer(p.nbytes, p), device.create_buffer(st.nbytes, st), device.create_buffer(4 * count)
    k = device.kernel("adjustParameters", cfg)
    for _ in range(2):
        g = np.where(rng.random(count) < 0.3, rng.normal(size=count), 0.0).astype(np.float32)
        g[:3] = [np.nan, np.inf, -0.0]
        gb.write(g)
        k.dispatch(AdjustParamsParams(sb.address, pb.address, gb.address, count), (count + 255) // 256)
        oracle.adjust_parameters(cfg, st, p, g)
    assert np.array_equal(pb.read(np.uint8), p.view(np.uint8))
    got = sb.read(np.uint8).view(C.ADAM_STATE_DTYPE)
    assert all(np.array_equal(got[f], st[f]) for f in ("mean", "variance", "iteration", "master"))
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
