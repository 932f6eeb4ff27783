"""The arithmetic of hidden activations in the kernels for widths up to 64, where it shows: the activation takes the
pre-activation as it is rounded to the storage type, and a pre-activation that rounds to zero, from either side, is a
zero (with fp32 storage it is not rounded and keeps its side)."""
import numpy as np
import pytest

from oracle import oracle
from slang_b200 import config as C

from mlp_testlib import layer_rel_errs, rel_err

pytestmark = pytest.mark.gpu

STORAGE = {"f16": (C.F16, 0), "bf16": (C.BF16, 0), "f32-f16": (C.F32, C.F16)}


@pytest.fixture(scope="module")
def device():
    from slang_b200.api import Device
    d = Device(0)
    yield d
    d.destroy()


def _config(dims, storage, act, **more):
    dtype, operand = STORAGE[storage]
    return C.make_config(dims, dtype, act, input_dtype=C.F32, target_dtype=C.F32, adam_master=0 if dtype == C.F32 else 1,
                         operand_dtype=operand, **more)


@pytest.mark.parametrize("alpha", [0.01, 0.3])
@pytest.mark.parametrize("storage", list(STORAGE))
@pytest.mark.parametrize("width", [12, 24, 40])
def test_leaky_relu_takes_the_rounded_preactivation(device, width, storage, alpha):
    """One sample through 2-width-width whose every sum is exact in fp32 and whose second layer is the identity: outputs
    and gradients have to equal the oracle's bit for bit."""
    from slang_b200.api import Trainer
    cfg = _config([2, width, width], storage, C.ACT_LEAKY_RELU, act_alpha=alpha)
    rng = np.random.default_rng(width)
    w_off, b_off, total = C.param_layout(cfg)
    p = np.zeros(total, dtype=np.float32)
    w0 = np.empty((width, 2), dtype=np.float32)
    w0[:, 0] = -rng.integers(64, 128, width) / 128.0    # times x_0: eleven bits, and a few more below them from x_1
    w0[:, 1] = rng.integers(-7, 8, width) / 8192.0
    p[w_off[0]:w_off[0] + 2 * width] = w0.ravel()
    p[w_off[1]:w_off[1] + width * width] = np.eye(width, dtype=np.float32).ravel()
    params = C.to_storage(p, cfg.dtype)
    x = np.array([[13.0 / 16.0, 1.0]], dtype=np.float32)
    t = rng.uniform(-1, 1, (1, width)).astype(np.float32)
    tr = Trainer(device, cfg, params)
    xb, tb, yb = device.create_buffer(x.nbytes, x), device.create_buffer(t.nbytes, t), device.create_buffer(4 * width)
    tr.forward(xb.address, yb.address, 1)
    assert np.array_equal(yb.read(np.float32), np.asarray(oracle.forward(cfg, params, x, 1), dtype=np.float32).ravel())
    want = np.zeros(total, dtype=np.float32)
    oracle.learn_gradient(cfg, params, want, x, t, 1)
    tr.learn_gradient(xb.address, tb.address, 1)
    assert np.array_equal(tr.read_grads(), want)


def _around_zero(device, dims, storage, act, count=500):
    """Three samples in four have one input, the smallest half above zero: every first-layer pre-activation is a product
    of less than half of it (biases are zero), of either sign.  Gradients, input gradients and loss against the oracle."""
    from slang_b200.api import Trainer
    cfg = _config(dims, storage, act, act_alpha=0.02)
    rng = np.random.default_rng(sum(dims))
    params = C.init_params(cfg, seed=4, scheme="xavier")
    p = C.from_storage(params, cfg.dtype).copy()
    w_off, b_off, total = C.param_layout(cfg)
    w0 = p[w_off[0]:w_off[0] + dims[0] * dims[1]]
    w0 *= 0.45 / np.abs(w0).max()
    for l in range(1, len(dims) - 1):
        p[b_off[l]:b_off[l] + dims[l + 1]] = rng.uniform(-0.5, 0.5, dims[l + 1])
    params = C.to_storage(p, cfg.dtype)
    x = rng.uniform(-1, 1, (count, dims[0])).astype(np.float32)
    small = np.arange(count) % 4 != 0
    x[small] = 0.0
    x[small, rng.integers(0, dims[0], count)[small]] = np.float32(2.0 ** -24)
    t = rng.uniform(-1, 1, (count, dims[-1])).astype(np.float32)
    want, words = np.zeros(total, dtype=np.float32), np.zeros(2, dtype=np.uint32)
    want_dx = oracle.learn_gradient_inputs(cfg, params, want, x, t, count, words)
    tr = Trainer(device, cfg, params)
    xb, tb = device.create_buffer(x.nbytes, x), device.create_buffer(t.nbytes, t)
    dxb = device.create_buffer(want_dx.nbytes)
    tr.learn_gradient(xb.address, tb.address, count, input_grads_address=dxb.address)
    # 1e-2: the bar of 16-bit gradients in these tests; a derivative of 0, 1/2, alpha or 1 in another's place is 0.1 to 1
    assert max(layer_rel_errs(cfg, tr.read_grads(), want)) < 1e-2
    dx = dxb.read(np.float32).reshape(want_dx.shape)
    assert rel_err(dx, want_dx) < 1e-2
    assert rel_err(dx[small], want_dx[small]) < 1e-2
    largest, total_loss = tr.read_loss()
    ref = words.view(np.float32)
    assert abs(largest - ref[0]) <= 1e-3 * ref[0] and abs(total_loss - ref[1]) <= 1e-3 * ref[1]


AROUND_ZERO = [[4, 32, 32, 4], [32, 24, 3], [6, 64, 48, 64, 3], [40, 64, 20]]


@pytest.mark.parametrize("storage", ["f16", "f32-f16"])
@pytest.mark.parametrize("dims", AROUND_ZERO, ids=lambda d: "-".join(map(str, d)))
def test_leaky_relu_around_zero(device, dims, storage):
    _around_zero(device, dims, storage, C.ACT_LEAKY_RELU)


@pytest.mark.parametrize("storage", ["f16", "f32-f16"])
@pytest.mark.parametrize("dims", AROUND_ZERO, ids=lambda d: "-".join(map(str, d)))
def test_relu_around_zero(device, dims, storage):
    """The derivative at zero is one half, from whichever side the pre-activation was rounded."""
    _around_zero(device, dims, storage, C.ACT_RELU)


# Batches from 1024 samples on (forward 4096) run in whole tiles of 128, networks up to width 128 among them.
@pytest.mark.parametrize("alpha", [0.01, 0.3])
@pytest.mark.parametrize("storage", ["f16", "bf16"])
@pytest.mark.parametrize("dims", [[2, 12, 12], [2, 24, 24], [2, 40, 40], [8, 100, 64]], ids=lambda d: "-".join(map(str, d)))
def test_leaky_relu_takes_the_rounded_preactivation_in_tiles(device, dims, storage, alpha):
    """The sample of the test above inside a batch of samples that are zero and have no gradient: still bit for bit."""
    from slang_b200.api import Trainer
    cfg = _config(dims, storage, C.ACT_LEAKY_RELU, act_alpha=alpha)
    count, width, out = 5001, dims[1], dims[2]
    rng = np.random.default_rng(width)
    w_off, b_off, total = C.param_layout(cfg)
    p = np.zeros(total, dtype=np.float32)
    w0 = np.zeros((width, dims[0]), dtype=np.float32)
    w0[:, 0] = -rng.integers(64, 128, width) / 128.0
    w0[:, 1] = rng.integers(-7, 8, width) / 8192.0
    p[w_off[0]:w_off[0] + w0.size] = w0.ravel()
    p[w_off[1]:w_off[1] + width * out] = np.eye(out, width, dtype=np.float32).ravel()
    params = C.to_storage(p, cfg.dtype)
    x, t = np.zeros((count, dims[0]), dtype=np.float32), np.zeros((count, out), dtype=np.float32)
    x[777, :2] = [13.0 / 16.0, 1.0]
    t[777] = rng.uniform(-1, 1, out)
    tr = Trainer(device, cfg, params)
    xb, tb, yb = device.create_buffer(x.nbytes, x), device.create_buffer(t.nbytes, t), device.create_buffer(4 * count * out)
    dxb = device.create_buffer(x.nbytes)
    tr.forward(xb.address, yb.address, count)
    assert np.array_equal(yb.read(np.float32), np.asarray(oracle.forward(cfg, params, x, count), dtype=np.float32).ravel())
    want, words = np.zeros(total, dtype=np.float32), np.zeros(2, dtype=np.uint32)
    oracle.learn_gradient_inputs(cfg, params, want, x, t, count, words)
    tr.learn_gradient(xb.address, tb.address, count, input_grads_address=dxb.address)
    assert np.array_equal(tr.read_grads(), want)
    dx = dxb.read(np.float32).reshape(x.shape)
    assert np.all(dx[777, :2] != 0) and np.count_nonzero(dx) == np.count_nonzero(dx[777])


@pytest.mark.parametrize("dims,act", [(d, a) for d in AROUND_ZERO + [[32, 128, 128, 3]] for a in (C.ACT_LEAKY_RELU, C.ACT_RELU)] + [([8, 100, 64], C.ACT_LEAKY_RELU)],
                         ids=lambda v: "-".join(map(str, v)) if isinstance(v, list) else {C.ACT_LEAKY_RELU: "leaky", C.ACT_RELU: "relu"}[v])
def test_around_zero_in_tiles(device, dims, act):
    """(ReLU through 8-100-64 runs in tiles from 131072 samples on: test_gpu_chain.py.)"""
    _around_zero(device, dims, "f16", act, count=5000)


@pytest.mark.parametrize("dims", [[1, 32, 3], [1, 40, 8], [1, 16, 1], [1, 24, 2], [1, 64, 4], [1, 33, 5]], ids=lambda d: "-".join(map(str, d)))
def test_output_sigmoid_is_as_exact_as_one_thread_per_sample(device, dims):
    """Outputs are returned in fp32, so the sigmoid is that of the general kernels bit for bit (the output layer copies
    the one input, so both kernels give it the same pre-activation)."""
    from slang_b200.api import Trainer
    cfg = _config(dims, "f16", C.ACT_RELU, output_act=C.ACT_SIGMOID)
    w_off, _, total = C.param_layout(cfg)
    p = np.zeros(total, dtype=np.float32)
    p[w_off[0]], p[w_off[0] + 1] = 1.0, -1.0                # x above zero, and -x above zero
    for o in range(dims[2]):
        p[w_off[1] + o * dims[1]:w_off[1] + o * dims[1] + 2] = [1.0, -1.0]
    params = C.to_storage(p, cfg.dtype)
    x = np.linspace(-12, 12, 5001, dtype=np.float32).reshape(-1, 1)
    xb, yb = device.create_buffer(x.nbytes, x), device.create_buffer(4 * x.size * dims[2])
    outputs = []
    for entry in ("forward", "forward_simt"):
        tr = Trainer(device, cfg, params, forward_entry=entry)
        tr.forward(xb.address, yb.address, x.size)
        outputs.append(yb.read(np.float32).copy())
    assert np.array_equal(outputs[0], outputs[1])


@pytest.mark.parametrize("storage", ["f16", "bf16"])
@pytest.mark.parametrize("dims", [[1, 32, 3], [1, 32, 9], [1, 24, 16], [1, 40, 20], [1, 64, 64]], ids=lambda d: "-".join(map(str, d)))
def test_output_sigmoid_of_every_value(device, dims, storage):
    """The same for every finite pre-activation of the storage type, for few outputs and many."""
    from slang_b200.api import Trainer
    cfg = _config(dims, storage, C.ACT_RELU, output_act=C.ACT_SIGMOID)
    w_off, _, total = C.param_layout(cfg)
    p = np.zeros(total, dtype=np.float32)
    p[w_off[0]], p[w_off[0] + 1] = 1.0, -1.0
    for o in range(dims[2]):
        p[w_off[1] + o * dims[1]:w_off[1] + o * dims[1] + 2] = [1.0, -1.0]
    params = C.to_storage(p, cfg.dtype)
    bits = np.arange(1 << 16, dtype=np.uint32)
    x = bits.astype(np.uint16).view(np.float16).astype(np.float32) if storage == "f16" else (bits << 16).view(np.float32)
    x = np.ascontiguousarray(x[np.isfinite(x)]).reshape(-1, 1)
    xb, yb = device.create_buffer(x.nbytes, x), device.create_buffer(4 * x.size * dims[2])
    outputs = []
    for entry in ("forward", "forward_simt"):
        tr = Trainer(device, cfg, params, forward_entry=entry)
        tr.forward(xb.address, yb.address, x.size)
        outputs.append(yb.read(np.float32).copy().reshape(x.size, dims[2]))
    differ = outputs[0] != outputs[1]
    assert not differ.any(), (int(differ.sum()), x[differ.any(1)][:4], outputs[0][differ][:4], outputs[1][differ][:4])
