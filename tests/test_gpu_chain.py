"""Kernels that run whole tiles of 128 samples on the tensor pipe: samples around a tile and around the SMs' shares, every padded
width and layer count, input rows of each kind, outputs that leave in each way, pre-activations that are zero."""
import numpy as np
import pytest

from oracle import layout_oracle as LO
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


def _run(device, cfg, count, p0=None, x=None, t=None, input_grads=False):
    """Gradients, loss, outputs and input gradients of the GPU and of the oracle."""
    from slang_b200.api import Trainer
    dims = cfg.layer_dims
    rng = np.random.default_rng(sum(dims) + count)
    width = 2 if cfg.encoding == C.ENC_FREQ2D else dims[0]
    if x is None:
        x = rng.uniform(0 if width == 2 else -1, 1, (count, width))
    x = C.to_storage(x, cfg.input_dtype)
    t = C.to_storage(rng.uniform(-1, 1, (count, dims[-1])) if t is None else t, cfg.target_dtype)
    p0 = C.init_params(cfg, seed=3, scheme="xavier") if p0 is None else p0
    tr = Trainer(device, cfg, p0)
    xb, tb = device.create_buffer(x.nbytes, x), device.create_buffer(t.nbytes, t)
    yb, gb = device.create_buffer(4 * count * dims[-1]), device.create_buffer(4 * count * dims[0])
    tr.learn_gradient(xb.address, tb.address, count, input_grads_address=gb.address if input_grads else 0)
    grads = np.zeros(tr.total, dtype=np.float32)
    ref = oracle.learn_gradient(cfg, p0, grads, x, t, count, n_threads=8).view(np.float32)
    loss = tr.read_loss()
    got = tr.read_grads()
    tr.forward(xb.address, yb.address, count)
    want = np.asarray(oracle.forward(cfg, p0, x, count)).reshape(count, dims[-1])
    out = yb.read(np.float32).reshape(count, dims[-1])
    return got, grads, loss, ref, out, want, gb.read(np.float32).reshape(count, dims[0])


def _check(cfg, result, bar):
    got, grads, loss, ref, out, want, _ = result
    assert max(layer_rel_errs(cfg, got, grads)) < bar
    assert abs(loss[0] - ref[0]) <= bar * ref[0] and abs(loss[1] - ref[1]) <= bar * ref[1]
    assert rel_err(out, want) < bar


@pytest.mark.parametrize("count", [1023, 1024, 1025, 1151, 4095, 4096, 4097, 148 * 128 * 3 + 1])
@pytest.mark.parametrize("dims", [[4, 32, 32, 32, 32, 4], [32, 64, 64, 64, 3], [64, 64, 64, 64, 64], [9, 17, 1], [32, 128, 128, 3]], ids=lambda d: "-".join(map(str, d)))
def test_counts_around_a_tile(device, dims, count):
    cfg = C.make_config(dims, C.F16, C.ACT_RELU, input_dtype=C.F32, target_dtype=C.F32, adam_master=1)
    _check(cfg, _run(device, cfg, count), 1e-2)


@pytest.mark.parametrize("dtype,act", [(C.F16, C.ACT_RELU), (C.BF16, C.ACT_RELU), (C.F16, C.ACT_LEAKY_RELU), (C.BF16, C.ACT_LEAKY_RELU)],
                         ids=["f16-relu", "bf16-relu", "f16-leaky", "bf16-leaky"])
@pytest.mark.parametrize("dims,input_dtype", [([1, 2, 1], C.F32), ([16, 32, 16], C.F32), ([31, 33, 33, 17], C.F32), ([12, 20, 20, 20, 20, 5], C.F32),
                                              ([24, 64, 64, 64, 16], None), ([40, 48, 48, 48, 64], None), ([33, 64, 64, 9], None),
                                              ([20, 50, 50, 50, 50, 8], C.F32), ([8, 32, 32, 32, 32], None), ([7, 40, 4], None), ([32, 128, 128, 3], None),
                                              ([64, 128, 64], None), ([24, 100, 66, 20], None), ([16, 65, 1], C.F32), ([40, 128, 128, 16], C.F32),
                                              ([8, 90, 128, 100, 16], None)],
                         ids=lambda v: "-".join(map(str, v)) if isinstance(v, list) else "f32" if v == C.F32 else "own")
def test_shapes_and_formats(device, dims, input_dtype, dtype, act):
    """Rows that are read as values, as whole pieces and converted one by one; every build but those of ReLU at width 128 that take larger batches
    only (test_relu_builds_of_large_batches).  In bf16 a sum that rounds the other way is 2^-8 of its value, and a few of them meet in a gradient."""
    cfg = C.make_config(dims, dtype, act, input_dtype=dtype if input_dtype is None else input_dtype, target_dtype=C.F32 if dims[-1] % 2 else dtype, adam_master=1)
    _check(cfg, _run(device, cfg, 5003), 2e-2 if dtype == C.BF16 else 1e-2)


@pytest.mark.parametrize("out", [3, 20])
def test_frequency_encoding(device, out):
    cfg = C.make_config([32, 64, 64, out], C.F16, C.ACT_RELU, output_act=C.ACT_SIGMOID, loss=C.LOSS_L2_SUM, encoding=C.ENC_FREQ2D, input_dtype=C.F32,
                        target_dtype=C.F32, adam_master=1)
    _check(cfg, _run(device, cfg, 6001), 1e-2)


@pytest.mark.parametrize("dims", [[8, 32, 32, 4], [32, 64, 64, 3], [36, 64, 64, 20], [32, 128, 128, 3]], ids=lambda d: "-".join(map(str, d)))
def test_zero_preactivations_pass_half_of_the_gradient(device, dims):
    """Samples whose inputs are all zero meet zero biases: their pre-activations are zero in every layer."""
    cfg = C.make_config(dims, C.F16, C.ACT_RELU, input_dtype=C.F32, target_dtype=C.F32, adam_master=1)
    rng = np.random.default_rng(1)
    x = rng.uniform(-1, 1, (3000, dims[0])) * (rng.random((3000, 1)) < 0.5)
    p0 = C.from_storage(C.init_params(cfg, seed=3, scheme="xavier"), C.F16)
    _, b_off, _ = C.param_layout(cfg)
    for l in range(cfg.n_layers):
        p0[b_off[l]:b_off[l] + dims[l + 1]] = 0.0
    _check(cfg, _run(device, cfg, 3000, C.to_storage(p0, C.F16), x), 1e-2)


@pytest.mark.parametrize("dims", [[8, 32, 32, 4], [32, 64, 64, 3], [40, 64, 64, 20], [7, 24, 3], [32, 128, 128, 3]], ids=lambda d: "-".join(map(str, d)))
def test_input_gradients(device, dims):
    """Against the chain rule in fp64 over the stored weights.  Roundings to half (2^-11) leave a row within a few 1e-3, except
    where a pre-activation lies so close to zero that they carry it over the kink: 2^-11 of a unit's range, some 192 units
    a sample, so one or two rows in a hundred differ by a whole slope."""
    cfg = C.make_config(dims, C.F16, C.ACT_LEAKY_RELU, input_dtype=C.F32, target_dtype=C.F32, adam_master=1)
    count = 2049
    p0 = C.init_params(cfg, seed=3, scheme="xavier")
    rng = np.random.default_rng(sum(dims) + count)
    x = rng.uniform(-1, 1, (count, dims[0])).astype(np.float32)
    t = rng.uniform(-1, 1, (count, dims[-1])).astype(np.float32)
    p = C.from_storage(p0, C.F16).astype(np.float64)
    w_off, b_off, _ = C.param_layout(cfg)
    a, zs = x.astype(np.float16).astype(np.float64), []
    for l in range(cfg.n_layers):
        w = p[w_off[l]:w_off[l] + dims[l] * dims[l + 1]].reshape(dims[l + 1], dims[l])
        z = a @ w.T + p[b_off[l]:b_off[l] + dims[l + 1]]
        zs.append(z)
        a = np.where(z < 0, cfg.act_alpha * z, z) if l < cfg.n_layers - 1 else z
    g = 2.0 / dims[-1] * (a - t)
    for l in reversed(range(cfg.n_layers)):
        w = p[w_off[l]:w_off[l] + dims[l] * dims[l + 1]].reshape(dims[l + 1], dims[l])
        g = g @ w
        if l > 0:
            g = g * np.where(zs[l - 1] < 0, cfg.act_alpha, 1.0)
    got = _run(device, cfg, count, p0, x, t, input_grads=True)[6]
    rows = np.linalg.norm(got - g, axis=1) / np.linalg.norm(g, axis=1)
    assert np.mean(rows > 1e-2) < 0.05, np.mean(rows > 1e-2)
    assert np.linalg.norm(got - g) / np.linalg.norm(g) < 0.1


@pytest.mark.parametrize("dims", [[20, 48, 64, 3], [4, 32, 32, 32, 32, 4], [32, 96, 128, 10]], ids=lambda d: "-".join(map(str, d)))
def test_optimal_layout_parameters(device, dims):
    """Parameters and gradients in 16x16 tiles: the outputs are those of the same parameters by rows, the gradients too (to the
    order of the CTAs' fp32 sums), each at its weight's place."""
    results = []
    for tiled in (False, True):
        cfg = C.make_config(dims, C.F16, C.ACT_RELU, input_dtype=C.F16, target_dtype=C.F32, adam_master=1)
        p0 = C.init_params(cfg, seed=5, scheme="xavier")
        w_off, b_off, total = C.param_layout(cfg)
        at = np.full(total, -1, dtype=np.int64)   # where each parameter lies
        if tiled:
            cfg.param_layout = C.PARAMS_OPTIMAL
            ow, ob, ototal = C.param_layout(cfg)
            for l in range(cfg.n_layers):
                out16 = LO.align16(dims[l + 1])
                for o in range(dims[l + 1]):
                    for i in range(dims[l]):
                        at[w_off[l] + o * dims[l] + i] = ow[l] + ((i // 16) * (out16 // 16) + o // 16) * 256 + LO.native_tile_pos(i % 16, o % 16)
                    at[b_off[l] + o] = ob[l] + o
            tp = np.zeros(ototal, dtype=p0.dtype)
            tp[at[at >= 0]] = p0[at >= 0]
            p0 = tp
        got, _, loss, _, out, _, _ = _run(device, cfg, 4100, p0)
        if tiled:
            rows = np.zeros(total, dtype=got.dtype)
            rows[at >= 0] = got[at[at >= 0]]
            got = rows
        results.append((got, loss, out))
    assert rel_err(results[1][0], results[0][0]) < 1e-5
    assert abs(results[1][1][1] - results[0][1][1]) <= 1e-5 * results[0][1][1]
    assert np.array_equal(results[1][2], results[0][2])


@pytest.mark.parametrize("count", [1024, 3000])
def test_a_sample_that_overflows_reaches_every_gradient(device, count):
    """Width 128: one sample's output is not a number, so no gradient it enters is, whichever ReLUs are off."""
    cfg = C.make_config([32, 128, 128, 3], C.F16, C.ACT_RELU, input_dtype=C.F16, target_dtype=C.F32, adam_master=1)
    x = np.random.default_rng(1).normal(size=(count, 32))
    x[77] = 6e4
    got, grads, loss, ref, _, _, _ = _run(device, cfg, count, None, x)
    assert np.isnan(ref[1]) and np.isnan(loss[1])
    assert np.array_equal(np.isnan(got), np.isnan(grads))


@pytest.mark.parametrize("where", ["output", "hidden"])
@pytest.mark.parametrize("dtype", [C.F16, C.BF16], ids=["f16", "bf16"])
@pytest.mark.parametrize("dims,count", [([32, 128, 128, 3], 1024), ([16, 96, 100, 3], 1100), ([64, 128, 64], 131072 + 77), ([40, 128, 128, 16], 65536 + 77),
                                        ([8, 90, 128, 100, 16], 65536 + 77)], ids=lambda v: "-".join(map(str, v)) if isinstance(v, list) else str(v))
def test_an_overflow_reaches_the_gradients_that_the_oracle_says(device, dims, count, dtype, where):
    """Width 128: one sample's dZ overflows, in the output layer (whose loss is finite in half), or first in the layer below, where weights of 1/2 keep
    a dA in range and weights of 30 do not.  A ReLU that is off turns an infinite dA into a NaN, a finite one into zero: the same
    entries as the oracle's are NaN, infinite and finite."""
    from slang_b200.api import Trainer
    cfg = C.make_config(dims, dtype, C.ACT_RELU, loss=C.LOSS_L2_SUM, input_dtype=dtype, target_dtype=C.F32, adam_master=1)
    rng = np.random.default_rng(count)
    p = C.from_storage(C.init_params(cfg, seed=3, scheme="xavier"), dtype).copy()
    x = C.to_storage(rng.uniform(-1, 1, (count, dims[0])), dtype)
    t = rng.uniform(-1, 1, (count, dims[-1])).astype(np.float32)
    w_off, _, total = C.param_layout(cfg)
    if where == "output":
        t[77, 0] = 5e4 if dtype == C.F16 else 3e38
    else:
        t[77, 0] = 1.5e4 if dtype == C.F16 else 5e37
        p[w_off[-1]:w_off[-1] + dims[-2]] = rng.choice([0.5, 30.0], dims[-2])
    params = C.to_storage(p, dtype)
    tr = Trainer(device, cfg, params)
    xb, tb, gb = device.create_buffer(x.nbytes, x), device.create_buffer(t.nbytes, t), device.create_buffer(4 * count * dims[0])
    tr.learn_gradient(xb.address, tb.address, count, input_grads_address=gb.address)
    want = np.zeros(total, dtype=np.float32)
    loss = oracle.learn_gradient(cfg, params, want, x, t, count, n_threads=8).view(np.float32)
    if where == "output" and dtype == C.F16:
        assert np.isfinite(loss).all()
    assert not np.isfinite(want).all() and np.isfinite(want).any()
    want_dx = oracle.learn_gradient_inputs(cfg, params, np.zeros(total, dtype=np.float32), x, t, 200, np.zeros(2, dtype=np.uint32)).ravel()
    for got, ref in ((tr.read_grads(), want), (gb.read(np.float32)[:want_dx.size], want_dx)):
        assert np.array_equal(np.isnan(got), np.isnan(ref))
        assert np.array_equal(np.isposinf(got), np.isposinf(ref)) and np.array_equal(np.isneginf(got), np.isneginf(ref))


@pytest.mark.parametrize("dims,dtype", [([16, 32, 3], C.F16), ([4, 32, 32, 32, 32, 4], C.F16), ([20, 24, 30, 16], C.BF16), ([32, 128, 128, 3], C.F16),
                                        ([64, 128, 64], C.F16), ([32, 128, 128, 128, 3], C.F16)], ids=lambda v: "-".join(map(str, v)) if isinstance(v, list) else {C.F16: "f16", C.BF16: "bf16"}[v])
def test_long_sums_are_not_cut_off(device, dims, dtype):
    """A sample over and over: the sums are one sample's gradients times the count.  (Values and weights are small multiples of powers of
    two, so one sample's arithmetic is the same in every kernel.)  Tensor memory drops what does not fit, at every addition and inside it: over four
    tiles of eight additions, to a sum that is half the final one on average, 32 / 2 * 2 * 2^-23 = 3.8e-6.  A CTA's 14 windows and 148 CTAs are added in fp32,
    (14 + 148) / 2 * 2^-24 = 4.8e-6 if every rounding goes the same way: 9e-6 in all.  Cut off over a CTA's 55 tiles the sums are 4e-5 short.
    Width 128: of dW_0 and the biases (the other dW are summed over all tiles)."""
    from slang_b200.api import Trainer
    cfg = C.make_config(dims, dtype, C.ACT_RELU, input_dtype=dtype, target_dtype=C.F32, adam_master=1)
    rng = np.random.default_rng(7)
    w_off, b_off, total = C.param_layout(cfg)
    p = np.zeros(total, dtype=np.float32)
    for l in range(cfg.n_layers):
        p[w_off[l]:w_off[l] + dims[l] * dims[l + 1]] = rng.integers(1, 8, dims[l] * dims[l + 1]) / 256.0
        p[b_off[l]:b_off[l] + dims[l + 1]] = rng.integers(1, 8, dims[l + 1]) / 16.0
    params = C.to_storage(p, dtype)
    count = (1 << 20) + 77
    x = np.tile(C.to_storage(rng.integers(1, 8, (1, dims[0])) / 8.0, dtype), (count, 1))
    t = np.tile(-rng.integers(8, 16, (1, dims[-1])).astype(np.float32) / 8, (count, 1))
    grads = []
    for n in (1, count):
        tr = Trainer(device, cfg, params)
        xb, tb = device.create_buffer(x[:n].nbytes, x[:n]), device.create_buffer(t[:n].nbytes, t[:n])
        tr.learn_gradient(xb.address, tb.address, n)
        grads.append(tr.read_grads().astype(np.float64))
        xb.destroy(); tb.destroy()
    want, got = grads[0] * count, grads[1]
    for l in range(cfg.n_layers):
        parts = [slice(b_off[l], b_off[l] + dims[l + 1])]
        if max(dims) <= 32 or l == 0:
            parts.append(slice(w_off[l], w_off[l] + dims[l] * dims[l + 1]))
        for part in parts:
            assert np.all(want[part] != 0)
            assert np.max(np.abs(got[part] / want[part] - 1)) < 9e-6


@pytest.mark.parametrize("dtype", [C.F16, C.BF16], ids=["f16", "bf16"])
@pytest.mark.parametrize("dims,count", [([64, 128, 64], 131072 + 77), ([24, 70, 40], 131072), ([40, 128, 128, 16], 65536 + 77), ([8, 90, 128, 100, 16], 65536 + 77),
                                        ([32, 128, 128, 128, 3], 65536)], ids=lambda v: "-".join(map(str, v)) if isinstance(v, list) else str(v))
def test_relu_builds_of_large_batches(device, dims, count, dtype):
    """Width 128, with input gradients; a third of the samples are zero and meet zero biases, so their pre-activations are zero in every layer."""
    cfg = C.make_config(dims, dtype, C.ACT_RELU, input_dtype=dtype, target_dtype=C.F32, adam_master=1)
    rng = np.random.default_rng(count)
    x = rng.uniform(-1, 1, (count, dims[0])) * (rng.random((count, 1)) < 0.7)
    t = rng.uniform(-1, 1, (count, dims[-1]))
    p0 = C.from_storage(C.init_params(cfg, seed=3, scheme="xavier"), dtype)
    w_off, b_off, total = C.param_layout(cfg)
    for l in range(cfg.n_layers):
        p0[b_off[l]:b_off[l] + dims[l + 1]] = 0.0
    p0 = C.to_storage(p0, dtype)
    bar = 2e-2 if dtype == C.BF16 else 1e-2
    result = _run(device, cfg, count, p0, x, t, input_grads=True)
    _check(cfg, result, bar)
    n = 300
    dx = oracle.learn_gradient_inputs(cfg, p0, np.zeros(total, dtype=np.float32), C.to_storage(x, dtype), C.to_storage(t, C.F32), n, np.zeros(2, dtype=np.uint32))
    assert rel_err(result[6][:n], dx[:n]) < bar


@pytest.mark.parametrize("dtype,act", [(C.F16, C.ACT_RELU), (C.BF16, C.ACT_RELU), (C.BF16, C.ACT_LEAKY_RELU)], ids=["f16-relu", "bf16-relu", "bf16-leaky"])
@pytest.mark.parametrize("dims", [[8, 32, 32, 4], [7, 24, 3], [32, 64, 64, 3], [40, 64, 64, 20], [32, 128, 128, 3]], ids=lambda d: "-".join(map(str, d)))
def test_input_gradients_against_the_oracle(device, dims, dtype, act):
    """The other formats and activations; the oracle rounds where the kernels do, so what is left is the order of sums of 16-bit values."""
    cfg = C.make_config(dims, dtype, act, input_dtype=C.F32, target_dtype=C.F32, adam_master=1)
    count = 1100
    rng = np.random.default_rng(sum(dims))
    x, t = rng.uniform(-1, 1, (count, dims[0])).astype(np.float32), rng.uniform(-1, 1, (count, dims[-1])).astype(np.float32)
    p0 = C.init_params(cfg, seed=3, scheme="xavier")
    want = oracle.learn_gradient_inputs(cfg, p0, np.zeros(C.param_layout(cfg)[2], dtype=np.float32), x, t, count, np.zeros(2, dtype=np.uint32))
    got = _run(device, cfg, count, p0, x, t, input_grads=True)[6]
    assert rel_err(got, want) < (2e-2 if dtype == C.BF16 else 1e-2)


@pytest.mark.parametrize("dims,input_dtype", [([8, 24, 8], C.F32), ([8, 24, 8], C.F16), ([16, 32, 16], C.F32), ([24, 32, 32, 4], C.F16), ([40, 64, 64, 20], C.F32),
                                              ([32, 64, 64, 64, 4], C.F16), ([32, 128, 128, 4], C.F16), ([32, 128, 128, 4], C.F32), ([32, 70, 70, 4], C.F16)],
                         ids=lambda v: "-".join(map(str, v)) if isinstance(v, list) else {C.F32: "f32", C.F16: "f16"}[v])
def test_memory_off_its_boundary(device, dims, input_dtype):
    """Rows, outputs, parameters and gradients one element past a 16-byte boundary (width 128: not its input rows): the values of aligned ones, the sums of
    gradients in another order.  (32-70-70-4 of this many samples runs in tc_kernels.cu.)"""
    from slang_b200.api import Trainer
    cfg = C.make_config(dims, C.F16, C.ACT_RELU, input_dtype=input_dtype, target_dtype=C.F32, adam_master=1)
    count = 4500
    rng = np.random.default_rng(sum(dims))
    x, t = C.to_storage(rng.uniform(-1, 1, (count, dims[0])), input_dtype), rng.uniform(-1, 1, (count, dims[-1])).astype(np.float32)
    p0 = C.init_params(cfg, seed=3, scheme="xavier")
    results = []
    for off in (0, 1):
        buffers = []

        def memory(nbytes, shift, data=None):
            b = device.create_buffer(nbytes + 64)
            buffers.append(b)
            if data is not None:
                b.write(data, offset=shift)
            return b.address + shift

        params, grads = memory(p0.nbytes, 2 * off), memory(4 * p0.size, 4 * off)
        tr = Trainer(device, cfg, p0, param_memory=(params, grads))
        xa = memory(x.nbytes, x.itemsize * off if max(dims) <= 64 else 0, x)
        ta = memory(t.nbytes, 4 * off, t)
        dx, y = memory(4 * count * dims[0], 4 * off), memory(4 * count * dims[-1], 4 * off)
        tr.learn_gradient(xa, ta, count, input_grads_address=dx)
        if max(dims) <= 64:   # (the other forward kernels want their memory aligned)
            tr.forward(xa, y, count)
        results.append([device.wrap_buffer(dx, 4 * count * dims[0]).read(np.float32), device.wrap_buffer(y, 4 * count * dims[-1]).read(np.float32), tr.read_grads(), tr.read_loss()])
    assert np.array_equal(results[0][0], results[1][0]) and np.array_equal(results[0][1], results[1][1])
    assert np.any(results[0][0]) and rel_err(results[1][2], results[0][2]) < 1e-5
    assert results[0][3][0] == results[1][3][0] and abs(results[0][3][1] - results[1][3][1]) <= 1e-5 * results[0][3][1]


@pytest.mark.parametrize("count", [500, 5000])
def test_misaligned_input_rows_of_wide_networks_are_refused(device, count):
    """By the host, in every batch."""
    from slang_b200.api import Trainer
    from slang_b200.lib import MlpError
    for input_dtype, shift in ((C.F16, 2), (C.F32, 4)):
        cfg = C.make_config([32, 128, 128, 3], C.F16, C.ACT_RELU, input_dtype=input_dtype, target_dtype=C.F32, adam_master=1)
        tr = Trainer(device, cfg, C.init_params(cfg, seed=3, scheme="xavier"))
        xb, tb = device.create_buffer(4 * 32 * count + 64), device.create_buffer(12 * count)
        with pytest.raises(MlpError):
            tr.learn_gradient(xb.address + shift, tb.address, count)
        tr.learn_gradient(xb.address, tb.address, count)
    device.wait()


@pytest.mark.parametrize("tiles", [4 * 148, 5 * 148, 8 * 148 - 1, 33 * 148 + 1])
@pytest.mark.parametrize("dims", [[9, 17, 1], [4, 32, 32, 32, 32, 4], [16, 100, 3]], ids=lambda d: "-".join(map(str, d)))
def test_windows_of_tiles(device, dims, tiles):
    """Gradients leave tensor memory every four tiles (width 32), every tile and every 16th (width 128): batches that end with a window, behind one, or before."""
    cfg = C.make_config(dims, C.F16, C.ACT_RELU, input_dtype=C.F16, target_dtype=C.F32, adam_master=1)
    _check(cfg, _run(device, cfg, 128 * tiles - 5), 1e-2)


@pytest.mark.parametrize("count", [4096 + 61, 20000])
@pytest.mark.parametrize("dims,dtype,input_dtype", [([20, 30, 30, 16], C.F16, C.F16), ([50, 44, 44, 40], C.F16, C.F32), ([50, 64, 48], C.BF16, C.BF16), ([37, 54, 6], C.BF16, C.F32), ([63, 40, 8], C.F16, C.F16),
                                                    ([18, 24, 5], C.F16, C.F32), ([25, 40, 8], C.F16, C.BF16), ([30, 40, 40, 8], C.F16, C.BF16), ([13, 41, 12], C.F16, C.F16), ([11, 20, 5], C.BF16, C.F32)],
                         ids=lambda v: "-".join(map(str, v)) if isinstance(v, list) else {C.F16: "f16", C.BF16: "bf16", C.F32: "f32"}[v])
def test_ragged_input_rows(device, dims, dtype, input_dtype, count):
    """Input rows that are no whole 16-byte pieces: even and odd widths, each number format, last tiles with few rows."""
    cfg = C.make_config(dims, dtype, C.ACT_RELU, input_dtype=input_dtype, target_dtype=C.F32, adam_master=1)
    _check(cfg, _run(device, cfg, count), 2e-2 if dtype == C.BF16 else 1e-2)


def test_a_first_call_with_fp32_rows_can_be_captured():
    """Width 128, fp32 input rows: nothing is converted in front and nothing allocated, so the first call of a device may be recorded."""
    from cuda.bindings import runtime as rt
    from slang_b200.api import Device, Trainer
    err, stream = rt.cudaStreamCreate()
    assert err == rt.cudaError_t.cudaSuccess
    for dims in ([32, 128, 128, 3], [32, 70, 70, 3]):
        d = Device(0, int(stream))
        cfg = C.make_config(dims, C.F16, C.ACT_RELU, input_dtype=C.F32, target_dtype=C.F32, adam_master=1)
        tr = Trainer(d, cfg, C.init_params(cfg, seed=3, scheme="xavier"))
        xb, tb = d.create_buffer(4 * 32 * 4096), d.create_buffer(4 * 3 * 4096)
        d.wait()
        assert rt.cudaStreamBeginCapture(stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal)[0] == rt.cudaError_t.cudaSuccess
        try:
            tr.learn_gradient(xb.address, tb.address, 4096)
        finally:
            err, graph = rt.cudaStreamEndCapture(stream)
        assert err == rt.cudaError_t.cudaSuccess
        rt.cudaGraphDestroy(graph)
        d.destroy()
    rt.cudaStreamDestroy(stream)
