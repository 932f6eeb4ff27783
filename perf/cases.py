"""The work a program gives this library, as measurable cases.

A case is a dict of plain values.  `listed()` names the fixed ones, `draw(rng)` gives further ones of the same
ranges, `prepare` makes what a program has in hand before the call (inputs on the device, or in pinned host memory
where the call takes host data, and the trainer it keeps), `run` makes one call of the public Python front ends, and
`work` / `tolerance` state the least traffic and arithmetic of a pass and how far two correct results may differ.

Kinds of work:
  example  one iteration of the literal example program's loop: clear the loss, learnGradient, adjustParameters
  train    one training step from tensors on the device (TorchTrainer.learn_gradient + adjust_parameters)
  encoded  one training step of a hash-grid encoder with a network behind it (EncodedTrainer)
  forward  inference from tensors on the device (TorchTrainer.forward)
  host     one training step whose batch starts in pinned host memory (HostStepper.step)
"""
import math
import weakref

import numpy as np
import torch

from slang_b200 import api
from slang_b200 import config as C
from slang_b200 import permuto as P
from slang_b200.encoded import EncodedTrainer
from slang_b200.host_step import HostStepper
from slang_b200.lib import load
from slang_b200.torch_api import TorchTrainer

DTYPES = {"f32": C.F32, "f16": C.F16, "bf16": C.BF16}
TORCH = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
ACTS = {"identity": C.ACT_IDENTITY, "relu": C.ACT_RELU, "leaky_relu": C.ACT_LEAKY_RELU, "sigmoid": C.ACT_SIGMOID,
        "gelu_tanh": C.ACT_GELU_TANH}
LARGEST_FLOPS = 376832.0 * (1 << 26)   # one step of the largest listed case


def _net(dims, dtype, act, **more):
    """The fields of a case that describe a network."""
    case = {"dims": "-".join(str(d) for d in dims), "dtype": dtype, "act": act, "out_act": "identity", "loss": "mse",
            "input": dtype, "target": dtype, "frequency": False, "operand": "", "lr": 1e-3}
    case.update(more)
    return case


def _c1(): return _net([2, 16, 16, 16, 1], "f32", "relu")
def _c2(): return _net([4, 32, 32, 32, 32, 4], "f16", "leaky_relu", input="f32", target="f32")
def _c3(): return _net([32, 64, 64, 64, 3], "f16", "relu", out_act="sigmoid", loss="l2", input="f32", frequency=True, lr=1e-2)
def _c4(): return _net([64, 128, 128, 128, 128, 64], "bf16", "gelu_tanh", lr=3e-4)
def _c5(width, dtype="f16"): return _net([width] * 5, dtype, "relu", target="f32")


def listed():
    return [
        # The example program's own loop: 16 samples through 4-16-4 in half; nothing but launches.
        {"name": "example_step", "kind": "example", "coopvec": False, "count": 16},
        # fp32 parity configuration at its stated batch: a small exact network in someone's inner loop.
        {"name": "train_f32_4k", "kind": "train", "count": 4096, **_c1()},
        # Small fp16 network at its stated batch (radiance caches and material networks are this size).
        {"name": "train_fp16_w32_1m", "kind": "train", "count": 1 << 20, **_c2()},
        # Neural-texture fit: every texel of a 4096 x 4096 image in one step, frequency encoding in front.
        {"name": "train_texture_16m", "kind": "train", "count": 1 << 24, **_c3()},
        # The wide bf16 network at its stated global batch: the largest call.
        {"name": "train_bf16_w128_64m", "kind": "train", "count": 1 << 26, **_c4()},
        # A network that is no benchmark configuration, at the batch of ordinary stochastic training; ragged.
        {"name": "train_widths_20k", "kind": "train", "count": 20011, **_net([32, 128, 128, 3], "f16", "relu")},
        # Hash-grid encoder and a small network, the usual 2^18 positions a step.
        {"name": "train_encoded_256k", "kind": "encoded", "count": 1 << 18, "space": 3, "features": 2, "log2_table": 19, "levels": 16,
         **_net([32, 64, 64, 3], "f16", "relu", out_act="sigmoid", loss="l2", input="f32", lr=1e-2)},
        # Inference as a server or a frame loop asks for it: a handful of samples, latency is all.
        {"name": "forward_w64_1k", "kind": "forward", "count": 1000, **_c5(64)},
        # Inference sweep, narrow network, ragged count.
        {"name": "forward_w32_1m", "kind": "forward", "count": 1000003, **_c5(32)},
        # Inference sweep, the widest network, the largest forward call.
        {"name": "forward_w128_16m", "kind": "forward", "count": 1 << 24, **_c5(128)},
        # A trained texture network rendered into a 1920 x 1080 view.
        {"name": "forward_texture_1080p", "kind": "forward", "count": 1920 * 1080, **_c3()},
        # A step of the wide network whose batch is still in host memory (a data loader in front); ragged.
        {"name": "train_host_1m", "kind": "host", "count": (1 << 20) + 77, **_c4()},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _any_network(rng):
    """A network of two to five layers with the library's usual number formats and activations."""
    dtype = rng.choice(["f16", "bf16"])
    act = rng.choice(["relu", "relu", "gelu_tanh", "leaky_relu"])
    n_layers = rng.randint(2, 5)
    if rng.random() < 0.5:   # every width up to 64
        dims = [rng.randint(2, 64)] + [rng.randint(16, 64)] * (n_layers - 1) + [rng.randint(1, 64)]
        return _net(dims, dtype, act, input=rng.choice([dtype, "f32"]), target=rng.choice([dtype, "f32"]))
    dims = [8 * rng.randint(1, 8)] + [rng.randint(65, 128)] * (n_layers - 1) + [rng.randint(1, 64)]
    return _net(dims, dtype, act, target=rng.choice([dtype, "f32"]))


def draw(rng):
    kind = rng.choice(["example", "f32", "train", "train", "train", "encoded", "forward", "forward", "host"])
    if kind == "example":
        return {"kind": "example", "coopvec": rng.random() < 0.5, "count": rng.randint(1, 256)}
    if kind == "f32":
        dims = rng.choice([[2, 16, 16, 16, 1], [2, rng.randint(4, 32), rng.randint(4, 32), 1], [3, 32, 32, 3]])
        return {"kind": "train", "count": _log_uniform(rng, 100, 1 << 16), **_net(dims, "f32", "relu")}
    if kind == "train":
        net = rng.choice([_c2, _c3, _c4, lambda: _any_network(rng), lambda: _any_network(rng)])()
        if net["dtype"] != "f32" and not net["frequency"] and net["input"] == "f32" and rng.random() < 0.3:
            net.update(operand=net["dtype"], dtype="f32", target="f32")   # fp32 storage, 16-bit operands
        most = 1 << 24 if net["operand"] == "" else 1 << 20
        return {"kind": "train", "count": _log_uniform(rng, 256, most), **net}
    if kind == "encoded":
        levels, features = rng.choice([(8, 2), (16, 2), (8, 4)])
        hidden = rng.choice([32, 64, 64, 128])
        out_act = "identity" if hidden > 64 else "sigmoid"
        net = _net([levels * features, hidden, hidden, rng.randint(1, 4)], "f16", "relu", out_act=out_act, loss="l2", input="f32", lr=1e-2)
        return {"kind": "encoded", "count": _log_uniform(rng, 1 << 12, 1 << 21), "space": rng.choice([2, 3]), "features": features,
                "log2_table": rng.randint(14, 19), "levels": levels, **net}
    if kind == "forward":
        net = rng.choice([lambda: _c5(rng.choice([16, 32, 64, 128]), rng.choice(["f16", "bf16"])),
                          lambda: _c5(rng.choice([16, 32, 64, 128]), rng.choice(["f16", "bf16"])),
                          _c3, _c4, lambda: _any_network(rng)])()
        return {"kind": "forward", "count": _log_uniform(rng, 100, 1 << 24), **net}
    net = rng.choice([_c2, _c4, lambda: _net([32, 128, 128, 3], "f16", "relu")])()
    return {"kind": "host", "count": _log_uniform(rng, 1 << 12, 1 << 21), **net}


def _dims(case):
    return [int(d) for d in case["dims"].split("-")]


def _config(case):
    dtype = DTYPES[case["dtype"]]
    return C.make_config(_dims(case), dtype, ACTS[case["act"]], output_act=ACTS[case["out_act"]],
                         loss=C.LOSS_L2_SUM if case["loss"] == "l2" else C.LOSS_MSE_MEAN,
                         encoding=C.ENC_FREQ2D if case["frequency"] else C.ENC_NONE, lr=case["lr"],
                         input_dtype=DTYPES[case["input"]], target_dtype=DTYPES[case["target"]],
                         adam_master=0 if case["dtype"] == "f32" else 1,
                         operand_dtype=DTYPES[case["operand"]] if case["operand"] else 0)


class _Memory:
    """A library buffer as torch sees it (no copy); keeps the buffer."""

    def __init__(self, buffer, n, typestr):
        self.buffer = buffer
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (buffer.address, False), "version": 3}


def _tensor(buffer, n, typestr):
    return torch.as_tensor(_Memory(buffer, n, typestr), device="cuda")


def _own(device, *buffers):
    """The handles are given back when the last reference to their wrappers goes."""
    for b in buffers:
        weakref.finalize(b, load().mlp_buffer_destroy, b.handle)
    if device is not None:
        weakref.finalize(device, load().mlp_device_destroy, device.handle)


def _own_trainer(device, tr):
    _own(device, tr.params, tr.grads, tr.states, tr.network, tr.loss)


class _State:
    """What the program keeps between calls."""

    def __init__(self, kind, device):
        self.kind, self.device = kind, device


def _optimizer_state(tr, prefix="", states=None, n=None):
    """Views of a trainer's Adam state: means and variances show the gradients, masters the parameters in fp32."""
    n = tr.total if n is None else n
    s = _tensor(tr.states if states is None else states, 4 * n, "<f4").view(n, 4)
    return {prefix + "mean": s[:, 0], prefix + "variance": s[:, 1], prefix + "iteration": s.view(torch.int32)[:, 2], prefix + "master": s[:, 3]}


def _loss(buffer):
    return _tensor(buffer, 2, "<f4")


def _texture(gen, x):
    """A procedural RGB image: sixteen seeded Gaussian blobs per channel."""
    out = torch.zeros((x.shape[0], 3), device="cuda")
    par = torch.rand((3, 16, 3), device="cuda", generator=gen).cpu()
    for ch in range(3):
        for cx, cy, s in par[ch].tolist():
            d2 = (x[:, 0] - cx).square_().add_((x[:, 1] - cy).square_())
            out[:, ch] += torch.exp_(d2.mul_(-0.5 / (0.01 + 0.09 * s) ** 2))
    return out.clamp_(0, 1)


def _inputs(case, gen, count):
    """Normal features in front of a wide network, U[-1, 1] otherwise; texel centres where the encoding takes coordinates."""
    width = 2 if case["frequency"] else _dims(case)[0]
    x = torch.empty((count, width), dtype=TORCH[case["input"]], device="cuda")
    for i in range(0, count, 1 << 22):
        shape = (min(1 << 22, count - i), width)
        if case["frequency"] and case["kind"] == "forward":   # a window of the texture, row by row
            at = torch.arange(i, i + shape[0], device="cuda")
            window = torch.rand(4, device="cuda", generator=gen)
            x[i:i + shape[0], 0] = window[0] * 0.5 + (at % 1920) * (0.5 / 1920)
            x[i:i + shape[0], 1] = window[1] * 0.5 + (at // 1920) * (0.5 / (count // 1920 + 1))
        elif case["frequency"]:                               # texels in random order
            x[i:i + shape[0]] = (torch.randint(0, 4096, shape, device="cuda", generator=gen) + 0.5) / 4096
        elif width >= 32 and case["kind"] != "forward":
            x[i:i + shape[0]] = torch.randn(shape, device="cuda", generator=gen)
        else:
            x[i:i + shape[0]] = torch.rand(shape, device="cuda", generator=gen) * 2 - 1
    return x


def _targets(case, gen, x):
    """A smooth function of the inputs of the size such networks are fitted to."""
    out = _dims(case)[-1]
    t = torch.empty((x.shape[0], out), dtype=TORCH[case["target"]], device="cuda")
    mix = torch.randn((x.shape[1], out), device="cuda", generator=gen) / math.sqrt(x.shape[1])
    for i in range(0, x.shape[0], 1 << 22):
        part = x[i:i + (1 << 22)]
        if case["frequency"]:
            t[i:i + (1 << 22)] = _texture(gen, part)
        elif case["out_act"] == "sigmoid":
            t[i:i + (1 << 22)] = 0.5 + 0.4 * torch.sin(7 * (part.float() @ mix))
        else:
            t[i:i + (1 << 22)] = 0.5 * torch.sin(2 * (part.float() @ mix))
    return t


def _prepare_example(case, gen, seed):
    """The example program's buffers (two-segment half parameters with 64-byte sub-allocations, zero gradients, Adam
    states, the per-layer address table) and its 2-D inputs."""
    dims, align = [4, 16, 4], 32
    rng = np.random.default_rng(seed)
    offsets, total = [], 0
    for l in range(2):
        w, b = total, total + (dims[l] * dims[l + 1] + align - 1) // align * align
        total = b + (dims[l + 1] + align - 1) // align * align
        offsets.append((w, b))
    p = np.zeros(total, dtype=np.float16)
    for l, (w, b) in enumerate(offsets):
        p[w:w + dims[l] * dims[l + 1]] = rng.uniform(-1, 1, dims[l] * dims[l + 1]) * math.sqrt(6.0 / (dims[l] + dims[l + 1]))
    dev = api.Device(0, torch.cuda.current_stream().cuda_stream)
    s = _State("example", dev)
    params = dev.create_buffer(p.nbytes, p)
    # the cooperative-vector flavour accumulates a weight gradient into one 16 x 16 tile per layer
    matrix = 256 if case["coopvec"] else 0
    grads = dev.create_buffer(p.nbytes + 2 * 2 * matrix)
    states = dev.create_buffer(8 * total)
    net = np.zeros((2, 4), dtype=np.uint64)
    for l, (w, b) in enumerate(offsets):
        dw = grads.address + (2 * (total + l * matrix) if case["coopvec"] else 2 * w)
        net[l] = [params.address + 2 * w, dw, params.address + 2 * b, grads.address + 2 * b]
    network = dev.create_buffer(net.nbytes, net)
    loss = dev.create_buffer(8)
    _own(dev, params, grads, states, network, loss)
    s.buffers = (params, grads, states, network, loss)
    s.loss, s.count = loss, case["count"]
    s.inputs = torch.rand((case["count"], 2), device="cuda", generator=gen)
    s.learn = dev.kernel("learnGradient_coopvec" if case["coopvec"] else "learnGradient")
    s.adjust = dev.kernel("adjustParameters")
    s.learn_args = api.LearnGradParams(network.address, loss.address, s.inputs.data_ptr(), case["count"])
    s.adjust_args = api.AdjustParamsParams(states.address, params.address, grads.address, total)
    s.groups = (api.groups_for(case["count"]), api.groups_for(total))
    s.moves = None
    if case["coopvec"]:   # the tiles back into row-major gradients, as that example's host loop does
        size = [api.matrix_size(dims[l + 1], dims[l], C.F16, api.MATRIX_TRAINING_OPTIMAL) for l in range(2)]
        src = [api.MatrixDesc(dims[l + 1], dims[l], C.F16, api.MATRIX_TRAINING_OPTIMAL, size[l], 2 * (total + l * matrix), 0) for l in range(2)]
        dst = [api.MatrixDesc(dims[l + 1], dims[l], C.F16, api.MATRIX_ROW_MAJOR, 2 * dims[l] * dims[l + 1], 2 * offsets[l][0], 2 * dims[l])
               for l in range(2)]
        s.moves, s.tiles = (grads, dst, src), (2 * total, 4 * matrix)
    half = _tensor(states, 4 * total, "<f2").view(total, 4)
    s.out = {"loss": _loss(loss)[:1], "params": _tensor(params, total, "<f2"), "mean": half[:, 0], "variance": half[:, 1],
             "iteration": _tensor(states, 2 * total, "<i4").view(total, 2)[:, 1]}
    return s


def _torch_trainer(case, seed):
    cfg = _config(case)
    tr = TorchTrainer(cfg, C.init_params(cfg, seed=seed, scheme="xavier"))
    s = _State(case["kind"], tr.device)
    s.tr = tr
    _own_trainer(tr.device, tr.trainer)
    return s


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind, count = case["kind"], case["count"]
    if kind == "example":
        return _prepare_example(case, gen, seed)
    if kind == "train":
        s = _torch_trainer(case, seed)
        s.x = _inputs(case, gen, count)
        s.t = _targets(case, gen, s.x)
        s.out = {"loss": _loss(s.tr.trainer.loss), "params": s.tr.params, **_optimizer_state(s.tr.trainer)}
        return s
    if kind == "forward":
        s = _torch_trainer(case, seed)
        s.x = _inputs(case, gen, count)
        return s
    dev = api.Device(0, torch.cuda.current_stream().cuda_stream)
    s = _State(kind, dev)
    cfg = _config(case)
    if kind == "host":
        tr = api.Trainer(dev, cfg, C.init_params(cfg, seed=seed, scheme="xavier"))
        _own_trainer(dev, tr)
        s.stepper = HostStepper(tr)
        x = _inputs(case, gen, count)
        t = _targets(case, gen, x)
        s.x = torch.empty(x.shape, dtype=x.dtype, pin_memory=True).copy_(x)
        s.t = torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t)
        s.out = {"params": _tensor(tr.states, 4 * tr.total, "<f4").view(-1, 4)[:, 3], **_optimizer_state(tr)}
        return s
    # encoded: positions in the unit square or cube, a table of small seeded features
    pcfg = P.prepare(case["space"], case["features"], case["log2_table"], case["levels"], 16.0, 0.5)
    rng = np.random.default_rng(seed)
    table = rng.random(pcfg.table_values, dtype=np.float32)
    table -= np.float32(0.5)
    table *= np.float32(2e-1)
    s.et = EncodedTrainer(dev, pcfg, cfg, table, C.init_params(cfg, seed=seed, scheme="xavier"), max_count=count)
    _own_trainer(dev, s.et.trainer)
    _own(None, s.et.table, s.et.d_table, s.et.table_states, s.et.features, s.et.d_features)
    s.x = torch.rand((count, case["space"]), device="cuda", generator=gen)
    s.t = _targets(case, gen, s.x)
    s.count = count
    s.out = {"loss": _loss(s.et.trainer.loss), "table": _tensor(s.et.table, s.et.n_table, "<f4"), **_optimizer_state(s.et.trainer),
             **_optimizer_state(None, "table_", s.et.table_states, s.et.n_table)}
    return s


def run(s):
    if s.kind == "train":
        s.tr.learn_gradient(s.x, s.t)
        s.tr.adjust_parameters()
        return s.out
    if s.kind == "forward":
        return s.tr.forward(s.x)
    if s.kind == "host":
        largest, mean = s.stepper.step(s.x, s.t)
        return {"largest": largest, "mean_loss": mean, **s.out}
    if s.kind == "encoded":
        s.et.learn_gradient(s.x.data_ptr(), s.t.data_ptr(), s.count)
        s.et.adjust_parameters()
        return s.out
    s.loss.clear()
    if s.moves is not None:
        s.moves[0].clear(*s.tiles)
    s.learn.dispatch(s.learn_args, s.groups[0])
    if s.moves is not None:
        grads, dst, src = s.moves
        s.device.matrix_convert(grads.address, dst, grads.address, src)
    s.adjust.dispatch(s.adjust_args, s.groups[1])
    return s.out


def work(case):
    """Inputs, targets, parameters and Adam states once each way; 2 flops per multiply-add of the layer products."""
    n = case["count"]
    if case["kind"] == "example":
        return {"bytes": 8.0 * n + 192 * 20, "flops": n * 6.0 * 128}
    cfg = _config(case)
    _, _, total = C.param_layout(cfg)
    size = C.DTYPE_SIZE
    row_in = cfg.input_width * size[cfg.input_dtype]
    if case["kind"] == "forward":
        return {"bytes": float(n * (row_in + 4 * cfg.out_dim) + total * size[cfg.dtype]), "flops": float(n) * C.flops_per_sample(cfg, False)}
    row_t = cfg.out_dim * size[cfg.target_dtype]
    adam = total * (32 + 2 * size[cfg.dtype])
    flops = float(n) * C.flops_per_sample(cfg)
    if case["kind"] == "encoded":
        # the table's gradient touches at most what the positions reach; its Adam step reads and writes every state
        table = case["levels"] * (1 << case["log2_table"]) * case["features"]
        flops += n * 2.0 * cfg.dims[0] * cfg.dims[1] + n * case["levels"] * (case["space"] + 1) * case["features"] * 6.0
        return {"bytes": float(n * (4 * case["space"] + row_t) + adam + table * (32 + 8)), "flops": flops}
    return {"bytes": float(n * (row_in + row_t) + adam), "flops": flops}


def tolerance(case):
    if case["kind"] == "example":
        return "exact"   # half arithmetic in the example's own order, one block: no freedom in the sums
    if case["dtype"] == "f32" and not case["operand"]:
        # fp32 sums over the batch in any order; a ReLU whose input is within rounding of zero moves one sample's share
        return {"rel": 1e-4, "max": 1e-2}
    if case["kind"] == "forward":
        return {"rel": 1e-2 if "bf16" in (case["dtype"], case["operand"]) else 2e-3}
    return {"rel": 1e-2}
