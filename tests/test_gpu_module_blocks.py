"""The stand-alone device module launched by a host of its own through the driver, with blocks of other sizes than the
example's 256: one block of 16 samples has the same sums whatever its size."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("entry,tile", [("learnGradient", 0), ("learnGradient_coopvec", 256)])
def test_module_blocks_of_other_sizes(entry, tile):
    from slang_b200.api import Device
    from slang_b200.lib import CUBIN_PATH
    device = Device(0)
    device.wait()
    cuda = ctypes.CDLL("libcuda.so.1")
    module, function = ctypes.c_void_p(), ctypes.c_void_p()
    assert cuda.cuModuleLoadData(ctypes.byref(module), open(CUBIN_PATH, "rb").read()) == 0
    assert cuda.cuModuleGetFunction(ctypes.byref(function), module, entry.encode()) == 0
    rng = np.random.default_rng(3)
    init = rng.uniform(-1, 1, 192).astype(np.float16)
    inputs = rng.uniform(0, 1, 32).astype(np.float32)
    offs = [(0, 128), (192, 320)]   # byte offsets of (weights, biases) of both layers
    results = {}
    for threads in (256, 176, 128, 64, 32):
        params, grads = device.create_buffer(384, init), device.create_buffer(384 + 4 * tile)
        net = np.array([[params.address + w, grads.address + (384 + 2 * tile * l if tile else w), params.address + b, grads.address + b]
                        for l, (w, b) in enumerate(offs)], dtype=np.uint64)
        network, xs, loss = device.create_buffer(64, net), device.create_buffer(128, inputs), device.create_buffer(8)
        device.wait()
        args = [ctypes.c_uint64(network.address), ctypes.c_uint64(loss.address), ctypes.c_uint64(xs.address), ctypes.c_uint32(16)]
        pointers = (ctypes.c_void_p * 4)(*[ctypes.cast(ctypes.byref(a), ctypes.c_void_p) for a in args])
        assert cuda.cuLaunchKernel(function, 1, 1, 1, threads, 1, 1, 0, None, pointers, None) == 0
        assert cuda.cuCtxSynchronize() == 0
        results[threads] = (grads.read(np.uint16).copy(), loss.read(np.uint32).copy())
    assert results[256][0].any() and results[256][1][0]
    for threads, (g, l) in results.items():
        assert np.array_equal(g, results[256][0]) and np.array_equal(l, results[256][1]), threads
    assert cuda.cuModuleUnload(module) == 0
    device.destroy()
