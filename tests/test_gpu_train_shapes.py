"""Training gradients at batch sizes around a tile and a grid of tiles, with
masked targets, against the FP64 reference with BF16 operands."""
import ctypes

import numpy as np
import pytest

from fluid_step import _abi
from fluid_step.learned import Model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 255, 257, 148 * 128 + 1])
def test_gradients_match_the_reference(n):
    """The tensor cores accumulate in FP32 in an order of their own and the
    SiLU's tanh is good to 2^-11: 1 % of the largest gradient of each block."""
    import torch

    import mlp_ref
    rng = np.random.default_rng(n)
    m = Model(seed=3)
    mean, std = rng.normal(size=12), rng.uniform(0.5, 2.0, 12)
    m.set_normalization(mean, std, [0.3, -0.2], [1.5, 0.7])
    x = (rng.normal(size=(n, 12)) * std + mean).astype(np.float32)
    y = rng.normal(size=(n, 2)).astype(np.float32)
    y[rng.random(n) < 0.4, 0] = np.nan
    p = m.parameters()
    norm = m.normalization()
    xs = (x - norm[:12]) / norm[12:24]
    ys = (y - norm[24:26]) / norm[26:28]
    xd, yd = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    g = np.empty(_abi.FE_MODEL_PARAMS, np.float32)
    loss = ctypes.c_float()
    _abi.check(m.lib, m.lib.fe_model_gradients(
        m.handle, ctypes.c_void_p(xd.data_ptr()), ctypes.c_void_p(yd.data_ptr()), n,
        g.ctypes.data_as(ctypes.c_void_p), ctypes.byref(loss)), "gradients")
    out, cache = mlp_ref.forward(p, xs)
    e = np.where(np.isnan(ys), 0.0, out - np.nan_to_num(ys))
    assert loss.value == pytest.approx(float((e ** 2).sum()), rel=2e-2, abs=1e-6)
    ref = reference_gradients(mlp_ref, p, xs, e)
    lo = 0
    for size in (1024, 4096, 128, 64, 64, 2):
        a, b = g[lo:lo + size], ref[lo:lo + size]
        assert np.abs(a - b).max() <= 1e-2 * np.abs(b).max() + 1e-7, lo
        lo += size
    # and again: bit for bit
    g2 = np.empty_like(g)
    _abi.check(m.lib, m.lib.fe_model_gradients(
        m.handle, ctypes.c_void_p(xd.data_ptr()), ctypes.c_void_p(yd.data_ptr()), n,
        g2.ctypes.data_as(ctypes.c_void_p), ctypes.byref(loss)), "gradients")
    assert np.array_equal(g.view(np.uint32), g2.view(np.uint32))


def reference_gradients(ref, p, xs, e):
    """Backward pass in FP64 with the operands rounded where the kernel does."""
    q = ref.bf16
    w1, w2, w3, b1, b2, _ = ref.unpack(p)
    X = q(ref.pad16(xs))
    z1 = X @ q(w1).T + b1
    h1 = q(ref.silu(z1))
    z2 = h1 @ q(w2).T + b2
    h2 = q(ref.silu(z2))
    do = 2.0 * e / len(e)
    dob = q(do)
    dz2 = (dob @ q(w3)) * ref.silu_grad(z2)
    dz2b = q(dz2)
    dz1 = (dz2b @ q(w2)) * ref.silu_grad(z1)
    return np.concatenate([(q(dz1).T @ X).reshape(-1), (dz2b.T @ h1).reshape(-1),
                           (dob.T @ h2).reshape(-1), dz1.sum(0), dz2.sum(0), do.sum(0)])


def test_a_step_that_failed_is_not_counted():
    """A step whose launches were refused (its stream's capture had been given up)
    has not updated the weights, so the next one's bias correction is that of a
    run without it."""
    import torch
    rng = np.random.default_rng(2)
    x = torch.from_numpy(rng.normal(size=(300, 12)).astype(np.float32)).cuda()
    y = torch.from_numpy(rng.normal(size=(300, 2)).astype(np.float32)).cuda()
    torch.cuda.synchronize()
    models = [Model(seed=3), Model(seed=3)]
    lib = models[0].lib
    rt = ctypes.CDLL("libcudart.so.12")      # the one torch has loaded

    def step(m, stream=None):
        return lib.fe_model_train_step(m.handle, ctypes.c_void_p(x.data_ptr()),
                                       ctypes.c_void_p(y.data_ptr()), 300, 1e-2, 0.0, stream, None)

    def refused(m):
        stream, graph = ctypes.c_void_p(), ctypes.c_void_p()
        assert rt.cudaStreamCreateWithFlags(ctypes.byref(stream), 1) == 0
        assert rt.cudaStreamBeginCapture(stream, 1) == 0          # thread-local
        assert rt.cudaStreamSynchronize(stream) != 0              # gives the capture up
        rc = step(m, stream)
        assert rt.cudaStreamEndCapture(stream, ctypes.byref(graph)) != 0
        rt.cudaGetLastError()
        assert rt.cudaStreamDestroy(stream) == 0
        return rc

    for m, fail in zip(models, (False, True)):
        assert step(m) == _abi.FE_OK
        if fail:
            assert refused(m) == _abi.FE_ERR_CUDA
        assert step(m) == _abi.FE_OK
    torch.cuda.synchronize()
    a, b = models[0].parameters(), models[1].parameters()
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    for m in models:
        m.close()
