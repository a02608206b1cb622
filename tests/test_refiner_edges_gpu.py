"""The refiner's tensor-core kernels at the edges of their tiles: images
narrower than, equal to and a little wider than one 128- or 64-pixel tile at some
pyramid level, single-row strips, strips and batches that do not divide evenly
among the resident blocks.

Each layer on its own: the FP64 convolution (and its two gradients) of the very
tensors the GPU stored, so that no rounding of an earlier layer enters.  Products
of two bf16 are exact in FP32; with S the sum of the products' magnitudes, an
accumulation of n FP32 additions is off by at most n 2^-23 S.  Activations and
input gradients add 9 cin / 16 <= 63 partial sums of 16 and round to bf16 (2^-8
of the value); a weight gradient's block adds at most one partial sum per 16
pixels (fewer than 1000 here), then the blocks' partials, at most 456."""
import importlib

import numpy as np
import pytest

from oracle import unet as U

pytestmark = pytest.mark.gpu

SIZES = [(1, 8, 8), (3, 8, 128), (1, 24, 136), (2, 40, 256), (1, 16, 1032), (5, 56, 72)]
# convolution -> (its output gradient, its input gradient, the ReLU output masking that)
BACK = {"c2": ("dz2", "dz1", "e0a"), "c3": ("dz3", "gp1", None), "c4": ("dz4", "dz3", "e1a"),
        "c5": ("dz5", "gp2", None), "c6": ("dz6", "dz5", "e2a"), "c7": ("dz7", "gp3", None),
        "c8": ("dz8", "dz7", "b3a"), "c9": ("dz9", "gu2", None), "c10": ("dz10", "gu1", None),
        "c11": ("dz11", "gu0", None)}


@pytest.mark.parametrize("n,h,w", SIZES)
def test_each_layer_at_tile_edges(cuda, n, h, w):
    rf = importlib.import_module("3deye_gb300.refiner")
    rng = np.random.default_rng(n * h * w)
    raw = rng.integers(500, 3000, (n, h, w)).astype(np.uint16)
    raw[rng.random(raw.shape) < 0.05] = 0
    tgt = np.clip(raw.astype(np.int64) + rng.integers(-6, 7, raw.shape), 0, 32767).astype(np.uint16)
    R = rf.Refiner(n, h, w, seed=5)
    theta = R.get_params()
    theta[-17:-1] = rng.normal(0, 0.1, 16)  # the head
    theta[:-17][theta[:-17] == 0] = 0.05    # biases
    R.set_params(theta)
    R.loss_grad(raw, tgt)
    assert R.status() == 0
    p, g = U.unflatten(theta), U.unflatten(R.grads())
    T = {k: R.tensor(k).astype(np.float64) for k in rf.ACTIVATIONS + rf.GRADIENTS}
    R.close()
    for name, _, a, _, mode, b, _, _, out in U.CONVS:
        x = T[a]
        x = U.pool2(x) if mode == U.POOL else U.up2(x) if mode == U.UP else x
        x = np.concatenate([x, T[b]], -1) if b else x
        wq, bias = U.bf16(p[name + ".w"]), p[name + ".b"]
        ref = np.maximum(U.conv3x3(x, wq, bias), 0)
        S = U.conv3x3(np.abs(x), np.abs(wq), np.abs(bias))
        assert np.all(np.abs(T[out] - ref) <= 2.0 ** -8 * ref + 80 * 2.0 ** -23 * S), name
        dz, gx, mask = BACK[name]
        ref = U.conv3x3_dgrad(T[dz], wq)
        S = U.conv3x3_dgrad(np.abs(T[dz]), np.abs(wq))
        ref = ref if mask is None else np.where(T[mask] > 0, ref, 0)
        assert np.all(np.abs(T[gx] - ref) <= 2.0 ** -8 * np.abs(ref) + 80 * 2.0 ** -23 * S), name + " input gradient"
        dw, db = U.conv3x3_wgrad(x, T[dz])
        Sw, Sb = U.conv3x3_wgrad(np.abs(x), np.abs(T[dz]))
        assert np.all(np.abs(g[name + ".w"] - dw) <= 1500 * 2.0 ** -23 * Sw + 1e-30), name + " weight gradient"
        assert np.all(np.abs(g[name + ".b"] - db) <= 1500 * 2.0 ** -23 * Sb + 1e-30), name + " bias gradient"


@pytest.mark.parametrize("n,h,w", SIZES)
def test_gradient_routing_at_row_ends(cuda, n, h, w):
    """The gradients routed through upsampling, pooling and skips equal the same
    FP32 operations on the stored tensors, rounded to bf16: rows of fewer items than
    a block, of whole blocks and of one item more, whole and split gradients."""
    import torch
    rf = importlib.import_module("3deye_gb300.refiner")
    rng = np.random.default_rng(n + h + w)
    raw = rng.integers(500, 3000, (n, h, w)).astype(np.uint16)
    tgt = np.clip(raw.astype(np.int64) + rng.integers(-6, 7, raw.shape), 0, 32767).astype(np.uint16)
    R = rf.Refiner(n, h, w, seed=9)
    theta = R.get_params()
    theta[-17:-1] = rng.normal(0, 0.1, 16)  # the head
    theta[:-17][theta[:-17] == 0] = 0.05    # biases
    R.set_params(theta)
    R.loss_grad(raw, tgt)
    assert R.status() == 0
    T = {k: R.tensor(k).astype(np.float32) for k in rf.ACTIVATIONS + rf.GRADIENTS}
    R.close()

    def bf16(x):
        return torch.from_numpy(np.ascontiguousarray(x)).bfloat16().float().numpy()

    def quad(x):  # the four pixels over each low-resolution one
        return [x[:, k >> 1::2, k & 1::2] for k in range(4)]

    for g, ca, y, dz in (("gu0", 32, "d1", "dz10"), ("gu1", 48, "d2", "dz9"), ("gu2", 64, "b3", "dz8")):
        s = np.float32(0)
        for q in quad(T[g][..., :ca]):
            s = s + q
        assert np.array_equal(T[dz], bf16(np.where(T[y] > 0, s, np.float32(0)))), dz
        assert np.any(T[dz])
    for g, ca, e, gp, dz in (("gu0", 32, "e0", "gp1", "dz2"), ("gu1", 48, "e1", "gp2", "dz4"),
                             ("gu2", 64, "e2", "gp3", "dz6")):
        ev, skip, got = quad(T[e]), quad(T[g][..., ca:]), quad(T[dz])
        top, taken = np.maximum(np.maximum(ev[0], ev[1]), np.maximum(ev[2], ev[3])), np.zeros(ev[0].shape, bool)
        for k in range(4):
            mine = (ev[k] == top) & ~taken
            taken |= mine
            v = skip[k] + np.where(mine, T[gp], np.float32(0))
            assert np.array_equal(got[k], bf16(np.where(ev[k] > 0, v, np.float32(0)))), (dz, k)
        assert np.any(T[dz])
