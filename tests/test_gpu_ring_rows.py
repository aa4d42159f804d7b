"""The streaming phases of the ring kernel at the edges of their tiles: rows that do not divide by the CTAs or pair up, rows of one to several segments with
ragged ends, rows longer than the prologue's staging area, more rows than their lanes' sums find room for, and activations on which the quantiser's shortcuts do not hold.  A feed-forward block
(norm, gate / up, silu * mul, down, residual) of the persistent kernel must equal the eager kernels bit for bit: both sum in one canonical order."""
import numpy as np
import pytest

from oracle import oracle as oc
from tests.blockgen import random_weight
from tests.gpu_common import make_device

pytestmark = pytest.mark.gpu


def rows(kind, n, rng):
    x = rng.standard_normal(n).astype(np.float32)
    if kind == "whole quotients":                    # every number a whole multiple of its block's step
        x = rng.integers(-127, 128, n).astype(np.float32) * np.float32(0.37)
        x[::32] = np.float32(127) * np.float32(0.37)
    elif kind == "zeros and extremes":
        x[: n // 2] = 0
        x[n // 2:: 3] *= np.float32(1e-30)
        x[n - 1] = np.float32(3e4)
    elif kind == "tiny":
        x *= np.float32(1e-32)
    return x


def block(dev, wt, dim, hid, x, w):
    from crabml_b200 import CudaTensor as T
    up = lambda b, r, c: T.from_cpu(b, [r, c], wt, dev)      # noqa: E731
    gate, upw, down = up(w["gate"], hid, dim), up(w["up"], hid, dim), up(w["down"], dim, hid)
    nw = T.from_cpu(w["norm"], [dim], oc.F32, dev)
    x = T.new(x.copy(), [1, dim], dev)
    orig = x.dup()
    x = x.rms_norm_inplace(1e-5).mul_inplace(nw)
    g, u = gate.matmul_vec(x), upw.matmul_vec(x)
    del x
    h = g.silu_inplace().mul_inplace(u)
    del g, u
    y = down.matmul_vec(h).add_inplace(orig)
    return y.export().copy()


@pytest.mark.parametrize("wt", [oc.Q8_0, oc.Q4_0])
@pytest.mark.parametrize("dim,hid", [(32, 32), (288, 768), (512, 4128), (4096, 12320), (4128, 2976), (12320, 160), (16448, 64), (320, 20000), (64, 24608), (32, 28672), (608, 29568), (96, 32768), (4128, 20000), (20512, 1216)])
def test_feed_forward_block_equals_the_eager_kernels(wt, dim, hid):
    rng = np.random.default_rng(dim * 7 + hid + wt)
    w = {"gate": random_weight(wt, hid, dim, rng), "up": random_weight(wt, hid, dim, rng), "down": random_weight(wt, dim, hid, rng),
         "norm": (1.0 + 0.1 * rng.standard_normal(dim)).astype(np.float32)}
    ring, eager = make_device(lazy=2), make_device(lazy=0)
    try:
        for kind in ("plain", "whole quotients", "zeros and extremes", "tiny"):
            x = rows(kind, dim, rng)
            a, b = block(ring, wt, dim, hid, x, w), block(eager, wt, dim, hid, x, w)
            np.testing.assert_array_equal(a.view(np.uint32), b.view(np.uint32), err_msg=kind)
        assert ring.mega_variant() == 2
    finally:
        ring.close()
        eager.close()
