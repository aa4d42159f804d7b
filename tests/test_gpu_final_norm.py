"""The end of a decoded token -- final norm, the last row's copy, the classifier -- as one phase of the persistent kernel where nobody else reads the normalised
row or its copy, and as phases of their own where somebody does: the same bits as the eager kernels, call after call at the same addresses."""
import numpy as np
import pytest

from oracle import oracle as oc
from tests.blockgen import random_weight
from tests.gpu_common import make_device

pytestmark = pytest.mark.gpu


def tail(dev, w, norm, x, wt, m, k, keep):
    from crabml_b200 import CudaTensor as T
    x = T.new(x.copy(), [1, k], dev)
    x = x.rms_norm_inplace(1e-5).mul_inplace(norm)
    last = T.alloc([k], oc.F32, dev)
    last.copy_rows_from(x, [0])
    y = w.matmul_vec(last)
    if keep != "row":
        del x
    if keep != "copy":
        del last
    out = [y.export().copy()]
    if keep == "row":
        out.append(x.export().copy())
    if keep == "copy":
        out.append(last.export().copy())
    return out


@pytest.mark.parametrize("wt,m,k", [(oc.Q8_0, 1000, 288), (oc.Q8_0, 34386, 288), (oc.Q4_0, 512, 4096), (oc.Q4_K, 300, 512), (oc.Q6_K, 300, 1024)])
def test_final_norm_and_classifier(wt, m, k):
    from crabml_b200 import CudaTensor as T
    rng = np.random.default_rng(k)
    blocks, nw = random_weight(wt, m, k, rng), (1.0 + 0.1 * rng.standard_normal(k)).astype(np.float32)
    fused, eager = make_device(lazy=2), make_device(lazy=0)
    try:
        side = [(d, T.from_cpu(blocks, [m, k], wt, d), T.from_cpu(nw, [k], oc.F32, d)) for d in (fused, eager)]
        for keep in ("nothing", "row", "nothing", "copy", "nothing"):
            x = rng.standard_normal(k).astype(np.float32)
            a, b = [tail(d, w, n, x, wt, m, k, keep) for d, w, n in side]
            for u, v in zip(a, b):
                np.testing.assert_array_equal(u.view(np.uint32), v.view(np.uint32), err_msg=keep)
        del side
    finally:
        fused.close()
        eager.close()


@pytest.mark.parametrize("lazy", [1, 2])
@pytest.mark.parametrize("rows,k,at", [(2, 32, 0), (5, 288, 4), (40, 512, 17)])
def test_a_prompts_row_is_normed_alone_only_where_the_others_are_dropped(lazy, rows, k, at):
    from crabml_b200 import CudaTensor as T
    rng = np.random.default_rng(rows)
    nw = (1.0 + 0.1 * rng.standard_normal(k)).astype(np.float32)
    devs = make_device(lazy=lazy), make_device(lazy=0)
    try:
        for keep in (False, True, False):
            x = rng.standard_normal((rows, k)).astype(np.float32)
            got = []
            for d in devs:
                t = T.new(x.reshape(-1).copy(), [rows, k], d).rms_norm_inplace(1e-5).mul_inplace(T.from_cpu(nw, [k], oc.F32, d))
                last = T.alloc([k], oc.F32, d)
                last.copy_rows_from(t, [at])
                if not keep:
                    del t
                got.append([last.export().copy()] + ([t.export().copy()] if keep else []))
            for a, b in zip(*got):
                np.testing.assert_array_equal(a.view(np.uint32), b.view(np.uint32))
            t = last = None
    finally:
        for d in devs:
            d.close()
