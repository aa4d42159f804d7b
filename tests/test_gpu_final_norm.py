"""The end of a decoded token -- final norm, the last row's copy, the classifier -- as one phase of the persistent kernel where nobody else reads the normalised
row or its copy, and as phases of their own where somebody does: the same bits as the eager kernels, call after call at the same addresses."""
import ctypes as C

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


def phases(dev):
    """phase types of the last plan that was made (device created with CRABML_MEGA_PROF): 0 norm, 1 product, 3 row copy (the first fills the row)"""
    cap = 8 * 4097
    ts, ty, n = (C.c_uint64 * cap)(), (C.c_int32 * cap)(), C.c_int32(0)
    dev.check(dev.lib.cc_lazy_mega_profile(dev.handle, ts, ty, cap, C.byref(n)))
    return [(t & 1023) // 16 for t in ty[:n.value]]


@pytest.mark.parametrize("wt,variant", [(oc.Q8_0, 2), (oc.Q4_0, 2), (oc.Q4_K, 1), (oc.Q6_K, 1)])
@pytest.mark.parametrize("keep,want", [("nothing", [3, 1]), ("row", [3, 0, 3, 1]), ("copy", [3, 0, 3, 1])])
def test_the_final_norm_is_no_phase_of_its_own_only_where_nobody_else_reads_it(monkeypatch, wt, variant, keep, want):
    from crabml_b200 import CudaTensor as T
    m, k = 300, 1024
    rng = np.random.default_rng(k)
    monkeypatch.setenv("CRABML_MEGA_PROF", "1")
    dev = make_device(lazy=2)
    try:
        w, n = T.from_cpu(random_weight(wt, m, k, rng), [m, k], wt, dev), T.from_cpu(np.ones(k, np.float32), [k], oc.F32, dev)
        tail(dev, w, n, rng.standard_normal(k).astype(np.float32), wt, m, k, keep)
        assert phases(dev) == want
        assert dev.mega_variant() == variant
        del w, n
    finally:
        dev.close()


@pytest.mark.parametrize("lazy", [1, 2])
def test_a_prompts_row_is_normed_alone_by_steps_that_are_no_graph(lazy):
    """norm, product and copy of all rows are a plan that is kept; the row alone is not: the count of uncached runs says which way was taken"""
    from crabml_b200 import CudaTensor as T
    dev = make_device(lazy=lazy)
    try:
        nw = T.from_cpu(np.ones(64, np.float32), [64], oc.F32, dev)
        for keep in (False, True, False):
            t = T.new(np.ones(5 * 64, np.float32), [5, 64], dev)
            before = dev.lazy_stats()["uncached"]
            t = t.rms_norm_inplace(1e-5).mul_inplace(nw)
            last = T.alloc([64], oc.F32, dev)
            last.copy_rows_from(t, [3])
            if not keep:
                del t
            last.export()
            assert dev.lazy_stats()["uncached"] - before == (0 if keep else 1)
            t = last = None
        del nw
    finally:
        dev.close()
