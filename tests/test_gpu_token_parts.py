"""Long tokens in parts of growing length (lazy.cu LZ_PART_GROWTH): the eager kernels' bits, one persistent kernel a part, and bounds that hold for any depth."""
import numpy as np
import pytest

from oracle import oracle as oc
from tests.gpu_common import make_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wt,ct", [(oc.Q8_0, oc.Q8_0), (oc.Q4_K, oc.Q6_K)])
def test_a_token_of_three_parts_has_the_eager_bits(wt, ct):
    from crabml_b200 import runner as R
    conf = R.LlamaConfig(4, 2, 16, 256, 512, 64, 512, 1e-5, 64)        # 16 layers of 26 ops: parts of 30, 150 and the rest
    res = {}
    for lazy in (0, 2):
        dev = make_device(lazy=lazy)
        try:
            r = R.LlamaRunner(dev, conf, R.synthetic_weights(dev, conf, wt, ct, seed=5), 64)
            first = [r.forward([t], p).copy() for p, t in enumerate([5, 6, 7])]
            launches = dev.launch_count()
            late = [r.forward([t], 3 + p).copy() for p, t in enumerate(range(11, 15))]
            res[lazy] = np.stack(first + late)
            if lazy:
                assert dev.launch_count() - launches == 4 * 3
            r.close()
        finally:
            dev.close()
    assert np.isfinite(res[0]).all() and np.abs(res[0]).max() > 0
    np.testing.assert_array_equal(res[2].view(np.uint32), res[0].view(np.uint32))


def deep(dev, layers):
    """a model of `layers` narrow layers, 26 ops each"""
    from crabml_b200 import runner as R
    conf = R.LlamaConfig(4, 2, layers, 256, 512, 600, 512, 1e-5, 64)
    return conf, R.synthetic_weights(dev, conf, oc.Q8_0, oc.Q8_0, seed=3)


@pytest.mark.parametrize("layers,parts", [(16, 3), (40, 4), (80, 4), (200, 4)])
def test_a_token_has_four_parts_at_most(layers, parts):
    from crabml_b200 import runner as R
    dev = make_device(lazy=2)
    try:
        r = R.LlamaRunner(dev, *deep(dev, layers), 16)
        for p in range(4):
            launches = dev.launch_count()
            r.forward([1 + p], p)
            assert dev.launch_count() - launches == parts
        r.close()
    finally:
        dev.close()


def test_sixty_four_sequences_of_long_tokens_replay_their_graphs():
    """40 layers are four parts a token, each a graph of every sequence with a cache of its own: 256 graphs, visited in turn, all stay cached."""
    from crabml_b200 import runner as R
    dev = make_device(lazy=2)
    try:
        conf, w = deep(dev, 40)
        runners = [R.LlamaRunner(dev, conf, w, 16) for _ in range(64)]
        captures = []
        for p in range(4):
            for r in runners:
                r.forward([1 + p], p)
            captures.append(dev.lazy_stats()["graph_captures"])
        assert captures[3] == captures[1], captures
        for r in runners:
            r.close()
    finally:
        dev.close()


def test_the_host_runs_eight_tokens_of_four_parts_ahead_of_the_gpu():
    """Eight tokens of 40 layers are recorded and submitted while the GPU is still at work on what was queued before them: a host that waited for a slot of
    per-token values would come back when that work is over."""
    import time
    from crabml_b200 import CudaTensor, runner as R
    from tests.blockgen import random_weight
    dev = make_device(lazy=2)
    try:
        r = R.LlamaRunner(dev, *deep(dev, 40), 64)
        w = CudaTensor.from_cpu(random_weight(oc.Q8_0, 4096, 4096, np.random.default_rng(0), 0.02), [4096, 4096], oc.Q8_0, dev)
        x = CudaTensor.new(np.ones((4096, 4096), np.float32), [4096, 4096], dev)

        def ahead(products):
            for _ in range(products):
                w.matmul_vec(x)
            dev.flush()
            t0 = time.perf_counter()
            for p in range(8):
                r.forward([1 + p], p, export=False)
            t1 = time.perf_counter()
            dev.synchronize()
            return t1 - t0, time.perf_counter() - t1
        for _ in range(3):
            ahead(20)                                      # plans, buffers and scratch are there now
        submit, left = min((ahead(600) for _ in range(3)), key=lambda t: t[0])
        assert submit < 0.5 * left, (submit, left)
        r.close()
    finally:
        dev.close()
