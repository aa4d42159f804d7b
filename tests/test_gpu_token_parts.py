"""A token long enough for three parts of growing length (lazy.cu LZ_PART_GROWTH): the eager kernels' bits, one persistent kernel a part."""
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
