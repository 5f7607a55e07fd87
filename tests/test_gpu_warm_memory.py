"""Device memory of the warm-start network's calls: a large batch's buffer does not stay with the handle."""
import numpy as np
import pytest

from oracle import warm_mlp
from woo_gb300 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["predict", "grad"])
def test_large_batches_give_their_memory_back(wdem_lib, what):
    """2M records take 136 MB on the device; no more than 32 MB stay (64 allowed for the allocator's own blocks), and
    the next calls, small and large, give what they gave before."""
    import torch
    rng = np.random.default_rng(0)
    h = abi.Handle(1)
    h.warm_set_weights(warm_mlp.init(3).astype(np.float32))
    small = rng.uniform(-0.8, 0.8, (300, 17)).astype(np.float32)
    large = np.tile(small, (6667, 1))
    call = (lambda R: h.warm_predict(np.ascontiguousarray(R[:, :13]))) if what == "predict" else (lambda R: h.warm_grad(R)[0])
    first = call(small)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    a = call(large)
    assert free - torch.cuda.mem_get_info()[0] <= 64 << 20
    b = call(large)
    if what == "predict":
        assert np.array_equal(a, b) and np.array_equal(a[:300], first) and np.array_equal(call(small), first)
    else:
        # FP32 sums in another order, of up to 2e6 terms: 1e-3 of the largest entry
        for g in (a, b, call(small)):
            assert np.abs(g - first).max() <= 1e-3 * np.abs(first).max()
    h.close()
