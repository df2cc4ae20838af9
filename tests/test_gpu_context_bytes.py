"""GPU test: the device memory that a context allocates stays below the figure for
admission control, also where a tall factor's copies outweigh V."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,k,arm", [(3000000, 64, 64, "fused"), (3000000, 40, 17, "bf16x3"), (64, 2000000, 64, "split_bf16"),
                                       (2000000, 70, 66, "plain"), (5000, 38, 3, "fused")])
def test_bound_holds(pkg, n, m, k, arm):
    import torch

    torch.cuda.empty_cache()
    pkg.load_library().nmfb_release_cached(0)
    before = torch.cuda.mem_get_info()[0]
    with pkg.NMF(n, m, k, arm=arm):
        taken = before - torch.cuda.mem_get_info()[0]
    pkg.load_library().nmfb_release_cached(0)
    assert taken <= pkg.context_bytes(n, m, k, arm)
