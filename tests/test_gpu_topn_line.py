"""msgb_topn on both sides of the line between selecting first and sorting everything
(2,800,000 keys more than twice the selected), against the rule itself: sort by (key,
index), keep the last n."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("total,n", [(2900000, 50000), (2900000, 50001), (2804097, 2049), (4200001, 262144), (3000000, 1500000)])
@pytest.mark.parametrize("zeros", [0.5, 0.999])
def test_lists_are_equal_on_both_sides(total, n, zeros):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from beamax_b200 import _lib

    rng = np.random.default_rng(total)
    keys = rng.random(total)
    keys[rng.random(total) < zeros] = 0.0
    dev = torch.device("cuda:0")
    kd = torch.from_numpy(keys).to(dev)
    c = torch.randn(total, 2, dtype=torch.float64, device=dev)
    nbytes = _lib.lib().msgb_topn_workspace_size(total, n)
    ws = torch.full((nbytes,), 0x5A, dtype=torch.uint8, device=dev)
    idx = torch.empty(n, dtype=torch.int64, device=dev)
    val = torch.empty(n, 2, dtype=torch.float64, device=dev)
    _lib.check(_lib.lib().msgb_topn(kd.data_ptr(), c.data_ptr(), total, n, idx.data_ptr(), val.data_ptr(), ws.data_ptr(),
                                    nbytes, torch.cuda.current_stream().cuda_stream), "msgb_topn")
    want = torch.sort(kd, stable=True).indices[-n:]  # equal keys in index order
    assert torch.equal(idx, want) and torch.equal(val, c[want])
