"""msgb_topn at the edges of its two routes (the full sort; the radix select
and a sort of the selected) against the rule itself: sort by (key, index), keep
the last n.  Index lists are equal, ties, zeros, infinities and NaN included
(NaN keys rank above infinity, as their bit patterns do)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _keys(kind, total, rng):
    if kind == "random":
        return rng.random(total)
    if kind == "ties":
        return rng.integers(0, 7, total) * 0.125
    if kind == "equal":
        return np.full(total, 3.0)
    if kind == "halfzero":
        k = rng.random(total) * 10.0 ** rng.integers(-300, 300, total)
        k[::2] = 0.0
        k[1::64] = -0.0
        return k
    k = rng.random(total)
    k[rng.integers(0, total, 9)] = np.inf
    k[rng.integers(0, total, 5)] = np.nan
    return k


@pytest.mark.parametrize("kind", ["random", "ties", "equal", "halfzero", "special"])
@pytest.mark.parametrize("total", [100, 8192, 8193, 20000, 300001, (1 << 21) - 1, (1 << 21) + 3])
def test_selected_indices_and_order(kind, total):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from beamax_b200 import _lib

    dev = torch.device("cuda:0")
    rng = np.random.default_rng(total)
    keys = _keys(kind, total, rng)
    bits = np.where(keys == 0, 0.0, keys).view(np.uint64)
    order = np.lexsort((np.arange(total), bits))
    kd = torch.from_numpy(keys).to(dev)
    c = torch.from_numpy(rng.standard_normal((total, 2))).to(dev)
    L = _lib.lib()
    for n in sorted({1, 2, 37, min(total, 2048), min(total, 2049), total // 3, total // 2, total // 2 + 1, total}):
        nbytes = L.msgb_topn_workspace_size(total, n)
        ws = torch.full((nbytes,), 0x5A, dtype=torch.uint8, device=dev)
        idx = torch.empty(n, dtype=torch.int64, device=dev)
        val = torch.empty(n, 2, dtype=torch.float64, device=dev)
        _lib.check(L.msgb_topn(kd.data_ptr(), c.data_ptr(), total, n, idx.data_ptr(), val.data_ptr(), ws.data_ptr(),
                               nbytes, torch.cuda.current_stream().cuda_stream), "msgb_topn")
        want = order[-n:]
        assert np.array_equal(idx.cpu().numpy(), want)
        assert torch.equal(val, c[idx])
