"""The order in which the FP32 sums add their beams: two beams' values are added in
plain FP32 before each compensated addition, no more.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda:0")


class _Case:
    """A problem of n beams and a row (or plane) of ns sensors through the C entry points."""

    def __init__(self, d, n, ns, nt, modes=0, width=None, N=256, seed=0):
        import beamax_b200 as bb
        from beamax_b200 import _lib
        from beamax_b200.solvers.msgb_solver import BeamTensors

        self.dev = dev = _dev()
        dx = 1e-4
        L = N * dx
        g = torch.Generator(device=dev).manual_seed(seed)
        rand = lambda *s: torch.rand(*s, generator=g, device=dev, dtype=torch.float64)
        p = rand(n, d) - 0.5
        p = 2 * np.pi * p / p.norm(dim=1, keepdim=True)
        om = (8 + 40 * rand(n)) / L
        w = (width or L / 12) * (0.6 + 0.8 * rand(n, d))
        a0 = torch.exp(2j * np.pi * rand(n)) * (0.2 + rand(n))
        self.bt = BeamTensors(rand(n, d) * L, p, (2j / (om[:, None] * w * w)).to(torch.complex128), a0,
                              torch.ones_like(a0), om, modes=modes)
        self.dom = bb.Domain(N=(N,) * d, dx=(dx,) * d, periodic=(False,) * d, cfl=0.3, c=1500.0)
        k = np.arange(ns)
        pos = np.stack([np.full(ns, 3), k % N, k // N][:d], -1) * dx if d > 1 else (k % N)[:, None] * dx
        if d == 2:
            pos[:, 0] += (k // N) * 20 * dx
        self.sens = bb.Sensor(self.dom, positions=pos)
        self.solver = bb.MSGBSolver(8, "top_n", 8, "spatial", bb.gb.gb_solvers.solve_hom_diag, "scan_real",
                                    precision="fp32")
        self.pr, self.keep = self.solver._problem(self.dom, self.sens, np.arange(nt) * 0.3 * dx / 1500.0, dev)
        self.opts = _lib.SumOpts(cutoff=16.0)
        self.nt, self.ns, self.n = nt, ns, n
        self.data = torch.randn(nt, ns, generator=g, device=dev)
        self.full = _lib.lib().msgb_sum_f32_workspace_size(_lib.ref(self.pr), n)

    def forward(self, nbytes, bt=None):
        from beamax_b200 import _lib

        bt = bt or self.bt
        bs = bt.beam_set()
        y = torch.full((self.nt, self.ns), float("nan"), dtype=torch.float32, device=self.dev)
        ws = torch.full((max(nbytes, 256),), 0x5A, dtype=torch.uint8, device=self.dev)
        st = _lib.lib().msgb_sum_fwd_f32(_lib.ref(self.pr), _lib.ref(bs), _lib.ref(self.opts), ws.data_ptr(), nbytes,
                                         y.data_ptr(), torch.cuda.current_stream().cuda_stream)
        return st, y


@pytest.mark.parametrize("n", [2, 3, 4, 7, 12, 31])
@pytest.mark.parametrize("d", [2, 3])
def test_two_beams_are_added_before_each_compensated_addition(d, n):
    """A pass of beams at full runs of sensors equals, bit for bit, the beams' own
    values added in pairs and then with Kahan's compensation."""
    c = _Case(d, n, 32, 32, modes=1, width=0.2, seed=n)
    st, y = c.forward(c.full)
    assert st == 0
    one = []
    for j in range(n):
        pick = lambda a: a[j:j + 1].contiguous()
        b = type(c.bt)(*(pick(getattr(c.bt, f)) for f in ("x0", "p0", "alpha", "a0", "a0_unit", "omega")), modes=1)
        one.append(c.forward(c.full, b)[1].cpu().numpy())
    acc, comp = np.zeros_like(one[0]), np.zeros_like(one[0])
    for j in range(0, n, 2):
        v = one[j] + (one[j + 1] if j + 1 < n else np.float32(0))
        t = v - comp
        s = acc + t
        comp = (s - acc) - t
        acc = s
    assert np.array_equal(y.cpu().numpy(), acc - comp)
