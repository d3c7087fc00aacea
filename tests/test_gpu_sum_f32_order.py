"""The order in which the FP32 sums add their beams.

Two beams' values are added in plain FP32 before each compensated addition, no
more.  The ranges into which a small problem's beams are split, and their order,
follow from the problem alone: the homogeneous sums are the same bits whatever the
size of the caller's workspace, and the entry point without a workspace gives them
too.  The trajectory sums pair other beams where a workspace has no room for the
limits: the same to FP32 rounding.
"""

import re

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

    def transpose(self, nbytes):
        from beamax_b200 import _lib

        bs = self.bt.beam_set(unit=True)
        g = torch.full((self.n, 2), float("nan"), dtype=torch.float64, device=self.dev)
        ws = torch.full((max(nbytes, 256),), 0x5A, dtype=torch.uint8, device=self.dev)
        st = _lib.lib().msgb_adj_gather_f32(_lib.ref(self.pr), _lib.ref(bs), _lib.ref(self.opts), ws.data_ptr(), nbytes,
                                            self.data.data_ptr(), g.data_ptr(), torch.cuda.current_stream().cuda_stream)
        return st, g

    def static(self):
        from beamax_b200 import _lib

        bs = self.bt.beam_set()
        y = torch.full((self.nt, self.ns), float("nan"), dtype=torch.float32, device=self.dev)
        _lib.check(_lib.lib().msgb_sum_fwd_f32_static(_lib.ref(self.pr), _lib.ref(bs), _lib.ref(self.opts), y.data_ptr(),
                                                      torch.cuda.current_stream().cuda_stream), "static")
        return y


def _least(call):
    """The smallest workspace the call accepts, from its refusal of an empty one."""
    from beamax_b200 import _lib

    st, _ = call(0)
    assert st == 2  # MSGB_ERR_WORKSPACE
    return int(re.search(r"need (\d+) bytes", _lib.last_error()).group(1))


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


@pytest.mark.parametrize("d,n,ns,nt", [(2, 2000, 128, 64), (2, 3000, 1024, 600), (3, 900, 300, 40), (1, 700, 100, 70),
                                       (2, 129, 17, 33)])
def test_results_do_not_depend_on_the_workspace(d, n, ns, nt):
    c = _Case(d, n, ns, nt, seed=ns)
    st, y = c.forward(c.full)
    assert st == 0 and bool(torch.isfinite(y).all())
    least = _least(c.forward)
    for extra in (0, 2 * 8 * ns * nt + 256 * n, 5 * 8 * ns * nt + 256 * n):
        st, z = c.forward(least + extra)
        assert st == 0 and torch.equal(y, z)
    assert torch.equal(y, c.static())
    st, g = c.transpose(c.full)
    assert st == 0 and bool(torch.isfinite(g).all())
    st, h = c.transpose(_least(c.transpose))
    assert st == 0 and torch.equal(g, h)


@pytest.mark.parametrize("nb,ns,nt", [(700, 128, 64), (300, 33, 40)])
def test_trajectory_results_with_less_workspace(nb, ns, nt):
    """Pairs of other beams are added before a compensated addition: a rounding of
    2^-24 of the beams' values, which are at most 1, on each side."""
    from beamax_b200 import _lib

    dev = _dev()
    c = _Case(2, (nb + 1) // 2, ns, nt, seed=nb)
    rec = np.zeros((nt, nb), np.dtype([("x", "f8", 2), ("wp", "f8", 2), ("q", "f4", 3), ("p", "f4", 3), ("a", "f4", 2)]))
    rng = np.random.default_rng(nb)
    rec["x"], rec["wp"] = rng.random((1, nb, 2)) * 0.0256, rng.standard_normal((1, nb, 2)) * 1e4
    rec["p"][..., 0] = rec["p"][..., 2] = 1e5
    rec["a"] = 1.0
    d_rec = torch.from_numpy(rec.view(np.uint8)).to(dev)
    box = np.zeros(((nt + 31) // 32, nb, 5), np.float32)
    box[..., 0:2] = box[..., 2:4] = rec["x"][0]
    box[..., 4] = 0.99e5
    d_box = torch.from_numpy(box).to(dev)
    tr = _lib.Trajectories(nb=nb, rec32=d_rec.data_ptr(), cull=d_box.data_ptr())
    bs = c.bt.beam_set()

    def forward(nbytes):
        y = torch.full((nt, ns), float("nan"), dtype=torch.float32, device=dev)
        ws = torch.full((max(nbytes, 256),), 0x5A, dtype=torch.uint8, device=dev)
        half = [_lib.Trajectories(nb=nb, rec32=d_rec.data_ptr(), cull=d_box.data_ptr())] * 2
        st = 0
        for k, t in enumerate(half):  # two chunks (of the same beams): the state is carried over
            st = st or _lib.lib().msgb_sum_fwd_f32_traj(_lib.ref(c.pr), _lib.ref(bs), _lib.ref(t), _lib.ref(c.opts),
                                                        k == 0, k == 1, ws.data_ptr(), nbytes, y.data_ptr(),
                                                        torch.cuda.current_stream().cuda_stream)
        return st, y

    st, y = forward(_lib.lib().msgb_sum_f32_traj_workspace_size(_lib.ref(c.pr), nb))
    assert st == 0 and bool(torch.isfinite(y).all())
    least = _least(forward)
    for extra in (0, 2 * 8 * ns * nt, 16 * 8 * ns * nt):
        st, z = forward(least + extra)
        assert st == 0 and float((y - z).abs().max()) <= 4 * 2 * nb * 2.0 ** -24
