"""The dense FP64 sums at the edges of their tiles, passes and cluster splits
against the same formula in plain torch, complex128.

Tolerance: both sides round the phase (up to about 300 rad here, 6e-14) and the
exponent; errors and values of different beams add alike, so rel-L2 <= 1e-12.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda:0")


def _reference(bt, modes, c0, ts, pos, data):
    """(field, per-coefficient transpose) of the beams at every time and position."""
    d = bt.x0.shape[1]
    np_ = bt.p0.norm(dim=1)
    u = bt.p0 / np_[:, None]
    eye = torch.eye(d, dtype=torch.complex128, device=pos.device)
    H = (eye - (u[:, :, None] * u[:, None, :]).to(torch.complex128)) / np_[:, None, None]
    M0 = torch.diag_embed(bt.alpha)
    y = torch.zeros(len(ts), len(pos), dtype=torch.float64, device=pos.device)
    g = torch.zeros(bt.n, dtype=torch.complex128, device=pos.device)
    for i, t in enumerate(ts):
        for c in modes:
            T = eye + c * c0 * t * (H @ M0)
            M = M0 @ torch.linalg.inv(T)
            D = pos[None] - (bt.x0 + c * c0 * t * u)[:, None, :]
            ph = (D * bt.p0[:, None, :]).sum(-1) + 0.5 * torch.einsum("bsi,bij,bsj->bs", D.to(torch.complex128), M,
                                                                      D.to(torch.complex128))
            K = torch.exp(1j * bt.omega[:, None] * ph) / torch.sqrt(torch.linalg.det(T))[:, None]
            y[i] += 2 * (bt.a0[:, None] * K).sum(0).real
            g += 2 * torch.conj(bt.a0_unit) * (torch.conj(K) @ data[i].to(torch.complex128))
    return y, g


def _run(d, n, ns, nt, modes=0, seed=0):
    import beamax_b200 as bb
    from beamax_b200.solvers.msgb_solver import BeamTensors

    dev = _dev()
    N, dx = 64, 1e-4
    L = N * dx
    gen = torch.Generator(device=dev).manual_seed(seed)
    rand = lambda *s: torch.rand(*s, generator=gen, device=dev, dtype=torch.float64)
    p = rand(n, d) - 0.5
    p = 2 * np.pi * p / p.norm(dim=1, keepdim=True)
    om = (4 + 20 * rand(n)) / L
    w = L / 6 * (0.6 + 0.8 * rand(n, d))
    a0 = torch.exp(2j * np.pi * rand(n)) * (0.2 + rand(n))
    bt = BeamTensors(rand(n, d) * L, p, 2j / (om[:, None] * w * w), a0, torch.exp(2j * np.pi * rand(n)), om, modes=modes)
    dom = bb.Domain(N=(N,) * d, dx=(dx,) * d, periodic=(False,) * d, cfl=0.3, c=1500.0)
    rng = np.random.default_rng(seed)
    pos = np.stack(np.unravel_index(rng.choice(N ** d, ns, replace=False), (N,) * d), -1) * dx
    sens = bb.Sensor(dom, positions=pos)
    ts = np.arange(nt) * 0.3 * dx / 1500.0
    s = bb.MSGBSolver(8, "top_n", 8, "spatial", bb.gb.gb_solvers.solve_hom_diag, "scan_real")
    data = torch.randn(nt, ns, generator=gen, device=dev, dtype=torch.float64)
    y, g = s.sum_forward(bt, dom, sens, ts), s.gather_adjoint(bt, dom, sens, ts, data)
    yr, gr = _reference(bt, {0: (1, -1), 1: (1,), 2: (-1,)}[modes], 1500.0, ts, torch.from_numpy(pos).to(dev), data)
    assert float((y - yr).norm()) <= 1e-12 * float(yr.norm())
    assert float((g - gr).norm()) <= 1e-12 * float(gr.norm())


@pytest.mark.parametrize("ns", [1, 31, 33, 63, 64, 65, 511, 513])
@pytest.mark.parametrize("nt", [1, 15, 17])
def test_tile_edges(ns, nt):
    _run(2, 70, ns, nt, seed=ns)


@pytest.mark.parametrize("n", [1, 16, 17, 255, 257, 1100])
def test_beam_counts_at_pass_and_split_edges(n):
    _run(2, n, 130, 20, seed=n)


@pytest.mark.parametrize("d,modes", [(1, 0), (3, 0), (2, 1), (2, 2)])
def test_dimensions_and_modes(d, modes):
    _run(d, 40, 60, 18, modes=modes, seed=d)


@pytest.mark.parametrize("scale", [1e6, -1.0, float("nan")])
def test_values_outside_the_reduced_functions_range(scale):
    """Exponents far beyond underflow, growing beams and a NaN M0: zero,
    finite, NaN where exp and cos say so."""
    import beamax_b200 as bb
    from beamax_b200.solvers.msgb_solver import BeamTensors

    dev = _dev()
    one = torch.ones(1, dtype=torch.complex128, device=dev)
    x0 = torch.tensor([[3e-3, 3e-3]], dtype=torch.float64, device=dev)
    p = torch.tensor([[2 * np.pi, 0.0]], dtype=torch.float64, device=dev)
    om = torch.tensor([3000.0], dtype=torch.float64, device=dev)
    al = 1j * torch.full((1, 2), 700.0, dtype=torch.float64, device=dev) * scale
    bt = BeamTensors(x0, p, al.to(torch.complex128), one, one, om)
    dom = bb.Domain(N=(64, 64), dx=(1e-4, 1e-4), periodic=(False, False), cfl=0.3, c=1500.0)
    pos = np.array([[3e-3, 3e-3], [1e-3, 5e-3], [6e-3, 1e-3]])
    sens = bb.Sensor(dom, positions=pos)
    s = bb.MSGBSolver(8, "top_n", 8, "spatial", bb.gb.gb_solvers.solve_hom_diag, "scan_real")
    ts = np.zeros(1)
    data = torch.ones(1, 3, dtype=torch.float64, device=dev)
    y, g = s.sum_forward(bt, dom, sens, ts)[0], s.gather_adjoint(bt, dom, sens, ts, data)[0]
    D = torch.from_numpy(pos).to(dev) - x0
    chi = 0.5 * om * (al.imag * D * D).sum(1)
    ref = 4 * torch.cos(om * (D * p).sum(1)) * torch.exp(-chi)  # both branches at t = 0
    assert torch.equal(torch.isnan(y), torch.isnan(ref)) and torch.equal(torch.isinf(y), torch.isinf(ref))
    fin = torch.isfinite(ref)
    assert bool((y[fin] - ref[fin]).abs().le(1e-12 * ref[fin].abs()).all())
    if bool(fin.all()):
        assert abs(float(g.real) - float(ref.sum())) <= 1e-12 * float(ref.abs().sum())
    else:
        assert not bool(torch.isfinite(g.real))
