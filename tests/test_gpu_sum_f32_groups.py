"""The FP32 sums at the sizes where their tiles, record passes, splits and
group masks have edges, against the dense FP64 sums of the same beams.

Tolerance: a value of the 16-sensor recurrence is off by at most
15^2 / 2 roundings of 2^-24 in its ratio plus the seed's few, below 1e-5 of the
beam's amplitude; errors and values of different beams add alike, so rel-L2
stays within 3e-5.  What the cutoff (16 e-folds) and the group test (20) leave
out is below e^-16 = 1.2e-7 of a beam's amplitude, per value (the only error
left where no beam comes near a sensor).  The transpose sums the same values.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

TOL = 3e-5


def _dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda:0")


def _beams(d, n, L, dev, seed, width=None, tilted=False):
    """Random beams over the domain: anisotropic widths of about L / 12, complex
    M0 (the general closed form) when tilted."""
    from beamax_b200.solvers.msgb_solver import BeamTensors

    g = torch.Generator(device=dev).manual_seed(seed)
    rand = lambda *s: torch.rand(*s, generator=g, device=dev, dtype=torch.float64)
    x0 = rand(n, d) * L
    p = rand(n, d) - 0.5
    p = 2 * np.pi * p / p.norm(dim=1, keepdim=True)
    om = (8 + 40 * rand(n)) / L
    w = (width or L / 12) * (0.6 + 0.8 * rand(n, d))
    al = 2j / (om[:, None] * w * w)
    if tilted:
        al = al + (rand(n, d) - 0.5) * al.abs()
    a0 = torch.exp(2j * np.pi * rand(n)) * (0.2 + rand(n))
    return BeamTensors(x0, p, al.to(torch.complex128), a0, torch.ones_like(a0), om)


def _compare(d, N, positions, nt, bt, cutoff=16.0):
    import beamax_b200 as bb

    dx = 1e-4
    dom = bb.Domain(N=(N,) * d, dx=(dx,) * d, periodic=(False,) * d, cfl=0.3, c=1500.0)
    sens = bb.Sensor(dom, positions=positions)
    ts = np.arange(nt) * 0.3 * dx / 1500.0
    hom = bb.gb.gb_solvers.solve_hom_diag
    s32 = bb.MSGBSolver(8, "top_n", 8, "spatial", hom, "scan_real", precision="fp32", cutoff=cutoff)
    s64 = bb.MSGBSolver(8, "top_n", 8, "spatial", hom, "scan_real")
    y64, y32 = s64.sum_forward(bt, dom, sens, ts), s32.sum_forward(bt, dom, sens, ts).double()
    left_out = 1.2e-7 * 4 * float(bt.a0.abs().sum()) * y64.numel() ** 0.5
    assert float((y32 - y64).norm()) <= TOL * float(y64.norm()) + left_out
    data = torch.randn(y64.shape, generator=torch.Generator(device=y64.device).manual_seed(3), device=y64.device,
                       dtype=torch.float64)
    g64, g32 = s64.gather_adjoint(bt, dom, sens, ts, data), s32.gather_adjoint(bt, dom, sens, ts, data)
    left_out = 1.2e-7 * 4 * float(data.norm()) * (y64.numel() * bt.n) ** 0.5
    assert float((g32 - g64).norm()) <= TOL * float(g64.norm()) + left_out


def _line(ns, N, dx=1e-4):
    return np.stack([np.full(ns, 3), (np.arange(ns) + 1) % N], -1) * dx


@pytest.mark.parametrize("ns", [1, 4, 15, 16, 17, 127, 128, 129, 200])
@pytest.mark.parametrize("nt", [1, 33])
def test_line_sensor_at_group_and_tile_edges(ns, nt):
    dev = _dev()
    _compare(2, 256, _line(ns, 256), nt, _beams(2, 150, 256e-4, dev, ns))


@pytest.mark.parametrize("n", [1, 2, 3, 5, 31, 33, 129, 1025])
def test_beam_counts_at_pass_scan_and_split_edges(n):
    dev = _dev()
    _compare(2, 256, _line(70, 256), 64, _beams(2, n, 256e-4, dev, n))


@pytest.mark.parametrize("case", ["cutoff0", "narrow", "tilted", "ring", "scattered"])
def test_variants_2d(case):
    """No culling; beams narrower than a sensor step (direct evaluation inside
    straight runs); the general closed form; off-grid and scattered sensors."""
    dev = _dev()
    L = 256e-4
    bt = _beams(2, 300, L, dev, 7, width=1.2e-4 if case == "narrow" else None, tilted=case == "tilted")
    pos = _line(150, 256)
    if case == "ring":
        th = 2 * np.pi * np.arange(170) / 170
        pos = 0.5 * L + 0.4 * L * np.stack([np.cos(th), np.sin(th)], -1)
    if case == "scattered":
        q = np.random.default_rng(0).choice(256 * 256, 145, replace=False)
        pos = np.stack([q // 256, q % 256], -1) * 1e-4
    _compare(2, 256, pos, 40, bt, cutoff=0.0 if case == "cutoff0" else 16.0)


@pytest.mark.parametrize("d,shape", [(1, (5,)), (3, (9, 17)), (3, (20, 40))])
def test_other_dimensions(d, shape):
    dev = _dev()
    N = 64
    if d == 1:
        pos = (np.arange(shape[0]) * 7 + 2)[:, None] * 1e-4
    else:
        a, b = np.meshgrid(np.arange(shape[0]), np.arange(shape[1]), indexing="ij")
        pos = np.stack([a.ravel(), b.ravel(), np.full(a.size, 0)], -1) * 1e-4
    _compare(d, N, pos, 35, _beams(d, 90, N * 1e-4, dev, d))


@pytest.mark.parametrize("d", [2, 3])
def test_trajectory_candidates_left_out_do_not_matter(d):
    """Beams in a strongly refracting medium: with culling (tile test, the test on
    four of a tile's records, group test) against every beam at every sensor."""
    import beamax_b200 as bb
    from beamax_b200.utils.interp import make_c_function_from_grid

    dev = _dev()
    N, dx = (128, 1e-4) if d == 2 else (48, 1e-4)
    ax = np.stack(np.meshgrid(*[np.arange(N)] * d, indexing="ij"), 0)
    c = 1500 * (1 + 0.08 * np.sin(2 * np.pi * ax[0] / 40) * np.cos(2 * np.pi * ax[-1] / 33))
    med = make_c_function_from_grid(c, (dx,) * d, method="bspline3", boundary="clamp")
    dom = bb.Domain(N=(N,) * d, dx=(dx,) * d, periodic=(False,) * d, cfl=0.3, c=med)
    mask = np.zeros((N,) * d)
    mask[0] = 1
    sens = bb.Sensor(dom, binary_mask=mask)
    ts = np.arange(300) * 0.3 * dx / 1620
    bt = _beams(d, 200, N * dx, dev, 11 + d, width=N * dx / 25)
    ode = bb.gb.gb_solvers.solve_ODE_base
    mk = lambda cut: bb.MSGBSolver(8, "top_n", 8, "spatial", ode, "scan_real", precision="fp32", cutoff=cut)
    y, y0 = (mk(cut).sum_forward(bt, dom, sens, ts).double() for cut in (16.0, 0.0))
    # focusing raises an amplitude by at most 10 here
    left_out = 1.2e-7 * 40 * float(bt.a0.abs().sum())
    assert float((y - y0).abs().max()) <= left_out + 1e-5 * float(y0.abs().max())
    data = torch.randn(y0.shape, generator=torch.Generator(device=dev).manual_seed(3), device=dev)
    g, g0 = (mk(cut).gather_adjoint(bt, dom, sens, ts, data) for cut in (16.0, 0.0))
    assert float((g - g0).norm()) <= 1e-5 * float(g0.norm())
