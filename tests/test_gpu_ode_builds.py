"""The mixed-precision beam ODE's builds and boxes.

The integrator is built for six and for seven blocks per SM, chosen by the number
of beams, and a lane that finishes takes another beam: the records of many beams in
one call equal, bit for bit, those of the same beams in calls of a few thousand.
The culling box of a time tile holds a lower bound on the eigenvalues of the
records' exponents, at every scale of the Hessian.
"""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda:0")


def _setup(dev, n, alpha_of, nt, N=24, d=2, method="bspline3"):
    """(solver, problem, medium, beam set, tensors kept alive) of n beams."""
    import beamax_b200 as bb
    from beamax_b200.solvers.msgb_solver import BeamTensors
    from beamax_b200.utils.interp import make_c_function_from_grid

    dx = 1e-4
    ax = np.stack(np.meshgrid(*[np.arange(N)] * d, indexing="ij"), 0)
    c = 1500 * (1 + 0.03 * np.sin(2 * np.pi * ax.sum(0) / N))
    dom = bb.Domain(N=(N,) * d, dx=(dx,) * d, periodic=(False,) * d, cfl=0.3,
                    c=make_c_function_from_grid(c, (dx,) * d, method=method, boundary="clamp"))
    sens = bb.Sensor(dom, positions=np.full((1, d), 2 * dx))
    g = torch.Generator(device=dev).manual_seed(5)
    rand = lambda *s: torch.rand(*s, generator=g, device=dev, dtype=torch.float64)
    p = rand(n, d) - 0.5
    p = 2 * np.pi * p / p.norm(dim=1, keepdim=True)
    om = (2 + 4 * rand(n)) / (N * dx)
    one = torch.ones(n, dtype=torch.complex128, device=dev)
    bt = BeamTensors(rand(n, d) * N * dx, p, alpha_of(om, rand(n, d)).to(torch.complex128), one, one, om)
    s = bb.MSGBSolver(8, "top_n", 8, "spatial", bb.gb.gb_solvers.solve_ODE_base, "scan_real", precision="fp32")
    pr, k1 = s._problem(dom, sens, np.arange(nt) * 0.3 * dx / 1500, dev)
    m, k2 = s._medium(dom, dev)
    return s, pr, m, bt.beam_set(), (bt, k1, k2, dom)


def _integrate(s, pr, m, bs, first, nb, dev):
    """(records, boxes) of beams [first, first + nb)."""
    d, n_tt = pr.ndim, (pr.nt + 31) // 32
    size = 16 * d + 4 * d * (d + 1) + 8
    per = pr.nt * size + n_tt * (2 * d + 1) * 4
    status = torch.zeros(2 * bs.n, dtype=torch.int32, device=dev)
    buf = torch.empty(per * nb + 4096, dtype=torch.uint8, device=dev)
    tr = s._trajectories(pr, m, bs, first, nb, False, per, n_tt, dev, torch.cuda.current_stream().cuda_stream, status, buf)
    torch.cuda.synchronize()
    assert int(status.max()) == 0
    at = (tr[0] if isinstance(tr, tuple) else tr).cull - buf.data_ptr()
    box = buf[at:at + 4 * n_tt * nb * (2 * d + 1)].view(torch.float32).reshape(n_tt, nb, 2 * d + 1)
    return buf[:pr.nt * nb * size].reshape(pr.nt, nb, size), box


@pytest.mark.parametrize("method,d", [("bspline3", 2), ("linear", 2), ("bspline3", 1)])
def test_many_beams_equal_the_same_beams_in_small_calls(method, d):
    """120,000 beams: more than the lanes of six or seven blocks on every SM."""
    dev = _dev()
    n, dx = 60000, 1e-4
    s, pr, m, bs, keep = _setup(dev, n, lambda om, r: 2j / (om[:, None] * (4 * dx) ** 2 * (1 + r)), 6, d=d, method=method)
    whole, _ = _integrate(s, pr, m, bs, 0, 2 * n, dev)
    for first, nb in ((0, 4000), (4000, 37), (57000, 6000), (63000, 43000), (2 * n - 5000, 5000)):
        part, _ = _integrate(s, pr, m, bs, first, nb, dev)
        assert torch.equal(part, whole[:, first:first + nb])


@pytest.mark.parametrize("scale", [1e-23, 1e-22, 1e-21, 1e-19, 1e-10, 1.0, 1e5])
def test_the_box_bounds_the_eigenvalues_at_every_scale(scale):
    """(w/2) lambda_min of the box against the records' own packed (w/2) Im M, in FP64.
    The records' three floats are rounded by 2^-24 each: an eigenvalue moves by at
    most the Frobenius norm of that, below 2^-23 of the largest one."""
    dev = _dev()
    s, pr, m, bs, keep = _setup(dev, 500, lambda om, r: 1j * scale * (1 + 9 * r), 40)
    rec, box = _integrate(s, pr, m, bs, 0, 1000, dev)
    P = rec.view(torch.float32).reshape(pr.nt, 1000, 16)[..., 11:14].double()
    h, mid = 0.5 * (P[..., 0] - P[..., 2]), 0.5 * (P[..., 0] + P[..., 2])
    r = torch.sqrt(h * h + 0.25 * P[..., 1] ** 2)
    lam = mid - r + 2.0 ** -23 * (mid + r)
    low = torch.stack([lam[t:t + 32].min(0).values for t in range(0, pr.nt, 32)])
    assert bool((box[..., 4].double() <= low).all())
    assert bool((box[..., 4] >= 0).all())
