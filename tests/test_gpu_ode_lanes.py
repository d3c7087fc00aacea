"""The beam ODE does not depend on which lanes and warps integrate the beams,
nor on the grid cells their stencils came from: the FP32 and FP64 records of a
set of beams equal, bit for bit, those of the same beams integrated in other
chunks (a lane's arithmetic is its own; chunk sizes around the warp, the block
and the spread of few beams over the GPU).  Beams start at the grid's edges and
leave it, under every boundary rule, in 1D, 2D and 3D, linear and cubic.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _records(s, pr, med, bs, b_first, nb, fp64, dev):
    d = pr.ndim
    size = (2 * d + 2 * d * d + 2) * 8 if fp64 else 16 * d + 4 * d * (d + 1) + 8
    n_tt = (pr.nt + 31) // 32
    per = pr.nt * size + n_tt * (2 * d + 1) * 4
    status = torch.zeros(2 * bs.n, dtype=torch.int32, device=dev)
    buf = torch.empty(per * nb + 4096, dtype=torch.uint8, device=dev)
    s._trajectories(pr, med, bs, b_first, nb, fp64, per, n_tt, dev, torch.cuda.current_stream().cuda_stream, status, buf)
    torch.cuda.synchronize()
    assert int(status.max()) == 0
    return buf[:pr.nt * nb * size].reshape(pr.nt, nb, size).clone()


@pytest.mark.parametrize("d,method,boundary", [(2, "bspline3", "clamp"), (2, "bspline3", "wrap"), (2, "bspline3", "mirror"),
                                               (2, "linear", "clamp"), (1, "bspline3", "clamp"), (3, "bspline3", "clamp")])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_records_do_not_depend_on_the_chunk(d, method, boundary, precision):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import beamax_b200 as bb
    from beamax_b200.solvers.msgb_solver import BeamTensors
    from beamax_b200.utils.interp import make_c_function_from_grid

    dev = torch.device("cuda:0")
    N, dx, n = 24, 1e-4, 350
    rng = np.random.default_rng(d)
    ax = np.stack(np.meshgrid(*[np.arange(N)] * d, indexing="ij"), 0)
    c = 1500 * (1 + 0.03 * np.sin(2 * np.pi * (ax.sum(0) + rng.uniform()) / N))
    med = make_c_function_from_grid(c, (dx,) * d, method=method, boundary=boundary)
    dom = bb.Domain(N=(N,) * d, dx=(dx,) * d, periodic=(False,) * d, cfl=0.3, c=med)
    sens = bb.Sensor(dom, positions=np.full((1, d), 2 * dx))
    ts = np.arange(41) * 0.3 * dx / 1500
    g = torch.Generator(device=dev).manual_seed(5)
    rand = lambda *s: torch.rand(*s, generator=g, device=dev, dtype=torch.float64)
    p = rand(n, d) - 0.5
    p = 2 * np.pi * p / p.norm(dim=1, keepdim=True)
    om = (2 + 4 * rand(n)) / (N * dx)
    bt = BeamTensors(rand(n, d) * N * dx, p, 2j / (om[:, None] * (4 * dx) ** 2 * (1 + rand(n, d))),
                     torch.ones(n, dtype=torch.complex128, device=dev), torch.ones(n, dtype=torch.complex128, device=dev), om)
    s = bb.MSGBSolver(8, "top_n", 8, "spatial", bb.gb.gb_solvers.solve_ODE_base, "scan_real", precision=precision)
    pr, k1 = s._problem(dom, sens, ts, dev)
    m, k2 = s._medium(dom, dev)
    bs = bt.beam_set()
    fp64 = precision == "fp64"
    whole = _records(s, pr, m, bs, 0, 2 * n, fp64, dev)
    first = 0
    for nb in (1, 2, 31, 33, 63, 65, 130, 375):
        part = _records(s, pr, m, bs, first, nb, fp64, dev)
        assert torch.equal(part, whole[:, first:first + nb])
        first += nb
    assert first == 2 * n
