"""Beams whose exponent has no positive lower bound, or none that is known, are in
every FP32 sum: the culling tests leave a beam out only where its exponent is
provably beyond the cutoff.

Not finite: a NaN in a beam's centre, momentum or Hessian reaches every output of
the forward and the beam's own entry of the transpose, as in the FP64 sums.
Growing: an indefinite Im M, whose exponent along a row of sensors is concave, in
the closed form and in trajectory records with an open culling box.  Varying:
records that come near a sensor at a few times of a tile only, or whose centre and
Hessian jump from time to time.

Tolerances: 3e-5 rel-L2 of the FP64 value, as for every FP32 sum (at most 15^2 / 2
roundings of 2^-24 in a run's ratio, plus the seed's); the trajectory cases also
leave out e^-16 of a beam's amplitude per value.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

TOL = 3e-5
DX = 1e-4
N = 256


def _dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda:0")


def _positions(kind):
    """line: one full tile of straight runs; run, runs: 16 and 32 sensors; short: a
    group that is not full; scattered: no straight run."""
    if kind == "scattered":
        rng = np.random.default_rng(0)
        q = rng.choice(90, 60, replace=False)
        return (np.stack([40 + q // 15, 40 + q % 15], -1) + 0.3 * rng.random((60, 2))) * DX
    ns = {"line": 128, "run": 16, "runs": 32, "short": 5}[kind]
    return np.stack([np.full(ns, 40), 40 + np.arange(ns)], -1) * DX


def _domain(positions):
    import beamax_b200 as bb

    dom = bb.Domain(N=(N, N), dx=(DX, DX), periodic=(False, False), cfl=0.3, c=1500.0)
    return dom, bb.Sensor(dom, positions=positions)


def _solvers():
    import beamax_b200 as bb

    hom = bb.gb.gb_solvers.solve_hom_diag
    return (bb.MSGBSolver(8, "top_n", 8, "spatial", hom, "scan_real", precision="fp32"),
            bb.MSGBSolver(8, "top_n", 8, "spatial", hom, "scan_real"))


def _beams(n, dev, x0, alpha, seed=1):
    from beamax_b200.solvers.msgb_solver import BeamTensors

    g = torch.Generator(device=dev).manual_seed(seed)
    p = torch.rand(n, 2, generator=g, device=dev, dtype=torch.float64) - 0.5
    p = 2 * np.pi * p / p.norm(dim=1, keepdim=True)
    a0 = torch.exp(2j * np.pi * torch.rand(n, generator=g, device=dev, dtype=torch.float64))
    om = torch.full((n,), 400.0, dtype=torch.float64, device=dev)
    return BeamTensors(x0, p, alpha.to(torch.complex128), a0, torch.ones_like(a0), om)


def _rel(a, b):
    return float((a - b).norm()) / float(b.norm())


@pytest.mark.parametrize("kind", ["line", "run", "short", "scattered"])
@pytest.mark.parametrize("field", ["x0", "p0", "alpha"])
def test_a_beam_that_is_not_finite_reaches_the_output(kind, field):
    dev = _dev()
    n, bad = 40, 17
    dom, sens = _domain(_positions(kind))
    ts = np.arange(34) * 0.3 * DX / 1500.0
    x0 = torch.rand(n, 2, generator=torch.Generator(device=dev).manual_seed(2), device=dev, dtype=torch.float64) * N * DX
    w = 400.0
    bt = _beams(n, dev, x0, torch.full((n, 2), 2j / (w * (10 * DX) ** 2), device=dev))
    getattr(bt, field)[bad] = float("nan")
    s32, s64 = _solvers()
    y = s32.sum_forward(bt, dom, sens, ts)
    assert bool(torch.isnan(s64.sum_forward(bt, dom, sens, ts)).all())
    assert bool(torch.isnan(y).all())
    data = torch.randn(y.shape, generator=torch.Generator(device=dev).manual_seed(3), device=dev, dtype=torch.float64)
    g32, g64 = s32.gather_adjoint(bt, dom, sens, ts, data), s64.gather_adjoint(bt, dom, sens, ts, data)
    nan = torch.isnan(torch.view_as_real(g32)).any(1)
    assert bool(nan[bad]) and int(nan.sum()) == 1
    ok = torch.arange(n, device=dev) != bad
    left_out = 1.2e-7 * 4 * float(data.norm()) * (y.numel() * n) ** 0.5
    assert float((g32[ok] - g64[ok]).norm()) <= TOL * float(g64[ok].norm()) + left_out


@pytest.mark.parametrize("kind", ["run", "runs", "short", "scattered"])
def test_a_growing_beam_is_in_every_group_of_sensors(kind):
    """chi = 25 - 0.1 k^2 from the sensor row's last group: 25 at its first sensor,
    2.5 at its last; scattered: 25 at the group's middle, less at its rim."""
    dev = _dev()
    pos = _positions(kind)
    dom, sens = _domain(pos)
    w, n = 400.0, 5
    off = {"run": 0, "runs": 16, "short": 0, "scattered": 7}[kind]
    grow = {"run": 0.1, "runs": 0.1, "short": 1.2, "scattered": 0.45}[kind]
    b0, b1 = 2 * 25.0 / (w * (10 * DX) ** 2), 2 * grow / (w * DX ** 2)
    x0 = torch.tensor([[30 * DX, (40 + off) * DX]] * n, dtype=torch.float64, device=dev)
    x0 = x0 + 1e-2 * DX * torch.arange(n, device=dev, dtype=torch.float64)[:, None]
    bt = _beams(n, dev, x0, torch.tensor([[1j * b0, -1j * b1]] * n, device=dev))
    ts = np.arange(3) * 1e-3 * DX / 1500.0
    s32, s64 = _solvers()
    y64 = s64.sum_forward(bt, dom, sens, ts)
    assert _rel(s32.sum_forward(bt, dom, sens, ts).double(), y64) <= TOL
    data = torch.randn(y64.shape, generator=torch.Generator(device=dev).manual_seed(3), device=dev, dtype=torch.float64)
    g64 = s64.gather_adjoint(bt, dom, sens, ts, data)
    assert _rel(s32.gather_adjoint(bt, dom, sens, ts, data), g64) <= TOL


# ---- trajectory records --------------------------------------------------------
PAIRS = {1: [(0, 0)], 2: [(0, 0), (0, 1), (1, 1)], 3: [(0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2)]}


def _rec(d):
    S = len(PAIRS[d])
    return np.dtype([("x", "f8", d), ("wp", "f8", d), ("q", "f4", S), ("p", "f4", S), ("ang", "f4"), ("amp", "f4")])


def _matrix(p, d):
    """Packed coefficients (off-diagonals doubled) -> symmetric matrices."""
    M = np.zeros(p.shape[:-1] + (d, d))
    for e, (i, k) in enumerate(PAIRS[d]):
        M[..., i, k] = M[..., k, i] = p[..., e] * (1.0 if i == k else 0.5)
    return M


class _Records:
    """Records of nb beams at nt times, their boxes, and the sums over them."""

    def __init__(self, rec, open_box, pos, cutoff=16.0):
        from beamax_b200 import _lib

        self.dev = _dev()
        self.rec, self.d = rec, rec["x"].shape[-1]
        d = self.d
        # 1D: along the row; 3D: the row lies in a plane
        pos = pos[:, 1:] if d == 1 else np.concatenate([pos, np.full((len(pos), d - 2), 40 * DX)], 1)
        self.pos = pos = np.ascontiguousarray(pos)
        nt, nb = rec.shape
        n_tt = (nt + 31) // 32
        box = np.zeros((n_tt, nb, 2 * d + 1), np.float32)
        for t in range(n_tt):
            r = rec[32 * t:32 * t + 32]
            lam = np.linalg.eigvalsh(_matrix(r["p"], d)).min(-1).min(0)
            box[t, :, :d], box[t, :, d:2 * d] = r["x"].min(0), r["x"].max(0)
            box[t, :, 2 * d] = np.maximum(lam * (1 - 1e-6), 0)
        box[:, open_box, :d], box[:, open_box, d:2 * d], box[:, open_box, 2 * d] = -3.4e38, 3.4e38, 0
        up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(self.dev)
        self.d_rec = up(rec.view(np.uint8))
        self.d_box = up(box)
        # the compact form: one block of 32 records per (tile, beam)
        pool = np.zeros((n_tt, nb, 32), rec.dtype)
        for t in range(n_tt):
            r = rec[32 * t:32 * t + 32]
            pool[t, :, :len(r)] = r.T
        self.d_pool, self.d_slot = up(pool.view(np.uint8)), up(np.arange(n_tt * nb, dtype=np.int32).reshape(n_tt, nb))
        self.ts, self.d_pos = up(np.arange(nt) * 1e-8), up(pos)
        n = (nb + 1) // 2
        self.one = up(np.tile([1.0, 0.0], n))
        self.z = up(np.ones((n, 2 * d)))
        z = self.z.data_ptr()
        self.bs = _lib.BeamSet(n=n, x0=z, p0=z, alpha=z, a0=self.one.data_ptr(), omega=z, modes=0)
        self.pr = _lib.Problem(ndim=d, c=1500.0, nt=nt, ts=self.ts.data_ptr(), ns=len(pos), sensors=self.d_pos.data_ptr())
        for a in range(3):
            self.pr.L[a] = N * DX
        self.opts = _lib.SumOpts(cutoff=cutoff)
        self.nt, self.nb = nt, nb

    def tr(self, compact):
        from beamax_b200 import _lib

        if compact:
            return _lib.Trajectories(nb=self.nb, slot=self.d_slot.data_ptr(), pool=self.d_pool.data_ptr(),
                                     pool_cull=self.d_box.data_ptr(), pool_blocks=self.d_slot.numel())
        return _lib.Trajectories(nb=self.nb, rec32=self.d_rec.data_ptr(), cull=self.d_box.data_ptr())

    def sums(self, compact, data):
        from beamax_b200 import _lib

        L, st = _lib.lib(), torch.cuda.current_stream().cuda_stream
        nbytes = L.msgb_sum_f32_traj_workspace_size(_lib.ref(self.pr), self.nb)
        ws = torch.full((nbytes,), 0x5A, dtype=torch.uint8, device=self.dev)
        y = torch.empty(self.nt, len(self.pos), dtype=torch.float32, device=self.dev)
        g = torch.empty(self.nb, 2, dtype=torch.float64, device=self.dev)
        tr = self.tr(compact)
        _lib.check(L.msgb_sum_fwd_f32_traj(_lib.ref(self.pr), _lib.ref(self.bs), _lib.ref(tr), _lib.ref(self.opts), 1, 1,
                                           ws.data_ptr(), nbytes, y.data_ptr(), st), "forward")
        _lib.check(L.msgb_adj_gather_f32_traj(_lib.ref(self.pr), _lib.ref(self.bs), _lib.ref(tr), _lib.ref(self.opts),
                                              ws.data_ptr(), nbytes, data.data_ptr(), g.data_ptr(), st), "transpose")
        return y.double().cpu().numpy(), torch.view_as_complex(g).cpu().numpy()

    def exact(self, data):
        """The same sums in 64 bits."""
        r = self.rec
        D = self.pos[None, None] - r["x"][:, :, None]  # (nt, nb, ns, d)
        dd = np.stack([D[..., i] * D[..., k] for i, k in PAIRS[self.d]], -1)
        th = (r["wp"][:, :, None] * D).sum(-1) + (r["q"][:, :, None].astype(float) * dd).sum(-1) + r["ang"][:, :, None]
        z = r["amp"][:, :, None] * np.exp(1j * th - (r["p"][:, :, None].astype(float) * dd).sum(-1))
        d = data.cpu().numpy().astype(float)
        return z.real.sum(1), (np.conj(z) * d[:, None]).sum((0, 2))


def _records(nt, nb, d=2, seed=5):
    rng = np.random.default_rng(seed)
    rec = np.zeros((nt, nb), _rec(d))
    rec["x"] = np.array([30.0, 47.0, 40.0][:d]) * DX + DX * rng.random((1, nb, d))
    rec["wp"] = rng.standard_normal((1, nb, d)) * 300
    rec["q"] = rng.standard_normal((1, nb, len(PAIRS[d]))) * 1e4
    _round(rec, slice(None), 2.0)
    rec["ang"], rec["amp"] = rng.random((1, nb)), 2.0
    return rec


def _round(rec, at, efolds):
    """Isotropic Hessians: `efolds` at ten grid steps."""
    for e, (i, k) in enumerate(PAIRS[rec["x"].shape[-1]]):
        rec["p"][at, :, e] = efolds / (10 * DX) ** 2 if i == k else 0.0


def _compare(R, compact):
    data = torch.randn(R.nt, len(R.pos), generator=torch.Generator(device=R.dev).manual_seed(3), device=R.dev)
    y, g = R.sums(compact, data)
    y0, g0 = R.exact(data)
    out = 1.2e-7 * 2 * R.nb
    assert np.linalg.norm(y - y0) <= TOL * np.linalg.norm(y0) + out * y0.size ** 0.5
    assert np.linalg.norm(g - g0) <= TOL * np.linalg.norm(g0) + 2.4e-7 * float(data.norm()) * (R.nb * y0.size) ** 0.5


@pytest.mark.parametrize("compact", [False, True])
@pytest.mark.parametrize("kind,d", [("line", 2), ("run", 2), ("runs", 2), ("short", 2), ("scattered", 2), ("line", 1), ("line", 3)])
def test_records_that_come_near_at_a_few_times_only(kind, d, compact):
    """Narrow beams (exponent 200 at the sensors) that are wide (2) at three of a
    tile's times."""
    rec = _records(40, 70, d)
    _round(rec, slice(None), 200.0)
    for k in (5, 13, 27, 33):
        _round(rec, k, 2.0)
    _compare(_Records(rec, np.zeros(70, bool), _positions(kind)), compact)


@pytest.mark.parametrize("kind,d", [("line", 1), ("line", 2), ("scattered", 2), ("line", 3)])
@pytest.mark.parametrize("nt", [1, 7, 32, 37])
@pytest.mark.parametrize("change", [0.02, 0.3, 3.0])
def test_records_that_change_from_time_to_time(change, nt, kind, d):
    """Centres that walk and Hessians that turn and stretch, by little and by much,
    at distances from within the beams to far beyond the cutoff."""
    rng = np.random.default_rng(int(100 * change) + nt)
    nb = 300
    rec = _records(nt, nb, d)
    rec["x"] = DX * (np.array([0.0, 0.0, 40.0][:d]) + rng.random((1, nb, d)) * [80.0, 200.0, 1e-9][:d])
    rec["x"] = rec["x"] + DX * 8 * change * rng.standard_normal((nt, nb, d)).cumsum(0)
    q, _ = np.linalg.qr(rng.standard_normal((1, nb, d, d)) + change * 0.3 * rng.standard_normal((nt, nb, d, d)).cumsum(0))
    lam = np.exp(rng.normal(0, 1.0, (1, nb, d)) + change * rng.standard_normal((nt, nb, d))) * 4.0 / (10 * DX) ** 2
    M = np.einsum("tbik,tbk,tbjk->tbij", q, lam, q)
    for e, (i, k) in enumerate(PAIRS[d]):
        rec["p"][..., e] = M[..., i, k] * (1 if i == k else 2)
    _compare(_Records(rec, np.zeros(nb, bool), _positions(kind)), True)


@pytest.mark.parametrize("curvature", [0.0, 1e-31, -1e-31, 1e-25])
def test_records_whose_exponent_falls_along_the_run(curvature):
    """An open box, chi = 25 - 1.5 k along a run: 25 at its first sensor, 2.5 at its
    last, with a curvature at the edge of FP32's range or none."""
    rec = _records(40, 70)
    rec["x"][:] = np.array([30.0, 40.0]) * DX
    rec["p"][:] = np.array([25.0 / (10 * DX) ** 2, -1.5 / (10 * DX * DX), curvature])
    _compare(_Records(rec, np.ones(70, bool), _positions("run")), False)


@pytest.mark.parametrize("compact", [False, True])
@pytest.mark.parametrize("kind", ["line", "run", "short", "scattered"])
def test_records_in_an_open_box(kind, compact):
    """An open culling box: growing beams are evaluated everywhere, and a record
    that is not finite reaches the outputs of its time."""
    rec = _records(40, 70)
    grow = {"line": 5e-3, "run": 0.1, "short": 1.2, "scattered": 0.45}[kind]
    off = {"line": 64, "run": 0, "short": 0, "scattered": 7}[kind]
    some = np.arange(70) % 3 == 0
    rec["x"][:, some] = np.array([30.0, 40.0 + off]) * DX
    rec["p"][:, some] = np.array([25.0 / (10 * DX) ** 2, 0.0, -grow / DX ** 2])
    _compare(_Records(rec, some, _positions(kind)), compact)
    rec["x"][35, 3] = np.nan
    R = _Records(rec, some, _positions(kind))
    data = torch.ones(R.nt, len(R.pos), device=R.dev)
    y, g = R.sums(compact, data)
    assert np.isnan(y[35]).all() and np.isfinite(np.delete(y, 35, 0)).all()
    assert np.isnan(g[3]) and np.isfinite(np.delete(g, 3)).all()
