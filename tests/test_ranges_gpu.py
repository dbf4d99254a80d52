"""States and physics outside the ranges of the step kernels' faces (gsw_face.cuh): their values
against the C oracle or another path, bit for bit, in the kernels of the production configuration
(a class table on the dense mesh, the L2 wave speed on the compressed one, the ensemble, the
adjoint), and what they cost, as a ratio of two times of the same kernels on one GPU.

Each bound on a ratio lies between what is measured (no-data beds 1.00 of the ordinary step,
lifted terrain 1.10, the operators alone 1.28 on the dense mesh and 1.41 on the compressed one,
films under the wave speed's floor 1.03) and what evaluating rows twice cost (1.39, 1.83, 1.86,
1.93, 1.86).
"""
import ctypes as C
import functools

import numpy as np
import pytest

import oracle
from tests._cases import pad_state, same
from tests.test_face_gpu import KINDS as _KINDS
from tests.test_face_gpu import extreme_state as _extreme_state

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

NTAB = np.array([0.02, 0.05, 0.09], np.float32)
KINDS = _KINDS + ["vast"]


def extreme_state(kind, nx, ny, seed):
    """As test_face_gpu's; "vast" is its "huge" with depths, beds and momenta eight times larger, which
    are then beyond the limit of the faces (2^17)."""
    if kind != "vast":
        return _extreme_state(kind, nx, ny, seed)
    q0, bed = _extreme_state("huge", nx, ny, seed)
    return q0 * np.float32(8.0), bed * np.float32(8.0)


def _classes(nx, ny, seed):
    return np.pad(np.random.default_rng(seed).integers(0, 3, (nx, ny)).astype(np.uint8), 2, mode="edge")


def _solver(q0, bed, cls=True, **cfg):
    from geoswe_b200 import Config, Mesh2D, Solver2D
    nx, ny = bed.shape
    kw = dict(bc_x="wall", bc_y="wall", friction="manning", arith="portable", h_min=1e-6)
    kw.update(cfg)
    s = Solver2D(Mesh2D(nx=nx, ny=ny, dx=2.0, dy=2.0, ngh=2), Config(**kw), q0, bed)
    if cls:
        s.set_manning_table(_classes(nx, ny, 1), NTAB)
    return s


def _oracle(q0, bed, **kw):
    nx, ny = bed.shape
    qp, bp = pad_state(q0, bed, 2, np.float32)
    return oracle.OracleSolver2D(qp, bp, 2, 2.0, 2.0, kinds=["wall"] * 4, friction="manning",
                                 ncls=_classes(nx, ny, 1), ntab=NTAB, **kw)


def _same_runs(q0, bed, steps=4, **phys):
    """Device-loop runs of the dense solver and the oracle."""
    s, o = _solver(q0, bed, **phys), _oracle(q0, bed, **phys)
    assert s.run(1e9, max_steps=steps) == o.run(1e9, max_steps=steps) == steps
    assert s.t == o.t
    assert same(s.q_interior.cpu().numpy(), o.q[:, 2:-2, 2:-2])


# ------------------------------------------------------------------- the production kernels
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("g,h_min", [(9.81, 1e-6), (981.0, 1e-6), (9.81, 1e-8)])
def test_extreme_states_with_a_class_table(kind, g, h_min):
    q0, bed = extreme_state(kind, 61, 64, seed=7)
    _same_runs(q0, bed, g=g, h_min=h_min)


def _compressed(q0, bed, fs=None, **cfg):
    from geoswe_b200.compressed import CompressedSolver
    nx, ny = bed.shape
    s = _solver(q0, bed, bc_x="fall", bc_y="fall", **cfg)
    mask = np.zeros((nx, ny), bool)
    mask[3:-3, 3:-3] = True
    mask[20:30, 20:40] = False
    s.set_inside_mask(mask)
    return CompressedSolver.from_dense(s, **(fs or {}))


def _flat_oracle(cs):
    q = [cs.flat(c).cpu().numpy() for c in range(3)]
    o = oracle.OracleFlat(cs.nbr, cs.is_active, q, cs._b[cs._slot].cpu().numpy(), cs.dx, g=cs.g,
                          ncls=cs._ncls[cs._slot].cpu().numpy(), ntab=NTAB, linf=cs.cfl_linf)
    o.h_min, o.h_min_cfl = cs.h_min, cs.h_min_cfl
    return o


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("fs", [{}, dict(g=981.0), dict(h_min=1e-8), dict(h_min=1e-7)],
                         ids=["earth", "g981", "h_min1e-8", "h_min1e-7"])
def test_extreme_states_on_the_compressed_mesh_with_the_l2_speed(kind, fs):
    """h_min 1e-7 leaves films under the wave speed's floor h_min_cfl (1e-6)."""
    q0, bed = extreme_state(kind, 61, 67, seed=9)
    cs = _compressed(q0, bed, fs)
    o = _flat_oracle(cs)
    assert cs.run(1e9, max_steps=4) == o.run(1e9, max_steps=4) == 4
    assert cs.t == o.t
    for c in range(3):
        assert same(cs.flat(c).cpu().numpy(), o.q[c]), c


@pytest.mark.parametrize("h_min,h_min_cfl", [(1e-6, 1e-3), (1e-6, 2.0), (1e-3, 1e-6)])
def test_wave_speed_floor_of_the_dense_step(h_min, h_min_cfl):
    q0, bed = extreme_state("film", 61, 64, seed=2)
    s, o = _solver(q0, bed, h_min=h_min, h_min_cfl=h_min_cfl), _oracle(q0, bed, h_min=h_min, h_cfl=h_min_cfl)
    assert s.run(1e9, max_steps=4) == o.run(1e9, max_steps=4)
    assert s.t == o.t and same(s.q_interior.cpu().numpy(), o.q[:, 2:-2, 2:-2])


@pytest.mark.parametrize("arith", ["portable", "exact"])
def test_extreme_members_equal_their_own_runs(arith):
    """Every kind of state, gravity and depth floor in one ensemble."""
    from geoswe_b200.ensemble import Ensemble
    specs = [(k, fs) for k in KINDS for fs in ({}, dict(g=981.0), dict(h_min=1e-7))]

    def member(k, i):
        return _compressed(*extreme_state(specs[k][0], 61, 67, seed=20 + i), specs[k][1], arith=arith)

    alone = [member(k, k) for k in range(len(specs))]
    ens = Ensemble([member(k, k) for k in range(len(specs))])
    assert ens.lean
    n = [cs.run(1e9, max_steps=5) for cs in alone]
    assert ens.run(1e9, max_steps=5) == n
    for k, cs in enumerate(alone):
        assert ens.members[k].t == cs.t, specs[k]
        for c in range(3):
            assert same(ens.flat(k, c).cpu().numpy(), cs.flat(c).cpu().numpy()), (specs[k], c)


@pytest.mark.parametrize("kind", ["huge", "vast", "still", "moving", "nodata"])
def test_adjoint_rows_equal_the_operators(kind):
    """The reverse step's recomputed rows against the operators: with gravity times 2^8, speeds
    times 2^4 and times over 2^4, every operation of the step scales by a power of two, so depths
    and their adjoints are the same bits and the momenta's scale, but gravity is then outside
    the faces' range and every row goes through the operators."""
    from geoswe_b200.adjoint import FlatAdjoint
    N, out, dts = 3, [], None
    for up in (1.0, 16.0):
        q0, bed = extreme_state(kind if kind in ("huge", "vast") else "still", 61, 67, seed=4)
        if kind == "moving":
            q0[1:] = q0[0] * np.random.default_rng(6).standard_normal(q0[1:].shape).astype(np.float32)
        if kind == "nodata":
            bed[:, 30:50] = 1.0e6
            q0[:, :, 26:54] = 0.0
        q0[1:] *= np.float32(up)
        cs = _compressed(q0, bed, dict(g=9.81 * up * up))
        cs.vcap = 1.0e12                              # the limiter's 1e-10 does not scale
        act = np.nonzero(cs.is_active != 0)[0]
        adj = FlatAdjoint(cs, gauges=act[::97], n_steps=N, window=N, snapshots=2, rain_times=np.array([0.0]),
                          rain_base=np.array([1e-5 * up]))
        adj.set_params(NTAB / up, 1.0)
        adj.forward()
        if dts is None:
            dts = adj.dt_tab.clone()
        adj.dt_tab.copy_(dts / up)                    # the rule's 1e-12 does not scale either
        adj._t_tab = np.concatenate([[0.0], np.cumsum(dts[:N].cpu().numpy() / up)])
        adj._build_state_table()
        series = adj.forward(replay=True).cpu().numpy()
        gn, gs, _ = adj.gradients(np.zeros_like(series) + 0.1)
        lam = [adj.adjoint_state(c)[cs._slot].cpu().numpy() * np.float32(1.0 if c == 0 else up) for c in range(3)]
        lam = [np.where(np.abs(x) < 2.0 ** -100, np.float32(0.0), x) for x in lam]
        out.append((series, gn.cpu().numpy() / up, gs, lam))
    (s0, n0, r0, l0), (s1, n1, r1, l1) = out
    assert same(s0, s1)
    assert np.abs(l0[0]).max() > 0
    for c in range(3):
        assert same(l0[c], l1[c]), c
    # sums over atomics in any order: binary64 rounding of at most 61 * 67 * 3 terms each
    assert np.abs(n0 - n1).max() <= 1e-12 * np.abs(n0).max() + 1e-300
    assert abs(r0 - r1) <= 1e-12 * abs(r0)


# ---------------------------------------------------------------------------- no-data beds
def _beds(value, seed=3, rim=True):
    """A flowing state whose right half is dry, behind dry ground four cells wide or a ragged
    shore, on beds of `value`."""
    q0, bed = extreme_state("plain", 90, 128, seed=seed)
    hit = np.zeros(bed.shape, bool)
    hit[:, 70:] = True
    if not rim:
        hit |= np.random.default_rng(seed).random(bed.shape) < 0.05
    q0[:, hit] = 0.0
    if rim:
        q0[:, :, 66:] = 0.0
        bed[:, 66:] = 50.0
    bed[hit] = value
    return q0, bed


@pytest.mark.parametrize("value", [99999.0, 1.0e6, -32768.0, 3.4e38])
@pytest.mark.parametrize("rim", [True, False])
def test_no_data_beds_match_oracle(value, rim):
    if not rim and value > 1e30:
        pytest.skip("water beside such a bed overflows")
    _same_runs(*_beds(value, rim=rim))


@pytest.mark.parametrize("arith", ["portable", "exact", "fast"])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_non_finite_beds_under_dry_ground(arith, value):
    """Beds that the solver refuses and a caller of the C entry points may hold: two dry cells
    exchange nothing whatever their beds, so the run is that of an ordinary high bed."""
    q0, bed = _beds(50.0)
    a, b = _solver(q0, bed, arith=arith), _solver(q0, bed, arith=arith)
    b._b[:, 72:] = value
    assert a.run(1e9, max_steps=6) == b.run(1e9, max_steps=6) == 6
    assert a.t == b.t
    assert torch.equal(a.q, b.q) and bool(torch.isfinite(b.q).all())
    assert torch.equal(a.residual(), b.residual())


# ----------------------------------------------------------------------------- what it costs
@functools.lru_cache(maxsize=None)
def _ground(nx=1536, ny=1500):
    g = torch.Generator(device="cuda").manual_seed(1)
    z = torch.zeros((nx, ny), device="cuda")
    n, amp = 4, 12.0
    while n <= 1024:
        c = torch.randn((1, 1, n, n), generator=g, device="cuda")
        z += amp * torch.nn.functional.interpolate(c, (nx, ny), mode="bilinear", align_corners=True)[0, 0]
        n, amp = 2 * n, amp / 2
    z -= z.min()
    level = z.reshape(-1)[::97].quantile(0.3)
    film = 0.003 * torch.rand((nx, ny), generator=g, device="cuda")
    h = torch.where(z < level, level - z, torch.where(film > 0.001, film, torch.zeros_like(film)))
    u = 0.3 * torch.randn((2, nx, ny), generator=g, device="cuda")
    cls = torch.randint(0, 3, (nx + 4, ny + 4), generator=g, device="cuda", dtype=torch.uint8)
    return torch.stack([h, h * u[0], h * u[1]]), z, cls


def _step_us(s, steps=16):
    s.run(1e12, max_steps=steps)
    best = 1e30
    for _ in range(5):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        e[0].record()
        s.run(1e12, max_steps=steps)
        e[1].record()
        torch.cuda.synchronize()
        best = min(best, e[0].elapsed_time(e[1]))
    return best * 1e3 / steps


def _cost(flat=False, fs=None, change=None, **cfg):
    from geoswe_b200.compressed import CompressedSolver
    q, z, cls = _ground()
    if change is not None:
        q, z = change(q.clone(), z.clone())
    s = _solver(q, z, cls=False, arith="exact", **dict(dict(bc_x="fall", bc_y="fall"), **cfg))
    s.set_manning_table(cls, NTAB)
    if flat:
        m = np.zeros(tuple(z.shape), bool)
        m[3:-3, 3:-3] = True
        s.set_inside_mask(m)
        s = CompressedSolver.from_dense(s, **(fs or {}))
    return _step_us(s)


def _costs_at_most(bound, changed, usual):
    """Whether the time of `changed` is under `bound` of that of `usual`, in one of a few tries: the
    host is shared and holds a launch up now and then."""
    return any(_cost(**changed) < bound * _cost(**usual) for _ in range(4))


def test_no_data_beds_cost_nothing_on_dry_rows():
    def half(value):
        def change(q, z):
            q[:, :, 746:] = 0.0
            z[:, 746:] = 60.0
            z[:, 750:] = value
            return q, z
        return change
    usual = dict(change=half(60.0))
    assert _costs_at_most(1.15, dict(change=half(3.4e38)), usual)
    assert _costs_at_most(1.15, dict(change=half(-3.4e38)), usual)


def test_lifted_terrain_costs_no_second_evaluation():
    assert _costs_at_most(1.3, dict(change=lambda q, z: (q, z + 20000.0)), {})


@pytest.mark.parametrize("cfg", [dict(g=981.0), dict(h_min=1e-8), dict(h_min_cfl=2.0)])
def test_physics_outside_the_ranges_costs_the_operators(cfg):
    assert _costs_at_most(1.5, cfg, {})


@pytest.mark.parametrize("fs,bound", [(dict(g=981.0), 1.6), (dict(h_min=1e-8), 1.6), (dict(h_min=1e-7), 1.2)])
def test_compressed_physics_outside_the_ranges_costs_the_operators(fs, bound):
    assert _costs_at_most(bound, dict(flat=True, fs=fs), dict(flat=True))


def test_wave_speed_of_a_narrow_grid():
    """The standalone wave speed of a grid a few cells wide keeps its warps busy: its cells take
    at most eight times as long as those of a wide grid (24 of 32 lanes have no cell)."""
    from geoswe_b200 import _lib as L
    from geoswe_b200.solver import _stream
    times = []
    for nx, ny in ((1 << 20, 8), (2896, 2896)):
        q0 = torch.rand((3, nx, ny), device="cuda") + 0.1
        s = _solver(q0, torch.zeros((nx, ny), device="cuda"), cls=False)
        a = s._dense_args(s._buf[0], s._buf[1], s._tables())
        bits = torch.zeros(1, dtype=torch.int64, device="cuda")
        best = 1e30
        for _ in range(6):
            bits.zero_()
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            L.call("gsw_dense_lammax", C.byref(a), C.c_void_p(bits.data_ptr()), _stream())
            e[1].record()
            torch.cuda.synchronize()
            best = min(best, e[0].elapsed_time(e[1]))
        h, hu, hv = s.q_interior
        want = torch.maximum((hu / h).abs(), (hv / h).abs()) + (9.81 * h).sqrt()
        got = bits.view(torch.float64).item()
        assert abs(got - float(want.max())) <= 4e-7 * got      # two roundings more or less
        times.append(best)
        del s, q0
    assert times[0] < 8.0 * times[1]


@pytest.mark.parametrize("nx,ny", [(7, 1), (70, 31), (70, 33), (130, 65), (9, 129), (33, 257), (40, 700)])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_wave_speed_matches_oracle(nx, ny, dtype):
    """Widths on both sides of each split of a block's warps between columns and rows."""
    from geoswe_b200 import Config, Mesh2D, Solver2D
    rng = np.random.default_rng(nx * ny)
    q0 = np.stack([rng.random((nx, ny)), *rng.standard_normal((2, nx, ny))]).astype(dtype)
    for at in ((0, 0), (nx - 1, ny - 1), (nx - 1, 0), (nx // 2, ny // 2)):
        q = q0.copy()
        q[1][at] = 900.0 * q[0][at]
        s = Solver2D(Mesh2D(nx=nx, ny=ny, dx=2.0, dy=2.0, ngh=2), Config(dtype=dtype, h_min=1e-6, h_min_cfl=1e-6), q,
                     np.zeros((nx, ny)))
        o = oracle.OracleSolver2D(*pad_state(q, np.zeros((nx, ny)), 2, np.dtype(dtype)), 2, 2.0, 2.0, h_min=1e-6)
        assert s.cfl_dt() == o.cfl_dt()


def test_ghost_fill_of_a_deep_halo():
    """More ghost layers than a launch has rows of blocks (13 GB)."""
    from geoswe_b200 import _lib as L
    from geoswe_b200.solver import _ptr, _stream
    n, ngh = 5, 16390
    free, _ = torch.cuda.mem_get_info()
    w = n + 2 * ngh
    if free < 5 * 4 * w * w:
        pytest.skip("needs 21 GB of free device memory")
    inner = torch.rand((n, n), device="cuda")
    a = L.GswBcArgs()
    a.abi_version, a.dtype, a.nxp, a.nyp, a.ngh, a.pitch = L.ABI_VERSION, L.F32, w, w, ngh, w
    q = [torch.zeros((w, w), device="cuda") for _ in range(3)]
    for x in q:
        x[ngh:-ngh, ngh:-ngh] = inner
    a.q0, a.q1, a.q2 = (_ptr(x) for x in q)
    for f in range(4):
        a.kinds[f] = L.BC_EXTRAPOLATE
    L.call("gsw_bc_fill", C.byref(a), _stream())
    rows = torch.arange(w, device="cuda").sub(ngh).clamp(0, n - 1)
    for lo in range(0, w, 4096):
        r = rows[lo:lo + 4096]
        want = inner[r][:, rows]
        for x in q:
            assert torch.equal(x[lo:lo + 4096], want), lo
