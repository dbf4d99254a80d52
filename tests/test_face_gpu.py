"""The binary32 faces and update without the IEEE operators (gsw_face.cuh).

Their roots and quotients are compared with the operators over the ranges they are used in;
states outside those ranges (non-finite values, tiny and subnormal momenta and depths, beds
and depths above 2^17, depth floors and gravity outside face_ranges) with the C oracle, bit for
bit, since they take the scalar operators instead. The portable arithmetic: a CPU cannot
reproduce CUDA's powf.
"""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

import oracle
from tests._cases import pad_state, same

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
HERE = Path(__file__).resolve().parent


def test_roots_and_quotients_are_correctly_rounded(tmp_path):
    from geoswe_b200 import build as B
    nvcc = B._nvcc()
    if shutil.which(nvcc) is None:
        pytest.skip("no nvcc")
    exe = tmp_path / "face_check"
    subprocess.run([nvcc, *B.ARCH, "-O3", "-std=c++17", *B.EXACT, "--expt-relaxed-constexpr", "-I", str(B.INCLUDE),
                    str(HERE / "native" / "face_check.cu"), str(B.CSRC / "gsw_loop.cu"), "-o", str(exe)], check=True)
    root, recip, hard, rand, tested = map(int, subprocess.run([str(exe)], check=True, capture_output=True,
                                                              text=True, timeout=120).stdout.split())
    assert tested > 10_000_000
    assert (root, recip, hard, rand) == (0, 0, 0, 0)


def extreme_state(kind, nx, ny, seed):
    """A flowing state with a tenth of its cells pushed to one kind of extreme."""
    rng = np.random.default_rng(seed)
    bed = (rng.random((nx, ny)) * 0.5).astype(np.float32)
    if kind == "flat":
        bed[:] = 0.0
    h = np.where(rng.random((nx, ny)) < 0.2, 0.0, rng.random((nx, ny))).astype(np.float32)
    u, v = rng.standard_normal((2, nx, ny))
    q = np.stack([h, h * u, h * v]).astype(np.float32)
    hit = rng.random((nx, ny)) < 0.1
    tiny = np.ldexp(rng.uniform(1.0, 2.0, (3, nx, ny)), rng.integers(-149, -60, (3, nx, ny))).astype(np.float32)
    sign = np.where(rng.random((2, nx, ny)) < 0.5, 1.0, -1.0).astype(np.float32)
    if kind in ("momentum", "flat"):
        q[1:] = np.where(hit, tiny[1:] * sign, q[1:])
    if kind in ("depth", "flat"):
        q[0] = np.where(rng.random((nx, ny)) < 0.1, tiny[0], q[0])
    if kind == "film":                                     # around the depth floor
        q[0] = np.where(hit, 1e-6 * rng.uniform(0.5, 1.5, (nx, ny)), q[0]).astype(np.float32)
        q[1:] = np.where(hit, q[0] * sign, q[1:])
    if kind == "bed":
        bed = np.where(hit, tiny[0], bed).astype(np.float32)
    if kind == "huge":
        q[0] = np.where(hit, 5.0e4, q[0])
        bed = np.where(rng.random((nx, ny)) < 0.05, 3.0e4, bed).astype(np.float32)
        q[1] = np.where(hit, q[0] * 3.0e4, q[1])
    if kind == "still":
        q[1:] = 0.0
        q[0] = np.maximum(np.float32(0.75) - bed, 0.0)
    return q.astype(np.float32), bed


KINDS = ["momentum", "depth", "flat", "film", "bed", "huge", "still"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("g,h_min", [(9.81, 1e-6), (0.5, 1e-6), (9.81, 1e-9)])
def test_extreme_states_match_oracle(kind, g, h_min):
    from geoswe_b200 import Config, Mesh2D, Solver2D
    nx, ny, ngh = 61, 64, 2
    q0, bed = extreme_state(kind, nx, ny, seed=3)
    cfg = dict(bc_x="wall", bc_y="wall", h_min=h_min, h_min_cfl=max(h_min, 1e-6), g=g, arith="portable")
    qp, bp = pad_state(q0, bed, ngh, np.float32)
    filled = qp.copy()
    oracle.bc_fill(filled, ngh, ["wall"] * 4)
    want = oracle.dense_rhs(filled, bp, 2.0, 2.0, g, h_min)
    mesh = Mesh2D(nx=nx, ny=ny, dx=2.0, dy=2.0, ngh=ngh)
    s = Solver2D(mesh, Config(**cfg), q0, bed)
    s.apply_bc()
    got = s.residual().cpu().numpy()
    for k in range(3):
        assert same(got[k], want[k]), f"residual {k}"
    for friction, n in ((None, 0.0), ("manning", 0.03)):
        s = Solver2D(mesh, Config(friction=friction, manning_n=n, **cfg), q0, bed)
        o = oracle.OracleSolver2D(qp, bp, ngh, 2.0, 2.0, g=g, h_min=h_min, h_cfl=max(h_min, 1e-6), kinds=["wall"] * 4,
                                  friction=friction, manning_n=n)
        for _ in range(3):
            dt = o.cfl_dt()
            assert s.cfl_dt() == dt
            s.step(dt)
            o.step(dt)
        inner = (slice(None), slice(ngh, -ngh), slice(ngh, -ngh))
        assert same(s.q.cpu().numpy()[inner], o.q[inner]), friction


@pytest.mark.parametrize("kind", KINDS)
def test_extreme_states_on_the_compressed_mesh(kind):
    """Compressed and dense residuals and steps are the same bits, extremes included."""
    from geoswe_b200 import Config, Mesh2D, Solver2D
    from geoswe_b200.compressed import CompressedSolver
    nx, ny = 61, 67
    q0, bed = extreme_state(kind, nx, ny, seed=5)
    mask = np.zeros((nx, ny), bool)
    mask[3:-3, 3:-3] = True
    mask[20:30, 20:40] = False
    s = Solver2D(Mesh2D(nx=nx, ny=ny, dx=2.0, dy=2.0, ngh=2), Config(bc_x="fall", bc_y="fall", friction="manning",
                                                                   manning_n=0.03), q0, bed)
    s.set_inside_mask(mask)
    cs = CompressedSolver.from_dense(s, cfl_linf=True)
    act = cs.is_active != 0
    ij = cs.ij_active[act]
    r = s.residual().cpu().numpy()
    f = cs.residual().cpu().numpy()
    for k in range(3):
        assert same(f[k][act], r[k][ij[:, 0], ij[:, 1]]), f"residual {k}"
    s.run(1e9, max_steps=1)
    cs.run(1e9, max_steps=1, dt_max=s.last_dt)
    assert cs.last_dt == s.last_dt
    for k in range(3):
        assert same(cs.flat(k).cpu().numpy()[act], s.q[k].cpu().numpy()[ij[:, 0], ij[:, 1]]), f"field {k}"


def test_non_finite_state_is_reported():
    from geoswe_b200 import Config, Mesh2D, Solver2D
    q0, bed = extreme_state("still", 40, 70, seed=1)
    for arith in ("exact", "fast"):
        for field in range(3):
            s = Solver2D(Mesh2D(nx=40, ny=70, dx=2.0, dy=2.0, ngh=2), Config(arith=arith, friction="manning",
                                                                           manning_n=0.03), q0, bed)
            s.run(1e9, max_steps=2)
            s.q[field, 20, 30] = float("nan")
            with pytest.raises(FloatingPointError):
                s.run(1e9, max_steps=3)


@pytest.mark.parametrize("nx,ny,ngh", [(5, 7, 2), (40, 300, 4), (2100, 2050, 2)])
@pytest.mark.parametrize("kinds", [("wall", "fall"), ("periodic", "extrapolate")])
def test_device_loop_equals_single_steps(nx, ny, ngh, kinds):
    """Runs of one and of several steps against the host's single steps, ghost cells included,
    on grids of a few cells and of several blocks per ghost row."""
    from geoswe_b200 import Config, Mesh2D, Solver2D
    q0, bed = extreme_state("film", nx, ny, seed=nx)
    mesh = Mesh2D(nx=nx, ny=ny, dx=2.0, dy=2.0, ngh=ngh)
    cfg = dict(bc_x=kinds[0], bc_y=kinds[1], friction="manning", manning_n=0.03)
    s, o = (Solver2D(mesh, Config(**cfg), q0, bed, use_graphs=g) for g in (True, False))
    for steps in (1, 3, 4):
        assert s.run(1e9, max_steps=steps) == steps
        for _ in range(steps):
            o.step()
        assert s.t == o.t and s.last_dt == o.last_dt
        assert torch.equal(s.q, o.q)
