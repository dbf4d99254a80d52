"""The step kernels of storage beyond 32-bit indices: 64-bit slots on the compressed mesh and in
the ensemble, the operators on dense rows too long for 32-bit offsets, and tiles cut to fit them.

Meshes of that size (2^31 slots take over 80 GB) are not built here: the library is compiled once
more with GSW_INDEX32_MAX = 900, which sends small meshes the same way, and every result
has to be the usual library's bit for bit.
"""
import hashlib
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

import numpy as np
import pytest

from tests._cases import flowing

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

ROOT = Path(__file__).resolve().parents[1]


def _mask(nx, ny):
    m = np.zeros((nx, ny), bool)
    m[3:-3, 3:-3] = True
    m[20:30, 20:40] = False
    return m


def _dense(nx, ny, cls=True, bc="wall", **cfg):
    from geoswe_b200 import Config, Mesh2D, Solver2D
    q0, bed = flowing(nx, ny, seed=nx + ny)
    s = Solver2D(Mesh2D(nx=nx, ny=ny, dx=2.0, dy=2.0, ngh=2),
                 Config(bc_x=bc, bc_y=bc, friction="manning", manning_n=0.03, h_min=1e-6, **cfg), q0, bed)
    if cls:
        s.set_manning_table(np.random.default_rng(1).integers(0, 3, s.mesh.padded_shape).astype(np.uint8),
                            [0.02, 0.04, 0.08])
    return s


def _digest(*parts):
    h = hashlib.sha256()
    for p in parts:
        h.update((p + 0.0).cpu().numpy().tobytes() if torch.is_tensor(p) else repr(p).encode())
    return h.hexdigest()


def results():
    """Name and digest of every run."""
    from geoswe_b200.compressed import CompressedSolver
    from geoswe_b200.ensemble import Ensemble
    for ny in (70, 300):                 # rows of 72 cells (tiles cut to eight rows) and of over 225
        # (the fast arithmetic's operators round otherwise than its faces: only rows of the faces)
        for arith in ("exact", "portable", "fast") if ny < 225 else ("exact", "portable"):
            for cls in (True, False):
                s = _dense(61, ny, cls, arith=arith)
                s._tile_rows = 32
                s.run(1e9, max_steps=5)
                s.apply_bc()
                yield f"dense {ny} {arith} {cls}", _digest(s.q, s.residual(), s.t)
        s = _dense(61, ny, h_min_cfl=1e-3, rainfall=1e-5)
        s.set_inside_mask(_mask(61, ny))
        s.run(1e9, max_steps=5)
        yield f"masked {ny}", _digest(s.q, s.t)

    def flat(nx, ny, arith="exact", **fs):
        s = _dense(nx, ny, bc="fall", arith=arith)
        s.set_inside_mask(_mask(nx, ny))
        return CompressedSolver.from_dense(s, **fs)

    for arith in ("exact", "portable", "fast"):
        for fs in ({}, dict(cfl_linf=True), dict(h_min=1e-7), dict(g=981.0)):
            for cap in (0, 3, 4, 5):
                cs = flat(61, 97, arith, **fs)
                cs.min_blocks = cap
                cs.run(1e9, max_steps=5)
                yield f"flat {arith} {fs} {cap}", _digest(*(cs.flat(c) for c in range(3)), cs.residual(), cs.t)
        for linf in (False, True):
            for cap in (0, 3, 4, 5):
                ens = Ensemble([flat(61, 97, arith, cfl_linf=linf), flat(40, 150, arith, cfl_linf=linf)])
                ens.min_blocks = cap
                ens.run(1e9, max_steps=5)
                yield f"ensemble {arith} {linf} {cap}", _digest(*(ens.flat(k, c) for k in range(2) for c in range(3)))


def _build(out):
    from geoswe_b200 import build as B
    nvcc = B._nvcc()

    def one(src):
        obj = out / (src.stem + ".o")
        if src.suffix == ".cpp":
            cmd = [nvcc, "-x", "c++", "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden"]
        else:
            cmd = [nvcc, *B.ARCH, *(B.FAST_FLAGS if src.name in B.FAST_SOURCES else B.NVCC_FLAGS),
                   "-DGSW_INDEX32_MAX=900"]
        subprocess.run([*cmd, "-I", str(B.INCLUDE), "-c", str(src), "-o", str(obj)], check=True)
        return str(obj)

    with ThreadPoolExecutor(8) as ex:
        objs = list(ex.map(one, B.sources()))
    lib = out / "libgsw_index64.so"
    subprocess.run([nvcc, *B.ARCH, "-shared", "-o", str(lib), *objs, "-lcudart"], check=True)
    return lib


def test_kernels_beyond_32_bit_indices(tmp_path):
    lib = _build(tmp_path)
    run = subprocess.run([sys.executable, "-c", "import sys; from pathlib import Path\n"
                          "from geoswe_b200 import _lib\n"
                          f"_lib.LIB_PATH = Path({str(lib)!r})\n"
                          "from tests.test_index64_gpu import results\n"
                          "for name, digest in results(): print(name, digest, sep='|')"],
                         cwd=ROOT, check=True, capture_output=True, text=True, timeout=300)
    wide = dict(line.rsplit("|", 1) for line in run.stdout.splitlines() if "|" in line)
    usual = dict(results())
    assert wide.keys() == usual.keys() and len(usual) > 60
    assert [k for k in usual if wide[k] != usual[k]] == []
