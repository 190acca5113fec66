"""Every chain of kernels that are placed while their predecessor ends, against
the same calls with each launch drained before the next (a process of its own
under CUDA_LAUNCH_BLOCKING): equal to the bit, or a kernel read or wrote too
early.  All sums are of a fixed order, so no tolerance is needed."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

from rapidfem_b200 import _native
from rapidfem_b200 import gpu as G
from rapidfem_b200 import operator as O

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ENGINES = {"tf32x3": _native.ENGINE_TF32X3, "fp32": _native.ENGINE_FP32,
           "fp32_small_tiles": _native.ENGINE_FP32_SMALL_TILES}
# a tile and a bit, tiles on part of the SMs, several tiles on each
MESHES = {"few": (2, 2, 1), "some": (5, 5, 4), "many": (13, 12, 11)}


def _f32_chains(gop, out, key, h):
    n = gop.n_dof()
    rng = np.random.default_rng(n)
    y, b = rng.standard_normal((2, n))
    g = rng.standard_normal(8)
    fun = [(rng.integers(0, n, 40), rng.standard_normal(40)), ([n - 1], [1.0])]
    probes = rng.integers(0, n, 37)
    out[key + "apply"] = gop.apply(y)
    series, yf = gop.transient_probes(y, 2 * h, 4, substeps=2, drive=("point", n // 3), g=g, probes=probes)
    out[key + "probes"], out[key + "probes_y"] = series, yf
    series, yf = gop.transient_functionals(y, 2 * h, 4, substeps=2, drive=("vector", b), g=g, functionals=fun)
    out[key + "functionals"], out[key + "functionals_y"] = series, yf
    # accepted, rejected (the first try is far too long) and surplus attempts
    traj, st = gop.transient_kcl(y, 6 * h, 3, drive=("vector", b), g=g[:3])
    out[key + "kcl"], out[key + "kcl_stats"] = traj, np.array(list(st.values()), dtype=np.float64)
    series, yf, _ = gop.transient_kcl_functionals(y, 6 * h, 3, drive=("point", 1), g=g[:3], functionals=fun)
    out[key + "kcl_functionals"], out[key + "kcl_functionals_y"] = series, yf
    _krylov(gop, out, key, y, b, h)


def _krylov(gop, out, key, y, b, h):
    out[key + "expmv"], dim = gop.expmv(y, 3 * h, 9)
    out[key + "expmv_dim"] = np.array(dim)
    # several chunks, steps past convergence skipped, a source
    out[key + "etd"], dim = gop.etd_step(y, b, 8 * h, 24, 1e-3)
    out[key + "etd_dim"] = np.array(dim)
    out[key + "poly"], dim, est = gop.etd_step_poly(y, b, [1.0, -0.5, 0.25], 2 * h, 12, 1e-2)
    out[key + "poly_est"] = np.array([dim, est])


def _f64_chains(gop, out, key, h):
    n = gop.n_dof()
    rng = np.random.default_rng(n)
    y, b = rng.standard_normal((2, n))
    g = rng.standard_normal(8)
    out[key + "apply64"] = gop.apply_f64(y)
    out[key + "free64"] = gop.transient_f64(y, 2 * h, 4, substeps=2)
    out[key + "driven64"] = gop.transient_f64(y, 2 * h, 4, substeps=2, drive=("vector", b), g=g, record=True)
    gop.set_krylov_precision(64)
    _krylov(gop, out, key + "k64_", y, b, h)
    gop.set_krylov_precision(32)


def _chains(order, mesh):
    cells = MESHES[mesh]
    ctx = G.GpuContext(0)
    m = O.structured_box_jittered(*cells, 1.0, 1.0, 1.0, 0.1, 5)
    gop = G.GpuOperator(ctx, O.MaxwellOperator(m, order, 1.0))
    h = 0.05 / (max(cells) * order * order)
    out = {}
    for name, engine in ENGINES.items():
        gop.set_engine(engine)
        _f32_chains(gop, out, name + "_", h)
    _f64_chains(gop, out, "", h)
    return out


def main(path):
    """The child: every chain of every case, drained, into an .npz."""
    import torch
    rt = ctypes.CDLL("libcudart.so.12")
    stream = torch.cuda.Stream()
    ctx = G.GpuContext(0)
    ctx.set_stream(stream.cuda_stream)
    gop = G.GpuOperator(ctx, O.MaxwellOperator(O.structured_box(8, 8, 8), 3, 1.0))
    gop.run_lserk(1e-3, 20)
    assert rt.cudaStreamQuery(ctypes.c_void_p(stream.cuda_stream)) == 0  # the launches are drained
    ctx.set_stream(None)
    np.savez(path, **{f"{order}/{mesh}/{k}": v for order in range(1, 6) for mesh in MESHES
                      for k, v in _chains(order, mesh).items()})


@pytest.fixture(scope="module")
def drained(tmp_path_factory):
    path = str(tmp_path_factory.mktemp("chains") / "drained.npz")
    env = dict(os.environ, CUDA_LAUNCH_BLOCKING="1")
    r = subprocess.run([sys.executable, "-c", f"from tests.test_gpu_overlap_chains import main; main({path!r})"],
                       cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return np.load(path)


@pytest.mark.parametrize("order", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("mesh", list(MESHES))
def test_chains_equal_their_drained_form(drained, order, mesh):
    for _ in range(2):
        for k, v in _chains(order, mesh).items():
            assert np.array_equal(v, drained[f"{order}/{mesh}/{k}"], equal_nan=True), k
