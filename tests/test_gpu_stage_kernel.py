"""The tensor-core stage kernel's tile edges: the flux units (groups of two face
nodes, four at order 4, whose last group may be partly padding), every face kind
in one tile, rough fields, tiles of which one element or all but one are real.

Tolerance: a right-hand side is a sum of at most 3 Np + 4 Nfp (252) f32-class
products; with random signs its relative error is about sqrt(252) 2^-24 times
the cancellation of the sum (5 to 10 on rough fields), i.e. 1e-6 x 2 to 5;
5e-6 is asked.
"""
import numpy as np
import pytest

from oracle import oracle as R
from rapidfem_b200 import _native
from rapidfem_b200 import gpu as G
from rapidfem_b200 import operator as O

from .conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return G.GpuContext(0)


def _mixed_box(n_tets):
    """A jittered box cut to its first n_tets elements (the cut faces are PEC
    walls) with an absorbing end and a severed pair of faces."""
    m = O.structured_box_jittered(5, 4, 3, 1.0, 0.8, 0.7, 0.1, 9)
    m = O.Mesh(m.nodes, np.ascontiguousarray(m.tets[:n_tets]))
    port = np.where(O.boundary_faces_on_plane(m, 2, 0.0), 0, -1)
    rng = np.random.default_rng(n_tets)
    K = m.n_tets
    mat = O.isotropic_materials(rng.uniform(1, 4, K), rng.uniform(1, 2, K), rng.uniform(0, 2, K), rng.uniform(0, 1, K))
    return m, port, mat


@pytest.mark.parametrize("order", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("n_tets", [1, 8, 9, 20, 21, 39, 161, 360])
@pytest.mark.parametrize("alpha", [1.0, 0.0, 0.3])
def test_rhs_of_rough_fields_at_tile_edges(ctx, order, n_tets, alpha):
    m, port, mat = _mixed_box(n_tets)
    prod = O.MaxwellOperator(m, order, alpha, face_port=port, materials=mat)
    orc = R.Operator(m.nodes, m.tets, order, alpha, face_port=port, materials=mat)
    gop = G.GpuOperator(ctx, prod)
    gop.set_engine(_native.ENGINE_TF32X3)
    y = np.random.default_rng(order).standard_normal(gop.n_dof()).astype(np.float32)
    assert rel_l2(gop.apply(y), orc.apply(y.astype(np.float64))) < 5e-6


@pytest.mark.parametrize("order", [1, 2, 3, 4, 5])
def test_a_nonfinite_element_stays_local(ctx, order):
    """One RHS spreads a NaN to the element's face neighbours and no further
    (the operand padding must not carry it to other rows)."""
    m, port, mat = _mixed_box(360)
    prod = O.MaxwellOperator(m, order, 1.0, face_port=port, materials=mat)
    gop = G.GpuOperator(ctx, prod)
    bs = 6 * prod.np
    y = np.random.default_rng(2).standard_normal(gop.n_dof()).astype(np.float32)
    clean = gop.apply(y).reshape(-1, bs)
    e = 173
    y[e * bs:(e + 1) * bs] = np.nan
    got = gop.apply(y).reshape(-1, bs)
    near = {e} | {int(q) for q in prod.get("nbr").reshape(-1, 4)[e] if q >= 0}
    far = np.array([q for q in range(m.n_tets) if q not in near])
    assert np.isnan(got[e]).all()
    assert np.array_equal(got[far], clean[far])


# ---- stages queued back to back (each kernel is placed while its predecessor
# ends) against the same stages with the stream drained in between: equal to
# the bit, or a kernel read its input too early

def _one_by_one(ctx, gop, h, steps, drive=None, g=None):
    for k in range(steps):
        for s in range(5):
            gop.lserk_stage(h, s, drive=drive, g=0.0 if g is None else float(g[k]))
            ctx.synchronize()


@pytest.mark.parametrize("engine", [_native.ENGINE_TF32X3, _native.ENGINE_FP32], ids=["tf32x3", "fp32"])
@pytest.mark.parametrize("order", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("cells,shuffled", [((1, 1, 1), False), ((3, 3, 3), False), ((8, 8, 8), False),
                                            ((8, 8, 8), True), ((14, 13, 11), False), ((14, 13, 11), True)],
                         ids=["one_tile", "few_tiles", "8", "8_shuffled", "14", "14_shuffled"])
def test_a_run_equals_its_stages(ctx, engine, order, cells, shuffled):
    m = O.structured_box_jittered(*cells, 1.0, 1.0, 1.0, 0.1, 5)
    if shuffled:
        m = O.Mesh(m.nodes, np.ascontiguousarray(m.tets[np.random.default_rng(1).permutation(m.n_tets)]))
    gop = G.GpuOperator(ctx, O.MaxwellOperator(m, order, 1.0))
    gop.set_engine(engine)
    n = gop.n_dof()
    rng = np.random.default_rng(order)
    y = rng.standard_normal(n).astype(np.float32)
    h = 0.05 / (max(cells) * order * order)
    g = rng.standard_normal(18)
    for steps, drive in ((1, None), (2, ("point", n // 2)), (18, None), (17, ("point", n - 1))):
        gop.upload(y)
        gop.run_lserk(h, steps, drive=drive, g=None if drive is None else g[:steps])
        got = gop.download()
        gop.upload(y)
        _one_by_one(ctx, gop, h, steps, drive, None if drive is None else g.astype(np.float32))
        assert np.array_equal(got, gop.download())


def test_runs_on_two_streams(ctx):
    """Two operators stepping at once on streams of their own."""
    other = G.GpuContext(0)
    m = O.structured_box(9, 8, 7)
    host = O.MaxwellOperator(m, 3, 1.0)
    ops = [G.GpuOperator(c, host) for c in (ctx, other)]
    y = np.random.default_rng(3).standard_normal(ops[0].n_dof()).astype(np.float32)
    for op in ops:
        op.upload(y)
    for _ in range(20):
        for op in ops:
            op.run_lserk(1e-3, 5)
    a, b = (op.download() for op in ops)
    ops[0].upload(y)
    for _ in range(20):
        ops[0].run_lserk(1e-3, 5)
    assert np.array_equal(a, b) and np.array_equal(a, ops[0].download())


@pytest.mark.parametrize("n_tets", [1, 6, 7, 8, 12, 13, 14, 15, 29, 360])
def test_order_4_pairs_at_tile_edges(ctx, n_tets):
    """The CUDA-core kernels of order 4 (two nodes per thread; tiles of 14, 7
    and 12 elements) on rough fields; f64 to the rounding of the same sums."""
    m, port, mat = _mixed_box(n_tets)
    prod = O.MaxwellOperator(m, 4, 0.3, face_port=port, materials=mat)
    orc = R.Operator(m.nodes, m.tets, 4, 0.3, face_port=port, materials=mat)
    gop = G.GpuOperator(ctx, prod)
    y = np.random.default_rng(4).standard_normal(gop.n_dof())
    y32 = y.astype(np.float32)
    want = orc.apply(y32.astype(np.float64))
    for engine in (_native.ENGINE_FP32, _native.ENGINE_FP32_SMALL_TILES):
        gop.set_engine(engine)
        assert rel_l2(gop.apply(y32), want) < 5e-6
    assert rel_l2(gop.apply_f64(y), orc.apply(y)) < 1e-11


@pytest.mark.parametrize("order", [1, 2, 3, 4, 5])
def test_wall_flux_of_a_nearly_normal_field(ctx, order):
    """E at an oblique PEC wall, all but normal to it: the wall's flux is of the
    tangential part (here 1e-3 of E) and has to be exact to the rounding of that
    part, not of E.  The field is constant, so only walls have a flux, and the
    difference of the upwind and the central right-hand side is its lifted
    penalty alone (the volume terms are the same bits).  Against the FP32 engine,
    which projects E first and reads the same records.

    Tolerance: the 3xTF32 products leave 2^-21 of each LIFT term; a LIFT row's
    terms cancel by a factor of up to about 10 over a face, so 5e-6.  Rounded as
    E is, the flux is off by the order of 2^-24 / 1e-3 = 6e-5."""
    box = O.structured_box(4, 4, 2)
    side = sum(O.boundary_faces_on_plane(box, a, v) for a in (0, 1) for v in (0.0, 1.0)).any(axis=1)
    wall = sum(O.boundary_faces_on_plane(box, 2, v) for v in (0.0, 1.0)).any(axis=1)
    q, _ = np.linalg.qr(np.array([[2.0, 0.3, 0.5], [0.1, 1.5, 0.7], [0.4, 0.2, 1.0]]))
    m = O.Mesh(np.ascontiguousarray(box.nodes @ q.T), box.tets)  # z walls: normal q[:, 2]
    field = np.zeros(6)
    field[:3] = q[:, 2] + 1e-3 * q[:, 0]
    got = {}
    for engine in (_native.ENGINE_TF32X3, _native.ENGINE_FP32):
        dy = []
        for alpha in (1.0, 0.0):
            gop = G.GpuOperator(ctx, O.MaxwellOperator(m, order, alpha))
            gop.set_engine(engine)
            y = np.tile(field, gop.n_dof() // 6).astype(np.float32)
            dy.append(gop.apply(y).astype(np.float64).reshape(m.n_tets, -1))
        got[engine] = (dy[0] - dy[1])[wall & ~side]  # the side walls see E as tangential
    assert rel_l2(got[_native.ENGINE_TF32X3], got[_native.ENGINE_FP32]) < 5e-6
