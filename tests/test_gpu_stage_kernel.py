"""The tensor-core stage kernel's tile edges: the flux units (groups of four
face nodes, whose last group is partly padding), every face kind in one tile,
rough fields, tiles of which one element or all but one are real.

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
