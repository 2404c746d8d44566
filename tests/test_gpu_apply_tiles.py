"""The complex128 operator at the edges of its tiles: 32 x 8 nodes, slabs of 4 to
32 planes (a tile and slab exactly filled, one node or plane more, less than
one), against the oracle's operator."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from aphid_git_b200 import Solver, model
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(3, 3, 3), (32, 8, 4), (33, 9, 5), (31, 16, 33), (66, 7, 34)])
def test_operator_at_tile_edges(dims):
    """Tolerance: a row adds some 20 complex products of four roundings each and
    multiplies by reciprocals where the oracle divides; 100 roundings of 1.1e-16
    of the rows' norm."""
    rng = np.random.default_rng(dims[0])
    axes = [np.cumsum(rng.uniform(50.0, 400.0, d)) for d in dims]
    cells = tuple(d - 1 for d in dims)
    sig = (10.0 ** rng.uniform(-3, 0, cells)).astype(np.float32)
    w = 2 * np.pi * 3.0
    g = O.Grid(*axes)
    sh = O.sigma_hat("R", w, sig_re=sig)
    with Solver() as s:
        s.set_nodes(*axes)
        k2 = s.gen_k2(np.asarray(sh).ravel(order="F"), w)
        x = rng.standard_normal(2 * g.n).view(np.complex128)
        y = s.inprod(k2, x)
    ref = O.inprod(g, k2, x)
    assert np.linalg.norm(y - ref) <= 100 * 1.1e-16 * np.linalg.norm(ref)
