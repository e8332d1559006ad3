"""Surface interactions at the edges of what the entry points accept, against
the oracle (oracle/ssint_oracle.c): tolerances as in tests/test_gpu_ssint.py."""
import numpy as np
import pytest

from ffea_gb300.params import nm
from oracle import oracle

pytestmark = pytest.mark.gpu


def _inputs(ssint_type, inc_self, seed):
    """Two spheres pushed into each other: the solver's arguments and the positions."""
    from tests.test_steric_oracle import overlapping_spheres
    pos, faces, apex, blob, h, grid = overlapping_spheres()
    rng = np.random.default_rng(seed)
    emin = rng.uniform(0.5, 2.0, (2, 2))
    kw = dict(num_nodes=len(pos), faces=faces, face_blob=blob, face_type=rng.integers(0, 2, len(faces)).astype(np.int32),
              emin=0.5 * (emin + emin.T), rmin=np.full((2, 2), nm(1.0)), num_blobs=2, cell_size=h, grid=grid,
              inc_self=inc_self, ssint_type=ssint_type, face_apex=apex, steric_factor=50.0, steric_dr=5e-3,
              k0=np.full((2, 2), 0.3))
    return kw, pos


def _oracle(kw, pos, **more):
    return oracle.ssint(pos, kw["faces"], kw["face_blob"], kw["face_type"], kw["emin"], kw["rmin"], kw["num_blobs"],
                        kw["cell_size"], kw["grid"], kw["inc_self"], kw["ssint_type"], kw["face_apex"], 50.0, 5e-3,
                        kw["k0"], **more)


def _compare(got, ref):
    (f, e, p), (f_ref, e_ref, p_ref) = got, ref
    assert p == p_ref and p_ref > 0
    np.testing.assert_allclose(f, f_ref, rtol=0, atol=1e-9 * np.abs(f_ref).max())
    np.testing.assert_allclose(e, e_ref, rtol=1e-9, atol=1e-9 * np.abs(e_ref).max())


def test_corrections_of_either_order_of_the_blobs():
    """set_pbc takes any matrix: the pair of faces (f1, f2) is shifted by
    blob_corr[blob of f2][blob of f1], whatever the other order's entry and
    the diagonal hold."""
    from ffea_gb300.surface import LJSurfaceSolver
    kw, pos = _inputs(0, 1, seed=17)
    corr = np.random.default_rng(3).uniform(-0.2, 0.2, (2, 2, 3)) * nm(1.0)
    s = LJSurfaceSolver(**kw)
    s.set_pbc(corr)
    got = s.forces(pos)
    s.close()
    _compare(got, _oracle(kw, pos, blob_corr=corr))


@pytest.mark.parametrize("ssint_type", [1, 3])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, -np.nan])
def test_fourth_nodes_that_are_not_finite(ssint_type, value):
    """A face whose element's fourth node is at infinity (a blob that blew up)
    has no overlap volume with the other blob's faces: those keep finite
    forces, the same as the oracle's, and the pairs stay the same."""
    from ffea_gb300.surface import LJSurfaceSolver
    kw, pos = _inputs(ssint_type, 0, seed=19)
    surface = np.unique(kw["faces"])
    inner = np.setdiff1d(kw["face_apex"][kw["face_blob"] == 1], surface)
    inner = inner[np.argsort(pos[inner, 0])][:12]  # those nearest the contact
    pos = pos.copy()
    pos[inner[::2], 0] = value
    pos[inner[1::2]] = value
    s = LJSurfaceSolver(**kw)
    got = s.forces(pos)
    s.close()
    ref = _oracle(kw, pos)
    own = np.arange(len(pos)) < len(pos) // 2
    assert np.isfinite(ref[0][own]).all()
    _compare((got[0][own], got[1], got[2]), (ref[0][own], ref[1], ref[2]))
