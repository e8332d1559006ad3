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


def _compare(got, ref, some=True):
    (f, e, p), (f_ref, e_ref, p_ref) = got, ref
    assert p == p_ref and (p_ref > 0 or not some)
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


def _two(r1, cell1, r2, cell2, gap, h):
    """Two spheres of given radius and element size, `gap` nm between them (negative: pushed into each other)."""
    from ffea_gb300.mesh import sphere_mesh
    from ffea_gb300.surface import surface_faces
    pos, faces, apex, blob, n = [], [], [], [], 0
    for k, (r, cell) in enumerate(((r1, cell1), (r2, cell2))):
        m = sphere_mesh(r, cell_nm=cell, seed=1 + k)
        tri, ap = surface_faces(m.pos, m.topology, with_apex=True)
        x = m.pos - m.pos.mean(0)
        if k:
            x = x + np.array([pos[0][:, 0].max() - x[:, 0].min() + nm(gap), 0.0, 0.0])
        pos.append(x)
        faces.append(tri + n)
        apex.append(ap + n)
        blob.append(np.full(len(tri), k, np.int32))
        n += len(x)
    pos, h = np.concatenate(pos), nm(h)
    grid = tuple(int(v) for v in 2 * np.ceil((pos.max(0) - pos.min(0)) / h))
    pos = pos - 0.5 * (pos.max(0) + pos.min(0)) + 0.5 * h * np.array(grid)
    faces = np.concatenate(faces).astype(np.int32)
    return pos, dict(num_nodes=len(pos), faces=faces, face_blob=np.concatenate(blob),
                     face_type=np.zeros(len(faces), np.int32), emin=np.ones((1, 1)), rmin=np.full((1, 1), nm(1.0)),
                     num_blobs=2, cell_size=h, grid=grid, face_apex=np.concatenate(apex).astype(np.int32),
                     steric_factor=50.0, steric_dr=5e-3, k0=np.full((1, 1), 0.3))


# faces that have candidates on 152 SMs: up to one an SM (65 and 83), up to three (168 and 176), more (1,676 and 1,142);
# small elements against ones of 6 nm: faces with up to 52 candidates, more than the 32 that are kept
@pytest.mark.parametrize("spheres,inc_self", [((4.0, 1.25, 4.0, 1.25, -0.6, 3.0), 0),
                                              ((8.0, 1.25, 8.0, 1.25, -0.6, 3.0), 0),
                                              ((8.0, 1.25, 8.0, 1.25, -0.6, 3.0), 1),
                                              ((8.0, 6.0, 8.0, 1.0, -0.5, 6.0), 0),
                                              ((12.0, 6.0, 12.0, 1.0, -1.0, 6.0), 0),
                                              ((8.0, 6.0, 8.0, 1.0, -0.5, 6.0), 1)])
@pytest.mark.parametrize("ssint_type,shifted", [(1, False), (1, True), (2, False)])
def test_steric_faces_few_and_many(spheres, inc_self, ssint_type, shifted):
    from ffea_gb300.surface import LJSurfaceSolver
    pos, kw = _two(*spheres)
    kw.update(inc_self=inc_self, ssint_type=ssint_type)
    s = LJSurfaceSolver(**kw)
    corr = None
    if shifted:  # the second blob one box length on in y, and 0.3 nm away in x (where 0.5 were in contact: none is left)
        pos = pos.copy()
        pos[kw["faces"][kw["face_blob"] == 1].min():, 1] += s.box[1]
        corr = np.zeros((2, 2, 3))
        corr[0, 1] = [-0.3 * nm(1.0), s.box[1], 0.0]
        corr[1, 0] = -corr[0, 1]
        s.set_pbc(corr)
    got = s.forces(pos)
    again = s.forces(pos)
    s.close()
    _compare(got, _oracle(kw, pos, blob_corr=corr), some=not shifted or spheres[4] < -0.5)
    # (the sums of a face are in the order of its candidates; the energies are summed with atomics)
    assert again[2] == got[2] and np.abs(again[0] - got[0]).max() <= 1e-12 * np.abs(got[0]).max()


def test_faces_without_partners_cost_a_search_only():
    """Two 20 nm spheres apart: of a steric solve nothing is left but the
    search for partners, as of a Lennard-Jones solve (LJ 0.14 ms; with a CTA
    of the clipping kernel for every face the steric solve took 0.9 ms)."""
    import torch
    from ffea_gb300.surface import LJSurfaceSolver
    pos, kw = _two(20.0, 1.25, 20.0, 1.25, 4.0, 3.0)
    d_pos = torch.tensor(pos, device="cuda")
    d_f, d_e = torch.zeros_like(d_pos), torch.zeros(4, dtype=torch.float64, device="cuda")
    best = {}
    for ssint_type in (0, 1):
        s = LJSurfaceSolver(inc_self=0, ssint_type=ssint_type, **kw)
        times = []
        for _ in range(12):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            with torch.cuda.stream(torch.cuda.ExternalStream(s.stream)):
                a.record()
                s.forces_device(d_pos.data_ptr(), d_f.data_ptr(), d_e.data_ptr())
                b.record()
            pairs = s.synchronize()
            times.append(a.elapsed_time(b))
        best[ssint_type] = min(times)
        s.close()
    assert pairs == 0 and not d_f.any() and best[1] < 3 * best[0], best
