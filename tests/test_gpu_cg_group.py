"""The solve of blobs that fit on chip (k_cg_group) at the edges of its launch
shapes: rows of a CTA around 256, 512 and 1024 (the variants' limits), one CTA
for a blob and several, more blobs than CTAs (a CTA with a list of segments),
pinned rows, and both precisions.

FFEA_GPU_CG_MAX_CTAS caps the grid, which makes segments longer (at most 1024
rows each).  The memory-resident solve runs the same arithmetic in the same
order, so with Jacobi both give the same bits; the true residual, which this
kernel sums in three FP32 parts and the other in FP64, agrees to the FP64
rounding of about a hundred terms a row (1e-12 relative).
"""
import numpy as np
import pytest

from ffea_gb300 import params as P
from tests.helpers import spec

pytestmark = pytest.mark.gpu


def _run(monkeypatch, specs, max_ctas, memory, steps=3, **kw):
    from ffea_gb300.world import World
    monkeypatch.setenv("FFEA_GPU_CG_MAX_CTAS", str(max_ctas))
    monkeypatch.setenv("FFEA_GPU_CG_MEMORY_STATE", "1" if memory else "0")
    with World(specs, **kw) as w:
        w.run(steps)
        return [w.blob(i).get_nodes() for i in range(len(specs))], [w.blob(i).status() for i in range(len(specs))], \
            [w.blob(i).rng_state() for i in range(len(specs))]


def _mixed(radius, seed, **kw):
    return spec(radius_nm=radius, seed=seed, rng_seed=80 + seed, precision=P.PRECISION_MIXED, epsilon=1e-6, **kw)


# (radii, CTA cap): 130 rows on one CTA; 437 rows on one CTA, and on two; 860 on one; 1,445 on two of about 720;
# a list of segments per CTA (5 blobs, 2 CTAs); 2,771 rows on 12 CTAs of about 230
CASES = [((3.0,), 1), ((5.0,), 1), ((5.0,), 2), ((6.4,), 1), ((8.0,), 2), ((3.0, 5.0, 4.0, 3.5, 6.0), 2), ((10.0,), 12)]


@pytest.mark.parametrize("radii,max_ctas", CASES)
@pytest.mark.parametrize("solver", [P.SOLVER_NOMASS, P.SOLVER_MASS])
def test_same_bits_as_the_memory_resident_solve(gpulib, monkeypatch, radii, max_ctas, solver):
    specs = [_mixed(r, i + 1, solver=solver, pinned=[0, 7] if i % 2 else None) for i, r in enumerate(radii)]
    on, s_on, g_on = _run(monkeypatch, specs, max_ctas, False, true_residual=True)
    mem, s_mem, g_mem = _run(monkeypatch, specs, max_ctas, True, true_residual=True)
    for i in range(len(specs)):
        for a, b in zip(on[i], mem[i]):
            assert np.array_equal(a, b), i
        assert np.array_equal(g_on[i], g_mem[i])
        assert s_on[i]["fail_bits"] == 0 and s_on[i]["cg_iters"] == s_mem[i]["cg_iters"]
        assert s_on[i]["true_relres"] == pytest.approx(s_mem[i]["true_relres"], rel=1e-12)


@pytest.mark.parametrize("radii,max_ctas", CASES)
def test_two_level_meets_the_true_residual(gpulib, monkeypatch, radii, max_ctas):
    specs = [_mixed(r, i + 1) for i, r in enumerate(radii)]
    _, st, _ = _run(monkeypatch, specs, max_ctas, False, true_residual=True, preconditioner=1)
    for s in st:
        assert s["fail_bits"] == 0 and s["true_relres"] < 1e-6, s


@pytest.mark.parametrize("radii,max_ctas", CASES)
@pytest.mark.parametrize("solver", [P.SOLVER_NOMASS, P.SOLVER_MASS])
def test_fp64_matches_oracle(gpulib, oracle, monkeypatch, radii, max_ctas, solver):
    specs = [spec(radius_nm=r, seed=i + 1, rng_seed=80 + i, solver=solver) for i, r in enumerate(radii)]
    on, st, _ = _run(monkeypatch, specs, max_ctas, False)
    for i, s in enumerate(specs):
        ref = oracle.blob_from_spec(s)
        assert ref.step(3) == 0 and st[i]["fail_bits"] == 0
        pos, vel, _ = ref.nodes()
        assert np.linalg.norm(on[i][1] - vel) <= 1e-9 * np.linalg.norm(vel), i
        assert np.abs(on[i][0] - pos).max() < 1e-10, i


@pytest.mark.parametrize("slots", [1, 8, 11])
@pytest.mark.parametrize("radii,max_ctas", [((5.0,), 1), ((8.0,), 2)])
def test_matrix_slots_in_each_memory(gpulib, monkeypatch, radii, max_ctas, slots):
    """The variants of more than 256 rows keep a row's first matrix slots in
    shared memory, more in tensor memory (an odd or an even number of them,
    the first or the last of a row's) and read the rest from L2; the
    environment variable caps the slots on chip."""
    monkeypatch.setenv("FFEA_GPU_CG_SMEM_SLOTS", str(slots))
    specs = [_mixed(r, i + 1, pinned=[0, 7]) for i, r in enumerate(radii)]
    on, s_on, _ = _run(monkeypatch, specs, max_ctas, False)
    mem, s_mem, _ = _run(monkeypatch, specs, max_ctas, True)
    for i in range(len(specs)):
        for a, b in zip(on[i], mem[i]):
            assert np.array_equal(a, b), i
        assert s_on[i]["fail_bits"] == 0 and s_on[i]["cg_iters"] == s_mem[i]["cg_iters"]


@pytest.mark.parametrize("radii,max_ctas", [((8.0, 7.9, 8.0, 10.0, 10.0, 10.0), 5), ((8.0, 3.0, 10.0, 3.5, 8.0), 4)])
def test_blobs_scheduled_in_rounds(gpulib, monkeypatch, radii, max_ctas):
    """Groups of two and three CTAs on five (two rounds' worth when a two and a
    three share each, more when the threes come first), and of one to three on four."""
    specs = [_mixed(r, i + 1) for i, r in enumerate(radii)]
    on, s_on, g_on = _run(monkeypatch, specs, max_ctas, False)
    mem, s_mem, g_mem = _run(monkeypatch, specs, max_ctas, True)
    for i in range(len(specs)):
        for a, b in zip(on[i], mem[i]):
            assert np.array_equal(a, b), i
        assert np.array_equal(g_on[i], g_mem[i])
        assert s_on[i]["fail_bits"] == 0 and s_on[i]["cg_iters"] == s_mem[i]["cg_iters"]


# two segments to a CTA: (radii, CTA cap) one CTA with both; four on two CTAs; three (one CTA has a single one)
# beside a blob of one
WIDE = [((8.0,), 1), ((10.0,), 2), ((10.0, 3.0), 2)]


@pytest.mark.parametrize("radii,max_ctas", WIDE)
@pytest.mark.parametrize("solver", [P.SOLVER_NOMASS, P.SOLVER_MASS])
def test_two_segments_to_a_cta_same_bits(gpulib, monkeypatch, radii, max_ctas, solver):
    specs = [_mixed(r, i + 1, solver=solver, pinned=[0, 7] if i % 2 == 0 else None) for i, r in enumerate(radii)]
    on, s_on, g_on = _run(monkeypatch, specs, max_ctas, False, true_residual=True)
    mem, s_mem, g_mem = _run(monkeypatch, specs, max_ctas, True, true_residual=True)
    for i in range(len(specs)):
        for a, b in zip(on[i], mem[i]):
            assert np.array_equal(a, b), i
        assert np.array_equal(g_on[i], g_mem[i])
        assert s_on[i]["fail_bits"] == 0 and s_on[i]["cg_iters"] == s_mem[i]["cg_iters"]
        assert s_on[i]["true_relres"] == pytest.approx(s_mem[i]["true_relres"], rel=1e-12)


@pytest.mark.parametrize("radii,max_ctas", WIDE)
def test_two_segments_to_a_cta_two_level(gpulib, monkeypatch, radii, max_ctas):
    specs = [_mixed(r, i + 1) for i, r in enumerate(radii)]
    _, st, _ = _run(monkeypatch, specs, max_ctas, False, true_residual=True, preconditioner=1)
    _, s_mem, _ = _run(monkeypatch, specs, max_ctas, True, true_residual=True, preconditioner=1)
    for s, m in zip(st, s_mem):
        assert s["fail_bits"] == 0 and s["true_relres"] < 1e-6, s
        assert abs(s["cg_iters"] - m["cg_iters"]) <= 1


@pytest.mark.parametrize("blobs", [2, 3, 5, 9, 65])
def test_start_sums_of_batches(gpulib, oracle, blobs):
    """r.u and f.f of every blob come from the last CTA of k_nodes: all its
    warps on one blob, four or two warps a blob, a warp per blob, and more
    blobs than it finishes at a time; FP64 steps against the oracle."""
    from ffea_gb300.world import World
    specs = [spec(radius_nm=3.0 + 0.25 * (i % 5), seed=i + 1, rng_seed=40 + i) for i in range(blobs)]
    with World(specs) as w:
        w.run(2)
        for i in sorted({0, 1, blobs // 2, blobs - 2, blobs - 1}):
            ref = oracle.blob_from_spec(specs[i])
            assert ref.step(2) == 0 and w.blob(i).status()["fail_bits"] == 0
            pos, vel, _ = ref.nodes()
            on = w.blob(i).get_nodes()
            assert np.linalg.norm(on[1] - vel) <= 1e-9 * np.linalg.norm(vel), i
            assert np.abs(on[0] - pos).max() < 1e-10, i


@pytest.mark.parametrize("radius,max_ctas", [(1.9, 1), (3.0, 2), (3.0, 1), (3.4, 1)])
@pytest.mark.parametrize("solver", [P.SOLVER_NOMASS, P.SOLVER_MASS])
def test_fp64_products_in_quarters(gpulib, oracle, monkeypatch, radius, max_ctas, solver):
    """FP64 segments of one to six slices, whose products run in quarters of a
    slice over the CTA's warps (not those of four slices), at the tolerances
    of the test above; the true residual is checked too."""
    s = spec(radius_nm=radius, seed=3, rng_seed=91, solver=solver, pinned=[1])
    on, st, _ = _run(monkeypatch, [s], max_ctas, False, true_residual=True)
    ref = oracle.blob_from_spec(s)
    assert ref.step(3) == 0 and st[0]["fail_bits"] == 0 and st[0]["true_relres"] < 1e-12
    pos, vel, _ = ref.nodes()
    assert np.linalg.norm(on[0][1] - vel) <= 1e-9 * np.linalg.norm(vel)
    assert np.abs(on[0][0] - pos).max() < 1e-10
