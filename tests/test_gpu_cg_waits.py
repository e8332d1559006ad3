"""The bounded waits of the solve on chip (k_cg_group): made to run out by a
short limit and a task left out of the schedule, they end in a status, and the
handle stays usable."""
import numpy as np
import pytest

from ffea_gb300 import params as P
from tests.helpers import spec

pytestmark = pytest.mark.gpu

FAIL_TIMEOUT = 8


def _world(monkeypatch, radii, max_ctas, epsilon=None, **kw):
    from ffea_gb300.world import World
    monkeypatch.setenv("FFEA_GPU_CG_MAX_CTAS", str(max_ctas))
    specs = [spec(radius_nm=r, seed=i + 1, rng_seed=60 + i, precision=P.PRECISION_MIXED,
                  epsilon=epsilon[i] if epsilon else 1e-6)
             for i, r in enumerate(radii)]
    return World(specs, **kw)


def _state(w):
    return [(*w.blob(i).get_nodes()[:2], w.blob(i).rng_state()) for i in range(w.num_blobs)]


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


# the first blob on both CTAs (a segment each of 720, of 220 rows; three segments, two to a CTA), the others queued
# behind it, two to each: the left-out segment starts the second CTA's task
@pytest.mark.parametrize("radii,segment", [((8.0, 3.0, 3.2, 3.4, 3.6), 1), ((5.0, 3.0, 3.0, 3.0, 3.0), 1),
                                           ((10.0, 3.0, 3.2, 3.4, 3.6), 2)])
@pytest.mark.parametrize("rng_mode,preconditioner", [(0, 0), (0, 1), (1, 0)])
def test_a_time_out_fails_every_blob_queued_behind_it(gpulib, monkeypatch, radii, segment, rng_mode, preconditioner):
    from ffea_gb300._lib import FfeaGpuError, check
    kw = dict(rng_mode=rng_mode, preconditioner=preconditioner)
    with _world(monkeypatch, radii, 2, **kw) as w, _world(monkeypatch, radii, 2, **kw) as free:
        w.run(1)
        free.run(1)
        before = _state(w)
        check(gpulib.ffea_gpu_selftest_solve_timeout(w.handle, 1024, 0, segment))
        for step in range(2):
            with pytest.raises(FfeaGpuError):
                w.run(1)
            free.run(1)
            bits = [w.blob(i).status()["fail_bits"] for i in range(w.num_blobs)]
            now, ref = _state(w), _state(free)
            for i, b in enumerate(bits):
                if b:  # not solved, or not to the end: stays at the failing step
                    assert b & FAIL_TIMEOUT and _same(now[i][:2], before[i][:2]), (step, i)
                    if rng_mode == 0:
                        assert np.array_equal(now[i][2], before[i][2]), (step, i)
                else:  # as without the time-out, its draws and its stream's state too
                    assert _same(now[i], ref[i]), (step, i)
            assert bits[0] and any(bits[1:]) and not all(bits[1:]), bits


# a CTA that is free early waits for its next blob's other CTA through the whole solve of the blob before: three and two
# CTAs of two segments each on four CTAs; a blob of two segments behind one solve that is long and one that is short
@pytest.mark.parametrize("radii,epsilon,max_ctas", [((10.0, 8.0), (1e-6, 1e-6), 4),
                                                    ((6.4, 6.4, 7.0), (1e-6, 0.5, 1e-6), 2)])
def test_a_wait_lasts_through_another_blobs_solve(gpulib, monkeypatch, radii, epsilon, max_ctas):
    """The limit, 256 reads (about 50 us), is many iterations long and shorter
    than a solve: a blob that waits longer than that for CTAs that get on with
    another solve is solved as with the default limit."""
    from ffea_gb300._lib import check
    with _world(monkeypatch, radii, max_ctas, epsilon) as w, _world(monkeypatch, radii, max_ctas, epsilon) as free:
        check(gpulib.ffea_gpu_selftest_solve_timeout(w.handle, 256, -1, 0))
        for step in range(3):
            free.run(1)
            w.run(1)
            for i, (a, b) in enumerate(zip(_state(w), _state(free))):
                assert w.blob(i).status()["fail_bits"] == 0 and _same(a, b), (step, i)
