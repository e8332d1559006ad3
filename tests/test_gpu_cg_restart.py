"""Restarts of the solve on chip (k_cg_group) from a failed FP64 residual: at
an epsilon below what FP32 vectors carry, the recursive residual passes before
the true one does, and the recurrences start again from that."""
import numpy as np
import pytest

from ffea_gb300 import params as P
from tests.helpers import spec

pytestmark = pytest.mark.gpu

FAIL_CG = 2


def _run(monkeypatch, radius, max_ctas, memory, epsilon, solver, true_residual, **kw):
    from ffea_gb300._lib import FfeaGpuError
    from ffea_gb300.world import World
    monkeypatch.setenv("FFEA_GPU_CG_MAX_CTAS", str(max_ctas))
    monkeypatch.setenv("FFEA_GPU_CG_MEMORY_STATE", "1" if memory else "0")
    s = spec(radius_nm=radius, rng_seed=80, precision=P.PRECISION_MIXED, epsilon=epsilon, solver=solver)
    with World([s], true_residual=true_residual, **kw) as w:
        try:
            w.run(1)
        except FfeaGpuError:
            pass
        return w.blob(0).get_nodes(), w.blob(0).status()


# one segment, two segments on two CTAs, and two on one; 5e-8 is met after restarts, 3e-8 is not with the four allowed
@pytest.mark.parametrize("radius,max_ctas", [(5.0, 1), (8.0, 2), (8.0, 1)])
@pytest.mark.parametrize("solver,preconditioner", [(P.SOLVER_NOMASS, 0), (P.SOLVER_MASS, 0), (P.SOLVER_NOMASS, 1)])
def test_restart_from_a_failed_true_residual(gpulib, monkeypatch, radius, max_ctas, solver, preconditioner):
    kw = dict(solver=solver, preconditioner=preconditioner)
    _, plain = _run(monkeypatch, radius, max_ctas, False, 5e-8, true_residual=False, **kw)
    on, st = _run(monkeypatch, radius, max_ctas, False, 5e-8, true_residual=True, **kw)
    assert plain["fail_bits"] == st["fail_bits"] == 0 and st["true_relres"] < 5e-8
    assert st["cg_iters"] > plain["cg_iters"]  # it went on after the recursive residual had passed
    _, bad = _run(monkeypatch, radius, max_ctas, False, 3e-8, true_residual=True, **kw)
    assert bad["fail_bits"] == FAIL_CG and bad["true_relres"] >= 3e-8
    if preconditioner == 0:  # the memory-resident solve restarts from the same bits
        mem, s_mem = _run(monkeypatch, radius, max_ctas, True, 5e-8, true_residual=True, **kw)
        assert st["cg_iters"] == s_mem["cg_iters"]
        for a, b in zip(on, mem):
            np.testing.assert_allclose(a, b, rtol=0, atol=1e-6 * np.abs(b).max())
