"""A tuning belongs to the kernels it was timed on (ffea_gb300.autotune), on the CPU."""
import json
import types

from ffea_gb300 import autotune as A


def test_a_tuning_of_other_kernels_is_not_reused(monkeypatch, tmp_path):
    import torch
    device = types.SimpleNamespace(name="GPU", multi_processor_count=152)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda d: device)
    src = tmp_path / "csrc"
    src.mkdir()
    (src / "solve.cu").write_text("slots in shared memory\n")
    timed = []
    monkeypatch.setattr(A, "time_config", lambda specs, cfg, pc, **kw: timed.append(cfg) or 1e-3)
    version = A.kernel_version
    monkeypatch.setattr(A, "kernel_version", lambda: version.__wrapped__(str(src)))
    space, cache = [{"FFEA_GPU_CG_SMEM_SLOTS": 3}], str(tmp_path / "tune.json")
    first = A.tune([], 2, space=space, cache=cache)
    assert A.tune([], 2, space=space, cache=cache) == first and len(timed) == 1
    (src / "solve.cu").write_text("slots in shared and tensor memory\n")
    A.tune([], 2, space=[{"FFEA_GPU_CG_SMEM_SLOTS": 64}], cache=cache)
    assert len(timed) == 2 and len(json.load(open(cache))) == 2


def test_the_version_is_that_of_the_sources():
    assert A.kernel_version() == A.kernel_version() and len(A.kernel_version()) == 16
