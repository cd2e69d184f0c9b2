"""CPU-only checks of the package layout, the build and the model bookkeeping."""
import math


def test_import_and_layout():
    import aws_ofi_nccl_b200
    import aws_ofi_nccl_b200.models
    import aws_ofi_nccl_b200.ops
    import aws_ofi_nccl_b200.parallel
    import aws_ofi_nccl_b200.utils

    assert aws_ofi_nccl_b200.__version__


def test_llama3_8b_parameter_count():
    from aws_ofi_nccl_b200.models.llama import LlamaConfig

    cfg = LlamaConfig.llama3_8b()
    n = cfg.num_params()
    assert abs(n - 8.03e9) < 0.01e9, n
    assert math.prod(dict(cfg.param_shapes())["l0.wqkv"]) == 6144 * 4096


def test_kernel_library_builds_for_sm100a(built):
    assert (built / "libb200ops.so").exists()
    import ctypes

    lib = ctypes.CDLL(str(built / "libb200ops.so"))
    for sym in ("b200_gemm_bf16", "b200_rmsnorm_fwd", "b200_adamw", "b200_cross_entropy"):
        assert hasattr(lib, sym)


def test_bench_reference_arm_reports_unavailable():
    import json
    import subprocess
    import sys
    from pathlib import Path

    root = Path(__file__).resolve().parent.parent
    out = subprocess.run([sys.executable, str(root / "bench.py"), "--impl", "reference"], capture_output=True,
                         text=True, check=True).stdout.strip().splitlines()[-1]
    d = json.loads(out)
    assert d["impl"] == "reference" and "unavailable" in d


def test_native_layers_are_rebuilt_for_another_torch_or_header(tmp_path, monkeypatch):
    """What the module was built against decides, not the age of its own source alone."""
    import os

    from aws_ofi_nccl_b200 import build

    runs = []
    monkeypatch.setattr(build, "LIB", tmp_path)
    monkeypatch.setattr(build, "_run", runs.append)
    out, header = tmp_path / "_b200torch.so", build.CSRC / "kernels" / "b200ops.h"
    out.write_bytes(b"")
    (tmp_path / "_b200torch.stamp").write_text(build.torch_ops_tag())
    build.build_torch_ops()
    assert not runs                                    # up to date
    (tmp_path / "_b200torch.stamp").write_text("torch 1.0 another-python")
    build.build_torch_ops()
    assert len(runs) == 1                              # another torch
    build.build_torch_ops()
    assert len(runs) == 1                              # and the stamp says so
    os.utime(out, (0, header.stat().st_mtime - 1))
    build.build_torch_ops()
    assert len(runs) == 2                              # a signature may have changed


def test_a_step_whose_kernels_gave_up_on_a_wait_raises(monkeypatch):
    """The status that the kernels leave, read behind the loss; a clean step returns that."""
    import pytest
    import torch

    from aws_ofi_nccl_b200.ops import _lib
    from aws_ofi_nccl_b200.parallel.engine import Trainer

    trainer = Trainer.__new__(Trainer)
    trainer.device, trainer._ids_dev, trainer.step_device = torch.device("cpu"), None, lambda ids, labels: torch.tensor(1.5)
    batch = torch.zeros(2, 4, dtype=torch.int64)
    status = [0]
    monkeypatch.setattr(_lib, "read_status", lambda: status[0])
    assert trainer.step(batch, batch) == 1.5
    status[0] = 7
    with pytest.raises(_lib.B200OpsError, match="status 7"):
        trainer.step(batch, batch)
