"""Kernels that run beside one another compute what they compute one after the other."""
import os
import pathlib
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu

HERE = pathlib.Path(__file__).resolve().parent


def test_programmatic_launches_change_no_bit(cuda_device, tmp_path):
    """With GFS_PDL=0 the same kernels, tiles and orders of summation run strictly one after the other. Weights fetched early,
    late-waiting weight gradients and dQ beside dK / dV must give the same bits: losses, gradients (added ones too), weights
    and logits of six models on both paths, and attention by itself."""
    results = []
    for on in "01":
        path = tmp_path / f"pdl{on}.pt"
        env = dict(os.environ, GFS_PDL=on, PYTHONPATH=str(HERE.parent))
        run = subprocess.run([sys.executable, str(HERE / "overlap_worker.py"), str(path)], env=env, cwd=HERE.parent, text=True,
                             capture_output=True, timeout=300)
        assert run.returncode == 0, run.stderr[-3000:]
        results.append(torch.load(path))
    assert results[0].keys() == results[1].keys()
    for name, serial in results[0].items():
        for i, (a, b) in enumerate(zip(serial, results[1][name], strict=True)):
            assert torch.equal(a, b), f"{name}, result {i}"
            assert a.isfinite().all(), f"{name}, result {i}"
