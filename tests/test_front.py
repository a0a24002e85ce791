"""The native front of quantized_matmul is an addition: a file that cannot be used takes no product down."""
import subprocess
import sys
import warnings
from pathlib import Path

import pytest
import torch

import mlx_kquant_b200 as kq
from mlx_kquant_b200 import _lib, ops

CSRC = Path(_lib.__file__).resolve().parent / "csrc"


@pytest.fixture
def fresh(monkeypatch):
    monkeypatch.setattr(_lib, "_front", None)
    monkeypatch.setattr(ops, "_front_qmm", ops._first_qmm)


def call():
    """As far as a call comes without a GPU: the weights are found not to be on one."""
    with pytest.raises(RuntimeError, match="CUDA device"):
        kq.quantized_matmul(torch.zeros(1, 256), torch.zeros(8, 144, dtype=torch.uint8), None, "q4_k")


def test_broken_file(fresh, monkeypatch, tmp_path):
    (tmp_path / "_kq_torch.so").write_bytes(b"not a shared object")
    monkeypatch.setattr(_lib, "HERE", tmp_path)
    with pytest.warns(RuntimeWarning, match="not used"):
        call()
    with warnings.catch_warnings():
        warnings.simplefilter("error")   # said once
        call()
    assert _lib.torch_front() is None


def test_absent(fresh, monkeypatch, tmp_path):
    monkeypatch.setattr(_lib, "HERE", tmp_path)
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        call()


def test_of_another_torch(fresh, monkeypatch):
    if not (CSRC.parent / "_kq_torch.so").exists():
        pytest.skip("not built")
    monkeypatch.setattr(torch, "__version__", "0.0")
    with pytest.warns(RuntimeWarning, match="built for torch"):
        assert _lib.torch_front() is None


def test_the_library_builds_without_torch(tmp_path):
    """What make would do with a python that has no torch: the library and nothing else."""
    stub = tmp_path / "python3"
    stub.write_text(f'#!/bin/sh\ncase "$*" in *torch*) exit 1;; esac\nexec {sys.executable} "$@"\n')
    stub.chmod(0o755)
    out = subprocess.run(["make", "-n", "-B", "-C", str(CSRC), f"PY={stub}"], capture_output=True, text=True)
    assert out.returncode == 0, out.stderr
    assert "libkquant_b200.so" in out.stdout and "kq_torch.cpp" not in out.stdout
    with_torch = subprocess.run(["make", "-n", "-B", "-C", str(CSRC), f"PY={sys.executable}"], capture_output=True, text=True)
    assert with_torch.returncode == 0 and "kq_torch.cpp" in with_torch.stdout
