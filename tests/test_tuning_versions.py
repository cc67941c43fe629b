"""Saved launch shapes of the batched engine: those timed with another version
of its kernel are timed again, those a user pins are kept."""

from __future__ import annotations

import json
import shutil
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT, two_phase

pytestmark = pytest.mark.gpu

COUNT = 160  # enough problems for the tuner


def key() -> str:
    import torch

    return f"{torch.cuda.get_device_name(0)}|side<=16|mixed|pc2|c2|s11|few"


def solve_with(monkeypatch, path, entry) -> list:
    from darcy_cpp_gb300 import capi

    path.write_text(json.dumps({key(): entry}))
    monkeypatch.setenv("DARCY_GPU_TUNE_FILE", str(path))
    a = np.stack([two_phase(16, seed=1)] * COUNT)
    assert capi.Context().solve_batch(a, form="mixed")["converged"].all()
    return json.loads(path.read_text())[key()]


def test_shapes_of_another_kernel_version_are_timed_again(monkeypatch, tmp_path) -> None:
    saved = solve_with(monkeypatch, tmp_path / "tune.json", [992, 0, 1])
    assert saved[:2] != [992, 0] and len(saved) == 3 and saved[2] > 1
    again = solve_with(monkeypatch, tmp_path / "again.json", [992, 0, saved[2]])
    assert again == [992, 0, saved[2]]  # of this version: taken as it is


def test_pinned_shapes_are_kept(monkeypatch, tmp_path) -> None:
    assert solve_with(monkeypatch, tmp_path / "tune.json", [992, 0]) == [992, 0]


def test_default_file_from_before_versions_is_timed_again(tmp_path) -> None:
    """The library in a folder of its own, beside the file an earlier build's
    tuner left there."""
    shutil.copy(ROOT / "darcy_cpp_gb300" / "libdarcy_gpu.so", tmp_path)
    (tmp_path / "_build").mkdir()
    file = tmp_path / "_build" / "autotune.json"
    file.write_text(json.dumps({key(): [992, 0]}))
    np.save(tmp_path / "a.npy", np.stack([two_phase(16, seed=1)] * COUNT))
    program = ("import os, sys, pathlib, numpy as np\n"
               "os.environ.pop('DARCY_GPU_TUNE_FILE', None)\n"
               "from darcy_cpp_gb300 import capi\n"
               "folder = pathlib.Path(sys.argv[1])\n"
               "capi.LIB_PATH = folder / 'libdarcy_gpu.so'\n"
               "assert capi.Context().solve_batch(np.load(folder / 'a.npy'), form='mixed')['converged'].all()\n")
    subprocess.run([sys.executable, "-c", program, str(tmp_path)], check=True, cwd=ROOT)
    saved = json.loads(file.read_text())[key()]
    assert saved[:2] != [992, 0] and len(saved) == 3
