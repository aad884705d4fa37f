"""Saved choices of the matrix products and the size of their kernel's ring, without a GPU."""
import os
import subprocess
import sys

import pytest
import torch

from llmserver_b200.ops import gemm_bf16
from llmserver_b200.ops.library import KernelError

KEY = (8, 4096, 4096, torch.bfloat16)
HEADER = "# row bucket,N,K,output,split of K (0: library product)"


@pytest.fixture
def choices(monkeypatch):
    monkeypatch.setattr(gemm_bf16, "_choice", {})
    return gemm_bf16


def test_what_is_written_is_read(choices, monkeypatch, tmp_path):
    path = str(tmp_path / "plan")
    gemm_bf16._choice.update({KEY: 6, (64, 128, 256, gemm_bf16.OWN_KERNEL): 3, (1, 151936, 4096, torch.float32): 1})
    gemm_bf16.save_plan(path)
    saved = dict(gemm_bf16._choice)
    gemm_bf16._choice.clear()
    assert gemm_bf16.load_plan(path) == 3 and gemm_bf16._choice == saved


@pytest.mark.parametrize("header,count", [(HEADER, 0), (HEADER + ", revision 1", 0), ("# mine", 1), (None, 1)])
def test_choices_of_other_kernels_are_not_read(choices, tmp_path, header, count):
    path = tmp_path / "plan"
    path.write_text("".join(line + "\n" for line in (header, "8,4096,4096,bf16,6") if line))
    assert gemm_bf16.load_plan(str(path)) == count
    assert gemm_bf16._choice == ({KEY: 6} if count else {})


def test_lines_that_are_no_choices_are_refused(choices, tmp_path):
    path = tmp_path / "plan"
    path.write_text("8,4096,4096\n")
    with pytest.raises(KernelError):
        gemm_bf16.load_plan(str(path))


@pytest.mark.parametrize("asked,want", [(None, [200, 100, 74]), ("64", [64, 64, 64]), ("120", [120, 120, 74]), ("8", [32, 32, 32]), ("999", [200, 200, 74])])
def test_ring_size_that_was_asked_for(asked, want):
    """LLMSERVER_B200_GEMM_RING_KIB holds for blocks that have an SM to themselves, share it with one other, and with two (as far as
    three fit)."""
    script = "from llmserver_b200.ops.library import library; print([library().llm_gemm_small_m_ring_kib(n) for n in (1, 2, 3)])"
    env = {key: value for key, value in os.environ.items() if key != "LLMSERVER_B200_GEMM_RING_KIB"}
    if asked is not None:
        env["LLMSERVER_B200_GEMM_RING_KIB"] = asked
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    done = subprocess.run([sys.executable, "-c", script], capture_output=True, text=True, cwd=root, env=dict(env, PYTHONPATH=root), timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
    assert done.stdout.split("\n")[-2] == str(want)
