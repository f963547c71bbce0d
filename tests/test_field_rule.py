"""The flip terms and counter adders the kernels use equal the acceptance rule
and a plain count on every spin/bond-count combination, with the draws at every
edge of every table."""
import pathlib
import shutil
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


def _build(tmp_path):
    exe = tmp_path / "field_rule_check"
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17",
                    f"-I{ROOT / 'spin-glass_b200' / 'csrc'}", str(ROOT / "tests" / "field_rule_check.cu"),
                    "-o", str(exe)], check=True, capture_output=True, timeout=600)
    return exe


@pytest.mark.gpu
def test_flip_terms_match_the_acceptance_rule(tmp_path):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    out = subprocess.run([str(_build(tmp_path))], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    words = out.stdout.split()
    assert int(words[1]) == 2000 * 30
    assert [int(w) for w in words[3::2]] == [0, 0, 0, 0], out.stdout
