"""The build rejects code that drops the error of a launch helper: a captured
graph would otherwise lack the kernels of a helper that failed."""
import re
import subprocess

import pytest

from perft_gpu_2026_b200 import build


def compiles(tmp_path, text):
    src = tmp_path / "snippet.cu"
    src.write_text(text)
    cmd = [build._nvcc()] + build.NVCC_FLAGS + ["-o", str(tmp_path / "snippet.so"), str(src)]
    return subprocess.run(cmd, capture_output=True, text=True).returncode == 0


def test_dropped_errors_do_not_build(tmp_path):
    kept = "#include <cuda_runtime.h>\n[[nodiscard]] cudaError_t f();\ncudaError_t g() { return f(); }\n"
    assert compiles(tmp_path, kept)
    assert not compiles(tmp_path, kept.replace("return f(); }", "f(); return cudaSuccess; }"))


@pytest.mark.parametrize("name", ["reset_counters", "launch_fold_kernel", "launch_fold_t", "launch_fold",
                                  "launch_tt_fold_t", "launch_tt_fold"])
def test_launch_helpers_return_errors_that_cannot_be_dropped(name):
    with open(build.CSRC + "/pb_engine.cu") as f:
        text = f.read()
    heads = re.findall(r"^.*cudaError_t %s\(pb_ctx" % name, text, re.M)
    assert len(heads) == 1 and heads[0].startswith("[[nodiscard]]"), heads
