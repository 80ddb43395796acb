"""The weight gradient's shared-memory layout holds 16, 32 or 64 channels; another
count does not compile (its chunk permutation would leave the voxel)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "3d_droplet_simulation_2007_gb300", "csrc")
USE = """
namespace dsg { namespace nn {
cudaError_t other(const bf16 *X, const bf16 *G, float *dW) { return wgrad_launch<%d, %d>(X, G, dW, 8, 8, 8, nullptr); }
} }
"""


@pytest.mark.parametrize("cin,cout", [(48, 16), (16, 48)])
def test_other_counts_do_not_compile(tmp_path, cin, cout):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("needs nvcc")
    with open(os.path.join(CSRC, "nn.cu")) as f:
        src = f.read()
    path = tmp_path / "nn_other.cu"
    path.write_text(src + USE % (cin, cout))
    r = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-I" + CSRC,
                        "-I" + os.path.join(ROOT, "include"), "-c", str(path), "-o", str(tmp_path / "nn.o")],
                       capture_output=True, text=True)
    assert r.returncode != 0 and "16, 32 or 64 channels" in r.stderr
