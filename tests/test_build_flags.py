"""The build refuses __shared__ variables whose type's constructor does something (a Tan pair's sets it to
zero): CUDA does not initialise them once per block, and each thread running the constructor at its own time
would race with the others' values."""
import os
import shutil
import subprocess

import pytest

from cosmolattice_b200 import build

CSRC = os.path.join(os.path.dirname(os.path.abspath(build.__file__)), "csrc")


@pytest.mark.skipif(shutil.which(os.environ.get("NVCC", "nvcc")) is None, reason="needs nvcc")
@pytest.mark.parametrize("type_,compiles", [("double", True), ("clb::Tan<double>", False)])
def test_shared_variables_have_no_constructor(tmp_path, type_, compiles):
    src = tmp_path / "t.cu"
    src.write_text('#include "clb_tangent.cuh"\n__global__ void k(double *o)\n{\n'
                   f"  __shared__ {type_} x[32];\n  o[threadIdx.x] = (double)sizeof(x);\n}}\n")
    r = subprocess.run([os.environ.get("NVCC", "nvcc"), *build.NVCC_FLAGS, f"-I{CSRC}", "-c", str(src), "-o", str(tmp_path / "t.o")],
                       capture_output=True, text=True, timeout=300)
    assert (r.returncode == 0) == compiles, r.stderr
    if not compiles:
        assert "dynamic initialization" in r.stderr, r.stderr
