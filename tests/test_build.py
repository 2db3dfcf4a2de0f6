"""The in-tree build (nvcc and g++ run here without a GPU)."""
import os
import shutil

import build
import pytest


@pytest.mark.parametrize("name", ["path", "name"])
def test_cuda_headers_are_found_for_any_form_of_NVCC(monkeypatch, name):
    nvcc = shutil.which(build.NVCC)
    if name == "name":  # as NVCC=nvcc in the environment, which the nvcc steps take through PATH
        monkeypatch.setenv("PATH", os.path.dirname(nvcc) + os.pathsep + os.environ["PATH"])
        nvcc = os.path.basename(nvcc)
    monkeypatch.setattr(build, "NVCC", nvcc)
    assert os.path.exists(os.path.join(build._cuda_include(), "cuda_runtime_api.h"))
