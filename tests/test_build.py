"""The in-tree build (nvcc and g++ run here without a GPU)."""
import importlib.util
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


@pytest.mark.parametrize("torch_there", [False, True])
def test_the_library_alone_needs_no_torch(monkeypatch, torch_there):
    def no_host(force):
        raise AssertionError("the host module was built")

    monkeypatch.setattr(build, "_build_host", no_host)
    if torch_there:
        assert build.build(host=False) == build.OUT
        with pytest.raises(AssertionError):
            build.build()
    else:
        find = importlib.util.find_spec
        monkeypatch.setattr(importlib.util, "find_spec", lambda name, *a: None if name == "torch" else find(name, *a))
        assert build.build() == build.OUT


def test_the_host_module_is_stale_for_another_torch_or_python(monkeypatch):
    import sysconfig
    import torch
    build.build()
    assert not build._host_stale()
    with monkeypatch.context() as m:
        m.setattr(torch, "__version__", "0.0.1")
        assert build._host_stale()
    with monkeypatch.context() as m:
        m.setattr(sysconfig, "get_config_var", lambda name: "cpython-300")
        assert build._host_stale()
    assert not build._host_stale()
