"""When the compiled parts are rebuilt, and what happens when that fails (no GPU needed)."""
import os
import shutil
import subprocess

import pytest
import torch

from ecml23_sparse_b200 import _lib, build


@pytest.fixture
def fresh(monkeypatch):
    build.build_binding()
    monkeypatch.setattr(_lib, "_binding", None)
    return monkeypatch


def test_binding_is_stale_for_another_torch(fresh):
    assert build.binding_torch() == torch.__version__ and not build._binding_stale()
    fresh.setattr(torch, "__version__", "1.0.0")
    assert build._binding_stale()


def test_a_source_that_does_not_compile_is_an_error(fresh, tmp_path):
    """... and not a reason to go on with the module built from the source before it."""
    src, old = tmp_path / "binding.cpp", tmp_path / "_native.so"
    shutil.copy(build.BINDING_PATH, old)
    src.write_text("this is no C++\n")
    os.utime(old, (1, 1))
    fresh.setattr(build, "BINDING_SRC", str(src))
    fresh.setattr(build, "BINDING_PATH", str(old))
    with pytest.raises(subprocess.CalledProcessError):
        _lib.binding()


@pytest.mark.parametrize("for_this_torch", [True, False])
def test_without_a_compiler_the_shipped_module_serves_its_own_torch(fresh, for_this_torch):
    def missing(*args, **kwargs):
        raise build.CompilerMissing("none here")

    fresh.setattr(build, "build_binding", missing)
    if for_this_torch:
        assert hasattr(_lib.binding(), "forward")
    else:
        fresh.setattr(torch, "__version__", "1.0.0")
        with pytest.raises(ImportError):
            _lib.binding()
