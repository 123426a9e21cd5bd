"""_host.so links torch's C++ internals: it says which torch and python it was built for, a build replaces one that was made
for others, and the loader refuses it before it loads it."""
import os
import shutil

import pytest

from open_ommx_serve_b200 import _lib, build


@pytest.fixture
def foreign(tmp_path):
    """A copy of the built module that says it was built for another torch."""
    path = str(tmp_path / "_host.so")
    with open(_lib.HOST_PATH, "rb") as f:
        data = f.read()
    here = _lib.host_target().encode()
    other = here.replace(b"torch ", b"TORCH ")
    assert data.count(_lib.HOST_MARK + here) == 1
    with open(path, "wb") as f:
        f.write(data.replace(_lib.HOST_MARK + here, _lib.HOST_MARK + other))
    return path


def test_the_module_says_what_it_was_built_for():
    import torch
    assert _lib.host_built_for() == _lib.host_target() and torch.__version__ in _lib.host_target()


def test_a_module_of_another_torch_is_refused_unloaded(foreign, monkeypatch):
    monkeypatch.setattr(_lib, "_HOST", None)
    monkeypatch.setattr(_lib, "HOST_PATH", foreign)
    with pytest.raises(RuntimeError, match="built for TORCH .*this is torch .*rebuild"):
        _lib.host()
    assert _lib._HOST is None
    monkeypatch.undo()
    assert _lib.host() is not None


@pytest.mark.parametrize("make", ["foreign", "silent", "same"])
def test_a_build_replaces_it(foreign, make, monkeypatch):
    if make == "silent":                                    # a module from before the text was put in
        with open(foreign, "rb") as f:
            data = f.read()
        with open(foreign, "wb") as f:
            f.write(data.replace(_lib.HOST_MARK, b"x" * len(_lib.HOST_MARK)))
        assert _lib.host_built_for(foreign) == ""
    elif make == "same":
        shutil.copy(_lib.HOST_PATH, foreign)
    os.utime(foreign)                                       # newer than its sources
    ran = []
    monkeypatch.setattr(build, "HOST_LIB", foreign)
    monkeypatch.setattr(build, "_run", lambda cmd: ran.append(cmd) or "")
    build.build_host()
    assert len(ran) == (0 if make == "same" else 1)
    if ran:
        assert any(_lib.host_target() in arg for arg in ran[0])
