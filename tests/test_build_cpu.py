"""What the build makes with and without torch; the compilers are replaced by a recorder, nothing is compiled."""
import os
import subprocess
import sys
import types

import pytest

from flashbias_b200 import build as fb_build


@pytest.fixture
def recorder(monkeypatch, tmp_path):
    made = []

    def run(cmd, **_):
        out = cmd[cmd.index("-o") + 1]
        made.append(os.path.basename(out))
        with open(out, "w") as f:
            f.write("built")
        return types.SimpleNamespace(returncode=0, stdout="", stderr="")

    monkeypatch.setattr(fb_build, "LIB", str(tmp_path / "libflashbias_b200.so"))
    monkeypatch.setattr(fb_build, "TORCH_OP", str(tmp_path / "_torch_op.so"))
    monkeypatch.setattr(fb_build, "OBJ", str(tmp_path / "build"))
    monkeypatch.setattr(fb_build, "_nvcc", lambda: "nvcc")
    monkeypatch.setattr(subprocess, "run", run)
    return made


def test_the_c_library_is_built_without_torch(recorder, monkeypatch):
    with monkeypatch.context() as m:
        m.setitem(sys.modules, "torch", None)  # any import of torch raises ImportError
        assert fb_build.build() == fb_build.LIB
    assert "libflashbias_b200.so" in recorder and "_torch_op.so" not in recorder
    recorder.clear()
    fb_build.build()  # with torch: the extension is added, the library is not built again
    assert recorder == ["_torch_op.so"]


def test_nothing_is_built_twice(recorder):
    fb_build.build()
    recorder.clear()
    fb_build.build()
    assert recorder == []
    fb_build.build(force=True)
    assert "libflashbias_b200.so" in recorder and "_torch_op.so" in recorder
