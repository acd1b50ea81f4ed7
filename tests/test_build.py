"""When the native host path is built again."""
import os

from tilus_b200 import build


def test_native_is_built_again_for_another_torch_or_abi(monkeypatch, tmp_path):
    """A binary made for another torch or interpreter does not load, however new it is; a change of the C ABI's header
    makes it stale too."""
    made = []

    class Done:
        returncode, stdout, stderr = 0, "", ""

    def compiler(cmd, **kw):
        made.append(cmd)
        open(build.NATIVE, "w").close()
        return Done

    header = tmp_path / "b200q.h"
    header.write_text("")
    monkeypatch.setattr(build, "NATIVE", str(tmp_path / "_native.so"))
    monkeypatch.setattr(build, "NATIVE_STAMP", str(tmp_path / "_native.stamp"))
    monkeypatch.setattr(build, "HEADER", str(header))
    monkeypatch.setattr(build.subprocess, "run", compiler)
    build.build_native()
    build.build_native()
    assert len(made) == 1
    stamp = open(build.NATIVE_STAMP).read()
    open(build.NATIVE_STAMP, "w").write(stamp.replace("torch ", "torch 0."))
    build.build_native()
    assert len(made) == 2 and open(build.NATIVE_STAMP).read() == stamp
    later = os.path.getmtime(build.NATIVE) + 10
    os.utime(header, (later, later))
    build.build_native()
    assert len(made) == 3
