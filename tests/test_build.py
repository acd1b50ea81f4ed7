"""When the native host path is built again, and what the kernels are built to."""
import os
import re
import subprocess

import pytest

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


@pytest.mark.parametrize("var", [2, 7, 13])
def test_two_ctas_of_the_small_batch_kernel_have_registers_on_an_sm(var, tmp_path):
    """Up to 32 rows its launches are planned to share SMs with the next launch of the stream: two CTAs of 512 threads have
    65536 registers, 64 each (2-, 4- and 7-bit integers; which types take more is said at batch_stages)."""
    cmd = [build._nvcc(), "-Xptxas", "-v", *build.NVCC_FLAGS, "-DB200Q_NPARTS=64", f"-DB200Q_PART={var}", "-c",
           os.path.join(build.CSRC, "batch_kernel.cu"), "-o", str(tmp_path / "batch.o")]
    log = subprocess.run(cmd, capture_output=True, text=True, check=True).stderr
    used = [int(r) for r in re.findall(r"batch_kernel.*?Used (\d+) registers", log, re.S)]
    assert len(used) == 2 and max(used) <= 64, used  # fp16, bf16
