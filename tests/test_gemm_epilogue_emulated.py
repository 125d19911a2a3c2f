"""The epilogue of the tensor-core GEMM under waits that give up in some warps and not in others, its source run on the CPU (no GPU is made to wait)."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_no_warp_is_left_waiting_where_another_gave_up(tmp_path):
    source = (ROOT / "layerstorm_b200/csrc/kernels/gemm_tc.cu").read_text()
    start = source.index("// ---------------- epilogue ----------------")
    (tmp_path / "epilogue_body.inc").write_text(source[start: source.index("} else if (ok) {", start)] + "}\n")
    exe = tmp_path / "emu"
    subprocess.run(["g++", "-O1", "-std=c++20", "-pthread", "-I", str(tmp_path), str(ROOT / "tests/simt_emu/gemm_epilogue_emu.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "bad=0" in r.stdout, r.stdout
