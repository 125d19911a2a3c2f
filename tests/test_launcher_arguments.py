"""Argument checks of the kernel launchers that need no GPU: nothing is launched."""
import subprocess
import sys
from pathlib import Path

import pytest

from layerstorm_b200.ops import _native as nat

ROOT = Path(__file__).resolve().parent.parent

pytestmark = pytest.mark.skipif(not nat.available(), reason="kernel library not built")


def _alone(code):
    """In a process of its own, as a division by zero would end it."""
    r = subprocess.run([sys.executable, "-c", "from layerstorm_b200.ops import _native as n; " + code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stderr[-500:])
    return r.stdout.split()


@pytest.mark.parametrize("N,K", [(16384, 1024), (512, 256)])
def test_no_rows_over_fp8_weights_are_no_work(N, K):
    assert _alone(f"print(n.load().lsb_gemv_fp8b(4096, 4096, 4096, 4096, None, 0, {N}, {K}, {K}, {N}, 1.0, 0, None, None) != -1)") == ["True"]


@pytest.mark.parametrize("half", ["gateup", "down"])
def test_no_groups_of_fp8_experts_are_refused(half):
    mid = {"gateup": "4096, 4, 0, 0.0, None, 0", "down": "4096, 0, 0"}[half]
    assert _alone("import ctypes; from layerstorm_b200.models.device_model import expert_layout; ef = expert_layout('fp8_e4m3', 1024, 512); "
                  f"print(n.load().lsb_moe_{half}(4096, 4096, 4096, ctypes.addressof(ef), 4096, 4096, 4096, 4096, {mid}, None) != 0)") == ["True"]
