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


@pytest.mark.parametrize("rows", [1, 2, 40])
def test_per_head_products_of_a_latent_layer_report_to_the_error_word(rows, monkeypatch):
    """Query absorption and value up-projection run on a pipelined product whose waits are bounded: the layer hands them the word that the engine reads behind a step,
    and the launcher hands it on."""
    from types import SimpleNamespace
    from unittest.mock import MagicMock

    from layerstorm_b200.models import device_model as dm

    seen, word = [], object()

    def call(name, *args):
        assert len(args) == len(nat.SIGS[name][0]), name
        seen.append((name, args))
    monkeypatch.setattr(dm.nat, "call", call)
    monkeypatch.setattr(dm.TcScratch, "get", classmethod(lambda cls, device: SimpleNamespace(err=word)))
    cfg = SimpleNamespace(kv_lora=512, qk_rope=64, qk_nope=128, v_head=128, q_lora=1536, index_head_dim=0, index_n_heads=0, has_indexer=False, index_kpool=1, rms_eps=1e-6,
                          softmax_scale=0.1)
    me = MagicMock(cfg=cfg, Hh=16, max_proj=4096, max_qb=4096, max_pages=4, page=64, kv_fmt="fp8", dcp=None, row_tier=None)
    L = {"mla_in": MagicMock(), "mla_qb": MagicMock(), "mla_o": MagicMock(), "qa_norm": 0, "kv_norm": 0, "k_b": "k_b", "v_b": "v_b"}
    dm.DeviceModel._mla(me, 0, L, MagicMock(NS=4), rows)
    products = [a for n, a in seen if L["k_b"] in a or L["v_b"] in a]
    assert len(products) == 2 and all(a[-1] is word for a in products)
    source = (ROOT / "layerstorm_b200/csrc/kernels/mla.cu").read_text()
    calls = [c.split(";")[0] for c in source.split("= lsb_gemm_bf16_tc_batched(")[1:]]
    assert calls and all(c.endswith("err, stream)") for c in calls)


@pytest.mark.parametrize("given,alone,peers", [(None, 5, 8), ("", 5, 8), ("8", 8, 8), ("3", 3, 3), ("0", 0, 0)])
def test_the_row_limit_of_the_cluster_kernel_is_taken_as_given(given, alone, peers):
    import os
    env = {k: v for k, v in os.environ.items() if k != "LSB_MHC_CLUSTER_MAX_ROWS"} | ({} if given is None else {"LSB_MHC_CLUSTER_MAX_ROWS": given})
    code = "from layerstorm_b200.models import device_model as m; print(m.mhc_cluster_rows(False), m.mhc_cluster_rows(True))"
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.stdout.split() == [str(alone), str(peers)], r.stderr[-500:]
