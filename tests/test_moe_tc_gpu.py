"""Tensor-core grouped expert FFN (sort -> gather -> gate/up+SwiGLU -> down) against an fp32
PyTorch reference built from the same (de-quantised) expert slots."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _setup(fmt, H, F, E, n_missing, seed, size=1.0):
    """``size``: factor on the gate and up matrices."""
    from layerstorm_b200.models.device_model import ExpertArena, QLinear, expert_layout
    dev = torch.device("cuda")
    g = torch.Generator(device="cpu").manual_seed(seed)
    ef = expert_layout(fmt, H, F)
    arena = ExpertArena(ef, E - n_missing, E, dev)
    ref = {}
    slot = 0
    for e in range(E):
        if e < n_missing:
            continue                                   # experts 0..n_missing-1 are not resident
        mats = [torch.randn(F, H, generator=g) * 0.05 * size, torch.randn(F, H, generator=g) * 0.05 * size, torch.randn(H, F, generator=g) * 0.05]
        arena.write_expert(slot, *(QLinear.from_float(m.to(dev), fmt, dev) for m in mats))
        arena.slot_of[e] = slot
        ref[e] = [m.double().cpu() for m in arena.read_expert(slot, fmt)]
        slot += 1
    return arena, ref


@pytest.mark.parametrize("fmt", ["nvfp4", "fp8_e4m3", "bf16", "gguf_q4_k"])
@pytest.mark.parametrize("BN,R", [(32, 40), (64, 150), (128, 300)])
def test_grouped_ffn_matches_reference(fmt, BN, R):
    from layerstorm_b200.ops import _native as nat
    dev = torch.device("cuda")
    H, F, E, S, limit = 256, (256 if fmt == "gguf_q4_k" else 128), 6, 3, 7.0
    arena, ref = _setup(fmt, H, F, E, n_missing=1, seed=1)
    g = torch.Generator(device="cpu").manual_seed(2)
    x = (torch.randn(R, H, generator=g) * 1.5).to(torch.bfloat16).to(dev)
    # skewed routing: expert E-1 gets every row (like a shared expert), the others are random; a few invalid ids
    ids = torch.stack([torch.randint(0, E - 1, (R,), generator=g), torch.randint(0, E - 1, (R,), generator=g), torch.full((R,), E - 1)], 1).int()
    ids[3, 0] = -1
    ids = ids.to(dev).contiguous()
    P = R * S
    i32 = dict(dtype=torch.int32, device=dev)
    tiles = P // BN + E + 1
    srt, te, tr, tn, cnt = (torch.zeros(P, **i32), torch.zeros(tiles, **i32), torch.zeros(tiles, **i32), torch.zeros(tiles, **i32), torch.zeros(2, **i32))
    xs = torch.zeros(P, H, dtype=torch.float16, device=dev)
    act = torch.zeros(P, F, dtype=torch.float16, device=dev)
    y = torch.full((P, H), float("nan"), device=dev)
    err, miss = torch.zeros(1, **i32), torch.zeros(1, **i32)
    efp = ctypes.addressof(arena.ef)
    for _ in range(2):                                  # twice: barriers, TMEM and scratch are reusable
        nat.call("lsb_moe_tc_sort", ids, P, E, BN, srt, te, tr, tn, cnt)
        nat.call("lsb_moe_tc_gather", x, srt, cnt, xs, P, S, H)
        nat.call("lsb_moe_tc_ffn", 1, xs, P, arena.data, arena.slot_of, efp, te, tr, tn, cnt, srt, act, BN, tiles, limit, miss, err, None)
        nat.call("lsb_moe_tc_ffn", 0, act, P, arena.data, arena.slot_of, efp, te, tr, tn, cnt, srt, y, BN, tiles, 0.0, None, err, None)
    torch.cuda.synchronize()
    assert int(err) == 0
    assert int(miss) == 1                               # expert 0 (+1) was routed to but is not resident
    n_valid = int((ids >= 0).sum())
    assert int(cnt[1]) == n_valid
    # the sort is a permutation of the valid pairs, grouped by expert
    sp = srt[:n_valid].cpu()
    assert sorted(sp.tolist()) == [i for i in range(P) if int(ids.view(-1)[i]) >= 0]
    es = ids.view(-1).cpu()[sp]
    assert torch.all(es[1:] >= es[:-1])
    # numerics
    xd = x.double().cpu()
    idc = ids.cpu()
    worst = 0.0
    for r in range(R):
        for s in range(S):
            e = int(idc[r, s])
            if e < 1:
                continue
            gate, up, down = ref[e]
            gv = torch.clamp(gate @ xd[r], max=limit)
            uv = torch.clamp(up @ xd[r], -limit, limit)
            want = down @ (torch.nn.functional.silu(gv) * uv)
            got = y[r * S + s].double().cpu()
            worst = max(worst, float((got - want).abs().max() / (want.abs().max() + 1e-6)))
    assert worst < 6e-3, worst


def test_engine_prefill_uses_grouped_path_and_matches_oracle():
    """Long enough chunks => the routed experts run on the tensor-core path; logits still match the fp32 oracle
    and the short-chunk (weight-streaming) path."""
    from layerstorm_b200.models.config import get_preset
    from layerstorm_b200.models.device_model import DeviceModel, TC_MOE_MIN_ROWS
    from layerstorm_b200.models.reference import Oracle
    from layerstorm_b200.models.weights import init_weights
    from layerstorm_b200.runtime.engine import Engine
    for name, eq in (("tiny-mla-moe", "bf16"), ("tiny-glm5-next", "nvfp4")):
        cfg = get_preset(name)
        m = DeviceModel.from_state_dict(cfg, init_weights(cfg, 5), "cuda", kv_fmt="bf16", page=16, expert_quant=eq)
        oracle = Oracle(cfg, m.effective_state_dict())
        g = torch.Generator().manual_seed(0)
        T = 30
        prompt = torch.randint(0, cfg.vocab, (T,), generator=g)
        want = oracle.forward(prompt)[T - 1]
        outs = []
        for chunk in (64, 8):                           # 64: one tensor-core chunk; 8: GEMV chunks
            assert (chunk >= TC_MOE_MIN_ROWS) == (chunk == 64)
            eng = Engine(m, max_seqs=2, max_ctx=256, prefill_chunk=chunk, use_graph=False)
            sid = eng.create_sequence()
            nxt, lg = eng.prefill(sid, prompt.tolist(), want_logits=True)
            assert nxt == int(want.argmax()), (name, chunk)
            assert float((lg - want).abs().max() / want.abs().max()) < 3e-2, (name, chunk)
            outs.append(lg)
            eng.free_sequence(sid)
        assert float((outs[0] - outs[1]).abs().max() / outs[1].abs().max()) < 2e-2


@pytest.mark.parametrize("fmt,H,F", [("nvfp4", 128, 128), ("nvfp4", 384, 640), ("nvfp4", 1152, 128), ("fp8_e4m3", 128, 384), ("fp8_e4m3", 640, 128), ("bf16", 128, 384),
                                     ("bf16", 1152, 128), ("gguf_q4_k", 256, 768), ("gguf_q4_k", 1280, 256)])
@pytest.mark.parametrize("BN", [32, 64, 128])
def test_widths_that_end_inside_boxes_and_operand_stages(fmt, H, F, BN):
    """Reduction lengths shorter than a weight box, that end inside one, inside an operand stage, and that wrap the rings."""
    from layerstorm_b200.ops import _native as nat
    dev = torch.device("cuda")
    E, R = 20, 2 * BN + 1
    arena, ref = _setup(fmt, H, F, E, n_missing=0, seed=3)
    g = torch.Generator(device="cpu").manual_seed(4)
    x = torch.randn(R, H, generator=g).to(torch.bfloat16).to(dev)
    ids = torch.stack([torch.full((R,), E - 1), torch.arange(R) % (E - 1)], 1).int().to(dev).contiguous()
    P, tiles = R * 2, R * 2 // BN + E + 1
    i32 = dict(dtype=torch.int32, device=dev)
    srt, te, tr, tn, cnt, err = (torch.zeros(n, **i32) for n in (P, tiles, tiles, tiles, 2, 1))
    xs, act = torch.zeros(P, H, dtype=torch.float16, device=dev), torch.zeros(P, F, dtype=torch.float16, device=dev)
    y = torch.full((P, H), float("nan"), device=dev)
    efp = ctypes.addressof(arena.ef)
    nat.call("lsb_moe_tc_sort", ids, P, E, BN, srt, te, tr, tn, cnt)
    nat.call("lsb_moe_tc_gather", x, srt, cnt, xs, P, 2, H)
    nat.call("lsb_moe_tc_ffn", 1, xs, P, arena.data, arena.slot_of, efp, te, tr, tn, cnt, srt, act, BN, tiles, 0.0, None, err, None)
    nat.call("lsb_moe_tc_ffn", 0, act, P, arena.data, arena.slot_of, efp, te, tr, tn, cnt, srt, y, BN, tiles, 0.0, None, err, None)
    torch.cuda.synchronize()
    assert int(err) == 0
    xd, idc, got = x.double().cpu(), ids.cpu(), y.double().cpu()
    for e in range(E):
        gate, up, down = ref[e]
        r, k = (idc == e).nonzero(as_tuple=True)
        want = (torch.nn.functional.silu(xd[r] @ gate.T) * (xd[r] @ up.T)) @ down.T
        # a hidden value rounded to fp16, at most 2^-11 relative per term (NVFP4 weights, bf16 weights of this size and FP8 weights with power-of-two block scales,
        # as `_setup` makes them, are exact in fp16).  Q4_K weights are d sc v - dmin m
        # with both products rounded to fp16, 2^-11 of terms up to 15 d sc and 8 d sc in size around weights of 4.6 d sc rms: 2.4e-3 at most
        assert float((got[r * 2 + k] - want).norm() / want.norm()) < (3e-3 if fmt == "gguf_q4_k" else 1e-3), e


@pytest.mark.parametrize("fmt,first", [("bf16", 3), ("fp8_e4m3", 16), ("nvfp4", 16), ("gguf_q4_k", 16)])
def test_steps_of_few_rows(fmt, first, monkeypatch):
    """Both sides of the row count from which a format's experts run on the grouped kernel and (NVFP4: 12 rows of 6 pairs) from which they run in groups, an id
    that takes no part among them."""
    from layerstorm_b200.models import device_model
    from layerstorm_b200.models.device_model import ModelBase, MoeBuffers
    monkeypatch.setattr(device_model, "TC_MOE_BF16_BYTES", 0)
    dev = torch.device("cuda")
    H, F, E, S = 256, 256, 9, 6
    arena, ref = _setup(fmt, H, F, E, n_missing=0, seed=5)
    m = ModelBase()
    m.device, m.tp_size, m.expert_shard = dev, 1, "ep"
    z = lambda *s, dtype=torch.float32: torch.zeros(*s, dtype=dtype, device=dev)
    for R in sorted({1, 2, first - 1, first, 12, 13, 15, 16}):
        g = torch.Generator(device="cpu").manual_seed(R)
        x = torch.randn(R, H, generator=g).to(torch.bfloat16).to(dev)
        ids = torch.stack([torch.randperm(E, generator=g)[:S] for _ in range(R)])
        mb = MoeBuffers()
        mb.alloc_moe(z, R, S, E, E, H, F, tc=True)
        mb.tc_xs, mb.tc_act = z(R * S, H, dtype=torch.float16), z(R * S, F, dtype=torch.float16)
        mb.ids.copy_(ids.int())
        mb.ids[R - 1, 2] = -1
        assert (m.moe_mode(arena, mb, R) == "tc") == (R >= first)
        mb.bs_ok = True                                  # block-scaled steps of few rows stay on the streaming kernels
        assert (m.moe_mode(arena, mb, R) == "tc") == (R >= 16)
        mb.bs_ok = False
        m.moe_prepare(arena, mb, x, R, E)
        m.moe_experts(arena, mb, x, R, E, 0.0, mb.miss)
        got, xd = mb.y.view(R, S, H).double().cpu(), x.double().cpu()
        for r in range(R):
            for k in range(S):
                if (r, k) == (R - 1, 2):
                    continue
                gate, up, down = ref[int(ids[r, k])]
                want = down @ (torch.nn.functional.silu(gate @ xd[r]) * (up @ xd[r]))
                # a hidden value in bf16 (2^-9 at most, averaged out) on the streaming kernels; Q4_K weights as above
                assert float((got[r, k] - want).norm() / want.norm()) < 4e-3, (R, r, k)
        assert int(mb.miss) == 0


@pytest.mark.parametrize("fmt,rows", [("fp8_e4m3", (1, 2, 9, 15)), ("gguf_q4_k", (1, 2, 9, 15)), ("bf16", (1, 2, 3, 9, 15))])
def test_steps_of_few_rows_keep_the_range_of_bf16(fmt, rows, monkeypatch):
    """Hidden values of about 1e6, FP8 block scales that are no powers of two and above 0.57 (where 256 of them times 448 passes fp16's largest number), and a
    row of activations beyond it (bf16 experts: on the grouped kernel with bf16 hidden values from 3 rows)."""
    from layerstorm_b200.models import device_model
    from layerstorm_b200.models.device_model import ModelBase, MoeBuffers
    monkeypatch.setattr(device_model, "TC_MOE_BF16_BYTES", 0)
    dev = torch.device("cuda")
    H, F, E, S = 256, 256, 9, 6
    arena, ref = _setup(fmt, H, F, E, n_missing=0, seed=9, size=2000.0)
    if fmt == "fp8_e4m3":
        for e in range(E):
            for off in (arena.ef.off_sg, arena.ef.off_su, arena.ef.off_sd):
                sc = arena.data[e][off: off + 16].view(torch.float32)
                sc *= 1.37
            assert float(arena.data[e][arena.ef.off_sg:][:16].view(torch.float32).min()) > 0.57
            ref[e] = [w.double().cpu() for w in arena.read_expert(e, fmt)]
    m = ModelBase()
    m.device, m.tp_size, m.expert_shard = dev, 1, "ep"
    z = lambda *s, dtype=torch.float32: torch.zeros(*s, dtype=dtype, device=dev)
    for R in rows:
        g = torch.Generator(device="cpu").manual_seed(R)
        x = torch.randn(R, H, generator=g)
        x[R - 1] *= 1e5
        x = x.to(torch.bfloat16).to(dev)
        ids = torch.stack([torch.randperm(E, generator=g)[:S] for _ in range(R)])
        mb = MoeBuffers()
        mb.alloc_moe(z, R, S, E, E, H, F, tc=True)
        mb.tc_xs, mb.tc_act = z(R * S, H, dtype=torch.float16), z(R * S, F, dtype=torch.float16)
        mb.ids.copy_(ids.int())
        m.moe_prepare(arena, mb, x, R, E)
        m.moe_experts(arena, mb, x, R, E, 0.0, mb.miss)
        got, xd = mb.y.view(R, S, H).double().cpu(), x.double().cpu()
        for r in range(R):
            for k in range(S):
                gate, up, down = ref[int(ids[r, k])]
                want = down @ (torch.nn.functional.silu(gate @ xd[r]) * (up @ xd[r]))
                # fp32 sums and a hidden value in bf16: 2^-9 of it at most, averaged out over 256 of them
                assert float((got[r, k] - want).norm() / want.norm()) < 4e-3, (R, r, k)


@pytest.mark.parametrize("fmt", ["nvfp4", "fp8_e4m3", "gguf_q4_k"])
def test_a_row_of_few_gets_the_same_experts_outputs_in_any_company(fmt):
    """Bit for bit, whatever the other rows of the step are: a draft's rows are checked together and were answered one by one."""
    from layerstorm_b200.models.device_model import ModelBase, MoeBuffers
    dev = torch.device("cuda")
    H, F, E, S, most = 256, 512, 20, 8, 15
    arena, _ = _setup(fmt, H, F, E, n_missing=0, seed=12)
    m = ModelBase()
    m.device, m.tp_size, m.expert_shard = dev, 1, "ep"
    z = lambda *s, dtype=torch.float32: torch.zeros(*s, dtype=dtype, device=dev)
    g = torch.Generator(device="cpu").manual_seed(13)
    x = torch.randn(most, H, generator=g).to(torch.bfloat16).to(dev)
    ids = torch.stack([torch.randperm(E, generator=g)[:S] for _ in range(most)]).int()
    alone = None
    for R in (1, 2, 5, 9, 10, 12, 15):
        for first in {0, most - R}:
            mb = MoeBuffers()
            mb.alloc_moe(z, R, S, E, E, H, F, tc=True)
            mb.tc_xs, mb.tc_act = z(R * S, H, dtype=torch.float16), z(R * S, F, dtype=torch.float16)
            mb.ids.copy_(ids[first: first + R])
            rows = x[first: first + R].contiguous()
            m.moe_prepare(arena, mb, rows, R, E)
            m.moe_experts(arena, mb, rows, R, E, 0.0, mb.miss)
            y = mb.y.view(R, S, H)
            if R == 1:
                alone = {**(alone or {}), first: y[0].clone()}
            for row, want in alone.items():
                if first <= row < first + R:
                    assert torch.equal(y[row - first], want), (R, first, row)


@pytest.mark.parametrize("E,H,F,S,slots,first", [(64, 4096, 2048, 8, 64, 3), (64, 4096, 2048, 8, 8, 16), (128, 2048, 768, 8, 128, 9), (8, 4096, 14336, 2, 8, 3),
                                                 (16, 1024, 512, 2, 16, 16), (64, 4096, 2048, 8, 16, 8)])
def test_few_rows_run_grouped_where_their_experts_are_many_bytes(E, H, F, S, slots, first):
    import types
    from layerstorm_b200.models.device_model import ModelBase, expert_layout
    fake = types.SimpleNamespace(ef=expert_layout("bf16", H, F), slot_of=torch.empty(E), n_slots=slots)
    assert [R for R in range(1, 40) if ModelBase.moe_grouped(fake, S, R)] == list(range(first, 40))
    fake.ef = expert_layout("bf16", H, F, gated=False)
    assert not ModelBase.moe_grouped(fake, S, 15) and ModelBase.moe_grouped(fake, S, 16)


def test_steps_of_few_rows_take_no_grouped_buffers(monkeypatch):
    """A workspace whose steps all stream their experts has neither the grouped kernel's buffers nor the block-scaled ones."""
    from layerstorm_b200.models import device_model
    monkeypatch.setattr(device_model, "TC_MOE_BF16_BYTES", 0)
    from layerstorm_b200.models.config import get_preset
    from layerstorm_b200.models.device_model import DeviceModel, Workspace
    from layerstorm_b200.models.weights import init_weights
    cfg = get_preset("tiny-glm5-next")
    w = init_weights(cfg, 5)
    for eq, first in (("nvfp4", 16), ("fp8_e4m3", 16), ("bf16", 3)):
        m = DeviceModel.from_state_dict(cfg, w, "cuda", kv_fmt="bf16", page=16, expert_quant=eq)
        for R in (1, 2, 3, 15, 16):
            ws = Workspace(m, R, 1, 64)
            assert ws.set_block_scaled(True) in (False, R >= 16)
            grouped = [n for n in ("tc_xs", "tc_act", "tc_sorted", "bs_xq", "bs_act") if hasattr(ws, n)]
            assert bool(grouped) == (R >= first and ws.tc_ok), (eq, R, grouped)


@pytest.mark.parametrize("H,F", [(128, 384), (640, 128), (1152, 256)])
@pytest.mark.parametrize("BN", [32, 64, 128])
@pytest.mark.parametrize("scaled", [False, True])
def test_bf16_rows_meet_bf16_experts_directly(H, F, BN, scaled):
    """Reductions of two sub-stages, that end inside an operand stage and that wrap the rings; an expert that is not resident; another gated unit with a factor
    per pair; weights and rows outside fp16's normal range."""
    from layerstorm_b200.ops import _native as nat
    dev = torch.device("cuda")
    E, R = 20, 2 * BN + 1
    arena, ref = _setup("bf16", H, F, E, n_missing=1, seed=6)
    g = torch.Generator(device="cpu").manual_seed(7)
    x = torch.randn(R, H, generator=g) * 0.5
    x[:, 0], x[:, 1] = 1e5, 1e-7                          # beyond fp16: the columns of the weights that meet them are as small and as large
    x = x.to(torch.bfloat16).to(dev)
    for e in range(1, E):
        v = arena.data[int(arena.slot_of[e])]
        for off in (arena.ef.off_gate, arena.ef.off_up):
            w = v[off: off + F * H * 2].view(torch.bfloat16).view(F, H)
            w[:, 0] *= 1e-6
            w[:, 1] *= 1e6
        ref[e] = [m.double().cpu() for m in arena.read_expert(int(arena.slot_of[e]), "bf16")]
    ids = torch.stack([torch.full((R,), E - 1), torch.arange(R) % (E - 1)], 1).int().to(dev).contiguous()
    P, tiles = R * 2, R * 2 // BN + E + 1
    i32 = dict(dtype=torch.int32, device=dev)
    srt, te, tr, tn, cnt, err, miss = (torch.zeros(n, **i32) for n in (P, tiles, tiles, tiles, 2, 1, 1))
    xs, act = torch.zeros(P, H, dtype=torch.bfloat16, device=dev), torch.zeros(P, F, dtype=torch.float16, device=dev)
    fac = torch.rand(P, generator=g).to(dev) if scaled else None
    limit, alpha, shift = (1.1, 1.702, 1.0) if scaled else (0.0, 1.0, 0.0)
    efp = ctypes.addressof(arena.ef)
    nat.call("lsb_moe_tc_sort", ids, P, E, BN, srt, te, tr, tn, cnt)
    nat.call("lsb_moe_tc_gather_bf16", x, srt, cnt, xs, P, 2, H)
    nat.call("lsb_moe_tc_gateup_bf16", xs, P, arena.data, arena.slot_of, efp, te, tr, tn, cnt, srt, act, BN, tiles, limit, alpha, shift, fac, miss, err)
    torch.cuda.synchronize()
    assert int(err) == 0 and int(miss) == 1
    pair, xd, got = srt.cpu().long(), x.double().cpu(), act.double().cpu()
    for pos in range(0, P, 7):
        r, e = int(pair[pos]) // 2, int(ids.view(-1)[int(pair[pos])])
        if e < 1:
            continue
        c = float(fac[int(pair[pos])]) if scaled else 1.0
        gv, uv = ref[e][0] @ xd[r] * c, ref[e][1] @ xd[r] * c
        if limit:
            gv, uv = gv.clamp(max=limit), uv.clamp(-limit, limit)
        want = gv * torch.sigmoid(alpha * gv) * (uv + shift)
        # fp32 sums, the unit rounded to fp16 (2^-11 relative at most)
        assert float((got[pos] - want).norm() / want.norm()) < 1e-3, (pos, e)


@pytest.mark.parametrize("H,F", [(128, 384), (640, 128), (1152, 640)])
@pytest.mark.parametrize("R", [1, 15])
@pytest.mark.parametrize("scaled", [False, True])
def test_few_rows_keep_bf16_hidden_values_over_bf16_experts(H, F, R, scaled):
    """Both halves of the direct form: reductions that end inside an operand stage and that wrap the rings, a full and a nearly empty tile, an expert that is not
    resident, another gated unit with a factor per pair, hidden values and down weights outside fp16's range."""
    from layerstorm_b200.ops import _native as nat
    dev = torch.device("cuda")
    E, S, BN = 20, 2, 32
    arena, ref = _setup("bf16", H, F, E, n_missing=1, seed=14, size=1.0 if scaled else 2000.0)
    for e in range(1, E):
        w = arena.data[int(arena.slot_of[e])][arena.ef.off_down:][: F * H * 2].view(torch.bfloat16)
        w *= 1e-7
        ref[e] = [m.double().cpu() for m in arena.read_expert(int(arena.slot_of[e]), "bf16")]
    g = torch.Generator(device="cpu").manual_seed(15)
    x = torch.randn(R, H, generator=g).to(torch.bfloat16).to(dev)
    ids = torch.stack([torch.full((R,), E - 1), torch.arange(R) % (E - 1)], 1).int().to(dev).contiguous()
    P, tiles = R * S, R * S // BN + E + 1
    i32 = dict(dtype=torch.int32, device=dev)
    srt, te, tr, tn, cnt, err, miss = (torch.zeros(n, **i32) for n in (P, tiles, tiles, tiles, 2, 1, 1))
    xs, act, y = torch.zeros(P, H, dtype=torch.bfloat16, device=dev), torch.zeros(P, F, dtype=torch.bfloat16, device=dev), torch.full((P, H), float("nan"), device=dev)
    fac = torch.rand(P, generator=g).to(dev) if scaled else None
    limit, alpha, shift = (1.1, 1.702, 1.0) if scaled else (0.0, 1.0, 0.0)
    efp = ctypes.addressof(arena.ef)
    nat.call("lsb_moe_tc_sort", ids, P, E, BN, srt, te, tr, tn, cnt)
    nat.call("lsb_moe_tc_gather_bf16", x, srt, cnt, xs, P, S, H)
    tl = (P, arena.data, arena.slot_of, efp, te, tr, tn, cnt, srt)
    nat.call("lsb_moe_tc_ffn_bf16", 1, xs, *tl, act, BN, tiles, limit, alpha, shift, fac, miss, err)
    nat.call("lsb_moe_tc_ffn_bf16", 0, act, *tl, y, BN, tiles, 0.0, 1.0, 0.0, None, None, err)
    torch.cuda.synchronize()
    assert int(err) == 0 and int(miss) == 1
    xd, got = x.double().cpu(), y.double().cpu()
    for p in range(P):
        r, e = p // S, int(ids.view(-1)[p])
        if e < 1:
            assert bool(got[p].isnan().all())
            continue
        c = float(fac[p]) if scaled else 1.0
        gv, uv = ref[e][0] @ xd[r] * c, ref[e][1] @ xd[r] * c
        if limit:
            gv, uv = gv.clamp(max=limit), uv.clamp(-limit, limit)
        want = ref[e][2] @ (gv * torch.sigmoid(alpha * gv) * (uv + shift))
        # fp32 sums and a hidden value in bf16: 2^-9 of it at most, averaged out over F of them
        assert float((got[p] - want).norm() / want.norm()) < 4e-3, (p, e)


@pytest.mark.parametrize("fmt", ["nvfp4", "fp8_e4m3", "bf16", "gguf_q4_k"])
def test_many_rows_stay_finite_beyond_fp16(fmt):
    """Hidden values of 4e4 rms, some of them beyond fp16, and a row of activations of 1e6 (hidden values of 1e15) count as fp16's largest number; a row with a NaN
    and one with an infinity give no numbers, and none of them touches its neighbours."""
    from layerstorm_b200.models.device_model import ModelBase, MoeBuffers
    dev = torch.device("cuda")
    H, F, E, S, R = 256, 256, 5, 2, 40
    arena, ref = _setup(fmt, H, F, E, n_missing=0, seed=16, size=300.0)
    m, mb = ModelBase(), MoeBuffers()
    m.device, m.tp_size, m.expert_shard = dev, 1, "ep"
    z = lambda *s, dtype=torch.float32: torch.zeros(*s, dtype=dtype, device=dev)
    mb.alloc_moe(z, R, S, E, E, H, F, tc=True)
    mb.tc_xs, mb.tc_act = z(R * S, H, dtype=torch.float16), z(R * S, F, dtype=torch.float16)
    g = torch.Generator(device="cpu").manual_seed(17)
    x = torch.randn(R, H, generator=g) * 0.8
    x[7] *= 1.25e6
    x[9, 3], x[11, 5] = float("nan"), float("inf")
    x = x.to(torch.bfloat16).to(dev)
    ids = torch.stack([torch.randperm(E, generator=g)[:S] for _ in range(R)])
    mb.ids.copy_(ids.int())
    m.moe_prepare(arena, mb, x, R, E)
    m.moe_experts(arena, mb, x, R, E, 0.0, mb.miss)
    got, xd = mb.y.view(R, S, H).double().cpu(), x.double().cpu()
    if fmt != "bf16":
        xd = xd.clamp(-65504.0, 65504.0)
    for r in range(R):
        for k in range(S):
            if r in (9, 11):
                assert not bool(got[r, k].isfinite().any()), (r, k)
                continue
            gate, up, down = ref[int(ids[r, k])]
            want = down @ (torch.nn.functional.silu(gate @ xd[r]) * (up @ xd[r])).clamp(-65504.0, 65504.0)
            if r == 7 and fmt == "gguf_q4_k":                 # every hidden value is at the limit, its sign that of sums whose weights are rounded
                assert bool(got[r, k].isfinite().all())
                continue
            # hidden values in fp16, 2^-11 at most of each; Q4_K weights d sc v - dmin m with both products rounded to fp16: 2^-11 of terms up to 15 d sc and 8 d sc
            # beside weights of 4.6 d sc rms is 2.4e-3 at most a matrix, three of them 4.2e-3 (most hidden values are inside the range: an error of those beyond it
            # would count against a norm that the limit has cut)
            assert float((got[r, k] - want).norm() / want.norm()) < (4.2e-3 if fmt == "gguf_q4_k" else 1e-3), (r, k)


@pytest.mark.parametrize("R", [16, 97, 340, 700])
def test_steps_of_fewer_rows_than_the_workspace(R):
    """The token tile follows the step's rows, not the workspace's: 32, 64 and 128 rows of a workspace whose own tile is 128."""
    from layerstorm_b200.models.device_model import ModelBase, MoeBuffers
    dev = torch.device("cuda")
    H, F, E, S = 128, 256, 8, 2
    arena, ref = _setup("nvfp4", H, F, E, n_missing=0, seed=8)
    m, mb = ModelBase(), MoeBuffers()
    m.device, m.tp_size, m.expert_shard = dev, 1, "ep"
    z = lambda *s, dtype=torch.float32: torch.zeros(*s, dtype=dtype, device=dev)
    mb.alloc_moe(z, 700, S, E, E, H, F, tc=True)
    mb.tc_xs, mb.tc_act = z(700 * S, H, dtype=torch.float16), z(700 * S, F, dtype=torch.float16)
    assert mb.tc_bn == 128 and mb.step_tiles(R * S, E)[0] == {16: 32, 97: 32, 340: 64, 700: 128}[R]
    g = torch.Generator(device="cpu").manual_seed(R)
    x = torch.randn(R, H, generator=g).to(torch.bfloat16).to(dev)
    ids = torch.stack([torch.randperm(E, generator=g)[:S] for _ in range(R)])
    mb.ids[:R].copy_(ids.int())
    m.moe_prepare(arena, mb, x, R, E)
    m.moe_experts(arena, mb, x, R, E, 0.0, mb.miss)
    got, xd = mb.y.view(700, S, H)[:R].double().cpu(), x.double().cpu()
    for e in range(E):
        gate, up, down = ref[e]
        r, k = (ids == e).nonzero(as_tuple=True)
        want = (torch.nn.functional.silu(xd[r] @ gate.T) * (xd[r] @ up.T)) @ down.T
        assert float((got[r, k] - want).norm() / want.norm()) < 1e-3, e
    assert float(mb.y.view(700, S, H)[R:].abs().sum()) == 0.0


@pytest.mark.parametrize("fmt", ["nvfp4", "fp8_e4m3", "bf16", "gguf_q4_k"])
@pytest.mark.parametrize("BN", [32, 64, 128])
@pytest.mark.parametrize("copies", [1, 12])
def test_tiles_of_every_number_of_rows(fmt, BN, copies):
    """One row, one below, at and above each piece of the epilogue, whole tiles and a remainder behind one, each beside experts with other numbers of rows; with
    copies, several tiles per thread block and reductions that end at every place of the rings."""
    from layerstorm_b200.ops import _native as nat
    dev, H, F = torch.device("cuda"), 1024, 768
    counts = [n for n in (1, 15, 16, 17, 31, 32, 33, 48, 63, 64, 65, 112, 127, 128, 129) if n <= BN + 1]
    E = len(counts)
    arena, ref = _setup(fmt, H, F, E, n_missing=0, seed=8)
    arena.slot_of = arena.slot_of.repeat(copies)                     # more experts with the same weights
    g = torch.Generator(device="cpu").manual_seed(9)
    ids = torch.cat([torch.full((n,), e + E * c) for c in range(copies) for e, n in enumerate(counts)])
    ids = ids[torch.randperm(len(ids), generator=g)].int()
    P = len(ids)
    x, tiles = torch.randn(P, H, generator=g).to(torch.bfloat16).to(dev), P // BN + E * copies + 1
    i32 = dict(dtype=torch.int32, device=dev)
    srt, te, tr, tn, cnt, err = (torch.zeros(n, **i32) for n in (P, tiles, tiles, tiles, 2, 1))
    xs, act = torch.zeros(P, H, dtype=torch.float16, device=dev), torch.zeros(P + 1, F, dtype=torch.float16, device=dev)
    y, efp = torch.zeros(P + 1, H, device=dev), ctypes.addressof(arena.ef)
    nat.call("lsb_moe_tc_sort", ids.to(dev), P, E * copies, BN, srt, te, tr, tn, cnt)
    nat.call("lsb_moe_tc_gather", x, srt, cnt, xs, P, 1, H)
    nat.call("lsb_moe_tc_ffn", 1, xs, P, arena.data, arena.slot_of, efp, te, tr, tn, cnt, srt, act, BN, tiles, 0.0, None, err, None)
    nat.call("lsb_moe_tc_ffn", 0, act, P, arena.data, arena.slot_of, efp, te, tr, tn, cnt, srt, y, BN, tiles, 0.0, None, err, None)
    torch.cuda.synchronize()
    assert int(err) == 0 and float(act[P].abs().sum()) == 0.0 and float(y[P].abs().sum()) == 0.0
    for e in range(E):
        r = (ids % E == e).nonzero()[:, 0].to(dev)
        gate, up, down = (m.to(dev) for m in ref[e])
        xd = x[r].double()
        want = (torch.nn.functional.silu(xd @ gate.T) * (xd @ up.T)) @ down.T
        # hidden values in fp16 (2^-11 each at most), bf16 weights converted to fp16 (the same); Q4_K weights are a scale times 0 .. 15 less an offset, both rounded
        # to fp16: 2^-11 of up to 15 steps where the weights' rms is 4.3 of them, 1.7e-3, in each of the three matrices
        assert float((y[r].double() - want).norm() / want.norm()) < (3 ** 0.5 * 1.7e-3 if fmt == "gguf_q4_k" else 1e-3), (e, counts[e])


@pytest.mark.parametrize("H,F", [(1024, 768), (128, 256)])
def test_bf16_experts_in_tiles_of_256_rows(H, F):
    """Gate/up over bf16 rows and down over fp16 hidden values in tiles of up to 256 rows: tiles of one and of two boxes of 128 side by side, whole, ragged and
    behind a full one; several tiles per thread block."""
    from layerstorm_b200.ops import _native as nat
    dev, BN, copies = torch.device("cuda"), 256, 6
    counts = [1, 127, 128, 129, 255, 256, 257, 300, 512, 513]
    E = len(counts)
    arena, ref = _setup("bf16", H, F, E, n_missing=0, seed=10)
    arena.slot_of = arena.slot_of.repeat(copies)
    g = torch.Generator(device="cpu").manual_seed(11)
    ids = torch.cat([torch.full((n,), e + E * c) for c in range(copies) for e, n in enumerate(counts)])
    ids = ids[torch.randperm(len(ids), generator=g)].int()
    P = len(ids)
    x, tiles = torch.randn(P, H, generator=g).to(torch.bfloat16).to(dev), P // BN + E * copies + 1
    i32 = dict(dtype=torch.int32, device=dev)
    srt, te, tr, tn, cnt, err, miss = (torch.zeros(n, **i32) for n in (P, tiles, tiles, tiles, 2, 1, 1))
    xs, act = torch.zeros(P, H, dtype=torch.bfloat16, device=dev), torch.zeros(P + 1, F, dtype=torch.float16, device=dev)
    y, efp = torch.zeros(P + 1, H, device=dev), ctypes.addressof(arena.ef)
    nat.call("lsb_moe_tc_sort", ids.to(dev), P, E * copies, BN, srt, te, tr, tn, cnt)
    nat.call("lsb_moe_tc_gather_bf16", x, srt, cnt, xs, P, 1, H)
    nat.call("lsb_moe_tc_gateup_bf16", xs, P, arena.data, arena.slot_of, efp, te, tr, tn, cnt, srt, act, BN, tiles, 0.0, 1.0, 0.0, None, miss, err)
    nat.call("lsb_moe_tc_ffn", 0, act, P, arena.data, arena.slot_of, efp, te, tr, tn, cnt, srt, y, BN, tiles, 0.0, None, err, None)
    torch.cuda.synchronize()
    assert int(err) == 0 and float(act[P].abs().sum()) == 0.0 and float(y[P].abs().sum()) == 0.0
    for e in range(E):
        r = (ids % E == e).nonzero()[:, 0].to(dev)
        gate, up, down = (m.to(dev) for m in ref[e])
        xd = x[r].double()
        want = (torch.nn.functional.silu(xd @ gate.T) * (xd @ up.T)) @ down.T
        assert float((y[r].double() - want).norm() / want.norm()) < 1e-3, counts[e]          # hidden values and down weights in fp16 (2^-11 each at most)


@pytest.mark.parametrize("H,F", [(640, 384), (384, 128), (128, 640)])
@pytest.mark.parametrize("BN", [32, 64, 128])
def test_fp8_reductions_of_an_odd_number_of_blocks_over_many_items(H, F, BN):
    """Each thread block computes several tiles one after another whose reductions end on an odd block of 128: what a converter set takes moves on by one each time."""
    from layerstorm_b200.ops import _native as nat
    dev = torch.device("cuda")
    E, copies = 12, 40 if H > 128 else 160
    arena, ref = _setup("fp8_e4m3", H, F, E, n_missing=0, seed=12)
    arena.slot_of = arena.slot_of.repeat(copies)                     # more experts with the same weights
    g = torch.Generator(device="cpu").manual_seed(13)
    ids = torch.arange(E * copies).repeat(2)[: 2 * E * copies - 5]
    ids = ids[torch.randperm(len(ids), generator=g)].int()
    P = len(ids)
    x, tiles = torch.randn(P, H, generator=g).to(torch.bfloat16).to(dev), P // BN + E * copies + 1
    i32 = dict(dtype=torch.int32, device=dev)
    srt, te, tr, tn, cnt, err = (torch.zeros(n, **i32) for n in (P, tiles, tiles, tiles, 2, 1))
    xs, act = torch.zeros(P, H, dtype=torch.float16, device=dev), torch.zeros(P + 1, F, dtype=torch.float16, device=dev)
    y, efp = torch.zeros(P + 1, H, device=dev), ctypes.addressof(arena.ef)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert E * copies * min(H, F) // 128 > 3 * sms                   # items of either half
    nat.call("lsb_moe_tc_sort", ids.to(dev), P, E * copies, BN, srt, te, tr, tn, cnt)
    nat.call("lsb_moe_tc_gather", x, srt, cnt, xs, P, 1, H)
    nat.call("lsb_moe_tc_ffn", 1, xs, P, arena.data, arena.slot_of, efp, te, tr, tn, cnt, srt, act, BN, tiles, 0.0, None, err, None)
    nat.call("lsb_moe_tc_ffn", 0, act, P, arena.data, arena.slot_of, efp, te, tr, tn, cnt, srt, y, BN, tiles, 0.0, None, err, None)
    torch.cuda.synchronize()
    assert int(err) == 0 and float(act[P].abs().sum()) == 0.0 and float(y[P].abs().sum()) == 0.0
    for e in range(E):
        r = (ids % E == e).nonzero()[:, 0].to(dev)
        gate, up, down = (m.to(dev) for m in ref[e])
        xd = x[r].double()
        want = (torch.nn.functional.silu(xd @ gate.T) * (xd @ up.T)) @ down.T
        assert float((y[r].double() - want).norm() / want.norm()) < 1e-3, e          # hidden values in fp16 (2^-11 at most)
