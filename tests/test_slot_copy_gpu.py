"""Sequence slots of several tensors copied in one launch."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from layerstorm_b200.ops import _native as nat


@pytest.mark.parametrize("n", [1, 5, 96, 97, 200])
def test_slots_of_any_size_and_alignment(n):
    """Sizes from one byte to more than a grid of 16-byte pieces, tensors at and off 16-byte addresses, more tensors than one launch takes; nothing else moves."""
    g = torch.Generator(device="cuda").manual_seed(n)
    sizes = [1, 7, 16, 48, 1000, 4096, 16384 * 3 + 16, 100003, 5 << 20][: max(1, min(9, n))]
    ts = []
    for k in range(n):
        b, off = sizes[k % len(sizes)], (k // len(sizes)) % 3
        b = min(b, 4096) if n > 9 and k >= 9 else b
        ts.append(torch.randint(0, 256, (3 * b + off,), generator=g, dtype=torch.uint8, device="cuda")[off:].view(3, b))
    want = [t.clone() for t in ts]
    for t in want:
        t[2] = t[0]
    table = np.array([(t.data_ptr(), t.shape[1]) for t in ts], dtype=np.int64)
    nat.call("lsb_copy_slots", table.ctypes.data, n, 0, 2)
    assert all(torch.equal(a, b) for a, b in zip(ts, want))


@pytest.mark.parametrize("where", ["first", "inside", "last", "all"])
def test_tensors_without_elements_take_no_part(where):
    """What a convolution of one tap keeps: nothing, at no address, with strides that say otherwise; more entries than one launch takes, too."""
    g = torch.Generator(device="cuda").manual_seed(3)
    ts = [torch.randn(3, 4, 40, generator=g, device="cuda") for _ in range(0 if where == "all" else 100)]
    none = torch.zeros(3, 4, 40, 0, device="cuda")
    at = {"first": [0, 0], "inside": [50, 95, 96], "last": [100], "all": [0]}[where]
    entries = [(t.data_ptr(), t.stride(0) * 4) for t in ts]
    for k in at:
        entries.insert(k, (none.data_ptr(), none.numel() * 4))
    want = [t.clone() for t in ts]
    for t in want:
        t[2] = t[0]
    table = np.array(entries, dtype=np.int64)
    nat.call("lsb_copy_slots", table.ctypes.data, len(entries), 0, 2)
    assert all(torch.equal(a, b) for a, b in zip(ts, want))
    wrong = np.array([(0, 16)], dtype=np.int64)                          # bytes at no address
    with pytest.raises(RuntimeError):
        nat.call("lsb_copy_slots", wrong.ctypes.data, 1, 0, 2)
