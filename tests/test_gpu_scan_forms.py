"""Scan and stream compaction where the default changes from one pass to two kernels (2^18
values), aligned and not, in place, and with an output that overlaps the input (which keeps the
single pass). Integer results: equality with numpy."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGE = 1 << 18


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _exclusive(a):
    return np.concatenate([[0], np.cumsum(a, dtype=np.int64)[:-1]]).astype(np.int32)


def _ws(torch, hhs, n):
    size = hhs.scan_workspace_size(n)
    return torch.full((size,), 0x5a, dtype=torch.uint8, device="cuda"), size


@pytest.mark.parametrize("shift", ["apart", "in_place", "behind"])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [EDGE - 1, EDGE, EDGE + 1, (1 << 20) + 4099, (1 << 22) - 1])
def test_scan_forms(cuda, hhs, n, offset, shift):
    torch = cuda
    a = np.random.default_rng(n + offset).integers(-1000, 1000, n).astype(np.int32)
    buf = torch.zeros(n + 8, dtype=torch.int32, device="cuda")
    src = buf[4 + offset:4 + offset + n]
    src.copy_(torch.from_numpy(a))
    dst = (src if shift == "in_place" else buf[offset:offset + n] if shift == "behind" else
           torch.zeros(n + 8, dtype=torch.int32, device="cuda")[offset:offset + n])
    ws, size = _ws(torch, hhs, n)
    hhs.scan_exclusive_i32(_ptr(src), _ptr(dst), n, _ptr(ws), size, None)
    assert hhs.scan_workspace_status(_ptr(ws), None) == 0
    assert np.array_equal(dst.cpu().numpy(), _exclusive(a))


@pytest.mark.parametrize("scan_out", ["none", "apart", "in_place"])
@pytest.mark.parametrize("idx_over_flags", [False, True])
@pytest.mark.parametrize("n", [EDGE - 1, EDGE, EDGE + 1, (1 << 20) + 4099])
def test_compaction_forms(cuda, hhs, n, idx_over_flags, scan_out):
    torch = cuda
    if idx_over_flags and scan_out == "in_place":
        pytest.skip("two outputs in one place")
    f = (np.random.default_rng(n).random(n) < 0.3).astype(np.int32)
    flags = torch.from_numpy(f).cuda()
    scan = {"none": None, "apart": torch.zeros(n, dtype=torch.int32, device="cuda"),
            "in_place": flags}[scan_out]
    idx = flags if idx_over_flags else torch.zeros(n, dtype=torch.int32, device="cuda")
    count = torch.zeros(1, dtype=torch.int32, device="cuda")
    ws, size = _ws(torch, hhs, n)
    hhs.compact_flags_i32(_ptr(flags), None if scan is None else _ptr(scan), _ptr(idx),
                          _ptr(count), n, _ptr(ws), size, None)
    assert hhs.scan_workspace_status(_ptr(ws), None) == 0
    ref = np.flatnonzero(f).astype(np.int32)
    assert int(count) == len(ref)
    assert np.array_equal(idx.cpu().numpy()[:len(ref)], ref)
    if scan is not None:
        assert np.array_equal(scan.cpu().numpy(), _exclusive(f))


@pytest.mark.parametrize("n,kernels", [(EDGE, 1), (EDGE + 1, 1), (3 << 17, 1), (1 << 19, 2)])
def test_scan_takes_a_second_kernel_where_it_pays(cuda, hhs, n, kernels):
    """Below 2^19 values a single call takes longer with two kernels (12.4 us against 10.6). The single
    pass clears the whole workspace, the two kernels write their chunk sums only."""
    torch = cuda
    a = torch.ones(n, dtype=torch.int32, device="cuda")
    out = torch.empty_like(a)
    ws, size = _ws(torch, hhs, n)
    hhs.scan_exclusive_i32(_ptr(a), _ptr(out), n, _ptr(ws), size, None)
    assert bool((ws == 0x5a).any()) == (kernels == 2)
    assert hhs.scan_workspace_status(_ptr(ws), None) == 0
    assert torch.equal(out, torch.arange(n, dtype=torch.int32, device="cuda"))
