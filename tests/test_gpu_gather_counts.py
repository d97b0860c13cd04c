"""gstex_batch_gather_counts, for callers that gather and scan in two calls
(gstex_inclusive_scan_picked_i32 does both)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 255, 256, 257, 100003])
def test_gathers_and_scans_like_the_picked_scan(n):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from gstex_cuda_gb300 import batch as B
    L, st = B._L(), torch.cuda.current_stream().cuda_stream
    g = torch.Generator().manual_seed(n)
    counts = torch.randint(0, 30, (n,), generator=g, dtype=torch.int32).cuda()
    order = torch.randperm(n, generator=g).int().cuda()
    out, picked, cum, cum2 = (torch.empty_like(counts) for _ in range(4))
    total = torch.zeros(2, dtype=torch.int64, device="cuda")
    ws = torch.empty(L.gstex_scan_workspace_bytes(n), dtype=torch.uint8, device="cuda")
    assert L.gstex_batch_gather_counts(n, order.data_ptr(), counts.data_ptr(), out.data_ptr(), st) == 0
    assert L.gstex_inclusive_scan_i32(n, out.data_ptr(), cum.data_ptr(), total.data_ptr(), ws.data_ptr(), ws.numel(),
                                      st) == 0
    assert L.gstex_inclusive_scan_picked_i32(n, counts.data_ptr(), order.data_ptr(), picked.data_ptr(),
                                             cum2.data_ptr(), total.data_ptr() + 8, ws.data_ptr(), ws.numel(), st) == 0
    assert torch.equal(out, counts[order.long()]) and torch.equal(picked, out)
    assert torch.equal(cum, cum2) and torch.equal(cum.long(), out.long().cumsum(0))
    assert total.tolist() == [int(counts.sum())] * 2
