"""A device batch scan replayed from its captured graph keeps to its matcher's
scratch: scans of another kind that replace the scratch's buffers in between
make the next call record its launches anew."""
import numpy as np
import pytest

import oracle
import workloads as w

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grow", ["host", "device", "stream", "batch"])
def test_replay_after_larger_scan_on_the_same_matcher(grow):
    import torch
    import warpstate_b200 as ws
    wl = w.regex(size=8 << 20, n=20, seed=31)
    pats = wl.patterns + [(0, b"literal one"), (0, b"another")]
    b = ws.PatternSet.builder()
    for k, p in pats:
        b = b.literal_bytes(p) if k == 0 else b.regex(p.decode() if isinstance(p, bytes) else p)
    m = ws.GpuMatcher.with_config(b.build(), ws.AutoMatcherConfig().max_matches(1 << 14))
    lens = np.full(64, 1000, dtype=np.uint64)
    ends = np.cumsum(lens).astype(np.uint32)
    items = [(int(e) - 1000, 1000) for e in ends]
    ids = np.arange(64, dtype=np.int64)
    small, cap = wl.data[: int(ends[-1])].copy(), 1 << 12
    small[500:511] = np.frombuffer(b"literal one", dtype=np.uint8)
    d_in, d_ends = torch.from_numpy(small).cuda(), torch.from_numpy(ends.view(np.int32)).cuda()
    d_ids, big = torch.from_numpy(ids).cuda(), torch.from_numpy(wl.data).cuda()
    d_out = torch.empty(cap * 3, dtype=torch.int64, device="cuda")
    d_big = torch.empty((1 << 22) * 3, dtype=torch.int64, device="cuda")
    d_cnt, d_cnt2 = (torch.zeros(1, dtype=torch.int64, device="cuda") for _ in range(2))
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    exp = oracle.batch_scan(pats, small, items, ids.astype(np.uint64))
    assert len(exp) > 0

    def run():
        m.scan_batch_device(d_in.data_ptr(), len(small), d_ends.data_ptr(), d_ids.data_ptr(), 64, d_out.data_ptr(),
                            cap, d_cnt.data_ptr(), s.cuda_stream)
        torch.cuda.synchronize()
        n = int(d_cnt.item())
        a = d_out[: 3 * n].view(n, 3).cpu().numpy().view(np.uint64)
        got = np.stack([a[:, 0], a[:, 1] & 0xFFFFFFFF, a[:, 1] >> 32, a[:, 2] & 0xFFFFFFFF], axis=1)
        assert np.array_equal(got[np.lexsort((got[:, 3], got[:, 1], got[:, 2], got[:, 0]))], exp)
        return m.info()["last_graph_replay"]

    assert [run() for _ in range(3)] == [0, 1, 1]
    if grow == "host":
        m.scan_array(wl.data)
    elif grow == "device":
        m.scan_device(big.data_ptr(), big.numel(), d_big.data_ptr(), 1 << 22, d_cnt2.data_ptr(), s.cuda_stream)
    elif grow == "stream":
        ws.StreamPipeline(m).scan_array(wl.data, block=4 << 20)
    else:
        one = torch.tensor([big.numel()], dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        m.scan_batch_device(big.data_ptr(), big.numel(), one.data_ptr(), d_ids.data_ptr(), 1, d_big.data_ptr(), 1 << 22,
                            d_cnt2.data_ptr(), s.cuda_stream)
    torch.cuda.synchronize()
    assert [run() for _ in range(3)] == [0, 1, 1]
