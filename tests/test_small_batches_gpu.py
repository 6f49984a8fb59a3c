"""Batches of at most four frames: the single-CTA GEMMs share the SMs (two CTAs each) and the scan runs beside the pack.
Every response and status equals the oracle's, on the host path, the device path launched directly and as a graph."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b", [1, 2, 3, 4])
@pytest.mark.parametrize("rows,record", [(2048, 2048), (4096, 6144), (65536, 2048)])
def test_batches_of_up_to_four_frames(gpu, oracle, svc, eng, rows, record, b):
    import torch
    p = svc.params(rows, record)
    st = svc.SyntheticState.make(p, seed=rows + b, keep_values=True)
    e = eng.Engine.from_state(st, threads=svc.threads())
    req = svc.synthetic_requests(p, b, seed=5 * b)
    if b == 3:  # one rejected frame among valid ones: its last z key is out of range
        req[1, 9 + 8 * p.count - 4:9 + 8 * p.count] = 0xFF
    frames = [req[i] for i in range(b)]
    _, want_status, want = oracle.answer(st, frames)
    ok = [i for i in range(b) if want_status[i] == 0]
    assert len(ok) == (2 if b == 3 else b)
    stride = (7 + e.request_len() + 255) // 256 * 256
    slots = np.zeros((b, stride), dtype=np.uint8)
    slots[:, 7:7 + e.request_len()] = req
    d_slots, d_out = torch.from_numpy(slots).cuda(), torch.zeros((b, e.response_len()), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    for mode in ("host", "device", "graph", "graph"):
        status = np.full(b, -1, dtype=np.int32)
        if mode == "host":
            out = np.zeros((b, e.response_len()), dtype=np.uint8)
            n, _ = e.answer(frames, out, status)
        else:
            e.set_graphs(mode == "graph")
            d_out.zero_()
            torch.cuda.synchronize()
            n = e.answer_device(d_slots.data_ptr(), stride, b, d_out.data_ptr(), e.response_len(), status)
            out = d_out.cpu().numpy()
        assert n == len(ok) and list(status) == list(want_status), mode
        assert np.array_equal(out[ok], want[ok]), mode
    e.close()
