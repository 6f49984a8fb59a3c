"""alto_answer's schedules against each other: statuses and responses where its column groups differ from the device
path's, and where it follows a batch still in flight."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("host_groups,groups", [("1", "2"), ("1", "8"), ("1", None), ("2", "1")])
def test_statuses_of_whole_frames_whatever_the_device_groups(gpu, svc, eng, monkeypatch, host_groups, groups):
    """24 frames of 82 KB (2 MB together, so they upload whole where alto_answer scans in one group) with 2.75 MB of
    responses (so the device path may take more groups).  The rejected frame moves from call to call: every call reports
    its own statuses, and a rejected frame's output stays untouched."""
    p = svc.params(4096, 32768)
    st = svc.SyntheticState.make(p, seed=61)
    b = 24
    frames = svc.synthetic_requests(p, b, seed=62)
    assert frames.nbytes <= 2 << 20
    plain = eng.Engine.from_state(st)
    want = np.zeros((b, plain.response_len()), dtype=np.uint8)
    assert want.nbytes >= 2 << 20
    assert plain.answer([frames[i] for i in range(b)], want, np.full(b, -1, dtype=np.int32))[0] == b
    plain.close()
    monkeypatch.setenv("ALTO_HOST_GROUPS", host_groups)
    if groups:
        monkeypatch.setenv("ALTO_GROUPS", groups)
    e = eng.Engine.from_state(st)
    for bad in (3, 0, 23, None, 11, 3, None):
        req = frames.copy()
        if bad is not None:
            req[bad, 9:13] = 0xFF  # y[0] >= Q: status 3
        out = np.full_like(want, 0x11)
        status = np.full(b, -1, dtype=np.int32)
        n, _ = e.answer([req[i] for i in range(b)], out, status)
        expect = want.copy()
        if bad is not None:
            expect[bad] = 0x11
        assert n == b - (bad is not None), bad
        assert list(status) == [3 if i == bad else 0 for i in range(b)], bad
        assert np.array_equal(out, expect), bad
    e.close()


@pytest.mark.parametrize("groups", ["1", "2"])
@pytest.mark.parametrize("piped", ["1", str(1 << 40)])
def test_answer_behind_a_batch_in_flight(gpu, svc, eng, monkeypatch, piped, groups):
    """alto_answer right behind alto_enqueue_device on the same engine, over two record chunks, with its query words
    uploaded chunk by chunk and all at once: it waits for the batch's scan sums before it clears them, so both batches
    return what they return alone."""
    import torch
    monkeypatch.setenv("ALTO_PIPED_BYTES", piped)
    monkeypatch.setenv("ALTO_GROUPS", groups)
    p = svc.params(65536, 16384)  # 40 frames: 13 MB uploaded, 2.3 MB of responses
    st = svc.SyntheticState.make(p, seed=71, keep_values=False, host_db=False)
    e = eng.Engine.from_state(st, threads=svc.threads(), tile=False)
    ahead, b = 64, 40
    ql, rl = e.request_len(), e.response_len()
    stride = (7 + ql + 255) // 256 * 256
    frames = svc.synthetic_requests(p, ahead + b, seed=72)
    slots = np.zeros((ahead, stride), dtype=np.uint8)
    slots[:, 7:7 + ql] = frames[:ahead]
    slots = torch.from_numpy(slots).cuda()
    req = [frames[ahead + i] for i in range(b)]

    def enqueue():
        out = torch.zeros((ahead, rl), dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        e.enqueue_device(slots.data_ptr(), stride, ahead, out.data_ptr(), rl)
        return out

    def answer():
        out, status = np.zeros((b, rl), dtype=np.uint8), np.full(b, -1, dtype=np.int32)
        assert e.answer(req, out, status)[0] == b
        return out

    first = enqueue()
    e.sync()
    want_ahead, want = first.cpu().numpy(), answer()
    for _ in range(5):
        out = enqueue()
        got = answer()
        e.sync()
        assert np.array_equal(got, want)
        assert np.array_equal(out.cpu().numpy(), want_ahead)
    e.close()


def test_column_groups_of_the_device_path_follow_the_setting(gpu, svc, eng, monkeypatch):
    """ALTO_GROUPS: a count holds for small batches too; 0 is the choice by size, as without the variable, which takes one
    launch of the scan for a small batch and two for one of more than 32 MB of responses."""
    import torch
    p = svc.params(2048, 32768)  # 16 response parts of 7 KB
    st = svc.SyntheticState.make(p, seed=81, keep_values=False, host_db=False)
    launches, outs = {}, {}
    small, large = 3, 300
    for setting in (None, "0", "1", "2", "4", "-3", "many"):
        monkeypatch.delenv("ALTO_GROUPS", raising=False)
        if setting is not None:
            monkeypatch.setenv("ALTO_GROUPS", setting)
        e = eng.Engine.from_state(st, threads=svc.threads(), tile=False)
        ql, rl = e.request_len(), e.response_len()
        assert small * rl < 2 << 20 and large * rl > 32 << 20
        stride = (7 + ql + 255) // 256 * 256
        slots = torch.zeros((large, stride), dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        svc.synthetic_requests_device(p, large, 82, slots.data_ptr(), stride)
        for b in (small, large):
            out = torch.zeros((b, rl), dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            assert e.answer_device(slots.data_ptr(), stride, b, out.data_ptr(), rl, np.zeros(b, dtype=np.int32)) == b
            launches[setting, b] = e.last_launches()
            outs[setting, b] = out.cpu().numpy()
        e.close()
    for setting in ("0", "-3", "many"):
        for b in (small, large):
            assert launches[setting, b] == launches[None, b], (setting, b)
    for b in (small, large):
        assert launches["1", b] == 4 and launches["2", b] == 8 and launches["4", b] == 12, (b, launches)
        for setting in ("0", "1", "2", "4", "-3", "many"):
            assert np.array_equal(outs[setting, b], outs[None, b]), (setting, b)
    assert launches[None, small] == 4 and launches[None, large] == 8
