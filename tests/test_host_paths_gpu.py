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
