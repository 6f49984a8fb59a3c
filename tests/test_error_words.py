"""Who is told about a kernel wait that ran out: the error word is set from the host, as a kernel would set it."""
import numpy as np
import pytest


def test_set_error_checks_its_arguments():
    import altopir_b200 as pkg
    assert pkg.lib().alto_engine_set_error(None, 0, 1) == -1


@pytest.mark.gpu
def test_offline_setup_leaves_an_earlier_batchs_error_to_sync(gpu, svc, eng):
    """A timeout of an enqueued batch is not the offline set-up's: the set-up returns its state, and the next sync
    reports the batch, once."""
    from altopir_b200 import offline
    p = svc.params(2048, 2048)
    db = np.random.default_rng(5).integers(0, 256, size=(p.record_bytes, p.rows), dtype=np.uint8)
    e = offline.blank_engine(p, db)
    want = offline.prepare(e, p, want=True)[1]
    e.set_lanes(2)
    for lane in (0, 1):
        e.set_error(4, lane)
        got = offline.prepare(e, p, want=True)[1]
        for k in want:
            assert np.array_equal(got[k], want[k]), (lane, k)
        with pytest.raises(eng.EngineError, match="0x4"):
            e.sync()
        e.sync()
        offline.prepare(e, p)
        e.sync()
    for lane, code in ((2, 1), (-1, 1), (0, 0), (0, 16)):
        with pytest.raises(eng.EngineError):
            e.set_error(code, lane)
    e.close()


@pytest.mark.gpu
def test_every_recorded_code_is_reported(gpu, svc, eng):
    """Two waits that ran out in one batch are both named; another lane's word is its own."""
    p = svc.params(2048, 2048)
    e = eng.Engine.from_state(svc.SyntheticState.make(p, seed=3))
    e.set_lanes(2)
    e.set_error(1)
    e.set_error(8)
    e.set_error(2, 1)
    with pytest.raises(eng.EngineError, match="0x9"):  # the main lane is looked at last
        e.sync()
    e.sync()
    e.close()
