"""The offline set-up at the smallest ring it takes, 16: its packing-matrix kernel writes 16 slots at a time."""
import numpy as np
import pytest


def test_engines_of_smaller_rings_are_refused(svc):
    """n = 8 never reaches the set-up: no engine is made for it."""
    import altopir_b200 as pkg
    from altopir_b200 import client, engine
    p = svc.Params(64, 32, n=8, tg=16)
    ub = np.zeros(4 * p.record_bytes * p.count, dtype=np.int8)
    pre = [np.zeros(p.part_len, dtype=np.uint8) for _ in range(p.instances)]
    that = [np.zeros(p.count, dtype=np.uint64) for _ in range(p.instances)]
    with pytest.raises(engine.EngineError, match="unsupported engine configuration"):
        engine.Engine.empty(p.rows, p.record_bytes, ub, 8, p.tg, pre, p.row1_off, 1 << p.q1_bits, p.q1_bits, that,
                            client.ntt_inverse_table(client.Ring(8)))
    assert "unsupported" in pkg.last_error()


@pytest.mark.gpu
@pytest.mark.parametrize("rows,record,tg", [(64, 32, 8), (128, 96, 16)])
def test_smallest_ring_equals_the_oracle(gpu, oracle, svc, rows, record, tg):
    from altopir_b200 import offline
    from oracle.scheme import SchemeState
    p = svc.Params(rows, record, n=16, tg=tg)
    db = np.random.default_rng(tg).integers(0, 256, size=(p.record_bytes, p.rows), dtype=np.uint8)
    st = SchemeState(p, db, oracle)
    e = offline.blank_engine(p, db)
    _, out = offline.prepare(e, p, want=True)
    for k in ("bold_t", "bold_t_bar", "that"):
        assert np.array_equal(out[k][0].astype(np.uint64), getattr(st, k)[0]), k
    req = svc.synthetic_requests(p, 3, seed=16)
    frames = [req[i] for i in range(3)]
    _, _, want = oracle.answer(st, frames)
    got = np.zeros((3, e.response_len()), dtype=np.uint8)
    status = np.full(3, -1, dtype=np.int32)
    assert e.answer(frames, got, status)[0] == 3
    assert np.array_equal(got, want)
    e.close()
