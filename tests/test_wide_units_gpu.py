"""The pair GEMMs' wide units (two sub-accumulators of 160 to 256 limb columns over one read of each A tile) against the
one-tile units and the oracle: widths, a half empty last unit, one block of K, rows of A past the last column."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,record,n,tg,batches", [
    (2048, 4096, 2048, 4, (65, 80, 81, 112, 128)),   # 2 x 160, 160, 192, 224, 256 columns
    (4096, 2048, 2048, 2, (129, 200, 257)),          # two and three units along the clients, the last partly empty
    (64, 96, 32, 4, (70, 129)),                      # one block of K; 96 columns in a tile of 256
    (3 * 32768 + 192, 2048, 2048, 1, (90,)),         # four record chunks, the last of two blocks
])
def test_wide_units_return_the_bytes_of_one_tile_units(gpu, oracle, svc, eng, monkeypatch, rows, record, n, tg,
                                                       batches):
    p = svc.Params(rows, record, n=n, tg=tg)
    st = svc.SyntheticState.make(p, seed=rows + n + tg, keep_values=True)
    st.db_col[::3] = 255
    e = eng.Engine.from_state(st, threads=svc.threads())
    for b in batches:
        req = svc.synthetic_requests(p, b, seed=b)
        outs = []
        for wide in ("1", "0", None):
            for k in ("ALTO_SCAN_WIDE", "ALTO_PACK_WIDE"):
                monkeypatch.delenv(k, raising=False)
                if wide:
                    monkeypatch.setenv(k, wide)
            out = np.zeros((b, e.response_len()), dtype=np.uint8)
            status = np.full(b, -1, dtype=np.int32)
            assert e.answer([req[i] for i in range(b)], out, status)[0] == b
            outs.append(out)
        pick = sorted({0, b // 2, 63, b - 1})
        _, _, want = oracle.answer(st, [req[i] for i in pick])
        assert np.array_equal(outs[0][pick], want), b
        assert np.array_equal(outs[0], outs[1]) and np.array_equal(outs[0], outs[2]), b
    e.close()


@pytest.mark.parametrize("rows,b", [(32768, 129), (32768, 257), (32768 + 9 * 128, 300)])
def test_scan_units_shortened_for_wide_batches(gpu, oracle, svc, eng, rows, b):
    """Batches of more than 512 limb columns cut their scan units to 128 or 64 blocks of K (a chunk has 256): one record
    chunk, and a second one of nine blocks."""
    p = svc.Params(rows, 2048, n=2048, tg=1) if rows % 2048 == 0 else svc.Params(rows, 96, n=32, tg=4)
    st = svc.SyntheticState.make(p, seed=rows + b, keep_values=True)
    st.db_col[::3] = 255
    e = eng.Engine.from_state(st, threads=svc.threads())
    req = svc.synthetic_requests(p, b, seed=b)
    out = np.zeros((b, e.response_len()), dtype=np.uint8)
    status = np.full(b, -1, dtype=np.int32)
    assert e.answer([req[i] for i in range(b)], out, status)[0] == b
    pick = sorted({0, 127, 128, b - 1})
    _, _, want = oracle.answer(st, [req[i] for i in pick])
    assert np.array_equal(out[pick], want)
    e.close()
