"""The arithmetic and the kernels of the offline set-up's register transforms."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "altopir-public_b200", "csrc")


def test_montgomery_products_and_lazy_sums(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "mont")
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", CSRC, os.path.join(HERE, "cpp", "test_mont.cpp"), "-o", exe],
                   check=True)
    assert subprocess.run([exe], capture_output=True, text=True, timeout=300).stdout.strip() == "0"


@pytest.mark.gpu
@pytest.mark.parametrize("rows,record,tg", [(2048, 2048, 2), (2048, 4096, 3), (2048 * 9, 4096, 5), (2048 * 20, 6144, 8)])
def test_register_transforms_equal_the_shared_memory_ones(gpu, svc, rows, record, tg, monkeypatch):
    """The hint on the tensor cores and the walk with register transforms on clusters of 2, 3, 5 and 8 CTAs (one a digit)
    give the values of the shared-memory transforms and the single-CTA walk, over a database of random bytes, all 255
    and all zero columns: from one polynomial a column to more than the loader's stages, and from fewer column groups
    than four an SM to a partial last round."""
    from altopir_b200 import offline
    p = svc.Params(rows, record, tg=tg)
    db = np.random.default_rng(tg).integers(0, 256, size=(p.record_bytes, p.rows), dtype=np.uint8)
    db[::3] = 255
    db[1::7] = 0
    got = []
    for variant in ({}, {"ALTO_OFFLINE_CLUSTER": "1", "ALTO_OFFLINE_ACT8": "0"}):
        for k, v in variant.items():
            monkeypatch.setenv(k, v)
        e = offline.blank_engine(p, db)
        got.append(offline.prepare(e, p, want=True)[1])
        e.close()
    for name in ("bold_t", "bold_t_bar", "that", "a_hat"):
        assert np.array_equal(got[0][name], got[1][name]), name


@pytest.mark.gpu
@pytest.mark.parametrize("n,tg", [(32, 4), (64, 8), (256, 4), (1024, 2)])
def test_packing_matrix_at_other_ring_dimensions(gpu, oracle, svc, n, tg):
    """Rings of 32 (several digits in one 128-byte tile row) to 1,024: the walk's values equal the oracle's, and the
    responses, which read every byte of the packing matrix, too."""
    from altopir_b200 import offline
    from oracle.scheme import SchemeState
    p = svc.Params(2 * n if n > 32 else 64, n, n=n, tg=tg)
    db = np.random.default_rng(n).integers(0, 256, size=(p.record_bytes, p.rows), dtype=np.uint8)
    st = SchemeState(p, db, oracle)
    e = offline.blank_engine(p, db)
    _, out = offline.prepare(e, p, want=True)
    for k in ("bold_t", "bold_t_bar", "that"):
        assert np.array_equal(out[k][0].astype(np.uint64), getattr(st, k)[0]), k
    req = svc.synthetic_requests(p, 3, seed=n)
    frames = [req[i] for i in range(3)]
    _, _, want = oracle.answer(st, frames)
    got = np.zeros((3, e.response_len()), dtype=np.uint8)
    status = np.full(3, -1, dtype=np.int32)
    assert e.answer(frames, got, status)[0] == 3
    assert np.array_equal(got, want)
    e.close()
