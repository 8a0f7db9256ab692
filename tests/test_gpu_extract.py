"""Record extraction at the edges of its kernel (32 records a block), its pipeline (16 384 records a piece) and of the
record format (arbitrary bits), page-locked and pageable, against the oracle."""
import threading

import numpy as np
import pytest

import oracle_lib as O
import tatara_b200 as tb

pytestmark = pytest.mark.gpu


def _check(psv, fs, **kw):
    got = tb.extract_batch(psv, tb.FEATURE_SETS[fs], **kw)
    want = O.psv_to_batch(fs, psv.tobytes())
    assert (got.nnz == want["nnz"]).all()
    assert (got.stm_indices == want["stm"]).all() and (got.nstm_indices == want["nstm"]).all()
    assert (got.score == want["score"]).all() and (got.wdl == want["wdl"]).all()
    if kw.get("with_bucket", True):
        assert (got.bucket_idx == want["bucket"]).all()
    else:
        assert got.bucket_idx is None


@pytest.mark.parametrize("n", [1, 31, 33, 16383, 16385, 40000])
@pytest.mark.parametrize("pinned,with_bucket", [(False, True), (True, True), (True, False)])
def test_extract_sizes(n, pinned, with_bucket):
    _check(tb.synthesize_psv(tb.SYNTH_SEED + n, n), "halfka-hm-merged", pinned=pinned, with_bucket=with_bucket)


@pytest.mark.parametrize("fs", ["halfkp", "halfka-split"])
def test_extract_arbitrary_bits(fs):
    rng = np.random.default_rng(3)
    psv = rng.integers(0, 256, (4000, 40), dtype=np.uint8)
    psv[0] = 255  # nothing but ones
    psv[1] = 0
    keep = []
    for i in range(len(psv)):
        try:
            O.psv_to_batch(fs, psv[i].tobytes())  # refuses a record of more pieces than the set has slots
            keep.append(i)
        except AssertionError:
            pass
    assert len(keep) > 1000
    _check(np.ascontiguousarray(psv[keep]), fs)


def test_extract_from_several_threads():
    psv = [tb.synthesize_psv(tb.SYNTH_SEED + i, 5000 + 777 * i) for i in range(4)]
    errors = []

    def work(i):
        try:
            for _ in range(3):
                _check(psv[i], "halfkp", pinned=bool(i & 1))
        except Exception as e:  # noqa: BLE001
            errors.append(e)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
