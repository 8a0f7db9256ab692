"""Weights uploaded from pageable memory and the tables derived from them."""
import numpy as np
import pytest

import tatara_b200 as tb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [tb.PrecisionFlags(), tb.PrecisionFlags(ft_fp16=True)])
def test_folded_table_follows_every_upload(precision):
    """The fold runs on a stream of its own: it has to wait for the last piece of the copy (the virtual rows)."""
    fs = tb.FeatureSetSpec("test", 4, 2, 1710, 40, True)
    F = 640
    rng = np.random.default_rng(3)
    tables = [rng.uniform(-0.2, 0.2, fs.train_ft_in * F).astype(np.float32) for _ in range(2)]
    want = []
    for w in tables:
        t = w.reshape(3, -1)
        c = (t[:2] + t[2]).reshape(-1)
        want.append(c.astype(np.float16).astype(np.float32) if precision.ft_fp16 else c)
    tr = tb.GpuTrainer(16, F, 8, 16, 9, fs, precision=precision, init=dict(tb.layerstack_default_init(fs, F, 8, 16, 9), ft_w=tables[1]))
    for i in range(200):
        tr.upload_group("ft_w", w=tables[i % 2])
        assert np.array_equal(tr.read_buffer("comb", fs.ft_in * F), want[i % 2]), i
