"""The order in which fp32 sums are added up.  It is part of what a step returns: AdamW's first steps are normalised and not
bias-corrected, so two correct orders can leave states that differ in the first digits after a few steps.  Every sum is added
up again here, term by term in the stated order, and has to come out bit for bit."""
import numpy as np
import pytest

import tatara_b200 as tb
from helpers import random_index_batch
from test_gpu_parity import LS_FS, _perturb

pytestmark = pytest.mark.gpu


def _same_bits(got, want, what):
    got, want = np.asarray(got, np.float32).reshape(-1), np.asarray(want, np.float32).reshape(-1)
    bad = np.flatnonzero(got.view(np.uint32) != want.view(np.uint32))
    assert bad.size == 0, "%s: %d of %d differ, first %d: %r, want %r" % (what, bad.size, got.size, bad[0], got[bad[0]], want[bad[0]])


@pytest.mark.parametrize("kb", [1, 9, 10, 16, 45, 46, 81, 82])
def test_virtual_row_gradient_is_one_chain_over_the_king_buckets(kb):
    """The fused kernel up to 81 king buckets, the two data-parallel ones above."""
    fs = tb.FeatureSetSpec("test", 4, kb, 24, 8, True)
    F, l1, l2, B = 256, 8, 16, 512
    rng = np.random.default_rng(kb)
    init = _perturb(tb.layerstack_default_init(fs, F, l1, l2, 9), rng, ["ft_w", "ft_b", "l1_b", "l1_shared_bias", "l2_b", "l3_b"])
    d = random_index_batch(rng, B, fs.max_active, fs.piece_inputs, 1, fs.max_active)
    for key in ("stm", "nstm"):
        d[key] = np.where(d[key] >= 0, d[key] + rng.integers(0, kb, B)[:, None] * fs.piece_inputs, d[key]).astype(np.int32)
    tr = tb.GpuTrainer(B, F, l1, l2, 9, fs, optimizer="adamw", init=init)
    tr.forward_backward(tb.BatchData(d["stm"], d["nstm"], d["nnz"], d["score"], d["wdl"], d["bucket"]), 0.0, tb.LossKind.sigmoid())
    tr.apply_optimizer(1e-3)
    g = tr.download_grad("ft_w").reshape(kb + 1, -1)
    want = np.zeros_like(g[0])
    for k in range(kb):
        want += g[k]
    assert np.count_nonzero(want) > want.size // 2
    _same_bits(g[kb], want, "virtual rows")
