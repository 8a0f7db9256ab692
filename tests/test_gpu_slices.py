"""Slice-resident FT kernels off the shapes they were first built for: the feature sets of 1710 rows per king bucket (a
narrower block in the forward), slices of very different sizes and empty ones."""
import numpy as np
import pytest

import oracle_lib as O
import tatara_b200 as tb
from helpers import random_index_batch
from test_gpu_parity import _check_step, _oracle_for, _perturb, _sync_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fs,F,B", [("halfka-hm-split", 384, 272), ("halfka-split", 256, 1040)])
def test_split_sets_step_matches_oracle(fs, F, B):
    fs = tb.FEATURE_SETS[fs].with_factorize(False)
    l1, l2 = 16, 32
    init = _perturb(tb.layerstack_default_init(fs, F, l1, l2, 9), np.random.default_rng(F), ["ft_b", "l1_b", "l1_shared_bias", "l2_b", "l3_b"])
    init["ft_w"] *= 30.0
    tr = tb.GpuTrainer(B, F, l1, l2, 9, fs, optimizer="adamw", init=init)
    ot = _oracle_for(tr, "layerstack", fs, F, l1, l2, 9, "adamw", (0.01, 0.01, 0.01), B)
    _sync_weights(tr, ot, init)
    _check_step(tr, ot, tb.synthetic_batch(tb.SYNTH_SEED + B, B, fs), tb.LossKind.sigmoid(), O.sigmoid_loss(), 1e-3, "layerstack", B, F, l1)


@pytest.mark.parametrize("B,share", [(16, 0.5), (4096, 0.6), (9008, 0.97)])
def test_uneven_slices_step_matches_oracle(B, share):
    """`share` of the items in one slice (runs of 4096, chunk groups of four), the rest in a few others, most slices empty."""
    F, l1, l2 = 256, 8, 16
    fs = tb.FEATURE_SETS["halfka-hm-merged"].with_factorize(False)
    rng = np.random.default_rng(B)
    init = _perturb(tb.layerstack_default_init(fs, F, l1, l2, 9), rng, ["ft_b", "l1_b", "l1_shared_bias", "l2_b", "l3_b"])
    init["ft_w"] *= 30.0
    d = random_index_batch(rng, B, fs.max_active, fs.piece_inputs, 0, fs.max_active)
    for key in ("stm", "nstm"):
        k = np.where(rng.random(B) < share, 7, rng.choice([0, 8, 44], B))
        d[key] = np.where(d[key] >= 0, d[key] + k[:, None] * fs.piece_inputs, d[key]).astype(np.int32)
    tr = tb.GpuTrainer(B, F, l1, l2, 9, fs, optimizer="adamw", init=init)
    ot = _oracle_for(tr, "layerstack", fs, F, l1, l2, 9, "adamw", (0.01, 0.01, 0.01), B)
    _sync_weights(tr, ot, init)
    batch = tb.BatchData(d["stm"], d["nstm"], d["nnz"], d["score"], d["wdl"], d["bucket"])
    _check_step(tr, ot, batch, tb.LossKind.sigmoid(), O.sigmoid_loss(), 1e-3, "layerstack", B, F, l1)
