"""Slice-resident FT kernels off the shapes they were first built for: the feature sets of 1710 rows per king bucket (a
narrower block in the forward), slices of very different sizes and empty ones."""
import numpy as np
import pytest

import oracle_lib as O
import tatara_b200 as tb
from helpers import assert_close, assert_close_scaled, random_index_batch
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


@pytest.mark.parametrize("kb", [1, 8, 9, 10, 46, 81, 82])
def test_factorized_optimizer_king_bucket_counts(kb):
    """Nine king buckets a warp, nine warps a block, two launches above that: the step's weights, moments and folded table."""
    fs = tb.FeatureSetSpec("test", 4, kb, 40, 8, True)
    F, l1, l2, B = 256, 8, 16, 64
    rng = np.random.default_rng(kb)
    init = _perturb(tb.layerstack_default_init(fs, F, l1, l2, 9), rng, ["ft_w", "ft_b", "l1_b", "l1_shared_bias", "l2_b", "l3_b"])
    d = random_index_batch(rng, B, fs.max_active, fs.piece_inputs, 1, fs.max_active)
    for key in ("stm", "nstm"):
        d[key] = np.where(d[key] >= 0, d[key] + rng.integers(0, kb, B)[:, None] * fs.piece_inputs, d[key]).astype(np.int32)
    tr = tb.GpuTrainer(B, F, l1, l2, 9, fs, optimizer="ranger", init=init)
    ot = _oracle_for(tr, "layerstack", fs, F, l1, l2, 9, "ranger", (0.01, 0.01, 0.01), B)
    _sync_weights(tr, ot, init)
    batch = tb.BatchData(d["stm"], d["nstm"], d["nnz"], d["score"], d["wdl"], d["bucket"])
    for _ in range(7):
        tr.train_step(batch, 1e-3, 0.0, tb.LossKind.sigmoid())
        ot.step(d, 1e-3, 0.0, O.sigmoid_loss())
    got = tr.download_group("ft_w", ("w", "m", "v", "slow"))
    assert_close(got["w"], ot.group("ft_w"), 1e-5, "w")
    assert_close(got["slow"], ot.group("ft_w", "slow"), 1e-5, "slow")
    assert_close_scaled(got["m"], ot.group("ft_w", "m"), 1e-4, "m")
    assert_close_scaled(got["v"], ot.group("ft_w", "v"), 1e-4, "v")
    w = got["w"].reshape(kb + 1, -1)
    assert np.array_equal(tr.read_buffer("comb", fs.ft_in * F), (w[:kb] + w[kb:]).reshape(-1))


def test_steps_alternate_between_inside_and_outside_batches():
    """The generic gradient kernels are launched only for the batches that have a row outside its slice: training steps on
    such a mix leave what gradient and optimizer run apart leave."""
    F, l1, l2, B = 256, 8, 16, 256
    fs = tb.FEATURE_SETS["halfka-hm-merged"]
    rng = np.random.default_rng(5)
    init = _perturb(tb.layerstack_default_init(fs, F, l1, l2, 9), rng, ["ft_b", "l1_b", "l1_shared_bias", "l2_b", "l3_b"])
    init["ft_w"][:fs.ft_in * F] *= 30.0
    a, b, c = (tb.GpuTrainer(B, F, l1, l2, 9, fs, optimizer="adamw", init=init) for _ in range(3))
    loss = tb.LossKind.sigmoid()
    for i in range(8):
        batch = tb.synthetic_batch(tb.SYNTH_SEED + i, B, fs)
        if i in (1, 2, 5):
            batch.nstm_indices[i, 3] = (batch.nstm_indices[i, 4] + fs.piece_inputs) % fs.ft_in
        a.train_step(batch, 1e-3, 0.25, loss)
        b.forward_backward(batch, 0.25, loss)
        b.apply_optimizer(1e-3)
        c.stage_batch(i % 3, batch)
        c.train_step_staged(i % 3, 1e-3, 0.25, loss)
    for name in a.group_names:
        x = a.download_group(name, ("w", "m", "v"))
        for other in (b, c):
            y = other.download_group(name, ("w", "m", "v"))
            assert all(np.array_equal(x[k].view(np.uint32), y[k].view(np.uint32)) for k in x), name
