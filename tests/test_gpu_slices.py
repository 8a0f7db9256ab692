"""Slice-resident FT kernels off the shapes they were first built for: the feature sets of 1710 rows per king bucket (a
narrower block in the forward), slices of very different sizes and empty ones."""
import numpy as np
import pytest

import oracle_lib as O
import tatara_b200 as tb
from helpers import assert_close, assert_close_scaled, ft_path, random_index_batch
from test_gpu_parity import _batch_dict, _check_step, _oracle_for, _perturb, _sync_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fs,F,B", [("halfka-hm-split", 384, 3920), ("halfka-split", 256, 6992)])
def test_split_sets_step_matches_oracle(fs, F, B):
    fs = tb.FEATURE_SETS[fs].with_factorize(False)
    l1, l2 = 16, 32
    init = _perturb(tb.layerstack_default_init(fs, F, l1, l2, 9), np.random.default_rng(F), ["ft_b", "l1_b", "l1_shared_bias", "l2_b", "l3_b"])
    init["ft_w"] *= 30.0
    tr = tb.GpuTrainer(B, F, l1, l2, 9, fs, optimizer="adamw", init=init)
    ot = _oracle_for(tr, "layerstack", fs, F, l1, l2, 9, "adamw", (0.01, 0.01, 0.01), B)
    _sync_weights(tr, ot, init)
    batch = tb.synthetic_batch(tb.SYNTH_SEED + B, B, fs)
    _check_step(tr, ot, batch, tb.LossKind.sigmoid(), O.sigmoid_loss(), 1e-3, "layerstack", B, F, l1)
    assert ft_path(tr, batch, tb.LossKind.sigmoid()) == "slices"


@pytest.mark.parametrize("B,share,rows", [(96, 0.5, 40), (4096, 0.6, 1629), (9008, 0.97, 1629)])
def test_uneven_slices_step_matches_oracle(B, share, rows):
    """`share` of the items in one slice (runs of 4096, chunk groups of four), the rest in a few others, most slices empty; the
    smallest batch on a table of few rows, since a large one would send it to the gather kernels."""
    F, l1, l2 = 256, 8, 16
    fs = tb.FeatureSetSpec("test", 4, 45, rows, 40, False)
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
    assert ft_path(tr, batch, tb.LossKind.sigmoid()) == "slices"


@pytest.mark.parametrize("arch,act", [("layerstack", ""), ("simple", "crelu"), ("simple", "screlu"), ("simple", "pairwise")])
def test_a_row_outside_its_slice_in_a_batch_large_enough_for_slices(arch, act):
    """Every activation on slices, and then with one row outside, where the generic kernels do the gradient behind slice kernels
    that return at once; the next batch is on slices again."""
    F, l1, l2, B = 256, 16, 32, 3680
    fs = tb.FEATURE_SETS["halfka-hm-merged"].with_factorize(False)
    rng = np.random.default_rng(len(act))
    for seed, outside in ((1, False), (2, True), (3, False)):
        if arch == "layerstack":
            init = _perturb(tb.layerstack_default_init(fs, F, l1, l2, 9), rng, ["ft_b", "l1_b", "l1_shared_bias", "l2_b", "l3_b"])
        else:
            init = _perturb(tb.simple_default_init(fs, F, l1, l2, pairwise=act == "pairwise"), rng, ["ft_b", "l1_b", "l2_b", "l3_b"])
        init["ft_w"] *= 30.0
        if arch == "layerstack":
            tr = tb.GpuTrainer(B, F, l1, l2, 9, fs, optimizer="adamw", init=init)
            ot = _oracle_for(tr, "layerstack", fs, F, l1, l2, 9, "adamw", (0.01, 0.01, 0.01), B)
        else:
            tr = tb.SimpleGpuTrainer(B, F, l1, l2, fs, activation=act, optimizer="adamw", weight_decay=0.0, init=init)
            ot = _oracle_for(tr, "simple", fs, F, l1, l2, 0, "adamw", (0.0, 0.0, 0.0), B, activation={"crelu": 0, "screlu": 1, "pairwise": 2}[act])
        _sync_weights(tr, ot, init)
        batch = tb.synthetic_batch(tb.SYNTH_SEED + seed, B, fs, with_bucket=arch == "layerstack")
        if outside:
            batch.nstm_indices[1234, 3] = (batch.nstm_indices[1234, 4] + fs.piece_inputs) % fs.ft_in
        if act == "pairwise":  # the raw sums are kept and the L1 input is ft_out wide
            tr.forward_backward(batch, 0.25, tb.LossKind.sigmoid())
            ot.step(_batch_dict(batch), 1e-3, 0.25, O.sigmoid_loss(), do_optimizer=False)
            assert np.array_equal(tr.read_buffer("ft_stm", B * F).view(np.uint32), ot.buffer("ft_stm").view(np.uint32))
            for name in ot.names:
                assert_close_scaled(tr.download_grad(name), ot.group(name, "grad"), 1e-4, "grad " + name)
        else:
            _check_step(tr, ot, batch, tb.LossKind.sigmoid(), O.sigmoid_loss(), 1e-3, arch, B, F, l1)
        assert ft_path(tr, batch, tb.LossKind.sigmoid()) == ("both" if outside else "slices")


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
    F, l1, l2, B = 256, 8, 16, 3680
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
        if i < 2:
            assert ft_path(b, batch, loss) == ("both" if i == 1 else "slices")
    for name in a.group_names:
        x = a.download_group(name, ("w", "m", "v"))
        for other in (b, c):
            y = other.download_group(name, ("w", "m", "v"))
            assert all(np.array_equal(x[k].view(np.uint32), y[k].view(np.uint32)) for k in x), name
