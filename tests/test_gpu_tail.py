"""The tiled tail (L2, L3, loss, their gradients) over its instantiations: hidden sizes, activations, ragged blocks of 128
positions, buckets without positions and positions without a bucket."""
import numpy as np
import pytest

import oracle_lib as O
import tatara_b200 as tb
from test_gpu_parity import KP_FS, LS_FS, _check_step, _oracle_for, _perturb, _sync_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("l1,l2,B,buckets", [(8, 16, 16, "one"), (16, 16, 400, "uneven"), (32, 32, 1040, "uneven"), (32, 16, 640, "none"),
                                             (16, 32, 272, "none")])
def test_layerstack_tail(l1, l2, B, buckets):
    F, fs = 256, LS_FS.with_factorize(False)
    rng = np.random.default_rng(l1 + l2 + B)
    init = _perturb(tb.layerstack_default_init(fs, F, l1, l2, 9), rng, ["ft_b", "l1_b", "l1_shared_bias", "l2_w", "l2_b", "l3_w", "l3_b"])
    init["ft_w"] *= 30.0
    init["l2_w"] *= 4.0
    tr = tb.GpuTrainer(B, F, l1, l2, 9, fs, optimizer="adamw", init=init)
    ot = _oracle_for(tr, "layerstack", fs, F, l1, l2, 9, "adamw", (0.01, 0.01, 0.01), B)
    _sync_weights(tr, ot, init)
    batch = tb.synthetic_batch(tb.SYNTH_SEED + B, B, fs)
    if buckets == "one":
        batch.bucket_idx[:] = 4
    else:  # one bucket with most positions, some with none
        batch.bucket_idx[:] = np.where(rng.random(B) < 0.7, 2, rng.choice([0, 8], B)).astype(np.int32)
    if buckets == "none":
        batch.bucket_idx[::3] = rng.choice([9, -1, 1000], len(batch.bucket_idx[::3])).astype(np.int32)
    _check_step(tr, ot, batch, tb.LossKind.sigmoid(), O.sigmoid_loss(), 1e-3, "layerstack", B, F, l1)


@pytest.mark.parametrize("l1,l2,B,act", [(8, 32, 16, "crelu"), (16, 16, 144, "screlu"), (32, 16, 1040, "crelu"), (32, 32, 400, "screlu")])
def test_simple_tail(l1, l2, B, act):
    F, fs = 128, KP_FS.with_factorize(False)
    rng = np.random.default_rng(l1 + l2 + B)
    init = _perturb(tb.simple_default_init(fs, F, l1, l2), rng, ["ft_b", "l1_b", "l2_w", "l2_b", "l3_w", "l3_b"])
    init["ft_w"] *= 10.0
    init["l2_w"] *= 4.0
    tr = tb.SimpleGpuTrainer(B, F, l1, l2, fs, activation=act, optimizer="adamw", weight_decay=0.0, init=init)
    ot = _oracle_for(tr, "simple", fs, F, l1, l2, 1, "adamw", (0.0, 0.0, 0.0), B, activation={"crelu": 0, "screlu": 1}[act])
    _sync_weights(tr, ot, init)
    _check_step(tr, ot, tb.synthetic_batch(tb.SYNTH_SEED + B, B, fs, with_bucket=False), tb.LossKind.wrm(), O.wrm_loss(600.0, 340.0, 270.0, 270.0, 380.0),
                1e-3, "simple", B, F, l1)
