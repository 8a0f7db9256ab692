"""Which FT kernels a batch takes is a matter of its size: slice-resident ones or the gather over global lists, the positions
sorted by one block or with the items.  Training steps and validation on both sides of every line, against the oracle."""
import numpy as np
import pytest

import oracle_lib as O
import tatara_b200 as tb
from helpers import assert_close
from test_gpu_parity import TOL_FWD, _batch_dict, _check_step, _oracle_for, _perturb, _sync_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fs,F,B", [
    ("halfka-hm-split", 256, 3840), ("halfka-hm-split", 256, 3856),    # four entries per table row
    ("halfka-hm-split", 256, 4800), ("halfka-hm-split", 256, 4816),    # validation: five
    ("halfka-split", 256, 8192), ("halfka-split", 256, 8208),          # one block sorts 8192 positions
    ("halfka-hm-merged", 1536, 1360), ("halfka-hm-merged", 1536, 1376),  # 640 MB of rows
    ("halfkp", 256, 16), ("halfkp", 256, 1056),
])
def test_step_and_validation_match_oracle(fs, F, B):
    fs = tb.FEATURE_SETS[fs].with_factorize(False)
    l1, l2 = 8, 16
    init = _perturb(tb.layerstack_default_init(fs, F, l1, l2, 9), np.random.default_rng(B), ["ft_b", "l1_b", "l1_shared_bias", "l2_b", "l3_b"])
    init["ft_w"] *= 30.0
    tr = tb.GpuTrainer(B, F, l1, l2, 9, fs, optimizer="adamw", init=init)
    ot = _oracle_for(tr, "layerstack", fs, F, l1, l2, 9, "adamw", (0.01, 0.01, 0.01), B)
    _sync_weights(tr, ot, init)
    batch = tb.synthetic_batch(tb.SYNTH_SEED + B, B, fs)
    _check_step(tr, ot, batch, tb.LossKind.sigmoid(), O.sigmoid_loss(), 1e-3, "layerstack", B, F, l1)
    loss, out = tr.validate_step(batch, 0.25, tb.LossKind.sigmoid())
    want_loss, want = ot.validate(_batch_dict(batch), 0.25, O.sigmoid_loss())
    assert_close(out, want, TOL_FWD, "net output")
    assert abs(loss - want_loss) <= TOL_FWD * (1 + abs(want_loss))
