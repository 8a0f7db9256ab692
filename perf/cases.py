"""What a user of this package has it do, as cases that can be prepared, run and compared.

Four kinds of work, all through the public entry points:

  train     STEPS training steps on two alternating host batches and the flush of the last loss: the inner loop of a
            trainer (LayerStack or Simple net, index arrays or 40-byte records as the feed, every precision mode)
  validate  forward and loss of one host batch, the net outputs read back
  extract   40-byte records on the host -> index arrays, buckets and targets on the host: what a data loader calls
  backward  the FT weight gradient alone on the caller's device tensors (the entry point that allocates nothing)

A case is a dict of plain values; `listed()` holds the ones that are always measured, `draw(rng)` gives more of the
same ranges.
"""
import ctypes as C
import math

import numpy as np
import torch

import tatara_b200 as tb

STEPS = 6          # one full period of the Ranger look-ahead, which touches a fourth table on every sixth step
LR = 8.75e-4       # the training command's default learning rate
PRECISIONS = {
    "fp32": tb.PrecisionFlags(),
    "tf32": tb.PrecisionFlags(tf32=True),
    "all-optim": tb.PrecisionFlags(tf32=True, ft_fp16=True, ft_fp16_out=True, fp16_opt_state=True),
}
LOSSES = {
    "sigmoid": tb.LossKind.sigmoid(1.0 / 290.0),
    "wrm": tb.LossKind.wrm(nnue2score=290.0, in_scaling=290.0, in_offset=0.0, target_offset=0.0, target_scaling=290.0),
}


# ---- the cases ---------------------------------------------------------------------------------------------------
def _layerstack(kind, name, **kw):
    c = dict(kind=kind, arch="layerstack", fs="halfka-hm-merged", ft_out=1536, l1=16, l2=32, batch=65536, optimizer="ranger",
             factorize=True, loss="sigmoid", precision="fp32", activation="pairwise", feed="arrays", pinned=True)
    c.update(kw)
    return dict(c, name=name) if name else c


def _simple(kind, name, **kw):
    c = dict(kind=kind, arch="simple", fs="halfkp", ft_out=256, l1=32, l2=32, batch=65536, optimizer="adamw", factorize=True,
             loss="wrm", precision="fp32", activation="crelu", feed="arrays", pinned=True)
    c.update(kw)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the headline configuration: the largest net, full batches, index arrays from the loader's page-locked buffers
        _layerstack("train", "train_ls1536"),
        # the same net in the reduced-precision mode that production runs use, fed with packed records
        _layerstack("train", "train_ls1536_alloptim", precision="all-optim", feed="records"),
        # the mid-size net at the default batch size, fed with packed records
        _layerstack("train", "train_ls768_b16k", ft_out=768, l1=8, batch=16384, feed="records"),
        # a small experiment: narrow net and small batches from ordinary arrays, where latency and launches count
        _layerstack("train", "train_ls256_b1k", ft_out=256, batch=1024, pinned=False),
        # the Simple architecture's standard net
        _simple("train", "train_simple256", feed="records"),
        # another feature set (split king planes), activation and optimizer, no factorizer, a ragged batch
        _simple("train", "train_simple512_split", fs="halfka-hm-split", ft_out=512, batch=10000, activation="screlu", optimizer="radam",
                factorize=False, loss="sigmoid", pinned=False),
        # the validation pass after a superbatch, in full batches
        _layerstack("validate", "validate_ls1536", pinned=False),
        # the smallest calls: a handful of positions scored with a small net
        _layerstack("validate", "validate_ls256_b256", ft_out=256, batch=256, pinned=False),
        # the data loader's work for one full batch, and for a small odd one
        dict(kind="extract", fs="halfka-hm-merged", batch=65536, bucket=True, pinned=True, name="extract_64k"),
        dict(kind="extract", fs="halfkp", batch=1000, bucket=False, pinned=False, name="extract_1k"),
        # the FT weight gradient alone, on lists spread over the whole feature space and on a small problem
        dict(kind="backward", fs="halfka-hm-merged", ft_out=1536, batch=16384, name="backward_1536_b16k"),
        dict(kind="backward", fs="halfkp", ft_out=256, batch=1000, name="backward_256_b1k"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(("train", "train", "train", "train", "validate", "validate", "extract", "backward"))
    fs = rng.choice(("halfka-hm-merged", "halfka-hm-merged", "halfka-hm-merged", "halfkp", "halfka-split", "halfka-merged", "halfka-hm-split"))
    spec = tb.FEATURE_SETS[fs]
    if kind == "extract":
        return dict(kind=kind, fs=fs, batch=int(_log(rng, 500, 65536)), bucket=rng.random() < 0.5, pinned=rng.random() < 0.5)
    # the sets with 81 king buckets have nearly twice the table rows: half the width
    ft_out = 128 * int(round(_log(rng, 256, 1536 if spec.king_buckets == 45 else 768) / 128))
    if kind == "backward":
        return dict(kind=kind, fs=fs, ft_out=ft_out, batch=int(_log(rng, 500, 655360 // spec.max_active)))
    top = min(65536, 65536 * 1024 // ft_out)
    if spec.piece_inputs == 1710:
        top = min(top, 65536 * 512 // ft_out)
    batch = 16 * int(_log(rng, 256, top) / 16)
    common = dict(fs=fs, ft_out=ft_out, batch=batch, optimizer=rng.choice(("ranger", "radam", "adamw")), factorize=rng.random() < 0.75,
                  l2=rng.choice((16, 32)), loss=rng.choice(("sigmoid", "wrm")), pinned=rng.random() < 0.5,
                  feed=rng.choice(("arrays", "records")) if kind == "train" else "arrays")
    if rng.random() < 0.7:
        return _layerstack(kind, None, l1=rng.choice((8, 16, 32)), precision=rng.choice(("fp32", "fp32", "tf32", "all-optim")), **common)
    return _simple(kind, None, l1=rng.choice((16, 32)), activation=rng.choice(("crelu", "screlu", "pairwise")), **common)


# ---- what a program has in hand before the call ---------------------------------------------------------------------
def _feature_set(case):
    return tb.FEATURE_SETS[case["fs"]].with_factorize(bool(case.get("factorize", True)))


def _weights(case, seed):
    """Initial weights with the ranges of the default initialisers, the FT rows scaled up so that the pre-activations
    spread over and beyond the clipped range as they do during training."""
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def uniform(n, half):
        return (torch.empty(n, device="cuda").uniform_(-half, half, generator=gen)).cpu().numpy()

    fs, F, l1, l2 = _feature_set(case), case["ft_out"], case["l1"], case["l2"]
    ft_w = uniform(fs.train_ft_in * F, 30.0 / math.sqrt(fs.ft_in))
    if case["arch"] == "layerstack":
        nb, l2in = 9, 2 * (l1 - 1)
        return {"ft_w": ft_w, "ft_b": uniform(F, 0.1), "l1_w": uniform(nb * l1 * F, 0.01), "l1_b": uniform(nb * l1, 0.1),
                "l1_shared_weight": uniform(F * l1, 0.01), "l1_shared_bias": uniform(l1, 0.1), "l2_w": uniform(nb * l2 * l2in, 0.1),
                "l2_b": uniform(nb * l2, 0.1), "l3_w": uniform(nb * l2, 0.1), "l3_b": uniform(nb, 0.1)}
    K = F if case["activation"] == "pairwise" else 2 * F
    return {"ft_w": ft_w, "ft_b": uniform(F, 0.1), "l1_w": uniform(K * l1, 0.01), "l1_b": uniform(l1, 0.1), "l2_w": uniform(l1 * l2, 0.1),
            "l2_b": uniform(l2, 0.1), "l3_w": uniform(l2, 0.1), "l3_b": uniform(1, 0.1)}


def _trainer(case, seed):
    fs = _feature_set(case)
    kw = dict(optimizer=case["optimizer"], precision=PRECISIONS[case["precision"]], init=_weights(case, seed))
    if case["arch"] == "layerstack":
        return tb.GpuTrainer(case["batch"], case["ft_out"], case["l1"], case["l2"], 9, fs, **kw)
    return tb.SimpleGpuTrainer(case["batch"], case["ft_out"], case["l1"], case["l2"], fs, activation=case["activation"],
                               weight_decay=0.01, **kw)


def _records(n, seed, pinned):
    psv = tb.synthesize_psv(tb.SYNTH_SEED + seed, n)
    if not pinned:
        return psv, None
    keep = tb.PinnedArray(psv.shape, np.uint8)
    keep.array[:] = psv
    return keep.array, keep


def _random_lists(n, A, lo, hi, space, gen):
    """Per position lo..hi distinct rows of the whole feature space in random order, padded with -1 to A slots."""
    rows = torch.randint(0, space - hi, (n, hi), generator=gen, device="cuda").sort(dim=1).values + torch.arange(hi, device="cuda")
    rows = rows.gather(1, torch.rand((n, hi), generator=gen, device="cuda").argsort(dim=1))
    nnz = torch.randint(lo, hi + 1, (n,), generator=gen, device="cuda", dtype=torch.int32)
    idx = torch.full((n, A), -1, dtype=torch.int32, device="cuda")
    idx[:, :hi] = rows.to(torch.int32)
    idx[torch.arange(A, device="cuda")[None, :] >= nnz[:, None]] = -1
    return idx, nnz


def prepare(case, seed):
    kind, n = case["kind"], case["batch"]
    fs = _feature_set(case)
    if kind == "extract":
        records, keep = _records(n, seed, case["pinned"])
        return dict(case=case, fs=fs, records=records, keep=keep)
    if kind == "backward":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        idx, nnz = _random_lists(n, fs.max_active, 30, 38, fs.ft_in, gen)
        dft = torch.randn((n, case["ft_out"]), generator=gen, device="cuda") * 1e-3
        return dict(case=case, fs=fs, lib=tb.load_library(), err=C.create_string_buffer(256), idx=idx, nnz=nnz, dft=dft,
                    grad=torch.empty((fs.ft_in, case["ft_out"]), device="cuda"))
    state = dict(case=case, loss=LOSSES[case["loss"]], trainer=_trainer(case, seed))
    count = 2 if kind == "train" else 1
    if case["feed"] == "records":
        state["batches"] = [_records(n, 2 * seed + i, case["pinned"]) for i in range(count)]
    else:
        state["batches"] = [tb.synthetic_batch(tb.SYNTH_SEED + 2 * seed + i, n, fs, with_bucket=case["arch"] == "layerstack",
                                               pinned=case["pinned"]) for i in range(count)]
    return state


# ---- one pass ---------------------------------------------------------------------------------------------------------
class TrainerState(dict):
    """Weights, moments and slow weights of every parameter group by name.  They stay on the GPU, as between the steps
    of a training run; looking an entry up downloads it."""

    def __init__(self, trainer):
        super().__init__(("%s.%s" % (g, which), None) for g in trainer.group_names for which in ("w", "m", "v", "slow"))
        self._trainer = trainer

    def __getitem__(self, key):
        group, which = key.rsplit(".", 1)
        return self._trainer.download_group(group, (which,))[which]


class Arrays(list):
    """The arrays of an extracted batch; page-locked ones live as long as their batch, which is kept here."""

    def __init__(self, batch):
        super().__init__(a for a in (batch.stm_indices, batch.nstm_indices, batch.nnz, batch.score, batch.wdl, batch.bucket_idx) if a is not None)
        self._batch = batch


def _train(state):
    tr, loss, records = state["trainer"], state["loss"], state["case"]["feed"] == "records"
    losses = []
    for i in range(STEPS):
        batch = state["batches"][i % 2]
        losses.append(tr.train_step_psv(batch[0], LR, 0.0, loss) if records else tr.train_step(batch, LR, 0.0, loss))
    losses.append(tr.flush_pending_loss())  # a step returns the loss of the one before it
    return {"losses": np.array(losses), "state": TrainerState(tr)}


def run(state):
    kind = state["case"]["kind"]
    if kind == "train":
        return _train(state)
    if kind == "validate":
        return state["trainer"].validate_step(state["batches"][0], 0.0, state["loss"])
    if kind == "extract":
        b = tb.extract_batch(state["records"], state["fs"], with_bucket=state["case"]["bucket"], pinned=state["case"]["pinned"])
        return Arrays(b)
    fs, F = state["fs"], state["case"]["ft_out"]
    rc = state["lib"].tb_ft_backward_static_scratch(state["dft"].data_ptr(), state["idx"].data_ptr(), state["nnz"].data_ptr(),
                                                    state["case"]["batch"], F, fs.ft_in, fs.max_active, state["grad"].data_ptr(),
                                                    torch.cuda.current_stream().cuda_stream, state["err"], 256)
    if rc != 0:
        raise RuntimeError(state["err"].value.decode())
    return state["grad"]


# ---- what a pass cannot do without, and how close two correct results are ------------------------------------------------
def work(case):
    fs = _feature_set(case)
    n, A = case["batch"], fs.max_active
    index_bytes = n * (2 * A + 4) * 4.0
    if case["kind"] == "extract":
        return {"bytes": 40.0 * n + index_bytes, "flops": 0.0}
    F = case["ft_out"]
    if case["kind"] == "backward":
        return {"bytes": 4.0 * n * F + 4.0 * n * (A + 1) + 4.0 * fs.ft_in * F, "flops": 34.0 * n * F}
    K = F if case["activation"] == "pairwise" else 2 * F
    gather = 2.0 * n * A * F                      # additions of one walk over every index list
    dense = 2.0 * n * (K * case["l1"] * (2 if case["arch"] == "layerstack" else 1))
    half = case["precision"] == "all-optim"
    if case["kind"] == "validate":
        rows = min(fs.ft_in, 2 * n * A)           # the table rows a batch touches at most
        return {"bytes": rows * F * (2.0 if half else 4.0) + index_bytes + 4.0 * n, "flops": gather + dense}
    table = float(fs.train_ft_in) * F
    state_bytes = table * (2 * 4.0 + 4 * (2.0 if half else 4.0))   # weights and both moments, in and out
    if case["optimizer"] == "ranger":
        state_bytes += table * 2 * 4.0 / STEPS                      # slow weights, in and out once in six steps
    feed_bytes = 40.0 * n if case["feed"] == "records" else index_bytes
    return {"bytes": STEPS * (state_bytes + feed_bytes), "flops": STEPS * (2 * gather + 3 * dense + 15 * table)}


def tolerance(case):
    if case["kind"] == "extract":
        return "exact"
    if case["kind"] == "backward":
        return {"rel": 1e-5}
    if case["kind"] == "validate":
        # 32-bit sums; TF32 products carry 10 bits, fp16 rows 11
        return {"rel": 1e-5} if case["precision"] == "fp32" else {"rel": 5e-3}
    # STEPS steps through clipped activations: a hidden unit within rounding of a clipping point (a few in the millions of a
    # pass) keeps its gradient in one correct implementation and drops it in another, which moves that position's share
    # of the moments by a whole term; the relative error of the tensors stays near one position's share of the batch
    return {"rel": 2e-3, "max": 0.5} if case["precision"] == "fp32" else {"rel": 2e-2, "max": 0.9}
