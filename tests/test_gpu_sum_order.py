"""The order in which fp32 sums are added up.  It is part of what a step returns: AdamW's first steps are normalised and not
bias-corrected, so two correct orders can leave states that differ in the first digits after a few steps.  Every sum is added
up again here, term by term in the stated order, and has to come out bit for bit."""
import ctypes as C

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


@pytest.mark.parametrize("kb,half", [(1, False), (9, False), (10, False), (16, False), (45, False), (46, False), (81, False), (82, False),
                                     (45, True), (82, True)])
def test_virtual_row_gradient_is_one_chain_over_the_king_buckets(kb, half):
    """The fused kernel up to 81 king buckets, the two data-parallel ones above.  half: gradient rows that carry a loss scale, here
    no power of two, which is taken out of every term, rounded, before it is added."""
    fs = tb.FeatureSetSpec("test", 4, kb, 24, 8, True)
    F, l1, l2, B = 256, 8, 16, 496
    rng = np.random.default_rng(kb)
    init = _perturb(tb.layerstack_default_init(fs, F, l1, l2, 9), rng, ["ft_w", "ft_b", "l1_b", "l1_shared_bias", "l2_b", "l3_b"])
    d = random_index_batch(rng, B, fs.max_active, fs.piece_inputs, 1, fs.max_active)
    for key in ("stm", "nstm"):
        d[key] = np.where(d[key] >= 0, d[key] + rng.integers(0, kb, B)[:, None] * fs.piece_inputs, d[key]).astype(np.int32)
    precision = tb.PrecisionFlags(ft_fp16=half, ft_fp16_out=half)
    tr = tb.GpuTrainer(B, F, l1, l2, 9, fs, optimizer="adamw", precision=precision, init=init)
    tr.forward_backward(tb.BatchData(d["stm"], d["nstm"], d["nnz"], d["score"], d["wdl"], d["bucket"]), 0.0, tb.LossKind.sigmoid())
    tr.apply_optimizer(1e-3)
    g = tr.download_grad("ft_w").reshape(kb + 1, -1)
    want = np.zeros_like(g[0])
    for k in range(kb):
        want += g[k]
    assert np.count_nonzero(want) > want.size // 2
    if half:  # downloaded gradients have the loss scale taken out, of the virtual rows once more
        want *= np.float32(1) / (np.float32(16384) * np.float32(B))
    _same_bits(g[kb], want, "virtual rows")


# ---- fp32 arithmetic of the kernels: a product and its addition are rounded once (80-bit sums of exact products, rounded to
# 24 bits: the same unless the 64-bit sum lies exactly between two floats, which random terms do not)
def _fma(a, b, c):
    return (np.asarray(a, np.longdouble) * np.asarray(b, np.longdouble) + np.asarray(c, np.longdouble)).astype(np.float32)


def _chain(u, v, c=None):
    """c + u[0] v[0] + u[1] v[1] + .., one after the other; the terms along the first axis."""
    acc = np.zeros(np.broadcast_shapes(u.shape[1:], v.shape[1:]), np.float32) if c is None else np.broadcast_to(c, np.broadcast_shapes(u.shape[1:], v.shape[1:]))
    for i in range(len(u)):
        acc = _fma(u[i], v[i], acc)
    return acc


def _halves(t):
    """Lane sums of a warp: lanes l and l + 16 first, then l and l + 8, .."""
    while len(t) > 1:
        t = t[: len(t) // 2] + t[len(t) // 2:]
    return t[0]


def _runs(u, v, order, seg, split):
    """Sums of u[b] v[b] over the segments' positions: equal runs of one chain each, added by a warp's lanes."""
    out = []
    for beg, end in zip(seg[:-1], seg[1:]):
        per = -(-(end - beg) // split)
        run = np.zeros((split,) + np.broadcast_shapes(u.shape[1:], v.shape[1:]), np.float32)
        for s in range(split):
            at = order[beg + min(s * per, end - beg): beg + min((s + 1) * per, end - beg)]
            if len(at):
                run[s] = _chain(u[at], v[at])
        lanes = np.zeros((32,) + run.shape[1:], np.float32)
        for s in range(split):
            lanes[s % 32] += run[s]
        out.append(_halves(lanes))
    return np.stack(out)


def _crelu(x):
    return np.clip(x, np.float32(0), np.float32(1))


def _masked(x, up):
    return np.where((x > 0) & (x < 1), up, np.float32(0)).astype(np.float32)


def _trainer(arch, B, F, l1, l2, act, seed, fs=LS_FS.with_factorize(False), capacity=None):
    rng = np.random.default_rng(seed)
    cap = capacity or B
    if arch == "layerstack":
        init = _perturb(tb.layerstack_default_init(fs, F, l1, l2, 9), rng, ["ft_b", "l1_b", "l1_shared_bias", "l2_w", "l2_b", "l3_w", "l3_b"])
        tr = tb.GpuTrainer(cap, F, l1, l2, 9, fs, optimizer="adamw", init=dict(init, ft_w=init["ft_w"] * 30))
    else:
        init = _perturb(tb.simple_default_init(fs, F, l1, l2, pairwise=act == "pairwise"), rng, ["ft_b", "l1_b", "l2_w", "l2_b", "l3_w", "l3_b"])
        tr = tb.SimpleGpuTrainer(cap, F, l1, l2, fs, activation=act, optimizer="adamw", init=dict(init, ft_w=init["ft_w"] * 30))
    batch = tb.synthetic_batch(tb.SYNTH_SEED + seed, B, fs, with_bucket=arch == "layerstack")
    if arch == "layerstack":
        batch.bucket_idx[:] = np.where(rng.random(B) < 0.4, 3, rng.choice([0, 1, 8, 9, -1], B)).astype(np.int32)  # some empty, some out of range
    tr.forward_backward(batch, 0.25, tb.LossKind.sigmoid())
    return tr, init, batch, rng


def _segments(batch, B, nb):
    key = np.zeros(B, np.int64) if nb == 0 else np.where((batch.bucket_idx >= 0) & (batch.bucket_idx < nb), batch.bucket_idx, nb)
    return np.argsort(key, kind="stable"), np.concatenate([[0], np.cumsum(np.bincount(key, minlength=nb + 1))])


@pytest.mark.parametrize("arch,l1,l2,B,act", [
    # blocks of 64, 32, 64 and 128 threads; l1 = 32: 64 and 128
    ("layerstack", 8, 16, 16, ""), ("layerstack", 16, 32, 1040, ""), ("layerstack", 16, 32, 8208, ""), ("layerstack", 16, 16, 21136, ""),
    ("layerstack", 8, 16, 36496, ""),
    ("layerstack", 32, 32, 400, ""), ("layerstack", 32, 16, 8208, ""), ("layerstack", 32, 32, 41616, ""),
    # blocks of 64, 32, 128 and 256 threads, the last one in one and in two rounds
    ("simple", 8, 32, 16, "crelu"), ("simple", 32, 32, 4112, "crelu"), ("simple", 16, 16, 16400, "screlu"),
    ("simple", 32, 32, 20000, "crelu"), ("simple", 32, 16, 33008, "pairwise")])
def test_small_layers(arch, l1, l2, B, act):
    F = 256
    tr, w, batch, _ = _trainer(arch, B, F, l1, l2, act, B + l1)
    ls = arch == "layerstack"
    x = tr.read_buffer("l1_total", B * l1).reshape(B, l1)
    dy, dl1 = tr.read_buffer("dy", B), tr.read_buffer("dl1_total", B * l1).reshape(B, l1)
    order, seg = _segments(batch, B, 9 if ls else 0)
    g = np.clip(batch.bucket_idx.astype(np.int64), 0, 8) if ls else np.zeros(B, np.int64)
    live = (batch.bucket_idx >= 0) & (batch.bucket_idx < 9) if ls else np.ones(B, bool)
    sqr = (lambda a: a * a) if act == "screlu" else (lambda a: a)
    if ls:
        m = x[:, : l1 - 1]
        v = _crelu(np.concatenate([m * m * np.float32(127.0 / 128.0), m], 1))
        w2, b2, w3 = w["l2_w"].reshape(9, l2, -1)[g], w["l2_b"].reshape(9, l2)[g], w["l3_w"].reshape(9, l2)[g]
        b3, skip = w["l3_b"][g], x[:, l1 - 1]
    else:
        v = sqr(_crelu(x))
        w2, b2, w3 = np.broadcast_to(w["l2_w"].reshape(l1, l2).T, (B, l2, l1)), w["l2_b"].reshape(1, l2), np.broadcast_to(w["l3_w"].reshape(1, l2), (B, l2))
        b3, skip = w["l3_b"][g], None
    a2 = _crelu(_chain(v.T[:, :, None], np.moveaxis(w2, 2, 0), b2))
    act2 = sqr(a2)
    if ls and l1 == 32:
        out = _chain(act2.T, w3.T, b3)
    else:
        t = np.zeros((32, B), np.float32)
        t[:l2] = (act2 * w3).T
        out = b3 + _halves(t)
    if ls:
        out = np.where(live, out, np.float32(0)) + skip
    _same_bits(tr.read_buffer("net_output", B), out, "net output")
    up = dy[:, None] * w3
    u = _masked(a2, up) if act != "screlu" else up * _masked(a2, 2 * a2)
    d2 = np.where(live[:, None], u, np.float32(0))
    dv = _chain(d2.T[:, :, None], np.moveaxis(w2, 1, 0))
    if ls:  # the squared and the plain half of L2's inputs meet again
        ds, dm = _masked(v[:, : l1 - 1], dv[:, : l1 - 1]), _masked(v[:, l1 - 1:], dv[:, l1 - 1:])
        k = (np.float32(2) * m) * np.float32(127.0 / 128.0)
        dm = _fma(k, ds, dm) if l1 == 32 else dm + k * ds
        _same_bits(dl1, np.concatenate([dm, dy[:, None]], 1), "dl1")
    else:
        a = _crelu(x)
        _same_bits(dl1, _masked(a, dv) if act != "screlu" else dv * _masked(a, 2 * a), "dl1")
    u, act2 = np.where(live[:, None], u, np.float32(0)), np.where(live[:, None], act2, np.float32(0))
    real = slice(0, 9 if ls else 1)
    split = 64 if ls else 128
    one = np.ones((B, 1), np.float32)
    got = {k: tr.download_grad(k) for k in ("l2_w", "l2_b", "l3_w", "l3_b", "l1_b")}
    w2g = _runs(u[:, :, None], v[:, None, :], order, seg, split)[real]
    _same_bits(got["l2_w"], w2g if ls else np.moveaxis(w2g, 1, 2), "l2_w")
    _same_bits(got["l2_b"], _runs(u, one, order, seg, split)[real], "l2_b")
    _same_bits(got["l3_w"], _runs(act2, dy[:, None], order, seg, split)[real], "l3_w")
    _same_bits(got["l3_b"], _runs(dy[:, None], one, order, seg, split)[real], "l3_b")
    b1 = _runs(dl1, one, order, seg, split)
    _same_bits(got["l1_b"], b1[real], "l1_b")
    if ls:
        total = np.zeros(l1, np.float32)
        for q in b1:
            total += q
        _same_bits(tr.download_grad("l1_shared_bias"), total, "l1_shared_bias")


@pytest.mark.parametrize("arch,F,l1,B", [
    # by batch size: units of 64, 128 and 256 positions; ragged tiles, short buckets, positions without a bucket
    ("layerstack", 256, 8, 16), ("layerstack", 640, 8, 9488), ("layerstack", 256, 8, 18960),
    ("layerstack", 256, 16, 272), ("layerstack", 384, 16, 9488), ("layerstack", 256, 16, 18960),
    ("layerstack", 256, 32, 272), ("layerstack", 256, 32, 9488), ("simple", 256, 32, 1040), ("simple", 128, 16, 18960)])
def test_l1_forward_is_one_chain_over_the_inputs(arch, F, l1, B):
    tr, w, batch, _ = _trainer(arch, B, F, l1, 16, "crelu", B + l1)
    ls = arch == "layerstack"
    K = F if ls else 2 * F
    x = tr.read_buffer("combined", B * K).reshape(B, K)
    ws = w["l1_shared_weight" if ls else "l1_w"].reshape(K, l1)
    bs = w["l1_shared_bias" if ls else "l1_b"]
    weff, beff = np.broadcast_to(ws, (10, K, l1)).copy(), np.broadcast_to(bs, (10, l1)).copy()
    if ls:
        weff[:9] = np.moveaxis(w["l1_w"].reshape(9, l1, K), 1, 2) + ws
        beff[:9] = w["l1_b"].reshape(9, l1) + bs
    order, seg = _segments(batch, B, 9 if ls else 0)
    want = np.empty((B, l1), np.float32)
    for g, (beg, end) in enumerate(zip(seg[:-1], seg[1:])):
        at = order[beg:end][:: max(1, (end - beg) // 300)]  # some of every bucket
        want[at] = _chain(x[at].T[:, :, None], weff[g][:, None, :]) + beff[g]
        _same_bits(tr.read_buffer("l1_total", B * l1).reshape(B, l1)[at], want[at], "bucket %d" % g)


@pytest.mark.parametrize("arch,F,l1,B", [
    ("layerstack", 256, 8, 16), ("layerstack", 640, 8, 9488), ("layerstack", 256, 16, 1040), ("layerstack", 256, 16, 19008),
    ("layerstack", 256, 32, 1040), ("simple", 256, 32, 1040), ("simple", 128, 8, 512), ("simple", 128, 16, 40016)])
def test_l1_weight_gradient_is_chains_of_256_positions(arch, F, l1, B):
    """Whatever the batch size: units of 256 positions of a bucket, the bucket's units in order, the buckets in order."""
    tr, w, batch, _ = _trainer(arch, B, F, l1, 16, "crelu", B + l1)
    ls = arch == "layerstack"
    K = F if ls else 2 * F
    cols = np.unique(np.linspace(0, K - 1, 37).astype(int))
    x = tr.read_buffer("combined", B * K).reshape(B, K)[:, cols]
    d = tr.read_buffer("dl1_total", B * l1).reshape(B, l1)
    order, seg = _segments(batch, B, 9 if ls else 0)
    total = np.zeros((len(cols), l1), np.float32)
    got = tr.download_grad("l1_w").reshape(9, l1, K) if ls else None
    for g, (beg, end) in enumerate(zip(seg[:-1], seg[1:])):
        bucket = np.zeros_like(total)
        for u in range(beg, end, 256):
            at = order[u: min(u + 256, end)]
            bucket += _chain(x[at][:, :, None], d[at][:, None, :])
        if ls and g < 9:
            _same_bits(got[g][:, cols].T, bucket, "bucket %d" % g)
        total += bucket
    shared = tr.download_grad("l1_shared_weight" if ls else "l1_w").reshape(K, l1)
    _same_bits(shared[cols], total, "all positions")


@pytest.mark.parametrize("arch,F,l1,B,capacity,act", [
    ("layerstack", 256, 8, 16, 16, ""), ("layerstack", 256, 16, 1040, 1040, ""), ("layerstack", 384, 32, 9488, 9488, ""),
    ("layerstack", 256, 16, 18960, 18960, ""), ("layerstack", 256, 16, 1040, 20000, ""),
    ("simple", 128, 32, 1040, 1040, "crelu"), ("simple", 128, 16, 9488, 9488, "screlu"), ("simple", 128, 32, 18960, 30000, "screlu"),
    ("layerstack", 1408, 8, 9488, 9488, ""),  # more dft rows than stay in L2
    ("layerstack", 256, 12, 1040, 1040, "")])
def test_ft_bias_gradient_is_chains_of_128_positions(arch, F, l1, B, capacity, act):
    """Whatever the batch size: half units of 128 positions, then a warp's lanes.  The general kernel (l1 = 12): tiles dealt to as
    many chains as the trainer's capacity gives."""
    tr, w, batch, _ = _trainer(arch, B, F, l1, 16, act, B + l1, capacity=capacity)
    ls = arch == "layerstack"
    dft = [tr.read_buffer(k, B * F).reshape(B, F) for k in ("dft_stm", "dft_nstm")]
    order, seg = _segments(batch, B, 9 if ls else 0)
    lane_rows = 2 * ((capacity // 32 + 11) // 8 + 11)
    lanes = np.zeros((32, F), np.float32)
    if l1 == 12:
        lane_rows = max(296, lane_rows)
        tiles = [order[b: min(b + 32, end)] for beg, end in zip(seg[:-1], seg[1:]) for b in range(beg, end, 32)]
        chains = [np.concatenate([t for t in tiles[r::lane_rows]] or [[]]).astype(int) for r in range(lane_rows)]
    else:
        chains = []
        for beg, end in zip(seg[:-1], seg[1:]):
            for u in range(beg, end, 256):
                unit = order[u: min(u + 256, end)]
                chains += [unit[:128], unit[128:]]
    for p in range(2):
        for r, at in enumerate(chains):
            row = np.zeros(F, np.float32)
            for b in at:
                row += dft[p][b]
            lanes[(p * lane_rows + r) % 32] += row
    _same_bits(tr.download_grad("ft_b"), _halves(lanes), "ft_b")


def _scalars(optimizer, step):
    """Step size, whether the value is divided by the root of the second moment, beta1 (pointwise/radam_step.rs:63-86)."""
    libm = C.CDLL("libm.so.6")
    libm.powf.restype, libm.powf.argtypes = C.c_float, [C.c_float, C.c_float]
    f = np.float32
    b1, b2, t = f(0.99 if optimizer == "ranger" else 0.9), f(0.999), f(step)
    if optimizer == "adamw":
        return f(1), True, b1
    b2t, top = f(libm.powf(b2, t)), f(2) / (f(1) - b2) - f(1)
    n, bc = top - f(2) * t * b2t / (f(1) - b2t), f(1) - f(libm.powf(b1, t))
    if not n > 5:
        return f(1) / bc, False, b1
    return np.sqrt((f(1) - b2t) * ((n - f(4)) / (top - f(4))) * ((n - f(2)) / n) * (top / (top - f(2)))) / bc, True, b1


@pytest.mark.parametrize("factorize", [False, True])
@pytest.mark.parametrize("optimizer", ["adamw", "radam", "ranger"])
def test_update_rounds_the_same_products(optimizer, factorize):
    """Which of two products is rounded before they are added, for every kernel and step: small groups, a plain table, a factorized
    one with its virtual rows; before and after the second moment counts (step 6), on the look-ahead (6) and beside it."""
    f = np.float32
    fs = tb.FeatureSetSpec("test", 4, 10, 40, 8, factorize)
    F, l1, l2, B, lr = 256, 8, 16, 256, 1e-3
    rng = np.random.default_rng(7)
    init = _perturb(tb.layerstack_default_init(fs, F, l1, l2, 9), rng, ["ft_w", "ft_b", "l1_b", "l1_shared_bias", "l2_b", "l3_b"])
    d = random_index_batch(rng, B, fs.max_active, fs.piece_inputs, 1, fs.max_active)
    for key in ("stm", "nstm"):
        d[key] = np.where(d[key] >= 0, d[key] + rng.integers(0, 10, B)[:, None] * fs.piece_inputs, d[key]).astype(np.int32)
    tr = tb.GpuTrainer(B, F, l1, l2, 9, fs, optimizer=optimizer, init=init)
    batch = tb.BatchData(d["stm"], d["nstm"], d["nnz"], d["score"], d["wdl"], d["bucket"])
    for step in range(1, 9):
        before = {g: tr.download_group(g, ("w", "m", "v", "slow")) for g in tr.group_names}
        tr.train_step(batch, lr, 0.0, tb.LossKind.sigmoid())
        size, denom, b1 = _scalars(optimizer, step)
        lerp = optimizer == "ranger" and step % 6 == 0
        rate, b2 = f(lr) * size, f(0.999)
        decay = _fma(-f(0.01), rate, f(1))
        for name in tr.group_names:
            old, new, g = before[name], tr.download_group(name, ("w", "m", "v", "slow")), tr.download_grad(name)
            gm, gv = f(1) - b1, (f(1) - b2) * g
            table = name == "ft_w"
            if table and factorize:
                m, v = _fma(gm, g, b1 * old["m"]), _fma(gv, g, b2 * old["v"])
            else:
                m, v = _fma(b1, old["m"], gm * g), _fma(b2, old["v"], gv * g)
            _same_bits(new["m"], m, "%s m, step %d" % (name, step))
            _same_bits(new["v"], v, "%s v, step %d" % (name, step))
            val = m / (np.sqrt(v) + f(1e-8)) if denom else m
            fused = np.full(g.size, lerp if table and not factorize else denom and not table)
            if table and factorize:
                fused[fs.ft_in * F + 3:: 4] = True
            w = np.where(fused, _fma(-rate, val, old["w"] * decay), _fma(old["w"], decay, -(rate * val)))
            if not table:
                w = np.clip(w, -f(127.0 / 64.0), f(127.0 / 64.0)) if name in ("l1_w", "l1_shared_weight", "l2_w", "l3_w") else w
            if lerp:
                w = f(0.5) * w + f(0.5) * old["slow"]
            _same_bits(new["w"], w, "%s w, step %d" % (name, step))
