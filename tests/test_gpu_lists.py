"""The FT weight gradient over global lists (counting sort, sorting in shared memory, column strips, split rows) at the
sizes where its pieces change: list lengths around the in-block sort's limits and around the parts of split rows, one and
four rows per warp, whole rows, even and ragged column strips, list room that crosses a scan block."""
import ctypes as C

import numpy as np
import pytest

import tatara_b200 as tb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,F,N,A,lengths", [
    (1, 128, 1, 1, (1,)),
    (513, 256, 4099, 5, (2, 63, 64, 65, 513)),               # four rows per warp
    (700, 384, 300, 7, (31, 33, 255, 256, 257, 700)),        # one row per warp
    (4099, 128, 2050, 4, (4095, 4096, 4097)),                # split rows
    (14000, 1408, 4200, 6, (8193, 300, 9)),                  # two strips, the second one shorter
    (20000, 1024, 2100, 3, (5000, 64)),                      # two equal strips
    (300, 4096, 97, 9, (300, 20)),                           # the widest rows
])
def test_lists_match_the_sequential_sum(B, F, N, A, lengths):
    torch = pytest.importorskip("torch")
    import oracle_lib as O
    from helpers import assert_close_scaled
    lib = tb.load_library()
    torch.cuda.set_device(0)
    rng = np.random.default_rng(B + F)
    dft = (rng.standard_normal((B, F)) * 1e-3).astype(np.float32)
    idx = rng.integers(len(lengths), max(N, len(lengths) + 1), (B, A)).astype(np.int32)   # may be out of range for N = 1
    nnz = np.full(B, A, np.int32)
    nnz[B // 2:B // 2 + 7] = 0
    for f, n in enumerate(lengths):                           # feature f is held by n positions, through one column
        if f < A:
            idx[rng.permutation(B)[:n], f] = f
    if B > 10:
        idx[5, :2] = len(lengths)                             # a feature twice in one row
        idx[6, 0] = -1
    want = np.zeros((N, F), np.float32)
    O.lib().ora_sparse_ft_backward(dft.reshape(-1), np.where(np.arange(A)[None] < nnz[:, None], idx, -1).reshape(-1).astype(np.int32),
                                   want.reshape(-1), B, F, N, A)
    d = [torch.from_numpy(x).cuda() for x in (dft, idx, nnz)]
    grad = torch.full((N, F), 7.0, device="cuda")
    err = C.create_string_buffer(256)
    rc = lib.tb_ft_backward_static_scratch(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), B, F, N, A, grad.data_ptr(),
                                           torch.cuda.current_stream().cuda_stream, err, 256)
    assert rc == 0, err.value
    got = grad.cpu().numpy()
    held = np.bincount(idx[(np.arange(A)[None] < nnz[:, None]) & (idx >= 0) & (idx < N)].reshape(-1), minlength=N)
    whole = held <= 4096                                      # these rows: the sequential sum itself
    assert np.array_equal(got[whole].view(np.uint32), want[whole].view(np.uint32))
    assert_close_scaled(got, want, 1e-5, "gradient")
