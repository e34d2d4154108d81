"""The FP64 LU and its solve at the sizes where their tiles, copies and fallbacks meet: panel and
row-block edges, odd orders (factored in a copy with aligned rows), row strides beyond the order
(odd and even), updates with fewer tiles than SMs and with several per group, and rejected panels factored
in shared memory and in place.  Against scipy's LAPACK."""

import numpy as np
import pytest
import scipy.linalg as la

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def _system(n, swapped, seed):
    """-2 pi I plus noise; the diagonal blocks of the `swapped` panels are antidiagonal, so that these
    panels interchange rows."""
    rng = np.random.default_rng(seed)
    A = rng.normal(size=(n, n)) * 1e-3 - 2 * np.pi * np.eye(n)
    for p in swapped:
        c0, m = 64 * p, min(64, n - 64 * p)
        A[c0:c0 + m, c0:c0 + m] = rng.normal(size=(m, m)) * 1e-3
        A[c0 + np.arange(m), c0 + m - 1 - np.arange(m)] -= 2 * np.pi
    return A, rng.normal(size=n)


@pytest.mark.parametrize("n,pad,swapped", [
    (1, 0, ()), (2, 1, ()), (63, 0, ()), (64, 3, ()), (65, 0, ()), (127, 1, ()), (128, 0, ()), (129, 2, ()),
    (192, 1, (0,)), (513, 0, (0, 8)), (640, 0, (0, 9)), (1023, 0, (15,)), (1024, 5, ()), (1281, 0, (13, 14)),
    (2110, 0, ()), (2178, 0, (1,)),
])
def test_lu_and_solve_match_lapack(n, pad, swapped):
    import torch

    from pyvl_b200 import _lib
    from pyvl_b200.device import ptr, stream_ptr

    A, b = _system(n, swapped, n + pad)
    lda = n + pad
    store = torch.full((n, lda), float("nan"), dtype=torch.float64, device="cuda")
    store[:, :n] = torch.as_tensor(A)
    ipiv = torch.zeros(2 * n, dtype=torch.int32, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    nb = int(_lib.query("pvl_lu_workspace", n))
    ws = torch.full((nb + 256,), 255, dtype=torch.uint8, device="cuda")  # NaNs: nothing is read before it is written
    x = torch.as_tensor(b, device="cuda")
    _lib.call("pvl_lu_factor", n, ptr(store), lda, ptr(ipiv), ptr(info), ptr(ws), nb, stream_ptr())
    _lib.call("pvl_lu_solve", n, ptr(store), lda, ptr(ipiv), ptr(x), ptr(err), ptr(ws), nb, stream_ptr())
    torch.cuda.synchronize()
    assert int(info.item()) == 0 and int(err.item()) == 0
    lu, piv = la.lu_factor(A)
    p = ipiv.cpu().numpy()
    assert np.array_equal(p[:n], piv)
    rows = np.arange(n)
    for i, q in enumerate(piv):
        rows[[i, q]] = rows[[q, i]]
    assert np.array_equal(p[n:], rows)
    assert rel(store[:, :n].cpu().numpy(), lu) <= 1e-13
    if pad:
        assert bool(torch.isnan(store[:, n:]).all())  # the rows' padding is not written
    assert rel(x.cpu().numpy(), la.lu_solve((lu, piv), b)) <= 1e-12


def test_solution_with_the_bits_of_the_not_ready_mark():
    """A NaN whose bits are those of the solve's "not ready" mark passes through as a NaN and does not
    make later blocks wait."""
    import torch

    from pyvl_b200 import _lib
    from pyvl_b200.device import ptr, stream_ptr

    n = 256
    A, b = _system(n, (), 1)
    LU = torch.as_tensor(A, device="cuda")
    ipiv = torch.zeros(2 * n, dtype=torch.int32, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    nb = int(_lib.query("pvl_lu_workspace", n))
    ws = torch.zeros(nb, dtype=torch.uint8, device="cuda")
    _lib.call("pvl_lu_factor", n, ptr(LU), n, ptr(ipiv), ptr(info), ptr(ws), nb, stream_ptr())
    x = torch.as_tensor(b, device="cuda")
    x.view(torch.int64)[70] = -1  # all bits set
    _lib.call("pvl_lu_solve", n, ptr(LU), n, ptr(ipiv), ptr(x), ptr(err), ptr(ws), nb, stream_ptr())
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    assert bool(torch.isnan(x).any())


def test_workspace_of_an_accepted_factorisation_reused_for_a_rejected_one():
    """The panels of the second matrix interchange rows where the first one's did not: their swaps and row
    blocks are formed although the workspace remembers accepted panels."""
    import torch

    from pyvl_b200 import _lib
    from pyvl_b200.device import ptr, stream_ptr

    n = 640
    ipiv = torch.zeros(2 * n, dtype=torch.int32, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    nb = int(_lib.query("pvl_lu_workspace", n))
    ws = torch.zeros(nb, dtype=torch.uint8, device="cuda")
    for swapped in ((), (0, 3, 4, 9), (), tuple(range(10))):
        A, _ = _system(n, swapped, 5)
        M = torch.as_tensor(A, device="cuda")
        _lib.call("pvl_lu_factor", n, ptr(M), n, ptr(ipiv), ptr(info), ptr(ws), nb, stream_ptr())
        lu, piv = la.lu_factor(A)
        assert np.array_equal(ipiv[:n].cpu().numpy(), piv)
        assert rel(M.cpu().numpy(), lu) <= 1e-13


@pytest.mark.parametrize("n", [1, 2, 31, 63, 65])
def test_backup_stays_inside_its_rows(n):
    """A panel's backup has n rows of 64 values at the head of the workspace; the region behind it, the FP32
    factorisation's top block, is not the FP64 one's to write."""
    import torch

    from pyvl_b200 import _lib
    from pyvl_b200.device import ptr, stream_ptr

    A, b = _system(n, (), n)
    M = torch.as_tensor(A, device="cuda")
    ipiv = torch.zeros(2 * n, dtype=torch.int32, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    nb = int(_lib.query("pvl_lu_workspace", n))
    ws = torch.full((nb,), 255, dtype=torch.uint8, device="cuda")
    _lib.call("pvl_lu_factor", n, ptr(M), n, ptr(ipiv), ptr(info), ptr(ws), nb, stream_ptr())
    begin = -(-n * 64 * 8 // 256) * 256
    assert bool((ws[begin:begin + 64 * 64 * 8] == 255).all())
    assert rel(M.cpu().numpy(), la.lu_factor(A)[0]) <= 1e-13


@pytest.mark.parametrize("n,pad,swapped", [
    (130, 3, ()), (130, 1, (2,)), (706, 1, ()), (706, 1, (0, 11)), (2110, 1, ()), (2110, 3, (31, 32)),
])
def test_odd_row_strides_with_ragged_last_panels(n, pad, swapped):
    """An even order with an odd row stride is factored in place with 8-byte copies: partial last panels
    after an update, and trailing tiles that are not full."""
    test_lu_and_solve_match_lapack(n, pad, swapped)


@pytest.mark.parametrize("n,lda,swapped", [(64, 64, ()), (130, 132, (2,)), (706, 706, ()), (706, 708, (0, 11))])
def test_matrix_that_is_not_16_byte_aligned(n, lda, swapped):
    """An even order and row stride, but a base 8 bytes off a 16-byte boundary."""
    import torch

    from pyvl_b200 import _lib
    from pyvl_b200.device import ptr, stream_ptr

    A, b = _system(n, swapped, n + lda)
    store = torch.full((n * lda + 1,), float("nan"), dtype=torch.float64, device="cuda")
    M = store[1:].view(n, lda)
    assert M.data_ptr() % 16 == 8
    M[:, :n] = torch.as_tensor(A)
    ipiv = torch.zeros(2 * n, dtype=torch.int32, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    nb = int(_lib.query("pvl_lu_workspace", n))
    ws = torch.full((nb,), 255, dtype=torch.uint8, device="cuda")
    x = torch.as_tensor(b, device="cuda")
    _lib.call("pvl_lu_factor", n, ptr(M), lda, ptr(ipiv), ptr(info), ptr(ws), nb, stream_ptr())
    _lib.call("pvl_lu_solve", n, ptr(M), lda, ptr(ipiv), ptr(x), ptr(err), ptr(ws), nb, stream_ptr())
    torch.cuda.synchronize()
    assert int(info.item()) == 0 and int(err.item()) == 0
    lu, piv = la.lu_factor(A)
    assert np.array_equal(ipiv[:n].cpu().numpy(), piv)
    assert rel(M[:, :n].cpu().numpy(), lu) <= 1e-13
    assert bool(torch.isnan(M[:, n:]).all()) and bool(torch.isnan(store[:1]).all())
    assert rel(x.cpu().numpy(), la.lu_solve((lu, piv), b)) <= 1e-12
