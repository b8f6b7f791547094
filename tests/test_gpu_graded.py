"""Graded operands keep FP64's entrywise accuracy.

The sums of a GEMM, an LU or an overlap are backward stable entry by entry in FP64: an
error of some K 2^-53 sum |a||b|, whatever the scales of rows, columns and modes.
Here rows, mode normalisations and fields are scaled by 20 decades or more in
opposite directions, which changes an exact result by known factors only; the results, with the
factors taken out, are held to the tolerance of the ungraded tests."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _grades(n, decades=20.0):
    return 2.0 ** np.round(np.linspace(0.0, -decades, n) * np.log2(10))


@pytest.mark.parametrize('n', [300, 700, 1300])
def test_fem_factor_of_a_badly_row_scaled_matrix(n):
    """A = D B: the interchanges and U's rows follow D, L's rows the inverse.  B is
    diagonally dominant (condition below 10): n x 10 x 2^-53 = 1.5e-12 of the largest
    entry of B^-1 at n = 1 300; 1e-11 is allowed."""
    import torch
    from emustack_b200._lib import check, lib, ptr, stream_ptr
    rng = np.random.default_rng(n)
    B = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(n) + 4 * np.eye(n)
    d = _grades(n, 60.0)
    A = torch.tensor(d[:, None] * B, device='cuda')
    ipiv = torch.empty(n, dtype=torch.int32, device='cuda')
    info = torch.zeros(1, dtype=torch.int32, device='cuda')
    cols = torch.arange(n, dtype=torch.int32, device='cuda')
    inv = torch.empty((n, n), dtype=torch.complex128, device='cuda')
    ws = torch.empty(lib().emu_fem_factor_workspace_size(n, n), dtype=torch.uint8, device='cuda')
    check(lib().emu_fem_factor(n, ptr(A), n, ptr(ipiv), ptr(info), n, ptr(cols), ptr(inv), n, ptr(ws),
                               C.c_size_t(ws.numel()), stream_ptr()), 'emu_fem_factor')
    assert int(info.item()) == 0
    ref = np.linalg.inv(B)
    got = inv.cpu().numpy() * d[None]
    assert np.abs(got - ref).max() <= 1e-11 * np.abs(ref).max()
