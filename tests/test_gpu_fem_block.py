"""The block step of the Krylov basis (emu_fem_orthonormalise) at the edges of its
tiles (32 rows per partial sum, 128 columns per CTA, 4 vectors per thread).

Tolerance: C and Q are sums of n products of entries of unit vectors, so V^H Q
and Q^H Q - I are off by at most n 2^-53 + the second pass's rest, 1e-13 for n <=
1 000; V C + Q R reproduces W to (m + b) 2^-53 of its column norms, 1e-13 too."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _step(V, W):
    from emustack_b200._lib import check, lib, ptr, stream_ptr
    n, m = V.shape
    b = W.shape[1]
    full = torch.zeros((n, m + b + 1), dtype=torch.complex128, device='cuda')
    full[:, :m] = torch.tensor(V)
    w = torch.tensor(W, device='cuda')
    out = torch.empty(m * b + b * b + 1, dtype=torch.complex128, device='cuda')
    ws = torch.empty(lib().emu_fem_orthonormalise_workspace_size(n, m, b), dtype=torch.uint8, device='cuda')
    check(lib().emu_fem_orthonormalise(n, m, b, ptr(full), full.stride(0), ptr(w), b, ptr(out), ptr(ws),
                                       C.c_size_t(ws.numel()), stream_ptr(None)), 'emu_fem_orthonormalise')
    o = out.cpu().numpy()
    f = full.cpu().numpy()
    np.testing.assert_array_equal(f[:, :m], V)
    assert (f[:, m + b] == 0).all()
    return f[:, m:m + b], o[:m * b].reshape(m, b), o[m * b:-1].reshape(b, b), o[-1].real


@pytest.mark.parametrize('n,m,b', [(2, 1, 1), (33, 4, 3), (64, 32, 4), (700, 129, 4), (1000, 300, 17), (257, 128, 5)])
def test_block_step_is_a_qr_step(n, m, b):
    rng = np.random.default_rng(n)
    cr = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
    V = np.ascontiguousarray(np.linalg.qr(cr(n, m))[0])
    W = cr(n, b) + V @ (100 * cr(m, b))
    Q, c, R, info = _step(V, W)
    assert info == 0
    assert np.abs(V.conj().T @ Q).max() < 1e-13
    assert np.abs(Q.conj().T @ Q - np.eye(b)).max() < 1e-13
    assert (np.tril(R, -1) == 0).all() and (np.diag(R).real > 0).all()
    np.testing.assert_allclose(V @ c + Q @ R, W, rtol=0, atol=1e-13 * np.linalg.norm(W, axis=0).max())


def test_block_step_reports_a_dependent_block():
    V = np.eye(40, 8, dtype=complex)
    assert _step(V, np.zeros((40, 4), complex))[3] > 0
    assert _step(V, np.full((40, 2), np.nan + 0j))[3] > 0


def test_block_step_checks_its_arguments():
    from emustack_b200 import _lib
    L = _lib.lib()
    assert L.emu_fem_orthonormalise_workspace_size(0, 1, 1) == 0
    assert L.emu_fem_orthonormalise(8, 4, 2, None, 5, None, 2, None, None, C.c_size_t(0), None) == _lib.EMU_E_SHAPE
    assert L.emu_fem_orthonormalise(8, 4, 2, None, 6, None, 2, None, None, C.c_size_t(0), None) == _lib.EMU_E_ARG
