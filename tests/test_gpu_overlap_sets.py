"""emu_overlap_batch with neither field set: the plane-wave order alone.

The C entry accepts d_sol1 = d_sol2 = NULL (with no outputs) and then gives
d_index_pw_inv, the order of backend/fortran/pw_ordering.f, on every path: direct
(up to 64 plane waves), residues and split TF32."""
import ctypes as C

import numpy as np
import pytest

from oracle import overlap as OV

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('precision', [0, 1])
@pytest.mark.parametrize('order,batch', [(0, 1), (3, 5), (5, 2), (9, 3)])
def test_order_without_fields(order, batch, precision):
    import torch
    from emustack_b200._lib import EmuOverlap, check, lib, ptr, stream_ptr
    from emustack_b200.films import grating_orders
    from emustack_b200.mesh import square_cell
    from emustack_b200.overlap import DeviceMesh
    rng = np.random.default_rng(order)
    dm = DeviceMesh(square_cell(3, radius=0.3))
    px, py = grating_orders(order, 500.0, 500.0)
    cu = lambda a: torch.tensor(np.asarray(a), device='cuda')
    bloch, k0 = rng.uniform(-1, 1, (batch, 2)), rng.uniform(5, 9, batch)
    t = [cu(px), cu(py), cu(bloch), cu(k0)]
    inv = torch.full((batch, len(px)), -1, dtype=torch.int32, device='cuda')
    d = EmuOverlap()
    d.batch, d.nval, d.nel, d.npt, d.n_pw, d.max_order = batch, 4, dm.nel, dm.npt, len(px), order
    d.d_px, d.d_py, d.d_bloch, d.d_k0 = map(ptr, t)
    d.d_x, d.d_table_nod, d.d, d.dy, d.area_norm = ptr(dm.x), ptr(dm.table_nod), 1.0, 1.0, 1.0
    d.d_index_pw_inv, d.precision = ptr(inv), precision
    n = lib().emu_overlap_workspace_size(C.byref(d))
    ws = torch.empty(n, dtype=torch.uint8, device='cuda')
    check(lib().emu_overlap_batch(C.byref(d), ptr(ws), C.c_size_t(n), stream_ptr()), 'emu_overlap_batch')
    for b in range(batch):
        np.testing.assert_array_equal(inv[b].cpu().numpy(), OV.pw_ordering(order, 1.0, 1.0, bloch[b], k0[b])[0])


@pytest.mark.parametrize('precision', ['fp64', 'tf32x3'])
@pytest.mark.parametrize('order', [3, 5, 6])
def test_prime_and_adjoint_fields_in_the_same_memory(order, precision):
    """One tensor given for both sets gives what two tensors of the same values give."""
    import torch
    from emustack_b200.films import grating_orders
    from emustack_b200.mesh import square_cell
    from emustack_b200.overlap import DeviceMesh, overlap_batch
    rng = np.random.default_rng(order)
    dm = DeviceMesh(square_cell(6, radius=0.3))
    cu = lambda a: torch.tensor(np.asarray(a), device='cuda')
    px, py = grating_orders(order, 500.0, 500.0)
    B, M = 2, 9
    sol = cu(rng.standard_normal((B, dm.nel, M, 13, 3)) + 1j * rng.standard_normal((B, dm.nel, M, 13, 3)))
    bloch, k0 = cu(rng.uniform(-1, 1, (B, 2))), cu(rng.uniform(5, 9, B))
    run = lambda a, b: overlap_batch(dm, px, py, order, bloch, k0, a, b, precision=precision)
    J, Jd, _ = run(sol, sol)
    rJ, rJd, _ = run(sol, sol.clone())
    assert torch.equal(J, rJ) and torch.equal(Jd, rJd)
