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


def _array_layer(P, M, B, graded, seed):
    """J with modes normalised by factors over 20 decades, J_dag by their inverses."""
    rng = np.random.default_rng(seed)
    cr = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
    J = cr(B, P, M) / np.sqrt(P)
    Jd = np.conj(J).swapaxes(1, 2) + 0.1 * cr(B, M, P) / np.sqrt(P)
    c = 1.0 / _grades(M) if graded else np.ones(M)
    kz = np.sqrt((25.0 - rng.uniform(0, 12, (B, P // 2)) ** 2).astype(complex))
    return kz, J * c, Jd / c[:, None], c


def _interfaces(P, M, B, graded, seed):
    import torch
    from emustack_b200.dense import interface_dense
    kz, J, Jd, c = _array_layer(P, M, B, graded, seed)
    cu = lambda a: torch.tensor(a, device='cuda')
    out = interface_dense(cu(kz), cu(np.ones(B, complex)), cu(np.full(B, 2 * np.pi / 5)), cu(J), cu(Jd))
    return kz, out, c


@pytest.mark.parametrize('P,M,B', [(58, 60, 3), (258, 300, 2), (400, 256, 1), (130, 513, 2)])
def test_interface_of_unevenly_normalised_modes(P, M, B):
    """A factor c of a mode leaves R12 as it is and goes to T12 as 1 / c, to T21 as c
    and to R21 as c_j / c_i.  Tolerance as for the ungraded interface (1e-11)."""
    _, ref, _ = _interfaces(P, M, B, False, P + M)
    _, got, c = _interfaces(P, M, B, True, P + M)
    ref, got = [t.cpu().numpy() for t in ref], [t.cpu().numpy() for t in got]
    assert not got[4].any()
    for r, g in zip(ref, (got[0], got[1] * c[:, None], got[2] * c[:, None] / c, got[3] / c)):
        np.testing.assert_allclose(g, r, rtol=0, atol=1e-11 * np.abs(r).max())


@pytest.mark.parametrize('P,M,B', [(58, 60, 2), (258, 300, 2)])
def test_cascade_of_unevenly_normalised_modes(P, M, B):
    """R_net, T_net and the lists do not depend on the modes' normalisation."""
    import torch
    from emustack_b200.dense import DenseLayer, DenseStackSolver, film_interface
    cu = lambda a: torch.tensor(a, device='cuda')
    res = []
    for graded in (False, True):
        kz, mid, _ = _interfaces(P, M, B, graded, 7)
        one, wln = cu(np.ones(B, complex)), cu(np.full(B, 2 * np.pi / 5))
        kzs = cu(np.sqrt(25.0 * 1.46 ** 2 - 25.0 + kz ** 2 + 0j))
        Rs, Ts = film_interface(cu(kz), one, kzs, 1.46 * one, wln)
        Ra, Ta = film_interface(cu(kz), one, cu(kz), one, wln)
        rng = np.random.default_rng(3)
        kzm = cu(5.0 * (rng.uniform(0, 2, (B, M)) + 1j * np.where(rng.uniform(size=(B, M)) < 0.2, 0.05, 8.0)))
        lay = [DenseLayer(Rs, Ts, -Rs, Ts, False)]
        lay += [DenseLayer(*mid[:4], True, kzm, 0.2), DenseLayer(*mid[:4], True, kzm, 0.1)]
        lay += [DenseLayer(Ra, Ta, -Ra, Ta, False)]
        i32 = lambda a: torch.tensor(a, dtype=torch.int32, device='cuda')
        o = DenseStackSolver().solve(lay, P, pol='TE', specular=i32([1] * B), num_prop=i32([[5, 5, 7]] * B))
        res.append({k: o[k].cpu().numpy() for k in ('R_net', 'T_net', 'a_list', 't_list', 'r_list')})
    for k, r in res[0].items():
        assert np.isfinite(r).all()
        np.testing.assert_allclose(res[1][k], r, rtol=0, atol=1e-10 * np.abs(r).max(), err_msg=k)


@pytest.mark.parametrize('order', [3, 5, 6])
@pytest.mark.parametrize('where', ['everywhere', 'smallest'])
def test_overlap_of_fields_that_follow_the_mesh(where, order):
    """Elements over 14 decades of area with fields that grow as they shrink, and modes
    that live in a few of the smallest elements only.  Bound: 5e-14 of sum |f| area / 3,
    which holds every element's share of an entry."""
    import torch
    from emustack_b200.films import grating_orders
    from emustack_b200.mesh import square_cell
    from emustack_b200.overlap import DeviceMesh, overlap_batch
    from oracle import overlap as OV
    rng = np.random.default_rng(order)
    mesh = square_cell(14, radius=0.3)
    mesh.x, mesh.table_nod = np.array(mesh.x), np.asarray(mesh.table_nod)
    mesh.x[:, 0] = mesh.x[:, 0] ** 12
    v = mesh.x[mesh.table_nod[:, :3] - 1]
    d1, d2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    area = 0.5 * np.abs(d1[:, 0] * d2[:, 1] - d1[:, 1] * d2[:, 0])
    assert area.max() / area.min() > 1e13
    M, B = 10, 2
    sol = [(rng.standard_normal((B, mesh.nel, M, 13, 3)) + 1j * rng.standard_normal((B, mesh.nel, M, 13, 3)))
           / area[None, :, None, None, None] for _ in range(2)]
    if where == 'smallest':
        keep = np.zeros((mesh.nel, M), bool)
        for m in range(M):
            keep[np.argsort(area)[m:2 * m + 1], m] = True
        sol = [s * keep[None, :, :, None, None] for s in sol]
    bloch, k0 = rng.uniform(-1, 1, (B, 2)), rng.uniform(5, 9, B)
    px, py = grating_orders(order, 500.0, 500.0)
    cu = lambda a: torch.tensor(a, device='cuda')
    J, Jd, _ = overlap_batch(DeviceMesh(mesh), px, py, order, cu(bloch), cu(k0), cu(sol[0]), cu(sol[1]))
    for b in range(B):
        inv, _, _ = OV.pw_ordering(order, 1.0, 1.0, bloch[b], k0[b])
        lim = [5e-14 * (np.abs(s[b][:, :, :6, :2]).sum((2, 3)) * area[:, None] / 3).sum(0) for s in sol]
        ref = OV.J_overlap(mesh.x, mesh.table_nod, sol[0][b], 1.0, 1.0, bloch[b], inv, order)
        assert (np.abs(J[b].cpu().numpy() - ref) <= lim[0][None]).all()
        ref = OV.J_dagger_overlap(mesh.x, mesh.table_nod, sol[1][b], 1.0, 1.0, bloch[b], inv, order)
        assert (np.abs(Jd[b].cpu().numpy() - ref) <= lim[1][:, None]).all()


@pytest.mark.parametrize('P,M,B', [(258, 300, 2), (130, 513, 1)])
def test_small_imaginary_parts_keep_their_digits(P, M, B):
    """Propagating orders only and nearly real overlaps: z is real and the matrices'
    imaginary parts are 1e-13 of the real ones.  FP64 sums give each part to its own
    rounding; 1e-9 of the largest imaginary part is allowed (condition below 1e3)."""
    import torch
    from emustack_b200.dense import interface_dense
    from oracle.gsm_oracle import r_t_mat_tf_ns
    rng = np.random.default_rng(P)
    cr = lambda *s: rng.standard_normal(s) + 1e-13j * rng.standard_normal(s)
    J = cr(B, P, M) / np.sqrt(P)
    Jd = J.swapaxes(1, 2) + 0.1 * cr(B, M, P) / np.sqrt(P)
    kz = np.sqrt((25.0 - rng.uniform(0, 4.5, (B, P // 2)) ** 2).astype(complex))
    cu = lambda a: torch.tensor(np.ascontiguousarray(a), device='cuda')
    out = interface_dense(cu(kz), cu(np.ones(B, complex)), cu(np.full(B, 2 * np.pi / 5)), cu(J), cu(Jd))
    for b in range(B):
        z = 5.0 / kz[b]
        for got, ref in zip(out, r_t_mat_tf_ns(np.concatenate([z, 1 / z]), J[b], Jd[b])):
            ref = np.asarray(ref)
            assert 0 < np.abs(ref.imag).max() < 1e-9
            np.testing.assert_allclose(got[b].cpu().numpy().imag, ref.imag, rtol=0, atol=1e-9 * np.abs(ref.imag).max())


def test_real_overlaps_give_exactly_real_interfaces():
    """Zero imaginary parts are sums of zeros, not small sums: exact, and not repeated."""
    import torch
    from emustack_b200.dense import interface_dense
    rng = np.random.default_rng(1)
    P, M = 258, 300
    J = rng.standard_normal((1, P, M)) / np.sqrt(P) + 0j
    kz = np.sqrt((25.0 - rng.uniform(0, 4.5, (1, P // 2)) ** 2).astype(complex))
    cu = lambda a: torch.tensor(np.ascontiguousarray(a), device='cuda')
    out = interface_dense(cu(kz), cu(np.ones(1, complex)), cu(np.full(1, 2 * np.pi / 5)), cu(J), cu(J.swapaxes(1, 2)))
    for t in out[:4]:
        assert np.isfinite(t.cpu().numpy()).all() and (t.cpu().numpy().imag == 0).all()
