"""A problem's results do not depend on the batch it is solved in.

Interfaces and cascades around max(P, M) = 256, where GEMMs begin to run as residues
(csrc/dense_multi.cuh): each problem alone, in small batches and in a batch larger than
the number of SMs, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inputs(P, M, B, seed=0):
    import torch
    rng = np.random.default_rng(seed + 1000 * P + M)
    cr = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
    J = cr(B, P, M) / np.sqrt(P)
    Jd = np.conj(J).swapaxes(1, 2) + 0.1 * cr(B, M, P) / np.sqrt(P)
    kz = np.sqrt((25.0 - rng.uniform(0, 12, (B, P // 2)) ** 2).astype(complex))
    cu = lambda a: torch.tensor(np.ascontiguousarray(a), device='cuda')
    return cu(kz), cu(np.ones(B, complex)), cu(np.full(B, 2 * np.pi / 5)), cu(J), cu(Jd)


@pytest.mark.parametrize('P,M', [(90, 250), (90, 256), (258, 100), (162, 300), (322, 260)])
def test_interface_alone_and_in_batches(P, M):
    from emustack_b200.dense import interface_dense
    B = 160
    a = _inputs(P, M, B)
    full = [t.cpu().numpy() for t in interface_dense(*a)]
    assert not full[4].any()
    for i0, n in ((0, 1), (5, 2), (60, 9), (159, 1)):
        part = interface_dense(*(t[i0:i0 + n].contiguous() for t in a))
        for x, y in zip(part, full):
            np.testing.assert_array_equal(x.cpu().numpy(), y[i0:i0 + n])


@pytest.mark.parametrize('P,M,B', [(90, 250, 6), (90, 256, 6), (262, 300, 5)])
def test_cascade_alone_and_in_batches(P, M, B):
    import torch
    from emustack_b200.dense import DenseLayer, DenseStackSolver, film_interface, interface_dense
    kz, one, wln, J, Jd = _inputs(P, M, B)
    mid = interface_dense(kz, one, wln, J, Jd)
    Ra, Ta = film_interface(kz, one, kz * 1.3, 1.3 * one, wln)
    rng = np.random.default_rng(4)
    kzm = torch.tensor(5.0 * (rng.uniform(0, 2, (B, M)) + 1j * rng.uniform(0, 3, (B, M))), device='cuda')
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device='cuda')

    def solve(sl):
        c = lambda t: t[sl].contiguous()
        film = DenseLayer(c(Ra), c(Ta), -c(Ra), c(Ta), False)
        lay = [film] + [DenseLayer(*(c(t) for t in mid[:4]), True, c(kzm), 0.15)] * 2 + [film]
        n = len(kz[sl])
        o = DenseStackSolver().solve(lay, P, pol='TM', specular=i32([2] * n), num_prop=i32([[5, 5, 6]] * n))
        return {k: o[k].cpu().numpy() for k in ('R_net', 'T_net', 'a_list', 't_list', 'r_list')}

    full = solve(slice(0, B))
    for i in range(B):
        one_ = solve(slice(i, i + 1))
        for k, v in full.items():
            np.testing.assert_array_equal(one_[k][0], v[i], err_msg=k)


@pytest.mark.parametrize('n,M,order,chunk', [
    (5, 3, 1, 0),        # 50 elements: one segment, folds of 16 and a rest of 2
    (16, 40, 3, 0),      # 512 elements: two segments
    (17, 70, 2, 0),      # 578 elements, three segments, two CTAs of modes
    (20, 20, 4, 0),      # 49 plane waves: one set per CTA
    (20, 20, 3, 300),    # spans of 304 elements
    (24, 30, 5, 0),      # residues (81 plane waves), K splits
    (24, 130, 6, 500),   # residues in chunks
])
def test_overlap_alone_and_in_batches(n, M, order, chunk):
    import torch
    from emustack_b200.films import grating_orders
    from emustack_b200.mesh import square_cell
    from emustack_b200.overlap import DeviceMesh, overlap_batch
    rng = np.random.default_rng(n)
    dm = DeviceMesh(square_cell(n, radius=0.3, jitter=0.2, seed=n))
    B = 40
    cu = lambda a: torch.tensor(np.ascontiguousarray(a), device='cuda')
    g = torch.Generator(device='cuda').manual_seed(n)
    sol = [torch.randn((B, dm.nel, M, 13, 3), dtype=torch.complex128, device='cuda', generator=g) for _ in range(2)]
    bloch, k0 = cu(rng.uniform(-1, 1, (B, 2))), cu(rng.uniform(5, 9, B))
    px, py = grating_orders(order, 500.0, 500.0)

    def run(i, m, sets=(0, 1)):
        c = lambda t: t[i:i + m].contiguous()
        return overlap_batch(dm, px, py, order, c(bloch), c(k0), *(c(sol[k]) if k in sets else None for k in (0, 1)),
                             elements_per_chunk=chunk)

    J, Jd, _ = run(0, B)
    for i, m in ((0, 1), (3, 2), (10, 7), (20, 20)):
        a, b, _ = run(i, m)
        assert torch.equal(a, J[i:i + m]) and torch.equal(b, Jd[i:i + m])


@pytest.mark.parametrize('n', [1, 8, 31, 33, 64, 100, 114, 130])
def test_systems_alone_and_in_batches(n):
    """LU solves: one system on a cluster, up to as many as SMs on a CTA each, more on
    two CTAs per SM."""
    import torch
    from emustack_b200.dense import zgesv_batched
    g = torch.Generator(device='cuda').manual_seed(n)
    A = torch.randn((320, n, n), dtype=torch.complex128, device='cuda', generator=g) + 2 * torch.eye(n, device='cuda')
    B = torch.randn((320, n, 5), dtype=torch.complex128, device='cuda', generator=g)
    solve = lambda i, m: zgesv_batched(A[i:i + m].clone(), B[i:i + m].clone())[0]
    full = solve(0, 320)
    ref = np.linalg.solve(A[:3].cpu().numpy(), B[:3].cpu().numpy())
    np.testing.assert_allclose(full[:3].cpu().numpy(), ref, rtol=1e-8, atol=1e-10)
    for i, m in ((0, 1), (7, 3), (40, 140)):
        assert torch.equal(solve(i, m), full[i:i + m])
