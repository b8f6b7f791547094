"""The FP64 overlap contraction as residues on the INT8 tensor cores
(csrc/residue_gemm.cuh) against the C oracle, at the edges of its tiles (128
field rows, 112 plane waves, 128 K values, 64 elements), with several chunks
and problems, and for rows that have no safe scale.

Tolerance: rounding a row to integers of 2-norm 2^57 .. 2^58 moves an entry by
at most sqrt(2 K) 2^-57 |e_s| |f_n| from both operands together; at K <= 3 000
that is 5.4e-16 |e_s| |f_n|, and the E~ table's own rounding (a few dozen
operations) adds as many ulps: 2e-14 |e_s| |f_n| is allowed, with |e_s|^2 <=
the sum over elements of 6 (area / 3)^2."""
import numpy as np
import pytest
import torch

from emustack_b200.mesh import square_cell
from oracle import overlap as OV

pytestmark = pytest.mark.gpu


def _bound(mesh, sol):
    v = mesh.x[mesh.table_nod[:, :3] - 1]
    d1, d2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    area = 0.5 * np.abs(d1[:, 0] * d2[:, 1] - d1[:, 1] * d2[:, 0])
    e = np.sqrt(6 * np.sum((area / 3) ** 2))
    f = np.sqrt((np.abs(sol[:, :, :6, :2]) ** 2).sum((0, 2, 3)))
    return 2e-14 * e * f


def _run(n, M, mo, B, sets, chunk=0, edit=None, jitter=0.2):
    from emustack_b200.films import grating_orders
    from emustack_b200.overlap import DeviceMesh, overlap_batch
    rng = np.random.default_rng(n * M + mo)
    mesh = square_cell(n, radius=0.3, jitter=jitter, seed=n)
    mesh.x, mesh.table_nod = np.asarray(mesh.x), np.asarray(mesh.table_nod)
    sol = [rng.standard_normal((B, mesh.nel, M, 13, 3)) + 1j * rng.standard_normal((B, mesh.nel, M, 13, 3))
           for _ in range(2)]
    if edit:
        edit(sol)
    bloch, k0 = rng.uniform(-1, 1, (B, 2)), rng.uniform(5, 9, B)
    px, py = grating_orders(mo, 500.0, 500.0)
    cu = lambda a: torch.tensor(a, device='cuda')
    J, Jd, inv = overlap_batch(DeviceMesh(mesh), px, py, mo, cu(bloch), cu(k0), cu(sol[0]) if 0 in sets else None,
                               cu(sol[1]) if 1 in sets else None, elements_per_chunk=chunk)
    return mesh, sol, bloch, k0, mo, J, Jd, inv


@pytest.mark.parametrize('n,M,mo,B,sets,chunk', [
    (3, 1, 0, 2, (0, 1), 0),       # one plane wave, one mode
    (6, 32, 5, 2, (0, 1), 0),      # 128 field rows exactly; 81 plane waves
    (7, 33, 6, 2, (0, 1), 0),      # 132 rows; 113 plane waves: two tiles of B
    (9, 65, 2, 3, (0,), 64),       # J only, chunks of 64 and 34 elements
    (10, 20, 3, 2, (1,), 70),      # J_dag only, uneven chunks
    (16, 40, 3, 1, (0, 1), 0),     # one problem above the small-problem rule
])
def test_residue_overlap_matches_oracle(n, M, mo, B, sets, chunk):
    mesh, sol, bloch, k0, mo, J, Jd, inv = _run(n, M, mo, B, sets, chunk)
    for b in range(B):
        oinv, _, _ = OV.pw_ordering(mo, 1.0, 1.0, bloch[b], k0[b])
        np.testing.assert_array_equal(inv[b].cpu().numpy(), oinv)
        if 0 in sets:
            ref = OV.J_overlap(mesh.x, mesh.table_nod, sol[0][b], 1.0, 1.0, bloch[b], oinv, mo)
            assert (np.abs(J[b].cpu().numpy() - ref) <= _bound(mesh, sol[0][b])[None]).all()
        if 1 in sets:
            ref = OV.J_dagger_overlap(mesh.x, mesh.table_nod, sol[1][b], 1.0, 1.0, bloch[b], oinv, mo)
            assert (np.abs(Jd[b].cpu().numpy() - ref) <= _bound(mesh, sol[1][b])[:, None]).all()


@pytest.mark.parametrize('n,M,mo,B,sets,chunk', [
    (2, 1, 0, 3, (0, 1), 0),       # one plane wave, one mode, one tile of 8 elements
    (3, 63, 1, 2, (0, 1), 0),      # 18 elements: a tile of 2 left over; 5 plane waves
    (7, 64, 2, 2, (0, 1), 0),      # one CTA of modes exactly; 13 plane waves
    (9, 65, 3, 2, (1,), 0),        # a second CTA with one mode; J_dag only; 29 plane waves
    (20, 20, 3, 30, (0, 1), 100),  # spans of 104 elements, the last one 72; 30 problems, sums folded several times
    (16, 70, 4, 1, (0, 1), 0),     # 49 plane waves: one set per CTA, tiles of 4 elements
    (40, 9, 4, 1, (0,), 0),        # 3 200 elements in many splits
])
def test_direct_overlap_matches_oracle(n, M, mo, B, sets, chunk):
    """At most 64 plane waves: the FP64 products themselves.  An entry's longest
    chain is 16 elements (192 products), then at most 8 folded sums, 20 splits of
    a thread and 8 threads: 230 x 2^-53 = 2.6e-14 |e_s| |f_n|, and a few dozen ulps
    of the E~ table: 3e-14 is allowed."""
    mesh, sol, bloch, k0, mo, J, Jd, inv = _run(n, M, mo, B, sets, chunk)
    for b in range(0, B, 7):
        oinv, _, _ = OV.pw_ordering(mo, 1.0, 1.0, bloch[b], k0[b])
        np.testing.assert_array_equal(inv[b].cpu().numpy(), oinv)
        if 0 in sets:
            ref = OV.J_overlap(mesh.x, mesh.table_nod, sol[0][b], 1.0, 1.0, bloch[b], oinv, mo)
            assert (np.abs(J[b].cpu().numpy() - ref) <= 1.5 * _bound(mesh, sol[0][b])[None]).all()
        if 1 in sets:
            ref = OV.J_dagger_overlap(mesh.x, mesh.table_nod, sol[1][b], 1.0, 1.0, bloch[b], oinv, mo)
            assert (np.abs(Jd[b].cpu().numpy() - ref) <= 1.5 * _bound(mesh, sol[1][b])[:, None]).all()


@pytest.mark.parametrize('mo', [3, 5])
def test_residue_overlap_rows_without_a_safe_scale(mo):
    """Modes with huge, tiny, infinite or NaN values are summed in FP64 and
    leave the others alone; a zero mode gives zeros."""
    def edit(sol):
        for s in sol:
            s[:, :, 1] *= 1e150
            s[:, :, 2] *= 1e-150
            s[:, 3, 3, 2, 0] = np.inf
            s[:, 4, 4, 1, 1] = np.nan
            s[:, :, 5] = 0
    mesh, sol, bloch, k0, mo, J, Jd, _ = _run(6, 12, mo, 2, (0, 1), 0, edit)
    for b in range(2):
        oinv, _, _ = OV.pw_ordering(mo, 1.0, 1.0, bloch[b], k0[b])
        for out, f, s in ((J[b].cpu().numpy(), OV.J_overlap, sol[0][b]),
                          (Jd[b].cpu().numpy().T, OV.J_dagger_overlap, sol[1][b])):
            ok = [m for m in range(12) if m not in (3, 4)]
            ref = f(mesh.x, mesh.table_nod, np.ascontiguousarray(s[:, ok]), 1.0, 1.0, bloch[b], oinv, mo)
            ref = ref if f is OV.J_overlap else ref.T
            assert (np.abs(out[:, ok] - ref) <= _bound(mesh, s[:, ok])[None]).all()
            assert (out[:, 5] == 0).all()
            assert not np.isfinite(out[:, 3:5]).any()


def _interface(P, M, B, seed):
    rng = np.random.default_rng(seed)
    cr = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
    J = cr(B, P, M) / np.sqrt(P)
    Jd = np.conj(J).swapaxes(1, 2) + 0.1 * cr(B, M, P) / np.sqrt(P)
    q = rng.uniform(0, 12, (B, P // 2))
    kz = np.sqrt((25.0 - q ** 2).astype(complex))
    return kz, J, np.ascontiguousarray(Jd)


def _interface_gpu(kz, J, Jd):
    from emustack_b200.dense import interface_dense
    cu = lambda a: torch.tensor(a, device='cuda')
    B = len(J)
    return [t.cpu().numpy() for t in interface_dense(cu(kz), cu(np.ones(B, complex)), cu(np.full(B, 2 * np.pi / 5)),
                                                     cu(J), cu(Jd))]


@pytest.mark.parametrize('P,M,B', [
    (258, 300, 2),      # the smallest matrices that use residues; a block of 44 after one of 256
    (400, 256, 1),      # one whole block
    (130, 513, 2),      # two blocks and one column; fewer plane waves than modes
])
def test_dense_residue_interface_matches_numpy(P, M, B):
    """Interfaces whose GEMMs run as residues (and whose LU recurses on
    blocks of 256) against numpy's solve: both are backward stable, so they
    agree to cond(I + B A) (below 1e3 here) x M x 2^-53, 6e-11 of the largest
    entry; 1e-11 is asked for."""
    from oracle.gsm_oracle import r_t_mat_tf_ns
    kz, J, Jd = _interface(P, M, B, P + M)
    out = _interface_gpu(kz, J, Jd)
    assert (out[4] == 0).all()
    for b in range(B):
        z = 5.0 / kz[b]
        for got, ref in zip(out, r_t_mat_tf_ns(np.concatenate([z, 1 / z]), J[b], Jd[b])):
            np.testing.assert_allclose(got[b], ref, rtol=0, atol=1e-11 * np.abs(ref).max())


def test_dense_residue_rows_without_a_safe_scale():
    """J x 1e140 and J_dag / 1e140 give the same R12 and R21 through the
    direct FP64 sums; a NaN spoils its own problem only."""
    kz, J, Jd = _interface(258, 300, 2, 7)
    ref = _interface_gpu(kz, J, Jd)
    out = _interface_gpu(kz, J * 1e140, Jd / 1e140)
    for i in (0, 2):
        np.testing.assert_allclose(out[i], ref[i], rtol=0, atol=1e-11 * np.abs(ref[i]).max())
    J[1, 5, 7] = np.nan
    out = _interface_gpu(kz, J, Jd)
    for i in range(4):
        np.testing.assert_array_equal(out[i][0], ref[i][0])
        assert not np.isfinite(out[i][1]).all()
