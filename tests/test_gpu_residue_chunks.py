"""The residue path of the overlaps (more than 64 plane waves) where its sums are put
together from parts, against the C oracle: residues added modulo p over chunks of
elements, a shorter last chunk that keeps the first one's K splits, K splits, spans of
elements with scales of their own, and one field set alone.  Tolerance as in
test_gpu_residue.py (2e-14 |e_s| |f_n|)."""
import numpy as np
import pytest

from oracle import overlap as OV
from test_gpu_residue import _bound, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n,M,mo,B,sets,chunk', [
    (9, 65, 5, 3, (0,), 64),       # J only, chunks of 64 and 34 elements
    (10, 20, 6, 2, (1,), 70),      # J_dag only, chunks of 128 and 72
    (8, 33, 5, 2, (0, 1), 50),     # both, three chunks
    (6, 1, 5, 2, (0, 1), 0),       # one mode
    (26, 12, 5, 1, (0, 1), 0),     # 1 352 elements: K = 8 112 in four splits
    (26, 12, 5, 2, (0,), 700),     # splits in chunks of 704 and 648
    (30, 5, 5, 1, (1,), 1000),     # splits, a last chunk of 800
])
def test_parts_of_residue_overlaps_match_the_oracle(n, M, mo, B, sets, chunk):
    mesh, sol, bloch, k0, mo, J, Jd, inv = _run(n, M, mo, B, sets, chunk)
    assert inv.shape[1] > 64        # the residue path
    for b in range(B):
        oinv, _, _ = OV.pw_ordering(mo, 1.0, 1.0, bloch[b], k0[b])
        if 0 in sets:
            ref = OV.J_overlap(mesh.x, mesh.table_nod, sol[0][b], 1.0, 1.0, bloch[b], oinv, mo)
            assert (np.abs(J[b].cpu().numpy() - ref) <= _bound(mesh, sol[0][b])[None]).all()
        if 1 in sets:
            ref = OV.J_dagger_overlap(mesh.x, mesh.table_nod, sol[1][b], 1.0, 1.0, bloch[b], oinv, mo)
            assert (np.abs(Jd[b].cpu().numpy() - ref) <= _bound(mesh, sol[1][b])[:, None]).all()


def test_spans_with_scales_of_their_own():
    """100 352 elements of 113 plane waves: E~ tables of 98 304 and 2 048 elements.  The
    second span's fields are 1e6 times the first one's."""
    edge = 98304

    def edit(sol):
        for s in sol:
            s[:, edge:] *= 1e6
    mesh, sol, bloch, k0, mo, J, Jd, inv = _run(224, 1, 6, 1, (0, 1), 0, edit)
    assert inv.shape[1] == 113 and 96 * 113 * edge < 1 << 30 < 96 * 113 * mesh.nel
    oinv, _, _ = OV.pw_ordering(mo, 1.0, 1.0, bloch[0], k0[0])
    # 25 times the elements of the tolerance's derivation: sqrt(25) for their rounding
    ref = OV.J_overlap(mesh.x, mesh.table_nod, sol[0][0], 1.0, 1.0, bloch[0], oinv, mo)
    assert (np.abs(J[0].cpu().numpy() - ref) <= 5 * _bound(mesh, sol[0][0])[None]).all()
    ref = OV.J_dagger_overlap(mesh.x, mesh.table_nod, sol[1][0], 1.0, 1.0, bloch[0], oinv, mo)
    assert (np.abs(Jd[0].cpu().numpy() - ref) <= 5 * _bound(mesh, sol[1][0])[:, None]).all()
