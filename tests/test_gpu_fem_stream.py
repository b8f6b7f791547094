"""A FEM solve on a stream that is not the current one.

The steps mix the library's kernels with torch operations; all of them follow the
stream that the caller names, so the result is that of the current stream, bit for bit
where no library reduction is involved (k_z to 1e-11 as in the other solver tests)."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MAIL = os.path.join(os.path.dirname(os.path.abspath(__file__)), 'golden', '4testing-600_120.mail')


@pytest.mark.parametrize('concurrent', [False, True])
def test_solve_on_a_named_stream(concurrent):
    import torch
    from emustack_b200.fem import FemMesh, FemModeSolver
    m = FemMesh.from_mail(MAIL)
    args = ([1.0, 3.6 + 0.05j], 0.9, [0.3, -0.2], 12)
    ref = FemModeSolver(m).solve_pair(*args, concurrent=False)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    # work on the current stream: a step that ran there by mistake would wait for it
    a = torch.randn(4096, 4096, device='cuda')
    for _ in range(20):
        a = a @ a / 64
    got = FemModeSolver(m).solve_pair(*args, stream=s, concurrent=concurrent)
    s.synchronize()
    for i in (0, 2):
        np.testing.assert_allclose(got[i], ref[i], rtol=1e-11, atol=1e-11)
        assert got[i + 1].shape == ref[i + 1].shape and bool(torch.isfinite(got[i + 1].real).all())
    torch.cuda.synchronize()
