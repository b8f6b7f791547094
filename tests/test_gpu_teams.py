"""Teams of 1, 2, 4 and 8 CTAs per stack give the same bits (csrc/cascade.cu).

How a team splits the work changes no entry's arithmetic, so every output of the
cascade and of the flux pass is compared bit for bit with one CTA per stack.  The
shapes are those at which a CTA may run ahead of its team: one plane wave against
many modes (products of one tile), P = M, P > M and P < M, films alone, arrays
alone and both, two layers and more."""
import numpy as np
import pytest
import torch

from test_gpu_stack_var import _random_stack, _uniform, _var_stack

pytestmark = pytest.mark.gpu

SHAPES = [(2, [130]), (2, [70, 0, 65]), (2, []), (10, []), (34, [34]), (34, [0, 34, 0]), (66, [20]), (66, [20, 66, 130]),
          (90, [64, 0]), (26, [46] * 4), (58, [0, 0, 78])]


def test_team_sizes_agree_bit_for_bit(monkeypatch):
    from emustack_b200 import dense
    rng = np.random.default_rng(5)
    sts = [_random_stack(rng, P, Ms, ('TE', 'TM', 'un')[i % 3], incoming=i % 4 == 3)
           for i, (P, Ms) in enumerate(SHAPES)]
    stacks = [_var_stack(s) for s in sts]
    solver = dense.StackVarSolver()

    def run(team):
        monkeypatch.setattr(dense, 'team_of', lambda costs, sms: team)
        o = solver.solve(stacks, want_fluxes=True)
        torch.cuda.synchronize()
        return {k: o[k].cpu().numpy() for k in ('R_net', 'T_net', 'a_list', 't_list', 'r_list', 'flags', 'info',
                                                'fluxes')}, o['rnet_off']

    ref, off = run(1)
    assert not ref['info'].any() and np.isfinite(ref['R_net']).all() and np.isfinite(ref['T_net']).all()
    for team in (2, 4, 8):
        for again in range(5):
            out, _ = run(team)
            for k in ref:
                np.testing.assert_array_equal(out[k], ref[k], err_msg='%s, team of %d' % (k, team))
    for s, o in zip(sts, off):          # and the uniform batch's own choice of team
        one, P = _uniform(s), s['P']
        for k in ('R_net', 'T_net'):
            np.testing.assert_array_equal(ref[k][o:o + P * P].reshape(P, P), one[k][0], err_msg=k)
