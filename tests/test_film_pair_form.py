"""The film kernels' division-free recursion (csrc/film_core.cuh) against the
reference's, and the teams of warps that solve one point of an uneven batch.

On the CPU, a numpy restatement: impedances z1 : z2 as A : B = 1 : t (TE) and
t : n^2 (TM) with t = k_z / k_z,air, the reflection as a pair rnet = (Z - V) /
(Z + V), the transmission as one product over the layers, and the outer layers'
square roots as sqrt(k_z) and +-sqrt(k_z) n.  Tolerance: about 40 roundings per
layer, 10 layers at most, amplified by the conditioning of a resonant entry (below
1e3 for these stacks): 40 x 10 x 1e3 x 2^-53 = 4.4e-11, so 1e-10 relative to the
entry (and 1e-12 absolute for entries that cancel) is allowed; 70 layers and
evanescent orders on the GPU take the 1e-9 of the other film tests."""
import numpy as np
import pytest

from oracle import gsm_oracle as O


def pair_form(ns, heights_nm, wl_nm, k_pll, period, max_order):
    air = O.make_air_ref(wl_nm, k_pll, period, None, max_order)
    npw = air.num_pw_per_pol
    ka = air.k_z[:npw].astype(complex)
    kz = [O.FilmModes(n, wl_nm, k_pll, period, None, max_order, air=air).k_z[:npw].astype(complex) for n in ns]

    def ab(l):
        t, nn = kz[l] / ka, np.full(npw, complex(ns[l]) ** 2)
        return np.concatenate([np.ones(npw), t]), np.concatenate([t, nn])

    def root(l):
        f = np.sqrt(kz[l])
        g = f * ns[l]
        s = f.real * complex(ns[l]).real + f.imag * complex(ns[l]).imag
        return np.concatenate([f, np.where(s < 0, -g, g)])

    Z, V = ab(0)
    num = root(0)
    for l in range(1, len(ns) - 1):
        A, B = ab(l)
        p = np.tile(np.exp(1j * kz[l] * heights_nm[l - 1] / period), 2)
        X, Y = A * V, B * Z
        u, w = X + Y, p * p * (Y - X)
        Z, V = A * (u + w), B * (u - w)
        num = num * 2 * A * B * p
    A, B = ab(len(ns) - 1)
    u, v = A * V + B * Z, B * Z - A * V
    return v / u, 2 * num * root(len(ns) - 1) / (np.tile(ka, 2) * u)


MEDIA = {
    'passive': lambda r, L: r.uniform(1.2, 4.0, L) + 1j * r.uniform(0.0, 0.4, L),
    'metal': lambda r, L: r.uniform(0.05, 0.5, L) + 1j * r.uniform(1.0, 6.0, L),
    'gain': lambda r, L: r.uniform(1.2, 3.0, L) - 1j * r.uniform(0.0, 0.05, L),
    'negative': lambda r, L: -r.uniform(1.2, 3.0, L) - 1j * r.uniform(0.01, 0.2, L),
    'air': lambda r, L: np.ones(L) + 0j,
}


@pytest.mark.parametrize('outer', sorted(MEDIA))
@pytest.mark.parametrize('inner', sorted(MEDIA))
@pytest.mark.parametrize('L', [2, 3, 8])
def test_pair_form_equals_reference(L, inner, outer):
    rng = np.random.default_rng(L)
    ns = MEDIA[inner](rng, L)
    ns[[0, -1]] = MEDIA[outer](rng, 2)
    heights = list(rng.uniform(20, 200, L - 2))
    wl = float(rng.uniform(350, 1100))
    kp = O.k_parallel_from_angles(wl, 0.4, 0.7)
    r, t = pair_form(ns, heights, wl, kp, 500.0, 2)
    ref = O.film_stack_point(list(ns), heights, wl, kp, 500.0, max_order=2, pol='TE')
    np.testing.assert_allclose(r, np.diag(ref.R_net), rtol=1e-10, atol=1e-12)
    np.testing.assert_allclose(t, np.diag(ref.T_net), rtol=1e-10, atol=1e-12)


@pytest.mark.gpu
@pytest.mark.parametrize('L,inner,order', [
    (2, 'passive', 3), (3, 'metal', 0), (6, 'gain', 4), (7, 'negative', 3), (5, 'air', 5),
    (9, 'metal', 8), (70, 'passive', 6),    # the pair is rescaled every fourth layer
])
def test_film_kernel_at_the_edges_of_the_recursion(L, inner, order):
    import torch
    from emustack_b200.films import FilmStackSolver
    rng = np.random.default_rng(10 * L + order)
    B = 3
    ns = np.stack([np.concatenate([[1.5 + 0j], MEDIA[inner](rng, L - 2), [1.0 + 0j]]) for _ in range(B)])
    h = rng.uniform(5, 900 if inner in ('metal', 'passive') else 100, L - 2)
    wl = rng.uniform(350, 900, B)
    kp = np.array([O.k_parallel_from_angles(w, 0.3, 0.2) for w in wl])
    s = FilmStackSolver(L, order, 500.0)
    cu = lambda a: torch.tensor(a, device=s.device)
    for pol in ('TE', 'TM', 'R Circ'):
        o = {k: v.cpu().numpy() for k, v in s.solve(cu(wl), cu(kp), cu(ns), cu(h), pol=pol).items()}
        for b in range(B):
            ref = O.film_stack_point(list(ns[b]), list(h), wl[b], kp[b], 500.0, max_order=order, pol=pol)
            np.testing.assert_allclose(o['R_net'][b], np.diag(ref.R_net), rtol=1e-9, atol=1e-10)
            np.testing.assert_allclose(o['T_net'][b], np.diag(ref.T_net), rtol=1e-9, atol=1e-10)
            for k in ('a_list', 't_list'):
                np.testing.assert_allclose(o[k][b], np.asarray(getattr(ref, k), float), rtol=1e-9, atol=1e-9)
        if inner == 'air':      # a film of air is no interface
            assert (np.abs(s.solve(cu(wl), cu(kp), cu(np.ones((B, L)) + 0j), cu(h), pol=pol)['R_net']
                           .cpu().numpy()) == 0).all()


@pytest.mark.gpu
@pytest.mark.parametrize('sizes', [[12], [12, 0], [11] + [0] * 400, [12, 9, 7, 5, 3, 1, 0] * 30,
                                   [12] * 3 + [2] * 3000])
def test_teams_of_warps_give_the_results_of_one_warp(sizes):
    """Points of 1 .. 441 orders on teams of 8, 4, 2 and 1 warps: R_net and T_net
    bit for bit those of one warp per point; the flux sums, added by atomics, to
    1e-13 as in the other tests of this kernel."""
    import torch
    from emustack_b200.films import FilmPoint, FilmVarSolver
    rng = np.random.default_rng(len(sizes))
    pts = []
    for i, m in enumerate(sizes):
        L = int(rng.integers(2, 9))
        wl = float(rng.uniform(400, 900))
        pts.append(FilmPoint(rng.uniform(1.2, 3.0, L) + 1j * rng.uniform(0, 0.2, L), rng.uniform(20, 200, L - 2), wl,
                             O.k_parallel_from_angles(wl, 0.2, 0.4), 500.0, m, pol=('TE', 'TM', 'L Circ')[i % 3]))
    s = FilmVarSolver()
    pl = s.plan(pts)
    run = lambda **k: {a: b.cpu().numpy().copy() for a, b in s.solve(pl, want_num_prop=True, **k).items()}
    ref = run(warps=1)
    for w in (2, 3, 8):
        for v in (0, 1):
            out = run(warps=w, variant=v)
            for k in ('R_net', 'T_net', 'flags', 'specular', 'num_prop'):
                np.testing.assert_array_equal(out[k], ref[k])
            for k in ('a_list', 't_list', 'r_list'):
                np.testing.assert_allclose(out[k], ref[k], rtol=1e-13, atol=1e-13)
    torch.cuda.synchronize()
