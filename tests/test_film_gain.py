"""Thick amplifying films: evanescent orders whose exp(i k_z h) grows.

In a film with Im n^2 < 0 the principal root gives evanescent orders Im k_z < 0, as
numpy's does in the reference (backend/mode_calcs.py:116-186), so |p| = |exp(i k_z h)|
passes 1e39 in one film of the cases below and |p|^2 over four films leaves the range
of a double.  The recursion of csrc/film_core.cuh scales such a layer by the exponent
of |p|.  Tolerance: that of the other film tests (1e-9 relative, 1e-10 absolute)."""
import numpy as np
import pytest

from oracle import gsm_oracle as O

TOL = dict(rtol=1e-9, atol=1e-10)
# films, n, height (nm), order
CASES = [(8, 2 - 0.02j, 900.0, 8), (8, 2 - 0.001j, 1500.0, 5), (7, 2 - 0.02j, 1000.0, 8), (9, 1.7 - 0.05j, 1200.0, 8),
         (70, 2 - 0.01j, 900.0, 5), (6, -1.5 + 0.1j, 1000.0, 6),
         (1, 2 - 0.02j, 2500.0, 8)]


def _stack(case, seed=0):
    films, n, h, order = case
    rng = np.random.default_rng(seed)
    ns = np.array([1.5 + 0j] + [n + 0.1 * i / films for i in range(films)] + [1.0 + 0j])
    wl = float(rng.uniform(500, 800))
    return ns, np.full(films, h), wl, O.k_parallel_from_angles(wl, 0.3, 0.5), order


def _oracle(ns, h, wl, kp, order, pol):
    ref = O.film_stack_point(list(ns), list(h), wl, kp, 500.0, max_order=order, pol=pol)
    return dict(R_net=np.diag(ref.R_net), T_net=np.diag(ref.T_net), a_list=np.asarray(ref.a_list, float),
                t_list=np.asarray(ref.t_list, float), r_list=np.asarray(ref.r_list, float))


@pytest.mark.parametrize('case', CASES)
def test_cases_grow_and_the_oracle_is_finite(case):
    ns, h, wl, kp, order = _stack(case)
    air = O.make_air_ref(wl, kp, 500.0, None, order)
    kz = O.FilmModes(ns[1], wl, kp, 500.0, None, order, air=air).k_z
    assert np.abs(np.exp(1j * kz * h[0] / 500.0)).max() > 1e20
    ref = _oracle(ns, h, wl, kp, order, 'TE')
    assert all(np.isfinite(v).all() for v in ref.values())


@pytest.mark.gpu
@pytest.mark.parametrize('case', CASES)
def test_growing_films_on_the_uniform_kernel(case):
    import torch
    from emustack_b200.films import FilmStackSolver
    pts = [_stack(case, i) for i in range(2)]
    L, order = len(pts[0][0]), case[3]
    s = FilmStackSolver(L, order, 500.0)
    cu = lambda a: torch.tensor(np.array(a), device=s.device)
    for pol in ('TE', 'TM', 'L Circ'):
        o = s.solve(cu([p[2] for p in pts]), cu([p[3] for p in pts]), cu([p[0] for p in pts]), cu(pts[0][1]), pol=pol,
                    want=('vec_coef', 'layer_rt'))
        o = {k: v.cpu().numpy() for k, v in o.items()}
        assert not (o['flags'] & 16).any()
        assert np.isfinite(o['vec_coef_down']).all() and np.isfinite(o['vec_coef_up']).all()
        for b, p in enumerate(pts):
            for k, v in _oracle(*p, pol).items():
                np.testing.assert_allclose(np.ravel(o[k][b]), v, **TOL, err_msg=k)


@pytest.mark.gpu
def test_growing_films_in_an_uneven_batch_and_the_request_loop():
    import torch
    from emustack_b200.films import FilmVarSolver
    from emustack_b200.serving import DeviceFilmServer, FilmRequest
    cases = [c for c in CASES if c[0] < 70]
    pts = [_stack(c) for c in cases]
    reqs = [FilmRequest(ns, h, wl, kp, 500.0, order, pol=('TE', 'TM', 'un')[i % 3])
            for i, (ns, h, wl, kp, order) in enumerate(pts)]
    s = FilmVarSolver()
    pl = s.plan(reqs)
    out = {k: v.cpu().numpy() for k, v in s.solve(pl).items()}
    torch.cuda.synchronize()
    uneven = s.unpack(pl, out)
    srv = DeviceFilmServer(capacity=64, idle_seconds=0.5)
    try:
        ring = [srv.take(t) for t in [srv.submit(r) for r in reqs]]
        assert srv.stop() == 0
    finally:
        srv.close()
    for p, r, a, b in zip(pts, reqs, uneven, ring):
        ref = _oracle(*p, r.pol)
        for k in ('R_net', 'T_net'):
            np.testing.assert_allclose(a[k], ref[k], **TOL)
            np.testing.assert_array_equal(a[k], b[k])
        np.testing.assert_allclose(a['a_list'], ref['a_list'], **TOL)
