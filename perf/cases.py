"""Timed cases: the work a program has this library do, through its public entry points.

Kinds
  film       one batch of all-film stacks (``FilmStackSolver.solve``)
  film_mix   an uneven batch of all-film stacks (``FilmVarSolver.solve``)
  overlap    overlap integrals J and J_dag of Bloch modes with plane waves (``overlap_batch``)
  interface  film / nanostructure interface matrices (``interface_dense``)
  cascade    S-matrix cascade and fluxes of stacks of arrays (``DenseStackSolver.solve``)
  stack_mix  an uneven batch of array stacks (``StackVarSolver.solve``)
  chain      a wavelength sweep of a one-array stack, fields to spectra (``NanoStackPipeline``)
  fem        Bloch modes of a layer on its mesh (``FemModeSolver.solve_pair``)
  fields     E on a grid inside a layer of solved stacks (``pw_fields``)

``exact`` restates each kind's formulas in plain torch / numpy complex128.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

c128, f64 = torch.complex128, torch.float64
POLS = ('TE', 'TM', 'un', 'R Circ', 'L Circ')


# ------------------------------------------------------------------ cases
def listed():
    return [
        # a single spectral point of one film on a substrate: the smallest call, all latency
        dict(name='film_one', kind='film', batch=1, films=1, order=2, pol='TE'),
        # a spectrum x angle map of a 10-film stack: the library's headline workload
        dict(name='film_sweep', kind='film', batch=32768, films=10, order=5, pol='TE'),
        # stacks of all shapes solved together, as a server batches them
        dict(name='film_mix', kind='film_mix', batch=4096),
        # one wavelength of one array on a 2048-triangle mesh, as the drop-in objects call it
        dict(name='overlap_one', kind='overlap', mesh=32, modes=60, order=3, batch=1, precision='fp64'),
        # a large cell: 20 000 triangles, 400 modes, 317 orders
        dict(name='overlap_large', kind='overlap', mesh=100, modes=400, order=10, batch=1, precision='fp64'),
        # the same through the opt-in single-precision fields and split-TF32 products
        dict(name='overlap_large_tf32x3', kind='overlap', mesh=100, modes=400, order=10, batch=1,
             precision='tf32x3'),
        # interfaces of a large array at a few wavelengths
        dict(name='interface_large', kind='interface', batch=16, order=10, modes=400),
        # four arrays of that size between a substrate and air
        dict(name='cascade_large', kind='cascade', batch=16, order=10, modes=400, arrays=4),
        # stacks of arrays of all sizes solved together
        dict(name='stack_mix', kind='stack_mix', batch=96),
        # a 50-wavelength sweep of one array, from mode fields to spectra
        dict(name='chain_sweep', kind='chain', batch=50, mesh=32, modes=60, order=3),
        # the modes themselves: one layer on a 512-triangle mesh, 40 modes, prime and adjoint
        dict(name='fem_layer', kind='fem', mesh=16, modes=40),
        # field maps in one layer of 256 solved stacks, on the reference's plotting grid
        dict(name='fields_grid', kind='fields', batch=256, order=5, nx=51, ny=51, nz=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(('film', 'film_mix', 'overlap', 'overlap', 'interface', 'cascade', 'stack_mix', 'chain',
                       'fem', 'fields'))
    if kind == 'film':
        films, order = rng.randint(1, 12), rng.randint(0, 8)
        most = 32768 * 12 * 81 // ((films + 2) * (3 * order * order + 1))
        return dict(kind=kind, batch=_log(rng, 1, max(2, min(32768, most))), films=films, order=order,
                    pol=rng.choice(POLS))
    if kind == 'film_mix':
        return dict(kind=kind, batch=_log(rng, 64, 4096))
    if kind == 'overlap':
        mesh, modes, order = _log(rng, 6, 100), _log(rng, 10, 400), rng.randint(1, 10)
        most = 20000 * 400 // (2 * mesh * mesh * modes)
        return dict(kind=kind, mesh=mesh, modes=modes, order=order, batch=rng.randint(1, max(1, min(8, most))),
                    precision=rng.choice(('fp64', 'fp64', 'tf32x3')))
    if kind in ('interface', 'cascade'):
        order, modes = rng.randint(2, 10), _log(rng, 20, 400)
        most = 16 * 618 ** 3 // max(modes, 6 * order * order) ** 3
        c = dict(kind=kind, batch=rng.randint(1, max(1, min(64, most))), order=order, modes=modes)
        if kind == 'cascade':
            c['arrays'] = rng.randint(1, 4)
        return c
    if kind == 'stack_mix':
        return dict(kind=kind, batch=_log(rng, 4, 96))
    if kind == 'chain':
        mesh, modes = rng.randint(6, 32), _log(rng, 15, 60)
        return dict(kind=kind, batch=rng.randint(1, 50), mesh=mesh, modes=modes, order=rng.randint(1, 3))
    if kind == 'fem':
        return dict(kind=kind, mesh=rng.randint(7, 15), modes=rng.randint(10, 40))
    return dict(kind='fields', batch=_log(rng, 1, 256), order=rng.randint(1, 5), nx=rng.randint(5, 51),
                ny=rng.randint(5, 51), nz=rng.randint(1, 4))


# ------------------------------------------------------------------ inputs
def _orders(order):
    """Orders inside the disc, px outer (backend/mode_calcs.py:61-74, square lattice)."""
    a = np.arange(-order, order + 1)
    px, py = np.meshgrid(a, a, indexing='ij')
    keep = px ** 2 + py ** 2 <= order ** 2
    return px[keep].astype(np.int32), py[keep].astype(np.int32)


def _npw(order):
    return len(_orders(order)[0])


def _k_pll(rng, wl, n):
    th, ph = np.radians(rng.uniform(0, 60, n)), np.radians(rng.uniform(0, 90, n))
    k = 2 * np.pi / wl
    return np.stack([k * np.sin(th) * np.cos(ph), k * np.sin(th) * np.sin(ph)], axis=1)


def _cu(a):
    return torch.as_tensor(np.ascontiguousarray(a)).cuda()


def _randn(g, *shape, dtype=c128):
    return torch.randn(shape, dtype=dtype, device='cuda', generator=g)


@functools.lru_cache(maxsize=8)
def _mesh(n, dy=1.0):
    from emustack_b200.mesh import square_cell
    return square_cell(n, dy=dy, radius=0.3 * dy, jitter=0.2, seed=n)


def _film_inputs(c, seed):
    rng = np.random.default_rng(seed)
    B, L = c['batch'], c['films'] + 2
    wl = rng.uniform(350, 1100, B)
    n = np.tile(np.concatenate([[1.46], rng.uniform(1.3, 4.0, L - 2) + 1j * rng.uniform(0, 0.5, L - 2),
                                [1.0]]).astype(complex), (B, 1))
    return dict(wl=_cu(wl), kp=_cu(_k_pll(rng, wl, B)), n=_cu(n), h=_cu(rng.uniform(20, 300, L - 2)))


def _film_points(c, seed):
    """Uneven film stacks: P = 2 Npw log-uniform in [50, 900], 2-12 films, four polarisations."""
    rng, shape = np.random.default_rng(seed), np.random.default_rng(c['batch'])
    tab = np.array([_npw(o) for o in range(17)])
    pts = []
    for i in range(c['batch']):
        order = int(np.argmin(np.abs(tab - math.exp(shape.uniform(math.log(50), math.log(900))) / 2)))
        F = int(shape.integers(2, 13))
        n = np.concatenate([[1.46], rng.uniform(1.3, 4.0, F) + 1j * rng.uniform(0, 0.5, F), [1.0]])
        wl = rng.uniform(350, 1100)
        pts.append((n, rng.uniform(20, 300, F), wl, _k_pll(rng, wl, 1)[0], order, POLS[i % 4]))
    return pts


def _overlap_inputs(c, seed):
    g = torch.Generator(device='cuda').manual_seed(seed)
    rng = np.random.default_rng(seed)
    B, M, nel = c['batch'], c['modes'], 2 * c['mesh'] ** 2
    wl = rng.uniform(400, 900, B) / 700.0
    dt = c128 if c['precision'] == 'fp64' else torch.complex64
    return dict(bloch=_cu(_k_pll(rng, wl, B)), k0=_cu(2 * np.pi / wl), sol1=_randn(g, B, nel, M, 13, 3, dtype=dt),
                sol2=_randn(g, B, nel, M, 13, 3, dtype=dt), scale2=_randn(g, B, M))


def _array_points(rng, g, B, order, M, arrays):
    """Films' k_z, and J, J_dag, Bloch k_z and heights of `arrays` layers, at B points (period 500 nm).
    J_dag is near J's adjoint, as biorthogonal modes give it, and most modes are evanescent."""
    period = 500.0
    wl = rng.uniform(350, 1100, B)
    kp = _cu(_k_pll(rng, wl, B) * period)
    wln = _cu(wl / period)
    px, py = (_cu(v).to(f64) for v in _orders(order))
    P = 2 * len(px)
    kz = {}
    sort = None
    for nm, n in (('air', 1.0), ('sub', 1.46)):
        k = 2 * np.pi * n / wln[:, None]
        z = torch.sqrt((k * k - (kp[:, :1] + 2 * np.pi * px) ** 2 - (kp[:, 1:] + 2 * np.pi * py) ** 2).to(c128))
        if sort is None:
            sort = torch.argsort(-z.real + z.imag, dim=1)
        kz[nm] = z.gather(1, sort)
    k0 = 2 * np.pi / wln[:, None]
    layers = []
    for _ in range(arrays):
        u = torch.rand((3, B, M), dtype=f64, device='cuda', generator=g)
        J = _randn(g, B, P, M) / math.sqrt(P)
        bm = torch.complex(2 * u[0] * (u[2] < 0.2), torch.where(u[2] < 0.2, 0.1 * u[1], 8 * u[1]))
        layers.append(dict(J=J, Jd=(J.mH + 0.1 * _randn(g, B, M, P) / math.sqrt(P)).contiguous(), kz=bm * k0,
                           h=float(rng.uniform(50, 200) / period)))
    spec = ((px == 0) & (py == 0)).nonzero()[0]
    return dict(B=B, P=P, M=M, wln=wln, kza=kz['air'], kzs=kz['sub'], layers=layers,
                spec=(sort == spec).to(torch.int32).argmax(dim=1).to(torch.int32),
                nprop=torch.stack([(kz[k].imag == 0).sum(1) for k in ('air', 'air', 'sub')], 1).to(torch.int32))


def _array_inputs(c, seed):
    g = torch.Generator(device='cuda').manual_seed(seed)
    return _array_points(np.random.default_rng(seed), g, c['batch'], c['order'], c['modes'], c.get('arrays', 1))


def _mix_shapes(c):
    """Shapes of uneven array stacks: P = 2 Npw log-uniform in [25, 260], M = P + 20, 2-6 arrays."""
    rng = np.random.default_rng(c['batch'])
    tab = np.array([_npw(o) for o in range(8)])
    return [(int(np.argmin(np.abs(tab - math.exp(rng.uniform(math.log(25), math.log(260))) / 2))),
             int(rng.integers(2, 7))) for _ in range(c['batch'])]


def _chain_inputs(c, seed):
    g = torch.Generator(device='cuda').manual_seed(seed)
    rng = np.random.default_rng(seed)
    B, M, nel = c['batch'], c['modes'], 2 * c['mesh'] ** 2
    wl = np.linspace(400.0, 900.0, B) if B > 1 else np.array([650.0])
    th, ph = np.radians(rng.uniform(1, 30)), np.radians(rng.uniform(5, 85))
    k = 2 * np.pi / wl
    kp = np.stack([k * np.sin(th) * np.cos(ph), k * np.sin(th) * np.sin(ph)], axis=1)
    k0 = 2 * np.pi / (wl / 600.0)
    beta = (rng.uniform(0.1, 2, (B, M)) + 1j * rng.uniform(0, 0.1, (B, M))) * k0[:, None]
    sol1 = 0.02 * _randn(g, B, nel, M, 13, 3)
    # adjoint modes near the conjugates of the prime ones, so that no <adjoint | prime> vanishes
    sol2 = sol1.conj().resolve_conj() + 0.002 * _randn(g, B, nel, M, 13, 3)
    return dict(wl=_cu(wl), kp=_cu(kp), sol1=sol1, sol2=sol2, beta=_cu(beta))


def _fields_inputs(c, seed):
    g = torch.Generator(device='cuda').manual_seed(seed)
    rng = np.random.default_rng(seed)
    B, period = c['batch'], 500.0
    px, py = _orders(c['order'])
    S = len(px)
    wl = rng.uniform(350, 1100, B)
    kp = _k_pll(rng, wl, B) * period
    al, be = kp[:, :1] + 2 * np.pi * px, kp[:, 1:] + 2 * np.pi * py
    k0 = 2 * np.pi / (wl / period)
    kza = np.sqrt((k0[:, None] ** 2 - al ** 2 - be ** 2).astype(complex))
    sort = np.argsort(-kza.real + kza.imag, axis=1, kind='stable')
    n = rng.uniform(1.3, 4.0, B) + 1j * rng.uniform(0, 0.5, B)
    kz = np.take_along_axis(np.sqrt((n * k0)[:, None] ** 2 - al ** 2 - be ** 2), sort, 1)
    h = rng.uniform(20, 300, B) / period
    decay = torch.exp(-0.3 * torch.arange(S, dtype=f64, device='cuda')).repeat(2)
    return dict(alphas=_cu(al), betas=_cu(be), sort_order=_cu(sort.astype(np.int32)), kz=_cu(kz), n=_cu(n),
                vec_coef_down=_randn(g, B, 2 * S) * decay, vec_coef_up=_randn(g, B, 2 * S) * decay,
                x=_cu(np.linspace(0, 1, c['nx'])), y=_cu(np.linspace(0, 1, c['ny'])),
                z=_cu(np.linspace(0, float(h.min()), c['nz'])), height_norm=_cu(h))


# ------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    kind, s = case['kind'], dict(case=case)
    if kind == 'film':
        from emustack_b200.films import FilmStackSolver
        s.update(_film_inputs(case, seed), solver=FilmStackSolver(case['films'] + 2, case['order'], 500.0))
    elif kind == 'film_mix':
        from emustack_b200.films import FilmPoint, FilmVarSolver
        pts = [FilmPoint(n, h, wl, kp, 500.0, order, pol=pol)
               for n, h, wl, kp, order, pol in _film_points(case, seed)]
        s['solver'] = FilmVarSolver()
        s['plan'] = s['solver'].plan(pts)
    elif kind == 'overlap':
        from emustack_b200.overlap import DeviceMesh
        px, py = _orders(case['order'])
        s.update(_overlap_inputs(case, seed), mesh=DeviceMesh(_mesh(case['mesh'])), px=_cu(px), py=_cu(py))
    elif kind in ('interface', 'cascade'):
        from emustack_b200.dense import DenseStackSolver
        s['pts'] = _array_inputs(case, seed)
        s['n_air'] = torch.ones(case['batch'], dtype=c128, device='cuda')
        if kind == 'cascade':
            s['layers'] = _device_layers(s['pts'])
            s['solver'] = DenseStackSolver()
    elif kind == 'stack_mix':
        from emustack_b200.dense import StackVarSolver, VarStack
        rng, g = np.random.default_rng(seed), torch.Generator(device='cuda').manual_seed(seed)
        s['stacks'] = []
        for order, arrays in _mix_shapes(case):
            p = _array_points(rng, g, 1, order, 2 * _npw(order) + 20, arrays)
            lays = [tuple(t[0].contiguous() for t in (ly.R12, ly.T12, ly.R21, ly.T21))
                    + (ly.dense, None if ly.kz is None else ly.kz[0].contiguous(), ly.height_norm)
                    for ly in _device_layers(p)]
            s['stacks'].append(VarStack(lays, p['P'], pol='TE', spec=int(p['spec'][0]),
                                        num_prop=[int(v) for v in p['nprop'][0]]))
        s['solver'] = StackVarSolver()
    elif kind == 'chain':
        from emustack_b200.pipeline import NanoStackPipeline
        i = _chain_inputs(case, seed)
        s['pipe'] = NanoStackPipeline(_mesh(case['mesh']), 600.0, case['order'], case['modes'], case['batch'], 100.0)
        s['pipe'].load(i['wl'], i['kp'], i['sol1'], i['sol2'], i['beta'])
        s['pipe'].capture()
    elif kind == 'fem':
        from emustack_b200.fem import FemMesh, FemModeSolver
        s['mesh'], s['n'], s['wl'] = _fem_inputs(case, seed)
        m = s['mesh']
        edge = (m.x == 0).any(1) | (m.x == m.x.max(0)).any(1)
        s['solver'] = FemModeSolver(FemMesh(m.x, edge.astype(np.int32), m.table_nod, m.type_el))
    else:
        s.update(args=_fields_inputs(case, seed))
    return s


def _fem_inputs(c, seed):
    """A high-index wire in air in a rectangular cell, at normal incidence."""
    rng = np.random.default_rng(seed)
    return _mesh(c['mesh'], 0.8), [1.0, complex(rng.uniform(3.4, 4.0), 0.05)], float(rng.uniform(0.8, 1.2))


def _device_layers(p):
    """The substrate, the arrays and the air above them as device layers."""
    from emustack_b200.dense import DenseLayer, film_interface, interface_dense
    na = torch.ones(p['B'], dtype=c128, device='cuda')
    Rs, Ts = film_interface(p['kza'], na, p['kzs'], 1.46 * na, p['wln'])
    Ra, Ta = film_interface(p['kza'], na, p['kza'], na, p['wln'])
    mid = []
    for ly in p['layers']:
        R12, T12, R21, T21, _ = interface_dense(p['kza'], na, p['wln'], ly['J'], ly['Jd'])
        mid.append(DenseLayer(R12, T12, R21, T21, True, ly['kz'], ly['h']))
    return [DenseLayer(Rs, Ts, -Rs, Ts, False)] + mid + [DenseLayer(Ra, Ta, -Ra, Ta, False)]


def run(s):
    c = s['case']
    kind = c['kind']
    if kind == 'film':
        o = s['solver'].solve(s['wl'], s['kp'], s['n'], s['h'], pol=c['pol'])
        return {k: o[k] for k in ('R_net', 'T_net', 'a_list', 't_list', 'r_list', 'flags')}
    if kind == 'film_mix':
        o = s['solver'].solve(s['plan'])
        return {k: o[k] for k in ('R_net', 'T_net', 'a_list', 't_list', 'r_list', 'flags')}
    if kind == 'overlap':
        from emustack_b200.overlap import overlap_batch
        J, Jd, inv = overlap_batch(s['mesh'], s['px'], s['py'], c['order'], s['bloch'], s['k0'], s['sol1'], s['sol2'],
                                   scale2=s['scale2'], precision=c['precision'])
        return dict(J=J, J_dag=Jd, order=inv)
    if kind == 'interface':
        from emustack_b200.dense import interface_dense
        p = s['pts']
        ly = p['layers'][0]
        R12, T12, R21, T21, info = interface_dense(p['kza'], s['n_air'], p['wln'], ly['J'], ly['Jd'])
        return dict(R12=R12, T12=T12, R21=R21, T21=T21, info=info)
    if kind == 'cascade':
        p = s['pts']
        o = s['solver'].solve(s['layers'], p['P'], pol='TE', specular=p['spec'], num_prop=p['nprop'])
        return {k: o[k] for k in ('R_net', 'T_net', 'a_list', 't_list', 'r_list', 'info')}
    if kind == 'stack_mix':
        o = s['solver'].solve(s['stacks'])
        return {k: o[k] for k in ('R_net', 'T_net', 'a_list', 't_list', 'r_list', 'info')}
    if kind == 'chain':
        o = s['pipe'].replay()
        return {k: o[k] for k in ('R_net', 'T_net', 'a_list', 't_list', 'r_list', 'info')}
    if kind == 'fem':
        b1, s1, b2, s2 = s['solver'].solve_pair(s['n'], s['wl'], (0.0, 0.0), c['modes'])
        return dict(beta=b1, sol=s1, beta_adjoint=b2, sol_adjoint=s2)
    from emustack_b200.fields import pw_fields
    E, Eabs = pw_fields(grid=True, **s['args'])
    return dict(E=E, abs=Eabs)


# ------------------------------------------------------------------ what a pass cannot do without
def _cascade_work(B, P, M, arrays):
    """Two LU solves and the products of each array, and of the air above."""
    lay = 8 / 3 * (P ** 3 + M ** 3) + 8 * (P * P * M + M * M * P)           # factor and solve
    lay += 8 * (P ** 3 + P * P * M + M * P * P + M * M * P)                 # gap products
    lay += 8 * (M ** 3 + P * M * P + P * M * M + P * M * P)                 # layer products
    top = 8 / 3 * P ** 3 + 24 * P ** 3
    io = 16 * (arrays * (P * P + M * M + 2 * P * M + M) + 6 * P + 2 * P * P)
    return dict(bytes=B * io, flops=B * (arrays * lay + top))


def work(c):
    kind = c['kind']
    if kind == 'film':
        B, L, S = c['batch'], c['films'] + 2, _npw(c['order'])
        return dict(bytes=B * (24 + 16 * L + 64 * S + 16 * (L - 1) + 12), flops=B * S * L * 244)
    if kind == 'film_mix':
        shapes = [(len(p[0]), _npw(p[4])) for p in _film_points(c, 0)]
        return dict(bytes=sum(120 + 24 * L + 64 * S + 16 * (L - 1) + 12 for L, S in shapes),
                    flops=sum(S * L * 244 for L, S in shapes))
    if kind == 'overlap':
        B, M, nel, S = c['batch'], c['modes'], 2 * c['mesh'] ** 2, _npw(c['order'])
        w = 16 if c['precision'] == 'fp64' else 8
        return dict(bytes=B * (2 * nel * M * 12 * w + 2 * 2 * S * M * 16), flops=B * 2 * 8 * S * 2 * M * 6 * nel)
    if kind == 'interface':
        B, P, M = c['batch'], 2 * _npw(c['order']), c['modes']
        return dict(bytes=B * 16 * (2 * P * M + P * P + M * M + 2 * P * M),
                    flops=B * (8 / 3 * M ** 3 + 8 * (M * M * P + M * M * P + M ** 3 + P * P * M + P * M * M)))
    if kind == 'cascade':
        return _cascade_work(c['batch'], 2 * _npw(c['order']), c['modes'], c['arrays'])
    if kind == 'stack_mix':
        each = [_cascade_work(1, 2 * _npw(o), 2 * _npw(o) + 20, k) for o, k in _mix_shapes(c)]
        return {k: sum(e[k] for e in each) for k in ('bytes', 'flops')}
    if kind == 'chain':
        B, M, nel, S = c['batch'], c['modes'], 2 * c['mesh'] ** 2, _npw(c['order'])
        w = _cascade_work(B, 2 * S, M, 1)
        return dict(bytes=B * nel * M * 16 * (12 + 22) + 16 * B * 4 * S * S,
                    flops=w['flops'] + B * nel * M * (12 * 22 * 4 + 2 * 8 * S * 2 * 6))
    if kind == 'fem':
        n, nt, M = 12 * 2 * c['mesh'] ** 2, 7.5 * 2 * c['mesh'] ** 2, c['modes']
        return dict(bytes=2 * 16 * (2 * c['mesh'] ** 2 * M * 39), flops=2 * (8 / 3 * n ** 3 + 8 * n * n * nt))
    Q, S = c['nx'] * c['ny'] * c['nz'], _npw(c['order'])
    return dict(bytes=c['batch'] * (S * 100 + Q * 56), flops=c['batch'] * Q * S * (24 + 6 / c['nz']))


# ------------------------------------------------------------------ exact
def _film_kz(n, wl, kp, order, period=500.0):
    """Sorted k_z [B, L, S], the specular position, in units of the period (backend/mode_calcs.py:116-186)."""
    px, py = (_cu(v).to(f64) for v in _orders(order))
    al, be = kp[:, :1] * period + 2 * np.pi * px, kp[:, 1:] * period + 2 * np.pi * py
    k0 = 2 * np.pi / (wl / period)
    z = lambda k: torch.sqrt((k * k)[:, None] - (al ** 2 + be ** 2).to(c128))
    air = z(k0.to(c128))
    sort = torch.argsort(-air.real + air.imag, dim=1, stable=True)
    kz = torch.stack([z(k0 * n[:, i]).gather(1, sort) for i in range(n.shape[1])], 1)
    kz_air = air.gather(1, sort)
    spec = (sort == ((px == 0) & (py == 0)).nonzero()[0]).to(torch.int32).argmax(dim=1)
    return kz, kz_air, spec, k0


def _impedance(n, k0, kz):
    q = (k0 * n)[:, None] / kz
    return torch.cat([q / n[:, None], 1 / (q * n[:, None])], 1)


def _film_rt(Z1, Z2):
    return (Z2 - Z1) / (Z2 + Z1), 2 * torch.sqrt(Z2) * torch.sqrt(Z1) / (Z2 + Z1)


def _incident(spec, S, pol):
    a = {'TE': (1, 0), 'TM': (0, 1), 'un': (2 ** -0.5, 2 ** -0.5), 'R Circ': (2 ** -0.5, 1j * 2 ** -0.5),
         'L Circ': (2 ** -0.5, -1j * 2 ** -0.5)}[pol]
    v = torch.zeros((len(spec), 2 * S), dtype=c128, device='cuda')
    b = torch.arange(len(spec), device='cuda')
    v[b, spec.long()], v[b, spec.long() + S] = a[0], a[1]
    return v


def _cascade(layers, props, inc, nprop, diag):
    """R_net, T_net and the a / t / r lists of a stack (backend/stack.py:162-426).  layers: (R12, T12, R21, T21);
    props: exp(i k_z h) of the finite layers [B, M]; diag: every matrix is given by its diagonal."""
    if diag:
        mm, solve, row, col = torch.mul, lambda a, b: b / a, torch.mul, torch.mul
        eye, vec = (lambda a: torch.ones_like(a)), torch.mul
    else:
        mm, solve = torch.matmul, torch.linalg.solve
        row, col = (lambda p, a: p[:, :, None] * a), (lambda a, p: a * p[:, None, :])
        eye = lambda a: torch.eye(a.shape[-1], dtype=c128, device='cuda').expand(a.shape)
        vec = lambda a, v: torch.matmul(a, v[..., None])[..., 0]
    L = len(layers)
    rnet, tnet = layers[0][0], layers[0][1]
    t0, rl, x21, x12 = tnet, [rnet], [], []
    for i in range(1, L):
        R12, T12, R21, T21 = layers[i]
        a = mm(R12, rnet)
        x = solve(eye(a) - a, T21)
        tnet, rnet = mm(tnet, x), R21 + mm(T12, mm(rnet, x))
        x21.append(x)
        rl.append(rnet)
        if i == L - 1:
            break
        p = props[i - 1]
        prp = row(p, col(rnet, p))
        a = mm(R21, prp)
        x = solve(eye(a) - a, T12)
        y = row(p, x)
        tnet, rnet = mm(tnet, y), R12 + mm(T21, mm(row(p, rnet), y))
        x12.append(x)
        rl.append(rnet)
    S = inc.shape[1] // 2
    idx = torch.arange(2 * S, device='cuda') % S
    power = lambda v, m: ((v.abs() ** 2) * (idx[None] < m[:, None])).sum(1)
    pol = torch.where(torch.arange(2 * S, device='cuda') < S, -1j, 1j).to(c128)

    def inner(d, u):
        pr = idx[None] < nprop[:, :1]
        x = pol * (d.conj() * u - u.conj() * d)
        return torch.where(pr, (d.abs() ** 2 - u.abs() ** 2).to(c128), x).sum(1)

    down, up0 = [power(inc, nprop[:, 1])], power(vec(rl[-1], inc), nprop[:, 1])
    f1 = vec(x21[-1], inc)
    for i in range(L - 2):
        down.append(inner(f1, vec(rl[-2 * i - 2], f1)).abs())
        f2 = vec(x12[-i - 1], f1)
        f1 = vec(x21[-i - 2], props[-i - 1] * f2)
    down.append(power(vec(t0, f1), nprop[:, 2]))
    D = torch.stack(down, 1)
    a = torch.cat([(D[:, 1:-1] - D[:, 2:]).abs(), (D[:, 0] - D[:, -1] - up0).abs()[:, None]], 1)
    t = torch.cat([D[:, 2:] / D[:, :-2], (D[:, -1] / D[:, 0])[:, None]], 1)
    return dict(R_net=rnet, T_net=tnet, a_list=a, t_list=t, r_list=up0 / D[:, 0])


def _films_exact(n, h, wl, kp, order, pol):
    kz, kz_air, spec, k0 = _film_kz(n, wl, kp, order)
    one = torch.ones_like(n[:, 0])
    Z0 = _impedance(one, k0, kz_air)
    layers = []
    for i in range(n.shape[1]):
        r, t = _film_rt(Z0, _impedance(n[:, i], k0, kz[:, i]))
        layers.append((r, t, -r, t))
    props = [torch.exp(1j * kz[:, i + 1] * h[:, i:i + 1] / 500.0).repeat(1, 2) for i in range(n.shape[1] - 2)]
    nprop = torch.stack([(z.imag == 0).sum(1) for z in (kz_air, kz[:, -1], kz[:, 0])], 1)
    return _cascade(layers, props, _incident(spec, kz.shape[2], pol), nprop, True)


def _interface_exact(Z, J, Jd):
    """R12, T12, R21, T21 of a film of impedances Z and an array (backend/mode_calcs.py:480-515)."""
    q = torch.sqrt(1 / Z)
    A, B = q[:, :, None] * J, Jd * q[:, None, :]
    BA = B @ A
    I = torch.eye(BA.shape[-1], dtype=c128, device='cuda')
    X = torch.linalg.solve(I + BA, torch.cat([B, I - BA, I.expand(BA.shape)], 2))
    P, M = J.shape[1:]
    DB, R21, Di = X[:, :, :P], X[:, :, P:P + M], X[:, :, P + M:]
    return 2 * A @ DB - torch.eye(P, dtype=c128, device='cuda'), 2 * DB, R21, 2 * A @ Di


def _arrays_exact(p):
    one = torch.ones(p['B'], dtype=c128, device='cuda')
    k0 = 2 * np.pi / p['wln']
    Z0, Zs = _impedance(one, k0, p['kza']), _impedance(1.46 * one, k0, p['kzs'])
    film = lambda Z: (lambda r, t: tuple(torch.diag_embed(v) for v in (r, t, -r, t)))(*_film_rt(Z0, Z))
    layers = [film(Zs)] + [_interface_exact(Z0, ly['J'], ly['Jd']) for ly in p['layers']] + [film(Z0)]
    props = [torch.exp(1j * ly['kz'] * ly['h']) for ly in p['layers']]
    return _cascade(layers, props, _incident(p['spec'], p['P'] // 2, 'TE'), p['nprop'], False)


def _quadrature():
    """The 16-point rule of Lyness and Jespersen (1975) on the unit triangle, its P2 basis."""
    w = np.array([1.443156076777862e-1 / 2] + [2.852749028018549e-1 / 6] * 3 + [9.737549286959440e-2 / 6] * 3
                 + [3.096521116041552e-1 / 6] * 3 + [1.633818850466092e-1 / 12] * 6)
    a1, b1, a2, b2 = 4.592925882927229e-1, 8.141482341455413e-2, 5.054722831703103e-2, 8.989055433659379e-1
    a3, b3 = 1.705693077517601e-1, 6.588613844964797e-1
    a4, b4, c4 = 7.284923929554041e-1, 2.63112829634638689e-1, 8.394777409957211e-3
    x = np.array([1 / 3, a1, a1, b1, a2, a2, b2, a3, a3, b3, a4, b4, b4, c4, c4, a4])
    y = np.array([1 / 3, a1, b1, a1, a2, b2, a2, a3, b3, a3, b4, a4, c4, b4, a4, c4])
    l = 1 - x - y
    return w, x, y, np.stack([l * (2 * l - 1), x * (2 * x - 1), y * (2 * y - 1), 4 * x * l, 4 * x * y, 4 * y * l], 1)


def _corners(mesh):
    v = np.asarray(mesh.x)[np.asarray(mesh.table_nod)[:, :3] - 1]
    return v[:, 0], np.stack([v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]], 2)


def _overlap_exact(mesh, order, bloch, k0, sol1, sol2, scale2):
    """J, J_dag and the plane waves' positions of one problem (J_overlap.f, J_dagger_overlap.f)."""
    w, xq, yq, phi = _quadrature()
    v0, Bm = _corners(mesh)
    pts = v0[:, None] + np.einsum('eij,qj->eqi', Bm, np.stack([xq, yq], 1))
    wd = _cu(w[None] * np.abs(np.linalg.det(Bm))[:, None])
    px, py = (_cu(v).to(f64) for v in _orders(order))
    al, be = bloch[0] + 2 * np.pi * px, bloch[1] + 2 * np.pi * py
    pos = torch.argsort(torch.argsort(-(k0 ** 2 - al ** 2 - be ** 2), stable=True))
    at = torch.argsort(pos)
    al, be = al[at], be[at]
    pts, phi = _cu(pts), _cu(phi)
    S, M, nel = len(al), sol1.shape[1], sol1.shape[0]
    G, Gd = (torch.zeros((S, 2 * M), dtype=c128, device='cuda') for _ in range(2))
    for e in range(0, nel, 2048):
        q = pts[e:e + 2048]
        ph = torch.exp(-1j * (al[:, None, None] * q[..., 0] + be[:, None, None] * q[..., 1])) * wd[e:e + 2048]
        E = torch.einsum('seq,qk->sek', ph, phi.to(c128)).reshape(S, -1)
        tr = lambda f: f[e:e + 2048, :, :6, :2].to(c128).permute(0, 2, 3, 1).reshape(E.shape[1], 2 * M)
        G += E @ tr(sol1)
        Gd += E.conj() @ tr(sol2)
    nm = torch.sqrt(al ** 2 + be ** 2)
    ca, cb = (al / nm)[:, None], (be / nm)[:, None]
    out = [torch.cat([cb * g[:, :M] - ca * g[:, M:], ca * g[:, :M] + cb * g[:, M:]]) for g in (G, Gd)]
    return out[0], (out[1] * scale2[None]).T.contiguous(), pos


def _mode_scale(mesh, k0, beta, sol1, sol2):
    """1 / <adjoint | prime> of every mode (orthogonal.f, normalisation.f), all materials with pp = 1."""
    w, xq, yq, phi2 = _quadrature()
    mono = lambda x, y: np.stack([x ** i * y ** j for i in range(4) for j in range(4 - i)], -1)
    third = np.array([(0, 0), (3, 0), (0, 3), (1, 0), (2, 0), (2, 1), (1, 2), (0, 2), (0, 1), (1, 1)]) / 3.0
    coef = np.linalg.inv(mono(third[:, 0], third[:, 1]))
    dx = np.stack([i * xq ** max(i - 1, 0) * yq ** j for i in range(4) for j in range(4 - i)], -1) @ coef
    dy = np.stack([j * xq ** i * yq ** max(j - 1, 0) for i in range(4) for j in range(4 - i)], -1) @ coef
    _, Bm = _corners(mesh)
    wd = w[None] * np.abs(np.linalg.det(Bm))[:, None]
    T = np.linalg.inv(Bm)                                               # [e][reference axis][x, y]
    mass = _cu(np.einsum('eq,qi,qj->eij', wd, phi2, phi2)).to(c128)
    grad = _cu(np.einsum('eq,qi,aqj,eac->eicj', wd, phi2, np.stack([dx, dy]), T)).to(c128)
    tr = sol1[:, :, :6, :2]
    z = torch.cat([sol1[:, :, :3, 2], sol1[:, :, 6:13, 2]], 2)
    f = torch.einsum('eij,emjc->emic', mass, tr) - torch.einsum('eicj,emj->emic', grad, z)
    return 1 / ((f * sol2[:, :, :6, :2]).sum((0, 2, 3)) * beta / k0)


def _chain_exact(c, seed):
    i, mesh = _chain_inputs(c, seed), _mesh(c['mesh'])
    period, M, S = 600.0, c['modes'], _npw(c['order'])
    n = torch.tensor([[1.46, 1.0]], dtype=c128, device='cuda').repeat(c['batch'], 1)
    kz, kz_air, spec, k0 = _film_kz(n, i['wl'], i['kp'], c['order'], period)
    J, Jd = [], []
    for b in range(c['batch']):
        s = _mode_scale(mesh, k0[b], i['beta'][b], i['sol1'][b], i['sol2'][b])
        j, d, _ = _overlap_exact(mesh, c['order'], i['kp'][b] * period, k0[b], i['sol1'][b], i['sol2'][b], s)
        J.append(j)
        Jd.append(d)
    nprop = torch.stack([(z.imag == 0).sum(1) for z in (kz_air, kz_air, kz[:, 0])], 1)
    return _arrays_exact(dict(B=c['batch'], P=2 * S, wln=2 * np.pi / k0, kza=kz_air, kzs=kz[:, 0], spec=spec,
                              nprop=nprop, layers=[dict(J=torch.stack(J), Jd=torch.stack(Jd), kz=i['beta'],
                                                        h=100.0 / period)]))


def _fields_exact(a):
    """E of TE and TM plane waves in a layer (backend/plotting.py:2896-2977)."""
    B, S = a['alphas'].shape
    s = a['sort_order'].long()
    al, be, ga, n = a['alphas'].gather(1, s), a['betas'].gather(1, s), a['kz'], a['n'][:, None]
    nm, k = torch.sqrt(al ** 2 + be ** 2), torch.sqrt(al ** 2 + be ** 2 + ga ** 2)
    te, tm = torch.sqrt(n * ga / k), torch.sqrt(n * k / ga)
    e_te = torch.stack([be / nm, -al / nm, 0 * nm], 1).to(c128) / te[:, None]
    e_tm = torch.stack([(al / nm).to(c128), (be / nm).to(c128), -nm / ga], 1) / tm[:, None]
    amp = lambda v: e_te * v[:, None, :S] + e_tm * v[:, None, S:]
    dn, up = amp(a['vec_coef_down']), amp(a['vec_coef_up'])
    X = torch.exp(1j * al[:, :, None] * a['x'])
    Y = torch.exp(1j * be[:, :, None] * a['y'])
    z, h = a['z'][None, None], a['height_norm'][:, None, None]
    Z = dn[..., None] * torch.exp(-1j * ga[:, :, None] * (z - h))[:, None]
    Z = Z + up[..., None] * torch.exp(1j * ga[:, :, None] * z)[:, None]
    E = torch.stack([torch.einsum('sx,sy,csz->cxyz', X[b], Y[b], Z[b]).reshape(3, -1) for b in range(B)])
    return dict(E=E, abs=torch.sqrt((E.abs() ** 2).sum(1)))


def exact(case, seed):
    kind = case['kind']
    if kind == 'film':
        i = _film_inputs(case, seed)
        o = _films_exact(i['n'], i['h'].expand(case['batch'], -1), i['wl'], i['kp'], case['order'], case['pol'])
        return dict(o, flags=None)
    if kind == 'film_mix':
        pts = _film_points(case, seed)
        groups, got = {}, [None] * len(pts)
        for j, p in enumerate(pts):
            groups.setdefault((p[4], len(p[0]), p[5]), []).append(j)
        for (order, _, pol), js in groups.items():
            col = lambda q: _cu(np.stack([np.asarray(pts[j][q]) for j in js]))
            o = _films_exact(col(0), col(1), col(2), col(3), order, pol)
            for r, j in enumerate(js):
                got[j] = {k: v[r].reshape(-1) for k, v in o.items()}
        return dict({k: torch.cat([g[k] for g in got]) for k in got[0]}, flags=None)
    if kind == 'overlap':
        i, mesh = _overlap_inputs(case, seed), _mesh(case['mesh'])
        o = [_overlap_exact(mesh, case['order'], i['bloch'][b], i['k0'][b], i['sol1'][b], i['sol2'][b],
                            i['scale2'][b]) for b in range(case['batch'])]
        J, Jd = torch.stack([v[0] for v in o]), torch.stack([v[1] for v in o])
        return dict(J=J, J_dag=Jd, order=None)
    if kind == 'interface':
        p = _array_inputs(case, seed)
        Z = _impedance(torch.ones(p['B'], dtype=c128, device='cuda'), 2 * np.pi / p['wln'], p['kza'])
        o = _interface_exact(Z, p['layers'][0]['J'], p['layers'][0]['Jd'])
        return dict(zip(('R12', 'T12', 'R21', 'T21'), o), info=None)
    if kind == 'cascade':
        return dict(_arrays_exact(_array_inputs(case, seed)), info=None)
    if kind == 'stack_mix':
        rng, g = np.random.default_rng(seed), torch.Generator(device='cuda').manual_seed(seed)
        o = [_arrays_exact(_array_points(rng, g, 1, order, 2 * _npw(order) + 20, k))
             for order, k in _mix_shapes(case)]
        return dict({k: torch.cat([v[k].reshape(-1) for v in o]) for k in o[0]}, info=None)
    if kind == 'chain':
        return dict(_chain_exact(case, seed), info=None)
    if kind == 'fields':
        return _fields_exact(_fields_inputs(case, seed))
    return None  # fem: a dense eigenproblem of thousands of unknowns takes minutes
