"""The workloads that the framework's performance is measured on.

Each case is one thing a SawSim user has the engine do: a field solve at the
resonance peak, a Y11 sweep of a band, the zoom sweeps of a locate, a lossy
template, a sweep of assembled matrices, the adjoint gradient, and the Hex27
slabs in FP64 and in mixed precision.  Cells and bands are the ones of
``sawsim_b200.cases``, ``templates`` and ``params`` at several sizes; the crystal
and the exact band edges come from the seed.

``exact`` solves the same inputs in 64 bits with plain torch: element matrices of
the tensor-product quadratic elements, the master / slave fold, and a block
tridiagonal elimination over the element layers of the depth axis with iterative
refinement.
"""
import math

import numpy as np
import torch

from sawsim_b200 import _lib, cases, params, templates
from sawsim_b200 import materials as mt
from sawsim_b200.engine import FrequencySolver

SCALE_Q9 = 6.173191780858575e-11       # row scaling of the mechanical equations, Q9 cells
SCALE_HEX = 6.723363908816403e-11      # the same for the Hex27 slabs


def listed():
    return [
        # the field at one frequency on the small plane-strain cell: a user plots the mode
        # at the peak of a finished sweep; latency and launches count
        dict(name='me0_16x64_field', call='field', cell='me0', cols=16, rows=64, points=1, precision='fp64'),
        # the same cell's whole band, the smallest full sweep
        dict(name='me0_16x64_sweep', call='sweep', cell='me0', cols=16, rows=64, points=101, precision='fp64'),
        # locate: coarse sweep, then a zoom; each reassembles with its own PML freeze
        # frequency on the analysed engine (16.5k DOF, an odd number of rows)
        dict(name='me1_16x67_zoom', call='zoom', cell='me1', cols=16, rows=67, points=41, precision='fp64'),
        # a lossy generic stack with a coating, as a configuration describes it: Rayleigh
        # damping and dielectric loss, ragged columns and layers
        dict(name='stack_loss', call='sweep', cell='stack', mesh_nm=97, layers=2, coatings=1, points=51, loss=True,
             precision='fp64'),
        # matrices assembled by the pipeline itself (no mesh: graph ordering)
        dict(name='me1_24x80_matrices', call='matrices', cell='me1', cols=24, rows=80, points=25, precision='fp64'),
        # an ordinary two-layer cell in FP64
        dict(name='me1_32x128_sweep', call='sweep', cell='me1', cols=32, rows=128, points=51, precision='fp64'),
        # a part of the full-size two-layer cell's band (262,664 active DOFs)
        dict(name='me1_64x256_sweep', call='sweep', cell='me1', cols=64, rows=256, points=11, precision='fp64'),
        # charges and the adjoint gradient of the four-layer cell: one optimiser step
        dict(name='me1_four_32x128_grad', call='gradient', cell='me1_four', cols=32, rows=128, points=16,
             precision='fp64'),
        # a thin Hex27 slab in FP64
        dict(name='hex_8x2x26_fp64', call='sweep', cell='hex', cols=8, ny=2, rows=26, points=33, precision='fp64'),
        # parts of the double- and four-layer slabs' bands in mixed precision (complex64
        # fronts, Krylov refinement to FP64)
        dict(name='hex_8x4x48_mixed', call='sweep', cell='hex', cols=8, ny=4, rows=48, points=16, precision='mixed'),
        dict(name='hex_four_12x4x48_mixed', call='sweep', cell='hex_four', cols=12, ny=4, rows=48, points=6,
             precision='mixed'),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(['field', 'sweep', 'zoom', 'stack', 'matrices', 'gradient', 'hex_fp64', 'hex_mixed'])
    if kind in ('field', 'sweep', 'zoom', 'matrices'):
        cell = rng.choice(['me0', 'me1', 'me1', 'me1_four'])
        cols = 8 * rng.randint(1, 4)
        rows = log_int(3 * cols, 5 * cols)
        points = 1 if kind == 'field' else log_int(9, 60 if cols < 32 else 30)
        return dict(call=kind, cell=cell, cols=cols, rows=rows, points=points, precision='fp64')
    if kind == 'stack':
        return dict(call='sweep', cell='stack', mesh_nm=log_int(85, 270), layers=rng.randint(1, 3),
                    coatings=rng.randint(0, 1), points=log_int(9, 60), loss=rng.random() < 0.7, precision='fp64')
    if kind == 'gradient':
        cols = 8 * rng.randint(1, 4)
        return dict(call='gradient', cell=rng.choice(['me1', 'me1_four']), cols=cols, rows=32 * rng.randint(1, 4),
                    points=log_int(3, 16), precision='fp64')
    cell = rng.choice(['hex', 'hex', 'hex_four'])
    ny = rng.randint(1, 3)
    return dict(call='sweep', cell=cell, cols=12 if cell == 'hex_four' else 8, ny=ny, rows=log_int(18, 44),
                points=log_int(4, 40 if ny < 2 else 12), precision='fp64' if kind == 'hex_fp64' else 'mixed')


# ----------------------------------------------------------------------------- inputs
def _stack_config(c, f):
    config = dict(model_id='sp_stack', pitch_um=1.085, electrode_um=0.17, substrate_um=0.6, metal_ratio=0.5,
                  mesh_um=c['mesh_nm'] * 1e-3, layers=[dict(thickness_um=t) for t in (0.5, 0.9, 1.7)[:c['layers']]],
                  coatings=[dict(thickness_um=0.31)] * c['coatings'], mode_extension=1, start_ghz=f[0] * 1e-9,
                  stop_ghz=f[-1] * 1e-9, points=len(f))
    if c['loss']:
        config.update(beta_dk=2e-13, eta_eps=2e-3)
    return config


def inputs(c, seed):
    """(cases.Case or HexCase, loss, Q9Model or None) of a case: the crystal and the band from the seed."""
    rng = np.random.default_rng(seed)
    f0, f1 = rng.uniform(1.58e9, 1.62e9), rng.uniform(1.98e9, 2.02e9)
    f = np.linspace(f0, f1, c['points']) if c['points'] > 1 else np.array([rng.uniform(f0, f1)])
    crystal = int(rng.integers(1 << 30))
    if c['cell'] == 'stack':
        xtal, euler = mt.seeded_3m(crystal)
        mats = [mt.rotate(xtal, euler), mt.al()] + [mt.sio2(), mt.poly_si(), mt.si_cubic()][:c['layers']]
        case, loss = templates.case_for(_stack_config(c, f), mats + [mt.sio2()] * c['coatings'])
        return case, loss, None
    if c['cell'].startswith('hex'):
        case = cases.make_hex_case('hex_8x4x48' if c['cell'] == 'hex' else 'hex_12x6x80', crystal, nx=c['cols'],
                                   ny=c['ny'], nz=c['rows'])
    elif c['call'] == 'gradient':
        model = params.Q9Model(cols=c['cols'], rows=c['rows'], seed=crystal, f0=f0, f1=f1,
                               stack='four_layer' if c['cell'] == 'me1_four' else 'two_layer')
        case = model.build(model.defaults())
        case.freqs = f
        return case, templates.Loss(), model
    else:
        name = {'me0': 'me0_16x64', 'me1': 'me1_64x256', 'me1_four': 'me1_128x512'}[c['cell']]
        case = cases.make_case(name, crystal, cols=c['cols'], rows=c['rows'])
    case.freqs = f
    return case, templates.Loss(), None


def _zoom(case):
    """The zoomed band of a locate: the middle fifth of the coarse one."""
    f = case.freqs
    mid, half = 0.5 * (f[0] + f[-1]), 0.1 * (f[-1] - f[0])
    return np.linspace(mid - half, mid + half, f.size)


def prepare(c, seed):
    case, loss, model = inputs(c, seed)
    engine = templates.engine_for(case, loss)
    if c['call'] == 'matrices':
        K, M = engine.export(_lib.SS_MAT_K), engine.export(_lib.SS_MAT_M)
        engine.close()
        engine = FrequencySolver.from_matrices(K, M, *case.bc)
    state = dict(call=c['call'], precision=c['precision'], engine=engine, freqs=case.freqs, top=case.omega_top)
    if c['call'] == 'zoom':
        state['zoom'] = _zoom(case)
    if c['call'] == 'gradient':
        state['seeds'] = model.seeds(model.defaults())
    return state


# ----------------------------------------------------------------------------- the pass
def run(s):
    e = s['engine']
    if s['call'] == 'field':
        disp, Q, _ = e.solve(2 * np.pi * s['freqs'][0], 1.0)
        return dict(disp=disp, Q=np.array([Q]))
    if s['call'] == 'zoom':
        e.set_freeze_frequency(s['top'])
        Q = e.sweep(s['freqs'], 1.0, s['precision'])
        e.set_freeze_frequency(2 * np.pi * s['zoom'][-1])
        return dict(Q=Q, Q_zoom=e.sweep(s['zoom'], 1.0, s['precision']))
    if s['call'] == 'gradient':
        Q, dQ, _ = e.gradient(2 * np.pi * s['freqs'], s['seeds'], 1.0, s['precision'])
        return dict(Q=Q, dQ=dQ)
    return dict(Q=e.sweep(s['freqs'], 1.0, s['precision']))


def _sizes(c):
    """About how many active DOFs there are, and how many in one cross-section."""
    if c['cell'].startswith('hex'):
        cross = 2 * c['cols'] * 2 * c['ny'] * 4
    elif c['cell'] == 'stack':
        h = c['mesh_nm'] * 1e-3
        deep = 2.17 / min(4 * h, 0.54)             # element rows of the PML, and of the stack above it
        depth = 0.6 + sum((0.5, 0.9, 1.7)[:c['layers']]) + 0.31 * c['coatings']
        return int(128 * math.ceil(0.27125 / h) * (max(8, deep) + depth / h)), 64 * math.ceil(0.27125 / h)
    else:
        cross = 2 * c['cols'] * (3 if c['cell'] == 'me0' else 4)
    return cross * 2 * c['rows'], cross


def work(c):
    """What a pass cannot do without: each point's factorisation by nested dissection as
    a symmetric matrix (operations fitted to the host analysis of these cells: n^1.5 in
    2D, n cross^2 for the slabs), a solve with its factors, the condensed matrices read
    and the results written once."""
    n, cross = _sizes(c)
    hexa = c['cell'].startswith('hex')
    flops = 7.5 * n * cross ** 2 if hexa else (430.0 if c['cell'] == 'me0' else 680.0) * n ** 1.5
    factors = 60.0 * n ** 1.5 if hexa else 31.0 * n * math.log2(max(4.0, n / 48.0))
    passes = c['points'] * (2 if c['call'] == 'zoom' else 1)
    solves = 2 if c['call'] == 'gradient' else 1
    entries = n * (190.0 if hexa else 62.0)
    return dict(flops=passes * (flops + solves * 8.0 * factors),
                bytes=32.0 * entries * passes / c['points'] + 16.0 * (n if c['call'] == 'field' else passes))


# ----------------------------------------------------------------------------- 64-bit values
# (component, Voigt row, derivative axis, stretch axis as a row and as a column of C) of
# each strain term
_STRAIN_Q9 = [(0, 0, 0, 0, 0), (0, 5, 1, 1, 1), (1, 1, 1, 1, 1), (1, 5, 0, 0, 0), (2, 3, 1, 1, 1), (2, 4, 0, 0, 0)]
_STRAIN_HEX = [(0, 0, 0, 0, 0), (0, 5, 1, 1, 0), (0, 4, 2, 2, 0), (1, 5, 0, 1, 0), (1, 1, 1, 1, 1), (1, 3, 2, 2, 1),
               (2, 4, 0, 2, 0), (2, 2, 2, 2, 2)]


def _grams(pos, conn):
    """Gradient Grams G[i][j] and the mass Gram (elements, nodes, nodes), and each element's
    centre node: quadratic Lagrange elements, 3 Gauss points per axis (the literals of
    the framework's reference)."""
    dim = pos.shape[1]
    x = pos[conn]
    lo, hi = x.min(1, keepdims=True), x.max(1, keepdims=True)
    loc = np.rint(2 * (x - lo) / (hi - lo)).astype(int)             # 0, 1, 2 per axis
    assert (loc == loc[:1]).all()
    loc = loc[0]
    g = np.array([-0.774596669241483, 0.0, 0.774596669241483])
    w = np.array([5.0, 8.0, 5.0]) / 9 if dim == 2 else np.array([0.555555555555556, 0.888888888888889,
                                                                0.555555555555556])
    one = np.array([[g * (g - 1) / 2, 1 - g * g, g * (g + 1) / 2], [g - 0.5, -2 * g, g + 0.5]])
    q = np.stack(np.meshgrid(*[np.arange(3)] * dim, indexing='ij'), -1).reshape(-1, dim)
    wq = w[q].prod(1)
    N = np.ones((len(q), len(loc)))
    D = np.ones((dim, len(q), len(loc)))
    for ax in range(dim):
        N *= one[0][loc[:, ax]][:, q[:, ax]].T
        for r in range(dim):
            D[r] *= one[int(r == ax)][loc[:, ax]][:, q[:, ax]].T
    J = np.einsum('rqa,eac->eqrc', D, x)
    wd = wq * np.abs(np.linalg.det(J))
    dN = np.einsum('eqir,rqa->eqia', np.linalg.inv(J), D)
    G = [[np.einsum('eq,eqa,eqb->eab', wd, dN[:, :, i], dN[:, :, j], optimize=True) for j in range(dim)]
         for i in range(dim)]
    return G, np.einsum('eq,qa,qb->eab', wd, N, N, optimize=True), int(np.flatnonzero((loc == 1).all(1))[0])


def _system(case, omega_top, loss):
    """COO entries (rows, cols, K, M, D values) of the unfolded system."""
    hexa = not hasattr(case, 'mesh')
    pos = np.asarray(case.pos_m if hexa else case.mesh.pos_m, float)
    conn = np.asarray(case.hexas if hexa else case.mesh.quads)
    tag = np.asarray(case.cell.hex_tag if hexa else case.mesh.elem_tag)
    dim, nn, ne = pos.shape[1], pos.shape[0], conn.shape[0]
    nd = 3 if hexa or case.mode_extension else 2
    mats = case.materials if hexa or case.mode_extension else [mt.lift_plane_strain(m) for m in case.materials]
    scale = SCALE_HEX if hexa else SCALE_Q9
    a = np.ones((3, ne), complex)
    G, GM, centre = _grams(pos, conn)
    xc = pos[conn[:, centre]]
    for reg in case.pml:
        sel = tag == reg.tag
        for ax, letter in enumerate('xyz'[:dim]):
            if letter in reg.kind:
                inner, outer = ((reg.xa, reg.xp), (reg.ya, reg.yp), (reg.za, reg.zp))[ax]
                r = (xc[sel, ax] - outer) ** 2 / (inner - outer) ** 2
                r = r if hexa else np.clip(r, 0.0, 1.0)
                a[ax, sel] = 1.0 + reg.dmax * (1.0 - r) ** reg.n / (1j * omega_top)
    vol = a.prod(0)
    idx = np.asarray(case.mat_idx)
    C, E, P = (np.stack([np.asarray(getattr(m, k), complex) for m in mats])[idx] for k in ('C', 'e', 'eps'))
    rho = np.array([m.rho for m in mats])[idx]
    strain = [s for s in (_STRAIN_HEX if hexa else _STRAIN_Q9) if s[0] < nd]
    dof = [3 * conn + c if hexa else c * nn + conn for c in range(nd)] + [nd * nn + conn]
    damp = np.where(idx == 0, loss.beta_dk, 0.0)
    rows, cols, vk, vm, vd = [], [], [], [], []

    def put(i, j, k, m=0.0, d=0.0):
        shape = (ne,) + GM.shape[1:]
        rows.append(np.broadcast_to(dof[i][:, :, None], shape).ravel())
        cols.append(np.broadcast_to(dof[j][:, None, :], shape).ravel())
        for out, v in ((vk, k), (vm, m), (vd, d)):
            out.append(np.broadcast_to(np.asarray(v, complex), shape).ravel())

    for c1 in range(nd):
        uf = 0.0
        for c2 in range(nd):
            k = 0.0
            for (ca, s, i, si, _) in strain:
                for (cb, t, j, _, sj) in strain:
                    if ca == c1 and cb == c2:
                        k = k + (C[:, s, t] * vol / (a[si] * a[sj]))[:, None, None] * G[i][j]
            put(c1, c2, scale * k, scale * (rho * vol)[:, None, None] * GM if c1 == c2 else 0.0,
                scale * damp[:, None, None] * k)
        for (ca, s, i, si, _) in strain:
            if ca == c1:
                for j in range(dim):
                    uf = uf + (E[:, j, s] * vol / (a[si] * a[j]))[:, None, None] * G[i][j]
        put(c1, nd, uf)
        put(nd, c1, scale * np.transpose(np.conj(uf) if hexa else uf, (0, 2, 1)))
    put(nd, nd, -sum((P[:, i, j] * vol / (a[i] * a[j]))[:, None, None] * G[i][j] for i in range(dim) for j in range(dim)))
    depth = np.concatenate([np.repeat(pos[:, -1], 3), pos[:, -1]]) if hexa else np.tile(pos[:, -1], nd + 1)
    return [np.concatenate(v) for v in (rows, cols, vk, vm, vd)] + [depth]


class _Exact:
    """The folded system in blocks of element layers, on the GPU."""

    def __init__(self, case, omega_top, loss):
        rows, cols, vk, vm, vd, depth = _system(case, omega_top, loss)
        fix, plus, minus, groups = case.bc[:4]
        ndof = depth.size
        rep = np.arange(ndof)
        for g in groups:
            for s in np.asarray(g).ravel()[1:]:
                rep[s] = np.asarray(g).ravel()[0]
        while (rep[rep] != rep).any():
            rep = rep[rep]
        free = rep == np.arange(ndof)
        free[np.concatenate([np.asarray(v).ravel() for v in (fix, plus, minus)])] = False
        level = np.unique(np.rint(depth * 1e13).astype(np.int64), return_inverse=True)[1]
        act = np.flatnonzero(free)
        act = act[np.argsort(level[act] // 2, kind='stable')]
        self.pos = np.full(ndof, -1)
        self.pos[act] = np.arange(act.size)
        self.rep, self.plus, self.minus, self.n = rep, np.asarray(plus), np.asarray(minus), act.size
        blk = level[act] // 2
        self.ptr = np.searchsorted(blk, np.arange(blk.max() + 2))
        self.dev = 'cuda' if torch.cuda.is_available() else 'cpu'
        s = np.zeros(ndof, bool)
        s[self.plus] = True
        t = lambda v: torch.as_tensor(v, device=self.dev)           # noqa: E731
        pr, pc = self.pos[rep[rows]], self.pos[rep[cols]]
        self.full = [t(v) for v in (rows, cols, vk)]
        on = (pr >= 0) & (pc >= 0)
        br, bc = blk[pr[on]], blk[pc[on]]
        assert (np.abs(br - bc) <= 1).all()
        self.r, self.c = t(pr[on]), t(pc[on])
        self.k, self.m, self.d = (t(v[on]) for v in (vk, vm, vd))
        self.part = {o: [np.flatnonzero((br == b) & (bc == b + o)) for b in range(blk.max() + 1)] for o in (-1, 0, 1)}
        self.part = {o: [t(v) for v in p] for o, p in self.part.items()}
        drive = s[rep[cols]] & (pr >= 0)          # columns of the + electrode
        self.dr = t(pr[drive])
        self.dk, self.dm, self.dd = (t(v[drive]) for v in (vk, vm, vd))
        self.spl = t(s)

    def values(self, w, k, m, d):
        w = w[:, None]
        return k[None] - w * w * m[None] + 1j * w * d[None]

    def block(self, a, o, b):
        p = self.part[o][b]
        r0, r1 = int(self.ptr[b]), int(self.ptr[b + 1])
        c0, c1 = int(self.ptr[b + o]), int(self.ptr[b + o + 1])
        out = torch.zeros((a.shape[0], (r1 - r0) * (c1 - c0)), dtype=a.dtype, device=self.dev)
        out.index_add_(1, (self.r[p] - r0) * (c1 - c0) + self.c[p] - c0, a[:, p])
        return out.view(-1, r1 - r0, c1 - c0)

    def solve(self, omega):
        """x (points, n) with the driven electrode at 1 V."""
        w = torch.as_tensor(omega, dtype=torch.float64, device=self.dev)
        a = self.values(w, self.k, self.m, self.d)
        rhs = torch.zeros((w.numel(), self.n), dtype=torch.complex128, device=self.dev)
        rhs.index_add_(1, self.dr, -self.values(w, self.dk, self.dm, self.dd))
        nb = len(self.ptr) - 1
        lu, up = [], []
        for b in range(nb):
            d = self.block(a, 0, b)
            if b:
                d = d - self.block(a, -1, b) @ up[-1]
            lu.append(torch.linalg.lu_factor(d))
            if b + 1 < nb:
                up.append(torch.linalg.lu_solve(*lu[-1], self.block(a, 1, b)))
        low = [None] + [self.block(a, -1, b) for b in range(1, nb)]

        def back(v):
            y = []
            for b in range(nb):
                t = v[:, self.ptr[b]:self.ptr[b + 1], None]
                t = t - low[b] @ y[-1] if b else t
                y.append(torch.linalg.lu_solve(*lu[b], t))
            for b in range(nb - 2, -1, -1):
                y[b] = y[b] - up[b] @ y[b + 1]
            return torch.cat(y, 1)[..., 0]

        x = back(rhs)
        for _ in range(3):
            ax = torch.zeros_like(rhs).index_add_(1, self.r, a * x[:, self.c])
            x = x + back(rhs - ax)
        return x

    def charge(self, x):
        """(Q, disp): every DOF's value, and the charge of the unfolded stiffness rows."""
        pos = torch.as_tensor(self.pos[self.rep], device=self.dev)
        disp = torch.where(pos >= 0, x[:, pos.clamp(min=0)], torch.zeros((), dtype=x.dtype, device=self.dev))
        disp[:, torch.as_tensor(self.plus, device=self.dev)] = 1.0
        disp[:, torch.as_tensor(self.minus, device=self.dev)] = 0.0
        r, c, k = self.full
        on = self.spl[r]
        return (k[on][None] * disp[:, c[on]]).sum(1), disp


def exact(c, seed):
    n, cross = _sizes(c)
    points = c['points'] * (2 if c['call'] == 'zoom' else 1)
    # elimination of `n / (2 cross)` blocks of 2 cross unknowns per point: the large
    # cells would take minutes
    if points * n * (2.0 * cross) ** 2 * 16 > 4e13:
        return None
    case, loss, _ = inputs(c, seed)
    step = max(1, int(12e9 / (16.0 * 8 * n * 2 * cross)))

    def charges(freqs, top):
        ex = _Exact(case, top, loss)
        out = []
        for i in range(0, freqs.size, step):
            Q, disp = ex.charge(ex.solve(2 * np.pi * freqs[i:i + step]))
            out.append(Q.cpu().numpy())
        return np.concatenate(out), disp

    Q, disp = charges(case.freqs, case.omega_top)
    if c['call'] == 'field':
        return dict(disp=disp[0].cpu().numpy(), Q=Q)
    if c['call'] == 'zoom':
        z = _zoom(case)
        return dict(Q=Q, Q_zoom=charges(z, 2 * np.pi * z[-1])[0])
    if c['call'] == 'gradient':
        return dict(Q=Q, dQ=None)
    return dict(Q=Q)
