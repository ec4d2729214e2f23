"""What the performance of the powder engine is measured on.

A case is one call (or the short run of calls) that a user's program repeats:
a powder FID of an uploaded spin system, an upload followed by a powder, a
graph of many systems' powders, a magic-angle-spinning powder, a pulse
sequence, or one gradient evaluation and one prediction of the orientation
surrogate.  Systems, grids and step counts are those of
spinach_gb300/workloads.py and bench.py; a seed draws another molecule of the
same kind.  FP32 runs carry single precision in the double arrays the engine
returns, so their results are handed on as single-precision values.
"""
import math

import numpy as np
import torch

from spinach_gb300 import batched, engine, singlerot, spin_system, workloads

DEVICE = 0


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # crystal.m: one orientation of a three-spin system, the smallest call, all latency
        {'name': 'crystal', 'kind': 'powder', 'system': 'nmr', 'spins': 3, 'relax': False, 'orient': 1,
         'steps': 1024, 'fp64': False},
        # a quick static powder of a small molecule (13C-1H-1H, dim 64), default precision
        {'name': 'small', 'kind': 'powder', 'system': 'nmr', 'spins': 3, 'relax': False, 'orient': 200,
         'steps': 1024, 'fp64': False},
        # the 2H powder pattern (quadratic coupling, dim 144) in double precision, every orientation kept
        {'name': 'deuterium64', 'kind': 'powder', 'system': 'deuterium', 'orient': 400, 'steps': 1024, 'fp64': True,
         'each': True},
        # the benchmark's headline: a seven-spin system (dim 1156) uploaded and its 1000-orientation powder run,
        # as a fit does at every parameter step
        {'name': 'upload_run', 'kind': 'powder', 'system': 'nmr', 'spins': 7, 'relax': True, 'orient': 1000,
         'steps': 2048, 'fp64': False, 'upload': True},
        # the same powder in double precision
        {'name': 'seven64', 'kind': 'powder', 'system': 'nmr', 'spins': 7, 'relax': True, 'orient': 1000,
         'steps': 2048, 'fp64': True},
        # an X-band radical (electron, 14N, ten 1H; dim 2736, complex values), 4000 orientations
        {'name': 'radical', 'kind': 'powder', 'system': 'radical', 'protons': 10, 'orient': 4000, 'steps': 4096,
         'fp64': False},
        # the largest full basis (six spins, dim 4096), grid and output resident on the device
        {'name': 'six_device', 'kind': 'powder', 'system': 'nmr', 'spins': 6, 'relax': True, 'orient': 400,
         'steps': 1024, 'fp64': False, 'device': True},
        # many molecules of uneven size as one tuned CUDA graph
        {'name': 'batch', 'kind': 'batch', 'spins': '3 7 4 5 8 3 6 5', 'orient': 400, 'steps': 1024, 'fp64': False},
        # magic-angle spinning (Fokker-Planck, 17 rotor points, dim 1088)
        {'name': 'mas', 'kind': 'mas', 'rank': 8, 'rate': 10000.0, 'orient': 200, 'steps': 1024, 'fp64': False},
        # a CPMG echo train on the seven-spin system
        {'name': 'cpmg', 'kind': 'cpmg', 'spins': 7, 'orient': 1000, 'points': 128, 'loops': 8, 'fp64': False},
        # a two-pulse echo decay of the radical
        {'name': 'eseem', 'kind': 'eseem', 'protons': 10, 'orient': 2000, 'points': 256, 'fp64': False},
        # the orientation surrogate: gradients over a coarse grid (a training step) and a dense prediction
        {'name': 'surrogate', 'kind': 'surrogate', 'train': 2000, 'dense': 20000, 'hidden': 256, 'layers': 4,
         'lmax': 12, 'out': 128},
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: small to large molecules, one to
    thousands of orientations, short and long acquisitions, odd counts, both
    precisions, one or two channels, with and without relaxation."""
    kind = rng.choice(['powder'] * 6 + ['batch', 'mas', 'cpmg', 'eseem', 'surrogate'])
    fp64 = rng.random() < 0.3
    if kind == 'powder':
        system = rng.choice(['nmr'] * 4 + ['radical', 'deuterium'])
        case = {'kind': 'powder', 'system': system, 'steps': _between(rng, 64, 2048), 'fp64': fp64,
                'upload': rng.random() < 0.25}
        if system == 'nmr':
            case['spins'] = rng.randint(3, 8)
            case['relax'] = rng.random() < 0.6
            case['channels'] = 1 if case['upload'] else rng.choice([1, 1, 2])
            top = {3: 1500, 4: 1200, 5: 600, 6: 300, 7: 1000, 8: 800}[case['spins']]
            case['orient'] = _between(rng, 1, max(2, top // 12 if fp64 else top))
        elif system == 'radical':
            case['protons'] = rng.choice([1, 2, 3, 10])
            case['orient'] = _between(rng, 1, 400 if fp64 else 3000)
        else:
            case['orient'] = _between(rng, 1, 2000)
        case['each'] = case['orient'] <= 500 and rng.random() < 0.3
        case['device'] = not (case['upload'] or case['each']) and rng.random() < 0.3
        return case
    if kind == 'batch':
        spins = [rng.choice([3, 3, 4, 4, 5, 7]) for _ in range(rng.randint(2, 6))]
        return {'kind': 'batch', 'spins': ' '.join(map(str, spins)), 'orient': _between(rng, 20, 400),
                'steps': _between(rng, 128, 1024), 'fp64': False}
    if kind == 'mas':
        return {'kind': 'mas', 'rank': rng.randint(3, 9), 'rate': rng.uniform(5e3, 2e4),
                'orient': _between(rng, 5, 60 if fp64 else 200), 'steps': _between(rng, 128, 1024), 'fp64': fp64}
    if kind == 'cpmg':
        return {'kind': 'cpmg', 'spins': rng.choice([3, 4, 5, 7]), 'orient': _between(rng, 10, 80 if fp64 else 800),
                'points': _between(rng, 16, 160), 'loops': rng.randint(1, 8), 'fp64': fp64}
    if kind == 'eseem':
        return {'kind': 'eseem', 'protons': rng.choice([1, 2, 3, 10]), 'orient': _between(rng, 10, 200 if fp64 else 1500),
                'points': _between(rng, 16, 256), 'fp64': fp64}
    return {'kind': 'surrogate', 'train': _between(rng, 100, 4000), 'dense': _between(rng, 500, 30000),
            'hidden': rng.choice([64, 96, 128, 256]), 'layers': rng.randint(2, 4), 'lmax': rng.randint(4, 12),
            'out': 2 * rng.randint(8, 64)}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _molecule(case, seed):
    """The workload of a case: a molecule of the stated kind, drawn by the seed."""
    system = case.get('system', 'nmr' if 'spins' in case else 'radical')
    if case['kind'] == 'mas':
        return workloads.nmr_molecule('mas', 3, seed, 'none', 0, 10e-6, case['steps'], case['orient'], False)
    if system == 'deuterium':
        return workloads.deuterium(seed)
    if system == 'radical':
        return workloads.c4(seed) if case['protons'] == 10 else workloads.c4_small(seed, case['protons'])
    spins = case['spins']
    full = 4 ** spins <= 4096
    dt = 5e-6 if spins == 7 else 10e-6
    return workloads.nmr_molecule('nmr', spins, seed, 'none' if full else 'IK-0', 0 if full else 3, dt,
                                  case.get('steps', 0), case['orient'], case.get('relax', True))


def _inputs(case, seed):
    """Matrices, states, pulse, grid and time step of one run."""
    w = _molecule(case, seed)
    L = workloads.build(w)
    x = {'I': L.I, 'terms': L.terms, 'R': L.R, 'rho0': L.rho0, 'coil': [L.coil], 'dt': w.dt, 'pulse': None,
         'grid': [np.ascontiguousarray(a) for a in workloads.zcwn_grid(case['orient'])]}
    if case['kind'] == 'mas':
        x['I'], x['terms'], x['R'], x['rho0'], coil = singlerot.fokker_planck(
            L.I, L.terms, L.R, L.rho0, L.coil, case['rank'], case['rate'], (1.0, 1.0, 1.0))
        x['coil'] = [coil]
    if case.get('channels', 1) > 1 or case['kind'] in ('cpmg', 'eseem'):
        ss = workloads.spin_system_of(w)
        fac = spin_system.factory_for(ss, spin_system.build_basis(ss, w.approximation, w.level))
        if case['kind'] in ('cpmg', 'eseem'):
            spin = '13C' if case['kind'] == 'cpmg' else 'E'
            x['rho0'] = fac.state('Lz', spin)
            x['pulse'] = sum(fac.operator([('Ly', i)]) for i, iso in enumerate(w.isotopes) if iso == spin)
            if case['kind'] == 'eseem':
                x['dt'] = 8e-9                      # a point of the echo decay; each half takes dt / 2
        else:
            x['coil'] = [fac.state('L+', '13C'), fac.state('Lx', '13C')]
    return x


def prepare(case, seed):
    dev = torch.device('cuda', DEVICE)
    precision = engine.FP64 if case.get('fp64') else engine.FP32
    if case['kind'] == 'surrogate':
        net = engine.Surrogate(DEVICE, lmax=case['lmax'], hidden=case['hidden'], layers=case['layers'],
                               n_out=case['out'], seed=seed)
        b, g, t, db, dg, params = _surrogate_inputs(case, seed, net.n_params)
        net.set_params(params)
        put = lambda a: torch.from_numpy(a).to(dev)
        return {'case': case, 'net': net, 'beta': put(b), 'gamma': put(g), 'targets': put(t), 'dense_beta': put(db),
                'dense_gamma': put(dg), 'out': torch.empty(case['dense'], case['out'], device=dev)}
    if case['kind'] == 'batch':
        ws = [_molecule({**case, 'kind': 'powder', 'spins': int(s)}, 100 * seed + i)
              for i, s in enumerate(case['spins'].split())]
        for w in ws:
            w.dt = 10e-6
        bp = batched.prepare(ws, n_orient=case['orient'], nsteps=case['steps'], device=DEVICE, precision=precision)
        return {'case': case, 'powders': bp, 'graph': batched.capture(bp, precision=precision)}
    x = _inputs(case, seed)
    eng = engine.Engine(DEVICE)
    state = {'case': case, 'engine': eng, 'precision': precision, **x}
    if case.get('upload'):
        state['host'] = engine.host_system(x['I'], x['terms'], x['R'], x['rho0'], x['coil'][0])
    else:
        eng.upload(x['I'], x['terms'], x['R'], x['rho0'], x['coil'][0])
        if len(x['coil']) > 1:
            eng.upload_coils(x['coil'])
    if case.get('device'):
        state['d_grid'] = torch.tensor(np.stack(x['grid']), device=dev)
        state['d_fid'] = torch.zeros(len(x['coil']) * (case['steps'] + 1), 2, dtype=torch.float64, device=dev)
    return state


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(state):
    case = state['case']
    if case['kind'] == 'surrogate':
        net = state['net']
        loss, grad = net.gradients(case['train'], state['beta'].data_ptr(), state['gamma'].data_ptr(),
                                   state['targets'].data_ptr())
        net.predict(case['dense'], state['dense_beta'].data_ptr(), state['dense_gamma'].data_ptr(),
                    state['out'].data_ptr())
        return {'loss': np.float32(loss), 'gradients': grad, 'prediction': state['out']}
    if case['kind'] == 'batch':
        state['graph'].launch()
        state['graph'].synchronize()
        return [f if case['fp64'] else f.float() for f in state['powders'].fids]
    eng, precision, grid = state['engine'], state['precision'], state['grid']
    if case.get('upload'):
        eng.upload_host(state['host'])
    if case.get('device'):
        d = state['d_grid']
        eng.run_device(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), d[3].data_ptr(), case['orient'],
                       state['dt'], case['steps'], state['d_fid'].data_ptr(), precision=precision)
        eng.synchronize()
        return state['d_fid'] if case['fp64'] else state['d_fid'].float()
    if case['kind'] == 'cpmg':
        res = eng.run_cpmg(*grid, state['dt'], case['points'], case['loops'], state['pulse'], precision=precision)
    elif case['kind'] == 'eseem':
        res = eng.run_eseem(*grid, state['dt'], case['points'], state['pulse'], precision=precision)
    else:
        res = eng.run(*grid, state['dt'], case['steps'], precision=precision,
                      per_orientation=bool(case.get('each')))
    out = [res.fid] if res.fids is None else [res.fid, res.fids]
    return out if case['fp64'] else [o.astype(np.complex64) for o in out]


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _coupled(system, case):
    """States that the detected coherence exchanges signal with."""
    if system == 'deuterium':
        return 8
    if system == 'radical':
        return 144 if case['protons'] == 10 else 9 * 2 ** case['protons']
    m = int(case['spins']) - 1
    return math.comb(2 * m, m) if 4 ** (m + 1) <= 4096 else 1 + m + 3 * m * (m - 1) // 2


def work(case):
    """Bytes: the grid in, the spectra out, and an uploaded system's entries.
    Flops: one complex multiply-add per coupled state, orientation and point."""
    if case['kind'] == 'surrogate':
        sizes = [(case['lmax'] + 1) ** 2] + [case['hidden']] * case['layers'] + [case['out']]
        mults = sum(a * b for a, b in zip(sizes, sizes[1:]))
        params = mults + sum(sizes[1:])
        return {'bytes': 4 * (2 * params + case['train'] * (4 + case['out']) + case['dense'] * (4 + case['out'])),
                'flops': 2.0 * mults * (3 * case['train'] + case['dense'])}
    no = case['orient']
    if case['kind'] == 'batch':
        spins = case['spins'].split()
        return {'bytes': len(spins) * (32 * no + 16 * (case['steps'] + 1)),
                'flops': 8.0 * no * (case['steps'] + 1) * sum(_coupled('nmr', {'spins': s}) for s in spins)}
    system = case.get('system', 'nmr' if 'spins' in case else 'radical')
    if case['kind'] == 'mas':
        points, n = case['steps'] + 1, (2 * case['rank'] + 1) * 6
    elif case['kind'] == 'cpmg':
        points, n = case['points'] * (1 + 2 * case['loops']), 2 * _coupled('nmr', case)
    elif case['kind'] == 'eseem':
        points, n = case['points'], 2 * _coupled('radical', case)
    else:
        points, n = case['steps'] + 1, _coupled(system, case) * case.get('channels', 1)
    out = 16 * points * case.get('channels', 1) * (1 + (no if case.get('each') else 0))
    matrices = 16 * 12 * 6800 if case.get('upload') else 0
    return {'bytes': 32 * no + out + matrices, 'flops': 8.0 * no * points * n}


# ---------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------
def _surrogate_inputs(case, seed, n_params):
    rng = np.random.default_rng(seed)
    angles = lambda n: (np.arccos(rng.uniform(-1, 1, n)), rng.uniform(0, 2 * np.pi, n))
    b, g = angles(case['train'])
    t = rng.normal(size=(case['train'], case['out'])).astype(np.float32)
    db, dg = angles(case['dense'])
    # trained networks have weights of the size 1/sqrt(fan-in) and small biases
    sizes = [(case['lmax'] + 1) ** 2] + [case['hidden']] * case['layers'] + [case['out']]
    parts = []
    for a, o in zip(sizes, sizes[1:]):
        parts += [rng.normal(0, 1.4 / math.sqrt(a), a * o), rng.normal(0, 0.05, o)]
    params = np.concatenate(parts).astype(np.float32)
    assert params.size == n_params
    return b, g, t, db, dg, params


def _features(beta, gamma, lmax):
    """Real spherical-harmonic features: per l Re Y_l0, then Re and Im Y_lm, m = 1..l."""
    x, s = torch.cos(beta), torch.sin(beta)
    P = {(0, 0): torch.full_like(x, math.sqrt(1 / (4 * math.pi)))}
    for m in range(1, lmax + 1):
        P[m, m] = -math.sqrt((2 * m + 1) / (2 * m)) * s * P[m - 1, m - 1]
    for m in range(lmax):
        P[m + 1, m] = math.sqrt(2 * m + 3) * x * P[m, m]
    for m in range(lmax + 1):
        for l in range(m + 2, lmax + 1):
            a = math.sqrt((4 * l * l - 1) / (l * l - m * m))
            b = math.sqrt(((l - 1) ** 2 - m * m) / (4 * (l - 1) ** 2 - 1))
            P[l, m] = a * (x * P[l - 1, m] - b * P[l - 2, m])
    cols = []
    for l in range(lmax + 1):
        cols.append(P[l, 0])
        for m in range(1, l + 1):
            cols += [P[l, m] * torch.cos(m * gamma), P[l, m] * torch.sin(m * gamma)]
    return torch.stack(cols, 1)


def _exact_surrogate(case, seed, dev):
    sizes = [(case['lmax'] + 1) ** 2] + [case['hidden']] * case['layers'] + [case['out']]
    n_params = sum(a * o + o for a, o in zip(sizes, sizes[1:]))
    b, g, t, db, dg, params = _surrogate_inputs(case, seed, n_params)
    put = lambda a: torch.from_numpy(a).to(dev).double()
    p = put(params).requires_grad_(True)

    def network(h):
        at = 0
        for i, (a, o) in enumerate(zip(sizes, sizes[1:])):
            weight, bias = p[at:at + a * o].reshape(o, a), p[at + a * o:at + a * o + o]
            at += a * o + o
            # products use weights rounded to 16 bits; the gradient passes straight through
            weight = weight + (weight.float().bfloat16().double() - weight).detach()
            h = h @ weight.T + bias
            if i + 2 < len(sizes):
                h = torch.nn.functional.gelu(h)
        return h

    loss = torch.mean((network(_features(put(b), put(g), case['lmax'])) - put(t)) ** 2)
    loss.backward()
    with torch.no_grad():
        dense = network(_features(put(db), put(dg), case['lmax']))
    return {'loss': loss.detach().cpu().numpy(), 'gradients': p.grad.cpu().numpy(), 'prediction': dense.cpu().numpy()}


def _wigner(rank, a, b, g):
    """D^rank for arrays of angles, rows and columns from +rank to -rank."""
    p = np.arange(rank, -rank - 1, -1)
    c, s = np.cos(b / 2), np.sin(b / 2)
    f = math.factorial
    d = np.zeros((b.size, p.size, p.size))
    for i, m1 in enumerate(p):
        for j, m2 in enumerate(p):
            pre = math.sqrt(f(rank + m1) * f(rank - m1) * f(rank + m2) * f(rank - m2))
            for k in range(max(0, m2 - m1), min(rank + m2, rank - m1) + 1):
                d[:, i, j] += pre * (-1.0) ** (m1 - m2 + k) / (f(rank + m2 - k) * f(k) * f(m1 - m2 + k) * f(rank - m1 - k)) \
                    * c ** (2 * rank + m2 - m1 - 2 * k) * s ** (m1 - m2 + 2 * k)
    return np.exp(-1j * p[None, :, None] * a[:, None, None]) * d * np.exp(-1j * p[None, None, :] * g[:, None, None])


def _components(n, matrices):
    """Labels of the sets of states that the matrices' entries connect."""
    top = max(abs(A).max() for A in matrices if A.nnz)
    r, c = [], []
    for A in matrices:
        A = A.tocoo()
        keep = np.abs(A.data) > 1e-14 * top
        r.append(A.row[keep])
        c.append(A.col[keep])
    r, c = np.concatenate(r), np.concatenate(c)
    lab = np.arange(n)
    while True:
        new = lab.copy()
        np.minimum.at(new, r, lab[c])
        np.minimum.at(new, c, lab[r])
        new = new[new]
        if np.array_equal(new, lab):
            return lab
        lab = new


class _Evolution:
    """Dense 64-bit evolution of the states that reach the coils, one block of
    connected states at a time, for a slice of the grid."""

    def __init__(self, x, grid, dev):
        self.dev = dev
        mats = [x['I']] + list(x['terms'].values())
        n = x['I'].shape[0]
        coils = np.array(x['coil'])
        joint = _components(n, mats + ([x['pulse']] if x['pulse'] is not None else []))
        live = np.isin(joint, joint[np.any(coils != 0, 0)]) & np.isin(joint, joint[x['rho0'] != 0])
        own = _components(n, mats)
        sets = [np.flatnonzero((own == v) & live) for v in np.unique(own[live])]
        sets.sort(key=len)
        self.order = np.concatenate(sets) if sets else np.zeros(0, int)
        put = lambda a: torch.from_numpy(np.ascontiguousarray(np.asarray(a, np.complex128))).to(dev)
        self.rho0, self.coils = put(x['rho0'][self.order]), put(coils[:, self.order])
        self.pulse = None if x['pulse'] is None else put(x['pulse'].tocsr()[self.order][:, self.order].toarray())
        d = {rank: _wigner(rank, *grid[:3]) for rank in {k[0] for k in x['terms']}}
        self.n, self.L, self.spans = grid[0].size, [], []
        at, i = 0, 0
        while i < len(sets):                                  # blocks of one size are stacked
            j = i
            while j < len(sets) and len(sets[j]) == len(sets[i]):
                j += 1
            group, size = sets[i:j], len(sets[i])
            stack = lambda A: np.stack([A[s][:, s].toarray() for s in group])
            H = put(stack(x['I'].tocsr()))[None].repeat(self.n, 1, 1, 1)
            for (rank, k, m), Q in x['terms'].items():
                H += put(d[rank][:, k, m])[:, None, None, None] * put(stack(Q.tocsr()))[None]
            H = 0.5 * (H + H.conj().transpose(-1, -2))
            if x['R'] is not None:
                H = H + 1j * put(stack(x['R'].tocsr()))[None]
            self.L.append(H)
            self.spans.append((at, len(group), size))
            at += len(group) * size
            i = j

    def step(self, dt):
        """exp(-i L dt) of every block; dt < 0 with adjoint gives the adjoint."""
        return [torch.linalg.matrix_exp(-1j * dt * H) for H in self.L]

    def apply(self, U, v):
        """U on states v (orientations x live states)."""
        out = torch.empty_like(v)
        for P, (at, cnt, size) in zip(U, self.spans):
            part = v[:, at:at + cnt * size].reshape(self.n, cnt, size, 1)
            out[:, at:at + cnt * size] = (P @ part).reshape(self.n, cnt * size)
        return out

    def turn(self, angle):
        return torch.linalg.matrix_exp(-1j * angle * self.pulse)

    def start(self, v):
        return v[None].repeat(self.n, 1)

    def record(self, U, v, steps):
        """Signals at 0..steps (orientations x channels x points) and the state at the last."""
        out = torch.empty(self.n, self.coils.shape[0], steps + 1, dtype=torch.complex128, device=self.dev)
        for k in range(steps + 1):
            out[:, :, k] = v @ self.coils.conj().T
            if k < steps:
                v = self.apply(U, v)
        return out, v


def exact(case, seed):
    dev = torch.device('cuda', DEVICE) if torch.cuda.is_available() else torch.device('cpu')
    if case['kind'] == 'surrogate':
        return _exact_surrogate(case, seed, dev)
    if case['kind'] == 'batch':
        out = []
        for i, s in enumerate(case['spins'].split()):
            one = {**case, 'kind': 'powder', 'spins': int(s)}
            x = _inputs(one, 100 * seed + i)
            x['dt'] = 10e-6
            out.append(_exact_fid(one, x, dev)[0].reshape(-1).view(np.float64))
        return out
    x = _inputs(case, seed)
    fid, each = _exact_fid(case, x, dev)
    if case.get('device'):
        return fid.reshape(-1).view(np.float64).reshape(-1, 2)
    squeeze = lambda a: a[..., 0, :] if len(x['coil']) == 1 else a
    return [squeeze(fid)] + ([squeeze(each)] if case.get('each') else [])


def _exact_fid(case, x, dev):
    no = x['grid'][0].size
    part = max(1, min(no, 1 << 8))
    each = []
    for o in range(0, no, part):
        ev = _Evolution(x, [a[o:o + part] for a in x['grid'][:3]], dev)
        if ev.order.size == 0:
            points = case.get('points', case.get('steps', 0) + 1) * (1 + 2 * case.get('loops', 0))
            each.append(torch.zeros(ev.n, len(x['coil']), points, dtype=torch.complex128, device=dev))
        elif case['kind'] == 'cpmg':
            U, half, full = ev.step(x['dt']), ev.turn(math.pi / 2), ev.turn(math.pi)
            sig, v = ev.record(U, ev.start(half @ ev.rho0), case['points'] - 1)
            got = [sig]
            for _ in range(case['loops']):
                sig, v = ev.record(U, v @ full.T, 2 * case['points'] - 1)
                got.append(sig)
            each.append(torch.cat(got, 2))
        elif case['kind'] == 'eseem':
            # point n: coil' U^n turn U^n rho, from the trajectories of rho and of the adjoint
            U, full = ev.step(x['dt'] / 2), ev.turn(math.pi)
            V = [P.conj().transpose(-1, -2) for P in U]
            u, v = ev.start(ev.turn(math.pi / 2) @ ev.rho0), ev.start(ev.coils[0])
            got = []
            for _ in range(case['points']):
                got.append((v.conj() * (u @ full.T)).sum(1))
                u, v = ev.apply(U, u), ev.apply(V, v)
            each.append(torch.stack(got, 1)[:, None, :])
        else:
            each.append(ev.record(ev.step(x['dt']), ev.start(ev.rho0), case['steps'])[0])
    each = torch.cat(each)
    weights = torch.from_numpy(x['grid'][3]).to(dev)
    fid = (weights[:, None, None] * each).sum(0)
    return fid.cpu().numpy(), each.cpu().numpy()
