"""Calls at the limits of the coupled-state kernels, the dense matrices and the
autotuner: what decides which kernels run, what a failed run leaves behind, and
options that have to reach every path."""
import numpy as np
import pytest
import scipy.linalg as sl
import scipy.sparse as sp

from spinach_gb300 import engine as E
from oracle_cases import rel_err
from test_gpu_coupled import ANGLES, WEIGHTS, _reference, _system

pytestmark = pytest.mark.gpu


def _chain(n, seed, rate=0.0):
    """A chain of n states, one real coupling between neighbours, all damped at
    the same rate (negative: growing)."""
    rng = np.random.default_rng(seed)
    H = np.diag(rng.normal(size=n))
    for i in range(1, n):
        H[i, i - 1] = H[i - 1, i] = rng.normal()
    rho0, coil = np.zeros(n, complex), np.zeros(n, complex)
    rho0[0], coil[min(2, n - 1)] = 1.0, 1.0 + 0.5j
    return H, -rate * np.eye(n), rho0, coil


def _upload(eng, H, R, rho0, coil):
    eng.upload(sp.csc_matrix(H.astype(complex)), {}, sp.csc_matrix(R.astype(complex)), rho0, coil)


def _fid(H, R, rho0, coil, dt, nsteps):
    U, v, out = sl.expm(-1j * (H + 1j * R) * dt), rho0, []
    for _ in range(nsteps + 1):
        out.append(np.vdot(coil, v))
        v = U @ v
    return np.array(out)


def _device_grid():
    import torch
    g = torch.tensor(np.stack([*ANGLES, WEIGHTS]), device='cuda')
    torch.cuda.synchronize()
    return g, [g[i].data_ptr() for i in range(4)]


@pytest.mark.parametrize('nchan', [2, 8])
@pytest.mark.parametrize('prec,tol', [(E.FP64, 1e-10), (E.FP32, 1e-5)])
def test_autotune_of_several_channels(engine_lib, nchan, prec, tol):
    """The tuner's output holds every channel's points."""
    H, R, rho0, coil = _chain(24, 1, 0.02)
    coils = [np.roll(coil, k) for k in range(nchan)]
    eng = E.Engine(0)
    try:
        _upload(eng, H, R, rho0, coil)
        eng.upload_coils(coils)
        g, ptr = _device_grid()
        eng.autotune(*ptr[:3], 3, 0.2, 600, prec)
        res = eng.run(*ANGLES, WEIGHTS, 0.2, 600, precision=prec)
        for ch in range(nchan):
            assert rel_err(res.fid[ch], _fid(H, R, rho0, coils[ch], 0.2, 600)) <= tol
    finally:
        eng.close()


def _shift_operator(n):
    return sp.csc_matrix(np.diag(np.ones(n - 1), 1) + np.diag(np.ones(n - 1), -1))


def test_steps_too_long_for_the_coupled_kernels_take_the_whole_system(gpu_engine):
    """Series of several thousand terms outgrow the coupled kernels' shared memory
    before they outgrow the whole system's: FP64 detection rows of a complex coil,
    FP32 trajectories.  The phases reach 1e4, which leaves FP64 about 1e-12 of
    them and FP32 1e-3."""
    n = 4
    H, R, rho0, coil = _chain(n, 5)
    P = _shift_operator(n)
    H *= 4800.0 / np.abs(H).sum(1).max()
    _upload(gpu_engine, H, R, rho0, coil)
    res = gpu_engine.run_sequence(*ANGLES, WEIGHTS, [P], [('evolve', 2, 1.0), ('pulse', 0, 0.3), ('evolve', 1, 1.0)],
                                  precision=E.FP64)
    first = _fid(H, R, rho0, coil, 1.0, 2)
    after = sl.expm(-0.3j * P.toarray()) @ sl.expm(-2j * H) @ rho0
    ref = np.concatenate([first, _fid(H, R, after, coil, 1.0, 1)])
    assert rel_err(res.fid, ref) <= 1e-10 and res.stats['coupled_dim'] == 0
    H *= 5300.0 / 4800.0
    _upload(gpu_engine, H, R, rho0, coil)
    res = gpu_engine.run_eseem(*ANGLES, WEIGHTS, 2.0, 3, P, precision=E.FP32)
    U, Pi = sl.expm(-1j * H), sl.expm(-1j * np.pi * P.toarray())
    v = sl.expm(-0.5j * np.pi * P.toarray()) @ rho0
    ref = [np.vdot(coil, np.linalg.matrix_power(U, j) @ Pi @ np.linalg.matrix_power(U, j) @ v) for j in range(3)]
    assert rel_err(res.fid, ref) <= 1e-3 and res.stats['coupled_dim'] == 0


@pytest.mark.parametrize('prec,tol', [(E.FP64, 1e-10), (E.FP32, 1e-5)])
def test_batch_follows_later_uploads(engine_lib, prec, tol):
    """A captured batch runs what its handles hold at the launch: initial states in
    another block (of other size), other coils, another system."""
    import torch
    H, Q, R, rho0, coil, block = _system(20, 70, False, True, 1, 2, 11)
    rest = np.setdiff1d(np.arange(90), block)
    H2, Q2, R2, rho2, coil2, block2 = _system(45, 60, True, True, 2, 1, 12)
    dt, nsteps = 0.3, 80
    eng, other = E.Engine(0), E.Engine(0)
    batch = None
    up = lambda e, *s: e.upload(sp.csc_matrix(s[0]), {(2, 2, 1): sp.csc_matrix(s[1])}, sp.csc_matrix(s[2]), s[3], s[4])
    try:
        up(eng, H, Q, R, rho0, coil)
        up(other, H2, Q2, R2, rho2, coil2)
        _, ptr = _device_grid()
        outs = [torch.zeros(2 * (nsteps + 1), dtype=torch.float64, device='cuda') for _ in range(2)]
        torch.cuda.synchronize()
        batch = E.Batch([(e, 3, *ptr, dt, nsteps, o.data_ptr(), prec) for e, o in zip((eng, other), outs)])
        full = np.arange(90)

        def check(ref):
            for _ in range(2):
                batch.launch()
                batch.synchronize()
                assert rel_err(outs[0].cpu().numpy().view(complex), WEIGHTS @ ref) <= tol
                ref2 = _reference(H2, Q2, R2, rho2, coil2, block2, dt, nsteps)
                assert rel_err(outs[1].cpu().numpy().view(complex), WEIGHTS @ ref2) <= tol

        check(_reference(H, Q, R, rho0, coil, block, dt, nsteps))
        far = np.zeros(90, complex)
        far[rest[3]], far[rest[40]] = 2.0, -1.0
        states = np.zeros((3, 90), complex)
        states[:, rest[0]] = [1.0, -2.0, 0.5]
        eng.upload_coils([far])
        eng.set_initial_states(states)
        check(np.array([_reference(H, Q, R, states[o], far, full, dt, nsteps)[o] for o in range(3)]))
        states[:, block[2]] = [0.3, 0.2, 0.1]
        eng.upload_coils([far + coil])
        eng.set_initial_states(states)
        check(np.array([_reference(H, Q, R, states[o], far + coil, full, dt, nsteps)[o] for o in range(3)]))
        up(eng, H2, Q2, R2, rho2, coil2)
        check(_reference(H2, Q2, R2, rho2, coil2, block2, dt, nsteps))
        eng.set_initial_states(np.zeros((2, 105), complex))
        with pytest.raises(E.SpxError, match='per-orientation initial states'):
            batch.launch()
    finally:
        if batch is not None:
            batch.close()
        eng.close()
        other.close()


@pytest.mark.parametrize('n', [1, 6, 20, 70])
@pytest.mark.parametrize('prec,tol', [(E.FP64, 1e-10), (E.FP32, 1e-5)])
def test_growing_states_are_refused_at_every_size(gpu_engine, n, prec, tol):
    """A relaxation matrix of the wrong sign: refused when the state may grow
    fourfold, whichever kernels the size would take; run when it cannot."""
    P = _shift_operator(n) if n > 1 else sp.csc_matrix((1, 1), dtype=complex)
    for rate in (0.05, 0.3, 3.0):                       # over 45 steps of 0.7: factors of 5 and more
        _upload(gpu_engine, *_chain(n, n, -rate))
        with pytest.raises(E.SpxError, match='series did not converge'):
            gpu_engine.run(*ANGLES, WEIGHTS, 0.7, 45, precision=prec)
        with pytest.raises(E.SpxError, match='series did not converge'):
            gpu_engine.run_sequence(*ANGLES, WEIGHTS, [P], [('evolve', 45, 0.7)], precision=prec)
        with pytest.raises(E.SpxError, match='series did not converge'):
            gpu_engine.run_eseem(*ANGLES, WEIGHTS, 45 * 1.4, 46, P, precision=prec)
    mild = _chain(n, n, -0.03)                          # 45 steps: 2.6
    _upload(gpu_engine, *mild)
    res = gpu_engine.run(*ANGLES, WEIGHTS, 0.7, 45, precision=prec)
    assert rel_err(res.fid, _fid(*mild, 0.7, 45)) <= tol
    # growth where nothing is detected is refused too
    H, R, rho0, coil = _chain(n, n, 0.01)
    H2, R2, rho2, _ = _chain(9, 2, -0.3)
    H, R = sl.block_diag(H, H2), sl.block_diag(R, R2)
    _upload(gpu_engine, H, R, np.concatenate([rho0, rho2]), np.concatenate([coil, np.zeros(9)]))
    with pytest.raises(E.SpxError, match='series did not converge'):
        gpu_engine.run(*ANGLES, WEIGHTS, 0.7, 45, precision=prec)


def _outlier(half=30, out=11.0, coupling=1e-3):
    """Two clusters of states at +-10 and one at `out`: two Lanczos steps find the
    clusters and miss it, so lanczos_its=2 gives an interval about 10.7 (with its
    margins) instead of 11.  Scaled by it the outlier lies at cosh(0.19), and a
    series of argument x amplifies its rounding by exp(x sinh 0.19)."""
    H = np.diag(np.concatenate([np.full(half, 10.0), np.full(half, -10.0), [out]]))
    for i in range(1, len(H)):
        H[i, i - 1] = H[i - 1, i] = coupling
    n = len(H)
    rho0, coil = np.ones(n, complex), np.zeros(n, complex)
    coil[0] = coil[n - 1] = 1.0
    return H, np.zeros((n, n)), rho0, coil


@pytest.mark.parametrize('size', [1.0, 1e25, 1e37, 1e-20, 1e-36])
def test_fp32_states_of_extreme_size(gpu_engine, size):
    """The FP32 kernels' norm check holds for initial states of any size: large and
    small ones run, and a violated spectral bound is noticed and mended."""
    H, R, rho0, coil = _chain(20, 3)
    _upload(gpu_engine, H, R, rho0 * size, coil)
    res = gpu_engine.run(*ANGLES, WEIGHTS, 0.7, 45, precision=E.FP32, fp32_check=False)
    assert rel_err(res.fid / size, _fid(H, R, rho0, coil, 0.7, 45)) <= 1e-5
    H, R, rho0, coil = _outlier()
    _upload(gpu_engine, H, R, rho0 * size, coil)
    # one chunk of argument 175: exp(34) of 2^-24, far above the fourfold growth
    res = gpu_engine.run(*ANGLES, WEIGHTS, 0.28, 59, precision=E.FP32, lanczos_its=2, fp32_check=False)
    assert res.stats['retries'] == 1 and res.stats['coupled_dim'] == len(H)
    assert rel_err(res.fid / size, _fid(H, R, rho0, coil, 0.28, 59)) <= 1e-5


def _call(eng, name, program, opt, npts, fill=None):
    """A pulse program or an echo on the three orientations through the C entry
    points: status, powder points and every orientation's."""
    import ctypes as C
    n = eng.dim
    P = E._CscHolder(_shift_operator(n), n)
    fid, fids = np.full(2 * npts, fill if fill else 0.0), np.full(2 * npts * 3, fill if fill else 0.0)
    grid = [E._dptr(np.ascontiguousarray(a)) for a in (*ANGLES, WEIGHTS)]
    if name == 'sequence':
        ops = (E.SpxSeqOp * len(program))(*[E.SpxSeqOp(E.SEQ_EVOLVE, 0, 0.0, ns, dt, 1, 0) for ns, dt in program])
        st = eng.lib.spx_run_sequence(eng.h, 3, *grid, 1, (E.SpxCsc * 1)(P.struct), len(program), ops, C.byref(opt),
                                      E._dptr(fid), E._dptr(fids))
    elif name == 'eseem':
        ns, dt = program
        st = eng.lib.spx_run_eseem(eng.h, 3, *grid, 2 * dt, ns + 1, C.byref(P.struct), C.byref(opt), E._dptr(fid),
                                   E._dptr(fids))
    else:
        ns, dt = program
        st = eng.lib.spx_run_deer(eng.h, 3, *grid, dt, ns, C.byref(P.struct), C.byref(P.struct), C.byref(opt),
                                  E._dptr(fid), E._dptr(fids))
    return st, fid, fids


@pytest.mark.parametrize('prec', [E.FP64, E.FP32])
@pytest.mark.parametrize('name', ['sequence', 'eseem', 'deer'])
def test_lanczos_steps_reach_sequences_and_echoes(engine_lib, name, prec):
    """Two Lanczos steps give the outlier's system an interval that misses it (and
    a refusal: these entry points do not retry); 32 and 48 hold it."""
    import ctypes as C
    eng = E.Engine(0)
    try:
        _upload(eng, *_outlier(half=12))                    # pulses connect all 25 states
        program, npts = ([(79, 0.33)], 80) if name == 'sequence' else ((79, 0.33), 80)
        half = {}
        for its in (0, 2, 32, 48):
            st, fid, _ = _call(eng, name, program, E.SpxOptions(prec, 0, 0, 0, 0.0, 0.0, its, 0), npts)
            s = E.SpxStats()
            eng.lib.spx_get_stats(eng.h, C.byref(s))
            half[its] = (st, s.max_half_width, fid)
            assert s.coupled_dim == 25
        assert half[2][1] < 0.99 * half[32][1]              # 10.46 and 10.61 by the formula of the bounds
        if name == 'sequence':                              # chunks long enough to grow
            assert half[2][0] == 5
        for its in (0, 48):
            assert half[its][0] == 0 and abs(half[its][1] / half[32][1] - 1) <= 1e-3
        assert np.array_equal(half[0][2], half[32][2])
    finally:
        eng.close()


@pytest.mark.parametrize('prec', [E.FP64, E.FP32])
def test_a_failed_run_leaves_the_output_untouched(engine_lib, prec):
    import ctypes as C
    eng = E.Engine(0)
    try:
        # whole system (growing) and coupled states (a violated bound, not retried)
        _upload(eng, *_chain(20, 3, -3.0))
        fid, fids = np.full(2 * 46, 7.0), np.full(2 * 46 * 3, 7.0)
        grid = [E._dptr(np.ascontiguousarray(a)) for a in (*ANGLES, WEIGHTS)]
        opt = E.SpxOptions(prec, 0, 0, 0, 0.0, 0.0, 0, 0)
        assert eng.lib.spx_run_powder(eng.h, 3, *grid, 0.7, 45, C.byref(opt), E._dptr(fid), E._dptr(fids)) == 5
        assert np.all(fid == 7.0) and np.all(fids == 7.0)
        _upload(eng, *_outlier(half=12))
        opt.lanczos_its = 2
        st, fid, fids = _call(eng, 'sequence', [(2, 0.01), (79, 0.33)], opt, 83, fill=7.0)
        assert st == 5 and np.all(fid == 7.0) and np.all(fids == 7.0)
        # the same program with the default bounds: every point is written
        opt.lanczos_its = 0
        st, fid, fids = _call(eng, 'sequence', [(2, 0.01), (79, 0.33)], opt, 83, fill=7.0)
        each = fids.view(complex).reshape(3, 83)
        assert st == 0 and rel_err(WEIGHTS @ each, fid.view(complex)) <= 1e-6 and not np.any(fids == 7.0)
    finally:
        eng.close()


def test_outputs_larger_than_the_pinned_stage(gpu_engine):
    """FIDs of more than 8 MB come straight from the device."""
    H, R, rho0, coil = _chain(6, 4)
    _upload(gpu_engine, H, R, rho0, coil)
    nsteps = 600000                                         # 9.6 MB
    res = gpu_engine.run(*[a[:1] for a in ANGLES], WEIGHTS[:1], 0.01, nsteps, precision=E.FP64)
    e, V = np.linalg.eigh(H)
    a = (coil.conj() @ V) * (V.T @ rho0)
    at = np.array([0, 1, 7777, 299999, nsteps])
    ref = WEIGHTS[0] * np.array([np.sum(a * np.exp(-1j * e * 0.01 * k)) for k in at])
    # rounding of 2400 chunks, of which each adds a few 2^-53
    assert np.abs(res.fid[at] - ref).max() <= 1e-10 * np.abs(ref).max()


def test_echo_in_several_batches(engine_lib):
    """With little free memory the trajectories of an echo come in batches; points
    and statistics are those of one batch (whose ladder of half-widths may lie a
    step of 1/16 octave off)."""
    import torch
    n, no, npoints, dt = 100, 200, 2048, 0.01
    H, R, rho0, coil = _chain(n, 6, 0.01)
    P = sp.csc_matrix(sl.block_diag(*[[[0.0, 1.0], [1.0, 0.0]]] * (n // 2)))
    rng = np.random.default_rng(2)
    grid = (*rng.uniform(0, 3, (3, no)), rng.uniform(0.1, 1, no))
    Q = sp.csc_matrix(np.diag(rng.normal(size=n)).astype(complex))
    res = []
    for limited in (True, False):
        eng, hold = E.Engine(0), None
        try:
            eng.upload(sp.csc_matrix(H.astype(complex)), {(2, 2, 1): Q}, sp.csc_matrix(R.astype(complex)), rho0, coil)
            if limited:
                # 3 GB left, of which a quarter takes 120 orientations' trajectories
                torch.cuda.empty_cache()
                hold = torch.empty(torch.cuda.mem_get_info()[0] - (3 << 30), dtype=torch.uint8, device='cuda')
            res.append(eng.run_eseem(*grid, 2 * dt, npoints, P, precision=E.FP64, per_orientation=True))
        finally:
            eng.close()
            del hold
            torch.cuda.empty_cache()
    a, b = res
    for o in range(no):
        assert rel_err(a.fids[o], b.fids[o]) <= 1e-10, o
    assert rel_err(a.fid, b.fid) <= 1e-10
    assert a.stats['coupled_dim'] == n and a.stats['n_orientations'] == no
    assert a.stats['chunk_steps'] == b.stats['chunk_steps']
    for key in ('min_half_width', 'max_half_width', 'matvecs', 'max_terms'):
        assert abs(a.stats[key] / b.stats[key] - 1) <= 0.1, key


@pytest.mark.parametrize('prec', [E.FP64, E.FP32])
def test_chunk_length_and_flags_of_the_caller_on_a_tuned_handle(engine_lib, prec):
    """A chunk length takes the whole system, tuned or not; a bit of the flags that
    means nothing does not turn a forced shape into the engine's own."""
    import ctypes as C
    eng = E.Engine(0)
    try:
        H, R, rho0, coil = _chain(40, 5)
        _upload(eng, H, R, rho0, coil)
        ref = WEIGHTS.sum() * _fid(H, R, rho0, coil, 0.3, 100)
        _, ptr = _device_grid()
        for tuned in (False, True):
            if tuned:
                eng.autotune(*ptr[:3], 3, 0.3, 100, prec)
            res = eng.run(*ANGLES, WEIGHTS, 0.3, 100, precision=prec, chunk_steps=10)
            assert res.stats['coupled_dim'] == 0 and res.stats['chunk_steps'] == 10
            assert rel_err(res.fid, ref) <= (1e-10 if prec else 1e-5)
            res = eng.run(*ANGLES, WEIGHTS, 0.3, 100, precision=prec)
            assert res.stats['coupled_dim'] == 40
            fid = np.zeros(2 * 101)
            grid = [E._dptr(np.ascontiguousarray(a)) for a in (*ANGLES, WEIGHTS)]
            opt = E.SpxOptions(prec, 0, 96, 1, 0.0, 0.0, 0, 1 << 30)
            assert eng.lib.spx_run_powder(eng.h, 3, *grid, 0.3, 100, C.byref(opt), E._dptr(fid), None) == 0
            assert eng.stats()['coupled_dim'] == 0 and eng.stats()['threads'] == 96
    finally:
        eng.close()


def test_autotuned_options_handed_back_keep_the_coupled_states(engine_lib):
    """What spx_autotune returns may be passed to runs of the handle, or of another
    one with such a system; a shape changed by the caller is forced."""
    import torch
    H, R, rho0, coil = _chain(41, 5, 0.02)
    ref = WEIGHTS.sum() * _fid(H, R, rho0, coil, 0.3, 700)
    _, ptr = _device_grid()
    eng, other = E.Engine(0), E.Engine(0)
    try:
        for e in (eng, other):
            _upload(e, H, R, rho0, coil)
        for prec, tol in ((E.FP64, 1e-10), (E.FP32, 1e-5)):
            untuned = eng.run(*ANGLES, WEIGHTS, 0.3, 700, precision=prec).stats
            best = eng.autotune(*ptr[:3], 3, 0.3, 700, prec)
            for e in (eng, other):
                res = e.run(*ANGLES, WEIGHTS, 0.3, 700, precision=prec, **best)
                assert res.stats['coupled_dim'] == 41 and rel_err(res.fid, ref) <= tol
                assert res.stats['threads'] == untuned['threads'] and res.stats['cluster'] == untuned['cluster']
                forced = dict(best, threads=best['threads'] + 32)
                res = e.run(*ANGLES, WEIGHTS, 0.3, 700, precision=prec, **forced)
                assert res.stats['coupled_dim'] == 0 and rel_err(res.fid, ref) <= tol
    finally:
        eng.close()
        other.close()


def test_autotune_where_the_whole_system_takes_short_chunks(engine_lib):
    """2370 states beside 30 coupled ones: the whole system's default has a shorter
    series per chunk than the coupled states', and both have to be tunable."""
    n, m, dt, nsteps = 2400, 2370, 0.05, 600
    rng = np.random.default_rng(n)
    A = sp.diags([rng.normal(size=m)] + [rng.normal(size=m - k) for k in (1, 2, 3, 5, 8, 13, 21, 34)],
                 [0, 1, 2, 3, 5, 8, 13, 21, 34])
    A = A + sp.triu(A, 1).T
    B, R, rho0, coil = _chain(n - m, 7)
    H = sp.block_diag([A, B], format='csc').astype(complex)
    z = np.zeros(m)
    eng = E.Engine(0)
    try:
        eng.upload(H, {}, sp.csc_matrix((n, n), dtype=complex), np.concatenate([z, rho0]), np.concatenate([z, coil]))
        _, ptr = _device_grid()
        for prec, tol in ((E.FP64, 1e-10), (E.FP32, 1e-5)):
            best = eng.autotune(*ptr[:3], 3, dt, nsteps, prec)
            for options in ({}, best):
                res = eng.run(*ANGLES, WEIGHTS, dt, nsteps, precision=prec, **options)
                assert res.stats['coupled_dim'] == n - m
                assert rel_err(res.fid, WEIGHTS.sum() * _fid(B, R, rho0, coil, dt, nsteps)) <= tol
    finally:
        eng.close()


@pytest.mark.parametrize('n', [4, 70])                     # 70: the pulse connects more states than the coupled path takes
def test_pulses_of_extreme_angles(gpu_engine, n):
    """A tiny rotation moves its tiny part of the state (relative to it, FP64's
    digits), and an angle that overflows the operator is an error."""
    H, R, _, _ = _chain(n, 8)
    P = _shift_operator(n)
    rho0, coil = np.zeros(n, complex), np.zeros(n, complex)
    rho0[0], coil[1] = 1.0, 1.0
    H[0, 1] = H[1, 0] = 0.0                                 # detected states are reached by the pulse alone
    _upload(gpu_engine, H, R, rho0, coil)
    for angle in (1e-3, 1e-16, 1e-200):
        res = gpu_engine.run_sequence(*ANGLES, WEIGHTS, [P], [('pulse', 0, angle), ('evolve', 20, 0.1)], precision=E.FP64)
        v = -1j * np.eye(n)[1] * angle if angle < 1e-10 else sl.expm(-1j * angle * P.toarray()) @ rho0
        assert rel_err(res.fid / angle, _fid(H, R, v / angle, coil, 0.1, 20)) <= 1e-10
    for op, angle in ((1e10 * P, 1e300), (1e308 * P, 1.0)):
        with pytest.raises(E.SpxError, match='overflows'):
            gpu_engine.run_sequence(*ANGLES, WEIGHTS, [op], [('pulse', 0, angle), ('evolve', 2, 0.1)], precision=E.FP64)


def test_fp64_runs_take_their_bounds_in_fp64(gpu_engine):
    """The Gershgorin interval of the retry after a violated bound, and the Lanczos
    interval, of a spectrum whose centre is 500 times its width: FP32 sums would
    widen the discs by a part in 1e6 of the centre."""
    shift, dt, nsteps = 1.05e4, 0.38, 8300                  # more steps than the dense matrices take
    H, R, rho0, coil = _outlier()
    H = H + shift * np.eye(len(H))
    _upload(gpu_engine, H, R, rho0, coil)
    d = np.diag(H)
    rad = np.abs(H).sum(1) - np.abs(d)
    safe = 0.505 * ((d + rad).max() - (d - rad).min()) + 1e-9 * d.max()
    e, V = np.linalg.eigh(H - shift * np.eye(len(H)))
    a = (coil.conj() @ V) * (V.T @ rho0)
    at = np.array([0, 1, 255, 256, nsteps])
    ref = np.array([np.sum(a * np.exp(-1j * e * dt * k)) * np.exp(-1j * shift * dt * k) for k in at])
    for its, retries in ((2, 1), (0, 0)):
        res = gpu_engine.run(*ANGLES, WEIGHTS, dt, nsteps, precision=E.FP64, lanczos_its=its)
        assert res.stats['coupled_dim'] == len(H) and res.stats['retries'] == retries
        # phases of 3e7: 4e-9 of them are lost to their rounding
        assert np.abs(res.fid[at] - ref).max() <= 1e-6 * np.abs(ref).max()
        if retries:
            assert abs(res.stats['max_half_width'] / safe - 1) <= 1e-9
        else:
            assert res.stats['max_half_width'] <= safe * (1 + 1e-9)
