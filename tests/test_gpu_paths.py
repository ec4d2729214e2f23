"""Which kernels a run takes, by its number of launches: three for one CTA per
orientation (dense matrices of few states), five for the series (bounds, tables,
propagation), more for the dense matrices of more states; each against dense
exponentials.  And programs that outgrow the coupled states' limits."""
import numpy as np
import pytest
import scipy.linalg as sl
import scipy.sparse as sp

from spinach_gb300 import engine as E
from oracle_cases import rel_err
from test_gpu_coupled import ANGLES, WEIGHTS, _reference, _system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('prec,tol', [(E.FP64, 1e-10), (E.FP32, 1e-5)])
@pytest.mark.parametrize('n,cplx,relax,dt,nsteps,path', [
    (1, False, True, 0.05, 45, 'one'), (16, True, False, 5.0, 300, 'one'), (16, False, True, 5.0, 2000, 'one'),
    (20, True, True, 0.05, 45, 'series'), (33, False, False, 0.05, 45, 'series'), (255, False, True, 0.05, 45, 'series'),
    (20, False, False, 5.0, 2000, 'matrices'), (40, True, False, 5.0, 2000, 'matrices'),
    (33, False, True, 5.0, 2000, 'matrices'), (65, False, False, 5.0, 2000, 'matrices')])
def test_kernels_by_size_and_length(gpu_engine, n, cplx, relax, dt, nsteps, path, prec, tol):
    H, Q, R, rho0, coil, block = _system(n, 7, cplx, relax, 1, 2, 1000 * n + nsteps)
    gpu_engine.upload(sp.csc_matrix(H), {(2, 2, 1): sp.csc_matrix(Q)}, sp.csc_matrix(R), rho0, coil)
    before = gpu_engine.stats()['kernel_launches']
    res = gpu_engine.run(*ANGLES, WEIGHTS, dt, nsteps, precision=prec, fp32_check=False)
    launches = res.stats['kernel_launches'] - before
    assert {3: 'one', 5: 'series'}.get(launches, 'matrices') == path, launches
    assert rel_err(res.fid, WEIGHTS @ _reference(H, Q, R, rho0, coil, block, dt, nsteps)) <= tol


@pytest.mark.parametrize('prec,tol', [(E.FP64, 1e-10), (E.FP32, 1e-5)])
@pytest.mark.parametrize('n,width,coupled', [(60, 60, True), (72, 70, False), (520, 2, False)])
def test_programs_beyond_the_coupled_limits_take_the_whole_system(gpu_engine, n, width, coupled, prec, tol):
    """A pulse operator that connects more than 64 states, and a set of more than 512
    rows; and one within the limits."""
    H, Q, R, rho0, coil, block = _system(n, 0, False, True, 0, 2, n)
    P = np.zeros((n, n))
    for at in range(0, n - width + 1, width):
        P[np.arange(at, at + width - 1), np.arange(at + 1, at + width)] = 0.5
    P = sp.csc_matrix(P + P.T)
    dt, steps = 0.2, (20, 9)
    gpu_engine.upload(sp.csc_matrix(H), {(2, 2, 1): sp.csc_matrix(Q)}, sp.csc_matrix(R), rho0, coil)
    res = gpu_engine.run_sequence(*ANGLES, WEIGHTS, [P], [('pulse', 0, 0.7), ('evolve', steps[0], dt), ('pulse', 0, 2.0),
                                                          ('evolve', steps[1], dt)], precision=prec)
    assert (res.stats['coupled_dim'] > 0) == coupled
    first, second = sl.expm(-0.7j * P.toarray()), sl.expm(-2j * P.toarray())
    ref = np.zeros(sum(steps) + 2, complex)
    for o in range(3):
        al, be, ga = (a[o] for a in ANGLES)
        A = H + np.sqrt(1.5) * np.sin(be) * np.cos(be) * np.exp(-1j * ga) * Q
        U = sl.expm(-1j * (0.5 * (A + A.conj().T) + 1j * R) * dt)
        v, f = first @ rho0, []
        for k in range(steps[0] + 1):
            f.append(np.vdot(coil, v))
            v = U @ v if k < steps[0] else v
        v = second @ v
        for _ in range(steps[1] + 1):
            f.append(np.vdot(coil, v))
            v = U @ v
        ref += WEIGHTS[o] * np.array(f)
    assert rel_err(res.fid, ref) <= tol


@pytest.mark.parametrize('prec,tol', [(E.FP64, 1e-10), (E.FP32, 1e-5)])
@pytest.mark.parametrize('n,cplx', [(31, False), (64, True), (256, False)])
def test_damped_systems_whole_and_on_the_coupled_states(gpu_engine, n, cplx, prec, tol):
    """Rates far below the spectral width: the whole-system kernel (whose norm check
    of the last series refuses rates near it) and the coupled states agree."""
    H, Q, R, rho0, coil, block = _system(n, 20, cplx, True, 1, 2, n)
    R = 0.02 * R
    dt, nsteps = 0.1, 600
    ref = WEIGHTS @ _reference(H, Q, R, rho0, coil, block, dt, nsteps)
    gpu_engine.upload(sp.csc_matrix(H), {(2, 2, 1): sp.csc_matrix(Q)}, sp.csc_matrix(R), rho0, coil)
    for options, states in (({}, n), ({'cluster': 1}, 0)):
        res = gpu_engine.run(*ANGLES, WEIGHTS, dt, nsteps, precision=prec, **options)
        assert res.stats['coupled_dim'] == states and rel_err(res.fid, ref) <= tol
