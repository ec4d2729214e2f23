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
