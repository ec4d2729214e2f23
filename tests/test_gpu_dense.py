"""FP32 runs that the dense FP64 matrices serve, rounded at the end, and the FP32
series on the same systems (the entry point without allocations always takes the
series): step counts around powers of two and the longest chunk, one orientation
and more than are checked, one and two channels, real and complex values."""
import numpy as np
import pytest
import scipy.sparse as sp

from spinach_gb300 import engine as E
from oracle_cases import rel_err
from test_gpu_coupled import ANGLES, WEIGHTS, _reference, _system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n,cplx,relax,nsteps', [
    (1, False, True, 1), (2, True, False, 3), (6, False, False, 0), (6, False, True, 255), (20, True, True, 256),
    (20, False, True, 257), (33, False, False, 511), (40, True, False, 45)])
def test_fp32_by_dense_matrices_and_by_series(gpu_engine, n, cplx, relax, nsteps):
    import torch
    H, Q, R, rho0, coil, block = _system(n, 7, cplx, relax, 1, 2, 100 * n + nsteps)
    dt = 0.05
    ref = _reference(H, Q, R, rho0, coil, block, dt, nsteps)
    gpu_engine.upload(sp.csc_matrix(H), {(2, 2, 1): sp.csc_matrix(Q)}, sp.csc_matrix(R), rho0, coil)
    for count in (1, 3):
        grid, w = [a[:count] for a in ANGLES], WEIGHTS[:count]
        res = gpu_engine.run(*grid, w, dt, nsteps, precision=E.FP32, per_orientation=True)
        assert rel_err(res.fid, w @ ref[:count]) <= 1e-5
        assert res.stats['fp32_checked'] == min(2, count)
        # the stated error is that of the checked orientations against FP64
        at = [((2 * j + 1) * count) // (2 * min(2, count)) for j in range(min(2, count))]
        true = max(rel_err(res.fids[o], ref[o]) for o in at)
        assert abs(res.stats['fp32_rel_error'] - true) <= 1e-9
    g = torch.tensor(np.stack([*ANGLES, WEIGHTS]), device='cuda')
    out = torch.zeros(2 * (nsteps + 1), dtype=torch.float64, device='cuda')
    torch.cuda.synchronize()
    gpu_engine.run_noalloc(*[g[i].data_ptr() for i in range(4)], 3, dt, nsteps, out.data_ptr(), precision=E.FP32)
    assert rel_err(out.cpu().numpy().view(complex), WEIGHTS @ ref) <= 1e-5


@pytest.mark.parametrize('n,cplx', [(6, False), (20, True), (33, False), (64, True)])
def test_long_fp32_runs_are_rounded_once(gpu_engine, n, cplx):
    """Long steps make the series long: the dense matrices take the FP32 run, and
    nothing but the rounding of its points is left of the error, on two channels."""
    H, Q, R, rho0, coil, block = _system(n, 5, cplx, False, 1, 2, 11 * n)
    gpu_engine.upload(sp.csc_matrix(H), {(2, 2, 1): sp.csc_matrix(Q)}, sp.csc_matrix(R), rho0, coil)
    other = np.zeros_like(coil)
    other[block[:12]] = np.linspace(1.0, 2.0, min(n, 12))
    gpu_engine.upload_coils([coil, other])
    dt, nsteps = 5.0, 2000
    f32 = gpu_engine.run(*ANGLES, WEIGHTS, dt, nsteps, precision=E.FP32, per_orientation=True)
    assert f32.stats['fp32_checked'] == 2 and f32.stats['fp32_rel_error'] <= 2.0 ** -24
    for ch, c in enumerate((coil, other)):
        ref = _reference(H, Q, R, rho0, c, block, dt, nsteps)
        for o in range(3):
            assert rel_err(f32.fids[o][ch], ref[o]) <= 1e-7
