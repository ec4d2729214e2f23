"""Runs restricted to the states that couple to the coils (block.cuh): random
block-diagonal systems whose coupled block has sizes around the layouts' edges
(one warp, 256 and 512 rows, 513 falls back to the whole system), hub rows
wider than one lane's entries, real and complex values, relaxation, coils of
one to many entries, against dense exponentials in FP64; and the same systems
run whole (a forced launch shape)."""
import numpy as np
import pytest
import scipy.linalg as sl
import scipy.sparse as sp

from spinach_gb300 import engine as E
from oracle_cases import rel_err

pytestmark = pytest.mark.gpu

ANGLES = (np.array([0.3, 1.1, 0.0]), np.array([0.4, 1.3, 2.2]), np.array([0.9, 0.0, 5.1]))
WEIGHTS = np.array([0.5, 0.2, 0.3])


def _system(n, extra, cplx, relax, hubs, ncoil, seed):
    """A coupled block of n states in a system of n + extra; the rest couples
    among itself only.  Returns I, one rank-2 term, R, rho0, coil, block rows."""
    rng = np.random.default_rng(seed)
    N = n + extra
    perm = rng.permutation(N)

    def part(rows):
        A = np.zeros((N, N), complex)
        for i, r in enumerate(rows[1:], 1):                 # a chain keeps the block connected
            A[r, rows[i - 1]] = rng.normal() + (1j * rng.normal() if cplx else 0)
        for h in range(min(hubs, len(rows))):
            for c in rng.choice(len(rows), min(len(rows), 70), replace=False):
                if rows[c] != rows[h]:
                    A[rows[h], rows[c]] = 0.2 * rng.normal()
        return A + A.conj().T + np.diag(rng.normal(size=N))

    block, rest = perm[:n], perm[n:]
    H = np.zeros((N, N), complex)
    H[np.ix_(block, block)] = part(block)[np.ix_(block, block)]
    if extra:
        H[np.ix_(rest, rest)] = part(rest)[np.ix_(rest, rest)]
    Q = np.diag(rng.normal(size=N)).astype(complex)
    R = -np.diag(rng.uniform(0.0, 0.3, N)) if relax else np.zeros((N, N))
    rho0, coil = np.zeros(N, complex), np.zeros(N, complex)
    rho0[block[rng.choice(n, min(n, 3), replace=False)]] = rng.normal(size=min(n, 3))
    if extra:
        rho0[rest[0]] = 1.0                                # excited, but never detected
    at = block[rng.choice(n, min(n, ncoil), replace=False)]
    coil[at] = rng.normal(size=at.size) + (1j * rng.normal(size=at.size) if ncoil > 1 else 0)
    return H, Q, R, rho0, coil, block


def _reference(H, Q, R, rho0, coil, block, dt, nsteps):
    out = []
    b = np.ix_(block, block)
    for al, be, ga in zip(*ANGLES):
        d = np.sqrt(1.5) * np.sin(be) * np.cos(be) * np.exp(-1j * ga)     # D^2(0, +1)
        A = H[b] + d * Q[b]
        L = 0.5 * (A + A.conj().T) + 1j * R[b]
        U = sl.expm(-1j * L * dt)
        v, f = rho0[block], []
        for _ in range(nsteps + 1):
            f.append(np.vdot(coil[block], v))
            v = U @ v
        out.append(np.array(f))
    return np.array(out)


@pytest.mark.parametrize('n,extra,cplx,relax,hubs,ncoil', [
    (1, 0, False, True, 0, 1), (1, 5, False, False, 0, 1), (2, 40, True, False, 0, 2), (31, 9, False, True, 1, 1),
    (32, 0, True, True, 0, 3), (33, 100, False, False, 2, 40), (64, 64, False, True, 0, 1), (65, 0, True, False, 3, 1),
    (255, 30, False, True, 4, 17), (256, 0, True, True, 0, 1), (300, 20, False, False, 6, 5),
    (480, 10, False, True, 0, 1), (512, 1, False, False, 0, 1), (513, 0, False, False, 0, 1)])
def test_coupled_states_match_dense_exponentials(gpu_engine, n, extra, cplx, relax, hubs, ncoil):
    H, Q, R, rho0, coil, block = _system(n, extra, cplx, relax, hubs, ncoil, 17 * n + extra)
    dt, nsteps = 0.7, 45
    ref = _reference(H, Q, R, rho0, coil, block, dt, nsteps)
    gpu_engine.upload(sp.csc_matrix(H), {(2, 2, 1): sp.csc_matrix(Q)}, sp.csc_matrix(R), rho0, coil)
    for prec, tol in ((E.FP64, 1e-10), (E.FP32, 1e-5)):
        res = gpu_engine.run(*ANGLES, WEIGHTS, dt, nsteps, precision=prec, per_orientation=True)
        for o in range(3):
            assert rel_err(res.fids[o], ref[o]) <= tol, (prec, o)
        assert rel_err(res.fid, WEIGHTS @ ref) <= tol
        assert res.stats['coupled_dim'] in ((n,) if n <= 480 else (0, n))
    assert gpu_engine.run(*ANGLES, WEIGHTS, dt, nsteps, precision=E.FP64).stats['dim'] == n + extra
    # FP64 of three orientations takes the dense matrices; the entry point
    # without allocations takes the series
    import torch
    g = torch.tensor(np.stack([*ANGLES, WEIGHTS]), device='cuda')
    out = torch.zeros(2 * (nsteps + 1), dtype=torch.float64, device='cuda')
    torch.cuda.synchronize()
    gpu_engine.run_noalloc(*[g[i].data_ptr() for i in range(4)], 3, dt, nsteps, out.data_ptr(), precision=E.FP64)
    assert rel_err(out.cpu().numpy().view(complex), WEIGHTS @ ref) <= 1e-10
    if relax:           # rates near the spectral width: the whole-system kernel takes its last series for growth
        return
    whole = gpu_engine.run(*ANGLES, WEIGHTS, dt, nsteps, precision=E.FP64, cluster=1)
    assert whole.stats['coupled_dim'] == 0 and rel_err(whole.fid, WEIGHTS @ ref) <= 1e-10


@pytest.mark.parametrize('nsteps', [0, 1, 2, 254, 255, 256, 257, 600])
def test_step_counts_around_the_chunk(gpu_engine, nsteps):
    """The longest chunk is 256 steps."""
    H, Q, R, rho0, coil, block = _system(20, 12, False, True, 1, 1, 3)
    dt = 0.05
    ref = _reference(H, Q, R, rho0, coil, block, dt, nsteps)
    gpu_engine.upload(sp.csc_matrix(H), {(2, 2, 1): sp.csc_matrix(Q)}, sp.csc_matrix(R), rho0, coil)
    for prec, tol in ((E.FP64, 1e-10), (E.FP32, 1e-5)):
        res = gpu_engine.run(*ANGLES, WEIGHTS, dt, nsteps, precision=prec)
        assert rel_err(res.fid, WEIGHTS @ ref) <= tol, prec


def test_channels_states_and_undetected_coils(gpu_engine):
    """Two channels with coils in different blocks, one of them never reached
    by the initial state; then per-orientation initial states that reach it."""
    H, Q, R, rho0, coil, block = _system(12, 9, False, True, 0, 2, 5)
    N = 21
    rest = np.setdiff1d(np.arange(N), block)
    rho0[rest] = 0.0
    far = np.zeros(N, complex)
    far[rest[3]] = 2.0
    gpu_engine.upload(sp.csc_matrix(H), {(2, 2, 1): sp.csc_matrix(Q)}, sp.csc_matrix(R), rho0, coil)
    gpu_engine.upload_coils([coil, far])
    ref = _reference(H, Q, R, rho0, coil, block, 0.3, 60)
    res = gpu_engine.run(*ANGLES, WEIGHTS, 0.3, 60, precision=E.FP64)
    assert rel_err(res.fid[0], WEIGHTS @ ref) <= 1e-10 and np.all(res.fid[1] == 0)
    states = np.zeros((3, N), complex)
    states[:, rest[0]] = [1.0, -2.0, 0.5]
    gpu_engine.set_initial_states(states)
    full = np.arange(N)
    each = np.array([_reference(H, Q, R, states[o], far, full, 0.3, 60)[o] for o in range(3)])
    res = gpu_engine.run(*ANGLES, WEIGHTS, 0.3, 60, precision=E.FP64)
    assert rel_err(res.fid[1], WEIGHTS @ each) <= 1e-10
    gpu_engine.set_initial_states(None)
