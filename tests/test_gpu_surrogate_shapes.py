"""GPU tests of the surrogate's kernels at the edges of their tiles, slabs and
vector loads: rows around multiples of 32 and 64, widths that are odd or below
a tile, gradients in one and in several launches, output that is not 8-byte
aligned.  Against the FP64 reference in oracle/surrogate_ref.py; tolerances as
in test_gpu_surrogate.py (FP32 products and sums: a few 1e-7 a layer)."""
import numpy as np
import pytest

from oracle import surrogate_ref as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n,lmax,hidden,layers,nout', [
    (1, 0, 1, 1, 1),
    (31, 1, 33, 2, 3),
    (64, 2, 64, 1, 64),
    (65, 5, 31, 3, 65),
    (255, 16, 130, 2, 129),       # 289 features; the largest row of sums without a split
    (257, 3, 100, 4, 17),         # two slabs of samples, the second with one row
    (20001, 4, 96, 2, 10),        # whole tiles, 32 slabs
    (4096, 4, 1024, 4, 6),        # weight gradients in more than one launch
])
def test_features_gradients_predictions(engine_lib, n, lmax, hidden, layers, nout):
    torch = pytest.importorskip('torch')
    if not torch.cuda.is_available():
        pytest.skip('no GPU')
    from spinach_gb300 import engine as E
    net = E.Surrogate(0, lmax=lmax, hidden=hidden, layers=layers, n_out=nout, seed=n)
    rng = np.random.default_rng(n)
    p = net.get_params()
    p = p + rng.normal(0, 0.05, p.size).astype(np.float32)
    net.set_params(p)
    b, g = np.arccos(rng.uniform(-1, 1, n)), rng.uniform(-7, 7, n)
    db, dg = torch.from_numpy(b).cuda(), torch.from_numpy(g).cuda()
    nfeat = (lmax + 1) ** 2
    X = S.sh_features(b, g, lmax)
    feat = torch.empty(n, nfeat, device='cuda', dtype=torch.float32)
    net.features(n, db.data_ptr(), dg.data_ptr(), feat.data_ptr())
    assert np.abs(feat.cpu().numpy() - X).max() <= 2e-6
    T = rng.normal(size=(n, nout)).astype(np.float32)
    dT = torch.empty(n * nout + 1, device='cuda', dtype=torch.float32)[1:]
    dT.copy_(torch.from_numpy(T).reshape(-1))
    loss, grad = net.gradients(n, db.data_ptr(), dg.data_ptr(), dT.data_ptr())
    shapes = S.layer_shapes(nfeat, hidden, layers, nout)
    rloss, rgrad = S.forward_backward(p.astype(np.float64), shapes, X, T.astype(np.float64))
    assert abs(loss - rloss) <= 1e-5 * rloss
    off = 0
    for o, i in shapes:
        for size in (o * i, o):
            blk = slice(off, off + size)
            assert np.linalg.norm(grad[blk] - rgrad[blk]) <= 1e-4 * np.linalg.norm(rgrad[blk]) + 1e-9
            off += size
    out = torch.full((n * nout + 3,), 7.0, device='cuda', dtype=torch.float32)
    net.predict(n, db.data_ptr(), dg.data_ptr(), out[1:].data_ptr())
    h = X
    pairs = S.unpack(p.astype(np.float64), shapes)
    for li, (W, bias) in enumerate(pairs):
        z = h @ S.bf16_round(W).T + bias
        h = S.gelu(z) if li + 1 < len(pairs) else z
    got = out.cpu().numpy()
    assert np.linalg.norm(got[1:-2].reshape(n, nout) - h) <= 1e-5 * np.linalg.norm(h)
    assert got[0] == 7.0 and np.all(got[-2:] == 7.0)
