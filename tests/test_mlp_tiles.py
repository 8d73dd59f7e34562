"""The planner kernels at the edges of their tiles: batches around one tile, around the sizes
where the tile changes, and inputs that are not 16-byte aligned, against the FP64 oracle."""
import numpy as np
import pytest

from oracle import mlp_oracle as M

SMS = 148  # the tile sizes change at multiples of the SM count


def _layers(p):
    out, at = [], 0
    for shape in ((M.IN, 64), (64,), (64, 64), (64,), (64, M.OUT), (M.OUT,)):
        n = int(np.prod(shape))
        out.append(p[at: at + n].reshape(shape))
        at += n
    return out


def _forward_bound(p, x):
    """Rounding bound of an fp32 forward pass with any summation order: every sum of n terms is
    within n * 2**-24 of its terms' magnitudes, and ReLU does not enlarge an error."""
    w1, b1, w2, b2, w3, b3 = (np.abs(a) for a in _layers(p))
    magnitude = ((np.abs(x) @ w1 + b1) @ w2 + b2) @ w3 + b3
    return (M.IN + 2 + 2 * (64 + 2)) * 2.0 ** -24 * magnitude


@pytest.mark.gpu
@pytest.mark.parametrize("batch", [1, 15, 16, 17, 63, 64, 65, 16 * 8 * SMS, 16 * 8 * SMS + 1, 64 * 8 * SMS + 65])
@pytest.mark.parametrize("shift", [0, 1])
def test_forward_tiles(batch, shift):
    import torch
    from mordred_b200 import _lib as L
    rng = np.random.default_rng(batch + shift)
    p = rng.normal(0, 0.2, M.NPARAMS).astype(np.float32)
    x = rng.normal(0, 1, (batch, M.IN)).astype(np.float32)
    dp = torch.from_numpy(p).cuda()
    dx = torch.empty(batch * M.IN + shift, dtype=torch.float32, device="cuda")
    dx[shift:] = torch.from_numpy(x).cuda().view(-1)
    dy = torch.full((batch * M.OUT + shift + 2,), 7.0, dtype=torch.float32, device="cuda")
    L.call("mb_mlp_forward", dp.data_ptr(), dx[shift:].data_ptr(), batch, dy[shift:].data_ptr(),
           torch.cuda.current_stream().cuda_stream)
    p64, x64 = p.astype(np.float64), x.astype(np.float64)
    ref, _ = M.forward(p64, x64)
    got = dy.cpu().numpy()
    assert (got[:shift] == 7.0).all() and (got[shift + batch * M.OUT:] == 7.0).all()  # nothing beyond the batch
    got = got[shift: shift + batch * M.OUT].reshape(batch, M.OUT)
    assert (np.abs(got - ref) <= _forward_bound(p64, x64)).all()


@pytest.mark.gpu
@pytest.mark.parametrize("batch", [1, 7, 8, 9, 8 * (SMS // 2), 8 * (SMS // 2) + 1, 32 * SMS + 33])
def test_backward_tiles(batch):
    import torch
    from mordred_b200 import _lib as L
    rng = np.random.default_rng(batch)
    p = rng.normal(0, 0.2, M.NPARAMS).astype(np.float32)
    x = rng.normal(0, 1, (batch, M.IN)).astype(np.float32)
    t = rng.normal(0, 1, (batch, M.OUT)).astype(np.float32)
    dp, dx, dt = (torch.from_numpy(a).cuda() for a in (p, x, t))
    g = torch.zeros(M.NPARAMS, dtype=torch.float32, device="cuda")
    loss = torch.zeros(1, dtype=torch.float32, device="cuda")
    L.call("mb_mlp_backward", dp.data_ptr(), dx.data_ptr(), dt.data_ptr(), batch, g.data_ptr(), loss.data_ptr(),
           torch.cuda.current_stream().cuda_stream)
    p64, x64, t64 = (a.astype(np.float64) for a in (p, x, t))
    ref = M.grad(p64, x64, t64)
    # the tolerances of the kernels' first test against the same oracle
    assert np.allclose(g.cpu().numpy(), ref, rtol=1e-3, atol=1e-5 * np.abs(ref).max())
    assert abs(loss.item() / batch - M.loss(p64, x64, t64)) <= 1e-4 * M.loss(p64, x64, t64) + 1e-6
