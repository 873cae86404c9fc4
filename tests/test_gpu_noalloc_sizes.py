"""gd2d_update_variables_noalloc over the sizes where its blocks can go wrong:
one cell, the edges of a 256-cell stretch, more stretches than blocks fit the
device at once, with velocities of every magnitude."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, 5000, 148 * 4 * 256 - 1, 148 * 4 * 256 + 1, 1_000_003])
def test_noalloc_update_sizes(pkg, n):
    import torch
    rng = np.random.default_rng(n)
    rho = 0.5 + rng.random(n)
    u = np.where(rng.random(n) < 0.2, 0.0, rng.choice([-1.0, 1.0], n) * 10.0 ** rng.uniform(-320, 1, n))
    v = 2.0 + rng.random(n)
    un = np.stack([rho, rho * u, rho * v, 2.5 + 0.5 * rho * (u * u + v * v)])
    uo = un * (1.0 + 1e-3 * rng.random((4, n)))
    d_un, d_uo = torch.from_numpy(un).cuda(), torch.from_numpy(uo.copy()).cuda()
    d_p, d_s = torch.zeros_like(d_un), torch.zeros(6, dtype=torch.float64, device="cuda")
    L = pkg._native.load()
    assert L.gd2d_update_variables_noalloc(d_un.data_ptr(), d_uo.data_ptr(), d_p.data_ptr(), n, 1.4, d_s.data_ptr(),
                                           torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    ux, uy = un[1] / un[0], un[2] / un[0]
    p = (1.4 - 1.0) * (un[3] - 0.5 * (un[1] * un[1] + un[2] * un[2]) / un[0])
    assert np.array_equal(d_p.cpu().numpy(), np.stack([un[0], ux, uy, p]))
    assert np.array_equal(d_uo.cpu().numpy(), un)
    st = d_s.cpu().numpy()
    # sums of n rounded squares in another order: within n ulp of each other
    assert np.allclose(st[:4], ((un - uo) ** 2).sum(axis=1), rtol=n * 2.3e-16 + 1e-15, atol=0)
    assert st[4] == (np.sqrt(ux * ux + uy * uy) + np.sqrt(1.4 * p / un[0])).max() and st[5] == 0.0
