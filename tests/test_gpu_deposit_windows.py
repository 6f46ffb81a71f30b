"""The deposition where a tile's window can go wrong: lattices shifted and
stretched against the grid (cells of one to nine particles), rarefied plasma
(several windows of a tile), scrambled plasma (particles outside all of them),
lattices mixed from global memory (too many coarse columns), masses outside
the fast arithmetic's range; every tile height."""
import numpy as np
import pytest

torch = pytest.importorskip('torch')

from conftest import GOLDEN  # noqa: E402, F401
from make_golden import make_config  # noqa: E402
from oracle import lcode_oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu

# (N, coarseness, fineness, smooth displacement, its wave number, random displacement, mass factor)
CASES = [(41, 3, 2, 0.0, 1.0, 0.0, 1.0), (61, 3, 2, 0.033, 0.0, 0.0, 1.0), (81, 3, 2, 0.3, 1.5, 0.0, 1.0),
         (121, 3, 2, 0.9, 1.6, 0.0, 1.0), (121, 3, 2, 0.3, 1.0, 1.5, 1.0), (161, 3, 2, 0.5, 1.2, 0.05, 1.0),
         (61, 1, 2, 0.2, 1.0, 0.02, 1.0), (61, 2, 3, 0.2, 1.0, 0.0, 1.0), (61, 3, 1, 0.2, 1.0, 0.1, 1.0),
         (61, 3, 4, 0.2, 1.0, 0.0, 1.0), (61, 3, 2, 0.2, 1.0, 0.0, 1e-150)]


@pytest.mark.parametrize('N, coarse, fine, amp, wave, noise, mass', CASES)
def test_deposit_matches_oracle(N, coarse, fine, amp, wave, noise, mass):
    import lcode3d_b200 as L
    from lcode3d_b200._lib import lib
    cfg = make_config(N, 0.1, 0.05, 10, amplitude=0.3)
    cfg.plasma_coarseness, cfg.plasma_fineness = coarse, fine
    cfg.reflect_padding_steps = max(cfg.reflect_padding_steps, coarse + 2)
    x0, y0, *_, m, q, ovirt = O.make_plasma(N - 2 * cfg.plasma_padding_steps, 0.1, coarse, fine)
    rng = np.random.default_rng(N)
    edge = (1 - (x0 / np.abs(x0).max()) ** 4) * (1 - (y0 / np.abs(y0).max()) ** 4)
    x = edge * (amp * np.sin(wave * (x0 + 0.6 * y0) + 1) + noise * rng.uniform(-.5, .5, x0.shape))
    y = edge * (amp * np.cos(wave * (0.7 * x0 - y0)) + noise * rng.uniform(-.5, .5, x0.shape))
    px, py, pz = (mass * rng.normal(size=x0.shape) for _ in range(3))
    args = [x, y, m * mass, q, px, py, pz]
    want = O.deposit(cfg, 0, *args, ovirt)
    virt = L.GPUArrays(**{k: getattr(ovirt, k) for k in ('influence_prev', 'influence_next', 'indices_prev',
                                                         'indices_next', 'fine_grid')})
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in args]
    s = L.solver_for(cfg)
    try:
        for rows in (0, 4, 8, 16):
            assert lib.lc3d_set_tiles(s.ctx, rows, 0) == 0
            got = L.deposit(cfg, 0, *dev, virt)
            again = L.deposit(cfg, 0, *dev, virt)
            for name, g, a, w in zip(('ro', 'jx', 'jy', 'jz'), got, again, want):
                assert torch.equal(g, a), (name, rows)   # sums in a fixed order
                assert O.relative_error(g.cpu().numpy(), w) < 1e-13, (name, rows)   # the particle stages' parity tolerance
    finally:
        lib.lc3d_set_tiles(s.ctx, 0, 0)
