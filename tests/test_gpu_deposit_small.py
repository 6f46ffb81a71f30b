"""The deposition on both sides of the rule for small lattices (240 fine
particles a side at fineness 2, 400 at others): one, two and four threads per cell below it, 12-row tiles
above, each where a window can go wrong (cells of many particles, several
windows of a tile, particles outside all of them); a launch over several
simulations takes each one's own shape."""
import numpy as np
import pytest

torch = pytest.importorskip('torch')

from conftest import GOLDEN  # noqa: E402, F401
from make_golden import make_config  # noqa: E402
from oracle import lcode_oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu

# (N, coarseness, fineness, smooth displacement, its wave number, random displacement)
CASES = [(141, 3, 2, 0.3, 1.5, 0.05), (143, 3, 2, 0.3, 1.5, 0.05),      # 240 and 244 fine particles a side
         (421, 3, 1, 0.3, 1.5, 0.05), (423, 3, 1, 0.3, 1.5, 0.05),      # 399 and 401
         (241, 3, 2, 0.9, 1.6, 0.0), (241, 3, 2, 0.0, 1.0, 4.0), (81, 3, 2, 0.0, 1.0, 4.0), (161, 3, 2, 0.9, 1.6, 0.0),
         (81, 1, 1, 0.9, 1.6, 0.0), (161, 3, 1, 0.3, 1.0, 1.5), (441, 3, 1, 0.3, 1.0, 0.1), (121, 2, 3, 0.9, 1.6, 0.1),
         (81, 3, 4, 0.9, 1.6, 0.0), (61, 3, 5, 0.3, 1.0, 1.5), (161, 3, 4, 0.3, 1.0, 0.1)]


@pytest.mark.parametrize('N, coarse, fine, amp, wave, noise', CASES)
def test_deposit_matches_oracle(N, coarse, fine, amp, wave, noise):
    import lcode3d_b200 as L
    h = 16.0 / (N - 1)
    cfg = make_config(N, h, 0.05, 10, amplitude=0.3)
    cfg.plasma_coarseness, cfg.plasma_fineness = coarse, fine
    x0, y0, *_, m, q, ovirt = O.make_plasma(N - 2 * cfg.plasma_padding_steps, h, coarse, fine)
    rng = np.random.default_rng(N + fine)
    edge = (1 - (x0 / np.abs(x0).max()) ** 4) * (1 - (y0 / np.abs(y0).max()) ** 4)
    x = edge * (amp * np.sin(wave * (x0 + 0.6 * y0) + 1) + noise * rng.uniform(-.5, .5, x0.shape))
    y = edge * (amp * np.cos(wave * (0.7 * x0 - y0)) + noise * rng.uniform(-.5, .5, x0.shape))
    args = [x, y, m, q, *(0.5 * rng.normal(size=x0.shape) for _ in range(3))]
    want = O.deposit(cfg, 0, *args, ovirt)
    virt = L.GPUArrays(**{k: getattr(ovirt, k) for k in ('influence_prev', 'influence_next', 'indices_prev',
                                                         'indices_next', 'fine_grid')})
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in args]
    got = L.deposit(cfg, 0, *dev, virt)
    again = L.deposit(cfg, 0, *dev, virt)
    for name, g, a, w in zip(('ro', 'jx', 'jy', 'jz'), got, again, want):
        assert torch.equal(g, a), name   # sums in a fixed order
        assert O.relative_error(g.cpu().numpy(), w) < 1e-13, name   # the particle stages' parity tolerance


def test_joint_deposition_of_both_shapes():
    from lcode3d_b200 import batch as B
    specs = [dict(grid_steps=n, grid_step_size=16.0 / (n - 1), xi_step_size=0.02, amplitude=0.4, sigma_r=1.0,
                  length_factor=1.0) for n in (161, 321, 41, 121)]
    runs = []
    for multi in (False, True):
        bt = B.Batch(specs, multi_deposit=multi)
        hist = bt.run(6)
        bt.check_errors()
        runs.append(([h.clone() for h in hist], [sim.state() for sim in bt.sims]))
    for k in range(len(specs)):
        assert torch.equal(runs[0][0][k], runs[1][0][k]), k
        assert torch.equal(runs[0][1][k].ro, runs[1][1][k].ro), k
