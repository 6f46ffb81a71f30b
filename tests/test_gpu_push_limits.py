"""Particles whose pz swamps their mass and transverse momenta, so that
gamma_m - pz rounds to exactly 0: the quotients are the infinities (NaN for
0 / 0) that the division gives."""
import numpy as np
import pytest

torch = pytest.importorskip('torch')

from conftest import GOLDEN  # noqa: E402, F401
from make_golden import make_config  # noqa: E402
from oracle import lcode_oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


def test_estimate_with_zero_denominator():
    import lcode3d_b200 as L
    cfg = make_config(41, 0.1, 0.05, 10, amplitude=0.3)
    O.init(cfg)
    x0, y0, *_, m, q, _ = O.make_plasma(21, 0.1)
    rng = np.random.default_rng(11)
    px, py = (rng.normal(size=m.shape) for _ in range(2))
    pz = rng.normal(size=m.shape)
    pz[::2] = 10.0 ** rng.uniform(12, 100, size=pz[::2].shape)
    px[0, :2] = 0.0
    off = [0.02 * rng.normal(size=m.shape) for _ in range(2)]
    args = [m, x0, y0, *off, px, py, pz]
    with np.errstate(all='ignore'):
        want = O.move_estimate_wo_fields(cfg, *args)
    got = L.move_estimate_wo_fields(cfg, *[torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in args])
    for g, w in zip(got, want):
        g = g.cpu().numpy()
        assert np.isinf(w[::2]).any() and np.isfinite(w[1::2]).all()
        assert np.array_equal(g[::2], w[::2], equal_nan=True)
        assert O.relative_error(g[1::2], w[1::2]) < 1e-13   # the particle stages' parity tolerance
