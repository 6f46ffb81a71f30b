"""The folded dense solves at the edges of their tiles: halves of one to a few
points, of a tile of rows or columns exactly and one more."""
import numpy as np
import pytest

torch = pytest.importorskip('torch')

from conftest import GOLDEN  # noqa: E402, F401
from make_golden import make_config  # noqa: E402
from oracle import lcode_oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('N', (5, 7, 9, 31, 63, 65, 67, 127, 129, 131, 235, 387))
def test_solvers_match_oracle(N):
    import lcode3d_b200 as L
    cfg = make_config(N, 16.0 / (N - 1), 0.01, 10, amplitude=0.1)
    cfg.plasma_padding_steps = 0
    cfg.plasma_coarseness = 1
    cfg.lc3d_fp64_transform = 'dense'
    rng = np.random.default_rng(N)
    a = [rng.normal(size=(N, N)) for _ in range(11)]
    t = [torch.from_numpy(v).cuda() for v in a]
    got = [v.cpu().numpy() for v in (*L.calculate_Ex_Ey_Bx_By(cfg, *t), L.calculate_Ez(cfg, t[0], t[1]),
                                     L.calculate_Bz(cfg, t[0], t[1]))]
    want = [*O.calculate_Ex_Ey_Bx_By(cfg, *a), O.calculate_Ez(cfg, a[0], a[1]), O.calculate_Bz(cfg, a[0], a[1])]
    for name, g, w in zip(('Ex', 'Ey', 'Bx', 'By', 'Ez', 'Bz'), got, want):
        assert O.relative_error(g, w) < 1e-12, name   # the solvers' parity tolerance
