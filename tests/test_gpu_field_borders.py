"""Grid rows and columns that a field's solve does not use (the Dirichlet
borders of Ey, Bx along x and of Ex, By along y) may hold anything."""
import numpy as np
import pytest

torch = pytest.importorskip('torch')

from conftest import GOLDEN  # noqa: E402, F401
from make_golden import make_config  # noqa: E402
from oracle import lcode_oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('form, N', [('fft', 5), ('fft', 41), ('fft', 161), ('fft', 433), ('dense', 43)])
@pytest.mark.parametrize('value', [1e40, float('nan'), float('inf')])
def test_unused_borders_do_not_matter(form, N, value):
    import lcode3d_b200 as L
    cfg = make_config(N, 16.0 / (N - 1), 0.01, 10, amplitude=0.1)
    cfg.plasma_padding_steps = 0
    cfg.plasma_coarseness = 1
    cfg.lc3d_fp64_transform = form
    rng = np.random.default_rng(N)
    a = [rng.normal(size=(N, N)) for _ in range(11)]   # Ex Ey Bx By averages, beam ro jx jy jz, previous jx jy
    want = O.calculate_Ex_Ey_Bx_By(cfg, *a)
    for k in (1, 2):
        a[k][[0, -1], :] = value
    for k in (0, 3):
        a[k][:, [0, -1]] = value
    got = L.calculate_Ex_Ey_Bx_By(cfg, *[torch.from_numpy(v).cuda() for v in a])
    for name, g, w in zip(('Ex', 'Ey', 'Bx', 'By'), got, want):
        assert O.relative_error(g.cpu().numpy(), w) < 1e-12, name   # the solvers' parity tolerance
