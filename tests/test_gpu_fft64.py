"""The float64 FFT solves at the edges of their plans: no middle radix, one,
two; every radix; grids of one partly filled CTA, of whole CTAs and one row
more; four and eight row pairs per CTA (the largest grids by shared memory)."""
import numpy as np
import pytest

torch = pytest.importorskip('torch')

from conftest import GOLDEN  # noqa: E402, F401
from make_golden import make_config  # noqa: E402
from oracle import lcode_oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu

# 385 / 401: either side of the small-grid rule; 751 and 811: two middle
# radices; 1441, 2001: past eight pairs' shared memory
SIZES = (5, 7, 17, 19, 33, 55, 101, 129, 151, 201, 271, 289, 385, 401, 433, 451, 577, 751, 811, 1153, 1441, 2001)


@pytest.mark.parametrize('N', SIZES)
def test_solvers_match_oracle(N):
    import lcode3d_b200 as L
    cfg = make_config(N, 16.0 / (N - 1), 0.01, 10, amplitude=0.1)
    cfg.plasma_padding_steps = 0
    cfg.plasma_coarseness = 1
    cfg.lc3d_fp64_transform = 'fft'
    rng = np.random.default_rng(N)
    a = [rng.normal(size=(N, N)) for _ in range(11)]
    t = [torch.from_numpy(v).cuda() for v in a]
    got = [v.cpu().numpy() for v in (*L.calculate_Ex_Ey_Bx_By(cfg, *t), L.calculate_Ez(cfg, t[0], t[1]),
                                     L.calculate_Bz(cfg, t[0], t[1]))]
    want = [*O.calculate_Ex_Ey_Bx_By(cfg, *a), O.calculate_Ez(cfg, a[0], a[1]), O.calculate_Bz(cfg, a[0], a[1])]
    for name, g, w in zip(('Ex', 'Ey', 'Bx', 'By', 'Ez', 'Bz'), got, want):
        assert O.relative_error(g, w) < 1e-12, name   # the solvers' parity tolerance
        # exact zeros on the Dirichlet borders
        if name in ('Ey', 'Bx', 'Ez'):
            assert not g[[0, -1]].any(), name
        if name in ('Ex', 'By', 'Ez'):
            assert not g[:, [0, -1]].any(), name


def test_grids_refused_before_stay_refused():
    import lcode3d_b200 as L
    from lcode3d_b200._lib import LC3DError
    for N in (387, 2049):   # 2 * 386 = 4 * 193; a longer FFT than the contexts take
        cfg = make_config(N, 16.0 / (N - 1), 0.01, 10, amplitude=0.1)
        cfg.lc3d_fp64_transform = 'fft'
        with pytest.raises(LC3DError):
            L.solver_for(cfg)
