"""The branch-free square root and quotients round as IEEE 754 does. With a
particle at the origin, py = 0 and a step of 1 the field-free estimate is
px / (sqrt(m^2 + pz^2 + px^2) - pz) itself; of 26-bit operands the squares are
exact, so numpy's result is the one correct rounding of every operation,
whatever the compiler fuses."""
import numpy as np
import pytest

torch = pytest.importorskip('torch')

from conftest import GOLDEN  # noqa: E402, F401
from make_golden import make_config  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('spread', [1, 3, 20, 200])   # binary orders of magnitude the operands span
@pytest.mark.parametrize('with_pz', [False, True])
def test_estimate_is_correctly_rounded(spread, with_pz):
    import lcode3d_b200 as L
    cfg = make_config(641, 1.0, 1.0, 10, amplitude=0.3)
    cfg.plasma_coarseness = cfg.plasma_fineness = 1
    n = L.solver_for(cfg).Nc
    rng = np.random.default_rng(spread)
    m, px, pz = (rng.integers(1 << 25, 1 << 26, size=(n, n)) * 2.0 ** (rng.integers(0, spread, size=(n, n)) - spread - 25)
                 for _ in range(3))
    pz = -pz if with_pz else np.zeros((n, n))   # the quotient stays within the reflecting boundary
    want = px / (np.sqrt(m * m + pz * pz + px * px) - pz)
    zero = np.zeros((n, n))
    args = [m, zero, zero, zero, zero, px, zero, pz]
    got = L.move_estimate_wo_fields(cfg, *[torch.from_numpy(a).cuda() for a in args])[0].cpu().numpy()
    assert np.array_equal(got, want)
