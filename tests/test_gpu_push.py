"""The pusher and the field-free estimate inside and outside the range of their
branch-free arithmetic, and a state's round trip through a context."""
import types

import numpy as np
import pytest

torch = pytest.importorskip('torch')

from conftest import GOLDEN  # noqa: E402, F401
from make_golden import make_config  # noqa: E402
from oracle import lcode_oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('mass', [1.0, 1e-100, 1e-150, 1e140])
def test_push_matches_oracle(mass):
    import lcode3d_b200 as L
    cfg = make_config(41, 0.1, 0.05, 10, amplitude=0.3)
    O.init(cfg)
    x0, y0, *_, m, q, _ = O.make_plasma(21, 0.1)
    rng = np.random.default_rng(7)
    p = [mass * rng.normal(size=m.shape) for _ in range(3)]
    off = [0.02 * rng.normal(size=m.shape) for _ in range(4)]
    fields = [mass * rng.normal(size=(41, 41)) for _ in range(6)]
    args = [m * mass, q, x0, y0, *off, *p, *fields]
    want = O.move_smart(cfg, *args)
    got = L.move_smart(cfg, *[torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in args])
    for k, (g, w) in enumerate(zip(got, want)):
        assert O.relative_error(g.cpu().numpy(), w) < 1e-13, k   # the particle stages' parity tolerance
    est = [m * mass, x0, y0, *off[:2], *p]
    want = O.move_estimate_wo_fields(cfg, *est)
    got = L.move_estimate_wo_fields(cfg, *[torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in est])
    for g, w in zip(got, want):
        assert O.relative_error(g.cpu().numpy(), w) < 1e-13


@pytest.mark.parametrize('N', [41, 43])
def test_state_round_trip(N):
    """lc3d_run of no steps copies the state in and out; arrays that start on
    odd words of an allocation take the unaligned copy."""
    from lcode3d_b200 import lcode as L
    cfg = make_config(N, 0.1, 0.05, 10, amplitude=0.3)
    _, _, const, virt, st = L.init(cfg)
    rng = np.random.default_rng(N)
    new = types.SimpleNamespace()
    for k, n in enumerate(('x_offt', 'y_offt', 'px', 'py', 'pz', 'Ex', 'Ey', 'Ez', 'Bx', 'By', 'Bz', 'ro', 'jx', 'jy',
                           'jz')):
        shape = getattr(st, n).shape
        buf = torch.from_numpy(rng.normal(size=shape.numel() + 1)).cuda()
        setattr(new, n, buf[k % 2:k % 2 + shape.numel()].view(shape))
    out, _ = L.run(cfg, const, virt, new, 0, 0)
    for n, v in vars(new).items():
        assert torch.equal(getattr(out, n), v), n
