"""lc3d_set_state / lc3d_get_state copy the 15 arrays as they are, whatever
their alignment: arrays packed at an odd number of elements lie on 8-byte
boundaries, those of a view at an even one on 16-byte boundaries."""
import ctypes

import pytest

torch = pytest.importorskip('torch')

from make_golden import make_config  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('N,shift,gap', [(41, 0, 0), (41, 1, 1), (41, 0, 1), (161, 1, 0)])
def test_state_round_trip(N, shift, gap):
    import lcode3d_b200 as L
    from lcode3d_b200 import _lib
    cfg = make_config(N, 0.1, 0.05, 10, amplitude=0.1)
    s = L.solver_for(cfg)
    _, _, _, _, st = L.init(cfg)
    names = _lib.STATE_NAMES
    sizes = [getattr(st, n).numel() for n in names]
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def packed(fill):
        # every array between guard elements, `shift` elements into the buffer
        buf = torch.full((shift + sum(sizes) + (gap + 1) * 16,), fill, dtype=torch.float64, device='cuda')
        at, views = shift, []
        for n in sizes:
            views.append(buf[at:at + n])
            at += n + gap
        return buf, views

    _, src = packed(0.0)
    for k, v in enumerate(src):
        v.copy_(torch.arange(v.numel(), dtype=torch.float64, device='cuda') + 1e6 * (k + 1))
    buf, dst = packed(-7.0)
    want = torch.full_like(buf, -7.0)
    for k, v in enumerate(dst):
        at = v.storage_offset()
        want[at:at + v.numel()] = src[k]
    sp, dp = (_lib.StatePtrs(*[v.data_ptr() for v in a]) for a in (src, dst))
    _lib.check(_lib.lib.lc3d_set_state(s.ctx, ctypes.byref(sp), stream), 'set_state')
    _lib.check(_lib.lib.lc3d_get_state(s.ctx, ctypes.byref(dp), stream), 'get_state')
    assert torch.equal(buf, want)   # the arrays, and nothing beside them
