"""lc3d_set_state / lc3d_get_state with arrays that the copy kernel may not
take: off 8-byte boundaries, in pinned host memory, overlapping (the copies
come in the order of the arrays, so the later one stays)."""
import ctypes

import pytest

torch = pytest.importorskip('torch')

from make_golden import make_config  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture
def ctx():
    import lcode3d_b200 as L
    from lcode3d_b200 import _lib
    cfg = make_config(41, 0.1, 0.05, 10, amplitude=0.1)
    s = L.solver_for(cfg)
    _, _, _, _, st = L.init(cfg)
    sizes = [getattr(st, n).numel() for n in _lib.STATE_NAMES]
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def call(name, pointers):
        p = _lib.StatePtrs(*pointers)
        _lib.check(getattr(_lib.lib, name)(s.ctx, ctypes.byref(p), stream), name)
        torch.cuda.synchronize()
    values = [torch.randn(n, dtype=torch.float64) for n in sizes]
    return call, sizes, values


def test_arrays_off_element_boundaries(ctx):
    call, sizes, values = ctx
    src = torch.zeros(8 * sum(sizes) + 4, dtype=torch.uint8, device='cuda')
    dst = torch.zeros_like(src)
    at = [4 + 8 * sum(sizes[:k]) for k in range(15)]
    for k, v in enumerate(values):
        src[at[k]:at[k] + 8 * sizes[k]] = v.view(torch.uint8).cuda()
    call('lc3d_set_state', [src.data_ptr() + o for o in at])
    call('lc3d_get_state', [dst.data_ptr() + o for o in at])
    assert torch.equal(src, dst)


def test_pinned_host_arrays(ctx):
    call, sizes, values = ctx
    src = [v.pin_memory() for v in values]
    dst = [torch.empty_like(v).pin_memory() for v in values]
    call('lc3d_set_state', [v.data_ptr() for v in src])
    call('lc3d_get_state', [v.data_ptr() for v in dst])
    assert all(map(torch.equal, src, dst))


def test_overlapping_arrays(ctx):
    call, sizes, values = ctx
    src = [v.cuda() for v in values]
    call('lc3d_set_state', [v.data_ptr() for v in src])
    n, g = sizes[0], sizes[5]
    for _ in range(20):
        dst = torch.zeros(5 * n + 9 * (g // 2) + g, dtype=torch.float64, device='cuda')
        want = torch.zeros_like(dst)
        at = [n * k for k in range(5)] + [5 * n + g // 2 * k for k in range(10)]   # every grid array half over the next
        for k, v in enumerate(src):
            want[at[k]:at[k] + sizes[k]] = v
        call('lc3d_get_state', [dst.data_ptr() + 8 * o for o in at])
        assert torch.equal(dst, want)
