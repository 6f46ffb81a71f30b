"""What a context holds on the device, in float64 planes of the grid: no more
than the arrays its form of the field solves reads."""
import ctypes

import pytest

torch = pytest.importorskip('torch')

from make_golden import make_config  # noqa: E402

pytestmark = pytest.mark.gpu


# 82.4 planes: the FFT form's context of one accumulator set and full-size transform matrices
@pytest.mark.parametrize('N, form, planes', [(1001, 'fft', 82.5), (1003, 'dense', 91.0)])
def test_context_memory(N, form, planes):
    import lcode3d_b200 as L
    from lcode3d_b200._lib import lib
    cfg = make_config(N, 16.0 / (N - 1), 0.05, 10, amplitude=0.1)
    cfg.lc3d_fp64_transform = form
    p = L.lcode.params_of(cfg)
    ctx = ctypes.c_void_p()
    used = []
    for _ in range(2):   # the first context also loads its kernels
        free = torch.cuda.mem_get_info()[0]
        assert lib.lc3d_create(ctypes.byref(p), torch.cuda.current_device(), ctypes.byref(ctx)) == 0
        used.append(free - torch.cuda.mem_get_info()[0])
        lib.lc3d_destroy(ctx)
    assert used[1] <= planes * 8 * N * N, used[1] / (8 * N * N)
