"""A context's two deposition accumulators pass between its calls: steps that
solve both passes, predicted steps (one pass), single depositions and captured
runs. Each call in turn on one context gives bit for bit what it gives on a
context of its own."""
import ctypes

import pytest

torch = pytest.importorskip('torch')

from conftest import GOLDEN  # noqa: E402, F401
from make_golden import beam_array, make_config  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('precision, form, N', [('fp64', 'fft', 81), ('fp64', 'dense', 83), ('fft32', 'fft', 161)])
def test_calls_in_turn_equal_calls_alone(precision, form, N):
    import lcode3d_b200 as L
    from lcode3d_b200 import _lib
    cfg = make_config(N, 0.1, 0.05, 10, amplitude=0.3)
    cfg.lc3d_precision, cfg.lc3d_fp64_transform = precision, form
    names = _lib.STATE_NAMES

    def fresh():
        L.lcode._solvers.clear()
        L.lcode._solvers_raw.clear()

    fresh()
    xs, ys, const, virt, st = L.init(cfg)
    for i in range(3):
        st = L.step(cfg, const, virt, st, beam_array(cfg, 40 + i, xs, ys))
    base = {n: getattr(st, n).clone() for n in names}
    beam = torch.from_numpy(beam_array(cfg, 43, xs, ys)).cuda()

    def state():
        return L.GPUArrays(**base)

    def arrays(s):
        return [getattr(s, n).clone() for n in names]

    def plain():
        return arrays(L.step(cfg, const, virt, state(), beam))

    def predicted():
        s = L.solver_for(cfg)
        s.set_const(const)
        s.set_virt(virt)
        out = {n: torch.empty_like(base[n]) for n in names}
        pred = [base[n] * 1.01 for n in ('Ex', 'Ey', 'Ez', 'Bx', 'By', 'Bz')]
        sp, op = (_lib.StatePtrs(*[d[n].data_ptr() for n in names]) for d in (base, out))
        _lib.check(_lib.lib.lc3d_step_arrays_predicted(
            s.ctx, ctypes.byref(sp), ctypes.byref(op), ctypes.c_void_p(beam.data_ptr()),
            (ctypes.c_void_p * 6)(*[p.data_ptr() for p in pred]), None, L.lcode._stream()), 'predicted step')
        torch.cuda.synchronize()
        return [out[n] for n in names]

    def deposit():
        return [t.clone() for t in L.deposit(cfg, 0, base['x_offt'], base['y_offt'], const.m, const.q, base['px'], base['py'],
                                             base['pz'], virt)]

    def run():
        s, ez = L.lcode.run(cfg, const, virt, state(), 43, 3, beam=(0.3, 1.0, 1.0))
        return arrays(s) + [ez.clone()]

    calls = (plain, predicted, plain, deposit, run, predicted, run, deposit, plain, predicted, deposit)
    fresh()
    together = [c() for c in calls]
    for k, c in enumerate(calls):
        fresh()
        for a, b in zip(together[k], c()):
            assert torch.equal(a, b), (k, c.__name__)
    fresh()
