"""A host allocation that fails while a context is set up is an error code, and
what was set up is given back. A child process runs with an operator new that
can be told to fail at the n-th large allocation of the calling thread."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SHIM = r'''
#include <cstdlib>
#include <new>
static thread_local long g_left = -1;   // large allocations until one fails; -1: none fails
extern "C" void fail_after(long n) { g_left = n; }
static void* take(size_t n) {
    if (n >= 65536 && g_left >= 0 && g_left-- == 0) throw std::bad_alloc();
    void* p = malloc(n ? n : 1);
    if (!p) throw std::bad_alloc();
    return p;
}
void* operator new(size_t n) { return take(n); }
void* operator new[](size_t n) { return take(n); }
void operator delete(void* p) noexcept { free(p); }
void operator delete[](void* p) noexcept { free(p); }
void operator delete(void* p, size_t) noexcept { free(p); }
void operator delete[](void* p, size_t) noexcept { free(p); }
'''

CHILD = r'''
import ctypes, sys
sys.path[:0] = [ROOT, ROOT + '/tests/golden']
import torch
import lcode3d_b200 as L
from lcode3d_b200 import _lib
from make_golden import make_config
shim = ctypes.CDLL(None)
for N, precision, form in ((161, 'fp64', 'fft'), (161, 'fp64', 'dense'), (161, 'fft32', 'fft'), (161, 'mixed', 'auto')):
    cfg = make_config(N, 0.1, 0.05, 10, amplitude=0.1)
    cfg.lc3d_precision, cfg.lc3d_fp64_transform = precision, form
    p = L.lcode.params_of(cfg)
    torch.cuda.init()
    ctx = ctypes.c_void_p()
    assert _lib.lib.lc3d_create(ctypes.byref(p), 0, ctypes.byref(ctx)) == 0   # loads every kernel of the set-up
    _lib.lib.lc3d_destroy(ctx)
    free = torch.cuda.mem_get_info()[0]
    for k in range(200):
        shim.fail_after(ctypes.c_long(k))
        rc = _lib.lib.lc3d_create(ctypes.byref(p), 0, ctypes.byref(ctx))
        shim.fail_after(ctypes.c_long(-1))
        if rc == 0:
            break
        assert 'size' in _lib.lib.lc3d_strerror(rc).decode() and not ctx.value, (rc, k)
        assert torch.cuda.mem_get_info()[0] >= free, k   # what the failed call took is back
    assert rc == 0 and k >= 4, (rc, k)
    _lib.lib.lc3d_destroy(ctx)
    print(precision, form, k)
'''


def test_failed_host_allocations(tmp_path):
    src = tmp_path / 'shim.cpp'
    src.write_text(SHIM)
    so = tmp_path / 'shim.so'
    subprocess.run(['g++', '-O1', '-shared', '-fPIC', '-o', str(so), str(src)], check=True)
    r = subprocess.run([sys.executable, '-c', f'ROOT = {ROOT!r}\n' + CHILD], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, LD_PRELOAD=str(so)))
    assert r.returncode == 0, r.stdout + r.stderr
    assert len(r.stdout.split('\n')) == 5, r.stdout
