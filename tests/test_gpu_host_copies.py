"""Copies of results and inputs between the device and the caller's memory, of each
kind that memory can be."""
import subprocess
import sys
import time

import numpy as np
import pytest

import instantgr_b200 as ig
from conftest import ROOT

pytestmark = pytest.mark.gpu


def _least(f, n=40):
    best = 1e9
    for _ in range(n):
        t0 = time.perf_counter()
        f()
        best = min(best, time.perf_counter() - t0)
    return best


def test_page_locked_memory_is_copied_directly(tmp_path):
    """Demand of 9 MB into a page-locked array: the copy itself (178 us) with a layout
    kernel and the wait around it (20 us), so 1.6 times a plain copy at most; through
    staging chunks and threads it took 2.3 times at the least."""
    import torch
    X, Y = 420, 600
    cap, net = str(tmp_path / "d.cap"), str(tmp_path / "d.net")
    ig.generate_custom(X, Y, 2000, seed=1, cap=cap, net=net)
    r = ig.Router(cap, net, rrr_iters=0)
    r.run()
    want = r.demand()
    locked = torch.full((9 * X * Y,), -1.0).pin_memory()
    get = lambda: ig._check(ig.lib().igr_router_demand(r.h, locked.numpy()))  # noqa: E731
    get()
    assert np.array_equal(locked.numpy(), want)
    mine = _least(get)
    dev = torch.from_numpy(want).cuda()
    plain = _least(lambda: (locked.copy_(dev), torch.cuda.synchronize()))
    r.close()
    assert mine <= 1.6 * plain, (mine, plain)


ONE_CORE = """
import os, sys, time
os.sched_setaffinity(0, {min(os.sched_getaffinity(0))})
sys.path.insert(0, sys.argv[1])
import numpy as np, torch
import instantgr_b200 as ig
X, Y = 840, 1140
cap, net = sys.argv[2] + "/d.cap", sys.argv[2] + "/d.net"
ig.generate_custom(X, Y, 2000, seed=1, cap=cap, net=net)
r = ig.Router(cap, net, rrr_iters=0)
r.run()
out, dev = torch.zeros(9 * X * Y), torch.zeros(9 * X * Y, device="cuda")
def least(f):
    t = []
    for _ in range(20):
        a = time.perf_counter(); f(); t.append(time.perf_counter() - a)
    return min(t[2:])
mine = least(lambda: ig._check(ig.lib().igr_router_demand(r.h, out.numpy())))
plain = least(lambda: (out.copy_(dev), torch.cuda.synchronize()))
print(mine / plain)
"""


def test_one_core_copies_as_the_driver_does(tmp_path):
    """34 MB into plain memory by a process of one core: the driver's copy and the layout
    kernel, so at most 1.35 times the driver's copy alone; chunk by chunk it took 1.7."""
    p = subprocess.run([sys.executable, "-c", ONE_CORE, ROOT, str(tmp_path)], capture_output=True, text=True,
                       timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]
    assert float(p.stdout.split()[-1]) <= 1.35


OWN_CONTEXT = """
import ctypes, sys
sys.path.insert(0, sys.argv[1])
if sys.argv[2] == "own":
    cu, ctx, dev = ctypes.CDLL("libcuda.so.1"), ctypes.c_void_p(), ctypes.c_int()
    assert cu.cuInit(0) == 0 and cu.cuDeviceGet(ctypes.byref(dev), 0) == 0
    assert cu.cuCtxCreate_v2(ctypes.byref(ctx), 0, dev) == 0
import hashlib
import numpy as np
import instantgr_b200 as ig
m = ig.Seed.load()
for X in (100, 400):
    print(hashlib.sha256(m.predict(np.random.default_rng(1).random((X, X, 16), np.float32)).tobytes()).hexdigest())
if sys.argv[2] == "thread":  # the first use of CUDA by its thread is a copy in chunks
    import threading
    m.set_tile(144, 16)
    x = np.random.default_rng(2).random((6, 144, 144, 16), np.float32)
    want, got = m.grad(x, x)[0], []
    t = threading.Thread(target=lambda: got.append(m.grad(x, x)[0]))
    t.start(); t.join()
    assert abs(got[0] - want) <= 1e-12 * want
m.close()
"""


def test_predictions_in_a_context_of_the_callers_own():
    """Inputs and results below and above the staging limit, in a process whose
    CUDA context is not the device's primary one: the primary one's predictions.
    (The loss of a second thread's call: sums of 1.2M squares in 64 bits, in any order.)"""
    out = []
    for kind in ("thread", "own"):
        p = subprocess.run([sys.executable, "-c", OWN_CONTEXT, ROOT, kind], capture_output=True, text=True, timeout=300)
        assert p.returncode == 0, p.stderr[-2000:]
        out.append(p.stdout)
    assert out[0] == out[1]
