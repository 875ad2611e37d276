"""The library's host code against a CUDA runtime of the host (harness/
fake_cudart.cpp, preloaded; CPU): what depends on the device that is current,
and what a call returns when a kernel reports a failure.  Kernels do not run,
so nothing here looks at numbers."""
import os
import subprocess
import sys

import pytest

from skkr_budapest_gb300 import build, native

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEAD = """
import ctypes, dataclasses
import numpy as np
from skkr_budapest_gb300 import api, native
from skkr_budapest_gb300 import workloads as W
rt = ctypes.CDLL(None)
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    if not os.path.exists(native.LIB_PATH):
        build.build()
    so = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I/usr/local/cuda/include", "-o", so,
                    os.path.join(ROOT, "tests", "harness", "fake_cudart.cpp")], check=True)

    def go(code):
        r = subprocess.run([sys.executable, "-c", HEAD + code], cwd=ROOT, capture_output=True, text=True, timeout=300,
                           env=dict(os.environ, LD_PRELOAD=so))
        assert r.returncode == 0 and "done" in r.stdout, (r.stdout[-500:], r.stderr[-2000:])
    return go


@pytest.mark.parametrize("n", [20, 100, 200])  # stacked tiles, 8-bit and 7-bit digits
def test_products_launch_on_every_device_of_the_process(run, n):
    run("""
a = np.ones((2, %d, %d), complex)
for dev in (0, 1, 0, 2):
    rt.cudaSetDevice(dev)
    for s in range(3, 9):
        native.zgemm_batch(a, a, precision="mixed", slices=s)
assert rt.fake_launches() > 0
print("done")
""" % (n, n))


def test_training_launches_on_every_device_of_the_process(run):
    run("""
layers = [(np.ones((5, 9), np.float32), np.zeros(9, np.float32))]
for dev in (0, 1):
    rt.cudaSetDevice(dev)
    native.mlp16_train(layers, np.ones((40, 5), np.float32), np.ones((40, 9), np.float32), np.ones(40, np.uint8), 2,
                       1e-3, 1e-4, eval_every=0)
print("done")
""")


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_an_expired_wait_fails_the_call_it_happened_in(run, precision):
    """tauij and the energy return the CUDA error and leave the caller's
    arrays alone; the call after them starts from a clear word."""
    run("""
ep = W.energy_problem(dataclasses.replace(W.plain_fcc(nset=1), pl=4), 8)   # 36 rows: tensor-core engines
ctx = api.Context.for_problem(ep, %r)
ctx.set_graphs(False)   # (the host runtime has no graphs)
def tauij():
    r = ctx.tauij(ep, [(0, 0, 0, 1)], [1.0, 0.0], [0.0, 1.0], np.zeros((ep.nintfc, 2)), np.eye(2).reshape(1, 4)
                  .repeat(len(ep.lg), 0), check=False)
    assert not r["tau_ij"].any()
    return r["status"]
def energy():
    return ctx.cpacoord(ep, check=False)["status"]
for call in (tauij, energy):
    rt.fake_expire_waits(1)
    assert call() == -2 and "bounded wait" in native.last_error(), call
    rt.fake_expire_waits(0)
    assert tauij() == 0
print("done")
""" % precision)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_a_rank_with_an_expired_wait_tells_the_others(run, precision):
    """Its sum does not join theirs: the flag goes into the reduction instead."""
    run("""
ep = W.energy_problem(dataclasses.replace(W.plain_fcc(nset=1), pl=4), 8)
ctx = api.Context.for_problem(ep, %r)
ctx.set_graphs(False)
flags = []
def reduce(buf):
    flags.append(buf[-1])
ctx.set_reduce(reduce)
rt.fake_expire_waits(1)
assert ctx.cpacoord(ep, check=False)["status"] == -2 and flags == [1.0], flags
rt.fake_expire_waits(0)
flags.clear()
ctx.cpacoord(ep, check=False)
assert flags[0] == 0.0
print("done")
""" % precision)
