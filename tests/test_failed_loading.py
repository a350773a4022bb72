"""A context whose filaments could not be loaded or laid out anew, one allocation
failing after another, on a CUDA runtime without a GPU
(tests/native/fake_cudart.c)."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

CHILD = r"""
import ctypes, sys
import numpy as np
sys.path.insert(0, %(root)r)
import simcore_b200 as sc
from simcore_b200 import workloads
fake = ctypes.CDLL(%(fake)r)
fake.fake_fail_after.argtypes = fake.fake_fail_from.argtypes = [ctypes.c_long]
fake.fake_launches.restype = fake.fake_live.restype = ctypes.c_long
cfg = workloads.make("C", scale=0.002, seed=1)


class Loading(sc.Context):  # keeps the handle of a failed construction
    def _check(self, rc):
        if rc != sc.SC_OK and not hasattr(self, "failed"):
            self.failed = rc
        else:
            super()._check(rc)


def load(n):
    ctx = Loading.__new__(Loading)
    orig = sc.lib.sc_add_filaments

    class Lib:  # the allocations of the loading alone are counted
        def __getattr__(self, name):
            return getattr(orig_lib, name)

        def sc_add_filaments(self, *args):
            fake.fake_fail_after(n)
            rc = orig(*args)
            fake.fake_fail_after(-1)
            return rc

    orig_lib, sc.lib = sc.lib, Lib()
    try:
        ctx.__init__(*cfg[:3])
    finally:
        sc.lib = orig_lib
    return ctx
"""

AFTER_FAILURE = CHILD + r"""
n = 0
while True:
    ctx = load(n)
    if not hasattr(ctx, "failed"):
        break
    assert ctx.failed == 2, (n, ctx.failed)  # SC_ERR_OOM
    before = fake.fake_launches()
    assert sc.lib.sc_synchronize(ctx.h) == sc.SC_OK
    assert fake.fake_launches() == before, "a kernel ran after allocation %%d failed" %% n
    ctx.close()
    n += 1
assert n > 50
"""

FAILED_LAYOUT = CHILD + r"""
ctx = load(-1)
assert not hasattr(ctx, "failed")
live = fake.fake_live()
n = 0
while True:
    fake.fake_fail_from(n)
    rc = sc.lib.sc_set_integrator_layout(ctx.h, 0, 256)
    fake.fake_fail_after(-1)
    if rc == sc.SC_OK:
        break
    assert rc == 2, (n, rc)
    assert fake.fake_live() == live, "the tables changed when allocation %%d failed" %% n
    n += 1
assert n > 3
ctx.close()
assert fake.fake_live() == 0
"""


def run_on_fake(tmp_path, code):
    """The code in a child process whose CUDA runtime is the fake."""
    fake = str(tmp_path / "libfake_cudart.so")
    subprocess.check_call(["/usr/bin/gcc", "-O1", "-shared", "-fPIC", "-o", fake,
                           os.path.join(ROOT, "tests", "native", "fake_cudart.c")])
    env = dict(os.environ, LD_PRELOAD=fake)
    out = subprocess.run([sys.executable, "-c", code % dict(root=ROOT, fake=fake)], env=env,
                         capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]


def test_synchronize_after_failed_loading_launches_nothing(tmp_path):
    """Whichever allocation of sc_add_filaments fails, sc_synchronize reads the
    status word and launches no kernel on arrays that do not exist."""
    run_on_fake(tmp_path, AFTER_FAILURE)


def test_failed_layout_keeps_the_old_tables(tmp_path):
    """When an allocation of a new integrator layout fails, and every one after
    it, the context keeps the tables that its launches read."""
    run_on_fake(tmp_path, FAILED_LAYOUT)
