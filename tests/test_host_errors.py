"""Calls after a failed one, on the CPU: the engine runs on a stand-in for the CUDA runtime (fake_cudart.c: host
memory, kernels skipped), one of whose allocations fails."""
import os
import subprocess
import sys

import pytest

from conftest import REPO

SETUP = """
import ctypes, sys
import numpy as np
from hfgpu import basis, engine, workloads

fake = ctypes.CDLL(sys.argv[1])
fake.fake_fail_malloc.argtypes = [ctypes.c_long]
fake.fake_uploads.restype = ctypes.c_long
Z, xyz = workloads.water_chain(2, np.random.default_rng(1))
e = engine.Engine(basis.pack("6-31G**", Z, xyz))
ns = e.nshells[0]
Q = np.exp(-6 * np.random.default_rng(2).random((ns, ns)) ** 2)  # pair products on both sides of the thresholds
Q = Q + Q.T
e.set_schwartz(Q)
D = np.eye(e.nao)
loose, tight = 1e-2, 1e-6

def uploads(f, *args, **kw):
    before = fake.fake_uploads()
    f(*args, **kw)
    return fake.fake_uploads() - before

def failing(after, f, *args, **kw):
    fake.fake_fail_malloc(after)
    try:
        f(*args, **kw)
    except engine.HfgError as x:
        assert x.code == -5, x  # HFG_ERR_NOMEM
    else:
        raise SystemExit("no allocation failed")
    finally:
        fake.fake_fail_malloc(-1)
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    from hfgpu import build

    build.build(verbose=False)
    lib = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", lib, os.path.join(REPO, "tests", "fake_cudart.c")], check=True)
    env = dict(os.environ, LD_PRELOAD=lib, PYTHONPATH=os.path.join(REPO, "hartree-fock_gb300"))

    def go(script, *args):
        r = subprocess.run([sys.executable, "-c", SETUP + script, lib, *map(str, args)], env=env, capture_output=True,
                           text=True, timeout=600)
        assert r.returncode == 0, r.stdout + r.stderr

    return go


@pytest.mark.parametrize("succeed", [0, 3, 11])
def test_failed_allocation_does_not_fail_the_next_call(run, succeed):
    run("""
e.fock(D, D, sthr=loose)
failing(int(sys.argv[2]), e.fock, D, D, sthr=tight)
e.fock(D, D, sthr=tight)
""", succeed)


@pytest.mark.parametrize("succeed", [0, 3, 11, 20])
@pytest.mark.parametrize("retry", ["the earlier threshold", "the failed one"])
def test_failed_sizing_of_the_lists_is_not_kept(run, succeed, retry):
    """Lists are sized class by class; a call that fails between two classes leaves some of them sized for its own
    threshold, so the next call, at whichever threshold, sizes all of them again."""
    run("""
first, again = uploads(e.fock, D, D, sthr=loose), uploads(e.fock, D, D, sthr=loose)
assert first > again  # the second call keeps the lists
failing(int(sys.argv[2]), e.fock, D, D, sthr=tight)
assert uploads(e.fock, D, D, sthr=loose if sys.argv[3] == "the earlier threshold" else tight) == first
""", succeed, retry)


def test_survivors_of_lists_that_are_gone_are_refused(run):
    """A call that fails while it sizes the lists has given the last build's lists back already."""
    run("""
e.fock(D, D, sthr=loose)
e.survivors()
failing(3, e.fock, D, D, sthr=tight)
try:
    e.survivors()
except engine.HfgError as x:
    assert x.code == -1, x  # HFG_ERR_INVALID
else:
    raise SystemExit("survivors read from new buffers")
e.fock(D, D, sthr=loose)
e.survivors()
""")
