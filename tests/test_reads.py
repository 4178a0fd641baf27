"""Reads of the status and the measurements: what reaches the caller when a
copy fails.  The CUDA runtime is a fake in host memory (fake_cudart.c), so
these run without a GPU, in a process of their own."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PRELUDE = """
import ctypes as C
from lceqcd_b200 import _lib
from lceqcd_b200.lattice import Params
fake = C.CDLL(None)
fake.fake_d2h_bytes.restype = fake.fake_d2h_copies.restype = C.c_size_t
lib = _lib.load()
REC = C.sizeof(_lib.LceMeas)

def create(n):
    p = (_lib.LceParams * n)(*[Params(L=(2, 2, 2), seed=i + 1).to_c() for i in range(n)])
    c = lib.lce_create_batch(p, n)
    assert c, lib.lce_last_error(None)
    return c
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    so = tmp_path_factory.mktemp("fake") / "fake_cudart.so"
    subprocess.check_call(["gcc", "-O1", "-shared", "-fPIC", "-o", str(so), os.path.join(ROOT, "tests", "fake_cudart.c")])

    def run(body):
        env = dict(os.environ, LD_PRELOAD=str(so), PYTHONPATH=ROOT)
        r = subprocess.run([sys.executable, "-c", PRELUDE + body], env=env, cwd=ROOT, capture_output=True, text=True,
                           timeout=120)
        assert r.returncode == 0, r.stdout + r.stderr
    return run


@pytest.mark.parametrize("copy,sync", [(1, 0), (0, 1)])
def test_failed_read_leaves_the_callers_record(fake, copy, sync):
    fake(f"""
c = create(3)
m, b = _lib.LceMeas(), (_lib.LceMeas * 3)()
C.memset(C.byref(m), 0x5a, REC)
C.memset(b, 0x5a, 3 * REC)
fake.fake_reset({copy}, {sync})
for chain in range(3):
    assert lib.lce_get_meas(c, chain, C.byref(m)) == _lib.LCE_ERR_CUDA
assert lib.lce_get_meas_batch(c, b) == _lib.LCE_ERR_CUDA
assert bytes(m) == b"\\x5a" * REC, "a record after a failed read"
assert bytes(b) == b"\\x5a" * 3 * REC, "records after a failed read"
fake.fake_reset(0, 0)
assert lib.lce_get_meas(c, 2, C.byref(m)) == 0 and bytes(m) == bytes(REC)
assert lib.lce_get_meas_batch(c, b) == 0 and bytes(b) == bytes(3 * REC)
lib.lce_destroy(c)
""")


@pytest.mark.parametrize("n", [1, 3, 1000])
def test_a_read_copies_what_it_returns(fake, n):
    """The state and the record asked for, not every chain's: a loop over the
    chains stays linear in their number.  A single chain's values and the last
    call's acceptance take one copy."""
    fake(f"""
n = {n}
c = create(n)
m, b, f = _lib.LceMeas(), (_lib.LceMeas * n)(), C.c_float(0.5)
def cost(call):
    fake.fake_reset(0, 0)
    assert call() == 0
    return fake.fake_d2h_bytes(), fake.fake_d2h_copies()
STATE = 256
assert cost(lambda: lib.lce_synchronize(c)) <= (STATE, 1)
for chain in {{0, n // 2, n - 1}}:
    size, copies = cost(lambda: lib.lce_get_meas(c, chain, C.byref(m)))
    assert size <= STATE + REC and copies <= (1 if chain == 0 else 2), (chain, size, copies)
for call in (lambda: lib.lce_ahiggs2(c, 1, C.byref(f)), lambda: lib.lce_ahiggs1(c, C.byref(f), 1, None)):
    size, copies = cost(call)
    assert size <= STATE + REC and copies == 1, (size, copies)
assert cost(lambda: lib.lce_get_meas_batch(c, b)) == (STATE + n * REC, 1)
lib.lce_destroy(c)
""")
