"""Waits inside the FP64 kernels that run out: the library with the limit of
one source file's waits set to nothing reports PQMC_ERR_TIMEOUT from the call
that launched the kernel, and the context stays usable."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import sys
import numpy as np
from pqmc_allinone_gb300 import abi
abi._LIB = abi.load_library(sys.argv[1])
from pqmc_allinone_gb300.engine import PqmcChain, PqmcError
from tests.helpers import SEED_WORDS, epsocz_small

def runs_out(call, *args):
    try:
        call(*args)
    except PqmcError as e:
        assert "PQMC_ERR_TIMEOUT" in str(e), e
        return
    raise AssertionError(f"{call.__name__}{args}: no error")

m, f = epsocz_small(L=4, ntime=8, ngroup=4)
c = PqmcChain(m, field=f, rng_words=SEED_WORDS)
c.init_expkv()
if sys.argv[2] == "linalg":
    runs_out(c.init_g, 1)
    runs_out(c.init_g, 1)
else:
    c.init_g(1)
    g = c.g()
    runs_out(c.sweep_slices, 2, 1, 1)      # one slice, no recompute after it
    runs_out(c.update_phonon_field, 1, 1)
    c.set_field(f)
    c.init_expkv()
    c.init_g(1)
    assert np.array_equal(c.g(), g)
print("reported")
"""


@pytest.mark.parametrize("source", ["update", "linalg"])
def test_waits_that_run_out_are_reported(tmp_path, source):
    from pqmc_allinone_gb300 import build as b
    b.build()
    obj, lib = str(tmp_path / "short.o"), str(tmp_path / "libshort.so")
    subprocess.run([b.nvcc(), *b.ARCH, *b.FLAGS, "-DPQMC_WAIT_CYCLES=0", "-c", os.path.join(b.CSRC, source + ".cu"), "-o",
                    obj], check=True, timeout=300)
    rest = [os.path.join(b.OUT, o) for o in sorted(os.listdir(b.OUT)) if o.endswith(".o") and o != source + ".o"]
    subprocess.run([b.nvcc(), *b.ARCH, "-shared", "-o", lib, obj, *rest, "-lcudart"], check=True, timeout=300)
    r = subprocess.run([sys.executable, "-c", SCRIPT, lib, source], cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "reported" in r.stdout, r.stdout + r.stderr
