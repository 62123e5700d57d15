"""k_transpose reads whole rows of the states, padding included, and flags codes
out of range among what it read: whatever buffer it is given, the bytes past
the last locus are zero (sdca_set_alignment's states, sdca_set_targets'
columns).  The library runs on the stand-in for the CUDA runtime, which looks
at the buffer when the kernel is launched.  No GPU."""
import json
import os

import pytest

import cuda_standin

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes as C, json, sys
import numpy as np
fake = C.CDLL(sys.argv[2], mode=C.RTLD_GLOBAL)
sys.path.insert(0, sys.argv[1])
from superdca_gb300 import Engine, FORM_GATHER
N, L, LT = json.loads(sys.argv[3])
with Engine(N, L, batch=1, form=FORM_GATHER) as E:
    E.set_alignment(np.ones((N, L), np.uint8), np.ones(N))
    E.set_targets(np.ones((N, LT), np.uint8))
    print(json.dumps([fake.standin_transposes(), fake.standin_bad_padding()]))
"""


@pytest.mark.parametrize("N,L,LT", [(5, 20, 7), (64, 64, 128), (130, 65, 63)])
def test_padding_is_zero(tmp_path, engine_lib, N, L, LT):
    so = cuda_standin.build(tmp_path)
    assert json.loads(cuda_standin.run(so, CHILD, ROOT, so, json.dumps([N, L, LT]))) == [2, 0]
