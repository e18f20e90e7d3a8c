"""The multipole evaluation of the drop-in entry points (mode_eval, compiled
for the host) against the oracle's, every (l, m), with both coefficient
settings of update_information (mode_cases.py: points and bound)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from mode_cases import BINARIES, LM, oracle_modes, params, rows

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("modes") / "libmodes.so"
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-o", str(out),
                           os.path.join(HERE, "native", "modes_host.cpp")])
    return ctypes.CDLL(str(out))


@pytest.mark.parametrize("use_hm", [0, 1])
@pytest.mark.parametrize("binary", BINARIES)
def test_every_mode(lib, oracle, binary, use_hm):
    dp = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
    q, par = rows(), params(*binary)
    out = np.zeros((len(LM), len(q), 2))
    lib.modes_eval(dp(par), use_hm, dp(q), len(q), ctypes.c_double(0.3), dp(out))
    got = out[..., 0] + 1j * out[..., 1]
    ref = oracle_modes(oracle, *binary, use_hm)
    for k, lm in enumerate(LM):
        assert np.max(np.abs(got[k] - ref[k])) <= 1e-12 * np.max(np.abs(ref[k])), (lm, use_hm)
