"""Rounding of the CFL rate against extended precision, rms over many levels.
Bound: the rate's error with every quotient a division, 2.8e-16 over these
levels (tables rounded to doubles in all)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import gpu_available

pytestmark = pytest.mark.gpu

if gpu_available():
    import heliocubed_b200 as hc


def test_rate_is_as_accurate_as_with_divisions(oracle_lib):
    if not gpu_available():
        pytest.skip("no CUDA device")
    err = []
    for nr, na in ((20, 16), (33, 21), (45, 33)):
        sh = hc.Shell(hc.Params(nr=nr, na=na))
        orc = oracle_lib.OracleLevel(oracle_lib.make_params(nr=nr, na=na))
        for seed in range(60):
            ju = sh.init_perturbed_wind(seed)
            err.append(orc.inv_dt_error(ju.cpu().numpy(), sh.inv_dt_max(ju).item()))
    assert np.sqrt(np.mean(np.square(err))) <= 2.8e-16
