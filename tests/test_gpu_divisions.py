"""The step kernels' divisions: fields of subnormal values, whose high words are
zero like a zero's."""
import numpy as np
import pytest

import pyoracle
from test_gpu_pairs import run_both
from test_gpu_parity import synth_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-308, 1e-313, 1e-317, 1e-322])
@pytest.mark.parametrize("scheme", [("MUSCL", "PPM", "FCT"), ("MFCT", "QR4C", "FCT"), ("MUSCL", "PPM", "NONE")])
@pytest.mark.parametrize("path", ["five", "fused"])
def test_subnormal_fields(api, oracle, scale, scheme, path):
    """Fields whose values, gradients and fluxes are subnormal, down to a few units
    of 2^-1074 and with half the domain at zero: the oracle's bits (no tolerance)."""
    K, uv, w, T, S, dt = synth_case(api, 14, 11, 16, True, 3)
    m = pyoracle.OracleMesh(oracle, 14, 11, 16, periodic=True, full_rings=True, node_K=K)
    T, S = np.asfortranarray(T * scale), np.asfortranarray(S * scale)
    S[:, : S.shape[1] // 2] = 0.0
    api.set_step_path(path)
    try:
        run_both(api, m, [T, S], uv, w, dt, scheme, 3)
    finally:
        api.set_step_path("five")
