"""The step kernels' divisions: the device functions on operands where they can go
wrong, and fields of subnormal values, whose high words are zero like a zero's."""
import ctypes

import numpy as np
import pytest

import pyoracle
from test_gpu_pairs import array_mesh, run_both
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


QUOTIENTS = ["div_fast", "div_any", "rcp", "div3", "div6", "limiter_ratio", "courant", "variation"]


def quotients(lib, kind, fp32, n, seed):
    wrong, flagged, ex = ctypes.c_longlong(-1), ctypes.c_longlong(-1), np.zeros(4)
    assert lib.tracer_selftest_quotients(QUOTIENTS.index(kind), fp32, n, seed, ctypes.byref(wrong), ctypes.byref(flagged),
                                         ex.ctypes.data_as(ctypes.c_void_p)) == 0
    return wrong.value, flagged.value, ex


@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("kind", QUOTIENTS[:5])
def test_straight_line_quotients(lib, kind, fp32):
    """Every result that is not flagged for a plain division is the IEEE quotient, on
    2^26 operand pairs; ordinary operands are flagged only for a divisor whose
    significand's high word (FP32: whole significand) is all ones, 1 in 2^20 (2^23)."""
    n = 1 << 26
    wrong, flagged, ex = quotients(lib, kind, fp32, n, 77 + fp32)
    assert wrong == 0, f"a={ex[0]!r} b={ex[1]!r} got={ex[2]!r} expected={ex[3]!r}"
    assert flagged <= (4 * n / 2 ** 20 if kind in ("div_any", "rcp") else 0)


@pytest.mark.parametrize("kind,fp32", [("limiter_ratio", 0), ("limiter_ratio", 1), ("courant", 1), ("variation", 1)])
def test_quotients_of_the_limiter_and_the_features(lib, kind, fp32):
    """FP64 quotients in the limiter ratios of every precision, IEEE quotients in the
    learned flux's features: the bits of the same expressions with plain divisions."""
    n = 1 << 26
    wrong, flagged, ex = quotients(lib, kind, fp32, n, 5)
    assert wrong == 0, f"a={ex[0]!r} b={ex[1]!r} got={ex[2]!r} expected={ex[3]!r}"
    assert flagged <= 4 * n / 2 ** 20


@pytest.mark.parametrize("h", [0.0, 5e-324, 1e-200, 1e200])
@pytest.mark.parametrize("scheme", [("MUSCL", "PPM", "FCT"), ("MUSCL", "PPM", "NONE"), ("MFCT", "QR4C", "FCT")])
def test_layers_of_extreme_thickness(api, oracle, h, scheme):
    """One old thickness (hnode, the divisor of PPM's Courant number) of zero, a
    subnormal and far outside any ocean, the same at every node, so that the level
    tables hold: the oracle's bits."""
    K, uv, w, T, S, dt = synth_case(api, 13, 12, 21, True, 9)
    names = ["elem2D_nodes", "edges", "edge_tri", "nlevels", "nlevels_nod2D", "ring_num", "ring_elem", "elem_area", "area",
             "areasvol", "edge_dxdy", "edge_cross_dxdy", "gradient_sca", "zbar", "hnode", "hnode_new", "helem", "coord"]
    arrays = {n: api.mesh_array(n) for n in names}
    arrays["elem_cos"] = np.ones(api.mesh_dims()["elem2D"])
    flat = np.array(arrays["hnode"])
    layers = flat.reshape(-1, 20)  # 20 layers of each node one after the other
    layers[:, 2] = h
    layers[:, 5] = h
    arrays["hnode"] = layers.reshape(arrays["hnode"].shape)
    m = array_mesh(api, oracle, arrays, 1.0e5, 1.0e5)
    with np.errstate(all="ignore"):
        run_both(api, m, [T, S], uv, w, dt, scheme, 1)
