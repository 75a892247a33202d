"""The step kernels' level pairs where they can go wrong: column depths around a
pair, a warp (64 levels) and its overlapping pieces, batches of 1 to 5 tracers,
meshes whose thicknesses differ from node to node (no level tables), operands
outside the fast divisions' range, caller buffers without vector alignment, and
the batch's member path over calls that leave its buffers swapped.  FP64 results
are compared bit for bit with the oracle, which evaluates the reference's
operations in their order, so no tolerance is involved."""
import ctypes

import numpy as np
import pytest

import pyoracle
from test_gpu_parity import assert_bitwise, synth_case

pytestmark = pytest.mark.gpu


def run_both(api, m, tracers, uv, w, dt, scheme, steps, refresh=True):
    """Steps tracers on the loaded mesh and on the oracle's mesh m, bit for bit."""
    api.allocate_tracers(len(tracers))
    for i, T in enumerate(tracers, 1):
        api.set_values(i, T)
        api.set_scheme(i, *scheme)
    api.set_velocity(uv, w)
    api.set_ab_refresh(refresh)
    ref, ab = [T.copy(order="F") for T in tracers], [T.copy(order="F") for T in tracers]
    for s in range(steps):
        api.advect_steps(1, dt)
        for i, T in enumerate(ref):
            m.step(T, T.copy(order="F") if refresh else ab[i], uv, w, dt, *scheme)
            assert_bitwise(api.get_tracer_values(i + 1), T, f"tracer {i + 1} step {s + 1}")


@pytest.mark.parametrize("nl", [3, 4, 5, 34, 64, 65, 66, 67, 96, 130, 200, 577])
@pytest.mark.parametrize("ntr", [1, 2])
def test_column_depths(api, oracle, nl, ntr):
    """2 to 576 layers (the most that a mesh may have) over random bathymetry: odd and even columns, columns that
    just fill a warp and those cut into two and up to ten overlapping pieces."""
    K, uv, w, T, S, dt = synth_case(api, 9, 8, nl, True, nl)
    K[:4] = [nl, max(3, nl - 1), max(3, nl - 2), 3]
    api.init_analytic(9, 8, nl, periodic=True, full_rings=True, node_K=K)
    uv, w = api.synth_velocity(seed=1, umax=1.0, mode2=0.5)
    m = pyoracle.OracleMesh(oracle, 9, 8, nl, periodic=True, full_rings=True, node_K=K)
    for scheme in (("MUSCL", "PPM", "FCT"), ("MFCT", "QR4C", "FCT")):
        run_both(api, m, [T, S][:ntr], uv, w, dt, scheme, 2)


@pytest.mark.parametrize("ntr", [3, 4, 5])
@pytest.mark.parametrize("refresh", [True, False])
def test_batch_sizes(api, oracle, ntr, refresh):
    """Batches of 2 + 1, 4 and 4 + 1 tracers, valuesAB equal to the values or not."""
    K, uv, w, T, S, dt = synth_case(api, 21, 17, 24, False, 5)
    m = pyoracle.OracleMesh(oracle, 21, 17, 24, periodic=False, full_rings=True, node_K=K)
    run_both(api, m, [api.synth_tracer(seed=40 + i, kind=i % 2) for i in range(ntr)], uv, w, dt, ("MUSCL", "PPM", "FCT"), 3,
             refresh)


def array_mesh(api, oracle, arrays, Lx, Ly):
    """The same mesh arrays in the library (tracer_set_mesh_arrays) and the oracle."""
    d = api.mesh_dims()
    num, flat = arrays["ring_num"], arrays["ring_elem"]
    ring = np.zeros((int(num.max()), d["nod2D"]), dtype=np.int32, order="F")
    start = np.concatenate([[0], np.cumsum(num)])
    for n in range(d["nod2D"]):
        ring[: num[n], n] = flat[start[n]:start[n + 1]]
    names = ["elem2D_nodes", "edges", "edge_tri", "nlevels", "nlevels_nod2D", "ring_num", None, "elem_area", "area", "areasvol",
             "edge_dxdy", "edge_cross_dxdy", "gradient_sca", "elem_cos", "zbar", "hnode", "hnode_new", "helem", "coord"]
    keep = [ring if n is None else np.ascontiguousarray(arrays[n]) for n in names]
    rc = api.lib.tracer_set_mesh_arrays(d["nl"], d["nod2D"], d["elem2D"], d["edge2D"], ring.shape[0],
                                        *[a.ctypes.data_as(ctypes.c_void_p) for a in keep], Lx, Ly)
    assert rc == 0, api.lib.tracer_last_error()
    full = dict(arrays)
    for n in ("nlevels_nod2D_min", "edge_up_dn_tri", "nboundary_lay"):
        full[n] = api.mesh_array(n)
    return pyoracle.OracleMesh.from_arrays(oracle, d["nl"], d["nod2D"], d["elem2D"], d["edge2D"], full, periodic=True, Lx=Lx,
                                           Ly=Ly)


@pytest.mark.parametrize("change", ["none", "hnode", "hnode_new", "one_cell"])
@pytest.mark.parametrize("scheme", [("MUSCL", "PPM", "FCT"), ("MUSCL", "PPM", "NONE"), ("UPW1", "UPW1", "FCT")])
def test_thicknesses_of_their_own(api, oracle, change, scheme):
    """Thicknesses that are not the same at every node take the kernels that form
    the PPM weights themselves; uniform ones given as arrays take the level tables."""
    K, uv, w, T, S, dt = synth_case(api, 13, 12, 21, True, 9)
    names = ["elem2D_nodes", "edges", "edge_tri", "nlevels", "nlevels_nod2D", "ring_num", "ring_elem", "elem_area", "area",
             "areasvol", "edge_dxdy", "edge_cross_dxdy", "gradient_sca", "zbar", "hnode", "hnode_new", "helem", "coord"]
    arrays = {n: api.mesh_array(n) for n in names}
    arrays["elem_cos"] = np.ones(api.mesh_dims()["elem2D"])
    rng = np.random.default_rng(3)
    if change == "one_cell":
        arrays["hnode_new"][7 * 20 + 1] *= 1.0 + 2.0 ** -52
    elif change != "none":
        arrays[change] = arrays[change] * rng.uniform(0.5, 1.5, arrays[change].size)
    m = array_mesh(api, oracle, arrays, 1.0e5, 1.0e5)
    run_both(api, m, [T, S], uv, w, dt, scheme, 2)


@pytest.mark.parametrize("scale", [1e-300, 1e-280, 1e-200, 1e160])
@pytest.mark.parametrize("scheme", [("MUSCL", "PPM", "FCT"), ("MFCT", "QR4C", "FCT")])
def test_operands_outside_the_fast_divisions(api, oracle, scale, scheme):
    """Fields below 2^-900, with differences that underflow, whose squares overflow,
    and fields that are zero over half the domain."""
    K, uv, w, T, S, dt = synth_case(api, 14, 11, 16, True, 3)
    m = pyoracle.OracleMesh(oracle, 14, 11, 16, periodic=True, full_rings=True, node_K=K)
    T, S = np.asfortranarray(T * scale), np.asfortranarray(S * scale)
    S[:, : S.shape[1] // 2] = 0.0
    T[3:6, ::3] = 0.0
    run_both(api, m, [T, S], uv, w, dt, scheme, 2)


@pytest.mark.parametrize("refresh", [True, False])
@pytest.mark.parametrize("scheme", [("MUSCL", "PPM", "FCT"), ("MFCT", "QR4C", "NONE"), ("UPW1", "UPW1", "FCT")])
def test_caller_buffers_without_vector_alignment(api, scheme, refresh):
    """tracer_advect_device_noalloc on buffers that are 8- but not 16-byte aligned."""
    import torch
    from test_zz_no_alloc import _padded, _setup
    T, dt = _setup(api, 22, 19, 13, 4, scheme)
    cur, _ = _padded(api, T)
    ab = cur if refresh else cur + 0.25 * torch.sin(torch.arange(cur.numel(), device="cuda", dtype=torch.float64)).reshape(cur.shape)
    got = []
    for offset in (0, 1):
        bufs = [torch.zeros(cur.numel() + 2, dtype=torch.float64, device="cuda")[offset:offset + cur.numel()] for _ in range(3)]
        bufs[0].copy_(cur.reshape(-1))
        bufs[1].copy_(ab.reshape(-1))
        assert all(b.data_ptr() % 16 == 8 * offset for b in bufs)
        torch.cuda.synchronize()
        assert api.lib.tracer_advect_device_noalloc(1, *[ctypes.c_void_p(b.data_ptr()) for b in bufs], dt) == 0
        got.append(bufs[2].cpu().numpy())
    assert np.array_equal(got[0].view(np.uint64), got[1].view(np.uint64))


def test_batch_member_path_keeps_its_state(lib):
    """Odd and even counts, a new velocity, new values, other paths and a new
    configuration between calls: the member path (work arrays and graph kept) gives
    the bits of the persistent path, which keeps nothing."""
    from fesom2_tracer_dwarf_b200 import FESOMTracerAdvection
    from fesom2_tracer_dwarf_b200.batch import TracerBatch
    from fesom2_tracer_dwarf_b200.workloads import layered_flow_case
    api = FESOMTracerAdvection()

    def run(path, graph):
        b, cases = TracerBatch(), []
        for i, (nx, nl, periodic) in enumerate([(33, 12, True), (24, 17, False)]):
            api.cleanup()
            c = layered_flow_case(api, nx, nl, periodic=periodic, seed=i)
            b.add_member(nx, nx, nl, 4, periodic=periodic, node_K=c.K)
            b.set_velocity(i, c.uv, c.w)
            for t in range(1, 5):
                b.set_values(i, t, api.synth_tracer(seed=10 * i + t, kind=t % 2))
            cases.append(c)
        api.cleanup()
        dts = [c.dt for c in cases]
        b.configure(dts)
        out = []

        def take(n, p=path):
            b.set_path(p)
            b.steps(n, graph=graph)
            out.append([b.get_values(i, t) for i in range(2) for t in range(1, 5)])

        for n in (1, 2, 5, 4, 3):
            take(n)
        b.set_velocity(0, 0.5 * cases[0].uv, 0.5 * cases[0].w)
        take(6)
        take(3, "phases")
        take(4)
        b.set_values(1, 3, cases[1].T)
        take(2)
        b.configure([0.5 * d for d in dts])
        take(4)
        b.close()
        return out

    ref = run("phases", False)
    for graph in (False, True):
        for k, (x, y) in enumerate(zip(ref, run("separate", graph))):
            assert all(np.array_equal(u, v) for u, v in zip(x, y)), (graph, k)


@pytest.mark.parametrize("S", [1, 127, 129, 257, 38000])
def test_mlp_gradients_at_tile_edges(lib, S):
    """One sample, one row short of and past a tile, an odd tile count and more tiles
    than CTAs, against the CPU restatement (which rounds weights and activations
    to BF16 alike).  What differs is the hardware tanh (2^-11 relative) in three
    places of each product and activations that round to the neighbouring BF16 (2^-8) on
    it, a few per thousand: 1e-2 of each block's norm holds both."""
    import mlp_oracle as mo
    from test_gpu_mlp import _mlp_case, from_bf16_bits
    X, p = _mlp_case(S, S + 3)
    dy = np.random.default_rng(S).standard_normal(S).astype(np.float32) / S
    g = np.zeros(mo.NPARAMS, dtype=np.float32)
    assert lib.tracer_mlp_grads(X.ctypes.data, dy.ctypes.data, S, p.ctypes.data, g.ctypes.data) == 0
    ref = mo.grads(from_bf16_bits(X), dy, p)
    for name, (a, b) in {"W1": (0, 1024), "b1": (1024, 1088), "W2": (1088, 5184), "b2": (5184, 5248), "w3": (5248, 5312),
                         "b3": (5312, 5313)}.items():
        rel = np.linalg.norm(g[a:b] - ref[a:b]) / (np.linalg.norm(ref[a:b]) + 1e-30)
        assert rel < 1e-2, (name, rel)
