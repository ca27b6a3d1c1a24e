"""The launch variants of the bond loops that depend on a scene's sizes, against
the variant that small scenes take, at the same lanes per node: 32-bit
neighbour columns (a body of more than 65 536 nodes), and the levels of the FP64
form's shared-memory stage (a wide window leaves node factors, dilatations and
bond data in global memory).

A node's bonds are summed in the same order by the same operations, so
everything is equal to the bit.
"""
import copy

import numpy as np
import pytest

from test_gpu_bonds_fp64 import LAWS, _scene

pytestmark = pytest.mark.gpu

BIG = 65537


def _with_big_body(sc):
    """The scene and, behind it, a body of 65 537 nodes without bonds."""
    s = copy.copy(sc)
    n, far = sc.n_nodes, sc.xref.max(axis=0) + 1e-2
    line = np.tile(far, (BIG, 1))
    line[:, 0] += 1e-4 * np.arange(BIG)
    line[:, sc.dim:] = 0.0
    s.xref, s.x = np.concatenate([sc.xref, line]), np.concatenate([sc.x, line])
    s.u = np.concatenate([sc.u, np.zeros((BIG, 3))])
    s.v = None
    for name, tail in (("vol", 1e-8), ("mx", 1.0), ("fix", 0), ("ptid", sc.n_particles)):
        a = getattr(sc, name)
        setattr(s, name, np.concatenate([a, np.full(BIG, tail, dtype=a.dtype)]))
    live = int(np.flatnonzero(sc.p_compute_force)[0])
    for name in vars(sc):
        a = getattr(sc, name)
        if name.startswith("p_") and isinstance(a, np.ndarray):
            setattr(s, name, np.concatenate([a, a[live:live + 1]]))
    s.p_start[-1], s.p_end[-1], s.p_center[-1] = n, n + BIG, n
    s.pd_rowptr = np.concatenate([sc.pd_rowptr, np.full(BIG, sc.pd_rowptr[-1], dtype=sc.pd_rowptr.dtype)])
    return s


def _run(sc, prec, **kw):
    from peridem_b200.model import GpuDEMModel, PREC_FP64, PREC_MIXED
    m = GpuDEMModel(sc, precision=PREC_FP64 if prec == "fp64" else PREC_MIXED, **kw)
    try:
        m.compute_pd_forces()
        return {k: m.field(k) for k in ("f", "Z", "bonds", "theta")}
    finally:
        m.close()


@pytest.mark.parametrize("prec,lanes,tile", [("fp64", 4, 0), ("fp64", 8, 129), ("fp64", 16, 17), ("fp64", 32, 5),
                                             ("mixed", 1, 130), ("mixed", 4, 0), ("mixed", 8, 33)])
@pytest.mark.parametrize("law", LAWS)
@pytest.mark.parametrize("dim", [2, 3])
def test_columns_of_32_bits(dim, law, prec, lanes, tile):
    sc = _scene(dim, law, inf_type=2 if lanes == 8 else 1)
    big = _with_big_body(sc)
    a, b = (_run(s, prec, pd_lanes=lanes, tile_nodes=tile) for s in (sc, big))
    n = sc.n_nodes
    assert np.any(a["f"]) and a["bonds"].sum() > 0
    assert np.array_equal(a["bonds"], b["bonds"])
    for k in ("f", "Z", "theta"):
        assert np.array_equal(a[k], b[k][:n]), k
        assert not np.any(b[k][n:]), k


def _tile_bytes(sc, nodes, keep):
    """Shared memory of the widest tile of `nodes` nodes with what `keep` names
    beside the window (1 node factors, 2 dilatations, 4 bond data), 3-D PD state,
    16-bit columns."""
    rp, col, most = sc.pd_rowptr.astype(np.int64), sc.pd_col.astype(np.int64), 0
    for p in np.flatnonzero(sc.p_compute_force):
        for b in range(int(sc.p_start[p]), int(sc.p_end[p]), nodes):
            e = min(b + nodes, int(sc.p_end[p]))
            k0, k1 = rp[b], rp[e]
            w = max(e, col[k0:k1].max() + 1) - min(b, col[k0:k1].min())
            n = 48 * w + (8 * w + 15) // 16 * 16
            if keep & 4:
                n += 2 * ((k1 + 7) // 8 * 8 - k0 // 8 * 8) + 4 * (((k1 + 31) // 32 + 3) // 4 * 4 - (k0 >> 5) // 4 * 4)
                n += 8 * ((e + 2) // 2 * 2 - b // 2 * 2)
            n += ((8 * w + 15) // 16 * 16 if keep & 2 else 0) + (16 * w if keep & 1 else 0)
            most = max(most, n)
    return most


@pytest.fixture(scope="module")
def wide():
    """A PD-state sphere of R / h = 10."""
    import pdoracle
    from peridem_b200 import scene as scn
    sc = scn.build_scene(scn.column_3d(n_spheres=1, median_r=1e-3, sigma=0.0, h_div=10, box=(3e-3, 3e-3, 6e-3), seed=1,
                                       material="PDState"))
    sc.multi_particle, sc.gravity, sc.ubc, sc.test = False, np.zeros(3), [], 0
    sc.pd_rowptr, sc.pd_col = pdoracle.build_pd_neighbors(sc)
    sc.mx = pdoracle.compute_mx(sc)
    rng = np.random.default_rng(7)
    h = float(sc.p_h[np.flatnonzero(sc.p_compute_force)[0]])
    sc.u = 0.01 * h * rng.normal(size=sc.xref.shape) * (sc.p_compute_force[sc.ptid] != 0)[:, None]
    sc.x = sc.xref + sc.u
    return sc


@pytest.mark.parametrize("lanes", [4, 8, 16])
def test_stage_levels(wide, lanes):
    room = 226 * 1024
    ref = None
    for nodes, keep in ((128, 7), (512, 6), (640, 4), (768, 0)):
        assert next(k for k in (7, 6, 4, 0) if _tile_bytes(wide, nodes, k) <= room) == keep
        got = _run(wide, "fp64", pd_lanes=lanes, tile_nodes=nodes)
        ref = ref or got
        assert 0 < ref["bonds"].sum() < wide.n_bonds and np.any(ref["theta"])
        for k, v in ref.items():
            assert np.array_equal(got[k], v), (nodes, k)
