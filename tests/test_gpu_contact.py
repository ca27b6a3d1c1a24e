"""The contact pass and the particle damping against the oracle, at the sizes
where their launch shapes change: more particles than a CTA stages at once,
more wall pairs than one warp orders, several scenes per CTA, and 8, 16 or 32
contact nodes per warp.

Forces are compared to 1e-12 of the largest: sums of at most a few hundred
FP64 terms, each below 20 times the largest total, in another order
(400 * 20 * 2^-53 = 9e-13).
"""
import numpy as np
import pytest

from peridem_b200 import scene as scn

pytestmark = pytest.mark.gpu

R = 1e-3


def _moving(sc, seed=1, shift=0.03):
    """Bodies shifted by a few per cent of the mesh size and moving."""
    rng = np.random.default_rng(seed)
    owner = sc.ptid.astype(np.int64)
    on = ((sc.p_type == 0) & (sc.p_compute_force != 0))[owner][:, None]
    u = rng.normal(0.0, shift, (sc.n_particles, 3))[owner] * sc.p_h[owner][:, None]
    v = rng.normal(0.0, 0.3, (sc.n_particles, 3))[owner] + rng.normal(0.0, 0.1, sc.xref.shape)
    sc.u, sc.v = np.where(on, u, 0.0), np.where(on, v, 0.0)
    sc.u[:, sc.dim:] = sc.v[:, sc.dim:] = 0.0
    sc.x = sc.xref + sc.u
    sc.ubc, sc.test = [], 0
    return sc


def _packing(n, h_div, width, radius_factor=0.95, gap=0.96, **kw):
    spec = scn.compressive_2d(n, r_range=(0.96 * R, R), h_div=h_div, width=width, gap=gap * 0.96 * R / h_div,
                              seed=2, **kw)
    for c in spec.contact.values():
        c.radius_factor = radius_factor
    return _moving(scn.build_scene(spec))


def _force(sc, **kw):
    from peridem_b200.model import GpuDEMModel, PREC_FP64
    if sc.pd_rowptr is None:
        kw["build_neighbors"] = True
    m = GpuDEMModel(sc, precision=PREC_FP64, **kw)
    try:
        m.integrate_begin()
        return m.field("f"), m.scalars()
    finally:
        m.close()


def _oracle_force(sc):
    import pdoracle
    ora = pdoracle.Oracle(sc)
    for name, a in (("po_u", sc.u), ("po_x", sc.x), ("po_v", sc.v)):
        np.ctypeslib.as_array(getattr(ora.L, name)(ora.m), shape=(sc.n_nodes, 3))[:] = a
    ora.integrate_begin()
    return ora.field("f")


SCENES = {
    "300 particles": lambda: _packing(300, 4, 40e-3),
    "wide wall contact": lambda: _packing(5, 10, 7e-3, radius_factor=4.0, gap=1.5, search_factor=2.0),
    "3-D": lambda: _moving(scn.build_scene(scn.column_3d(12, median_r=R, sigma=0.05, h_div=4, footprint=(2, 2),
                                                         seed=3, material="PDElasticBond")), shift=0.3),
}


@pytest.mark.parametrize("lanes", [1, 4])
@pytest.mark.parametrize("name", sorted(SCENES))
def test_forces_match_oracle(name, lanes):
    sc = SCENES[name]()
    fo = _oracle_force(sc)
    f, s = _force(sc, contact_lanes=lanes, wall_pair_capacity=4096)
    assert s["contact_entries"] > 0
    e = float(np.max(np.abs(f - fo)) / np.max(np.abs(fo)))
    print(f"{name}: {sc.n_particles} particles, {s['contact_entries']} candidates, f {e:.1e}")
    assert e <= 1e-12


@pytest.mark.parametrize("n,ctas", [(40, 1), (260, 1), (260, 4)])
def test_nodes_per_warp(n, ctas):
    """8, 16 and 32 contact nodes per warp against one node per lane group."""
    sc = _packing(n, 18, 18e-3 if n < 100 else 40e-3)
    a, s = _force(sc, contact_lanes=1, contact_ctas=ctas)
    b, _ = _force(sc, contact_lanes=2)
    print(f"{n} particles, {s['contact_entries']} candidates")
    assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b))


def test_damping_of_several_scenes_per_cta():
    """Scenes of a batch give the forces of the same scenes alone."""
    alone = [_packing(n, 5, 12e-3) for n in (3, 21, 6, 9)]
    for k, sc in enumerate(alone):
        sc.test = 2
    both = scn.merge_scenes(alone)
    both.u = np.concatenate([sc.u for sc in alone])
    both.v = np.concatenate([sc.v for sc in alone])
    f, _ = _force(both)
    at = 0
    for sc in alone:
        g, _ = _force(sc)
        e = np.max(np.abs(f[at:at + sc.n_nodes] - g)) / np.max(np.abs(g))
        # the shift of a scene moves coordinates by their rounding, 2^-53 of
        # 0.1 m against distances of 1e-4 m
        assert e <= 1e-9, e
        at += sc.n_nodes
