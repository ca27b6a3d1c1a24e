"""The FP64 bond loop and PD state pre-pass over their tile shapes and
launch variants, against the oracle's per-bond restatement of the reference.

Forces of a node are sums of at most 122 terms whose order differs; each term
is the oracle's to the bit except RNP's exp().  122 * 2^-53 * sum|terms| is
below 1e-12 of the largest force for the states used (terms do not exceed 70
times the largest sum), the tolerance of the parity tests.  Damage to the
reference's own 2e-5; bond states equal.
"""
import numpy as np
import pytest

from peridem_b200 import scene as scn

pytestmark = pytest.mark.gpu

LAWS = ("RNPBond", "PMBBond", "PDElasticBond", "PDState")
R = 1e-3


def _scene(dim, law, inf_type=1):
    """A scene of free bodies (no contact, no gravity) with a rough, partly
    overstretched displacement and some bonds broken from both ends."""
    import pdoracle
    if dim == 2:
        spec = scn.compressive_2d(n_particles=3, r_range=(R, 1.2 * R), h_div=7, width=8e-3, seed=3, material=law)
    else:
        spec = scn.column_3d(n_spheres=2, median_r=R, sigma=0.1, h_div=4, box=(3e-3, 3e-3, 6e-3), seed=1,
                             material=law)
    for z in spec.zones:
        z.material.influence_type = inf_type
    sc = scn.build_scene(spec)
    sc.multi_particle, sc.gravity, sc.ubc, sc.test = False, np.zeros(3), [], 0
    sc.pd_rowptr, sc.pd_col = pdoracle.build_pd_neighbors(sc)
    sc.mx = pdoracle.compute_mx(sc)
    rng = np.random.default_rng(5)
    owner = sc.ptid.astype(np.int64)
    h = sc.p_h[owner][:, None]
    rel = sc.xref - sc.xref[sc.p_center][owner]
    e = rng.uniform(-3e-2, 3e-2, (sc.n_particles, 3, 3))
    sc.u = np.einsum("nab,nb->na", e[owner], rel) + 2e-3 * h * rng.normal(size=rel.shape)
    sc.u[:, dim:] = 0.0
    sc.x = sc.xref + sc.u
    rp, col = sc.pd_rowptr.astype(np.int64), sc.pd_col.astype(np.int64)
    i = np.repeat(np.arange(sc.n_nodes), np.diff(rp))
    sc.bond_state = (((i * col) % 53 == 0) & (rel[i, 0] > 0) & (rel[col, 0] > 0)).astype(np.uint8)
    return sc


def _oracle(sc):
    import pdoracle
    ora = pdoracle.Oracle(sc)
    N = sc.n_nodes
    for name, a in (("po_u", sc.u), ("po_x", sc.x)):
        np.ctypeslib.as_array(getattr(ora.L, name)(ora.m), shape=(N, 3))[:] = a
    np.ctypeslib.as_array(ora.L.po_bonds(ora.m), shape=(sc.n_bonds,))[:] = sc.bond_state
    ora.integrate_begin()
    return ora.field("f"), ora.field("Z"), ora.field("bonds")


def _run(sc, **kw):
    from peridem_b200.model import GpuDEMModel, PREC_FP64
    m = GpuDEMModel(sc, precision=PREC_FP64, **kw)
    try:
        m.integrate_begin()
        return m.field("f"), m.field("Z"), m.field("bonds"), m.field("theta")
    finally:
        m.close()


@pytest.mark.parametrize("lanes,tile", [(0, 0), (4, 129), (8, 33), (16, 16), (32, 5)])
@pytest.mark.parametrize("law", LAWS)
@pytest.mark.parametrize("dim", [2, 3])
def test_tile_shapes_match_oracle(dim, law, lanes, tile):
    sc = _scene(dim, law, inf_type={0: 1, 4: 1, 8: 0, 16: 2, 32: 1}[lanes])
    f, z, b, th = _run(sc, pd_lanes=lanes, tile_nodes=tile)
    fo, zo, bo = _oracle(sc)
    assert bo.sum() > sc.bond_state.sum() or law == "PDElasticBond", "no bond breaks in this state"
    assert np.array_equal(b, bo), int(np.sum(b != bo))
    ef = float(np.max(np.abs(f - fo)) / np.max(np.abs(fo)))
    ez = float(np.max(np.abs(z - zo) / np.maximum(np.abs(zo), 1e-6)))
    print(f"{law} {dim}-D lanes {lanes} tile {tile}: f {ef:.1e} Z {ez:.1e}")
    assert ef <= 1e-12 and ez <= 2e-5, (ef, ez)


@pytest.mark.parametrize("law", ("PMBBond", "PDElasticBond", "PDState"))
@pytest.mark.parametrize("dim", [2, 3])
def test_lengths_beyond_the_unchecked_root(dim, law):
    """Lengths scaled by 2^460 (and volumes by 2^-460, which keeps m_x and the
    forces in range) take the launch that checks every root's range and reads
    the bond data from global memory.  A power of two scales every operand of
    these laws by one, so stretches, dilatations, damage and bond states are
    the same to the bit and forces by 2^-460."""
    s = 2.0 ** 460
    sc, big = _scene(dim, law), _scene(dim, law)
    for name in ("xref", "u", "x", "mx", "p_horizon", "p_h", "p_rc"):
        setattr(big, name, getattr(big, name) * s)
    big.vol, big.p_kn = big.vol / s, big.p_kn / s
    f, z, b, th = _run(sc, pd_lanes=8)
    F, Z, B, TH = _run(big, pd_lanes=8)
    assert np.any(f) and np.array_equal(F, f / s)
    assert np.array_equal(Z, z) and np.array_equal(B, b) and np.array_equal(TH, th)
