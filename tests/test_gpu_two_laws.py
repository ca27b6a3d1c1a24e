"""Two material laws in one scene, FP64 form: a launch per law, a shared-memory
stage that holds the widest tile of either, the state pre-pass by the first
particle's law.  Against the oracle, tolerance as in test_gpu_bonds_fp64.py.
"""
import numpy as np
import pytest

from peridem_b200 import scene as scn
from test_gpu_bonds_fp64 import R, _oracle, _run

pytestmark = pytest.mark.gpu


def _scene(first, second):
    import pdoracle

    def spec(law):
        return scn.compressive_2d(n_particles=4, r_range=(R, 1.2 * R), h_div=7, width=8e-3, seed=3, material=law)
    s = spec(first)
    last = [k for k, z in enumerate(s.zones) if not z.is_wall][-1]
    s.zones[last].material = spec(second).zones[last].material
    sc = scn.build_scene(s)
    sc.multi_particle, sc.gravity, sc.ubc, sc.test = False, np.zeros(3), [], 0
    sc.pd_rowptr, sc.pd_col = pdoracle.build_pd_neighbors(sc)
    sc.mx = pdoracle.compute_mx(sc)
    rng = np.random.default_rng(2)
    owner = sc.ptid.astype(np.int64)
    rel = sc.xref - sc.xref[sc.p_center][owner]
    e = rng.uniform(-1e-2, 1e-2, (sc.n_particles, 3, 3))
    sc.u = np.einsum("nab,nb->na", e[owner], rel)
    sc.u[:, 2:] = 0.0
    sc.x = sc.xref + sc.u
    sc.bond_state = np.zeros(len(sc.pd_col), dtype=np.uint8)
    return sc


@pytest.mark.parametrize("lanes,tile", [(0, 0), (8, 257)])
@pytest.mark.parametrize("first,second", [("RNPBond", "PDState"), ("PDState", "PMBBond"), ("PDElasticBond", "PDState"),
                                          ("PMBBond", "RNPBond")])
def test_two_laws(first, second, lanes, tile):
    sc = _scene(first, second)
    assert len(set(sc.p_material[sc.p_compute_force != 0])) == 2
    f, z, b, th = _run(sc, pd_lanes=lanes, tile_nodes=tile)
    fo, zo, bo = _oracle(sc)
    assert np.array_equal(b, bo)
    for law in set(sc.p_material[sc.p_compute_force != 0]):
        on = (sc.p_material[sc.ptid] == law) & (sc.p_compute_force[sc.ptid] != 0)
        assert np.any(fo[on])
        assert np.max(np.abs(f - fo)[on]) <= 1e-12 * np.max(np.abs(fo[on]))
        assert np.max(np.abs(z - zo)[on] / np.maximum(np.abs(zo[on]), 1e-6)) <= 2e-5
