"""The FP32 bond loop and PD state pre-pass over lanes per node and tile sizes,
against one lane per node (2-D) or four (3-D) on the same state.

Stretch and damage of a bond do not depend on the launch shape, so damage and
bond states are equal; forces are FP32 sums of at most 122 terms in another
order: 122 * 2^-24 of sum|terms|, which the rough states used keep below 10
times the largest force: 1e-4.
"""
import numpy as np
import pytest

from test_gpu_bonds_fp64 import LAWS, _scene

pytestmark = pytest.mark.gpu


def _run(sc, **kw):
    from peridem_b200.model import GpuDEMModel, PREC_MIXED
    m = GpuDEMModel(sc, precision=PREC_MIXED, **kw)
    try:
        m.set_field("u", sc.u)
        m.set_field("bonds", sc.bond_state)
        m.compute_pd_forces()
        return m.field("f"), m.field("Z"), m.field("bonds")
    finally:
        m.close()


@pytest.mark.parametrize("lanes,tile", [(1, 1), (1, 130), (2, 65), (4, 127), (8, 33), (16, 9), (32, 3)])
@pytest.mark.parametrize("law", LAWS)
@pytest.mark.parametrize("dim", [2, 3])
def test_launch_shapes_agree(dim, law, lanes, tile):
    sc = _scene(dim, law, inf_type=2 if lanes == 8 else 1)
    f0, z0, b0 = _run(sc)
    f, z, b = _run(sc, pd_lanes=lanes, tile_nodes=tile)
    assert np.array_equal(b, b0), int(np.sum(b != b0))
    assert np.array_equal(z, z0)
    assert np.max(np.abs(f - f0)) <= 1e-4 * np.max(np.abs(f0))
