"""A model keeps running beside a later one whose bond tiles need less shared
memory: the limit of a kernel is the process's, not the model's."""
import numpy as np
import pytest

from test_gpu_bonds_fp64 import _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("dim", [2, 3])
def test_smaller_tiles_after_larger(dim, prec):
    from peridem_b200.model import GpuDEMModel, PREC_FP64, PREC_MIXED
    p = PREC_FP64 if prec == "fp64" else PREC_MIXED
    sc = _scene(dim, "PDState")
    # 4 lanes: 512 nodes a tile against 4 (above and below 48 KB in 3-D)
    a = GpuDEMModel(sc, precision=p, pd_lanes=4, tile_nodes=512)
    try:
        a.compute_pd_forces()
        want = a.field("f")
        b = GpuDEMModel(sc, precision=p, pd_lanes=4, tile_nodes=4)
        try:
            b.compute_pd_forces()
            a.set_field("bonds", sc.bond_state)
            a.compute_pd_forces()
            assert np.any(want) and np.array_equal(a.field("f"), want)
            assert np.array_equal(b.field("f"), want)
        finally:
            b.close()
        a.integrate_begin()
        a.integrate_step(4, graph_steps=2)
        a.sync()
    finally:
        a.close()
