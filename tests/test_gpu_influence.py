"""An influence function set after the first evaluation holds for the next one
(FP64 form), as one set before."""
import numpy as np
import pytest

from test_gpu_bonds_fp64 import LAWS, _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first,then", [(1, 2), (2, 0), (0, 2)])
@pytest.mark.parametrize("law", LAWS)
def test_influence_set_again(law, first, then):
    import ctypes
    from peridem_b200.model import GpuDEMModel, PREC_FP64
    a, b, other = _scene(2, law, inf_type=first), _scene(2, law, inf_type=first), _scene(2, law, inf_type=then)
    b.inf_type, b.inf_params = other.inf_type, other.inf_params  # all other constants stay
    m, n = GpuDEMModel(a, precision=PREC_FP64), GpuDEMModel(b, precision=PREC_FP64)
    try:
        m.compute_pd_forces()
        old = m.field("f")
        par = (ctypes.c_double * 2)(*[float(v) for v in b.inf_params])
        m._check(m.lib.pdgpu_set_influence(m.ctx, int(b.inf_type), par))
        m.set_field("bonds", a.bond_state)
        m.compute_pd_forces()
        n.compute_pd_forces()
        f = n.field("f")
        assert np.array_equal(m.field("f"), f) and not np.array_equal(old, f)
    finally:
        m.close()
        n.close()
