"""Damage of nodes whose bonds' stretch overflows is infinite in the FP64 form,
as the quotient is."""
import numpy as np
import pytest

from test_gpu_bonds_fp64 import LAWS, _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes", [4, 16])
@pytest.mark.parametrize("law", LAWS)
@pytest.mark.parametrize("dim", [2, 3])
def test_damage_of_an_overflowed_stretch(dim, law, lanes):
    from peridem_b200.model import GpuDEMModel, PREC_FP64
    sc = _scene(dim, law)
    at = int(sc.p_center[np.flatnonzero(sc.p_compute_force)[0]])
    sc.u[at, :dim] = (1e306, 1.5e306, 2e306)[:dim]
    i = np.repeat(np.arange(sc.n_nodes), np.diff(sc.pd_rowptr.astype(np.int64)))
    j = sc.pd_col.astype(np.int64)
    d, e = sc.xref[j] - sc.xref[i], sc.u[j] - sc.u[i]
    with np.errstate(over="ignore"):
        r2 = (d * d).sum(1)
        y = d + e
        s = (d * e).sum(1) / r2 if law == "RNPBond" else (np.sqrt((y * y).sum(1)) - np.sqrt(r2)) / np.sqrt(r2)
    want = np.zeros(sc.n_nodes, dtype=bool)
    want[i[np.abs(s) > 1e60]] = True  # damage is kept as a float
    assert 10 < want.sum() < sc.n_nodes // 2
    m = GpuDEMModel(sc, precision=PREC_FP64, pd_lanes=lanes)
    try:
        m.compute_pd_forces()
        z = m.field("Z")
    finally:
        m.close()
    assert np.array_equal(np.isinf(z), want)
    assert np.all(z[~want] < 1e6)
