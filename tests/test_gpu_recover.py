"""A context whose contact rebuild stopped at a barrier recovers through a
snapshot and continues as an untouched one does, to the bit."""
import numpy as np
import pytest

from test_gpu_contact import _packing

pytestmark = pytest.mark.gpu

STEPS = 90  # more than two search intervals


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_stopped_rebuild_then_snapshot(prec, tmp_path):
    from peridem_b200 import api
    from peridem_b200.model import GpuDEMModel, PREC_FP64, PREC_MIXED
    p = PREC_FP64 if prec == "fp64" else PREC_MIXED
    sc = _packing(40, 10, 18e-3)
    path = str(tmp_path / "state.pdsnap")

    def new():
        return GpuDEMModel(sc, precision=p, build_neighbors=True, compute_mx=True)

    a = new()
    try:
        a.integrate_begin()
        a.integrate_step(5)
        a.save_state(path)
        a.integrate_step(STEPS)
        a.sync()
        want = {k: a.field(k) for k in ("x", "u", "v", "f", "bonds")}
        rows = a.contact_lists()
    finally:
        a.close()
    b = new()  # its first lists are built
    try:
        # the blocks that come first to the rebuild's first barrier give up at
        # once: nodes are counted in their cells, the lists are not built
        b._check(b.lib.pdgpu_set_barrier_limit(b.ctx, 0))
        with pytest.raises(api.PdgpuError, match="gave up waiting"):
            b.integrate_begin()
        b._check(b.lib.pdgpu_set_barrier_limit(b.ctx, 30 * 10**9))
        b.load_state(path)
        b.integrate_step(STEPS)
        b.sync()
        for k, v in want.items():
            assert np.array_equal(b.field(k), v), k
        got = b.contact_lists()
        assert rows[1].size and np.array_equal(got[0], rows[0]) and np.array_equal(got[1], rows[1])
    finally:
        b.close()
