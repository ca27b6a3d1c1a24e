"""Contact nodes per warp (8, 16 or 32, by the nodes that have candidates and
the warps of the launch), each against a node pass with two lanes per node, and
that the three scenes do take the three group sizes.

Tolerance as in test_gpu_contact.py: 1e-12 of the largest force.
"""
import numpy as np
import pytest

from test_gpu_contact import _packing

pytestmark = pytest.mark.gpu


def _force(sc, **kw):
    from peridem_b200.model import GpuDEMModel, PREC_FP64
    m = GpuDEMModel(sc, precision=PREC_FP64, build_neighbors=True, compute_mx=True, **kw)
    try:
        m.integrate_begin()
        return m.field("f"), int(np.count_nonzero(np.diff(m.contact_lists()[0].astype(np.int64))))
    finally:
        m.close()


@pytest.mark.parametrize("n,width,group", [(40, 16e-3, 8), (160, 30e-3, 16), (320, 42e-3, 32)])
def test_each_group_size(n, width, group):
    import torch
    sc = _packing(n, 10, width)
    f, nodes = _force(sc, contact_lanes=1, contact_ctas=1)
    warps = 8 * torch.cuda.get_device_properties(0).multi_processor_count
    assert group == (8 if nodes <= 8 * warps else 16 if nodes <= 16 * warps else 32), (nodes, warps)
    g, _ = _force(sc, contact_lanes=2)
    assert np.any(f) and np.max(np.abs(f - g)) <= 1e-12 * np.max(np.abs(g))
