"""Steps replayed from a graph of several steps, whose inner steps end and begin
in one kernel, against the same steps issued one by one: the same operations in
the same order, so every field, the test history and the scalars are equal to
the bit.  The graph lengths put test-output steps (every tenth) inside a graph
and at its end."""
import numpy as np
import pytest

import scenarios
from peridem_b200 import scene as scn

pytestmark = pytest.mark.gpu

CASES = dict(scenarios.CASES)
CASES["two_particle_pmb_verlet"] = (lambda: _verlet(scn.two_particle(h_div=7, material="PMBBond", v0=-1.0,
                                                                     gap=0.02e-3 / 7)), 60, [])


def _verlet(spec):
    spec.time_scheme = "velocity_verlet"
    return spec


def _run(sc, prec, steps, graph_steps):
    from peridem_b200.model import GpuDEMModel
    m = GpuDEMModel(sc, precision=prec, build_neighbors=True, compute_mx=True)
    try:
        m.integrate_begin()
        m.integrate_step(steps, graph_steps=graph_steps)
        m.sync()
        out = {k: m.field(k) for k in ("x", "u", "v", "f", "Z", "vMag", "bonds")}
        out["history"] = m.history()
        out["scalars"] = np.array([float(v) for _, v in sorted(m.scalars().items())])
        return out
    finally:
        m.close()


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("case", sorted(CASES))
def test_graph_steps_equal_single_steps(case, prec):
    from peridem_b200.model import PREC_FP64, PREC_MIXED
    sc = scn.build_scene(CASES[case][0]())
    sc.test_interval = 10
    p = PREC_FP64 if prec == "fp64" else PREC_MIXED
    a = _run(sc, p, 57, 0)
    for graph_steps in (2, 19):
        b = _run(sc, p, 57, graph_steps)
        for k in a:
            assert np.array_equal(a[k], b[k], equal_nan=True), (case, graph_steps, k)
