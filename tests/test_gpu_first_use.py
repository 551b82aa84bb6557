"""The first work on new buffers: what fills them is complete before a stream that has no
order with the default one reads it."""
import numpy as np
import pytest

import atmmetaforce as atm
from atmmetaforce import synthetic as S

pytestmark = pytest.mark.gpu


def test_first_evaluation_launched_eagerly():
    """Kernel by kernel (no graph to record, which would leave the fills time to finish),
    with kept lists, whose decision counts from a zeroed status."""
    c = S.water_ligand_box(1500, 2.5, [9], [(1.1, 1.0, 1.2)], S.CUTOFF_PERIODIC, 0.9, seed=150)
    sys_ = atm.system_from_case(c)[0]
    want = atm.ReplicaBatch([sys_], 0, {"ListSkin": 0.1}).evaluate(c.pos, as_array=True)
    for _ in range(20):
        b = atm.ReplicaBatch([sys_], 0, {"ListSkin": 0.1})
        b.setProfiling(True)
        E, F, r = b.evaluate(c.pos, as_array=True)
        assert np.array_equal(F, want[1]) and np.array_equal(r, want[2])
        assert b.listInfo()["builds"] == 1


def test_first_steps_from_new_positions():
    c = S.water_ligand_box(1500, 2.5, [9], [(1.1, 1.0, 1.2)], S.PME, 0.9, seed=151, use_disp_corr=False)
    terms, _ = S.md_terms_ligand_centroid(c)
    sys_ = atm.md_system_from_case(c, terms)[0]
    vel = np.random.default_rng(1).normal(0.0, 0.1, c.pos.shape)
    out = []
    for _ in range(5):
        integ = atm.LangevinIntegrator(300.0, 1.0, 0.0005)
        integ.setRandomNumberSeed(5)
        sim = atm.ReplicaSimulation([sys_], integ, 0, {"ListSkin": 0.1})
        for _ in range(2):  # the second time over work of the first
            sim.setPositions(c.pos)
            sim.setVelocities(vel)
            sim.step(3)
        s = sim.getState(getPositions=True, getVelocities=True)
        out.append((s.getPositions(), s.getVelocities()))
    for x, v in out[1:]:
        assert np.array_equal(x, out[0][0]) and np.array_equal(v, out[0][1])
