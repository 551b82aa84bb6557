"""MD steps that are neither recorded nor checked run without the evaluation's force output:
the update merges the forces itself, to the same bits."""
import numpy as np
import pytest

import atmmetaforce as atm
from atmmetaforce import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("diff", [0, 1], ids=["two-states", "difference"])
@pytest.mark.parametrize("direction", [1.0, -1.0])
def test_steps_with_and_without_output_are_the_same_bits(diff, direction):
    """Every step checked (all with output), checks every 7 steps, and records every 3
    steps: positions, velocities, forces and energies of 20 steps, and the records."""
    cases = [S.water_ligand_box(1100 + 3 * k, 2.25, [9], [(1.1, 1.0, 1.2)], S.PME, 0.9, seed=140 + k,
                                params=S.default_params(0.2, 0.4, 0.1, 60.0, 0.5, direction=direction)) for k in range(2)]
    systems = []
    for c in cases:
        terms, _ = S.md_terms_ligand_centroid(c)
        systems.append(atm.md_system_from_case(c, terms)[0])
    out = []
    for check, record in ((1, 0), (7, 0), (20, 3), (1, 3)):
        integ = atm.LangevinIntegrator(300.0, 1.0, 0.0005)
        integ.setRandomNumberSeed(5)
        sim = atm.ReplicaSimulation(systems, integ, 0, {"DifferencePath": diff, "CheckInterval": check, "ListSkin": 0.1})
        sim.setPositions(np.concatenate([c.pos for c in cases]))
        sim.setVelocitiesToTemperature(300.0, 5)
        if record:
            sim.setRecording(record, 16)
        sim.step(20)
        s = sim.getState(getPositions=True, getVelocities=True, getForces=True, getEnergy=True)
        out.append((s.getPositions(), s.getVelocities(), s.getForces(), s.getPotentialEnergy(), s.getKineticEnergy(),
                    sim.getRecords() if record else None))
    for o in out[1:]:
        for a, b in zip(o[:5], out[0][:5]):
            assert np.array_equal(a, b)
    for key in ("steps", "results", "matrices"):
        assert np.array_equal(out[2][5][key], out[3][5][key])
    assert list(out[2][5]["steps"]) == [0, 3, 6, 9, 12, 15, 18]
