"""The transforms' wide CTAs (few large planes) against the FP64 oracle: planes just below and
at the size from which they are used, odd and with a prime stage, and a batch with too many."""
import numpy as np
import pytest

import atmmetaforce as atm
import oracle as O
from atmmetaforce import synthetic as S

pytestmark = pytest.mark.gpu

U_TOL, F_TOL = 0.01, 1e-4  # kJ/mol, force RMS relative: the parity tests' tolerances


@pytest.mark.parametrize("grid,replicas", [((50, 54, 54), 1), ((53, 55, 52), 2), ((56, 57, 68), 1), ((20, 96, 90), 1),
                                           ((88, 56, 56), 2)])
@pytest.mark.parametrize("diff", [0, 1], ids=["two-states", "difference"])
def test_few_large_planes(grid, replicas, diff):
    cases = []
    for k in range(replicas):
        c = S.water_ligand_box(1100, 2.25, [9], [(1.1, 1.0, 1.2)], S.PME, 0.9, seed=80 + k)
        c.spec.grid = grid
        cases.append(c)
    b = atm.ReplicaBatch([atm.system_from_case(c)[0] for c in cases], 0, {"DifferencePath": diff})
    E, F, r = b.evaluate(np.concatenate([c.pos for c in cases]))
    for k, c in enumerate(cases):
        ref = O.atm_eval(c.spec, c.pos, c.displ, c.params)
        f = F[b.offsets[k]:b.offsets[k + 1]]
        assert abs(r[k]["pert"] - ref["usc"]) <= U_TOL
        assert np.sqrt(((f - ref["forces"]) ** 2).sum() / (ref["forces"] ** 2).sum()) <= F_TOL
