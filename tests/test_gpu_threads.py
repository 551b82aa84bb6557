"""Host threads, each with an engine of its own, that build, record and evaluate at once."""
import threading

import numpy as np
import pytest

import atmmetaforce as atm
from atmmetaforce import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fused", [0, 1], ids=["find-tiles", "fused"])
def test_engines_of_several_threads(fused):
    """The first use of every kernel's launch in this process may be any thread's: the
    sizes that a launch takes from the device are each engine's own."""
    cases = [S.water_ligand_box(1100 + 300 * k, 2.25 + 0.2 * k, [9], [(1.1, 1.0, 1.2)], S.PME, 0.9, seed=160 + k)
             for k in range(6)]
    for c, K in zip(cases, (24, 27, 50, 53, 56, 60)):
        c.spec.grid = (K, K, K)
    systems = [atm.system_from_case(c)[0] for c in cases]
    got, errors = [None] * len(cases), []
    start = threading.Barrier(len(cases))

    def work(k):
        try:
            start.wait(60)
            b = atm.ReplicaBatch([systems[k]], 0, {"FusedTiles": fused})
            got[k] = [b.evaluate(cases[k].pos, as_array=True) for _ in range(3)]
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(cases))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for k, c in enumerate(cases):
        E, F, r = atm.ReplicaBatch([systems[k]], 0, {"FusedTiles": fused}).evaluate(c.pos, as_array=True)
        for e, f, q in got[k]:
            assert np.array_equal(f, F) and np.array_equal(q, r)


def test_engines_of_other_grid_sizes_record_at_once():
    """Engines whose transforms and bricks need 10 to 80 KB of shared memory, recorded from
    several threads over and over: none takes back what another's launch needs."""
    cases = [S.water_ligand_box(1100 + 100 * k, 2.25, [9], [(1.1, 1.0, 1.2)], S.PME, 0.9, seed=170 + k) for k in range(4)]
    for c, K in zip(cases, (20, 64, 22, 60)):
        c.spec.grid = (K, K, K)
    systems = [atm.system_from_case(c)[0] for c in cases]

    def evaluate(k, brick):
        return atm.ReplicaBatch([systems[k]], 0, {"SpreadBrick": brick}).evaluate(cases[k].pos, as_array=True)

    want = [evaluate(k, 0) for k in range(len(cases))]
    errors, different = [], [0] * len(cases)
    start = threading.Barrier(len(cases))

    def work(k):
        try:
            start.wait(60)
            for n in range(60):
                E, F, r = evaluate(k, 16 * (n % 2))
                different[k] += not (np.array_equal(F, want[k][1]) and np.array_equal(r, want[k][2]))
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(cases))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors and not any(different)
