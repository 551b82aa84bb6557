"""The autotuner times each launch once and names what it launches."""
import numpy as np
import pytest

import atmmetaforce as atm
from atmmetaforce import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("replicas,kinds", [
    # 126 rows, one pass of 567 CTAs: fewer than 4 per SM are (608), more than 3 (456) or 2
    (3, ["tiles/SM=4", "tiles in one pass, 80 registers", "fused lists+tiles"]),
    # 168 rows, 756 CTAs
    (4, ["tiles in one pass, 64 registers", "tiles in one pass, 80 registers", "fused lists+tiles"]),
    # 3,360 rows: one pass at 4 (4,864 warps) and 3 (3,648), from a counter at 2 (2,432)
    (80, ["tiles in one pass, 64 registers", "tiles in one pass, 80 registers", "tiles/SM=2", "fused lists+tiles"]),
])
def test_each_launch_is_timed_once(tmp_path, monkeypatch, replicas, kinds):
    monkeypatch.setenv("ATM_AUTOTUNE_CACHE", str(tmp_path / "tune.txt"))
    c = S.water_ligand_box(1300, 2.4, [9], [(1.1, 1.0, 1.2)], S.CUTOFF_PERIODIC, 0.9, seed=180)
    b = atm.ReplicaBatch([atm.system_from_case(c)[0]] * replicas, 0, {"DifferencePath": 1})
    pos = np.tile(c.pos, (replicas, 1))
    E, F, r = b.evaluate(pos, as_array=True)
    lines = b.autotune(trials=1, use_cache=False).strip().splitlines()
    timed = [l.split(" brick=")[0] for l in lines[:-1]]
    assert timed == kinds
    assert lines[-1].startswith("chosen: ") and lines[-1][len("chosen: "):].split(" brick=")[0] in kinds
    E1, F1, r1 = b.evaluate(pos, as_array=True)
    assert np.array_equal(F1, F)
