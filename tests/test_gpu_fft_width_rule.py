"""Which transforms run with wide CTAs, and that a replica's results do not depend on it."""
import numpy as np
import pytest

import atmmetaforce as atm
from atmmetaforce import synthetic as S
import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

U_TOL, F_TOL = 0.01, 1e-4  # kJ/mol, force RMS relative: the parity tests' tolerances


def _case(grid):
    c = S.water_ligand_box(1100, 2.25, [9], [(1.1, 1.0, 1.2)], S.PME, 0.9, seed=90)
    c.spec.grid = grid
    return c


def _wide(batch, pos):
    """Whether the plane kernels and the slab kernel of an evaluation ran with 512 threads,
    by their names in a trace; None where there is no trace to be had."""
    batch.setProfiling(True)  # (kernel by kernel)
    batch.evaluate(pos)
    names = []
    for _ in range(3):  # (the first trace of a process can be empty)
        if not names:
            with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
                batch.evaluate(pos)
                torch.cuda.synchronize()
            names = [e.name for e in prof.events() if "k_" in e.name]
    batch.setProfiling(False)
    wide = {}
    for k in ("k_fft_zy", "k_fft_x_conv", "k_ifft_yz"):
        hits = [n for n in names if k in n]
        if not hits:
            return None
        wide[k] = "512" in hits[0]
    assert wide["k_fft_zy"] == wide["k_ifft_yz"]
    return wide["k_fft_zy"], wide["k_fft_x_conv"]


@pytest.mark.parametrize("grid,replicas,planes,slabs", [
    ((20, 276, 9), 1, False, False),  # 1,380 points (the twiddles of a long dimension are no points)
    ((20, 280, 9), 1, True, False),   # 1,400 points; slabs of 100
    ((51, 51, 51), 1, False, False),  # 1,326 and 1,326
    ((52, 52, 52), 1, True, True),    # 1,404 and 1,404
    ((55, 55, 52), 2, True, True),    # 1,485 and 1,485
    ((56, 56, 56), 2, True, True),    # 224 planes, 112 slabs
    ((56, 56, 56), 3, False, False),  # 336 planes, 168 slabs: more than two and one per SM
])
def test_width_follows_the_points(grid, replicas, planes, slabs):
    c = _case(grid)
    b = atm.ReplicaBatch([atm.system_from_case(c)[0]] * replicas, 0, {"DifferencePath": 1})
    pos = np.tile(c.pos, (replicas, 1))
    E, F, r = b.evaluate(pos)
    ref = O.atm_eval(c.spec, c.pos, c.displ, c.params)
    assert abs(r[0]["pert"] - ref["usc"]) <= U_TOL
    f = F[:c.n]
    assert np.sqrt(((f - ref["forces"]) ** 2).sum() / (ref["forces"] ** 2).sum()) <= F_TOL
    got = _wide(b, pos)
    if got is None:
        pytest.skip("no kernel trace on this machine")
    assert got == (planes, slabs)


@pytest.mark.parametrize("grid", [(56, 56, 56), (55, 57, 58), (54, 68, 46)])
def test_both_widths_give_the_same_bits(grid):
    """One replica alone (wide CTAs) and among as many as make the CTAs narrow."""
    c = _case(grid)
    sys_ = atm.system_from_case(c)[0]
    E, F, r = atm.ReplicaBatch([sys_], 0, {"DifferencePath": 1}).evaluate(c.pos, as_array=True)
    n = 4
    E4, F4, r4 = atm.ReplicaBatch([sys_] * n, 0, {"DifferencePath": 1}).evaluate(np.tile(c.pos, (n, 1)), as_array=True)
    for k in range(n):
        assert np.array_equal(F4[k * c.n:(k + 1) * c.n], F) and np.array_equal(r4[k], r[0])
