"""PME grids of several sizes and factors on the GPU, against the FP64 oracle."""
import numpy as np
import pytest

import atmmetaforce as atm
from atmmetaforce import synthetic as S
import oracle as O

pytestmark = pytest.mark.gpu

U_TOL, F_TOL = 0.01, 1e-4  # kJ/mol, force RMS relative: the parity tests' tolerances


def _check(grids, diff):
    cases = []
    for k, g in enumerate(grids):
        c = S.water_ligand_box(1100, 2.25, [9], [(1.1, 1.0, 1.2)], S.PME, 0.9, seed=60 + k)
        c.spec.grid = tuple(g)
        cases.append(c)
    b = atm.ReplicaBatch([atm.system_from_case(c)[0] for c in cases], 0, {"DifferencePath": diff})
    E, F, r = b.evaluate(np.concatenate([c.pos for c in cases]))
    for k, c in enumerate(cases):
        ref = O.atm_eval(c.spec, c.pos, c.displ, c.params)
        f = F[b.offsets[k]:b.offsets[k + 1]]
        assert abs(r[k]["pert"] - ref["usc"]) <= U_TOL, grids[k]
        assert np.sqrt(((f - ref["forces"]) ** 2).sum() / (ref["forces"] ** 2).sum()) <= F_TOL, grids[k]


@pytest.mark.parametrize("diff", [0, 1], ids=["two-states", "difference"])
def test_grids_of_odd_and_multiple_of_four_sizes_in_one_batch(diff):
    """Two grids of an odd size are 2 mod 4 floats long; the next replicas' grids,
    whose rows are read and written as float4, must start on 16 bytes all the same."""
    _check([(23, 23, 23), (24, 24, 24), (23, 25, 21), (25, 23, 28), (24, 24, 24)], diff)


@pytest.mark.parametrize("diff", [0, 1], ids=["two-states", "difference"])
def test_grids_with_prime_factors_beyond_the_dedicated_radices(diff):
    """The direct DFT stage: primes 11 to 37, one or five past a multiple of its
    outputs per work item, alone (23, 29, 31, 37) and after other stages (22, 26,
    33, 34, 38, 39)."""
    _check([(22, 23, 26), (31, 29, 37), (34, 39, 38), (33, 22, 22), (26, 22, 34)], diff)


@pytest.mark.parametrize("grid", [(121, 24, 22), (24, 121, 26), (22, 26, 121), (101, 23, 24), (143, 20, 21)])
def test_grids_with_two_prime_stages_or_a_long_one(grid):
    """Roots of a prime stage after another one (121, 143), and of one prime (101)."""
    _check([grid], 1)


@pytest.mark.parametrize("ligand", [7, 8, 9, 33], ids=lambda n: f"ligand{n}")
def test_default_spreading_gives_the_bricks_bits(ligand):
    """Per-atom spreading (the default) against bricks: blocks that end one atom
    before, at and after a warp's share of a block, and a moving block of one atom."""
    c = S.water_ligand_box(1300 + ligand, 2.6, [ligand], [(1.3, 1.2, 1.1)], S.PME, 0.9, seed=70)
    out = []
    for props in ({}, {"SpreadBrick": 16}, {"SpreadByOwner": 0}):
        b = atm.ReplicaBatch([atm.system_from_case(c)[0]], 0, props)
        out.append(b.evaluate(c.pos, as_array=True))
    for E, F, r in out[1:]:
        assert np.array_equal(F, out[0][1]) and np.array_equal(r, out[0][2])


@pytest.mark.parametrize("n,edge", [(31, 1.9), (33, 1.9), (65, 9.0), (65, 3.6), (1500, 2.5), (16384, 5.6)])
def test_noalloc_skips_no_pair(n, edge):
    """Tiles and steps left out hold no counted pair: one block, one particle past a
    block, blocks mostly beyond the cutoff, a dense box and the largest count, with
    particles outside the cell and blocks that span it, against the oracle."""
    import ctypes as C

    import torch
    from atmmetaforce import _lib

    rng = np.random.default_rng(n)
    side = int(np.ceil(n ** (1 / 3)))
    g = (np.arange(side) + 0.5) * (edge / side)
    pos = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)[rng.permutation(side ** 3)[:n]]
    pos += rng.uniform(-0.02, 0.02, (n, 3)) + edge * rng.integers(-2, 3, (n, 3))
    q, sig, eps = rng.uniform(-0.4, 0.4, n), rng.uniform(0.15, 0.2, n), rng.uniform(0.1, 0.5, n)
    ei = np.arange(0, n - 1, 2, dtype=np.int32)
    zero = np.zeros(len(ei))
    spec = S.NonbondedSpec(q, sig, eps, ei, ei + 1, zero, zero + 1.0, zero, S.CUTOFF_PERIODIC, 0.9, np.full(3, edge))
    start = np.concatenate([[0], np.cumsum(np.arange(n) < 2 * len(ei))]).astype(np.int32)
    flat = (np.arange(2 * len(ei)) ^ 1).astype(np.int32)
    d = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    args = [d(a) for a in (pos, q, sig, eps, start, flat)]
    e = torch.zeros(1, dtype=torch.float64, device="cuda")
    f = torch.zeros(n, 3, dtype=torch.float64, device="cuda")
    _lib.call("atm_rf_nonbonded_noalloc", n, *(C.c_void_p(a.data_ptr()) for a in args), (C.c_double * 3)(*spec.box), 0.9,
              78.5, C.c_void_p(e.data_ptr()), C.c_void_p(f.data_ptr()), None)
    torch.cuda.synchronize()
    E, F, T = O.nonbonded(spec, pos)
    assert abs(e.item() - E) <= 2e-6 * (sum(abs(v) for v in T.values()) + 1.0)
    # (no pair at all in the sparsest box: both are zero)
    assert np.sqrt(((f.cpu().numpy() - F) ** 2).sum()) <= F_TOL * np.sqrt((F ** 2).sum())


@pytest.mark.parametrize("method", [S.PME, S.CUTOFF_PERIODIC], ids=["pme", "rf"])
def test_dispersion_correction_follows_parameters_and_box(method):
    """The dispersion correction of each replica after new epsilons of one of them and
    after a new box, against the oracle."""
    cases = [S.water_ligand_box(1100, 2.25, [9], [(1.1, 1.0, 1.2)], method, 0.9, seed=80 + k, use_disp_corr=True)
             for k in range(2)]
    b = atm.ReplicaBatch([atm.system_from_case(c)[0] for c in cases], 0)
    pos = np.concatenate([c.pos for c in cases])

    def check(E):
        for k, c in enumerate(cases):
            ref = O.atm_eval(c.spec, c.pos, c.displ, c.params)
            _, _, T = O.nonbonded(c.spec, c.pos)
            assert abs(E[k] - ref["energy"]) <= 2e-6 * (sum(abs(v) for v in T.values()) + 1.0) + U_TOL

    check(b.evaluate(pos)[0])
    cases[1].spec.epsilon = cases[1].spec.epsilon * 1.7
    b.setNonbondedParameters(1, cases[1].spec.charge, cases[1].spec.sigma, cases[1].spec.epsilon)
    check(b.evaluate(pos)[0])
    cases[0].spec.box = cases[0].spec.box * 1.01
    L = cases[0].spec.box
    b.setPeriodicBoxVectors(0, (L[0], 0, 0), (0, L[1], 0), (0, 0, L[2]))
    check(b.evaluate(pos)[0])


@pytest.mark.parametrize("diff", [0, 1], ids=["two-states", "difference"])
@pytest.mark.parametrize("n,L,ligand", [(1506, 2.78, 9), (2703, 3.4, 33), (8009, 4.86, 29)])
def test_triclinic_rows_by_groups(n, L, ligand, diff):
    """Rhombic dodecahedral cells whose rows keep or drop whole groups of j slots: too
    small for any group to be dropped, partial blocks before the moving ones (their
    groups straddle half blocks), and a cell where most groups are dropped."""
    c = S.triclinic_water_ligand_box(n, (L, L, L * 0.5 ** 0.5), (0.0, 0.5 * L, 0.5 * L), [ligand],
                                     [(0.35 * L, 0.35 * L, 0.3 * L)], S.PME, 0.9, seed=120 + ligand)
    b = atm.ReplicaBatch([atm.system_from_case(c)[0]], 0, {"DifferencePath": diff})
    E, F, r = b.evaluate(c.pos)
    ref = O.atm_eval(c.spec, c.pos, c.displ, c.params)
    assert abs(r[0]["pert"] - ref["usc"]) <= U_TOL
    assert np.sqrt(((F - ref["forces"]) ** 2).sum() / (ref["forces"] ** 2).sum()) <= F_TOL


@pytest.mark.parametrize("atoms", [(1103, 2207, 1500), (9001, 1103)])
def test_octets_of_blocks_across_replicas(atoms):
    """Octets that belong to two replicas, that hold the last blocks of one, moving blocks
    at their displaced positions, and rows in one part (enough replicas) and in several,
    against batches of one replica."""
    cases = [S.water_ligand_box(n, (n / 98.85) ** (1 / 3), [9 + k], [(0.9, 1.0, 0.8)], S.PME, 0.9, seed=130 + k)
             for k, n in enumerate(atoms)]
    many = [cases[k % len(cases)] for k in range(48 if len(atoms) == 3 else 2)]
    for diff in (0, 1):
        one = [atm.ReplicaBatch([atm.system_from_case(c)[0]], 0, {"DifferencePath": diff}) for c in cases]
        want = [b.evaluate(c.pos, as_array=True) for b, c in zip(one, cases)]
        systems = [atm.system_from_case(c)[0] for c in cases]
        b = atm.ReplicaBatch([systems[k % len(cases)] for k in range(len(many))], 0, {"DifferencePath": diff})
        E, F, r = b.evaluate(np.concatenate([c.pos for c in many]), as_array=True)
        for k in range(len(many)):
            e, f, q = want[k % len(cases)]
            got = F[b.offsets[k]:b.offsets[k + 1]]
            # rows in another number of parts group their pairs otherwise: FP32 sums of at
            # most 16 terms, a few 2^-24 of the pair forces
            assert np.sqrt(((got - f) ** 2).sum() / (f ** 2).sum()) <= 2e-6, (diff, k)
            assert abs(r[k][atm.RES_KEYS.index("u")] - q[0][atm.RES_KEYS.index("u")]) <= U_TOL
