"""Device inputs right after new device buffers, before any evaluation has run on them."""
import numpy as np
import pytest

import atmmetaforce as atm
from atmmetaforce import synthetic as S

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from atmmetaforce.autograd import batch_tensors  # noqa: E402

PROPS = {"DifferencePath": 1, "Adjoint": 1}


def _cases():
    return [S.water_ligand_box(n, edge, [11], [(1.1, 1.0, 1.2)], S.PME, 0.9, seed=60 + n,
                               params=S.default_params(0.2, 0.4, 0.1, 60.0, 0.5), use_disp_corr=False)
            for n, edge in ((1103, 2.3), (1502, 2.55))]


def _batch(cases):
    return atm.ReplicaBatch([atm.system_from_case(c)[0] for c in cases], 0, PROPS)


def _set(batch, tensors):
    x, d, p, q, s, e = tensors
    batch.setInputsDevice(d.data_ptr(), q.data_ptr(), s.data_ptr(), e.data_ptr(), p.data_ptr())


@pytest.mark.parametrize("evaluated", [False, True], ids=["first-buffers", "buffers-anew"])
def test_new_charges_after_a_stored_tuning(tmp_path, monkeypatch, evaluated):
    """A tuning read from the file makes buffers (or, with another spreading brick, makes them
    anew) without an evaluation; charges set then give a new batch's energies."""
    cache = tmp_path / "tune.txt"
    monkeypatch.setenv("ATM_AUTOTUNE_CACHE", str(cache))
    cases = _cases()
    pos = np.concatenate([c.pos for c in cases])
    first = _batch(cases)
    first.evaluate(pos)
    first.autotune(trials=1, use_cache=False)
    key = cache.read_text().rstrip("\n").split("\t")[0]
    cache.write_text(key + "\t4 16 1 0\n")  # bricks of 16: not the default

    batch = _batch(cases)
    if evaluated:
        batch.evaluate(pos)
    else:
        for r, c in enumerate(cases):
            batch.setPositions(r, c.pos)
    assert batch.autotune(trials=1, use_cache=True).startswith("cached")
    t = list(batch_tensors(batch, cases))
    t[3] *= 1.01
    _set(batch, t)
    E, F, res = batch.evaluate(pos, as_array=True)

    for c in cases:
        c.spec.charge = c.spec.charge * 1.01
    want = _batch(cases)
    E0, F0, res0 = want.evaluate(pos, as_array=True)
    # equal but for the order of the FP64 sum of squared charges in the self energy (some
    # 1e5 kJ/mol here: its rounding errors are a few 1e-11)
    assert np.array_equal(F, F0)
    assert np.allclose(E, E0, rtol=1e-12, atol=1e-12 * np.abs(res0).max())
    assert np.allclose(res, res0, rtol=1e-12, atol=1e-12 * np.abs(res0).max())
