"""Device inputs given on a stream of the caller's: in force, on every stream, when the call
returns."""
import numpy as np
import pytest

import atmmetaforce as atm
from atmmetaforce import synthetic as S

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from atmmetaforce.autograd import batch_tensors  # noqa: E402


@pytest.mark.parametrize("changed", ["charge", "lj"])
def test_inputs_on_a_side_stream_are_in_force_at_return(changed):
    # (12,000 atoms: the update's kernel takes some tens of microseconds, more than the
    # return of the call)
    case = S.water_ligand_box(12000, 4.95, [30], [(1.9, 2.0, 2.1)], S.PME, 0.9, seed=17, use_disp_corr=False)
    sys_ = atm.system_from_case(case)[0]
    batch = atm.ReplicaBatch([sys_], 0, {"DifferencePath": 1, "Adjoint": 1})
    batch.evaluate(case.pos)
    side = torch.cuda.Stream()
    for factor in (1.01, 0.99, 1.02):
        t = list(batch_tensors(batch, [case]))
        for k in (3,) if changed == "charge" else (4, 5):
            t[k] = t[k] * factor
        torch.cuda.synchronize()
        batch.setInputsDevice(*(t[k].data_ptr() for k in (1, 3, 4, 5, 2)), side.cuda_stream)
        assert side.query()
        E, F, res = batch.evaluate(case.pos, as_array=True)
        # a batch that took the same inputs while nothing else ran
        fresh = atm.ReplicaBatch([sys_], 0, {"DifferencePath": 1, "Adjoint": 1})
        fresh.evaluate(case.pos)
        fresh.setInputsDevice(*(t[k].data_ptr() for k in (1, 3, 4, 5, 2)))
        torch.cuda.synchronize()
        E0, F0, res0 = fresh.evaluate(case.pos, as_array=True)
        assert np.array_equal(F, F0) and np.array_equal(res, res0)
        # and one built with them, but for its energies (the self energy is summed in
        # another order)
        host = atm.ReplicaBatch([sys_], 0, {"DifferencePath": 1, "Adjoint": 1})
        host.setNonbondedParameters(0, *(t[k].cpu().numpy() for k in (3, 4, 5)))
        assert np.array_equal(F, host.evaluate(case.pos)[1])
