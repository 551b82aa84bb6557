"""A context's forces are summed over the requested groups on the device, from positions that
the first kernel reads in the staging buffer: every mask, fresh or of the same evaluation again."""
import numpy as np
import pytest

import atmmetaforce as atm
from atmmetaforce import synthetic as S

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)


def _forces(ctx, groups):
    return ctx.getState(getEnergy=True, getForces=True, groups=groups).getForces().copy()


# a partial last warp; whole warps; no PME chain (the exceptions on the main stream)
@pytest.mark.parametrize("n,method", [(1103, S.PME), (1504, S.PME), (1502, S.CUTOFF_PERIODIC)])
def test_group_masks_fresh_and_repeated(n, method):
    case = S.water_ligand_box(n, 2.55, [14], [(1.1, 1.0, 1.2)], method, 0.9, seed=17,
                              params=S.default_params(0.2, 0.4, 0.1, 60.0, 0.5))
    ctx = atm.Context(atm.system_from_case(case)[0], 0)
    batch = atm.ReplicaBatch([atm.system_from_case(case)[0]], 0, {"DifferencePath": 0})  # (a context's path)
    masks = ({1}, {2}, {1, 2})
    for shift in (0.0, 0.013):
        pos = case.pos + shift
        want = batch.evaluate(pos, as_array=True)[1].reshape(-1, 3)
        fresh = []
        for g in masks:
            ctx.setPositions(pos)
            fresh.append(_forces(ctx, g))
        # the batch's forces are the same kernels' on copied positions; the sum of the
        # groups is one FP64 addition
        assert np.array_equal(fresh[1], want)
        assert np.array_equal(fresh[2], fresh[0] + fresh[1])
        for g, f in zip(masks, fresh):  # without another evaluation
            assert np.array_equal(_forces(ctx, g), f)
        assert not _forces(ctx, {5}).any()
        # an evaluation for the energy alone, its forces asked for afterwards
        ctx.setPositions(pos)
        ctx.getState(getEnergy=True, groups={1})
        assert np.array_equal(_forces(ctx, {2}), fresh[1])
