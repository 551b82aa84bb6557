"""Differentiable calls whose inputs stay on the device: new parameters are taken over by a
kernel, without the host's layout; the results must be those of a batch built with them."""
import numpy as np
import pytest

import atmmetaforce as atm
from atmmetaforce import synthetic as S

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from atmmetaforce.autograd import atm_softplus_energy, batch_tensors  # noqa: E402

PROPS = {"DifferencePath": 1, "Adjoint": 1}


def _cases(method, dispersion):
    # odd counts: partial blocks, a partial last warp of the update and of the exceptions
    out = []
    for k, (n, lig) in enumerate([(1103, 11), (1502, 14)]):
        edge = 2.3 if k == 0 else 2.55
        out.append(S.water_ligand_box(n, edge, [lig], [(1.1, 1.0, 1.2)], method, 0.9, seed=90 + k,
                                      params=S.default_params(0.2, 0.4, 0.1, 60.0, 0.5), use_disp_corr=dispersion))
    return out


def _batch(cases):
    return atm.ReplicaBatch([atm.system_from_case(c)[0] for c in cases], 0, PROPS)


def _run(batch, tensors):
    x, d, p, q, s, e = [t.clone().requires_grad_() for t in tensors]
    w = atm_softplus_energy(batch, x, d, p, q, s, e)
    g = torch.autograd.grad((w * torch.arange(1.0, len(w) + 1, device=w.device, dtype=w.dtype)).sum(), (x, d, p, q, s, e))
    E, F, r = batch.evaluate(x.detach().cpu().numpy(), as_array=True)
    return [w.detach().cpu().numpy(), F, r] + [t.cpu().numpy() for t in g]


def _same(got, want):
    # the forces and gradients are the same bits; energies differ by the order of the FP64
    # sum of squared charges in the self energy (at most n rounding errors of 2^-53 of it)
    for k, (a, b) in enumerate(zip(got, want)):
        assert np.allclose(a, b, rtol=1e-12, atol=1e-12 * np.abs(b).max()), k


@pytest.mark.parametrize("method,dispersion", [(S.PME, False), (S.PME, True), (S.CUTOFF_PERIODIC, True)])
def test_changed_inputs_give_a_new_batchs_results(method, dispersion):
    cases = _cases(method, dispersion)
    batch = _batch(cases)
    base = batch_tensors(batch, cases)
    _run(batch, base)
    rng = np.random.default_rng(3)
    # charges only; sigmas and epsilons of one replica; softplus parameters only;
    # displacements (the layout follows) with new charges; back to the first inputs
    for step in ("charge", "lj", "params", "displacements", "back"):
        t = [v.clone() for v in base]
        n0 = cases[0].n
        if step in ("charge", "displacements"):
            t[3] *= torch.as_tensor(rng.uniform(0.98, 1.02, len(t[3])), device=t[3].device)
        if step == "lj":
            t[4][n0:] *= 1.01
            t[5][n0:] *= 0.97
        if step == "params":
            t[2][:, 0] += 0.05
        if step == "displacements":
            t[1][t[1] != 0] += 0.03
        new = [S.ATMCase(c.spec.__class__(**c.spec.__dict__), c.pos, c.displ.copy(), c.params.copy(), c.ligands) for c in cases]
        for k, c in enumerate(new):
            a, b = (0, n0) if k == 0 else (n0, n0 + cases[1].n)
            c.displ = t[1][a:b].cpu().numpy()
            c.params[:5] = t[2][k].cpu().numpy()
            c.spec.charge, c.spec.sigma, c.spec.epsilon = (t[q][a:b].cpu().numpy() for q in (3, 4, 5))
        fresh = _batch(new)
        _same(_run(batch, t), _run(fresh, t))


def test_host_setters_and_other_tensor_types_between_device_inputs():
    """Host setters after device inputs, and float32 inputs (which go through the host),
    act on the values in force."""
    cases = _cases(S.PME, True)
    batch = _batch(cases)
    base = batch_tensors(batch, cases)
    first = _run(batch, base)
    changed = [v.clone() for v in base]
    changed[3] *= 1.01
    _run(batch, changed)
    # one replica set through the host: the other keeps what the device call set
    c = cases[0]
    batch.setNonbondedParameters(0, c.spec.charge, c.spec.sigma, c.spec.epsilon)
    _, F, _ = batch.evaluate(base[0].cpu().numpy(), as_array=True)
    assert np.array_equal(F[: c.n], first[1][: c.n])
    assert not np.array_equal(F[c.n:], first[1][c.n:])
    # float32 charges, then float64 ones again
    low = [v.clone() for v in base]
    low[3] = low[3].float()
    w32 = atm_softplus_energy(batch, *low)
    exact = [v.clone() for v in base]
    exact[3] = low[3].double()
    assert torch.allclose(w32, atm_softplus_energy(batch, *exact), rtol=1e-12)
    _same(_run(batch, base), first)
