"""Tau of the models of a context: the kernels take uniform values from launch
parameters and others from the model's planes.  A model uploaded in place of
another, with the time loop captured before, and models of different tau in
one context give the results of a context of their own, bit for bit."""
import numpy as np
import pytest

from ifos_b200.solver import ShotSolver
from tests.golden.cases import build_case
from tests.gpu_helpers import bit_equal, gpu_shot

pytestmark = pytest.mark.gpu
NAMES = ["psv_visc_o4", "sh_visc_o4", "ac_visc_o4_p"]


def _models(p, model):
    """The same medium with the parameter file's tau, with twice it, and with tau varying over the grid."""
    rng = np.random.default_rng(2)
    tau = np.full(model["vp"].shape, p.tau, np.float32)
    vary = (tau * rng.uniform(0.6, 1.4, tau.shape)).astype(np.float32)
    return [dict(model, taup=t, taus=t) for t in (tau, tau * 2, vary)]


def _same(a, b):
    return all(bit_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("order", [(0, 1), (1, 2, 0), (2, 1)])
@pytest.mark.parametrize("name", NAMES)
def test_a_model_uploaded_in_place_of_another(name, order):
    p, model, g, sig, adj = build_case(name, nt=60)
    models = _models(p, model)
    want = {k: gpu_shot(p, models[k], g, sig, adj) for k in order}
    with ShotSolver(p, max_rec=g.recpos.shape[1]) as s:
        s.setup_shot(0, g.srcpos, sig, g.recpos)
        for k in order:
            s.upload_model(models[k])
            for _ in range(2):
                assert _same((s.forward(1)[0], s.adjoint(adj[None])[0]), (want[k]["sections"], want[k]["grads"])), k
    assert not bit_equal(want[order[0]]["sections"], want[order[1]]["sections"])


@pytest.mark.parametrize("order", [(0, 1), (1, 0), (0, 2), (2, 0, 1)])
@pytest.mark.parametrize("name", NAMES)
def test_models_of_different_tau_in_one_context(name, order):
    p, model, g, sig, adj = build_case(name, nt=60)
    models, n = _models(p, model), len(order)
    with ShotSolver(p, max_shots=n, max_models=n, max_rec=g.recpos.shape[1]) as s:
        for slot, k in enumerate(order):
            s.upload_model(models[k], slot)
            s.setup_shot(slot, g.srcpos, sig, g.recpos, model=slot)
        sec, grads = s.forward(n), s.adjoint(np.stack([adj] * n), n)
    for slot, k in enumerate(order):
        want = gpu_shot(p, models[k], g, sig, adj)
        assert _same((sec[slot], grads[slot]), (want["sections"], want["grads"])), k
