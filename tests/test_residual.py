"""The residual kernel at the edges of its 32-trace x 32-sample blocks: the
residual traces are bit-identical to sequential float32 running sums, and the
sums equal the FP64 sums of their squares; several slots and components in
one launch equal the single calls."""
import numpy as np
import pytest

from ifos_b200 import workloads as W
from ifos_b200.solver import ShotSolver
from tests.golden.cases import build_case
from tests.gpu_helpers import bit_equal

pytestmark = pytest.mark.gpu


def _expected(obs, syn, dt):
    dt = np.float32(dt)
    r = np.cumsum(syn, axis=1, dtype=np.float32) * dt - (d := np.cumsum(obs, axis=1, dtype=np.float32) * dt)
    return r[:, ::-1], float((r.astype(np.float64) ** 2).sum()), float((d.astype(np.float64) ** 2).sum())


@pytest.mark.parametrize("ntr,ns", [(1, 1), (1, 33), (31, 32), (32, 31), (33, 64), (64, 65), (100, 257), (3, 500)])
def test_residual_blocks(ntr, ns):
    p, *_ = build_case("psv_el_o4")
    p.nt, p.dtinv = ns, 1
    rng = np.random.default_rng(ntr * 1000 + ns)
    obs, syn = rng.standard_normal((2, ntr, ns), dtype=np.float32)
    with ShotSolver(p, max_rec=ntr, snapshots=False) as s:
        diff, l2, en = s.calc_res(obs, syn)
    want, l2_w, en_w = _expected(obs, syn, p.dt)
    assert bit_equal(diff, want)
    # sums of ns * ntr non-negative FP64 terms in another order: n * 2^-53 each way
    tol = 2.0 * ntr * ns * 2.0 ** -53 + 2.0 ** -52
    assert abs(l2 - l2_w) <= tol * l2_w and abs(en - en_w) <= tol * en_w


@pytest.mark.parametrize("case,planes", [("psv_el_o4", (0, 1)), ("sh_el_o6", (2,)), ("acoustic_o4_p", (2,))])
def test_slots_and_components_in_one_launch(case, planes):
    p, model, g, sig, _ = build_case(case)
    ntr = g.recpos.shape[1]
    sec_plane = {0: 0, 1: 1, 2: 3 if p.acoustic else 2}
    rng = np.random.default_rng(9)
    obs = (rng.standard_normal((2, 3, ntr, p.nt)) * 1e-6).astype(np.float32)
    kill = np.zeros((2, ntr), np.int32)
    kill[1, ntr // 2] = 1
    adj = np.zeros((2, 3, ntr, p.nt), np.float32)
    with ShotSolver(p, max_shots=2, max_rec=ntr) as s:
        s.upload_model(model)
        s.setup_shot(0, g.srcpos, sig, g.recpos)
        s.setup_shot(1, g.srcpos, sig, np.ascontiguousarray(g.recpos[:, :ntr - 1]))  # fewer traces than the other slot
        sec = s.forward(2, store=False)
        l2, en = s.residual_adjoint(obs, 2, kill=kill)
        for slot, live in ((0, np.arange(ntr)), (1, np.delete(np.arange(ntr - 1), ntr // 2))):
            want = np.zeros(2)
            for k in planes:
                diff, a, b = s.calc_res(obs[slot, k][live], sec[slot, sec_plane[k]][live])
                want += (a, b)
                adj[slot, k, live] = diff
            np.testing.assert_allclose((l2[slot], en[slot]), want, rtol=1e-13)
        # the residual traces: the adjoint of the staged ones equals that of the single calls' traces
        s.forward(2, store=True, fetch=False)
        s.residual_adjoint(obs, 2, kill=kill)
        staged = s.adjoint(None, 2)
        assert bit_equal(staged, s.adjoint(adj, 2))
        assert all(np.abs(staged[slot]).max() > 0 for slot in range(2))
