"""Sources, receivers and the free surface inside the SH and acoustic
kernels: receiver layouts that fit the cell map and ones that do not, sources
that share a cell or a row with receivers, both seismogram and adjoint types.
Bit-identical to the oracle."""
import numpy as np
import pytest

from ifos_b200 import workloads as W
from ifos_b200.solver import ShotSolver
from tests.golden.cases import build_case
from tests.gpu_helpers import bit_equal, forward_fields_mask, gpu_shot, oracle_shot

pytestmark = pytest.mark.gpu


def _receivers(p, layout):
    if layout == "three_rows":
        xs = np.concatenate([np.arange(10, 55, 4), np.arange(12, 50, 5), np.arange(9, 57, 6)])
        ys = np.concatenate([np.full(12, 3), np.full(8, 11), np.full(8, 20)])
    elif layout == "vertical_line":  # more rows than the cell map holds: the separate receiver kernels
        ys = np.arange(3, 36, 3)
        xs = np.full(ys.shape, 30)
    elif layout == "surface":
        xs, ys = np.arange(5, 60, 7), np.full(8, 1)
    else:  # the probe's cell, and the last cells of a row
        xs, ys = np.array([p.nx // 2, p.nx, p.nx - 1, 1]), np.array([p.ny // 2, 3, 3, 3])
    return np.stack([xs, ys]).astype(np.int32)


@pytest.mark.parametrize("layout", ["three_rows", "vertical_line", "surface", "centre"])
@pytest.mark.parametrize("name,seismo,adjoint_type", [("sh_el_o6", 1, 1), ("sh_visc_o4", 1, 1), ("acoustic_o4_p", 2, 4),
                                                      ("acoustic_o4_p", 1, 1), ("acoustic_o4_p", 1, 2),
                                                      ("acoustic_o4_p", 5, 4), ("ac_visc_o4_p", 2, 4),
                                                      ("ac_visc_o2_nofs", 2, 4)])
def test_receivers(name, seismo, adjoint_type, layout):
    p, model, g, sig, _ = build_case(name, nt=60)
    p.seismo, p.adjoint_type = seismo, adjoint_type
    rec = _receivers(p, layout)
    g = W.Geometry(g.srcpos, rec)
    adj = (np.random.default_rng(5).standard_normal((3, rec.shape[1], p.nt)) * 1e-3).astype(np.float32)
    gpu, ref = gpu_shot(p, model, g, sig, adj), oracle_shot(p, model, g, sig, adj)
    m = forward_fields_mask()
    for key in ("sections", "grads", "adj_fields"):
        assert bit_equal(gpu[key], ref[key]), key
    assert bit_equal(gpu["fields"][m], ref["fields"][m]), "fields"
    if layout != "surface":  # the pressure of row 1 is zero
        assert np.abs(ref["sections"]).max() > 0 and np.abs(ref["grads"]).max() > 0


@pytest.mark.parametrize("cells", [[(30, 3), (30, 3)], [(30, 1), (31, 1), (33, 2)], [(64, 40), (1, 1), (17, 9), (18, 9)]])
@pytest.mark.parametrize("name", ["sh_el_o6", "sh_visc_o4", "acoustic_o4_p", "ac_visc_o4_p", "psv_el_o4", "psv_visc_o4"])
def test_several_sources(name, cells):
    p, model, g, sig, adj = build_case(name, nt=60)
    src = np.repeat(g.srcpos, len(cells), axis=1)
    for k, (i, j) in enumerate(cells):
        src[0, k], src[1, k] = i, j
    sig = np.concatenate([sig * np.float32(1.0 + 0.3 * k) for k in range(len(cells))])
    g = W.Geometry(np.ascontiguousarray(src), g.recpos)
    gpu, ref = gpu_shot(p, model, g, sig, adj), oracle_shot(p, model, g, sig, adj)
    m = forward_fields_mask()
    for key in ("sections", "grads"):
        assert bit_equal(gpu[key], ref[key]), key
    assert bit_equal(gpu["fields"][m], ref["fields"][m]), "fields"


@pytest.mark.parametrize("name", ["sh_el_o6", "sh_visc_o4"])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("layout", ["three_rows", "vertical_line"])
def test_sh_has_no_pressure_residual(name, precision, layout):
    """An SH run takes its residuals in vz under every ADJOINT_TYPE: the
    pressure residual of type 4 has no plane to go to."""
    p, model, g, sig, _ = build_case(name, nt=60)
    rec = _receivers(p, layout)
    g = W.Geometry(g.srcpos, rec)
    adj = (np.random.default_rng(6).standard_normal((3, rec.shape[1], p.nt)) * 1e-3).astype(np.float32)
    got = []
    for p.adjoint_type in (1, 4):
        got.append(gpu_shot(p, model, g, sig, adj, precision=precision))
    for key in ("sections", "grads", "adj_fields"):
        assert bit_equal(got[0][key], got[1][key]), key
    assert np.abs(got[0]["grads"]).max() > 0


@pytest.mark.parametrize("name", ["psv_el_o4", "psv_visc_o8_holberg", "sh_el_o6", "sh_visc_o4", "acoustic_o4_p",
                                  "ac_visc_o4_p", "psv_el_o2_nofs"])
def test_shots_at_several_depths_in_one_batch(name):
    """Slots whose sources and receivers lie in different rows, some in two
    distant ones, some without receivers or sources in most rows of the span
    that the batch's cover: every slot equals the oracle's single shot."""
    p, model, g, sig, _ = build_case(name, nx=100, ny=61, nt=60)
    rng = np.random.default_rng(8)
    rows = [(3, [3, 57]), (31, [30]), (58, [8, 9]), (16, [17, 40, 55])]
    shots = []
    for k, (js, jr) in enumerate(rows):
        src = g.srcpos.copy()
        src[0], src[1] = 20 + 17 * k, js
        xs = np.arange(6 + k, 95, 7)
        rec = np.stack([np.tile(xs, len(jr)), np.repeat(jr, len(xs))]).astype(np.int32)
        adj = (rng.standard_normal((3, rec.shape[1], p.nt)) * 1e-3).astype(np.float32)
        shots.append((src, rec, adj))
    ntr = max(r.shape[1] for _, r, _ in shots)
    want = [oracle_shot(p, model, W.Geometry(src, rec), sig, adj) for src, rec, adj in shots]
    all_adj = np.zeros((len(shots), 3, ntr, p.nt), np.float32)
    with ShotSolver(p, max_shots=len(shots), max_rec=ntr) as s:
        s.upload_model(model)
        for k, (src, rec, adj) in enumerate(shots):
            s.setup_shot(k, src, sig, rec)
            all_adj[k, :, :rec.shape[1]] = adj
        sec, grads = s.forward(len(shots)), s.adjoint(all_adj, len(shots))
    for k, (_, rec, _) in enumerate(shots):
        assert bit_equal(sec[k, :, :rec.shape[1]], want[k]["sections"]), k
        assert bit_equal(grads[k], want[k]["grads"]), k
    for k in (0, 1):  # sources beside receivers: the waves arrive within the run
        assert np.abs(want[k]["sections"]).max() > 0 and np.abs(want[k]["grads"]).max() > 0
