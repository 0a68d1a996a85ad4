"""The pipelined stencils at the edges of their cell groups: every remainder
of NX by the four cells a thread owns (and by the vector widths of the
snapshots and the correlation), CPML strips that start and end inside a
group or share one, tiles with no plain warp, steps whose 1/DH is not exact,
and CPML profiles with K above 1.  Bit-identical to the oracle, as the
aligned cases are."""
import numpy as np
import pytest

from ifos_b200.solver import ShotSolver
from tests.golden.cases import build_case
from tests.gpu_helpers import bit_equal, forward_fields_mask, gpu_shot, oracle_shot

pytestmark = pytest.mark.gpu
NAMES = ["psv_el_o4", "psv_el_o8_holberg", "psv_visc_o8_holberg", "sh_el_o6", "sh_visc_o4", "acoustic_o4_p",
         "ac_visc_o2_nofs", "psv_el_o2_nofs", "psv_el_o12_ref"]


def _same(p, model, g, sig, adj):
    gpu, ref = gpu_shot(p, model, g, sig, adj), oracle_shot(p, model, g, sig, adj)
    m = forward_fields_mask()
    for key in ("sections", "grads", "adj_fields"):
        assert bit_equal(gpu[key], ref[key]), key
    assert bit_equal(gpu["fields"][m], ref["fields"][m]), "fields"
    assert np.abs(ref["grads"]).max() > 0


@pytest.mark.parametrize("nx,ny,fw", [(64, 40, 8), (65, 41, 7), (66, 39, 9), (67, 38, 6), (129, 33, 10), (190, 35, 11)])
@pytest.mark.parametrize("name", NAMES)
def test_every_remainder(name, nx, ny, fw):
    _same(*build_case(name, nx=nx, ny=ny, nt=50, fw=fw))


@pytest.mark.parametrize("nx,fw", [(41, 20), (42, 20), (43, 19), (66, 31), (78, 39)])
@pytest.mark.parametrize("name", ["psv_el_o4", "psv_visc_o4_kmax2", "sh_el_o4_kmax3", "acoustic_o4_p"])
def test_strips_that_meet_in_a_group(name, nx, fw):
    """2 FW up to NX: a group of four cells holds cells of both x strips, and
    strips too wide for the table a block stages read the global profiles."""
    p, model, g, sig, adj = build_case(name, nx=90, ny=2 * fw + 8, nt=40, fw=fw)
    keep = slice(0, nx)
    p.nx = nx
    model = {k: np.ascontiguousarray(v[:, keep]) for k, v in model.items()}
    g.recpos = np.ascontiguousarray(g.recpos[:, g.recpos[0] <= nx])
    g.srcpos[0] = np.minimum(g.srcpos[0], nx // 2)
    _same(p, model, g, sig, np.ascontiguousarray(adj[:, :g.recpos.shape[1]]))


@pytest.mark.parametrize("dh", [2.5, 0.7, 3.0, 12.5])
@pytest.mark.parametrize("name", ["psv_el_o4", "sh_el_o6", "acoustic_o4_p"])
def test_inexact_reciprocal_of_dh(name, dh):
    """x/DH by the reciprocal rounds as the division; the first steps hold
    zero and tiny values, which take the division itself."""
    p, model, g, sig, adj = build_case(name, nt=60)
    p.dt *= dh / p.dh
    p.dh = dh
    _same(p, model, g, sig, adj)


@pytest.mark.parametrize("nx", [64, 65, 66, 67, 130])
@pytest.mark.parametrize("name,snap", [("psv_el_o4", "fp16s"), ("psv_visc_o8_holberg", "fp16s"), ("sh_el_o6", "fp16s"),
                                       ("acoustic_o4_p", "fp16s"), ("psv_el_o4", "i16s")])
def test_segment_snapshots_of_ragged_rows(name, snap, nx):
    """Segment snapshots of every row remainder against the fp32 snapshots
    quantised on the host: the maximum of a 64-cell segment maps to the top of
    the format (65472 for fp16, 32767 for int16), each value within half a
    unit in the last place of its own magnitude (fp16) or of the segment
    (int16), plus the few fp32 roundings of the scale; a segment whose maximum
    is below 1e-30 is stored as zeros."""
    p, model, g, sig, adj = build_case(name, nx=nx, ny=37, nt=60)
    ntr, index = g.recpos.shape[1], p.nt // p.dtinv - 1
    got = {}
    for fmt in ("fp32", snap):
        with ShotSolver(p, max_rec=ntr, snap_format=fmt) as s:
            s.upload_model(model)
            s.setup_shot(0, g.srcpos, sig, g.recpos)
            s.forward(1, store=True, fetch=False)
            got[fmt] = s.snapshot(index).astype(np.float64)
    want = got["fp32"]
    for c0 in range(0, nx, 64):
        w, v = want[:, :, c0:c0 + 64], got[snap][:, :, c0:c0 + 64]
        top = np.abs(w).max(axis=2, keepdims=True)
        w = np.where(top >= np.float32(1e-30), w, 0.0)
        if snap == "fp16s":
            # fp16: 2^-11 relative for normal values, else half the smallest subnormal (2^-25) of the scaled range
            tol = np.maximum(np.abs(w) * 2.0 ** -11, top / 65472.0 * 2.0 ** -25)
        else:
            tol = top / 32767.0 * 0.5
        assert (np.abs(v - w) <= tol * (1 + 1e-5) + np.abs(w) * 2.0 ** -20).all()
    assert np.abs(want).max() > 0


@pytest.mark.parametrize("nx", [64, 66, 67])
@pytest.mark.parametrize("name", ["psv_el_o4", "sh_el_o6", "acoustic_o4_p"])
@pytest.mark.parametrize("snap", ["fp16s", "i16s"])
def test_correlation_of_segment_snapshots(name, snap, nx):
    """The raw correlation sums with segment snapshots against the same
    float32 terms formed on the host from the fetched snapshots and the
    adjoint fields of one snapshot step (NT = DTINV: one term, bit for bit)."""
    p, model, g, sig, adj = build_case(name, nx=nx, ny=33, nt=60)
    p.dtinv = p.nt
    p.dt *= 0.9
    ntr = g.recpos.shape[1]
    with ShotSolver(p, max_rec=ntr, snap_format=snap) as s:
        s.upload_model(model)
        sig = np.ascontiguousarray(sig[:, ::-1])  # energy in the first step, the one that is stored
        s.setup_shot(0, g.srcpos, sig, g.recpos)
        s.forward(1, store=True, fetch=False)
        f = s.snapshot(0)
        grads = s.adjoint(adj[None])[0]
        a = s.fields(0)
    if name == "sh_el_o6":
        want = {7: f[0] * a[10]}
    elif name == "acoustic_o4_p":
        want = {0: f[2] * a[11], 2: a[5] * f[0] + a[6] * f[1]}
    else:
        want = {0: (f[2] + f[3]) * (a[2] + a[3]), 2: a[5] * f[0] + a[6] * f[1]}
    for plane, w in want.items():
        assert bit_equal(grads[plane] + 0.0, w.astype(np.float32) + np.float32(0.0)), plane


def test_shared_coefficients_match_single_shots():
    """A batch large enough that the viscoelastic stress takes the model's
    coefficients past its ring (two models, ragged rows): every slot equals
    the same shot alone."""
    nx, ny, n = 703, 431, 14  # 303 000 cells, 4.2 million in the batch
    p, model, g, sig, adj = build_case("psv_visc_o8_holberg", nx=nx, ny=ny, nt=12, fw=20)
    p.dtinv = 3
    ntr = g.recpos.shape[1]
    models = [model, {k: (v * np.float32(1.01) if k != "rho" else v) for k, v in model.items()}]
    alone = []
    for m in models:
        with ShotSolver(p, max_rec=ntr) as s:
            s.upload_model(m)
            s.setup_shot(0, g.srcpos, sig, g.recpos)
            alone.append((s.forward(1)[0], s.adjoint(adj[None])[0]))
    with ShotSolver(p, max_shots=n, max_models=2, max_rec=ntr) as s:
        s.set_options(tile_order=3)
        for k, m in enumerate(models):
            s.upload_model(m, k)
        for k in range(n):
            s.setup_shot(k, g.srcpos, sig, g.recpos, model=k % 2)
        sec = s.forward(n)
        grads = s.adjoint(np.stack([adj] * n), n)
    for k in range(n):
        assert bit_equal(sec[k], alone[k % 2][0]) and bit_equal(grads[k], alone[k % 2][1]), k


@pytest.mark.parametrize("nx", [129, 130, 131, 132])
@pytest.mark.parametrize("name", ["psv_el_o4", "psv_el_o2_nofs"])
def test_batches_match_single_shots_of_a_tile_per_sm(name, nx):
    """FDORDER 2 and 4 elastic launches of at most a tile per SM use two cells
    a thread, larger ones four: a batch of 12 (180 tiles) equals the single
    shot (15 tiles), which equals the oracle."""
    p, model, g, sig, adj = build_case(name, nx=nx, ny=33, nt=40, fw=9)
    ntr, n = g.recpos.shape[1], 12
    ref = oracle_shot(p, model, g, sig, adj)
    with ShotSolver(p, max_shots=n, max_rec=ntr) as s:
        s.upload_model(model)
        for k in range(n):
            s.setup_shot(k, g.srcpos, sig, g.recpos)
        sec = s.forward(n)
        grads = s.adjoint(np.stack([adj] * n), n)
    for k in range(n):
        assert bit_equal(sec[k], ref["sections"]) and bit_equal(grads[k], ref["grads"]), k


@pytest.mark.parametrize("nx", [130, 131])
@pytest.mark.parametrize("name,n", [("psv_el_o4", 42), ("psv_el_o2_nofs", 42), ("psv_el_o8_holberg", 12),
                                    ("psv_el_o12_ref", 12), ("psv_el_o12_ref", 42)])
def test_batches_of_few_and_more_tiles_per_sm(name, n, nx):
    """The P-SV launches change from two to four cells a thread above one or
    four tiles per SM (by FDORDER): batches on both sides (12 and 42 shots, 180
    and 630 tiles) and the single shot (15 tiles) equal the oracle."""
    p, model, g, sig, adj = build_case(name, nx=nx, ny=33, nt=40, fw=9)
    ntr = g.recpos.shape[1]
    ref = oracle_shot(p, model, g, sig, adj)
    for shots in (1, n):
        with ShotSolver(p, max_shots=shots, max_rec=ntr) as s:
            s.upload_model(model)
            for k in range(shots):
                s.setup_shot(k, g.srcpos, sig, g.recpos)
            sec = s.forward(shots)
            grads = s.adjoint(np.stack([adj] * shots), shots)
        for k in range(shots):
            assert bit_equal(sec[k], ref["sections"]) and bit_equal(grads[k], ref["grads"]), k


@pytest.mark.parametrize("fdorder,L", [(2, 3), (4, 3), (6, 1), (8, 1), (12, 1), (12, 3), (4, 4), (8, 4), (8, 2), (10, 3)])
def test_large_viscoelastic_batches_by_order_and_mechanisms(fdorder, L):
    """Each form that a large viscoelastic batch takes by FDORDER and L
    (coefficients in registers or through the ring, with and without CPML in
    the stress): every slot equals the same shot alone, which takes the ring."""
    nx, ny, n = 703, 431, 14  # 303 000 cells, 4.2 million in the batch
    p, model, g, sig, adj = build_case("psv_visc_o4", nx=nx, ny=ny, nt=9, fw=20)
    p.dtinv, p.fdorder = 3, fdorder
    p.L, p.fl = L, [5.0 * 2 ** k for k in range(L)]
    ntr = g.recpos.shape[1]
    with ShotSolver(p, max_rec=ntr) as s:
        s.upload_model(model)
        s.setup_shot(0, g.srcpos, sig, g.recpos)
        alone = s.forward(1)[0], s.adjoint(adj[None])[0]
    with ShotSolver(p, max_shots=n, max_rec=ntr) as s:
        s.set_options(tile_order=3)
        s.upload_model(model)
        for k in range(n):
            s.setup_shot(k, g.srcpos, sig, g.recpos)
        sec = s.forward(n)
        grads = s.adjoint(np.stack([adj] * n), n)
    for k in range(n):
        assert bit_equal(sec[k], alone[0]) and bit_equal(grads[k], alone[1]), k
    assert np.abs(alone[1]).max() > 0
