"""Which kernels a batch takes (dn_last_run_route), and every elastic way against the float
restatement (itself pinned to the reference): the sizes of the other tests lie below the line of
the small kernels, so the paired kernels with and without the work folded into them, which larger
batches take, are asked for here."""
import numpy as np
import pytest

import denise_b200 as dn
from denise_b200 import synth

import oracles as O
import test_gpu_parity as P
from test_gpu_fused import _case
from test_gpu_parity import gpu_shot, small_case

pytestmark = pytest.mark.gpu

WAYS = {"paired": {"DN_SMALL": "0"}, "separate": {"DN_SRC_IN_KERNEL": "0"}}


def _take(monkeypatch, way):
    for k, v in WAYS.get(way, {}).items():
        monkeypatch.setenv(k, v)


def _taken(way, L=0):
    names, _ = dn.last_run_route()
    assert ("small" in names) == (way == "default" and L == 0), names
    assert ("src" in names) == (way != "separate"), names
    assert "paired" in names


@pytest.mark.parametrize("nx,ny,L,fw,nsrc,env,small,src,rows", [
    (546, 549, 0, 10, 1, {}, True, True, 1),          # 299,754 cells: the last of the small kernels
    (546, 550, 0, 10, 1, {}, False, True, 1),
    (64, 48, 1, 10, 1, {}, False, True, 1),           # elastic only
    (39, 60, 0, 20, 1, {}, False, True, 1),           # a column in both CPML sides
    (40, 40, 0, 20, 1, {}, True, True, 1),
    (64, 48, 0, 10, 9, {}, False, False, 1),          # more source cells than the kernels take
    (64, 48, 0, 10, 1, {"DN_SMALL": "0"}, False, True, 1),
    (64, 48, 0, 10, 1, {"DN_SRC_IN_KERNEL": "0"}, False, False, 1),
    (1300, 1000, 0, 10, 1, {}, False, True, 2),
    (2500, 2000, 0, 10, 1, {}, False, False, 4),
])
def test_route_of_a_batch(monkeypatch, nx, ny, L, fw, nsrc, env, small, src, rows):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    p = synth.c0_params(nx=nx, ny=ny, nt=4, fw=fw, L=L, fl=(2.0,)[:L], ts=0.1, seismo=1)
    one = np.ones((nx, ny), np.float32)
    m = dn.Model(p, 3000 * one, 1700 * one, 2000 * one, *([50 * one] * 2 if L else []))
    si = np.arange(10, 10 + 2 * nsrc, 2, dtype=np.int32)
    s = dn.Shot(m, si, np.full(nsrc, 3, np.int32), np.ones((nsrc, p.nt), np.float32), si, np.full(nsrc, 4, np.int32))
    dn.run([s], dn.MODE_FORWARD)
    names, got = dn.last_run_route()
    assert (("small" in names), ("src" in names), got) == (small, src, rows), names


@pytest.mark.parametrize("fdorder,ny,shots,seismo,small", [
    (12, 166, 2, 4, True), (12, 167, 2, 4, False),     # 4 x 166 x 2 of at most 9 x 148 blocks
    (12, 167, 2, 1, True), (10, 167, 2, 4, True), (12, 334, 1, 4, True)])
def test_route_past_one_wave_of_blocks(fdorder, ny, shots, seismo, small):
    """FDORDER 12 shots without folded work leave the small kernels soon after one wave of their blocks."""
    p = synth.c0_params(nx=500, ny=ny, nt=4, fw=10, fdorder=fdorder, free_surf=0, seismo=seismo)
    one = np.ones((500, ny), np.float32)
    m = dn.Model(p, 3000 * one, 1700 * one, 2000 * one)
    at = [np.array([k], np.int32) for k in (50, 60, 40)]
    batch = [dn.Shot(m, at[0], at[2], np.ones((1, 4), np.float32), at[1], at[2]) for _ in range(shots)]
    dn.run(batch, dn.MODE_FORWARD)
    assert ("small" in dn.last_run_route()[0]) == small


FORWARD = [c for c in P.CASES + P.ODD if c.get("L", 0) == 0]
FORWARD += [dict(L=0, fdorder=6, nx=65, ny=33, free_surf=0, styp=4), dict(L=0, fdorder=10, nx=131, ny=37, free_surf=0),
            dict(L=0, fdorder=10, nx=130, ny=40, styp=1)]


@pytest.mark.parametrize("way", list(WAYS))
@pytest.mark.parametrize("case", FORWARD, ids=lambda c: "-".join(f"{k}{v}" for k, v in c.items()))
def test_forward_by_way(monkeypatch, case, way):
    """All five sections (k_seismo) and the final fields."""
    _take(monkeypatch, way)
    P.test_forward_bitexact(case)
    _taken(way)


@pytest.mark.parametrize("quelltypb", [1, 4])
@pytest.mark.parametrize("way", ["default"] + list(WAYS))
@pytest.mark.parametrize("fdorder", [2, 6, 8, 10, 12])
def test_gradient_by_way(monkeypatch, fdorder, way, quelltypb):
    """Snapshots, adjoint forces and (QUELLTYPB 4) pressures in a mirrored row, correlation."""
    _take(monkeypatch, way)
    p, model, src, rec = _case(fdorder=fdorder, nx=141, ny=39, nt=90, store_snapshots=1)
    p = p.replace(quelltypb=quelltypb, seismo=1)
    rec = (rec[0], np.full_like(rec[1], 2))
    m, s = gpu_shot(p, model, src, rec)
    dn.run([s], dn.MODE_FORWARD)
    _taken(way)
    ref = O.Restatement(p, model, src, rec, "f")
    ref.forward(store=True)
    for c in (0, 1):
        np.testing.assert_array_equal(s.sections(c), ref.sections(c))
    rvx, rvy = P._residuals(p, s.sections(0), s.sections(1))
    rp = (0.5 * rvx).astype(np.float32) if quelltypb >= 4 else None
    s.set_residuals(rvx, rvy, rp)
    ref.adjoint(rvx, rvy, rp)
    dn.run([s], dn.MODE_ADJOINT)
    _taken(way)
    s.accumulate_gradient()
    for a, b in zip(m.gradient(), ref.gradient()):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("way", list(WAYS))
def test_checkpoints_by_way(monkeypatch, way):
    _take(monkeypatch, way)
    P.test_checkpointed_adjoint_equals_stored_snapshots(0, dn.SNAP_F32, 39)
    _taken(way)


@pytest.mark.parametrize("L,prec", [(0, dn.SNAP_F32), (3, dn.SNAP_F32), (0, dn.SNAP_F16)])
def test_two_row_tiles_beside_four_row_snapshots(L, prec):
    """Thirty small gradient shots make a batch of 1.35 M cells: stencil tiles of two rows, the
    snapshots' own of four.  FP32 against the restatement, FP16 against the shot run alone (one-row
    stencil tiles), whose snapshots have the same tiles and scales."""
    p, model, src, rec = small_case(L=L, nx=301, ny=150, nt=60, store_snapshots=1, snap_precision=prec)
    m = dn.Model(p, *model[:3], *(model[3:5] if L else ()))
    shots = [dn.Shot(m, src[0], src[1], src[2], rec[0], rec[1], src_type=src[3], src_azi=src[4]) for _ in range(30)]

    def gradient(batch):
        dn.run(batch, dn.MODE_FORWARD)
        rows = dn.last_run_route()[1]
        rvx, rvy = P._residuals(p, batch[-1].sections(0), batch[-1].sections(1))
        for s in batch:
            s.set_residuals(rvx, rvy, None)
        dn.run(batch, dn.MODE_ADJOINT)
        assert dn.last_run_route()[1] == rows
        m.zero_gradient()
        batch[-1].accumulate_gradient()
        return rows, (rvx, rvy), m.gradient()

    rows, res, got = gradient(shots)
    assert rows == 2
    if prec == dn.SNAP_F32:
        ref = O.Restatement(p, model, src, rec, "f")
        ref.forward(store=True)
        np.testing.assert_array_equal(shots[-1].sections(0), ref.sections(0))
        ref.adjoint(*res, None)
        want = ref.gradient()
    else:
        rows, _, want = gradient(shots[-1:])
        assert rows == 1
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("way", ["default", "paired"])
@pytest.mark.parametrize("L", [0, 2])
def test_receiver_counts_of_a_folded_batch(monkeypatch, L, way):
    """More receivers than the receiver blocks' threads, few, none of the usual multiples; one shot
    keeps its surface kernel (moment tensor) beside shots that do not."""
    _take(monkeypatch, way)
    cases = []
    for n, styp, seed in ((2100, 1, 1), (7, 5, 2), (129, 3, 3)):
        p, model, src, _ = _case(nx=211, ny=37, nt=70, L=L, styp=styp, seed=seed)
        k = np.arange(n)
        cases.append((p.replace(seismo=1), model, src, ((5 + k % 200).astype(np.int32), (2 + k // 200).astype(np.int32))))
    pairs = [gpu_shot(*c) for c in cases]
    dn.run([s for _, s in pairs], dn.MODE_FORWARD)
    names, _ = dn.last_run_route()
    assert "fold" in names
    for c, (_, s) in zip(cases, pairs):
        ref = O.Restatement(*c, "f")
        ref.forward(store=False)
        for comp in (0, 1):
            np.testing.assert_array_equal(s.sections(comp), ref.sections(comp))
        for name, fid in (("vx", 0), ("vy", 1), ("sxx", 2), ("syy", 3), ("sxy", 4)):
            np.testing.assert_array_equal(s.field(fid), ref.field(fid), err_msg=name)


@pytest.mark.parametrize("L", [0, 2])
@pytest.mark.parametrize("shots,fold", [
    (((1, 1, 1),), True), (((1, 4, 1),), True), (((0, 1, 1),), True),
    (((0, 4, 1),), False),                   # neither launch goes
    (((1, 4, 1), (1, 4, 5)), False),         # a moment tensor keeps k_surface_*, stress sections k_seismo
    (((1, 1, 1), (1, 4, 5)), False),
    (((1, 1, 1), (0, 4, 1)), True),          # k_surface_* goes
    (((1, 1, 5), (0, 1, 1)), True),          # k_seismo goes
])
def test_folds_only_where_a_launch_goes(monkeypatch, shots, fold, L):
    """Shots (free surface, SEISMO, source type) of one batch in the paired kernels: the variants
    with the surface rows and receiver blocks run only if k_surface_* or k_seismo is spared."""
    _take(monkeypatch, "paired")
    cases = [_case(nx=131, ny=37, nt=80, L=L, free_surf=fs, styp=styp, seed=k) for k, (fs, _, styp) in enumerate(shots)]
    cases = [(c[0].replace(seismo=se), *c[1:]) for c, (_, se, _) in zip(cases, shots)]
    pairs = [gpu_shot(*c) for c in cases]
    dn.run([s for _, s in pairs], dn.MODE_FORWARD)
    assert ("fold" in dn.last_run_route()[0]) == fold
    for c, (_, s) in zip(cases, pairs):
        ref = O.Restatement(*c, "f")
        ref.forward(store=False)
        for comp in ((0, 1) if c[0].seismo == 1 else range(5)):
            np.testing.assert_array_equal(s.sections(comp), ref.sections(comp))
        for name, fid in (("vx", 0), ("vy", 1), ("sxx", 2), ("syy", 3), ("sxy", 4)):
            np.testing.assert_array_equal(s.field(fid), ref.field(fid), err_msg=name)
