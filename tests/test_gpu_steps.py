"""The kernels of small batches (sources, surface and receivers folded into the two updates,
overlapping launches), bit-identical to the float restatement (itself pinned to the reference),
against the separate kernels at the sizes where the folding can go wrong."""
import numpy as np
import pytest

import denise_b200 as dn

import oracles as O
from test_gpu_fused import _case
from test_gpu_parity import _residuals, gpu_shot

pytestmark = pytest.mark.gpu

FIELDS = (("vx", 0), ("vy", 1), ("sxx", 2), ("syy", 3), ("sxy", 4))


def _check(p, model, src, rec, shot, comps):
    ref = O.Restatement(p, model, src, rec, "f")
    ref.forward(store=False)
    for c in comps:
        np.testing.assert_array_equal(shot.sections(c), ref.sections(c), err_msg=f"section {c}")
    for name, fid in FIELDS:
        np.testing.assert_array_equal(shot.field(fid), ref.field(fid), err_msg=name)


# odd and lone last columns, tiles of one row and more, fewer rows than a tile, sources in the
# surface row and on tile edges, every order, several mechanisms
SMALL = [
    dict(nx=131, ny=37, fdorder=8, src_ij=[(66, 1)]),
    dict(nx=131, ny=37, fdorder=8, src_ij=[(66, 2), (128, 5)]),
    dict(nx=129, ny=20, fdorder=12, styp=3, src_ij=[(128, 7)]),
    dict(nx=63, ny=41, fdorder=2, styp=2),
    dict(nx=300, ny=70, fdorder=4, free_surf=0, styp=4),
    dict(nx=140, ny=33, fdorder=10, L=1),
    dict(nx=90, ny=29, fdorder=6, L=3, src_ij=[(45, 1)]),
    dict(nx=19, ny=15, fdorder=8, src_ij=[(9, 3)]),   # CPML sides overlap
    dict(nx=257, ny=24, fdorder=8, L=5, free_surf=0, styp=2),
]
IDS = [f"{c['nx']}x{c['ny']}-fd{c['fdorder']}-L{c.get('L', 0)}-{k}" for k, c in enumerate(SMALL)]


@pytest.mark.parametrize("way", ["default", "paired", "injected"])
@pytest.mark.parametrize("case", SMALL, ids=IDS)
def test_small_batch_steps_bitexact(monkeypatch, case, way):
    """The default way (the small kernels for L = 0), without the small kernels, and with the surface,
    receivers and sources in kernels of their own; the launch count tells a folded step (two
    launches) from the last."""
    if way != "default":
        monkeypatch.setenv("DN_SMALL", "0")
    if way == "injected":
        monkeypatch.setenv("DN_SRC_IN_KERNEL", "0")
    p, model, src, rec = _case(nt=120, **case)
    p = p.replace(seismo=1)
    m, s = gpu_shot(p, model, src, rec)
    dn.run([s], dn.MODE_FORWARD)
    assert (dn.last_run_stats()[1] <= 2 * 150 + 3) == (way != "injected")
    _check(p, model, src, rec, s, (0, 1))


@pytest.mark.parametrize("rows", [1, 3])
def test_small_batch_of_unequal_shots(monkeypatch, rows):
    """Shots of different sizes and step counts, tiles of one row and of three; a second run repeats
    the first."""
    monkeypatch.setenv("DN_TILE", f"128x{rows}")
    cases = [_case(nx=131, ny=37, nt=90, seed=1), _case(nx=300, ny=21, nt=140, styp=2, seed=2),
             _case(nx=64, ny=64, nt=61, free_surf=0, seed=5)]
    pairs = [gpu_shot(*c) for c in cases]
    for _ in range(2):
        dn.run([s for _, s in pairs], dn.MODE_FORWARD)
        for c, (_, s) in zip(cases, pairs):
            _check(*c, s, range(5))


@pytest.mark.parametrize("quelltypb", [1, 4])
@pytest.mark.parametrize("rec_row", [1, 2, 4])
@pytest.mark.parametrize("L", [0, 2])
def test_small_batch_gradient_bitexact(L, rec_row, quelltypb):
    """Forward with snapshots and adjoint; adjoint pressures in the surface row (its own kernel),
    in a mirrored row (the image follows the injection) and below."""
    p, model, src, rec = _case(nx=150, ny=41, nt=120, L=L, store_snapshots=1)
    p = p.replace(quelltypb=quelltypb, seismo=1)
    rec = (rec[0], np.full_like(rec[1], rec_row))
    m, s = gpu_shot(p, model, src, rec)
    dn.run([s], dn.MODE_FORWARD)
    ref = O.Restatement(p, model, src, rec, "f")
    ref.forward(store=True)
    rvx, rvy = _residuals(p, s.sections(0), s.sections(1))
    rp = (0.5 * rvx).astype(np.float32) if quelltypb >= 4 else None
    s.set_residuals(rvx, rvy, rp)
    ref.adjoint(rvx, rvy, rp)
    dn.run([s], dn.MODE_ADJOINT)
    s.accumulate_gradient()
    for a, b in zip(m.gradient(), ref.gradient()):
        np.testing.assert_array_equal(a, b)
