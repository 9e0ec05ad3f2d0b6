"""FP64 drop-in path on the GPU against the FP64 CPU oracle, phase by phase,
through the C ABI.  Tolerances are relative to the largest magnitude of the
oracle's output (FP64; the GPU sums in a different order and the ADI solve is
a reassociated Thomas recurrence)."""
import math

import numpy as np
import pytest

from genesis4_cuda_port_b200 import device as dev
from genesis4_cuda_port_b200._lib import G4BError
from oracle import pyoracle as orc
from tests import synth

pytestmark = pytest.mark.gpu

TOL = 1e-12


@pytest.fixture(scope="module")
def ctx():
    c = dev.Context(0)
    yield c
    c.synchronize()


def _beam(ctx, off, parts, current=None):
    b = dev.BeamState(ctx, off, synth.GAMMA0)
    b.upload(parts)
    b.set_current(current if current is not None else np.full(len(off) - 1, synth.CURRENT))
    return b


@pytest.mark.parametrize("ngrid,nslice", [(7, 3), (33, 2), (64, 2), (151, 1), (201, 2), (301, 1)])
def test_adi_without_source(ctx, ngrid, nslice):
    gridmax = 200e-6
    f0 = synth.field(nslice, ngrid, gridmax, seed=ngrid)
    step = synth.drift_step(delz=0.015)
    off = np.zeros(nslice + 1, np.int64)
    parts = {k: np.zeros(0) for k in synth.copy_parts(synth.beam(1, 1)[1])}
    fld = dev.FieldState(ctx, nslice, ngrid, gridmax, synth.LAMBDA0)
    fld.upload(f0)
    beam = _beam(ctx, off, {k: np.zeros(0) for k in parts})
    adi = dev.FieldSolverADICUDA(ctx)
    adi.init(step.delz, fld.dgrid, fld.xks, ngrid)
    ref = f0.copy()
    for _ in range(3):
        adi.advance(fld, beam, step, fc=0.0)
        orc.adi_advance(ref, harm=1, gridmax=gridmax, xks=fld.xks, delz=step.delz, fc=0.0,
                        enabled=True, step=step, off=off, current=np.zeros(nslice), parts=parts)
    got = fld.download()
    assert synth.rel_err(got, ref) < TOL


# the row solve at the edges of its lanes (one element, a last lane of one or of
# all its elements) and of its coefficients: r = delz / (4 ks dgrid^2) from the
# configurations' 0.02 to 40 (|q| near 1), backwards
# and zero.  The recurrences are stable and the matrix's condition number is
# below 1 + 4 |r|, so a step errs by at most some n (1 + 4 |r|) roundings.
@pytest.mark.parametrize("r", [0.02, 1.0, 40.0, -0.5, 0.0])
@pytest.mark.parametrize("ngrid", [2, 3, 16, 32, 33, 80, 81, 160, 161, 257])
def test_adi_row_solve_at_its_edges(ctx, ngrid, r):
    nslice, gridmax = 2, 200e-6
    f0 = synth.field(nslice, ngrid, gridmax, seed=ngrid)
    xks, dgrid = 2 * np.pi / synth.LAMBDA0, 2 * gridmax / (ngrid - 1)
    step = synth.drift_step(delz=4 * r * xks * dgrid ** 2)
    off = np.zeros(nslice + 1, np.int64)
    parts = {k: np.zeros(0) for k in dev.BeamState.NAMES}
    ref = f0.copy()
    for _ in range(2):
        orc.adi_advance(ref, harm=1, gridmax=gridmax, xks=xks, delz=step.delz, fc=0.0,
                        enabled=True, step=step, off=off, current=np.zeros(nslice), parts=parts)
    bound = 4 * ngrid * (1 + 4 * abs(r))
    fld = dev.FieldState(ctx, nslice, ngrid, gridmax, synth.LAMBDA0)
    fld.upload(f0)
    adi = dev.FieldSolverADICUDA(ctx)
    adi.init(step.delz, fld.dgrid, fld.xks, ngrid)
    beam = _beam(ctx, off, parts)
    for _ in range(2):
        adi.advance(fld, beam, step, fc=0.0)
    assert synth.rel_err(fld.download(), ref) < bound * 2.0 ** -53
    run = dev.Run(ctx, off, fields=[(1, ngrid, gridmax)], lambda0=synth.LAMBDA0,
                  gamma_ref=synth.GAMMA0, time_run=False)
    run.upload_field(0, f0)
    run.set_lattice([step] * 2, [[0.0]] * 2, [0.0] * 2)
    for layout in {run.layouts()[0], 107 if ngrid == 81 else run.layouts()[0]}:
        run.upload_field(0, f0)
        run.set_layouts([layout])
        run.advance(0, 2, graph=False)
        assert synth.rel_err(run.download_field(0)[0], ref) < bound * 2.0 ** -24
    run.close()


# Far from a localised field the solution falls by |q| per cell, over hundreds of
# orders of magnitude, and stays relatively accurate: each cell is a product of
# up to 2 n powers, so some 4 n roundings.
@pytest.mark.parametrize("ngrid", [64, 151, 182, 201])
def test_adi_far_field_is_relatively_accurate(ctx, ngrid):
    gridmax = 200e-6
    f0 = np.zeros((1, ngrid, ngrid), np.complex128)
    f0[0, ngrid // 2, ngrid // 2] = 1e12
    fld = dev.FieldState(ctx, 1, ngrid, gridmax, synth.LAMBDA0)
    fld.upload(f0)
    step = synth.drift_step(delz=0.015)
    off = np.zeros(2, np.int64)
    parts = {k: np.zeros(0) for k in dev.BeamState.NAMES}
    adi = dev.FieldSolverADICUDA(ctx)
    adi.init(step.delz, fld.dgrid, fld.xks, ngrid)
    adi.advance(fld, _beam(ctx, off, parts), step, fc=0.0)
    orc.adi_advance(f0, harm=1, gridmax=gridmax, xks=fld.xks, delz=step.delz, fc=0.0,
                    enabled=True, step=step, off=off, current=np.zeros(1), parts=parts)
    got = fld.download()
    ok = np.abs(f0) > 1e-280
    assert ok.sum() > 0.5 * ok.size
    assert np.max(np.abs(got[ok] - f0[ok]) / np.abs(f0[ok])) < 4 * ngrid * 2.0 ** -53


@pytest.mark.parametrize("ngrid,nslice,first", [(33, 3, 1), (151, 2, 0), (201, 3, 2)])
def test_adi_with_deposited_source(ctx, ngrid, nslice, first):
    gridmax = 200e-6
    off, parts = synth.beam(nslice, 3000, seed=ngrid, ragged=True)
    f0 = synth.field(nslice, ngrid, gridmax, seed=7)
    step = synth.und_step()
    fc = synth.coupling()
    cur = np.linspace(1000, 3000, nslice)
    fld = dev.FieldState(ctx, nslice, ngrid, gridmax, synth.LAMBDA0)
    fld.upload(f0)
    fld.first = first
    beam = _beam(ctx, off, parts, cur)
    adi = dev.FieldSolverADICUDA(ctx)
    adi.init(step.delz, fld.dgrid, fld.xks, ngrid)
    adi.advance(fld, beam, step, fc=fc)
    ref = f0.copy()
    orc.adi_advance(ref, harm=1, gridmax=gridmax, xks=fld.xks, delz=step.delz, fc=fc,
                    enabled=True, step=step, off=off, current=cur, parts=parts, first=first)
    got = fld.download()
    assert synth.rel_err(got, ref) < TOL
    # the source alone (field zero) is also reproduced
    fld.upload(np.zeros_like(f0))
    adi.advance(fld, beam, step, fc=fc)
    ref = np.zeros_like(f0)
    orc.adi_advance(ref, harm=1, gridmax=gridmax, xks=fld.xks, delz=step.delz, fc=fc,
                    enabled=True, step=step, off=off, current=cur, parts=parts, first=first)
    assert synth.rel_err(fld.download(), ref) < 1e-11


def test_deposit_is_deterministic(ctx):
    nslice, ngrid, gridmax = 2, 151, 200e-6
    off, parts = synth.beam(nslice, 20000, seed=11)
    step = synth.und_step()
    outs = []
    for _ in range(2):
        fld = dev.FieldState(ctx, nslice, ngrid, gridmax, synth.LAMBDA0)
        beam = _beam(ctx, off, parts)
        adi = dev.FieldSolverADICUDA(ctx)
        adi.init(step.delz, fld.dgrid, fld.xks, ngrid)
        adi.advance(fld, beam, step, fc=synth.coupling())
        outs.append(fld.download())
    assert np.array_equal(outs[0], outs[1])


def test_source_off_outside_undulator_and_for_even_harmonics(ctx):
    nslice, ngrid, gridmax = 1, 33, 200e-6
    off, parts = synth.beam(nslice, 500, seed=12)
    beam = _beam(ctx, off, parts)
    for step, harm in [(synth.drift_step(delz=0.015), 1), (synth.und_step(), 2)]:
        fld = dev.FieldState(ctx, nslice, ngrid, gridmax, synth.LAMBDA0 / harm, harm=harm)
        adi = dev.FieldSolverADICUDA(ctx)
        adi.init(step.delz, fld.dgrid, fld.xks, ngrid)
        adi.advance(fld, beam, step, fc=synth.coupling())
        assert not np.any(fld.download())


@pytest.mark.parametrize("kind", ["drift", "fquad", "und", "chicane", "corrector"])
def test_transverse_track(ctx, kind):
    off, parts = synth.beam(3, 700, seed=13, ragged=True)
    steps = {
        "drift": (synth.drift_step(delz=0.2), False),
        "fquad": (synth.drift_step(delz=0.1, qf=1.5, dqx=1e-5, dqy=-2e-5), False),
        "und": (synth.und_step(ax=3e-6, ay=-2e-6, kx=0.3 * synth.KU ** 2), False),
        "chicane": (synth.drift_step(delz=0.1, chic_angle=2e-3, chic_lb=0.02,
                                     chic_ld=0.01, chic_lt=0.1), False),
        "corrector": (synth.drift_step(delz=0.1, cx=1e-6, cy=-3e-6), True),
    }
    step, last = steps[kind]
    beam = _beam(ctx, off, parts)
    beam.track(step, step.delz * 0.5, last)
    ref = synth.copy_parts(parts)
    orc.track(ref, step, step.delz * 0.5, last)
    got = beam.download()
    for k in ("x", "y", "px", "py"):
        assert synth.rel_err(got[k], ref[k]) < TOL, k


def test_r56(ctx):
    off, parts = synth.beam(2, 500, seed=14)
    step = synth.drift_step(delz=0.1, chic_angle=2e-3, chic_lb=0.02, chic_ld=0.01, chic_lt=0.1)
    beam = _beam(ctx, off, parts)
    beam.apply_r56(step, synth.LAMBDA0)
    ref = synth.copy_parts(parts)
    orc.r56(ref, step, synth.LAMBDA0)
    assert synth.rel_err(beam.download()["theta"], ref["theta"]) < TOL


@pytest.mark.parametrize("nfield", [1, 2])
def test_push(ctx, nfield):
    nslice, ngrid, gridmax = 3, 65, 150e-6
    off, parts = synth.beam(nslice, 2000, seed=15, ragged=True)
    step = synth.und_step(autophase=0.1)
    eloss = np.array([1e-3, -2e-3, 0.0])
    beam = _beam(ctx, off, parts)
    beam.set_eloss(eloss)
    flds, views, fcs = [], [], []
    for i in range(nfield):
        h = 1 + 2 * i
        cells = synth.field(nslice, ngrid, gridmax, seed=20 + i, amplitude=3e13)
        f = dev.FieldState(ctx, nslice, ngrid, gridmax, synth.LAMBDA0 / h, harm=h)
        f.upload(cells)
        f.first = i % nslice
        flds.append(f)
        fcs.append(synth.coupling(harm=h))
        views.append(dict(cells=cells, first=i % nslice, harm=h, gridmax=gridmax,
                          xlambda=synth.LAMBDA0 / h, fc=fcs[-1]))
    beam.advance(flds, fcs, step)
    ref = synth.copy_parts(parts)
    orc.push(off, step, views, ref, slice_eloss=eloss)
    got = beam.download()
    # gamma changes by a small amount: compare the change
    dg = got["gamma"] - parts["gamma"]
    dg_ref = ref["gamma"] - parts["gamma"]
    assert np.max(np.abs(dg_ref)) > 1e-6
    assert synth.rel_err(dg, dg_ref) < 1e-10
    assert synth.rel_err(got["theta"], ref["theta"]) < TOL


def test_slippage_bit_exact(ctx):
    nslice, ngrid = 6, 17
    f0 = synth.field(nslice, ngrid, 100e-6, seed=30)
    fld = dev.FieldState(ctx, nslice, ngrid, 100e-6, synth.LAMBDA0)
    fld.upload(f0)
    ref = f0.copy()
    acc, first = 0.0, 0
    for shift in [1.0, 2.6, -0.4, -1.7, 0.5, 3.0]:
        n_gpu = fld.apply_slippage(shift, 1.0)
        acc, first, n_ref = orc.slippage(ref, shift, 1.0, True, False, acc, first)
        assert n_gpu == n_ref and fld.first == first
        assert fld.accuslip == acc
    assert np.array_equal(fld.download(), ref)


@pytest.mark.parametrize("need_aux,nharm", [(True, 1), (False, 3), (True, 10)])
def test_beam_diagnostics(ctx, need_aux, nharm):
    off, parts = synth.beam(4, 1500, seed=31, ragged=True)
    beam = _beam(ctx, off, parts)
    stats, bre, bim = beam.diagnostics(nharm, need_aux)
    rs, rbre, rbim = orc.diag_beam(off, parts, nharm, need_aux)
    np.testing.assert_allclose(stats, rs, rtol=1e-12, atol=1e-300)
    np.testing.assert_allclose(bre, rbre, rtol=1e-9, atol=1e-9)
    np.testing.assert_allclose(bim, rbim, rtol=1e-9, atol=1e-9)


def test_field_diagnostics(ctx):
    nslice, ngrid = 4, 45
    f0 = synth.field(nslice, ngrid, 100e-6, seed=32)
    fld = dev.FieldState(ctx, nslice, ngrid, 100e-6, synth.LAMBDA0)
    fld.upload(f0)
    fld.first = 3
    stats, center = fld.diagnostics()
    rs, rc = orc.diag_field(f0, 3)
    np.testing.assert_allclose(stats, rs, rtol=1e-11, atol=1e-12 * np.max(np.abs(rs)))
    np.testing.assert_array_equal(center, rc)


def test_full_steps_match_oracle(ctx):
    """Five Gencore steps (beam track/advance/R56/track, field track, slippage)
    in the reference order, through the per-phase entry points."""
    nslice, ngrid, gridmax = 4, 65, 160e-6
    off, parts = synth.beam(nslice, 1500, seed=40)
    cells = synth.field(nslice, ngrid, gridmax, seed=41, amplitude=1e12)
    cur = np.full(nslice, synth.CURRENT)
    fc = synth.coupling()
    beam = _beam(ctx, off, parts, cur)
    fld = dev.FieldState(ctx, nslice, ngrid, gridmax, synth.LAMBDA0)
    fld.upload(cells)
    adi = dev.FieldSolverADICUDA(ctx)
    ref_parts = synth.copy_parts(parts)
    ref_field = dict(cells=cells.copy(), gridmax=gridmax, xlambda=synth.LAMBDA0, fc=fc,
                     first=0, accuslip=0.0)
    steps = [synth.und_step(), synth.und_step(), synth.drift_step(delz=0.05, qf=1.5),
             synth.und_step(), synth.und_step()]
    for st in steps:
        slip = 1.0 if st.in_undulator else 0.3
        fcs = fc if st.in_undulator else 0.0
        beam.track(st, st.delz * 0.5, False)
        beam.advance([fld], [fcs], st)
        beam.apply_r56(st, synth.LAMBDA0)
        beam.track(st, st.delz * 0.5, True)
        adi.init(st.delz, fld.dgrid, fld.xks, ngrid)
        adi.advance(fld, beam, st, fc=fcs)
        fld.apply_slippage(slip, 1.0)
        ref_field["fc"] = fcs
        orc.step(off, cur, st, synth.LAMBDA0, slip, 1.0, True, False, [ref_field], ref_parts)
    got = beam.download()
    for k in parts:
        assert synth.rel_err(got[k], ref_parts[k]) < 1e-11, k
    assert fld.first == ref_field["first"]
    assert synth.rel_err(fld.download(), ref_field["cells"]) < 1e-11


# slices split over several CTAs (down to 512 particles and 16 rows each) and
# not, one harmonic pass and several, particle counts off every tile.  The sums
# are FP64 additions of at most N terms: a few N roundings of the largest.
@pytest.mark.parametrize("nslice,npart,ngrid,nharm", [(1, 1, 2, 1), (1, 513, 17, 2), (1, 9001, 151, 4),
                                                      (3, 2047, 64, 5), (40, 700, 33, 9),
                                                      (700, 300, 9, 1)])
def test_diagnostics_split_over_ctas(ctx, nslice, npart, ngrid, nharm):
    off, parts = synth.beam(nslice, npart, seed=nslice, ragged=nslice > 1)
    beam = _beam(ctx, off, parts)
    got, want = beam.diagnostics(nharm, True), orc.diag_beam(off, parts, nharm, True)
    for g, w in zip(got, want):
        assert np.max(np.abs(g - w) / np.maximum(np.max(np.abs(w), 0), 1.0)) < 8 * npart * 2.0 ** -53
    f0 = synth.field(nslice, ngrid, 160e-6, seed=3, amplitude=2e12)
    fld = dev.FieldState(ctx, nslice, ngrid, 160e-6, synth.LAMBDA0)
    fld.upload(f0)
    fld.first = nslice // 2
    st, cen = fld.diagnostics()
    rs, rc = orc.diag_field(f0, nslice // 2)
    assert np.max(np.abs(st - rs) / np.max(np.abs(rs), 0)) < 8 * ngrid ** 2 * 2.0 ** -53
    assert np.array_equal(cen, rc)


# One particle per slice, so each sum is one cosine or sine: within the 2 ulp of
# CUDA's sincos and the rounding of the correction for the product h theta, 3 x
# 2^-53, at every harmonic and phase (the product itself is exact in 64 bits).
@pytest.mark.parametrize("nharm", [1, 4, 5, 9])
@pytest.mark.parametrize("span", [0.1, 3.2, 400.0])
def test_bunching_harmonics_are_single_sines(ctx, nharm, span):
    ns = 1000
    off, parts = synth.beam(ns, 1, seed=nharm)
    parts["theta"] = np.random.default_rng(nharm).uniform(-span, span, ns)
    beam = _beam(ctx, off, parts)
    _, re, im = beam.diagnostics(nharm, True)
    for h in range(nharm):
        ph = parts["theta"].astype(np.longdouble) * (h + 1)
        assert np.max(np.abs(re[:, h] - np.cos(ph))) <= 3 * 2.0 ** -53
        assert np.max(np.abs(im[:, h] - np.sin(ph))) <= 3 * 2.0 ** -53
    beam.close()


# split slices (up to 148), whole ones in the caller's layout above; sums of up to
# 700 terms round 9 (terms per thread) + 5 + 8 + 9 (parts) times at most, the
# field's of 33^2 up to 5 + 33 + 5 + 8 + 3
@pytest.mark.parametrize("ns", [1, 148, 149, 600])
@pytest.mark.parametrize("nharm, aux", [(1, True), (5, False)])
def test_diagnostics_of_split_and_whole_slices(ctx, ns, nharm, aux):
    off, parts = synth.beam(ns, 700, seed=ns, ragged=True)
    beam = _beam(ctx, off, parts)
    st, re, im = beam.diagnostics(nharm, aux)
    p = {k: v.astype(np.longdouble) for k, v in parts.items()}
    cols = [p["gamma"], p["gamma"] ** 2, p["x"], p["x"] ** 2, p["y"], p["y"] ** 2, p["px"],
            p["px"] ** 2, p["py"], p["py"] ** 2, p["x"] * p["px"], p["y"] * p["py"]]
    cols += [f(p["theta"] * (h + 1)) for h in range(nharm) for f in (np.cos, np.sin)]
    got = [st[:, k] for k in range(12)] + [a[:, h] for h in range(nharm) for a in (re, im)]
    assert np.array_equal(st[:, 12], np.diff(off))
    for s in range(ns):
        o = slice(off[s], off[s + 1])
        for v, g in zip(cols, got):
            assert abs(g[s] - v[o].sum()) <= (31 + 3) * 2.0 ** -53 * np.abs(v[o]).sum() + 1e-300
        for k, (name, lo, hi) in enumerate((("x", 1e5, -1e5), ("px", 1e5, -1e5), ("y", 1e5, -1e5),
                                            ("py", 1e5, -1e5), ("gamma", 1e7, 1.0))):
            want = (min([lo, *parts[name][o]]), max([hi, *parts[name][o]])) if aux else (0.0, 0.0)
            assert tuple(st[s, 13 + 2 * k:15 + 2 * k]) == want
    n = 33
    fld = dev.FieldState(ctx, ns, n, 150e-6, synth.LAMBDA0)
    cells = synth.field(ns, n, 150e-6, seed=5, amplitude=1e11)
    fld.upload(cells)
    stats, center = fld.diagnostics()
    u, d = cells.astype(np.clongdouble), np.arange(n) - np.longdouble(0.5 * (n - 1))
    w = u.real ** 2 + u.imag ** 2
    for k, v in enumerate((w, w * d, w * d * d, w * d[:, None], w * d[:, None] ** 2, u.real, u.imag)):
        assert np.all(np.abs(stats[:, k] - v.sum((1, 2))) <= 58 * 2.0 ** -53 * np.abs(v).sum((1, 2)))
    assert np.array_equal(center, np.stack([cells.real, cells.imag], -1)[:, n // 2, n // 2])
    for o in (fld, beam):
        o.close()


def test_deposition_takes_every_weight_up_to_its_limit(ctx):
    """Charge weights up to 1e300 are taken: with gamma 2^-980 of its value and
    the current 2^-200 the source is 2^780 times as large, bit for bit; a weight
    above the limit is reported."""
    ngrid, gridmax = 33, 150e-6
    off, parts = synth.beam(2, 500, seed=61)
    step, got = synth.und_step(), []
    for eg, ec in ((0, 0), (-980, -200), (-1020, -200)):
        p = dict(parts, gamma=parts["gamma"] * 2.0 ** eg)
        beam = _beam(ctx, off, p, np.full(2, synth.CURRENT * 2.0 ** ec))
        fld = dev.FieldState(ctx, 2, ngrid, gridmax, synth.LAMBDA0)
        fld.upload(np.zeros((2, ngrid, ngrid), np.complex128))
        adi = dev.FieldSolverADICUDA(ctx)
        adi.init(step.delz, fld.dgrid, fld.xks, ngrid)
        adi.advance(fld, beam, step, fc=synth.coupling())
        if eg == -1020:
            with pytest.raises(G4BError, match="fixed-point range"):
                ctx.synchronize()
        else:
            ctx.synchronize()
            got.append(fld.download())
        for o in (adi, fld, beam):
            o.close()
    assert np.max(np.abs(got[0])) > 0
    assert np.array_equal(got[1] * 2.0 ** -780, got[0])
