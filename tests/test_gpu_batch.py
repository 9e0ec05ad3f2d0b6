"""Batched runs: runs of different grids, particle counts, slice counts,
tapers and lengths advanced together give exactly the results they give
alone (every work item is computed as in the single-run kernels)."""
import numpy as np
import pytest

from genesis4_cuda_port_b200 import device as dev
from tests import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = dev.Context(0)
    yield c
    c.synchronize()


CONFIGS = [
    # nslice, npart/slice, ngrid, taper, detuning, time_run, nsteps
    dict(nslice=1, npart=1024, ngrid=45, taper=0.02, dgam=0.0, time_run=False, nsteps=8),
    dict(nslice=1, npart=2048, ngrid=71, taper=0.0, dgam=3e-4, time_run=False, nsteps=8),
    dict(nslice=3, npart=512, ngrid=33, taper=0.01, dgam=-2e-4, time_run=True, nsteps=6),
    dict(nslice=2, npart=768, ngrid=101, taper=0.0, dgam=0.0, time_run=True, nsteps=7),
    # 32-lane ADI rows (the grids above use 16-lane rows): a batch of mixed
    # row layouts runs their ADI kernels on concurrent streams
    dict(nslice=2, npart=512, ngrid=151, taper=0.005, dgam=1e-4, time_run=True, nsteps=6),
]


def _inputs(k, cfg):
    off, parts = synth.beam(cfg["nslice"], cfg["npart"], seed=200 + k)
    parts["gamma"] = parts["gamma"] * (1 + cfg["dgam"])
    cells = synth.field(cfg["nslice"], cfg["ngrid"], 160e-6, seed=300 + k, amplitude=2e12)
    n = cfg["nsteps"]
    steps = [synth.und_step(aw=synth.AW * (1 - cfg["taper"] * i / n)) for i in range(n - 1)]
    steps.append(synth.drift_step(delz=0.05, qf=1.0))
    fc = [[synth.coupling(st.aw) if st.in_undulator else 0.0] for st in steps]
    slip = [st.delz * (1 + st.aw ** 2) / (2 * synth.GAMMA0 ** 2) / synth.LAMBDA0 for st in steps]
    return off, parts, cells, steps, fc, slip


def _make(ctx, k, cfg):
    off, parts, cells, steps, fc, slip = _inputs(k, cfg)
    run = dev.Run(ctx, off, fields=[(1, cfg["ngrid"], 160e-6)], lambda0=synth.LAMBDA0,
                  gamma_ref=synth.GAMMA0, sample=1.0, time_run=cfg["time_run"], nbunch=1)
    run.upload_beam(parts)
    run.upload_field(0, cells, 0)
    run.set_current(np.full(cfg["nslice"], synth.CURRENT))
    run.set_lattice(steps, fc, slip)
    return run


def _result(run, nsteps):
    beam = run.download_beam()
    cells, first = run.download_field(0)
    hist = [run.history(i) for i in range(nsteps)]
    return beam, cells, first, hist


def _same(a, b):
    for k in a[0]:
        assert np.array_equal(a[0][k], b[0][k]), k
    assert np.array_equal(a[1], b[1])
    assert a[2] == b[2]
    for (hb1, hf1), (hb2, hf2) in zip(a[3], b[3]):
        assert np.array_equal(hb1, hb2) and np.array_equal(hf1, hf2)


def _alone(ctx):
    out = []
    for k, cfg in enumerate(CONFIGS):
        run = _make(ctx, k, cfg)
        run.advance(0, cfg["nsteps"], graph=False)
        out.append(_result(run, cfg["nsteps"]))
        run.close()
    return out


@pytest.mark.parametrize("graph, tune", [(False, False), (True, False), (True, True)])
def test_batch_equals_runs_alone(ctx, graph, tune):
    alone = _alone(ctx)
    batch = dev.Batch(ctx, 8)
    runs = [_make(ctx, k, cfg) for k, cfg in enumerate(CONFIGS)]
    slots = [batch.attach(r, 0, cfg["nsteps"]) for r, cfg in zip(runs, CONFIGS)]
    if tune:
        batch.tune()
    longest = max(cfg["nsteps"] for cfg in CONFIGS)
    batch.step(longest + 2, graph=graph)  # runs leave at their own end
    ctx.synchronize()
    for s, r, cfg, ref in zip(slots, runs, CONFIGS, alone):
        assert batch.status(s) == (cfg["nsteps"], 0)
        _same(_result(r, cfg["nsteps"]), ref)
    if tune:
        g = batch.shapes()
        assert all(v > 0 for v in g.values())
    batch.close()


def test_run_joins_a_batch_in_progress(ctx):
    """A run attached while others are mid-way (continuous batching) ends
    with the results it has alone."""
    alone = _alone(ctx)
    batch = dev.Batch(ctx, len(CONFIGS))
    runs = [_make(ctx, k, cfg) for k, cfg in enumerate(CONFIGS)]
    batch.attach(runs[0], 0, CONFIGS[0]["nsteps"])
    batch.attach(runs[1], 0, CONFIGS[1]["nsteps"])
    batch.step(3, graph=True)
    batch.attach(runs[2], 0, CONFIGS[2]["nsteps"])
    batch.step(2, graph=True)
    batch.attach(runs[3], 0, CONFIGS[3]["nsteps"])
    batch.attach(runs[4], 0, CONFIGS[4]["nsteps"])
    batch.step(12, graph=True)
    ctx.synchronize()
    for r, cfg, ref in zip(runs, CONFIGS, alone):
        _same(_result(r, cfg["nsteps"]), ref)
    batch.close()


def test_many_slices_alone_graphed_and_batched_agree(ctx):
    """A 150-slice time-dependent run with slippage every step: direct
    launches, graph replay and the batch engine give the same bits, state and
    the diagnostics of every step."""
    cfg = dict(nslice=150, npart=256, ngrid=65, taper=0.0, dgam=0.0, time_run=True, nsteps=5)
    alone = _make(ctx, 9, cfg)
    alone.advance(0, cfg["nsteps"], graph=False)
    ref = _result(alone, cfg["nsteps"])
    alone.close()
    graphed = _make(ctx, 9, cfg)
    graphed.advance(0, cfg["nsteps"], graph=True)
    _same(_result(graphed, cfg["nsteps"]), ref)
    graphed.close()
    batch = dev.Batch(ctx, 2)
    run = _make(ctx, 9, cfg)
    batch.attach(run, 0, cfg["nsteps"])
    batch.step(cfg["nsteps"], graph=False)
    ctx.synchronize()
    _same(_result(run, cfg["nsteps"]), ref)
    batch.close()


def test_row_layout_tuner_keeps_batch_equal_to_alone(ctx):
    """g4b_batch_tune_layouts times both ADI row layouts of every grid on a
    scratch field before the first step; every step then runs in the chosen
    layouts, so each run equals an alone run given the same layouts."""
    lib = ctx.lib
    # a grid with at least 32 slices in the batch (ngrid 101: 40 + 2) is
    # timed in both layouts; the others keep their defaults
    cfgs = CONFIGS + [dict(nslice=40, npart=256, ngrid=101, taper=0.0, dgam=0.0,
                           time_run=True, nsteps=6)]
    batch = dev.Batch(ctx, 8)
    runs = [_make(ctx, k, cfg) for k, cfg in enumerate(cfgs)]
    for r, cfg in zip(runs, cfgs):
        batch.attach(r, 0, cfg["nsteps"])
    batch.tune_layouts()
    longest = max(cfg["nsteps"] for cfg in cfgs)
    batch.step(longest + 2, graph=True)
    ctx.synchronize()
    per_grid = {}
    for cfg in cfgs:
        per_grid[cfg["ngrid"]] = per_grid.get(cfg["ngrid"], 0) + cfg["nslice"]
    for k, (r, cfg) in enumerate(zip(runs, cfgs)):
        if per_grid[cfg["ngrid"]] < 32:  # too few slices of this grid to time
            assert r.layouts()[0] == lib.g4b_default_layout(cfg["ngrid"])
        lay = r.layouts()
        default = lib.g4b_default_layout(cfg["ngrid"])
        assert lay[0] == default or (lay[0] >= 100) != (default >= 100)
        alone = _make(ctx, k, cfg)
        alone.set_layouts(lay)
        alone.advance(0, cfg["nsteps"], graph=False)
        _same(_result(r, cfg["nsteps"]), _result(alone, cfg["nsteps"]))
        alone.close()
    batch.close()


def test_both_row_layouts_solve_the_same_system(ctx):
    """The other row layout of a grid changes only the FP32 rounding of the
    row solve; a layout that is not one of the grid's two is refused."""
    # ngrid 101: 16 lanes x 7 by default, 32 lanes x 5 the other; steady
    # state, so the field stays in the window
    k, cfg = 3, dict(CONFIGS[3], time_run=False)
    a = _make(ctx, k, cfg)
    a.advance(0, cfg["nsteps"], graph=False)
    ra = _result(a, cfg["nsteps"])
    b = _make(ctx, k, cfg)
    lay = b.layouts()
    other = 5 if lay[0] >= 100 else 107
    b.set_layouts([other])
    assert b.layouts() == [other]
    b.advance(0, cfg["nsteps"], graph=False)
    rb = _result(b, cfg["nsteps"])
    scale = np.max(np.abs(ra[1]))
    assert scale > 0
    assert not np.array_equal(ra[1], rb[1])
    assert np.max(np.abs(ra[1] - rb[1])) < 1e-4 * scale
    with pytest.raises(Exception):
        b.set_layouts([9])
    a.close()
    b.close()


@pytest.mark.parametrize("graph", [False, True])
def test_more_row_layouts_than_concurrent_branches(ctx, graph):
    """Sixteen row layouts in a batch: some branches carry two chains of an ADI
    pass X and its pass Y."""
    lanes16 = [100 + m for m in (5, 7, 9, 11, 13, 15, 17, 21)]
    lanes32 = [3, 5, 7, 9, 11, 13, 15, 17]
    cfgs, want = [], []
    for n in (75, 101, 130, 170, 201, 240, 260, 330):
        cfgs += 2 * [dict(nslice=1, npart=512, ngrid=n, taper=0.0, dgam=0.0, time_run=False,
                          nsteps=4)]
        want += [next(m for m in lanes16 if 16 * (m - 100) >= n),
                 next(m for m in lanes32 if 32 * m >= n)]
    assert len(set(want)) > 12
    runs = [_make(ctx, k, cfg) for k, cfg in enumerate(cfgs)]
    batch = dev.Batch(ctx, len(runs))
    for r, m in zip(runs, want):
        r.set_layouts([m])
        batch.attach(r, 0, 4)
    batch.step(4, graph=graph)
    ctx.synchronize()
    for k, (r, cfg, m) in enumerate(zip(runs, cfgs, want)):
        alone = _make(ctx, k, cfg)
        alone.set_layouts([m])
        alone.advance(0, 4, graph=False)
        _same(_result(r, 4), _result(alone, 4))
        alone.close()
    batch.close()


# the deposition and the beam diagnostics of a slice are split by the number of
# slices in the launch (dep_split, dep_split_batch: shared tile up to 21 slices,
# two CTAs per slice up to 147 in a run and 592 in a batch, one CTA above); widths 1 and 6 make tiles
# of one band and of several, the slices start at odd offsets
@pytest.mark.parametrize("width", [1.0, 6.0])
@pytest.mark.parametrize("fill", [18, 19, 71, 72, 144, 145, 589, 590])
def test_results_do_not_depend_on_how_the_slices_are_split(ctx, width, fill):
    ns, ngrid, gm, n = 3, 151, 160e-6, 5
    off, parts = synth.beam(ns, 1500, seed=11, ragged=True)
    for k in ("x", "y"):
        parts[k] = np.clip(parts[k] * width, -0.99 * gm, 0.99 * gm)
    cells = synth.field(ns, ngrid, gm, seed=12, amplitude=2e12)
    steps = [synth.und_step() for _ in range(n)]
    fc = [[synth.coupling()]] * n
    slip = [0.4] * n

    def make(offsets, p, c, grid):
        run = dev.Run(ctx, offsets, fields=[(1, grid, gm)], lambda0=synth.LAMBDA0,
                      gamma_ref=synth.GAMMA0, time_run=True)
        run.upload_beam(p)
        run.upload_field(0, c, 0)
        run.set_current(synth.CURRENT)
        run.set_lattice(steps, fc, slip)
        return run

    alone = make(off, parts, cells, ngrid)
    alone.advance(0, n, graph=True)
    want = _result(alone, n)
    foff, fparts = synth.beam(fill, 64, seed=13)
    filler = make(foff, fparts, None, 33)
    run = make(off, parts, cells, ngrid)
    batch = dev.Batch(ctx, 2)
    batch.attach(run, 0, n)
    batch.attach(filler, 0, n)
    batch.step(n)
    got = _result(run, n)
    assert np.any(want[1] != cells)
    for k in want[0]:
        assert np.array_equal(got[0][k], want[0][k])
    assert np.array_equal(got[1], want[1]) and got[2] == want[2]
    for a, b in zip(got[3], want[3]):
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    for o in (batch, run, filler, alone):
        o.close()


@pytest.mark.parametrize("graph", [False, True])
def test_a_layout_switched_after_attaching_takes_effect(ctx, graph):
    """set_layouts on a run that a batch already steps (from a captured graph
    too): the later steps equal those of an alone run switched at that step."""
    cfgs = [dict(nslice=2, npart=512, ngrid=n, taper=0.0, dgam=0.0, time_run=False, nsteps=9)
            for n in (101, 151, 201, 240)]
    other = [5, 111, 7, 9]  # by default 16 x 7, 32 x 5, 16 x 13, 16 x 15
    runs = [_make(ctx, k, cfg) for k, cfg in enumerate(cfgs)]
    batch = dev.Batch(ctx, len(runs))
    for r in runs:
        batch.attach(r, 0, 9)
    batch.step(5, graph=graph)
    for r, m in zip(runs, other):
        assert r.layouts() != [m]
        r.set_layouts([m])
    batch.step(4, graph=graph)
    ctx.synchronize()
    for k, (r, cfg, m) in enumerate(zip(runs, cfgs, other)):
        alone = _make(ctx, k, cfg)
        alone.advance(0, 5, graph=False)
        alone.set_layouts([m])
        alone.advance(5, 4, graph=False)
        _same(_result(r, 9), _result(alone, 9))
        alone.close()
    batch.close()


@pytest.mark.parametrize("ngrid, layouts", [(33, (105, 3)), (351, (11, 125)), (400, (125, 13)),
                                            (528, (133, 17)), (672, (21,)), (700, (25,)),
                                            (880, (33,))])
def test_batched_rows_equal_single_rows_in_the_longest_layouts(ctx, ngrid, layouts):
    """The batched row solve reads its coefficients from an image in memory,
    the single-run one from its parameters: the same bits, to the widest grid."""
    cfg = dict(nslice=1, npart=256, ngrid=ngrid, taper=0.0, dgam=0.0, time_run=False, nsteps=3)
    for layout in layouts:
        got = []
        for batched in (False, True):
            run = _make(ctx, 3, cfg)
            run.set_layouts([layout])
            if batched:
                batch = dev.Batch(ctx, 1)
                batch.attach(run, 0, 3)
                batch.step(3, graph=False)
                ctx.synchronize()
                batch.close()
            else:
                run.advance(0, 3, graph=False)
            got.append(_result(run, 3))
            run.close()
        _same(*got)


# the splits of a single run: up to 21 slices shared by several CTAs (tile: 3001
# and 33001 particles; alone: 1500, or 13 slices and more; bands: width 6, and
# 301^2 for a box above the tile's 65536 cells), pairs of 512 threads to 74 and of
# 256 to 147 (up to 2048 particles, else of 512 to 98), one CTA per slice above.
# The second step focuses x to half its width, so that in every split the bounds
# taken from the step before fail and the deposition is redone.
@pytest.mark.parametrize("ngrid, npart, width, counts", [
    (151, 1500, 1.0, (1, 12, 13, 21, 22, 74, 75, 147, 148, 295, 296)),
    (151, 1500, 6.0, (1, 13, 21, 22, 75, 147, 148, 296)),
    (151, 3001, 1.0, (1, 12, 13, 22, 75, 98, 99, 148)),
    (151, 3001, 6.0, (1, 21, 22, 75, 98, 99)),
    (151, 40000, 6.0, (1, 8, 9, 22, 99)),
    (301, 2999, 8.0, (1, 21, 22, 75, 99)),
])
@pytest.mark.parametrize("nbunch", [1, 3])
def test_a_slice_does_not_depend_on_the_slices_beside_it(ctx, ngrid, npart, width, counts, nbunch):
    gm, n = 160e-6, 4
    sizes = [npart - 1, npart // 2 | 1, npart]  # the second and third start at odd offsets
    off, parts = synth.beam(3, sizes, seed=21)
    for k in ("x", "y"):
        parts[k] = np.clip(parts[k] * width, -0.99 * gm, 0.99 * gm)
    for k in ("x", "y", "px", "py", "gamma"):  # the first slice in beamlets of four
        parts[k][:sizes[0]] = np.repeat(parts[k][:sizes[0] // 4 + 1], 4)[:sizes[0]]
    k60 = (np.pi / (3 * synth.LAMBDA_U)) ** 2  # 60 degrees of phase advance
    steps = [synth.und_step(), synth.und_step(qf=k60), synth.und_step(), synth.und_step()]

    def go(which, ns, graph):
        """These of the three slices, spread over a run of ns; the others hold 64."""
        order = [0, ns // 2, ns - 1][:len(which)]
        few = synth.beam(1, 64, seed=22)[1]
        cols = [few] * ns
        for i, s in zip(which, order):
            cols[s] = {k: parts[k][off[i]:off[i + 1]] for k in parts}
        p = {k: np.concatenate([c[k] for c in cols]) for k in parts}
        o = np.concatenate([[0], np.cumsum([len(c["x"]) for c in cols])])
        run = dev.Run(ctx, o, fields=[(1, ngrid, gm)], lambda0=synth.LAMBDA0,
                      gamma_ref=synth.GAMMA0, time_run=False, nbunch=nbunch)
        run.upload_beam(p)
        run.upload_field(0, None)
        run.set_current(synth.CURRENT)
        run.set_lattice(steps, [[synth.coupling()]] * n, [0.0] * n)
        run.advance(0, n, graph=graph)
        beam = run.download_beam()
        field = run.download_field(0)[0]
        hist = [run.history(i) for i in range(n)]
        run.close()
        return [([beam[k][o[s]:o[s + 1]] for k in beam], field[s],
                 [(b[s], f[:, s]) for b, f in hist]) for s in order]

    want = go((0, 1, 2), 3, False)
    assert all(np.any(w[1]) for w in want)
    for ns in counts:
        got = go((0, 1, 2), ns, ns % 2 == 0) if ns > 1 else [go((i,), 1, False)[0] for i in range(3)]
        for g, w in zip(got, want):
            for a, b in zip(g[0], w[0]):
                assert np.array_equal(a, b), ns
            assert np.array_equal(g[1], w[1]), ns
            for (b1, f1), (b2, f2) in zip(g[2], w[2]):
                assert np.array_equal(b1, b2) and np.array_equal(f1, f2), ns


def test_tuner_leaves_the_deposition_grid_that_a_split_ignores(ctx):
    """Few slices take several CTAs each, whatever the tuned grid: timings of
    that launch say nothing about it, so it keeps its default."""
    batch = dev.Batch(ctx, 2)
    default = batch.shapes()
    run = _make(ctx, 3, CONFIGS[3])
    batch.attach(run, 0, 7)
    for _ in range(5):  # repeated: timings picked one of four grids by chance
        batch.tune()
        batch.step(4, graph=False)
        assert batch.shapes()["deposit"] == default["deposit"]
        batch.detach(0)
        batch.attach(run, 0, 7)
    batch.close()
    run.close()


def test_runs_of_different_harmonics_share_a_batch(ctx):
    """The diagnostics' order of sums follows the run's own number of bunching
    harmonics: in a batch whose kernel serves several, every run has its bits."""
    n = 4

    def make(k, nbunch):
        off, parts = synth.beam(2, [5000, 1111], seed=80 + k)
        run = dev.Run(ctx, off, fields=[(1, 65, 160e-6)], lambda0=synth.LAMBDA0,
                      gamma_ref=synth.GAMMA0, time_run=False, nbunch=nbunch)
        run.upload_beam(parts)
        run.upload_field(0, None)
        run.set_current(synth.CURRENT)
        run.set_lattice([synth.und_step()] * n, [[synth.coupling()]] * n, [0.0] * n)
        return run

    kinds = [1, 2, 5, 8]
    batch = dev.Batch(ctx, len(kinds))
    runs = [make(k, nb) for k, nb in enumerate(kinds)]
    for r in runs:
        batch.attach(r, 0, n)
    batch.step(n, graph=False)
    ctx.synchronize()
    for k, (r, nb) in enumerate(zip(runs, kinds)):
        alone = make(k, nb)
        alone.advance(0, n, graph=False)
        _same(_result(r, n), _result(alone, n))
        alone.close()
        r.close()
    batch.close()
