"""The on-chip solves (one planet per thread-block cluster) against the kernel schedule: the
same phases and reduction trees, so every result is the same bits - planets alone and in
batches, left-out planets, every precision, sweep setting and ending of the iteration."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def inputs_of(mesh, seed):
    from planet_game_gb300 import workloads as W

    return W.step_inputs(mesh, seed=seed, edge_diffusivity=W.lognormal_edge_diffusivity(mesh.edge_count, 300 + seed))


def step(batch, inputs, **options):
    keep = options.pop("keep", range(len(inputs)))
    pick = lambda f: [f(i) if k in keep else None for k, i in enumerate(inputs)]
    active = [k in keep for k in range(len(inputs))]
    return batch.transport_step(pick(lambda i: i.t0), pick(lambda i: i.source), 4e7, inputs[0].dt,
                                edge_conductance=[i.edge_conductance for i in inputs],
                                active=None if all(active) else active, **options)


def same(a, b):
    (out_a, rep_a), (out_b, rep_b) = a, b
    for x, y in zip(out_a, out_b):
        assert (x is None) == (y is None)
        assert x is None or np.array_equal(x, y)
    for x, y in zip(rep_a, rep_b):
        assert (x.status, x.refinements, x.iterations) == (y.status, y.refinements, y.iterations)
        assert x.relative_residual == y.relative_residual


# levels 3 (two levels, 42 coarsest rows) to 6 (the largest that fits a cluster in FP32)
@pytest.mark.parametrize("level,precision", [(3, "fp64"), (3, "mixed"), (4, "fp64"), (4, "mixed"), (5, "fp64"),
                                             (5, "mixed"), (6, "mixed"), (6, "fp64")])
def test_one_planet_equals_the_kernel_schedule(meshes, level, precision):
    import planet_game_gb300 as pg

    m = meshes(level, 3.4e6)
    batch, inputs = pg.Batch([m]), [inputs_of(m, level)]
    for options in ({}, {"pre_sweeps": 1, "post_sweeps": 1, "jacobi_omega": 1.0}, {"pre_sweeps": 1, "post_sweeps": 0},
                    {"pre_sweeps": 3, "post_sweeps": 2}, {"max_iterations": 2, "max_refinements": 3},
                    {"tolerance": 1e-3}):
        same(step(batch, inputs, precision=precision, **options),
             step(batch, inputs, precision=precision, schedule="kernels", **options))


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_batches_of_several_levels(meshes, precision):
    """Several sizes of cluster side by side, and a batch that one planet keeps off chip; some
    planets left out of the step."""
    import planet_game_gb300 as pg

    for levels in ((5, 3, 4, 5, 4), (5, 3, 7, 4, 5)):
        ms = [meshes(l, 3.0e6 + 0.4e6 * i) for i, l in enumerate(levels)]
        inputs = [inputs_of(m, i) for i, m in enumerate(ms)]
        batch = pg.Batch(ms)
        for keep in (range(5), (0, 2), (1, 4), (2,)):
            same(step(batch, inputs, precision=precision, keep=keep),
                 step(batch, inputs, precision=precision, keep=keep, schedule="kernels"))


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_tuned_sweeps(meshes, precision):
    """Block-local coarse sweeps (whole tiles per block) and a scaled coarse correction."""
    import planet_game_gb300 as pg

    ms = [meshes(l, 3.2e6 + 0.3e6 * i) for i, l in enumerate((5, 6, 4, 5, 3))]
    inputs = [inputs_of(m, 20 + i) for i, m in enumerate(ms)]
    batch = pg.Batch(ms)
    depth = batch.tuning["levels"]
    for inner, correction, omega in ((6, 1.0, 1.0), (3, 2.0, 0.9), (1, 1.5, 0.8)):
        batch.set_tuning({"pre_sweeps": [1] + [2] * (depth - 1), "post_sweeps": [1] + [2] * (depth - 1),
                          "stencil_tiles": [1] * depth, "vector_tiles": [1] * depth,
                          "block_sweeps": [1] + [inner] * (depth - 1), "jacobi_omega": omega,
                          "coarse_correction": correction})
        same(step(batch, inputs, precision=precision), step(batch, inputs, precision=precision, schedule="kernels"))


def test_non_finite_source_reports_and_keeps_the_other_planets(meshes):
    import planet_game_gb300 as pg

    ms = [meshes(4, 3.3e6), meshes(5, 4.1e6)]
    inputs = [inputs_of(m, 40 + i) for i, m in enumerate(ms)]
    bad = inputs[0].source.copy()
    bad[7] = np.nan
    batch = pg.Batch(ms)
    args = lambda s0: ([i.t0 for i in inputs], [s0, inputs[1].source], 4e7, inputs[0].dt)
    edges = [i.edge_conductance for i in inputs]
    good = batch.transport_step(*args(inputs[0].source), edge_conductance=edges, precision="mixed")
    with pytest.raises(Exception, match="non-finite"):
        batch.transport_step(*args(bad), edge_conductance=edges, precision="mixed")
    same(good, batch.transport_step(*args(inputs[0].source), edge_conductance=edges, precision="mixed"))


def launches_of(family, call):
    """The launches of a kernel family during a call, and the call's result."""
    import ctypes as C

    from planet_game_gb300 import capi

    lib = capi.load()
    ms, count, swept = C.c_double(), C.c_uint64(), C.c_uint64()
    capi.check(lib.psgb_profile_begin(family.encode()))
    try:
        out = call()
    finally:
        capi.check(lib.psgb_profile_end(C.byref(ms), C.byref(count), C.byref(swept)))
    assert (ms.value > 0.0) == (count.value > 0)
    return count.value, out


@pytest.mark.parametrize("levels,precision", [((4,), "fp64"), ((5, 3, 4, 5), "mixed")])
def test_a_recording_profile_times_the_solves_that_run_without_it(meshes, levels, precision):
    import planet_game_gb300 as pg

    ms = [meshes(l, 3.3e6 + 2e5 * i) for i, l in enumerate(levels)]
    batch, inputs = pg.Batch(ms), [inputs_of(m, 60 + i) for i, m in enumerate(ms)]
    plain = step(batch, inputs, precision=precision)
    for schedule in ("auto", "kernels"):
        call = lambda: step(batch, inputs, precision=precision, schedule=schedule)
        onchip, recorded = launches_of("onchip", call)
        smooth, again = launches_of("smooth", call)
        same(plain, recorded)
        same(plain, again)
        if schedule == "auto":   # a launch a planet shape, no sweep of the kernel schedule
            assert onchip == len(set(levels)) and smooth == 0
        else:
            assert onchip == 0 and smooth > 0


# every form of the kernel that a batch's planets take: rows a thread, with block-local coarse
# sweeps and a scaled correction too, and batches that keep the kernel schedule
@pytest.mark.parametrize("precision,levels,onchip", [("fp64", (4,), True), ("fp64", (5,), True), ("fp64", (5, 4, 5, 3), True),
                                                     ("fp64", (6,), False), ("mixed", (5,), True), ("mixed", (6,), True),
                                                     ("mixed", (5, 6, 4, 5, 3), True), ("mixed", (5, 7), False)])
def test_which_batches_go_on_chip(meshes, precision, levels, onchip):
    """Tuned and untuned: that the path is the one meant, and the kernel schedule's bits."""
    import planet_game_gb300 as pg

    ms = [meshes(l, 3.1e6 + 3e5 * i) for i, l in enumerate(levels)]
    inputs = [inputs_of(m, 80 + i) for i, m in enumerate(ms)]
    batch = pg.Batch(ms)
    depth = batch.tuning["levels"]
    for inner, correction, omega in ((0, 1.0, 0.8), (6, 1.0, 1.0), (3, 2.0, 0.9), (1, 1.5, 0.8)):
        if inner:
            batch.set_tuning({"pre_sweeps": [1] + [2] * (depth - 1), "post_sweeps": [1] + [2] * (depth - 1),
                              "stencil_tiles": [1] * depth, "vector_tiles": [1] * depth,
                              "block_sweeps": [1] + [inner] * (depth - 1), "jacobi_omega": omega,
                              "coarse_correction": correction})
        count, got = launches_of("onchip", lambda: step(batch, inputs, precision=precision))
        assert count == (len(set(levels)) if onchip else 0)
        same(got, step(batch, inputs, precision=precision, schedule="kernels"))


def test_priority_and_masks_change_nothing(meshes):
    """After a solve, set_priority drops the plans with their streams; a changing mask keeps them."""
    import planet_game_gb300 as pg

    ms = [meshes(l, 3.0e6 + 2e5 * i) for i, l in enumerate((5, 3, 4, 5, 4))]
    inputs = [inputs_of(m, 100 + i) for i, m in enumerate(ms)]
    batch = pg.Batch(ms)
    masks = (range(5), (0, 2), (4,), (1, 3), range(5))
    want = [step(batch, inputs, precision="mixed", keep=keep, schedule="kernels") for keep in masks]
    for high in (None, True, False):
        if high is not None:
            batch.set_priority(high)
        for keep, ref in zip(masks, want):
            count, got = launches_of("onchip", lambda: step(batch, inputs, precision="mixed", keep=keep))
            assert count == 3
            same(got, ref)


def test_batches_side_by_side(meshes):
    """Two batches solved on chip from two threads, beside one on the kernel schedule."""
    import threading

    import planet_game_gb300 as pg

    jobs = []
    for k, (levels, precision) in enumerate((((5, 4, 3), "mixed"), ((4, 5), "fp64"), ((7,), "mixed"))):
        ms = [meshes(l, 3.0e6 + 2e5 * i + 1e5 * k) for i, l in enumerate(levels)]
        inputs = [inputs_of(m, 120 + 10 * k + i) for i, m in enumerate(ms)]
        batch = pg.Batch(ms)
        jobs.append((batch, inputs, precision, step(batch, inputs, precision=precision, schedule="kernels"), []))

    def work(batch, inputs, precision, _, out):
        for _ in range(5):
            out.append(step(batch, inputs, precision=precision))

    threads = [threading.Thread(target=work, args=job) for job in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for *_, want, got in jobs:
        assert len(got) == 5
        for g in got:
            same(g, want)


def test_more_sweep_settings_than_plans_are_kept(meshes):
    import planet_game_gb300 as pg

    ms = [meshes(l, 3.2e6 + 2e5 * i) for i, l in enumerate((4, 5, 3))]
    inputs = [inputs_of(m, 150 + i) for i, m in enumerate(ms)]
    batch = pg.Batch(ms)
    settings = [dict(pre_sweeps=a, post_sweeps=b, precision=p) for p in ("mixed", "fp64") for a, b in ((1, 0), (1, 1), (2, 1), (3, 3))]
    want = [step(batch, inputs, schedule="kernels", **s) for s in settings]
    for _ in range(2):
        for s, ref in zip(settings, want):
            count, got = launches_of("onchip", lambda: step(batch, inputs, **s))
            assert count == 3
            same(got, ref)
