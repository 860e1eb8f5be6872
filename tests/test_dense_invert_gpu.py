"""The coarsest levels' inverses: the same bits however many blocks a planet's inverse is shared
out over (the more planets a batch holds, the fewer), at sizes around a warp and a block's rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 42 and 162 coarsest rows; 1, 8, 16, 37 planets: clusters of 8 and 16, 8, 4, 2 blocks
@pytest.mark.parametrize("level,count", [(3, 8), (3, 16), (3, 37), (4, 8), (4, 16), (4, 37)])
def test_a_batch_of_any_size_inverts_as_one_planet_does(meshes, level, count):
    import planet_game_gb300 as pg
    from planet_game_gb300 import workloads as W

    ms = [meshes(level, 3.0e6 + 1.0e5 * i) for i in range(count)]
    inputs = [W.step_inputs(m, seed=i) for i, m in enumerate(ms)]
    out, reports = pg.Batch(ms).transport_step([i.t0 for i in inputs], [i.source for i in inputs], 4e7, inputs[0].dt,
                                               conductance=[4e13] * count, schedule="kernels")
    assert all(r.status == 0 for r in reports)
    for k in (0, count // 2, count - 1):
        (alone,), (report,) = pg.Batch([ms[k]]).transport_step([inputs[k].t0], [inputs[k].source], 4e7, inputs[0].dt,
                                                               conductance=[4e13], schedule="kernels")
        assert np.array_equal(alone, out[k]) and report.iterations == reports[k].iterations


def test_inverse_solves_the_coarsest_system(meshes):
    """A level-2 planet's one level is its coarsest: the V-cycle is the inverse alone."""
    import planet_game_gb300 as pg

    m = meshes(2, 5.0e6)
    mg = pg.GraphMultigrid(m)
    a = m.arrays()
    mg.set_matrix(1.5e15 + 4e13 * a["graph_weight_sum"], -4e13 * a["graph_weight"])
    lv = m.hierarchy_level(0)
    rows = len(lv["offset"]) - 1
    diagonal, off = mg.level_values(0)
    dense = np.diag(diagonal)
    for i in range(rows):
        k = slice(lv["offset"][i], lv["offset"][i + 1])
        dense[i, lv["column"][k]] += off[k]
    b = np.random.default_rng(2).normal(0.0, 1.0, rows)
    want = np.linalg.solve(dense, b)
    # Gauss-Jordan on a diagonally dominant matrix of condition c: n c eps
    bound = rows * np.linalg.cond(dense) * np.finfo(float).eps
    assert np.linalg.norm(mg.precondition(b) - want) <= bound * np.linalg.norm(want)
