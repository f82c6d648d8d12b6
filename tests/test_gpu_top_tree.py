"""The top tree built on the device against the prep's build_sah over the same units, node for node (the same f32
operations, so the tolerance is none): numbers of units around what a warp, a shared-memory subtree and a block split,
spread evenly, in clusters that peel a few units off at each split, and all in one place."""
import numpy as np
import pytest

from threert_b200 import RenderError, prep, scenes

pytestmark = pytest.mark.gpu

SPREADS = {
    "even": lambda rng, n: rng.uniform(-100.0, 100.0, (n, 3)),
    # (each unit 1.3 times as far out as the last: the splits are uneven, and the depth's room ends them)
    "peeling": lambda rng, n: np.sign(rng.normal(size=(n, 3))) * (1.3 ** np.minimum(np.arange(n), 60))[:, None] * 1e-2,
    "one place": lambda rng, n: np.zeros((n, 3)),
    "a row": lambda rng, n: np.stack([np.arange(n, dtype=float), np.zeros(n), np.zeros(n)], 1),
}


@pytest.mark.parametrize("spread", list(SPREADS))
@pytest.mark.parametrize("n", [1, 2, 3, 10, 11, 33, 127, 128, 129, 256, 257, 700, 2049, 5003])
def test_the_devices_top_tree_is_the_preps(gpu, n, spread):
    rng = np.random.default_rng(n)
    at = SPREADS[spread](rng, n)
    world = lambda p: scenes.translate_rot_y(p, rng.uniform(0, 3.0))
    insts = [prep.Instance(0, [0], scenes.translate_rot_y((k, 0, 0)), object=k) for k in range(n)]
    cam = prep.Camera.look_at((0, 4, 14), (0, 0, 0), 50, 8, 8)
    P = prep.prepare(prep.SceneDescription([scenes.box_mesh(1, 1, 1)], [prep.lambert(0.5)], insts, cam))
    S = gpu.upload(P)
    S.deform_setup(np.zeros((0, 16), np.float32), np.zeros((0, 8), np.uint32))
    t_inst, first = int(P.params[124 + 7]), int(P.params[70])
    rec = P.tables[4 * t_inst: 4 * t_inst + 40 * n].reshape(n, 40)
    roots = rec[:, 15]
    box = P.nodes.view(np.float32)[roots][:, [0, 1, 2, 4, 5, 6]]
    for frame in range(2):  # (a second build, over the lists the first left)
        worlds = np.stack([world(p) for p in at])
        S.update(3, t_inst * 16, prep.unit_records(worlds, rec[:, 24:28], roots, np.ones(n, np.uint32)))
        st = S.deform(P.params, np.zeros((0, 12), np.float32))
        assert st["errors"] == 0
        want, _ = prep.units_top(worlds, box)
        got = S.read(2, 32 * first, 32 * (2 * n - 1), np.uint32).reshape(-1, 8)
        assert np.array_equal(got[:, [3, 7]], want[:, [3, 7]])
        # (boxes as floats: a zero's sign may differ between folds)
        assert np.array_equal(got.view(np.float32)[:, [0, 1, 2, 4, 5, 6]], want.view(np.float32)[:, [0, 1, 2, 4, 5, 6]])
    S.close()


def turned(rng, n):
    return np.stack([scenes.translate_rot_y(p, rng.uniform(0, 3.0)) for p in rng.uniform(-50.0, 50.0, (n, 3))])


# Nodes that a warp splits without bins and with them, one block, and a launch a level; the NaN in a unit's place or in
# its rotation, in the first unit, the last, or several.
@pytest.mark.parametrize("row,col", [(0, 3), (1, 3), (2, 0)])
@pytest.mark.parametrize("n", [2, 3, 6, 10, 11, 40, 128, 129, 300, 2049])
def test_a_unit_whose_box_is_not_a_number_is_refused(gpu, n, row, col):
    rng = np.random.default_rng(n)
    insts = [prep.Instance(0, [0], scenes.translate_rot_y((k, 0, 0)), object=k) for k in range(n)]
    cam = prep.Camera.look_at((0, 4, 14), (0, 0, 0), 50, 8, 8)
    P = prep.prepare(prep.SceneDescription([scenes.box_mesh(1, 1, 1)], [prep.lambert(0.5)], insts, cam))
    S = gpu.upload(P)
    S.deform_setup(np.zeros((0, 16), np.float32), np.zeros((0, 8), np.uint32))
    t_inst, first = int(P.params[124 + 7]), int(P.params[70])
    rec = P.tables[4 * t_inst: 4 * t_inst + 40 * n].reshape(n, 40)
    box = P.nodes.view(np.float32)[rec[:, 15]][:, [0, 1, 2, 4, 5, 6]]

    def frame(worlds):
        S.update(3, t_inst * 16, prep.unit_records(worlds, rec[:, 24:28], rec[:, 15], np.ones(n, np.uint32)))
        return S.deform(P.params, np.zeros((0, 12), np.float32))

    for bad in ([0], [n - 1], [0, n // 2]):
        worlds = turned(rng, n)
        worlds[bad, row, col] = np.nan
        with pytest.raises(RenderError, match="TRT_EGUARD.*not a number"):
            frame(worlds)
        # the next frame is as if none had failed; a unit far out (its centre's sum overflows) is none to refuse
        worlds = turned(rng, n)
        worlds[n // 2, 0, 3] = 3e38
        assert frame(worlds)["errors"] == 0
        want, _ = prep.units_top(worlds, box)
        got = S.read(2, 32 * first, 32 * (2 * n - 1), np.uint32).reshape(-1, 8)
        assert np.array_equal(got[:, [3, 7]], want[:, [3, 7]])
    S.close()
