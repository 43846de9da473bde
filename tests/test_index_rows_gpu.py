"""The index build against the oracle where its kernels change over: term lists
around the sort's run lengths, nodes with more partners than the row table
takes, and terms that list a node twice."""
import numpy as np
import pytest

from multiviewdynrecon_b200 import abi, synth

pytestmark = pytest.mark.gpu

ARRAYS = (abi.ARRAY_NODE2TERM_OFFSET, abi.ARRAY_NODE2TERM_INDEX, abi.ARRAY_HALF_NODEPAIR_KEY,
          abi.ARRAY_NODEPAIR_TERM_INDEX, abi.ARRAY_NODEPAIR_KEY, abi.ARRAY_NODEPAIR_TERM_RANGE,
          abi.ARRAY_BLKROW_OFFSET, abi.ARRAY_BINBLOCK_COLPTR)


def _few_nodes(nodes, width, height):
    scene = synth.sphere_single_view(seed=8, num_nodes=nodes, width=width, height=height)
    scene.surfel_knn_weight[:] = (0.4, 0.3, 0.2, 0.1)
    return scene


def _crowded(nodes, twice):
    scene = synth.torso_multi_view(seed=9, num_nodes=nodes, num_views=2, width=160, height=120, features_per_view=40,
                                   cross_per_pair=40)
    scene.surfel_knn_weight[:] = (0.4, 0.3, 0.2, 0.1)
    rng = np.random.default_rng(2)
    scene.surfel_knn[:] = rng.permuted(np.tile(np.arange(nodes), (scene.num_surfels, 1)), axis=1)[:, :4]
    if twice:
        scene.surfel_knn[::7, 3] = scene.surfel_knn[::7, 1]
    return scene


@pytest.mark.parametrize("scene,long_lists", [
    (lambda: _few_nodes(12, 24, 18), (None, 257)),       # within one run
    (lambda: _few_nodes(40, 96, 72), (257, 4096)),       # merged runs
    (lambda: _few_nodes(10, 110, 83), (4097, None)),     # past the merge
    (lambda: _crowded(230, False), (None, None)),        # more than 192 partners
    (lambda: _crowded(60, True), (None, None)),          # a node twice in a term
])
def test_index_equals_the_oracle(scene, long_lists, oracle_mod):
    _check(scene(), long_lists, oracle_mod, None)


@pytest.mark.parametrize("max_nodes", [4095, 4096])  # a CTA or a warp per row
@pytest.mark.parametrize("scene", [lambda: _few_nodes(40, 96, 72), lambda: _crowded(230, False),
                                   lambda: _crowded(60, True)])
def test_index_at_the_change_of_row_kernels(scene, max_nodes, oracle_mod):
    _check(scene(), (None, None), oracle_mod, max_nodes)


def _check(scene, long_lists, oracle_mod, max_nodes):
    from multiviewdynrecon_b200.solver import NonRigidSolver
    cfg = abi.make_config(scene)
    cfg.max_nodes = max_nodes or cfg.max_nodes
    cfg.max_node_pairs = max(16 * scene.num_nodes, scene.num_nodes ** 2)
    cfg.max_terms_per_node = 16384
    g = NonRigidSolver(cfg)
    g.set_solver_input(scene)
    g.build_index()
    assert g.counts().error_flags == 0
    o = oracle_mod.Oracle(scene, cfg)
    o.build_index()
    for a in ARRAYS:
        assert np.array_equal(g.get_array(a), o.get(a)), a
    lens = np.diff(g.get_array(abi.ARRAY_NODE2TERM_OFFSET).astype(np.int64))
    low, high = long_lists
    assert (low is None or lens.max() >= low) and (high is None or lens.max() <= high)
    if scene.num_nodes == 230:
        keys = g.get_array(abi.ARRAY_HALF_NODEPAIR_KEY)
        assert np.bincount(keys // 4096).max() > 192
    g.close()
