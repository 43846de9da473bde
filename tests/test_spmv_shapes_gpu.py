"""The SpMV tile shapes at capacities whose launches store the most partial sums (a
shape with four block rows per CTA stores N / 4 of them per sum)."""
import numpy as np
import pytest
import torch
from scipy.spatial import cKDTree

from conftest import rel_norm_error, small_scene
from multiviewdynrecon_b200 import abi, synth
from multiviewdynrecon_b200.solver import BatchSolver

pytestmark = pytest.mark.gpu


def _increments(scene, shapes, precision, pcg, **capacity):
    cfg = abi.make_config(scene, precision=precision)
    for name, value in capacity.items():
        setattr(cfg, name, value)
    b = BatchSolver(cfg, 2)
    out = []
    for shape in shapes:
        b.set_spmv_shape(shape)
        for i in range(2):
            b.set_input(i, scene)
        b.solve(1, pcg)
        torch.cuda.synchronize()
        assert b.instance(0).counts().error_flags == 0
        out.append([b.instance(i).get_array(abi.ARRAY_INCREMENT) for i in range(2)])
        assert np.array_equal(out[-1][0], out[-1][1])
    b.close()
    return [o[0] for o in out]


@pytest.mark.parametrize("precision", [abi.PRECISION_MIXED, abi.PRECISION_FP32])
def test_capacity_does_not_change_the_increments(precision):
    """CTAs past the bound nodes store zeros, so every shape's sums are the same
    whatever the capacity."""
    scene, shapes = small_scene("torso"), range(abi.NUM_SPMV_SHAPES)
    pairs = 64 * scene.num_nodes
    want = _increments(scene, shapes, precision, 6, max_node_pairs=pairs)
    for nodes in (4769, 6000, 16000, 65535):
        got = _increments(scene, shapes, precision, 6, max_nodes=nodes, max_node_pairs=pairs)
        for shape, (a, b) in enumerate(zip(got, want)):
            assert np.array_equal(a, b), (nodes, abi.SPMV_SHAPES[shape])


def test_every_shape_solves_a_large_graph():
    """6,000 nodes: 1,500 CTAs of the narrowest shape. A float sum of the about 120
    products of a row is off by at most 120 x 2^-24 of their magnitudes, so two
    shapes differ by less than 1e-4 after five iterations."""
    scene = synth.sphere_single_view(seed=5, num_nodes=40, width=320, height=240)
    rng = np.random.default_rng(2)
    nodes = scene.surfel_position[rng.choice(scene.num_surfels, 6000, replace=False)]
    tree = cKDTree(nodes)
    scene.canonical_nodes = np.concatenate([nodes, np.ones((6000, 1))], 1).astype(np.float32)
    scene.node_se3 = np.tile(np.array([0, 0, 0, 1, 0.002, -0.001, 0.003, 0], np.float32), (6000, 1))
    scene.surfel_knn = tree.query(scene.surfel_position, 4)[1].astype(np.uint16)
    scene.surfel_knn_weight = np.tile(np.array([0.4, 0.3, 0.2, 0.1], np.float32), (scene.num_surfels, 1))
    near = tree.query(nodes, 9)[1][:, 1:]
    scene.node_graph = np.stack([np.repeat(np.arange(6000), 8), near.reshape(-1)], 1).astype(np.uint16)
    got = _increments(scene, range(abi.NUM_SPMV_SHAPES), abi.PRECISION_MIXED, 5)
    assert np.abs(got[0]).max() > 1e-4
    for shape, x in enumerate(got):
        assert rel_norm_error(x, got[0]) < 1e-4, abi.SPMV_SHAPES[shape]
