"""Node errors at the edges of the kernel's pixel tiles, and with skinning weights
that its summed form does not take (negative, above 2^18): equal to the oracle."""
import numpy as np
import pytest
import torch

from multiviewdynrecon_b200 import abi, synth
from multiviewdynrecon_b200.solver import NonRigidSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height,weights", [(97, 65, None), (64, 72, None), (129, 57, "large"), (65, 67, "mixed")])
def test_node_error_equals_the_oracle(oracle_mod, width, height, weights):
    scene = synth.sphere_single_view(seed=4, num_nodes=40, width=width, height=height)
    rng = np.random.default_rng(6)
    w = rng.uniform(0.05, 0.4, scene.surfel_knn_weight.shape).astype(np.float32)
    if weights == "large":
        w *= np.float32(1 << 22)
    elif weights == "mixed":
        some = rng.random(len(w)) < 0.02
        w[some] *= np.float32(-3e6)
    scene.surfel_knn_weight[:] = w
    # (a node twice among a surfel's four is added twice)
    scene.surfel_knn[::7, 3] = scene.surfel_knn[::7, 0]
    solver = NonRigidSolver(abi.make_config(scene))
    solver.set_solver_input(scene)
    got = solver.compute_alignment_error_on_nodes(maps=True)
    torch.cuda.synchronize()
    want = oracle_mod.node_error(scene, scene.node_se3, maps=True)
    for k in ("accumulated_error", "accumulated_weight", "united_error", "large_error_mark"):
        assert np.array_equal(got[k].cpu().numpy().astype(want[k].dtype), want[k], equal_nan=True), k
    for k in ("alignment_error_map", "node_error_map"):
        assert np.array_equal(got[k][0].cpu().numpy(), want[k][0], equal_nan=True), k
    assert (want["accumulated_error"] != 0).sum() > 10
    solver.close()


@pytest.mark.parametrize("width,height,nodes,times", [(97, 65, 1, 4), (96, 64, 2, 3), (129, 57, 40, 3), (65, 67, 40, 4)])
def test_node_error_of_surfels_that_repeat_a_node(oracle_mod, width, height, nodes, times):
    """A node three or four times among each surfel's four, as every scene of one or
    two nodes has it: up to 128 entries of a tile for one node."""
    scene = synth.sphere_single_view(seed=4, num_nodes=40, width=width, height=height)
    rng = np.random.default_rng(8)
    scene.canonical_nodes, scene.node_se3 = scene.canonical_nodes[:nodes], scene.node_se3[:nodes]
    scene.node_graph = scene.node_graph[:0]
    scene.surfel_knn_weight[:] = rng.uniform(0.05, 0.4, scene.surfel_knn_weight.shape)
    scene.surfel_knn[:] %= nodes
    for column in range(1, times):
        scene.surfel_knn[:, column] = scene.surfel_knn[:, 0]
    solver = NonRigidSolver(abi.make_config(scene))
    solver.set_solver_input(scene)
    got = solver.compute_alignment_error_on_nodes(maps=True)
    torch.cuda.synchronize()
    want = oracle_mod.node_error(scene, scene.node_se3, maps=True)
    for k in ("accumulated_error", "accumulated_weight", "united_error", "large_error_mark"):
        assert np.array_equal(got[k].cpu().numpy().astype(want[k].dtype), want[k], equal_nan=True), k
    for k in ("alignment_error_map", "node_error_map"):
        assert np.array_equal(got[k][0].cpu().numpy(), want[k][0], equal_nan=True), k
    assert (want["accumulated_weight"] > 10).any()
    solver.close()


@pytest.mark.parametrize("nodes,spread", [(40, False), (200, False), (3000, False), (3000, True)])
def test_node_error_of_tiles_with_few_and_many_nodes(oracle_mod, nodes, spread):
    """Tiles on both sides of the limit of nearest nodes (up to 32), summed and added
    pixel by pixel; `spread`: four nodes of each surfel's own."""
    scene = synth.sphere_single_view(seed=9, num_nodes=40, width=131, height=99)
    rng = np.random.default_rng(3)
    pos = scene.surfel_position[rng.choice(scene.num_surfels, nodes, replace=False)]
    scene.canonical_nodes = np.concatenate([pos, np.ones((nodes, 1))], 1).astype(np.float32)
    scene.node_se3 = np.tile(np.array([0, 0, 0, 1, 0.001, -0.002, 0.001, 0], np.float32), (nodes, 1))
    scene.node_graph = scene.node_graph[:0]
    d = ((scene.surfel_position[:, None] - pos[None, :]) ** 2).sum(-1)
    knn = np.argsort(d, 1)[:, :4]
    scene.surfel_knn = (rng.integers(0, nodes, knn.shape) if spread else knn).astype(np.uint16)
    scene.surfel_knn_weight = rng.uniform(0.05, 0.4, knn.shape).astype(np.float32)
    solver = NonRigidSolver(abi.make_config(scene))
    solver.set_solver_input(scene)
    got = solver.compute_alignment_error_on_nodes(maps=True)
    torch.cuda.synchronize()
    want = oracle_mod.node_error(scene, scene.node_se3, maps=True)
    for k in ("accumulated_error", "accumulated_weight", "united_error", "large_error_mark"):
        assert np.array_equal(got[k].cpu().numpy().astype(want[k].dtype), want[k], equal_nan=True), k
    for k in ("alignment_error_map", "node_error_map"):
        assert np.array_equal(got[k][0].cpu().numpy(), want[k][0], equal_nan=True), k
    # the number of nearest nodes of the tiles of 8 x 4 pixels
    index = scene.views[0].index_map
    drawn = index != 0xFFFFFFFF
    near = np.where(drawn, scene.surfel_knn[np.where(drawn, index, 0), 0].astype(np.int64), -1)
    count = [len(np.unique(near[y:y + 4, x:x + 8])) for y in range(0, 99, 4) for x in range(0, 131, 8)]
    assert min(count) <= 6
    if nodes >= 200:
        assert max(count) > 6
    solver.close()
