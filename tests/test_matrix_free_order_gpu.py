"""The matrix-free J.d takes the pixel terms last in small launches and first in large
ones: the same bits either way."""
import numpy as np
import pytest
import torch

from conftest import small_scene
from multiviewdynrecon_b200 import abi
from multiviewdynrecon_b200.solver import BatchSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.PRECISION_MIXED, abi.PRECISION_FP32])
@pytest.mark.parametrize("recompute", [False, True])
@pytest.mark.parametrize("kind", ["sphere", "torso"])
def test_both_orders_give_the_same_increments(kind, precision, recompute):
    scene = small_scene(kind)
    got = []
    # (instances, capacity): small, more than four, at the largest small and the smallest large one
    for count, nodes in ((1, 0), (5, 0), (1, 16384), (1, 16385)):
        cfg = abi.make_config(scene, precision=precision, mode=abi.MODE_MATRIX_FREE, recompute_jacobians=recompute)
        if nodes:
            cfg.max_nodes, cfg.max_node_pairs = nodes, 32 * scene.num_nodes
        b = BatchSolver(cfg, count)
        for i in range(count):
            b.set_input(i, scene)
        b.solve(2, 6)
        torch.cuda.synchronize()
        got += [b.instance(i).get_array(abi.ARRAY_INCREMENT) for i in range(count)]
        b.close()
    assert np.abs(got[0]).max() > 0
    for x in got[1:]:
        assert np.array_equal(x, got[0])
