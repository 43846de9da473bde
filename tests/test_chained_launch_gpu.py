"""Chained kernel launches inside a caller's graph, behind a node that is not a kernel:
two replayed iterations give the bits of two plain ones."""
import numpy as np
import pytest
import torch

from conftest import small_scene
from multiviewdynrecon_b200 import abi
from multiviewdynrecon_b200.solver import NonRigidSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,mode", [(abi.PRECISION_FP32, abi.MODE_MATERIALIZED),
                                            (abi.PRECISION_MIXED, abi.MODE_MATERIALIZED),
                                            (abi.PRECISION_MIXED, abi.MODE_MATRIX_FREE)])
def test_captured_iterations_equal_plain_ones(precision, mode):
    scene = small_scene("torso")
    solver = NonRigidSolver(abi.make_config(scene, precision=precision, mode=mode))
    solver.set_solver_input(scene)
    solver.build_index()
    for _ in range(2):
        solver.gn_iteration(5)
    torch.cuda.synchronize()
    want = solver.get_array(abi.ARRAY_INCREMENT), solver.get_array(abi.ARRAY_NODE_SE3)
    solver.set_solver_input(scene)
    solver.build_index()
    torch.cuda.synchronize()
    graph, stream, cleared = torch.cuda.CUDAGraph(), torch.cuda.Stream(), torch.ones(1000, device="cuda")
    with torch.cuda.stream(stream):
        graph.capture_begin(capture_error_mode="relaxed")
        cleared.zero_()
        solver.gn_iteration(5, stream=stream)
        graph.capture_end()
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(solver.get_array(abi.ARRAY_INCREMENT), want[0])
    assert np.array_equal(solver.get_array(abi.ARRAY_NODE_SE3), want[1])
    solver.close()


@pytest.mark.parametrize("precision,mode", [(abi.PRECISION_FP32, abi.MODE_MATERIALIZED),
                                            (abi.PRECISION_MIXED, abi.MODE_MATERIALIZED),
                                            (abi.PRECISION_MIXED, abi.MODE_MATRIX_FREE)])
@pytest.mark.parametrize("count", [1, 2, 3, 4])
def test_chained_streams_equal_plain_graphs(precision, mode, count):
    """Up to three instances are launched chained on a stream and plainly in the batch's
    graph: the same bits."""
    from multiviewdynrecon_b200.solver import BatchSolver
    scene = small_scene("torso")
    b = BatchSolver(abi.make_config(scene, precision=precision, mode=mode), count)
    got = []
    for use_graph in (False, True, True, False):
        for i in range(count):
            b.set_input(i, scene)
        b.solve(3, 7, use_graph=use_graph)
        torch.cuda.synchronize()
        got.append([b.instance(i).get_array(abi.ARRAY_NODE_SE3) for i in range(count)])
    for x in got:
        assert all(np.array_equal(a, got[0][0]) for a in x)
    b.close()
