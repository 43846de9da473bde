"""The PCG of a single solve as one resident launch against the launched form
(which a convergence tolerance selects): the same bits, at the edges of the
CTAs' rows, with more entries than fit in shared memory, and with several
solvers at work at once."""
import threading

import numpy as np
import pytest

from multiviewdynrecon_b200 import abi, synth

pytestmark = pytest.mark.gpu


def _scene(nodes, crowded=False):
    scene = synth.torso_multi_view(seed=6, num_nodes=nodes, num_views=2, width=96, height=72, features_per_view=30,
                                   cross_per_pair=30)
    scene.surfel_knn_weight[:] = (0.4, 0.3, 0.2, 0.1)
    if crowded:  # every node a neighbour of nearly every other one
        rng = np.random.default_rng(1)
        scene.surfel_knn[:] = rng.permuted(np.tile(np.arange(nodes), (scene.num_surfels, 1)), axis=1)[:, :4]
    return scene


def _solver(scene, tolerance):
    from multiviewdynrecon_b200.solver import NonRigidSolver
    cfg = abi.make_config(scene, precision=abi.PRECISION_MIXED, pcg_tolerance=tolerance)
    cfg.max_node_pairs = max(16 * scene.num_nodes, scene.num_nodes * min(scene.num_nodes, 128))
    return NonRigidSolver(cfg)


@pytest.mark.parametrize("nodes,crowded,iterations", [(16, False, 1), (33, False, 2), (64, True, 7), (100, True, 15),
                                                      (1000, False, 15), (1025, False, 4)])
def test_resident_matches_launched(nodes, crowded, iterations):
    scene = _scene(nodes, crowded)
    got = []
    for tolerance in (0.0, 1e-30):  # (never reached: the fixed count, launch by launch)
        g = _solver(scene, tolerance)
        g.set_solver_input(scene)
        g.solve_non_rigid_alignment(2, iterations)
        got.append((g.solved_node_se3().cpu().numpy(), g.get_array(abi.ARRAY_INCREMENT),
                    g.get_array(abi.ARRAY_PCG_RESIDUALS)))
        if crowded:
            rows = np.diff(g.get_array(abi.ARRAY_BLKROW_OFFSET).astype(np.int64))
            assert rows[:32].sum() > 736
        g.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b, equal_nan=True)


def test_solvers_on_several_streams():
    import torch
    scenes = [_scene(n) for n in (300, 700, 1000)]
    solvers = [_solver(s, 0.0) for s in scenes]
    inputs, want = [], []
    for g, s in zip(solvers, scenes):
        inputs.append(g.set_solver_input(s))
        g.solve_non_rigid_alignment(3, 10)
        want.append(g.solved_node_se3().cpu())
    torch.cuda.synchronize()
    wrong = []

    def work(k):
        stream = torch.cuda.Stream()
        out = torch.empty_like(want[k]).pin_memory()
        for _ in range(10):
            solvers[k].set_solver_input(inputs[k], stream=stream)
            solvers[k].solve_non_rigid_alignment(3, 10, stream=stream)
            solvers[k].solved_node_se3_async(out, stream=stream)
            if solvers[k].counts(stream=stream).error_flags or not torch.equal(out, want[k]):
                wrong.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def _rounds(solver, inputs, want, count):
    """`count` solves on a stream of its own; a failed call raises in the caller."""
    import torch
    stream = torch.cuda.Stream()
    out = torch.empty_like(want).pin_memory()
    for k in range(count):
        out.zero_()
        solver.set_solver_input(inputs, stream=stream)
        solver.solve_non_rigid_alignment(3, 10, stream=stream)
        solver.solved_node_se3_async(out, stream=stream)
        assert solver.counts(stream=stream).error_flags == 0, k
        assert torch.equal(out, want), k
    return count


def test_launches_that_do_not_fit_together():
    """Each solver's launch takes most or all of the SMs, so no two of them can be
    resident at once: the launches take turns, and no barrier waits for the other."""
    import torch
    from concurrent.futures import ThreadPoolExecutor
    from multiviewdynrecon_b200.solver import NonRigidSolver
    scene, work = _scene(700), []
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for nodes in (4096, 32 * sms, 3000):
        cfg = abi.make_config(scene, precision=abi.PRECISION_MIXED)
        cfg.max_nodes, cfg.max_node_pairs = nodes, 16 * nodes
        g = NonRigidSolver(cfg)
        inputs = g.set_solver_input(scene)
        g.solve_non_rigid_alignment(3, 10)
        work.append((g, inputs, g.solved_node_se3().cpu()))
    torch.cuda.synchronize()
    with ThreadPoolExecutor(len(work)) as pool:
        done = [pool.submit(_rounds, g, inputs, want, 20) for g, inputs, want in work]
        assert [d.result() for d in done] == [20, 20, 20]


def test_one_instance_lanes_as_graphs():
    """Two lanes of one instance each, whose graphs hold a resident launch per
    iteration, replayed side by side: the results of single solvers."""
    import torch
    from multiviewdynrecon_b200.solver import NonRigidSolver, StreamedBatch
    scenes = [_scene(700), _scene(600)]
    cfg = abi.make_config(None, max_nodes=4096, max_views=2, width=96, height=72, use_foreground=True,
                          use_feature=True, use_cross_view=True, max_surfels=max(s.num_surfels for s in scenes),
                          max_feature_terms=max(s.feature.count for s in scenes),
                          max_cross_terms=max(s.cross_view.count for s in scenes))
    want = []
    for s in scenes:
        g = NonRigidSolver(cfg)
        g.set_solver_input(s)
        g.solve_non_rigid_alignment(3, 10)
        want.append(g.solved_node_se3())
    lanes = StreamedBatch(cfg, 2, lanes=2)
    for _ in range(20):
        for i, s in enumerate(scenes):
            lanes.set_input(i, s)
        lanes.solve(3, 10)
        for i in range(2):
            assert torch.equal(lanes.node_se3(i), want[i])
    lanes.close()
