"""The off-diagonal blocks at the edges of their kernels' ranges: the pairs that
16 lanes take together (more than a hundred entries, up to more than the length
buckets tell apart) and the pairs a thread takes, in less than a warp of pairs,
about one ordering window and several windows."""
import numpy as np
import pytest

from multiviewdynrecon_b200 import abi, synth

pytestmark = pytest.mark.gpu


def _twist_rows(p):
    z = np.zeros(len(p))
    x, y, c = p.T
    skew = np.stack([z, c, -y, -c, z, x, y, -x, z], -1).reshape(-1, 3, 3)
    return np.concatenate([skew, np.broadcast_to(np.eye(3), (len(p), 3, 3))], 2)


def _expected(scene, get, lam_smooth):
    """Upper blocks in float64 from the exported term data, the sums of the
    absolute values of their addends, and the pairs' entry counts."""
    jac = get(abi.ARRAY_TERM_JACOBIAN).astype(np.float64)[:, :6]
    knn = get(abi.ARRAY_DENSE_KNN).astype(np.int64)
    w = get(abi.ARRAY_DENSE_KNN_WEIGHT).astype(np.float64)
    sm = get(abi.ARRAY_SMOOTH_TERMS).astype(np.float64)
    index = get(abi.ARRAY_NODEPAIR_TERM_INDEX).astype(np.int64)
    key = get(abi.ARRAY_NODEPAIR_KEY).astype(np.int64)
    rg = get(abi.ARRAY_NODEPAIR_TERM_RANGE).astype(np.int64)
    upper = key // 4096 < key % 4096
    i, j = key[upper] // 4096, key[upper] % 4096
    rg = rg[upper]
    length = rg[:, 1] - rg[:, 0]
    pair = np.repeat(np.arange(len(i)), length)
    entry = np.concatenate([np.arange(a, b) for a, b in rg])
    t = index[entry]
    blocks, size = np.zeros((len(i), 36)), np.zeros((len(i), 36))

    def add(p, m):
        np.add.at(blocks, p, m.reshape(-1, 36))
        np.add.at(size, p, np.abs(m).reshape(-1, 36))

    d = t < len(knn)
    p, td = pair[d], t[d]
    wi = (w[td] * (knn[td] == i[p][:, None])).sum(1)
    wj = (w[td] * (knn[td] == j[p][:, None])).sum(1)
    add(p, (wi * wj)[:, None, None] * jac[td][:, :, None] * jac[td][:, None, :])
    p, k = pair[~d], t[~d] - len(knn)
    p, k = p[sm[k, 6] != 0], k[sm[k, 6] != 0]
    first = scene.node_graph[k, 0] == i[p]
    a, b = sm[k, 0:3], sm[k, 3:6]
    fi, fj = (_twist_rows(np.where(first[:, None], x, y)) for x, y in ((a, b), (b, a)))
    add(p, -lam_smooth ** 2 * np.einsum("ncr,nck->nrk", fi, fj))
    return blocks.reshape(-1, 6, 6), size.reshape(-1, 6, 6), length, upper


@pytest.mark.parametrize("precision", [abi.PRECISION_MIXED, abi.PRECISION_FP32])
@pytest.mark.parametrize("nodes,width,height", [(12, 24, 18), (30, 120, 90), (140, 96, 72), (700, 160, 120)])
def test_upper_blocks_at_every_pair_length(precision, nodes, width, height):
    from multiviewdynrecon_b200.solver import NonRigidSolver
    scene = synth.sphere_single_view(seed=3, num_nodes=nodes, width=width, height=height)
    # (so few nodes lie too far apart for the distance weights)
    scene.surfel_knn_weight[:] = (0.4, 0.3, 0.2, 0.1)
    g = NonRigidSolver(abi.make_config(scene, precision=precision))
    g.set_solver_input(scene)
    g.build_index()
    g.gn_iteration(4)
    g.solved_node_se3()  # raises on a device-side error
    want, size, length, upper = _expected(scene, g.get_array, 5.0)
    got = g.get_array(abi.ARRAY_OFFDIAG_BLOCKS).astype(np.float64)[upper].reshape(-1, 6, 6).transpose(0, 2, 1)
    if nodes == 30:
        assert length.max() > 1020 and length.min() < 100
    # running float sums of n addends, each a product of rounded factors: n + 8
    # half-ulps of the addends' sizes; double sums are rounded to float once
    half_ulps = length + 8 if precision == abi.PRECISION_FP32 else np.full(len(length), 2)
    assert np.all(np.abs(got - want) <= half_ulps[:, None, None] * 2.0 ** -24 * size + 1e-30)
    g.close()


def test_blocks_do_not_depend_on_the_share_taken_by_group():
    """max_nodes sets how many pairs of a window go to the 16-lane groups (512, 256,
    128 or 32 of 1024); both forms give the same bits."""
    from multiviewdynrecon_b200.solver import NonRigidSolver
    scene = synth.torso_multi_view(seed=3, num_nodes=400, num_views=2, width=160, height=120, features_per_view=40,
                                   cross_per_pair=40)
    got = []
    for max_nodes in (400, 5119, 5120, 10239, 10240, 16383, 16384):
        cfg = abi.make_config(scene)
        cfg.max_nodes = max_nodes
        solver = NonRigidSolver(cfg)
        solver.set_solver_input(scene)
        solver.build_index()
        solver.gn_iteration(5)
        got.append(solver.get_array(abi.ARRAY_OFFDIAG_BLOCKS))
        assert solver.counts().half_pairs > 1024  # several windows
        solver.close()
    for blocks in got[1:]:
        assert np.array_equal(blocks, got[0])


@pytest.mark.parametrize("precision", [abi.PRECISION_MIXED, abi.PRECISION_FP32])
@pytest.mark.parametrize("count,capacity", [(4, 1279), (4, 1280), (5, 1300), (4, 3071), (4, 3072)])
def test_batches_at_each_share_of_pairs(precision, count, capacity):
    """A batch with little image per node takes fewer pairs by group from 5,120 nodes of
    capacity on: the bits of a single solve on both sides of the line."""
    import torch
    from multiviewdynrecon_b200.solver import BatchSolver, NonRigidSolver
    scene = synth.sphere_single_view(seed=3, num_nodes=300, width=160, height=120)
    cfg = abi.make_config(scene, precision=precision)
    single = NonRigidSolver(cfg)
    single.set_solver_input(scene)
    single.solve_non_rigid_alignment(2, 6)
    want = single.get_array(abi.ARRAY_INCREMENT)
    cfg.max_nodes, cfg.max_node_pairs = capacity, 32 * scene.num_nodes
    b = BatchSolver(cfg, count)
    for i in range(count):
        b.set_input(i, scene)
    b.solve(2, 6)
    torch.cuda.synchronize()
    for i in range(count):
        assert np.array_equal(b.instance(i).get_array(abi.ARRAY_INCREMENT), want)
    b.close()
    single.close()
