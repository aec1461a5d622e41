"""Sizes at which a kernel takes another path or a partial tile: the tree's
1024-position tiles, one narrow level or a grid of them in the multipoles, the
sort's single block (4096 keys) and its tile sizes (2^17, 2^20), walk groups shared by
two warps, and the copies of device arrays.  Build results are whole numbers:
equal to the oracle; forces of shared groups equal, bit for bit, those of the
same system inside an ensemble too large for sharing."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tree(pos, nleaf, ncrit, ls=5):
    import bonsai2_b200 as B
    t = B.Treecode(eps=0.01, theta=0.5, ncrit=ncrit, nleaf=nleaf)
    t.alloc(pos.shape[0])
    t.h_ptclPos[:] = pos
    t.ptcl_h2d()
    t.buildTree(nleaf)
    t.computeMultipoles()
    t.makeGroups(ls, ncrit)
    return t


@pytest.mark.parametrize("n,nleaf,ncrit,same", [
    (1, 16, 64, 0), (2, 1, 1, 0), (33, 16, 64, 0), (1023, 1, 64, 0), (1024, 64, 128, 0), (1025, 16, 64, 0),
    (4095, 8, 32, 0), (4096, 16, 64, 0), (4097, 16, 64, 0), (8193, 63, 16, 0), (5000, 5, 64, 2000),
    (1 << 17, 16, 64, 0), ((1 << 17) + 1, 16, 64, 0), (1 << 20, 16, 64, 0), ((1 << 20) + 3, 16, 64, 0)])
@pytest.mark.filterwarnings("ignore:.*deeper than 21 levels")
def test_build_matches_oracle(oracle, lib, n, nleaf, ncrit, same):
    pos, _ = oracle.plummer_float4(n, n % 97 + 1)
    pos[:same] = pos[0]
    t = _tree(pos, nleaf, ncrit)
    S = oracle.OracleStep(pos, theta=0.5, eps=0.01, nleaf=nleaf, ncrit=ncrit, level_split=5).build().groups()
    k, c, g = t.keys(), t.cells(), t.groups()
    tk = oracle.tree_keys(pos, S.box)
    tp = oracle.argsort_u64(tk)
    assert np.array_equal(k["tree_keys"], tk[tp]) and np.array_equal(k["tree_perm"], tp)
    assert np.array_equal(k["ph_keys"], S.ph_sorted) and np.array_equal(k["ph_perm"], S.ph_perm)
    assert np.array_equal(c["cell_data"], S.tree.cell_data())
    assert np.array_equal(g[:, 0], S.gbeg) and np.array_equal(g[:, 1], S.gnp)
    # mass and centre of mass of every cell, from prefix sums over the sorted
    # particles: doubles rounded to float once, and the prefix sums' own
    # cancellation (1e-16 of the whole sum)
    cd, j = c["cell_data"], pos[tp].astype(np.float64)
    pre = np.concatenate([np.zeros((1, 4)), np.cumsum(np.column_stack([j[:, :3] * j[:, 3:], j[:, 3]]), axis=0)])
    s = pre[cd[:, 3]] - pre[cd[:, 2]]
    m = s[:, 3]
    assert np.allclose(c["mono"][:, 3], m, rtol=1e-7, atol=1e-13)
    size = np.abs(j[:, :3]).max()
    assert np.allclose(c["mono"][:, :3], s[:, :3] / m[:, None], rtol=1e-7, atol=size * (1e-7 + 1e-12 / m.min()))
    t.close()


# each system small enough for shared groups, their ensemble too large (layout 1
# shares one row of 32 between two warps); groups of nCrit 16 are one row of 16
# and never shared, alone or together
@pytest.mark.parametrize("ncrit,layout,sizes", [
    (64, 0, (1, 15, 1000, 30011, 85000)), (32, 0, (2, 300, 12001, 14001)), (128, 0, (5, 4000, 200001, 330000)),
    (64, 1, (1, 33, 700, 20011, 40000)), (16, 0, (700, 20000))])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("theta_mode", [0, 1, 3])
def test_shared_groups_bit_identical(lib, ncrit, layout, sizes, precision, theta_mode):
    """Four steps: in the network's and the relative mode (1, 3) the first walk is
    at the fixed angle, and from the third on the features are those of a
    relative walk's statistics, which one of a shared group's warps records."""
    import bonsai2_b200 as B
    from bonsai2_b200 import learned
    from bonsai2_b200.ensemble import plummer_ensemble
    counts = np.array(sizes, np.int32)
    pos, vel = plummer_ensemble(counts, base_seed=11)
    prm = dict(eps=0.01, theta=0.7, ncrit=ncrit)
    w = learned.init_weights(3)

    def run(t, p, v):
        if precision:
            t.set_precision(1)
        t.set_walk_layout(layout)
        if theta_mode == 1:
            assert lib.bonsai_set_mlp_weights(t.handle, w.ctypes.data_as(ctypes.c_void_p), w.size) == 0
        if theta_mode:
            assert lib.bonsai_set_theta_mode(t.handle, theta_mode, *((1e-2, 1e-2) if theta_mode == 3 else
                                                                     (learned.YLO, learned.YHI))) == 0
        t.h_ptclPos[:] = p
        t.h_ptclVel[:] = v
        t.ptcl_h2d()
        t.step(4)
        assert t.synchronize() == 0
        t.ptcl_d2h()
        out = t.h_ptclPos.copy(), t.h_ptclVel.copy(), t.get_acc()
        t.close()
        return out

    t = B.Treecode(**prm)
    t.set_systems(counts)
    whole = run(t, pos, vel)
    off = np.concatenate([[0], np.cumsum(counts)])
    for s in range(len(counts)):
        a, b = off[s], off[s + 1]
        u = B.Treecode(**prm)
        u.alloc(int(counts[s]))
        alone = run(u, pos[a:b], vel[a:b])
        for x, y in zip(whole, alone):
            assert np.array_equal(x[a:b], y)


@pytest.mark.parametrize("n", [1, 255, 257, 70001])
@pytest.mark.parametrize("shift", [0, 1, 4])
def test_device_arrays(lib, n, shift):
    """Device arrays at 16-byte boundaries (read and written by kernels) and
    beside them (copied): the same particles either way."""
    import torch

    import bonsai2_b200 as B
    pos, vel = B.plummer(n, 3)
    t = B.Treecode(eps=0.01, theta=0.6)
    t.alloc(n)
    flat = [torch.zeros(4 * n + 8, device="cuda") for _ in range(5)]
    part = [x[shift:shift + 4 * n] for x in flat]
    part[0].copy_(torch.from_numpy(pos.ravel()))
    part[1].copy_(torch.from_numpy(vel.ravel()))
    torch.cuda.synchronize()
    ptr = [ctypes.c_void_p(x.data_ptr()) for x in part]
    assert lib.bonsai_set_particles_device(t.handle, ptr[0], ptr[1], n) == 0
    t.step(1)
    assert lib.bonsai_get_particles_device(t.handle, ptr[2], ptr[3], ptr[4]) == 0
    assert t.synchronize() == 0
    t.ptcl_d2h()
    acc = t.get_acc()
    for x, y in zip(part[2:], (t.h_ptclPos, t.h_ptclVel, acc)):
        assert np.array_equal(x.cpu().numpy().reshape(n, 4), y)
    for x in flat[2:]:  # nothing beside the arrays
        assert x[:shift].count_nonzero() == 0 and x[shift + 4 * n:].count_nonzero() == 0
    # one array alone
    part[4].zero_()
    torch.cuda.synchronize()
    assert lib.bonsai_get_particles_device(t.handle, None, None, ptr[4]) == 0
    assert np.array_equal(part[4].cpu().numpy().reshape(n, 4), acc)
    t.close()


@pytest.mark.parametrize("n", [1, 2, 3, 4, 4097, 70000])
@pytest.mark.parametrize("precision", [0, 1])
def test_double_positions_round_trip(lib, n, precision):
    """Positions split into float pairs on the device and joined again: exactly
    what the same split gives on the host, for even and odd counts."""
    import bonsai2_b200 as B
    rng = np.random.default_rng(n)
    pos = np.column_stack([rng.normal(size=(n, 3)) * 10.0 ** rng.uniform(-6, 6, (n, 1)), rng.uniform(0.1, 1, n)])
    vel = rng.normal(size=(n, 4)).astype(np.float32)
    t = B.Treecode()
    t.alloc(n)
    t.set_precision(precision)
    t.set_particles_f64(pos, vel)
    p, v, _ = t.get_particles_f64()
    hi = pos.astype(np.float32)
    want = hi.astype(np.float64)
    if precision:
        want[:, :3] += (pos[:, :3] - want[:, :3]).astype(np.float32)
    assert np.array_equal(p, want) and np.array_equal(v, vel)
    t.close()


@pytest.mark.parametrize("n,ns", [(1, 1), (7, 3), (300, 1), (300, 257), (2049, 1000), (5000, 5000), (1000, 40000),
                                  (2000, 200000)])
@pytest.mark.parametrize("include_self", [True, False])
def test_direct_sum_slices(oracle, lib, n, ns, include_self):
    """The direct sum at 444 slices (also of fewer sources), 481, 148, 18 (runs of
    two and three) and 3 (empty runs).  FP64 on both sides: the difference is
    a few roundings of 2^-53 for each of at most 5000 terms, 1e-12 of the terms'
    magnitudes, which the near pairs dominate."""
    import bonsai2_b200 as B
    pos, _ = B.plummer(n, 6)
    t = B.Treecode(eps=0.05)
    t.alloc(n)
    t.h_ptclPos[:] = pos
    t.ptcl_h2d()
    sample = np.random.default_rng(n).integers(0, n, ns).astype(np.int32)
    got = t.direct_fp64(sample, include_self)
    t.close()
    want = oracle.direct_fp64(pos, sample, 0.05, include_self)
    assert np.allclose(got, want, rtol=1e-12, atol=1e-12 * max(1.0, np.abs(want).max()))


def test_handles_in_threads(lib):
    """Handles stepped from threads of their own at once give what each gives
    alone: their steps share the GPU, grid-wide barriers of the multipoles'
    level launches among them."""
    import threading

    import bonsai2_b200 as B
    sizes = [300007, 40000, 300007, 150001, 9000]
    steps = 12

    inputs = [B.plummer(n, k + 1) for k, n in enumerate(sizes)]  # (one rand() stream: not in the threads)

    def run(n, out, k):
        pos, vel = inputs[k]
        t = B.Treecode(eps=0.01, theta=0.8)
        t.alloc(n)
        t.h_ptclPos[:] = pos
        t.h_ptclVel[:] = vel
        t.ptcl_h2d()
        t.step(steps)
        status = t.synchronize()
        t.ptcl_d2h()
        out[k] = (status, t.h_ptclPos.copy(), t.get_acc())
        t.close()

    alone, together = {}, {}
    for k, n in enumerate(sizes):
        run(n, alone, k)
    threads = [threading.Thread(target=run, args=(n, together, k)) for k, n in enumerate(sizes)]
    for x in threads:
        x.start()
    for x in threads:
        x.join()
    for k in range(len(sizes)):
        assert alone[k][0] == 0 and together[k][0] == 0
        assert np.array_equal(alone[k][1], together[k][1]) and np.array_equal(alone[k][2], together[k][2])
