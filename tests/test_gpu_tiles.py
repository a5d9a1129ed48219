"""The pass at the edges of its kernels' tiles, against the oracle and the
host build.

Tolerances are those of the parity tests: FP64 1e-9 on the gradient (1e-7
from P = 9, where the equivalent densities are as ill-conditioned as FP64
holds and two FP64 implementations agree to that), FP32-mixed 1e-5.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def uniform01(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.random((n, 3))
    q = rng.random(n) * 2 - 1
    return x, q - q.mean()


def l2(a, b):
    return float(np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(np.asarray(b)))


def args(pkg, P, ncrit, images, precision, stages=None):
    return pkg.Argument(P=P, ncrit=ncrit, images=images, cycle=1.0, x=(0.5, 0.5, 0.5), dipole_correction=0,
                        divide_4pi=1, precision=precision, stages=pkg.STAGE_ALL if stages is None else stages)


# far field at every order with its own transform kernels and at two without
# (2, 11), with 9 and with 73 target parents (the Hadamard's tiles hold 8, 24
# and 96), periodic and free
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("P,n,ncrit,images", [(2, 900, 24, 1), (4, 900, 24, 2), (5, 700, 12, 0), (6, 2500, 8, 1),
                                              (7, 900, 24, 3), (8, 900, 24, 0), (9, 900, 24, 2), (10, 2500, 8, 1),
                                              (11, 600, 24, 1)])
def test_far_field_at_every_order(pkg, oracle, P, n, ncrit, images, precision):
    x, q = uniform01(n, 100 + P)
    # from P = 9 the two pseudo-inverses (two SVDs, cut at 4e-16) differ by up
    # to 1e-7 of the whole field, of which the far part is a tenth here
    stages = "far" if P < 9 else "all"
    f = pkg.LaplaceFMM(x, q, args(pkg, P, ncrit, images, precision, pkg.STAGE_FAR if P < 9 else pkg.STAGE_ALL))
    phi, grad = f.solve()
    f.close()
    rphi, rgrad = oracle.FMM(x, q, P, ncrit, images, 1.0, center=(0.5, 0.5, 0.5), divide_4pi=1).solve(stages=stages)
    tol = 1e-5 if precision else 1e-9 if P < 9 else 1e-7
    assert l2(grad, rgrad) < tol
    assert l2(phi - phi.mean(), rphi - rphi.mean()) < max(tol, 1e-8)


# near field where source lists are cut into parts: a leaf of 200 bodies
# beside leaves of one to eight, and lists of many tiny leaves (more than 32
# entries); target groups of 1, 4, 5, 16, 17, 32 and 33 bodies
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("images", [0, 1])
def test_near_field_with_long_lists(pkg, oracle, images, precision):
    rng = np.random.default_rng(7)
    sizes = [200, 33, 32, 17, 16, 5, 4, 1]
    corners = np.array([[i, j, k] for i in (0, 1) for j in (0, 1) for k in (0, 1)])
    parts = [(c + rng.random((m, 3))) * 0.25 for c, m in zip(corners, sizes)]  # eight leaves of edge 1/4
    parts.append(0.5 + 0.02 * rng.standard_normal((1500, 3)))  # a dense cluster at their corner
    x = np.clip(np.concatenate(parts), 1e-6, 1 - 1e-6)
    q = rng.standard_normal(len(x))
    q -= q.mean()
    f = pkg.LaplaceFMM(x, q, args(pkg, 4, 8 if images else 200, images, precision, pkg.STAGE_NEAR))
    phi, grad = f.solve()
    f.setup()
    lo, src, _ = f.leaf_lists()
    ints, _ = f.cells()
    leaf = ints[:f.info()["ncell"]]
    bnum = leaf[(leaf[:, 3] == 0) & (leaf[:, 5] > 0), 5][:f.info()["nleaf"]]
    bodies = np.add.reduceat(bnum[src], lo[:-1])
    assert bodies.max() > 512, "a list long enough to be cut"
    f.close()
    rphi, rgrad = oracle.FMM(x, q, 4, 8 if images else 200, images, 1.0, center=(0.5, 0.5, 0.5),
                             divide_4pi=1).solve(stages="near")
    tol = 1e-5 if precision else 1e-12  # FP64: a sum of 2000 terms, ~1e-15 each
    assert l2(grad, rgrad) < tol and l2(phi, rphi) < tol


# a part of a list may hold no entry at all: leaves of 625 bodies beside parts
# of 256
@pytest.mark.parametrize("precision", [0, 1])
def test_near_field_with_entries_above_a_part(pkg, precision):
    x, q = uniform01(5000, 12)
    f = pkg.LaplaceFMM(x, q, args(pkg, 4, 900, 0, precision, pkg.STAGE_NEAR))
    phi, grad = f.solve()
    assert f.info()["nleaf"] == 8  # each beside all others: the near field is the direct sum
    f.close()
    d = x[:, None] - x[None]
    r2 = (d * d).sum(2)
    np.fill_diagonal(r2, np.inf)
    t = q / np.sqrt(r2) / (4 * np.pi)
    tol = 1e-5 if precision else 1e-12
    assert l2(phi, t.sum(1)) < tol
    assert l2(grad, -np.einsum("ij,ijk->ik", t / r2, d)) < tol


# FP32 terms meet in FP64: neither the two halves of a packed sum nor the terms
# of two small leaves are added in FP32, where a term of 2^-30 beside one of 1
# is lost.  One leaf of 3 bodies, one of 40 (the form for long entries), and
# 26 leaves of one body around a target
@pytest.mark.parametrize("case", ["leaf of 3", "leaf of 40", "leaves of 1"])
def test_fp32_terms_meet_in_fp64(pkg, case):
    if case == "leaves of 1":
        x = (np.stack(np.meshgrid(*[np.arange(3)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) / 4
        target, strong, weak, ncrit = 13, 4, [k for k in range(27) if k not in (4, 13)], 1
    else:
        n = 3 if case == "leaf of 3" else 40
        x = np.random.default_rng(3).random((n, 3)) * 0.2
        x[:3] = [[0.25, 0.5, 0.5], [0.5, 0.75, 0.5], [0.5, 0.5, 0.5]]  # sources 0 and 1 of a pair
        target, strong, weak, ncrit = 2, 0, [1], 64
    q = np.zeros(len(x))
    f = pkg.LaplaceFMM(x, q, args(pkg, 4, ncrit, 0, 1, pkg.STAGE_NEAR))
    f.setup()
    q[strong] = 1.0
    phi0, grad0 = f.evaluate(q)
    q[weak] = 2.0 ** -30
    phi, grad = f.evaluate(q)
    f.close()
    d = x[target] - x[weak]
    t = 2.0 ** -30 / np.linalg.norm(d, axis=1) / (4 * np.pi)
    g = t[:, None] * d / (d * d).sum(1)[:, None]
    # the weak terms' own FP32 rounding (reciprocal square root: 2^-22)
    assert abs(phi[target] - phi0[target] - t.sum()) < 1e-5 * t.sum()
    assert np.abs(grad[target] - grad0[target] + g.sum(0)).max() < 1e-5 * np.abs(g).sum()


# octrees below the first sorted digits (12 levels), and leaves above the size
# ordered by counting (1500 bodies)
@pytest.mark.parametrize("ncrit,scale", [(4, 2e-4), (1500, 1.0)])
def test_device_tree_beyond_its_fast_paths(pkg, ncrit, scale):
    x, q = uniform01(6000, 8)
    x = 0.3 + scale * (x - 0.3)
    a = args(pkg, 4, ncrit, 1, 1)
    h = pkg.LaplaceFMM(x, q, a)
    h.setup()
    d = pkg.LaplaceFMM(x, q, a)
    xd, qd = torch.from_numpy(x).cuda(), torch.from_numpy(q).cuda()
    torch.cuda.synchronize()
    for _ in range(2):  # a second set-up reuses every buffer
        d.setup_device(xd.data_ptr(), qd.data_ptr(), len(q))
    if ncrit == 4:
        assert h.info()["depth_max"] > 10
    assert all(np.array_equal(u, v) for u, v in zip(h.cells(), d.cells()))
    assert np.array_equal(h.perm(), d.perm())
    assert all(np.array_equal(u, v) for u, v in zip(h.leaf_lists(), d.leaf_lists()))
    ph, gh = h.evaluate()
    d.evaluate_device()
    pd, gd = d.download()
    assert np.array_equal(ph, pd) and np.array_equal(gh, gd)
    h.close()
    d.close()


# the first pass of a plan is issued launch by launch, the second captured,
# the third replayed: the same outputs
@pytest.mark.parametrize("precision", [0, 1])
def test_first_pass_equals_replayed_ones(pkg, precision):
    x, q = uniform01(5000, 9)
    f = pkg.LaplaceFMM(x, q, args(pkg, 5, 40, 2, precision))
    first = f.solve()
    for _ in range(3):
        again = f.evaluate()
        assert all(np.array_equal(u, v) for u, v in zip(first, again))
    f.close()


# 15000 leaves run their operators in 64 x 64 tiles, a sixteenth of them in
# 16 x 32 ones: every body's outputs are the same bit for bit
def test_small_and_large_operator_tiles_agree(pkg):
    x, q = uniform01(30000, 10)
    a, n, R = args(pkg, 6, 4, 0, 0), 30000, 16
    f = pkg.LaplaceFMM(x, q, a)
    f.setup()
    phi, grad = f.evaluate()
    f.close()
    hs = []
    for r in range(R):
        f = pkg.LaplaceFMM(x, q, a)
        f.shard(r, R)
        f.setup()
        f.upload()
        hs.append(f)
    total = torch.zeros(hs[0].shard_sizes()[1], dtype=torch.float64, device="cuda")
    for f in hs:
        buf = torch.zeros_like(total)
        torch.cuda.synchronize()
        f.shard_upward(buf.data_ptr())  # returns when buf is complete
        total += buf
    p = torch.zeros(n, dtype=torch.float64, device="cuda")
    g = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for f in hs:
        f.shard_downward(total.data_ptr(), p.data_ptr(), g.data_ptr())
        idx = f.shard_bodies()
        assert np.array_equal(p.cpu().numpy()[idx], phi[idx]) and np.array_equal(g.cpu().numpy()[idx], grad[idx])
        f.close()


# a forward and backward step repeated on one set-up: the adjoint's transposed
# pass is issued launch by launch, then captured, then replayed, with other
# weights each time
@pytest.mark.parametrize("precision", [0, 1])
def test_repeated_adjoints_agree(pkg, precision):
    x, q = uniform01(6000, 11)
    f = pkg.LaplaceFMM(x, q, args(pkg, 5, 40, 1, precision))
    f.setup()
    w = [np.random.default_rng(k).standard_normal(len(q)) for k in (1, 2)]
    first = [f.adjoint(v) for v in w]
    for _ in range(2):
        f.evaluate(q)
        for v, ref in zip(w, first):
            assert all(np.array_equal(a, b) for a, b in zip(f.adjoint(v), ref))
    f.close()
