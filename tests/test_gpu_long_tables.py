"""Pixels that open more nodes, or meet more expansions, than a warp's shared
tables hold: the tiles left for the long tables, groups narrower than a warp
there, pixels that are past those as well, through every entry point that
descends.  Indices and path probabilities equal the CPU oracle's bit for bit;
and an image several times taller than wide takes about as long per pixel as
any other."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
PRECISION = 0.01
# entries of the tables in csrc/uds_sample.cu: WarpTables (nodes, expansions) and LongTables
SHORT, LONG = (224, 192), 8192


def T(a):
    return torch.as_tensor(np.ascontiguousarray(a)).to(device=DEV, dtype=torch.float32)


@pytest.fixture(scope="module")
def smp():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from unbiased_differentiable_splatting_gb300 import _lib
    from unbiased_differentiable_splatting_gb300.cudaExtensions import sampling
    _lib.load()
    return sampling


def cloud(seed, N, W, H, f, sd):
    rng = np.random.default_rng(seed)
    z = rng.uniform(-2.4, -1.6, N)
    u = rng.uniform(0.0, 1.0, size=(N, 2))
    pts = np.stack([(u[:, 0] - 0.5) * -z * W / f, (u[:, 1] - 0.5) * -z * H / f, z], 1)
    n = rng.normal(size=(N, 3))
    n[:, 2] = np.abs(n[:, 2]) + 0.5
    n /= np.linalg.norm(n, axis=1, keepdims=True)
    return pts.astype(np.float32), n.astype(np.float32), np.full((N, 2), sd, np.float32)


def table_sizes(tree, W, H):
    """(nodes opened, expansions met) of the image's pixel with most of them."""
    t = tree.export()
    radius = np.sqrt(2.0) * tree.h * np.sqrt(-np.log(PRECISION / t["count"]))
    worst = (0, 0)
    for i in range(0, W, max(W // 4, 1)):
        for j in range(0, H, max(H // 8, 1)):
            level, opened, met = np.array([0]), 0, 0
            while level.size:
                met += int((t["degree"][level] >= 0).sum())
                level = level[t["degree"][level] < 0]
                b = t["box"][level]
                d = np.hypot(i - np.clip(i, b[:, 0], b[:, 2]), j - np.clip(j, b[:, 1], b[:, 3]))
                level = level[d < radius[level]]
                opened += level.size
                level = np.concatenate([t["left"][level], t["right"][level]])
            worst = max(worst, (opened, met))
    return worst


def case(N, W, H, f, sd, degree):
    pts, nrm, s = cloud(N, N, W, H, f, sd)
    h = oracle.view_bandwidth(W, H, f, pts, nrm, s, 0.0)
    tree = oracle.Tree(W, H, f, pts, h, oracle.cull_radius(h, PRECISION), PRECISION, max_degree=degree)
    return pts, nrm, s, h, tree


# splats, image, focal length, std-dev, largest degree: a lone pixel past the shared tables
WITHIN = [(6_000, 5, 41, 8.0, 0.1, 1), (3_000, 19, 9, 20.0, 0.1, 0), (2_500, 7, 33, 9.0, 0.2, 2)]
BEYOND = (30_000, 5, 12, 8.0, 0.3, 0)  # and past the long ones


@pytest.mark.parametrize("K,leaf", [(8, 0), (4, 0), (1, 0), (9, 0), (16, 0), (17, 0), (40, 0), (64, 0), (8, 20)])
@pytest.mark.parametrize("which", range(len(WITHIN)))
def test_indices_match_oracle(smp, which, K, leaf):
    N, W, H, f, sd, degree = WITHIN[which]
    pts, nrm, s, h, tree = case(*WITHIN[which])
    opened, met = table_sizes(tree, W, H)
    assert (opened > SHORT[0] or met > SHORT[1]) and opened <= LONG
    ref = tree.sample(W, H, K, PRECISION, seed=31, leaf_size=leaf)
    assert (ref >= 0).any()
    for tile in (4, 8):
        for spread in (0, 1):
            got = smp.sample(W, H, f, T(pts[None]), T(nrm[None]), None, T(s[None]), K, 0.0, PRECISION, seed=31,
                             h=T([h]), max_degree=degree, leaf_size=leaf, tile_x=tile, spread=spread)
            np.testing.assert_array_equal(got.cpu().numpy()[0], ref)


@pytest.mark.parametrize("K", [8, 17])
def test_past_the_long_tables(smp, K):
    N, W, H, f, sd, degree = BEYOND
    pts, nrm, s, h, tree = case(*BEYOND)
    assert table_sizes(tree, W, H)[0] > LONG
    ref = tree.sample(W, H, K, PRECISION, seed=32)
    got = smp.sample(W, H, f, T(pts[None]), T(nrm[None]), None, T(s[None]), K, 0.0, PRECISION, seed=32, h=T([h]),
                     max_degree=degree)
    np.testing.assert_array_equal(got.cpu().numpy()[0], ref)
    ri, rp = tree.sample_stochastic(W, H, K, PRECISION, seed=33)
    gi, gp = smp.sample_stochastic(W, H, f, T(pts[None]), T(nrm[None]), T(s[None]), K, 0.0, PRECISION, seed=33,
                                   h=T([h]), max_degree=degree)
    np.testing.assert_array_equal(gi.cpu().numpy()[0], ri)
    np.testing.assert_array_equal(gp.cpu().numpy()[0], rp)


@pytest.mark.parametrize("which", range(len(WITHIN)))
def test_stochastic_matches_oracle(smp, which):
    N, W, H, f, sd, degree = WITHIN[which]
    pts, nrm, s, h, tree = case(*WITHIN[which])
    ri, rp = tree.sample_stochastic(W, H, 5, PRECISION, seed=34)
    gi, gp = smp.sample_stochastic(W, H, f, T(pts[None]), T(nrm[None]), T(s[None]), 5, 0.0, PRECISION, seed=34,
                                   h=T([h]), max_degree=degree)
    np.testing.assert_array_equal(gi.cpu().numpy()[0], ri)
    np.testing.assert_array_equal(gp.cpu().numpy()[0], rp)


@pytest.mark.parametrize("K", [3, 8, 12])
def test_batches_of_views(smp, K):
    """Several views of one size and of different sizes: each view's tiles go
    to the long tables with its own tree, seed counters and output."""
    N, W, H, f, sd, degree = WITHIN[0]
    pts, nrm, s, h, tree = case(*WITHIN[0])
    few = cloud(7, N, W, H, f, sd)[0].copy()
    few[200:, 2] = 1.0  # behind the camera
    P = T(np.stack([few, pts, pts]))
    args = (P, T(np.stack([nrm] * 3)), None, T(s[None]), K, 0.0, PRECISION)
    got = smp.sample(W, H, f, *args, seed=35, h=T([h] * 3), max_degree=degree).cpu().numpy()
    for v in (1, 2):
        np.testing.assert_array_equal(got[v], tree.sample(W, H, K, PRECISION, seed=35, view=v))
    views = [(W, H, f), (W, H, f), (W + 4, H - 9, f)]
    got = smp.sample_views(views, *args, seed=35, h=T([h] * 3), max_degree=degree)
    np.testing.assert_array_equal(got[1].cpu().numpy()[0], tree.sample(W, H, K, PRECISION, seed=35, view=1))
    other = oracle.Tree(W + 4, H - 9, f, pts, h, oracle.cull_radius(h, PRECISION), PRECISION, max_degree=degree)
    np.testing.assert_array_equal(got[2].cpu().numpy()[0],
                                  other.sample(W + 4, H - 9, K, PRECISION, seed=35, view=2))


def test_descent_entry_point_repeated(smp):
    """The list of tiles is empty again after each descent of one tree."""
    from unbiased_differentiable_splatting_gb300 import _lib
    N, W, H, f, sd, degree = WITHIN[0]
    pts, nrm, s, h, tree = case(*WITHIN[0])
    built = smp.build_tree(W, H, f, T(pts[None]), T(nrm[None]), T(s[None]), 8, 0.0, PRECISION, h=T([h]),
                           max_degree=degree)
    prm, ws = built["_prm"], built["_ws"]
    for seed in (1, 2, 3):
        prm.seed = seed
        out = torch.full((W, H, 8), -1, dtype=torch.int32, device=DEV)
        _lib.check(_lib.load().uds_sample_descent(prm, 0, None, out.data_ptr(), ws.data_ptr(), ws.numel(),
                                                  _lib.stream_ptr(out.device)), "descent")
        np.testing.assert_array_equal(out.cpu().numpy(), tree.sample(W, H, 8, PRECISION, seed=seed))


def test_proposal_draws(smp):
    """Every pixel with a mass gets its draws, also in tiles left for the long
    tables, and the weights' mean is 1: mean over S draws of a weight with
    variance v has a standard error of sqrt(v / S), and five of them are
    allowed."""
    from unbiased_differentiable_splatting_gb300 import proposal
    W, H, f, N = 16, 512, 20.0, 60_000
    pts, nrm, s = cloud(3, N, W, H, f, 0.1)
    h = oracle.view_bandwidth(W, H, f, pts, nrm, s, 0.0)
    tree = oracle.Tree(W, H, f, pts, h, oracle.cull_radius(h, PRECISION), PRECISION)
    opened, met = table_sizes(tree, W, H)
    assert opened > SHORT[0] or met > SHORT[1]
    net = proposal.ProposalNet(DEV, seed=2)
    idx, w, fb, nfb = proposal.sample(W, H, f, T(pts[None]), T(nrm[None]), T(s[None]), 16, 0.0, PRECISION, net=net,
                                      ess_tau=0.0, seed=5, h=T([h]))
    mass = np.array([[tree.node_weight(0, (i, j)) for j in range(H)] for i in range(W)])
    has = torch.as_tensor(mass >= PRECISION).to(DEV)
    assert bool(((idx[0] >= 0).all(-1) == has).all()) and not net.failed()
    per_pixel = w[0][has].double().mean(1)  # independent between pixels
    error = float(per_pixel.std()) / per_pixel.numel() ** 0.5
    assert abs(float(per_pixel.mean()) - 1.0) < 5 * error


def test_time_of_a_tall_image(smp):
    """300k splats at 128 x 1024 (131k pixels) against 1024 x 1024 (1M
    pixels): a tall image's pixels meet several times as many expansions, and
    a factor of 40 is allowed; with one lane at a time for pixels past the
    shared tables it was over 1000."""
    from unbiased_differentiable_splatting_gb300 import scenes

    def time(W, H):
        sc = scenes.harmonic_scene(n=300_000, sd_range=(0.003, 0.01), width=W, seed=1)
        P, Nn = scenes.camera_space(sc, DEV)
        Nn = torch.where(Nn[..., 2:] > 0, -Nn, Nn).contiguous()
        sd = sc["stddevs"].to(DEV)
        best = float("inf")
        for _ in range(3):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            smp.sample(W, H, sc["focal"], P, Nn, None, sd, 8, 0.0, PRECISION, seed=1, tile_x=8, spread=0)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    assert time(128, 1024) < 40 * time(1024, 1024)
