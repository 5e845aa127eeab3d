"""Kernels at the sizes where a branch of their dispatch or an edge of their
tiles could go wrong, against the oracle.  Whole numbers and moved values are
compared bit for bit."""
import math

import numpy as np
import pytest

from neslgpu_gb300 import ops, workloads as W

pytestmark = pytest.mark.gpu


def _group(gpu):
    """Draws that one pass of RAND's largest grid makes (16 CTAs of 1024 draws per SM)."""
    return gpu.cvl.gcvl_sm_count() * 16 * 1024


@pytest.mark.parametrize("n", [1, 255, 256, 257, 1023, 1024, 1025, "g-1", "g", "g+1", "2g+777"])
def test_rand_group_edges(gpu, oracle, n):
    if isinstance(n, str):
        n = {"g-1": _group(gpu) - 1, "g": _group(gpu), "g+1": _group(gpu) + 1, "2g+777": 2 * _group(gpu) + 777}[n]
    r = W.rng(n % 9973)
    bounds = r.integers(1, 2 ** 31, size=n, dtype=np.int64).astype(np.int32)
    assert np.array_equal(ops.rand_u(gpu, bounds, seed=n + 5), ops.rand_u(oracle, bounds, seed=n + 5))


# ----------------------------------------------------------------- ranks ---
# sizes of neslgpu_gb300/csrc/rank.cuh and rank.cu: a CTA's segments start in
# 2048 elements and hold at most 2048; one CTA ranks a whole vector of 4096;
# digit passes take smaller tiles up to 2^18 and up to 2^20 and write ranks by window past 2^23
LR_T = LR_MAX = 2048


def _keys(r, n, typ, dist):
    if dist == "few":
        x = r.integers(0, 5, size=n)
    elif dist == "equal":
        x = np.full(n, -7)
    elif dist == "clusters":  # two narrow ranges far apart: crowded buckets
        x = np.where(r.random(n) < 0.5, r.integers(-40, 40, size=n), 2 ** 31 - 1 - r.integers(0, 900, size=n))
    else:
        x = W.int32_uniform(r, n) if typ == "z" else W.float64_normal(r, n)
    x = np.asarray(x, dtype=np.float64 if typ == "d" else np.int32)
    if typ == "d" and dist == "special":
        x[r.random(n) < 0.2] = np.inf
        x[r.random(n) < 0.2] = -np.inf
        x[r.random(n) < 0.1] = 0.0
        x[r.random(n) < 0.1] = -0.0
        x[r.random(n) < 0.1] *= 2.0 ** -1030
    return x


def _segments(r, shape):
    if shape == "ones":
        return np.ones(LR_T * 2 + 5, dtype=np.int32)
    if shape == "limit":  # around the longest segment one CTA takes, at every place in a tile
        return np.array([2047, 1, 2048, 3, 2049, 0, 2048, 2048, 1, 4097, 2049, 0, 5, 2046], dtype=np.int32)
    if shape == "long":  # long segments over several tiles among short ones
        s = W.geometric_lengths(r, 60_000, 20)
        return np.insert(s, [3, 3, 900, len(s)], [30_001, 2049, 70_000, 9_000]).astype(np.int32)
    if shape == "empties":
        return W.with_empty(r, W.geometric_lengths(r, 50_001, 300), 0.3)
    if shape == "whole":
        return W.with_empty(r, W.geometric_lengths(r, 4096, 64), 0.2)
    return W.lognormal_lengths(r, 400_003, 5, 2, 1 << 18)


@pytest.mark.parametrize("shape", ["ones", "limit", "long", "empties", "whole", "lognormal"])
@pytest.mark.parametrize("dist", ["uniform", "few", "equal", "clusters", "special"])
@pytest.mark.parametrize("name", ["rku_lez", "rkd_lez", "rku_led", "rkd_led"])
def test_rank_segments(gpu, oracle, name, dist, shape):
    r = W.rng(sum(map(ord, name + dist + shape)))
    lens = _segments(r, shape)
    x = _keys(r, int(lens.sum()), name[-1], dist)
    assert np.array_equal(ops.rank_e(gpu, name, x, lens), ops.rank_e(oracle, name, x, lens))


@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, 257, 2047, 2049, 4095, 4096, 4097, 1 << 18, (1 << 18) + 1, 1 << 20, (1 << 20) + 1])
@pytest.mark.parametrize("name,dist", [("rku_luz", "uniform"), ("rkd_luz", "few"), ("rku_lud", "special"),
                                       ("rkd_lud", "uniform"), ("rku_luz", "clusters")])
def test_rank_whole_vectors(gpu, oracle, name, dist, n):
    x = _keys(W.rng(n + len(dist)), n, name[-1], dist)
    assert np.array_equal(ops.rank_u(gpu, name, x), ops.rank_u(oracle, name, x))


@pytest.mark.parametrize("name,n", [("rku_lez", (1 << 23) + 1), ("rkd_led", (1 << 23) + 12_345)])
def test_rank_long_segments_by_window(gpu, oracle, name, n):
    """Past 2^23 elements the long segments' ranks go through windows of the index that they fill only in part."""
    r = W.rng(n)
    lens = W.bimodal_lengths(r, n)
    x = _keys(r, n, name[-1], "uniform")
    assert np.array_equal(ops.rank_e(gpu, name, x, lens), ops.rank_e(oracle, name, x, lens))


@pytest.mark.parametrize("n", [4097, 1 << 18, (1 << 18) + 1, 1 << 20, (1 << 20) + 1])
@pytest.mark.parametrize("name", ["rkd_lez", "rku_led"])
def test_rank_long_segments_captured(gpu, oracle, name, n):
    """The passes over the long segments inside a CUDA graph, replayed on other keys, in each of their tile sizes
    (one launch that meets between passes); then the same call outside it."""
    r = W.rng(n + 3)
    lens = np.array([2049, 0, 7, n - 2056], dtype=np.int32)
    if n == 4097:
        lens = np.array([2048, 2049], dtype=np.int32)
    c, t = gpu.cvl, name[-1]
    x = [_keys(r, n, t, "uniform"), _keys(r, n, t, "few")]
    sd, _, m = gpu.segd(lens)
    k, d = gpu.vec(x[0], t), gpu.out(n, "z")
    scr = gpu.units(gpu.fn(name + "_scratch")(n, m))
    assert c.gcvl_graph_begin() == 0
    gpu.fn(name)(d.ptr, k.ptr, sd.ptr, n, m, scr.ptr)
    g = c.gcvl_graph_end()
    for keys in x:
        k.upload(keys)
        c.gcvl_graph_launch(g)
        assert np.array_equal(gpu.get(d, n), ops.rank_e(oracle, name, keys, lens))
    c.gcvl_graph_destroy(g)
    assert np.array_equal(ops.rank_e(gpu, name, x[0], lens), ops.rank_e(oracle, name, x[0], lens))
    assert c.gcvl_sync() == 0


# ------------------------------------------------------------------ puts ---
# the owner passes take 2048 elements a CTA, up to 3 * 2^24 destinations
def _put_case(r, n_s, n_d, order):
    if order == "ascending":
        return np.sort(r.permutation(n_d)[:n_s]).astype(np.int32)
    if order == "one":
        return np.full(n_s, n_d - 1, dtype=np.int32)
    return r.integers(0, n_d, size=n_s).astype(np.int32)


@pytest.mark.parametrize("n_s,n_d", [(1, 1), (5, 3), (2047, 2049), (2048, 2048), (2049, 6000), (3, 100_001)])
@pytest.mark.parametrize("order", ["ascending", "one", "random"])
@pytest.mark.parametrize("t", "zbd")
def test_put_by_owner(gpu, oracle, t, order, n_s, n_d):
    r = W.rng(n_s * 7 + n_d + ord(t))
    if order == "ascending" and n_s > n_d:
        pytest.skip("more values than places")
    idx = _put_case(r, n_s, n_d, order)
    x = _keys(r, n_s, t, "few" if t == "b" else "uniform")
    v = _keys(r, n_d, t, "few" if t == "b" else "uniform")
    flags = (r.random(n_s) < 0.6).astype(np.int32)
    for R in (gpu, oracle):
        R.got = [ops.dpe_u(R, f"dpe_pu{t}", x, idx, v), ops.fpm_u(R, f"fpm_pu{t}", x, idx, flags, n_d, v),
                 ops.fpm_u(R, f"dfp_pu{t}", x, idx, flags, n_d, v)]
    for a, b in zip(gpu.got, oracle.got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("t", "zd")
def test_put_default_in_place(gpu, oracle, t):
    """The destination may be the default itself."""
    r = W.rng(77)
    n_s, n_d = 3001, 9999
    idx, x, v = _put_case(r, n_s, n_d, "random"), _keys(r, n_s, t, "uniform"), _keys(r, n_d, t, "uniform")
    c = gpu.cvl
    d, s, i = gpu.vec(v, t), gpu.vec(x, t), gpu.vec(idx, "z")
    scr = gpu.units(gpu.fn(f"dpe_pu{t}_scratch")(n_s, n_d))
    gpu.fn(f"dpe_pu{t}")(d.ptr, s.ptr, i.ptr, d.ptr, n_s, n_d, scr.ptr)
    assert np.array_equal(gpu.get(d, n_d), ops.dpe_u(oracle, f"dpe_pu{t}", x, idx, v))
    assert c.gcvl_sync() == 0


@pytest.mark.parametrize("t", "zd")
def test_put_segments(gpu, oracle, t):
    r = W.rng(78)
    len_s = W.with_empty(r, W.geometric_lengths(r, 20_011, 9), 0.2)
    len_d = (len_s * 2 + r.integers(0, 3, size=len_s.size)).astype(np.int32)
    len_d[len_s > 0] += 1
    idx = W.seg_indices(r, len_d, len_s)
    x, v = _keys(r, int(len_s.sum()), t, "uniform"), _keys(r, int(len_d.sum()), t, "uniform")
    flags = (r.random(x.size) < 0.6).astype(np.int32)
    for R in (gpu, oracle):
        R.got = [ops.dpe_e(R, f"dpe_pe{t}", x, idx, v, len_s, len_d),
                 ops.fpm_e(R, f"fpm_pe{t}", x, idx, flags, len_s, len_d, v),
                 ops.fpm_e(R, f"dfp_pe{t}", x, idx, flags, len_s, len_d, v)]
    for a, b in zip(gpu.got, oracle.got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n_d", [3 << 24, (3 << 24) + 1])
def test_put_either_side_of_the_owner_limit(gpu, oracle, n_d):
    r = W.rng(n_d)
    idx = r.integers(0, n_d, size=100_003).astype(np.int32)
    x, v = _keys(r, idx.size, "z", "uniform"), np.arange(n_d, dtype=np.int32)
    assert np.array_equal(ops.dpe_u(gpu, "dpe_puz", x, idx, v), ops.dpe_u(oracle, "dpe_puz", x, idx, v))


# ----------------------------------- one-launch forms of scans and friends ---
# one tile: 4096 ints, 2048 doubles; segment descriptors: ranges of 8192
# elements, 4096 lengths scanned in the CTA; packs: tiles of 4096, 1024 summed
def _lens(r, n, shape):
    if shape == "one-element":
        return np.ones(n, dtype=np.int32)
    if shape == "long":
        return np.array([0, n - n // 3, 0, 0, n // 3, 0], dtype=np.int32)
    if shape in ("fours", "fives"):  # either side of the mean from which warps reduce ranges of their own
        k = 4 if shape == "fours" else 5
        return np.array([k] * (n // k) + [n % k] * (n % k > 0), dtype=np.int32)
    return W.with_empty(r, W.geometric_lengths(r, n, 37), 0.3)


@pytest.mark.parametrize("n", [1, 63, 64, 65, 2047, 2048, 2049, 2559, 2561, 4095, 4096, 4097, 8191, 8192, 8193, 300_007])
@pytest.mark.parametrize("shape", ["one-element", "fours", "fives", "long", "geometric"])
def test_segmented_at_tile_edges(gpu, oracle, shape, n):
    r = W.rng(n * 3 + len(shape))
    lens = _lens(r, n, shape)
    assert int(lens.sum()) == n
    xi, xb = W.int32_uniform(r, n), (r.random(n) < 0.4).astype(np.int32)
    xd = W.float64_normal(r, n)
    for R in (gpu, oracle):
        R.got = [ops.scan_e(R, "add_sez", xi, lens), ops.scan_e(R, "max_sed", xd, lens), ops.scan_e(R, "xor_seb", xb, lens),
                 ops.reduce_e(R, "max_rez", xi, lens), ops.reduce_e(R, "min_red", xd, lens),
                 ops.reduce_e(R, "ior_reb", xb, lens), ops.pk1_e(R, xb, lens), *ops.pack_e(R, "pk2_lez", xi, xb, lens),
                 *ops.pack_e(R, "pk2_led", xd, xb, lens), ops.dis_e(R, "dis_vez", np.arange(lens.size), lens)]
    for k, (a, b) in enumerate(zip(gpu.got, oracle.got)):
        assert np.array_equal(a, b), k
    # sums within 1e-12 of the magnitudes summed, as for every float64 sum
    start = np.cumsum(lens) - lens
    c = np.concatenate([[0.0], np.cumsum(np.abs(xd))])
    mag = c[start + lens] - c[start]
    g, o = ops.reduce_e(gpu, "add_red", xd, lens), ops.reduce_e(oracle, "add_red", xd, lens)
    assert np.all(np.abs(g - o) <= 1e-12 * mag)
    g, o = ops.scan_e(gpu, "add_sed", xd, lens), ops.scan_e(oracle, "add_sed", xd, lens)
    assert np.all(np.abs(g - o) <= 1e-12 * np.repeat(mag, lens))


@pytest.mark.parametrize("m,n", [(4096, 5000), (4097, 5000), (4096, 2 ** 22 + 17), (3, 8192 * 304), (3, 8192 * 304 + 1),
                                 (1, 8192), (5, 0)])
def test_segment_descriptor_forms(gpu, oracle, m, n):
    """Either side of the lengths and the elements that the one-launch form takes."""
    r = W.rng(m + n)
    cut = np.sort(r.integers(0, n + 1, size=m - 1))
    lens = np.diff(np.concatenate([[0], cut, [n]])).astype(np.int32)
    x = W.int32_uniform(r, n)
    for R in (gpu, oracle):
        R.got = [ops.scan_e(R, "add_sez", x, lens), ops.reduce_e(R, "max_rez", x, lens),
                 ops.dis_e(R, "dis_vez", np.arange(m), lens)]
    for a, b in zip(gpu.got, oracle.got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n", [1, 511, 512, 513, 8191, 8192, 8193, 4096 * 1024, 4096 * 1024 + 1])
def test_reduce_and_pack_edges(gpu, oracle, n):
    r = W.rng(n)
    x, f = W.int32_uniform(r, n), (r.random(n) < 0.5).astype(np.int32)
    for name in ("add_ruz", "min_ruz", "xor_ruz"):
        assert ops.reduce_u(gpu, name, x) == ops.reduce_u(oracle, name, x)
    assert ops.pk1_u(gpu, f) == ops.pk1_u(oracle, f)
    assert np.array_equal(ops.pack_u(gpu, "pk2_luz", x, f), ops.pack_u(oracle, "pk2_luz", x, f))


@pytest.mark.parametrize("ranges", [1, 2, 1024, 1025, 2049])
def test_reduction_fix_up_by_one_cta_or_several(gpu, oracle, ranges):
    """One segment over every tile but the ends: each tile's result needs the tiles before it."""
    n = ranges * 2048 + 3
    lens = np.array([2, n - 3, 1], dtype=np.int32)
    x = W.rng(ranges).integers(-9, 10, size=n).astype(np.float64)  # sums exact in any order
    for name in ("add_red", "max_red"):
        assert np.array_equal(ops.reduce_e(gpu, name, x, lens), ops.reduce_e(oracle, name, x, lens))
    assert np.array_equal(ops.reduce_e(gpu, "add_rez", x, lens), ops.reduce_e(oracle, "add_rez", x, lens))


@pytest.mark.parametrize("ones", [0, 1_000_000, 1_999_999])
def test_reductions_of_nearly_one_element_segments(gpu, oracle, ones):
    """Results put together in shared memory: one-element segments, some empty, one long at the end."""
    r = W.rng(ones)
    lens = np.concatenate([np.ones(ones, dtype=np.int32), r.integers(0, 3, size=2_000_000 - ones).astype(np.int32),
                           np.array([5000, 0, 1], dtype=np.int32)])
    n = int(lens.sum())
    xi, xd = W.int32_uniform(r, n), r.integers(-9, 10, size=n).astype(np.float64)  # sums exact in any order
    for name, x in (("max_rez", xi), ("add_rez", xi), ("add_red", xd), ("max_red", xd)):
        assert np.array_equal(ops.reduce_e(gpu, name, x, lens), ops.reduce_e(oracle, name, x, lens)), name


@pytest.mark.parametrize("n", [1, 31, 191, 192, 193, 767, 768, 769, 20_003])
@pytest.mark.parametrize("shape", ["one-element", "long", "geometric"])
@pytest.mark.parametrize("t", "zbd")
def test_segmented_permutes_at_warp_edges(gpu, oracle, t, shape, n):
    """A warp takes 192 elements (32 lanes of 6), a CTA 768."""
    r = W.rng(n + ord(t))
    lens = _lens(r, n, shape)
    x = _keys(r, n, t, "few" if t == "b" else "uniform")
    perm = W.seg_permutation(r, lens)
    len_s = (lens + r.integers(0, 4, size=lens.size)).astype(np.int32)  # as many source segments
    xs = _keys(r, int(len_s.sum()), t, "few" if t == "b" else "uniform")
    idx = W.seg_indices(r, len_s, lens)
    v, ii = _keys(r, lens.size, t, "few" if t == "b" else "uniform"), W.int32_uniform(r, lens.size)
    for R in (gpu, oracle):
        R.got = [ops.smp_e(R, f"smp_pe{t}", x, perm, lens), ops.bck_e(R, f"bck_pe{t}", xs, idx, len_s, lens),
                 ops.dis_e(R, f"dis_ve{t}", v, lens), ops.ind_e(R, ii, ii[::-1].copy(), lens)]
    for a, b in zip(gpu.got, oracle.got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("name,n", [("add_sez", 1 << 22), ("add_sez", (1 << 22) + 1), ("max_sed", 1 << 22),
                                    ("max_sed", (1 << 22) + 1), ("add_suz", 1 << 21), ("add_suz", (1 << 21) + 1),
                                    ("min_sud", (1 << 21) + 1)])
def test_scans_either_side_of_the_ring(gpu, oracle, name, n):
    r = W.rng(n)
    x = _keys(r, n, name[-1], "uniform")
    if name[5] == "u":
        assert np.array_equal(ops.scan_u(gpu, name, x), ops.scan_u(oracle, name, x))
    else:
        lens = W.with_empty(r, W.lognormal_lengths(r, n, 5, 2, 1 << 20), 0.1)
        assert np.array_equal(ops.scan_e(gpu, name, x, lens), ops.scan_e(oracle, name, x, lens))


@pytest.mark.parametrize("n", [1 << 19, (1 << 19) + 1])
@pytest.mark.parametrize("name", ["add_sed", "add_sud"])
def test_float_sums_either_side_of_the_ring(gpu, oracle, name, n):
    """Within 1e-12 of the magnitudes summed, as for every float64 sum."""
    r = W.rng(n + 5)
    x = W.float64_normal(r, n) * 2.0 ** r.integers(-40, 40, size=n)
    lens = W.lognormal_lengths(r, n, 5, 2, 1 << 18) if name == "add_sed" else np.array([n], dtype=np.int32)
    c = np.concatenate([[0.0], np.cumsum(np.abs(x))])
    mag = c[np.arange(n)] - np.repeat(c[np.cumsum(lens) - lens], lens)
    if name == "add_sed":
        g, o = ops.scan_e(gpu, name, x, lens), ops.scan_e(oracle, name, x, lens)
    else:
        g, o = ops.scan_u(gpu, name, x), ops.scan_u(oracle, name, x)
    assert np.all(np.abs(g - o) <= 1e-12 * np.maximum(mag, np.abs(o)))


@pytest.mark.parametrize("mean", [1, 2, 15, 16, 17, 349, 350, 351])
def test_float_sums_of_even_segments(gpu, oracle, mean):
    """Either side of the mean from which the sums fold in fixed point; rows hold 16 elements, tiles 2048."""
    r = W.rng(mean)
    m = 700_003 // mean
    lens = np.full(m, mean, dtype=np.int32)
    x = W.float64_normal(r, m * mean) * 2.0 ** r.integers(-40, 40, size=m * mean)
    mag = np.add.reduceat(np.abs(x), np.arange(m) * mean)
    g, o = ops.reduce_e(gpu, "add_red", x, lens), ops.reduce_e(oracle, "add_red", x, lens)
    assert np.all(np.abs(g - o) <= 1e-12 * mag)


@pytest.mark.parametrize("where", ["spread", "one place", "end", "start"])
@pytest.mark.parametrize("n,m", [(1, 5000), (63, 8193), (4097, 8193), (4097, 8194), (4097, 8195), (8192 * 3 + 5, 40_000),
                                 (50_000, 99_999), (50_000, 100_000), (50_000, 300_000), (3_000_001, 1_200_000)])
def test_descriptors_of_mostly_empty_segments(gpu, oracle, n, m, where):
    """Either side of two segments per element, from which every element searches its segment, and of the
    segments that a CTA walks over 8192 elements (32768, and 131072 beyond two ranges per SM)."""
    r = W.rng(n + m)
    lens = np.zeros(m, dtype=np.int32)
    if where == "spread":
        lens = np.diff(np.concatenate([[0], np.sort(r.integers(0, n + 1, size=m - 1)), [n]])).astype(np.int32)
    else:  # the elements in few segments, the others empty in one place
        k = min(n, 20)
        cut = np.diff(np.concatenate([[0], np.sort(r.choice(np.arange(1, n), size=k - 1, replace=False)), [n]])) if k > 1 else [n]
        at = {"one place": k // 2, "end": k, "start": 0}[where]
        lens[:at], lens[m - (k - at):] = cut[:at], cut[at:]
    x, v = W.int32_uniform(r, n), np.arange(m, dtype=np.int32)
    for R in (gpu, oracle):
        R.got = [ops.scan_e(R, "add_sez", x, lens), ops.reduce_e(R, "max_rez", x, lens), ops.dis_e(R, "dis_vez", v, lens)]
    for a, b in zip(gpu.got, oracle.got):
        assert np.array_equal(a, b)


def test_float_sums_keep_the_small_items_of_a_row(gpu):
    """Rows of 16 whose last item is 2^52 times the others: every sum on the way is a float64, so the results are
    exact unless items are cut off at the unit of a row's largest."""
    m, per = 3, 8 * 2048  # segments of eight tiles
    row = np.zeros(16)
    row[:8], row[15] = 2.0 ** -53, 1.0
    x = np.tile(row, m * per // 16)
    got = ops.reduce_e(gpu, "add_red", x, np.full(m, per, dtype=np.int32))
    assert np.array_equal(got, np.full(m, per // 16 * (1.0 + 2.0 ** -50)))


@pytest.mark.parametrize("n", [500, 512])
def test_float_sum_of_a_short_vector_folds_its_warps_pairwise(gpu, n):
    """The first warp's 32 elements sum to 1, each other warp's to what a running sum rounds up every time: pairwise,
    an element takes part in at most 5 + 4 inexact additions, 2^-53 each."""
    x = np.full(n, 2.0 ** -58 * (1 + 2.0 ** -7))
    x[:32] = 2.0 ** -5
    exact = math.fsum(x)
    assert abs(ops.reduce_u(gpu, "add_rud", x) - exact) <= 9 * 2.0 ** -53 * exact


def _dpe_in_place(R, name, x, idx, v, lens=None):
    """dpe_* whose destination is its own default, as the interpreter issues it when the default dies there."""
    t = name[-1]
    d, s, i = R.vec(v, t), R.vec(x, t), R.vec(idx, "z")
    if lens is None:
        sizes = a = (len(x), len(v))
    else:
        (sds, n_s, m_s), (sdd, n_d, m_d) = R.segd(lens[0]), R.segd(lens[1])
        sizes, a = (n_s, m_s, n_d, m_d), (R.p(sds), n_s, m_s, R.p(sdd), n_d, m_d)
    scr = R.units(R.fn(name + "_scratch")(*sizes))
    R.fn(name)(R.p(d), R.p(s), R.p(i), R.p(d), *a, R.p(scr))
    r = R.get(d, len(v))
    R.done()
    return r


# few values for many destinations: from 2^23 destinations and 32 of them per value on, 2^25 and 128 where the
# default is copied; owners left from other puts lie in the scratch
@pytest.mark.parametrize("n_d,n_s", [((1 << 23) - 1, 40), (1 << 23, 1), (1 << 23, 40), (1 << 23, 1 << 18), (1 << 23, (1 << 18) + 1),
                                     ((1 << 25) - 1, 1000), (1 << 25, 2049), (1 << 25, 1 << 18), (1 << 25, (1 << 18) + 1)])
@pytest.mark.parametrize("t", "zd")
def test_put_of_few_values(gpu, oracle, t, n_d, n_s):
    r = W.rng(n_d + n_s)
    v, x = _keys(r, n_d, t, "few"), _keys(r, n_s, t, "uniform")
    flags = (r.random(n_s) < 0.6).astype(np.int32)
    for idx in (r.integers(0, n_d, size=n_s), r.integers(n_d - 9, n_d, size=n_s), np.arange(n_s) * (n_d // n_s)):
        idx = idx.astype(np.int32)
        want = v.copy()  # the last value stays
        want[idx] = x
        keep = v.copy()
        keep[idx[flags != 0]] = x[flags != 0]
        assert np.array_equal(ops.dpe_u(gpu, f"dpe_pu{t}", x, idx, v), want)
        assert np.array_equal(_dpe_in_place(gpu, f"dpe_pu{t}", x, idx, v), want)
        assert np.array_equal(ops.fpm_u(gpu, f"fpm_pu{t}", x, idx, flags, n_d, v), keep)
        assert np.array_equal(ops.fpm_u(gpu, f"dfp_pu{t}", x, idx, flags, n_d, v), keep)
    assert np.array_equal(ops.dpe_u(oracle, f"dpe_pu{t}", x, idx, v), want)


@pytest.mark.parametrize("m,ratio", [(3000, 31), (3000, 33), (3000, 130), (1, 130)])
@pytest.mark.parametrize("t", "zd")
def test_put_of_few_values_by_segments(gpu, oracle, t, m, ratio):
    r = W.rng(m + ratio)
    len_s = r.multinomial((1 << 25) // ratio, np.ones(m) / m).astype(np.int32)
    len_d = (len_s * ratio + ((1 << 25) % ratio > 0)).astype(np.int32)
    len_d[-1] += max(0, (1 << 25) - int(len_d.sum()))
    idx = W.seg_indices(r, len_d, len_s)
    x, v = _keys(r, int(len_s.sum()), t, "uniform"), _keys(r, int(len_d.sum()), t, "few")
    flags = (r.random(x.size) < 0.6).astype(np.int32)
    for R in (gpu, oracle):
        R.got = [ops.dpe_e(R, f"dpe_pe{t}", x, idx, v, len_s, len_d), _dpe_in_place(R, f"dpe_pe{t}", x, idx, v, (len_s, len_d)),
                 ops.fpm_e(R, f"fpm_pe{t}", x, idx, flags, len_s, len_d, v)]
    for a, b in zip(gpu.got, oracle.got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("name,n,mean", [("add_sez", 4097, 7), ("add_sez", 4097, 8), ("xor_sez", 20_003, 7), ("min_sez", 20_003, 8),
                                         ("add_sez", 3 << 18, 8), ("add_sez", (3 << 18) + 1, 8), ("max_sed", 1 << 20, 256),
                                         ("max_sed", (1 << 20) + 1, 257), ("min_sed", 1 << 21, 255), ("min_sed", (1 << 21) + 1, 255),
                                         ("mul_sed", 3 << 19, 50), ("mul_sed", (3 << 19) + 1, 50), ("max_sud", 1 << 20, 0),
                                         ("max_sud", (1 << 20) + 1, 0), ("mul_sud", 1 << 20, 0), ("mul_sud", (1 << 20) + 1, 0)])
def test_scans_either_side_of_their_lines(gpu, oracle, name, n, mean):
    """The sizes and mean segment lengths up to which scans take a tile per CTA."""
    r = W.rng(n + mean)
    x = _keys(r, n, name[-1], "uniform")
    if name[:3] == "mul":  # products exact in any order
        x = np.where(r.random(n) < 0.5, -1.0, 1.0)
    if name[5] == "u":
        assert np.array_equal(ops.scan_u(gpu, name, x), ops.scan_u(oracle, name, x))
    else:
        lens = np.array([mean] * (n // mean) + [n % mean] * (n % mean > 0), dtype=np.int32)
        assert np.array_equal(ops.scan_e(gpu, name, x, lens), ops.scan_e(oracle, name, x, lens))


@pytest.mark.parametrize("n", [6000, 1 << 20, (1 << 24) + 1025])
@pytest.mark.parametrize("mean", [5, 6, 8, 9])
@pytest.mark.parametrize("shape", ["even", "uneven"])
def test_reductions_either_side_of_the_warp_ranges(gpu, oracle, shape, mean, n):
    """Warp ranges from 6 elements a segment on, three times as many below 9; short segments and long ones apart."""
    r = W.rng(n + mean)
    if shape == "even":
        lens = np.array([mean] * (n // mean) + [n % mean] * (n % mean > 0), dtype=np.int32)
    else:  # mean * m elements: m - 2 segments of half the mean among two long ones
        m = n // mean
        lens = np.full(m, max(1, mean // 2), dtype=np.int32)
        lens[m // 5] = lens[m // 2] = 0
        lens[m // 5] = (n - int(lens.sum())) // 2
        lens[m // 2] = n - int(lens.sum())
    x, b = W.int32_uniform(r, n), (r.random(n) < 0.4).astype(np.int32)
    for R in (gpu, oracle):
        R.got = [ops.reduce_e(R, "max_rez", x, lens), ops.reduce_e(R, "add_rez", x, lens), ops.pk1_e(R, b, lens),
                 ops.reduce_e(R, "ior_reb", b, lens)]
    for g, o in zip(gpu.got, oracle.got):
        assert np.array_equal(g, o)


@pytest.mark.parametrize("n", [4095, 4096, 4097, 8191, 8192, 8193])
def test_float_reductions_by_one_cta_or_several(gpu, oracle, n):
    x = W.rng(n).integers(-9, 10, size=n).astype(np.float64)  # sums exact in any order
    for name in ("add_rud", "max_rud", "min_rud"):
        assert ops.reduce_u(gpu, name, x) == ops.reduce_u(oracle, name, x)


@pytest.mark.parametrize("lens", [(127,), (128,), (129,), (100, 155), (100, 156), (100, 157), (5, 1111, 0, 3000)])
@pytest.mark.parametrize("form", ["add_red", "spmv"])
def test_float_sums_either_side_of_the_fold(gpu, oracle, form, lens):
    """The mean of 128 elements a segment from which warps without a segment boundary fold theirs in fixed point, for
    sums and for the fused row sums of a sparse matrix; the last has warps with and without a boundary in one tile."""
    r = W.rng(sum(lens))
    lens = np.array(lens * (600_000 // sum(lens)), dtype=np.int32)
    n, m = int(lens.sum()), lens.size
    x = W.float64_normal(r, n) * 2.0 ** r.integers(-40, 40, size=n)
    if form == "add_red":
        g = ops.reduce_e(gpu, "add_red", x, lens)
    else:
        c = gpu.cvl
        w = W.float64_normal(r, 5000)
        cols = r.integers(0, w.size, size=n).astype(np.int32)
        sd, _, _ = gpu.segd(lens)
        vv, cv, wv, y = gpu.vec(x, "d"), gpu.vec(cols, "z"), gpu.vec(w, "d"), gpu.out(m, "d")
        scr = gpu.units(c.gcvl_spmv_csr_scratch(n, m))
        c.gcvl_spmv_csr(y.ptr, vv.ptr, cv.ptr, wv.ptr, sd.ptr, n, m, scr.ptr)
        g = gpu.get(y, m)
        assert c.gcvl_sync() == 0
        x = x * w[cols]
    o = ops.reduce_e(oracle, "add_red", x, lens)
    e = np.cumsum(lens.astype(np.int64))
    mag = np.where(lens > 0, np.add.reduceat(np.append(np.abs(x), 0.0), np.minimum(e - lens, n - 1)), 0.0)
    assert np.all(np.abs(g - o) <= 1e-12 * mag)


@pytest.mark.parametrize("shape", ["ones", "limit", "empties", "whole", "vector"])
@pytest.mark.parametrize("name", ["rku", "rkd"])
def test_ranks_with_nans(gpu, oracle, name, shape):
    """NaNs rank by their bits, beyond the infinities of their sign; the buckets of a local rank put them at the ends."""
    r = W.rng(len(shape))
    lens = np.array([4000], dtype=np.int32) if shape == "vector" else _segments(r, shape)
    x = _keys(r, int(lens.sum()), "d", "special")
    nan = r.random(x.size) < 0.2
    bits = r.integers(1, 1 << 52, size=x.size, dtype=np.uint64) | np.uint64(0x7FF << 52)
    bits[r.random(x.size) < 0.5] |= np.uint64(1 << 63)
    x[nan] = bits.view(np.float64)[nan]
    if shape == "vector":
        assert np.array_equal(ops.rank_u(gpu, name + "_lud", x), ops.rank_u(oracle, name + "_lud", x))
    else:
        assert np.array_equal(ops.rank_e(gpu, name + "_led", x, lens), ops.rank_e(oracle, name + "_led", x, lens))


@pytest.mark.parametrize("m", [2, 255, 256, 257, 1000])
@pytest.mark.parametrize("name", ["rku_lez", "rkd_led"])
def test_ranks_of_few_long_segments(gpu, oracle, name, m):
    """The passes by segment number cover as many long segments as there are segments, not as many as would fit."""
    r = W.rng(m)
    lens = r.integers(2049, 30_000, size=m).astype(np.int32)
    lens[m // 2] = 600_000
    x = _keys(r, int(lens.sum()), name[-1], "few")
    assert np.array_equal(ops.rank_e(gpu, name, x, lens), ops.rank_e(oracle, name, x, lens))


@pytest.mark.parametrize("n,m", [(0, 1), (0, 4096), (0, 4097), (0, 100_000), (1, 5000), (8192, 20_000), (8193, 20_000), (8193, 4097),
                                 (8192 * 304 + 1, 8192 * 304 * 4 + 4), (8192 * 304, 8192 * 304 * 2)])
def test_descriptors_end_where_their_size_says(gpu, n, m):
    """Nothing is written past the units that siz_fos gives, nor past the scratch that mke_fov_scratch gives."""
    c = gpu.cvl
    lens = np.zeros(m, dtype=np.int32)
    lens[: min(n, m)] = 1
    lens[m // 2] += n - int(lens.sum())
    guard = np.full(4096, 0x5A5A5A5A, dtype=np.int32)
    room, scr_room = c.siz_fos(n, m), c.mke_fov_scratch(n, m)
    sd = gpu.vec(np.concatenate([np.zeros(2 * room, dtype=np.int32), guard]), "z")
    scr = gpu.vec(np.concatenate([np.zeros(2 * scr_room, dtype=np.int32), guard]), "z")
    lv = gpu.vec(lens, "z")
    c.mke_fov(sd.ptr, lv.ptr, n, m, scr.ptr)
    assert np.array_equal(sd.numpy(2 * room + guard.size)[2 * room:], guard)
    assert np.array_equal(scr.numpy(2 * scr_room + guard.size)[2 * scr_room:], guard)
    d = gpu.out(m, "z")
    c.len_fos(d.ptr, sd.ptr, n, m, None)
    assert np.array_equal(gpu.get(d, m), lens)
    assert c.gcvl_sync() == 0


@pytest.mark.parametrize("n", [2049, 4096, 4097, 100_003, 1 << 18, (1 << 18) + 1])
@pytest.mark.parametrize("shape", ["one-element", "long", "geometric", "across"])
@pytest.mark.parametrize("name", ["min_red", "max_red"])
def test_float_min_max_either_side_of_the_look_back(gpu, oracle, name, shape, n):
    """Up to 2^18 elements a tile takes the earlier tiles' part of its first result by look-back; vectors on and off a
    16-byte boundary."""
    r = W.rng(n + len(shape))
    lens = np.array([3, 0, n - 5, 0, 2], dtype=np.int32) if shape == "across" else _lens(r, n, shape)
    x = _keys(r, n, "d", "special")
    want = ops.reduce_e(oracle, name, x, lens)
    assert np.array_equal(ops.reduce_e(gpu, name, x, lens), want)
    assert np.array_equal(ops.reduce_e(ops.DeviceRunner(gpu.cvl, offset=1), name, x, lens), want)
