"""Failure detection without a GPU fault.  Every device wait in the library
is bounded: when it runs out the kernel records a status instead of hanging
and the host reads it as error 3 (timeout); the context stays usable.  Host
errors are recorded, never abort."""
import numpy as np
import pytest

from neslgpu_gb300 import ops, workloads as W


def test_host_error_is_recorded_not_fatal():
    from neslgpu_gb300.cvl import load
    c = load()
    c.gcvl_clear_error()
    assert c.alo_foz(-1) is None          # negative size (or no device): NULL, no abort
    assert c.gcvl_last_error() != 0
    assert c.gcvl_error_string()
    c.gcvl_clear_error()
    assert c.gcvl_last_error() == 0


@pytest.mark.gpu
def test_wait_that_nothing_releases_times_out(gpu):
    c = gpu.cvl
    c.gcvl_clear_error()
    assert c.gcvl_selftest_timeout(2000) == 3
    assert "bounded device wait" in c.gcvl_error_string().decode()
    c.gcvl_clear_error()
    # the context is still usable afterwards
    r = W.rng(3)
    x = W.int32_uniform(r, 10_000)
    lens = W.geometric_lengths(r, 10_000, 30)
    from oracle.oracle import HostRunner, load_oracle
    assert np.array_equal(ops.scan_e(gpu, "add_sez", x, lens),
                          ops.scan_e(HostRunner(load_oracle()), "add_sez", x, lens))


@pytest.mark.gpu
def test_injected_spin_limit_never_hangs(gpu):
    """With the wait limit forced to 1, look-back waits on tiles that have not
    published yet give up at once: the call finishes (correct or flagged),
    and after restoring the limit results are right again."""
    c = gpu.cvl
    old = c.gcvl_get_spin_limit()
    r = W.rng(4)
    n = 1 << 22
    x = W.float64_normal(r, n)
    one = np.array([n], dtype=np.int32)
    from cases import compare, seg_abs_prefix
    from oracle.oracle import HostRunner, load_oracle
    want = ops.scan_e(HostRunner(load_oracle()), "add_sed", x, one)
    S = seg_abs_prefix(x, one)
    try:
        c.gcvl_set_spin_limit(1)
        R = ops.DeviceRunner(c, checked=False)
        flagged = ops.scan_e(R, "add_sed", x, one)
        code = c.gcvl_sync()
        assert code in (0, 3)
        if code == 0:  # no wait ran out: the result must be right
            compare("sum", flagged, want, S)
        else:
            assert "bounded device wait" in c.gcvl_error_string().decode()
    finally:
        c.gcvl_set_spin_limit(old)
        c.gcvl_clear_error()
    compare("sum", ops.scan_e(gpu, "add_sed", x, one), want, S)


def _rank_case(r, name, n):
    """Keys and, for a segmented rank, lengths among which are some that the digit passes take."""
    x = W.float64_normal(r, n) if name[-1] == "d" else W.int32_uniform(r, n)
    if name[5] == "u":
        return x, None
    return x, np.array([5, n // 2, 0, 1, n - n // 2 - 6], dtype=np.int32)


def _rank(R, name, x, lens):
    return ops.rank_u(R, name, x) if lens is None else ops.rank_e(R, name, x, lens)


# sizes of the digit passes' three tile sizes; past 2^23 the ranks go through windows
@pytest.mark.gpu
@pytest.mark.parametrize("n", [200_003, 1_000_003, (1 << 23) + 5])
@pytest.mark.parametrize("name", ["rku_luz", "rkd_lud", "rkd_lez", "rku_led"])
def test_ranks_whose_waits_run_out(gpu, oracle, name, n):
    """With the wait limit forced to 1 the digit passes' look-back and meetings give up: the ranks are right, or
    flagged and then nothing is written past their vector; the next call is right again."""
    c = gpu.cvl
    x, lens = _rank_case(W.rng(n), name, n)
    want = _rank(oracle, name, x, lens)
    old = c.gcvl_get_spin_limit()
    k, d = gpu.vec(x, name[-1]), gpu.vec(np.full(n + 4096, -1, dtype=np.int32), "z")
    sd, sizes = (None, (n,)) if lens is None else (gpu.segd(lens)[0], (n, lens.size))
    scr = gpu.units(gpu.fn(name + "_scratch")(*sizes))
    assert c.gcvl_sync() == 0
    try:
        c.gcvl_set_spin_limit(1)
        gpu.fn(name)(d.ptr, k.ptr, *([sd.ptr] if sd else []), *sizes, scr.ptr)
        code = c.gcvl_sync()
        got = d.numpy(n + 4096)
        assert code in (0, 3)
        assert np.all(got[n:] == -1)
        if code == 0:
            assert np.array_equal(got[:n], want)
    finally:
        c.gcvl_set_spin_limit(old)
        c.gcvl_clear_error()
    assert np.array_equal(_rank(gpu, name, x, lens), want)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [300_000, (1 << 23) + 5])
@pytest.mark.parametrize("name", ["rku_lez", "rkd_led", "rku_luz"])
def test_ranks_after_an_earlier_call_gave_up(gpu, oracle, name, n):
    """A wait that gave up stays noted until gcvl_sync; the calls before that are carried out all the same."""
    c = gpu.cvl
    old = c.gcvl_get_spin_limit()
    r = W.rng(n + 1)
    y = W.float64_normal(r, 1 << 22)
    x, lens = _rank_case(r, name, n)
    R = ops.DeviceRunner(c, checked=False)
    try:
        c.gcvl_set_spin_limit(1)
        ops.scan_e(R, "add_sed", y, np.array([y.size], dtype=np.int32))
        c.gcvl_set_spin_limit(old)
        got = _rank(R, name, x, lens)
        assert c.gcvl_sync() in (0, 3)
    finally:
        c.gcvl_set_spin_limit(old)
        c.gcvl_clear_error()
    assert np.array_equal(got, _rank(oracle, name, x, lens))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [(1 << 23) + 5, (1 << 25) + 3])
@pytest.mark.parametrize("name", ["smp_puz", "bck_puz", "smp_pud", "bck_pud"])
def test_random_permutes_whose_waits_run_out(gpu, name, n):
    """With the wait limit forced to 1 the scan of the window split's counts may give up: the result is right, or
    flagged and then nothing is written past its vector; the next call is right again."""
    c = gpu.cvl
    r = W.rng(n)
    x = W.float64_normal(r, n) if name[-1] == "d" else W.int32_uniform(r, n)
    perm = r.permutation(n).astype(np.int32)
    want = np.empty_like(x)
    if name[0] == "s":
        want[perm] = x
    else:
        want = x[perm]
    sizes = (n,) if name[0] == "s" else (n, n)
    guard = x[:4096]
    s, p, d = gpu.vec(x, name[-1]), gpu.vec(perm, "z"), gpu.vec(np.concatenate([x, guard]), name[-1])
    scr = gpu.units(gpu.fn(name + "_scratch")(*sizes))
    old = c.gcvl_get_spin_limit()
    assert c.gcvl_sync() == 0
    try:
        for limit in (1, old):
            c.gcvl_set_spin_limit(limit)
            gpu.fn(name)(d.ptr, s.ptr, p.ptr, *sizes, scr.ptr)
            code = c.gcvl_sync()
            got = d.numpy(n + guard.size)
            assert code in ((0, 3) if limit == 1 else (0,))
            assert np.array_equal(got[n:], guard)
            if code == 0:
                assert np.array_equal(got[:n], want)
            c.gcvl_clear_error()
    finally:
        c.gcvl_set_spin_limit(old)
        c.gcvl_clear_error()


@pytest.mark.gpu
@pytest.mark.parametrize("n,m", [(1 << 20, 300_001), (1 << 25, (1 << 22) + 3), (3_000_000, 1 << 20)])
def test_descriptors_whose_waits_run_out(gpu, oracle, n, m):
    """With the wait limit forced to 1 the scan of the lengths gives up and leaves offsets that do not ascend: nothing
    is written past the descriptor, and the next call is right again.  Lengths apart and in place."""
    c = gpu.cvl
    r = W.rng(m)
    lens = np.diff(np.concatenate([[0], np.sort(r.integers(0, n + 1, size=m - 1)), [n]])).astype(np.int32)
    units, guard = c.siz_fos(n, m), np.arange(4096, dtype=np.int32)
    old = c.gcvl_get_spin_limit()
    scr = gpu.units(c.mke_fov_scratch(n, m))
    x = W.int32_uniform(r, n)
    want = ops.reduce_e(oracle, "max_rez", x, lens)
    xv, y = gpu.vec(x, "z"), gpu.out(m, "z")
    rscr = gpu.units(gpu.fn("max_rez_scratch")(n, m))
    for in_place in (False, True):
        sd = gpu.vec(np.zeros(2 * units + guard.size, dtype=np.int32), "z")
        lv = gpu.vec(lens, "z")
        tail = c.add_fov(sd.ptr, units)
        try:
            for limit in (1, old):
                c.c2v_fuz(tail, guard.ctypes.data, guard.size, None)
                if in_place:
                    c.c2v_fuz(sd.ptr, lens.ctypes.data, m, None)
                assert c.gcvl_sync() == 0
                c.gcvl_set_spin_limit(limit)
                c.mke_fov(sd.ptr, sd.ptr if in_place else lv.ptr, n, m, scr.ptr)
                code = c.gcvl_sync()
                assert code in ((0, 3) if limit == 1 else (0,))
                c.gcvl_clear_error()
                got = np.empty(guard.size, dtype=np.int32)
                c.v2c_fuz(got.ctypes.data, tail, guard.size, None)
                assert np.array_equal(got, guard)
        finally:
            c.gcvl_set_spin_limit(old)
            c.gcvl_clear_error()
        gpu.fn("max_rez")(y.ptr, xv.ptr, sd.ptr, n, m, rscr.ptr)
        assert np.array_equal(gpu.get(y, m), want)


@pytest.mark.gpu
def test_float_min_max_whose_waits_run_out(gpu, oracle):
    """With the wait limit forced to 1 the look-back of a short reduction may give up: right or flagged, nothing past
    the results, and the next call is right."""
    c = gpu.cvl
    r = W.rng(9)
    n = 200_000
    lens = np.array([n - 40_000, 30_000, 0, 10_000], dtype=np.int32)
    x = W.float64_normal(r, n)
    want = ops.reduce_e(oracle, "max_red", x, lens)
    sd, _, m = gpu.segd(lens)
    xv, d = gpu.vec(x, "d"), gpu.vec(np.full(m + 512, 7.5), "d")
    scr = gpu.units(gpu.fn("max_red_scratch")(n, m))
    old = c.gcvl_get_spin_limit()
    assert c.gcvl_sync() == 0
    try:
        for limit in (1, old):
            c.gcvl_set_spin_limit(limit)
            gpu.fn("max_red")(d.ptr, xv.ptr, sd.ptr, n, m, scr.ptr)
            code = c.gcvl_sync()
            assert code in ((0, 3) if limit == 1 else (0,))
            got = d.numpy(m + 512)
            assert np.all(got[m:] == 7.5)
            if code == 0:
                assert np.array_equal(got[:m], want)
            c.gcvl_clear_error()
    finally:
        c.gcvl_set_spin_limit(old)
        c.gcvl_clear_error()
