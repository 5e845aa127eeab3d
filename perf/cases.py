"""What programs have this library do, as cases that can be timed.

A case is one call sequence of the C ABI (or one VCODE program), as a caller
with its vectors on the GPU issues it: vectors and scratch are torch tensors
whose addresses are the vec_p arguments, scratch is sized by the F_scratch
functions, and nothing is read back that the sequence itself does not read.
The distributions restate the configurations of ``neslgpu_gb300/workloads.py``
and ``bench.py``: uniform int32 keys, N(0,1) float64 values, segment lengths
that are geometric, log-normal, power-law or bimodal.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from neslgpu_gb300 import vcode, vcode_programs
from neslgpu_gb300.cvl import load

DEV = "cuda"
FLT_1E36 = float(np.float32(1e36))  # the serial CVL's starting value of float min and max


# ------------------------------------------------------------------ cases ---
def listed():
    return [
        # the vector operations of a program on a short vector: the inner
        # calls of a divide-and-conquer program, where launches are the time
        {"name": "block_1k", "kind": "block", "n": 1000, "mean": 64},
        # the primitive suite at the size the reference's CPU library is run at
        {"name": "block_1m", "kind": "block", "n": 1 << 20, "mean": 64},
        # bench.py's headline step: scan and sum of long uneven segments
        {"name": "scan_reduce_256m", "kind": "scan_reduce", "n": 1 << 28, "type": "d", "op": "add",
         "segs": "lognormal", "mean": 1100},
        # PACK of a nested float sequence (a filter inside an apply-to-each)
        {"name": "pack_double", "kind": "pack", "n": 40_000_003, "type": "d", "segs": "geometric", "mean": 32,
         "keep": 0.5},
        # a permutation of a large table and its inverse (transposes, sort results)
        {"name": "permute_random", "kind": "permute", "n": 1 << 27, "type": "z"},
        # rank of one long key vector (sort, group-by)
        {"name": "rank_int", "kind": "rank", "n": 1 << 26, "type": "z", "up": True},
        # rank inside many short segments (sorting each row of a nested sequence)
        {"name": "rank_segments", "kind": "rank_seg", "n": 1 << 24, "type": "z", "up": True, "segs": "geometric",
         "mean": 64},
        # moves inside a nested sequence: DIST, INDEX, BPERMUTE, PERMUTE
        {"name": "moves_nested", "kind": "moves", "n": 33_000_001, "type": "d", "segs": "geometric", "mean": 64},
        # writes with a default: the interleave of a flattened program, then
        # a random put whose destinations repeat
        {"name": "put_default", "kind": "put", "n": 5_000_011, "type": "d"},
        # a whole VCODE program from host keys to host keys
        {"name": "quicksort_4m", "kind": "quicksort", "n": 1 << 22},
        # thousands of uneven vectors flattened into one: scan, filter, RAND, gather
        {"name": "batch_flat", "kind": "batch", "vectors": 4096, "n": 1 << 25, "type": "d"},
        # sparse matrix times vector over CSR rows, as its VCODE sequence runs it
        {"name": "spmv_rows", "kind": "spmv", "rows": 1 << 22, "fused": False},
    ]


def _size(rng, lo, hi):
    return int(2.0 ** rng.uniform(lo, hi))


def draw(rng):
    kind = rng.choice(["block", "scan_reduce", "scan_reduce", "pack", "permute", "rank", "rank_seg", "moves", "put",
                       "quicksort", "batch", "spmv"])
    segs = rng.choice(["geometric", "lognormal", "powerlaw", "bimodal", "empties"])
    mean = int(2.0 ** rng.uniform(2, 11))
    typ = rng.choice("zd")
    if kind == "block":
        return {"kind": kind, "n": _size(rng, 8, 22), "mean": mean}
    if kind == "scan_reduce":
        typ = rng.choice("zdb")
        return {"kind": kind, "n": _size(rng, 10, 27.5), "type": typ,
                "op": "ior" if typ == "b" else rng.choice(["add", "max", "min"]), "segs": segs, "mean": mean}
    if kind == "pack":
        return {"kind": kind, "n": _size(rng, 10, 27), "type": typ, "segs": segs, "mean": mean,
                "keep": round(rng.uniform(0.05, 0.95), 3)}
    if kind == "permute":
        return {"kind": kind, "n": _size(rng, 10, 26.5), "type": typ}
    if kind == "rank":
        return {"kind": kind, "n": _size(rng, 10, 25.5), "type": typ, "up": rng.random() < 0.5}
    if kind == "rank_seg":
        return {"kind": kind, "n": _size(rng, 10, 24.5), "type": typ, "up": rng.random() < 0.5, "segs": segs,
                "mean": mean}
    if kind == "moves":
        return {"kind": kind, "n": _size(rng, 10, 26), "type": typ, "segs": segs, "mean": mean}
    if kind == "put":
        return {"kind": kind, "n": _size(rng, 10, 24), "type": typ}
    if kind == "quicksort":
        return {"kind": kind, "n": _size(rng, 8, 22)}
    if kind == "batch":
        n = _size(rng, 16, 25)
        return {"kind": kind, "vectors": max(1, min(8192, int(n / 2.0 ** rng.uniform(9, 14)))), "n": n, "type": typ}
    return {"kind": kind, "rows": _size(rng, 10, 22), "fused": rng.random() < 0.5}


# ----------------------------------------------------------------- inputs ---
def _gen(seed, salt):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1000003 + salt) & 0x7FFFFFFFFFFF)
    return g


def _int32(n, g):
    return torch.randint(-(1 << 31), 1 << 31, (n,), generator=g, device=DEV, dtype=torch.int64).to(torch.int32)


def _values(typ, n, g):
    if typ == "d":
        return torch.randn(n, generator=g, device=DEV, dtype=torch.float64)
    if typ == "b":
        return (torch.rand(n, generator=g, device=DEV) < 0.02).to(torch.int32)
    return _int32(n, g)


def _fit(lens, n):
    """A length sequence cut (or padded) to sum to n."""
    c = torch.cumsum(lens, 0)
    k = int(torch.searchsorted(c, n))
    if k >= lens.numel():
        return torch.cat([lens, lens.new_tensor([n - int(c[-1])])])
    lens = lens[: k + 1].clone()
    lens[k] -= c[k] - n
    return lens


def _power_law(k, g, alpha, hi):
    """k draws of about x^-alpha on [1, hi]."""
    u = torch.rand(k, generator=g, device=DEV, dtype=torch.float64)
    a = 1.0 - alpha
    return (1.0 + u * (float(hi + 1) ** a - 1.0)).pow(1.0 / a).long().clamp(1, hi)


def _lengths(dist, n, mean, g):
    """int64 segment lengths summing to n, of about the given mean."""
    mean = max(2, min(mean, n))
    if dist == "lognormal":  # sigma 2: the mean is e^2 times the median
        k = int(n / mean * 2) + 4096
        x = torch.randn(k, generator=g, device=DEV, dtype=torch.float64)
        return _fit((x * 2.0 + math.log(mean) - 2.0).exp().round().long().clamp(1, 1 << 24), n)
    if dist == "powerlaw":  # alpha 2.1 on [1, 2^16]: short rows and a few long ones
        return _fit(_power_law(n // 3 + 64, g, 2.1, 1 << 16), n)
    if dist == "bimodal":  # half the elements in four long segments, the rest in ones to fours
        half = n // 2
        short = _fit(torch.randint(1, 5, (half // 2 + 16,), generator=g, device=DEV), n - half)
        long = torch.full((4,), half // 4, device=DEV, dtype=torch.int64)
        long[3] += half - 4 * (half // 4)
        at = torch.rand(short.numel() + 4, generator=g, device=DEV)
        return torch.cat([short, long])[torch.argsort(at)]
    k = int(n / mean * 1.3) + 64
    lens = _fit(torch.empty(k, device=DEV, dtype=torch.float64).geometric_(1.0 / mean, generator=g).long(), n)
    if dist == "empties":  # a fifth of the segments empty
        keep = torch.rand(lens.numel() * 5 // 4 + 1, generator=g, device=DEV) >= 0.2
        at = torch.nonzero(keep).flatten()[: lens.numel()]
        out = torch.zeros(keep.numel() + lens.numel() - at.numel(), device=DEV, dtype=torch.int64)
        out[at] = lens[: at.numel()]
        if at.numel() < lens.numel():
            out[keep.numel():] = lens[at.numel():]
        return out
    return lens


def _room(case):
    """A bound on the number of segments that a case of any seed has."""
    n, dist = case["n"], "batch" if case["kind"] == "batch" else case.get("segs", "geometric")
    mean = max(2, min(case.get("mean", 32), n))
    return {"lognormal": int(n / mean * 2) + 4097, "powerlaw": n // 3 + 65, "bimodal": n // 2 + 32,
            "empties": int(n / mean * 3) + 160, "geometric": int(n / mean * 1.3) + 65,
            "batch": n // 24 + 65 + case.get("vectors", 0)}[dist]


def _vec(typ, n):
    """An output vector; where fewer results are written than it has room for, the rest stays zero."""
    return torch.zeros(max(n, 1), device=DEV, dtype=torch.float64 if typ == "d" else torch.int32)


def _units(u):
    return torch.empty(max(int(u), 1), device=DEV, dtype=torch.int64)


def _scratch(c, *calls):
    """One scratch vector for all the calls: (name, its size arguments)."""
    return _units(max([1] + [getattr(c, name + "_scratch")(*a) for name, *a in calls]))


def _segdes(c, lens32, n):
    m = lens32.numel()
    sd = _units(c.siz_fos(n, m))
    scr = _scratch(c, ("mke_fov", n, m))
    c.mke_fov(sd.data_ptr(), lens32.data_ptr(), n, m, scr.data_ptr())
    c.gcvl_sync()
    return sd


_VM = {}


def _interpreter():
    """The VCODE interpreter a program keeps: parsed once, its vectors reused."""
    if "qsort" not in _VM:
        _VM["qsort"] = vcode.Interpreter(vcode_programs.qsort_program())
    return _VM["qsort"]


def _inputs(case, seed):
    """The values a case works on: a dict of tensors (exact() has them too)."""
    kind, g = case["kind"], _gen(seed, 1)
    n = case.get("n", 0)
    if kind == "block":
        return {"x": _int32(n, g), "lens": _lengths("geometric", n, case["mean"], g),
                "perm": torch.randperm(n, generator=g, device=DEV).to(torch.int32)}
    if kind == "scan_reduce":
        return {"x": _values(case["type"], n, g), "lens": _lengths(case["segs"], n, case["mean"], g)}
    if kind == "pack":
        return {"x": _values(case["type"], n, g), "lens": _lengths(case["segs"], n, case["mean"], g),
                "f": (torch.rand(n, generator=g, device=DEV) < case["keep"]).to(torch.int32)}
    if kind == "permute":
        return {"x": _values(case["type"], n, g),
                "perm": torch.randperm(n, generator=g, device=DEV, dtype=torch.int64).to(torch.int32)}
    if kind == "rank":
        return {"x": _values(case["type"], n, g)}
    if kind == "rank_seg":
        return {"x": _values(case["type"], n, g), "lens": _lengths(case["segs"], n, case["mean"], g)}
    if kind == "moves":
        lens = _lengths(case["segs"], n, case["mean"], g)
        m = lens.numel()
        seg = torch.repeat_interleave(torch.arange(m, device=DEV), lens, output_size=n)
        start = (torch.cumsum(lens, 0) - lens)[seg]
        u = torch.rand(n, generator=g, device=DEV, dtype=torch.float64)
        idx = (u * lens[seg]).long().minimum(lens[seg] - 1).to(torch.int32)
        order = torch.argsort(u + seg)  # a permutation within every segment
        perm = torch.empty(n, device=DEV, dtype=torch.int32)
        perm[order] = (torch.arange(n, device=DEV) - start).to(torch.int32)
        return {"x": _values(case["type"], n, g), "v": _values(case["type"], m, g), "lens": lens, "idx": idx,
                "perm": perm, "i0": _int32(m, g), "stride": _int32(m, g)}
    if kind == "put":
        return {"x": _values(case["type"], n, g), "default": _values(case["type"], 3 * n, g),
                "asc": torch.arange(n, device=DEV, dtype=torch.int32) * 3 + 1,
                "idx": torch.randint(0, 3 * n, (n,), generator=g, device=DEV, dtype=torch.int32)}
    if kind == "quicksort":
        return {"keys": _int32(n, g)}
    if kind == "batch":
        k = case["vectors"]  # vector lengths log-normal, sigma 1.6; inner segments geometric, mean 32
        w = (torch.randn(k, generator=g, device=DEV, dtype=torch.float64) * 1.6).exp()
        vec = (w * (n / float(w.sum()))).long().clamp(min=1)
        big = int(torch.argmax(vec))
        vec[big] = max(1, int(vec[big]) + n - int(vec.sum()))
        n = int(vec.sum())
        ends = torch.cumsum(torch.empty(n // 24 + 64, device=DEV, dtype=torch.float64).geometric_(
            1.0 / 32, generator=g).long(), 0)
        ends = torch.unique(torch.cat([ends[ends < n], torch.cumsum(vec, 0)]))
        lens = torch.diff(ends, prepend=ends.new_zeros(1))
        x = _values("d", n, g) if case["type"] == "d" else torch.randint(
            -1000, 1001, (n,), generator=g, device=DEV, dtype=torch.int32)
        return {"x": x, "lens": lens}
    lens = _power_law(case["rows"], g, 2.1, 1 << 16)
    nnz = int(lens.sum())
    return {"lens": lens, "vals": _values("d", nnz, g), "x": _values("d", case["rows"], g),
            "cols": torch.randint(0, case["rows"], (nnz,), generator=g, device=DEV, dtype=torch.int32)}


def prepare(case, seed):
    c = load()
    I = _inputs(case, seed)
    kind, typ = case["kind"], case.get("type", "z")
    S = {"kind": kind, "c": c, "in": I, "case": case}
    if "lens" in I:
        I["lens"] = I["lens"].to(torch.int32)
        m = I["lens"].numel()
        S["m"] = m
    torch.cuda.synchronize()
    n = S["n"] = I["x"].numel() if "x" in I else case["n"]
    O = S["out"] = {}
    if kind == "block":
        O.update(y=_vec("z", n), inc=_vec("z", n), mx=_vec("z", _room(case)), f=_vec("z", n), cnt=_vec("z", _room(case)), p=_vec("z", n),
                 pm=_vec("z", n), rk=_vec("z", n))
        S["zero"] = torch.zeros(n, device=DEV, dtype=torch.int32)
        S["sd"], S["sd2"] = _units(c.siz_fos(n, m)), _units(c.siz_fos(n, m))
        S["scr"] = _scratch(c, ("mke_fov", n, m), ("add_sez", n, m), ("max_rez", n, m), ("pk1_lev", n, m),
                            ("add_ruz", m), ("pk2_lez", n, m, n, m), ("smp_puz", n), ("rku_luz", n))
    elif kind == "scan_reduce":
        S["sd"] = _segdes(c, I["lens"], n)
        O.update(y=_vec(typ, n), r=_vec(typ, _room(case)))
        S["scan"], S["red"] = (getattr(c, f"{case['op']}_{q}e{typ}") for q in "sr")
        S["scr"] = _scratch(c, (f"{case['op']}_se{typ}", n, m), (f"{case['op']}_re{typ}", n, m))
    elif kind == "pack":
        S["sd"], S["sd2"] = _segdes(c, I["lens"], n), _units(c.siz_fos(n, m))
        O.update(cnt=_vec("z", _room(case)), p=_vec(typ, n))
        S["pk2"] = getattr(c, f"pk2_le{typ}")
        S["scr"] = _scratch(c, ("pk1_lev", n, m), ("add_ruz", m), ("mke_fov", n, m), (f"pk2_le{typ}", n, m, n, m))
    elif kind == "permute":
        O.update(y=_vec(typ, n), z=_vec(typ, n))
        S["smp"], S["bck"] = getattr(c, f"smp_pu{typ}"), getattr(c, f"bck_pu{typ}")
        S["scr"] = _scratch(c, (f"smp_pu{typ}", n), (f"bck_pu{typ}", n, n))
    elif kind in ("rank", "rank_seg"):
        name = f"rk{'u' if case['up'] else 'd'}_l{'u' if kind == 'rank' else 'e'}{typ}"
        O["rk"] = _vec("z", n)
        S["fn"] = getattr(c, name)
        if kind == "rank":
            S["scr"] = _scratch(c, (name, n))
        else:
            S["sd"], S["scr"] = _segdes(c, I["lens"], n), _scratch(c, (name, n, m))
    elif kind == "moves":
        S["sd"] = _segdes(c, I["lens"], n)
        O.update(dist=_vec(typ, n), ind=_vec("z", n), g=_vec(typ, n), s=_vec(typ, n))
        S["dis"], S["bck"], S["smp"] = (getattr(c, f"{q}e{typ}") for q in ("dis_v", "bck_p", "smp_p"))
        S["scr"] = _scratch(c, (f"bck_pe{typ}", n, m, n, m), (f"smp_pe{typ}", n, m))
    elif kind == "put":
        O.update(a=_vec(typ, 3 * n), b=_vec(typ, 3 * n))
        S["dpe"], S["scr"] = getattr(c, f"dpe_pu{typ}"), _scratch(c, (f"dpe_pu{typ}", n, 3 * n))
    elif kind == "quicksort":
        S["vm"], S["keys"] = _interpreter(), I["keys"].cpu().numpy()
    elif kind == "batch":
        O.update(y=_vec(typ, n), f=_vec("z", n), cnt=_vec("z", _room(case)), p=_vec(typ, n), bnd=_vec("z", n),
                 idx=_vec("z", n), g=_vec(typ, n))
        S["zeros"] = _vec(typ, n)
        S["sd"], S["sd2"] = _units(c.siz_fos(n, m)), _units(c.siz_fos(n, m))
        for q in ("add_se", "dis_vu", "grt_wu", "pk2_le", "bck_pe"):
            S[q] = getattr(c, q + typ)
        S["scr"] = _scratch(c, ("mke_fov", n, m), (f"add_se{typ}", n, m), ("pk1_lev", n, m), ("add_ruz", m),
                            (f"pk2_le{typ}", n, m, n, m), (f"bck_pe{typ}", n, m, n, m))
    else:
        nnz = S["nnz"] = I["vals"].numel()
        S["sd"] = _segdes(c, I["lens"], nnz)
        O["y"] = _vec("d", m)
        if case["fused"]:
            S["scr"] = _scratch(c, ("gcvl_spmv_csr", nnz, m))
        else:
            S["xg"] = _vec("d", nnz)
            S["scr"] = _scratch(c, ("bck_pud", n, nnz), ("add_red", nnz, m))
    S["p"] = {k: v.data_ptr() for d in (I, O, S) for k, v in d.items() if isinstance(v, torch.Tensor)}
    torch.cuda.synchronize()
    return S


def run(S):
    c, p, O, kind = S["c"], S["p"], S["out"], S["kind"]
    n, m = S.get("n"), S.get("m")
    scr = p.get("scr")
    if kind == "block":
        c.mke_fov(p["sd"], p["lens"], n, m, scr)
        c.add_sez(p["y"], p["x"], p["sd"], n, m, scr)
        c.add_wuz(p["inc"], p["y"], p["x"], n, None)  # inclusive scan
        c.max_rez(p["mx"], p["x"], p["sd"], n, m, scr)
        c.grt_wuz(p["f"], p["x"], p["zero"], n, None)
        c.pk1_lev(p["cnt"], p["f"], p["sd"], n, m, scr)
        n2 = c.add_ruz(p["cnt"], m, scr)
        c.mke_fov(p["sd2"], p["cnt"], n2, m, scr)
        c.pk2_lez(p["p"], p["x"], p["f"], p["sd"], n, m, p["sd2"], n2, m, scr)
        c.smp_puz(p["pm"], p["x"], p["perm"], n, scr)
        c.rku_luz(p["rk"], p["x"], n, scr)
        return [O["y"], O["inc"], O["mx"], O["f"], O["cnt"], O["p"], O["pm"], O["rk"]]
    if kind == "scan_reduce":
        S["scan"](p["y"], p["x"], p["sd"], n, m, scr)
        S["red"](p["r"], p["x"], p["sd"], n, m, scr)
        return [O["y"], O["r"]]
    if kind == "pack":
        c.pk1_lev(p["cnt"], p["f"], p["sd"], n, m, scr)
        n2 = c.add_ruz(p["cnt"], m, scr)
        c.mke_fov(p["sd2"], p["cnt"], n2, m, scr)
        S["pk2"](p["p"], p["x"], p["f"], p["sd"], n, m, p["sd2"], n2, m, scr)
        return [O["cnt"], O["p"]]
    if kind == "permute":
        S["smp"](p["y"], p["x"], p["perm"], n, scr)
        S["bck"](p["z"], p["x"], p["perm"], n, n, scr)
        return [O["y"], O["z"]]
    if kind == "rank":
        S["fn"](p["rk"], p["x"], n, scr)
        return [O["rk"]]
    if kind == "rank_seg":
        S["fn"](p["rk"], p["x"], p["sd"], n, m, scr)
        return [O["rk"]]
    if kind == "moves":
        S["dis"](p["dist"], p["v"], p["sd"], n, m, None)
        c.ind_lez(p["ind"], p["i0"], p["stride"], p["sd"], n, m, None)
        S["bck"](p["g"], p["x"], p["idx"], p["sd"], n, m, p["sd"], n, m, scr)
        S["smp"](p["s"], p["x"], p["perm"], p["sd"], n, m, scr)
        return [O["dist"], O["ind"], O["g"], O["s"]]
    if kind == "put":
        S["dpe"](p["a"], p["x"], p["asc"], p["default"], n, 3 * n, scr)
        S["dpe"](p["b"], p["x"], p["idx"], p["default"], n, 3 * n, scr)
        return [O["a"], O["b"]]
    if kind == "quicksort":
        vm = S["vm"]
        lv = vm.from_host("I", [n])
        sd = vm.segdes_from_lengths(lv)
        vm.drop(lv)
        stack = vm.run("QSORT", [sd, vm.from_host("I", S["keys"])])
        out = vm.to_host(stack[-1])
        for v in stack:
            vm.drop(v)
        return [out]
    if kind == "batch":
        c.rnd_foz(12345)
        c.mke_fov(p["sd"], p["lens"], n, m, scr)
        S["add_se"](p["y"], p["x"], p["sd"], n, m, scr)
        S["dis_vu"](p["zeros"], 0, n, None)
        S["grt_wu"](p["f"], p["x"], p["zeros"], n, None)
        c.pk1_lev(p["cnt"], p["f"], p["sd"], n, m, scr)
        n2 = c.add_ruz(p["cnt"], m, scr)
        c.mke_fov(p["sd2"], p["cnt"], n2, m, scr)
        S["pk2_le"](p["p"], p["y"], p["f"], p["sd"], n, m, p["sd2"], n2, m, scr)
        c.dis_vez(p["bnd"], p["cnt"], p["sd2"], n2, m, None)
        c.rnd_wuz(p["idx"], p["bnd"], n2, None)
        S["bck_pe"](p["g"], p["p"], p["idx"], p["sd2"], n2, m, p["sd2"], n2, m, scr)
        return [O["y"], O["f"], O["cnt"], O["p"], O["bnd"], O["idx"], O["g"]]
    if S["case"]["fused"]:
        c.gcvl_spmv_csr(p["y"], p["vals"], p["cols"], p["x"], p["sd"], S["nnz"], m, scr)
    else:
        c.bck_pud(p["xg"], p["x"], p["cols"], n, S["nnz"], scr)
        c.mul_wud(p["xg"], p["xg"], p["vals"], S["nnz"], None)
        c.add_red(p["y"], p["xg"], p["sd"], S["nnz"], m, scr)
    return [O["y"]]


def work(case):
    """Bytes of the inputs and outputs, each once, and one operation per
    element and primitive (a sort's comparisons for ranks and quicksort)."""
    kind = case["kind"]
    e = 8 if case.get("type") == "d" else 4
    n = case.get("n", 0)
    m = n / max(2, case.get("mean", 32))
    if case.get("segs") in ("powerlaw", "bimodal"):
        m = n / 5
    lg = math.log2(max(n, 2))
    if kind == "block":  # x, perm, lens in; y, inc, flags, half of x, permuted, ranks, 2 per segment out
        return {"bytes": 4 * (7.5 * n + 3 * m), "flops": n * (5 + lg)}
    if kind == "scan_reduce":
        return {"bytes": 2 * e * n + (4 + e) * m, "flops": 2 * n}
    if kind == "pack":
        return {"bytes": n * (4 + e + e * case["keep"]) + 8 * m, "flops": n}
    if kind == "permute":
        return {"bytes": n * (4 + 3 * e), "flops": 0}
    if kind in ("rank", "rank_seg"):
        return {"bytes": n * (e + 4) + (4 * m if kind == "rank_seg" else 0), "flops": n * lg}
    if kind == "moves":
        return {"bytes": n * (4 * e + 12) + m * (e + 12), "flops": n}
    if kind == "put":
        return {"bytes": n * (e + 8 + 9 * e), "flops": 0}
    if kind == "quicksort":
        return {"bytes": 8 * n, "flops": n * lg}
    if kind == "batch":
        return {"bytes": n * (e + e + 4 + (2 * e + 8) / 2) + 8 * n / 32, "flops": 4 * n}
    nnz = 4.8 * case["rows"]
    return {"bytes": nnz * 12 + case["rows"] * 20, "flops": 2 * nnz}


# --------------------------------------------------------- 64-bit results ---
def _heads(lens):
    """For every element: the start of its segment, and the segments' ends."""
    end = torch.cumsum(lens, 0)
    n = int(end[-1])
    return torch.repeat_interleave(end - lens, lens, output_size=n), end


def _scan(x, lens, op, init):
    """(exclusive scan, reduction) of every segment, by doubling."""
    start, end = _heads(lens)
    n, d, longest = x.numel(), 1, int(lens.max())
    f = {"add": torch.add, "max": torch.maximum, "min": torch.minimum}[op]
    y = x.clone()
    while d < longest:
        ok = start[d:] <= torch.arange(n - d, device=DEV)
        y[d:] = torch.where(ok, f(y[:-d], y[d:]), y[d:])
        d *= 2
        del ok
    y = f(y, torch.full((), init, device=DEV, dtype=y.dtype))
    r = torch.full((lens.numel(),), init, device=DEV, dtype=y.dtype)
    r[lens > 0] = y[end[lens > 0] - 1]
    ex = torch.full_like(y, init)
    ex[1:] = y[:-1]
    ex[end[(lens > 0)][:-1]] = init
    return ex, r


def _lrand48(seed, n):
    """n draws of the 31-bit lrand48 stream."""
    M = (1 << 48) - 1
    a, c = 0x5DEECE66D, 0xB
    x = torch.tensor([(a * ((seed << 16) | 0x330E) + c) & M], device=DEV, dtype=torch.int64)
    while x.numel() < n:  # (a, c) is the step over all the draws there are
        to_signed = a - (1 << 64) if a >= 1 << 63 else a
        x = torch.cat([x, (x * to_signed + c) & M])
        a, c = (a * a) & M, (a * c + c) & M
    return (x[:n] >> 17).to(torch.int32)


def _padded(v, n):
    return torch.cat([v, v.new_zeros(max(n, 1) - v.numel())])


def exact(case, seed):
    """Floating results in 64 bits; whole numbers are compared as they are."""
    kind, typ = case["kind"], case.get("type", "z")
    if kind in ("block", "rank", "rank_seg", "quicksort") or (kind not in ("spmv",) and typ != "d"):
        return None
    I = _inputs(case, seed)
    lens = I.get("lens")
    if kind == "scan_reduce":
        init = {"add": 0.0, "max": -FLT_1E36, "min": FLT_1E36}[case["op"]]
        y, r = _scan(I["x"], lens, case["op"], init)
        return [y, _padded(r, _room(case))]
    if kind == "pack":
        return [None, _padded(I["x"][I["f"] != 0], case["n"])]
    if kind == "permute":
        y = torch.empty_like(I["x"])
        y[I["perm"].long()] = I["x"]
        return [y, I["x"][I["perm"].long()]]
    if kind == "moves":
        start, _ = _heads(lens)
        s = torch.empty_like(I["x"])
        s[start + I["perm"]] = I["x"]
        return [torch.repeat_interleave(I["v"], lens), None, I["x"][start + I["idx"]], s]
    if kind == "put":
        a, b = I["default"].clone(), I["default"].clone()
        a[I["asc"].long()] = I["x"]
        last = torch.full((b.numel(),), -1, device=DEV, dtype=torch.int64)  # the last writer stays
        last.scatter_reduce_(0, I["idx"].long(), torch.arange(case["n"], device=DEV), "amax")
        b[last >= 0] = I["x"][last[last >= 0]]
        return [a, b]
    if kind == "batch":
        y, _ = _scan(I["x"], lens, "add", 0.0)
        keep = I["x"] > 0
        p = y[keep]
        seg = torch.repeat_interleave(torch.arange(lens.numel(), device=DEV), lens)[keep]
        cnt = torch.bincount(seg, minlength=lens.numel())
        start, _ = _heads(cnt)
        at = _lrand48(12345, p.numel()).long() % cnt[seg]
        return [y, None, None, _padded(p, y.numel()), None, None, _padded(p[start + at], y.numel())]
    return [_scan(I["vals"] * I["x"][I["cols"].long()], lens, "add", 0.0)[1]]
