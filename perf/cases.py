"""The engine's work as its users call it: decode, filter, encode and expression selection at the sizes and value
distributions of the benchmark configurations, through the package's public entry points.

listed() names the cases, draw() makes more of the same ranges, prepare() builds what a program has in hand before
the call (device buffers, plans, weights), run() is one pass, work() the bytes it cannot do without, and exact()
the decoded values (or the selector's float64 result) in plain torch.
"""
import functools
import math

import numpy as np
import torch

from fastlanes_b200 import _lib as L
from fastlanes_b200 import pages as PG
from fastlanes_b200 import primitives as P
from fastlanes_b200 import rowgroups as RG
from fastlanes_b200 import select as SL
from fastlanes_b200 import strings as S
from fastlanes_b200 import workloads as W

DEV = "cuda"
UNSIGNED = {8: torch.uint8, 16: torch.uint16, 32: torch.uint32, 64: torch.uint64}
SIGNED = {8: torch.int8, 16: torch.int16, 32: torch.int32, 64: torch.int64}
PAGE_TYPES = {"int32": (PG.INT32, 32), "uint32": (PG.UINT32, 32), "int64": (PG.INT64, 64), "uint64": (PG.UINT64, 64)}
EXPR_IDS = {"raw": 0, "ffor": 1, "rle": 6, "delta": 11}
FAMILIES = {"for_u32": 1, "for_i64": 1, "delta_i64": 3, "rle_i32": 2, "rle_i64": 2, "dict_i32": 4, "dict_rle_i32": 5}
THRESHOLD, STRIDE = 0.7, 16  # the learned selector's confidence threshold and sampling of the benchmark


def listed():
    return [
        # the smallest call in earnest: one primitive over 1024 vectors (FFOR u32 at 7 bits), launch and host bound
        {"name": "unffor_u32_1k", "kind": "primitive", "op": "unffor", "width": 32, "max_bw": 7, "n_vec": 1024,
         "order": 0},
        # a scan of bit-packed data of every width: u32 and u64 vectors mixed, one plan, original order
        {"name": "bw_sweep", "kind": "sweep", "n32": 65536, "n64": 32768, "order": 1},
        # a sorted timestamp column, DELTA page
        {"name": "delta_i64", "kind": "page", "expr": "delta", "dtype": "int64", "n_vec": 32768},
        # a column of runs, RLE page
        {"name": "rle_i32", "kind": "page", "expr": "rle", "dtype": "int32", "n_vec": 32768},
        # a WHERE clause on the timestamp column: predicate on the compressed page, bitmaps, then row positions
        {"name": "filter_delta_i64", "kind": "filter", "expr": "delta", "dtype": "int64", "n_vec": 16001, "keep": 0.5},
        # writing a column: transpose, deltas, widths and bases, bit packing, all on the device
        {"name": "encode_delta_i64", "kind": "encode", "scheme": "delta", "width": 64, "signed": True, "n_vec": 16385},
        # a string column with a dictionary (DICT over an FSST dictionary), the most common string encoding
        {"name": "strings_dict", "kind": "dict_strings", "n_vec": 16384, "n_dict": 4096},
        # a string column without one (FSST column), some rows with bytes outside the symbol table
        {"name": "strings_fsst", "kind": "fsst_strings", "n_vec": 8192, "n_dict": 4096, "escaped": 0.02},
        # a table's row groups: integer columns of every encoding in one plan, string columns in one set
        {"name": "rowgroups", "kind": "rowgroups", "int_columns": 20, "str_columns": 5, "max_vec": 2048},
        # choosing every chunk's encoding exactly (wizard) for integer and string columns
        {"name": "wizard", "kind": "wizard", "int_columns": 28, "str_columns": 6, "max_vec": 2048},
        # choosing it with the learned selector (statistics, MLP, wizard for the unsure chunks)
        {"name": "learned", "kind": "learned", "int_columns": 56, "max_vec": 2048},
        # the C API on host memory: encode a pinned column into a page, decode the page back
        {"name": "host_ffor_u64", "kind": "host", "expr": "ffor", "dtype": "uint64", "n_vec": 8192},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["primitive", "sweep", "page", "page", "filter", "encode", "dict_strings", "fsst_strings",
                       "rowgroups", "wizard", "learned", "host"])
    if kind == "primitive":
        op = rng.choice(["unpack", "unffor", "unffor_rsum", "rsum", "untranspose"])
        width = rng.choice([16, 32, 64] if op in ("unffor_rsum", "rsum") else [8, 16, 32, 64])
        return {"kind": kind, "op": op, "width": width, "max_bw": rng.randint(1, width), "n_vec": _log(rng, 1, 32768),
                "order": rng.randint(0, 1)}
    if kind == "sweep":
        return {"kind": kind, "n32": _log(rng, 256, 65536), "n64": _log(rng, 256, 32768), "order": rng.randint(0, 1)}
    if kind in ("page", "filter"):
        c = {"kind": kind, "expr": rng.choice(["raw", "ffor", "delta", "rle", "dict", "dict_rle"]),
             "dtype": rng.choice(list(PAGE_TYPES)), "n_vec": _log(rng, 3, 32768)}
        return dict(c, keep=round(rng.uniform(0.01, 0.99), 3), n_vec=min(c["n_vec"], 16384)) if kind == "filter" else c
    if kind == "encode":
        return {"kind": kind, "scheme": rng.choice(["ffor", "delta"]), "width": rng.choice([16, 32, 64]),
                "signed": rng.random() < 0.5, "n_vec": _log(rng, 5, 16384)}
    if kind == "dict_strings":
        return {"kind": kind, "n_vec": _log(rng, 16, 16384), "n_dict": _log(rng, 16, 4096)}
    if kind == "fsst_strings":
        return {"kind": kind, "n_vec": _log(rng, 16, 8192), "n_dict": _log(rng, 16, 4096),
                "escaped": rng.choice([0.0, round(rng.uniform(0, 0.2), 3)])}
    if kind in ("rowgroups", "wizard"):
        return {"kind": kind, "int_columns": rng.randint(4, 20), "str_columns": rng.randint(1, 5),
                "max_vec": _log(rng, 65, 2048)}
    if kind == "learned":
        return {"kind": kind, "int_columns": rng.randint(4, 56), "max_vec": _log(rng, 65, 2048)}
    return {"kind": "host", "expr": rng.choice(["raw", "ffor", "delta", "rle"]), "dtype": rng.choice(list(PAGE_TYPES)),
            "n_vec": _log(rng, 8, 8192)}


# ---- values, made from the seed in plain torch (shared by prepare and exact) ------------------------------------
def _gen(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1_000_003 + salt) & (2**62 - 1))
    return g


def _original_index():
    k = torch.arange(1024, device=DEV)
    order = torch.tensor([0, 4, 2, 6, 1, 5, 3, 7], device=DEV)
    return (k % 16) * 64 + order[(k // 16) % 8] * 8 + k // 128


def _transposed(v):
    return v.view(-1, 1024)[:, _original_index()].reshape(-1)


def _narrow(v, width):
    """int64 values to the width's unsigned type (low bits)."""
    if width == 64:
        return v.view(torch.uint64)
    return (v & ((1 << width) - 1)).to(torch.int64).to(SIGNED[width]).view(UNSIGNED[width])


def _mixed_width(g, width, n_vec, max_bw):
    """Per-vector width uniform in 0..max_bw, base uniform, values base + uniform (wrapping in the type):
    (int64 values, bit widths, int64 bases)."""
    bw = torch.randint(0, max_bw + 1, (n_vec,), generator=g, device=DEV)
    base = torch.randint(-(1 << 62), 1 << 62, (n_vec,), generator=g, device=DEV)
    if width < 64:
        base = base & ((1 << width) - 1)
    bits = torch.randint(-(1 << 63), (1 << 63) - 1, (n_vec, 1024), generator=g, device=DEV)
    mask = torch.where(bw >= 64, torch.full_like(bw, -1), (torch.ones_like(bw) << bw.clamp(max=63)) - 1)
    return ((bits & mask[:, None]) + base[:, None]).view(-1), bw.to(torch.uint8), base


def _geometric(g, n, mean):
    u = torch.rand(n, generator=g, device=DEV, dtype=torch.float64).clamp_(min=1e-300)
    return (torch.log(u) / math.log1p(-1.0 / mean)).floor().to(torch.int64) + 1 if mean > 1.0 else torch.ones(
        n, dtype=torch.int64, device=DEV)


def _runs(g, n, mean):
    """Run number of each of n positions, geometric lengths."""
    ends = torch.cumsum(_geometric(g, int(n / mean * 1.5) + 2048, mean), 0)
    return torch.searchsorted(ends, torch.arange(n, device=DEV), right=True)


def _zipf(g, n, d, a):
    cdf = torch.cumsum(torch.arange(1, d + 1, device=DEV, dtype=torch.float64).pow(-a), 0)
    u = torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * cdf[-1]
    return torch.searchsorted(cdf, u).clamp_(max=d - 1)


def _sorted_values(g, n, mean, start):
    return torch.cumsum(_geometric(g, n, mean), 0) + start


def _column(case, seed):
    """The int64 values of a page / filter / host case."""
    g, n, width = _gen(seed, 7), case["n_vec"] * 1024, PAGE_TYPES[case["dtype"]][1]
    e = case["expr"]
    if e == "delta":
        return _sorted_values(g, n, 10.0, 1_600_000_000_000_000_000 if width == 64 else 1_000_000)
    if e == "rle":
        run = _runs(g, n, 8.0)
        return torch.randint(0, 10**6, (int(run[-1]) + 1,), generator=g, device=DEV)[run]
    if e in ("dict", "dict_rle"):
        dic = torch.randint(0, 1 << 30, (3000,), generator=g, device=DEV)
        if e == "dict":
            return dic[_zipf(g, n, 3000, 1.1)]
        run = _runs(g, n, 8.0)
        return dic[_zipf(g, int(run[-1]) + 1, 3000, 1.1)[run]]
    return _mixed_width(g, width, case["n_vec"], min(width - 1, 40))[0]


def _typed(v, dtype):
    signed, width = not dtype.startswith("u"), PAGE_TYPES[dtype][1]
    u = _narrow(v, width)
    return u.view(SIGNED[width]) if signed else u


def _lengths(case, count, salt):
    """Vectors of each column of a table, spread evenly over 64..max_vec (set by the case, not the seed)."""
    return [64 + int((0.618034 * (i + salt) + 0.37) % 1.0 * (case["max_vec"] - 63)) for i in range(count)]


def _int_columns(case, seed):
    """Integer columns of a table: (tensor int32 / int64, is_signed, family)."""
    rng = np.random.default_rng(seed)
    names = list(FAMILIES)
    cols = []
    for i, n in enumerate(_lengths(case, case["int_columns"], 0)):
        fam, n = names[i % len(names)], n * 1024
        g = _gen(seed, 100 + i)
        if fam == "for_u32":
            bw = int(rng.integers(0, 33))
            v = torch.randint(0, 1 << bw, (n,), generator=g, device=DEV) + int(rng.integers(0, 2**32 - 2**bw + 1))
            cols.append((_narrow(v, 32).view(torch.int32), False, fam))
        elif fam == "for_i64":
            bw = int(rng.integers(0, 63))
            v = torch.randint(0, 1 << bw, (n,), generator=g, device=DEV) + int(rng.integers(-2**61, 2**61))
            cols.append((v, True, fam))
        elif fam == "delta_i64":
            cols.append((_sorted_values(g, n, float(np.exp(rng.uniform(0.1, 8))), 1_600_000_000_000_000_000), True, fam))
        elif fam.startswith("rle"):
            run = _runs(g, n, float(rng.uniform(2, 64)))
            v = torch.randint(0, 1 << int(rng.integers(4, 31)), (int(run[-1]) + 1,), generator=g, device=DEV)[run]
            cols.append((v if fam == "rle_i64" else v.to(torch.int32), True, fam))
        else:
            d, a = int(np.exp(rng.uniform(np.log(16), np.log(65536)))), float(rng.uniform(0.8, 1.5))
            dic = torch.randint(-2**30, 2**30, (d,), generator=g, device=DEV)
            if fam == "dict_i32":
                code = _zipf(g, n, d, a)
            else:
                run = _runs(g, n, float(rng.uniform(2, 64)))
                code = _zipf(g, int(run[-1]) + 1, d, a)[run]
            cols.append((dic[code].to(torch.int32), True, fam))
    return cols


def _dictionary(seed, n_dict):
    """String dictionary entries (bytes, offsets): 5..40-byte token strings."""
    return W.string_dictionary(seed=seed % (2**31), n_dict=n_dict)


# ---- prepare ----------------------------------------------------------------------------------------------------
def _place(page):
    """A page's bytes on the device, its packed buffer 16-byte aligned: (buffer, address)."""
    shift = PG.placement(page)
    buf = torch.zeros(page.size + 64, dtype=torch.uint8, device=DEV)
    buf[shift:shift + page.size] = torch.from_numpy(page).to(DEV)
    return buf, buf.data_ptr() + shift


def _prepare_primitive(case, seed):
    g, w, op = _gen(seed), case["width"], case["op"]
    if op in ("unffor_rsum", "rsum"):
        mean = 2.0 ** min(max(case["max_bw"] - 4, 1), 20)
        tr = P.transpose_i(_narrow(_sorted_values(g, case["n_vec"] * 1024, mean, 1000), w))
        lane = tr.view(SIGNED[w]).view(-1, 1024)[:, :1024 // w].contiguous().view(UNSIGNED[w])
        d = P.unrsum(tr)
        if op == "rsum":
            return {"deltas": d, "lane": lane}
        bw, base = P.analyze(d)
        packed, off = P.ffor(d, bw, base)
        return {"packed": packed, "off": off, "bw": bw, "base": base, "lane": lane}
    v, bw, base = _mixed_width(g, w, case["n_vec"], case["max_bw"])
    if op == "unpack":
        v = (v.view(-1, 1024) - base[:, None]).reshape(-1)
    tr = P.transpose_i(_narrow(v, w))
    if op == "untranspose":
        return {"tr": tr}
    base = _narrow(base, w)
    packed, off = P.ffor(tr, bw, base if op == "unffor" else None)
    return {"packed": packed.view(UNSIGNED[w]), "off": off, "bw": bw, "base": base}


def _prepare_sweep(case, seed):
    cols = []
    for w, n in ((32, case["n32"]), (64, case["n64"])):
        v, bw, base = _mixed_width(_gen(seed, w), w, n, w)
        base = _narrow(base, w)
        packed, off = P.ffor(P.transpose_i(_narrow(v, w)), bw, base)
        cols.append(W.FforColumn(w, packed, off, bw, base))
    items = torch.cat([torch.arange(case["n32"], device=DEV), (1 << 24) | torch.arange(case["n64"], device=DEV)])
    queue = items[torch.randperm(items.numel(), generator=_gen(seed, 3), device=DEV)].to(torch.int32)
    outs = [torch.empty(c.n_vec * 1024, dtype=SIGNED[c.width], device=DEV) for c in cols]
    return {"plan": W.Plan(cols, outs, case["order"], queue), "outs": outs}


def _encode_page(case, values):
    host = values.cpu().numpy()
    if case["expr"] in ("dict", "dict_rle"):
        return PG.encode_int_dict(host, rle=case["expr"] == "dict_rle")
    return PG.encode_from_memory(host, PAGE_TYPES[case["dtype"]][0], EXPR_IDS[case["expr"]])[0], None


def _prepare_page(case, seed):
    code, _ = PAGE_TYPES[case["dtype"]]
    values = _typed(_column(case, seed), case["dtype"])
    page, dic = _encode_page(case, values)
    buf, addr = _place(page)
    d_dict = None if dic is None else torch.from_numpy(dic).to(DEV)
    col = dict(d_page=addr, page_size=page.size, d_dict=None if dic is None else d_dict.data_ptr(),
               dict_size=0 if dic is None else dic.size, data_type=code, order=1)
    keep = {"buf": buf, "dict": d_dict}
    if case["kind"] == "page":
        out = torch.empty_like(values)
        return dict(keep, out=out, plan=PG.PagePlan([dict(col, d_out=out.data_ptr())]))
    n = case["n_vec"]
    bitmap = torch.empty(n * 16, dtype=torch.int64, device=DEV)
    idx = torch.zeros(n * 1024, dtype=torch.int16, device=DEV)
    count = torch.empty(n, dtype=torch.int16, device=DEV)
    plan = PG.FilterPlan([dict(col, d_out=bitmap.data_ptr())], PG.PRED_LE, _cut(case, values, seed))
    return dict(keep, plan=plan, n=n, bitmap=bitmap, idx=idx, count=count)


def _cut(case, values, seed):
    """The filter's constant: about case["keep"] of a sample of the values are at or below it."""
    keep = min(1.0, case["keep"] * float(np.random.default_rng(seed).uniform(0.9, 1.1)))
    sample = values.view(SIGNED[PAGE_TYPES[case["dtype"]][1]])[::max(1, values.numel() // 65536)].cpu().numpy()
    if case["dtype"].startswith("u"):
        sample = sample.view(case["dtype"])
    return int(np.sort(sample)[int(keep * (sample.size - 1))])


def _prepare_encode(case, seed):
    """Every vector's bit width is set by the case (the packed size must not depend on the seed): the widest value
    of a vector, or its widest gap, is put in."""
    g, w, n = _gen(seed), case["width"], case["n_vec"]
    by_case = np.random.default_rng(n)
    if case["scheme"] == "delta":
        top = torch.from_numpy((1 << by_case.choice([6, 7, 8], n, p=[0.25, 0.65, 0.1])) - 1).to(DEV)[:, None]
        gap = torch.minimum(_geometric(g, n * 1024, 10.0).view(n, 1024), top)
        gap[:, 517] = top[:, 0]
        v = torch.cumsum(gap.view(-1), 0) + (1_600_000_000_000_000_000 if w == 64 else 1000)
    else:
        bw = torch.from_numpy(by_case.integers(0, min(w - 1, 40) + 1, n)).to(DEV)[:, None]
        top = (torch.ones_like(bw) << bw) - 1
        bits = torch.randint(0, 1 << 62, (n, 1024), generator=g, device=DEV) & top
        bits[:, 3], bits[:, 700] = 0, top[:, 0]
        low = torch.randint(0, 1 << (w - 2), (n, 1), generator=g, device=DEV)
        v = (torch.minimum(low, (1 << (w - 1)) - 1 - top) + bits).view(-1)
    return {"values": _narrow(v, w)}


def _prepare_dict_strings(case, seed):
    dbytes, doffs = _dictionary(seed, case["n_dict"])
    codes = _zipf(_gen(seed, 1), case["n_vec"] * 1024, case["n_dict"], 1.1).to(torch.int32).cpu().numpy()
    page, dic = S.encode_string_dict(dbytes, doffs, codes.view(np.uint32))
    buf, addr = _place(page)
    d_dict = torch.from_numpy(dic).to(DEV)
    return _string_state(S.StringPlan(addr, page.size, d_dict.data_ptr(), dic.size), [buf, d_dict])


def _string_outputs(plan):
    """Offsets and bytes of a column's rows (at most 40 bytes each)."""
    return (torch.empty(plan.n_rows + 1, dtype=torch.int32, device=DEV),
            torch.zeros(plan.n_rows * 40 + 16, dtype=torch.uint8, device=DEV))


def _string_state(plan, keep):
    offsets, data = _string_outputs(plan)
    return {"plan": plan, "keep": keep, "offsets": offsets, "data": data}


def _prepare_fsst_strings(case, seed):
    """Every row compressed with the dictionary entries' table; a share of the entries holds bytes the table has no
    symbol for, so that their rows carry escapes."""
    rng = np.random.default_rng(seed)
    dbytes, doffs = _dictionary(seed, case["n_dict"])
    dbytes = dbytes.copy()
    for e in np.nonzero(rng.random(case["n_dict"]) < case["escaped"])[0]:
        at = rng.integers(int(doffs[e]), int(doffs[e + 1]), 2)
        dbytes[at] = rng.integers(128, 256, 2)
    table, comp, coffs = S.fsst_compress(dbytes, doffs)
    codes = _zipf(_gen(seed, 1), case["n_vec"] * 1024, case["n_dict"], 1.1)
    rows, offs = W.dict_rows_device(comp, coffs, codes.cpu().numpy(), DEV)
    n = int(offs[-1])
    page, dic = S.fsst_page(table, rows[:n].cpu().numpy(), offs.cpu().numpy().view(np.uint64))
    d_page, d_dict = torch.from_numpy(page).to(DEV), torch.from_numpy(dic).to(DEV)
    return _string_state(S.StringPlan(d_page.data_ptr(), page.size, d_dict.data_ptr(), dic.size), [d_page, d_dict])


def _prepare_rowgroups(case, seed):
    cols = _int_columns(case, seed)
    col, first, count, choice = [], [], [], []
    for c, (t, _, fam) in enumerate(cols):
        n = t.numel() // 1024
        for v in range(0, n, 64):
            col.append(c), first.append(v), count.append(min(64, n - v)), choice.append(FAMILIES[fam])
    ints = RG.RowGroupSet([(t, s) for t, s, _ in cols], (col, first, count), choice, DEV)
    strs = [_prepare_dict_strings({"n_vec": n, "n_dict": 4096}, seed + i)
            for i, n in enumerate(_lengths(case, case["str_columns"], 3))]
    group = S.StringSet([s["plan"] for s in strs])
    group.bind([s["offsets"] for s in strs], [s["data"] for s in strs])
    return {"ints": ints, "strs": strs, "set": group}


def _alphabet_rows(g, n):
    """n rows of 5..40 random letters: (bytes, offsets int64)."""
    lens = torch.randint(5, 41, (n,), generator=g, device=DEV)
    offs = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    offs[1:] = torch.cumsum(lens, 0)
    return torch.randint(97, 123, (int(offs[-1]),), generator=g, device=DEV).to(torch.uint8), offs


def _prepare_wizard(case, seed):
    ints = SL.SelectionPlan([(t, s) for t, s, _ in _int_columns(case, seed)])
    strs = []
    for i, n in enumerate(_lengths(case, case["str_columns"], 3)):
        g = _gen(seed, 900 + i)
        if i % 3 == 2:  # every row another string
            byts, offs = _alphabet_rows(g, n * 1024)
        else:  # dictionary strings, in runs in every other such column
            dbytes, doffs = _dictionary(seed + i, 2048)
            run = _runs(g, n * 1024, 12.0) if i % 3 else torch.arange(n * 1024, device=DEV)
            codes = _zipf(g, int(run[-1]) + 1, 2048, 1.1)[run]
            byts, offs = W.dict_rows_device(dbytes, doffs, codes.cpu().numpy(), DEV)
        end = int(offs[2048])
        table, _, _ = S.fsst_compress(byts[:end].cpu().numpy(), offs[:2049].cpu().numpy().view(np.uint64))
        strs.append((byts, offs, table))
    return {"ints": ints, "strs": SL.StrSelectionPlan(strs)}


def _prepare_learned(case, seed):
    cols = [(t, s) for t, s, _ in _int_columns(case, seed)]
    return {"plan": SL.SelectionPlan(cols), "params": _selector_params().float()}


def _prepare_host(case, seed):
    code, _ = PAGE_TYPES[case["dtype"]]
    t = _typed(_column(case, seed), case["dtype"])
    values = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    values.copy_(t)
    back = torch.zeros(t.shape, dtype=t.dtype, pin_memory=True)
    page = torch.zeros(values.numel() * values.element_size() * 2 + 65536, dtype=torch.uint8, pin_memory=True)
    return {"values": values, "page": page, "back": back, "code": code, "expr": EXPR_IDS[case["expr"]],
            "size": PG._u64(), "meta": PG._u64()}


PREPARE = {"primitive": _prepare_primitive, "sweep": _prepare_sweep, "page": _prepare_page, "filter": _prepare_page,
           "encode": _prepare_encode, "dict_strings": _prepare_dict_strings, "fsst_strings": _prepare_fsst_strings,
           "rowgroups": _prepare_rowgroups, "wizard": _prepare_wizard, "learned": _prepare_learned,
           "host": _prepare_host}


def prepare(case, seed):
    state = PREPARE[case["kind"]](case, seed)
    state["case"] = case
    torch.cuda.synchronize()
    return state


# ---- run --------------------------------------------------------------------------------------------------------
def _run_primitive(s):
    return _primitive(s, s["case"]).view(SIGNED[s["case"]["width"]])


def _primitive(s, c):
    op, order = c["op"], c["order"]
    if op == "unffor":
        return P.unffor(s["packed"], s["bw"], s["base"], s["off"], order)
    if op == "unpack":
        return P.unpack(s["packed"], s["bw"], s["off"], order, c["width"])
    if op == "unffor_rsum":
        return P.unffor_rsum(s["packed"], s["bw"], s["base"], s["lane"], s["off"], order)
    if op == "rsum":
        return P.rsum(s["deltas"], s["lane"], order)
    return P.untranspose_i(s["tr"])


def _run_sweep(s):
    s["plan"].decode()
    return s["outs"]


def _run_page(s):
    s["plan"].decode()
    return s["out"]


def _run_filter(s):
    s["plan"].decode()
    PG.bitmap_to_selection(s["bitmap"].data_ptr(), s["n"], s["idx"].data_ptr(), s["count"].data_ptr())
    return [s["bitmap"], s["idx"], s["count"]]


def _run_encode(s):
    c, w = s["case"], s["case"]["width"]
    tr = P.transpose_i(s["values"])
    out = {}
    if c["scheme"] == "delta":
        out["lane"] = tr.view(SIGNED[w]).view(-1, 1024)[:, :1024 // w].contiguous()
        tr = P.unrsum(tr)
    out["bw"], base = P.analyze(tr, c["signed"])
    out["packed"], off = P.ffor(tr, out["bw"], base)
    return dict(out, base=base.view(SIGNED[w]), off=off.view(torch.int64))


def _run_strings(s):
    s["plan"].decode_into(s["offsets"], s["data"])
    return [s["offsets"], s["data"]]


def _run_rowgroups(s):
    s["ints"].decode()
    s["set"].decode()
    return {"ints": s["ints"].outputs, "strs": [[c["offsets"], c["data"]] for c in s["strs"]]}


def _run_wizard(s):
    return [list(s["ints"].wizard()), list(s["strs"].wizard())]


def _run_learned(s):
    choice, conf, n = s["plan"].learned(s["params"], STRIDE, THRESHOLD)
    return {"choice": choice, "conf": conf, "fallback": n}


def _run_host(s):
    v, page = s["values"], s["page"]
    ok = L.lib.encode_from_memory(v.data_ptr(), v.numel(), page.numel(), page.data_ptr(), s["size"], s["meta"],
                                  s["code"], s["expr"])
    L.lib.decode_to_memory(page.data_ptr(), s["back"].data_ptr(), s["code"])
    return {"ok": int(ok), "size": s["size"].value, "page": page, "back": s["back"]}


RUN = {"primitive": _run_primitive, "sweep": _run_sweep, "page": _run_page, "filter": _run_filter,
       "encode": _run_encode, "dict_strings": _run_strings, "fsst_strings": _run_strings, "rowgroups": _run_rowgroups,
       "wizard": _run_wizard, "learned": _run_learned, "host": _run_host}


def run(state):
    return RUN[state["case"]["kind"]](state)


# ---- work: each input read once, each output written once (expected figures of the distributions) ---------------
def _page_bytes(expr, dtype, n):
    """Expected page bytes of n vectors."""
    size = PAGE_TYPES[dtype][1] // 8
    return n * {"raw": 1024 * size, "ffor": 128 * min(8 * size - 1, 40) / 2 + 1 + size, "delta": 128 * 7 + 129 + size,
                "rle": 128 * size + 259, "dict": 128 * 12 + 5, "dict_rle": 128 * 4 + 259}[expr]


def work(case):
    k, b = case["kind"], 0.0
    if k == "primitive":
        w, n = case["width"], case["n_vec"]
        read = {"unpack": 64 * case["max_bw"] + 9, "unffor": 64 * case["max_bw"] + 9 + w // 8,
                "unffor_rsum": 128 * min(case["max_bw"], w) + 137 + w // 8, "rsum": 128 * w + 128,
                "untranspose": 128 * w}[case["op"]]
        b = n * (read + 128 * w)
    elif k == "sweep":
        b = sum(n * (64 * w + 9 + w // 8 + 4 + 128 * w) for n, w in ((case["n32"], 32), (case["n64"], 64)))
    elif k == "page":
        b = _page_bytes(case["expr"], case["dtype"], case["n_vec"]) + case["n_vec"] * 128 * PAGE_TYPES[case["dtype"]][1]
    elif k == "filter":
        b = _page_bytes(case["expr"], case["dtype"], case["n_vec"]) + case["n_vec"] * (130 + 2048 * case["keep"])
    elif k == "encode":
        w = case["width"]
        out = 128 * 7 + 128 if case["scheme"] == "delta" else 64 * min(w, 40)
        b = case["n_vec"] * (128 * w + out + 9 + w // 8)
    elif k == "dict_strings":
        b = case["n_vec"] * 1024 * (12 / 8 + 4 + 22.5)
    elif k == "fsst_strings":
        b = case["n_vec"] * 1024 * (4 + 9 + 4 + 22.5)
    elif k in ("rowgroups", "wizard", "learned"):
        vec = (64 + case["max_vec"]) / 2
        size = 1024 * 40 / 7  # mean value bytes of a vector over the families (three of 8 bytes, four of 4)
        if k == "rowgroups":
            b = case["int_columns"] * vec * size * 1.3 + case["str_columns"] * vec * 1024 * 28
        elif k == "wizard":
            b = case["int_columns"] * vec * size + case["str_columns"] * vec * 1024 * (22.5 + 8)
        else:
            b = case["int_columns"] * vec * size / STRIDE
            n = case["int_columns"] * vec / STRIDE
            return {"bytes": b, "flops": 2 * n * (32 * 128 + 128 * 128 + 128 * 6)}
    else:
        b = 2 * (_page_bytes(case["expr"], case["dtype"], case["n_vec"]) +
                 case["n_vec"] * 128 * PAGE_TYPES[case["dtype"]][1])
    return {"bytes": float(b), "flops": 0.0}


# ---- the learned selector in float64 torch ----------------------------------------------------------------------
def _bits(d):
    """Bit length of int64 patterns read as unsigned."""
    out = torch.zeros_like(d)
    x = d
    for s in (32, 16, 8, 4, 2, 1):
        hi = (x >> s) & ((1 << (64 - s)) - 1)
        up = hi != 0
        out = torch.where(up, out + s, out)
        x = torch.where(up, hi, x)
    return out + (x != 0)


def _statistics(x, width, signed):
    """The selector's 32 statistics of every row of x (n x 1024, int64: values of the column's type, sign- or
    zero-extended), float64."""
    n, w, size = x.shape[0], float(width), width // 8
    mask = (1 << width) - 1 if width < 64 else -1
    flip = -(1 << 63) if (width == 64 and not signed) else 0  # orders unsigned 64-bit patterns

    def span(v, dim=1):
        k = v ^ flip
        return _bits((k.amax(dim) - k.amin(dim)) & mask)

    def wrap(d):  # difference in the type, as its signed or unsigned value
        d = d & mask
        return d if width == 64 or not signed else torch.where(d >= 1 << (width - 1), d - (1 << width), d)

    diff = torch.zeros_like(x)
    diff[:, 1:] = x[:, 1:] - x[:, :-1]
    chain = wrap(diff).view(n, -1, 64 if width == 64 else 32).clone()
    chain[:, :, 0] = 0
    bw_f, bw_d = span(x), span(chain.view(n, 1024))
    start = torch.ones_like(x, dtype=torch.bool)
    start[:, 1:] = x[:, 1:] != x[:, :-1]
    runs = start.sum(1)
    bw_i = (start.view(n, 64, 16)[:, :, 1:]).flatten(1).any(1).long()

    def longest(first):  # longest stretch of a row's positions that a True begins
        pos = torch.arange(1024, device=x.device).expand(n, 1024)
        since = torch.cummax(torch.where(first, pos, torch.zeros_like(pos)), 1).values
        return (pos - since).amax(1) + 1

    srt = torch.sort(x, 1).values
    new = torch.ones_like(start)
    new[:, 1:] = srt[:, 1:] != srt[:, :-1]
    dv, top, maxrun = new.sum(1), longest(new), longest(start)
    key = x ^ flip
    inc, dec = (key[:, 1:] > key[:, :-1]).sum(1), (key[:, 1:] < key[:, :-1]).sum(1)
    d = diff[:, 1:] & mask
    neg = ((d >> (width - 1)) & 1) != 0
    bw_a = _bits(torch.where(neg, (-d) & mask, d)).amax(1)
    mn, mx = key.amin(1) ^ flip, key.amax(1) ^ flip
    above = (x - mn[:, None]) & mask
    cnt_top = torch.where(bw_f[:, None] > 0, (above >> (bw_f - 1).clamp(min=0)[:, None]) & 1, 0).sum(1)
    blk = span(x.view(n, 32, 32), 2).sum(1)
    mag = _bits(torch.where(x < 0, -x, x) if signed else x).amax(1)
    nzero, nmin, nmax = (x == 0).sum(1), (x == mn[:, None]).sum(1), (x == mx[:, None]).sum(1)
    raw, cb = 1024.0 * size, _bits(dv - 1)
    f = [bw_f / w, bw_d / w, runs / 1024, bw_i / 16, dv / 1024, torch.log2(dv.double()) / 10, cb / 16, inc / 1023,
         dec / 1023, bw_a / w, maxrun / 1024, torch.log2(1024 / runs.double()) / 10, top / 1024, cnt_top / 1024,
         blk / (32 * w), torch.full_like(dv, width) / 64, torch.full_like(dv, int(signed)),
         (1 + size + 128 * bw_f) / raw, (129 + size + 128 * bw_d) / raw, (runs * size + 131 + 128 * bw_i) / raw,
         (dv * size + 5 + 128 * cb) / raw, (dv * size + 4 * runs + 131 + 128 * bw_i) / raw, mag / w, nzero / 1024,
         dv.double() / runs.double(), torch.log2(maxrun.double()) / 10, _bits(top) / 11, nmin / 1024, nmax / 1024,
         (bw_f.double() - blk.double() / 32) / w, bw_f == 0, dec == 0]
    return torch.stack([v.double() for v in f], 1)


def _sampled(t, signed):
    """Sampled vectors of a column (every STRIDE-th of each 64-vector chunk) as int64 rows, and their chunks."""
    n = t.numel() // 1024
    v = torch.tensor([c + i for c in range(0, n, 64) for i in range(0, min(64, n - c), STRIDE)], device=t.device)
    x = t.view(-1, 1024)[v].long()
    if not signed and t.dtype == torch.int32:
        x = x & 0xFFFFFFFF
    return x, v // 64


def _mlp(p, x):
    shapes, out, at = ((32, 128), (128,), (128, 128), (128,), (128, 6), (6,)), [], 0
    for s in shapes:
        out.append(p[at:at + math.prod(s)].view(s))
        at += math.prod(s)
    w1, b1, w2, b2, w3, b3 = out
    return torch.log_softmax(torch.relu(torch.relu(x @ w1 + b1) @ w2 + b2) @ w3 + b3, 1)


@functools.lru_cache(1)
def _selector_params():
    """A selector's weights: the MLP trained in torch on columns labelled with their family's encoding."""
    xs, ys = [], []
    for seed in range(6):
        for t, signed, fam in _int_columns({"int_columns": 28, "max_vec": 128}, 10_000 + seed):
            x, _ = _sampled(t, signed)
            xs.append(_statistics(x, t.element_size() * 8, signed))
            ys += [FAMILIES[fam]] * x.shape[0]
    x, y = torch.cat(xs), torch.tensor(ys, device=DEV)
    r = np.random.default_rng(5)
    init = [r.normal(size=(i, o)) * math.sqrt(2 / i) if o else np.zeros(i)
            for i, o in ((32, 128), (128, 0), (128, 128), (128, 0), (128, 6), (6, 0))]
    p = torch.from_numpy(np.concatenate([a.reshape(-1) for a in init])).to(DEV).requires_grad_(True)
    opt = torch.optim.Adam([p], lr=2e-3)
    for _ in range(150):
        opt.zero_grad()
        torch.nn.functional.nll_loss(_mlp(p, x), y).backward()
        opt.step()
    return p.detach()


def _exact_learned(case, seed):
    p, conf = _selector_params().float().double(), []
    for t, signed, _ in _int_columns(case, seed):
        x, chunk = _sampled(t, signed)
        lp = _mlp(p, _statistics(x, t.element_size() * 8, signed))
        n = int(chunk[-1]) + 1
        vote = torch.zeros(n, 6, dtype=torch.float64, device=DEV).index_add_(0, chunk, lp)
        prob = torch.zeros(n, 6, dtype=torch.float64, device=DEV).index_add_(0, chunk, lp.exp())
        rows = torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, chunk, torch.ones_like(lp[:, 0]))
        conf.append(prob.gather(1, vote.argmax(1, keepdim=True))[:, 0] / rows)
    return {"choice": None, "conf": torch.cat(conf), "fallback": None}


# ---- exact: the decoded values (plain torch), None where an output is bytes or indexes ---------------------------
def exact(case, seed):
    k = case["kind"]
    if k == "primitive":
        w, op = case["width"], case["op"]
        if op in ("unffor_rsum", "rsum"):
            v = _sorted_values(_gen(seed), case["n_vec"] * 1024, 2.0 ** min(max(case["max_bw"] - 4, 1), 20), 1000)
        else:
            v, _, base = _mixed_width(_gen(seed), w, case["n_vec"], case["max_bw"])
            if op == "unpack":
                v = (v.view(-1, 1024) - base[:, None]).reshape(-1)
        return _narrow(v if case["order"] or op == "untranspose" else _transposed(v), w).view(SIGNED[w])
    if k == "sweep":
        vals = [_mixed_width(_gen(seed, w), w, n, w)[0] for w, n in ((32, case["n32"]), (64, case["n64"]))]
        return [_narrow(v if case["order"] else _transposed(v), w).view(SIGNED[w]) for v, w in zip(vals, (32, 64))]
    if k == "page":
        return _typed(_column(case, seed), case["dtype"])
    if k == "rowgroups":
        return {"ints": [t for t, _, _ in _int_columns(case, seed)], "strs": [[None, None]] * case["str_columns"]}
    if k == "learned":
        return _exact_learned(case, seed)
    if k == "host":
        return {"ok": None, "size": None, "page": None, "back": _typed(_column(case, seed), case["dtype"]).cpu()}
    return None
