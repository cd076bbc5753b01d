"""The performance cases of this repository: what a user of the index has it do.

A case is a dict of plain values; `listed()` gives the fixed ones, `draw(rng)`
one more of the same ranges.  `prepare(case, seed)` makes a user's state on the
GPU (a built tree, a forest plan, query batches), `run(state)` one pass through
the public Python entry points, `work(case)` the bytes a pass cannot do
without, and `exact(case, seed)` the same answers by torch alone.

Kinds of case:
  point    Tree.point_search / point_search_found of a device batch
  count    Tree.range_count
  ids      Tree.range_search (counts, offsets and the sorted hit IDs)
  rect     rect_search over Morton-keyed points
  forest   ForestPlan.run over many uneven trees
  build    Tree.build_unsorted, a first batch of look-ups, close
  train    Tree.learned_train, then a first batch of learned look-ups
"""
import importlib
import math

import numpy as np
import torch

bt = importlib.import_module("b-tree-index-searching_b200")

_INT = {2: torch.int16, 4: torch.int32, 8: torch.int64}
_UINT = {2: torch.uint16, 4: torch.uint32, 8: torch.uint64}


def listed():
    return [
        # one request of a serving process: a small batch on a small table
        dict(name="point_small", kind="point", keys=1_000_003, kb=4, vb=4, queries=1000,
             mode="basic", dist="uniform", found=False),
        # the repository's small configuration: 2^20 keys, 2^20 look-ups, half of them hits
        dict(name="point_l2", kind="point", keys=1 << 20, kb=4, vb=4, queries=1 << 20,
             mode="basic", dist="half", found=False),
        # membership test (value and found flag) with mixed widths and ragged sizes
        dict(name="point_found_odd", kind="point", keys=9_999_991, kb=8, vb=4, queries=1_500_007,
             mode="basic", dist="uniform", found=True),
        # the radix-grouped configuration: skewed look-ups on 2^26 keys
        dict(name="point_grouped_zipf", kind="point", keys=1 << 26, kb=4, vb=4, queries=1 << 24,
             mode="grouped", dist="zipf", found=False),
        # the largest single table: 2^28 64-bit keys, plain search
        dict(name="point_u64", kind="point", keys=1 << 28, kb=8, vb=8, queries=1 << 24,
             mode="basic", dist="uniform", found=False),
        # the headline: the same table through its learned index
        dict(name="point_learned", kind="point", keys=1 << 28, kb=8, vb=8, queries=1 << 24,
             mode="learned", dist="uniform", found=False),
        # range counts in the reference's Z-order grouping
        dict(name="count_zorder", kind="count", keys=1 << 26, kb=4, vb=4, queries=1 << 22,
             mode="zorder", width=64),
        # range look-ups returning row IDs that do not ascend with the keys
        dict(name="ids_shuffled", kind="ids", keys=1 << 24, kb=4, vb=4, queries=1 << 20,
             mode="basic", width=64, shuffled=True),
        # map windows: points of 2^20 boxes with sides up to 256
        dict(name="rect", kind="rect", points=1 << 24, vb=4, boxes=1 << 20, side=256,
             mode="basic"),
        # one batch over 4,096 tables of very different sizes
        dict(name="forest", kind="forest", trees=4096, size_log2=20, batch_log2=16, tile=8192),
        # (re)loading a table from unsorted rows, and its first look-ups
        dict(name="build_unsorted", kind="build", keys=1 << 26, kb=4, vb=4, queries=1 << 22),
        # (re)training the learned index of a table, and its first look-ups
        dict(name="train_learned", kind="train", keys=1 << 26, kb=8, vb=8, queries=1 << 21,
             segments=65536),
    ]


def draw(rng):
    def size(lo, hi):
        n = int(round(2.0 ** rng.uniform(math.log2(lo), math.log2(hi))))
        return n if rng.random() < 0.3 else n | 1

    kind = rng.choice(["point", "point", "point", "count", "ids", "rect", "forest", "build", "train"])
    if kind == "point":
        mode = rng.choice(["basic", "basic", "grouped", "learned"])
        kb = 8 if mode == "learned" else rng.choice([4, 8])
        dist = rng.choice(["uniform", "half", "zipf"])
        cap = 1 << 26 if kb == 4 or dist == "zipf" else 1 << 28
        return dict(kind=kind, keys=size(1 << 14, cap), kb=kb, vb=rng.choice([4, 8]),
                    queries=size(64, 1 << 24), mode=mode, dist=dist,
                    found=rng.random() < 0.25)
    if kind == "count":
        return dict(kind=kind, keys=size(1 << 14, 1 << 26), kb=rng.choice([4, 8]),
                    vb=rng.choice([4, 8]), queries=size(64, 1 << 22),
                    mode=rng.choice(["basic", "2d", "zorder"]), width=size(8, 1024))
    if kind == "ids":
        q = size(64, 1 << 20)
        return dict(kind=kind, keys=size(1 << 16, 1 << 25), kb=rng.choice([4, 8]),
                    vb=rng.choice([4, 8]), queries=q,
                    mode=rng.choice(["basic", "2d", "zorder"]),
                    width=size(8, max(16, min(600, (1 << 26) // q))),
                    shuffled=rng.random() < 0.5)
    if kind == "rect":
        points, boxes = size(1 << 16, 1 << 24), size(64, 1 << 20)
        side = min(1024, int(120000 * math.sqrt((1 << 26) / (boxes * points))))
        return dict(kind=kind, points=points, vb=rng.choice([4, 8]), boxes=boxes,
                    side=size(8, max(16, side)), mode=rng.choice(["basic", "2d", "zorder"]))
    if kind == "forest":
        return dict(kind=kind, trees=size(16, 4096), size_log2=rng.choice([14, 16, 18, 20]),
                    batch_log2=rng.choice([10, 12, 14, 16]), tile=rng.choice([512, 2048, 8192]))
    if kind == "build":
        kb = rng.choice([4, 8])
        return dict(kind=kind, keys=size(1 << 12, 1 << 26 if kb == 4 else 1 << 25), kb=kb,
                    vb=rng.choice([4, 8]), queries=size(1 << 10, 1 << 20))
    n = size(1 << 16, 1 << 26)
    return dict(kind=kind, keys=n, kb=8, vb=rng.choice([4, 8]), queries=size(1 << 10, 1 << 20),
                segments=min(65536, max(64, n >> 10)))


# ------------------------------------------------------------------ inputs


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _ints(hi, n, g):
    """n integers uniform in [0, hi)."""
    return torch.randint(0, hi, (n,), generator=g, device="cuda", dtype=torch.int64)


def _pack(x, nbytes):
    """int64 values as the unsigned type of that width."""
    return x.to(_INT[nbytes]).view(_UINT[nbytes])


def _keys(n, kb, g):
    """n distinct ascending keys: uniform over 32 bits, or 64-bit keys whose
    gaps are lognormal(4, 2)."""
    if kb == 4:
        m = n + n // 16 + 4096
        while True:
            v = torch.unique(_ints(1 << 32, m, g))
            if len(v) >= n:
                break
            m += m // 8
        if len(v) > n:
            keep = torch.ones(len(v), dtype=torch.bool, device="cuda")
            keep[torch.randperm(len(v), generator=g, device="cuda")[: len(v) - n]] = False
            v = v[keep]
        return v
    gap = torch.empty(n, dtype=torch.float64, device="cuda").normal_(4.0, 2.0, generator=g)
    return torch.cumsum(gap.exp_().floor_().to(torch.int64) + 1, 0)


def _queries(keys, m, kb, dist, g):
    """m look-ups: 90% keys (50% for "half"), uniform or Zipf(0.99) over a
    random order of them; the rest uniform over the key range."""
    n = len(keys)
    if dist == "zipf":
        # ranks by the inverse of the continuous distribution function
        # (x^(1-s) - 1) / (n^(1-s) - 1), s = 0.99
        u = torch.rand(m, dtype=torch.float64, generator=g, device="cuda")
        r = (1.0 + u * (float(n + 1) ** 0.01 - 1.0)).pow_(100.0).floor_()
        r = (r.to(torch.int64) - 1).clamp_(0, n - 1)
        r = torch.randperm(n, generator=g, device="cuda")[r]
    else:
        r = _ints(n, m, g)
    miss = torch.rand(m, generator=g, device="cuda") < (0.5 if dist == "half" else 0.1)
    top = 1 << 32 if kb == 4 else int(keys[-1]) + 1
    return torch.where(miss, _ints(top, m, g), keys[r])


def _spread(v):
    for s, k in ((8, 0x00FF00FF), (4, 0x0F0F0F0F), (2, 0x33333333), (1, 0x55555555)):
        v = (v | (v << s)) & k
    return v


def _forest_shape(case):
    """Tree sizes, point batch and range batch of every tree (the case's own,
    whatever the seed)."""
    r = np.random.default_rng([case["trees"], case["size_log2"], case["batch_log2"]])
    t = case["trees"]
    n = np.rint(2.0 ** r.uniform(10, case["size_log2"], size=t)).astype(np.int64)
    q = np.rint(2.0 ** r.uniform(6, case["batch_log2"], size=t)).astype(np.int64)
    return n, q, np.rint(0.01 * q).astype(np.int64)


def _offsets(n):
    return np.concatenate([[0], np.cumsum(n)]).astype(np.uint64)


def _each(n):
    """The tree of every element, for per-tree counts n (on the GPU)."""
    return torch.repeat_interleave(torch.arange(len(n), device="cuda"),
                                   torch.from_numpy(n).to("cuda"))


def _inputs(case, seed):
    """The inputs as int64 tensors."""
    g = _gen(seed)
    kind = case["kind"]
    if kind == "rect":
        # points and boxes of the case, moved and mirrored by the seed, with
        # the seed's own IDs and box order: every seed finds as many points
        n, m, top = case["points"], case["boxes"], 60000
        c = _gen(n)
        x, y = _ints(top, n, c), _ints(top, n, c)
        x0, y0 = _ints(top, m, c), _ints(top, m, c)
        x1 = (x0 + _ints(case["side"], m, c)).clamp_(max=top - 1)
        y1 = (y0 + _ints(case["side"], m, c)).clamp_(max=top - 1)
        p = torch.randperm(m, generator=g, device="cuda")
        x0, y0, x1, y1 = x0[p], y0[p], x1[p], y1[p]
        turn, dx, dy = (int(v) for v in (_ints(2, 1, g), _ints(65536 - top, 1, g),
                                         _ints(65536 - top, 1, g)))
        if turn:
            x, x0, x1 = top - 1 - x, top - 1 - x1, top - 1 - x0
            x, y, x0, y0, x1, y1 = y, x, y0, x0, y1, x1
        z, at = torch.sort(_spread(x + dx) | (_spread(y + dy) << 1))
        ids = torch.randperm(n, generator=g, device="cuda")[at]
        return dict(keys=z, vals=ids, box=(x0 + dx, y0 + dy, x1 + dx, y1 + dy))
    if kind == "forest":
        n, q, nr = _forest_shape(case)
        ko = _offsets(n)
        dn = torch.from_numpy(n).to("cuda")
        t = _each(n)
        gap = torch.rand(len(t), generator=g, device="cuda", dtype=torch.float64)
        gap = (gap * (0xFFFFFFFF // dn)[t]).floor_().to(torch.int64) + 1
        keys = torch.cumsum(gap, 0)
        start = torch.from_numpy(ko[:-1].astype(np.int64)).to("cuda")
        base = torch.where(start > 0, keys[(start - 1).clamp(min=0)], 0)
        keys -= base[t]
        vals = torch.arange(len(t), device="cuda") - start[t]
        del t, gap
        tq, tr = _each(q), _each(nr)
        pick = start[tq] + (torch.rand(len(tq), generator=g, device="cuda", dtype=torch.float64)
                            * dn[tq]).to(torch.int64)
        hit = torch.rand(len(tq), generator=g, device="cuda") < 0.8
        qs = torch.where(hit, keys[pick], _ints(1 << 32, len(tq), g))
        a = (torch.rand(len(tr), generator=g, device="cuda", dtype=torch.float64)
             * dn[tr]).to(torch.int64)
        b = torch.minimum(a + _ints(1 << 12, len(tr), g), dn[tr] - 1)
        return dict(keys=keys, vals=vals, ko=ko, q=qs, qo=_offsets(q), tq=tq, start=start,
                    lo=keys[start[tr] + a], hi=keys[start[tr] + b], ro=_offsets(nr), tr=tr)
    n, kb = case["keys"], case["kb"]
    keys = _keys(n, kb, g)
    if kind == "build":
        order = torch.randperm(n, generator=g, device="cuda")
        return dict(keys=keys, vals=torch.arange(n, device="cuda"), order=order,
                    q=_queries(keys, case["queries"], kb, "uniform", g))
    vals = (torch.randperm(n, generator=g, device="cuda") if case.get("shuffled")
            else torch.arange(n, device="cuda"))
    if kind in ("count", "ids"):
        m, width = case["queries"], case["width"]
        w = _ints(width, m, _gen(m))  # the case's widths, in the seed's order
        w = w[torch.randperm(m, generator=g, device="cuda")]
        a = _ints(n - width, m, g)
        b = a + w
        return dict(keys=keys, vals=vals, lo=keys[a], hi=keys[b])
    q = _queries(keys, case["queries"], kb, case.get("dist", "uniform"), g)
    return dict(keys=keys, vals=vals, q=q)


def _segments(n):
    """Segment target of a user's index: about 4,096 keys a segment."""
    return max(16, n >> 12)


def prepare(case, seed):
    kind, d = case["kind"], _inputs(case, seed)
    s = dict(case=case)
    if kind == "rect":
        s["tree"] = bt.Tree.build(_pack(d["keys"], 4), _pack(d["vals"], case["vb"]))
        s["box"] = [_pack(x, 2) for x in d["box"]]
        return s
    if kind == "forest":
        s["forest"] = bt.Forest(_pack(d["keys"], 4), _pack(d["vals"], 4), d["ko"])
        s["out"] = torch.empty(len(d["q"]), dtype=torch.uint32, device="cuda")
        s["counts"] = torch.empty(len(d["lo"]), dtype=torch.uint64, device="cuda")
        s["plan"] = s["forest"].plan(_pack(d["q"], 4), d["qo"], s["out"], _pack(d["lo"], 4),
                                     _pack(d["hi"], 4), d["ro"], s["counts"],
                                     tile=case["tile"])
        return s
    kb, vb = case["kb"], case["vb"]
    keys, vals = _pack(d["keys"], kb), _pack(d["vals"], vb)
    if kind == "build":
        s["keys"] = _pack(d["keys"][d["order"]], kb)
        s["vals"] = _pack(d["vals"][d["order"]], vb)
        s["q"] = _pack(d["q"], kb)
        return s
    s["tree"] = bt.Tree.build(keys, vals)
    if kind in ("count", "ids"):
        s["lo"], s["hi"] = _pack(d["lo"], kb), _pack(d["hi"], kb)
        return s
    s["q"] = _pack(d["q"], kb)
    if case.get("mode") == "learned":
        s["tree"].learned_train(num_segments=_segments(case["keys"]))
    return s


def _int(x):
    """The signed view of an unsigned tensor (same bits)."""
    return x.view(_INT[x.element_size()])


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "point":
        if case["found"]:
            v, f = state["tree"].point_search_found(state["q"], mode=case["mode"])
            return dict(values=_int(v), found=f)
        return dict(values=_int(state["tree"].point_search(state["q"], mode=case["mode"])))
    if kind == "count":
        c = state["tree"].range_count(state["lo"], state["hi"], mode=case["mode"])
        return dict(counts=_int(c))
    if kind == "ids":
        c, o, i = state["tree"].range_search(state["lo"], state["hi"], mode=case["mode"])
        return dict(counts=_int(c), offsets=_int(o), ids=_int(i))
    if kind == "rect":
        c, o, i = bt.rect_search(state["tree"], *state["box"], mode=case["mode"])
        return dict(counts=_int(c), offsets=_int(o), ids=_int(i))
    if kind == "forest":
        state["plan"].run()
        return dict(values=_int(state["out"]), counts=_int(state["counts"]))
    if kind == "build":
        t = bt.Tree.build_unsorted(state["keys"], state["vals"])
        v = t.point_search(state["q"])
        got = dict(values=_int(v), keys=int(t.info.num_keys), first=int(t.info.min_key),
                   last=int(t.info.max_key), sorted_values=int(t.info.values_sorted))
        t.close()
        return got
    r = state["tree"].learned_train(num_segments=case["segments"])
    v = state["tree"].point_search_learned(state["q"])
    return dict(values=_int(v), segments=r["num_segments"], max_error=r["max_error"],
                eps_max=r["eps_max"], eps_mean=r["eps_mean"], index_bytes=r["index_bytes"],
                loss_initial=r["root_loss_initial"], loss_final=r["root_loss_final"])


def work(case):
    kind = case["kind"]
    if kind == "rect":
        per = case["points"] * ((case["side"] + 1) / 2 / 60000.0) ** 2
        hits = case["boxes"] * per
        return dict(bytes=case["boxes"] * (8 + 16) + hits * (4 + 2 * case["vb"]), flops=0)
    if kind == "forest":
        n, q, r = _forest_shape(case)
        q, r = int(q.sum()), int(r.sum())
        return dict(bytes=q * (4 + 4 + 32 + 0.8 * 32) + r * (8 + 8 + 64), flops=0)
    n, kb, vb, m = case["keys"], case["kb"], case["vb"], case["queries"]
    leaf = n * (kb + vb)
    if kind == "point":
        hit = 0.5 if case["dist"] == "half" else 0.9
        return dict(bytes=m * (kb + vb + int(case["found"])) + min(leaf, m * 32 * (1 + hit)),
                    flops=0)
    if kind == "count":
        return dict(bytes=m * (2 * kb + 8) + min(n * kb, m * 64), flops=0)
    if kind == "ids":
        hits = m * (case["width"] + 1) / 2.0
        return dict(bytes=m * (2 * kb + 16) + min(n * kb, m * 64) + hits * 2 * vb, flops=0)
    if kind == "build":  # rows in, tree out, first look-ups
        return dict(bytes=2 * leaf + m * (kb + vb + 64), flops=0)
    return dict(bytes=n * kb + m * (kb + vb + 64), flops=0)


def _lookup(keys, vals, q):
    p = torch.searchsorted(keys, q).clamp_(max=len(keys) - 1)
    f = keys[p] == q
    return torch.where(f, vals[p], -1), f


def exact(case, seed):
    kind = case["kind"]
    if kind == "rect":
        return None  # a scan of every point for every box
    d = _inputs(case, seed)
    if kind == "forest":
        key = (_each(_forest_shape(case)[0]) << 32) | d["keys"]
        v, _ = _lookup(key, d["vals"], (d["tq"] << 32) | d["q"])
        c = (torch.searchsorted(key, (d["tr"] << 32) | d["hi"], right=True)
             - torch.searchsorted(key, (d["tr"] << 32) | d["lo"]))
        return dict(values=v, counts=c)
    if kind in ("count", "ids"):
        a = torch.searchsorted(d["keys"], d["lo"])
        c = torch.searchsorted(d["keys"], d["hi"], right=True) - a
        if kind == "count":
            return dict(counts=c)
        o = torch.cumsum(c, 0) - c
        seg = torch.repeat_interleave(torch.arange(len(c), device="cuda"), c)
        at = a[seg] + torch.arange(len(seg), device="cuda") - o[seg]
        ids = torch.sort((seg << 32) | d["vals"][at]).values & 0xFFFFFFFF
        return dict(counts=c, offsets=o, ids=ids)
    v, f = _lookup(d["keys"], d["vals"], d["q"])
    if kind == "point":
        return dict(values=v, found=f.to(torch.uint8)) if case["found"] else dict(values=v)
    if kind == "build":
        return dict(values=v, keys=case["keys"], first=int(d["keys"][0]), last=int(d["keys"][-1]),
                    sorted_values=1)
    return dict(values=v, segments=None, max_error=None, eps_max=None, eps_mean=None,
                index_bytes=None, loss_initial=None, loss_final=None)
