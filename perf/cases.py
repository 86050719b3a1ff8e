"""The block-tensor calls that a tensor-network program spends its time in, as
cases to be timed: permutes, eager contractions, captured networks, batches,
grouped sector GEMMs on a caller's own buffers, and the SVD that closes an
iTEBD step; in FP64, split precision and the fast tensor-core modes.

A case is a dict of plain values; its "kind" names the call, the rest the
sizes.  The bond structure of a ragged case comes from its "struct" number,
the elements from the seed that prepare() is given.
"""
import functools
import itertools
import math

import numpy as np
import torch

from trim_gb300 import capi
from trim_gb300 import uni10 as tu
from trim_gb300 import workloads as wl

IN, OUT = wl.IN, wl.OUT


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a user's eager contraction of small U(1) tensors (chi 64): copy,
        # permute, contract; 2 848 elements, so launches and host work count
        dict(name="contract_u1_chi64", kind="u1", scale=1.0, struct=0, mode="fp64"),
        # a dense rank-6 operator reordered, 3 GB moved (chi 24, the MERA operator)
        dict(name="permute_rank6_chi24", kind="permute_dense", rank=6, dim=24, order="450123"),
        # a complex U(1) rank-4 tensor with ragged sectors regrouped
        dict(name="permute_u1_c128", kind="permute_u1", chi=1500, phys=3, struct=7),
        # the contraction half of an iTEBD step, replayed as a CUDA graph
        dict(name="itebd_theta_chi512", kind="itebd", chi=512, mode="fp64"),
        # the other half: per-sector SVD of theta, truncation to chi
        dict(name="itebd_svd_chi512", kind="svd", chi=512),
        # a batch of uneven contractions with persistent operands, replayed
        dict(name="batch64_fp64", kind="batch", n=64, lo=16, hi=256, struct=4004, mode="fp64"),
        # 1024 uneven contractions in one grouped call on the caller's buffers
        dict(name="sectors1024_fp64", kind="sectors", n=1024, lo=16, hi=256, struct=4004, mode="fp64"),
        dict(name="sectors1024_split", kind="sectors", n=1024, lo=16, hi=256, struct=4004, mode="split"),
        # Z2 iPEPS corner quadrant through Network::launch, by precision
        dict(name="ipeps_chi64_D6_fp64", kind="ipeps", chi=64, D=6, mode="fp64"),
        dict(name="ipeps_chi128_D8_split", kind="ipeps", chi=128, D=8, mode="split"),
        dict(name="ipeps_chi128_D8_bf16", kind="ipeps", chi=128, D=8, mode="bf16_tc"),
        # one ascending diagram of the dense ternary MERA (the largest)
        dict(name="mera_left_chi24_split", kind="mera", chi=24, diagram="left", mode="split"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same kinds, its sizes over the whole range."""
    kind = rng.choice(["u1", "permute_dense", "permute_u1", "itebd", "svd", "batch", "sectors", "ipeps", "mera"])
    s = rng.randrange(1, 1 << 20)
    if kind == "u1":
        return dict(kind=kind, scale=round(math.exp(rng.uniform(math.log(0.25), math.log(6.0))), 3), struct=s, mode="fp64")
    if kind == "permute_dense":
        rank = rng.randrange(3, 7)
        dim = _log(rng, 4, int((1.9e8) ** (1.0 / rank)))
        order = list(range(rank))
        while order == sorted(order):
            rng.shuffle(order)
        return dict(kind=kind, rank=rank, dim=dim, order="".join(map(str, order)))
    if kind == "permute_u1":
        return dict(kind=kind, chi=_log(rng, 16, 1500), phys=rng.randrange(2, 4), struct=s)
    if kind == "itebd":
        return dict(kind=kind, chi=_log(rng, 32, 1024), mode="fp64")
    if kind == "svd":
        return dict(kind=kind, chi=_log(rng, 32, 512))
    if kind == "batch":
        return dict(kind=kind, n=_log(rng, 8, 64), lo=16, hi=_log(rng, 48, 256), struct=s, mode=rng.choice(["fp64", "split"]))
    if kind == "sectors":
        return dict(kind=kind, n=_log(rng, 64, 1024), lo=16, hi=_log(rng, 64, 256), struct=s, mode=rng.choice(["fp64", "split"]))
    if kind == "ipeps":
        mode = rng.choice(["fp64", "split", "split", "bf16_tc", "tf32_tc"])
        if mode == "fp64":
            return dict(kind=kind, chi=_log(rng, 16, 72), D=rng.choice([3, 4, 5, 6]), mode=mode)
        return dict(kind=kind, chi=_log(rng, 48, 128), D=rng.choice([4, 5, 6, 7, 8]), mode=mode)
    return dict(kind="mera", chi=_log(rng, 9, 24), diagram=rng.choice(["left", "center", "right"]), mode="split")


# ------------------------------------------------------------------ structure
def _charges(bonds):
    """Block order of the joint index of `bonds`: {charge: flat indices in the
    order a block lists them} -- by run tuple, then by position in the runs."""
    at, per = [], []
    for _, runs in bonds:
        off = 0
        lst = []
        for (u, p, f, d) in runs:
            lst.append(((u, p), off, d))
            off += d
        per.append(lst)
        at.append(off)
    strides = [int(np.prod(at[i + 1:], dtype=np.int64)) for i in range(len(at))]
    out = {}
    for combo in itertools.product(*per):
        u, p = 0, 0
        idx = np.zeros(1, dtype=np.int64)
        for ((cu, cp), off, d), st in zip(combo, strides):
            u, p = u + cu, p ^ cp
            idx = (idx[:, None] + (off + np.arange(d, dtype=np.int64))[None, :] * st).reshape(-1)
        out.setdefault((u, p), []).append(idx)
    return {q: np.concatenate(v) for q, v in out.items()}, int(np.prod(at, dtype=np.int64))


def _layout(bonds):
    """[(charge, row indices, column indices)] in block order, and the dense extents."""
    r, nr = _charges([b for b in bonds if b[0] == IN])
    c, nc = _charges([b for b in bonds if b[0] == OUT])
    return [(q, r[q], c[q]) for q in sorted(r, key=lambda q: q[0] * 4 + q[1] * 2) if q in c], nr, nc


def _dims(bonds):
    return [sum(x[3] for x in runs) for _, runs in bonds]


def _to_dense(bonds, elem):
    lay, nr, nc = _layout(bonds)
    m = torch.zeros(nr, nc, dtype=elem.dtype, device=elem.device)
    off = 0
    for _, r, c in lay:
        ri, ci = torch.from_numpy(r).to(elem.device), torch.from_numpy(c).to(elem.device)
        m[ri[:, None], ci[None, :]] = elem[off:off + r.size * c.size].view(r.size, c.size)
        off += r.size * c.size
    return m.view(_dims([b for b in bonds if b[0] == IN] + [b for b in bonds if b[0] == OUT]))


def _from_dense(bonds, t):
    lay, nr, nc = _layout(bonds)
    m = t.reshape(nr, nc)
    return torch.cat([m[torch.from_numpy(r).to(t.device)[:, None], torch.from_numpy(c).to(t.device)[None, :]].reshape(-1)
                      for _, r, c in lay])


def _product(a, b):
    """(tensor, labels) pairs contracted over their common labels."""
    (x, lx), (y, ly) = a, b
    com = [l for l in lx if l in ly]
    t = torch.tensordot(x, y, dims=([lx.index(l) for l in com], [ly.index(l) for l in com]))
    return t, [l for l in lx if l not in com] + [l for l in ly if l not in com]


def _flops(rows, mid, cols):
    """Multiply-adds x 2 of a contraction's sector products."""
    h = [{q: v for q, v in wl._hist(b).items()} for b in (rows, mid, cols)]
    return 2.0 * sum(h[0][q] * h[1][q] * h[2][q] for q in h[0] if q in h[1] and q in h[2])


@functools.lru_cache(maxsize=8)
def _gauss_degs(chi):
    """chi states over charges -8..8, a discretised Gaussian (sigma 3)."""
    if chi == 512:
        return wl.ITEBD_DEGS
    w = np.exp(-0.5 * (np.arange(-8, 9) / 3.0) ** 2)
    w = w / w.sum() * chi
    d = np.floor(w).astype(int)
    for i in np.argsort(d - w)[: chi - d.sum()]:
        d[i] += 1
    return tuple(int(v) for v in d)


def _bond(t, degs, c0):
    return wl.u1_bond(t, range(c0, c0 + len(degs)), degs)


def _u1(case):
    degs = wl.CHI64_DEGS
    if case["scale"] != 1.0 or case["struct"]:
        r = np.random.default_rng(case["struct"])
        degs = [max(1, int(round(d * case["scale"] * r.uniform(0.7, 1.3)))) for d in degs]
    v = lambda t: _bond(t, degs, -3)  # noqa: E731
    s = lambda t: wl.u1_bond(t, (1, -1), (1, 1))  # noqa: E731
    return [v(IN), s(IN), s(IN), v(OUT)], [v(IN), s(IN), s(OUT), v(OUT)], [v(IN), s(IN), v(OUT), wl.change(s(IN), OUT)]


def _permute_bonds(case):
    """(source bonds, destination bonds, bond order)."""
    if case["kind"] == "permute_dense":
        n, rn = case["rank"], case["rank"] // 2
        order = [int(c) for c in case["order"]]
        src = [wl.dense_bond(IN if i < rn else OUT, case["dim"]) for i in range(n)]
    else:
        rn, order = 2, [0, 2, 1, 3]
        r = np.random.default_rng(case["struct"])
        degs = [wl._dirichlet_degs(r, case["chi"], 7) for _ in range(2)]
        ph = lambda t: wl.u1_bond(t, range(case["phys"]), [1 + i % 2 for i in range(case["phys"])])  # noqa: E731
        src = [_bond(IN, degs[0], -3), ph(IN), ph(OUT), _bond(OUT, degs[1], -3)]
    dst = [wl.change(src[o], IN if i < rn else OUT) for i, o in enumerate(order)]
    return src, dst, order


@functools.lru_cache(maxsize=4)
def _sectors(n, lo, hi, struct):
    """The sector products of n uneven contractions T1[x|y,z] . T2[y,z|w]:
    (M, N, K, a_off, b_off, c_off) and the three buffers' lengths."""
    lst, a, b, c = [], 0, 0, 0
    for t1, t2 in wl.batched(n, lo, hi, struct)["pairs"]:
        x, yz, w = (wl._hist(bs) for bs in (t1.bonds[:1], t1.bonds[1:], t2.bonds[2:]))
        for q in sorted(x):
            if q in yz and q in w:
                lst.append((x[q], w[q], yz[q], a, b, c))
                a, b, c = a + x[q] * yz[q], b + yz[q] * w[q], c + x[q] * w[q]
    return tuple(lst), (a, b, c)


def _pairs(case):
    return wl.batched(case["n"], case["lo"], case["hi"], case["struct"])["pairs"]


def _ipeps(case):
    chi, D = case["chi"], case["D"]
    vD = lambda t: wl.z2_bond(t, D // 2, D - D // 2)  # noqa: E731
    dd = lambda t: wl.combine(t, [vD(IN), vD(OUT)])  # noqa: E731
    c = lambda t: wl.z2_bond(t, chi // 2, chi - chi // 2)  # noqa: E731
    return {"C": ([c(IN), c(OUT)], [1, 2]), "T1": ([c(IN), dd(IN), c(OUT)], [2, 10, 3]),
            "T2": ([c(IN), dd(IN), c(OUT)], [4, 20, 1]), "A2": ([dd(IN), dd(IN), dd(OUT), dd(OUT)], [10, 20, 30, 40])}


def _itebd(case):
    return wl.itebd(_gauss_degs(case["chi"]))


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(n, g):
    return torch.rand(n, generator=g, dtype=torch.float64, device="cuda") * 2 - 1


def _normal(n, g):
    return torch.randn(n, generator=g, dtype=torch.float64, device="cuda")


def _tensor(bonds, labels, elem):
    """A UniTensor holding a device array's elements."""
    t = tu.UniTensor(bonds, labels)
    elem = elem.contiguous()
    torch.cuda.synchronize()
    capi.call("tn_tensor_set_elem_device", t.h, elem.data_ptr(), elem.numel())
    tu.sync()
    return t


class _View:
    """A tensor handle's device elements for torch (no copy)."""

    def __init__(self, t):
        self.t = t
        self.__cuda_array_interface__ = {"shape": (t.elem_num(),), "typestr": "<f8", "data": (t.device_ptr(), False), "version": 2}


def _view(t):
    return torch.as_tensor(_View(t), device="cuda")


def _elems(case, seed):
    """The input elements of a case, by name, on the device."""
    g, k = _gen(seed), case["kind"]
    if k == "u1":
        a, b, _ = _u1(case)
        return {"A": _uniform(wl.elem_count(a), g), "B": _uniform(wl.elem_count(b), g)}
    if k in ("permute_dense", "permute_u1"):
        n = wl.elem_count(_permute_bonds(case)[0])
        x = _uniform(n * (2 if k == "permute_u1" else 1), g)
        return {"x": torch.view_as_complex(x.view(n, 2)) if k == "permute_u1" else x}
    if k in ("itebd", "svd"):
        spec = _itebd(case)
        out = {}
        for s in spec["tensors"]:
            if s.kind == "diag":  # positive, descending in every block
                v = [torch.sort(torch.rand(r, generator=g, dtype=torch.float64, device="cuda") * 0.9 + 0.1, descending=True)[0]
                     for _, r, _ in wl.block_shapes(s.bonds)]
                out[s.name] = torch.cat([torch.diag(d).reshape(-1) for d in v])
            elif s.kind == "given":
                out[s.name] = torch.from_numpy(np.asarray(s.extra["elems"])).cuda()
            else:
                out[s.name] = _uniform(wl.elem_count(s.bonds), g)
        return out
    if k == "batch":
        return {"ab": [(_uniform(wl.elem_count(a.bonds), g), _uniform(wl.elem_count(b.bonds), g)) for a, b in _pairs(case)]}
    if k == "sectors":
        _, (na, nb, _) = _sectors(case["n"], case["lo"], case["hi"], case["struct"])
        return {"a": _uniform(na, g), "b": _uniform(nb, g)}
    if k == "ipeps":
        return {n: _normal(wl.elem_count(b), g) for n, (b, _) in _ipeps(case).items()}
    chi = case["chi"]
    iso = lambda r, c: torch.linalg.qr(_normal(r * c, g).view(r, c))[0].contiguous().view(-1)  # noqa: E731
    w, u = iso(chi ** 3, chi), iso(chi ** 2, chi ** 2)
    o = _normal(chi ** 6, g).view(chi ** 3, chi ** 3)
    o = (o + o.T).mul_(0.5).view(-1)
    return {"W1": w, "W2": w, "U": u, "O": o, "Ud": u, "W1d": w, "W2d": w}


def _itebd_network(case, seed):
    spec, el = _itebd(case), _elems(case, seed)
    net, keep = tu.Network(spec["net"]), []
    for s in spec["tensors"]:
        if s.kind == "diag":  # the Lambdas, as a program builds them: block by block, diagonal
            t = tu.UniTensor(s.bonds, s.labels)
            for q, r, c, d in wl.diag_blocks(s.bonds, el[s.name].cpu().numpy()):
                t.put_block(q, (r, c, d), diag=True)
        else:
            t = _tensor(s.bonds, s.labels, el[s.name])
        net.put_tensor(s.name, t)
        keep.append(t)
    return net, keep


def prepare(case, seed):
    k = case["kind"]
    st = {"kind": k, "mode": case.get("mode")}
    if k == "u1":
        a, b, _ = _u1(case)
        el = _elems(case, seed)
        st.update(a=_tensor(a, [0, 1, 2, 3], el["A"]), b=_tensor(b, [3, 2, 4, 5], el["B"]))
    elif k in ("permute_dense", "permute_u1"):
        src, dst, order = _permute_bonds(case)
        x = _elems(case, seed)["x"]
        st.update(src=tu.SectorMap(src), dst=tu.SectorMap(dst), order=order, x=x, y=torch.empty_like(x))
    elif k in ("itebd", "svd"):
        net, keep = _itebd_network(case, seed)
        if k == "itebd":
            net.capture(case["mode"])
            st.update(net=net, keep=keep, out=_view(net.output()))
        else:
            th = net.launch("fp64")
            blocks, off = th.sector_map().blocks(), [0, 0, 0]
            lst, cnt = [], []
            for _, m, n, a in blocks:
                r = min(m, n)
                lst.append((m, n, a, *off))
                cnt.append(r)
                off = [off[0] + m * r, off[1] + r, off[2] + r * n]
            st.update(theta=th, a=th.device_ptr(), lst=lst, cnt=cnt, chi=case["chi"],
                      usv=[torch.zeros(v, dtype=torch.float64, device="cuda") for v in off])
    elif k == "batch":
        el = _elems(case, seed)["ab"]
        ts = [(_tensor(a.bonds, a.labels, x), _tensor(b.bonds, b.labels, y)) for (a, b), (x, y) in zip(_pairs(case), el)]
        bt = tu.Batch([a for a, _ in ts], [b for _, b in ts])
        bt.capture(case["mode"])
        st.update(batch=bt, out=[_view(bt.output(i)) for i in range(case["n"])])
    elif k == "sectors":
        lst, (_, _, nc) = _sectors(case["n"], case["lo"], case["hi"], case["struct"])
        el = _elems(case, seed)
        st.update(lst=(capi.SectorGemm * len(lst))(*[capi.SectorGemm(*g) for g in lst]), a=el["a"], b=el["b"],
                  c=torch.empty(nc, dtype=torch.float64, device="cuda"), m=capi.MODES[case["mode"]])
    elif k == "ipeps":
        el = _elems(case, seed)
        ts = {n: _tensor(b, l, el[n]) for n, (b, l) in _ipeps(case).items()}
        net = tu.Network(wl.IPEPS_NET)
        for n, t in ts.items():
            net.put_tensor(n, t)
        st.update(net=net, ts=ts)
    else:
        el = _elems(case, seed)
        b = lambda i, o: [wl.dense_bond(IN, case["chi"])] * i + [wl.dense_bond(OUT, case["chi"])] * o  # noqa: E731
        shape = {"W": (3, 1), "U": (2, 2), "O": (3, 3)}
        ts = {n: _tensor(b(*shape[n[0]]), list(range(sum(shape[n[0]]))), e) for n, e in el.items()}
        st.update(net=tu.Network(wl.MERA_NETS[case["diagram"]]), ts=ts)
    tu.sync()
    torch.cuda.synchronize()
    return st


# ------------------------------------------------------------------ one pass
def run(st):
    k = st["kind"]
    if k == "u1":
        p = st["a"].copy()
        p.permute([0, 1, 3, 2], 2)
        c = tu.contract(p, st["b"], fast=True, mode=st["mode"])
        return [_view(p), _view(c)]
    if k == "permute_dense":
        tu.permute_device(st["src"], st["dst"], st["order"], st["x"].data_ptr(), st["y"].data_ptr())
        return st["y"]
    if k == "permute_u1":
        tu.permute_device_c128(st["src"], st["dst"], st["order"], st["x"].data_ptr(), st["y"].data_ptr())
        return st["y"]
    if k == "itebd":
        st["net"].replay()
        return st["out"]
    if k == "svd":
        u, s, vt = st["usv"]
        tu.svd_sectors(st["lst"], st["a"], u.data_ptr(), s.data_ptr(), vt.data_ptr())
        kept, norm = tu.truncate_sectors([g[4] for g in st["lst"]], st["cnt"], s.data_ptr(), st["chi"])
        return [u, s, vt, np.array(kept), norm]
    if k == "batch":
        st["batch"].replay()
        return st["out"]
    if k == "sectors":
        capi.call("tn_contract_sectors", None, st["m"], len(st["lst"]), st["lst"], st["a"].data_ptr(), st["b"].data_ptr(),
                  st["c"].data_ptr())
        return st["c"]
    if k == "mera":
        for n, t in st["ts"].items():
            st["net"].put_tensor(n, t)
    return _view(st["net"].launch(st["mode"]))


# ------------------------------------------------------------------ the work
def work(case):
    k = case["kind"]
    if k == "u1":
        a, b, p = _u1(case)
        n = [wl.elem_count(x) for x in (a, b, p, p[:2] + b[2:])]
        return {"bytes": 8.0 * sum(n), "flops": _flops(p[:2], p[2:], b[2:])}
    if k in ("permute_dense", "permute_u1"):
        return {"bytes": (16.0 if k == "permute_dense" else 32.0) * wl.elem_count(_permute_bonds(case)[0]), "flops": 0}
    if k in ("itebd", "svd"):
        La, A, _, B, _, U = _itebd(case)["tensors"]
        v, s = La.bonds[0], A.bonds[1]
        o = lambda b: wl.change(b, OUT)  # noqa: E731
        theta = wl.elem_count([v, s, o(s), (OUT, v[1])])
        if k == "svd":  # 14 n^3 multiply-adds a block of n, as LAPACK counts an SVD with vectors
            blocks = [r for _, r, _ in wl.block_shapes([v, s, o(s), (OUT, v[1])])]
            return {"bytes": 24.0 * theta, "flops": 14.0 * sum(r ** 3 for r in blocks)}
        n = sum(wl.elem_count(t.bonds) for t in (A, B, U)) + 3 * sum(_dims([v])) + theta
        return {"bytes": 8.0 * n, "flops": _flops([v, s], [v], [wl.change(s, OUT), (OUT, v[1])]) + 2.0 * 2 * theta}
    if k in ("batch", "sectors"):
        lst, n = _sectors(case["n"], case["lo"], case["hi"], case["struct"])
        return {"bytes": 8.0 * sum(n), "flops": 2.0 * sum(m * c * d for m, c, d, *_ in lst)}
    if k == "ipeps":
        b = {n: x for n, (x, _) in _ipeps(case).items()}
        c, dd = b["C"][:1], b["T1"][1:2]
        fl = _flops(c, c, dd + c) + _flops(dd + c, c, c + dd) + _flops(c + c, dd + dd, dd + dd)
        return {"bytes": 8.0 * (sum(wl.elem_count(x) for x in b.values()) + wl.elem_count([c[0], c[0], (OUT, dd[0][1]), (OUT, dd[0][1])])),
                "flops": fl}
    chi = case["chi"]
    big = {"left": 3, "center": 4, "right": 4}[case["diagram"]]  # chi^8 products of its ORDER
    return {"bytes": 8.0 * (chi ** 6 + 6 * chi ** 4 + chi ** 4), "flops": 2.0 * big * chi ** 8}


# ------------------------------------------------------------------ 64 bits
def _theta(case, el):
    t = {}
    for s in _itebd(case)["tensors"]:
        t[s.name] = (_to_dense(s.bonds, el[s.name]), list(s.labels))
    x = t["La"]
    for n in ("A", "Lb", "B", "Lc", "U"):
        x = _product(x, t[n])
    th = x[0].permute([x[1].index(l) for l in (-1, -2, -4, -3)]).contiguous()
    La, A, *_ = _itebd(case)["tensors"]
    v, s = La.bonds[0], A.bonds[1]
    return [v, s, wl.change(s, OUT), (OUT, v[1])], th


def exact(case, seed):
    k, el = case["kind"], _elems(case, seed)
    if k == "u1":
        a, b, p = _u1(case)
        pe = _from_dense(p, _to_dense(a, el["A"]).permute(0, 1, 3, 2).contiguous())
        blocks = lambda bonds, e: dict(zip([q for q, _, _ in _layout(bonds)[0]], _split(bonds, e)))  # noqa: E731
        pa, bb, out = blocks(p, pe), blocks(b, el["B"]), []
        for q, r, c in _layout(p[:2] + b[2:])[0]:
            out.append((pa[q] @ bb[q] if q in pa and q in bb else torch.zeros(r.size, c.size, dtype=torch.float64, device="cuda")).reshape(-1))
        return [pe, torch.cat(out)]
    if k in ("permute_dense", "permute_u1"):
        src, dst, order = _permute_bonds(case)
        if k == "permute_dense":
            return el["x"].view(_dims(src)).permute(order).contiguous().view(-1)
        return _from_dense(dst, _to_dense(src, el["x"]).permute(order).contiguous())
    if k == "itebd":
        return _from_dense(*_theta(case, el))
    if k == "svd":
        bonds, th = _theta(case, el)
        sv = [torch.linalg.svdvals(m) for m in _split(bonds, _from_dense(bonds, th))]
        cut = torch.sort(torch.cat(sv), descending=True)[0][: case["chi"]]
        norm = torch.linalg.norm(cut)
        return [None, torch.cat([torch.where(v >= cut[-1], v / norm, v) for v in sv]), None,
                np.array([int((v >= cut[-1]).sum()) for v in sv]), float(norm)]
    if k == "batch":
        out = []
        for (a, b), (x, y) in zip(_pairs(case), el["ab"]):
            m = _to_dense(a.bonds, x).reshape(_dims(a.bonds)[0], -1) @ _to_dense(b.bonds, y).reshape(-1, _dims(b.bonds)[2])
            out.append(_from_dense([a.bonds[0], b.bonds[2]], m))
        return out
    if k == "sectors":
        lst, _ = _sectors(case["n"], case["lo"], case["hi"], case["struct"])
        return torch.cat([(el["a"][a:a + m * d].view(m, d) @ el["b"][b:b + d * n].view(d, n)).reshape(-1) for m, n, d, a, b, _ in lst])
    if k == "ipeps":
        spec = _ipeps(case)
        t = {n: (_to_dense(b, el[n]), l) for n, (b, l) in spec.items()}
        x = _product(_product(_product(t["C"], t["T1"]), t["T2"]), t["A2"])
        th = x[0].permute([x[1].index(l) for l in (3, 4, 30, 40)]).contiguous()
        c, dd = spec["C"][0][0], spec["T1"][0][1]
        return _from_dense([c, c, (OUT, dd[1]), (OUT, dd[1])], th)
    text = dict(line.split(":", 1) for line in wl.MERA_NETS[case["diagram"]].strip().splitlines())
    label = lambda n: [int(v) for v in text[n].replace(";", " ").split()]  # noqa: E731
    env = {n: (e.view([case["chi"]] * len(label(n))), label(n)) for n, e in el.items()}
    x = _bracket(text["ORDER"].replace("(", " ( ").replace(")", " ) ").split(), env)
    return x[0].permute([x[1].index(l) for l in label("TOUT")]).contiguous().view(-1)


def _split(bonds, e):
    out, off = [], 0
    for _, r, c in _layout(bonds)[0]:
        out.append(e[off:off + r.size * c.size].view(r.size, c.size))
        off += r.size * c.size
    return out


def _bracket(tok, env):
    """A pair tree in brackets, contracted in its order."""
    stack = []
    for w in tok:
        if w == "(":
            stack.append(w)
        elif w == ")":
            b, a = stack.pop(), stack.pop()
            stack.pop()
            stack.append(_product(a, b))
        else:
            stack.append(env[w])
    return stack[0]
