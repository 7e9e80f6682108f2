"""Performance cases: the calls a program makes on one process's share of a
tensor contraction or coupled-cluster iteration, through the package's public
entry points.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges,
``prepare(case, seed)`` makes what the program holds before the call,
``run(state)`` is one pass, ``work(case)`` the bytes and operations a pass
cannot do without, and ``exact(case, seed)`` the same outputs from plain torch
in 64 bits.
"""
import ctypes
import itertools
import math
import random

import numpy as np
import torch

from dtcf_gb300 import cc, dltc, leaves, rrr
from dtcf_gb300._lib import check, lib


def listed():
    return [
        # one 8^4 block permuted: the call DTCF's per-block loop makes, where latency counts
        dict(name="transpose_block", kind="transpose", widths="8,8,8,8", perm="2,3,0,1"),
        # a dense amplitude-sized tensor reordered once (ragged extents, no index keeps its place)
        dict(name="transpose_dense", kind="transpose", widths="47,53,61,39", perm="2,0,3,1"),
        # every block of an operand permuted in one call, each with the permutation its un-flip needs
        dict(name="transpose_blocks", kind="blocks", count=2000, widths="8,8,8,8", layout=1),
        # all 1296 blocks of a 48^4 integral tensor packed into the big matrix and unpacked again
        dict(name="big_matrix", kind="bigmatrix", vgrid="6,6,6,6", rpb=64, cpb=64, rows=2, layout=2),
        # one block pair's product: the small dgemm of the block loops
        dict(name="gemm_block", kind="gemm", m=64, n=48, k=96, at=0, bt=1),
        # a packed operand pair's product, ragged, A and B stored the other way round
        dict(name="gemm_packed", kind="gemm", m=1021, n=765, k=1531, at=1, bt=0),
        # the particle ladder over unique blocks, o = 16, v = 48, block 8, FP64
        dict(name="ladder_fp64", kind="plan", form="ladder", o=16, v=48, block=8, mode="fp64", slices=0),
        # the same at o = 32, v = 128, block 16 on the split engine
        dict(name="ladder_split", kind="plan", form="ladder", o=32, v=128, block=16, mode="split", slices=6),
        # block triples of mixed shapes (8 to 256) planned as one batch
        dict(name="triples", kind="group", count=2000, mode=2, layout=3),
        # the CCD-T2 residual table as a program over dense tensors
        dict(name="residual_ccd", kind="residual", O=12, V=36, wbO=4, wbV=6, mode="fp64"),
        # CCSD iterations of a small molecule's job, FP64, kernel graph: launches and latency
        dict(name="ccsd_small", kind="cc", o=8, v=24, nirrep=1, max_block=16, min_block=1, method="ccsd",
             engine="fp64", slices=0, graph=1, niter=4, molecule=1),
        # CCSD iterations with 8 irreps and uneven blocks at o = 48, v = 240 on the split engine
        dict(name="ccsd_large", kind="cc", o=48, v=240, nirrep=8, max_block=40, min_block=4, method="ccsd",
             engine="split", slices=4, graph=2, niter=4, molecule=1),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["transpose", "blocks", "bigmatrix", "gemm", "plan", "group", "residual", "cc"])
    if kind == "transpose":
        rank = rng.choice([2, 3, 4, 4, 4, 5, 6])
        total = _log(rng, 512, 6000000)
        w = [max(2, int(round(total ** (1.0 / rank) * rng.uniform(0.6, 1.6)))) for _ in range(rank)]
        p = list(range(rank))
        rng.shuffle(p)
        return dict(kind=kind, widths=",".join(map(str, w)), perm=",".join(map(str, p)))
    if kind == "blocks":
        w = [rng.randint(3, 16) for _ in range(4)]
        count = _log(rng, 2, max(2, min(4000, 8000000 // math.prod(w))))
        return dict(kind=kind, count=count, widths="%d,%d,%d,%d" % (w[0], w[0], w[2], w[2]), layout=rng.randint(1, 999))
    if kind == "bigmatrix":
        g = [rng.randint(1, 6) for _ in range(4)]
        return dict(kind=kind, vgrid=",".join(map(str, g)), rpb=rng.randint(9, 100), cpb=rng.randint(9, 64), rows=2,
                    layout=rng.randint(1, 999))
    if kind == "gemm":
        while True:
            m, n, k = (_log(rng, 1, 2000) for _ in range(3))
            if m * n * k <= 1.2e9 and m * n <= 2000000 and max(m, n) * k <= 3000000:
                return dict(kind=kind, m=m, n=n, k=k, at=rng.randint(0, 1), bt=rng.randint(0, 1))
    if kind == "plan":
        mode = rng.choice(["fp64", "split"])
        b = rng.randint(5, 10)
        nv = rng.randint(2, 6) if mode == "fp64" else rng.randint(4, 8)
        return dict(kind=kind, form=rng.choice(["ladder", "ring", "fock"]), o=b * rng.randint(1, 2), v=b * nv, block=b,
                    mode=mode, slices=0 if mode == "fp64" else rng.randint(4, 7))
    if kind == "group":
        return dict(kind=kind, count=_log(rng, 10, 2000), mode=rng.randint(0, 2), layout=rng.randint(1, 999))
    if kind == "residual":
        wo, wv = rng.randint(2, 4), rng.randint(3, 7)
        return dict(kind=kind, O=wo * rng.randint(2, 3), V=wv * rng.randint(2, 5), wbO=wo, wbV=wv,
                    mode=rng.choice(["fp64", "split"]))
    o = rng.randint(6, 16)
    return dict(kind=kind, o=o, v=int(o * rng.uniform(2.5, 4)), nirrep=rng.choice([1, 1, 2, 4, 8]),
                max_block=rng.randint(5, 16), min_block=1, method=rng.choice(["ccd", "ccsd"]),
                engine=rng.choice(["fp64", "split"]), slices=rng.randint(4, 6), graph=rng.randint(1, 2), niter=4,
                molecule=rng.randint(1, 9))


def _ints(text):
    return [int(x) for x in text.split(",")]


class _Gen:
    """Seeded device values: uniform in (-1, 1), or sign * 10^u with u in [-6, 6)."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(seed)

    def uniform(self, n):
        return torch.rand(n, generator=self.g, device="cuda", dtype=torch.float64) * 2 - 1

    def graded(self, n):
        x = self.uniform(n)
        u = torch.rand(n, generator=self.g, device="cuda", dtype=torch.float64) * 12 - 6
        return torch.where(x < 0, -1.0, 1.0).double() * torch.pow(10.0, u)


# ---- permutes and packs ------------------------------------------------------


def _inverse(p):
    q = [0] * len(p)
    for i, x in enumerate(p):
        q[x] = i
    return q


def _block_perms(case):
    """Each block's permutation: the operand's, after the un-flip of either index pair."""
    rng = random.Random(case["layout"])
    base = [2, 3, 0, 1]
    out = []
    for _ in range(case["count"]):
        p = list(base)
        if rng.random() < 0.5:
            p[0], p[1] = p[1], p[0]
        if rng.random() < 0.5:
            p[2], p[3] = p[3], p[2]
        out.append(p)
    return out


def _pack_layout(case):
    """The blocks' permuted addresses in stored order: every block of the grid, shuffled."""
    g = _ints(case["vgrid"])
    addr = list(itertools.product(*[range(x) for x in g]))
    random.Random(case["layout"]).shuffle(addr)
    return g, addr


def _pack_exact(case, tiles):
    g, addr = _pack_layout(case)
    r, c, nr = case["rpb"], case["cpb"], case["rows"]
    rows = list(itertools.product(*[range(x) for x in g[:nr]]))
    cols = list(itertools.product(*[range(x) for x in g[nr:]]))
    big = torch.empty(len(rows), len(cols), r, c, dtype=torch.float64, device=tiles.device)
    ri = torch.tensor([rows.index(a[:nr]) for a in addr], device=tiles.device)
    ci = torch.tensor([cols.index(a[nr:]) for a in addr], device=tiles.device)
    big[ri, ci] = tiles.view(-1, r, c)
    return big.permute(0, 2, 1, 3).reshape(-1)


# ---- contractions over unique blocks -----------------------------------------

# (symmetry string, spaces, index string) of A, B and C
FORMS = {
    "ladder": (("aabb", "vvvv", "a,b,e,f"), ("aabb", "vvoo", "e,f,i,j"), ("aabb", "vvoo", "a,b,i,j")),
    "ring": (("cccc", "vovo", "a,i,e,m"), ("cccc", "vovo", "e,m,b,j"), ("cccc", "vovo", "a,i,b,j")),
    "fock": (("cc", "vv", "a,e"), ("ccbb", "vvoo", "e,b,i,j"), ("ccbb", "vvoo", "a,b,i,j")),
}


def _plan_tensors(case):
    out = []
    for sym, spaces, _ in FORMS[case["form"]]:
        size = [case["o"] if s == "o" else case["v"] for s in spaces]
        out.append(rrr.Tensor(sym, size, [s // case["block"] for s in size]))
    return out


def _unique(sym, grid):
    """Stored block addresses: coordinates not increasing inside a symmetry group, lexicographic."""
    out = []
    for c in itertools.product(*[range(x) for x in grid]):
        if all(c[i] >= c[j] for i in range(len(c)) for j in range(i + 1, len(c))
               if sym[i] == sym[j] and sym[i] in "ab"):
            out.append(c)
    return out


def _dense(case, which, tiles):
    """The dense antisymmetric tensor that the stored blocks stand for."""
    sym, spaces, _ = FORMS[case["form"]][which]
    b = case["block"]
    grid = [(case["o"] if s == "o" else case["v"]) // b for s in spaces]
    r = len(grid)
    D = torch.zeros(grid + [b] * r, dtype=torch.float64, device=tiles.device)
    pairs = [[d for d in range(r) if sym[d] == x] for x in "ab" if sym.count(x) == 2]
    for t, c in zip(tiles.view([-1] + [b] * r), _unique(sym, grid)):
        for flips in itertools.product([0, 1], repeat=len(pairs)):
            p, sign, skip = list(range(r)), 1.0, False
            for f, (i, j) in zip(flips, pairs):
                if f:
                    skip = skip or c[i] == c[j]
                    p[i], p[j], sign = p[j], p[i], -sign
            if not skip:
                D[tuple(c[x] for x in p)] = sign * t.permute(p)
    return D.permute([x for d in range(r) for x in (d, r + d)]).reshape([x * b for x in grid])


def _stored(case, D):
    sym, spaces, _ = FORMS[case["form"]][2]
    b, r = case["block"], len(spaces)
    grid = [s // b for s in D.shape]
    B = D.reshape([x for g in grid for x in (g, b)]).permute([2 * d for d in range(r)] + [2 * d + 1 for d in range(r)])
    return torch.stack([B[c] for c in _unique(sym, grid)]).reshape(-1)


def _triple_dims(case):
    rng = np.random.default_rng(case["layout"])
    return np.exp(rng.uniform(np.log(8), np.log(256), size=(case["count"], 3))).round().astype(np.int64)


# ---- the CCD-T2 residual ------------------------------------------------------

# tensor, spaces (h hole, p particle); the inputs a program fills
CCD_INPUTS = {"F_OO": "hh", "F_VV": "pp", "T_VVOO": "pphh", "V_OOOO": "hhhh", "V_VVOO": "pphh", "V_OOVV": "hhpp",
              "V_OVOV": "hphp", "V_VVVV": "pppp"}
CCD_RESULTS = ["R_VVOO", "I_OO", "I_VV", "I_OOOO", "I_OVOV"]


def _ccd_exact(x):
    T, e = x["T_VVOO"], torch.einsum
    out = {
        "I_OO": x["F_OO"] + e("pqlm,nmpq->nl", T, x["V_OOVV"]),
        "I_VV": x["F_VV"] + e("prmn,mnqr->pq", T, x["V_OOVV"]),
        "I_OOOO": x["V_OOOO"] + e("pqij,mnpq->mnij", T, x["V_OOVV"]),
        "I_OVOV": x["V_OVOV"] + e("prim,nmqr->npiq", T, x["V_OOVV"]),
    }
    out["R_VVOO"] = (x["V_VVOO"] + e("pqij,rspq->rsij", T, x["V_VVVV"]) + e("abik,kj->abij", T, out["I_OO"])
                     + e("acij,bc->abij", T, out["I_VV"]) + e("abmn,mnij->abij", T, out["I_OOOO"])
                     + e("acim,mbjc->abij", T, out["I_OVOV"]))
    return [out[n].reshape(-1) for n in CCD_RESULTS]


# ---- coupled-cluster jobs -------------------------------------------------------


def _cc_save(job, t1, t2):
    check(lib().gbx_cc_save_amplitudes(job.handle, ctypes.c_void_p(t1.data_ptr()) if t1 is not None else None,
                                       ctypes.c_void_p(t2.data_ptr()),
                                       ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))


def _cc_start(seed):
    """The amplitudes a program resumes from: the guess, damped or enlarged (any factor keeps its antisymmetry)."""
    return random.Random(seed).uniform(0.7, 1.3)


_M64 = (1 << 64) - 1


def _mix(z):
    z ^= z >> 30
    z = z * 0xBF58476D1CE4E5B9 & _M64
    z ^= z >> 27
    z = z * 0x94D049BB133111EB & _M64
    return z ^ (z >> 31)


def _numbers(seed, stream):
    s = _mix((seed ^ (0x9E3779B97F4A7C15 * (stream + 1))) & _M64)
    while True:
        s = (s + 0x9E3779B97F4A7C15) & _M64
        yield _mix(s)


def _cc_system(case, seed):
    """Orbital energies and dense <pq||rs> of the synthetic job without spatial symmetry."""
    o, v = case["o"], case["v"]
    n = o + v
    so, sv = _numbers(seed, 3), _numbers(seed, 4)
    eo = np.array([-2.0 + 1.5 * ((next(so) >> 11) * 2.0 ** -53) for _ in range(o)])
    ev = np.array([0.2 + 2.8 * ((next(sv) >> 11) * 2.0 ** -53) for _ in range(v)])
    p, q, r, s = np.meshgrid(*[np.arange(n, dtype=np.uint64)] * 4, indexing="ij")
    x, y = np.minimum(p, q) * np.uint64(n) + np.maximum(p, q), np.minimum(r, s) * np.uint64(n) + np.maximum(r, s)
    with np.errstate(over="ignore"):
        z = np.minimum(x, y) * np.uint64(0x9E3779B97F4A7C15) + np.maximum(x, y) * np.uint64(0xC2B2AE3D27D4EB4F)
        z ^= np.uint64(next(_numbers(seed, 5)))
        z ^= z >> np.uint64(30)
        z *= np.uint64(0xBF58476D1CE4E5B9)
        z ^= z >> np.uint64(27)
        z *= np.uint64(0x94D049BB133111EB)
        z ^= z >> np.uint64(31)
    i = [a.astype(np.int64) for a in (p, q, r, s)]
    V = 1e-2 * np.exp(-(np.abs(i[0] - i[1]) + np.abs(i[2] - i[3])) / 8.0) * np.where(z >> np.uint64(63), -1.0, 1.0)
    return eo, ev, torch.from_numpy(V * np.sign(i[1] - i[0]) * np.sign(i[3] - i[2]))


def _cc_exact(case, seed):
    """The amplitudes after the case's Jacobi iterations from the scaled MP2 guess: the spin-orbital CCSD equations
    of Stanton, Gauss, Watts and Bartlett, J. Chem. Phys. 94, 4334 (1991); CCD is their t1 = 0."""
    o = case["o"]
    eo, ev, V = _cc_system(case, case["molecule"])
    V = V.cuda()
    f = {c: (slice(0, o) if c in "ijklmn" else slice(o, None)) for c in "ijklmnabef"}

    def I(names):  # noqa: E743
        return V[tuple(f[c] for c in names)]

    e = torch.einsum
    eo, ev = torch.from_numpy(eo).cuda(), torch.from_numpy(ev).cuda()
    d1 = eo[:, None] - ev
    d2 = d1[:, None, :, None] + d1[None, :, None, :]
    oovv = I("ijab")
    t1, t2 = torch.zeros_like(d1), oovv / d2 * _cc_start(seed)

    def pij(x):
        return x - x.transpose(0, 1)

    def pab(x):
        return x - x.transpose(2, 3)

    for _ in range(case["niter"]):
        tt = pij(e("ia,jb->ijab", t1, t1))
        tau, taut = t2 + tt, t2 + tt / 2
        Fae = e("mf,mafe->ae", t1, I("mafe")) - e("mnaf,mnef->ae", taut, oovv) / 2
        Fmi = e("ne,mnie->mi", t1, I("mnie")) + e("inef,mnef->mi", taut, oovv) / 2
        Fme = e("nf,mnef->me", t1, oovv)
        Wo = I("mnij") + pab(e("je,mnie->mnij", t1, I("mnie"))) + e("ijef,mnef->mnij", tau, oovv) / 4
        Wv = I("abef") - pij(e("mb,amef->abef", t1, I("amef"))) + e("mnab,mnef->abef", tau, oovv) / 4
        Wr = (I("mbej") + e("jf,mbef->mbej", t1, I("mbef")) - e("nb,mnej->mbej", t1, I("mnej"))
              - e("jnfb,mnef->mbej", t2 / 2 + e("jf,nb->jnfb", t1, t1), oovv))
        R1 = (e("ie,ae->ia", t1, Fae) - e("ma,mi->ia", t1, Fmi) + e("imae,me->ia", t2, Fme)
              - e("nf,naif->ia", t1, I("naif")) - e("imef,maef->ia", t2, I("maef")) / 2
              - e("mnae,nmei->ia", t2, I("nmei")) / 2)
        Fbe, Fmj = Fae - e("mb,me->be", t1, Fme) / 2, Fmi + e("je,me->mj", t1, Fme) / 2
        R2 = (oovv + pab(e("ijae,be->ijab", t2, Fbe)) - pij(e("imab,mj->ijab", t2, Fmj))
              + e("mnab,mnij->ijab", tau, Wo) / 2 + e("ijef,abef->ijab", tau, Wv) / 2
              + pij(pab(e("imae,mbej->ijab", t2, Wr) - e("ie,ma,mbej->ijab", t1, t1, I("mbej"))))
              + pij(e("ie,abej->ijab", t1, I("abej"))) - pab(e("ma,mbij->ijab", t1, I("mbij"))))
        if case["method"] == "ccsd":
            t1 = R1 / d1
        t2 = R2 / d2
    return [_tiles(t1, case), _tiles(t2, case)] if case["method"] == "ccsd" else [_tiles(t2, case)]


def _tiles(t, case):
    """A dense amplitude tensor in the job's tile order: blocks as even as possible, of at most max_block orbitals."""
    cuts = []
    for n in t.shape:
        nb = -(-n // case["max_block"])
        ext = [n // nb + (1 if k < n % nb else 0) for k in range(nb)]
        cuts.append([slice(sum(ext[:k]), sum(ext[:k + 1])) for k in range(nb)])
    return torch.cat([t[c].reshape(-1) for c in itertools.product(*cuts)]).cpu()


# ---- the cases ---------------------------------------------------------------------


def prepare(case, seed):
    g, k = _Gen(seed), case["kind"]
    s = dict(case=case)
    if k == "transpose":
        w = _ints(case["widths"])
        x = g.uniform(math.prod(w))
        s.update(x=x, y=torch.empty_like(x), w=w, p=_ints(case["perm"]))
    elif k == "blocks":
        w = _ints(case["widths"])
        x = g.uniform(case["count"] * math.prod(w))
        s.update(x=x, y=torch.empty_like(x), w=w, p=np.array(_block_perms(case), dtype=np.int32))
    elif k == "bigmatrix":
        grid, addr = _pack_layout(case)
        x = g.uniform(len(addr) * case["rpb"] * case["cpb"])
        s.update(x=x, big=torch.empty_like(x), back=torch.empty_like(x), grid=grid, addr=np.array(addr, dtype=np.int32))
    elif k == "gemm":
        m, n, kk = case["m"], case["n"], case["k"]
        s.update(A=g.uniform(m * kk), B=g.uniform(n * kk), C=g.uniform(m * n))
    elif k == "plan":
        A, B, C = _plan_tensors(case)
        for t in (A, B, C):
            t.tiles.copy_(g.uniform(t.tiles.numel()))
        c = rrr.Contraction(A, B, C, mode=case["mode"], sign=-1, slices=case["slices"])
        idx = [f[2] for f in FORMS[case["form"]]]
        c.plan(*idx)
        s.update(c=c, idx=idx)
    elif k == "group":
        d = _triple_dims(case)
        oa, ob, oc = (np.concatenate([[0], np.cumsum(d[:, i] * d[:, j])]) for i, j in ((0, 2), (1, 2), (0, 1)))
        A, B = g.graded(int(oa[-1])), g.graded(int(ob[-1]))
        C = torch.zeros(int(oc[-1]), dtype=torch.float64, device="cuda")
        tri = [leaves.Triple(A.data_ptr() + 8 * int(a), B.data_ptr() + 8 * int(b), C.data_ptr() + 8 * int(c), int(z), 1,
                             int(z), 1, int(y), int(x), int(y), int(z), 1.0, 0)
               for (x, y, z), a, b, c in zip(d, oa, ob, oc)]
        s.update(A=A, B=B, C=C, group=leaves.Group(tri, mode=case["mode"]))
    elif k == "residual":
        prog = dltc.Program("ccd_t2", dltc.dims(case["O"], case["V"], case["wbO"], case["wbV"]), mode=case["mode"])
        at = {name: i for i, (name, _) in enumerate(prog.table["tensors"])}
        for name in CCD_INPUTS:
            t = prog.tensor(at[name])
            t.copy_(g.uniform(t.numel()))
        made = [prog.tensor(at[name]) for name in CCD_RESULTS]  # the program's own memory, gone with it
        s.update(prog=prog, made=made, out=[torch.empty_like(t) for t in made])
    else:
        job = cc.Job(nocc=case["o"], nvir=case["v"], nirrep=case["nirrep"], max_block=case["max_block"],
                     min_block=case["min_block"], method=case["method"], engine=case["engine"], slices=case["slices"],
                     use_graph=case["graph"], seed=case["molecule"])
        n1, n2 = job.amplitude_elems()
        pin = [torch.zeros(n, dtype=torch.float64).pin_memory() if n else None for n in (n1, n2, n1, n2)]
        _cc_save(job, pin[0], pin[1])  # the guess the job starts from
        torch.cuda.current_stream().synchronize()
        pin[1].mul_(_cc_start(seed))
        s.update(job=job, start=pin[:2], out=pin[2:])
    return s


def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "transpose":
        return leaves.transpose(s["x"], s["y"], s["p"], s["w"])
    if k == "blocks":
        return leaves.transpose_blocks(s["x"], s["y"], s["p"], s["w"])
    if k == "bigmatrix":
        p = list(range(len(s["grid"])))
        leaves.create_big_matrix(s["grid"], p, s["x"], s["addr"], case["rpb"], case["cpb"], case["rows"], s["big"])
        leaves.revert_big_matrix(s["grid"], p, s["addr"], case["rpb"], case["cpb"], case["rows"], s["big"], s["back"])
        return [s["big"], s["back"]]
    if k == "gemm":
        return leaves.local_contraction(case["m"], case["n"], case["k"], s["A"], s["B"], s["C"], case["at"], case["bt"],
                                        0.5)
    if k == "plan":
        return s["c"].contract(*s["idx"], alpha=0.5).tiles
    if k == "group":
        s["group"].execute()
        return s["C"]
    if k == "residual":
        for t in s["made"]:
            t.zero_()
        s["prog"].run()
        for t, r in zip(s["made"], s["out"]):
            r.copy_(t)
        return s["out"]
    # a step of a longer run: the amplitudes come from the host, some iterations, and they go back
    job, start, out = s["job"], s["start"], s["out"]
    job.set_amplitudes(start[0].data_ptr() if start[0] is not None else 0, start[1].data_ptr())
    job.enqueue(case["niter"])
    _cc_save(job, out[0], out[1])
    return [t for t in out if t is not None]


def work(case):
    k = case["kind"]
    if k == "transpose":
        return {"bytes": 16 * math.prod(_ints(case["widths"])), "flops": 0}
    if k == "blocks":
        return {"bytes": 16 * case["count"] * math.prod(_ints(case["widths"])), "flops": 0}
    if k == "bigmatrix":
        return {"bytes": 32 * math.prod(_ints(case["vgrid"])) * case["rpb"] * case["cpb"], "flops": 0}
    if k == "gemm":
        m, n, kk = case["m"], case["n"], case["k"]
        return {"bytes": 8 * (m * kk + n * kk + 2 * m * n), "flops": 2 * m * n * kk}
    if k == "plan":
        size, total = [], 0
        for sym, spaces, _ in FORMS[case["form"]]:
            grid = [(case["o"] if s == "o" else case["v"]) // case["block"] for s in spaces]
            n = 1
            for x in sorted(set(sym)):
                d = [grid[i] for i in range(len(sym)) if sym[i] == x]
                n *= d[0] * (d[0] + 1) // 2 if x in "ab" and len(d) == 2 else math.prod(d)
            size.append(n * case["block"] ** len(spaces))
        total = 8 * (size[0] + size[1] + 2 * size[2])
        o, v = case["o"], case["v"]
        return {"bytes": total, "flops": 2 * size[2] * {"ladder": v * v, "ring": v * o, "fock": v}[case["form"]]}
    if k == "group":
        d = _triple_dims(case).astype(float)
        return {"bytes": float(8 * np.sum(d[:, 0] * d[:, 2] + d[:, 1] * d[:, 2] + d[:, 0] * d[:, 1])),
                "flops": float(2 * np.sum(d[:, 0] * d[:, 1] * d[:, 2]))}
    if k == "residual":
        O, V = case["O"], case["V"]
        n = sum(math.prod([O if c == "h" else V for c in sp]) for sp in CCD_INPUTS.values())
        n += O * O * V * V + O * O + V * V + O ** 4 + O * O * V * V
        return {"bytes": 8 * n, "flops": 2 * (O ** 2 * V ** 4 + 2 * O ** 4 * V ** 2 + 2 * O ** 3 * V ** 3
                                              + 2 * O ** 3 * V ** 2 + 2 * O ** 2 * V ** 3)}
    # the antisymmetric unique parts of the ladder, the rings and W_mnij; the unique integrals and the amplitudes
    o, v, h, sd = case["o"], case["v"], case["nirrep"], case["method"] == "ccsd"
    flops = (o * o * v ** 4 / 4 + 4 * o ** 3 * v ** 3 + (o ** 3 * v ** 3 if sd else 0) + o ** 4 * v * v / 2) / h
    ints = (v ** 4 / 8 + o ** 2 * v ** 2 * 1.25 + o ** 4 / 8 + ((o * v ** 3 + o ** 3 * v) / 2 if sd else 0)) / h
    return {"bytes": 8 * case["niter"] * (ints + o * o * v * v / 2 / h), "flops": case["niter"] * flops}


def exact(case, seed):
    g, k = _Gen(seed), case["kind"]
    if k == "transpose":
        w, p = _ints(case["widths"]), _ints(case["perm"])
        return g.uniform(math.prod(w)).view(w).permute(_inverse(p)).reshape(-1)
    if k == "blocks":
        w = _ints(case["widths"])
        x = g.uniform(case["count"] * math.prod(w)).view([-1] + w)
        return torch.cat([t.permute(_inverse(p)).reshape(-1) for t, p in zip(x, _block_perms(case))])
    if k == "bigmatrix":
        x = g.uniform(math.prod(_ints(case["vgrid"])) * case["rpb"] * case["cpb"])
        return [_pack_exact(case, x), x]
    if k == "gemm":
        m, n, kk = case["m"], case["n"], case["k"]
        A, B, C = g.uniform(m * kk), g.uniform(n * kk), g.uniform(m * n)
        A = A.view(kk, m).T if case["at"] else A.view(m, kk)
        B = B.view(n, kk).T if case["bt"] else B.view(kk, n)
        return (C.view(m, n) + 0.5 * (A @ B)).reshape(-1)
    if k == "plan":
        sizes = [len(_unique(sym, [(case["o"] if s == "o" else case["v"]) // case["block"] for s in spaces]))
                 * case["block"] ** len(spaces) for sym, spaces, _ in FORMS[case["form"]]]
        tiles = [g.uniform(n) for n in sizes]
        A, B, C = (_dense(case, i, t) for i, t in enumerate(tiles))
        ia, ib, ic = (f[2].replace(",", "") for f in FORMS[case["form"]])
        return _stored(case, C + 0.5 * torch.einsum("%s,%s->%s" % (ia, ib, ic), A, B))
    if k == "group":
        d = _triple_dims(case)
        A, B = g.graded(int(np.sum(d[:, 0] * d[:, 2]))), g.graded(int(np.sum(d[:, 1] * d[:, 2])))
        out, a, b = [], 0, 0
        for m, n, kk in d.tolist():
            out.append((A[a:a + m * kk].view(m, kk) @ B[b:b + n * kk].view(n, kk).T).reshape(-1))
            a, b = a + m * kk, b + n * kk
        return torch.cat(out)
    if k == "residual":
        x = {}
        for name, sp in CCD_INPUTS.items():
            shape = [case["O"] if c == "h" else case["V"] for c in sp]
            x[name] = g.uniform(math.prod(shape)).view(shape)
        return _ccd_exact(x)
    # jobs with spatial symmetry or too large for dense tensors have no plain counterpart here
    return _cc_exact(case, seed) if case["nirrep"] == 1 and case["o"] + case["v"] <= 48 else None
