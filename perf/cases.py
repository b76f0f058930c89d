"""The work that users of this package have it do, as measurable cases.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same
ranges, ``prepare(case, seed)`` makes a program's operands on the GPU,
``run(state)`` is one pass through the package's public calls, ``work(case)``
the bytes and operations that pass cannot do without, and ``exact(case, seed)``
what it computes, by plain torch in FP64.

Kinds of cases:
  heff      one two-site effective-Hamiltonian apply (``qn.HeffOperator``): the
            step that a DMRG solve repeats, in FP64 (ragged sector blocks, or the
            zero-padded blocks of the reference's layout) or 3xTF32
  env       one environment update (``qn.make_L`` / ``qn.make_R``)
  eigsolve  one Lanczos solve of a bond (``krylov.eigsolve``, krylovdim 3)
  pxp       the two-site matvec of the PXP chain, whose MPO is a COOTensor
  apply     MPO x MPS on one site, the MPO in COO storage
  permute   ``permutedims`` of a block-sparse environment
  qr, svd   the block factorisations that move the orthogonality centre
"""
import math

import numpy as np
import torch

import sparsebackends_b200 as sb
from sparsebackends_b200 import krylov, pxp, qn

DEVICE = "cuda:0"
PHYS = (1, -1)  # 2Sz of the two spin states


def listed():
    return [
        # a bond in the middle of a 16-site Heisenberg chain (MPO w = 5): small blocks, latency counts
        dict(name="heff_n16_chi60", kind="heff", chi_l=60, chi_r=60, sectors=5, c0=3, c2=1, layout="ragged",
             precision="f64", w12=False),
        # an early sweep of a cylinder (MPO w = 38): many blocks, none of them large
        dict(name="heff_chi256", kind="heff", chi_l=256, chi_r=256, sectors=11, c0=14, c2=12, layout="ragged",
             precision="f64", w12=False),
        # the full-size bond of the J1-J2 cylinder, the benchmark's headline
        dict(name="heff_chi2048", kind="heff", chi_l=2048, chi_r=2048, sectors=11, c0=14, c2=12, layout="ragged",
             precision="f64", w12=False),
        # the same model for a caller that keeps the reference's zero-padded blocks; odd, unequal links
        dict(name="heff_padded_chi1023", kind="heff", chi_l=1023, chi_r=1001, sectors=11, c0=14, c2=12,
             layout="padded", precision="f64", w12=False),
        # the full-size bond in the mixed-precision form of a DMRG sweep
        dict(name="heff_tf32x3_chi2048", kind="heff", chi_l=2048, chi_r=2048, sectors=11, c0=14, c2=12,
             layout="ragged", precision="tf32x3", w12=True),
        # after every bond: the environment that moves with the centre
        dict(name="env_left_chi1024", kind="env", side="left", chi_l=1024, chi_r=1000, sectors=11, c0=10, c2=8),
        # a whole bond solve as a sweep does it: three applies and the vector operations between them
        dict(name="eigsolve_chi512", kind="eigsolve", chi_l=512, chi_r=512, sectors=11, c0=10, c2=8),
        # the constrained chain without a charge: four blocks, MPO entries in COO
        dict(name="pxp_matvec_chi256", kind="pxp", n=18, chi=256),
        dict(name="apply_mpo_chi512", kind="apply", chi_l=512, chi_r=512),
        # an environment in the other index order
        dict(name="permute_env_chi1024", kind="permute", chi=1024, sectors=11, c0=14, c2=12, perm="321654"),
        # moving the orthogonality centre of a sparse-prefix MPS tensor
        dict(name="left_qr_256x160", kind="qr", nl=128, nr=160, ds=2, fill=0.5),
        dict(name="svd_64x96", kind="svd", nl=64, nr=96, d1=2, d2=2, fill=0.5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["heff", "heff", "heff", "heff", "env", "eigsolve", "pxp", "apply", "permute", "qr", "svd"])
    if kind == "heff":
        layout, precision = rng.choice([("ragged", "f64"), ("ragged", "f64"), ("padded", "f64"), ("ragged", "tf32x3")])
        chi = _log(rng, 48, 1100 if layout == "padded" else 2000)
        c2 = rng.choice([1, 4, 8, 12])
        return dict(kind=kind, chi_l=chi, chi_r=max(40, chi - rng.randrange(0, 1 + chi // 6)),
                    sectors=rng.choice([5, 7, 9, 11]) if chi < 256 else rng.choice([9, 11]), c0=c2 + 2, c2=c2,
                    layout=layout, precision=precision, w12=rng.random() < 0.4)
    if kind in ("env", "eigsolve"):
        chi = _log(rng, 48, 1100 if kind == "env" else 800)
        c2 = rng.choice([1, 4, 8])
        d = dict(kind=kind, chi_l=chi, chi_r=max(40, chi - rng.randrange(0, 1 + chi // 6)),
                 sectors=rng.choice([7, 9, 11]), c0=c2 + 2, c2=c2)
        return dict(d, side=rng.choice(["left", "right"])) if kind == "env" else d
    if kind == "pxp":
        return dict(kind=kind, n=rng.choice([12, 14, 16, 18]), chi=_log(rng, 24, 256))
    if kind == "apply":
        return dict(kind=kind, chi_l=_log(rng, 16, 600), chi_r=_log(rng, 16, 600))
    if kind == "permute":
        return dict(kind=kind, chi=_log(rng, 64, 1500), sectors=rng.choice([5, 7, 9, 11]), c0=rng.choice([3, 6, 14]),
                    c2=rng.choice([1, 4, 12]), perm=rng.choice(["321654", "123546", "213465", "132645", "312564"]))
    if kind == "qr":
        return dict(kind=kind, nl=_log(rng, 8, 160), nr=_log(rng, 8, 200), ds=rng.choice([2, 3]), fill=0.5)
    return dict(kind="svd", nl=_log(rng, 4, 80), nr=_log(rng, 8, 120), d1=rng.choice([2, 3]), d2=rng.choice([2, 3]),
                fill=0.5)


# ── sectors, keys and block extents ────────────────────────────────────────

def _link(chi, sectors, shift=0):
    """(charges, dims): ``sectors`` charges around ``shift`` with a Gaussian profile that sums to ``chi``."""
    charges = [2 * i - (sectors - 1) + shift for i in range(sectors)]
    charges = [c + (1 if (c - shift) % 2 else 0) for c in charges]  # one parity whatever the count
    w = np.exp(-((np.asarray(charges, float) - shift) / 2.0) ** 2 / (2 * (sectors / 5.5) ** 2))
    raw = w / w.sum() * max(chi, sectors)
    dims = np.maximum(1, np.floor(raw)).astype(int)
    dims[int(np.argmax(dims))] += max(chi, sectors) - int(dims.sum())
    return charges, [int(d) for d in dims]


def _mpo_link(c0, c2):
    return [-2, 0, 2], [c2, c0, c2]


def _sorted(keys):
    return sorted(keys, key=lambda k: k[::-1])


def _psi_keys(l, r):
    return _sorted((a + 1, s + 1, t + 1, b + 1) for a, qa in enumerate(l[0]) for s in range(2) for t in range(2)
                   for b, qb in enumerate(r[0]) if qa + PHYS[s] + PHYS[t] == qb)


def _site_keys(l, r):
    return _sorted((a + 1, s + 1, b + 1) for a, qa in enumerate(l[0]) for s in range(2) for b, qb in enumerate(r[0])
                   if qa + PHYS[s] == qb)


def _env_keys(link, w):
    return _sorted((p + 1, c + 1, q + 1) for p, qp in enumerate(link[0]) for c, qc in enumerate(w[0])
                   for q, qq in enumerate(link[0]) if qp - qq == qc)


def _mpo_keys(w):
    return _sorted((a + 1, s + 1, t + 1, b + 1) for a, qa in enumerate(w[0]) for s in range(2) for t in range(2)
                   for b, qb in enumerate(w[0]) if qb == qa + PHYS[s] - PHYS[t])


class _Blocks:
    """Block-sparse operand in plain torch: sorted keys, true block extents, and the flat column-major payload."""

    def __init__(self, labels, n2, keys, exts, flat, pdims, tdims):
        self.labels, self.n2, self.keys, self.exts, self.flat = labels, n2, keys, exts, flat
        self.pdims, self.tdims = pdims, tdims
        self.P = len(labels) - n2

    @property
    def dims(self):
        return tuple(self.pdims) + tuple(self.tdims)

    def blocks(self):
        """{key: array with axes in label order}, views of the payload."""
        out, o = {}, 0
        for k, e in zip(self.keys, self.exts):
            n = int(np.prod(e))
            out[k] = self.flat[o:o + n].view(tuple(reversed(e))).permute(tuple(reversed(range(len(e)))))
            o += n
        return out

    def padded(self):
        """The payload with every block zero-padded to the tail extents."""
        out = torch.zeros((len(self.keys),) + tuple(reversed(self.tdims)), dtype=torch.float64, device=DEVICE)
        for i, b in enumerate(self.blocks().values()):
            out[i].permute(tuple(reversed(range(self.n2))))[tuple(slice(0, x) for x in b.shape)] = b
        return out.reshape(-1)


def _env_exts(keys, link, w):
    return [(link[1][k[0] - 1], w[1][k[1] - 1], link[1][k[2] - 1]) for k in keys]


def _gaussian(gen, keys, exts, scale):
    n = sum(int(np.prod(e)) for e in exts)
    return torch.randn(n, generator=gen, dtype=torch.float64, device=DEVICE).mul_(scale)


def _grade(flat, keys, exts):
    """Schmidt-like weights: both bond indices of every block fall off over three decades."""
    o = 0
    for e in exts:
        n = e[0] * e[1]
        b = flat[o:o + n].view(e[1], e[0])
        b *= torch.logspace(0, -3, e[0], dtype=torch.float64, device=DEVICE)[None, :]
        b *= torch.logspace(0, -3, e[1], dtype=torch.float64, device=DEVICE)[:, None]
        o += n
    return flat


LAB = {"psi": ["ql", "s1", "s2", "qr", "ml", "mr"], "L": ["qlp", "qwl", "ql", "mlp", "mwl", "ml"],
       "W1": ["qwl", "s1p", "s1", "qwm", "mwl", "mwm"], "W2": ["qwm", "s2p", "s2", "qwr", "mwm", "mwr"],
       "R": ["qrp", "qwr", "qr", "mrp", "mwr", "mr"], "A": ["ql", "s1", "qr", "ml", "mr"]}


def _operands(case, seed):
    """The operands of the heff, env and eigsolve kinds, by name."""
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    env = case["kind"] == "env"
    l = _link(case["chi_l"], case["sectors"])
    r = _link(case["chi_r"], case["sectors"], 1 if env else 0)
    w = _mpo_link(case["c0"], case["c2"])
    S, D = (lambda x: len(x[0])), (lambda x: max(x[1]))
    out = {}

    def add(name, keys, exts, scale, pdims, tdims):
        out[name] = _Blocks(LAB[name], len(tdims), keys, exts, _gaussian(gen, keys, exts, scale), pdims, tdims)

    mk = _mpo_keys(w)
    me = [(w[1][k[0] - 1], w[1][k[3] - 1]) for k in mk]
    for name in (("W1",) if env else ("W1", "W2")):
        add(name, mk, me, 0.3, (S(w), 2, 2, S(w)), (D(w), D(w)))
    for name, link in (("L", l), ("R", r)):
        keys = _env_keys(link, w)
        add(name, keys, _env_exts(keys, link, w), 0.05, (S(link), S(w), S(link)), (D(link), D(w), D(link)))
    if env:
        keys = _site_keys(l, r)
        add("A", keys, [(l[1][k[0] - 1], r[1][k[2] - 1]) for k in keys], 0.05, (S(l), 2, S(r)), (D(l), D(r)))
        del out["R" if case["side"] == "left" else "L"]
        return out, l, r, w
    keys = _psi_keys(l, r)
    exts = [(l[1][k[0] - 1], r[1][k[3] - 1]) for k in keys]
    add("psi", keys, exts, 1.0, (S(l), 2, 2, S(r)), (D(l), D(r)))
    _grade(out["psi"].flat, keys, exts)
    out["psi"].flat /= out["psi"].flat.norm()
    if case["kind"] == "eigsolve":  # a symmetric operator: average with the transpose over w -> conjugate channel
        conj = {1: 3, 2: 2, 3: 1}
        for name in ("L", "R", "W1", "W2"):
            src = {k: b.clone() for k, b in out[name].blocks().items()}
            for k, b in out[name].blocks().items():
                if name in ("L", "R"):
                    t = src[(k[2], conj[k[1]], k[0])].permute(2, 1, 0)
                else:
                    t = src[(conj[k[0]], k[2], k[1], conj[k[3]])]
                b.copy_(0.5 * (src[k] + t))
    return out, l, r, w


# ── tensors of the package over device values ──────────────────────────────

class _Payload:
    def __init__(self, tensor):
        ptr, n = tensor.device_ptr()
        self.tensor = tensor  # the payload lives as long as the view
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False), "version": 3,
                                         "stream": None}


def _view(tensor):
    """The payload of a tensor of the package as a torch vector, without a copy."""
    return torch.as_tensor(_Payload(tensor), device=DEVICE)


def _tensor(b, layout="ragged"):
    n = len(b.keys) * int(np.prod(b.tdims)) if layout == "padded" else b.flat.numel()
    t = sb.NewBlockSparseSorted(b.dims, b.n2, b.keys, data=np.zeros(n),
                                block_dims=None if layout == "padded" else b.exts)
    t.ctx.synchronize()
    _view(t).copy_(b.padded() if layout == "padded" else b.flat)
    return t


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("heff", "env", "eigsolve"):
        ops, l, r, w = _operands(case, seed)
        t = {n: _tensor(b, case.get("layout", "ragged")) for n, b in ops.items()}
        torch.cuda.synchronize()
        if kind == "env":
            return dict(kind=kind, side=case["side"], E=t["L" if case["side"] == "left" else "R"], A=t["A"], W=t["W1"])
        layout = qn.HeffLayout(qn.U1Link(*l), qn.U1Link(*r), qn.U1Link(*w))
        op = qn.HeffOperator(layout, t["L"], t["W1"], t["W2"], t["R"], w12=case.get("w12", False),
                             precision=case.get("precision", "f64"))
        return dict(kind=kind, op=op, psi=t["psi"])
    if kind == "pxp":
        p = pxp.PxpProblem(n=case["n"], chi=case["chi"], seed=seed)
        return dict(kind=kind, p=p)
    if kind == "apply":
        p = pxp.PxpProblem(n=4, chi=4, seed=1)
        return dict(kind=kind, p=p, A=_tensor(_site(case, seed), "padded"))
    if kind == "permute":
        return dict(kind=kind, A=_tensor(_permute_operand(case, seed)), perm=[int(c) for c in case["perm"]])
    b = _factor_operand(case, seed)
    return dict(kind=kind, A=_tensor(b, "padded"))


def run(state):
    kind = state["kind"]
    if kind == "heff":
        return [_view(state["op"](state["psi"]))]
    if kind == "env":
        make = qn.make_L if state["side"] == "left" else qn.make_R
        return [_view(make(state["E"], state["A"], state["W"]))]
    if kind == "eigsolve":
        values, vectors, _ = krylov.eigsolve(state["op"], state["psi"], 1, "SR", krylovdim=3, maxiter=1)
        return [values[0], _view(vectors[0])]
    if kind == "pxp":
        return [_view(state["p"].apply(state["p"].psi))]
    if kind == "apply":
        return [_view(state["p"].apply_mpo(state["A"]))]
    if kind == "permute":
        return [_view(sb.permutedims(state["A"], state["perm"]))]
    if kind == "qr":
        q, r, lv, rv = sb.blocksparse_left_qr(state["A"])
        return [_view(q), _view(r)]
    u, sv, svs, spec = sb.blocksparse_svd(state["A"], cutoff=1e-10)
    return [_view(u), _view(sv), svs]


# ── further operands ───────────────────────────────────────────────────────

def _site(case, seed):
    """A site tensor of the PXP chain (ql, s, qr | l, r): one block per physical value."""
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    l, r = case["chi_l"], case["chi_r"]
    keys, exts = [(1, 1, 1), (1, 2, 1)], [(l, r), (l, r)]
    return _Blocks(["ql", "s", "qr", "l", "r"], 2, keys, exts, _gaussian(gen, keys, exts, 1.0 / math.sqrt(2 * l)),
                   (1, 2, 1), (l, r))


def _permute_operand(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    link, w = _link(case["chi"], case["sectors"]), _mpo_link(case["c0"], case["c2"])
    keys = _env_keys(link, w)
    exts = _env_exts(keys, link, w)
    return _Blocks(LAB["L"], 3, keys, exts, _gaussian(gen, keys, exts, 1.0), (len(link[0]), 3, len(link[0])),
                   (max(link[1]), max(w[1]), max(link[1])))


def _factor_operand(case, seed):
    """qr: (l, r | s); svd: (L, R | s1, s2), a share ``fill`` of the blocks, none of the prefix values empty."""
    rs = np.random.RandomState(7)  # the block structure is the model's, the values come from the seed
    nl, nr = case["nl"], case["nr"]
    have = rs.rand(nl, nr) < case["fill"]
    have[np.arange(nl), np.arange(nl) % nr] = True
    have[np.arange(nr) % nl, np.arange(nr)] = True
    keys = _sorted((int(a) + 1, int(b) + 1) for a, b in zip(*np.nonzero(have)))
    tail = (case["ds"],) if case["kind"] == "qr" else (case["d1"], case["d2"])
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    exts = [tail] * len(keys)
    labels = ["l", "r", "s1", "s2"][:2 + len(tail)]
    return _Blocks(labels, len(tail), keys, exts, _gaussian(gen, keys, exts, 1.0), (nl, nr), tail)


# ── the same results by plain torch in FP64 ────────────────────────────────

def _contract(A, B, labels, n2):
    """C(labels) = sum over the labels that A and B share, block pair by block pair."""
    shared = [x for x in A.labels if x in B.labels]
    PA, PB = A.labels[:A.P], B.labels[:B.P]
    tA, tB = A.labels[A.P:], B.labels[B.P:]
    pshared = [x for x in PA if x in PB]
    red = [x for x in tA if x in tB]
    assert set(shared) == set(pshared) | set(red)
    kept = [x for x in tA if x not in red] + [x for x in tB if x not in red]
    tail = labels[len(labels) - n2:]
    by = {}
    bb = B.blocks()
    for k in B.keys:
        by.setdefault(tuple(k[PB.index(x)] for x in pshared), []).append(k)
    axes = ([tA.index(x) for x in red], [tB.index(x) for x in red])
    acc = {}
    for ka, a in A.blocks().items():
        for kb in by.get(tuple(ka[PA.index(x)] for x in pshared), ()):
            kv = dict(zip(PA, ka))
            kv.update(zip(PB, kb))
            kc = tuple(kv[x] for x in labels[:len(labels) - n2])
            c = torch.tensordot(a, bb[kb], dims=axes)
            acc[kc] = acc[kc].add_(c) if kc in acc else c
    order = [kept.index(x) for x in tail]
    keys = _sorted(acc)
    parts, exts = [], []
    for k in keys:
        c = acc.pop(k).permute(order)
        exts.append(tuple(c.shape))
        parts.append(c.permute(tuple(reversed(range(c.dim())))).reshape(-1))
    dim = dict(zip(A.labels, A.dims))
    dim.update(zip(B.labels, B.dims))
    return _Blocks(labels, n2, keys, exts, torch.cat(parts), [dim[x] for x in labels[:len(labels) - n2]],
                   [dim[x] for x in tail])


def _heff(o, psi):
    t1 = _contract(o["L"], psi, ["qlp", "s2", "qr", "qwl", "s1", "mr", "mlp", "mwl"], 3)
    t2 = _contract(t1, o["W1"], ["qlp", "qr", "s1p", "qwm", "s2", "mr", "mlp", "mwm"], 3)
    del t1
    t3 = _contract(t2, o["W2"], ["qlp", "s1p", "s2p", "qwr", "qr", "mwr", "mr", "mlp"], 3)
    del t2
    return _contract(o["R"], t3, ["qlp", "s1p", "s2p", "qrp", "mlp", "mrp"], 2)


def _env(o, side):
    a = o["A"]
    bar = _Blocks(["qlp", "s1p", "qrp", "mlp", "mrp"], 2, a.keys, a.exts, a.flat, a.pdims, a.tdims)
    if side == "left":
        e = _contract(o["L"], a, ["qlp", "qwl", "s1", "qr", "mr", "mlp", "mwl"], 3)
        e = _contract(e, o["W1"], ["qlp", "qr", "s1p", "qwm", "mr", "mlp", "mwm"], 3)
        return _contract(e, bar, ["qrp", "qwm", "qr", "mrp", "mwm", "mr"], 3)
    env = o["R"]
    env = _Blocks(["qrp", "qwm", "qr", "mrp", "mwm", "mr"], 3, env.keys, env.exts, env.flat, env.pdims, env.tdims)
    e = _contract(env, a, ["qrp", "qwm", "ql", "s1", "ml", "mrp", "mwm"], 3)
    e = _contract(e, o["W1"], ["qrp", "ql", "s1p", "qwl", "ml", "mrp", "mwl"], 3)
    return _contract(e, bar, ["qlp", "qwl", "ql", "mlp", "mwl", "ml"], 3)


def exact(case, seed):
    kind = case["kind"]
    if kind == "heff":
        o, l, r, w = _operands(case, seed)
        t = _heff(o, o["psi"])
        return [t.padded() if case["layout"] == "padded" else t.flat]
    if kind == "env":
        o, l, r, w = _operands(case, seed)
        return [_env(o, case["side"]).flat]
    if kind == "eigsolve":
        return _exact_eigsolve(case, seed)
    if kind == "pxp":
        return [_exact_pxp(case, seed)]
    if kind == "apply":
        a = torch.stack([b for b in _site(case, seed).blocks().values()], 1)  # l, s, r
        w = torch.from_numpy(pxp.mpo_dense()).to(DEVICE)                      # s', s, wl, wr
        full = torch.einsum("xsab,lsr->xablr", w, a)
        have = (w != 0).any(1)                                                # a block exists for every nonzero entry
        keys = sorted((tuple(int(i) for i in k) for k in have.nonzero()), key=lambda k: k[::-1])
        return [torch.cat([full[k].t().reshape(-1) for k in keys])]
    if kind == "permute":
        b = _permute_operand(case, seed)
        p = [int(c) - 1 for c in case["perm"]]
        new = {tuple(k[q] for q in p[:3]): blk.permute([q - 3 for q in p[3:]]) for k, blk in b.blocks().items()}
        return [torch.cat([new[k].permute(2, 1, 0).reshape(-1) for k in _sorted(new)])]
    b = _factor_operand(case, seed)
    if kind == "qr":
        nl, nr, ds = case["nl"], case["nr"], case["ds"]
        m = torch.zeros(nl * ds, nr, dtype=torch.float64)
        for k, blk in b.blocks().items():
            m[(k[0] - 1) * ds:k[0] * ds, k[1] - 1] = blk.cpu()
        q, r = torch.linalg.qr(m)
        n = q.shape[1]
        return [q.view(nl, ds, n).permute(0, 2, 1).reshape(-1), r.t().reshape(-1)]
    groups, blocks = {}, b.blocks()
    for k in b.keys:
        groups.setdefault(k[0], []).append(blocks[k].cpu())
    sv = []
    for g in sorted(groups):
        s = torch.linalg.svdvals(torch.cat(groups[g], 1))
        sv.append(s)
    return [None, None, torch.cat(sv)]  # the vectors are fixed up to their signs only


def _exact_eigsolve(case, seed):
    """Three Lanczos steps from psi and the lowest Ritz pair."""
    o, l, r, w = _operands(case, seed)
    p = o["psi"]
    apply = lambda v: _heff(o, _Blocks(p.labels, 2, p.keys, p.exts, v, p.pdims, p.tdims)).flat  # noqa: E731
    V, a, b = [p.flat / p.flat.norm()], [], []
    for k in range(3):
        x = apply(V[k])
        a.append(float(V[k] @ x))
        for _ in range(2):
            for v in V:
                x = x - (v @ x) * v
        b.append(float(x.norm()))
        V.append(x / b[-1])
    d, u = np.linalg.eigh(np.diag(a) + np.diag(b[:2], 1) + np.diag(b[:2], -1))
    return [float(d[0]), sum(float(c) * v for c, v in zip(u[:, 0], V))]


def _exact_pxp(case, seed):
    sites, psi, c = pxp.random_mps(case["n"], case["chi"], seed)
    t = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to(DEVICE)  # noqa: E731
    w = t(pxp.mpo_dense())  # s', s, wl, wr
    L = torch.zeros(1, 4, 1, dtype=torch.float64, device=DEVICE)
    L[0, 3, 0] = 1.0
    for k in range(1, c):
        a = t(sites[k - 1])
        e = torch.einsum("pwq,qsr->pwsr", L, a)
        e = torch.einsum("pwsr,tswx->ptxr", e, w)
        L = torch.einsum("ptxr,ptm->mxr", e, a)
    R = torch.zeros(1, 4, 1, dtype=torch.float64, device=DEVICE)
    R[0, 0, 0] = 1.0
    for k in range(case["n"], c + 1, -1):
        a = t(sites[k - 1])
        e = torch.einsum("pwq,lsq->pwsl", R, a)
        e = torch.einsum("pwsl,tsxw->ptxl", e, w)
        R = torch.einsum("ptxl,mtp->mxl", e, a)
    x = torch.einsum("pwl,labr->pwabr", L, t(psi))
    x = torch.einsum("pwabr,cawm->pcmbr", x, w)
    x = torch.einsum("pcmbr,dbmn->pcdnr", x, w)
    x = torch.einsum("pcdnr,qnr->pcdq", x, R)
    return torch.cat([x[:, s, u, :].t().reshape(-1) for u in range(2) for s in range(2)])


# ── the work that a pass cannot do without ─────────────────────────────────

def _structure(case):
    """Keys and extents of the operands of heff, env and eigsolve, without values."""
    env = case["kind"] == "env"
    l = _link(case["chi_l"], case["sectors"])
    r = _link(case["chi_r"], case["sectors"], 1 if env else 0)
    w = _mpo_link(case["c0"], case["c2"])
    dim = {"ql": l, "qlp": l, "qr": r, "qrp": r, "qwl": w, "qwm": w, "qwr": w}
    keys = {"L": _env_keys(l, w), "R": _env_keys(r, w), "W1": _mpo_keys(w), "W2": _mpo_keys(w)}
    keys.update({"A": _site_keys(l, r)} if env else {"psi": _psi_keys(l, r)})
    return keys, lambda q, v: dim[q][1][v - 1]


GRADE = {"ml": "ql", "mlp": "qlp", "mr": "qr", "mrp": "qrp", "mwl": "qwl", "mwm": "qwm", "mwr": "qwr"}


def _walk(steps, keys, labels, size):
    """FLOPs of a chain of contractions, and the values of its last result."""
    total, values = 0.0, 0
    keys, labels = dict(keys), dict(labels)
    for c, lc, n2, a, b in steps:
        la, lb = labels[a], labels[b]
        pa, pb = [x for x in la if x not in GRADE], [x for x in lb if x not in GRADE]
        sh = [x for x in pa if x in pb]
        by = {}
        for k in keys[b]:
            by.setdefault(tuple(k[pb.index(x)] for x in sh), []).append(k)
        out = {}
        for ka in keys[a]:
            for kb in by.get(tuple(ka[pa.index(x)] for x in sh), ()):
                kv = dict(zip(pa, ka))
                kv.update(zip(pb, kb))
                n = 2.0
                for x in {*la, *lb} & GRADE.keys():
                    n *= size(GRADE[x], kv[GRADE[x]])
                total += n
                kc = tuple(kv[x] for x in lc[:len(lc) - n2])
                if kc not in out:
                    out[kc] = float(np.prod([size(GRADE[x], kv[GRADE[x]]) for x in lc[len(lc) - n2:]]))
        keys[c], labels[c] = list(out), lc
        values = sum(out.values())
    return total, values


HEFF = (("T1", ["qlp", "s2", "qr", "qwl", "s1", "mr", "mlp", "mwl"], 3, "L", "psi"),
        ("T2", ["qlp", "qr", "s1p", "qwm", "s2", "mr", "mlp", "mwm"], 3, "T1", "W1"),
        ("T3", ["qlp", "s1p", "s2p", "qwr", "qr", "mwr", "mr", "mlp"], 3, "T2", "W2"),
        ("T4", ["qlp", "s1p", "s2p", "qrp", "mlp", "mrp"], 2, "R", "T3"))
ENV_L = (("E1", ["qlp", "qwl", "s1", "qr", "mr", "mlp", "mwl"], 3, "L", "A"),
         ("E2", ["qlp", "qr", "s1p", "qwm", "mr", "mlp", "mwm"], 3, "E1", "W1"),
         ("E3", ["qrp", "qwm", "qr", "mrp", "mwm", "mr"], 3, "E2", "B"))
ENV_R = (("E1", ["qrp", "qwr", "ql", "s1", "ml", "mrp", "mwr"], 3, "R", "A"),
         ("E2", ["qrp", "ql", "s1p", "qwl", "ml", "mrp", "mwl"], 3, "E1", "W"),
         ("E3", ["qlp", "qwl", "ql", "mlp", "mwl", "ml"], 3, "E2", "B"))


def work(case):
    kind = case["kind"]
    if kind in ("heff", "env", "eigsolve"):
        keys, size = _structure(case)
        values = {n: sum(float(np.prod([size(GRADE[x], k[[y for y in LAB[n] if y not in GRADE].index(GRADE[x])])
                                        for x in LAB[n] if x in GRADE])) for k in ks) for n, ks in keys.items()}
        labels = dict(LAB)
        if kind == "env":
            keys["B"], labels["B"] = keys["A"], ["qlp", "s1p", "qrp", "mlp", "mrp"]
            keys["W"], labels["W"] = keys["W1"], ["qwl", "s1p", "s1", "qwr", "mwl", "mwr"]
            flops, out = _walk(ENV_L if case["side"] == "left" else ENV_R, keys, labels, size)
            ins = values["L" if case["side"] == "left" else "R"] + values["A"] + values["W1"]
            return {"bytes": 8.0 * (ins + out), "flops": flops}
        flops, out = _walk(HEFF, keys, labels, size)
        ins = values["L"] + values["R"] + values["W1"] + values["W2"] + values["psi"]
        n = 3 if kind == "eigsolve" else 1
        return {"bytes": 8.0 * (ins + out), "flops": n * flops}
    if kind == "pxp":
        d = pxp.bond_dims(case["n"], case["chi"])
        c = case["n"] // 2
        l, r = d[c - 1], d[c + 1]
        return {"bytes": 8.0 * (4 * l * l + 4 * r * r + 8 * l * r), "flops": 2.0 * 4 * 4 * (l * l * r + l * r * r)}
    if kind == "apply":
        n = float(case["chi_l"] * case["chi_r"])
        return {"bytes": 8.0 * (2 + 8) * n, "flops": 16.0 * n}
    if kind == "permute":
        link, w = _link(case["chi"], case["sectors"]), _mpo_link(case["c0"], case["c2"])
        n = sum(float(np.prod(e)) for e in _env_exts(_env_keys(link, w), link, w))
        return {"bytes": 16.0 * n, "flops": 0.0}
    if kind == "qr":
        m, n = case["nl"] * case["ds"], case["nr"]
        k = min(m, n)
        return {"bytes": 8.0 * (m * n + m * k + k * n), "flops": 4.0 * m * n * k}
    m, n = case["d1"], case["nr"] * case["fill"] * case["d2"]
    return {"bytes": 8.0 * case["nl"] * (2 * m * n + m * m), "flops": 8.0 * case["nl"] * m * m * n}
