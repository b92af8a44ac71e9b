"""Performance cases of the library: what its users run, at the sizes they run it.

A case is one pass through the public Python entry points (api.py, autograd.py)
on inputs that are already on the device:

  kernel    one lib_cc contraction (cpsd_<name>) on DPD tensors, FP64 or mixed
  cis       the SF-CIS program (Davidson)
  pipeline  SF-CIS + ground CPS(D) + EE-CPS(D-3) of one molecule, FP64 or mixed
  batch     several molecules in one call, mixed
  grad3     energies up to w^(3) and their gradient through torch.autograd
  grcpsd    CIS(D-infinity), grCPS(D) and EE-grCPS(D)

Systems come from the seeded generator of synth.py (the shapes of its named
workloads and of its batch draw, and odd sizes between them).  exact() restates
the same quantities densely in FP64 torch, from the packed integrals alone.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    if "cpsd_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location("_graft_entry", os.path.join(_ROOT, "__graft_entry__.py"))
        mod = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(mod)
        mod.load_package()
    from cpsd_b200 import api, autograd, synth
    return api, autograd, synth


# layouts of the integral lists and amplitudes: spaces and pair packing (0: p < q)
LAYOUT = {"ai": ("vozz", (1, 1)), "oo": ("oozz", (1, 1)), "vv": ("vvzz", (1, 1)), "abij": ("vvoo", (0, 0)),
          "ijkl": ("oooo", (0, 0)), "ijka": ("ooov", (0, 1)), "iabj": ("vovo", (1, 1)), "abci": ("vvvo", (0, 1)),
          "abcd": ("vvvv", (0, 0))}
LISTS = ("ijkl", "ijka", "abij", "iabj", "abci", "abcd")

# contraction -> layouts of (out, amplitude, integral), letters of the dense product, factor on them (packed sums
# count once), which output pairs are antisymmetrised
KERNELS = {
    "c2_r2abcd": (("abij", "abij", "abcd"), "efij,abef->abij", 0.5, ""),
    "c2_r2Wmbej": (("abij", "abij", "iabj"), "aeim,embj->abij", 1.0, "pr"),
    "c2_r2Fae": (("abij", "abij", "vv"), "aeij,be->abij", 1.0, "p"),
    "c2_r1abci": (("abij", "ai", "abci"), "ei,abej->abij", 1.0, "r"),
    "c1_r2abci": (("ai", "abij", "abci"), "feim,feam->ai", 0.5, ""),
    "c1_r1iabj": (("ai", "ai", "iabj"), "fn,fnai->ai", 1.0, ""),
    "Fae_r1abci": (("vv", "ai", "abci"), "fm,efam->ae", 1.0, ""),
    "Wmbej_r1abci": (("iabj", "ai", "abci"), "fj,febm->embj", 1.0, ""),
    "Wmbej_r2abij": (("iabj", "abij", "abij"), "bfjn,fenm->embj", 0.5, ""),
    "Wkbij_r2abci": (("ijka", "abij", "abci"), "cdij,dcbk->ijkb", 0.5, ""),
}
TIGHT = dict(davidson_conv=12, davidson_cyc=100, diis_max_err=1e-12, diis_cyc=200)


def _mol(nmo, nocc_a, nirrep, roots=1, **kw):
    return dict(nmo=nmo, nocc_a=nocc_a, nocc_b=nocc_a - 2, nirrep=nirrep, roots=roots, **kw)


def listed():
    return [
        # the smallest program: the spin-flip CIS spectrum of a small C2v molecule; short launches one after another
        dict(name="cis_c2v_nmo48", kind="cis", **_mol(48, 5, 4, 3)),
        # one small contraction call, as a caller of the boundary makes them by the hundred: host path and launches
        dict(name="ring_c2v_nmo48", kind="kernel", op="c2_r2Wmbej", digits=0, **_mol(48, 5, 4)),
        # the particle ladder, the largest contraction of every order: mixed at the size of the single-molecule
        # workload, FP64 on an unsymmetric molecule of an odd size
        dict(name="ladder_d2h_nmo200_5d", kind="kernel", op="c2_r2abcd", digits=5, **_mol(200, 10, 8)),
        dict(name="ladder_c1_nmo71", kind="kernel", op="c2_r2abcd", digits=0, **_mol(71, 5, 1)),
        # doubles into singles over the (vv|vo) list: once per root and order, bound by reading the list
        dict(name="c1_r2abci_d2h_nmo200", kind="kernel", op="c1_r2abci", digits=0, **_mol(200, 10, 8)),
        # the (vv|vo) list against one CIS vector, at an odd size
        dict(name="wmbej_r1abci_c2v_nmo151", kind="kernel", op="Wmbej_r1abci", digits=0, **_mol(151, 9, 4)),
        # the whole chain of one molecule: the small workload in FP64, ordinary FP64, the large one mixed
        dict(name="pipeline_c2v_nmo48", kind="pipeline", digits=0, **_mol(48, 5, 4, 3)),
        dict(name="pipeline_c2v_nmo120", kind="pipeline", digits=0, **_mol(120, 8, 4, 4)),
        dict(name="pipeline_d2h_nmo200_5d", kind="pipeline", digits=5, **_mol(200, 10, 8, 5)),
        # a screening run: many independent molecules of mixed sizes and symmetries in one call
        dict(name="batch_8_nmo60-100_6d", kind="batch", digits=6, molecules=8, nmo_min=60, nmo_max=100, shape_seed=0),
        # response properties: energies and the gradient with respect to every integral (forward and backward)
        dict(name="grad3_c2v_nmo80", kind="grad3", digits=0, **_mol(80, 8, 4, 2)),
        # the second-order programs over (R1, R2) vectors
        dict(name="grcpsd_c2v_nmo48", kind="grcpsd", digits=0, **_mol(48, 5, 4, 2)),
    ]


# largest number of orbitals per irrep count: the (vv|vv) list stays below that of the largest listed molecule
NMO_CAP = {1: 90, 2: 120, 4: 150, 8: 200}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["kernel"] * 5 + ["pipeline"] * 3 + ["cis", "batch", "grad3", "grcpsd"])
    nirrep = rng.choice([1, 2, 4, 8])
    if kind == "batch":
        lo = rng.randint(40, 70)
        return dict(kind=kind, digits=rng.choice([0, 5, 6]), molecules=rng.randint(2, 8), nmo_min=lo,
                    nmo_max=rng.randint(lo + 5, 100), shape_seed=rng.randint(1, 10 ** 6))
    # vectors of the grCPS(D) programs no longer than the listed molecule's
    cap = {"grad3": min(80, NMO_CAP[nirrep]), "grcpsd": {1: 26, 2: 34, 4: 46, 8: 60}[nirrep]}.get(kind, NMO_CAP[nirrep])
    nmo = _log(rng, {"cis": 32, "grcpsd": 20}.get(kind, 24), cap)
    m = _mol(nmo, rng.randint(4, 5 if kind == "grcpsd" else min(12, nmo // 6)) if nmo >= 24 else 4, nirrep)
    if kind == "kernel":
        op = rng.choice(sorted(KERNELS))
        return dict(kind=kind, op=op, digits=rng.choice([0, 0, 5, 6]), **m)
    m.update(roots=rng.randint(1, 2 if kind in ("grad3", "grcpsd") else 6))
    return dict(kind=kind, digits=rng.choice([0, 5, 6]) if kind == "pipeline" else 0, **m)


# ------------------------------------------------------------------ inputs
def _batch_shapes(case):
    """molecules of a batch case, drawn like the batching workload"""
    rng = np.random.default_rng(case["shape_seed"])
    out = []
    for _ in range(case["molecules"]):
        nirrep = int(rng.choice([1, 2, 4, 8]))
        nmo = int(rng.integers(case["nmo_min"], min(case["nmo_max"], NMO_CAP[nirrep]) + 1))
        out.append(_mol(nmo, int(rng.integers(4, 11)), nirrep, int(rng.integers(3, 7))))
    return out


def _system(synth, m, seed):
    # the lowest roots, as the large workloads ask for; the close-lying ones of unsymmetric molecules take up to a
    # hundred Davidson cycles
    return synth.System(m["nmo"], m["nocc_a"], m["nocc_b"], m["nirrep"], seed=seed, roots=m["roots"],
                        run_opts=dict(lowest=1, davidson_cyc=100), host_ints=False)


class _Shape:
    """populations of a molecule without its integrals"""

    def __init__(self, m):
        n = m["nirrep"]
        self.n, self.nmo = n, m["nmo"]
        pop = np.zeros((4, 8), np.int64)  # alpha occupied, beta occupied, alpha virtual, beta virtual
        for k in range(m["nmo"]):
            pop[0 if k < m["nocc_a"] else 2, k % n] += 1
            pop[1 if k < m["nocc_b"] else 3, k % n] += 1
        self.oa, self.ob, self.va, self.vb = pop
        self.o, self.v = pop[0] + pop[1], pop[2] + pop[3]
        self.z = np.array([1] + [0] * 7, np.int64)

    def pops(self, layout):
        return [{"o": self.o, "v": self.v, "z": self.z}[c] for c in LAYOUT[layout][0]]

    def pairs(self, p, q, iop):
        """stored (irrep index, p, q) pairs per pair irrep, in storage order, as orbital numbers"""
        offp, offq = np.concatenate([[0], np.cumsum(p)]), np.concatenate([[0], np.cumsum(q)])
        out = []
        for irr in range(self.n):
            P, Q = [], []
            for iq in range(self.n):
                ip = iq ^ irr
                if iop == 0 and ip > iq:
                    continue
                b, a = np.meshgrid(np.arange(q[iq]), np.arange(p[ip]), indexing="ij")
                keep = a < b if iop == 0 and ip == iq else np.ones_like(a, bool)
                P.append(offp[ip] + a[keep])
                Q.append(offq[iq] + b[keep])
            out.append((np.concatenate(P), np.concatenate(Q)))
        return out

    def length(self, layout):
        p, (i0, i1) = self.pops(layout), LAYOUT[layout][1]
        left, right = self.pairs(p[0], p[1], i0), self.pairs(p[2], p[3], i1)
        return sum(len(l[0]) * len(r[0]) for l, r in zip(left, right))


def prepare(case, seed):
    api, autograd, synth = _package()
    kind = case["kind"]
    if kind == "kernel":
        sh = _Shape(case)
        layouts = KERNELS[case["op"]][0]
        g = torch.Generator(device="cuda").manual_seed(seed)
        # amplitudes are integrals over orbital-energy denominators of about 1 to 10 Eh
        n_amp, n_int = sh.length(layouts[1]), sh.length(layouts[2])
        amp = 0.02 * torch.randn(n_amp, dtype=torch.float64, device="cuda", generator=g)
        amp /= 1.0 + 9.0 * torch.rand(n_amp, dtype=torch.float64, device="cuda", generator=g)
        ints = torch.randn(n_int, dtype=torch.float64, device="cuda", generator=g).mul_(0.05)
        out = torch.zeros(sh.length(layouts[0]), dtype=torch.float64, device="cuda")
        dirprd = synth.xor_dirprd(case["nirrep"])
        api.init(case["nirrep"], dirprd)
        opts = [api.opt(sh.pops(l), LAYOUT[l][1], 1, t) for l, t in zip(layouts, (out, amp, ints))]
        return dict(kind=kind, case=case, tensors=(out, amp, ints), opts=opts, dirprd=dirprd)
    if kind == "batch":
        mols = [_system(synth, m, 1000 * seed + k) for k, m in enumerate(_batch_shapes(case))]
        ints = [api.DeviceIntegrals.from_tensors(synth.device_integrals(s)) for s in mols]
        for s in mols:
            s.L = None
        return dict(kind=kind, case=case, mols=mols, ints=ints, params=[api.make_params(s) for s in mols])
    s = _system(synth, case, seed)
    t = synth.device_integrals(s)
    s.L = None  # the generator's factors are not needed any more
    st = dict(kind=kind, case=case, s=s, t=t)
    if kind == "grad3":
        w = np.random.default_rng(seed).uniform(0.5, 1.5, (3, s.nroots))
        st.update(weights=torch.from_numpy(w), t={k: v.requires_grad_(True) for k, v in t.items()})
        return st
    st.update(ints=api.DeviceIntegrals.from_tensors(t), sysc=api.make_system(s), par=api.make_params(s))
    return st


def run(state):
    api, autograd, _ = _package()
    kind, case = state["kind"], state["case"]
    api.use_torch_stream()
    api.set_mixed(case.get("digits", 0))
    if kind == "kernel":
        out = state["tensors"][0]
        api.init(case["nirrep"], state["dirprd"])
        out.zero_()
        api.kernel(case["op"], *state["opts"])
        return out
    if kind == "batch":
        res = api.pipeline_batch(state["mols"], state["ints"], state["params"], nworkers=8)
        return [list(r) for r in res]
    s = state["s"]
    if kind == "grad3":
        t = state["t"]
        w = autograd.cpsd3_energies(s, t, 1, s.nroots, **TIGHT)
        E = sum((g * x).sum() for g, x in zip(state["weights"], w))
        grads = torch.autograd.grad(E, list(t.values()))
        return dict(energies=[x.detach() for x in w], grads=dict(zip(t, grads)))
    args = (s, state["sysc"], state["ints"], state["par"])
    if kind == "cis":
        om, R, _ = api.cis_run(*args)
        return dict(omega=om, vectors=R)
    if kind == "pipeline":
        om, w2, w3 = api.pipeline(*args)
        return dict(omega=om, w2=w2, w3=w3)
    g = api.grcpsd_ground(*args)
    om, R0, _ = api.cisdoo_run(*args)
    r = api.eegrcpsd_roots(*args, g, om, R0)
    # the root vectors are left out: their sign is the general eigen-solver's, which rounding decides
    return dict(T1=g["T1"], T2=g["T2"], E=g["E"], omega=om, w=r["w"])


# ------------------------------------------------------------- the work of a pass
def _kernel_work(op, sh):
    layouts, spec, _, _ = KERNELS[op]
    a, rest = spec.split(",")
    b, c = rest.split("->")
    space = {x: y for l, t in zip((a, b, c), layouts[1:] + layouts[:1]) for x, y in zip(l, LAYOUT[t][0])}
    f = 2.0
    for x in set(a + b + c):
        f *= float({"o": sh.o, "v": sh.v}[space[x]].sum())
    f /= sh.n ** 2  # two symmetry constraints
    for letters, t in ((a, layouts[1]), (b, layouts[2])):  # packed pairs kept by both of their tensors run once
        for k in (0, 1):
            if LAYOUT[t][1][k] == 0 and len(letters) == 4:
                pair = set(letters[2 * k:2 * k + 2])
                others = [l for l in (a, b, c) if l != letters]
                if any(pair <= set(l) for l in others):
                    f /= 2.0 if letters == a or not pair <= set(a) else 1.0
    return dict(bytes=8.0 * sum(sh.length(t) for t in layouts), flops=f)


def _pipeline_work(sh, roots):
    doubles = sum(_kernel_work(op, sh)["flops"] for op in ("c2_r2abcd", "c2_r2Wmbej", "c2_r1abci", "Wmbej_r1abci"))
    return dict(bytes=8.0 * sum(sh.length(t) for t in LISTS), flops=(roots + 1) * doubles)


def work(case):
    if case["kind"] == "kernel":
        return _kernel_work(case["op"], _Shape(case))
    if case["kind"] == "batch":
        w = [_pipeline_work(_Shape(m), m["roots"]) for m in _batch_shapes(case)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    sh = _Shape(case)
    if case["kind"] == "cis":  # the operator of irrep 1 is read once; about ten products per root
        w = _kernel_work("c1_r1iabj", sh)
        return dict(bytes=w["bytes"], flops=10.0 * case["roots"] * w["flops"])
    w = _pipeline_work(sh, case["roots"])
    if case["kind"] == "grad3":  # each list is read and its gradient written; two products reverse each product
        return dict(bytes=2.0 * w["bytes"], flops=3.0 * w["flops"])
    return dict(bytes=w["bytes"] + 8.0 * 6 * sh.length("abij"), flops=w["flops"])


def tolerance(case):
    """Four times the largest relative change seen over about sixty drawn cases.  FP64: a contraction against exact();
    a program with every contraction through 7 digits instead (a disturbance of 1e-13).  Mixed: a contraction against
    exact(); a program with every contraction through its digits instead of the large ones."""
    digits = case.get("digits", 0)
    if case["kind"] == "kernel":
        return {"rel": {0: 1.2e-14, 5: 1.4e-8, 6: 7e-11}[digits]}
    if case["kind"] in ("pipeline", "batch"):
        return {"rel": {0: 1e-9, 5: 1.2e-6, 6: 1e-8}[digits]}
    return {"rel": {"cis": 2e-11, "grad3": 6e-11, "grcpsd": 6e-11}[case["kind"]]}


# ------------------------------------------------------------------ exact values
class _Dense:
    """The packed lists of a molecule as dense spin-orbital tensors (FP64 torch, differentiable)."""

    def __init__(self, m, t):
        self.sh, self.t = _Shape(m), t
        self.maps = {}

    def _pairs(self, p, q, iop):
        """position, sign and irrep of every (p, q) in its packed pair space, and the pairs per irrep"""
        sh = self.sh
        lists = sh.pairs(p, q, iop)
        pos = np.zeros((p.sum(), q.sum()), np.int64)
        sgn = np.zeros((p.sum(), q.sum()))
        irr = np.zeros((p.sum(), q.sum()), np.int64)
        for h, (a, b) in enumerate(lists):
            k = np.arange(len(a))
            pos[a, b], sgn[a, b], irr[a, b] = k, 1.0, h
            if iop == 0:
                pos[b, a], sgn[b, a], irr[b, a] = k, -1.0, h
        return [torch.from_numpy(x).cuda() for x in (pos, sgn, irr)] + [[len(a) for a, _ in lists]]

    def __getitem__(self, layout):
        return self.unpack(self.t[layout], layout)

    def unpack(self, vec, layout):
        if layout not in self.maps:
            p, (i0, i1) = self.sh.pops(layout), LAYOUT[layout][1]
            pl, sl, hl, nl = self._pairs(p[0], p[1], i0)
            pr, sr, hr, nr = self._pairs(p[2], p[3], i1)
            base = torch.tensor(np.concatenate([[0], np.cumsum(np.array(nl) * np.array(nr))]), device="cuda")
            nl = torch.tensor(nl, device="cuda")
            idx = (base[hr] + pr * nl[hr])[None, None] + pl[:, :, None, None]
            s = sl[:, :, None, None] * sr[None, None] * (hl[:, :, None, None] == hr[None, None])
            self.maps[layout] = (torch.where(s != 0, idx, 0), s)
        idx, s = self.maps[layout]
        return vec[idx] * s if LAYOUT[layout][0][2:] != "zz" else (vec[idx] * s)[:, :, 0, 0]

    def pack(self, D, layout):
        p, (i0, i1) = self.sh.pops(layout), LAYOUT[layout][1]
        if D.dim() == 2:
            D = D[:, :, None, None]
        out = []
        for (a, b), (c, d) in zip(self.sh.pairs(p[0], p[1], i0), self.sh.pairs(p[2], p[3], i1)):
            a, b, c, d = (torch.from_numpy(x).cuda() for x in (a, b, c, d))
            out.append(D[a[None, :], b[None, :], c[:, None], d[:, None]].reshape(-1))
        return torch.cat(out)

    def ladder(self, r):
        """0.5 V(ab,ef) r(ef,ij) by the blocks of the packed (vv|vv) list"""
        sh, vec, off = self.sh, self.t["abcd"], 0
        out = torch.zeros_like(r)
        for a, b in sh.pairs(sh.v, sh.v, 0):
            n = len(a)
            a, b = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
            x = vec[off:off + n * n].view(n, n).T @ r[a, b].reshape(n, -1)
            x = x.reshape(n, *r.shape[2:])
            out = out.index_put((a, b), x).index_put((b, a), -x)
            off += n * n
        return out


def _pq(x):
    return x - x.transpose(0, 1)


def _rs(x):
    return x - x.transpose(2, 3)


def _chain(m, t, grads=None):
    """(w0, w^(2), w^(3)) of the lowest spin-flip roots of irrep 1; with grads (3 x roots weights) also the gradient of
    the weighted sum with respect to every list and the orbital energies.  No w^(3) where the singles equations are
    indefinite: the programs' DIIS loop then ends at its cycle limit."""
    e = torch.einsum
    if grads is not None:
        t = {k: v.detach().clone().requires_grad_(True) for k, v in t.items()}
    d = _Dense(m, t)
    sh = d.sh
    no = int(sh.o.sum())
    ijkl, ijka, abij, iabj, abci = (d[k] for k in LISTS[:5])
    eo, ev = t["eorb"][:no], t["eorb"][no:]
    e1 = ev[:, None] - eo[None]
    e2 = e1[:, None, :, None] + e1[None, :, None, :]
    # singles of irrep 1; the spin-flip block takes an alpha electron to a beta orbital
    irr = [np.repeat(np.arange(8), x) for x in (sh.v, sh.o)]
    beta = [np.concatenate([np.arange(a + b) >= a for a, b in zip(*x)]) for x in ((sh.va, sh.vb), (sh.oa, sh.ob))]
    a, i = np.nonzero(irr[0][:, None] == irr[1][None])
    flip = torch.from_numpy(np.nonzero(beta[0][a] & ~beta[1][i])[0]).cuda()
    a, i = torch.from_numpy(a).cuda(), torch.from_numpy(i).cuda()
    A = iabj[:, :, a, i][a, i].T + torch.diag(e1[a, i])  # rows (ai), columns (fn)
    _, X = torch.linalg.eigh((0.5 * (A + A.T)).detach()[flip][:, flip])

    def ladder(r):
        return d.ladder(r)

    def c1_doubles(r):
        return 0.5 * e("feam,feim->ai", abci, r) - 0.5 * e("aemn,mnie->ai", r, ijka)

    def c2_doubles(r):
        ring = _rs(_pq(e("aeim,embj->abij", r, iabj)))
        return ring + 0.5 * e("abmn,mnij->abij", r, ijkl) + ladder(r)

    def fock(r):
        return 0.5 * e("efin,efmn->mi", r, abij), -0.5 * e("afmn,efmn->ae", r, abij)

    T2 = -abij / e2
    C1 = c1_doubles(T2)
    T2b = -c2_doubles(T2) / e2
    T1b = torch.zeros_like(e1).index_put((a, i), torch.linalg.solve(A, -C1[a, i]))
    foo, fvv = fock(T2)
    wvo = e("bfjn,fenm->embj", T2, abij)
    woo = _pq(e("klic,bcjl->ijkb", ijka, T2)) + 0.5 * e("dcbk,cdij->ijkb", abci, T2)
    foo3, fvv3 = fock(T2b)
    foo3 = foo3 + e("en,mnie->mi", T1b, ijka)
    fvv3 = fvv3 + e("fm,efam->ae", T1b, abci)
    wvo3 = e("bfjn,fenm->embj", T2b, abij) + e("fj,febm->embj", T1b, abci) - e("bn,nmje->embj", T1b, ijka)
    res = []
    for k in range(m["roots"]):
        x = torch.zeros(len(a), dtype=torch.float64, device="cuda")
        x[flip] = X[:, k]
        if grads is not None:  # one Newton step on A x = w x, |x| = 1 from the solution: its derivative is the response
            A0, n = A.detach(), len(a)
            w = x @ A0 @ x
            J = torch.zeros(n + 1, n + 1, dtype=torch.float64, device="cuda")
            J[:n, :n] = A0 - w * torch.eye(n, dtype=torch.float64, device="cuda")
            J[:n, n], J[n, :n] = -x, x
            x = x - torch.linalg.solve(J, torch.cat([A @ x - w * x, torch.zeros_like(x[:1])]))[:n]
        w0 = x @ (A @ x)
        L = torch.zeros_like(e1).index_put((a, i), x)

        def energy(r2, f_oo, f_vv, w):
            c = c1_doubles(r2) + e("fn,fnai->ai", L, w) + f_vv @ L - L @ f_oo
            return (L * c).sum()

        R2 = (_pq(e("ijmb,am->abij", ijka, L)) - _rs(e("abej,ei->abij", abci, L))) / (e2 - w0)
        w2 = energy(R2, foo, fvv, wvo)
        C2 = (c2_doubles(R2) - _pq(e("ijmb,am->abij", woo, L))
              + 0.5 * e("abmn,mnij->abij", T2, _rs(e("ej,mnie->mnij", L, ijka)))
              + _rs(_pq(e("aeim,embj->abij", T2, e("fj,febm->embj", L, abci))))
              - _rs(e("abim,mj->abij", T2, e("en,mnie->mi", L, ijka)))
              + _pq(e("aeij,be->abij", T2, e("fm,efam->ae", L, abci))))
        res.append((w0, w2, energy(-C2 / (e2 - w0), foo3, fvv3, wvo3)))
    w = [torch.stack(x) for x in zip(*res)]
    if grads is None:
        stable = torch.linalg.eigvalsh(0.5 * (A + A.T)).min() > 0.05
        return [w[0].cpu(), w[1].cpu(), w[2].cpu() if stable else None]
    g = torch.autograd.grad(sum((x.cuda() * y).sum() for x, y in zip(grads, w)), list(t.values()))
    return w, dict(zip(t, g))


def exact(case, seed):
    st = prepare(case, seed)
    kind = case["kind"]
    if kind == "kernel":
        layouts, spec, f, anti = KERNELS[case["op"]]
        out, amp, ints = st["tensors"]
        d = _Dense(case, {layouts[2]: ints})
        r = d.unpack(amp, layouts[1])
        x = d.ladder(r) if case["op"] == "c2_r2abcd" else f * torch.einsum(spec, r, d[layouts[2]])
        x = _pq(x) if "p" in anti else x
        x = _rs(x) if "r" in anti else x
        return d.pack(x, layouts[0])
    if kind == "batch":
        return [_chain(m, i.t) for m, i in zip(_batch_shapes(case), st["ints"])]
    if kind == "grcpsd":
        return None  # eigenproblems and linear systems over all doubles
    if kind == "grad3":
        w, g = _chain(case, st["t"], st["weights"])
        return dict(energies=[x.detach().cpu() for x in w], grads=g)
    w = _chain(case, st["t"])
    if kind == "cis":
        return dict(omega=w[0], vectors=None)  # a vector is fixed up to its sign
    return dict(omega=w[0], w2=w[1], w3=w[2])
