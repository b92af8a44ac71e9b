"""The kernels that read the packed (vv|vo) list (Wmbej_r1abci, Fae_r1abci)
against the oracle where they can go wrong: one to seven chunks of 32 (64)
rows with remainders, row tiles of 8 and strips of 8 at and beside their edges,
more than eight columns, singles of another irrep than 1, irreps without
occupied orbitals, both tile-count instances.

Operands are standard normal, so an output is a sum of at most 2 x 212 terms of
size 1: its FP64 rounding is below 424 eps sqrt(424) = 2e-12, in either order.
"""
import numpy as np
import pytest

import kernel_specs as ks
import oracle_ffi as of
from cpsd_b200 import api, synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["Wmbej_r1abci", "Fae_r1abci"])
@pytest.mark.parametrize("nmo,nocc,nirrep,symr", [
    (110, (3, 1), 1, 1),   # v = 216: seven chunks of 32, four of 64
    (52, (5, 3), 1, 1),    # v = 96: three full chunks of 32
    (53, (5, 4), 1, 1),    # v = 97, nine columns
    (20, (4, 2), 1, 1),    # v = 34: two rows past a chunk of 32
    (13, (2, 1), 1, 1),    # v = 23: less than a chunk
    (90, (7, 5), 2, 2),    # irreps of 84, singles of irrep 2
    (37, (5, 3), 4, 3),
    (35, (3, 1), 8, 1),    # irreps without occupied orbitals
    (35, (9, 7), 8, 6),
])
def test_packed_pair_matches_oracle(name, nmo, nocc, nirrep, symr):
    rng = np.random.default_rng(nmo)
    s = synth.System(nmo=nmo, nocc_a=nocc[0], nocc_b=nocc[1], nirrep=nirrep, seed=2, naux=nirrep, skip_abcd=True,
                     host_ints=False)
    api.use_torch_stream()
    api.init(s.nirrep, s.dirprd)
    of.set_symmetry(s.nirrep, s.dirprd)
    lo, la, lb, _ = ks.KERNELS[name]
    ops = []
    for layout, sym in ((lo, symr), (la, symr), (lb, 1)):
        pops, iops = ks.pops_of(layout, s.popo, s.popv)
        n = s.sym.idsymsoc(sym, pops[0], pops[1], iops[0], pops[2], pops[3], iops[1])
        ops.append((pops, iops, sym, rng.standard_normal(n)))
    ref = ops[0][3].copy()
    args = [of.opt(p, i, y, x) for p, i, y, x in ops]
    args[0] = of.opt(*ops[0][:3], ref)
    assert of.call_kernel(name, *args, 0.7) == 0
    dev = [torch.from_numpy(x).cuda() for _, _, _, x in ops]
    api.contract_timing(True)
    try:
        api.kernel(name, *[api.opt(p, i, y, t) for (p, i, y, _), t in zip(ops, dev)], 0.7)
        _, _, kinds, _ = api.contract_records()
    finally:
        api.contract_timing(False)
    assert 23 in kinds and 40 not in kinds, "the list was expanded"
    assert float(np.max(np.abs(dev[0].cpu().numpy() - ref))) < 2e-12 * (1 + np.max(np.abs(ref)) / 50)


@pytest.mark.parametrize("name", ["Wmbej_r1abci", "Fae_r1abci"])
def test_second_pair_packed(name):
    """A list whose second pair is packed too (its two spaces of the same populations) is a call of the general path,
    which expands both pairs: the result is that of the list with the second pair full."""
    n, rng = 6, np.random.default_rng(1)
    p, z = np.array([n] + [0] * 7, np.int64), np.array([1] + [0] * 7, np.int64)
    api.use_torch_stream()
    api.init(1, np.ones((8, 8), np.int64))
    np2 = n * (n - 1) // 2
    packed = rng.standard_normal((np2, np2))  # column (x, m), x < m; rows (p, q), p < q
    full = np.zeros((n, n, np2))
    cols = [(x, m) for m in range(n) for x in range(m)]
    for k, (x, m) in enumerate(cols):
        full[m, x], full[x, m] = packed[k], -packed[k]
    r = torch.from_numpy(rng.standard_normal(n * n)).cuda()
    pops = [p, p, p, p] if name[0] == "W" else [p, p, z, z]
    got = []
    for iop, x in ((0, packed), (1, full)):
        out = torch.zeros(int(np.prod([q.sum() for q in pops])), dtype=torch.float64, device="cuda")
        api.kernel(name, api.opt(pops, (1, 1), 1, out), api.opt([p, p, z, z], (1, 1), 1, r),
                   api.opt([p] * 4, (0, iop), 1, torch.from_numpy(x.reshape(-1).copy()).cuda()), 0.7)
        got.append(out)
    assert float(got[1].abs().max()) > 0.1
    assert float((got[0] - got[1]).abs().max()) < 1e-13  # sums of up to 36 products of size 1


@pytest.mark.parametrize("name", ["Wmbej_r1abci", "Fae_r1abci"])
def test_records_hold_the_flops(name):
    n, z = 20, np.array([1] + [0] * 7, np.int64)
    v, o = np.array([n] + [0] * 7, np.int64), np.array([3] + [0] * 7, np.int64)
    api.use_torch_stream()
    api.init(1, np.ones((8, 8), np.int64))
    pops = [v, o, v, o] if name[0] == "W" else [v, v, z, z]
    t = [torch.ones(m, dtype=torch.float64, device="cuda")
         for m in (int(np.prod([q.sum() for q in pops])), 3 * n, n * (n - 1) // 2 * 3 * n)]
    ops = [api.opt(pops, (1, 1), 1, t[0]), api.opt([v, o, z, z], (1, 1), 1, t[1]), api.opt([v, v, v, o], (0, 1), 1, t[2])]
    api.contract_timing(True)
    try:
        api.kernel(name, *ops, 0.7)
        _, flops, kinds, _ = api.contract_records()
    finally:
        api.contract_timing(False)
    assert 2.0 * n * 3 * n * n * (3 if name[0] == "W" else 1) in [f for f, k in zip(flops, kinds) if k == 23]
