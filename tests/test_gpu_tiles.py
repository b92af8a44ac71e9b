"""The FP64 tile kernel at the edges of its tile shapes and K split: one column
to one beside each tile width, rows beside the tile heights, contracted ranges
of one, around a stage of 16, around the shortest part (32) and across several
irrep segments, against torch FP64 products.  Operands are standard normal: an
output is a sum of K products of size 1, its rounding below K eps sqrt(K)."""
import numpy as np
import pytest

from cpsd_b200 import api
from cpsd_b200.dpd import Symmetry, xor_dirprd

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def pops(n, nirrep):
    p = np.zeros(8, np.int64)
    p[:nirrep] = n // nirrep
    p[:n % nirrep] += 1
    return p


# M, N, K as products of two free letters each: (a b), (i j), (e f)
@pytest.mark.parametrize("a,b,i,j,e,f,nirrep", [
    (9, 9, 5, 5, 1, 1, 1),        # K = 1
    (13, 10, 15, 1, 5, 3, 1),     # 130 x 15, K = 15
    (16, 8, 17, 1, 16, 1, 1),     # 128 x 17, K = 16
    (17, 8, 33, 1, 17, 1, 1),     # 136 x 33, K = 17
    (13, 5, 65, 1, 21, 3, 1),     # 65 x 65, K = 63: one part
    (40, 30, 16, 2, 64, 1, 1),    # 1200 x 32, K = 64: two parts
    (33, 31, 43, 3, 37, 31, 1),   # 1023 x 129, K = 1147
    (90, 80, 2, 4, 61, 53, 2),    # long K in two segments, eight columns
    (21, 23, 9, 11, 13, 17, 4),
    (21, 23, 9, 11, 13, 17, 8),
])
def test_tiles_match_torch(a, b, i, j, e, f, nirrep):
    sym = Symmetry(nirrep, xor_dirprd(nirrep))
    api.init(nirrep, xor_dirprd(nirrep))
    api.use_torch_stream()
    P = {k: pops(n, nirrep) for k, n in zip("abijef", (a, b, i, j, e, f))}
    off = {k: np.concatenate([[0], np.cumsum(p)]) for k, p in P.items()}

    def layout(letters):
        """(orbital numbers of every stored element) of a full 4-index tensor, storage order"""
        p, q, r, s = letters
        out = []
        for R in range(nirrep):
            right = [(x, y) for y in range(nirrep) for x in [y ^ R]]
            rr = [(off[r][x] + u, off[s][y] + w) for x, y in right for w in range(P[s][y]) for u in range(P[r][x])]
            ll = [(off[p][x] + u, off[q][y] + w) for x, y in right for w in range(P[q][y]) for u in range(P[p][x])]
            if rr and ll:
                rr, ll = np.array(rr), np.array(ll)
                out.append(np.concatenate([np.tile(ll, (len(rr), 1)), np.repeat(rr, len(ll), 0)], 1))
        return np.concatenate(out)

    g = torch.Generator(device="cuda").manual_seed(7)

    def tensor(letters):
        ix = torch.from_numpy(layout(letters)).cuda()
        v = torch.randn(len(ix), dtype=torch.float64, device="cuda", generator=g)
        D = torch.zeros([int(P[c].sum()) for c in letters], dtype=torch.float64, device="cuda")
        D[tuple(ix.T)] = v
        return ix, v, D

    # interleaved letters, so that no pair stays whole and every index goes by its stride
    _, v1, d1 = tensor("aebf")
    _, v2, d2 = tensor("eifj")
    ix, v3, d3 = tensor("aibj")
    desc = lambda t: ([P[c] for c in t], (1, 1), 1)  # noqa: E731
    api.vv2v_dpd_444(v1, desc("aebf"), "aebf", v2, desc("eifj"), "eifj", v3, desc("aibj"), "aibj", 0.5, 1.0)
    ref = (d3 + 0.5 * torch.einsum("aebf,eifj->aibj", d1, d2))[tuple(ix.T)]
    K = e * f
    assert float((v3 - ref).abs().max()) < 4 * K * 2.3e-16 * np.sqrt(K) + 1e-14


def test_small_workspace_keeps_the_fixed_tiles():
    """A caller's workspace too small for the chosen K parts still serves a contraction that the fixed rule (parts of
    256 and more) does without partial tiles."""
    n, k = 40, 176
    api.init(1, xor_dirprd(1))
    api.use_torch_stream()
    P = {"a": pops(n, 1), "b": pops(n, 1), "e": pops(k, 1), "z": pops(1, 1)}
    g = torch.Generator(device="cuda").manual_seed(3)
    A, B = (torch.randn(n * k, dtype=torch.float64, device="cuda", generator=g) for _ in range(2))
    C = torch.zeros(n * n, dtype=torch.float64, device="cuda")
    ws = torch.empty(256, dtype=torch.float64, device="cuda")
    z = P["z"]
    args = (A, ([P["a"], P["e"], z, z], (1, 1), 1), "ae..", B, ([P["e"], P["b"], z, z], (1, 1), 1), "eb..", C,
            ([P["a"], P["b"], z, z], (1, 1), 1), "ab..", 1.0, 0.0)
    api.check(api.lib().cpsd_set_workspace(api.dptr(ws), api.ctypes.c_size_t(ws.numel() * 8)), "workspace")
    try:
        api.vv2v_dpd_444(*args)
    finally:
        api.check(api.lib().cpsd_set_workspace(None, api.ctypes.c_size_t(0)), "workspace")
    ref = (B.view(n, k) @ A.view(k, n)).reshape(-1)  # column-major storage
    assert float((C - ref).abs().max()) < 4 * k * 2.3e-16 * np.sqrt(k)
