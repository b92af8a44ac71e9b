"""FP64 contractions with interleaved indices against torch products: small ones, most of which the narrow and short-K
kernels take (contracted range of at most 64, or at most 16 columns), and those of the tile kernel (a record of its
shape is asserted): its tile shapes, whole and split K, both orders in which each operand is contiguous, columns and
rows at and beside the tile edges, contracted ranges beside multiples of a stage of 16, segments shorter than the ring
of three or four stages.  Operands are standard normal: an output is a sum of K products of size 1, its rounding below
K eps sqrt(K)."""
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
SMALL = [
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
]
# the same with the tile shape that takes it, and the letters of the operands: A or B contiguous along its rows
# (columns) or along the contracted index
ROWS, KS = "aebf", "eafb"
COLS, KB = "ifje", "eifj"
TILES = [
    # edges of the tiles and of a stage, one segment
    (16, 8, 17, 1, 13, 5, 1, ROWS, KB, (64, 64)),     # 128 x 17, K = 65
    (17, 8, 33, 1, 79, 1, 1, ROWS, KB, (64, 64)),     # 136 x 33, K = 79
    (13, 5, 65, 1, 16, 5, 1, KS, COLS, (64, 64)),     # 65 x 65, K = 80
    (40, 30, 16, 2, 81, 1, 1, ROWS, COLS, (64, 64)),  # 1200 x 32, K = 81
    (64, 1, 128, 1, 65, 1, 1, KS, KB, (64, 64)),      # 64 x 128, K = 65
    (13, 10, 15, 1, 11, 9, 1, ROWS, KB, (128, 32)),   # 130 x 15, K = 99: at most 16 columns
    (57, 6, 5, 28, 36, 8, 1, KS, KB, (128, 32)),
    (33, 31, 43, 3, 37, 31, 1, ROWS, KB, (64, 64)),
    # whole K
    (20, 7, 7, 68, 7, 11, 1, KS, KB, (64, 64)),
    (16, 5, 51, 29, 13, 6, 1, ROWS, COLS, (64, 64)),
    (38, 28, 70, 47, 37, 9, 2, KS, COLS, (64, 128)),
    (13, 49, 71, 63, 19, 32, 8, KS, KB, (64, 128)),
    (39, 17, 69, 69, 36, 37, 8, ROWS, COLS, (64, 128)),
    (58, 26, 61, 34, 35, 13, 4, KS, KB, (128, 32)),
    (69, 71, 38, 12, 30, 9, 4, ROWS, COLS, (128, 32)),
    (53, 20, 57, 70, 20, 37, 4, KS, KB, (128, 64)),
    (18, 66, 61, 55, 32, 36, 4, ROWS, KB, (128, 64)),
    # parts of K
    (23, 19, 55, 18, 46, 33, 1, ROWS, KB, (64, 128)),
    (19, 17, 46, 26, 40, 20, 1, ROWS, COLS, (128, 64)),
    (11, 43, 52, 17, 38, 23, 1, KS, KB, (128, 64)),
    (22, 15, 28, 10, 16, 35, 2, ROWS, COLS, (128, 32)),
    # segments of 4 to 20, columns of 1 to 16, parts that begin and end inside a segment
    (2, 3, 1, 34, 15, 37, 8, KS, KB, (128, 32)),
    (16, 17, 17, 16, 35, 17, 8, KS, COLS, (128, 32)),
    (27, 13, 14, 37, 20, 30, 8, KS, KB, (128, 32)),
    (29, 42, 37, 9, 11, 29, 4, KS, COLS, (128, 32)),
    (6, 18, 27, 4, 21, 28, 8, KS, KB, (64, 64)),
    (90, 80, 2, 4, 61, 53, 2, ROWS, KB, (128, 32)),   # long K in two segments
]


@pytest.mark.parametrize("a,b,i,j,e,f,nirrep", SMALL)
def test_tiles_match_torch(a, b, i, j, e, f, nirrep):
    contraction(a, b, i, j, e, f, nirrep, "aebf", "eifj")


@pytest.mark.parametrize("a,b,i,j,e,f,nirrep,left,right,shape", TILES)
def test_tile_kernel_matches_torch(a, b, i, j, e, f, nirrep, left, right, shape):
    api.contract_timing(True)
    try:
        contraction(a, b, i, j, e, f, nirrep, left, right)
        kinds = api.contract_records()[2].tolist()
    finally:
        api.contract_timing(False)
    assert kinds == [[(128, 64), (128, 32), (64, 128), (64, 64)].index(shape)]


def contraction(a, b, i, j, e, f, nirrep, left, right):
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
    _, v1, d1 = tensor(left)
    _, v2, d2 = tensor(right)
    ix, v3, d3 = tensor("aibj")
    desc = lambda t: ([P[c] for c in t], (1, 1), 1)  # noqa: E731
    api.vv2v_dpd_444(v1, desc(left), left, v2, desc(right), right, v3, desc("aibj"), "aibj", 0.5, 1.0)
    ref = (d3 + 0.5 * torch.einsum(f"{left},{right}->aibj", d1, d2))[tuple(ix.T)]
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
