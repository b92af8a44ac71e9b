"""The Davidson and DIIS step kernels at the sizes where their split over a
cluster of CTAs changes: one CTA, the first split, the largest portable
cluster, 16 CTAs with the vectors in shared memory and beyond it, more than
eight roots (two coefficient passes, a collapse of more than eight vectors).

SF-CIS roots against dense diagonalisation: the eigenvalue error is second
order in the residual (1e-10 here) and rounding leaves about n eps |A| (n up
to 4000, |A| of a few Eh), so 1e-11 Eh bounds both.  The DIIS loop against
the oracle's, which takes the same steps: rounding differences of 1e-16 grow
through the extrapolations of a converging loop, 1e-9 of the amplitudes'
size, the loop's own tolerance being 1e-7.  Nine and more roots get a basis of
32: in one of 20 they take 86 to over 300 cycles from seed to seed (and end at
the cycle limit at some, as one-CTA steps do), a count that rounding decides.
"""
import numpy as np
import pytest

import oracle_ffi as of
from cpsd_b200 import api, synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# nmo, nocc_a, nirrep, roots -> vector length of irrep 1
@pytest.mark.parametrize("nmo,nocc_a,nirrep,roots", [
    (19, 4, 1, 2),    # 192: one CTA, full
    (20, 4, 1, 3),    # 204: two CTAs
    (31, 5, 1, 9),    # 432: four CTAs, nine roots
    (48, 9, 1, 5),    # 1280: eight CTAs
    (85, 10, 1, 4),   # 2736: 16 CTAs, vectors in shared memory
    (85, 10, 1, 12),  # the same, vectors in global memory
    (101, 12, 1, 2),  # 3960: 16 CTAs, in shared memory
    (105, 12, 1, 5),  # 4136: longer than the shared memory holds, collapses of ten vectors
])
def test_cis_roots_match_dense(nmo, nocc_a, nirrep, roots):
    s = synth.System(nmo=nmo, nocc_a=nocc_a, nocc_b=nocc_a - 2, nirrep=nirrep, seed=3, roots=roots, skip_abcd=True,
                     run_opts=dict(lowest=1, davidson_conv=10, davidson_cyc=300, davidson_dim=20 if roots < 9 else 32))
    api.use_torch_stream()
    ints = api.DeviceIntegrals(s)
    om, R, it = api.cis_run(s, api.make_system(s), ints, api.make_params(s))
    check_cis(s, om, R, roots)


def check_cis(s, om, R, roots):
    """roots against dense diagonalisation of the spin-flip block: alpha occupied to beta virtual"""
    o, v = int(s.popo.sum()), int(s.popv.sum())
    n = o * v
    V = torch.from_numpy(s.ints["iabj"]).cuda().view(n, n)  # element (fn, ai) of the column-major block: row (ai)
    e1 = (torch.from_numpy(s.eorb[o:])[None, :] - torch.from_numpy(s.eorb[:o])[:, None]).reshape(-1).cuda()
    A = V + torch.diag(e1)
    a, i = np.meshgrid(np.arange(v), np.arange(o))
    flip = torch.from_numpy(np.nonzero((a.reshape(-1) >= s.vrta[0]) & (i.reshape(-1) < s.popa[0]))[0]).cuda()
    w = torch.linalg.eigvalsh(A[flip][:, flip])[:roots].cpu().numpy()
    assert np.max(np.abs(np.sort(om) - w)) < 1e-11
    X = R.view(roots, n)
    res = X @ A.T - torch.from_numpy(om).cuda()[:, None] * X
    assert float(res.abs().max()) < 1e-9
    G = X @ X.T
    assert float((G - torch.eye(roots, dtype=torch.float64, device="cuda")).abs().max()) < 1e-8


# basis, roots: a collapse that keeps roots + 5, then those where that is the whole basis or more (the roots are kept)
@pytest.mark.parametrize("dim,roots", [(20, 14), (20, 15), (20, 16), (20, 19), (32, 27), (32, 28), (32, 31)])
@pytest.mark.parametrize("nmo", [28, 101])  # 384 elements: four CTAs, in shared memory; 3960: 16, in global memory
def test_many_roots_in_a_small_basis(nmo, dim, roots):
    s = synth.System(nmo=nmo, nocc_a=5 if nmo < 50 else 12, nocc_b=3 if nmo < 50 else 10, nirrep=1, seed=3, roots=roots,
                     skip_abcd=True,
                     run_opts=dict(lowest=1, davidson_conv=10, davidson_cyc=3000, davidson_dim=dim))
    s.ints["iabj"] *= 0.02 if nmo < 50 else 0.004  # one to six free places: weakly coupled configurations converge
    api.use_torch_stream()
    om, R, _ = api.cis_run(s, api.make_system(s), api.DeviceIntegrals(s), api.make_params(s))
    check_cis(s, om, R, roots)


@pytest.mark.parametrize("nmo,nocc_a,nirrep", [(28, 5, 1), (36, 6, 1), (44, 8, 1), (44, 9, 1), (80, 14, 2), (56, 16, 1),
                                               (72, 24, 1)])
def test_diis_loop_matches_oracle(nmo, nocc_a, nirrep):
    """T1^(2) vectors of 384 elements (one CTA), 620 (two), 1036, 1152 and 1744 (four), 2460 (eight), 4508 (16)"""
    s = synth.System(nmo=nmo, nocc_a=nocc_a, nocc_b=nocc_a - 2, nirrep=nirrep, seed=4, roots=1)
    # weaker integrals keep the singles equations definite at these sizes, so that the loop converges
    for k, x in s.ints.items():
        x *= 0.1
    api.use_torch_stream()
    g = api.ground(s, api.make_system(s), api.DeviceIntegrals(s), api.make_params(s))
    r = of.Oracle(s, nthreads=8).ground()
    t = g["T1_2"].cpu().numpy()
    ref = r["T1_2"]
    assert g["iters"] == r["iters"]
    assert np.linalg.norm(t - ref) < 1e-9 * np.linalg.norm(ref)
    assert abs(g["E3"] - r["E3"]) < 1e-11 * max(1.0, abs(r["E3"]))


@pytest.mark.parametrize("cap", [1, 2, 4, 8])
def test_smaller_clusters(cap):
    """A device that holds only smaller clusters: the same roots and amplitudes from fewer CTAs."""
    s = synth.System(nmo=60, nocc_a=9, nocc_b=7, nirrep=1, seed=5, roots=3,
                     run_opts=dict(lowest=1, davidson_conv=9, davidson_cyc=100))
    for x in s.ints.values():  # the singles equations converge, as above
        x *= 0.1
    api.use_torch_stream()
    ints, sysc, par = api.DeviceIntegrals(s), api.make_system(s), api.make_params(s)
    om, R, _ = api.cis_run(s, sysc, ints, par)
    g = api.ground(s, sysc, ints, par)
    api.check(api.lib().cpsd_debug_team_cap(api.I64(cap)), "cap")
    try:
        om1, R1, _ = api.cis_run(s, sysc, ints, par)
        g1 = api.ground(s, sysc, ints, par)
    finally:
        api.check(api.lib().cpsd_debug_team_cap(api.I64(16)), "cap")
    assert np.max(np.abs(om1 - om)) < 1e-11
    assert float((R1 - R).abs().max()) < 1e-7
    assert g["iters"] == g1["iters"]
    assert float((g1["T1_2"] - g["T1_2"]).norm()) < 1e-9 * float(g["T1_2"].norm())
