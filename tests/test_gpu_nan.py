"""NaN and infinities in the solvers.  Symmetric Ritz problem: the eigen-solve and the SF-CIS program end without an error,
with NaN values and without a write outside their buffers, for even and odd subspaces (an odd one is padded by one
place).  DIIS: the same of the loop whose pivots are NaN."""
import numpy as np
import pytest

from cpsd_b200 import api, synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 4, 5, 19, 31, 32])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_eigen_solve_takes_nan(n, bad):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n))
    A = A + A.T
    A[0, n - 1] = A[n - 1, 0] = bad
    w, V = api.syev(A)
    assert np.isnan(w).all()
    B = np.diag(np.arange(1.0, n + 1))  # the next call's result is not touched by this one
    w, V = api.syev(B)
    assert np.array_equal(w, np.arange(1.0, n + 1)) and np.array_equal(V, np.eye(n))


@pytest.mark.parametrize("roots", [2, 3, 4, 5])
def test_cis_takes_nan(roots):
    s = synth.System(nmo=20, nocc_a=4, nocc_b=2, nirrep=1, seed=5, roots=roots, skip_abcd=True,
                     run_opts=dict(lowest=1))
    api.use_torch_stream()
    good, _, _ = api.cis_run(s, api.make_system(s), api.DeviceIntegrals(s), api.make_params(s))
    s.ints["iabj"][:] = np.nan
    om, R, it = api.cis_run(s, api.make_system(s), api.DeviceIntegrals(s), api.make_params(s))
    assert np.isnan(om).all()
    s = synth.System(nmo=20, nocc_a=4, nocc_b=2, nirrep=1, seed=5, roots=roots, skip_abcd=True,
                     run_opts=dict(lowest=1))
    again, _, _ = api.cis_run(s, api.make_system(s), api.DeviceIntegrals(s), api.make_params(s))
    assert np.array_equal(good, again)


def test_diis_takes_nan():
    s = synth.System(nmo=24, nocc_a=5, nocc_b=3, nirrep=2, seed=6, roots=1)
    api.use_torch_stream()
    good = api.ground(s, api.make_system(s), api.DeviceIntegrals(s), api.make_params(s))
    for x in s.ints.values():
        x[:] = np.nan
    bad = api.ground(s, api.make_system(s), api.DeviceIntegrals(s), api.make_params(s))
    assert np.isnan(bad["E3"]) and torch.isnan(bad["T1_2"]).any()
    s = synth.System(nmo=24, nocc_a=5, nocc_b=3, nirrep=2, seed=6, roots=1)
    again = api.ground(s, api.make_system(s), api.DeviceIntegrals(s), api.make_params(s))
    assert good["E3"] == again["E3"] and torch.equal(good["T1_2"], again["T1_2"])
