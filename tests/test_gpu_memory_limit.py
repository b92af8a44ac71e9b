"""Fresh plans on a card without free memory: their tables take the place of what the library keeps between calls (idle
buffers of cached copies) and, inside a program, of cached copies themselves; the results are those of a card with
room."""
import ctypes

import numpy as np
import pytest

from cpsd_b200 import api, synth
from cpsd_b200.dpd import xor_dirprd

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture
def full_card():
    """fill() takes all device memory but the last MB; released at the end (or by calling fill.free())"""
    rt = ctypes.CDLL("libcudart.so.12")
    held = []

    def fill():
        torch.cuda.synchronize()
        size = 64 << 30
        while size >= 1 << 20:
            p = ctypes.c_void_p()
            if rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(size)) == 0:
                held.append(p)
            else:
                rt.cudaGetLastError()
                size //= 2

    def free():
        torch.cuda.synchronize()
        while held:
            assert rt.cudaFree(held.pop()) == 0

    fill.free = free
    yield fill
    free()


def molecule(nmo, nirrep, seed):
    s = synth.System(nmo=nmo, nocc_a=6, nocc_b=4, nirrep=nirrep, seed=seed, roots=1, host_ints=False)
    t = synth.device_integrals(s)
    return s, api.make_system(s), api.DeviceIntegrals.from_tensors(t), api.make_params(s)


@pytest.fixture
def mixed():
    api.use_torch_stream()
    api.set_mixed(6, 0.0)
    yield
    api.set_mixed(0)


def test_tables_take_idle_buffers(full_card, mixed):
    api.ground(*molecule(60, 1, 1))  # leaves its digit tiles as idle buffers
    api.set_mixed(0)
    api.init(8, xor_dirprd(8))
    g = torch.Generator(device="cuda").manual_seed(1)
    calls = []
    for k in range(9):  # a few MB of tables each
        p = np.full(8, 4, np.int64)
        p[:k] += 1
        n = sum(sum(p[a] * p[a ^ r] for a in range(8)) ** 2 for r in range(8))
        v1, v2 = (torch.randn(int(n), dtype=torch.float64, device="cuda", generator=g) for _ in range(2))
        calls.append((([p] * 4, (1, 1), 1), v1, v2, torch.zeros_like(v1)))

    def run(d, v1, v2, v3):
        api.vv2v_dpd_444(v1, d, "aebf", v2, d, "eifj", v3, d, "aibj", 1.0, 0.0)

    run(*calls[0])  # the kernels are loaded
    full_card()
    for c in calls:
        run(*c)
    full_card.free()
    for c in calls:
        kept = c[3].clone()
        run(*c)
        assert torch.equal(kept, c[3]) and float(kept.abs().max()) > 0.0


@pytest.mark.parametrize("nirrep", [1, 2])
def test_program_at_the_limit(full_card, mixed, nirrep):
    small = molecule(53, nirrep, 2 + nirrep)  # shapes that no other test has
    api.ground(*molecule(61, nirrep, 3))
    room = [torch.empty(20 << 20, dtype=torch.uint8, device="cuda") for _ in range(4)]  # the caller's own outputs
    del room
    full_card()
    got = api.ground(*small)
    full_card.free()
    ref = api.ground(*small)
    assert torch.equal(got["T1_2"], ref["T1_2"]) and got["E3"] == ref["E3"] and not np.isnan(got["E3"])
