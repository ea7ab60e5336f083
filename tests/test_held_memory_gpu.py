"""Device memory the library holds between calls: pa_basis_cache_clear gives back
the scratch memory and pools, and a batch that is not recorded for replay does not
leave more behind than the bound in pa_b200.h."""

import pytest

from pysisyphus_addons import _native as nat
from pysisyphus_addons.common.synthetic import make_workload

pytestmark = pytest.mark.gpu

BOUND = 4 << 30  # scratch of an unrecorded batch that stays with the library


def run_batch(natoms, nmol):
    """The same molecule nmol times; (bytes of its metric, outputs)."""
    torch = pytest.importorskip("torch")
    w = make_workload(natoms, 3, 4, 6, seed=1)
    orb, aux = nat.Basis(w.shells, "orbital"), nat.Basis(w.shells_aux, "aux")
    D = torch.from_numpy(w.densities.copy()).cuda()
    outs = [torch.empty(6**4, dtype=torch.float64, device="cuda") for _ in range(nmol)]
    nat.df_4d_batch([orb] * nmol, [aux] * nmol, [D] * nmol, [6] * nmol, outs, use_graph=False)
    return 8 * aux.nsph**2, outs


def free(torch):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


@pytest.fixture(autouse=True)
def exact_boys():
    nat.set_boys_mode("exact")
    nat.set_metric_shift(1e-7)
    yield
    nat.set_metric_shift(0.0)
    nat.set_boys_mode("reference")


def test_cleared_memory_is_given_back():
    torch = pytest.importorskip("torch")
    one, outs = run_batch(30, 4)
    held = free(torch)
    nat.clear_basis_cache()
    assert free(torch) - held >= 4 * one
    again = run_batch(30, 4)[1]  # and the next call takes it again
    for a, b in zip(outs, again):
        assert torch.equal(a, b)


def test_large_batch_is_not_kept():
    torch = pytest.importorskip("torch")
    run_batch(5, 2)  # kernels and contexts are loaded
    nat.clear_basis_cache()
    before = free(torch)
    run_batch(35, 32)
    # (reserving adds a quarter and 64 MiB; another 64 MiB for what else a first call may map)
    assert before - free(torch) <= BOUND * 5 // 4 + (128 << 20)
