"""The byte model of the tracer kernels: the winds' fields once a launch, the
tracer's own fields once a tracer, one launch for up to four tracers."""
import importlib

import pytest


@pytest.fixture(scope="module")
def rf():
    return importlib.import_module("pynicam-dc_b200.roofline")


def test_one_tracer_counts_every_field_once(rf):
    n, n2 = 1000, 25
    for k, (reads, writes, planes) in rf.KERNELS.items():
        want = sum(rf.esize(c, "mixed") for _, c in reads + writes) * n + len(planes) * 4 * n2
        assert rf.kernel_bytes(k, n, n2, "mixed") == want
        assert rf.kernel_passes(k) == (len(reads) + len(writes), len(planes))


@pytest.mark.parametrize("nq", [1, 3, 4, 5, 17])
def test_batches_read_the_winds_fields_once(rf, nq):
    n, n2 = 1000, 25
    launches, b = rf.step_launches(nq=nq), rf.step_bytes(n, n2, 0, nq=nq)
    batches = (nq + 3) // 4
    assert launches["trc_vadv"] == 2 and launches["trc_remap"] == launches["trc_apply"] == batches
    assert sum(rf.launch_tracers("trc_grad", nq)) == nq and len(rf.launch_tracers("trc_grad", nq)) == batches
    # k_trc_remap: centroids and masks (12) a launch; q, three gradients, three faces a tracer; 3 planes
    assert b["trc_remap"] == 8 * (n * (12 * batches + 7 * nq) + 3 * n2 * batches)
    # k_trc_apply: masks and fluxes (9) a launch; faces, q, bounds and the mass (read, written) a tracer
    assert b["trc_apply"] == 8 * n * (9 * batches + 8 * nq)
    # k_trc_vadv: density, flux and tendency a launch; the mass read and written a tracer, two sweeps
    assert b["trc_vadv"] == 8 * n * 2 * (3 + 2 * nq)
    one = rf.step_bytes(n, n2, 0, nq=1)
    assert all(b[k] == one[k] for k in b if not k.startswith("trc_") and k not in ("comm", "total"))
    assert rf.field_passes(nq=nq) >= rf.field_passes(nq=1)
