"""Every candidate that the autotuner times is a launch of its own: the settings
that a limit would make equal are listed once."""
from voxelmapping_b200 import autotune as AT
from voxelmapping_b200 import build as B


def test_candidates_differ():
    for f, values in AT.CANDIDATES.items():
        assert len(set(values)) == len(values) >= 2, f


def test_mesh_candidates_differ_below_the_resident_grid():
    """The mesh kernels run CTAs of 128 threads, twice the setting and at most what an SM holds."""
    report = {k: r for k, r in B.ptxas_report().items() if "mesh_kernel" in k}
    counting = [r for k, r in report.items() if ", false>" in k]
    assert len(report) == 8 and len(counting) == 4

    def fit(r):  # resident CTAs by registers (in eights), shared memory (1 KB a CTA reserved) and threads
        return min(65536 // (128 * (-(-r["registers"] // 8) * 8)), 227 * 1024 // (r["smem"] + 1024), 16)
    most = min(fit(r) for r in counting)
    grids = [min(2 * c, most) for c in AT.CANDIDATES["mesh_ctas_per_sm"]]
    assert len(set(grids)) == len(grids), (grids, most)
