"""The benchmark's roofline: the work that it counts per update is what the kernel does."""
import numpy as np

import bench


def test_backprojection_bytes_are_those_the_kernel_reads():
    """The roofline's shared-memory bytes per update against a count of the bins that
    patches at drawn ray coordinates read (the last one only where its weight is not 0)."""
    w = bench.WORKLOAD
    th = np.arange(w["n_par_proj"])[:, None] * np.pi / w["n_par_proj"]
    a, b = (w["n_par_det"] / w["n_pixels"] * np.abs(f(th)) for f in (np.cos, np.sin))
    g = np.random.default_rng(0).uniform(0.0, 1.0, (w["n_par_proj"], 4000))  # the lowest pixel above its bin
    far = g + a + b  # the farthest pixel's coordinate
    mid = np.minimum(np.floor(a + b), 2) + 1  # the middle of the three bins it may weigh
    read = mid + 1 + (far > mid)
    # 16 B per bin and quad of slices, 4 pixels x 4 slices; the draw's own error is 2e-4
    assert abs(read.mean() - bench.bp_smem_bytes_per_update("patch_2x2")) < 2e-3
    assert bench.bp_smem_bytes_per_update("staged_s4_a8") == 8.0
