"""The committed counters that bench.py divides by a peak are of bytes that were moved: at the
capture's own times they stay below the rates that this GPU's L2 and HBM reach. CPU only."""
import bench

SAMPLES = 480 * 270 * 64  # of the captured frame
L2_READ, HBM = 18.6e12, 6.8e12  # bytes a second, as probed


def test_counters_stay_below_the_peaks():
    kernels = bench.kernel_profile()
    for name in ("k_wf_extend", "k_wf_shadow", "k_wf_shade"):
        k = kernels[name]
        seconds = k["device_ms_cold"] * 1e-3
        assert 0.0 < k["l2_read_bytes_per_sample"] * SAMPLES / seconds < L2_READ
        assert 0.0 < k["dram_bytes_per_sample"] * SAMPLES / seconds < HBM
