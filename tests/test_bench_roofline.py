"""The bench's roofline records (host arithmetic): a kernel is credited with the products of its own formulation over the rows
that it sees, so no record of a real run passes its peak."""
import pytest

from conftest import ROOT  # noqa: F401 -- puts the repository's root on the path

import bench

PEAKS = dict(bf16_tflops_sustained=1404.3, hbm_gbs=6568.7, source="measured")


# label, milliseconds and launches of a run, workload, heads, chunk; what one launch computes, per head
@pytest.mark.parametrize("label,count,ms,cfg,bh,flops", [
    # the causal blocks of four chunks of 2048 tokens and one of 1808, 8 d products a pair
    ("fm_dense_tc_dkdv", 20, 178.6, "c3", 1024, 8 * 64 * (4 * 2048 * 2049 // 2 + 1808 * 1809 // 2)),
    ("fm_dense_tc_fwd", 20, 75.0, "c3", 1024, 4 * 64 * (4 * 2048 * 2049 // 2 + 1808 * 1809 // 2)),
    ("fm_moments_tc_readout_a", 40, 156.0, "c3", 1024, 2 * 64 * 40 * 65 * (10000 - 2048)),
    ("fm_moments_tc_state", 40, 148.0, "c3", 1024, 2 * 2080 * 64 * 8192)])
def test_moment_family_kernels_get_what_they_compute(label, count, ms, cfg, bh, flops):
    per = {label: (count, ms), "fm_moments_prefix_bf16": (1, 0.1)}
    r = bench.roofline_of(per, bench.cfg_of(cfg), bh, PEAKS, 0)
    assert r["kernel"] == label and r["alg_flops_per_launch"] == flops * bh and r["frac"] < 1
    assert r["achieved"] == pytest.approx(flops * bh / (ms / count * 1e-3) / 1e12)


def test_whole_rows_get_the_cheaper_form():
    for n, form in ((500, 6 * 64 * (500 * 501 // 2)), (100000, 4 * (64 + 64 * 64) * 65 * 100000)):
        cfg = (1, 8, n, 64, "bf16", 1, 2, 1)
        r = bench.roofline_of({"fm_dense_tc_dq": (1, 1.0)}, cfg, 8, PEAKS, 0)
        assert r["alg_flops_per_launch"] == 8 * form


def test_decode_step_moves_a_triangle_in_and_a_square_out():
    assert bench.decode_step_bytes(64, 2) == 4 * 65 * (65 + 36 * 64 + 65 + 4096)
    assert bench.decode_step_bytes(64, 1) == 4 * 65 * 130
