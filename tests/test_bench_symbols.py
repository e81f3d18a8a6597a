"""Kernel names that the bench prints for a handle's own launch configuration (CPU)."""

from __future__ import annotations

import bench

CONFIG = {"fused_transverse": False, "persistent_z": True, "slabs": 1, "launches_per_step": 8, "tma_staging": False}


def test_odd_rows_run_the_persistent_z_passes():
    assert bench.slot_symbols((64, 63, 64), config=CONFIG)[3] == "kfp_zpass_u<64>"
    assert bench.slot_symbols((64, 63, 320), config=CONFIG)[3::4] == ["kfp_zpass_u<320>", "kfp_zpass_p<320,false>"]
    one_tile = {**CONFIG, "persistent_z": False}
    assert bench.slot_symbols((64, 63, 64), config=one_tile)[3] == "kf_zpass_u<64>"
    assert bench.slot_symbols((64, 63, 320), config=one_tile)[3] == "kfp_zpass_u<320>"  # no one-tile kernel
    assert bench.slot_symbols((64, 63, 405), config=CONFIG)[3] == "k_zpass_u"


def test_one_x_plane_runs_a_transverse_chain_in_one_kernel():
    names = bench.slot_symbols((1, 96, 128), config={**CONFIG, "launches_per_step": 4})
    assert names[0] == "kf_plane<96,false>" and names[4] == "kf_plane<96,true>"
    assert [n for n in names if n] == [names[0], names[3], names[4], names[7]]
    assert bench.slot_symbols((1, 405, 16), config=CONFIG)[0] == "k_ypass"


def test_even_rows_are_named_as_without_a_configuration():
    tma = {**CONFIG, "tma_staging": True}
    assert bench.slot_symbols((192, 192, 256), config=tma) == bench.slot_symbols((192, 192, 256), tma=True)
