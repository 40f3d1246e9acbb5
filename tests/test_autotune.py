"""The autotuner times a setting only where the workload's world has a launch that it shapes."""
from beamlab_b200 import autotune


def test_candidates_by_world_size():
    assert set(autotune.candidates(943132, 8870418)) == {"beams_per_sm", "force_block", "integrate_block"}
    assert set(autotune.candidates(6001, 4000000)) == {"force_block", "integrate_block"}
    assert set(autotune.candidates(400, 3121)) == {"integrate_block"}
    src = open(autotune.HERE + "/csrc/bl_world.cu").read()
    assert f"kPlainBeams = {autotune.PLAIN_BEAMS}, kWideNodes = {autotune.WIDE_NODES};" in src
