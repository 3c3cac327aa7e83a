"""Which models the block sweep takes for their constants (no GPU needed)."""
import math

import pytest

from sapien_gb300 import PinocchioModel, synthetic as syn

LINK = '<link name="{}"><inertial><origin xyz="{}" rpy="0 0 0"/><mass value="{}"/><inertia ixx="{}" iyy="0.02" izz="0.03" ixy="0" ixz="0" iyz="0"/></inertial></link>'


def arm(rpy="0 0 0", com="0.1 0 0.2", mass=1.5, ixx=0.01, xyz="0 0.3 0.1", gravity=(0, 0, -9.81)):
    return PinocchioModel(
        '<robot name="r">' + LINK.format("base", "0 0 0", 1, 0.01) + LINK.format("a", com, mass, ixx)
        + LINK.format("b", com, mass, ixx)
        + f'<joint name="j" type="revolute"><origin xyz="{xyz}" rpy="{rpy}"/><parent link="base"/><child link="a"/>'
        '<axis xyz="0 0 1"/><limit effort="0" velocity="0" lower="-1" upper="1"/></joint>'
        f'<joint name="k" type="continuous"><origin xyz="{xyz}" rpy="{rpy}"/><parent link="a"/><child link="b"/>'
        '<axis xyz="1 0 0"/></joint></robot>', gravity)


@pytest.mark.parametrize("rpy", [f"{r!r} {p!r} {y!r}" for r in (0.0, math.pi / 2, math.pi, -math.pi / 2)
                                 for p in (0.0, math.pi / 2, math.pi) for y in (0.0, math.pi, math.pi / 2)])
def test_residues_of_right_angles_are_in_range(rpy):
    assert arm(rpy).block_sweep


def test_small_entries_beside_larger_ones_are_in_range():
    assert arm(com="1e-40 0.1 -3e-200", xyz="0 1e-33 0.4", gravity=(1e-60, 0, -9.81)).block_sweep
    assert arm(com="0 0 0", xyz="0 0 0", gravity=(0, 0, 0)).block_sweep


@pytest.mark.parametrize("what", [{"com": "1e31 0 0"}, {"xyz": "0 0 1e-40"}, {"mass": 1e-35}, {"mass": 1e40},
                                  {"ixx": 1e35}, {"gravity": (0, 0, 1e-32)}, {"gravity": (0, 1e32, 0)}])
def test_blocks_out_of_range_are_not(what):
    assert not arm(**what).block_sweep


def test_trees_that_do_not_fit_a_block_and_settings_that_ask_for_fp64():
    assert PinocchioModel(syn.serial_chain(40, seed=1).urdf).block_sweep
    assert not PinocchioModel(syn.serial_chain(63, seed=1).urdf).block_sweep
    m = arm()
    m.set_lanes(1)
    assert not m.block_sweep
    m.set_lanes(0)
    assert m.block_sweep
