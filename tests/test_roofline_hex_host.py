"""The FP64 operations that the element-by-element rooflines divide by time."""
from solvix_b200.roofline import HEX_ELEMENT_FLOPS, HEX_NODE_FLOPS, hex_iteration_flops


def test_operations_of_the_160x16x16_cantilever():
    assert HEX_ELEMENT_FLOPS == 1605 and HEX_NODE_FLOPS == 54
    assert hex_iteration_flops(40_960, 46_529) == 1605 * 40_960 + 54 * 46_529
