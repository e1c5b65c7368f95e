"""Names of the network's Python interface that programs call besides its passes."""
from hemelb_gb300 import nn


def test_tc_tiles():
    assert nn.tc_tiles(1, 1, 1, 1) == 1
    assert nn.tc_tiles(4, 96, 96, 96) == 4 * 48 * 6 * 12
    assert nn.tc_tiles(2, 3, 17, 9) == 2 * 2 * 2 * 2
