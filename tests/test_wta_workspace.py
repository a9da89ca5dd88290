"""The winner selection's workspace: the scan's candidates are F32's alone."""

from spyker_b200 import _lib


def test_integer_input_needs_the_keys_alone():
    conv, fc = _lib.lib.spk_rank_convwta_workspace, _lib.lib.spk_rank_fcwta_workspace
    assert conv(4096, 0, 30, 28, 28) == 0  # keys in shared memory
    assert conv(4096, 15, 30, 28, 28) >= 4096 * 30 * 784 * 6
    assert conv(2, 0, 60, 28, 28) == 2 * 60 * 784 * 4  # keys in global memory
    assert fc(64, 1000, 100) == 0 and fc(64, 0, 50000) == 64 * 50000 * 4
