"""What the emulation of several ranks on one GPU refuses, before it looks for one. No call here has tensors."""
import ctypes

import pytest

from switchml_b200._native import last_error, lib

F32, I32, BF16 = 0, 1, 2
SUM, QUANT = 0, 1
STAGED, ONESHOT, PUSH = 0, 1, 3


def _call(elem=F32, mode=QUANT, algo=STAGED, block=256, slot_bytes=131072, slots=2, n=2):
    none = (ctypes.c_void_p * n)()
    rc = lib().sml_emu_allreduce(n, none, none, 1 << 18, elem, mode, algo, block, slot_bytes, slots, 0, 1.0, 1, -1)
    return rc, last_error()


def _looked_for_tensors(rc, why):
    return rc == -1 and why == "a rank has no tensor"


@pytest.mark.parametrize("algo", [STAGED, PUSH])
@pytest.mark.parametrize("block", [1, 16, 31, 48, 100, 384, 2048])
def test_blocks_that_the_exact_kernels_have_no_room_for(algo, block):
    for elem in (F32, BF16):
        rc, why = _call(elem=elem, algo=algo, block=block, slot_bytes=16384)
        assert rc == -1 and "power of two" in why
    for elem, mode in ((F32, SUM), (BF16, SUM), (I32, QUANT)):  # plain sums have no blocks
        assert _looked_for_tensors(*_call(elem=elem, mode=mode, algo=algo, block=block, slot_bytes=16384))


def test_no_block_at_all():
    for algo in (STAGED, ONESHOT, PUSH):
        for block in (0, -5):
            assert _call(algo=algo, block=block)[0] == -1


@pytest.mark.parametrize("block", [32, 64, 128, 256, 512, 1024])
def test_blocks_of_contexts(block):
    for algo in (STAGED, ONESHOT, PUSH):
        assert _looked_for_tensors(*_call(algo=algo, block=block))


def test_slots_without_room():
    assert _call(slots=0)[0] == -1 and _call(slot_bytes=0)[0] == -1 and _call(slot_bytes=1023)[0] == -1
    assert _call(elem=BF16, slot_bytes=1024)[0] == -1 and _looked_for_tensors(*_call(elem=BF16, slot_bytes=2048))
    assert _looked_for_tensors(*_call(slot_bytes=1024)) and _looked_for_tensors(*_call(slot_bytes=100001))
    assert _looked_for_tensors(*_call(algo=ONESHOT, slots=0, slot_bytes=0))


def test_numbers_of_other_types():
    """Python converts what the native call would not take."""
    import torch
    from switchml_b200.ops.emulation import emulated_allreduce
    xs = [torch.ones(4) for _ in range(2)]
    for options in ({"exponent_lookahead": 2.0}, {"exponent_lookahead": "2"}, {"post_scale": "0.5"}, {"post_scale": 1}):
        with pytest.raises(AssertionError):  # the tensors are not on a GPU: nothing else is wrong
            emulated_allreduce(xs, mode="sum", **options)
