"""The page-locked blocks that a step runner's logits live in, over a fake allocator: no GPU."""
import ctypes
import gc

import numpy as np

from easy_gpt.cpp_b200.native import _HostBlocks


class FakeLibrary:
    def __init__(self):
        self.live = {}

    def ege_host_alloc(self, size):
        memory = ctypes.create_string_buffer(size)
        self.live[ctypes.addressof(memory)] = memory
        return ctypes.addressof(memory)

    def ege_host_free(self, address):
        del self.live[address]                                     # a second free of a block is a KeyError


def test_blocks_are_taken_again_only_when_every_view_is_gone():
    lib = FakeLibrary()
    blocks = _HostBlocks(lib)
    a = blocks.array(3, 40000)
    a[:] = 1.0
    row = a[2]
    del a
    b = blocks.array(3, 40000)
    b[:] = 2.0
    assert len(lib.live) == 2 and np.all(row == 1.0)
    del row
    gc.collect()
    c = blocks.array(3, 40000)
    assert len(lib.live) == 2 and c.shape == (3, 40000) and c.dtype == np.float32 and c.flags.writeable
    assert blocks.array(1, 100) is None                            # small arrays live in plain memory


def test_the_limit_holds_other_sizes_make_room_and_close_frees_all():
    lib = FakeLibrary()
    blocks = _HostBlocks(lib)
    blocks.LIMIT = 4 << 20
    held = [blocks.array(1, 1 << 18) for _ in range(4)]            # 1 MB each
    assert all(h is not None for h in held) and blocks.array(1, 1 << 18) is None
    del held[1:]
    gc.collect()
    big = blocks.array(1, 3 << 18)                                 # the three free blocks go for it
    assert big is not None and len(lib.live) == 2
    blocks.close()
    assert len(lib.live) == 2                                      # both are handed out still
    del held, big
    gc.collect()
    assert not lib.live
