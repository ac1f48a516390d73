"""The blocks that a step runner's logits live in: over a fake allocator, and on a GPU what their users see of them."""
import ctypes
import gc
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from easy_gpt.cpp_b200.native import _HostBlocks


class FakeLibrary:
    def __init__(self):
        self.live = {}

    def ege_host_pin(self, address):
        assert address in self.live
        return 1

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


class CountingLibrary(FakeLibrary):
    def __init__(self):
        super().__init__()
        self.allocated, self.pinned = 0, []

    def ege_host_alloc(self, size):
        self.allocated += 1
        return super().ege_host_alloc(size)

    def ege_host_pin(self, address):
        self.pinned.append(address)
        return super().ege_host_pin(address)


def test_only_blocks_that_come_back_are_page_locked_and_each_once():
    lib = CountingLibrary()
    blocks = _HostBlocks(lib)
    kept = [blocks.array(8, 100000) for _ in range(5)]             # 3.2 MB each, kept: nothing is locked
    assert lib.allocated == 5 and not lib.pinned
    del kept
    gc.collect()
    for _ in range(5):
        blocks.array(8, 100000)                                    # dropped at once: one block goes round
    assert lib.allocated == 5 and len(lib.pinned) == 1
    for use in range(5):                                           # 0.6 MB: less than half of the free blocks
        blocks.array(1, 151936)
    assert lib.allocated == 6 and len(lib.pinned) == 2
    assert blocks.array(300, 151936) is None and lib.allocated == 6     # 182 MB: plain memory


def test_sizes_that_change_from_step_to_step_share_blocks():
    lib = CountingLibrary()
    blocks = _HostBlocks(lib)
    rng = np.random.default_rng(0)
    held = []
    for n in rng.integers(1, 33, 2000):                            # the last eight arrays are kept
        a = blocks.array(int(n), 151936)
        assert a is not None and a.shape == (n, 151936)
        held = (held + [a])[-8:]
        del a
    assert lib.allocated <= 60 and sum(len(m) for m in lib.live.values()) <= blocks.LIMIT


def test_a_forked_child_frees_nothing():
    lib = FakeLibrary()
    blocks = _HostBlocks(lib)
    a = blocks.array(3, 40000)
    blocks._process += 1                                           # as in a child: another process than the one that made it
    blocks.close()
    del a
    gc.collect()
    assert len(lib.live) == 1


_FORK = """
import os
import numpy as np
from easy_gpt.cpp_b200.native import NativeStepRunner
from easy_gpt.cpp_b200.weights.random_init import write_random_model
write_random_model({folder!r}, {config!r}, 3)
runner = NativeStepRunner({folder!r}, "bfloat16", page_size=16, num_pages=64, max_slots=20)
ids = list(range(16))
def step(k):
    return runner.run([(i, [k + i], [0]) for i in ids])
for k in range(4):                       # each dropped before the next: the block is taken again and page-locked
    step(k)
mine = step(50)
there = mine.ctypes.data
want = mine.copy()
to_child, from_parent = os.pipe()[::-1]
from_child, to_parent = os.pipe()
pid = os.fork()
if pid == 0:
    os.read(from_parent, 1)              # the parent has dropped its array and run further steps by now
    same = bool(np.all(mine == want))
    mine[:] = -7.0
    os.write(to_parent, b"x")
    os.read(from_parent, 1)
    os._exit(0 if same else 3)
del mine
after = step(90)
assert after.ctypes.data == there, "the block is taken again"
again = after.copy()
os.write(to_child, b"x")
os.read(from_child, 1)
assert np.array_equal(after, again), "a child's write reached the parent"
last = step(91)                          # another block; the first is still in use
os.write(to_child, b"x")
assert os.WEXITSTATUS(os.waitpid(pid, 0)[1]) == 0, "the parent's steps reached the child"
fresh = NativeStepRunner({folder!r}, "bfloat16", page_size=16, num_pages=64, max_slots=20)
for k in (0, 1, 2, 3, 50, 90):
    rows = fresh.run([(i, [k + i], [0]) for i in ids])
assert np.array_equal(rows, again), "page-locked memory that the process forked from holds what the device wrote"
print("all right")
"""


def test_the_librarys_blocks_lie_apart_and_go_back():
    """The library's own allocator, without a GPU: blocks of one mapping and of their own, written from end to end."""
    from easy_gpt.cpp_b200 import native

    lib, rng, live = native.library(), np.random.default_rng(1), {}
    for turn in range(300):
        if live and rng.random() < 0.45:
            address = list(live)[int(rng.integers(len(live)))]
            memory, value = live.pop(address)
            assert memory[0] == memory[-1] == value and np.all(memory[:: 4096] == value)
            lib.ege_host_free(address)
            continue
        size = int(rng.integers(1, 9 << 20) if turn % 2 else rng.integers(1, 1 << 20))
        address = lib.ege_host_alloc(size)
        assert address and address % 4096 == 0 and address not in live
        memory = np.frombuffer((ctypes.c_uint8 * size).from_address(address), dtype=np.uint8)
        memory[:] = turn % 251
        live[address] = (memory, turn % 251)
    for address, (memory, value) in live.items():
        assert np.all(memory == value)
        lib.ege_host_free(address)
    assert not lib.ege_host_alloc(0)
    lib.ege_host_free(None)


@pytest.mark.gpu
def test_a_forked_child_has_its_own_copy_of_the_logits(tmp_path):
    root = Path(__file__).resolve().parent.parent
    config = {"architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "num_hidden_layers": 1, "hidden_size": 64, "num_attention_heads": 2,
              "num_key_value_heads": 1, "intermediate_size": 64, "vocab_size": 50000, "rope_theta": 10000.0, "rms_norm_eps": 1e-6,
              "tie_word_embeddings": True, "max_position_embeddings": 512, "bos_token_id": -1, "eos_token_id": -1, "use_sliding_window": False}
    code = _FORK.format(config=config, folder=str(tmp_path / "model"))
    out = subprocess.run([sys.executable, "-W", "ignore", "-c", code], capture_output=True, text=True, cwd=root, env=dict(os.environ), timeout=300)
    assert out.returncode == 0 and "all right" in out.stdout, out.stdout[-2000:] + out.stderr[-3000:]
