"""What is remembered about a tensor ends with it: another tensor at the same address,
or the same one written to, is looked at again (CPU: the host logic alone)."""

import gc

import torch

from tsb import _lib as L


def _two_in_turn(first, second):
    """The answers for two index tensors of which the second may take the first one's
    address (it does on the CPU allocator within a few tries)."""
    for _ in range(50):
        a = torch.repeat_interleave(torch.arange(len(first)), torch.tensor(first))
        at, got = a.data_ptr(), [L.max_system_atoms(a, len(first))]
        del a
        gc.collect()
        b = torch.repeat_interleave(torch.arange(len(second)), torch.tensor(second))
        got.append(L.max_system_atoms(b, len(second)))
        if b.data_ptr() == at:
            break
    return got


def test_largest_system_of_a_new_tensor_at_an_old_address():
    assert _two_in_turn([25, 25, 25, 25], [10, 30, 30, 30]) == [25, 30]
    assert _two_in_turn([32, 28], [0, 60]) == [32, 60]


def test_largest_system_is_kept_while_the_tensor_lives(monkeypatch):
    idx = torch.tensor([0, 0, 0, 1, 1])
    reads = []
    count = torch.bincount
    monkeypatch.setattr(torch, "bincount", lambda *a, **k: reads.append(1) or count(*a, **k))
    assert [L.max_system_atoms(idx, 2) for _ in range(3)] == [3, 3, 3] and len(reads) == 1
    idx[2] = 1  # written to in place
    idx[1] = 1
    assert L.max_system_atoms(idx, 2) == 4 and len(reads) == 2
    assert L.max_system_atoms(idx, 5) == 4  # other numbers of systems ask again
    assert L.max_system_atoms(torch.zeros(0, dtype=torch.int64), 1) == 0


def test_nothing_is_kept_of_a_tensor_that_is_gone():
    before = len(L._MAX_SYS)
    for n in range(1, 200):
        L.max_system_atoms(torch.zeros(n, dtype=torch.int64), 1)
    gc.collect()
    assert len(L._MAX_SYS) <= before
