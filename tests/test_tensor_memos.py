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


def test_species_of_other_atoms_at_an_old_address():
    from tsb import models

    model = models.kob_andersen_model(device="cpu")
    for _ in range(50):
        a = torch.tensor([1, 1, 2, 2] * 100)
        at = a.data_ptr()
        assert torch.equal(model._species(a), (a - 1).int())
        del a
        b = torch.tensor([2, 1, 2, 1] * 100)
        assert torch.equal(model._species(b), (b - 1).int())
        if b.data_ptr() == at:
            break


def test_order_of_other_systems_at_an_old_address():
    from tsb import integrators

    class State:
        pass

    st = State()
    for _ in range(50):
        st.system_idx, st.n_atoms, st.n_systems = torch.tensor([0] * 300 + [1] * 20), 320, 2
        at = st.system_idx.data_ptr()
        assert integrators._system_order(st)[0].tolist() == [0, 1]
        st.system_idx = None
        st.system_idx = torch.tensor([0] * 20 + [1] * 300)
        order, most = integrators._system_order(st)
        assert order.tolist() == [1, 0] and most == 300
        if st.system_idx.data_ptr() == at:
            break
    st.system_idx[20:] = 0  # written to in place
    assert integrators._system_order(st)[1] == 320


def test_what_counts_as_the_same_tensor():
    import copy
    import pickle

    a = torch.arange(12)
    seen = L.Seen(a)
    assert seen.same(a) and seen.same(a.view(12)) and not seen.same(a.clone())
    assert not seen.same(a[:6]) and not seen.same(a.view(3, 4))
    assert not L.Seen(a[:6]).same(a[::2])  # one address, one length
    assert not copy.deepcopy(seen).same(a) and not pickle.loads(pickle.dumps(seen)).same(a)
    a[0] = 5
    assert not seen.same(a) and not L.Seen().same(a)


def test_what_counts_as_the_same_periodic_axes():
    for flags in (True, [True] * 3, torch.tensor([True] * 3), torch.tensor(True)):
        seen = L.SeenPbc(flags)
        assert seen.same(flags) and not seen.same([True, False, True]) and not seen.same(False)
    assert L.SeenPbc([True, False, True]).same(torch.tensor([1, 0, 1]))
    cpu = torch.tensor([True] * 3)
    seen = L.SeenPbc(cpu)
    cpu[1] = False
    assert not seen.same(cpu) and not L.SeenPbc().same(cpu)
