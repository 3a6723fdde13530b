"""checkpoint_every bounds what a trajectory's gradients keep: within a fixed factor of the
checkpoints and one segment, whatever the number of steps."""

import pytest
import torch


def _states(n_steps, every):
    return 2 * -(-n_steps // every) + min(every, n_steps)


@pytest.mark.parametrize("every", [1, 7, 20, 100, 1000])
def test_kept_positions_stay_within_the_bound(every):
    from tsb.adjoint import _Blocks

    for n_steps in [*range(1, 400), 1000, 5000, 10**5, 10**7]:
        whole = _Blocks.keeps_all(n_steps, every, 24)
        assert (n_steps if whole else 0) <= _Blocks.KEEP * _states(n_steps, every)
        assert whole or n_steps > _Blocks.KEEP * _states(n_steps, every)
    assert not _Blocks.keeps_all(100, every, _Blocks.TRAJ_BYTES // 99)
    assert not _Blocks.keeps_all(10**6, 1000, 24)  # k = sqrt(T): O(sqrt(T)) states


@pytest.mark.gpu
def test_memory_follows_checkpoint_every():
    from test_gpu_adjoint_blocks import _close, _problem
    from tsb import adjoint

    P, s, e, q, p = _problem([60] * 40, 1200)
    step = 8 * q.numel()
    got = {}
    for every in (1200, 35):
        P.checkpoint_every = every
        adjoint.loss_and_grad(s, e, q, p, P)
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        got[every] = adjoint.loss_and_grad(s, e, q, p, P)
        peak = torch.cuda.max_memory_allocated() - before
        # (some tens of vectors besides: results, histograms)
        assert peak < step * (1200 if every == 1200 else 2 * 35 + 35) + 64 * step
    # a trajectory that is integrated again rebuilds its lists at other steps, so sums
    # differ in order; 1,200 steps amplify 1e-16 (4e-12 over 60 steps is what the
    # instability of this density allows; 1e-3 is far below any lost segment)
    for a, b in zip(got[1200], got[35], strict=True):
        _close(a, b, 1e-3)


@pytest.mark.gpu
def test_no_room_for_every_step_takes_the_segments(monkeypatch):
    from test_gpu_adjoint_blocks import _close, _problem
    from tsb import adjoint

    P, s, e, q, p = _problem([30, 40], 50)
    want = adjoint.loss_and_grad(s, e, q, p, P)
    empty = torch.empty

    def full(shape, *a, **k):
        if not isinstance(shape, int) and tuple(shape)[0] == 50:
            raise torch.cuda.OutOfMemoryError("no room")
        return empty(shape, *a, **k)

    monkeypatch.setattr(torch, "empty", full)
    for a, b in zip(adjoint.loss_and_grad(s, e, q, p, P), want, strict=True):
        _close(a, b)
