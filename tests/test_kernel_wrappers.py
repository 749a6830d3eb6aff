"""Host side of the kernel wrappers, without a GPU: what reaches the C entries."""
import pytest
import torch

from torchft_b200.ops import kernels as K


class _OnGpu(torch.Tensor):
    """A CPU tensor that says it is on the GPU."""

    is_cuda = True


@pytest.fixture
def calls(monkeypatch):
    """The arguments of every C entry called, by name, instead of the calls."""
    seen = []
    monkeypatch.setattr(K, "_fn", lambda name: lambda *args: seen.append((name, args)) or 0)
    monkeypatch.setattr(K, "_status_ptr", lambda device: 0)
    stream = [1]
    monkeypatch.setattr(K, "_stream", lambda: stream[0])
    seen_on = lambda s: stream.__setitem__(0, s)  # noqa: E731
    return seen, seen_on


def test_rmsnorm_bwd_partial_sums_are_a_stream_s_own(calls, monkeypatch):
    """The two kernels of a call meet in the scratch memory, so calls on different streams do not share it."""
    monkeypatch.setattr(K, "_rms_scratch", {})
    seen, on_stream = calls
    x, w, rstd = (torch.zeros(*s).as_subclass(_OnGpu) for s in ((4, 64), (64,), (4,)))
    for s in (1, 2, 1, 2):
        on_stream(s)
        K.rmsnorm_bwd(x, x, w, rstd, dx=x, dw=w)
    scratch = [args[7] for _, args in seen]
    assert scratch[0] == scratch[2] and scratch[1] == scratch[3] and scratch[0] != scratch[1]


def test_rmsnorm_bwd_takes_the_caller_s_scratch(calls):
    seen, _ = calls
    x, w, rstd = (torch.zeros(*s).as_subclass(_OnGpu) for s in ((4, 64), (64,), (4,)))
    need = K.rmsnorm_bwd_scratch_floats(64)
    own = torch.empty(need + 4)
    K.rmsnorm_bwd(x, x, w, rstd, dx=x, dw=w, scratch=own)
    assert seen[0][1][7] == own.data_ptr()
    for bad in (own[: need - 1], own.double(), own[1:], torch.empty(2 * need)[::2]):
        with pytest.raises(ValueError):
            K.rmsnorm_bwd(x, x, w, rstd, dx=x, dw=w, scratch=bad)
    assert len(seen) == 1
