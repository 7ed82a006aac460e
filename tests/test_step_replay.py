"""The call that replays a captured step, with a library in its place that only records what it is given (no GPU)."""
from types import SimpleNamespace

import pytest
import torch

from aegean_tge_b200 import ops


class _Tokens(SimpleNamespace):
    """As much of a device tensor of token ids as the call looks at."""
    is_cuda, dtype = True, torch.int32

    def numel(self):
        return self.count

    def is_contiguous(self):
        return True

    def data_ptr(self):
        return 0


@pytest.fixture
def library(monkeypatch):
    calls, lib = [], SimpleNamespace(rc=0, tge_last_error=lambda: b"refused")
    lib.tge_replay_step = lambda *args: calls.append(args) or lib.rc
    lib.calls = calls
    monkeypatch.setattr(ops, "core", lambda: lib)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    return lib


def _replay(tokens, event=None):
    dev, host = torch.zeros(40, dtype=torch.int32), torch.zeros(40, dtype=torch.int32)
    event = event or SimpleNamespace(_handle=None, _recorded=False)
    ops.replay_step(1, dev, host, 40, event, tokens, 8, 4)


@pytest.mark.parametrize("count", [1, 4, 5, 32, 33])
def test_more_token_ids_than_the_captured_step_has_places_for_are_refused(library, count):
    """Ids beyond the step's rows would fall on positions, sequence numbers and tables."""
    if count <= 4:
        _replay(_Tokens(count=count))
        assert library.calls[0][6] == 4 * count
    else:
        with pytest.raises(ops.KernelError):
            _replay(_Tokens(count=count))
        assert not library.calls


def test_a_replay_that_fails_half_way_leaves_its_buffer_in_use(library):
    """The copy out of the pinned buffer may be queued when a later part of the call fails: whoever takes the buffer next waits."""
    library.rc = -2
    event = SimpleNamespace(_handle=None, _recorded=False)
    with pytest.raises(ops.KernelError):
        _replay(None, event)
    assert event._recorded
