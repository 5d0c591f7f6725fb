"""profiling.region as a context manager and as a decorator."""
import contextlib

import pytest

from flowmc_gb300 import profiling


@pytest.fixture
def seen(monkeypatch):
    """What regions record, without a GPU: the timed part is replaced by a list."""
    out = []

    @contextlib.contextmanager
    def record(name, units):
        out.append((name, units))
        yield

    monkeypatch.setattr(profiling, "_timed", record)
    monkeypatch.setattr(profiling, "_nvtx", False)
    return out


def test_decorator_made_while_nothing_records(seen):
    @profiling.region("f", 3.0)
    def f(n):
        return n if n == 0 else f(n - 1)

    assert f(1) == 0 and seen == []
    with profiling.Profiler():
        assert f(2) == 0
    assert seen == [("f", 3.0)] * 3


def test_region_made_before_the_profiler_records(seen):
    r = profiling.region("g")
    with profiling.Profiler():
        with r:
            pass
    assert seen == [("g", 0.0)]


def test_exceptions_pass_through(seen):
    for on in (False, True):
        with contextlib.ExitStack() as s:
            if on:
                s.enter_context(profiling.Profiler())
            with pytest.raises(KeyError):
                with profiling.region("h"):
                    raise KeyError("k")
