"""What goes wrong while the pair list gets its room is raised as it is.  Needs no GPU: the library is a stand-in that asks
for room and reports none."""
import numpy as np
import pytest

import riggle_b200 as rg
from riggle_b200 import _lib, api


class _Library:
    def __init__(self, count):
        self.count = count

    def rgl_query_pairs_alloc(self, handle, batch, alloc, user, n):
        return _lib.RGL_OK if alloc(None, self.count) else _lib.RGL_ERR_OOM

    def rgl_last_error(self):
        return b"no room"

    def rgl_context_destroy(self, handle):
        pass


def _context(monkeypatch, count):
    monkeypatch.setattr(api, "load", lambda: _Library(count))
    ctx = api.Context.__new__(api.Context)
    ctx._h = None
    return ctx


def test_no_room_is_a_memory_error(monkeypatch):
    ctx = _context(monkeypatch, 2**58)  # 2^63 bytes: more than any address space
    with pytest.raises((MemoryError, ValueError)) as e:
        ctx.query_pairs({0: np.array([[1, 2, 0]], np.uint32)}, 1)
    assert not isinstance(e.value, rg.RiggleError)


@pytest.mark.parametrize("error", [MemoryError, KeyboardInterrupt])
def test_errors_pass(monkeypatch, error):
    ctx = _context(monkeypatch, 7)
    empty = np.empty

    def fail(shape, *args, **kw):
        if shape == (7, 8):
            raise error()
        return empty(shape, *args, **kw)

    monkeypatch.setattr(np, "empty", fail)
    with pytest.raises(error):
        ctx.query_pairs({0: np.array([[1, 2, 0]], np.uint32)}, 1)


def test_the_list_comes_back(monkeypatch):
    ctx = _context(monkeypatch, 7)
    assert ctx.query_pairs({0: np.array([[1, 2, 0]], np.uint32)}, 1).shape == (7, 8)
