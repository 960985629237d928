"""CPU: the compositing shape and the long tiles that the library chooses can be left and returned to.  What the
get calls report restores what was in force, whatever came between, each direction and the split by itself; and the
autotuner times the library's choice first and installs it where nothing beats it.  (Host-only calls.)"""
import ctypes as C

import pytest
import torch

from filtergs_b200 import _lib, autotune

RULE = (0, 0, 0, 0, 0, -1)


@pytest.fixture(autouse=True)
def library():
    try:
        cfg, split = _lib.get_render_config(), _lib.get_render_split()
    except Exception as e:  # the library is not built: nothing to test on this machine
        pytest.skip(f"library unavailable: {e}")
    _lib.set_render_config()
    _lib.set_render_split()
    yield
    _lib.set_render_config(*cfg)
    _lib.set_render_split(*split)


def _c_values():
    cfg, split = (C.c_int * 4)(), (C.c_int * 2)()
    assert _lib.lib().fgs_get_render_config(C.cast(cfg, C.c_void_p)) == _lib.FGS_OK
    assert _lib.lib().fgs_get_render_split(C.cast(split, C.c_void_p)) == _lib.FGS_OK
    return tuple(cfg) + tuple(split)


@pytest.mark.parametrize("shape", [None, (1, 64, 1, 64), (2, 256, 2, 256), (2, 128, 2, 256), (4, 128, 2, 64)])
@pytest.mark.parametrize("split", [None, (0, 0), (512, 3)])
def test_what_was_read_restores_what_was_in_force(shape, split):
    assert _c_values() == RULE
    cfg, sp = _lib.get_render_config(), _lib.get_render_split()
    assert cfg == (2, 128, 2, 256) and sp == (0, 0)      # what is in use
    if shape:
        _lib.set_render_config(*shape)
        assert _lib.get_render_config() == shape and _c_values()[:4] == shape
    if split:
        _lib.set_render_split(*split)
        assert _lib.get_render_split() == split and _c_values()[4:] == split
    was = _lib.get_render_config(), _lib.get_render_split(), _c_values()
    _lib.set_render_config(4, 64, 4, 64)
    _lib.set_render_split(1024, 1)
    _lib.set_render_config(*was[0])
    _lib.set_render_split(*was[1])
    assert _c_values() == was[2]
    _lib.set_render_config(*cfg)
    _lib.set_render_split(*sp)
    assert _c_values() == RULE


def test_each_direction_by_itself():
    cfg = _lib.get_render_config()
    _lib.set_render_config(4, 64, *cfg[2:])
    assert _c_values() == (4, 64, 0, 0, 0, -1)
    _lib.set_render_config(cfg[0], cfg[1], 1, 128)
    assert _c_values() == (0, 0, 1, 128, 0, -1)
    _lib.set_render_config(4)                            # one argument: the rest of its direction as ever
    assert _c_values()[:4] == (4, 256, 0, 0)
    _lib.set_render_split(256)
    assert _c_values()[4:] == (256, 0)
    _lib.set_render_split(0)
    assert _c_values()[4:] == (0, 0)
    _lib.set_render_config()
    _lib.set_render_split()
    assert _c_values() == RULE


@pytest.mark.parametrize("bad", [(0, 64, 2, 64), (2, 0, 2, 64), (2, 64, 0, 64), (2, 64, 4, 0), (-1, 64, 2, 64)])
def test_half_a_choice_is_refused(bad):
    assert _lib.lib().fgs_set_render_config(*bad) == _lib.FGS_ERR_ARG
    assert _c_values() == RULE


@pytest.mark.parametrize("bad", [(1, -1), (-1, -1), (-1, 0), (0, -2), (0, 4)])
def test_half_a_split_is_refused(bad):
    assert _lib.lib().fgs_set_render_split(*bad) == _lib.FGS_ERR_ARG
    assert _c_values() == RULE


def _tune(monkeypatch, fwd, bwd, **kw):
    """tune_render on a cost table: fwd and bwd map the C settings to milliseconds."""
    pending, seen = [0.0, 0.0], []

    def run_step():
        seen.append(_c_values())
        pending[0] += fwd(seen[-1])
        pending[1] += bwd(seen[-1])

    def profile_read(reset=True):
        out = {"render_fwd": (pending[0], 1), "render_bwd": (pending[1], 1)}
        pending[:] = [0.0, 0.0]
        return out

    monkeypatch.setattr(_lib, "profile_read", profile_read)
    monkeypatch.setattr(_lib, "profile_enable", lambda on=True: None)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda *a, **k: None)
    monkeypatch.setattr(autotune, "_cache", {})
    best, table = autotune.tune_render(run_step, key="k", splits=((0, 0), (512, 3)), **kw)
    assert seen[0] == RULE
    return best, table, run_step


def test_tuning_keeps_the_library_choice_where_nothing_beats_it(monkeypatch):
    _lib.set_render_config(1, 64, 1, 64)
    fwd = lambda c: 1.0 if c[0] == 0 and c[5] == -1 else (1.5 if c[5] == 3 else 6.0)  # noqa: E731
    bwd = lambda c: 2.0 if c[2] in (0, 2) else 3.0                                     # noqa: E731
    best, table, run_step = _tune(monkeypatch, fwd, bwd)
    assert _c_values() == RULE and best == (2, 128, 2, 256)
    assert table[("split", "library")] == pytest.approx((1.0, 2.0))
    assert table[("split", 512, 3)][0] == pytest.approx(1.5)
    _lib.set_render_config(4, 64, 4, 64)
    _lib.set_render_split(0, 0)
    assert autotune.tune_render(run_step, key="k")[0] == best and _c_values() == RULE   # from the cache


@pytest.mark.parametrize("slow", ["forward", "backward"])
def test_tuning_leaves_the_library_choice_by_direction(monkeypatch, slow):
    fwd = lambda c: 9.0 if c[0] == 0 else (4.0 if c[:2] == (4, 64) else 5.0) + (0.5 if c[5] == 3 else 0.0)  # noqa: E731
    bwd = lambda c: 7.0 if c[2] == 0 else (3.0 if c[2] == 4 else 8.0)                                       # noqa: E731
    if slow == "forward":
        _tune(monkeypatch, fwd, lambda c: 1.0)
        assert _c_values() == (4, 64, 0, 0, 0, 0)
    else:
        _tune(monkeypatch, lambda c: 1.0, bwd)
        assert _c_values()[:2] == (0, 0) and _c_values()[2] == 4 and _c_values()[4:] == (0, -1)
