"""Context.download into host arrays that are too small: the ones it returns have
the caller's layout (pinned memory, the fields left out, the depth) and room for
the world, and what it hands to mac_download_state are their pointers. On CPU,
with a stand-in for the library's two calls and for pinned allocation.
"""
import pytest

from mac_b200.gpu import CELL_F64, Context, HostState
from mac_b200.state import Params


class _Lib:
    """A world of nb bricks and npart particles; records the pointers it is given."""

    def __init__(self, nb, npart):
        self.nb, self.npart = nb, npart

    def mac_query_sizes(self, h, nb, npart):
        nb._obj.value, npart._obj.value = self.nb, self.npart
        return 0

    def mac_download_state(self, h, st):
        self.given = st._obj
        assert st._obj.nbricks == self.nb and st._obj.nparticles == self.npart
        return 0


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("depth", [False, True])
@pytest.mark.parametrize("stage", [False, True])
@pytest.mark.parametrize("need", [(5, 9), (2, 30), (6, 40)])
def test_grown_arrays_keep_the_layout(monkeypatch, pinned, depth, stage, need):
    import torch
    empty, pins = torch.empty, []

    def fake(*a, pin_memory=False, **k):
        pins.append(pin_memory)
        return empty(*a, **k)
    monkeypatch.setattr(torch, "empty", fake)
    host = HostState(4, 20, pinned=pinned, depth=depth, stage_buffers=stage)
    ctx = Context.__new__(Context)
    ctx.h, ctx.params, ctx.lib = None, Params(depth_mode=int(depth)), _Lib(*need)
    del pins[:]
    got = ctx.download(host=host, to_state=False)
    assert got is not host and (got.nbricks, got.nparticles) == need
    assert got.cap_bricks == max(4, need[0]) and got.cap_particles == max(20, need[1])
    assert (len(pins) > 0 and all(pins)) == pinned
    assert list(got.f64) == list(host.f64) == [n for n in CELL_F64 if stage or n not in HostState.STAGE]
    assert (got.depth is not None) == depth
    assert all(len(a) >= 512 * need[0] for a in got.f64.values()) and len(got.pos) >= 3 * need[1]
    assert bool(ctx.lib.given.u[1][0]) == stage and bool(ctx.lib.given.depth) == depth


def test_arrays_with_room_are_used_as_they_are():
    host = HostState(4, 20, stage_buffers=False)
    ctx = Context.__new__(Context)
    ctx.h, ctx.params, ctx.lib = None, Params(), _Lib(4, 20)
    assert ctx.download(host=host, to_state=False) is host
