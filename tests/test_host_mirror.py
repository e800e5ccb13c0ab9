"""No-GPU checks of the Python mirror's weights and workspaces: what a call keeps with an object it was
given must not change what that object is afterwards. The planes are CPU tensors that say they are on a
device; nothing here launches a kernel."""
from __future__ import annotations

import copy
import pickle

import pytest
import torch

from ignis_b200 import _lib, moe, nvfp4, trellis


class OnDevice(torch.Tensor):
    """A CPU tensor that answers ``is_cuda`` as a device tensor would."""

    is_cuda = True

    def __deepcopy__(self, memo):
        return on_device(self.as_subclass(torch.Tensor).clone())


def on_device(t: torch.Tensor) -> torch.Tensor:
    return t.as_subclass(OnDevice)


def nvfp4_weight() -> nvfp4.Weight:
    n, k = 128, 256
    return nvfp4.Weight(on_device(torch.arange(n * k // 2, dtype=torch.int64).to(torch.uint8).reshape(n, k // 2)),
                        on_device(torch.ones(n * k // 16, dtype=torch.uint8)), n, k, 448.0, 96.0)


def trellis_weight() -> trellis.Weight:
    in_ = out = 128
    return trellis.Weight(on_device(torch.arange(8 * 8 * trellis.tile_words16(6), dtype=torch.int16)), on_device(torch.ones(in_, dtype=torch.float16)),
                          on_device(torch.ones(out, dtype=torch.float16)), 6, in_, out)


class Recorder:
    """Stands in for the library: every entry point succeeds, the last call's arguments are kept."""

    def __init__(self) -> None:
        self.args = ()

    def __getattr__(self, name):
        def entry(*args):
            self.args = args
            return 0
        return entry


@pytest.fixture
def lib(monkeypatch):
    lib = Recorder()
    monkeypatch.setattr(_lib, "load", lambda: lib)
    for module in (nvfp4, trellis, moe):
        monkeypatch.setattr(module, "_stream", lambda: 0)
    return lib


def planes(w) -> list[torch.Tensor]:
    return [w.codes, w.scales] if isinstance(w, nvfp4.Weight) else [w.trellis, w.suh, w.svh]


def activations(w) -> torch.Tensor:
    return on_device(torch.ones(2, w.k if isinstance(w, nvfp4.Weight) else w.in_, dtype=torch.bfloat16))


def addresses_in_a_call(lib, w) -> list[int]:
    """The plane addresses in the struct that the library is handed."""
    if isinstance(w, nvfp4.Weight):
        nvfp4.linear_split(activations(w), w, [w.n])
        s = lib.args[0]
        return [s.codes, s.scales]
    trellis.linear(w, activations(w))
    s = lib.args[0]
    return [s.trellis, s.suh, s.svh]


@pytest.mark.parametrize("make", [nvfp4_weight, trellis_weight])
@pytest.mark.parametrize("duplicate", [copy.deepcopy, lambda w: pickle.loads(pickle.dumps(w)), copy.copy])
def test_a_weight_that_was_called_can_be_copied(lib, make, duplicate):
    w = make()
    w.label = "layer 0"   # what a program adds goes along
    before = addresses_in_a_call(lib, w)
    assert before == [t.data_ptr() for t in planes(w)]
    twin = duplicate(w)
    assert type(twin) is type(w) and twin.label == "layer 0"
    assert all(torch.equal(a, b) for a, b in zip(planes(w), planes(twin)))
    assert addresses_in_a_call(lib, twin) == [t.data_ptr() for t in planes(twin)]   # its own planes
    assert addresses_in_a_call(lib, w) == before


@pytest.mark.parametrize("make", [nvfp4_weight, trellis_weight])
def test_planes_reseated_in_place_are_the_ones_a_call_reads(lib, make):
    """A plane can get another memory without its field being assigned: through ``.data``, ``set_`` or ``resize_``."""
    w = make()
    for i in range(len(planes(w))):
        addresses_in_a_call(lib, w)
        kept = planes(w)[i].data   # keeps the old memory alive: the new one lies elsewhere
        planes(w)[i].data = on_device(planes(w)[i].as_subclass(torch.Tensor).clone())
        assert planes(w)[i].data_ptr() != kept.data_ptr()
        assert addresses_in_a_call(lib, w) == [t.data_ptr() for t in planes(w)]
    planes(w)[1].set_(on_device(planes(w)[1].as_subclass(torch.Tensor).clone()))
    assert addresses_in_a_call(lib, w) == [t.data_ptr() for t in planes(w)]


@pytest.mark.parametrize("make", [nvfp4_weight, trellis_weight])
def test_a_weight_moved_off_the_device_is_refused(lib, make):
    w = make()
    addresses_in_a_call(lib, w)
    name = "codes" if isinstance(w, nvfp4.Weight) else "trellis"
    setattr(w, name, getattr(w, name).as_subclass(torch.Tensor).clone())
    with pytest.raises((nvfp4.Nvfp4Error, trellis.TrellisError)):
        addresses_in_a_call(lib, w)


@pytest.mark.parametrize("make,module,kind", [(nvfp4_weight, nvfp4, nvfp4.Workspace), (trellis_weight, trellis, trellis.WorkspaceBuffer)])
def test_a_call_takes_the_workspace_struct_that_is_there_now(lib, make, module, kind):
    ws = kind(512, device="cpu")
    w = make()
    x = activations(w)
    for base in (ws.c.base, ws.c.base + 256):   # another struct put in its place: a part of a larger region
        ws.c = _lib.Workspace(base, 256)
        module.linear(*((x, w) if module is nvfp4 else (w, x)), workspace=ws)
        seen = next(a for a in lib.args if isinstance(a, _lib.Workspace))
        assert seen.base == base and seen.bytes == 256


def test_a_geometry_struct_is_the_callers_own():
    g = moe.Geometry(256, 128, 8, 2)
    g.c_struct().hidden = 512
    assert g.c_struct().hidden == 256
    assert pickle.loads(pickle.dumps(g)) == g and set(vars(g)) == {"hidden", "inter", "experts", "top_k"}
