"""Which calls the native host path stands in for, checked on the CPU with a stand-in for the extension."""

import os
import struct
import sys
import types

import pytest
import torch

import turboquant as tq
from turboquant import _native as N
from turboquant import cache

pytestmark = pytest.mark.filterwarnings("ignore::RuntimeWarning")


class _OnCuda:
    """Enough of a CUDA tensor for the routing."""
    is_cuda, device, dtype = True, "cuda:0", torch.float16

    def __init__(self, *shape):
        self.shape = shape

    def __getitem__(self, _index):
        return self


@pytest.fixture
def unloaded(monkeypatch):
    monkeypatch.setattr(N, "_host", None)              # what host() leaves there goes with the test


@pytest.mark.parametrize("reason", ["does not load", "of another torch"])
def test_calls_take_the_general_path_without_the_extension(unloaded, monkeypatch, tmp_path, reason):
    if reason == "does not load":
        monkeypatch.setitem(sys.modules, "turboquant._tq_host", None)
        monkeypatch.delattr(tq, "_tq_host", raising=False)
    else:
        (tmp_path / "_tq_host.built_for").write_text("torch 1.0 other\n")
        monkeypatch.setattr(N, "_HERE", str(tmp_path))
    with pytest.warns(RuntimeWarning, match="is not used"):
        host = N.host()
    assert host.compress(None, None) is None and host.step_plan([], 0) is None
    assert N.host() is host                                                  # said once


def test_the_extension_that_is_here_loads(unloaded):
    assert not isinstance(N.host(), N._GeneralPath)


def test_a_build_for_another_torch_is_stale(monkeypatch, tmp_path):
    sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(tq.__file__))))
    import build
    out, stamp = tmp_path / "_tq_host.so", tmp_path / "_tq_host.built_for"
    built = []
    monkeypatch.setattr(build, "HOST_OUT", str(out))
    monkeypatch.setattr(build, "HOST_STAMP", str(stamp))
    monkeypatch.setattr(build.subprocess, "check_call", lambda cmd: (built.append(cmd), out.write_bytes(b"")))
    build.build_host()
    build.build_host()
    assert len(built) == 1 and stamp.read_text() == build.host_built_for()
    stamp.write_text("torch 1.0 other\n")
    build.build_host()
    assert len(built) == 2 and stamp.read_text() == build.host_built_for()


def test_a_cache_that_the_native_step_refuses_is_not_looked_over_again(monkeypatch):
    tried = []
    monkeypatch.setattr(N, "host", lambda: types.SimpleNamespace(step_plan=lambda states, window: tried.append(window)))
    monkeypatch.setattr(torch.cuda, "current_device", lambda: device)
    device = 0
    c = cache.V3Cache(n_layers=2)
    monkeypatch.setattr(c, "_step_general", lambda keys, values, views: "general")
    for l in range(2):
        c._layers[l] = types.SimpleNamespace(k=_OnCuda(1, 2, 16, 16))
    tokens = [None, None]
    assert [c.step(tokens, tokens) for _ in range(3)] == ["general"] * 3 and len(tried) == 1
    device = 1                                                               # another device may hold what this one does not
    c.step(tokens, tokens)
    c.step(tokens, tokens)
    assert len(tried) == 2
    c._native_plan = None                                                    # a layer was made or grown
    c.step(tokens, tokens)
    c.residual_window += 1
    c.step(tokens, tokens)
    assert len(tried) == 4


def test_a_step_before_the_layers_exist_makes_its_plan_afterwards(monkeypatch):
    """Layers that update() creates drop the answer that there is no plan."""
    c = cache.V3Cache(n_layers=2, residual_window=128)
    token = [torch.zeros(1, 2, 1, 16) for _ in range(2)]
    c.step(token, token)
    assert c._native_plan is None
    assert c.get_seq_length(1) == 1


def _record(*layers):
    """The record of one native step: (first token, tokens, four offsets) of every layer."""
    firsts, counts, offsets = zip(*layers)
    return struct.pack(f"{6 * len(layers)}q", *firsts, *counts, *(o for four in offsets for o in four))


def test_native_steps_are_read_where_they_are_recorded():
    """Nothing is left for a later call: the entries of a layer come from its own list and from the steps' records, in token
    order, and asking for them changes neither."""
    c = cache.V3Cache(n_layers=3)
    for l in range(3):
        c._layers[l] = types.SimpleNamespace(packed=[])
    c._layers[0].packed.append((0, 5, "update"))
    c._step_log.append(("first", _record((5, 1, (0, 16, 32, 48)), (0, 2, (64, 80, 96, 112)))))
    c._layers[0].packed.append((6, 2, "update again"))
    c._step_log.append(("second", _record((8, 0, (0, 0, 0, 0)), (2, 1, (0, 16, 32, 48)), (0, 1, (64, 80, 96, 112)))))
    for _ in range(2):
        assert c._entries(0) == [(0, 5, "update"), (5, 1, "first", (0, 16, 32, 48)), (6, 2, "update again")]
        assert c._entries(1) == [(0, 2, "first", (64, 80, 96, 112)), (2, 1, "second", (0, 16, 32, 48))]
        assert c._entries(2) == [(0, 1, "second", (64, 80, 96, 112))]
    assert len(c._step_log) == 2 and len(c._layers[0].packed) == 2 and not hasattr(c, "_file_steps")


@pytest.mark.parametrize("entry", ["tq_score_workspace_bytes", "tq_decode_attention_workspace_bytes", "tq_qjl_scores_packed_workspace_bytes"])
def test_a_replaced_scratch_size_is_asked(monkeypatch, entry):
    """The extension holds the library's own size entries; a call whose entry was replaced takes the path that asks it."""
    assert N.attention_host(entry) is N.host()
    with monkeypatch.context() as m:
        m.setattr(N.lib(), entry, lambda *a: 0)
        assert isinstance(N.attention_host(entry), N._GeneralPath)
    assert N.attention_host(entry) is N.host()
