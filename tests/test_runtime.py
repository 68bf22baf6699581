"""CPU tests of the host-side plumbing: what makes a model pack its weights again and drop its captured launches."""
import copy
import gc
import pickle
import random
import weakref

import numpy as np
import pytest
import torch
from torch.func import functional_call

from vtpack_b200 import runtime
from vtpack_b200.models.dge import deit_dge, pvt_dge
from vtpack_b200.models.dge.deit_dge import _param_key


def _tiny():
    return deit_dge.VisionTransformer(img_size=64, patch_size=16, embed_dim=64, depth=2, num_heads=1, num_classes=10,
                                      split_sizes=[4, 2, 1])


class _Keyed(torch.nn.Module):
    """A model whose forward returns the key of its weight pack."""

    def __init__(self, model):
        super().__init__()
        self.model = model

    def forward(self):
        return _param_key(self.model, torch.bfloat16)


def test_weight_key_follows_tensors_in_the_parameters_place():
    """functional_call puts plain tensors where the parameters are: an in-place update of one between two calls (a moving
    average) makes another key, the same tensors untouched the same key."""
    m = _Keyed(_tiny())
    ema = {k: v.detach().clone() for k, v in m.named_parameters()}
    keys = [functional_call(m, ema, ())]
    assert functional_call(m, ema, ()) == keys[0]
    for name in ("model.head.weight", "model.blocks.1.attn.q.bias", "model.cls_token"):
        ema[name].mul_(0.5)
        keys.append(functional_call(m, ema, ()))
    keys.append(m())                                         # the module's own parameters again
    assert len(set(keys)) == len(keys)
    with torch.no_grad():
        m.model.head.weight.add_(1.0)
    assert m() not in keys


class _Plan:
    pass


@pytest.fixture
def no_capture(monkeypatch):
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)


@pytest.mark.parametrize("move", ["update", "replace"])
def test_pvt_plans_of_replaced_weights_are_dropped(no_capture, move):
    """A plan holds its weights' device copies: none of the old ones is left when the weights are others."""
    m = pvt_dge.pvt_dge_s124_tiny_256()
    made = []

    def capture():
        p = _Plan()
        made.append(weakref.ref(p))
        return p

    for step in range(3):
        m._param_generation()
        for key in ("a", "b"):
            for _ in range(20):
                m._plans.get(key, lambda p: True, capture)
        gc.collect()
        assert len(made) == 2 * (step + 1) and sum(r() is not None for r in made) == 2
        with torch.no_grad():
            if move == "update":
                m.head.bias.add_(1.0)
            else:
                m.head.bias = torch.nn.Parameter(m.head.bias.clone())
    m._param_generation()
    gc.collect()
    assert all(r() is None for r in made)


def test_replay_registers_its_stream_with_all_that_the_plan_holds(monkeypatch):
    """The allocator may not hand on a plan's memory while a stream that replayed it still works on it, whichever stream
    that was and whoever else has let go of the buffers."""
    class Graph:
        def replay(self):
            pass

    seen = []
    monkeypatch.setattr(torch.Tensor, "record_stream", lambda t, s: seen.append((t.data_ptr(), s)))
    held = [torch.zeros(3) for _ in range(5)]
    keep = (held[0], {"a": held[1], "b": (1.0, held[2])}, [{"c": held[3]}, None])
    plan = deit_dge._CapturedTrunk(Graph(), keep, 0, held[4])
    for stream in ("x", "y", "x"):
        monkeypatch.setattr(torch.cuda, "current_stream", lambda d=None, s=stream: s)
        plan.replay(None)
    assert sorted(seen) == sorted((t.data_ptr(), s) for t in held for s in "xy")


@pytest.mark.parametrize("make", [_tiny, pvt_dge.pvt_dge_s124_tiny_256])
def test_whole_models_saved_before_there_were_plans_load(make, no_capture):
    """Files of whole models, also from a version without watches and plans, load into models that work; a copy starts
    without plans."""
    m = make()
    m._plans.earn = 3
    old = dict(m.__dict__)
    old["_consts"] = {"norm": ((), None)}                    # an entry of another form
    for name in ("_plans", "_graph") + (("_pack",) if "_graph" in old else ()):
        old.pop(name, None)
    fresh = type(m).__new__(type(m))
    fresh.__setstate__(old)
    for model in (fresh, copy.deepcopy(m), pickle.loads(pickle.dumps(m))):
        key = _param_key(model, torch.float32)
        assert key == _param_key(model, torch.float32)
        assert model._plans.get("a", lambda p: True, _Plan) is None
        if isinstance(model, pvt_dge.PyramidVisionTransformer):
            assert model._graph is None and "_consts" not in model.__dict__
            assert model._param_generation() == model._param_generation()
    pack = pickle.loads(pickle.dumps(m.blocks[0]._pack if hasattr(m, "blocks") else m.block1[0]._pack))
    assert pack.watch is None and deit_dge._WeightPack.__new__(deit_dge._WeightPack).watch is None


def test_stage_forward_refuses_tokens_of_another_width(monkeypatch):
    """The stage's launches take the width from the blocks: narrower tokens would be read and written beyond their end."""
    monkeypatch.setattr(pvt_dge, "require_cuda", lambda *t: None)
    stage = pvt_dge.pvt_dge_s124_tiny_256().block1
    monkeypatch.setattr(pvt_dge, "_launch_stage", lambda *a: pytest.fail("launched"))
    with pytest.raises(ValueError, match="32 channels"):
        pvt_dge.stage_forward(stage, torch.zeros(1, 64, 32), 8, 8)


def test_constants_follow_a_tensor_that_took_the_address_of_another():
    """Weights handed over as new tensors on every call (functional_call) may lie where the ones before lay."""
    m = pvt_dge.pvt_dge_s124_tiny_256()
    memory = np.zeros(4, dtype=np.float32)
    for value in (1.0, 2.0):
        memory[:] = value
        source = torch.from_numpy(memory)                    # another tensor at the same address, version 0
        got = m._const("c", (source,), lambda: source.detach().clone())
        assert got.tolist() == [value] * 4
        assert m._const("c", (source,), lambda: None) is got
        del source


def test_plans_are_earned_by_calls(no_capture):
    """A shape that is seen often gets a plan and keeps it; many shapes in turn pay for few captures, and for fewer the
    longer it goes on."""
    plans, made = runtime.LaunchPlans(most=4, earn=8), []

    def call(key):
        def capture():
            made.append(key)
            return _Plan()
        return plans.get(key, lambda p: True, capture)

    got = [call("a") for _ in range(20)]
    assert got[:7] == [None] * 7 and all(p is got[7] for p in got[7:]) and made == ["a"]
    rng = random.Random(0)
    for _ in range(2000):
        call(rng.randrange(30))                              # within the shapes that calls are counted for
    first = len(made)
    for _ in range(2000):
        call(rng.randrange(30))
    assert first < 2000 / 8 / 1.5 and len(made) - first < first / 2
    assert len(plans._plans) == 4 and len(plans._calls) <= 32
    for key in range(1000, 3000):
        assert call(key) is None
    assert len(plans._calls) <= 32


def test_a_plan_that_no_longer_fits_is_made_again_at_once(no_capture):
    plans = runtime.LaunchPlans(most=4, earn=2)
    assert plans.get("a", lambda p: True, _Plan) is None
    p = plans.get("a", lambda p: True, _Plan)
    q = plans.get("a", lambda p: False, _Plan)
    assert q is not p and plans.get("a", lambda p: True, _Plan) is q
    plans.clear()
    assert plans.get("a", lambda p: True, _Plan) is None and copy.deepcopy(plans).earn == 2


class _OnDevice:
    """What the training path looks at of a tensor before it picks a kernel, as if on a GPU."""

    def __init__(self, shape, index=0, dtype=torch.float32):
        self.shape, self.device, self.dtype, self.is_cuda = torch.Size(shape), torch.device("cuda", index), dtype, True

    def dim(self):
        return len(self.shape)

    def element_size(self):
        return self.dtype.itemsize

    def data_ptr(self):
        return 256


@pytest.mark.parametrize("other", [None, "x", "comp", "gate", "ref", "patches"])
def test_gated_decompress_in_one_launch_takes_operands_of_one_device(monkeypatch, other):
    """Operands of two GPUs are refused by the operations that the launch stands for; the launch would read the other GPU's addresses."""
    from vtpack_b200.layers import grained_sample as gs
    monkeypatch.setattr(gs._GatedDecompress, "apply", lambda *a: "launched")
    monkeypatch.setattr(gs, "_by_region", lambda *a: True)
    t = {n: _OnDevice(shape, 1 if n == other else 0) for n, shape in
         dict(x=(9, 64), comp=(9, 64), gate=(1, 2, 2, 3), ref=(1, 65, 64), patches=(9, 4)).items()}
    t["patches"]._vtp_regions, t["patches"]._vtp_offsets = (None, None, [4, 2, 1], 4, 2, 2, 1), None
    got = gs.gated_decompress(t["x"], t["comp"], t["gate"], t["ref"], t["patches"], 8, 1)
    assert got == ("launched" if other is None else None)


@pytest.mark.parametrize("index", [0, 1])
def test_ragged_attention_as_one_node_takes_operands_of_one_device(monkeypatch, index):
    from vtpack_b200.layers import sparse_ops
    monkeypatch.setattr(sparse_ops._RaggedAttention, "apply", lambda *a: "launched")
    got = sparse_ops.ragged_attention(_OnDevice((9, 64)), _OnDevice((2, 5, 128), index), torch.tensor([4, 5]), 1, 0.125, torch.nn.Dropout(0.0))
    assert got == ("launched" if index == 0 else None)
