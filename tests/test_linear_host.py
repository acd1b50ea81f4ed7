"""What QuantizedLinear hands to its native host path, without a GPU."""
import copy
import pickle
import types

import pytest
import torch

from tilus_b200 import QuantizedLinear, float16
from tilus_b200 import dtypes as D
from tilus_b200 import linear as linear_module


@pytest.fixture
def calls(monkeypatch):
    seen = []

    def record(*args):
        seen.append(args)
        return args

    stub = types.SimpleNamespace(linear=record, linear_host=record, gate_up_cast=record)
    monkeypatch.setattr(linear_module, "native", lambda: stub)
    return seen


def _layer():
    return QuantizedLinear(float16, D.uint4b, 128, 512, 64, zero_point=8)


def test_calls_follow_the_layers_attributes(calls):
    """Constants changed after construction are the ones the next call uses."""
    layer, x = _layer(), torch.zeros(1, 512, dtype=torch.float16)
    layer(x)
    assert calls[-1][3] == (D.uint4b.code, 8, 128, 512, 64)
    layer.zero_point = 0
    layer.w_dtype = D.int4b
    layer(x)
    layer.forward_host(x, torch.zeros(1, 64, dtype=torch.float16))
    layer.forward_swiglu_cast(x)
    assert [c[i] for c, i in zip(calls[1:], (3, 4, 3))] == [(D.int4b.code, 0, 128, 512, 64)] * 3


def test_weights_that_are_not_parameters(calls):
    layer, x = _layer(), torch.zeros(1, 512, dtype=torch.float16)
    qw, scales = layer.quantized_weight.data, layer.scales.data
    del layer.quantized_weight, layer.scales
    layer.register_buffer("quantized_weight", qw)
    layer.scales = scales  # a plain attribute
    layer(x)
    assert calls[-1][1] is qw and calls[-1][2] is scales


def test_copies_and_pickles_of_other_versions_call(calls):
    """A module object saved whole carries attributes only; none that a call needs may be one it lacks."""
    x = torch.zeros(1, 512, dtype=torch.float16)
    for layer in (copy.deepcopy(_layer()), pickle.loads(pickle.dumps(_layer()))):
        for name in [n for n in vars(layer) if n.startswith("_") and n not in vars(torch.nn.Module())]:
            del layer.__dict__[name]
        layer(x)
        assert calls[-1][3] == (D.uint4b.code, 8, 128, 512, 64)
