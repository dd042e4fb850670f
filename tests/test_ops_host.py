"""Host side of the single operators: what is built once is built again when what it describes changes."""
import ctypes as C

import numpy as np
import pytest
import torch

from dyninfer_b200 import _lib, ops, synth


def described(weight):
    return C.cast(weight.ref(), C.POINTER(_lib.Weight)).contents


@pytest.fixture
def weight(native_lib):
    t = synth.random_weight("mlx.affine.u4", 4, 128, 1)
    return ops.DeviceWeight("mlx.affine.u4", 4, 128, t["packed"], t["scales"], t["biases"], device="cpu")


def test_the_descriptor_is_kept_while_nothing_changes(weight):
    assert weight.ref() is weight.ref()


@pytest.mark.parametrize("field", ["data", "scales", "biases"])
def test_a_replaced_tensor_is_described_anew(weight, field):
    weight.ref()
    fresh = getattr(weight, field).clone()
    setattr(weight, field, fresh)
    assert getattr(described(weight), field) == fresh.data_ptr()


@pytest.mark.parametrize("field,value,name", [("rows", 3, "rows"), ("cols", 64, "cols"), ("group", 32, "group"),
                                              ("aux", "plain.f16", "aux_type"), ("encoding", "gguf.q4_0", "encoding")])
def test_changed_fields_are_described_anew(weight, field, value, name):
    weight.ref()
    setattr(weight, field, value)
    assert getattr(described(weight), name) == (_lib.ENC[value] if isinstance(value, str) else value)


@pytest.mark.parametrize("missing", ["_raw_stream", "_raw_device"])
def test_the_stream_comes_the_public_way_from_a_torch_without_raw_getters(monkeypatch, missing):
    class Stream:
        cuda_stream = 1234
    monkeypatch.setattr(ops, missing, None)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: Stream)
    assert ops._stream() == 1234
