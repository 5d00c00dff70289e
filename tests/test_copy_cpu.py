"""What a packed model keeps for its foreign calls, when the model is copied or pickled (no device needed)."""
import copy
import ctypes as C
import pickle

import torch

from paligemma_multimodal_system_b200 import _lib


def test_layer_addresses_belong_to_the_copy():
    names = [n for n, _ in _lib.GemmaLayer._fields_]
    packed = dict(layers=[{n: torch.randn(3) for n in names} for _ in range(2)])
    first = _lib.layer_array(_lib.GemmaLayer, packed)
    assert _lib.layer_array(_lib.GemmaLayer, packed) is first
    for other in (copy.deepcopy(packed), pickle.loads(pickle.dumps(packed))):
        array = _lib.layer_array(_lib.GemmaLayer, other)
        assert C.addressof(array) != C.addressof(first)
        for i, layer in enumerate(other["layers"]):
            for n in names:
                assert getattr(array[i], n) == layer[n].data_ptr() != packed["layers"][i][n].data_ptr()
                assert torch.equal(layer[n], packed["layers"][i][n])
