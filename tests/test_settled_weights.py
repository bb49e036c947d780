"""Matrices that several tensors are joined into are there before the first step: the products'
kernels read their weights while the kernel ahead of them may still run."""
import gc

import pytest
import torch

from pretrained_rstr_b200 import load_lm
from pretrained_rstr_b200.config.registry import named_size
from pretrained_rstr_b200.engine.batch import Runtime
from pretrained_rstr_b200.parts.latent_attention import FusedInput
from pretrained_rstr_b200.parts.linear import ResultProduct
from pretrained_rstr_b200.weights import make_random_model
from pretrained_rstr_b200.weights.loader import load_weights

TINY = ["tiny-a", "redisun-tiny", "pezarax-tiny", "devalorn-tiny", "vakilorn-tiny", "musilorn-tiny", "lemunex-tiny"]


def _unbuilt(runtime):
    gc.collect()
    return [o for o in gc.get_objects() if type(o) in (FusedInput, ResultProduct) and
            o.runtime is runtime and o.host is None and o._linear is None]


def _folder(tmp_path, size, dtype):
    arch, cfg = named_size(size)
    make_random_model(str(tmp_path), cfg, seed=1, dtype=dtype)
    return arch, cfg, str(tmp_path)


@pytest.mark.parametrize("size", TINY)
def test_settle_builds_every_joined_matrix(tmp_path, size):
    arch, cfg, folder = _folder(tmp_path, size, torch.float32)
    runtime = Runtime(device=torch.device("cpu"), dtype=torch.float32)
    store = load_weights(folder, arch.expected_tensors(cfg), torch.device("cpu"),
                         strip_prefixes=arch.strip_prefixes, ignorable=arch.ignorable)
    model = arch.build(cfg, store, runtime)
    model.settle()
    assert _unbuilt(runtime) == []


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("size", TINY)
def test_a_loaded_model_has_nothing_left_to_build(tmp_path, size, dtype):
    _arch, _cfg, folder = _folder(tmp_path, size, getattr(torch, dtype))
    m = load_lm(folder, dtype=dtype, max_lanes=2, max_batched_tokens=64)
    assert _unbuilt(m.loaded.runtime) == []
