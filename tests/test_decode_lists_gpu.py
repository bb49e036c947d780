"""Decode attention of launches of more than 64 tokens, up to the most the ring kernel takes, by itself
and in an engine made for as many requests."""
import random

import pytest
import torch

from pretrained_rstr_b200 import load_lm
from pretrained_rstr_b200.config import GPT2Config
from pretrained_rstr_b200.engine.batch import Entry
from pretrained_rstr_b200.settings import SETTINGS
from pretrained_rstr_b200.weights import make_random_model

from test_kernels_gpu import _ops, _paged_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", [64, 65, 128, 255, 256])
@pytest.mark.parametrize("nh,nkv,ps,window", [(12, 12, 64, None), (4, 2, 16, 100), (3, 1, 32, None)])
def test_ring_attention_of_long_token_lists(t, nh, nkv, ps, window):
    ops = _ops()
    rng = random.Random(t + nh)
    lengths = [rng.choice([1, 31, 32, 33, 64, 65, 200, 513, 1000]) + rng.randrange(20) for _ in range(t)]
    q, k, v, table, seq, pos = _paged_case(t, nh, nkv, 64, ps, lengths, [1] * t, torch.bfloat16)
    order = list(range(t))
    rng.shuffle(order)
    tokens = torch.tensor(order, dtype=torch.int32, device="cuda")
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    ref = torch.empty_like(q)
    ops.attention_generic(ref, q, k, v, table, seq, pos, t, nh, 0.2, window, 1024, status)
    ws = torch.full((ops.decode_ring_workspace(t, nh, 64),), float("nan"), device="cuda")
    counters = torch.zeros(t * nh, dtype=torch.int32, device="cuda")
    for used in (t, t - 3):
        count = torch.tensor([used], dtype=torch.int32, device="cuda")
        out = torch.full_like(q, float("nan"))
        ops.attention_decode_ring(out, q, k, v, table, seq, pos, tokens, count, t, nh, 0.2, window, ws, counters,
                                  status, new_keys=4, max_context=1024)
        # weights of a sum of one, each rounded to bfloat16 (2^-9), times values of up to five or so,
        # and the result's own rounding
        assert float((out[order[:used]].float() - ref[order[:used]].float()).abs().max()) <= 2e-2
        assert bool(torch.isnan(out[order[used:]]).all())
        assert int(counters.abs().sum()) == 0
    assert status.tolist() == [0, 0, 0, 0]


@pytest.mark.parametrize("blocks", [2, 5, 8])
def test_ring_attention_merges_in_one_order(blocks):
    """Blocks of 32 keys, a warp each: in the warps of one CTA where a token an SM is asked for, in a CTA each
    where few are.  Either way their states are merged in the keys' order: the same bits."""
    ops = _ops()
    sms = min(ops.sm_count(), ops.decode_ring_max_list())
    few = max(1, sms // blocks)
    _q, k, v, table, seq, pos = _paged_case(blocks, 1, 1, 64, 64, [32 * blocks - i % 32 for i in range(sms)],
                                            [1] * sms, torch.bfloat16)
    ws = torch.zeros(ops.decode_ring_workspace(sms, 1, 64), device="cuda")
    counters = torch.zeros(sms, dtype=torch.int32, device="cuda")
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    for seed in range(40):
        q = torch.randn(sms, 64, generator=torch.Generator().manual_seed(seed)).to(torch.bfloat16).cuda()
        many, apart = torch.full_like(q, float("nan")), torch.full_like(q, float("nan"))
        ops.attention_decode_ring(many, q, k, v, table, seq, pos, None, None, sms, 1, 0.2, None, ws, counters, status)
        for first in range(0, sms, few):
            tokens = torch.arange(first, min(sms, first + few), dtype=torch.int32, device="cuda")
            ops.attention_decode_ring(apart, q, k, v, table, seq, pos, tokens, None, len(tokens), 1, 0.2, None, ws,
                                      counters, status)
        assert torch.equal(many, apart)
    assert status.tolist() == [0, 0, 0, 0] and int(counters.abs().sum()) == 0


@pytest.mark.parametrize("requests,context", [(100, 600), (130, 70)])
def test_an_engine_of_many_requests_by_either_decode_attention(tmp_path, monkeypatch, requests, context):
    cfg = GPT2Config.from_dict(dict(n_layer=2, n_embd=256, n_head=4, n_inner=512, vocab_size=512, n_positions=1024))
    make_random_model(str(tmp_path), cfg, seed=3, dtype=torch.bfloat16)
    rng = random.Random(requests)
    prompts = [[rng.randrange(512) for _ in range(context - rng.randrange(40))] for _ in range(requests)]
    given = [[rng.randrange(512) for _ in range(requests)] for _ in range(3)]
    results = []
    for ring in (False, True, None):
        monkeypatch.setattr(SETTINGS, "decode_ring", ring)
        m = load_lm(str(tmp_path), dtype="bfloat16", max_lanes=requests, max_batched_tokens=2048, maxpos=1024)
        runner, cache = m.loaded.runner, m.loaded.cache
        for b, prompt in enumerate(prompts):
            cache.open(b)
            runner.step([Entry(b, prompt, [len(prompt) - 1])])
        logits = [runner.step([Entry(b, [step[b]], [0]) for b in range(requests)]).clone() for step in given]
        results.append(torch.stack(logits))
    size = float(results[0].float().pow(2).mean().sqrt())
    # (two layers whose attention is rounded to bfloat16 in other places)
    assert float((results[1] - results[0]).abs().max()) <= 0.1 * size
    assert float((results[2] - results[0]).abs().max()) <= 0.1 * size


def test_few_requests_take_the_split_key_attention():
    """A request or eight by the ring kernel: 1 to 8 % more a decode step, at every context and size."""
    ops = _ops()
    for heads in (12, 16, 25):
        for context in (64, 256, 512, 1024):
            assert not ops.decode_ring_prefers(1, heads, context)
            assert not ops.decode_ring_prefers(8, 12, context)
    assert ops.decode_ring_prefers(32, 12, 1024) and ops.decode_ring_prefers(256, 12, 1024)
