"""Copy-on-write in steps that follow one another without a wait between them."""
import pytest
import torch

from helpers import ATOL, TINY, make_folder, oracle_logits, random_tokens

pytestmark = pytest.mark.gpu


def test_forks_in_steps_launched_one_behind_the_other(tmp_path):
    """Every step forks another context off the root and runs a token of all of them: the description of a
    step's page copies must stay as it is until the copies have run, however far ahead the host is."""
    from pretrained_rstr_b200 import load_lm
    from pretrained_rstr_b200.engine.batch import Entry
    raw, seed = TINY["A"]
    folder = make_folder(str(tmp_path), raw, seed, "float32")
    base = random_tokens(70, raw["vocab_size"], 3)
    tails = {f"kid{i}": random_tokens(6 - i, raw["vocab_size"], 20 + i) for i in range(6)}
    oracle = oracle_logits(folder, {rid: base + tail for rid, tail in tails.items()})
    lm = load_lm(folder, gpu=True, dtype="float32", max_lanes=8, max_batched_tokens=256, share_prefixes=False)
    cache, runner = lm.loaded.cache, lm.loaded.runner
    cache.open("root")
    runner.step([Entry("root", base, [69])])
    filler = torch.randn(4096, 4096, device="cuda")
    for _ in range(8):
        filler = filler @ filler * 1e-2                    # the stream is busy while the host goes on
    got = []
    for k in range(6):
        cache.fork("root", f"kid{k}")
        live = [f"kid{i}" for i in range(k + 1)]
        logits = runner.step([Entry(rid, [tails[rid][k - i]], [0]) for i, rid in enumerate(live)])
        got.append(logits.clone())
    assert runner.counters["cow_copies"] >= 6
    for k, rows in enumerate(got):
        for i in range(k + 1):
            want = oracle[f"kid{i}"][70 + k - i]
            assert float((rows[i].double().cpu() - want.double()).abs().max()) <= ATOL["float32"]
    for rid in ["root"] + list(tails):
        cache.close(rid)
