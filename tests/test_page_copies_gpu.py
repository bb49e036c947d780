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


def test_pages_copied_in_a_step_are_those_its_decode_attention_asks_for_early(tmp_path, monkeypatch):
    """bfloat16, head size 64: the ring attention asks for cached pages before the kernel ahead of it has ended, among
    them the pages that the step has just copied.  Steps one behind the other give the bits of steps waited for."""
    from pretrained_rstr_b200 import load_lm
    from pretrained_rstr_b200.engine.batch import Entry
    from pretrained_rstr_b200.settings import SETTINGS
    monkeypatch.setattr(SETTINGS, "decode_ring", True)
    raw, seed = TINY["C"]
    folder = make_folder(str(tmp_path), raw, seed, "bfloat16")
    base = random_tokens(230, raw["vocab_size"], 5)              # (the last of four pages is filled in part)
    kids = [random_tokens(13, raw["vocab_size"], 40 + i) for i in range(12)]
    runs = []
    for waits in (True, False):
        lm = load_lm(folder, gpu=True, dtype="bfloat16", max_lanes=16, max_batched_tokens=512, share_prefixes=False)
        cache, runner = lm.loaded.cache, lm.loaded.runner
        cache.open("root")
        runner.step([Entry("root", base, [229])])
        torch.cuda.synchronize()
        filler = torch.randn(4096, 4096, device="cuda")
        for _ in range(8):
            filler = filler @ filler * 1e-2                      # the stream is busy while the host goes on
        got = []
        for k in range(len(kids)):
            cache.fork("root", k)
            logits = runner.step([Entry(i, [kids[i][k - i]], [0]) for i in range(k + 1)])
            got.append(logits.clone())
            if waits:
                torch.cuda.synchronize()
        assert runner.counters["cow_copies"] >= len(kids)
        runner.fetch_result()
        runs.append(torch.cat(got))
    assert torch.equal(runs[0], runs[1])
    # (the same tokens without a copy: a request of its own that holds all of them)
    cache.open("alone")
    runner.step([Entry("alone", base + kids[0][:1], [230])])
    alone = [runner.step([Entry("alone", [t], [0])]).clone() for t in kids[0][1:12]]
    for k, row in enumerate(alone):
        at = sum(range(1, k + 2))                                # kid 0 is the first row of every step
        assert float((runs[1][at].float() - row[0].float()).abs().max()) <= ATOL["bfloat16"]
