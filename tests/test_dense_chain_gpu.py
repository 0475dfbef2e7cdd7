"""The layers behind one call give the bits that the parts give one by one."""
import pytest
import torch

import replay_util as ru

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def model_of(**changes):
    from dispec_b200 import load_model_config
    from dispec_b200.weights import load_random_model
    cfg = dict(ru.CONFIG_B)
    cfg.update(changes)
    return load_random_model(load_model_config(cfg), 3, 0.05, "bfloat16", DEV)


def run(model, chain, lengths, steps, page_size, graph=False):
    """A step that reads prompts of ``lengths`` together, then ``steps`` steps in which each takes a token, the last of
    them beside a new prompt."""
    from dispec_b200.engine import ModelRunner, SeqEntry
    model.dense_chain = chain
    runner = ModelRunner(model, page_size=page_size, num_pages=200, max_num_seqs=len(lengths) + 1, cuda_graph=graph)
    ids = [ru.random_ids(n + steps + 1, model.spec.vocab_size, 5 + i) for i, n in enumerate(lengths)]
    for i in range(len(lengths)):
        runner.admit(i)
    out = [runner.step([SeqEntry(i, s[:n], 0, [n - 1, n // 2]) for i, (s, n) in enumerate(zip(ids, lengths))]).clone()]
    for t in range(steps):
        entries = [SeqEntry(i, s[n + t:n + t + 1], n + t, [0]) for i, (s, n) in enumerate(zip(ids, lengths))]
        if t == steps - 1:
            runner.admit("late")
            entries.append(SeqEntry("late", ru.random_ids(19, model.spec.vocab_size, 4), 0, [18]))
        out.append(runner.step(entries).clone())
    runner.check_device()
    return out, runner


@pytest.mark.parametrize("changes,lengths,page_size", [
    ({}, [1], 16), ({}, [7, 3], 8), ({}, [63], 16), ({}, [64], 16), ({}, [65, 1], 32), ({}, [128], 16), ({}, [129], 8),
    ({}, [300, 40, 2], 16),
    (dict(tie_word_embeddings=True, num_attention_heads=4, num_key_value_heads=4), [33, 5], 16),
    # a window in some layers, pages that the tiles of 128 rows do not take
    (dict(use_sliding_window=True, sliding_window=24, max_window_layers=1), [90, 20], 16),
    (dict(use_sliding_window=True, sliding_window=24, max_window_layers=1), [90, 20], 4),
    (dict(head_dim=64, num_attention_heads=4, num_key_value_heads=2), [150, 9], 16),
    (dict(head_dim=128, num_attention_heads=6, num_key_value_heads=1), [200], 16),
    (dict(head_dim=80, num_attention_heads=4, num_key_value_heads=2), [70, 30], 16),
])
def test_same_bits_as_the_parts(changes, lengths, page_size):
    from dispec_b200.ops.library import LaunchCounter
    model = model_of(**changes)
    assert model.dense_chain
    n0 = LaunchCounter.n
    mine, _ = run(model, True, lengths, 3, page_size)
    n1 = LaunchCounter.n
    parts, _ = run(model, False, lengths, 3, page_size)
    assert LaunchCounter.n - n1 == n1 - n0
    for a, b in zip(mine, parts):
        assert torch.equal(a, b)


def test_from_captured_steps():
    model = model_of()
    mine, runner = run(model, True, [40, 70, 12], 4, 16, graph=True)
    assert runner._graphs
    parts, _ = run(model, False, [40, 70, 12], 4, 16, graph=True)
    for a, b in zip(mine, parts):
        assert torch.equal(a, b)


@pytest.mark.parametrize("changes", [dict(intermediate_size=232), dict(head_dim=24)])
def test_sizes_that_stay_with_the_parts(changes):
    assert not model_of(**changes).dense_chain


def test_weights_off_sixteen_bytes_stay_with_the_parts():
    """A source may serve views of one slab at any offset: the parts' products take them, the chain's do not."""
    from dispec_b200.ops.library import LaunchCounter
    model = model_of()
    for part, name in ((model.layers[0].mixer, "w_o"), (model.layers[-1].feed_forward, "w_down")):
        w = getattr(part, name)
        slab = torch.empty(w.numel() + 3, dtype=w.dtype, device=w.device)
        slab[3:].copy_(w.flatten())
        setattr(part, name, slab[3:].view(w.shape))
    n0 = LaunchCounter.n
    mine, _ = run(model, True, [70, 9], 2, 16)
    n1 = LaunchCounter.n
    parts, _ = run(model, False, [70, 9], 2, 16)
    assert LaunchCounter.n - n1 == n1 - n0
    for a, b in zip(mine, parts):
        assert torch.equal(a, b)


def test_a_bias_off_eight_bytes():
    """At sizes where the product on CTA pairs is chosen, which takes no such bias: another kernel runs, as in the parts."""
    from dispec_b200.ops import gemm, tuning
    model = model_of(hidden_size=1536, intermediate_size=2048, num_attention_heads=12, num_key_value_heads=2, head_dim=128)
    mixer = model.layers[0].mixer
    slab = torch.empty(1536 + 1, dtype=torch.bfloat16, device=DEV).normal_()
    mixer.b_o = slab[1:]
    assert model.dense_chain and tuning.pairs_are_faster(536, 1536, 1536)
    x = torch.zeros((536, 1536), dtype=torch.bfloat16, device=DEV)
    assert gemm.pairs_supported(x, mixer.w_o, None, x, x) and not gemm.pairs_supported(x, mixer.w_o, mixer.b_o, x, x)
    mine, _ = run(model, True, [500, 36], 2, 16)
    parts, _ = run(model, False, [500, 36], 2, 16)
    for a, b in zip(mine, parts):
        assert torch.equal(a, b)


@pytest.mark.parametrize("prompts,stored", [([137], 0), ([536], 0), ([700, 40], 0), ([1900], 0), ([24, 5], 4200), ([300], 9000)])
def test_same_bits_at_the_sizes_where_c_chooses(prompts, stored):
    """Two layers of the 1.5B sizes: few-row products above 128 rows, products that let their successor start late, norms a
    warp a row, and (``stored``) a single token whose keys are cut into ranges beyond a cluster."""
    from dispec_b200.engine import ModelRunner, SeqEntry
    from dispec_b200.ops import attention as A, tuning
    dev = torch.device(DEV)
    model = model_of(hidden_size=1536, intermediate_size=8960, num_hidden_layers=2, num_attention_heads=12,
                     num_key_value_heads=2, head_dim=128, max_position_embeddings=16384)
    assert model.dense_chain
    T = sum(prompts) + (stored > 0)
    assert tuning.rows_in_chunks_is_faster(T, 1536, 8960, dev) is (T <= 1152) and 2 * 1536 * 8960 >= tuning.STREAM_LATE_TRIGGER_BYTES
    if stored:
        splits = A.choose_splits(1, 2, stored + 1, dev)
        assert A.choose_outer(1, 2, stored + 1, splits, dev) > 1
    vocab, out = model.spec.vocab_size, []
    for chain in (True, False):
        model.dense_chain = chain
        runner = ModelRunner(model, page_size=16, num_pages=(stored + sum(prompts)) // 16 + 40, max_num_seqs=4)
        entries = []
        if stored:
            runner.admit("long")
            ids = ru.random_ids(stored + 1, vocab, 11)
            for at in range(0, stored, 1500):
                runner.step([SeqEntry("long", ids[at:min(stored, at + 1500)], at)])
            entries.append(SeqEntry("long", ids[stored:], stored, [0]))
        for i, n in enumerate(prompts):
            runner.admit(i)
            entries.append(SeqEntry(i, ru.random_ids(n, vocab, 20 + i), 0, [n - 1, n // 2]))
        out.append(runner.step(entries).clone())
        runner.check_device()
    assert torch.equal(*out) and out[0].isfinite().all()
