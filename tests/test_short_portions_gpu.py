"""Many requests that bring a few tokens each beside long contexts: steps that queue up behind one another."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
WIDTH, HEADS, DIM, VOCAB = 1536, 12, 128, 4000


def model_of(kinds):
    from dispec_b200 import load_model_config
    from dispec_b200.weights import load_random_model
    mlp = {"kind": "dense", "ff": 8960}
    mixers = {"attention": {"heads": HEADS, "kv_heads": 2, "dim": DIM, "vdim": DIM, "scale": DIM ** -0.5,
                            "rot": {"base": 1e6, "dims": DIM}},
              "delta": {"heads": HEADS, "kv_heads": HEADS, "dim": DIM, "vdim": DIM, "conv": 4}}
    cfg = {"architecture": "Pikalorn", "vocab": VOCAB, "width": WIDTH, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-6},
           "layers": [{"type": k, "mlp": mlp, "mixer": mixers[k]} for k in kinds]}
    return load_random_model(load_model_config(cfg), 3, 0.02, "bfloat16", DEV)


@pytest.mark.parametrize("kinds,requests,stored,new,steps", [
    (("delta", "attention", "delta", "attention"), 64, 1000, 2, 24),
    (("delta", "attention", "delta", "attention"), 64, 1000, 4, 24),
])
def test_no_wait_runs_out(kinds, requests, stored, new, steps):
    """Portions of two and four tokens of 64 requests after 1,000 stored ones, without a look at the device in between."""
    from dispec_b200 import ModelRunner, SeqEntry
    runner = ModelRunner(model_of(kinds), page_size=16, num_pages=requests * ((stored + steps * new) // 16 + 2),
                         max_num_seqs=requests)
    g = torch.Generator().manual_seed(1)
    ids = torch.randint(0, VOCAB, (requests, stored + steps * new), generator=g).tolist()
    for i in range(requests):
        runner.admit(i)
    at = 0
    while at < stored:
        n = min(stored - at, 125)
        runner.step([SeqEntry(i, ids[i][at:at + n], at) for i in range(requests)])
        at += n
    for _ in range(steps):
        logits = runner.step([SeqEntry(i, ids[i][at:at + new], at, [new - 1]) for i in range(requests)])
        at += new
    runner.check_device()
    assert logits.isfinite().all()
