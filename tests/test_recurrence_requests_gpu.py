"""Long requests of a recurrence are cut into segments: by their own tokens alone, so that a request has the same bits alone,
among others and with little memory."""
import pytest
import torch

from test_recurrence_segments_gpu import scan

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F = torch.float64
LENS = [300, 1, 128, 129, 0, 40, 127, 192, 257, 3]  # cut from 128 on; 257 and 300 in segments of 128 with three at most


def inputs(H, d, dv, mode, seed):
    from dispec_b200.ops import recurrence as R
    g = torch.Generator().manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=g)
    T, N, rank = sum(LENS), len(LENS), 5
    proj, dt, state = rnd(T, 2 * H * d + H * dv + rank), torch.rand(T, H, generator=g), rnd(N, H, d, dv)
    kw, code = {"fixed": (dict(decay=torch.linspace(0.9, 1.0, H)), R.FIXED_DECAY),
                "gate": (dict(gate_bias=2.0 + rnd(H * d), lower=0.9 * torch.rand(H * d, generator=g)), R.FORGET_GATE),
                "key": (dict(gate_map=rnd(rank, H * d) / 3, gate_bias=2.0 + rnd(H * d), low_off=proj.shape[1] - rank, power=0.3),
                        R.KEY_DECAY),
                "step": (dict(skip=rnd(H), num_groups=H), R.STEP_DECAY)}[mode]
    kw = {k: v.to(DEV) if isinstance(v, torch.Tensor) else v for k, v in kw.items()}
    return proj.to(DEV), dt, state, kw, code


def run(H, d, dv, mode, who, data, known=True):
    """The requests ``who`` in one step: (outputs, state) of each."""
    from dispec_b200.ops import recurrence as R
    proj, dt, state, kw, code = data
    starts = [sum(LENS[:i]) for i in range(len(LENS))]
    rows = torch.cat([torch.arange(starts[s], starts[s] + LENS[s]) for s in who])
    if mode == "step":
        kw = dict(kw, steps=torch.stack([dt, torch.exp(-0.05 * dt)], 1)[rows].contiguous().to(DEV))
    if known:
        kw = dict(kw, host_q_len=[LENS[s] for s in who])
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    st = state[who].contiguous().to(DEV)
    q0 = [0]
    for s in who:
        q0.append(q0[-1] + LENS[s])
    out = R.linear_recurrence(proj[rows.to(DEV)].contiguous(), 0, H * d, 2 * H * d, code, H, d, dv, st, i32(list(range(len(who)))),
                              i32(q0), i32([t for s in who for t in range(LENS[s])]), **kw)
    return [(out[a:b], st[i]) for i, (a, b) in enumerate(zip(q0, q0[1:]))]


def same(a, b):
    return torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])


@pytest.mark.parametrize("H,d,dv", [(2, 20, 33), (3, 64, 32), (2, 100, 70), (4, 128, 128), (1, 200, 40)])
@pytest.mark.parametrize("mode", ["fixed", "gate", "key", "step"])
def test_the_same_bits_alone_and_among_others(H, d, dv, mode, monkeypatch):
    from dispec_b200.ops import recurrence as R
    monkeypatch.setattr(R, "SEGMENTS_MIN_TOKENS", 128)
    monkeypatch.setattr(R, "_MAX_SEGMENTS", 3)
    data, all_of_them = inputs(H, d, dv, mode, d + dv), list(range(len(LENS)))
    together = run(H, d, dv, mode, all_of_them, data, known=False)
    for s, n in enumerate(LENS):
        if n > 2:  # (single tokens alone take a kernel of their own)
            assert same(run(H, d, dv, mode, [s], data, known=False)[0], together[s]), n
    assert all(map(same, together, run(H, d, dv, mode, all_of_them, data)))
    monkeypatch.setattr(R, "_SEGMENTS_BYTES", 1)  # one head at a time
    assert all(map(same, together, run(H, d, dv, mode, all_of_them, data)))


@pytest.mark.parametrize("H,d,dv", [(2, 20, 33), (3, 64, 32), (2, 100, 70), (4, 128, 128), (1, 200, 40)])
def test_against_one_scan(H, d, dv, monkeypatch):
    from dispec_b200.ops import recurrence as R
    monkeypatch.setattr(R, "SEGMENTS_MIN_TOKENS", 128)
    monkeypatch.setattr(R, "_MAX_SEGMENTS", 3)
    proj, dt, state, kw, _ = data = inputs(H, d, dv, "gate", 7)
    x, lower, bias = proj.cpu().to(F), kw["lower"].cpu().to(F), kw["gate_bias"].cpu().to(F)
    f = lower + (1 - lower) * torch.sigmoid(x[:, H * d:2 * H * d] + bias)
    q, v = torch.nn.functional.silu(x[:, :H * d]), x[:, 2 * H * d:2 * H * d + H * dv]
    at = 0
    for s, (got, got_state) in enumerate(run(H, d, dv, "gate", list(range(len(LENS))), data)):
        n = LENS[s]
        if n == 0:
            continue
        a, rows = f[at:at + n].view(n, H, d, 1), slice(at, at + n)
        want, want_state = scan(q[rows].view(n, H, d), 1 - a[..., 0], a, v[rows].view(n, H, dv), state[s].to(F))
        # sums of up to d (products) and 300 (tokens) terms in 32 bits
        assert (got.cpu().to(F).view(n, H, dv) - want).abs().max() < 3e-5 * want.abs().max()
        assert (got_state.cpu().to(F) - want_state).abs().max() < 3e-5 * want_state.abs().max()
        at += n


@pytest.mark.parametrize("mode", ["gate", "step"])
def test_a_long_request_beside_many_single_tokens(mode, monkeypatch):
    """The single tokens have the bits of a step without the long request, whether the host knows the lengths or not."""
    from dispec_b200.ops import recurrence as R
    monkeypatch.setattr(R, "SEGMENTS_MIN_TOKENS", 128)
    monkeypatch.setitem(globals(), "LENS", [200] + [1] * 250)
    data = inputs(2, 64, 64, mode, 9)
    together = run(2, 64, 64, mode, list(range(251)), data)
    assert all(map(same, together, run(2, 64, 64, mode, list(range(251)), data, known=False)))
    assert all(map(same, together[1:], run(2, 64, 64, mode, list(range(1, 251)), data)))
    assert same(together[0], run(2, 64, 64, mode, [0], data)[0])


def test_memory_that_is_refused_gives_the_same_bits(monkeypatch):
    from dispec_b200.ops import recurrence as R
    monkeypatch.setattr(R, "SEGMENTS_MIN_TOKENS", 128)
    who = [0, 1, 7]
    data = inputs(4, 128, 128, "fixed", 3)
    want = run(4, 128, 128, "fixed", who, data)
    refused, empty = [], torch.empty

    def scarce(size, *a, **k):
        if isinstance(size, int) and size > R._segment_floats(sum(LENS[s] for s in who), 1, 128, 128):
            refused.append(size)
            raise torch.OutOfMemoryError("CUDA out of memory.")
        return empty(size, *a, **k)

    monkeypatch.setattr(R.torch, "empty", scarce)
    got = run(4, 128, 128, "fixed", who, data)
    monkeypatch.undo()
    assert len(refused) == 2  # four heads, two heads, one
    assert all(map(same, want, got))
