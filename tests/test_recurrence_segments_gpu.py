"""Recurrences of steps that are cut into segments of tokens: requests of one and of several segments, cut at edges of a
segment, carried on by a second step, single tokens and a padding row among them."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F = torch.float64


def scan(q, b, a, v, S):
    out = []
    for t in range(q.shape[0]):
        S = a[t] * S + b[t][:, :, None] * v[t][:, None, :]
        out.append((S * q[t][:, :, None]).sum(1))
    return torch.stack(out), S


@pytest.mark.parametrize("H,d,dv", [(2, 20, 33), (1, 64, 32), (2, 100, 70), (1, 128, 128), (1, 200, 40)])
@pytest.mark.parametrize("mode", ["fixed", "gate", "key", "step"])
def test_segments_against_one_scan(H, d, dv, mode, monkeypatch):
    from dispec_b200.ops import recurrence as R
    monkeypatch.setattr(R, "_MAX_SEGMENTS", 4)  # segments of 128 tokens in the first step, of 64 in the second
    g = torch.Generator().manual_seed(d + dv)
    rnd = lambda *s: torch.randn(*s, generator=g)
    steps = [[300, 1, 128, 129, 0, 40], [64, 65, 1, 60, 3, 63]]  # tokens of each request in each step
    N, slots, rank = len(steps[0]), [5, 0, 3, 1, 6, 2], 5
    cols = 2 * H * d + H * dv + rank
    state = torch.full((8, H, d, dv), float("nan"), device=DEV)
    state[slots] = rnd(N, H, d, dv).to(DEV)
    want_state = {s: state[slots[s]].cpu().to(F) for s in range(N)}
    decay, bias, lower = torch.tensor([0.97, 1.0])[:H], 2.0 + rnd(H * d), 0.9 * torch.rand(H * d, generator=g)
    gate_map, skip = rnd(rank, H * d) / 3, rnd(H)
    seen = [0] * N
    for lens in steps:
        T = sum(lens)
        proj, dt = rnd(T + 1, cols), torch.rand(T + 1, H, generator=g)
        proj[T] = float("nan")  # a padding row: position -1, its slot is not touched
        alpha = torch.exp(-0.05 * dt)
        starts, positions = [0], []
        for s, n in enumerate(lens):
            starts.append(starts[-1] + n)
            positions += list(range(seen[s], seen[s] + n))
        starts.append(T + 1)
        i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
        kw, code = {"fixed": (dict(decay=decay), R.FIXED_DECAY),
                    "gate": (dict(gate_bias=bias, lower=lower), R.FORGET_GATE),
                    "key": (dict(gate_map=gate_map, gate_bias=bias, low_off=cols - rank, power=0.3), R.KEY_DECAY),
                    "step": (dict(steps=torch.stack([dt, alpha], 1).contiguous(), skip=skip, num_groups=H), R.STEP_DECAY)}[mode]
        kw = {k: v.to(DEV) if isinstance(v, torch.Tensor) else v for k, v in kw.items()}
        got = R.linear_recurrence(proj.to(DEV), 0, H * d, 2 * H * d, code, H, d, dv, state, i32(slots + [7]), i32(starts),
                                  i32(positions + [-1]), **kw).cpu().to(F)
        for s, n in enumerate(lens):
            if n == 0:
                continue
            rows = slice(starts[s], starts[s] + n)
            x = proj[rows].to(F)
            q, k, v = x[:, :H * d].view(n, H, d), x[:, H * d:2 * H * d].view(n, H, d), x[:, 2 * H * d:2 * H * d + H * dv].view(n, H, dv)
            if mode == "fixed":
                a = decay.to(F)[None, :, None, None].expand(n, H, 1, 1)
            elif mode == "gate":
                f = lower.to(F) + (1 - lower.to(F)) * torch.sigmoid(x[:, H * d:2 * H * d] + bias.to(F))
                q, k, a = torch.nn.functional.silu(q), (1 - f).view(n, H, d), f.view(n, H, d, 1)
            elif mode == "key":
                a = (torch.sigmoid(x[:, cols - rank:] @ gate_map.to(F) + bias.to(F)) ** 0.3).view(n, H, d, 1)
            else:
                a = alpha[rows].to(F)[:, :, None, None]
            w = v * dt[rows].to(F)[:, :, None] if mode == "step" else v
            o, want_state[s] = scan(q, k, a, w, want_state[s])
            if mode == "step":
                o = o + skip.to(F)[:, None] * v
            # sums of up to d (products) and 300 (tokens) terms in 32 bits
            assert (got[rows].view(n, H, dv) - o).abs().max() < 3e-5 * o.abs().max(), (lens, s)
            assert (state[slots[s]].cpu().to(F) - want_state[s]).abs().max() < 3e-5 * want_state[s].abs().max(), (lens, s)
            seen[s] += n
    assert torch.isnan(state[[4, 7]]).all()
