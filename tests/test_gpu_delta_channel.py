"""The delta rule with a decay per key channel in chunks of 64 tokens: the three kernels between the layer's projections
against the plain formulas in 64 bits and against the kernels that go token by token, at lengths around the edges of blocks of
16 and chunks of 64, with states of earlier steps, with decays from none at all to ones that leave nothing of the token before."""

import pytest
import torch

from tests.plain import pofadra as plain
from tests.test_gpu_kernels import DEV, F, rand

pytestmark = pytest.mark.gpu
EPS = 1e-5


def i32(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


class Layer:
    def __init__(self, lens, H, G, d, dv, taps, decay, seed):
        self.sizes, self.lens = (H, G, d, dv, taps), lens
        T, C = sum(lens), 2 * G * d + H * dv
        self.C = C
        width = -(-(C + H) // 8) * 8
        self.proj = rand(T, width, seed=seed).to(torch.bfloat16)
        self.low = rand(T, H * (d + dv), seed=seed + 1).float()
        self.conv_w = rand(C, taps, seed=seed + 2, scale=0.5).float()
        self.a_log = (rand(H, seed=seed + 3) * 0.7).float() + decay
        self.dt_bias = rand(H * d, seed=seed + 4).float()
        self.norm = 1 + 0.1 * rand(dv, seed=seed + 5).float()
        self.slots = torch.randperm(len(lens) + 2, generator=torch.Generator().manual_seed(seed))[:len(lens)].tolist()
        self.state = rand(len(lens) + 2, H, d, dv, seed=seed + 6).float()
        self.conv = rand(len(lens) + 2, max(taps - 1, 1), C, seed=seed + 7).float()

    def run(self, chunked, wave_bytes=None):
        H, G, d, dv, taps = self.sizes
        f, starts = F(), [0]
        for n in self.lens:
            starts.append(starts[-1] + n)
        seq = [i for i, n in enumerate(self.lens) for _ in range(n)]
        pos = [t for n in self.lens for t in range(n)]
        state, conv = self.state.to(DEV), self.conv.to(DEV)
        proj, low, conv_w, a_log, dt_bias, norm = (t.to(DEV) for t in (self.proj, self.low, self.conv_w, self.a_log, self.dt_bias, self.norm))
        if chunked:
            assert f.delta_channel_ok(proj, low, dt_bias, norm, conv if taps > 1 else None, state, d, dv, taps)
            y = f.delta_channel(proj, low, conv_w, conv if taps > 1 else None, a_log, dt_bias, norm, EPS, state, i32(starts), i32(self.slots),
                                len(self.lens), max(self.lens), H, G, d, dv, taps)
        else:
            parts = f.delta_prepare(proj, low, conv_w, conv if taps > 1 else None, a_log, dt_bias, i32(pos), i32(seq), i32(starts), i32(self.slots),
                                    H, G, d, dv, taps)
            if taps > 1:
                f.conv_roll(proj, conv, i32(starts), i32(self.slots), len(self.lens), self.C)
            o = f.delta_scan(*parts, state, i32(starts), i32(self.slots), len(self.lens))
            y = f.head_norm_gate(o, norm, low, H * d, EPS, torch.bfloat16)
        return y.double().cpu(), state.double().cpu(), conv.double().cpu()

    def oracle(self):
        """The plain formulas in 64 bits, token by token: gated read-outs and states."""
        H, G, d, dv, taps = self.sizes
        state, outs, at = self.state.double().clone(), [], 0
        for n, slot in zip(self.lens, self.slots):
            x = self.proj[at:at + n].double()
            before = self.conv[slot].double() if taps > 1 else x.new_zeros(0, self.C)
            full = torch.cat([before, x[:, :self.C]])
            act = plain.silu(sum(full[j:j + n] * self.conv_w.double()[:, j] for j in range(taps)))
            q = plain.unit(act[:, :G * d].view(n, G, d)) * d**-0.5
            k = plain.unit(act[:, G * d:2 * G * d].view(n, G, d))
            v = act[:, 2 * G * d:].view(n, H, dv)
            low = self.low[at:at + n].double()
            step = torch.nn.functional.softplus(low[:, :H * d] + self.dt_bias.double()).view(n, H, d)
            g = torch.exp(-torch.exp(self.a_log.double())[None, :, None] * step)
            beta = torch.sigmoid(x[:, self.C:self.C + H])
            S, o = state[slot], torch.empty(n, H, dv, dtype=torch.float64)
            own = torch.arange(H) // (H // G)
            for t in range(n):
                S = S * g[t][:, :, None]
                u = beta[t][:, None] * (v[t] - (k[t][own][:, None, :] @ S)[:, 0])
                S = S + k[t][own][:, :, None] * u[:, None, :]
                o[t] = (q[t][own][:, None, :] @ S)[:, 0]
            state[slot] = S
            o = o / (o.pow(2).mean(-1, keepdim=True) + EPS).sqrt() * self.norm.double() * torch.sigmoid(low[:, H * d:].view(n, H, dv))
            outs.append(o.view(n, H * dv))
            at += n
        return torch.cat(outs), state


def relative(got, want):
    return ((got - want).norm() / want.norm()).item()


# decay: the centre of log(-log g): -9 keeps all, 3 leaves e^-20 and less of a token before
@pytest.mark.parametrize("lens,H,G,d,dv,taps,decay", [
    ([1], 1, 1, 128, 128, 4, -1.0), ([15, 16, 17], 2, 1, 128, 128, 4, -1.0), ([63, 1, 64, 65], 4, 2, 128, 128, 4, -1.0),
    ([129, 3, 200], 2, 2, 64, 64, 4, -1.0), ([2, 100], 3, 3, 64, 16, 1, -1.0), ([33, 2], 2, 1, 128, 48, 2, -1.0), ([130, 48], 2, 2, 128, 112, 3, 0.0),
    ([300], 2, 1, 128, 128, 4, -9.0), ([190], 2, 2, 128, 128, 4, 3.0), ([190], 2, 2, 64, 64, 4, 5.0)])
def test_chunks_against_the_plain_formulas_and_the_token_by_token_kernels(lens, H, G, d, dv, taps, decay):
    layer = Layer(lens, H, G, d, dv, taps, decay, seed=7 * len(lens) + d + dv)
    want, want_state = layer.oracle()
    y, state, conv = layer.run(True)
    y0, state0, conv0 = layer.run(False)
    assert torch.equal(conv, conv0)
    used = layer.slots
    idle = [s for s in range(state.shape[0]) if s not in used]
    assert torch.equal(state[idle], layer.state.double()[idle])  # no other slot was touched
    # 32-bit operands and sums: a rounding of 2^-24 of the state a token, which decays may carry away, and those of the inputs
    assert relative(state[used], want_state[used]) < (16 + max(lens)) * 2.0**-24
    # no further from 64 bits than token by token; the margin is for sizes where both are a few roundings
    assert relative(state[used], want_state[used]) < 1.5 * relative(state0[used], want_state[used]) + 1e-7
    # the read-outs are rounded to bfloat16 at the end: half a place of eight bits each
    assert ((y - want).abs() <= 2.0**-8 * want.abs() + 1e-4 * want.abs().max()).all()
    assert relative(y, want) < 1.05 * relative(y0, want) + 1e-5


def test_a_prompt_in_waves_and_in_portions_is_the_whole_prompt(monkeypatch):
    """More chunks than the workspace holds at a time, and a prompt cut where the convolution and the state have to carry over."""
    whole = Layer([333], 2, 1, 128, 128, 4, -1.0, seed=3)
    y, state, conv = whole.run(True)
    f = F()
    monkeypatch.setattr(f, "DELTA_WORKSPACE_BYTES", 2 * 2 * 4 * f.library().gk_delta_channel_work(128))
    y2, state2, conv2 = whole.run(True)
    assert torch.equal(y, y2) and torch.equal(state, state2) and torch.equal(conv, conv2)
    monkeypatch.undo()
    parts, at = [], 0
    cut = Layer([333], 2, 1, 128, 128, 4, -1.0, seed=3)
    for n in (100, 1, 2, 64, 166):
        piece = Layer([n], 2, 1, 128, 128, 4, -1.0, seed=3)
        for name in ("conv_w", "a_log", "dt_bias", "norm", "slots", "state", "conv"):
            setattr(piece, name, getattr(cut, name))
        piece.proj, piece.low = whole.proj[at:at + n].contiguous(), whole.low[at:at + n].contiguous()
        y3, state3, conv3 = piece.run(True)
        cut.state, cut.conv = state3.float(), conv3.float()
        parts.append(y3)
        at += n
    assert torch.equal(conv3, conv) and relative(state3, state) < 2e-6
    assert relative(torch.cat(parts), y) < 2e-3


@pytest.mark.parametrize("lens,decay", [([192], -1.0), ([260, 40], -1.0), ([400], -2.0), ([192, 64], -9.0)])
def test_states_are_no_further_from_64_bits_than_token_by_token(lens, decay):
    """What a product leaves out (2^-27.5 of it, root mean square) is less than a rounded addition, and there are fewer additions than token by token."""
    chunks = tokens = 0.0
    for seed in range(1, 9):
        layer = Layer(lens, 4, 4, 128, 128, 4, decay, seed=seed)
        _, want = layer.oracle()
        used = layer.slots
        chunks += relative(layer.run(True)[1][used], want[used])
        tokens += relative(layer.run(False)[1][used], want[used])
    assert chunks <= tokens


@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf")])
@pytest.mark.parametrize("where", ["q", "k", "v", "beta", "decay", "gate", "state", "conv"])
def test_what_is_no_number_comes_out_where_it_does_token_by_token(where, value):
    """Of one token (in the middle of a block of 16, behind other tokens of its chunk) or of the state: the tokens in front, the other heads and
    the other sequence stay numbers, and nothing that is no number is lost."""
    H, G, d, dv = 2, 2, 128, 128
    for at in (0, 87, 127):
        layer = Layer([150, 40], H, G, d, dv, 4, -1.0, seed=11)
        column = {"q": d + 3, "k": G * d + d + 3, "v": 2 * G * d + dv + 5, "beta": layer.C + 1}
        if where in column:
            layer.proj[at, column[where]] = value
        elif where in ("decay", "gate"):
            layer.low[at, d + 7 if where == "decay" else H * d + dv + 7] = value
        elif where == "state":
            layer.state[layer.slots[0], 1, 9, 5] = value
        else:
            layer.conv[layer.slots[0], 2, 2 * G * d + dv + 5] = value
        y, state, conv = layer.run(True)
        y0, state0, conv0 = layer.run(False)
        assert torch.equal(conv.isnan(), conv0.isnan()) and torch.equal(conv[~conv.isnan()], conv0[~conv0.isnan()])
        # a head's row at a token; for infinities 0 * infinity decides which of a row's entries are none, so rows and states' columns as a whole
        lost = lambda t, t0: (~t0.isfinite()).any(-1) & t.isfinite().all(-1)
        made = lambda t, t0: (~t.isfinite()).any(-1) & t0.isfinite().all(-1)
        rows, rows0 = y.view(190, H, dv), y0.view(190, H, dv)
        turned, turned0 = state.transpose(-1, -2), state0.transpose(-1, -2)
        assert not lost(rows, rows0).any() and not lost(turned, turned0).any()
        assert not made(rows, rows0).any() and not made(turned, turned0).any()
        if value != value:
            assert torch.equal(y.isnan(), y0.isnan()) and torch.equal(state.isnan(), state0.isnan())
        # what stays a number is what it was
        fine, fine0 = y.isfinite() & y0.isfinite(), state.isfinite() & state0.isfinite()
        assert ((y - y0).abs()[fine] <= 2.0**-7 * y0.abs()[fine] + 1e-4).all() and ((state - state0).abs()[fine0] <= 1e-5).all()


def test_many_sequences_stay_within_the_workspace_and_go_in_groups(monkeypatch):
    """One run beside many single tokens: the workspace is bounded whatever the number of sequences, and a sequence's result does not depend on it."""
    layer = Layer([200] + [1] * 40 + [70], 8, 8, 128, 128, 4, -1.0, seed=5)
    whole = layer.run(True)
    f = F()
    monkeypatch.setattr(f, "DELTA_WORKSPACE_BYTES", 5 * 8 * 4 * f.library().gk_delta_channel_work(128))
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    sizes, empty = [], torch.empty
    monkeypatch.setattr(torch, "empty", lambda shape, **kw: sizes.append(4 * shape[0]) or empty(shape, **kw) if len(shape) == 1 else empty(shape, **kw))
    grouped = layer.run(True)
    assert sizes and max(sizes) <= f.DELTA_WORKSPACE_BYTES
    assert all(torch.equal(a, b) for a, b in zip(whole, grouped))


def test_a_long_run_beside_many_single_tokens_goes_token_by_token(monkeypatch):
    from gtar_kimik3_public_b200.engine.step import SequenceStep, plan_step
    from gtar_kimik3_public_b200.parts.base import build_part

    part = build_part("mixer", "channel_delta", hidden_size=256, n_heads=2, n_kv_heads=2, key_dim=128, value_dim=128, conv_taps=4, norm_eps=EPS)
    b = lambda *shape: rand(*shape, seed=sum(shape), scale=0.05).to(torch.bfloat16).to(DEV)
    wide = 256
    part.load({"q": b(wide, 256), "k": b(wide, 256), "v": b(wide, 256), "q.conv": b(wide, 4), "k.conv": b(wide, 4), "v.conv": b(wide, 4), "b": b(2, 256),
               "A_log": b(2), "norm": b(128), "a1": b(64, 256), "a2": b(wide, 64), "dt_bias": b(wide), "g1": b(64, 256), "g2": b(wide, 64), "o": b(256, wide)})
    taken, chunks = [], F().delta_channel
    monkeypatch.setattr(F(), "delta_channel", lambda *a: taken.append(1) or chunks(*a))
    for counts, want in (([512], 1), ([512] + [1] * 127, 0), ([100, 100], 0)):
        taken.clear()
        cache = tuple(torch.zeros((len(counts), *r.shape), dtype=r.dtype, device=DEV) for r in part.cache_request())
        ctx = plan_step([SequenceStep(i, 0, [0] * c, []) for i, c in enumerate(counts)], torch.bfloat16, torch.device(DEV), 1)
        part.forward(b(sum(counts), 256), ctx, cache)
        assert len(taken) == want, counts
