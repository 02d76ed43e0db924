"""The recurrences with all chunks side by side, alone, against the formulas in 64 bits; the kernels that walk the same chunks one by one
say what 32 bits give in chunks of 32 (running sums of logarithms: where a decay is strong these differ from the token-by-token rule)."""
import pytest
import torch

from test_kernels_gpu import DEV

pytestmark = pytest.mark.gpu


def _slots(lens, floats, seed):
    g = torch.Generator().manual_seed(seed)
    slots = torch.randperm(len(lens) + 2, generator=g)[:len(lens)].to(torch.int32)
    start = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32)
    return g, slots, start, torch.randn(len(lens) + 2, floats + 8, generator=g) * 0.3


def _delta(qkv, bg, state, lens, slots, H, G, d, e):
    out, after, t = torch.zeros(qkv.shape[0], H * e, dtype=torch.float64), state.double().clone(), 0
    for s, n in enumerate(lens):
        S = after[slots[s], :H * e * d].view(H, e, d).clone()
        for _ in range(n):
            row = qkv[t].double()
            q, k = (row[i * G * d:(i + 1) * G * d].view(G, d).repeat_interleave(H // G, 0) for i in (0, 1))
            v = row[2 * G * d:].view(H, e)
            S = S * torch.exp(bg[t, H:].double()).view(H, 1, 1)
            u = bg[t, :H].double().view(H, 1) * (v - (S @ k.unsqueeze(2)).squeeze(2))
            S = S + u.unsqueeze(2) * k.unsqueeze(1)
            out[t] = (S @ q.unsqueeze(2)).reshape(-1)
            t += 1
        after[slots[s], :H * e * d] = S.reshape(-1)
    return out, after


def _errors(got, want):
    return [((a.double().cpu() - b).abs().max() / b.abs().max()).item() for a, b in zip(got, want)]


@pytest.mark.parametrize("H,G,d,e,lens", [(2, 1, 64, 64, [100, 3, 32, 33]), (3, 3, 16, 24, [31, 65, 1]), (1, 1, 40, 130, [96, 257]),
                                          (4, 2, 64, 64, [300])])
@pytest.mark.parametrize("fade", ["slow", "fast", "none"])
def test_delta_rule(H, G, d, e, lens, fade):
    """Chunk edges (31, 32, 33, 65 tokens), sizes that are no multiple of a tile, states that begin somewhere; requests of fewer
    than 32 tokens are left to the other kernel, and so is what lies behind a slot's state."""
    from sandyrt_b200.csrc import ops

    g, slots, start, state = _slots(lens, H * e * d, seed=d + e)
    T = sum(lens)
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)
    q, k = unit(torch.randn(T, G, d, generator=g)) * d ** -0.5, unit(torch.randn(T, G, d, generator=g))
    qkv = torch.cat([q.reshape(T, -1), k.reshape(T, -1), torch.randn(T, H * e, generator=g)], 1)
    rate = {"slow": 0.05, "fast": 40.0, "none": 0.0}[fade]
    bg = torch.cat([torch.rand(T, H, generator=g), -rate * torch.rand(T, H, generator=g)], 1)
    want = _delta(qkv, bg, state, lens, slots, H, G, d, e)
    errors = {}
    for form, long_from in (("walk", 32), ("chunks", 32)):
        st, out = state.to(DEV), torch.full((T, H * e), float("nan"), device=DEV)
        args = (qkv.to(DEV), bg.to(DEV), st, start.to(DEV), slots.to(DEV), out)
        kw = dict(n_heads=H, n_qk_heads=G, qk_dim=d, v_dim=e, long_from=long_from)
        ops.delta_scan(*args, **kw)
        ops.delta_scan(*args, **kw, max_q_len=max(lens), form=form)
        assert torch.equal(st[:, H * e * d:].cpu(), state[:, H * e * d:])
        errors[form] = _errors((out, st), want)
    # sums of up to 64 + 32 products instead of 64, and two products with A in place of one: twice the rounding
    for a, b in zip(errors["chunks"], errors["walk"]):
        assert a < 2 * b + 1e-6, errors


@pytest.mark.parametrize("keys", ["apart", "alike"])
@pytest.mark.parametrize("strength", [1.0, 0.05])
@pytest.mark.parametrize("rate", [0.0, 0.01, 0.3])
def test_delta_rule_is_no_less_precise_than_the_walk(keys, strength, rate):
    """The error of the state and of the read-outs (2-norm, against 64 bits) over 8 chunks of 6 heads from an empty state and from
    a large one.  Both forms round 24 k sums of the same size in another order: beside the walk's it may come out a tenth larger by chance."""
    from sandyrt_b200.csrc import ops

    T, H, d = 256, 6, 64
    g = torch.Generator().manual_seed(int(100 * strength + 1000 * rate))
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)
    mean = torch.randn(1, H, d, generator=g) if keys == "alike" else torch.zeros(1, H, d)
    noise = 0.05 if keys == "alike" else 1.0
    q, k = unit(torch.randn(T, H, d, generator=g)) * d ** -0.5, unit(mean + noise * torch.randn(T, H, d, generator=g))
    qkv = torch.cat([q.reshape(T, -1), k.reshape(T, -1), torch.randn(T, H * d, generator=g)], 1)
    bg = torch.cat([strength * torch.rand(T, H, generator=g), -rate * torch.rand(T, H, generator=g)], 1)
    start, slots = torch.tensor([0, T], dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    for size in (0.0, 3.0):
        state = size * torch.randn(1, H * d * d, generator=g)
        want = _delta(qkv, bg, state, [T], slots.cpu(), H, H, d, d)
        errors = {}
        for form in ("walk", "chunks"):
            st, out = state.to(DEV), torch.empty(T, H * d, device=DEV)
            ops.delta_scan(qkv.to(DEV), bg.to(DEV), st, start, slots, out, n_heads=H, n_qk_heads=H, qk_dim=d, v_dim=d, long_from=1,
                           max_q_len=T, form=form)
            errors[form] = [((a.double().cpu() - b).norm() / b.norm()).item() for a, b in zip((out, st), want)]
        assert all(a < 1.1 * b for a, b in zip(errors["chunks"], errors["walk"])), errors


def _memory(q, k, v, li, lf, state, lens, slots, H, d, e):
    Z = (e + 15) // 16
    out, after, t = torch.zeros(q.shape[0], H * e, dtype=torch.float64), state.double().clone(), 0
    a, b = H * e * d, H * e * d + H * Z * d
    for s, n in enumerate(lens):
        S = after[slots[s], :a].view(H, e, d).clone()
        nn = after[slots[s], a:b].view(H, Z, d)[:, 0].clone()
        m = after[slots[s], b:b + H * Z].view(H, Z)[:, 0].clone()
        for _ in range(n):
            new = torch.maximum(lf[t] + m, li[t])
            x, y, m = torch.exp(lf[t] + m - new), torch.exp(li[t] - new), new
            S = x.view(H, 1, 1) * S + y.view(H, 1, 1) * v[t].unsqueeze(2) * k[t].unsqueeze(1)
            nn = x.view(H, 1) * nn + y.view(H, 1) * k[t]
            den = torch.maximum((nn * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
            out[t] = ((S @ q[t].unsqueeze(2)).squeeze(2) / den.unsqueeze(1)).reshape(-1)
            t += 1
        after[slots[s], :a] = S.reshape(-1)
        after[slots[s], a:b] = nn.unsqueeze(1).expand(H, Z, d).reshape(-1)
        after[slots[s], b:b + H * Z] = m.unsqueeze(1).expand(H, Z).reshape(-1)
    return out, after


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,d,e,lens", [(2, 64, 128, [100, 3, 32, 33]), (3, 16, 20, [31, 65, 1]), (1, 40, 130, [96, 257]), (2, 64, 64, [600])])
@pytest.mark.parametrize("bias", [(0.0, 4.0), (6.0, -6.0), (-8.0, 8.0)])
def test_matrix_memory(dtype, H, d, e, lens, bias):
    """As above; gates that keep, that forget at once, and that let little in (the denominator's exp(-m) then decides)."""
    from sandyrt_b200.csrc import ops

    Z, cap, scale = (e + 15) // 16, 12.0, d ** -0.5
    g, slots, start, state = _slots(lens, H * e * d + H * Z * d + H * Z, seed=d + e)
    a, b = H * e * d, H * e * d + H * Z * d
    state[:, a:b] = state[:, a:b].view(-1, H, Z, d)[:, :, :1].expand(-1, H, Z, d).reshape(-1, H * Z * d)
    state[:, b:b + H * Z] = state[:, b:b + H * Z].view(-1, H, Z)[:, :, :1].expand(-1, H, Z).reshape(-1, H * Z)
    T = sum(lens)
    proj = torch.randn(T, H * (2 * d + e) + 5, generator=g).to(dtype)
    gates, gb = torch.randn(T, 2 * H + 3, generator=g), torch.cat([torch.full((H,), bias[0]), torch.full((H,), bias[1])])
    q, k = (proj[:, i * H * d:(i + 1) * H * d].double().view(T, H, d) for i in (0, 1))
    v = proj[:, 2 * H * d:2 * H * d + H * e].double().view(T, H, e)
    z = cap * torch.tanh((gates[:, :2 * H].double() + gb.double()) / cap)
    want = _memory(q * scale, k, v, z[:, :H], torch.nn.functional.logsigmoid(z[:, H:]), state, lens, slots, H, d, e)
    errors = {}
    for form, long_from in (("walk", 32), ("chunks", 32)):
        st, out = state.to(DEV), torch.full((T, H * e), float("nan"), device=DEV)
        args = (proj.to(DEV), 0, H * d, 2 * H * d, gates.to(DEV), gb.to(DEV), st, start.to(DEV), slots.to(DEV), out)
        kw = dict(cap=cap, q_scale=scale, n_heads=H, qk_dim=d, v_dim=e, long_from=long_from)
        ops.mlstm_scan(*args, **kw)
        ops.mlstm_scan(*args, **kw, max_q_len=max(lens), form=form)
        assert torch.equal(st[:, b + H * Z:].cpu(), state[:, b + H * Z:])
        rows = (out.double().cpu() - want[0]).view(T, H, e).norm(dim=-1) / (1e-3 + want[0].view(T, H, e).norm(dim=-1))
        errors[form] = [rows.max().item(), _errors((st,), want[1:])[0]]
    # a read-out is divided by a sum that may nearly cancel: what 32 bits give there is what the other kernel gives, twice that allowed
    for a, b in zip(errors["chunks"], errors["walk"]):
        assert a < 2 * b + 2e-6, errors


@pytest.mark.parametrize("kind", ["delta", "memory"])
def test_a_value_that_is_not_finite_does_not_reach_earlier_tokens(kind):
    from sandyrt_b200.csrc import ops

    T, d, e, bad = 100, 64, 64, 41
    g = torch.Generator().manual_seed(1)
    proj = torch.randn(T, 2 * d + e, generator=g) * 0.1
    proj[bad, 2 * d + 3] = float("nan")
    proj[bad, d + 5] = float("inf")
    state, out = torch.zeros(1, 8192, device=DEV), torch.zeros(T, e, device=DEV)
    start, slots = torch.tensor([0, T], dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    gates = torch.cat([torch.rand(T, 1, generator=g), -0.1 * torch.rand(T, 1, generator=g)], 1).to(DEV)
    if kind == "delta":
        ops.delta_scan(proj.to(DEV), gates, state, start, slots, out, n_heads=1, n_qk_heads=1, qk_dim=d, v_dim=e, long_from=1, max_q_len=T, form="chunks")
    else:
        ops.mlstm_scan(proj.to(DEV), 0, d, 2 * d, gates, torch.zeros(2, device=DEV), state, start, slots, out, cap=12.0, q_scale=0.125,
                       n_heads=1, qk_dim=d, v_dim=e, long_from=1, max_q_len=T, form="chunks")
    assert torch.isfinite(out[:bad]).all() and not torch.isfinite(out[bad]).all()
