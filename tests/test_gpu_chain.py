"""jb200_forward_layers (whole layers in one native call) against the kernel-by-kernel path, and the loss kernel against
torch, at the sizes where they can go wrong."""
import copy
import io

import pytest
import torch

from jarvis_b200 import _lib, modules as jm, ops

pytestmark = pytest.mark.gpu


def _model(layers=3):
    torch.manual_seed(12)
    return jm.ternary_init_(jm.Jarvis(vocab_size=320, d_model=128, n_layers=layers, n_heads=2, max_seq_len=640)).cuda().eval()


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30))


# All forms of a stage give the same bits: every product is one chain over K in steps of 16, and the kernels for few tokens
# keep the order of the sums and the roundings of those they stand for.  So a token's experts do not depend on how many
# others share its call, and the two paths are compared with torch.equal.  Only l_balance has another order of roundings
# (f64 throughout, rounded to f32 once: one ulp).
ULP = 2.0 ** -23


@pytest.mark.parametrize("B,T", [(1, 1), (5, 1), (1, 2), (3, 9), (2, 64), (1, 129), (4, 256), (2, 600)])
def test_chain_matches_the_kernel_by_kernel_path(B, T):
    model = _model()
    gen = torch.Generator(device="cuda").manual_seed(B * 1000 + T)
    idx = torch.randint(0, 320, (B, T), generator=gen, device="cuda")
    pos = torch.randint(0, 20, (B,), generator=gen, device="cuda", dtype=torch.int32)
    state = {"h": [torch.randn(B, 128, generator=gen, device="cuda") for _ in range(3)],
             "S": [torch.randn(B, 2, 64, 64, generator=gen, device="cuda") for _ in range(3)]}
    got = {}
    for chain in (False, True):
        model.use_chain = chain
        st = {k: [t.clone() for t in v] for k, v in state.items()}
        logits, new = model.step(idx, pos, st, max_position=640)
        into, same = model.step(idx, pos, st, max_position=640, inplace=True)
        assert all(a is b for a, b in zip(same["S"] + same["h"], st["S"] + st["h"])) or not chain
        model.reset_state()
        first, loss = model(idx, targets=idx, persist_state=True)
        second, _ = model(idx, persist_state=True)
        assert model._token_pos == 2 * T
        aux = torch.stack(model.last_aux)                          # a list on either path
        idxs = [b.moe.last_routing[0].clone() for b in model.blocks]
        got[chain] = [logits, into, torch.stack(new["h"]), torch.stack(new["S"]), torch.stack(same["h"]), torch.stack(same["S"]),
                      first, second, torch.stack(idxs), aux[:, 1:], aux[:, 0], loss.reshape(1)]
    assert _lib.device_status() == 0
    for a, b in zip(got[True][:-2], got[False][:-2]):
        assert torch.equal(a, b)
    assert rel(got[True][-2], got[False][-2]) <= 2 * ULP
    # the penalty is made of the same two scalars by f32 operations on either path (four roundings), three layers of it
    assert rel(got[True][-1], got[False][-1]) <= 16 * ULP


def test_chain_follows_changed_parameters_and_modules():
    model = _model(2)
    idx = torch.arange(24, device="cuda").view(1, 24)
    a = model(idx)[0].clone()
    with torch.no_grad():
        model.blocks[1].attn.q_proj.weight.neg_()
    b = model(idx)[0].clone()
    assert not torch.equal(a, b)
    with torch.no_grad():
        model.blocks[1].attn.q_proj.weight.neg_()
    assert torch.equal(model(idx)[0], a)
    model.blocks[0].moe.w1[2] = jm.ternary_init_(jm.TernaryLinear(128, 256)).cuda()
    model.use_chain = False
    want = model(idx)[0].clone()
    model.use_chain = True
    assert torch.equal(model(idx)[0], want) and not torch.equal(want, a)


@pytest.mark.parametrize("rows,V,ld", [(1, 1, 8), (3, 7, 8), (5, 8, 128), (37, 4095, 4096), (9, 4101, 4224), (300, 50257, 50304)])
def test_cross_entropy_matches_torch(rows, V, ld):
    gen = torch.Generator(device="cuda").manual_seed(V)
    buf = (torch.randn(rows, ld, generator=gen, device="cuda") * 5).bfloat16()
    logits = buf[:, :V].view(1, rows, V) if V == ld else buf.view(1, rows, ld)[..., :V]
    y = torch.randint(0, V, (1, rows), generator=gen, device="cuda")
    if rows > 2:
        y[0, 1] = -100
    aux, refl = torch.rand(4, 3, generator=gen, device="cuda"), torch.rand(4, generator=gen, device="cuda")
    got = ops.cross_entropy(logits, y, aux, refl)
    want = torch.nn.functional.cross_entropy(logits[0].double(), y[0]) + aux[:, 0].double().sum() + refl.double().sum()
    # f32 exponentials (2 ulp each) and an f32 logarithm and subtraction at magnitude |max| + log V <= 32: 32 * 2^-23 * 4
    assert abs(float(got) - float(want)) < 2e-5 * max(1.0, abs(float(want)))
    assert _lib.device_status() == 0


@pytest.mark.parametrize("V", [1, 7, 4101, 50257])
def test_cross_entropy_of_values_that_are_not_finite(V):
    """A NaN anywhere makes the loss NaN, also where a thread has met nothing else yet; -inf logits count as nothing."""
    gen = torch.Generator(device="cuda").manual_seed(V)
    clean = (torch.randn(1, 2, (V + 7) // 8 * 8, generator=gen, device="cuda") * 5).bfloat16()
    y = torch.full((1, 2), V - 1, device="cuda", dtype=torch.int64)
    none = torch.zeros(1, 3, device="cuda"), torch.zeros(1, device="cuda")
    nan, inf = float("nan"), float("inf")
    for value, spans in ((nan, [(0, 1), (0, 8), (max(V - 8, 0), V), (0, V)]), (-inf, [(0, 8), (0, max(V - 1, 0)), (0, V)]), (inf, [(0, 1)])):
        for a, b in spans:
            buf = clean.clone()
            buf[0, 1, a:min(b, V)] = value
            logits = buf[..., :V]
            got, want = float(ops.cross_entropy(logits, y, *none)), float(torch.nn.functional.cross_entropy(logits[0].double(), y[0]))
            assert (got != got) == (want != want), (value, a, b, got, want)
            assert want != want or got == want or abs(got - want) < 2e-5 * max(1.0, abs(want))
    mixed = clean.clone()
    mixed[0, 0, :8] = -inf
    mixed[0, 0, 0] = nan                                            # NaN among -inf in one thread's first values
    assert bool(torch.isnan(ops.cross_entropy(mixed[..., :V], y, *none)))


@pytest.mark.parametrize("B,T", [(1, 1), (4, 1), (5, 1), (8, 1), (9, 1), (16, 1), (17, 1), (33, 1), (64, 1), (65, 1), (128, 1),
                                 (129, 1), (1, 2), (3, 3), (1, 16), (2, 20), (1, 64), (1, 65), (2, 64), (1, 128), (1, 129),
                                 (1, 256), (1, 257), (257, 1), (1, 640), (1, 960), (1, 961), (1, 40), (1, 41)])
def test_chain_at_full_width_around_the_edges_of_its_small_kernels(B, T):
    """d_model 1024: the kernels for few tokens (GEMM forms up to 16, up to 960 and beyond, router up to 256, row cluster up to
    128 steps or 192 tokens of prompts) against the kernel-by-kernel path; mixed routing, carried state, one expert without tokens
    at the smallest sizes."""
    from jarvis_b200 import chain
    torch.manual_seed(7)
    blk = jm.ternary_init_(jm.JarvisBlock(1024, 16, max_seq_len=1024)).cuda().eval()
    gen = torch.Generator(device="cuda").manual_seed(B * 1000 + T)
    x = torch.randn(B * T, 1024, generator=gen, device="cuda")
    h = torch.randn(B, 1024, generator=gen, device="cuda")
    S = torch.randn(B, 16, 64, 64, generator=gen, device="cuda")
    norm = (torch.rand(1024, generator=gen, device="cuda") + 0.5, 1e-6)
    xa, xb = x.clone(), x.clone()
    acc, hist = torch.zeros(6, dtype=torch.float64, device="cuda"), torch.zeros(4, dtype=torch.int32, device="cuda")
    ha, sa, Sa = blk.forward_rows(xa, B, T, h, 5, S, want_attn_state=True, scratch=(acc, hist, torch.zeros(3, device="cuda")))
    idx_a, gates_a, _ = blk.moe.last_routing
    r = chain.run(chain.table_of(blk, [blk]), xb, B, T, start_pos=5, h_in=[h], s_in=[S], want_state=True, final_norm=norm)
    assert torch.equal(xb, xa) and torch.equal(r.h[0], ha) and torch.equal(r.S[0], Sa)
    assert torch.equal(r.hidden, ops.rmsnorm(xb, *norm))
    assert torch.equal(r.scalars[0][1:], sa[1:]) and rel(r.scalars[0][:1], sa[:1]) <= 2 * ULP
    idx, gates, (counts, offsets, scatter, gather, gate_idx) = blk.moe.last_routing
    assert torch.equal(idx, idx_a) and torch.equal(gates, gates_a)
    want = ops.moe_metadata(idx.contiguous(), 4)
    for got, ref in zip((counts, offsets, scatter, gather, gate_idx), want):
        assert torch.equal(got, ref)                                          # dispatch order: bit-exact
    assert int(torch.bincount(idx.flatten(), minlength=4).sum()) == 2 * B * T
    assert _lib.device_status() == 0


@pytest.mark.parametrize("B,T", [(1, 48), (1, 80), (1, 100), (100, 1), (160, 1), (161, 1), (192, 1), (300, 1), (1, 160), (1, 161), (1, 448), (1, 449)])
def test_chain_around_the_edges_of_its_gemm_tiles(B, T):
    """Products in tiles of 64 and of 128 out-features, one and several token tiles, all rows for every expert and dispatched ones."""
    test_chain_at_full_width_around_the_edges_of_its_small_kernels(B, T)


@pytest.mark.parametrize("B,T", [(1, 192), (1, 193), (2, 96), (64, 3), (21, 9), (11, 17), (10, 19), (5, 33), (24, 8)])
def test_chain_around_the_edges_of_its_tail_cluster(B, T):
    """Runs of up to 8, 16 and more tokens, more of them than warps, tokens for every warp of a CTA and for few."""
    test_chain_at_full_width_around_the_edges_of_its_small_kernels(B, T)


@pytest.mark.parametrize("skew", [0.5, 4.0])
@pytest.mark.parametrize("T", [17, 64, 129, 256, 640, 960])
def test_chain_with_uneven_experts(T, skew):
    """Tokens that lean one way go to the same experts: token tiles beyond an even share, groups without rows."""
    from jarvis_b200 import chain
    torch.manual_seed(7)
    blk = jm.ternary_init_(jm.JarvisBlock(1024, 16, max_seq_len=2048)).cuda().eval()
    gen = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, 1024, generator=gen, device="cuda") + skew * torch.randn(1, 1024, generator=gen, device="cuda")
    norm = (torch.ones(1024, device="cuda"), 1e-6)
    xa, xb = x.clone(), x.clone()
    acc, hist = torch.zeros(6, dtype=torch.float64, device="cuda"), torch.zeros(4, dtype=torch.int32, device="cuda")
    blk.forward_rows(xa, 1, T, None, 0, None, scratch=(acc, hist, torch.zeros(3, device="cuda")))
    chain.run(chain.table_of(blk, [blk]), xb, 1, T, start_pos=0, final_norm=norm)
    assert torch.equal(xb, xa)
    counts = torch.bincount(blk.moe.last_routing[0].flatten(), minlength=4)
    assert int(counts.max()) > T * (5 if skew < 1 else 8) // 10, counts
    assert _lib.device_status() == 0


@pytest.mark.parametrize("B,T,D", [(1, 129, 1024), (1, 256, 64), (3, 777, 1024), (2, 1023, 200), (9, 300, 1024), (10, 300, 1024)])
def test_residual_scan_with_its_tiles_side_by_side(B, T, D):
    """The fused scan of sequences of two to eight tiles against the recurrence in f64; the membrane is updated in place."""
    gen = torch.Generator(device="cuda").manual_seed(T)
    m = torch.randn(B, T, D, generator=gen, device="cuda").bfloat16()
    h0 = torch.randn(B, D, generator=gen, device="cuda")
    x = torch.randn(B, T, D, generator=gen, device="cuda")
    alpha, h, want = torch.tensor([0.97], device="cuda"), h0.double(), x.double()
    a = float(alpha)
    for t in range(T):
        h = a * h + (1.0 - a) * m[:, t].double()
        want[:, t] += h
    got, last = x.clone(), h0.clone()
    ops.lsf_scan(m, alpha_scalar=alpha, h0=last, resid=got, want_out=False, last_out=last)
    # every step rounds values below 5 three times (2^-24 of them), and errors fade by alpha: 3 * 5 * 2^-24 / 0.03 = 3e-5
    assert float((got.double() - want).abs().max()) < 3e-5 and float((last.double() - h).abs().max()) < 3e-5
    assert _lib.device_status() == 0


@pytest.mark.parametrize("E", [1, 4, 16])
@pytest.mark.parametrize("N", [1, 17, 511, 512, 513, 1000, 1024, 1025])
def test_dispatch_metadata_around_the_one_cta_form(N, E):
    """One round, two rounds, three kernels; expected maps from a stable sort on the host."""
    idx = torch.randint(0, E, (N, 2), generator=torch.Generator().manual_seed(N))
    idx[N // 2:] = E - 1                                                       # uneven
    flat = idx.flatten()
    order = torch.argsort(flat, stable=True)
    counts = torch.bincount(flat, minlength=E)
    slots = torch.empty(2 * N, dtype=torch.long)
    slots[order] = torch.arange(2 * N)
    offsets = torch.cat([torch.zeros(1, dtype=torch.long), counts.cumsum(0)])
    for got, want in zip(ops.moe_metadata(idx.cuda(), E), (counts, offsets, slots, order // 2, order % 2)):
        assert torch.equal(got.cpu().flatten().long(), want)


@pytest.mark.parametrize("T", [1, 5])
def test_carried_state_that_does_not_fit_is_refused(T):
    """Wrong batch, host memory, too few layers, a membrane that cannot be updated in place: an error before any launch."""
    model = _model(2)
    idx = torch.zeros((3, T), dtype=torch.int64, device="cuda")

    def state(B=3, n=2, dev="cuda", dtype=torch.float32):
        return {"h": [torch.zeros(B, 128, device=dev, dtype=dtype) for _ in range(n)],
                "S": [torch.zeros(B, 2, 64, 64, device=dev) for _ in range(n)]}
    model(idx)
    launches = _lib.kernel_launches()
    for bad in (state(B=2), state(n=1), state(dev="cpu"), {"h": state()["h"], "S": state(B=2)["S"]}):
        for inplace in (False, True):
            with pytest.raises((RuntimeError, IndexError)):
                model.step(idx, 0, bad, max_position=16, inplace=inplace)
    with pytest.raises(RuntimeError):
        model.step(idx, torch.zeros(2, dtype=torch.int32, device="cuda"), state(), max_position=16)
    strided = {"h": [torch.zeros(128, 3, device="cuda").t() for _ in range(2)], "S": state()["S"]}
    with pytest.raises(RuntimeError):
        model.step(idx, 0, strided, max_position=16, inplace=True)
    if T > 1:
        with pytest.raises(RuntimeError):
            model.step(idx, 0, state(dtype=torch.bfloat16), max_position=16, inplace=True)
    assert _lib.kernel_launches() == launches
    model.step(idx, 0, strided, max_position=16)                   # converted where nothing has to alias
    st = state()
    st["S"][1] = st["h"][0] = None                                 # layers without a state get a new one, the others are updated
    _, new = model.step(idx, 0, st, max_position=16, inplace=True)
    assert new["S"][0] is st["S"][0] and new["h"][1] is st["h"][1] and float(st["S"][0].abs().sum()) > 0
    assert new["S"][1] is not None and new["h"][0].shape == (3, 128)
    with pytest.raises(RuntimeError):
        model.blocks[0].forward_rows(torch.zeros(3 * T + 1, 128, device="cuda"), 3, T)
    assert _lib.device_status() == 0


def test_weights_left_on_the_host_are_refused():
    model = _model(1)
    idx = torch.zeros((2, 3), dtype=torch.int64, device="cuda")
    model(idx)
    for name in ("tok_emb", "final_norm"):
        getattr(model, name).cpu()
        with pytest.raises(RuntimeError):
            model(idx)
        getattr(model, name).cuda()
    model.blocks[0].moe.w2 = torch.nn.ModuleList(jm.ternary_init_(jm.TernaryLinear(384, 128)).cuda() for _ in range(4))
    with pytest.raises(RuntimeError):
        model(idx)
    assert _lib.device_status() == 0


@pytest.mark.parametrize("B,T", [(3, 1), (130, 1), (2, 2), (2, 9), (1, 64), (1, 200), (2, 300)])
@pytest.mark.parametrize("inplace", [False, True])
def test_membranes_on_an_8_byte_boundary(B, T, inplace):
    """The LSF scan takes them; the fused tails, which read 16 bytes at a time, leave them to it.  Same bits."""
    torch.manual_seed(3)
    blk = jm.ternary_init_(jm.JarvisBlock(256, 4, max_seq_len=512)).cuda().eval()
    gen = torch.Generator(device="cuda").manual_seed(B * 1000 + T)
    x, h = torch.randn(B * T, 256, generator=gen, device="cuda"), torch.randn(B, 256, generator=gen, device="cuda")
    odd = torch.empty(B * 256 + 2, device="cuda")[2:].view(B, 256).copy_(h)
    assert odd.data_ptr() % 16 == 8
    xa, xb, aligned = x.clone(), x.clone(), h.clone()
    ha = blk.forward_rows(xa, B, T, aligned, inplace_state=inplace)[0]
    hb = blk.forward_rows(xb, B, T, odd, inplace_state=inplace)[0]
    assert torch.equal(xa, xb) and torch.equal(ha, hb) and (hb is odd) == inplace
    assert _lib.device_status() == 0


@pytest.mark.parametrize("B,T,mult", [(1, 1, 8), (8, 1, 7), (9, 1, 5), (2, 8, 5), (16, 1, 4)])
def test_few_tokens_with_wide_experts(B, T, mult):
    """Expert widths whose rows do not fit the shared memory of the kernel for a few tokens (from 4800 at 9 to 16 tokens, 7200
    below), and the widest that does."""
    torch.manual_seed(5)
    blk = jm.JarvisBlock(1024, 16, max_seq_len=64)
    blk.moe = jm.SparseMoELayer(1024, hidden_mult=mult)
    blk = jm.ternary_init_(blk).cuda().eval()
    x = torch.randn(B * T, 1024, generator=torch.Generator(device="cuda").manual_seed(B), device="cuda")
    xa, xb = x.clone(), x.clone()
    blk.forward_rows(xa, B, T, scratch=(torch.zeros(6, dtype=torch.float64, device="cuda"),
                                        torch.zeros(4, dtype=torch.int32, device="cuda"), torch.zeros(3, device="cuda")))
    blk.forward_rows(xb, B, T)
    assert torch.equal(xa, xb)
    assert _lib.device_status() == 0


def test_overrides_and_penalties_of_the_callers_own_are_honoured():
    model = _model(2)
    idx = torch.arange(24, device="cuda").view(1, 24)
    base, loss = model(idx, targets=idx)
    calls = []
    moe, plain = model.blocks[1].moe, model.blocks[1].moe.run_rows
    moe.run_rows = lambda *a, **k: (calls.append(1), plain(*a, **k))[1]           # after the table was made
    assert torch.equal(model(idx)[0], base) and calls == [1]
    model.blocks[1](torch.randn(1, 4, 128, device="cuda"))
    assert calls == [1, 1]
    del moe.run_rows
    assert torch.equal(model(idx)[0], base) and calls == [1, 1]
    model.step(idx)

    class Attn(jm.AssociativeLinearAttention):
        def scan_rows(self, *a, **k):
            o, s = super().scan_rows(*a, **k)
            return torch.zeros_like(o), s
    stock, ours = model.blocks[0].attn, Attn(128, 2, max_seq_len=640).cuda().eval()
    ours.load_state_dict(stock.state_dict())
    model.blocks[0].attn = ours
    assert not torch.equal(model(idx)[0], base) and not torch.equal(model.step(idx)[0], base)
    model.blocks[0].attn = stock
    assert torch.equal(model(idx)[0], base)

    # the penalty: its running mean moves in training, hooks see the call, and it may return a number
    refl = model.blocks[0].reflect
    refl.train()
    before = refl.mu_t.clone()
    model(idx, targets=idx)
    assert not torch.equal(refl.mu_t, before)
    refl.eval().mu_t = before
    seen = []
    hook = refl.register_forward_hook(lambda m, args, out: seen.append(float(out)))
    got = model(idx, targets=idx)[1]
    hook.remove()
    assert len(seen) == 1 and abs(float(got) - float(loss)) < 1e-5 * abs(float(loss))
    zero = torch.nn.Module()
    zero.forward = lambda mean, var: 0.25
    model.blocks[0].reflect = zero
    shifted = model(idx, targets=idx)[1]
    assert abs(float(shifted) - (float(loss) - seen[0] + 0.25)) < 1e-5 * abs(float(shifted))
    assert _lib.device_status() == 0


def test_a_model_that_has_run_can_be_copied_and_saved():
    model = _model(2)
    idx = torch.arange(24, device="cuda").view(1, 24)
    want = model(idx)[0].clone()
    model.blocks[0](torch.randn(1, 4, 128, device="cuda"))
    buf = io.BytesIO()
    torch.save(model, buf)
    buf.seek(0)
    for twin in (copy.deepcopy(model), torch.load(buf, weights_only=False)):
        assert torch.equal(twin(idx)[0], want)
        with torch.no_grad():
            twin.blocks[0].attn.gamma_raw.neg_()
        assert not torch.equal(twin(idx)[0], want) and torch.equal(model(idx)[0], want)


def test_a_captured_step_outlives_the_layer_table():
    """An in-place edit of a norm weight makes the next eager call build a new table; what the graph reads must stay."""
    model = _model(2)
    gen = torch.Generator(device="cuda").manual_seed(3)
    idx = torch.randint(0, 320, (5, 1), generator=gen, device="cuda")
    state = {"h": [torch.randn(5, 128, generator=gen, device="cuda") for _ in range(2)],
             "S": [torch.randn(5, 2, 64, 64, generator=gen, device="cuda") for _ in range(2)]}
    pos = torch.full((5,), 3, dtype=torch.int32, device="cuda")
    session = jm.DecodeSession(model, {k: [s.clone() for s in v] for k, v in state.items()}, pos, 640).capture()
    gammas = [b.attn.decays() for b in model.blocks]
    with torch.no_grad():
        model.blocks[0].norm1.weight.mul_(1.5)
    model(idx)
    assert all(b.attn.decays() is g for b, g in zip(model.blocks, gammas))
    junk = [torch.full((2,), 0.01, device="cuda") for _ in range(2000)]             # freed blocks of that size would be taken
    session.load_state(state, pos)
    got = session.step(idx).clone()
    want, _ = model.step(idx, pos, state, max_position=640)
    assert torch.equal(got, want) and len(junk) == 2000
    assert _lib.device_status() == 0


@pytest.mark.parametrize("B", [1, 5, 13])
def test_a_captured_step_follows_edits_in_place(B):
    """Norms, router and var_scale are read from the parameters themselves, by the one-launch step as by the kernels."""
    torch.manual_seed(12)
    model = jm.ternary_init_(jm.Jarvis(vocab_size=320, d_model=1024, n_layers=2, n_heads=16, max_seq_len=64)).cuda().eval()
    gen = torch.Generator(device="cuda").manual_seed(3)
    idx = torch.randint(0, 320, (B, 1), generator=gen, device="cuda")
    state = {"h": [torch.randn(B, 1024, generator=gen, device="cuda") for _ in range(2)],
             "S": [torch.randn(B, 16, 64, 64, generator=gen, device="cuda") for _ in range(2)]}
    pos = torch.full((B,), 3, dtype=torch.int32, device="cuda")
    session = jm.DecodeSession(model, {k: [s.clone() for s in v] for k, v in state.items()}, pos, 64).capture()
    router, var_scale = model.blocks[0].moe.router.weight, model.blocks[1].liquid.var_scale
    edits = [lambda: None, lambda: model.blocks[0].norm2.weight.mul_(1.5), lambda: router.copy_(router.flip(0)), lambda: var_scale.add_(2.0)]
    seen = []
    for edit in edits:
        with torch.no_grad():
            edit()
        session.load_state(state, pos)
        seen.append(session.step(idx).clone())
        want, new = model.step(idx, pos, state, max_position=64)
        assert torch.equal(seen[-1], want)
        assert all(torch.equal(a, b) for a, b in zip(session.state["h"] + session.state["S"], new["h"] + new["S"]))
    assert not any(torch.equal(a, b) for a, b in zip(seen, seen[1:]))
    assert _lib.device_status() == 0


def test_a_captured_step_outlives_its_angle_tables():
    """A longer prompt makes the model's angle tables anew; the graph goes on with those it was captured with."""
    torch.manual_seed(12)
    model = jm.ternary_init_(jm.Jarvis(vocab_size=320, d_model=128, n_layers=2, n_heads=2, max_seq_len=256)).cuda().eval()
    idx = torch.arange(5, device="cuda").view(5, 1)
    state = {"h": [torch.ones(5, 128, device="cuda") for _ in range(2)],
             "S": [torch.ones(5, 2, 64, 64, device="cuda") for _ in range(2)]}
    pos = torch.full((5,), 200, dtype=torch.int32, device="cuda")
    want, _ = model.step(idx, pos, state, max_position=250)
    session = jm.DecodeSession(model, {k: [s.clone() for s in v] for k, v in state.items()}, pos, 250).capture()
    model(torch.zeros((1, 700), dtype=torch.int64, device="cuda"))
    junk = [torch.full((256, 32), 9.0, device="cuda") for _ in range(50)]
    session.load_state(state, pos)
    assert torch.equal(session.step(idx), want) and len(junk) == 50


@pytest.mark.parametrize("N", [3, 64, 65, 200])
def test_dispatch_maps_of_tokens_whose_router_is_nan(N):
    """A token without finite logits has no second expert (-1); the maps still hold every assignment, as the general sort's do."""
    torch.manual_seed(9)
    blk = jm.ternary_init_(jm.JarvisBlock(256, 4, max_seq_len=256)).cuda().eval()
    x = torch.randn(N, 256, device="cuda")
    x[N // 2] = float("nan")
    blk.forward_rows(x, 1, N)
    idx, _, got = blk.moe.last_routing
    assert int(idx.min()) == -1
    for a, b in zip(got, ops.moe_metadata(idx.contiguous(), 4)):
        assert torch.equal(a, b)
    assert _lib.device_status() == 0


@pytest.mark.parametrize("B,T,C", [(1, 1, 1024), (3, 1, 1024), (8, 1, 1024), (13, 1, 1024), (56, 1, 1024), (64, 1, 1024), (1, 3, 1024),
                                   (1, 16, 1024), (2, 20, 1024), (1, 64, 1024), (1, 65, 1024), (2, 150, 1024), (7, 1, 128), (2, 20, 128)])
def test_both_assignments_of_a_token_whose_router_is_nan_run(B, T, C):
    """Logits that overflow where everything else of the token is finite: its two assignments are expert 0's, as the maps say, in every
    form, and the other tokens of the call do not notice."""
    torch.manual_seed(9)
    model = jm.ternary_init_(jm.Jarvis(vocab_size=320, d_model=C, n_layers=2, n_heads=C // 64, max_seq_len=512)).cuda().eval()
    with torch.no_grad():
        model.tok_emb.weight[:, 0] = 0.0                           # token 7 alone has a channel that overflows in the first router
        model.tok_emb.weight[7, 0] = 5.0
        model.blocks[0].attn.out_proj.weight[0] = 0.0
        model.blocks[0].moe.router.weight[:, 0] = 3e38
    gen = torch.Generator(device="cuda").manual_seed(3)
    idx = torch.randint(8, 320, (B, T), generator=gen, device="cuda")
    idx.view(-1)[B * T // 2] = 7
    state = {"h": [torch.randn(B, C, generator=gen, device="cuda") for _ in range(2)],
             "S": [torch.randn(B, C // 64, 64, 64, generator=gen, device="cuda") for _ in range(2)]}
    pos = torch.full((B,), 3, dtype=torch.int32, device="cuda")
    got = []
    for model.use_chain in (False, True, True):                    # twice: the one-launch step lays its weights out first
        logits, st = model.step(idx, pos, state, max_position=512)
        ids, _, maps = model.blocks[0].moe.last_routing
        got.append([logits, torch.stack(st["h"]), torch.stack(st["S"]), ids, *maps])
    assert got[0][3].view(-1, 2)[B * T // 2].tolist() == [0, -1] and int((got[0][3] < 0).sum()) == 1
    assert all(bool(torch.isfinite(t).all()) for t in got[0][:3])
    for other in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0], other))
    assert _lib.device_status() == 0


@pytest.mark.parametrize("B,layers,states,skew", [(1, 3, True, 0.0), (1, 2, False, 0.0), (2, 34, True, 0.0), (3, 3, True, 3.0), (3, 2, False, 0.0),
                                                  (4, 3, True, 0.0), (7, 3, True, 3.0), (8, 3, True, 0.0), (13, 3, True, 3.0),
                                                  (15, 3, True, 0.0), (29, 2, True, 0.0), (49, 3, True, 3.0), (56, 3, True, 0.0),
                                                  (57, 2, True, 0.0), (5, 2, False, 0.0)])
def test_one_launch_step_against_the_kernels_it_stands_for(B, layers, states, skew, monkeypatch):
    """All layers of a single-token step in one launch, bit for bit: one and several clusters, one to eight sequences in each, no states,
    more layers than a launch takes, experts nobody wants (skew: most tokens go to two), states updated in place over several
    steps; beyond the last size the kernels themselves run on either side."""
    from jarvis_b200 import chain
    torch.manual_seed(B)
    model = jm.ternary_init_(jm.Jarvis(vocab_size=320, d_model=1024, n_layers=layers, n_heads=16, max_seq_len=64)).cuda().eval()
    with torch.no_grad():
        for b in model.blocks:
            b.moe.router.weight[:2] += skew * b.moe.router.weight[2:].abs().mean() * torch.sign(torch.randn(1024, device="cuda"))
    gen = torch.Generator(device="cuda").manual_seed(B)
    state = {"h": [torch.randn(B, 1024, generator=gen, device="cuda") for _ in range(layers)],
             "S": [torch.randn(B, 16, 64, 64, generator=gen, device="cuda") for _ in range(layers)]} if states else None
    pos = torch.randint(0, 20, (B,), generator=gen, device="cuda", dtype=torch.int32)
    idx = torch.randint(0, 320, (4, B, 1), generator=gen, device="cuda")
    _, first = model.step(idx[0], pos, None, max_position=64)             # weights are packed, on the next call laid out
    model.step(idx[0], pos, first, max_position=64)
    few = B <= min(56, _lib.load().jb200_step_max_sequences())
    got = {}
    for one_launch in (True, False):
        if not one_launch:
            monkeypatch.setattr(chain.LayerTable, "step_weights", lambda self, B: None)
        st = state and {k: [t.clone() for t in v] for k, v in state.items()}
        out, before = [], _lib.kernel_launches()
        for t in range(4):
            logits, st = model.step(idx[t], pos + t, st, max_position=64, inplace=st is not None)
            out += [logits, torch.stack([b.moe.last_routing[0] for b in model.blocks]), torch.stack([b.moe.last_routing[1] for b in model.blocks])]
            out += [torch.cat([m.flatten() for m in b.moe.last_routing[2]]) for b in model.blocks]
        got[one_launch] = out + st["h"] + st["S"], _lib.kernel_launches() - before
    assert all(torch.equal(a, b) for a, b in zip(got[True][0], got[False][0]))
    assert got[True][1] < got[False][1] if few else got[True][1] <= got[False][1]
    assert _lib.device_status() == 0


def test_states_that_overlap_go_kernel_by_kernel():
    """The one-launch step fetches states layers ahead: a state that another layer writes is left to the kernels, in their order."""
    torch.manual_seed(3)
    model = jm.ternary_init_(jm.Jarvis(vocab_size=320, d_model=1024, n_layers=2, n_heads=16, max_seq_len=64)).cuda().eval()
    idx = torch.tensor([[5], [9]], device="cuda")
    h, S = torch.randn(2, 1024, device="cuda"), torch.randn(2, 16, 64, 64, device="cuda")
    apart, shared = [{"h": [h.clone()] * 2, "S": [S.clone()] * 2} for _ in range(2)]
    model.use_chain = False
    want, _ = model.step(idx, 0, apart, max_position=64, inplace=True)
    model.use_chain = True
    got, _ = model.step(idx, 0, shared, max_position=64, inplace=True)
    assert torch.equal(got, want) and torch.equal(shared["S"][0], apart["S"][0]) and torch.equal(shared["h"][1], apart["h"][1])
    assert _lib.device_status() == 0


@pytest.mark.parametrize("E,C", [(4, 1024), (8, 136)])
@pytest.mark.parametrize("N", [1, 63, 64, 65, 257, 4095, 4097, 70000])
def test_dispatch_in_one_launch_against_metadata_and_gather(N, E, C):
    """Chunk edges, one to a thousand chunks, an expert nobody takes, assignments without an expert."""
    gen = torch.Generator(device="cuda").manual_seed(N)
    first = torch.randint(0, E - 1, (N,), generator=gen, device="cuda")
    idx = torch.stack([first, (first + torch.randint(1, E - 1, (N,), generator=gen, device="cuda")) % (E - 1)], 1)
    idx[N // 2, 1] = -1
    idx[N // 3] = 0
    x = torch.randn(N, C, generator=gen, device="cuda").bfloat16()
    got, rows = ops.moe_dispatch(x, idx, E)
    want = ops.moe_metadata(idx, E)
    assert all(torch.equal(a, b) for a, b in zip(got, want)) and torch.equal(rows, ops.dispatch_gather(x, want[3]))
    with pytest.raises(RuntimeError):
        ops.moe_dispatch(x, idx[:, :1].contiguous(), E)
    assert _lib.device_status() == 0


@pytest.mark.parametrize("E,C", [(4, 1024), (8, 136)])
@pytest.mark.parametrize("N", [1024, 1025, 16384, 16385, 262144, 262145])
def test_dispatch_around_the_sizes_of_its_one_launch_form(N, E, C):
    gen = torch.Generator(device="cuda").manual_seed(N)
    first = torch.randint(0, E, (N,), generator=gen, device="cuda")
    idx = torch.stack([first, (first + torch.randint(1, E, (N,), generator=gen, device="cuda")) % E], 1)
    idx[N // 2, 1] = -1
    x = torch.randn(N, C, generator=gen, device="cuda").bfloat16()
    got, rows = ops.moe_dispatch(x, idx, E)
    want = ops.moe_metadata(idx, E)
    assert all(torch.equal(a, b) for a, b in zip(got, want)) and torch.equal(rows, ops.dispatch_gather(x, want[3]))
    assert _lib.device_status() == 0


def _chain_against_kernels(C, E, mult, B, T):
    """One block with E experts of mult * C features, carried states: chain and kernel by kernel, rows, states, routes and maps."""
    from jarvis_b200 import chain
    torch.manual_seed(7)
    blk = jm.JarvisBlock(C, C // 64, num_experts=E, max_seq_len=256)
    blk.moe = jm.SparseMoELayer(C, num_experts=E, hidden_mult=mult)
    blk = jm.ternary_init_(blk).cuda().eval()
    gen = torch.Generator(device="cuda").manual_seed(B * 1000 + T)
    x, h = torch.randn(B * T, C, generator=gen, device="cuda"), torch.randn(B, C, generator=gen, device="cuda")
    S = torch.randn(B, C // 64, 64, 64, generator=gen, device="cuda")
    norm = (torch.rand(C, generator=gen, device="cuda") + 0.5, 1e-6)
    xa, xb = x.clone(), x.clone()
    acc, hist = torch.zeros(2 + E, dtype=torch.float64, device="cuda"), torch.zeros(E, dtype=torch.int32, device="cuda")
    ha, sa, Sa = blk.forward_rows(xa, B, T, h, 5, S, want_attn_state=True, scratch=(acc, hist, torch.zeros(3, device="cuda")))
    idx_a, gates_a, _ = blk.moe.last_routing
    r = chain.run(chain.table_of(blk, [blk]), xb, B, T, start_pos=5, h_in=[h], s_in=[S], want_state=True, final_norm=norm)
    idx, gates, maps = blk.moe.last_routing
    assert torch.equal(idx, idx_a) and torch.equal(gates, gates_a)
    assert all(torch.equal(a, b) for a, b in zip(maps, ops.moe_metadata(idx.contiguous(), E)))
    assert torch.equal(xb, xa) and torch.equal(r.h[0], ha) and torch.equal(r.S[0], Sa)
    assert torch.equal(r.hidden, ops.rmsnorm(xb, *norm))
    assert torch.equal(r.scalars[0][1:], sa[1:]) and rel(r.scalars[0][:1], sa[:1]) <= 2 * ULP
    assert _lib.device_status() == 0


@pytest.mark.parametrize("E,mult,B,T", [(8, 2, 1, 17), (8, 2, 1, 37), (8, 2, 64, 1), (8, 2, 1, 65), (8, 2, 100, 1), (8, 2, 3, 30), (8, 2, 1, 160),
                                        (8, 2, 1, 161), (8, 1, 1, 129), (4, 4, 1, 37), (4, 4, 1, 100), (4, 4, 1, 161), (8, 4, 1, 20), (8, 4, 1, 160),
                                        (8, 4, 1, 300), (4, 5, 1, 12)])
def test_chain_with_eight_experts_and_with_wide_ones(E, mult, B, T):
    """All rows for every expert and dispatched ones, maps by the router and by the first expert matrix, more tiles than SMs."""
    _chain_against_kernels(1024, E, mult, B, T)


@pytest.mark.parametrize("C", [384, 512, 640, 768, 896])
@pytest.mark.parametrize("B,T", [(1, 20), (1, 72), (7, 10), (9, 8), (1, 120), (2, 96)])
def test_chain_at_other_widths(C, B, T):
    """The tail in clusters of C / 64 CTAs, up to twelve tokens for each of them, and beyond that in kernels of its own."""
    _chain_against_kernels(C, 4, 2, B, T)


@pytest.mark.parametrize("B,T,C", [(160, 1, 1024), (100, 1, 1024), (1, 100, 1024), (1, 160, 1024), (1, 20, 128)])
def test_a_token_whose_router_is_nan_where_the_first_expert_matrix_makes_the_maps(B, T, C):
    """65 to 160 tokens: its row is stored once and combine, or the tail cluster, takes it twice; and the smallest tail cluster."""
    test_both_assignments_of_a_token_whose_router_is_nan_run(B, T, C)


@pytest.mark.parametrize("C,E,mult,B,T", [(128, 4, 1, 1, 18), (128, 8, 2, 1, 200), (640, 4, 1, 1, 47), (384, 4, 3, 1, 500), (1024, 4, 4, 1, 33),
                                          (1024, 4, 8, 1, 170), (1024, 8, 4, 1, 900), (896, 4, 5, 2, 480)])
def test_chain_where_codes_and_weights_outgrow_their_rings(C, E, mult, B, T):
    """The latency GEMM with one chunk and part of a box of codes (128 in-features), odd numbers of chunks, more boxes than its ring
    has, and several tiles a CTA, whose chunks begin anywhere in the rings."""
    _chain_against_kernels(C, E, mult, B, T)


@pytest.mark.parametrize("C,E,N", [(1024, 4, 161), (1024, 8, 257), (1024, 4, 512), (1024, 8, 513), (1024, 4, 1184), (128, 8, 1185), (1024, 4, 2368),
                                   (128, 4, 2369)])
def test_chain_where_maps_and_rows_come_from_the_ids(C, E, N):
    """161 to 2368 tokens: eight or sixteen tokens a CTA, around the lines of the routers and of the form with maps made before."""
    _chain_against_kernels(C, E, 2, 1, N)


@pytest.mark.parametrize("B,T", [(1, 961), (1, 1536), (1, 1537), (2, 2304), (1, 4609)])
def test_chain_where_the_attention_products_leave_the_latency_form(B, T):
    """One wave of tiles of 256 rows: q|k|v up to 1536 tokens, the out-projection up to 4608 (148 SMs)."""
    _chain_against_kernels(1024, 4, 2, B, T)


@pytest.mark.parametrize("B,T,C", [(2, 300, 1024), (3, 234, 1024), (2, 481, 1024), (3, 500, 128), (5, 473, 1024), (5, 474, 1024)])
def test_a_token_whose_router_is_nan_where_the_router_leaves_counts_of_eight(B, T, C):
    """513 to 2368 tokens, and just beyond: the router's counts, the ranks of the dispatch and the segments of the first expert matrix (the
    latency form's up to 960, the pair form's beyond) agree on where an assignment without an expert goes."""
    test_both_assignments_of_a_token_whose_router_is_nan_run(B, T, C)


@pytest.mark.parametrize("skew", [0.5, 4.0])
@pytest.mark.parametrize("T", [513, 961, 1500, 2048])
def test_chain_with_uneven_experts_whose_segments_are_counted_by_the_router(T, skew):
    """Very long segments and empty ones, from counts, in the latency form and in the pair form."""
    test_chain_with_uneven_experts(T, skew)
