"""The work a user of this framework has it do, as cases that can be timed and compared.

A case is a dict of plain values.  `listed()` names the standing ones, `draw(rng)` gives another one of the same
ranges, `prepare(case, seed)` makes what a user's program holds before the call (inputs, weights, carried state),
`run(state)` makes one pass through the public entry points, `work(case)` says what the pass cannot do without and
`tolerance(case)` how far two correct implementations may lie apart.

The model is the 24-layer 606M configuration (d_model 1024, 16 heads x 64, 4 experts, top-2, vocabulary 50257) with
seeded Gaussian ternary weights and per-head decays U[0.90, 0.999]; token ids are uniform over the vocabulary.
The path is inference only (there is no backward), so its two directions are prefill and decode.
"""
import math

import torch

import jarvis_b200  # noqa: F401
from jarvis_b200 import modules as jm
from jarvis_b200 import ops, synthetic

VOCAB, C, LAYERS, HEADS, D, EXPERTS = 50257, 1024, 24, 16, 64, 4
HID = 2 * C
PRIOR_MAX = 4096          # longest context a decode or a continued prompt starts from
TOKENS_MAX = 16384        # tokens of the largest model call (8 x 2048)
ROWS_MAX = 65536          # tokens of the largest single-layer call
BF16 = torch.bfloat16


def listed():
    return [
        # a short interactive prompt: the latency of one small forward, an odd length
        dict(name="prefill_1x37", kind="prefill", B=1, T=37, loss=False),
        # corpus evaluation: one 256-token window with its loss
        dict(name="score_1x256", kind="prefill", B=1, T=256, loss=True),
        # batch prefill at the size the benchmark quotes
        dict(name="prefill_8x2048", kind="prefill", B=8, T=2048, loss=False),
        # one long document
        dict(name="prefill_1x16384", kind="prefill", B=1, T=16384, loss=False),
        # continued prompts with carried state and their own positions: chunked prefill, admission to a serving slot
        dict(name="chunk_3x777", kind="chunk", B=3, T=777),
        # one token per step: a single conversation, a serving batch of 64 slots, 256 ragged sequences
        dict(name="decode_1", kind="decode", B=1),
        dict(name="decode_64", kind="decode", B=64),
        dict(name="decode_256", kind="decode", B=256),
        # one block as a drop-in module of a host model that keeps float32 activations
        dict(name="block_1x512_f32", kind="block", B=1, T=512, dtype="f32"),
        # one MoE layer alone on many tokens, expert loads skewed by Zipf(1.2)
        dict(name="moe_65536", kind="moe", N=65536, dtype="bf16"),
        # the two scans alone, as in the scan sweep
        dict(name="attn_32x2048", kind="attn", B=32, T=2048, carry=False),
        dict(name="lsf_32x2048", kind="lsf", B=32, T=2048, per_element=False, dtype="bf16"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _batch_and_length(rng, b_max, t_min, t_max, rows):
    T = _log_int(rng, t_min, t_max)
    B = _log_int(rng, 1, max(1, min(b_max, rows // T)))
    return B, T


def draw(rng):
    kind = rng.choice(["prefill", "prefill", "prefill", "chunk", "decode", "decode", "block", "moe", "attn", "lsf"])
    if kind == "prefill":
        B, T = _batch_and_length(rng, 16, 16, TOKENS_MAX, TOKENS_MAX)
        return dict(kind=kind, B=B, T=T, loss=B * T <= 2048 and rng.random() < 0.3)
    if kind == "chunk":
        B, T = _batch_and_length(rng, 16, 16, 2048, 8192)
        return dict(kind=kind, B=B, T=T)
    if kind == "decode":
        return dict(kind=kind, B=_log_int(rng, 1, 256))
    if kind == "block":
        B, T = _batch_and_length(rng, 8, 16, 2048, TOKENS_MAX)
        return dict(kind=kind, B=B, T=T, dtype=rng.choice(["f32", "bf16"]))
    if kind == "moe":
        return dict(kind=kind, N=_log_int(rng, 64, ROWS_MAX), dtype=rng.choice(["f32", "bf16"]))
    B, T = _batch_and_length(rng, 32, 64, 8192, ROWS_MAX)
    if kind == "attn":
        return dict(kind=kind, B=B, T=T, carry=rng.random() < 0.5)
    return dict(kind=kind, B=B, T=T, per_element=rng.random() < 0.4, dtype=rng.choice(["f32", "bf16"]))


# ----------------------------------------------------------------------------------------------
# what a program holds before the call
# ----------------------------------------------------------------------------------------------
def _ternary_init(module, gen):
    """The benchmark's weights: every ternary matrix ~ N(0, 0.02^2), decays U[0.90, 0.999]."""
    with torch.no_grad():
        for m in module.modules():
            if isinstance(m, jm.TernaryLinear):
                m.weight.normal_(0.0, 0.02, generator=gen)
            elif isinstance(m, jm.AssociativeLinearAttention):
                m.gamma_raw.copy_(torch.logit(torch.rand(m.n_heads, generator=gen, device="cuda") * 0.099 + 0.9))
    return module.eval()


def _model(gen, max_seq_len):
    torch.manual_seed(gen.initial_seed())
    with torch.device("cuda"):
        model = jm.Jarvis(VOCAB, C, LAYERS, HEADS, EXPERTS, max_seq_len=max_seq_len)
    _ternary_init(model, gen)
    model(torch.zeros((1, 1), dtype=torch.int64, device="cuda"))       # a loaded model has packed its weights
    return model


def _tokens(gen, *shape):
    return torch.randint(0, VOCAB, shape, generator=gen, device="cuda")


def _normal(gen, *shape, dtype=torch.float32):
    return torch.randn(*shape, generator=gen, device="cuda").to(dtype)


def _dtype(case):
    return torch.float32 if case["dtype"] == "f32" else BF16


def _context(model, gen, B, seed, limit):
    """Ragged prior lengths and the state after the last (up to) 32 tokens of each context."""
    prior = synthetic.ragged_prior_lengths(B, PRIOR_MAX, seed).to("cuda")
    start = (prior - 32).clamp_min(0).to(torch.int32)
    _, state = model.step(_tokens(gen, B, 32), positions=start, max_position=limit)
    return state, start + 32


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    st = dict(kind=kind)
    if kind == "prefill":
        st["model"] = _model(gen, max(case["T"], 256))
        st["idx"] = _tokens(gen, case["B"], case["T"])
        st["targets"] = _tokens(gen, case["B"], case["T"]) if case["loss"] else None
    elif kind == "chunk":
        limit = PRIOR_MAX + 32 + case["T"]
        st["model"] = _model(gen, limit)
        st["state"], st["positions"] = _context(st["model"], gen, case["B"], seed, limit)
        st["idx"] = _tokens(gen, case["B"], case["T"])
        st["limit"] = limit
    elif kind == "decode":
        B, limit = case["B"], 4 * PRIOR_MAX
        model = _model(gen, limit)
        first, positions = _context(model, gen, B, seed, limit)
        # the carried state of all layers in one buffer each, handed to the session layer by layer
        st["h"], st["S"] = torch.stack(first["h"]), torch.stack(first["S"])
        session = jm.DecodeSession(model, {"h": list(st["h"].unbind(0)), "S": list(st["S"].unbind(0))}, positions, limit)
        session.capture()
        session.load_state(first, positions)
        st["session"], st["idx"] = session, _tokens(gen, B, 1)
    elif kind == "block":
        torch.manual_seed(seed)
        with torch.device("cuda"):
            block = jm.JarvisBlock(C, HEADS, EXPERTS, max_seq_len=case["T"])
        st["block"] = _ternary_init(block, gen)
        st["x"] = _normal(gen, case["B"], case["T"], C, dtype=_dtype(case))
        st["h"] = _normal(gen, case["B"], C)
    elif kind == "moe":
        torch.manual_seed(seed)
        with torch.device("cuda"):
            moe = jm.SparseMoELayer(C, EXPERTS)
        st["moe"] = _ternary_init(moe, gen)
        x = _normal(gen, 1, case["N"], C)
        x[..., 0] = 1.0                                   # a constant channel carries the skew of the expert loads
        with torch.no_grad():
            moe.router.weight[:, 0] = 1.6 * torch.log(synthetic.zipf_shares(EXPERTS)).cuda()
        st["x"] = x.to(_dtype(case))
    elif kind == "attn":
        B, T = case["B"], case["T"]
        st.update(B=B, T=T, qkv=_normal(gen, B * T, 3 * C, dtype=BF16))
        st["gamma"] = torch.rand(HEADS, generator=gen, device="cuda") * 0.099 + 0.9
        st["cos"], st["sin"] = jm.RotaryEmbedding(D, T).half_tables(T, st["qkv"].device)
        st["S"] = _normal(gen, B, HEADS, D, D) if case["carry"] else None
    else:
        B, T, dt = case["B"], case["T"], _dtype(case)
        st["x"], st["h"] = _normal(gen, B, T, C, dtype=dt), _normal(gen, B, C)
        if case["per_element"]:
            st["alpha"] = (torch.rand(B, T, C, generator=gen, device="cuda") * 0.89 + 0.1).to(dt)
            st["lsf"] = jm.LiquidStateFusionExt()
        else:
            st["alpha"], st["lsf"] = None, jm.LiquidStateFusion(C).cuda()
            st["act_var"] = torch.rand((), generator=gen, device="cuda") + 0.05
    return st


# ----------------------------------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------------------------------
def run(st):
    kind = st["kind"]
    with torch.no_grad():
        if kind == "prefill":
            return st["model"](st["idx"], targets=st["targets"])
        if kind == "chunk":
            return st["model"].step(st["idx"], positions=st["positions"], state=st["state"], max_position=st["limit"])
        if kind == "decode":
            return st["session"].step(st["idx"]), st["h"], st["S"], st["session"].positions
        if kind == "block":
            return st["block"](st["x"], st["h"])
        if kind == "moe":
            return st["moe"](st["x"])
        if kind == "attn":
            q, k, v = st["qkv"][:, :C], st["qkv"][:, C:2 * C], st["qkv"][:, 2 * C:]
            return ops.attn_scan(q, k, v, st["gamma"], st["cos"], st["sin"], st["B"], st["T"], HEADS, state_in=st["S"],
                                 want_state=True)
        if st["alpha"] is not None:
            return st["lsf"](st["alpha"], st["x"], st["h"])
        return st["lsf"](st["x"], st["act_var"], st["h"])


# ----------------------------------------------------------------------------------------------
# what the pass cannot do without
# ----------------------------------------------------------------------------------------------
STATE_BYTES = HEADS * D * D * 4                       # attention state of one sequence and layer
MOE_FLOPS = 2 * 2 * (2 * C * HID)                     # one token: two experts of two matrices
BLOCK_FLOPS = 2 * 4 * C * C + MOE_FLOPS + HEADS * 2 * 2 * D * D
EXPERT_BYTES = 2 * C * HID // 4                       # 2 bits per weight
BLOCK_BYTES = 4 * C * C // 4 + EXPERT_BYTES * EXPERTS


def work(case):
    kind = case["kind"]
    if kind in ("prefill", "chunk", "decode"):
        B, T = case["B"], case.get("T", 1)
        n = B * T
        flops = n * (LAYERS * BLOCK_FLOPS + 2 * C * VOCAB)
        # packed weights of the experts that n tokens can reach, the head, the embedding rows, the logits
        layer = C * C + EXPERT_BYTES * min(EXPERTS, 2 * n)
        byts = LAYERS * layer + 2 * C * VOCAB + n * (8 + 4 * C) + 2 * n * VOCAB
        if kind != "prefill":
            byts += 2 * LAYERS * B * (STATE_BYTES + 4 * C)
        return dict(bytes=byts, flops=flops)
    if kind == "block":
        n = case["B"] * case["T"]
        es = 4 if case["dtype"] == "f32" else 2
        return dict(bytes=BLOCK_BYTES + 2 * n * C * es + 2 * case["B"] * C * 4, flops=n * BLOCK_FLOPS)
    if kind == "moe":
        es = 4 if case["dtype"] == "f32" else 2
        return dict(bytes=EXPERT_BYTES * EXPERTS + 2 * case["N"] * C * es, flops=case["N"] * MOE_FLOPS)
    n = case["B"] * case["T"]
    if kind == "attn":
        return dict(bytes=n * 4 * C * 2 + case["B"] * STATE_BYTES * (2 if case["carry"] else 1), flops=n * HEADS * 4 * D * D)
    es = 4 if case["dtype"] == "f32" else 2
    return dict(bytes=n * C * es * (3 if case["per_element"] else 2) + 2 * case["B"] * C * 4, flops=n * C * 4)


def tolerance(case):
    kind = case["kind"]
    if kind in ("prefill", "chunk", "decode"):
        # bf16 GEMM and scan inputs through 24 layers: two orders of rounding lie 3e-3 to 6e-3 apart (the feature map
        # in the projection's epilogue or in the scan), single logits up to 0.05.  `max` leaves room for a token whose
        # second and third expert are all but tied and which may go to either of them.
        return dict(rel=1e-2, max=0.2)
    if kind == "lsf":
        return dict(rel=1e-5) if case["dtype"] == "f32" else dict(rel=5e-3)
    return dict(rel=1e-2)
