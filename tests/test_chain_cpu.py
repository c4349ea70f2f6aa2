"""Host side of the native forward call (chain.py) without a GPU: what it refuses before anything is launched."""
import copy
import ctypes as C
import gc
import pickle
import types
import weakref

import pytest
import torch
from torch.nn.utils import prune

from jarvis_b200 import _lib, chain, modules as jm, ops

CPU = torch.device("cpu")


def test_carried_states_are_checked_before_their_addresses_are_taken():
    good = [torch.zeros(3, 128), None, torch.zeros(3, 128, dtype=torch.bfloat16)]
    out = chain._carried(good, 3, (3, 128), CPU, "h")
    assert out[0] is good[0] and out[1] is None and out[2].dtype is torch.float32
    assert len(chain._carried(good + [None], 3, (3, 128), CPU, "h")) == 3          # more entries than layers: the first ones count
    with pytest.raises(RuntimeError, match="2 entries for 3 layers"):
        chain._carried(good[:2], 3, (3, 128), CPU, "h")
    for exact, shape in ((True, (2, 128)), (False, (2, 128)), (True, (3, 1, 128)), (False, (4, 128))):
        with pytest.raises(RuntimeError, match="of shape"):
            chain._carried([torch.zeros(shape)], 1, (3, 128), CPU, "h", exact=exact)
    chain._carried([torch.zeros(3, 1, 128)], 1, (3, 128), CPU, "h", exact=False)
    with pytest.raises(RuntimeError, match="on meta, expected cpu"):
        chain._carried([torch.zeros(3, 128, device="meta")], 1, (3, 128), CPU, "h")
    with pytest.raises(RuntimeError, match="in place"):
        chain._carried(good, 3, (3, 128), CPU, "h", must_alias=lambda t: True)
    with pytest.raises(RuntimeError, match="in place"):
        chain._carried([torch.zeros(128, 3).t()], 1, (3, 128), CPU, "h", must_alias=lambda t: t.dtype is torch.float32)


def test_states_are_updated_in_place_layer_by_layer():
    a, b = torch.zeros(3, 8), torch.zeros(3, 8)
    got = chain._results(4, [a, None, b, None], True, (3, 8), CPU)
    assert got[0] is a and got[2] is b and got[1].shape == got[3].shape == (3, 8) and got[1].data_ptr() != got[3].data_ptr()
    assert all(g is not a and g is not b for g in chain._results(2, [a, b], False, (3, 8), CPU))
    assert all(g is t for g, t in zip(chain._results(2, [a, b], True, (3, 8), CPU), (a, b)))


def test_a_table_is_made_for_weights_of_one_size():
    """The native call knows no weight's size: a block with one that differs takes the kernel-by-kernel path, which checks."""
    def block():
        return jm.JarvisBlock(128, 2)

    def fits(b):
        return chain._fits(b, b.attn, 128, 256, 4)
    assert fits(block())
    narrow, wide, odd, short, few = block(), block(), block(), block(), block()
    narrow.moe.w2[1] = jm.TernaryLinear(128, 128)
    wide.moe.w1[3] = jm.TernaryLinear(128, 512)
    odd.attn.k_proj = jm.TernaryLinear(256, 128)
    short.norm2.weight = torch.nn.Parameter(torch.ones(64))
    few.moe.w2 = few.moe.w2[:3]
    assert not any(map(fits, (narrow, wide, odd, short, few)))


def _call(**over):
    """An argument block with made-up addresses: for calls that end before anything is launched."""
    lib, n = _lib.load(), 2
    layers = (_lib.Layer * n)()
    for d in layers:
        for i, (name, kind) in enumerate(_lib.Layer._fields_):
            if kind is C.c_void_p:
                setattr(d, name, 0x10000 + 0x1000 * i)
    f = _lib.Forward()
    f.B, f.T, f.C, f.H, f.E, f.hidden = 2, 1, 128, 2, 4, 256
    for i, name in enumerate(("x", "cos_tab", "sin_tab", "accumulators", "scalars", "routing", "workspace")):
        setattr(f, name, 0x100000 + 0x1000 * i)
    states = {k: (C.c_void_p * n)(*(0x200000 + 0x1000 * i for i in range(n))) for k in ("h_in", "h_out", "s_in", "s_out")}
    for k, v in states.items():
        setattr(f, k, C.addressof(v))
    for k, v in over.items():
        if k in states:
            states[k][1] = v
        elif hasattr(layers[1], k):
            setattr(layers[1], k, v)
        else:
            setattr(f, k, v)
    return lib.jb200_forward_layers(layers, n, C.byref(f), None), _lib.last_error()


@pytest.mark.parametrize("over,text", [
    (dict(x=0x100004), "16-byte aligned"), (dict(workspace=0x100080), "workspace 256"), (dict(routing=0x100008), "16-byte aligned"),
    (dict(accumulators=0x100004), "accumulators 8"), (dict(w_router=0x10004), "layer 1"), (dict(w_norm2=0x10008), "layer 1"),
    (dict(w1=0x10008), "layer 1"), (dict(w2=None), "layer 1 is missing"), (dict(h_out=None), "layer 1 is missing"),
    (dict(h_in=0x200004), "membranes 8"), (dict(h_out=0x20000C), "membranes 8"), (dict(s_in=0x200008), "attention states"),
    (dict(s_out=0x200004), "attention states"), (dict(ids=0x300000), "embedding table")])
def test_forward_arguments_are_checked_before_the_first_launch(over, text):
    rc, message = _call(**over)
    assert rc == _lib.ERR_ARG and text in message


def test_overridden_methods_need_the_kernel_by_kernel_path(monkeypatch):
    class Attn(jm.AssociativeLinearAttention):
        def scan_rows(self, *a, **k):
            return super().scan_rows(*a, **k)

    class Harmless(jm.JarvisBlock):
        def extra_repr(self):
            return "named"

    def block(cls=jm.JarvisBlock):
        return cls(128, 2)
    assert chain._stock(block()) and chain._stock(block(Harmless))
    sub, inst, other, packed = block(), block(), block(), block()
    sub.attn = Attn(128, 2)
    inst.moe.run_rows = lambda *a, **k: None
    other.attn = torch.nn.Identity()
    packed.attn.out_proj.packed = lambda: None
    assert not any(map(chain._stock, (sub, inst, other, packed)))
    monkeypatch.setattr(jm.JarvisBlock, "step_rows", lambda *a, **k: None)
    assert not chain._stock(block())


def test_modules_that_hold_a_table_can_be_copied_and_pickled():
    block = jm.JarvisBlock(128, 2)
    tab = object.__new__(chain.LayerTable)
    tab.array = (_lib.Layer * 1)()                 # ctypes structures with pointers cannot be pickled
    block.__dict__["_layer_table"] = tab
    for twin in (copy.deepcopy(block), pickle.loads(pickle.dumps(block))):
        assert twin.__dict__["_layer_table"] is None and block.__dict__["_layer_table"] is tab
        assert torch.equal(twin.attn.q_proj.weight, block.attn.q_proj.weight)


def test_decays_are_kept_while_their_parameter_is():
    """Captured graphs hold their address, so an edit of another parameter must not make new ones."""
    at = jm.AssociativeLinearAttention(128, 2)
    first = at.decays()
    with torch.no_grad():
        at.q_proj.weight.add_(1.0)
    assert at.decays() is first and torch.equal(first, torch.sigmoid(at.gamma_raw))
    with torch.no_grad():
        at.gamma_raw.add_(1.0)
    assert at.decays() is not first and torch.equal(at.decays(), torch.sigmoid(at.gamma_raw))


def test_what_a_captured_session_keeps():
    model = jm.Jarvis(vocab_size=32, d_model=128, n_layers=1, n_heads=2)
    at = model.blocks[0].attn
    at._qkv.packed, at._qkv.alpha = torch.zeros(3), torch.ones(3)
    made = [at.decays(), at._qkv.packed, at.rotary.half_tables(8, CPU)[0], jm._f32(model.final_norm.weight)]
    model.blocks[0].moe = torch.nn.Identity()                       # a part of the caller's own
    flat = [t for entry in jm._made_from_parameters(model) if isinstance(entry, tuple) for t in entry]
    assert all(any(t is m for t in flat) for m in made)


def test_last_aux_is_a_list_on_either_path():
    model = jm.Jarvis(vocab_size=32, d_model=128, n_layers=2, n_heads=2)
    assert model.last_aux is None
    rows = torch.arange(6.0).view(2, 3)
    for aux in (rows, list(rows.unbind(0))):
        model._aux = aux
        assert isinstance(model.last_aux, list) and torch.equal(torch.stack(model.last_aux), rows)
    model._reflect = rows
    model.last_aux = model.blocks[0].moe.last_routing = ["of an override"]
    assert model._aux == model.blocks[0].moe._routing == ["of an override"] and model._reflect is None


@pytest.fixture
def tables_on_cpu(monkeypatch):
    """Layer tables without a GPU: the packing is made up, nothing is ever launched with them."""
    monkeypatch.setattr(ops, "pack_ternary", lambda w, alpha=None: (torch.zeros(w.shape[0], w.shape[1] // 4, dtype=torch.uint8), torch.ones(1)))
    monkeypatch.setattr(ops, "prepare_weights", lambda p: p.clone())
    monkeypatch.setattr(chain, "supported", lambda blocks: all(map(chain._stock, blocks)))


def test_a_dropped_block_goes_at_once(tables_on_cpu):
    """Its own table must not keep it until the next collection: the memory of a replaced model is wanted right away."""
    block = jm.JarvisBlock(128, 2).eval()
    assert chain.table_of(block, [block]) is not None and block.__dict__["_layer_table"] is not None
    gone = [weakref.ref(t) for t in (block, block.attn, block.moe.w1[0].weight)]
    gc.disable()
    try:
        del block
        assert all(ref() is None for ref in gone)
    finally:
        gc.enable()


def test_a_table_follows_overrides_and_replaced_parts(tables_on_cpu):
    blocks = [jm.JarvisBlock(128, 2).eval() for _ in range(2)]
    owner = torch.nn.Module()
    tab = chain.table_of(owner, blocks)
    assert chain.table_of(owner, blocks) is tab
    for part, name in ((blocks[1], "forward_rows"), (blocks[0], "step_rows"), (blocks[1].attn, "scan_rows"), (blocks[0].moe, "packed"),
                       (blocks[0].attn.rotary, "half_tables")):
        setattr(part, name, lambda *a, **k: None)
        assert chain.table_of(owner, blocks) is None
        delattr(part, name)
        assert chain.table_of(owner, blocks) is not None
    with torch.no_grad():
        blocks[0].norm1.weight.mul_(2.0)
    assert chain.table_of(owner, blocks) is not tab
    blocks[0].reflect.train()
    assert chain.table_of(owner, blocks) is None
    blocks[0].reflect.eval()
    prune.identity(blocks[0].attn.q_proj, "weight")          # the weight is no parameter any more
    assert chain.table_of(owner, blocks) is None


def test_refused_tokens_do_not_move_the_position():
    model = jm.Jarvis(vocab_size=32, d_model=128, n_layers=1, n_heads=2).eval()
    with pytest.raises(RuntimeError):
        model(torch.zeros((1, 5), dtype=torch.int64), persist_state=True)
    assert model._token_pos == 0


def test_which_single_token_steps_run_in_one_launch():
    """Several sequences in a cluster only with the sums of four and more, and those only with states, however few clusters fit."""
    lib = _lib.load()
    for resident in range(10):
        for B in range(0, 80):
            for carried in (0, 1):
                n = lib.jb200_step_clusters(B, resident, carried)
                if n == 0:
                    continue
                assert 1 <= n <= min(resident, 8, B) and -(-B // n) <= 8
                assert B >= 4 or n == B                  # the kernels sum two or three sequences another way
                assert carried or B < 4
    whole = [lib.jb200_step_clusters(B, 7, 1) for B in range(1, 60)]
    assert whole == [1, 2, 3, 4, 5, 6, 7, 4, 5, 5, 6, 6] + [7] * 44 + [0] * 3
    assert [lib.jb200_step_clusters(B, 7, 0) for B in range(1, 6)] == [1, 2, 3, 0, 0]
    assert [lib.jb200_step_clusters(B, 1, 1) for B in (1, 2, 3, 4, 8, 9)] == [1, 0, 0, 1, 1, 0]
    assert [lib.jb200_step_clusters(B, 2, c) for B in (2, 3) for c in (0, 1)] == [2, 2, 0, 0]


class _StepLibrary:
    """The library with a one-launch step of layouts of 64 bytes; counts the layers that are laid out."""

    def __init__(self, lib):
        self._lib, self.laid = lib, 0

    def __getattr__(self, name):
        return getattr(self._lib, name)

    def jb200_step_max_sequences(self):
        return 56

    def jb200_step_weight_bytes(self, *sizes):
        return 64

    def jb200_prepare_step_weights(self, *args):
        self.laid += 1
        return _lib.OK


@pytest.fixture
def step_library(tables_on_cpu, monkeypatch):
    lib = _StepLibrary(_lib.load())
    monkeypatch.setattr(_lib, "load", lambda: lib)
    monkeypatch.setattr(ops, "_stream", lambda: None)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev=None: types.SimpleNamespace(synchronize=lambda: None))
    return lib


def test_without_memory_for_a_second_layout_steps_go_kernel_by_kernel(step_library, monkeypatch):
    blocks = [jm.JarvisBlock(128, 2).eval() for _ in range(2)]
    tab, asked = chain.LayerTable(blocks), []

    def empty(*a, **k):
        asked.append(a)
        raise torch.OutOfMemoryError("out of memory")
    monkeypatch.setattr(chain.torch, "empty", empty)
    assert tab.step_weights(1) is None and tab.step_weights(1) is None and len(asked) == 1


def test_an_edited_layer_alone_is_laid_out_again(step_library):
    blocks = [jm.JarvisBlock(128, 2).eval() for _ in range(3)]
    owner = torch.nn.Module()

    def layouts():
        tab = chain.table_of(owner, blocks)
        return list(tab.step_weights(1)), tab
    first, tab = layouts()
    assert step_library.laid == 3 and len(set(first)) == 3 and layouts()[1] is tab
    with torch.no_grad():                    # read from the parameters themselves
        for p in (blocks[0].norm1.weight, blocks[1].moe.router.weight, blocks[2].liquid.var_scale):
            p.mul_(1.5)
    second, other = layouts()
    assert other is not tab and second == first and step_library.laid == 3
    with torch.no_grad():
        blocks[1].moe.w2[3].weight.mul_(1.5)
        blocks[2].attn.gamma_raw.add_(1.0)
    third, _ = layouts()
    assert step_library.laid == 5 and third[0] == first[0] and third[1] != first[1] and third[2] != first[2]
    held = [weakref.ref(tab), weakref.ref(other)]
    del tab, other
    gc.collect()
    assert all(ref() is None for ref in held)            # a table does not keep the one before it


@pytest.mark.parametrize("E", [4, 8])
@pytest.mark.parametrize("hidden", [1024, 2048, 4096])
def test_expert_tiles_are_no_larger_than_their_rows(E, hidden):
    """However many tiles the experts need, a token tile ends with the rows there are: the smallest that leaves the launch on half of the
    SMs (all rows for every expert) or on all of them, else one for all rows.  Its ring is one that the kernel has, in chunks of four
    K-blocks or of two."""
    lib, out, of = _lib.load(), (C.c_int32 * 6)(), (C.c_int32 * 4)()
    rings = lambda tile, K: [of[0] for coarse in (0, 1) if lib.jb200_host_mid_ring(tile, K, coarse, of)]
    up = lambda n: (n + 15) // 16 * 16
    for tokens in range(1, 961):
        assert lib.jb200_host_expert_tiles(tokens, 0, 1024, E, hidden, 148, out) == 1
        all_rows, bm, bn, bn_max, ring, ring_max = out
        rows = tokens if all_rows else -(-2 * tokens // E)
        assert all_rows == (tokens <= 160) and bn <= bn_max <= min(256, up(2 * tokens)) and ring >= ring_max >= 2
        assert ring in rings(bn, 1024) and ring_max in rings(bn_max, 1024)
        if all_rows:
            tiles = lambda n: hidden // bm * E * -(-tokens // n)
            assert bn == bn_max <= up(tokens)
            assert tiles(bn) <= 74 or bn == up(tokens)
            assert bn <= 64 or tiles(bn - 16) > 74
        else:
            assert bn <= up(rows + -(-rows // 8))
        assert lib.jb200_host_expert_tiles(tokens, 1, 1024, E, hidden, 148, out) == 1 and out[2] <= out[3] <= min(256, up(2 * tokens))
        assert out[4] in rings(out[2], hidden) and out[5] in rings(out[3], hidden)
    assert lib.jb200_host_expert_tiles(961, 0, 1024, E, hidden, 148, out) == 0


@pytest.mark.parametrize("K", [128, 256, 384, 1024, 1152, 2048, 8192])
def test_the_ring_of_the_latency_gemm_fits_its_memories(K):
    """Accumulator (f32, bn columns in steps of 64) and weights (32 columns a K-block of 64) in the 512 columns of tensor memory; codes (boxes of
    128 rows x 512 in-features, at most four) and rows (bf16) in 227 KB; never more chunks than K has or the kernel has barriers for."""
    lib, out = _lib.load(), (C.c_int32 * 4)()
    for bn in range(16, 257, 16):
        for coarse in (0, 1):
            kb = 4 if coarse else 2
            ok = lib.jb200_host_mid_ring(bn, K, coarse, out)
            if K % (64 * kb):
                assert not ok
                continue
            boxes, acc, rows = 16384 * min(-(-K // 512), 4), -(-bn // 64) * 64, 128 * bn * kb
            assert out[1] == kb and out[2] == acc + out[0] * kb * 32 <= 512
            assert out[3] == boxes + out[0] * rows + 1024 <= 223 * 1024       # beside them control words and the epilogue's row lists, 3 KB
            assert out[0] <= min(8, K // (64 * kb))
            # and no chunk is left out that all of them would hold
            assert out[0] == min(8, K // (64 * kb)) or out[2] + kb * 32 > 512 or out[3] + rows > 223 * 1024
            assert ok == (out[0] >= 1) and (coarse or out[0] >= min(2, K // 128))


@pytest.mark.parametrize("sms", [8, 37, 59, 60, 132, 148, 160])
def test_whoever_reads_maps_and_counts_finds_them_made_on_a_device_of_any_size(sms):
    """161 to 512 tokens count the ids whatever the device; counts of every eight tokens need a router of a single pass (two CTAs of eight
    tokens an SM); and the first expert matrix takes its segments from counts only where the router leaves them."""
    lib, out = _lib.load(), (C.c_int32 * 2)()
    ROUTER, EXPERT_GEMM, FROM_IDS, FROM_EIGHTS, METADATA = range(5)
    for tokens in range(1, 3001):
        for hidden in (2048, 8192):
            assert lib.jb200_host_dispatch_plan(tokens, 1024, hidden, sms, out) == 1
            maps, load = out
            if tokens <= 160:
                want = ROUTER if tokens <= (16 if hidden == 2048 else 0) else EXPERT_GEMM
            else:
                want = FROM_IDS if tokens <= 512 else FROM_EIGHTS if tokens <= min(16 * sms, 2368) else METADATA
            assert maps == want and load == (maps in (FROM_IDS, FROM_EIGHTS)), (tokens, hidden)
    assert lib.jb200_host_dispatch_plan(0, 1024, 2048, sms, out) == 0
