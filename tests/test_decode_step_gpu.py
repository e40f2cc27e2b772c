"""Decode steps of the Reasoner on the kernels: what surrounds the layers (csrc/step_edges.cu) and the order of the launches."""
import pytest
import torch

from cosmos_b200 import ops
from cosmos_b200.config import get_model_config
from cosmos_b200.serve.decoder import TPDecoder

pytestmark = pytest.mark.gpu

DEV = "cuda"


@pytest.fixture(autouse=True)
def _status_clean():
    ops.load_extension()
    yield
    torch.cuda.synchronize()
    ops.check_status()


def _decoder(batch, prompt=40, room=16, **kw):
    cfg = get_model_config("tiny128", **{"n_layers": 2, **kw})
    dec = TPDecoder(cfg, 1, 0, None, DEV, page_size=16, max_batch=batch, max_len=prompt + room)
    dec.prefill_synthetic(batch, prompt, room)
    return dec


@pytest.mark.parametrize("batch,d,inner", [(1, 512, 8192), (3, 1024, 16384), (33, 512, 16384), (128, 2048, 8192)])
def test_eager_step_behind_a_kernel_that_writes_a_weight(batch, d, inner):
    """The GEMM in front of an eager step writes the weight that the step's first projection reads (and reads ahead), with
    nothing between them; again with that weight long in place. The same bits: the same kernels on the same numbers."""
    dec = _decoder(batch, d_model=d, n_heads=d // 128, n_kv_heads=2, ffn_dim=2 * d)
    tokens, lens = dec.tokens.clone(), dec.lens.clone()
    w = dec.layers[0]["wqkv"]
    right = (torch.randn(d, inner, device=DEV) * inner ** -0.5).bfloat16()
    dec.step()
    for seed in range(3):
        torch.manual_seed(seed)
        left = (torch.randn(w.shape[0], inner, device=DEV) * 0.05).bfloat16()
        dec.tokens.copy_(tokens)
        dec.lens.copy_(lens)
        ops.gemm(left, right, out=w)
        dec.step()
        got = dec.last_logits.clone()
        torch.cuda.synchronize()
        dec.tokens.copy_(tokens)
        dec.lens.copy_(lens)
        torch.cuda.synchronize()
        dec.step()
        assert torch.equal(got, dec.last_logits)


def _logits_and_tokens(dec, steps=2):
    out = []
    for _ in range(steps):
        dec.step()
        out += [dec.last_logits.clone(), dec.next_tokens.clone().long(), dec.lens.clone().long()]
    return out


@pytest.mark.parametrize("name,dtype,forms", [
    ("tokens", torch.int32, ("tokens",)), ("step_inc", torch.long, ()), ("pos_delta", torch.int32, ()), ("next_tokens", torch.int32, ("next_tokens",)),
    ("step_inc", torch.int32, ("scalar",)), ("next_tokens", torch.long, ("strided",)), ("inv_freq", torch.float32, ("strided",))])
def test_step_takes_its_state_in_other_forms(name, dtype, forms):
    """State that the kernels at both ends of a step do not take: the same logits and tokens as with theirs."""
    dec, same = _decoder(3), _decoder(3)
    for d in (dec, same):
        d.step_inc = torch.ones(3, dtype=torch.int32, device=DEV)
        d.pos_delta = torch.tensor([0, -3, -40], device=DEV)
    t = getattr(dec, name).to(dtype)
    if "scalar" in forms:
        t = t[0]
    if "strided" in forms:
        t = torch.stack([t, t], dim=-1)[..., 0]
    setattr(dec, name, t)
    for x, y in zip(_logits_and_tokens(dec), _logits_and_tokens(same)):
        # the kernel's rotary tables may differ from torch's in the last bits, which bf16 sums over two layers hardly show
        assert torch.equal(x, y) if x.dtype == torch.long else (x.float() - y.float()).norm() <= 1e-2 * y.float().norm()


def test_first_own_op_of_a_program_is_a_step(monkeypatch):
    """The step loads the kernel library itself: nothing before it may have."""
    import cosmos_b200.serve.paged as paged
    monkeypatch.setattr(paged.ops, "load_extension", lambda **kw: False)
    dec = _decoder(1)
    monkeypatch.undo()
    calls = []
    load = ops.load_extension
    monkeypatch.setattr(ops, "load_extension", lambda *a, **kw: calls.append(1) or load(*a, **kw))
    real = ops.rmsnorm
    seen = []
    monkeypatch.setattr(ops, "rmsnorm", lambda *a, **kw: seen.append(len(calls)) or real(*a, **kw))
    dec.step()
    assert seen and seen[0] > 0


def test_step_in_fp32_needs_no_kernel_library(monkeypatch):
    """A decoder of another type runs on the plain definitions, on a host without the library too."""
    cfg = get_model_config("tiny128", n_layers=1)
    dec = TPDecoder(cfg, 1, 0, None, DEV, page_size=16, max_batch=2, max_len=64, dtype=torch.float32)
    assert all(dec.cache.reserve(i, 28) for i in range(2))
    dec.table, dec.max_len = dec.cache.tables([0, 1])[0], 28
    dec.lens, dec.tokens = torch.full((2,), 20, dtype=torch.int32, device=DEV), torch.tensor([5, 9], device=DEV)
    dec.next_tokens = torch.zeros_like(dec.tokens)
    monkeypatch.setattr(ops, "_loaded", False)
    monkeypatch.setattr(ops, "load_extension", lambda *a, **kw: False)
    monkeypatch.setattr(torch.ops, "cosmos_b200", None)
    dec.step()
    assert dec.last_logits.isfinite().all()


def test_step_counts_negative_token_ids_from_the_end():
    dec = _decoder(4)
    dec.tokens = torch.tensor([-1, 0, -dec.cfg.vocab_size, 7], device=DEV)
    x = torch.ops.cosmos_b200.decode_begin(dec.lens, None, None, dec.inv_freq, dec.table, dec.page_size, dec.tokens, dec.embed)[0]
    assert torch.equal(x, dec.embed[dec.tokens])


@pytest.mark.parametrize("bad", ["length past the row", "far past it", "negative length", "unused entry", "page beyond the cache", "token"])
def test_step_without_a_place_for_its_token_stores_nothing(bad):
    """One sequence of three has a bad length, table entry or token. It is reported; its keys and values are not stored, the others' are;
    the lengths stay inside the table."""
    dec = _decoder(3)
    room = dec.table.shape[1] * dec.page_size
    lens = torch.tensor([40, 32, 47], dtype=torch.int32, device=DEV)   # the second one's next token begins a page
    if bad == "unused entry":
        dec.table[1, 32 // dec.page_size] = -1
    elif bad == "page beyond the cache":
        dec.table[1, 32 // dec.page_size] = dec.cache.k[0].shape[0]
    elif bad == "token":
        dec.tokens[1] = dec.cfg.vocab_size
    else:
        lens[1] = {"length past the row": room, "far past it": 2 ** 31 - 1, "negative length": -5}[bad]
    dec.lens = lens.clone()
    before = [(k.clone(), v.clone()) for k, v in zip(dec.cache.k, dec.cache.v)]
    slots = torch.ops.cosmos_b200.decode_begin(lens.clone(), None, None, dec.inv_freq, dec.table, dec.page_size, dec.tokens, dec.embed,
                                               dec.cache.k[0].shape[0])[3].tolist()
    with pytest.raises(RuntimeError, match="index out of range at " + ("decoder stack token" if bad == "token" else "decode_qkv_post slot")):
        ops.check_status()
    assert [s < 0 for s in slots] == [False, bad != "token", False]
    want = {"length past the row": room, "far past it": room, "negative length": 0, "token": 33}.get(bad, 32)
    if bad in ("far past it", "negative length"):   # no state that a sequence gets into: up to the first layer's store
        x, cos, sin, at = torch.ops.cosmos_b200.decode_begin(dec.lens, None, None, dec.inv_freq, dec.table, dec.page_size, dec.tokens,
                                                             dec.embed, dec.cache.k[0].shape[0])
        p = dec.layers[0]
        ops.gemm_decode_qkv_post(x, p["wqkv"], dec.hq, cos, sin, p["q_norm"], p["k_norm"], 1e-6, at, dec.cache.k[0], dec.cache.v[0])
    else:
        dec.max_len = room
        dec.step()
    with pytest.raises(RuntimeError, match="index out of range"):
        ops.check_status()
    assert dec.lens.tolist() == [41, want, 48]
    for li, pair in enumerate(before):
        for old, new in zip(pair, (dec.cache.k[li], dec.cache.v[li])):
            for s in slots:
                if s >= 0:
                    assert li > 0 or not torch.equal(old[s // 16, :, s % 16], new[s // 16, :, s % 16])
                    old[s // 16, :, s % 16] = new[s // 16, :, s % 16]
            assert torch.equal(old, new)


def test_engine_hands_out_nothing_after_a_report():
    """A request whose next page is taken away: the engine raises before the request is finished."""
    from cosmos_b200.models.mot import MoTModel
    from cosmos_b200.serve.engine import BatchEngine
    cfg = get_model_config("tiny128", n_layers=1)
    model = MoTModel(cfg, dtype=torch.bfloat16, device=DEV)
    eng = BatchEngine(model, max_batch=2, max_len=64, page_size=16)
    r = eng.submit(list(range(1, 16)), max_new_tokens=4)
    eng.step()                                # the prompt and one token: a page is full
    assert int(eng.dec.lens[r.slot]) == 16
    eng.dec.table[r.slot, 1] = -1
    with pytest.raises(RuntimeError, match="index out of range"):
        eng.run_until_done()
    assert r.rid not in eng.finished


@pytest.mark.parametrize("setting", ["0", "1"])
def test_programmatic_edges_of_a_captured_step(setting, monkeypatch):
    """COSMOS_DECODE_PDL=0 leaves no launch of the step, first and last kernel included, that may start before its predecessor ends.
    The same logits with and without."""
    from cuda.bindings import runtime
    monkeypatch.setenv("COSMOS_DECODE_PDL", setting)
    dec, same = _decoder(2), _decoder(2)
    monkeypatch.setenv("COSMOS_DECODE_PDL", "1")
    same.step()
    monkeypatch.setenv("COSMOS_DECODE_PDL", setting)
    dec.step()
    assert torch.equal(dec.last_logits, same.last_logits)
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g), torch.no_grad():
        dec._step_impl()
    raw = runtime.cudaGraph_t(g.raw_cuda_graph())
    n = runtime.cudaGraphGetEdges_v2(raw)[-1]
    data = runtime.cudaGraphGetEdges_v2(raw, n)[3]
    early = sum(d.type == int(runtime.cudaGraphDependencyType.cudaGraphDependencyTypeProgrammatic) for d in data)
    assert n > 15 and (early == 0 if setting == "0" else early > 15), (n, early)
    assert torch.ops.cosmos_b200.launch_overlap(1) == 1    # the thread's own level again
