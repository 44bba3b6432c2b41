"""Prompt portions of the Llama / Qwen3 decoders through the native call against the loop over
the layers' modules: the same bits, and every module that a program has changed is called.  Steps
whose inputs were staged behind the step before against steps that stage their own."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

VOCAB = 512


def engine(layout, qk_norm, bias, ff=1024, hidden=512, layers=2):
    from fastkernels_b200.candidate.L4.llama import LlamaConfig
    from fastkernels_b200.engine import DecodeEngine
    cfg = LlamaConfig(hidden_size=hidden, intermediate_size=ff, num_hidden_layers=layers,
                      num_attention_heads=4, num_key_value_heads=2, head_dim=128, vocab_size=VOCAB,
                      max_position_embeddings=1024, rope_theta=1e4, qkv_bias=bias, qk_norm=qk_norm,
                      kv_block_size=16 if layout == "HND" else 64, kv_layout=layout)
    eng = DecodeEngine(cfg, max_num_seqs=4, max_model_len=1024, num_kv_blocks=300, seed=3,
                       init_scale=0.05)
    g = torch.Generator(device="cuda").manual_seed(5)
    with torch.no_grad():
        for n, p in eng.model.named_parameters():
            if "norm" in n or n.endswith("bias"):
                p.normal_(1.0 if "norm" in n else 0.0, 0.2, generator=g)
    return eng


def logits(eng, portions):
    """Prompts in portions of given lengths; the last logits and the pools after them."""
    rs = np.random.RandomState(1)
    seqs = [eng.open_sequence() for _ in portions]
    out = []
    for step in range(max(map(len, portions))):
        part = [(s, rs.randint(0, VOCAB, p[step]).tolist()) for s, p in zip(seqs, portions)
                if step < len(p)]
        out += eng.feed(part)
    pool = eng.kv_cache.clone()
    for s in reversed(seqs):
        eng.finish(s)
    return torch.cat(out), pool


@pytest.mark.parametrize("layout,qk_norm,bias", [("NHD", True, False), ("HND", False, True),
                                                 ("HND", True, True)])
@pytest.mark.parametrize("portions", [[[1]], [[17, 3], [64]], [[130, 127]], [[300, 2], [257]]])
def test_same_bits_as_the_modules(layout, qk_norm, bias, portions, monkeypatch):
    from fastkernels_b200.candidate.L4 import llama
    # one launch of gate/up and SiLU for few rows (ff 9600), and the sizes without one
    for ff in (1024, 9600):
        eng = engine(layout, qk_norm, bias, ff=ff)
        calls, native = [], llama.PromptRun.layer

        def counted(*a):
            r = native(*a)
            calls.append(r is not None)
            return r
        with monkeypatch.context() as m:
            m.setattr(llama.PromptRun, "layer", counted)
            got = logits(eng, portions)
        rows = [sum(p[i] for p in portions if i < len(p)) for i in range(max(map(len, portions)))]
        assert calls == [ff == 9600 or n > 256 for n in rows for _ in range(2)]
        eng.kv_cache.zero_()
        with monkeypatch.context() as m:
            m.setattr(llama.PromptRun, "begin", lambda *a: None)
            want = logits(eng, portions)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


def _hook(eng, seen):
    return eng.model.model.layers[1].mlp.down_proj.register_forward_hook(
        lambda *a: seen.append(1))


def _forward(eng, seen):
    m = eng.model.model.layers[0].self_attn.q_norm
    m.forward = lambda *a, f=m.forward: (seen.append(1), f(*a))[1]
    # q/k norms run inside the fused chain, which a replaced forward has never stopped
    eng.model.model.layers[0].self_attn.fused = False


def _class(eng, seen):
    m = eng.model.model.layers[0].post_attention_layernorm
    m.__class__ = type("Mine", (type(m),), {
        "forward": lambda self, *a: (seen.append(1), super(type(self), self).forward(*a))[1]})


def _operator(eng, seen, monkeypatch):
    from fastkernels_b200 import ops
    f = ops.qkv_rope_store
    monkeypatch.setattr(ops, "qkv_rope_store", lambda *a, **k: (seen.append(1), f(*a, **k))[1])


@pytest.mark.parametrize("change", [_hook, _forward, _class, _operator])
def test_what_a_program_changed_is_called(change, monkeypatch):
    eng, seen = engine("NHD", True, False, ff=9600), []
    want = logits(eng, [[40]])[0]
    change(eng, seen, *([monkeypatch] if change is _operator else []))
    got = logits(eng, [[40]])[0]
    assert seen
    # the op-by-op chain rounds between norm and rotation
    torch.testing.assert_close(got, want, atol=3e-2 * float(want.std()), rtol=3e-2) \
        if change is _forward else torch.testing.assert_close(got, want, atol=0.0, rtol=0.0)


@pytest.mark.parametrize("graphs", [[], [4]])
def test_steps_staged_ahead(graphs, monkeypatch):
    """Tokens that the program replaces, sequences that come and go, another stream, steps that
    do not wait, and prompts in between: the same tokens as without staging ahead."""
    from fastkernels_b200 import engine as E

    def run(ahead):
        monkeypatch.setattr(E, "_NO_PREPARE_AHEAD", not ahead)
        eng, rs, out = engine("HND", True, False, ff=9600), np.random.RandomState(2), []
        if graphs:
            eng.capture_cudagraph(graphs)
        eng.prefill([rs.randint(0, VOCAB, n).tolist() for n in (15, 33, 7)])
        staged = 0
        for i in range(24):
            if i == 5:
                eng.seqs[1].last_token = 11
            if i == 8:
                eng.finish(eng.seqs[0])
            if i == 10:
                eng.prefill([rs.randint(0, VOCAB, 20).tolist()])
            if i == 16:
                s = eng.open_sequence()
                eng.feed([(s, [1, 2, 3])])
                out.append(eng.feed([(s, [4])])[0])
                eng.finish(s)
            staged += eng._staged_ahead is not None and eng._ahead is not None
            if i == 13:
                with torch.cuda.stream(torch.cuda.Stream()):
                    out.append(torch.from_numpy(eng.step()))
                    torch.cuda.current_stream().synchronize()
            elif i == 19:
                eng.step(sync=False)
                torch.cuda.synchronize()
                for q, t in zip(eng.seqs, eng.host_np["token_ids"]):
                    q.last_token = int(t)
            else:
                out.append(torch.from_numpy(eng.step()))
        assert eng.device_status() == 0
        return out, staged
    got, staged = run(True)
    want, none = run(False)
    assert staged >= 16 and none == 0
    assert all(torch.equal(a, b) for a, b in zip(got, want))
