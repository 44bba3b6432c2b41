"""Whole decode step on the GPU against the CPU oracle: logits within tolerance
and greedy tokens identical over 32 steps (tiny Qwen3-style decoder)."""
import numpy as np
import pytest
import torch

import cases
from oracle import decode_oracle as O

pytestmark = pytest.mark.gpu


def make_engine(cfg_d, w, lens, block=64, eager=False, fused=True, graphs=(), layout="NHD",
                decode_block=False):
    from fastkernels_b200.candidate.L4.llama import LlamaConfig
    from fastkernels_b200.engine import DecodeEngine
    cfg = LlamaConfig(hidden_size=cfg_d["hidden"], intermediate_size=cfg_d["ffn"],
                      num_hidden_layers=cfg_d["num_layers"],
                      num_attention_heads=cfg_d["num_heads"],
                      num_key_value_heads=cfg_d["num_kv_heads"], head_dim=cfg_d["head_dim"],
                      vocab_size=cfg_d["vocab"], max_position_embeddings=cfg_d["max_pos"],
                      rms_norm_eps=cfg_d["eps"], rope_theta=cfg_d["theta"],
                      qk_norm=cfg_d["qk_norm"], kv_block_size=block,
                      fused_attention_prologue=fused, kv_layout=layout,
                      decode_block=decode_block)
    nb = sum((L + 40 + block - 1) // block for L in lens) + 2
    eng = DecodeEngine(cfg, max_num_seqs=len(lens), max_model_len=max(lens) + 64,
                       num_kv_blocks=nb, enforce_eager=eager)
    eng.load_full_weights(w)
    if graphs:
        eng.capture_cudagraph(graphs)
    return eng


def seed_context(eng, lens, seed):
    """Random K/V for the first L-1 positions of every sequence, written both to
    the GPU pool and to numpy caches for the oracle."""
    cfg = eng.config
    rs = np.random.RandomState(seed)
    first = rs.randint(0, cfg.vocab_size, size=len(lens))
    eng.add_sequences(lens, first)
    nb, bs = eng.num_kv_blocks, eng.block_size
    shape = (nb, bs, cfg.num_key_value_heads, cfg.head_dim)
    hnd = cfg.kv_layout == "HND"
    kcs, vcs = [], []
    for li in range(cfg.num_hidden_layers):
        k = cases.randn_bf16(rs, shape, 0.5)          # the oracle always sees NHD
        v = cases.randn_bf16(rs, shape, 0.5)
        eng.kv_cache[0, li].copy_(torch.from_numpy(k.transpose(0, 2, 1, 3) if hnd else k))
        eng.kv_cache[1, li].copy_(torch.from_numpy(v.transpose(0, 2, 1, 3) if hnd else v))
        kcs.append(k)
        vcs.append(v)
    return first, kcs, vcs


def bf16_ulp(x):
    return 2.0 ** (np.floor(np.log2(max(abs(float(x)), 1e-30))) - 7)


def lockstep(cfg_d, w, eng, first, kcs, vcs, steps):
    """Run engine and oracle side by side for `steps` greedy steps.  The oracle is
    fed the ENGINE's tokens (so both walk the same trajectory and every step is
    checked, not only those before a first divergence) and the engine's own
    host-side schedule.  Returns (tokens equal, near ties, first-step logits)."""
    cs = O.bf16_round(eng.model.model.rotary_emb.cos_sin_cache.cpu().numpy())
    dec = O.DecoderOracle(cfg_d, w, cs)
    ids = np.array(first)
    bs = eng.block_size
    equal = near = 0
    first_logits = None
    for step in range(steps):
        lens = np.array([s.num_tokens for s in eng.seqs])
        got = eng.step(sync=True)
        tables = [list(s.block_table) for s in eng.seqs]      # after page appends
        cols = max(len(t) for t in tables)
        bt = np.full((len(lens), cols), -1, np.int32)
        for i, t in enumerate(tables):
            bt[i, :len(t)] = t
        slots = np.array([tables[i][(L - 1) // bs] * bs + (L - 1) % bs
                          for i, L in enumerate(lens)])
        logits, want = dec.step(ids, lens - 1, kcs, vcs, slots, lens.astype(np.int32), bt)
        if first_logits is None:
            first_logits = logits
        for i in range(len(lens)):
            if got[i] == want[i]:
                equal += 1
                continue
            # a different token is acceptable only at a near tie of the oracle's
            # bf16 logits: the engine's choice within 2 bf16 steps of the maximum
            gap = float(logits[i, want[i]] - logits[i, got[i]])
            assert gap <= 2 * bf16_ulp(logits[i, want[i]]), (
                f"step {step} seq {i}: engine token {got[i]} (oracle logit "
                f"{logits[i, got[i]]}) vs oracle argmax {want[i]} ({logits[i, want[i]]})")
            near += 1
        ids = got.copy()
    return equal, near, first_logits


# "*_block": everything between two attention calls as one persistent launch
# (fk_decode_block); the other modes run one kernel per op, "unfused" as the
# reference's op-by-op chain on the L1 ops
@pytest.mark.parametrize("mode", ["eager_fused", "eager_unfused", "graph", "graph_hnd16",
                                  "eager_unfused_hnd16", "eager_block", "graph_block",
                                  "graph_block_hnd16"])
def test_greedy_tokens_match_oracle_32_steps(mode):
    cfg_d = cases.TINY_QWEN3
    w = cases.decoder_weights(5, cfg_d, scale=0.05)
    lens = [1, 30, 64, 65, 127, 200]
    hnd = mode.endswith("hnd16")
    eng = make_engine(cfg_d, w, lens, eager=not mode.startswith("graph"),
                      fused=not mode.startswith("eager_unfused"),
                      graphs=(len(lens),) if mode.startswith("graph") else (),
                      block=16 if hnd else 64, layout="HND" if hnd else "NHD",
                      decode_block="block" in mode)
    first, kcs, vcs = seed_context(eng, lens, 17)
    equal, near, _ = lockstep(cfg_d, w, eng, first, kcs, vcs, 32)
    assert int(eng.status.item()) == 0
    total = 32 * len(lens)
    assert equal + near == total
    # identical tokens except at bf16 near-ties of the top two logits, which a
    # random-init model produces now and then
    assert equal >= 0.95 * total, (equal, near)
    # the KV cache the engine built matches the oracle's.  Layer 0 comes from one
    # projection (per-op tolerance); deeper layers inherit the rounding of a whole
    # layer chain, so they get the harness rule: >= 99 % inside 2e-2, none far off
    for li in range(cfg_d["num_layers"]):
        for which, ref in ((0, kcs[li]), (1, vcs[li])):
            g = eng.kv_cache[which, li].float().cpu().numpy()
            if hnd:
                g = g.transpose(0, 2, 1, 3)
            if li == 0:
                np.testing.assert_allclose(g, ref, atol=2e-2, rtol=2e-2)
            else:
                inside = np.abs(g - ref) <= 2e-2 + 2e-2 * np.abs(ref)
                assert inside.mean() >= 0.999 and np.abs(g - ref).max() <= 0.125


def test_logits_within_tolerance_first_step():
    """Whole-step logits: >= 99 % of the elements inside atol/rtol 2e-2 (the
    reference harness' acceptance rule, fastkernels/bench.py:141-156) and no
    element further than 4 bf16 steps."""
    cfg_d = cases.TINY_QWEN3
    w = cases.decoder_weights(6, cfg_d, scale=0.05)
    lens = [5, 300]
    eng = make_engine(cfg_d, w, lens, eager=True)
    first, kcs, vcs = seed_context(eng, lens, 3)
    _, _, ref = lockstep(cfg_d, w, eng, first, kcs, vcs, 1)
    got = eng.graph_vars["lm_logits"][:2].float().cpu().numpy()
    inside = np.abs(got - ref) <= 2e-2 + 2e-2 * np.abs(ref)
    assert inside.mean() >= 0.99, inside.mean()
    assert np.abs(got - ref).max() <= 0.0625


def test_graph_replay_equals_eager_bitwise():
    cfg_d = cases.TINY_QWEN3
    w = cases.decoder_weights(7, cfg_d, scale=0.05)
    lens = [3, 64, 129]
    outs = []
    for eager in (True, False):
        eng = make_engine(cfg_d, w, lens, eager=eager, graphs=() if eager else (4,))
        seed_context(eng, lens, 9)
        toks = eng.decode(8)
        outs.append((toks, eng.graph_vars["lm_logits"][:3].clone()))
    assert np.array_equal(outs[0][0], outs[1][0])
    assert torch.equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("mode", ["paged", "dense", "chunked", "paged_hnd16"])
def test_prefill_then_decode_matches_oracle(mode):
    """Prompts go through engine.prefill (whole, over dense K/V, or in chunks of 48
    tokens over the pages), then 8 decode steps: first tokens, the KV pages the
    prefill wrote and the following greedy tokens against the oracle."""
    cfg_d = cases.TINY_QWEN3
    w = cases.decoder_weights(8, cfg_d, scale=0.05)
    rs = np.random.RandomState(23)
    plens = [1, 17, 64, 130, 201]
    prompts = [rs.randint(0, cfg_d["vocab"], size=n).tolist() for n in plens]
    hnd = mode.endswith("hnd16")
    block = 16 if hnd else 64
    eng = make_engine(cfg_d, w, [n + 1 for n in plens], eager=True, block=block,
                      layout="HND" if hnd else "NHD")
    got = eng.prefill(prompts, chunk_tokens=48 if mode == "chunked" else None,
                      use_block_tables=mode != "dense")
    assert int(eng.status.item()) == 0

    cs = O.bf16_round(eng.model.model.rotary_emb.cos_sin_cache.cpu().numpy())
    dec = O.DecoderOracle(cfg_d, w, cs)
    shape = (eng.num_kv_blocks, block, cfg_d["num_kv_heads"], cfg_d["head_dim"])
    kcs = [np.zeros(shape, np.float32) for _ in range(cfg_d["num_layers"])]
    vcs = [np.zeros(shape, np.float32) for _ in range(cfg_d["num_layers"])]
    cu = np.concatenate([[0], np.cumsum(plens)]).astype(np.int32)
    slots = np.concatenate([[s.block_table[t // block] * block + t % block for t in range(n)]
                            for s, n in zip(eng.seqs, plens)])
    ids = np.concatenate(prompts)
    pos = np.concatenate([np.arange(n) for n in plens])
    logits, want = dec.prefill(ids, pos, cu, kcs, vcs, slots)
    for i in range(len(plens)):
        if got[i] != want[i]:
            gap = float(logits[i, want[i]] - logits[i, got[i]])
            assert gap <= 2 * bf16_ulp(logits[i, want[i]]), (i, got[i], want[i])
    for li in range(cfg_d["num_layers"]):
        for which, ref in ((0, kcs[li]), (1, vcs[li])):
            g = eng.kv_cache[which, li].float().cpu().numpy()
            if hnd:
                g = g.transpose(0, 2, 1, 3)
            inside = np.abs(g - ref) <= 2e-2 + 2e-2 * np.abs(ref)
            assert inside.mean() >= 0.999 and np.abs(g - ref).max() <= 0.125
    # hand-over to decode: the engine continues from its own first tokens
    equal, near, _ = lockstep(cfg_d, w, eng, got, kcs, vcs, 8)
    assert equal + near == 8 * len(plens) and equal >= 0.9 * 8 * len(plens)


@pytest.mark.parametrize("graphs", [(), (3,)])
def test_step_and_feed_raise_on_device_status(graphs):
    """A status bit that a kernel left makes the step whose tokens come back raise, also from a
    replayed graph; it is cleared, and the engine goes on."""
    from fastkernels_b200 import ops
    cfg_d = cases.TINY_QWEN3
    w = cases.decoder_weights(5, cfg_d, scale=0.05)
    lens = [30, 64, 127]
    eng = make_engine(cfg_d, w, lens, graphs=graphs)
    seed_context(eng, lens, 17)
    eng.step()
    for word in (eng.status, ops.default_status("cuda")):
        word.fill_(4)
        with pytest.raises(RuntimeError, match="device status word 4"):
            eng.step()
        assert len(eng.step()) == 3 and eng.device_status() == 0
    eng.finish(eng.seqs[-1])
    s = eng.open_sequence()
    for tokens in ([1, 2, 3], [4]):
        eng.status.fill_(1)
        with pytest.raises(RuntimeError, match="device status word 1"):
            eng.feed([(s, tokens)])
        assert eng.feed([(s, tokens)])[0].shape[0] == 1 and eng.device_status() == 0
