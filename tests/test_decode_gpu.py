"""KV-cache greedy decoding against the numpy oracle (full-prefix recomputation), through the
C-ABI: prefill logits, token-by-token agreement, cache consistency (prefill + steps == longer
prefill), limits and errors."""
import numpy as np
import pytest
import torch

from oracle import model as om

pytestmark = pytest.mark.gpu
F32 = np.float32

CASES = [
    dict(vocab_size=320, hidden_size=128, intermediate_size=256, num_hidden_layers=2, num_attention_heads=4,
         num_key_value_heads=2, head_dim=64, rms_norm_eps=1e-5, rope_theta=10000.0),
    dict(vocab_size=384, hidden_size=128, intermediate_size=256, num_hidden_layers=2, num_attention_heads=2,
         num_key_value_heads=1, head_dim=128, rms_norm_eps=1e-6, rope_theta=1000000.0, qk_norm=True),
]


def build(kw, seed):
    from emberlm_b200 import engine as E
    ocfg, ecfg = om.LlamaConfig(**kw), E.make_config(**kw)
    params = om.init_params(ocfg, seed=seed, std=0.08)
    rng = np.random.default_rng(seed + 1)
    for k in params:
        if params[k].ndim == 1:
            params[k] = (params[k] + rng.uniform(-0.2, 0.2, params[k].shape)).astype(F32)
    return ocfg, ecfg, params


@pytest.mark.parametrize("kw", CASES)
def test_greedy_decode_matches_oracle(kw):
    from emberlm_b200 import engine as E
    ocfg, ecfg, params = build(kw, 41)
    prompt = np.random.default_rng(5).integers(0, ocfg.vocab_size, size=19)
    dec = E.Decoder(ecfg, max_seq_len=64)
    dec.load_parameters(params)
    got = dec.generate(prompt, 12).cpu().tolist()
    want, margins = om.greedy_generate(params, ocfg, prompt, 12, acc=np.float64)
    # tokens must agree wherever the oracle's top-2 logit margin is larger than TF32 noise; after a
    # (legitimate) near-tie divergence the continuations differ, so stop comparing there
    for i, (g, w, m) in enumerate(zip(got, want, margins)):
        if g != w:
            assert m < 2e-3, (i, g, w, m)
            break
    assert len(got) == 12
    # logits of the last processed position against the oracle on the same prefix
    prefix = np.concatenate([prompt, np.array(got[:-1], dtype=np.int64)])
    ref = om.forward_logits(params, ocfg, prefix[None, :], acc=np.float64)[0, -1]
    z = dec.last_logits().cpu().numpy()
    assert np.abs(z - ref).max() <= 5e-3 * max(np.abs(ref).max(), 1.0)


def test_cached_steps_equal_longer_prefill():
    from emberlm_b200 import engine as E
    ocfg, ecfg, params = build(CASES[0], 43)
    prompt = np.random.default_rng(6).integers(0, ocfg.vocab_size, size=33)
    dec = E.Decoder(ecfg, max_seq_len=80)
    dec.load_parameters(params)
    toks = dec.generate(prompt, 9).cpu().numpy()
    z_cached = dec.last_logits().cpu().numpy().copy()
    longer = np.concatenate([prompt, toks[:-1]])
    dec2 = E.Decoder(ecfg, max_seq_len=80, params=dec.params)
    dec2.generate(longer, 1)
    z_prefill = dec2.last_logits().cpu().numpy()
    # tests/test_integration_kvcache.cpp: prefill + decode == full forward within 5e-4 (fp32 there;
    # TF32 projections in the prefill here)
    assert np.abs(z_cached - z_prefill).max() <= 5e-3 * max(np.abs(z_prefill).max(), 1.0)


def test_decode_limits_and_errors():
    from emberlm_b200 import engine as E
    ocfg, ecfg, params = build(CASES[0], 45)
    dec = E.Decoder(ecfg, max_seq_len=24)
    dec.load_parameters(params)
    assert dec.generate(np.arange(20), 100).numel() == 5      # stops at max_seq_len: 24 - 20 cache positions + the token that needs none
    with pytest.raises(RuntimeError):
        dec.generate([], 4)
    with pytest.raises(RuntimeError):
        dec.generate(np.arange(24), 1)                        # prompt must leave room for one token


@pytest.mark.parametrize("kw", CASES)
def test_portions_of_given_tokens(kw):
    """extend(): a prompt cut anywhere gives the logits of the whole prompt, also after a reset."""
    from emberlm_b200 import engine as E
    ocfg, ecfg, params = build(kw, 47)
    t = np.random.default_rng(8).integers(0, ocfg.vocab_size, size=30)
    want = om.forward_logits(params, ocfg, t[None, :], acc=np.float64)[0]
    dec = E.Decoder(ecfg, max_seq_len=32)
    dec.load_parameters(params)
    for sizes in ([30], [17, 13], [1, 1, 28], [29, 1]):
        dec.reset()
        got, at = [], 0
        for n in sizes:
            got.append(dec.extend(t[at:at + n], range(n)).cpu().numpy())
            at += n
        assert np.abs(np.concatenate(got) - want).max() <= 5e-3 * max(np.abs(want).max(), 1.0), sizes
    assert np.abs(dec.step(int(t[0])).cpu().numpy() - om.forward_logits(
        params, ocfg, np.append(t, t[0])[None, :], acc=np.float64)[0, -1]).max() <= 5e-3 * max(np.abs(want).max(), 1.0)


@pytest.mark.parametrize("case, context", [(0, 190), (0, 200), (0, 700), (1, 94), (1, 101), (1, 510)])
def test_token_pass_over_key_ranges(case, context):
    """The token kernel on both sides of the switch from one key range per head to several (192 positions at head
    size 64, 96 at 128) and with many ranges: logits against the oracle over the same prefix, for a burst of
    greedy tokens and for single chosen ones. fp32 sums over at most 700 keys behind a TF32 prompt (2^-11 per
    operand, two layers): 5e-3 of the largest logit, as the tests above."""
    from emberlm_b200 import engine as E
    ocfg, ecfg, params = build(CASES[case], 51)
    prompt = np.random.default_rng(context).integers(0, ocfg.vocab_size, size=context)
    dec = E.Decoder(ecfg, max_seq_len=context + 8)
    dec.load_parameters(params)
    got = dec.generate(prompt, 6).cpu().numpy()
    prefix = np.concatenate([prompt, got[:-1]])
    ref = om.forward_logits(params, ocfg, prefix[None, :], acc=np.float64)[0, -1]
    assert np.abs(dec.last_logits().cpu().numpy() - ref).max() <= 5e-3 * max(np.abs(ref).max(), 1.0)
    dec.reset()
    dec.extend(prompt)
    for token in got[:-1]:
        z = dec.step(int(token)).cpu().numpy()
    assert np.abs(z - ref).max() <= 5e-3 * max(np.abs(ref).max(), 1.0)


@pytest.mark.parametrize("one_launch", [True, False])
@pytest.mark.parametrize("kw", CASES)
def test_ids_outside_the_vocabulary(kw, one_launch, monkeypatch):
    """Behind a prompt too such an id is an embedding row of zeros and is counted, by the token kernel as by the kernel
    per phase. The oracle has the row of zeros behind the vocabulary; tolerance as above."""
    import ctypes as C

    from emberlm_b200 import engine as E
    monkeypatch.setenv("CTDK_DECODE_PERSISTENT", "1" if one_launch else "0")
    ocfg, ecfg, params = build(kw, 53)
    V = ocfg.vocab_size
    wider = dict(params)
    wider["model.embed_tokens.weight"] = np.concatenate([params["model.embed_tokens.weight"], np.zeros((1, ocfg.hidden_size), F32)])
    t = np.random.default_rng(8).integers(0, V, size=30)
    given = t.copy()
    given[[20, 22, 29]] = [-1, V, 1 << 40]   # inside a portion, first of one, a lone token
    want = om.forward_logits(wider, om.LlamaConfig(**dict(kw, vocab_size=V + 1)), np.where((given < 0) | (given >= V), V, given)[None, :],
                             acc=np.float64)[0, :, :V]
    dec = E.Decoder(ecfg, max_seq_len=40)
    dec.load_parameters(params)
    counts = []
    for lo, hi in ((0, 17), (17, 22), (22, 29), (29, 30)):
        words = (C.c_int * 4)()
        z = dec.extend(given[lo:hi], want=range(hi - lo)).cpu().numpy()
        E.lib.check(E._L.ctdk_device_status(dec.stream.cuda_stream, words))
        counts.append(words[2])
        assert np.abs(z - want[lo:hi]).max() <= 5e-3 * max(np.abs(want).max(), 1.0), (lo, hi)
    assert [b - a for a, b in zip(counts, counts[1:])] == [1, 1, 1]


@pytest.mark.parametrize("one_launch", [True, False])
def test_decoders_of_different_sizes_take_turns(one_launch, monkeypatch):
    """Decoders share the kernels of their head size, and with them the limit of dynamic shared memory: a small one between
    two passes of a large one leaves the large one's limit alone."""
    from emberlm_b200 import engine as E
    monkeypatch.setenv("CTDK_DECODE_PERSISTENT", "1" if one_launch else "0")
    made = []
    for inter, max_seq in ((8192, 8192), (256, 64)):   # 32 KB of staged vector against 18, 3 KB of scores against 1
        ocfg, ecfg, params = build(dict(CASES[0], intermediate_size=inter), 55)
        dec = E.Decoder(ecfg, max_seq_len=max_seq)
        dec.load_parameters(params)
        made.append((dec, ocfg, params))
    t = np.random.default_rng(9).integers(0, 320, size=12)
    for dec, _, _ in made:
        dec.extend(t[:8])
    for n in (8, 9, 10):
        for dec, ocfg, params in made:
            ref = om.forward_logits(params, ocfg, t[None, :n + 1], acc=np.float64)[0, -1]
            assert np.abs(dec.step(int(t[n])).cpu().numpy() - ref).max() <= 5e-3 * max(np.abs(ref).max(), 1.0)


# Shares of rows that differ from CTA to CTA (576 and 1 000 over 148), a warp with several units; two passes over the heads
# of a key, the second full and partial; rows of several loads a warp, and (20 480) parts longer than one batch of loads.
WIDE = [
    dict(vocab_size=1000, hidden_size=576, intermediate_size=1536, num_hidden_layers=2, num_attention_heads=9,
         num_key_value_heads=3, head_dim=64, rms_norm_eps=1e-5, rope_theta=10000.0),
    dict(vocab_size=1001, hidden_size=1096, intermediate_size=4104, num_hidden_layers=2, num_attention_heads=8,
         num_key_value_heads=1, head_dim=128, rms_norm_eps=1e-6, rope_theta=1000000.0, qk_norm=True),
    dict(vocab_size=640, hidden_size=2048, intermediate_size=8192, num_hidden_layers=2, num_attention_heads=12,
         num_key_value_heads=2, head_dim=64, rms_norm_eps=1e-5, rope_theta=10000.0),
    dict(vocab_size=320, hidden_size=128, intermediate_size=20480, num_hidden_layers=2, num_attention_heads=2,
         num_key_value_heads=1, head_dim=128, rms_norm_eps=1e-5, rope_theta=10000.0),
]


@pytest.mark.parametrize("one_launch", [True, False])
@pytest.mark.parametrize("case", range(len(WIDE)))
def test_sizes_of_either_token_path(case, one_launch, monkeypatch):
    """Greedy and chosen tokens of the token kernel and of the kernel per phase against the oracle; tolerance as above
    (weights are drawn so that a layer keeps the size of what passes through it)."""
    from emberlm_b200 import engine as E
    monkeypatch.setenv("CTDK_DECODE_PERSISTENT", "1" if one_launch else "0")
    kw = WIDE[case]
    ocfg, ecfg = om.LlamaConfig(**kw), E.make_config(**kw)
    params = om.init_params(ocfg, seed=61, std=0.5 * kw["hidden_size"] ** -0.5)
    prompt = np.random.default_rng(case).integers(0, ocfg.vocab_size, size=21)
    dec = E.Decoder(ecfg, max_seq_len=40)
    dec.load_parameters(params)
    if not one_launch and kw["intermediate_size"] > 12288:   # the kernel per phase stages a vector in 48 KB
        with pytest.raises(E.lib.CtdkError):
            dec.generate(prompt, 6)
        return
    got = dec.generate(prompt, 6).cpu().numpy()
    prefix = np.concatenate([prompt, got[:-1]])
    ref = om.forward_logits(params, ocfg, prefix[None, :], acc=np.float64)[0, -6:]
    limit = 5e-3 * max(np.abs(ref).max(), 1.0)
    assert np.abs(dec.last_logits().cpu().numpy() - ref[-1]).max() <= limit
    dec.reset()
    dec.extend(prompt)
    for token, want in zip(got[:-1], ref[1:]):
        assert np.abs(dec.step(int(token)).cpu().numpy() - want).max() <= limit


@pytest.mark.parametrize("case, context, inter", [(0, 9, 256), (1, 12, 256), (0, 30, 256), (1, 21, 26048), (0, 33, 13056)])
def test_token_pass_over_few_keys_and_long_rows(case, context, inter):
    """Tokens on both sides of the first cut of the keys into ranges (16 keys), and rows that pass through the weight ring in
    many pieces with one place for the vector (26 048 floats) and with two; tolerance as above."""
    from emberlm_b200 import engine as E
    ocfg, ecfg, params = build(dict(CASES[case], intermediate_size=inter), 63)
    prompt = np.random.default_rng(context).integers(0, ocfg.vocab_size, size=context)
    dec = E.Decoder(ecfg, max_seq_len=context + 12)
    dec.load_parameters(params)
    got = dec.generate(prompt, 10).cpu().numpy()
    ref = om.forward_logits(params, ocfg, np.concatenate([prompt, got[:-1]])[None, :], acc=np.float64)[0, -10:]
    limit = 5e-3 * max(np.abs(ref).max(), 1.0)
    assert np.abs(dec.last_logits().cpu().numpy() - ref[-1]).max() <= limit
    dec.reset()
    dec.extend(prompt)
    for token, want in zip(got[:-1], ref[1:]):
        assert np.abs(dec.step(int(token)).cpu().numpy() - want).max() <= limit


@pytest.mark.parametrize("heads, kv_heads, dim, contexts", [(48, 48, 64, (190, 195, 390)), (96, 16, 64, (570, 640)), (48, 48, 128, (94, 100, 290)),
                                                            (96, 24, 128, (190, 300))])
def test_ranges_of_several_tiles(heads, kv_heads, dim, contexts):
    """Many key/value heads leave few CTAs for each, so that a range of keys is longer than one and two tiles (32 or 64 keys, of
    128 values half as many), also with more query heads than are taken at once; tolerance as above."""
    from emberlm_b200 import engine as E
    kw = dict(CASES[0], num_hidden_layers=1, num_attention_heads=heads, num_key_value_heads=kv_heads, head_dim=dim)
    ocfg, ecfg, params = build(kw, 65)
    prompt = np.random.default_rng(heads).integers(0, ocfg.vocab_size, size=max(contexts) + 3)
    ref = om.forward_logits(params, ocfg, prompt[None, :], acc=np.float64)[0]
    dec = E.Decoder(ecfg, max_seq_len=max(contexts) + 8)
    dec.load_parameters(params)
    for context in contexts:
        dec.reset()
        dec.extend(prompt[:context])
        for i in range(context, context + 3):
            assert np.abs(dec.step(int(prompt[i])).cpu().numpy() - ref[i]).max() <= 5e-3 * max(np.abs(ref[i]).max(), 1.0), (context, i)


@pytest.mark.parametrize("gate", [-87.5, -88.0, -88.5, -40.0])
def test_gates_at_the_edge_of_the_range(gate):
    """Gates whose 1 + exp(-gate) lies between 2^126 and 2^128, where an approximate division gives zero, against up values that
    make a product of ordinary size of it; tolerance as above."""
    from emberlm_b200 import engine as E
    ocfg, ecfg, params = build(dict(CASES[0], num_hidden_layers=1), 67)
    hid, inter, p = ocfg.hidden_size, 256, "model.layers.0."
    rng = np.random.default_rng(68)
    params["model.embed_tokens.weight"][7] = 1.0   # the token's row, which reaches the gate as it is
    params[p + "post_attention_layernorm.weight"][:] = 1.0
    params[p + "self_attn.o_proj.weight"][:] = 0.0
    params[p + "mlp.gate_proj.weight"][:] = gate / hid
    params[p + "mlp.up_proj.weight"][:] = (rng.uniform(-1.0, 1.0, (inter, 1)) * (1.0 + np.exp(-gate)) / -gate / hid).astype(F32)
    dec = E.Decoder(ecfg, max_seq_len=8)
    dec.load_parameters(params)
    dec.extend([7])
    got = dec.step(7).cpu().numpy()
    ref = om.forward_logits(params, ocfg, np.array([[7, 7]]), acc=np.float64)[0, 1]
    silent = dict(params, **{p + "mlp.down_proj.weight": 0.0 * params[p + "mlp.down_proj.weight"]})
    quiet = om.forward_logits(silent, ocfg, np.array([[7, 7]]), acc=np.float64)[0, 1]
    limit = 5e-3 * max(np.abs(ref).max(), 1.0)
    assert np.abs(quiet - ref).max() > 20 * limit
    assert np.abs(got - ref).max() <= limit


@pytest.mark.parametrize("hid, inter, heads, kv_heads, dim, contexts", [(128, 26048, 48, 48, 64, (10, 190, 390)), (128, 20480, 96, 24, 128, (190, 300)),
                                                                       (1024, 31616, 16, 2, 128, (9, 600)), (128, 33024, 4, 2, 64, (9, 190)),
                                                                       (128, 45056, 4, 2, 64, (9, 190))])
def test_tiles_over_the_place_of_the_vector(hid, inter, heads, kv_heads, dim, contexts):
    """Rows so long that the attention's tiles lie over the second place of the vector, that there is one place only, or that the ring
    takes pieces of 128 and 64 chunks, with ranges of one and several tiles; tolerance as above (weights are drawn so that a layer keeps the size of what passes through it)."""
    from emberlm_b200 import engine as E
    kw = dict(CASES[0], hidden_size=hid, intermediate_size=inter, num_attention_heads=heads, num_key_value_heads=kv_heads, head_dim=dim)
    ocfg, ecfg = om.LlamaConfig(**kw), E.make_config(**kw)
    params = om.init_params(ocfg, seed=69, std=0.5 * hid ** -0.5)
    prompt = np.random.default_rng(heads).integers(0, ocfg.vocab_size, size=max(contexts) + 3)
    ref = om.forward_logits(params, ocfg, prompt[None, :], acc=np.float64)[0]
    dec = E.Decoder(ecfg, max_seq_len=max(contexts) + 8)
    dec.load_parameters(params)
    for context in contexts:
        dec.reset()
        dec.extend(prompt[:context])
        for i in range(context, context + 3):
            assert np.abs(dec.step(int(prompt[i])).cpu().numpy() - ref[i]).max() <= 5e-3 * max(np.abs(ref[i]).max(), 1.0), (context, i)


@pytest.mark.parametrize("heads, kv_heads, dim", [(32, 1, 128), (5, 1, 64), (9, 3, 64), (2, 2, 128), (17, 1, 64), (96, 1, 128), (10, 2, 64)])
def test_groups_of_query_heads(heads, kv_heads, dim):
    """Groups of one, two, three and more query heads, which share the walk over the keys, with as many blocks of 32 columns as a
    range's warps, fewer and more; tolerance as above."""
    from emberlm_b200 import engine as E
    kw = dict(CASES[0], num_hidden_layers=1, num_attention_heads=heads, num_key_value_heads=kv_heads, head_dim=dim)
    ocfg, ecfg, params = build(kw, 71)
    prompt = np.random.default_rng(heads).integers(0, ocfg.vocab_size, size=1400)
    ref = om.forward_logits(params, ocfg, prompt[None, :], acc=np.float64)[0]
    dec = E.Decoder(ecfg, max_seq_len=1408)
    dec.load_parameters(params)
    for context in (1, 15, 70, 700, 1397):
        dec.reset()
        dec.extend(prompt[:context])
        for i in range(context, context + 3):
            assert np.abs(dec.step(int(prompt[i])).cpu().numpy() - ref[i]).max() <= 5e-3 * max(np.abs(ref[i]).max(), 1.0), (context, i)
