"""Prompt prefill on the tensor cores against the decode path it replaces.

The reference feeds a prompt token by token through the decode path (crates/inferi-chat/src/chat_llama2.rs:137-155); that loop
is the anchor: after `prefill` the logits of the last prompt position must agree with the loop's within 2e-2 and the greedy
tokens that follow must be identical."""
import numpy as np
import pytest
import torch

import oracle
from helpers import LOGITS_MAX_ABS
from inferi_b200 import quant
from inferi_b200.llama2 import LLAMA_3_2_1B, Llama2, Llama2Config, Llama2Weights, Q4_K_M, synth_weights, weights_to_host
from inferi_b200.ops import InferiError

pytestmark = pytest.mark.gpu


def loop_vs_prefill(backend, cfg, dev_w, prompt, n_gen):
    loop = Llama2(backend, cfg, dev_w, kv_f16=True)
    fast = Llama2(backend, cfg, dev_w, kv_f16=True)
    first = loop.generate(prompt, 1)                       # the prompt through the decode path
    want_logits = loop.last_logits()
    want = first.tolist() + loop.generate(first, n_gen - 1, start_pos=len(prompt)).tolist()
    nxt = fast.prefill(prompt)                             # the prompt through the GEMMs
    got_logits = fast.last_logits()
    err = float(np.abs(got_logits - want_logits).max())
    assert err <= LOGITS_MAX_ABS, f"logits of the last prompt position differ by {err}"
    got = [nxt] + fast.generate([nxt], n_gen - 1, start_pos=len(prompt)).tolist()
    assert got == want, f"greedy tokens after the prompt differ (logits agreed to {err:.2e})"
    loop.close()
    fast.close()
    return err, want


def test_llama_3_2_1b_architecture_prefill_then_64_tokens(backend):
    cfg = LLAMA_3_2_1B
    w = synth_weights(cfg, seed=3001, device="cuda")
    dev_w = Llama2Weights(backend, cfg, w)
    del w
    prompt = np.random.default_rng(3002).integers(0, cfg.vocab_size, 32).tolist()
    err, _ = loop_vs_prefill(backend, cfg, dev_w, prompt, 65)
    print(f"1B-architecture prefill: logits of the last prompt position agree with the decode loop to {err:.3e}")
    dev_w.close()


def test_long_prompt_goes_in_chunks_and_matches_the_oracle(backend):
    """300 prompt tokens = three chunks of a GEMM pass; a later turn continues from start_pos > 0.  Small model, also against the oracle."""
    cfg = Llama2Config(512, 1024, 2, 8, 2, 512, 512, 500000.0, 1e-5)
    recipe = dict(Q4_K_M, token_embd=quant.Q4_K, attn_v=quant.Q5_K, ffn_down=quant.Q8_0, output=quant.Q4_K)   # 512 columns: no Q6_K rows here
    w = synth_weights(cfg, seed=21, recipe=recipe)
    dev_w = Llama2Weights(backend, cfg, w)
    prompt = np.random.default_rng(22).integers(0, cfg.vocab_size, 300).tolist()
    _, want = loop_vs_prefill(backend, cfg, dev_w, prompt, 12)
    ref = oracle.Llama(dict(hidden=512, ffn=1024, n_layers=2, n_heads=8, n_kv_heads=2, vocab=512, max_pos=512, rope_theta=500000.0, rms_eps=1e-5),
                       weights_to_host(w), kv_f16=True)
    toks, out = list(prompt), []
    for pos in range(len(prompt) + 11):
        lg = ref.forward(toks[pos], pos)
        if pos >= len(prompt) - 1:
            out.append(oracle.argmax(lg))
            toks.append(out[-1])
    ref.close()
    assert want == out
    # second turn: 40 more prompt tokens on top of the kept cache
    m = Llama2(backend, cfg, dev_w, kv_f16=True)
    a = m.prefill(prompt)
    more = np.random.default_rng(23).integers(0, cfg.vocab_size, 40).tolist()
    b = m.prefill(more, start_pos=len(prompt))
    loop = Llama2(backend, cfg, dev_w, kv_f16=True)
    assert int(loop.generate(prompt + more, 1)[0]) == b and a == want[0]
    m.close()
    loop.close()
    dev_w.close()


# q, k (Q4_K or Q5_K) and v (Q6_K) in one GEMM launch, and beyond two chunks of tokens in two: one SM per tile and pairs, a partial and a second chunk
@pytest.mark.parametrize("qk,heads", [(quant.Q4_K, 32), (quant.Q5_K, 16)])
def test_formats_that_share_a_launch(backend, qk, heads):
    cfg = Llama2Config(2048, 2048, 2, heads, heads // 4, 512, 512, 500000.0, 1e-5)
    w = synth_weights(cfg, seed=31, device="cuda", recipe=dict(Q4_K_M, attn_q=qk, attn_k=qk, token_embd=quant.Q4_K))
    dev_w = Llama2Weights(backend, cfg, w)
    for n in (1, 9, 16, 17, 64, 65, 128, 129, 256, 257, 400):
        loop_vs_prefill(backend, cfg, dev_w, np.random.default_rng(n).integers(0, cfg.vocab_size, n).tolist(), 3)
    dev_w.close()


# From 512 tokens on the norm's CTAs hold rows of 2048 and 4096 columns of two tokens, others of up to 4096 of four, longer ones of one; a token count that leaves
# padding rows.  Without a nudge (eps 0) the padding rows' norm is infinite: they stay zero all the same.
@pytest.mark.parametrize("hidden,eps", [(2048, 0.0), (3072, 0.0), (4096, 1e-5), (4608, 1e-5), (8704, 0.0)])
@pytest.mark.parametrize("n", [9, 517, 601])
def test_norms_of_many_tokens(backend, hidden, eps, n):
    cfg = Llama2Config(hidden, 512, 1, hidden // 128, hidden // 512, 512, 640, 500000.0, eps)
    w = synth_weights(cfg, seed=hidden, device="cuda", recipe={**{k: quant.Q4_K for k in Q4_K_M}, "token_embd": quant.Q4_K})
    dev_w = Llama2Weights(backend, cfg, w)
    loop_vs_prefill(backend, cfg, dev_w, np.random.default_rng(n).integers(0, cfg.vocab_size, n).tolist(), 2)
    dev_w.close()


@pytest.mark.parametrize("hidden,heads,n,start", [(512, 8, 17, 0), (512, 8, 1, 300), (512, 4, 65, 0), (512, 4, 15, 470), (512, 8, 200, 130)])
def test_prompt_attention_at_the_edges_of_its_tiles(backend, hidden, heads, n, start):
    """16-token and 64-position tiles with remainders, positions divided between the CTAs of a cluster (few tokens far into the
    context), both head sizes: against the decode loop's attention, whose cache rows are the same f16 values."""
    cfg = Llama2Config(hidden, 1024, 1, heads, heads // 4, 512, 512, 500000.0, 1e-5)
    recipe = dict(Q4_K_M, token_embd=quant.Q4_K, attn_v=quant.Q5_K, ffn_down=quant.Q8_0, output=quant.Q4_K)
    w = synth_weights(cfg, seed=31, recipe=recipe, std=0.06)      # sharper scores than 0.02 gives
    dev_w = Llama2Weights(backend, cfg, w)
    toks = np.random.default_rng(32 + n).integers(0, cfg.vocab_size, start + n).tolist()
    loop, fast = Llama2(backend, cfg, dev_w, kv_f16=True), Llama2(backend, cfg, dev_w, kv_f16=True)
    loop.generate(toks, 0)
    if start:
        fast.prefill(toks[:start])
    fast.prefill(toks[start:], start_pos=start)
    a, b = loop.hidden_state(), fast.hidden_state()
    # the loop's activations are 16-bit block fixed point (2^-15 of a group's largest value per GEMV, seven GEMVs deep)
    assert np.abs(a - b).max() <= 2e-3 * np.abs(a).max()
    loop.close()
    fast.close()
    dev_w.close()


def test_prompts_and_gemms_go_in_shorter_passes_where_memory_is_short(backend):
    """1024 tokens through layers of the 8B architecture take 330 MB of buffers at once, 128 tokens 45 MB: with 150 MB free on the device the
    prompt goes through in shorter passes, to the same result, and so do 1024 rows through one matrix.  (Sums of f32
    that are split differently: 1e-6; where that rounds a cache value the other way, 2^-11 of one of the 1500 rows that are averaged.)"""
    from inferi_b200.ops import Backend, GemmQuant
    cfg = Llama2Config(4096, 14336, 1, 32, 8, 512, 2048, 500000.0, 1e-5)
    w = synth_weights(cfg, seed=51, device="cuda", recipe=dict(Q4_K_M, token_embd=quant.Q4_K, output=quant.Q4_K))
    toks = np.random.default_rng(52).integers(0, 512, 1500).tolist()
    x = torch.randn(1024, 4096, device="cuda")

    def results(free):
        be = Backend(0)
        dev_w = Llama2Weights(be, cfg, w)
        model = Llama2(be, cfg, dev_w, kv_f16=True)
        out = torch.zeros(1024, 14336, device="cuda")
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        hog = torch.empty(torch.cuda.mem_get_info()[0] - free, dtype=torch.uint8, device="cuda") if free else None
        model.prefill(toks)
        hidden = model.hidden_state()
        model.prefill(toks[:9])
        model.prefill(toks)          # the buffers that a long prompt got are kept
        assert np.array_equal(hidden, model.hidden_state())
        GemmQuant(be).launch(out, dev_w.layers[0]["ffn_gate"], x)
        torch.cuda.synchronize()
        del hog
        torch.cuda.empty_cache()
        model.close()
        dev_w.close()
        be.close()
        return hidden, out

    (h0, g0), (h1, g1) = results(0), results(150 << 20)
    assert np.abs(h0 - h1).max() <= 1e-4 * np.abs(h0).max()
    assert float((g0 - g1).abs().max()) <= 1e-5 * float(g0.abs().max())


def test_prefill_refuses_what_the_tensor_core_path_does_not_take(backend):
    cfg = Llama2Config(256, 2048, 2, 4, 2, 512, 64, 500000.0, 1e-5)     # 2 query heads per kv head, 256-row matrices... kv_mul = 2
    w = synth_weights(cfg, seed=5, recipe=dict(Q4_K_M, token_embd=quant.Q4_K, attn_v=quant.Q4_K, ffn_down=quant.Q4_K, output=quant.Q4_K))
    dev_w = Llama2Weights(backend, cfg, w)
    m = Llama2(backend, cfg, dev_w, kv_f16=True)
    with pytest.raises(InferiError) as e:
        m.prefill([1, 2, 3])
    assert e.value.code == 4      # IB_ERR_UNSUPPORTED: the caller feeds the prompt through generate()
    assert m.generate([1, 2, 3], 4).shape == (4,)
    m.close()
    dev_w.close()
