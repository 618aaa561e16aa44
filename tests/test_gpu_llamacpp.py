"""Greedy-token parity through the reference's REAL llama.cpp: identical greedy-decoded tokens over 128 steps.

oracle/_ref/llama_harness (the unmodified src/llama.cpp + ggml_backend_sched compiled from /root/reference) decodes a synthetic
GGUF twice: on the reference CPU backend, and with libkcpp_b200.so attached by ggml_backend_register (Route 2).  Asserted:
  * the two greedy token streams are identical (prompt logits + 128 generated tokens);
  * the logits of every step agree to a stated relative L2 (the CPU path quantises activations to q8_0 / q8_K, the B200 path to
    q8_1 for decode and bf16 for prompt batches: noise of ~1e-2);
  * the scheduler left only the token-embedding GET_ROWS on the CPU backend (llama.cpp keeps token_embd in a host buffer).
The models are random-init with the reference quantiser (tools/make_gguf.py "margin model"; the margin statistics are asserted
too, so a degenerate fixture cannot make the token check vacuous).
"""
from __future__ import annotations

import os
import tempfile

import numpy as np
import pytest

import gguf_fixtures as G
import llamacpp as LC

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not LC.available(), reason="oracle/_ref/llama_harness not built")]

# Relative L2 of a step's logits, B200 vs the reference CPU backend.  Deep random-init models amplify rounding differences: the
# reference's OWN builds disagree with each other by several percent on the C1 fixture (AVX2 vs AVX-512 build 4.5e-2, flash
# attention on vs off 5.1e-2, f16 vs q8_0 KV 5.5e-2: measured with tools in this repo).  The bar is therefore stated
# against that spread, measured in the same test: B200-vs-CPU <= 1.5 x (CPU flash-attention-on vs CPU flash-attention-off), with
# an absolute floor for the shallow fixtures where the spread is tiny.
LOGIT_TOL_FLOOR = 2.5e-2
LOGIT_TOL_SPREAD_FACTOR = 1.5
ONLY_EMBD = [("GET_ROWS", "inp_embd")]


def both(model, n_prompt, n_gen, **opts):
    with tempfile.TemporaryDirectory() as d:
        lc, lg = os.path.join(d, "cpu.bin"), os.path.join(d, "gpu.bin")
        cpu = LC.run(model, "cpu", n_prompt=n_prompt, n_gen=n_gen, exe=LC.harness_path(), logits_out=lc, threads=min(32, os.cpu_count() or 8), **opts)
        gpu = LC.run(model, "b200", n_prompt=n_prompt, n_gen=n_gen, sched_debug=True, logits_out=lg, **opts)
        nv = cpu["n_vocab"]
        a = np.fromfile(lc, dtype=np.float32).reshape(-1, nv)
        b = np.fromfile(lg, dtype=np.float32).reshape(-1, nv)
        # the reference's own spread: the same run with the other attention path (flash attention toggled)
        o2 = dict(opts)
        o2["fa"] = 0 if int(opts.get("fa", 1)) else 1
        if o2.get("type_kv") in ("q8_0", "q4_0") and o2["fa"] == 0:
            o2.pop("type_kv")  # a quantised V cache needs flash attention (src/llama.cpp:19447-19450): compare against f16 KV instead
        LC.run(model, "cpu", n_prompt=n_prompt, n_gen=n_gen, exe=LC.harness_path(), logits_out=lc, threads=min(32, os.cpu_count() or 8), **o2)
        a2 = np.fromfile(lc, dtype=np.float32).reshape(-1, nv)
        cpu["spread"] = float((np.linalg.norm(a - a2, axis=1) / np.linalg.norm(a, axis=1)).max()) if a2.shape == a.shape else 0.0
    return cpu, gpu, a, b


def check_parity(cpu, gpu, a, b, min_margin_sigma):
    assert gpu["n_devices"] >= 1
    assert gpu["sched"]["cpu_nodes"] == ONLY_EMBD, gpu["sched"]
    assert a.shape == b.shape and np.isfinite(b).all()
    rel = np.linalg.norm(a - b, axis=1) / np.linalg.norm(a, axis=1)
    m = np.array(cpu["margins"]) / np.array(cpu["logit_std"])
    # the fixture is not degenerate: the layers move the logits (std well above 0) and the argmax margin is what we rely on
    assert m.min() > min_margin_sigma, m.min()
    first_diff = next((i for i, (x, y) in enumerate(zip(cpu["tokens"], gpu["tokens"])) if x != y), None)
    assert cpu["tokens"] == gpu["tokens"], f"greedy streams differ at step {first_diff}; rel L2 of logits there {rel[first_diff]:.3e}"
    tol = max(LOGIT_TOL_FLOOR, LOGIT_TOL_SPREAD_FACTOR * cpu["spread"])
    assert rel.max() < tol, (float(rel.max()), int(rel.argmax()), cpu["spread"])
    return float(rel.max()), float(np.median(rel))


def test_c1_tinyllama_q4_0_pp128_tg128_identical_tokens():
    """TinyLlama-1.1B-shaped Q4_0 (output Q6_K), pp128 + tg128 greedy, f16 KV, flash attention."""
    model = G.build_fixture("tinyllama-1.1b-q4_0", layer_gain=3.0)
    cpu, gpu, a, b = both(model, 128, 128)
    assert len(cpu["tokens"]) == 129
    worst, med = check_parity(cpu, gpu, a, b, min_margin_sigma=1.0)
    print(f"C1 logits rel L2: worst {worst:.3e} median {med:.3e} (reference FA on/off spread {cpu['spread']:.3e}); cpu tg {cpu['tg_tok_s']:.1f} tok/s, b200 tg {gpu['tg_tok_s']:.1f} tok/s (through llama_decode)")


def test_7b_shaped_2_layer_q4_k_m_q8_0_kv_identical_tokens():
    """Llama-2-7B layer shapes (4096 / 11008 / 32 heads), Q4_K + Q6_K mix, q8_0 KV cache: 2 layers keep the fixture small."""
    model = G.build_fixture("llama2-7b-q4_k_m", n_layer=2, layer_gain=4.0)
    cpu, gpu, a, b = both(model, 128, 128, type_kv="q8_0")
    worst, med = check_parity(cpu, gpu, a, b, min_margin_sigma=1.0)
    print(f"7B-shaped x2 logits rel L2: worst {worst:.3e} median {med:.3e}")


def test_q4_0_kv_cache_identical_tokens():
    """N4: a q4_0 KV cache (koboldcpp's quantkv = 2): K and V rows stored by CPY f32 -> q4_0 (bit-exact quantize_row_q4_0_ref), attention
    over q4_0 tiles on the tensor-core kernel, prompt and decode."""
    model = G.build_fixture("test-dense", layer_gain=1.5)
    cpu, gpu, a, b = both(model, 40, 32, type_kv="q4_0")
    check_parity(cpu, gpu, a, b, min_margin_sigma=0.5)


@pytest.mark.parametrize("ftype", ("Q4_1", "Q5_0", "Q5_1", "Q2_K", "Q3_K", "IQ4_NL", "IQ4_XS"))
def test_legacy_quant_types_identical_tokens(ftype):
    """N4: the 32-value formats Q4_1 / Q5_0 / Q5_1 the small K-quants Q2_K / Q3_K and the non-linear IQ4_NL / IQ4_XS, every matrix of the type (output.weight Q6_K) through llama_decode: prompt on the tensor-core GEMM,
    decode on the GEMV, token embedding rows by GET_ROWS on the CPU as always."""
    model = G.build_fixture("test-dense", layer_gain=1.5, ftype=ftype)
    cpu, gpu, a, b = both(model, 40, 32)
    check_parity(cpu, gpu, a, b, min_margin_sigma=0.5)


def test_moe_prompt_and_decode_identical_tokens():
    """Mixtral-style graph: MUL_MAT_ID batches (grouped tensor-core GEMM) in the prompt, expert GEMV in decode, fused router."""
    model = G.build_fixture("test-moe", layer_gain=1.5)
    cpu, gpu, a, b = both(model, 40, 32)
    check_parity(cpu, gpu, a, b, min_margin_sigma=0.5)


def test_context_shift_identical_tokens():
    """koboldcpp ContextShift (K-shift graph on the backend: in-place f16 ROPE over the cache) in the middle of generation."""
    model = G.build_fixture("test-dense", layer_gain=1.5)
    cpu, gpu, a, b = both(model, 48, 24, shift_at=8, shift_by=16)
    check_parity(cpu, gpu, a, b, min_margin_sigma=0.5)


def test_context_shift_q8_0_cache():
    """K-shift over a q8_0 cache: CPY(q8_0 -> f32) -> ROPE -> CPY(f32 -> q8_0) (src/llama.cpp:10165-10180).  The reference CPU
    backend cannot run this graph at all (ggml.c:9073 fatal error in ggml_compute_forward_dup for a q8_0 source), so the check is
    against the reference's f16-cache run of the same shift: identical greedy tokens, logits within the q8_0-vs-f16 cache noise."""
    model = G.build_fixture("test-dense", layer_gain=1.5)
    with tempfile.TemporaryDirectory() as d:
        lc, lg = os.path.join(d, "cpu.bin"), os.path.join(d, "gpu.bin")
        cpu = LC.run(model, "cpu", n_prompt=48, n_gen=24, exe=LC.harness_path(), logits_out=lc, shift_at=8, shift_by=16)
        gpu = LC.run(model, "b200", n_prompt=48, n_gen=24, sched_debug=True, logits_out=lg, type_kv="q8_0", shift_at=8, shift_by=16)
        a = np.fromfile(lc, dtype=np.float32).reshape(-1, cpu["n_vocab"])
        b = np.fromfile(lg, dtype=np.float32).reshape(-1, cpu["n_vocab"])
    assert gpu["sched"]["cpu_nodes"] == ONLY_EMBD
    assert cpu["tokens"] == gpu["tokens"]
    rel = np.linalg.norm(a - b, axis=1) / np.linalg.norm(a, axis=1)
    assert rel.max() < 6e-2, float(rel.max())


def test_batched_prompt_in_ubatches_and_fa_off():
    model = G.build_fixture("test-dense", layer_gain=1.5)
    cpu, gpu, a, b = both(model, 200, 8, n_batch=64, n_ubatch=64)
    check_parity(cpu, gpu, a, b, min_margin_sigma=0.5)
    cpu, gpu, a, b = both(model, 40, 8, fa=0)
    check_parity(cpu, gpu, a, b, min_margin_sigma=0.5)


def test_split_mode_row_matches_single_gpu():
    """LLAMA_SPLIT_MODE_ROW over the row-split buffer type (a13 / a14): same greedy tokens as one GPU."""
    from koboldcpp_b200.lib import lib
    if lib().b200_device_count() < 2:
        pytest.skip("needs 2 GPUs")
    model = G.build_fixture("test-dense", layer_gain=1.5)
    one = LC.run(model, "b200", n_prompt=40, n_gen=24, env_extra={"CUDA_VISIBLE_DEVICES": "0"})
    two = LC.run(model, "b200", n_prompt=40, n_gen=24, split_mode="row", sched_debug=True)
    assert two["n_devices"] >= 2 and two["sched"]["cpu_nodes"] == ONLY_EMBD
    assert one["tokens"] == two["tokens"]
