"""How far the kernels are from 64-bit arithmetic on the same packed weights, against what fp32 arithmetic throughout
reaches.  (The error of a product: 2-norm of the difference over 2-norm of the result.)"""
import functools

import numpy as np
import pytest

from tie_b200 import synth, workloads

N_EXACT = 6  # tokens whose outputs are worked out in 64 bits


def dequant(blocks, ggml_type, k):
    """[rows][k] in 64 bits (dequantize_row_q4_k, _q6_k: math_scalar.c:216-287)."""
    if ggml_type == synth.GGML_Q4_K:
        b = np.ascontiguousarray(blocks).reshape(-1, synth.Q4K_BYTES)
        d, dmin = b[:, 0:2].copy().view(np.float16).astype(np.float64), b[:, 2:4].copy().view(np.float16).astype(np.float64)
        s = b[:, 4:16].astype(int)
        sc = np.concatenate([s[:, 0:4] & 63, (s[:, 8:12] & 15) | (s[:, 0:4] >> 6) << 4], axis=1)
        mn = np.concatenate([s[:, 4:8] & 63, s[:, 8:12] >> 4 | (s[:, 4:8] >> 6) << 4], axis=1)
        qs = b[:, 16:].reshape(-1, 4, 1, 32)
        q = np.concatenate([qs & 15, qs >> 4], axis=2).reshape(-1, 8, 32)
        w = d[:, :, None] * sc[:, :, None] * q - dmin[:, :, None] * mn[:, :, None]
    else:
        b = np.ascontiguousarray(blocks).reshape(-1, synth.Q6K_BYTES)
        ql, qh = b[:, :128].reshape(-1, 2, 2, 32), b[:, 128:192].reshape(-1, 2, 1, 32).astype(int)
        lo = np.stack([ql[:, :, 0] & 15, ql[:, :, 1] & 15, ql[:, :, 0] >> 4, ql[:, :, 1] >> 4], axis=2)
        q = lo + ((qh >> np.array([0, 2, 4, 6]).reshape(4, 1) & 3) << 4) - 32
        w = q.reshape(-1, 16, 16) * b[:, 192:208].view(np.int8).astype(np.float64)[:, :, None] * b[:, 208:210].copy().view(np.float16).astype(np.float64)[:, :, None]
    return w.reshape(-1, k)


def error(got, want):
    return np.sqrt(((got - want) ** 2).sum() / (want ** 2).sum())


@pytest.mark.parametrize("ggml_type", [synth.GGML_Q4_K, synth.GGML_Q6_K])
def test_dequantisation_agrees_with_the_restatement(ggml_type, port_lib):
    w = (synth.q4k_blocks if ggml_type == synth.GGML_Q4_K else synth.q6k_blocks)(3, 9, 64 * 2)
    x = synth.make_x(3, 1, 512)[0]
    assert error(port_lib.mat_vec(x, w, ggml_type, 512, 64), dequant(w, ggml_type, 512) @ x.astype(np.float64)) < 1e-6


@pytest.fixture(scope="module")
def block(layer0, ref_silu_table):
    """Layer 0 with a Q6_K down tensor, layer 1 the same with Q4_K; the first tokens' outputs in 64 bits."""
    from tie_b200 import moe
    s = synth.MoeShape()
    q4 = synth.MoeLayer(s, layer0.router_w, layer0.gate, layer0.up, synth.q4k_blocks(77, synth.STREAM_DOWN, s.n_expert * s.hidden * (s.ffn_dim // 256)),
                        gate_type=synth.GGML_Q4_K, up_type=synth.GGML_Q4_K, down_type=synth.GGML_Q4_K)
    b = moe.MoeBackend(max_tokens=512, silu_table=ref_silu_table, n_layers=2)
    b.upload_layer(0, layer0)
    b.upload_layer(1, q4)
    x, tab = synth.make_x(3, 512, first_token=1000), ref_silu_table.astype(np.float64)
    idx, w, _ = b.route(0, x[:N_EXACT])

    @functools.lru_cache(None)
    def weights(which, e):
        t, kind, k = {"gate": (layer0.gate, synth.GGML_Q4_K, s.hidden), "up": (layer0.up, synth.GGML_Q4_K, s.hidden),
                      "q6_k": (layer0.down, synth.GGML_Q6_K, s.ffn_dim), "q4_k": (q4.down, synth.GGML_Q4_K, s.ffn_dim)}[which]
        return dequant(np.asarray(t).reshape(s.n_expert, -1)[e], kind, k)

    want = np.zeros((2, N_EXACT, s.hidden))
    for t in range(N_EXACT):
        xt = x[t].astype(np.float64)
        for j, e in enumerate(idx[t]):
            g, u = weights("gate", e) @ xt, weights("up", e) @ xt
            pos = (g + 10.0) * 8191.0 * 0.05  # the table's SwiGLU (math_avx2.c:908-950)
            i = np.clip(np.rint(pos), 0, 8190).astype(int)
            h = (tab[i] + (tab[i + 1] - tab[i]) * (pos - i)) * u
            for layer, kind in enumerate(("q6_k", "q4_k")):
                want[layer, t] += float(w[t, j]) * (weights(kind, e) @ h)
    yield b, x, want
    b.close()


# fp32 arithmetic throughout (the kernels before their products moved to the tensor cores) was 2.9e-7 off with a Q6_K down
# tensor and 1.1e-7 with Q4_K, at the most.  Products on the tensor cores whose parts lie on no grid: 3.3e-7 .. 4.5e-7.
@pytest.mark.gpu
@pytest.mark.parametrize("layer,bound", [(0, 2.9e-7), (1, 1.12e-7)], ids=["q6k_down", "q4k_down"])
@pytest.mark.parametrize("n_tokens", [1, 2, 4, 7, 8, 13, 31])
def test_small_batches_are_as_exact_as_fp32(block, n_tokens, layer, bound):
    b, x, want = block
    n = min(n_tokens, N_EXACT)
    assert error(b.moe_ffn(layer, x[:n_tokens])[:n], want[layer, :n]) < bound


# fp16 hi + lo halves (22 bits), with accumulators of their own for the two: 1.09e-6 and 1.37e-6 at the most; with their
# products in turn in one accumulator 1.5e-6 and 1.9e-6.
@pytest.mark.gpu
@pytest.mark.parametrize("layer,bound", [(0, 1.1e-6), (1, 1.38e-6)], ids=["q6k_down", "q4k_down"])
@pytest.mark.parametrize("n_tokens", [32, 512])
def test_prompt_batches(block, n_tokens, layer, bound):
    b, x, want = block
    assert error(b.moe_ffn(layer, x[:n_tokens])[:N_EXACT], want[layer]) < bound


# The same for one product: 2.9e-7 and 6.0e-7.
@pytest.mark.gpu
@pytest.mark.parametrize("batch", [37, 256])
@pytest.mark.parametrize("ggml_type,in_dim,out_dim", [(synth.GGML_Q4_K, 4096, 2048), (synth.GGML_Q6_K, 2048, 512)])
def test_dense_products(block, ggml_type, in_dim, out_dim, batch):
    b = block[0]
    w = np.ascontiguousarray((synth.q4k_blocks if ggml_type == synth.GGML_Q4_K else synth.q6k_blocks)(5, 9, in_dim // 256 * out_dim))
    b.register_tensor(w, ggml_type, in_dim)
    x = synth.make_x(4, batch, in_dim)
    got = b.mat_mat(w, x, np.empty((batch, out_dim), dtype=np.float32), batch, in_dim, out_dim)
    assert error(got, x.astype(np.float64) @ dequant(w, ggml_type, in_dim).T) < 4e-7
