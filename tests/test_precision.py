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


# ---- Q6_K scales over the whole of int8, as quantisers write them (the synthetic blocks stop at +-32) ----

def pack_q6k(q, scales, d):
    """Q6_K blocks (gguf.h:109-113) of quants [n][256] from 0 to 63, scales [n][16] and d [n]."""
    n = len(q)
    g = q.reshape(n, 2, 4, 32).astype(np.uint8)  # [half][quarter]: low bits in two nibbles of ql, high bits in four fields of qh
    ql = (g[:, :, :2] & 15) | (g[:, :, 2:] & 15) << 4
    qh = (g >> 4 << np.array([0, 2, 4, 6], dtype=np.uint8).reshape(4, 1)).sum(axis=2, dtype=np.uint8)
    return np.concatenate([ql.reshape(n, 128), qh.reshape(n, 64), scales.astype(np.int8).view(np.uint8).reshape(n, 16),
                           d.astype(np.float16).reshape(n, 1).view(np.uint8)], axis=1).reshape(-1)


def q6k_operand(blocks, k):
    """What the grouped product multiplies, [rows][k] in 64 bits: scale * (quant - 32) rounded to a half, times d."""
    d = np.repeat(np.ascontiguousarray(blocks).reshape(-1, synth.Q6K_BYTES)[:, 208:210].copy().view(np.float16).astype(np.float64), 256, axis=1).reshape(-1, k)
    return (dequant(blocks, synth.GGML_Q6_K, k) / d).astype(np.float16).astype(np.float64) * d


def every_scale_and_quant(rows, nb):
    """Blocks in which each of the 256 x 64 pairs stands in each of the 16 sub-blocks: [rows][nb], rows * nb >= 1024."""
    c = np.arange(rows * nb).reshape(-1, 1, 1)
    j, e = np.arange(16).reshape(1, 16, 1), np.arange(16).reshape(1, 1, 16)
    q = 16 * (c // 256 % 4) + (e + 5 * (c // 256) + j) % 16
    return pack_q6k(q.reshape(-1, 256), np.broadcast_to(c.reshape(-1, 1) % 256 - 128, (rows * nb, 16)), np.full(rows * nb, 2.0 ** -6))


def test_every_scale_and_quant_is_there(port_lib):
    w = every_scale_and_quant(256, 4)
    sub = np.rint(dequant(w, synth.GGML_Q6_K, 1024) * 64).astype(int).reshape(-1, 16, 16)
    for j in range(16):
        assert set(sub[:, j].ravel()) == {s * q for s in range(-128, 128) for q in range(-32, 32)}
    x = synth.make_x(3, 1, 1024)[0]
    assert error(port_lib.mat_vec(x, w, synth.GGML_Q6_K, 1024, 256), dequant(w, synth.GGML_Q6_K, 1024) @ x.astype(np.float64)) < 1e-6
    assert np.abs(q6k_operand(w, 1024) - dequant(w, synth.GGML_Q6_K, 1024)).max() <= 2.0 ** -6  # (4096 is reached: 11 bits are steps of 2)


@pytest.fixture(scope="module")
def dense():
    from tie_b200 import moe
    b = moe.MoeBackend(max_tokens=1024)
    yield b
    b.close()


# Unit vectors read the operand itself: one product with the half 1, all others with 0, so no bit may differ.  1024 of them
# against 1024 rows: tiles of 64 on pairs of CTAs; 640: single CTAs; 512 and 384: the same with tiles of 32; 256: rows split.
@pytest.mark.gpu
@pytest.mark.parametrize("out_dim", [1024, 640, 512, 384, 256])
def test_q6k_operand_over_all_scales_and_quants(dense, out_dim):
    b, k = dense, 1024
    w = every_scale_and_quant(out_dim, k // 256)
    b.register_tensor(w, synth.GGML_Q6_K, k)
    got = b.mat_mat(w, np.eye(k, dtype=np.float32), np.full((k, out_dim), np.nan, dtype=np.float32), k, k, out_dim)
    assert np.array_equal(got, q6k_operand(w, k).T)


@pytest.fixture(scope="module", params=["q6k_down", "q6k_gate_up"])
def wide(request, layer0, ref_silu_table):
    """A block with Q6_K tensors of all scales; the first tokens' outputs per expert in 64 bits, from the exact weights and
    from the operand that the grouped product makes of them."""
    from tie_b200 import moe
    s = synth.MoeShape()
    n_gu, n_dn = s.n_expert * s.ffn_dim * (s.hidden // 256), s.n_expert * s.hidden * (s.ffn_dim // 256)

    def q6k(stream, n):
        b = np.array(synth.q6k_blocks(61, stream, n)).reshape(n, synth.Q6K_BYTES)
        b[:, 192:208] = np.random.default_rng(stream).integers(-128, 128, (n, 16), dtype=np.int8).view(np.uint8)
        b[:, 208:210] = (b[:, 208:210].copy().view(np.float16) * np.float16(0.25)).view(np.uint8)  # (weights of the usual size)
        return b.reshape(-1)

    if request.param == "q6k_down":
        layer = synth.MoeLayer(s, layer0.router_w, layer0.gate, layer0.up, q6k(synth.STREAM_DOWN, n_dn))
    else:
        layer = synth.MoeLayer(s, layer0.router_w, q6k(synth.STREAM_GATE, n_gu), q6k(synth.STREAM_UP, n_gu), synth.q4k_blocks(77, synth.STREAM_DOWN, n_dn),
                               gate_type=synth.GGML_Q6_K, up_type=synth.GGML_Q6_K, down_type=synth.GGML_Q4_K)
    b = moe.MoeBackend(max_tokens=512, silu_table=ref_silu_table)
    b.upload_layer(0, layer)
    x, tab = synth.make_x(3, 512, first_token=2000), ref_silu_table.astype(np.float64)
    idx, w, _ = b.route(0, x[:N_EXACT])
    rows = np.zeros((2, N_EXACT, s.top_k, s.hidden))
    for i, rounded in enumerate((False, True)):
        def weights(t, kind, e, k):
            t = np.asarray(t).reshape(s.n_expert, -1)[e]
            return q6k_operand(t, k) if rounded and kind == synth.GGML_Q6_K else dequant(t, kind, k)

        for t in range(N_EXACT):
            xt = x[t].astype(np.float64)
            for j, e in enumerate(idx[t]):
                g, u = weights(layer.gate, layer.gate_type, e, s.hidden) @ xt, weights(layer.up, layer.up_type, e, s.hidden) @ xt
                pos = (g + 10.0) * 8191.0 * 0.05  # the table's SwiGLU (math_avx2.c:908-950)
                p = np.clip(np.rint(pos), 0, 8190).astype(int)
                rows[i, t, j] = weights(layer.down, layer.down_type, e, s.ffn_dim) @ ((tab[p] + (tab[p + 1] - tab[p]) * (pos - p)) * u)
    yield b, x, idx, rows, np.einsum("tj,itjh->ith", w.astype(np.float64), rows)
    b.close()


# A weight above 2048 is off by 1 at the most, 2^-11 of itself: 1.4e-4 of a product with scales uniform over int8, 2.5e-4 where
# gate and up both have them.  Against the rounded weights what is left is the activations' 22 bits: 8.0e-7 to 9.1e-7 here,
# twice the bound of prompts of the usual weights allowed.
WIDE, WIDE_OPERAND = 3e-4, 2.8e-6


# 32 and 64 tokens: tiles of 32; 512: of 64.  Gate and up in pairs of CTAs, down in pairs at 512, or all of them single.
@pytest.mark.gpu
@pytest.mark.parametrize("path", ["auto", "no_pair"])
@pytest.mark.parametrize("n_tokens", [32, 64, 512])
def test_q6k_scales_of_prompt_batches(wide, n_tokens, path):
    from tie_b200 import moe
    b, x, _, _, want = wide
    got = b.moe_ffn(0, x[:n_tokens], path=moe.PATH_NO_PAIR if path == "no_pair" else moe.PATH_AUTO)[:N_EXACT]
    assert error(got, want[1]) < WIDE_OPERAND
    assert error(got, want[0]) < WIDE


@pytest.mark.gpu
def test_q6k_scales_of_expert_rows(wide):
    import torch
    from tie_b200 import moe
    b, x, idx, rows, _ = wide
    xr, e = np.repeat(x[:N_EXACT], idx.shape[1], axis=0), np.ascontiguousarray(idx, dtype=np.int32).reshape(-1)
    y = torch.full(xr.shape, float("nan"), device="cuda")
    b.expert_rows_ptr(0, torch.from_numpy(xr).cuda(), torch.from_numpy(e).cuda(), len(e), y, moe.DEVICE | moe.PATH_TENSOR)
    assert error(y.cpu().numpy(), rows[1].reshape(xr.shape)) < WIDE_OPERAND
    assert error(y.cpu().numpy(), rows[0].reshape(xr.shape)) < WIDE


# Rows split among a cluster (37 tokens) and not (600).
@pytest.mark.gpu
@pytest.mark.parametrize("batch", [37, 600])
def test_q6k_scales_of_dense_products(dense, batch):
    b, k, out_dim = dense, 2048, 512
    w = every_scale_and_quant(out_dim, k // 256)
    b.register_tensor(w, synth.GGML_Q6_K, k)
    x = synth.make_x(4, batch, k)
    got = b.mat_mat(w, x, np.empty((batch, out_dim), dtype=np.float32), batch, k, out_dim)
    assert error(got, x.astype(np.float64) @ q6k_operand(w, k).T) < 4e-7  # as with the usual weights
    assert error(got, x.astype(np.float64) @ dequant(w, synth.GGML_Q6_K, k).T) < WIDE
