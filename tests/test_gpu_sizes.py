"""Sizes where one form of a kernel hands over to another, or where a tile has a remainder: token
tiles of the router, of the grouped products and of the dispatch sort, the step from the per-row
decode kernels to the grouped ones, and the copies of pageable host buffers.  Against the CPU
restatement, or bit for bit against another route to the same kernels.
"""
import numpy as np
import pytest

from tie_b200 import synth, workloads

pytestmark = pytest.mark.gpu

TOL = 1e-3


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)


@pytest.fixture(scope="module")
def be(layer0, ref_silu_table):
    from tie_b200 import moe
    b = moe.MoeBackend(max_tokens=1100, silu_table=ref_silu_table)
    b.upload_layer(0, layer0, keep_host=True)
    yield b
    b.close()


@pytest.fixture(scope="module")
def port0(port_lib, layer0, ref_silu_table):
    return port_lib.PortMoe(layer0, silu=ref_silu_table)


# The smaller expert shape of the grouped products: 4 super-blocks per gate / up row (pairs of CTAs), 1 per
# down row; Q6_K down, and the same with all three tensors as Q4_K.
@pytest.fixture(scope="module", params=["q6k_down", "q4k_down"])
def grouped(request, port_lib, ref_silu_table):
    from tie_b200 import moe
    s = synth.MoeShape(hidden=1024, n_expert=32, top_k=4, ffn_dim=256)
    layer = synth.make_layer(workloads.BASE_SEED + 5, s)
    if request.param == "q4k_down":
        n_down = s.n_expert * s.hidden * (s.ffn_dim // 256)
        layer = synth.MoeLayer(s, layer.router_w, layer.gate, layer.up, synth.q4k_blocks(5, synth.STREAM_DOWN, n_down),
                               gate_type=synth.GGML_Q4_K, up_type=synth.GGML_Q4_K, down_type=synth.GGML_Q4_K)
    b = moe.MoeBackend(hidden=s.hidden, n_expert=s.n_expert, top_k=s.top_k, ffn_dim=s.ffn_dim, max_tokens=512, silu_table=ref_silu_table)
    b.upload_layer(0, layer, keep_host=True)
    yield b, port_lib.PortMoe(layer, silu=ref_silu_table), s
    b.close()


# A tile of the batched router is 4, 8, 16, 32 or 64 tokens wide, by how many CTAs the batch makes.
@pytest.mark.parametrize("n_tokens", [5, 13, 31, 33, 65, 129, 257, 511, 1023, 1100])
def test_router_tiles_and_both_selections(be, port0, n_tokens):
    x = synth.make_x(0, n_tokens, first_token=7)
    idx, w, logits = be.route(0, x)
    i_r, w_r, l_r = port0.route(x)
    assert np.array_equal(bits(logits), bits(l_r)) and np.array_equal(idx, i_r)
    assert np.abs(w - w_r).max() <= 2e-7
    idx, w, _ = be.route(0, x, lfm2=True)
    i_r, w_r, _ = port0.route_lfm2(x)
    assert np.array_equal(idx, i_r)
    assert np.abs(w / w_r - 1).max() < 2e-6


# 7 tokens are the last batch of the per-row kernels with 128 experts and top-8.
@pytest.mark.parametrize("n_tokens", [6, 8, 9, 12])
def test_per_row_and_grouped_products_around_the_change(be, port0, n_tokens):
    x = synth.make_x(0, n_tokens, first_token=90)
    ref, ref_idx, _ = port0.moe_ffn(x)
    out = be.moe_ffn(0, x)
    assert workloads.rel_rms_err(out, ref).max() < (1e-5 if n_tokens <= 8 else TOL)
    assert be.last_active_experts() == len(np.unique(ref_idx))


# 128 row tiles a token: the Q4_K down kernel runs with two CTAs per SM at 2 and 4 tokens, with three at 3.
@pytest.mark.parametrize("n_tokens", [2, 3, 4, 8])
def test_per_row_q4k_down_around_a_wave(n_tokens, port_lib, ref_silu_table):
    from tie_b200 import moe
    s = synth.MoeShape(hidden=2048, n_expert=128, top_k=8, ffn_dim=256)
    q6 = synth.make_layer(workloads.BASE_SEED + 6, s)
    down = synth.q4k_blocks(6, synth.STREAM_DOWN, s.n_expert * s.hidden * (s.ffn_dim // 256))
    layer = synth.MoeLayer(s, q6.router_w, q6.gate, q6.up, down, gate_type=synth.GGML_Q4_K, up_type=synth.GGML_Q4_K, down_type=synth.GGML_Q4_K)
    b = moe.MoeBackend(ffn_dim=s.ffn_dim, max_tokens=8, silu_table=ref_silu_table)
    b.upload_layer(0, layer, keep_host=True)
    x = synth.make_x(0, n_tokens, first_token=50)
    ref, _, _ = port_lib.PortMoe(layer, silu=ref_silu_table).moe_ffn(x)
    out = b.moe_ffn(0, x)
    b.close()
    assert workloads.rel_rms_err(out, ref).max() < 1e-5


# Rows per expert at the edges of 16-, 32- and 64-row tiles: tiles of 32 up to 24 rows an expert on average, of 64
# above; the dispatch sort is one CTA up to 1024 rows.
_EDGES = [0, 1, 15, 16, 17, 31, 32, 33, 63, 64, 65]


@pytest.mark.parametrize("flags", [0, "no_pair"])
@pytest.mark.parametrize("counts", [_EDGES, _EDGES + [48] * 9, _EDGES + [127, 128, 129, 1, 47], [32] * 32, [32] * 31 + [31], [32] * 31 + [33]],
                         ids=["337rows", "769rows", "769rows_wide", "1024rows", "1023rows", "1025rows"])
def test_grouped_tile_edges(grouped, counts, flags):
    import torch
    from tie_b200 import moe
    b, port, s = grouped
    row_expert = np.repeat(np.arange(len(counts), dtype=np.int32), counts)
    row_expert = row_expert[np.random.default_rng(11).permutation(row_expert.size)]
    rows = synth.make_x(13, row_expert.size, s.hidden)
    ref = port.expert_rows(rows, row_expert)
    x, e = torch.from_numpy(rows).cuda(), torch.from_numpy(row_expert).cuda()
    y = torch.full_like(x, float("nan"))
    b.expert_rows_ptr(0, x, e, row_expert.size, y, moe.DEVICE | moe.PATH_TENSOR | (moe.PATH_NO_PAIR if flags else 0))
    # (a row whose gates are all far below zero has no output to speak of: relative to the usual row then)
    rms = np.sqrt((ref.astype(np.float64) ** 2).mean(1))
    assert (np.abs(y.cpu().numpy() - ref).max(1) / np.maximum(rms, 1e-2 * np.median(rms))).max() < TOL


# One registered tensor: its batch in tiles of 64, or of 32 where 64 leave SMs idle; Q4_K rows beyond 2048 inputs
# (9 super-blocks: a second segment of the input sums).
@pytest.mark.parametrize("ggml_type,in_dim,out_dim", [(12, 2304, 256), (14, 512, 256), (12, 256, 9472)])
@pytest.mark.parametrize("batch", [1, 32, 33, 64, 65, 129])
def test_dense_batches(be, port_lib, ggml_type, in_dim, out_dim, batch):
    nb = out_dim * (in_dim // 256)
    w = np.ascontiguousarray(synth.q4k_blocks(78, 9, nb) if ggml_type == 12 else synth.q6k_blocks(78, 9, nb))
    be.register_tensor(w, ggml_type, in_dim)
    x = synth.make_x(4, batch, in_dim)
    rows = sorted({0, batch // 2, batch - 1, min(31, batch - 1), min(32, batch - 1)})
    ref = np.stack([port_lib.mat_vec(x[i], w, ggml_type, in_dim, out_dim) for i in rows])
    got = be.mat_mat(w, x, np.full((batch, out_dim), np.nan, dtype=np.float32), batch, in_dim, out_dim)
    scale = np.sqrt((ref.astype(np.float64) ** 2).mean(axis=1, keepdims=True))
    assert (np.abs(got[rows] - ref) / scale).max() < TOL
    assert np.isfinite(got).all()


# Pageable buffers of 256 KB (32 tokens) and more go through the chunked copies; pinned ones do not.
@pytest.mark.parametrize("n_tokens", [1, 31, 32, 33, 333])
@pytest.mark.parametrize("pinned", [(False, False), (True, False), (False, True), (True, True)])
def test_host_buffers_pageable_and_pinned(be, n_tokens, pinned):
    import torch
    from tie_b200 import moe
    x = torch.from_numpy(synth.make_x(0, n_tokens, first_token=400))
    want = torch.empty(n_tokens, 2048, device="cuda")
    be.moe_ffn_ptr(0, x.cuda(), want, n_tokens, moe.DEVICE)
    xh = x.pin_memory() if pinned[0] else x
    out = torch.full((n_tokens, 2048), float("nan"), pin_memory=pinned[1])
    for _ in range(2):
        be.moe_ffn_ptr(0, xh, out, n_tokens, moe.HOST)
        assert np.array_equal(bits(out.numpy()), bits(want.cpu().numpy()))
        out.fill_(float("nan"))


# The threads that help copying a pageable batch sleep once the call has returned: the process uses no processor time while
# its caller sleeps (three helpers that poll on for 400 us would take up to 24 ms in 20 calls).
def test_copy_helpers_sleep_after_the_call(be):
    import time
    from tie_b200 import moe
    x = synth.make_x(0, 333)
    out = np.empty_like(x)
    used = 0.0
    for _ in range(20):
        be.moe_ffn_ptr(0, x, out, 333, moe.HOST | moe.GRAPH)
        t0 = time.process_time()
        time.sleep(0.002)
        used += time.process_time() - t0
    assert used < 6e-3


# One launch for a run of blocks with the same gate / up kind: down tensors of both kinds in it, and a block in the
# middle that needs a launch of its own.
def test_one_token_stack_of_mixed_blocks(small_shape, ref_silu_table):
    import torch
    from tie_b200 import moe
    s = small_shape
    n_gu, n_dn = s.n_expert * s.ffn_dim * (s.hidden // 256), s.n_expert * s.hidden * (s.ffn_dim // 256)
    b = moe.MoeBackend(hidden=s.hidden, n_expert=s.n_expert, top_k=s.top_k, ffn_dim=s.ffn_dim, max_tokens=4, silu_table=ref_silu_table,
                       n_layers=7)
    try:
        for l in range(7):
            m = synth.make_layer(30 + l, s)
            if l in (1, 2, 5):
                m.down, m.down_type = synth.q4k_blocks(30 + l, synth.STREAM_DOWN, n_dn), synth.GGML_Q4_K
            if l == 3:
                m.gate, m.gate_type = synth.q6k_blocks(33, synth.STREAM_GATE, n_gu), synth.GGML_Q6_K
                m.up, m.up_type = synth.q6k_blocks(33, synth.STREAM_UP, n_gu), synth.GGML_Q6_K
            b.upload_layer(l, m, ffn_norm_w=None if l == 4 else np.linspace(0.9, 1.1, s.hidden, dtype=np.float32))
        h0 = torch.from_numpy(synth.make_x(6, 1, s.hidden)).cuda()
        want, got = h0.clone(), h0.clone()
        for l in range(7):
            b.moe_block_inplace_ptr(l, want, 1, moe.DEVICE)
        l0 = b.launch_count
        b.moe_stack_inplace_ptr(0, 7, got, 1, moe.DEVICE)
        assert b.launch_count - l0 == 3
        assert np.array_equal(bits(got.cpu().numpy()), bits(want.cpu().numpy())) and np.isfinite(got.cpu().numpy()).all()
    finally:
        b.close()


# One token on host buffers: the result comes without a copy, also when the stream is still busy and from a graph.
def test_one_token_host_calls(be):
    import torch
    from tie_b200 import moe
    out = np.empty((1, 2048), np.float32)
    big = torch.from_numpy(synth.make_x(0, 1100)).cuda()
    big_out = torch.empty_like(big)
    for i in range(4):
        x = synth.make_x(0, 1, first_token=700 + i)
        want = torch.empty(1, 2048, device="cuda")
        be.moe_ffn_ptr(0, torch.from_numpy(x).cuda(), want, 1, moe.DEVICE)
        for flags in (0, moe.GRAPH):
            for _ in range(3):
                be.moe_ffn_ptr(0, big, big_out, 1100, moe.DEVICE | moe.NO_SYNC)
            out[:] = np.nan
            be.moe_ffn_ptr(0, x, out, 1, moe.HOST | flags)
            assert np.array_equal(bits(out), bits(want.cpu().numpy()))


# Up to some 70 tokens the router makes the RMSNorm of a block's tokens itself: the same bits as behind the norm kernel (what the
# chain flag asks for), around the router's tiles of 4 and 8 tokens, rows of fewer float4 than its threads, and above its last size.
@pytest.mark.parametrize("hidden", [512, 1536, 2048])
@pytest.mark.parametrize("n_tokens", [2, 3, 4, 5, 8, 9, 31, 33, 63, 65, 90])
def test_block_norm_inside_the_router(hidden, n_tokens, ref_silu_table):
    import torch
    from tie_b200 import moe
    s = synth.MoeShape(hidden=hidden, n_expert=32, top_k=4, ffn_dim=256)
    b = moe.MoeBackend(hidden=s.hidden, n_expert=s.n_expert, top_k=s.top_k, ffn_dim=s.ffn_dim, max_tokens=96, silu_table=ref_silu_table)
    try:
        b.upload_layer(0, synth.make_layer(40, s), ffn_norm_w=np.linspace(0.5, 1.5, s.hidden, dtype=np.float32))
        h0 = torch.from_numpy(synth.make_x(8, n_tokens, s.hidden)).cuda()
        want, got = h0.clone(), h0.clone()
        b.moe_block_inplace_ptr(0, want, n_tokens, moe.DEVICE | moe.PATH_DECODE_CHAIN)
        b.moe_block_inplace_ptr(0, got, n_tokens, moe.DEVICE)
        assert np.array_equal(bits(got.cpu().numpy()), bits(want.cpu().numpy())) and not torch.equal(got, h0)
    finally:
        b.close()


# RMSNorm of rows of one CTA each: hidden below, at and above what its threads keep in registers (2048).
@pytest.mark.parametrize("hidden", [512, 2048, 2304])
def test_rms_norm_row_lengths(hidden, port_lib, ref_silu_table):
    import torch
    from tie_b200 import moe
    s = synth.MoeShape(hidden=hidden, n_expert=16, top_k=2, ffn_dim=256)
    layer = synth.make_layer(17, s)
    norm = np.linspace(0.8, 1.2, hidden, dtype=np.float32)
    b = moe.MoeBackend(hidden=hidden, n_expert=16, top_k=2, ffn_dim=256, max_tokens=8, silu_table=ref_silu_table)
    try:
        b.upload_layer(0, layer, ffn_norm_w=norm)
        h0 = synth.make_x(18, 5, hidden)
        normed = np.stack([port_lib.rms_norm(h0[i], norm, 1e-6) for i in range(5)])
        ref = h0 + port_lib.PortMoe(layer, silu=ref_silu_table).moe_ffn(normed)[0]
        h = torch.from_numpy(h0.copy()).cuda()
        b.moe_block_inplace_ptr(0, h, 5, moe.DEVICE)
        assert workloads.rel_rms_err(h.cpu().numpy(), ref).max() < TOL
    finally:
        b.close()


# Below twice as many rows as experts every product is exact to fp32, as for one token: rows grouped by expert, four to
# a group (8 tokens on with 128 experts and top-8), have the bits of their tokens alone, whichever experts they share.
@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("n_tokens", [7, 8, 9, 20, 31])
def test_small_batches_have_the_bits_of_single_tokens(be, port0, n_tokens, shared):
    x = synth.make_x(0, n_tokens, first_token=600)
    bias = None
    if shared:  # all tokens on the same eight experts: groups of four and a remainder
        bias = np.zeros(128, dtype=np.float32)
        bias[[0, 3, 17, 44, 45, 90, 126, 127]] = 1000.0
    out = be.moe_ffn(0, x, router_bias=bias)
    active = be.last_active_experts()
    alone = np.concatenate([be.moe_ffn(0, x[i:i + 1], router_bias=bias) for i in range(n_tokens)])
    assert np.array_equal(bits(out), bits(alone))
    ref, ref_idx, _ = port0.moe_ffn(x, router_bias=bias)
    assert workloads.rel_rms_err(out, ref).max() < 1e-5
    assert active == len(np.unique(ref_idx))


# Activations far from 1, and Q6_K scales over their whole range (products beyond 11 bits), with every kind of tensor.  The
# CPU restatement itself is up to 1.0e-5 from 64-bit arithmetic at 0.03 (SwiGLU rounds gate + 10) and 1.4e-6 at 1 and 2e4.
@pytest.mark.parametrize("kinds", ["q4k_q6k", "q6k_q4k", "q4k_q4k"])
@pytest.mark.parametrize("scale", [0.03, 1.0, 2e4])
@pytest.mark.parametrize("n_tokens", [5, 9, 15])
def test_small_batches_over_the_range_of_activations(n_tokens, scale, kinds, small_shape, port_lib, ref_silu_table):
    import torch
    from tie_b200 import moe
    s = small_shape  # 32 experts, top-4: grouped from 5 to 15 tokens
    n_gu, n_dn = s.n_expert * s.ffn_dim * (s.hidden // 256), s.n_expert * s.hidden * (s.ffn_dim // 256)

    def blocks(kind, stream, n):
        if kind == "q4k":
            return synth.q4k_blocks(55, stream, n), synth.GGML_Q4_K
        b = np.array(synth.q6k_blocks(55, stream, n)).reshape(n, synth.Q6K_BYTES)
        b[:, 192:208] = np.random.default_rng(stream).integers(-128, 128, (n, 16), dtype=np.int8).view(np.uint8)
        return b.reshape(-1), synth.GGML_Q6_K

    gu, dn = kinds.split("_")
    (gate, gt), (up, _), (down, dt) = blocks(gu, synth.STREAM_GATE, n_gu), blocks(gu, synth.STREAM_UP, n_gu), blocks(dn, synth.STREAM_DOWN, n_dn)
    layer = synth.MoeLayer(s, synth.make_layer(55, s).router_w, gate, up, down, gate_type=gt, up_type=gt, down_type=dt)
    b = moe.MoeBackend(hidden=s.hidden, n_expert=s.n_expert, top_k=s.top_k, ffn_dim=s.ffn_dim, max_tokens=16, silu_table=ref_silu_table)
    try:
        b.upload_layer(0, layer, keep_host=True)
        x = synth.make_x(9, n_tokens, s.hidden) * np.float32(scale)
        ref, _, _ = port_lib.PortMoe(layer, silu=ref_silu_table).moe_ffn(x)
        out = b.moe_ffn(0, x)
        assert np.isfinite(out).all() and workloads.rel_rms_err(out, ref).max() < (3e-5 if scale < 1 else 1e-5)
        # as many rows through the building block of expert parallelism (rows without an output to speak of: see above)
        rows, row_expert = np.repeat(x, s.top_k, axis=0), np.random.default_rng(3).integers(0, s.n_expert, n_tokens * s.top_k).astype(np.int32)
        y = torch.empty(rows.shape, device="cuda")
        b.expert_rows_ptr(0, torch.from_numpy(rows).cuda(), torch.from_numpy(row_expert).cuda(), len(rows), y, moe.DEVICE)
        y_ref = port_lib.PortMoe(layer, silu=ref_silu_table).expert_rows(rows, row_expert)
        rms = np.sqrt((y_ref.astype(np.float64) ** 2).mean(1))
        assert (np.abs(y.cpu().numpy() - y_ref).max(1) / np.maximum(rms, 1e-2 * np.median(rms))).max() < (1e-4 if scale < 1 else 3e-5)
        alone = np.concatenate([b.moe_ffn(0, x[i:i + 1]) for i in range(n_tokens)])
        assert np.array_equal(bits(out), bits(alone))
    finally:
        b.close()
