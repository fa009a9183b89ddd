"""Kernels at the sizes where they can go wrong: edges of tiles, remainders, one-tile and many-tile
launches, through the C ABI."""
import ctypes as C

import numpy as np
import pytest

from conftest import rel_err
from test_gpu_parity import _attn_case

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,M,N,K", [(0, 20480, 1544, 520), (0, 33000, 768, 64), (0, 20481, 1000, 1096), (1, 20483, 1032, 136),
                                        (2, 5000, 5008, 72), (2, 6144, 1032, 2056), (0, 19200, 1024, 8)])
@pytest.mark.parametrize("c_f32", [0, 1])
def test_many_tile_gemm_vs_fp32(pkg, mode, M, N, K, c_f32):
    """More output tiles than CTA pairs: ragged last rows, columns and k-blocks, one k-block alone (no
    odd chain), every operand arrangement, both output types."""
    lib = pkg.library()
    g = torch.Generator(device="cuda").manual_seed(M + N + K + mode)
    a = torch.randn((K, M) if mode == 2 else (M, K), generator=g, device="cuda").bfloat16()
    if mode == 2 and M % 8:
        pytest.skip("rows of a transposed operand are 16-byte aligned")
    b = torch.randn((N, K) if mode == 0 else (K, N), generator=g, device="cuda").bfloat16()
    ref = (a.float().T if mode == 2 else a.float()) @ (b.float().T if mode == 0 else b.float())
    c = torch.full((M, N), float("nan"), device="cuda", dtype=torch.float32 if c_f32 else torch.bfloat16)
    assert lib.nncu_gemm_bf16(pkg.abi.GEMM_TCGEN05, mode, M, N, K, a.data_ptr(), a.shape[1], b.data_ptr(), b.shape[1],
                              c.data_ptr(), N, c_f32, None) == 0, lib.nncu_last_error()
    assert (c.float() - ref).abs().max().item() < (5e-5 if c_f32 else 5e-3) * ref.abs().max().item()
    if mode == 0:   # the rows of a one-tile launch, which takes the other kernel, are the same bits
        part = torch.zeros(40, N, device="cuda", dtype=c.dtype)
        off = M - 40
        assert lib.nncu_gemm_bf16(pkg.abi.GEMM_TCGEN05, 0, 40, N, K, a[off:].data_ptr(), K, b.data_ptr(), K,
                                  part.data_ptr(), N, c_f32, None) == 0, lib.nncu_last_error()
        assert torch.equal(part, c[off:])


@pytest.mark.parametrize("B,H,dk,T,M,P,alen", [(1, 1, 64, 1, 1, 2, 0), (2, 1, 64, 64, 65, 129, 0), (1, 2, 32, 16, 48, 33, 0),
                                               (2, 1, 128, 64, 256, 300, 0), (3, 1, 16, 17, 64, 81, 30), (1, 2, 128, 64, 1, 65, 2)])
def test_attention_edges_bf16(pkg, oracle, B, H, dk, T, M, P, alen):
    """One query, one key more than the blocks hold, a table that ends inside the left pad, a window of two keys."""
    _attn_case(pkg, oracle, B, H, dk, T, M, P, alen, True, 7)


@pytest.mark.parametrize("dk,T,M,P,alen", [(16, 20, 100, 50, 0), (32, 64, 300, 364, 0), (64, 64, 513, 577, 0), (64, 70, 64, 90, 100),
                                           (128, 33, 256, 289, 200)])
def test_attention_single_queries_equal_the_segment_bitwise(pkg, dk, T, M, P, alen):
    """The one-query kernel against the segment kernel, every query: output and log-sum-exp bit for bit."""
    lib = pkg.library()
    B, H, L = 3, 2, T + M
    g = torch.Generator(device="cuda").manual_seed(dk + T + M)
    q = torch.randn(T * B, H * dk, generator=g, device="cuda").bfloat16()
    kv = torch.randn(L * B, 2 * H * dk, generator=g, device="cuda").bfloat16()
    w_r = 0.1 * torch.randn(H, P, dk, generator=g, device="cuda")
    b_r = 0.1 * torch.randn(H, L, generator=g, device="cuda")
    outs = []
    for ranges in ([(0, T)], [(t, t + 1) for t in range(T)]):
        out, lse = torch.zeros_like(q), torch.zeros(B * H, T, device="cuda")
        for t0, t1 in ranges:
            shp = pkg.abi.AttnShape(B, H, dk, T, M, P, alen, t0, t1, float(np.sqrt(dk * 512.0)), 1)
            assert lib.nncu_attention_forward(C.byref(shp), q.data_ptr(), kv.data_ptr(), w_r.data_ptr(), b_r.data_ptr(),
                                              out.data_ptr(), lse.data_ptr(), None) == 0, lib.nncu_last_error()
        torch.cuda.synchronize()
        outs.append((out, lse))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


def test_attention_edges_fp32(pkg, oracle):
    """The CUDA-core kernels: a head size that is no multiple of four, one that fills the shared memory up
    to the narrow row pitch, a left pad of most of the table."""
    for B, H, dk, T, M, P, alen in ((2, 2, 6, 7, 9, 16, 0), (1, 1, 64, 32, 120, 152, 0), (2, 1, 32, 31, 40, 3, 20)):
        _attn_case(pkg, oracle, B, H, dk, T, M, P, alen, False, 8)


@pytest.mark.parametrize("ln,act,D,n_head", [(1, 1, 256, 4), (2 | 4 | 16, 2, 384, 3)])
def test_gradients_of_a_long_memory_match_the_other_engine(pkg, ln, act, D, n_head):
    """Projection gradients over 9216 rows: the memory rows' query part is left out in both passes, the
    contraction is split over idle CTA pairs; rows that are no multiple of 512 bytes go through the norms."""
    kw = dict(n_layer=1, d_model=D, n_head=n_head, d_key=D // n_head, d_inner=2 * D, d_pos=192, mem_len=128, seg_len=64,
              n_streams=48, n_symbols=512, use_bf16=1, init_range=0.05, ln_flags=ln, ff_act=act)
    rng = np.random.default_rng(3)
    ids, tg = (rng.integers(0, 512, (3, 64, 48)).astype(np.int32) for _ in range(2))
    got = []
    for backend in (1, 2):
        m = pkg.TrfModel(pkg.abi.make_params(gemm_backend=backend, **kw))
        m.reset()
        for s in range(3):
            m.eval(-1, ids[s], read=False)
            loss = m.eval_gradient(tg[s])
            m.memory_shift()
        got.append(({n: m.get_grad(n) for n in m.info}, loss))
        m.close()
    assert abs(got[0][1] - got[1][1]) < 1e-3 * abs(got[0][1])
    for n in got[0][0]:
        assert rel_err(got[1][0][n], got[0][0][n]) < 2e-2, n


@pytest.mark.parametrize("kw", [
    dict(n_layer=3, d_model=96, n_head=3, d_key=32, d_inner=208, d_pos=20, mem_len=17, seg_len=9, n_streams=1, n_symbols=256),
    dict(n_layer=2, d_model=256, n_head=8, d_key=32, d_inner=1024, d_pos=32, mem_len=32, seg_len=8, n_streams=16, n_symbols=256),
    dict(n_layer=2, d_model=512, n_head=4, d_key=64, d_inner=272, d_pos=9, mem_len=5, seg_len=7, n_streams=19, n_symbols=300, ff_act=0),
    dict(n_layer=2, d_model=64, n_head=1, d_key=16, d_inner=64, d_pos=4, mem_len=0, seg_len=6, n_streams=50, n_symbols=37, use_w_r=0,
         use_bias=0, query_bias=0),
    dict(n_layer=1, d_model=48, n_head=12, d_key=4, d_inner=16, d_pos=20, mem_len=40, seg_len=5, n_streams=56, n_symbols=64, attn_len=[11])])
def test_one_launch_steps_equal_whole_segment_bitwise(pkg, kw):
    """The one-launch time step of small fp32 models, one to four streams per cluster: probabilities, and
    through the gradients everything it leaves for the backward pass, bit for bit those of the segment."""
    p = pkg.abi.make_params(use_bf16=0, init_range=0.3, lr=1e-3, **kw)
    T, B, V = p.seg_len, p.n_streams, p.n_symbols
    rng = np.random.default_rng(3)
    seg, one = pkg.TrfModel(p), pkg.TrfModel(p)
    seg.reset(); one.reset()
    for _ in range(3):   # both memory twins
        ids, tg = rng.integers(0, V, (T, B)).astype(np.int32), rng.integers(0, V, (T, B)).astype(np.int32)
        a = seg.eval(-1, ids)
        b = np.concatenate([one.eval(t, ids) for t in range(T)])
        assert np.array_equal(a, b)
        for m in (seg, one):
            m.eval_gradient(tg)
            m.update()
        assert seg.weights_hash() == one.weights_hash()
    seg.close(); one.close()


@pytest.mark.parametrize("V", [16, 256, 300, 16384])
def test_decoder_walk_of_improbable_branches(pkg, V):
    """Trees of nearly certain branches and payloads that keep taking the others (two payload bytes a bit), over the
    end of the payload: the device's symbols against the host's walk of the same trees."""
    p = pkg.abi.make_params(n_layer=1, d_model=64, n_head=2, d_key=32, d_inner=64, d_pos=8, mem_len=8, seg_len=4, n_streams=7,
                            n_symbols=V, init_range=0.05)
    T, B, L = 4, 7, pkg.host.library()
    rng = np.random.default_rng(V)
    bias = np.zeros(V, np.float32)
    bias[rng.integers(0, V, max(2, V // 8))] = 25.0
    for payload in (b"\xff" * 900, b"\x00" * 900, b"\x00\xff\xfe" * 300, bytes(rng.integers(0, 2, 900, dtype=np.uint8) * 255), b"\xff" * 40):
        dev, ref = pkg.TrfModel(p), pkg.TrfModel(p)
        for m in (dev, ref):
            m.set_param("out_bias", bias)
            m.reset()
        dev.decoder_begin(payload)
        got = dev.decode_steps(0, T, np.zeros(B, np.int32))
        buf = C.create_string_buffer(payload, len(payload))
        hd, ids, want = L.nch_dec_new(buf, len(payload)), np.zeros((T, B), np.int32), np.zeros((T, B), np.int32)
        for t in range(T):
            ids[t] = want[t - 1] if t else 0
            ref.eval(t, ids, read=False)
            trees = np.ascontiguousarray(ref.coder_trees(t, 1))
            for b in range(B):
                want[t, b] = L.nch_read_sym_tree(hd, trees[b].ctypes.data_as(C.c_void_p), V)
        L.nch_dec_free(hd)
        assert np.array_equal(got, want)
        dev.decoder_end()
        dev.close(); ref.close()


@pytest.mark.parametrize("V", [257, 511, 514, 1027, 2050, 4099, 8191, 9208, 16383])
def test_coder_paths_of_any_alphabet_by_subtrees(pkg, oracle, V):
    """Every depth that the kernel of 256 subtrees takes (9 to 14), least and most two-symbol nodes, rows on and off
    16-byte boundaries: the integers of write_sym, equal."""
    m = pkg.TrfModel(pkg.abi.make_params(n_layer=1, d_model=64, n_head=2, d_key=32, d_inner=128, d_pos=16, mem_len=8, seg_len=8,
                                         n_streams=3, n_symbols=V, init_range=0.5))
    rng = np.random.default_rng(V)
    ids, syms = (rng.integers(0, V, (8, 3)).astype(np.int32) for _ in range(2))
    syms[0], syms[1] = [0, V - 1, V // 2], [V // 2 - 1, V // 256, V // 256 + 1]
    probs, paths = m.eval(-1, ids), m.coder_paths(0, 8, syms)
    for t in range(8):
        for b in range(3):
            want = oracle.sym_path(probs[t, b], syms[t, b])
            got = paths[t * 3 + b]
            assert np.array_equal(got[:len(want)], want) and not got[len(want):].any(), (t, b)
    m.close()


@pytest.mark.parametrize("kw", [
    dict(d_model=256, n_head=4, d_key=64, d_pos=150, mem_len=130, seg_len=20, n_streams=130),                        # three key blocks
    dict(d_model=256, n_head=4, d_key=64, d_pos=40, mem_len=130, seg_len=20, n_streams=130),                         # copies of table row 0
    dict(d_model=256, n_head=2, d_key=128, d_pos=90, mem_len=64, seg_len=26, n_streams=256),
    dict(d_model=256, n_head=2, d_key=128, d_pos=220, mem_len=200, seg_len=20, n_streams=256, attn_len=[70, 1]),     # windows
    dict(d_model=128, n_head=2, d_key=64, d_pos=5, mem_len=0, seg_len=5, n_streams=256, use_w_r=0)])                 # one key, no table
def test_one_query_by_a_warp_equals_whole_segment_bitwise(pkg, kw):
    """Time steps of many streams: a warp for every (stream, head), against the segment kernel, bit for bit."""
    p = pkg.abi.make_params(n_layer=2, d_inner=256, n_symbols=64, use_bf16=1, init_range=0.3, lr=1e-3, **kw)
    T, B, V = p.seg_len, p.n_streams, p.n_symbols
    rng = np.random.default_rng(5)
    seg, one = pkg.TrfModel(p), pkg.TrfModel(p)
    seg.reset(); one.reset()
    for _ in range(3):
        ids, tg = rng.integers(0, V, (T, B)).astype(np.int32), rng.integers(0, V, (T, B)).astype(np.int32)
        a = seg.eval(-1, ids)
        assert np.array_equal(a, np.concatenate([one.eval(t, ids) for t in range(T)]))
        for m in (seg, one):
            m.eval_gradient(tg)
            m.update()
        assert seg.weights_hash() == one.weights_hash()
    seg.close(); one.close()


@pytest.mark.parametrize("mode,M,N,K", [(0, 2048, 1024, 1024), (0, 2000, 1000, 72), (1, 1930, 1032, 136), (2, 2056, 1000, 1096), (0, 18900, 72, 520),
                                        (0, 2041, 1016, 8)])
@pytest.mark.parametrize("c_f32", [0, 1])
def test_one_round_gemm_vs_fp32(pkg, mode, M, N, K, c_f32):
    """Outputs of 75 to 148 tiles of 128 x 128, one to an SM: ragged edges, one k-block to more than the ring holds, and
    the rows of a launch that takes narrower tiles."""
    lib = pkg.library()
    g = torch.Generator(device="cuda").manual_seed(M + N + K + mode)
    a = torch.randn((K, M) if mode == 2 else (M, K), generator=g, device="cuda").bfloat16()
    b = torch.randn((N, K) if mode == 0 else (K, N), generator=g, device="cuda").bfloat16()
    ref = (a.float().T if mode == 2 else a.float()) @ (b.float().T if mode == 0 else b.float())
    c = torch.full((M, N), float("nan"), device="cuda", dtype=torch.float32 if c_f32 else torch.bfloat16)
    assert lib.nncu_gemm_bf16(pkg.abi.GEMM_TCGEN05, mode, M, N, K, a.data_ptr(), a.shape[1], b.data_ptr(), b.shape[1],
                              c.data_ptr(), N, c_f32, None) == 0, lib.nncu_last_error()
    assert (c.float() - ref).abs().max().item() < (5e-5 if c_f32 else 5e-3) * ref.abs().max().item()
    if mode == 0:
        part = torch.zeros(40, N, device="cuda", dtype=c.dtype)
        off = M - 40
        assert lib.nncu_gemm_bf16(pkg.abi.GEMM_TCGEN05, 0, 40, N, K, a[off:].data_ptr(), K, b.data_ptr(), K,
                                  part.data_ptr(), N, c_f32, None) == 0, lib.nncu_last_error()
        assert torch.equal(part, c[off:])


@pytest.mark.parametrize("B,H,dk,T,M,P,alen", [(1, 1, 16, 64, 20, 84, 0), (2, 2, 32, 40, 30, 50, 0), (3, 2, 8, 16, 40, 56, 21), (1, 3, 6, 15, 9, 20, 0),
                                               (75, 2, 8, 16, 5, 21, 0), (37, 2, 16, 33, 8, 41, 0), (1, 2, 32, 32, 1, 33, 2)])
def test_fp32_attention_by_clusters(pkg, oracle, B, H, dk, T, M, P, alen):
    """One to eight CTAs per (stream, head): as many as the shape gives, rows and results that do not divide evenly.  (Of a window of
    one key the gradients of queries and keys are rounding only: dS = P (dP - D) is zero.)"""
    _attn_case(pkg, oracle, B, H, dk, T, M, P, alen, False, 9)


@pytest.mark.parametrize("kw", [dict(n_layer=1), dict(n_layer=2), dict(n_layer=3), dict(n_layer=5, ln_flags=2 | 4 | 16, ff_act=2),
                                dict(n_layer=3, use_bf16=0), dict(n_layer=4, use_bf16=0, tied_w_r=1, tied_b_r=1),
                                dict(n_layer=4, ln_flags=1 | 8), dict(n_layer=5, ln_flags=2 | 4 | 8, attn_len=[48, 20, 7, 33, 1])])
def test_gradients_with_and_without_the_side_stream_are_the_same_bits(pkg, monkeypatch, kw):
    """Weight gradients and reductions run up to two layers behind the main stream, from buffers that layers take in
    turn: every gradient of several steps and models, against one stream."""
    base = dict(d_model=256, n_head=4, d_key=64, d_inner=512, d_pos=48, mem_len=16, seg_len=32, n_streams=4, n_symbols=512,
                use_bf16=1, lr=1e-3, init_range=0.03)
    p = pkg.abi.make_params(**dict(base, **kw))
    rng = np.random.default_rng(2)
    steps = [tuple(rng.integers(0, 512, (32, 4)).astype(np.int32) for _ in range(2)) for _ in range(3)]

    def run():
        m, got = pkg.TrfModel(p), []
        m.reset()
        for ids, tg in steps:
            m.eval(-1, ids, read=False)
            m.eval_gradient(tg)
            got.append({n: m.get_grad(n) for n in m.info})
            m.update()
        m.close()
        return got

    monkeypatch.setenv("NNCU_NO_OVERLAP", "1")
    want = run()
    monkeypatch.delenv("NNCU_NO_OVERLAP")
    for _ in range(6):
        for a, b in zip(want, run()):
            for n in a:
                assert np.array_equal(a[n], b[n]), n


@pytest.mark.parametrize("B,H,dk,T,M,P,alen", [(1, 1, 64, 64, 64, 128, 0), (2, 1, 64, 64, 65, 100, 0), (3, 2, 64, 1, 127, 128, 0), (40, 4, 64, 33, 160, 193, 0),
                                               (1, 2, 64, 63, 400, 30, 90), (2, 2, 128, 64, 192, 256, 0), (1, 1, 128, 17, 112, 60, 0),
                                               (75, 2, 128, 16, 130, 146, 0), (1, 2, 128, 64, 500, 564, 70)])
def test_attention_adjoint_on_128_key_blocks_bf16(pkg, oracle, B, H, dk, T, M, P, alen):
    """The persistent kernel of head sizes 64 and 128: whole and ragged key blocks, one query, more (stream, head) pairs
    than CTAs, tables that end inside the left pad, windows that leave whole blocks out."""
    _attn_case(pkg, oracle, B, H, dk, T, M, P, alen, True, 11)


@pytest.mark.parametrize("B,H,dk,T,M,P,alen", [(1, 2, 64, 64, 1368, 1432, 0), (1, 2, 64, 64, 1369, 1433, 0), (1, 2, 64, 40, 1393, 700, 0), (2, 1, 64, 64, 1400, 1464, 200),
                                               (1, 2, 128, 64, 1240, 1304, 0), (1, 2, 128, 64, 1241, 1305, 0), (1, 1, 128, 33, 1300, 500, 0),
                                               (1, 2, 128, 64, 1250, 1314, 130)])
def test_attention_adjoint_where_b_r_outgrows_its_place_bf16(pkg, oracle, B, H, dk, T, M, P, alen):
    """The most keys whose two copies of b_r fit beside the tiles of 128 keys (1432 at head size 64, 1304 at 128), one more, and more than
    that: the warp-level kernel, with tables that end inside the left pad and with windows."""
    _attn_case(pkg, oracle, B, H, dk, T, M, P, alen, True, 13)


@pytest.mark.parametrize("B,H,dk,T,M,P,alen", [(40, 4, 64, 20, 30, 50, 0), (20, 8, 64, 64, 0, 40, 0), (40, 4, 64, 16, 150, 166, 0), (38, 4, 64, 9, 170, 100, 0),
                                               (19, 8, 64, 33, 90, 123, 20), (37, 4, 64, 20, 30, 50, 0)])
def test_attention_adjoint_of_short_windows_bf16(pkg, oracle, B, H, dk, T, M, P, alen):
    """Head size 64, more pairs than SMs: one 64-key block, three of them for one tile of queries, two that a window puts into two
    128-key blocks; and one block with a pair to an SM."""
    _attn_case(pkg, oracle, B, H, dk, T, M, P, alen, True, 12)


@pytest.mark.parametrize("kw", [
    dict(n_head=8, n_streams=74, d_pos=64),                                       # four pairs to a CTA, heads that start in mid-CTA
    dict(n_head=8, n_streams=75, d_pos=50),                                       # four or five; copies of table row 0
    dict(n_head=9, n_streams=66, d_pos=324, mem_len=300, attn_len=[60]),          # a window: zero rows of the table
    dict(n_head=9, n_streams=66, d_pos=310, mem_len=300, n_layer=4, attn_len=[60, 324, 90, 25]),  # layers in turn over the same partials
    dict(n_head=12, n_streams=50, d_pos=33, d_key=128, n_layer=2, tied_w_r=1),    # one table of two layers
    dict(n_head=200, n_streams=3, d_pos=64),                                      # several heads' ends in a CTA
    dict(n_head=8, n_streams=73, d_pos=64)])                                      # a part for each stream
def test_position_table_gradients_summed_over_streams(pkg, kw):
    """The table's gradient where CTAs of the adjoint sum the streams they take, element by element against two models that have
    half the streams each, which write a part for each stream.  Every row of activations and gradients has the same bits in both, so
    what differs is the association of at most 75 fp32 parts (a layer): 75 x 2^-24 of the sum of their magnitudes, which for parts
    of random sign is some sqrt(75) times the sum: 4e-5 of the head's largest element (2^-24 x 75 x 8.7), and a tied table's two layers
    as much again.  A row that is lost, stale or counted twice is of the size of the others."""
    base = dict(n_layer=1, d_model=128, d_key=64, d_inner=128, mem_len=60, seg_len=24, n_symbols=64, init_range=0.05, use_bf16=1)
    kw = dict(base, **kw)
    B, rng = kw.pop("n_streams"), np.random.default_rng(6)
    ids, tg = (rng.integers(0, 64, (3, 24, B)).astype(np.int32) for _ in range(2))

    def grads(s0, s1):
        p = pkg.abi.make_params(n_streams=s1 - s0, n_streams_total=B, **kw)
        m = pkg.TrfModel(p)
        m.reset()
        for s in range(3):
            m.eval(-1, np.ascontiguousarray(ids[s][:, s0:s1]), read=False)
            m.eval_gradient(np.ascontiguousarray(tg[s][:, s0:s1]))
            m.memory_shift()
        got = {n: m.get_grad(n).reshape(p.n_head, -1).astype(np.float64) for n in m.info if "w_r" in n}
        m.close()
        return got

    whole, halves = grads(0, B), (grads(0, B // 2), grads(B // 2, B))
    assert whole
    for n in whole:
        a, b = whole[n], halves[0][n] + halves[1][n]
        assert (np.abs(a - b) <= 4e-5 * (1 + kw.get("tied_w_r", 0)) * np.abs(b).max(axis=1, keepdims=True)).all(), n


@pytest.mark.parametrize("dk,B,alen,P", [(64, 2, 60, 340), (64, 2, 60, 200), (128, 2, 60, 340), (128, 3, 60, 200), (64, 80, 60, 340)])
def test_adjoint_reads_no_block_that_no_query_sees(pkg, dk, B, alen, P):
    """A window whose first 64-key block is the upper half of a 128-key block (keys 192 on): what the keys before it, and the table
    rows that only they would meet, hold does not matter, and their gradients are zeros even for queries that are not finite."""
    lib = pkg.library()
    H, T, M = 2, 40, 300
    L, HD = T + M, H * dk
    g = torch.Generator(device="cuda").manual_seed(dk + P)
    q, dout = (torch.randn(T * B, HD, generator=g, device="cuda").bfloat16() for _ in range(2))
    kv = torch.randn(L * B, 2 * HD, generator=g, device="cuda").bfloat16()
    w_r, b_r = 0.1 * torch.randn(H, P, dk, generator=g, device="cuda"), 0.1 * torch.randn(H, L, generator=g, device="cuda")
    shp = C.byref(pkg.abi.AttnShape(B, H, dk, T, M, P, alen, 0, T, float(np.sqrt(dk * 512.0)), 1))
    unseen = 192 * B                      # rows of kv
    unmet = max(0, 192 + P - M - 64)      # rows of the table below those of the first block's window

    def run(fill, query=None):
        k, w, x = kv.clone(), w_r.clone(), q.clone()
        k[:unseen] = fill
        w[:, 1:unmet] = fill              # row 0 stands for all rows before the table
        if P == L:
            w[:, :unmet] = fill
        if query is not None:
            x[query] = float("inf")
        out, lse, dq, dkv = torch.zeros_like(q), torch.zeros(B * H, T, device="cuda"), torch.full_like(q, 7), torch.full_like(kv, 7)
        pw, pb = torch.full((B, H, P, dk), 7.0, device="cuda"), torch.full((B, H, L), 7.0, device="cuda")
        ptr = [C.c_void_p(t.data_ptr()) for t in (x, k, w, b_r, out, lse, dout, dq, dkv, pw, pb)]
        assert lib.nncu_attention_forward(shp, *ptr[:6], None) == 0, lib.nncu_last_error()
        assert lib.nncu_attention_backward(shp, *ptr, None) == 0, lib.nncu_last_error()
        torch.cuda.synchronize()
        return out, lse, dq, dkv, pw, pb

    want = run(0.0)
    assert all(t.isfinite().all() for t in want)
    for fill in (float("nan"), float("inf")):
        assert all(torch.equal(a, b) for a, b in zip(want, run(fill)))
    got = run(0.0, query=5 * B)
    assert (got[3][:unseen] == 0).all()
    if P == L:
        assert (got[4][:, :, :unmet] == 0).all()


@pytest.mark.parametrize("dk", [64, 128])
def test_table_rows_that_no_window_meets_do_not_matter_to_a_step(pkg, dk):
    p = pkg.abi.make_params(n_layer=1, d_model=2 * dk, n_head=2, d_key=dk, d_inner=128, d_pos=340, mem_len=300, seg_len=40, n_streams=2, n_symbols=64,
                            use_bf16=1, attn_len=[60], init_range=0.1)
    rng = np.random.default_rng(4)
    ids, tg = (rng.integers(0, 64, (40, 2)).astype(np.int32) for _ in range(2))
    got = []
    for fill in (0.0, float("nan")):
        m = pkg.TrfModel(p)
        w = m.get_param("w_r_0").reshape(2, 340, dk).copy()
        w[:, :168] = fill
        m.set_param("w_r_0", w.reshape(-1))
        m.reset()
        m.eval(-1, ids, read=False)
        m.eval_gradient(tg)
        got.append({n: m.get_grad(n) for n in m.info})
        m.close()
    for n in got[0]:
        assert np.isfinite(got[0][n]).all() and np.array_equal(got[0][n], got[1][n]), n


def test_partial_tables_take_the_room_of_the_sums_that_are_kept(pkg):
    """Many pairs, whose CTAs sum the table's gradient over their streams: a model's memory grows by a few tables with the
    table's length (a table has the same weights, gradients and moments besides), not by one for each stream."""
    def taken(d_pos):
        kw = dict(n_layer=1, d_model=64, n_head=8, d_key=64, d_inner=64, d_pos=d_pos, mem_len=400, seg_len=32, n_streams=128, n_symbols=64, use_bf16=1)
        m = pkg.TrfModel(pkg.abi.make_params(**kw))
        m.close()
        before = torch.cuda.mem_get_info()[0]
        m = pkg.TrfModel(pkg.abi.make_params(**kw))
        now = torch.cuda.mem_get_info()[0]
        m.close()
        return before - now

    table = 8 * 431 * 64 * 4
    # two sets of at most ceil(128 / 6) + 1 parts, and the copies of the parameter; allocations in pieces of 2 MB
    assert taken(432) - taken(1) < (2 * 23 + 4) * table + 4 * 2 ** 20 < 128 * table


@pytest.mark.parametrize("kw", [
    dict(d_model=256, n_head=4, d_key=64, n_streams=100),                           # a warp for every (stream, head)
    dict(d_model=256, n_head=2, d_key=128, n_streams=130, attn_len=[90, 0, 30]),
    dict(d_model=256, n_head=4, d_key=64, n_streams=5, d_pos=90),                   # four warps for one, tiles by TMA; copies of table row 0
    dict(d_model=256, n_head=2, d_key=128, n_streams=3, ln_flags=2 | 4 | 16, ff_act=2),
    dict(d_model=128, n_head=4, d_key=32, n_streams=6, mem_len=400, d_pos=412)])    # tiles by every thread, more than one round
def test_device_decoder_over_several_key_blocks(pkg, kw):
    """Steps of a decoder, launched to overlap one another, read the keys of earlier steps, the tables and the weights before they
    wait: over memories of several key blocks, both memory twins and weights that have just been updated, the symbols are those of the
    host's walk of a whole segment's trees, and probabilities and updated weights have that segment's bits."""
    p = pkg.abi.make_params(**dict(dict(n_layer=3, d_inner=256, d_pos=162, mem_len=150, seg_len=12, n_symbols=300, use_bf16=1, init_range=0.2, lr=1e-3), **kw))
    T, B, V, L = p.seg_len, p.n_streams, p.n_symbols, pkg.host.library()
    rng = np.random.default_rng(9)
    dev, ref, streams = pkg.TrfModel(p), pkg.TrfModel(p), [torch.cuda.Stream() for _ in range(2)]
    for m, st in zip((dev, ref), streams):
        m.set_stream(st.cuda_stream)
        m.reset()
    for seg in range(6):   # the third pass over a memory twin replays graphs
        payload = rng.integers(0, 256, 40 * B, dtype=np.uint8).tobytes()
        first = rng.integers(0, V, B).astype(np.int32)
        dev.decoder_begin(payload)
        got = dev.decode_steps(0, T, first)
        dev.decoder_end()
        ids = np.concatenate([first[None], got[:-1]])
        assert np.array_equal(ref.eval(-1, ids), dev.read_probs(0, T))
        buf = C.create_string_buffer(payload, len(payload))
        hd, trees = L.nch_dec_new(buf, len(payload)), np.ascontiguousarray(ref.coder_trees(0, T))
        want = [L.nch_read_sym_tree(hd, trees[i].ctypes.data_as(C.c_void_p), V) for i in range(T * B)]
        L.nch_dec_free(hd)
        assert np.array_equal(got.reshape(-1), want)
        for m in (dev, ref):
            m.eval_gradient(got)
            m.update()
        assert dev.weights_hash() == ref.weights_hash()
    dev.close(); ref.close()
