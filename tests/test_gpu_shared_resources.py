"""Shapes at which paths that share or outgrow a resource meet: workspaces of two streams, associations of
two kernels for one row, CTAs without a share of the work."""
import ctypes as C

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


def test_split_head_gradients_beside_each_other(pkg, monkeypatch):
    """8192 symbols, d_model 256, 128 streams x 64: the head's weight gradient (side stream) and its dX (main
    stream) are both split over the contraction.  The gradients are the other engine's, the same every time,
    and those of a model without a side stream bit for bit."""
    kw = dict(n_layer=1, d_model=256, n_head=4, d_key=64, d_inner=256, d_pos=80, mem_len=16, seg_len=64, n_streams=128,
              n_symbols=8192, use_bf16=1, init_range=0.05)
    rng = np.random.default_rng(5)
    ids, tg = (rng.integers(0, 8192, (64, 128)).astype(np.int32) for _ in range(2))
    got = []
    for backend, no_overlap, times in ((2, "0", 6), (2, "1", 1), (1, "0", 1)):
        monkeypatch.setenv("NNCU_NO_OVERLAP", no_overlap)
        m = pkg.TrfModel(pkg.abi.make_params(gemm_backend=backend, **kw))
        m.reset()
        for _ in range(times):
            m.eval(-1, ids, read=False)
            m.eval_gradient(tg)
            got.append({n: m.get_grad(n) for n in m.info})
        m.close()
    first, other = got[0], got[-1]
    for g in got[1:-1]:
        for n in first:
            assert np.array_equal(g[n], first[n]), n
    for n in first:  # bf16 operands of both engines, fp32 sums: as in the other comparisons of engines
        assert rel_err(first[n], other[n]) < 2e-2, n


@pytest.mark.parametrize("V,D", [(1024, 64), (3072, 96), (4096, 32)])
def test_one_launch_steps_of_wide_alphabets_equal_whole_segment_bitwise(pkg, V, D):
    """fp32 models whose alphabet is a multiple of 1024: whole segments take the softmax that keeps a row in
    registers, and the one-launch step the same sums in the same order; so the symbols coded from a whole
    segment's probabilities come back."""
    p = pkg.abi.make_params(n_layer=2, d_model=D, n_head=2, d_key=16, d_inner=128, d_pos=12, mem_len=9, seg_len=6, n_streams=3,
                            n_symbols=V, use_bf16=0, init_range=0.5)
    T, B, L = 6, 3, pkg.host.library()
    rng = np.random.default_rng(V)
    seg, one = pkg.TrfModel(p), pkg.TrfModel(p)
    seg.reset(); one.reset()
    ids, tg = (rng.integers(0, V, (T, B)).astype(np.int32) for _ in range(2))
    ids[1:] = tg[:-1]
    a = seg.eval(-1, ids)
    b = np.concatenate([one.eval(t, ids) for t in range(T)])
    assert np.array_equal(a, b)
    for m in (seg, one):
        m.eval_gradient(tg)
        m.update()
    assert seg.weights_hash() == one.weights_hash()
    one.eval_end()
    # the next segment: coded from whole-segment probabilities, decoded step by step
    ids[0] = tg[-1]
    tg = rng.integers(0, V, (T, B)).astype(np.int32)
    ids[1:] = tg[:-1]
    seg.eval(-1, ids, read=False)
    paths = seg.coder_paths(0, T, tg)
    enc, data = L.nch_enc_new(), C.c_void_p()
    L.nch_write_sym_paths_any(enc, paths.ctypes.data_as(C.c_void_p), V, tg.ctypes.data_as(C.c_void_p), T * B)
    n = L.nch_enc_finish(enc, C.byref(data))
    payload = C.string_at(data.value, n)
    L.nch_enc_free(enc)
    one.decoder_begin(payload)
    assert np.array_equal(one.decode_steps(0, T, np.ascontiguousarray(ids[0])), tg)
    one.decoder_end()
    seg.close(); one.close()


@pytest.mark.parametrize("D,H,dk,F,B", [(16, 1, 16, 16, 3), (48, 12, 4, 16, 40), (112, 7, 16, 112, 5), (64, 1, 16, 64, 9), (96, 3, 32, 208, 1),
                                        (64, 4, 16, 48, 17)])
def test_one_launch_steps_of_narrow_models_equal_whole_segment_bitwise(pkg, D, H, dk, F, B):
    """Products too narrow to give every CTA of a cluster a share, and ones that only just do."""
    p = pkg.abi.make_params(n_layer=3, d_model=D, n_head=H, d_key=dk, d_inner=F, d_pos=14, mem_len=9, seg_len=6, n_streams=B, n_symbols=72,
                            use_bf16=0, init_range=0.4, lr=1e-3)
    rng = np.random.default_rng(D + F)
    seg, one = pkg.TrfModel(p), pkg.TrfModel(p)
    seg.reset(); one.reset()
    for _ in range(4):
        ids, tg = (rng.integers(0, 72, (6, B)).astype(np.int32) for _ in range(2))
        assert np.array_equal(seg.eval(-1, ids), np.concatenate([one.eval(t, ids) for t in range(6)]))
        for m in (seg, one):
            m.eval_gradient(tg)
            m.update()
        assert seg.weights_hash() == one.weights_hash()
    seg.close(); one.close()


def test_models_of_other_shapes_leave_a_models_launches_alone(pkg):
    """Shared-memory limits are the kernels', not the models': a smaller model made later, on the same
    device, must not lower them.  Coder trees, two open decoders, one-launch steps."""
    def model(V, B, F=64):
        m = pkg.TrfModel(pkg.abi.make_params(n_layer=1, d_model=64, n_head=2, d_key=32, d_inner=F, d_pos=8, mem_len=8, seg_len=4,
                                             n_streams=B, n_symbols=V, use_bf16=0, init_range=0.05))
        m.reset()
        return m

    big, small = model(16384, 2), model(8192, 2)
    ids = np.zeros((4, 2), np.int32)
    big.eval(-1, ids, read=False)
    big.coder_trees(0, 1)
    big.close(); small.close()
    big, small = model(4096, 50, 512), model(4096, 2)
    big.decoder_begin(b"\x55" * 9000)
    small.decoder_begin(b"\x55" * 900)
    for m, B in ((big, 50), (small, 2), (big, 50)):
        m.decode_steps(0, 2, np.zeros(B, np.int32))
        m.eval_end()
    big.close(); small.close()


def test_two_devices_of_one_process(pkg):
    """fp32 and bf16 models on a second device after the first."""
    torch = pytest.importorskip("torch")
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two devices")
    kw = dict(n_layer=1, d_model=64, n_head=2, d_key=32, d_inner=64, d_pos=8, mem_len=8, seg_len=4, n_streams=2, n_symbols=256)
    ids = np.zeros((4, 2), np.int32)
    for bf16 in (0, 1):
        probs = []
        for device in (0, 1):
            m = pkg.TrfModel(pkg.abi.make_params(use_bf16=bf16, device=device, **kw))
            m.reset()
            probs.append(m.eval(-1, ids))
            m.eval_gradient(ids)
            m.synchronize()
            m.close()
        assert np.array_equal(*probs)


@pytest.mark.parametrize("dk", [64, 128])
def test_query_kernel_table_tiles_by_hand_and_by_copy(pkg, dk):
    """A table that ends inside the left pad: the one-query kernel writes a warp's first tiles of it by
    ordinary stores and has the later ones copied to the same place; every step is the segment's, bit for bit."""
    p = pkg.abi.make_params(n_layer=2, d_model=2 * dk, n_head=2, d_key=dk, d_inner=128, d_pos=200, mem_len=500, seg_len=8, n_streams=5,
                            n_symbols=256, use_bf16=1, init_range=0.3)
    rng = np.random.default_rng(dk)
    seg, one = pkg.TrfModel(p), pkg.TrfModel(p)
    seg.reset(); one.reset()
    for _ in range(2):
        ids = rng.integers(0, 256, (8, 5)).astype(np.int32)
        assert np.array_equal(seg.eval(-1, ids), np.concatenate([one.eval(t, ids) for t in range(8)]))
        for m in (seg, one):
            m.memory_shift()
    seg.close(); one.close()


def test_launches_of_a_models_creation_are_counted(pkg):
    """Every launch is checked and counted: one for each parameter whose initial values are not zero."""
    prof = pkg.abi.Profile()
    lib = pkg.library()
    lib.nncu_profile_begin(0)
    m = pkg.TrfModel(pkg.abi.make_params(n_layer=2, d_model=64, n_head=2, d_key=32, d_inner=64, d_pos=8, mem_len=8, seg_len=4, n_streams=2,
                                         n_symbols=64, use_bf16=0))
    lib.nncu_profile_end(C.byref(prof))
    assert prof.launches == sum(n.startswith(("ln_g", "w_", "ff1", "ff2", "embed")) for n in m.info)
    m.close()


def test_profiled_work_leaves_out_what_is_not_computed(pkg):
    """A long memory: the memory rows' queries are neither projected nor part of the weight gradient."""
    D, F, T, M, B, V = 512, 1024, 64, 512, 32, 1024
    lib, prof = pkg.library(), pkg.abi.Profile()
    m = pkg.TrfModel(pkg.abi.make_params(n_layer=1, d_model=D, n_head=8, d_key=64, d_inner=F, d_pos=M + T, mem_len=M, seg_len=T, n_streams=B,
                                         n_symbols=V, use_bf16=1, init_range=0.05))
    m.reset()
    ids = np.zeros((T, B), np.int32)
    work = []
    for step in (lambda: m.eval(-1, ids, read=False), lambda: m.eval_gradient(ids)):
        lib.nncu_profile_begin(1)
        step()
        lib.nncu_profile_end(C.byref(prof))
        work.append(prof.gemm_flops)
    m.close()
    rows, dense = T * B, 2 * T * B * D * (D + 2 * F + V)   # output projection, feed-forward, head
    project = 2 * (M * B * 2 * D + rows * 3 * D) * D
    assert work[0] == dense + project
    assert work[1] == 2 * dense + project + 2 * rows * 3 * D * D


@pytest.mark.parametrize("B,V", [(11500, 256), (12690, 256), (10900, 300)])
def test_decoder_of_very_many_streams(pkg, B, V):
    """The payload window of so many streams leaves room for a few trees only: they still go through the
    ring, and the symbols are those of the host's walk of the same trees."""
    p = pkg.abi.make_params(n_layer=1, d_model=16, n_head=1, d_key=16, d_inner=16, d_pos=2, mem_len=0, seg_len=2, n_streams=B, n_symbols=V,
                            use_bf16=0, init_range=0.5)
    L = pkg.host.library()
    payload = np.random.default_rng(B).integers(0, 256, 20000, dtype=np.uint8).tobytes()
    dev, ref = pkg.TrfModel(p), pkg.TrfModel(p)
    dev.reset(); ref.reset()
    dev.decoder_begin(payload)
    got = dev.decode_steps(0, 2, np.zeros(B, np.int32))
    buf = C.create_string_buffer(payload, len(payload))
    hd, ids, want = L.nch_dec_new(buf, len(payload)), np.zeros((2, B), np.int32), np.zeros((2, B), np.int32)
    for t in range(2):
        ids[t] = want[t - 1] if t else 0
        ref.eval(t, ids, read=False)
        trees = np.ascontiguousarray(ref.coder_trees(t, 1))
        for b in range(B):
            want[t, b] = L.nch_read_sym_tree(hd, trees[b].ctypes.data_as(C.c_void_p), V)
    L.nch_dec_free(hd)
    assert np.array_equal(got, want)
    dev.close(); ref.close()


@pytest.mark.parametrize("dk,T,M,alen", [(16, 20, 300, 0), (32, 64, 500, 90), (64, 64, 836, 0), (64, 64, 600, 130), (128, 33, 500, 200),
                                           (64, 64, 1368, 0), (64, 64, 1369, 300), (128, 33, 1271, 0), (128, 33, 1272, 200)])
def test_attention_of_operands_inside_larger_buffers(pkg, dk, T, M, alen):
    """An fp32 table, results and partials that start between 16-byte boundaries, as views of larger buffers do, with
    more keys than the CUDA-core kernels hold: the bits of the aligned call, segments and single queries."""
    torch = pytest.importorskip("torch")
    lib = pkg.library()
    B, H, L, P = 2, 3, T + M, T + M - 5
    g = torch.Generator(device="cuda").manual_seed(dk + M)
    q, dout = (torch.randn(T * B, H * dk, generator=g, device="cuda").bfloat16() for _ in range(2))
    kv = torch.randn(L * B, 2 * H * dk, generator=g, device="cuda").bfloat16()
    w_r, b_r = 0.1 * torch.randn(H, P, dk, generator=g, device="cuda"), 0.1 * torch.randn(H, L, generator=g, device="cuda")

    def place(t, by):   # the same values, `by` elements into a buffer
        room = torch.full((t.numel() + 16,), float("nan"), device="cuda", dtype=t.dtype)
        view = room[by:by + t.numel()].view(t.shape)
        view.copy_(t)
        return view

    got = []
    for off in (0, 1):
        table = place(w_r, off)
        out, one, dq, dkv = (place(torch.full_like(t, float("nan")), 2 * off) for t in (q, q, q, kv))
        lse = torch.zeros(B * H, T, device="cuda")
        part, dbr = place(torch.full((B, H, P, dk), float("nan"), device="cuda"), 2 * off), torch.full((B, H, L), float("nan"), device="cuda")

        def shape(t0, t1):
            return C.byref(pkg.abi.AttnShape(B, H, dk, T, M, P, alen, t0, t1, float(np.sqrt(dk * 512.0)), 1))

        calls = [lib.nncu_attention_forward(shape(0, T), q.data_ptr(), kv.data_ptr(), table.data_ptr(), b_r.data_ptr(), out.data_ptr(),
                                            lse.data_ptr(), None)]
        calls += [lib.nncu_attention_forward(shape(t, t + 1), q.data_ptr(), kv.data_ptr(), table.data_ptr(), b_r.data_ptr(), one.data_ptr(),
                                             None, None) for t in range(T)]
        calls += [lib.nncu_attention_backward(shape(0, T), q.data_ptr(), kv.data_ptr(), table.data_ptr(), b_r.data_ptr(), out.data_ptr(),
                                              lse.data_ptr(), dout.data_ptr(), dq.data_ptr(), dkv.data_ptr(), part.data_ptr(), dbr.data_ptr(),
                                              None)]
        assert not any(calls), lib.nncu_last_error()
        torch.cuda.synchronize()
        got.append((out, one, lse, dq, dkv, part, dbr))
    for a, b in zip(*got):
        assert torch.equal(a, b) and not a.isnan().any()
    assert torch.equal(got[0][0], got[0][1])
