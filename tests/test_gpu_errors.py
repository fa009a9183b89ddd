"""The error path of a bounded device-side wait: it runs out, the kernel returns, the host reads
NNCU_ERR_TIMEOUT once, and the model computes the same step afterwards as one that never saw it."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

KW = dict(n_layer=2, d_model=256, n_head=4, d_key=64, d_inner=512, d_pos=48, mem_len=16, seg_len=32,
          n_streams=4, n_symbols=512, use_bf16=1, lr=1e-3, init_range=0.03)


def test_expired_wait_is_reported_once_and_the_model_survives(pkg):
    p = pkg.abi.make_params(**KW)
    a, b = pkg.TrfModel(p), pkg.TrfModel(p)
    rng = np.random.default_rng(2)
    ids = rng.integers(0, 512, (32, 4)).astype(np.int32)
    tg = rng.integers(0, 512, (32, 4)).astype(np.int32)
    assert a.lib.nncu_selftest_expired_wait(a.h) == 0
    assert a.lib.nncu_synchronize(a.h) == pkg.abi.ERR_TIMEOUT
    assert b"bounded device-side wait" in a.lib.nncu_last_error()
    assert a.lib.nncu_synchronize(a.h) == 0          # the flag was cleared by the report
    for m in (a, b):
        m.reset()
        m.eval(-1, ids, read=False)
        m.eval_gradient(tg)
        m.update()
    assert a.weights_hash() == b.weights_hash()
    a.close()
    b.close()


@pytest.fixture(scope="module")
def expired(tmp_path_factory, pkg):
    """The attention kernels compiled with waits that give up after one look (tests/expired_waits.cu)."""
    nvcc = pkg.loader._nvcc()
    if nvcc is None:
        pytest.skip("needs nvcc")
    out = str(tmp_path_factory.mktemp("expired") / "expired.so")
    subprocess.run([nvcc] + pkg.loader.NVCC_FLAGS + ["-I", os.path.join(ROOT, "include"), "-I", pkg.loader.CSRC, "-o", out,
                                                     os.path.join(ROOT, "tests", "expired_waits.cu")], check=True, capture_output=True)
    lib = C.CDLL(out)
    lib.expired_error.restype = C.c_char_p
    return lib


@pytest.mark.parametrize("dk,B,alen,sums", [(64, 19, 0, 0), (64, 75, 0, 1), (64, 2, 70, 0), (128, 19, 0, 0), (128, 2, 70, 0)])
def test_expired_waits_of_attention_leave_no_result(pkg, expired, dk, B, alen, sums):
    """Segment, single queries and adjoint without their operands' arrival: the kernels return, the flag names a wait, and every
    value they owe is NaN, those that no key block reaches among them.  The same call with the usual waits is right afterwards."""
    torch = pytest.importorskip("torch")
    lib = pkg.library()
    H, T, M = 8, 40, 150
    L, P, HD = T + M, T + M - 5, H * dk
    g = torch.Generator(device="cuda").manual_seed(dk + B)
    q, dout = (torch.randn(T * B, HD, generator=g, device="cuda").bfloat16() for _ in range(2))
    kv = torch.randn(L * B, 2 * HD, generator=g, device="cuda").bfloat16()
    w_r, b_r = 0.1 * torch.randn(H, P, dk, generator=g, device="cuda"), 0.1 * torch.randn(H, L, generator=g, device="cuda")
    w16 = w_r.bfloat16()

    def shape(t0=0, t1=T):
        return C.byref(pkg.abi.AttnShape(B, H, dk, T, M, P, alen, t0, t1, float(np.sqrt(dk * 512.0)), 1))

    def results():
        new = lambda *s, t=torch.float32: torch.ones(*s, device="cuda", dtype=t)
        return [new(T * B, HD, t=torch.bfloat16), new(B * H, T), new(T * B, HD, t=torch.bfloat16), new(L * B, 2 * HD, t=torch.bfloat16),
                new(B, H, P, dk), new(B, H, L)]

    def ptr(*ts):
        return [C.c_void_p(t.data_ptr()) for t in ts]

    def usual():
        r = results()
        assert lib.nncu_attention_forward(shape(), *ptr(q, kv, w_r, b_r, r[0], r[1]), None) == 0
        assert lib.nncu_attention_backward(shape(), *ptr(q, kv, w_r, b_r, r[0], r[1], dout, r[2], r[3], r[4], r[5]), None) == 0
        torch.cuda.synchronize()
        return r

    before = usual()
    out, lse, dq, dkv, dwr, dbr = results()
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    if dk == 64:
        for t0, t1 in ((0, T), (T - 1, T)):
            out.fill_(1), lse.fill_(1), flag.zero_()
            assert expired.expired_forward(shape(t0, t1), *ptr(q, kv, w_r, w16, b_r, out, lse, flag)) == 0, expired.expired_error()
            torch.cuda.synchronize()
            assert flag.item() != 0
            assert out[t0 * B:t1 * B].isnan().all() and lse[:, t0:t1].isnan().all()
    flag.zero_()
    assert expired.expired_backward(shape(), sums, *ptr(q, kv, w_r, b_r, before[0], before[1], dout, dq, dkv, dwr, dbr, flag)) == 0, expired.expired_error()
    torch.cuda.synchronize()
    assert flag.item() != 0
    assert dq.isnan().all() and dkv.isnan().all() and dbr.isnan().all()
    if sums:    # a part for each CTA that has pairs of the head, the places behind them untouched
        at = dwr.view(B, H, P * dk)
        ends = [c * (B * H // 148) + min(c, B * H % 148) for c in range(149)]
        for h in range(H):
            parts = sum(ends[c] < (h + 1) * B and ends[c + 1] > h * B for c in range(148))
            assert at[:parts, h].isnan().all() and (at[parts:, h] == 1).all()
    else:
        assert dwr.isnan().all()
    assert all(torch.equal(a, b) for a, b in zip(before, usual()))
