"""Shapes at which paths that share or outgrow a resource meet: workspaces of two streams, associations of
two kernels for one row, CTAs without a share of the work."""
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
