"""Q8_0 products with one to four activation rows at input widths that are no multiple of the kernels' 2048-input segment:
the short last segment, the short last 512-input chunk in it, and rows padded in shared memory.  The ring kernel takes one row
and a multiple of four columns, the register kernel the rest.  Tolerance: the single-row one (fp32 sums in another order)."""
import numpy as np
import pytest

from helpers import DECODE_TOL, rel_err
from test_q8_decoder_gpu import BLOCK_TOL, _make_block

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import shainet_b200 as S
    c = S.AttnContext(0)
    yield c
    c.close()


@pytest.mark.parametrize("M", [1, 2, 3, 4])
@pytest.mark.parametrize("K,N", [(128, 4), (384, 1001), (512, 256), (1024, 4096), (1536, 2304), (2176, 257), (3072, 1000),
                                 (4608, 516), (6144, 64), (12288, 40)], ids=lambda v: str(v))
def test_widths_against_f64(ctx, K, N, M):
    import torch
    import shainet_b200 as S
    rng = np.random.default_rng(K + N + M)
    q = rng.integers(-128, 128, (N, K)).astype(np.int8)
    s = (0.001 * (0.5 + rng.random((N, K // 32)))).astype(np.float32)
    x = rng.standard_normal((M, K)).astype(np.float32)
    W = S.Q8Weight.from_quantized(ctx, q, s)
    dev = torch.device("cuda:0")
    tx = torch.from_numpy(x).to(dev)
    ty = torch.full((M + 1, N), float("nan"), device=dev)
    torch.cuda.synchronize()
    W.gemv_dev(tx.data_ptr(), ty.data_ptr(), M)
    ctx.sync()
    truth = x.astype(np.float64) @ (q.astype(np.float64) * s.astype(np.float64).repeat(32, 1)).T
    got = ty.cpu().numpy()
    assert np.isfinite(got[:M]).all() and np.isnan(got[M]).all()
    assert rel_err(got[:M], truth) <= DECODE_TOL, rel_err(got[:M], truth)
    W.close()


@pytest.mark.parametrize("d,H,KV,hd,ffn", [(1536, 24, 8, 64, 4608), (640, 10, 2, 64, 1408), (3072, 24, 8, 128, 9216)], ids=lambda v: str(v))
def test_block_of_other_widths(ctx, d, H, KV, hd, ffn):
    """Norm prologue, residual and SwiGLU epilogues with padded rows: one to four tokens, then single ones."""
    rng = np.random.default_rng(d)
    ob, gb, owned = _make_block(ctx, rng, d, H, KV, hd, ffn, 5e5, 1e-5, False)
    for T in (1, 3, 1, 2):
        x = rng.standard_normal((T, d)).astype(np.float32)
        ref, got = ob.forward_cached(x), gb.forward_cached(x)
        assert rel_err(got, ref) <= BLOCK_TOL, (T, rel_err(got, ref))
    for o in owned:
        o.close()
