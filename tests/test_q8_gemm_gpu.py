"""Q8_0 products with several activation rows on the tensor cores, against an f64 product with the dequantised weight.

Tolerance: the products are exact (int8 weights are bfloat16 values, an fp32 activation is the sum of three of them), what
is left are fp32 sums of K <= 8192 terms; with the error normalised by the largest output, sqrt(K) 2^-24 times a few for
the tensor core's truncating adds stays below 1e-5, the tolerance of the single-row kernels."""
import numpy as np
import pytest

from helpers import DECODE_TOL, rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import shainet_b200 as S
    c = S.AttnContext(0)
    yield c
    c.close()


# token tiles of 16, 32, 64 and 128 with their edges; weight tiles of 256 rows; one and many splits of the contraction
@pytest.mark.parametrize("K,N,M", [(128, 1, 2), (128, 256, 16), (384, 257, 17), (2048, 255, 32), (1536, 640, 33), (2048, 512, 64),
                                   (640, 300, 65), (2048, 3072, 128), (512, 20000, 129), (8192, 512, 3), (3584, 1000, 300),
                                   (2048, 2048, 1000)], ids=lambda v: str(v))
def test_several_rows_against_f64(ctx, K, N, M):
    import torch
    import shainet_b200 as S
    rng = np.random.default_rng(K + 3 * N + 7 * M)
    q = rng.integers(-128, 128, (N, K)).astype(np.int8)
    s = (0.001 * (0.5 + rng.random((N, K // 32)))).astype(np.float32)
    # activations over thirty binary orders of magnitude: every bit of every one of them counts
    x = (rng.standard_normal((M, K)) * np.exp2(rng.integers(-30, 1, (M, K)))).astype(np.float32)
    x[:, ::7] = rng.standard_normal((M, (K + 6) // 7)).astype(np.float32)
    W = S.Q8Weight.from_quantized(ctx, q, s)
    dev = torch.device("cuda:0")
    tx = torch.from_numpy(x).to(dev)
    ty = torch.full((M + 1, N), float("nan"), device=dev)
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    for stream in (st.cuda_stream, None):   # two streams share the context's scratch
        W.gemv_dev(tx.data_ptr(), ty.data_ptr(), M, stream)
    torch.cuda.synchronize()
    ctx.sync()
    w = torch.from_numpy(q).to(dev).double() * torch.from_numpy(s).to(dev).double().repeat_interleave(32, 1)
    truth = (tx.double() @ w.T).cpu().numpy()
    got = ty.cpu().numpy()
    assert np.isfinite(got[:M]).all() and np.isnan(got[M]).all()
    assert rel_err(got[:M], truth) <= DECODE_TOL, rel_err(got[:M], truth)
    W.close()
