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
    # activations over thirty binary orders of magnitude (the error is normalised by the largest output here)
    x = (rng.standard_normal((M, K)) * np.exp2(rng.integers(-30, 1, (M, K)))).astype(np.float32)
    x[:, ::7] = rng.standard_normal((M, (K + 6) // 7)).astype(np.float32)
    W = S.Q8Weight.from_quantized(ctx, q, s)
    dev = torch.device("cuda:0")
    tx = torch.from_numpy(x).to(dev)
    ty = torch.full((M + 1, N), float("nan"), device=dev)
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    for stream in (st.cuda_stream, None):   # on a caller's stream, then on the context's, over the same output
        W.gemv_dev(tx.data_ptr(), ty.data_ptr(), M, stream)
    torch.cuda.synchronize()
    ctx.sync()
    w = torch.from_numpy(q).to(dev).double() * torch.from_numpy(s).to(dev).double().repeat_interleave(32, 1)
    truth = (tx.double() @ w.T).cpu().numpy()
    got = ty.cpu().numpy()
    assert np.isfinite(got[:M]).all() and np.isnan(got[M]).all()
    assert rel_err(got[:M], truth) <= DECODE_TOL, rel_err(got[:M], truth)
    W.close()


@pytest.mark.parametrize("M", [16, 64, 200])   # planes side by side, and passes of their own
@pytest.mark.parametrize("K", [2048, 8192])
def test_error_is_that_of_fp32_sums(ctx, K, M):
    """2-norm of the error over that of the result: the row kernels' 1.04e-7 and 1.21e-7 (K = 2048, 8192) with a tenth of
    room, on normal activations; and rows of very different magnitude, zeros, infinities and NaN keep to themselves."""
    import torch
    import shainet_b200 as S
    rng = np.random.default_rng(K + M)
    N = 512
    q = rng.integers(-127, 128, (N, K)).astype(np.int8)
    s = (0.001 * rng.random((N, K // 32))).astype(np.float32)
    x = rng.standard_normal((M, K)).astype(np.float32)
    x[1] *= np.float32(2.0 ** 100)
    x[2] *= np.float32(2.0 ** -100)
    x[3] = 0.0
    x[4, 7] = np.inf
    x[5, 9] = np.nan
    W = S.Q8Weight.from_quantized(ctx, q, s)
    dev = torch.device("cuda:0")
    tx = torch.from_numpy(x).to(dev)
    ty = torch.empty((M, N), device=dev)
    torch.cuda.synchronize()
    W.gemv_dev(tx.data_ptr(), ty.data_ptr(), M)
    ctx.sync()
    truth = x.astype(np.float64) @ (q.astype(np.float64) * s.astype(np.float64).repeat(32, 1)).T
    got = ty.cpu().numpy().astype(np.float64)
    plain = [i for i in range(M) if i not in (3, 4, 5)]
    for rows in (plain[:1], [1], [2], plain[3:]):
        err = np.linalg.norm(got[rows] - truth[rows]) / np.linalg.norm(truth[rows])
        assert err <= {2048: 1.15e-7, 8192: 1.33e-7}[K] * (1.0 if len(rows) > 1 else 1.2), (rows[0], err)
    assert (got[3] == 0).all() and not np.isfinite(got[4]).any() and np.isnan(got[5]).all()
    W.close()


def test_products_on_two_streams_keep_to_themselves(ctx):
    """The scratch of a context's products is shared by calls on different streams: other activations, weights and outputs
    on each of them, back and forth, long enough to overlap."""
    import torch
    import shainet_b200 as S
    rng = np.random.default_rng(8)
    dev = torch.device("cuda:0")
    K, N, M = 2048, 4096, 1500
    jobs = []
    for i in range(2):
        q = rng.integers(-127, 128, (N, K)).astype(np.int8)
        s = (0.001 * (0.5 + rng.random((N, K // 32)))).astype(np.float32)
        x = rng.standard_normal((M - 700 * i, K)).astype(np.float32)
        W = S.Q8Weight.from_quantized(ctx, q, s)
        w = torch.from_numpy(q).to(dev).double() * torch.from_numpy(s).to(dev).double().repeat_interleave(32, 1)
        tx = torch.from_numpy(x).to(dev)
        jobs.append((W, tx, [torch.full((len(x), N), float("nan"), device=dev) for _ in range(6)], (tx.double() @ w.T).cpu().numpy(), torch.cuda.Stream()))
    torch.cuda.synchronize()
    for r in range(6):
        for W, tx, ys, _, st in jobs:
            W.gemv_dev(tx.data_ptr(), ys[r].data_ptr(), len(tx), st.cuda_stream)
    torch.cuda.synchronize()
    ctx.sync()
    for W, _, ys, truth, _ in jobs:
        for y in ys:
            assert rel_err(y.cpu().numpy(), truth) <= DECODE_TOL
        W.close()


def test_a_block_and_products_on_other_streams(ctx):
    """A block of several tokens on one stream and products on two others use the same scratch: block, product, block,
    product without a synchronisation between them give what they give one by one."""
    import torch
    import shainet_b200 as S
    from test_q8_decoder_gpu import _make_block
    rng = np.random.default_rng(81)
    d, T, K, N, M = 2048, 300, 2048, 8192, 900
    _, block, owned = _make_block(ctx, rng, d, 32, 8, 64, 8192, 5e5, 1e-5, False)
    q = rng.integers(-127, 128, (N, K)).astype(np.int8)
    s = (0.001 * (0.5 + rng.random((N, K // 32)))).astype(np.float32)
    W = S.Q8Weight.from_quantized(ctx, q, s)
    xb, xw = torch.randn(3, T, d, device="cuda"), torch.randn(3, M, K, device="cuda")
    streams = [torch.cuda.Stream() for _ in range(3)]
    results = []
    for one_by_one in (True, False):
        block.clear_cache()
        yb, yw = torch.full_like(xb, float("nan")), torch.full((3, M, N), float("nan"), device="cuda")
        torch.cuda.synchronize()
        for r in range(3):   # the block always on the first stream: its cache grows in order
            block.forward_cached_dev(xb[r].data_ptr(), yb[r].data_ptr(), T, streams[0].cuda_stream)
            if one_by_one:
                torch.cuda.synchronize()
            W.gemv_dev(xw[r].data_ptr(), yw[r].data_ptr(), M, streams[1 + r % 2].cuda_stream)
            if one_by_one:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        ctx.sync()
        results.append((yb, yw))
    assert torch.isfinite(results[0][0]).all() and torch.isfinite(results[0][1]).all()
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])
    W.close()
    for o in owned:
        o.close()


@pytest.mark.parametrize("K,N,M", [(2048, 512, 6), (2048, 512, 200), (1536, 300, 40)], ids=lambda v: str(v))
def test_several_rows_under_stream_capture(ctx, K, N, M):
    """A captured product of several rows replays with new activations, on a context that has made no such product before
    and whatever is called beside the graph."""
    import torch
    import shainet_b200 as S
    rng = np.random.default_rng(K + N + M)
    q = rng.integers(-127, 128, (N, K)).astype(np.int8)
    s = (0.001 * (0.5 + rng.random((N, K // 32)))).astype(np.float32)
    w = q.astype(np.float64) * s.astype(np.float64).repeat(32, 1)
    c = S.AttnContext(0)
    W = S.Q8Weight.from_quantized(c, q, s)
    tx, ty = torch.empty((M, K), device="cuda"), torch.empty((M, N), device="cuda")
    other = torch.empty((M, N), device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        W.gemv_dev(tx.data_ptr(), ty.data_ptr(), M, torch.cuda.current_stream().cuda_stream)
    for _ in range(2):
        x = rng.standard_normal((M, K)).astype(np.float32)
        tx.copy_(torch.from_numpy(x))
        torch.cuda.synchronize()
        graph.replay()
        W.gemv_dev(tx.data_ptr(), other.data_ptr(), M)   # on the context's stream, beside the replay
        torch.cuda.synchronize()
        c.sync()
        truth = x.astype(np.float64) @ w.T
        assert rel_err(ty.cpu().numpy(), truth) <= DECODE_TOL
        assert rel_err(other.cpu().numpy(), truth) <= DECODE_TOL
    del graph
    W.close()
    c.close()


def test_a_block_of_several_tokens_under_stream_capture(ctx):
    """After one plain call with as many tokens a captured block call finds all its scratch; its replay is the plain call's
    result to the block's tolerance (other kernels)."""
    import torch
    import shainet_b200 as S
    from test_q8_decoder_gpu import BLOCK_TOL, _make_block
    rng = np.random.default_rng(82)
    d, T = 2048, 9
    c = S.AttnContext(0)
    _, block, owned = _make_block(c, rng, d, 32, 8, 64, 4096, 5e5, 1e-5, False)
    x, y, z = (torch.randn(T, d, device="cuda") for _ in range(3))
    torch.cuda.synchronize()
    block.forward_cached_dev(x.data_ptr(), y.data_ptr(), T)
    c.sync()
    block.clear_cache()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        block.forward_cached_dev(x.data_ptr(), z.data_ptr(), T, torch.cuda.current_stream().cuda_stream)
    for seed in range(2):
        x.copy_(torch.randn(T, d, device="cuda"))
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        block.clear_cache()
        block.forward_cached_dev(x.data_ptr(), y.data_ptr(), T)
        c.sync()
        assert rel_err(z.cpu().numpy(), y.cpu().numpy()) <= BLOCK_TOL
    del graph
    for o in owned:
        o.close()
    c.close()


def test_more_rows_than_one_pass(ctx):
    """A product and a block of more tokens than a pass takes: the rows of the second pass are those of a call of their own."""
    import torch
    import shainet_b200 as S
    from test_q8_decoder_gpu import _make_block
    rng = np.random.default_rng(83)
    K, N, M, P = 256, 300, 8192 + 130, 8192
    q = rng.integers(-127, 128, (N, K)).astype(np.int8)
    s = (0.001 * (0.5 + rng.random((N, K // 32)))).astype(np.float32)
    W = S.Q8Weight.from_quantized(ctx, q, s)
    x = torch.randn(M, K, device="cuda")
    y, z = torch.full((M, N), float("nan"), device="cuda"), torch.full((M - P, N), float("nan"), device="cuda")
    torch.cuda.synchronize()
    W.gemv_dev(x.data_ptr(), y.data_ptr(), M)
    W.gemv_dev(x[P:].data_ptr(), z.data_ptr(), M - P)
    ctx.sync()
    truth = x.cpu().numpy().astype(np.float64) @ (q.astype(np.float64) * s.astype(np.float64).repeat(32, 1)).T
    assert rel_err(y.cpu().numpy(), truth) <= DECODE_TOL and torch.equal(y[P:], z)
    W.close()
    for ffn in (512, 0):
        _, block, owned = _make_block(ctx, rng, 256, 4, 2, 64, ffn, 5e5, 1e-5, False)
        x, y = torch.randn(M, 256, device="cuda"), torch.empty(M, 256, device="cuda")
        z = torch.empty(M - P, 256, device="cuda")
        torch.cuda.synchronize()
        block.forward_cached_dev(x.data_ptr(), y.data_ptr(), M)
        ctx.sync()
        block.clear_cache()
        first = torch.empty(P, 256, device="cuda")
        torch.cuda.synchronize()
        block.forward_cached_dev(x.data_ptr(), first.data_ptr(), P)
        block.forward_cached_dev(x[P:].data_ptr(), z.data_ptr(), M - P)
        block.clear_cache()
        inplace = x.clone()
        torch.cuda.synchronize()
        block.forward_cached_dev(inplace.data_ptr(), inplace.data_ptr(), M)
        ctx.sync()
        assert torch.equal(y[:P], first) and torch.equal(y[P:], z) and torch.equal(inplace, y)
        for o in owned:
            o.close()


@pytest.mark.parametrize("free_mb", [110, 36])
def test_without_memory_for_the_planes(free_mb):
    """Where the device has no room for the planes of all rows the product of several rows takes fewer at a time, and the row
    kernels, which need no scratch, where it has none at all."""
    import torch
    import shainet_b200 as S
    rng = np.random.default_rng(84)
    K, N, M = 51200, 64, 2048   # planes of 2048 rows: 400 MB and more, of 256 rows: more than 48
    c = S.AttnContext(0)
    q = rng.integers(-127, 128, (N, K)).astype(np.int8)
    s = (0.001 * (0.5 + rng.random((N, K // 32)))).astype(np.float32)
    W = S.Q8Weight.from_quantized(c, q, s)
    x = torch.randn(M, K, device="cuda")
    short, roomy = torch.empty(M, N, device="cuda"), torch.empty(M, N, device="cuda")
    torch.cuda.synchronize()
    W.gemv_dev(x.data_ptr(), short.data_ptr(), 1)   # loads the row kernel
    c.sync()
    assert c.scratch_bytes() < 16 << 20
    held = []
    for size in (1 << 30, 1 << 26, 12 << 20):   # down to at most 12 MB more than free_mb
        while torch.cuda.mem_get_info()[0] > size + (free_mb << 20):
            held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
    W.gemv_dev(x.data_ptr(), short.data_ptr(), M)
    c.sync()
    assert (c.scratch_bytes() < 16 << 20) if free_mb == 36 else ((48 << 20) < c.scratch_bytes() < (122 << 20))
    del held
    torch.cuda.empty_cache()
    W.gemv_dev(x.data_ptr(), roomy.data_ptr(), M)
    c.sync()
    assert c.scratch_bytes() >= 400 << 20
    assert rel_err(short.cpu().numpy(), roomy.cpu().numpy()) <= 2 * DECODE_TOL   # either is within DECODE_TOL of the exact product
    W.close()
    c.close()


@pytest.mark.parametrize("M", [16, 64, 200])
@pytest.mark.parametrize("outlier", [1e4, 1e6])
def test_small_activations_beside_a_large_one(ctx, outlier, M):
    """One channel 10^4 or 10^6 times the others, with zero weights: the outputs are those of the others, to the error of
    the row kernels (2-norm; 1.04e-7 with a tenth of room)."""
    import torch
    import shainet_b200 as S
    rng = np.random.default_rng(M)
    K, N = 2048, 512
    q = rng.integers(-127, 128, (N, K)).astype(np.int8)
    q[:, 77] = 0
    s = (0.001 * rng.random((N, K // 32))).astype(np.float32)
    x = rng.standard_normal((M, K)).astype(np.float32)
    x[:, 77] *= np.float32(outlier)
    W = S.Q8Weight.from_quantized(ctx, q, s)
    tx = torch.from_numpy(x).cuda()
    ty = torch.empty((M, N), device="cuda")
    torch.cuda.synchronize()
    W.gemv_dev(tx.data_ptr(), ty.data_ptr(), M)
    ctx.sync()
    truth = x.astype(np.float64) @ (q.astype(np.float64) * s.astype(np.float64).repeat(32, 1)).T
    err = np.linalg.norm(ty.cpu().numpy() - truth) / np.linalg.norm(truth)
    assert err <= 1.15e-7, err
    W.close()


@pytest.mark.parametrize("K,M,tensor", [(10240, 4, False), (10368, 4, True), (10368, 2, False), (12288, 3, True), (20480, 2, False),
                                        (20608, 2, False), (20608, 3, True), (2176, 4, False), (256, 5, True)], ids=lambda v: str(v))
def test_which_rows_the_row_kernels_keep(K, M, tensor):
    """Two rows stay with the row kernels, three and four while one of their row tiles holds them; the tensor path shows by the
    scratch it needs."""
    import torch
    import shainet_b200 as S
    rng = np.random.default_rng(K + M)
    N = 260
    c = S.AttnContext(0)
    q = rng.integers(-127, 128, (N, K)).astype(np.int8)
    s = (0.001 * (0.5 + rng.random((N, K // 32)))).astype(np.float32)
    x = rng.standard_normal((M, K)).astype(np.float32)
    W = S.Q8Weight.from_quantized(c, q, s)
    tx, ty = torch.from_numpy(x).cuda(), torch.empty((M, N), device="cuda")
    torch.cuda.synchronize()
    before = c.scratch_bytes()
    W.gemv_dev(tx.data_ptr(), ty.data_ptr(), M)
    c.sync()
    assert (c.scratch_bytes() > before) == tensor
    truth = x.astype(np.float64) @ (q.astype(np.float64) * s.astype(np.float64).repeat(32, 1)).T
    assert rel_err(ty.cpu().numpy(), truth) <= DECODE_TOL
    W.close()
    c.close()
