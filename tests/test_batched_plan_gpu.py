"""Batched decode over sequences of very different lengths: slices that are all resident at once, and the four-wave plan where
the sequences are too many or too uneven for that.  And bfloat16 caches widened for the kernels that read fp32 rows."""
import numpy as np
import pytest

from helpers import DECODE_TOL, make_pair, qkv, rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import shainet_b200 as S
    c = S.AttnContext(0)
    yield c
    c.close()


@pytest.mark.parametrize("H,KV,hd,fmt,lens", [
    (32, 8, 64, "f32", [0, 1, 700, 3000, 63]), (8, 2, 128, "f32", [5000, 17]), (8, 2, 128, "bf16", [900, 31, 2500]),
    (32, 4, 128, "f32", [int(v) for v in np.linspace(1, 900, 33)]),        # 33 x 4 slices at least, resident at once
    (16, 16, 64, "bf16", [int(v) for v in np.linspace(5, 400, 21)]),       # 21 x 16: more than are resident
], ids=["five", "two", "three_bf16", "thirty_three", "twenty_one_bf16"])
def test_ragged_batch_against_the_oracle(ctx, H, KV, hd, fmt, lens):
    import torch
    from shainet_b200.attention import forward_batched_dev
    rng = np.random.default_rng(len(lens) + hd)
    shape = dict(H=H, KV=KV, hd=hd, theta=10000.0)
    pairs = []
    for L in lens:
        o, g = make_pair(ctx, shape, rng, kv_format=fmt, initial_capacity=L + 2)
        if L:
            kc, vc = (rng.standard_normal((KV, L, hd), dtype=np.float32) for _ in range(2))
            o.import_cache(kc, vc)
            g.cache.import_(kc, vc)
        pairs.append((o, g))
    for step in range(2):
        q, k, v = qkv(rng, shape, len(lens))
        dev = [torch.from_numpy(t).cuda() for t in (q, k, v)]
        out = torch.full((len(lens), H * hd), float("nan"), device="cuda")
        torch.cuda.synchronize()
        forward_batched_dev(ctx, [g.cache for _, g in pairs], *[t.data_ptr() for t in dev], out.data_ptr(), 1.0 / hd ** 0.5)
        ctx.sync()
        got = out.cpu().numpy()
        for b, (o, g) in enumerate(pairs):
            ref = o.attend_cached(q[b:b + 1], k[b:b + 1], v[b:b + 1], threads=4)
            # a rotated K element at a bfloat16 rounding boundary may land one step (2^-8 of it) away
            tol = DECODE_TOL if fmt == "f32" or np.array_equal(o.export_cache()[0], g.cache.export()[0]) else 5e-3
            assert rel_err(got[b:b + 1], ref) <= tol, (step, lens[b], rel_err(got[b:b + 1], ref))
    for _, g in pairs:
        g.close()


@pytest.mark.parametrize("hd,pre,T", [(64, 33, 70), (128, 200, 64), (24, 65, 5), (20, 9, 3)], ids=lambda v: str(v))
def test_widened_bf16_cache(ctx, hd, pre, T):
    """Tensor-core and generic kernels over the fp32 image: rows of whole 16-byte vectors and others, old and new rows; a second
    call finds the image of the first."""
    shape = dict(H=8, KV=2, hd=hd, theta=10000.0)
    rng = np.random.default_rng(hd)
    o, g = make_pair(ctx, shape, rng, kv_format="bf16")
    kc, vc = (rng.standard_normal((2, pre, hd), dtype=np.float32) for _ in range(2))
    o.import_cache(kc, vc)
    g.cache.import_(kc, vc)
    for n in (T, T + 1):
        q, k, v = qkv(rng, shape, n)
        ref = o.attend_cached(q, k, v, threads=4)
        got = g.forward_cached(q, k, v)
        same = np.array_equal(o.export_cache()[0], g.cache.export()[0])
        assert rel_err(got, ref) <= (2e-3 if n >= 64 and hd >= 64 else DECODE_TOL if same else 5e-3), rel_err(got, ref)
    g.close()


@pytest.mark.parametrize("hd", [64, 128])
def test_widened_image_holds_nothing_of_an_earlier_cache(ctx, hd):
    """The fp32 image ends on a whole position tile: what a longer cache with infinities left there does not reach a shorter
    one, whose masked positions the tensor cores multiply by zero probabilities."""
    shape = dict(H=4, KV=2, hd=hd, theta=10000.0)
    rng = np.random.default_rng(hd)
    _, a = make_pair(ctx, shape, rng, kv_format="bf16")
    q, k, v = qkv(rng, shape, 128)
    v[:, ::2] = np.inf
    a.forward_cached(q, k, v)
    o, b = make_pair(ctx, shape, rng, kv_format="bf16")
    q, k, v = qkv(rng, shape, 70)
    ref = o.attend_cached(q, k, v, threads=4)
    got = b.forward_cached(q, k, v)
    assert rel_err(got, ref) <= 2e-3, rel_err(got, ref)   # TF32 operands
    a.close()
    b.close()
