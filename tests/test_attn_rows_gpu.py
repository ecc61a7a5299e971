"""The row-tile attention kernel (a few query rows of a kv head, fp32) against the oracle, with the decode tolerance: the
arithmetic is fp32 throughout, only the order of the sums differs."""
import numpy as np
import pytest

from helpers import DECODE_TOL, make_pair, qkv, rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import shainet_b200 as S
    from shainet_b200 import build
    build.build()
    c = S.AttnContext(0)
    yield c
    c.close()


# (group size, new tokens): row tiles of 16, 32 and 64 with their remainders, one to sixteen tiles, causal edges inside a tile
@pytest.mark.parametrize("G,T", [(7, 1), (16, 1), (3, 1), (1, 2), (4, 5), (16, 2), (8, 3), (5, 13), (4, 17), (16, 63), (1, 63)],
                         ids=lambda v: str(v))
@pytest.mark.parametrize("hd,fmt", [(64, "f32"), (128, "f32"), (64, "bf16"), (128, "bf16")])
def test_rows_against_the_oracle(ctx, G, T, hd, fmt):
    rng = np.random.default_rng(hd + 1000 * G + T)
    shape = dict(H=2 * G, KV=2, hd=hd, theta=10000.0)
    for L in (0, 1, 63, 64, 65, 200, 1031, 3000):   # position tiles of 64, one and many slices
        o, g = make_pair(ctx, shape, rng, kv_format=fmt)
        if L:
            kc = rng.standard_normal((2, L, hd), dtype=np.float32)
            vc = rng.standard_normal((2, L, hd), dtype=np.float32)
            o.import_cache(kc, vc)
            g.cache.import_(kc, vc)
        q, k, v = qkv(rng, shape, T)
        ref = o.attend_cached(q, k, v, threads=8)
        got = g.forward_cached(q, k, v)
        ko, vo = o.export_cache()
        kg, vg = g.cache.export()
        assert np.array_equal(vo, vg)
        # a rotated K element at a bfloat16 rounding boundary may land one step (2^-8 of it) away: its row's score moves by
        # that much of one product, its probability by as much, the output by that share of one row among L + T
        tol = DECODE_TOL if fmt == "f32" or np.array_equal(ko, kg) else 5e-3
        assert rel_err(got, ref) <= tol, (L, rel_err(got, ref))
        assert np.isfinite(got).all()
        g.close()


def test_batched_tokens_of_an_odd_group_size(ctx):
    """Ragged lock-step decode at seven query heads per kv head, biased projections."""
    import torch
    import shainet_b200 as S
    rng = np.random.default_rng(9)
    shape = dict(H=14, KV=2, hd=128, theta=1e6)
    dev = torch.device("cuda:0")
    bias = dict(b_q=rng.standard_normal(14 * 128).astype(np.float32), b_k=rng.standard_normal(256).astype(np.float32),
                b_v=rng.standard_normal(256).astype(np.float32))
    for fmt in ("f32", "bf16"):
        lens = [1, 63, 64, 700, 5000]
        pairs = [make_pair(ctx, shape, rng, kv_format=fmt, **bias) for _ in lens]
        for (o, g), L in zip(pairs, lens):
            kc = rng.standard_normal((2, L, 128), dtype=np.float32)
            vc = rng.standard_normal((2, L, 128), dtype=np.float32)
            o.import_cache(kc, vc)
            g.cache.import_(kc, vc)
        q, k, v = qkv(rng, shape, len(lens))
        tq, tk, tv = (torch.from_numpy(x).to(dev) for x in (q, k, v))
        out = torch.empty_like(tq)
        torch.cuda.synchronize()
        S.forward_batched_dev(ctx, [g.cache for _, g in pairs], tq.data_ptr(), tk.data_ptr(), tv.data_ptr(), out.data_ptr(),
                              pairs[0][1].scale)
        ctx.sync()
        got = out.cpu().numpy()
        for b, (o, g) in enumerate(pairs):
            ref = o.attend_cached(q[b:b + 1], k[b:b + 1], v[b:b + 1])
            same = np.array_equal(o.export_cache()[0], g.cache.export()[0])
            assert rel_err(got[b:b + 1], ref) <= (DECODE_TOL if fmt == "f32" or same else 5e-3), (fmt, b)
            g.close()


@pytest.mark.parametrize("T", [2, 5, 40, 63])
@pytest.mark.parametrize("hd,fmt", [(64, "f32"), (128, "f32"), (64, "bf16"), (128, "bf16")])
def test_non_finite_rows_of_later_tokens_do_not_reach_earlier_ones(ctx, hd, fmt, T):
    """A drafted token whose V or K row holds an infinity or NaN: the tokens before it are bit for bit what they are with
    finite rows in its place."""
    rng = np.random.default_rng(hd + T)
    shape = dict(H=8, KV=2, hd=hd, theta=10000.0)
    for L in (0, 61, 700):
        kc, vc = (rng.standard_normal((2, L, hd), dtype=np.float32) for _ in range(2))
        q, k, v = qkv(rng, shape, T)
        outs = []
        bad = T // 2   # the first bad token
        for value in (1.0, np.inf, np.nan):
            _, g = make_pair(ctx, shape, rng, kv_format=fmt)
            if L:
                g.cache.import_(kc, vc)
            vb, kb = v.copy(), k.copy()
            vb[bad:, 3::hd] = value
            if value != 1.0:
                kb[T - 1] = np.nan
            outs.append(g.forward_cached(q, kb, vb))
            g.close()
        for out in outs[1:]:
            assert np.array_equal(out[:bad], outs[0][:bad]), (L, np.isnan(out[:bad]).sum())
            assert not np.isfinite(out[bad:].reshape(T - bad, 8, hd)[:, :, 3]).any()


@pytest.mark.parametrize("hd,fmt", [(64, "f32"), (128, "bf16")])
def test_an_infinite_cached_column_stays_infinite(ctx, hd, fmt):
    """Every cached V row holds +Inf in one column: so does every output, also where a short last tile of positions lies
    where an earlier tile lay."""
    rng = np.random.default_rng(hd)
    shape = dict(H=16, KV=16, hd=hd, theta=10000.0)
    for L, T in ((130, 2), (9001, 40)):
        kc, vc = (rng.standard_normal((16, L, hd), dtype=np.float32) for _ in range(2))
        vc[:, :, 3] = np.inf
        q, k, v = qkv(rng, shape, T)
        v[:, 3::hd] = np.inf
        _, g = make_pair(ctx, shape, rng, kv_format=fmt)
        g.cache.import_(kc, vc)
        out = g.forward_cached(q, k, v).reshape(T, 16, hd)
        assert (out[:, :, 3] == np.inf).all()
        assert np.isfinite(np.delete(out, 3, axis=2)).all()
        g.close()
