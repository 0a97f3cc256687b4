"""Kernels at the sizes where their tiles, splits and dispatch rules end, against dense attention in 64 bits."""
import numpy as np
import pytest
import torch

from chunk_attn import cabi
from gpu_helpers import CabiEngine

pytestmark = pytest.mark.gpu


def dense(q, contexts, scale):
    """q [n, H, d]; contexts: (k, v) [T, H, .] per row."""
    out = []
    for x, (k, v) in zip(q.double(), contexts):
        p = torch.softmax(torch.einsum("hd,thd->ht", x, k.double()) * scale, -1)
        out.append(torch.einsum("ht,thd->hd", p, v.double()))
    return torch.stack(out)


@pytest.mark.parametrize("dtype,d", [(torch.float16, 16), (torch.float16, 40), (torch.float16, 64), (torch.float16, 72), (torch.float16, 136),
                                     (torch.float16, 256), (torch.float32, 4), (torch.float32, 36), (torch.float32, 68), (torch.float32, 256),
                                     (torch.float16, 20), (torch.float32, 30)])
@pytest.mark.parametrize("chunk,lens", [(7, [1, 2, 6, 7, 8, 50]), (64, [1, 15, 16, 17, 63, 64, 65, 700]), (32, [33, 512]), (16, [9] * 70)])
@pytest.mark.parametrize("direct", [0, 1])
def test_split_rows(dtype, d, chunk, lens, direct):
    # every lane layout (4 or 8 lanes per token, 1 to 8 granules each; the last two have rows of no whole granules), blocks that
    # end inside a chunk, clusters of 1 to 8 CTAs, warps without a block; by default, fp16 rows of up to 128 elements may go to the
    # one-launch kernel instead.  The pool's unused rows hold NaN.
    if direct and (dtype == torch.float32 or d > 128 or d % 8 or chunk < 16):
        pytest.skip("these have one kernel")
    H, n = 3, len(lens)
    g = torch.Generator().manual_seed(d + chunk)
    eng = CabiEngine(H, d, chunk, dtype, max_chunks=sum(x // chunk + 2 for x in lens), direct=direct)
    kv = [(torch.randn(x, H, d, generator=g).to(dtype), torch.randn(x, H, d, generator=g).to(dtype)) for x in lens]
    for i, (k, v) in enumerate(kv):
        eng.add_seq([1000 * i + j for j in range(lens[i])], k, v)
    q = torch.randn(n, H, d, generator=g).to(dtype)
    # fp32 sums over up to 700 tokens, results rounded to the dtype: the repository's bars for both types
    tol = 1e-3 if dtype == torch.float16 else 1e-4
    assert (eng.forward(q).cpu().double() - dense(q, kv, d ** -0.5)).abs().max() < tol
    if chunk > 7:
        return
    k1, v1 = torch.randn(n, H, d, generator=g).to(dtype), torch.randn(n, H, d, generator=g).to(dtype)
    eng.append_token([5] * n, k1, v1)  # a token more than the work list says, some of them in a chunk of their own
    kv = [(torch.cat([k, a[None]]), torch.cat([v, b[None]])) for (k, v), a, b in zip(kv, k1, v1)]
    assert (eng.forward(q).cpu().double() - dense(q, kv, d ** -0.5)).abs().max() < tol


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(8, 2, 64, 64, 64), (40, 8, 40, 24, 18), (2, 1, 128, 48, 128), (3, 1, 256, 256, 6), (96, 4, 16, 16, 0)])
@pytest.mark.parametrize("lens", [[888], [889], [1, 1750, 64]])
def test_stored_heads_of_more_tokens_than_ctas(shape, dtype, lens):
    # The store walks tokens with a grid of at most 888 CTAs: exactly one each, one more, three for some; groups of 8 and 16
    # lanes with one and two granules each; heads that fill a pass, a part of one, several; a rotated part that ends inside a granule.
    import chunk_attn
    import gagorax_oracle as oracle
    from chunk_attn import SpanBatch
    from test_gpu_block_ops import close, oracle_attention, rnd
    H, G, dk, dv, rot = shape
    eps, base, scale, dev = 1e-4, 1000.0, dk ** -0.5, torch.device("cuda:0")
    cache = chunk_attn.Attention.shaped(n_heads=H, n_kv_heads=G, d_key=dk, d_value=dv, scale=scale, sink=True, chunk_size=64, memory_mb=64,
                                        dtype=dtype, device=dev)
    qn, kn = rnd(1, dk) * 0.2 + 1, rnd(2, dk) * 0.2 + 1
    freq = lambda n: torch.from_numpy(oracle.pair_frequencies(n, base)).float().to(dev)
    x = rnd(3, sum(lens), (H + G) * dk + G * dv).to(dtype)
    tokens = [[10_000 * i + t for t in range(n)] for i, n in enumerate(lens)]
    cache.extend([-1] * len(lens), tokens)
    spans = SpanBatch(tokens, [0] * len(lens), list(range(len(lens))), dev)
    q = cache.store_qkv(x.to(dev), spans.positions, qn.to(dev), kn.to(dev), eps, rot, freq(rot) if rot else None, freq(dv))
    o = cache.forward_rows(q, spans.positions, freq(dv), spans.entry_of).split(lens)
    for xs, part in zip(x.split(lens), o):
        close(part, oracle_attention(xs.double().numpy(), shape, qn.double().numpy(), kn.double().numpy(), eps, base, scale), dtype)
    assert cache.device_status() == 0


@pytest.mark.parametrize("shape", [(2, 2, 64, 64), (6, 2, 128, 64), (32, 8, 128, 128), (128, 1, 64, 128)])
@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("lens", [[1, 63, 64, 65, 129, 300], [40] * 80, [1] * 40])
def test_prompts_in_pieces(shape, sign, lens):
    # Portions on tcgen05: 1, 3, 4 and 128 query heads to a key/value head (blocks of 128, 126 and 128 rows of 128, 42, 32 and 1 tokens;
    # angles shared by a token's rows or not), pieces of one tile, last tiles of 1 token to all of them, more pieces than CTAs, a
    # negative scale.  What one sequence's values are must not reach another: the last one's are infinite.
    import chunk_attn
    import gagorax_oracle as oracle
    from chunk_attn import SpanBatch
    from test_gpu_block_ops import close, oracle_attention, rnd
    H, G, dk, dv = shape
    eps, base, scale, dev = 1e-4, 1000.0, sign * dk ** -0.5, torch.device("cuda:0")
    cache = chunk_attn.Attention.shaped(n_heads=H, n_kv_heads=G, d_key=dk, d_value=dv, scale=scale, sink=True, chunk_size=64, memory_mb=64,
                                        dtype=torch.bfloat16, device=dev)
    freq = lambda n: torch.from_numpy(oracle.pair_frequencies(n, base)).float().to(dev)
    qn, kn = rnd(1, dk) * 0.2 + 1, rnd(2, dk) * 0.2 + 1
    x = rnd(3, sum(lens), (H + G) * dk + G * dv).to(torch.bfloat16)
    x[-lens[-1]:, (H + G) * dk:] = float("inf")
    tokens = [[10_000 * i + t for t in range(n)] for i, n in enumerate(lens)]
    cache.extend([-1] * len(lens), tokens)
    spans = SpanBatch(tokens, [0] * len(lens), list(range(len(lens))), dev)
    q = cache.store_qkv(x.to(dev), spans.positions, qn.to(dev), kn.to(dev), eps, 32, freq(32), freq(dv))
    o = cache.forward_rows(q, spans.positions, freq(dv), spans.entry_of).split(lens)
    for xs, part in list(zip(x.split(lens), o))[:-1]:
        close(part, oracle_attention(xs.double().numpy(), shape + (32,), qn.double().numpy(), kn.double().numpy(), eps, base, scale), torch.bfloat16)
    assert cache.device_status() == 0


@pytest.mark.parametrize("shape", [(2, 2, 128, 128), (8, 1, 64, 64), (6, 2, 128, 64), (4, 2, 80, 48), (16, 2, 256, 256), (9, 1, 64, 128)])
@pytest.mark.parametrize("chunk", [64, 16])
@pytest.mark.parametrize("direct", [0, 1])
def test_decoded_rows_of_small_groups(shape, chunk, direct):
    # Items of at most 8 rows (groups of 1 to 8) and of 9, whose tokens end on every side of the 16 that a warp takes; tiles staged
    # verbatim and granule by granule.
    import chunk_attn
    H, G, dk, dv = shape
    lens = [1, 2, 15, 16, 17, 31, 33, 48, 63, 64, 65, 80, 127, 128, 700]
    g = torch.Generator().manual_seed(H + dk)
    cache = chunk_attn.Attention.shaped(n_heads=H, n_kv_heads=G, d_key=dk, d_value=dv, scale=dk ** -0.5, sink=False, chunk_size=chunk, memory_mb=64,
                                        dtype=torch.bfloat16, device="cuda:0")
    cache.set_option(cabi.CA_OPT_DIRECT, direct)
    kv = []
    for i, n in enumerate(lens):
        k, v = torch.randn(n, G, dk, generator=g).bfloat16(), torch.randn(n, G, dv, generator=g).bfloat16()
        cache.add_seq(tokens=[10_000 * i + t for t in range(n)], k=k.cuda(), v=v.cuda())
        kv.append((k.repeat_interleave(H // G, 1), v.repeat_interleave(H // G, 1)))
    q = torch.randn(len(lens), H, dk, generator=g).bfloat16()
    o = cache.forward_rows(q.cuda(), torch.tensor([n - 1 for n in lens], dtype=torch.int32, device="cuda:0"))
    want = dense(q, kv, dk ** -0.5)
    # the result's rounding to bf16 (2^-9 of it) and that of the weights (2^-17): far below this
    assert (o.cpu().double() - want).abs().max() < 8e-3 * max(1.0, float(want.abs().max()))
    assert cache.device_status() == 0 and (direct or cache.plan_stats()["kernels_per_step"] == 2)


@pytest.mark.parametrize("n,H", [(64, 8), (310, 16), (700, 16)])
@pytest.mark.parametrize("shared,most", [(0, 63), (256, 63), (256, 64)])
def test_short_tails_walked_by_half_warps(n, H, shared, most):
    # Private tails of up to 64 tokens (rounds of eight, both items of a warp of different lengths): 512 of them for the grid's 4736
    # half-warps, 4960 (a second item for some), 11200 (a third for some); with other partials to combine and without; a token appended,
    # into a chunk of its own for some.  Tails of 64 have a next chunk already and are not short: where there are some the merge kernel
    # finishes the rows, else the kernel itself does.
    g = torch.Generator().manual_seed(n)
    eng = CabiEngine(H, 128, 64, torch.float16, max_chunks=4 + 2 * n)
    eng.ctx.set_option(cabi.CA_OPT_NUM_CTAS, 8)  # the tails are many by comparison and take their own kernel
    sk, sv = torch.randn(shared, H, 128, generator=g).half(), torch.randn(shared, H, 128, generator=g).half()
    kv = []
    for i in range(n):
        own = (7 * i) % (most + 1) if shared else 1 + (7 * i) % 63
        k, v = torch.randn(own, H, 128, generator=g).half(), torch.randn(own, H, 128, generator=g).half()
        kv.append((torch.cat([sk, k]), torch.cat([sv, v])))
        eng.add_seq(list(range(shared)) + [100_000 + 1000 * i + j for j in range(own)], *kv[-1])
    q = torch.randn(n, H, 128, generator=g).half()

    def check():
        want = dense(q.cuda(), [(k.cuda(), v.cuda()) for k, v in kv], 128 ** -0.5)
        # the result's rounding to fp16, 2^-11 of it, and that of a shared run's weights: 2^-11 of the mean |value|, 0.8
        assert ((eng.forward(q).double() - want).abs() - want.abs() * 2.0 ** -11).max() < 4e-4

    check()
    rows = sum(k.shape[0] < shared + 64 for k, _ in kv)
    launches = []
    for finish in (0, 1):
        eng.ctx.set_option(cabi.CA_OPT_FINISH_IN_TAILS, finish)
        launches.append(eng.ctx.stats()["kernels_per_step"])
    assert eng.ctx.stats()["n_items_short"] == rows * H and launches[0] - launches[1] == (rows == n)
    check()
    k1, v1 = torch.randn(n, H, 128, generator=g).half(), torch.randn(n, H, 128, generator=g).half()
    eng.append_token([5] * n, k1, v1)
    kv = [(torch.cat([k, a[None]]), torch.cat([v, b[None]])) for (k, v), a, b in zip(kv, k1, v1)]
    check()


def test_queries_from_host_memory_of_any_alignment():
    # from 256 bytes to a megabyte, from an address that is a multiple of 16 bytes and from one of 8
    import chunk_attn
    for n, H in ((1, 1), (3, 32), (8, 32), (33, 8), (129, 31)):
        attn = chunk_attn.Attention(n_heads=H, d_head=128, chunk_size=64, memory_mb=256, dtype=torch.float16, device="cuda:0")
        for i in range(n):
            k = torch.randn(5 + i % 3, H, 128).half().cuda()
            attn.add_seq(tokens=[1000 * i + j for j in range(k.shape[0])], k=k, v=-k)
        room = torch.randn(n * H * 128 + 8).half().pin_memory()
        for at in (0, 4):
            q = room[at:at + n * H * 128].view(n, H, 128)
            assert torch.equal(attn.forward_host(q=q), attn.forward(q=q.cuda()).cpu())


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shape", [(4, 2, 64, 64), (4, 2, 40, 48), (4, 2, 128, 128), (2, 1, 256, 64)])
def test_head_norms_are_rounded_as_fp32_operations(dtype, shape):
    # Whole numbers, whose squares add up exactly in any order: mean, root, reciprocal and weights, one fp32 rounding each, then the
    # result's.  Every bit of it (an approximate root turns the rounding of some of the 16-bit results).
    import chunk_attn
    from chunk_attn import SpanBatch
    H, G, dk, dv = shape
    n, eps, dev = 700, 1e-5, torch.device("cuda:0")
    g = torch.Generator().manual_seed(dk)
    cache = chunk_attn.Attention.shaped(n_heads=H, n_kv_heads=G, d_key=dk, d_value=dv, scale=dk ** -0.5, sink=False, chunk_size=64, memory_mb=64,
                                        dtype=dtype, device=dev)
    x = torch.randint(-30, 31, (n, (H + G) * dk + G * dv), generator=g).float()
    w = torch.randn(dk, generator=g) * 0.2 + 1
    tokens = [list(range(n))]
    cache.extend([-1], tokens)
    spans = SpanBatch(tokens, [0], [0], dev)
    q = cache.store_qkv(x.to(dev, dtype), spans.positions, w.to(dev), w.to(dev), eps, 0, None, None)
    heads = x[:, :H * dk].view(n, H, dk).numpy()
    mean = np.square(heads).sum(-1, keepdims=True) / np.float32(dk)
    inv, w = np.float32(1) / np.sqrt(mean + np.float32(eps)), w.numpy()
    want = heads * inv * w if dtype == torch.float32 and dk == 256 else heads * (inv * w)  # heads of more than 32 granules: weights last
    assert want.dtype == np.float32
    assert torch.equal(q.view(n, H, -1)[..., :dk].cpu(), torch.from_numpy(want).to(dtype))


@pytest.mark.parametrize("shape", [(6, 2, 64, 64), (32, 8, 128, 128), (2, 2, 128, 64), (8, 1, 64, 128)])
@pytest.mark.parametrize("lens", [[1, 63, 64, 65, 129, 300], [40] * 80])
def test_prompts_on_each_kernel(shape, lens):
    # The weights of the softmax as one bf16 number (each within 2^-9 of itself, so a row within 2^-9 of the largest value) and as
    # two, and the mma.sync kernel; every result is rounded to bf16, another 2^-9 of it.
    import chunk_attn
    from chunk_attn import SpanBatch
    H, G, dk, dv = shape
    dev, n = torch.device("cuda:0"), len(lens)
    cache = chunk_attn.Attention.shaped(n_heads=H, n_kv_heads=G, d_key=dk, d_value=dv, scale=dk ** -0.5, sink=True, chunk_size=64, memory_mb=128,
                                        dtype=torch.bfloat16, device=dev)
    tokens = [[10_000 * i + t for t in range(x)] for i, x in enumerate(lens)]
    cache.extend([-1] * n, tokens)
    spans = SpanBatch(tokens, [0] * n, list(range(n)), dev)
    x = torch.randn(sum(lens), (H + G) * dk + G * dv, generator=torch.Generator().manual_seed(dk)).to(dev, torch.bfloat16)
    q = cache.store_qkv(x, spans.positions, None, None, 1e-5, 0, None, None)
    out = []
    for option in (0, 1, 2):
        cache.set_option(cabi.CA_OPT_SPAN_TENSOR, option)
        out.append(cache.forward_rows(q, spans.positions, None, spans.entry_of).double())
    start, at = 0, (H + G) * dk
    for length in lens:
        xs = x[start:start + length].double()
        kk = xs[:, H * dk:at].view(length, G, dk).repeat_interleave(H // G, 1)
        vv = xs[:, at:].view(length, G, dv).repeat_interleave(H // G, 1)
        s = torch.einsum("ihd,jhd->hij", xs[:, :H * dk].view(length, H, dk), kk) * dk ** -0.5
        s = s.masked_fill(torch.ones(length, length, dtype=torch.bool, device=dev).triu(1), float("-inf"))
        m = s.amax(-1, keepdim=True).clamp(min=0)  # the unit term: a score of zero without a value
        e = torch.exp(s - m)
        want = torch.einsum("hij,jhd->ihd", e / (e.sum(-1, keepdim=True) + torch.exp(-m)), vv)
        for o, weights in zip(out, (2.0 ** -16, 2.0 ** -16, 2.0 ** -9)):
            # the fast exponentials and the scores' fp32 sums: 2^-14 of the largest value
            bound = want.abs() * 2.0 ** -8 + (weights + 2.0 ** -14) * vv.abs().max()
            assert ((o[start:start + length].view_as(want) - want).abs() <= bound).all()
        start += length
    assert cache.device_status() == 0
