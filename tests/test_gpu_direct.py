"""The one-launch kernel against dense attention in 64 bits, and against the kernels it stands in for."""
import ctypes as C

import numpy as np
import pytest
import torch

from chunk_attn import cabi
from gpu_helpers import CabiEngine
from test_gpu_kernel_edges import dense

pytestmark = pytest.mark.gpu


def engine(H, d, chunk, max_chunks, mode=2):
    eng = CabiEngine(H, d, chunk, torch.float16, max_chunks=max_chunks)
    eng.ctx.set_option(cabi.CA_OPT_DIRECT, mode)
    return eng


def fill(eng, g, shared, lens, scale=1.0):
    """Sequences of `lens` own tokens over `shared` common ones; their contexts by row."""
    H, d = eng.H, eng.d
    rnd = lambda n: (torch.randn(n, H, d, generator=g) * scale).half()
    pk, pv = rnd(shared), rnd(shared)
    ctx = []
    for i, n in enumerate(lens):
        k, v = torch.cat([pk, rnd(n)]), torch.cat([pv, rnd(n)])
        row = eng.add_seq(list(range(shared)) + [10_000 * (i + 1) + j for j in range(n)], k, v)
        ctx.insert(row, (k, v))
    return ctx


# Scores and sums are fp32, weights have 22 bits (or fp16's 11 with 64-token chunks of 128, where they had them before); what is
# left is the rounding of the result: 2^-11 of values that are below 2 here, and the repository's bar for fp16 above it.
TOL = 1e-3


@pytest.mark.parametrize("d,chunk", [(128, 64), (128, 32), (64, 64), (64, 16), (96, 40), (72, 24), (40, 64), (32, 16), (8, 17), (120, 64)])
@pytest.mark.parametrize("shared,lens", [(0, [1]), (0, [15, 16, 17]), (0, [700]), (64, [1, 63, 64, 65]), (130, [5, 5, 5, 5, 5]), (200, [33] * 8),
                                         (100, [7] * 9), (64, [300, 1, 20] * 6)])
def test_edges(d, chunk, shared, lens):
    # instances of every width, 1 to 8 rows a block and several blocks, clusters of every size, ranges that end inside a chunk.
    # The pool's unused rows hold NaN.
    H = 3
    g = torch.Generator().manual_seed(d + chunk + shared)
    eng = engine(H, d, chunk, max_chunks=sum(n // chunk + 3 for n in lens) + shared // chunk + 4)
    ctx = fill(eng, g, shared, lens)
    q = torch.randn(len(lens), H, d, generator=g).half()
    for step in range(3):  # tokens beyond what the work list says
        got = eng.forward(q).cpu().double()
        assert eng.ctx.stats()["kernels_per_step"] == 1
        want = dense(q, ctx, d ** -0.5)
        assert (got - want).abs().max() < TOL
        if step == 0:  # and the kernels it stands in for
            eng.ctx.set_option(cabi.CA_OPT_DIRECT, 0)
            eng.valid = False
            assert (eng.forward(q).cpu().double() - want).abs().max() < TOL
            eng.ctx.set_option(cabi.CA_OPT_DIRECT, 2)
            eng.valid = False
        k1, v1 = torch.randn(len(lens), H, d, generator=g).half(), torch.randn(len(lens), H, d, generator=g).half()
        eng.append_token([7] * len(lens), k1, v1)
        ctx = [(torch.cat([k, a[None]]), torch.cat([v, b[None]])) for (k, v), a, b in zip(ctx, k1, v1)]


@pytest.mark.parametrize("d,chunk", [(128, 64), (64, 32)])
def test_two_levels_and_scores_that_rise(d, chunk):
    # groups of rows over prompts of their own: the rows that see a chunk change along a warp's range; scores that grow by
    # more than the step in which the reference follows them, and by less
    H, g = 2, torch.Generator().manual_seed(5)
    eng = engine(H, d, chunk, max_chunks=200)
    root = (torch.randn(2 * chunk, H, d, generator=g).half(), torch.randn(2 * chunk, H, d, generator=g).half())
    ctx = []
    for i in range(11):
        grp = torch.Generator().manual_seed(i // 3)
        gk, gv = torch.randn(chunk, H, d, generator=grp).half() * 2, torch.randn(chunk, H, d, generator=grp).half()
        own = 20 + 13 * i
        k = torch.cat([root[0], gk, torch.randn(own, H, d, generator=g).half() * torch.linspace(0.5, 6, own)[:, None, None]]).half()
        v = torch.cat([root[1], gv, torch.randn(own, H, d, generator=g).half()])
        row = eng.add_seq(list(range(2 * chunk)) + [500 * (i // 3 + 1) + j for j in range(chunk)] + [10_000 * (i + 1) + j for j in range(own)], k, v)
        ctx.insert(row, (k, v))
    q = torch.randn(11, H, d, generator=g).half()
    assert (eng.forward(q).cpu().double() - dense(q, ctx, d ** -0.5)).abs().max() < 2 * TOL  # values up to 4


@pytest.mark.parametrize("d,chunk", [(128, 64), (64, 64)])
def test_a_row_with_infinities_stays_alone(d, chunk):
    H, g, lens = 2, torch.Generator().manual_seed(9), [50, 90, 20, 64]
    eng = engine(H, d, chunk, max_chunks=40)
    rnd = lambda n: torch.randn(n, H, d, generator=g).half()
    pk, pv = rnd(chunk), rnd(chunk)
    ctx = []
    for i, n in enumerate(lens):
        k, v = torch.cat([pk, rnd(n)]), torch.cat([pv, rnd(n)])
        if i == 1:
            v[chunk + 3], k[chunk + 5] = float("inf"), float("nan")
        eng.add_seq(list(range(chunk)) + [1000 * (i + 1) + j for j in range(n)], k, v)
        ctx.append((k, v))
    q = rnd(4)
    got, want = eng.forward(q).cpu().double(), dense(q, ctx, d ** -0.5)
    assert torch.isnan(got[1]).all()
    keep = [0, 2, 3]
    assert (got[keep] - want[keep]).abs().max() < TOL


@pytest.mark.parametrize("d,chunk", [(128, 64), (64, 64), (128, 32), (96, 40), (40, 64), (8, 17)])
@pytest.mark.parametrize("shared,lens", [(0, [1]), (0, [900]), (64, [50, 90, 20, 64]), (130, [5, 70, 1, 200, 33, 16, 17, 40]), (64, [30] * 11)])
@pytest.mark.parametrize("where", ["own", "shared"])
def test_infinite_values(d, chunk, shared, lens, where):
    # weights of 1 (a single token) down to 2^-20, blocks of 1 to 8 rows: an infinite value comes out as it is, infinities of both signs as
    # NaN, and neither reaches another element or, from a row's own tokens, another row
    if where == "shared" and not shared:
        pytest.skip("no shared tokens")
    H, g, n = 2, torch.Generator().manual_seed(d + chunk + len(lens)), len(lens)
    eng = engine(H, d, chunk, max_chunks=sum(x // chunk + 3 for x in lens) + shared // chunk + 4)
    rnd = lambda k, scale=1.0: (torch.randn(k, H, d, generator=g) * scale).half()
    pk, pv = rnd(shared, 2.0), rnd(shared)
    if where == "shared":
        pv[3, :, 0], pv[40, :, 1], pv[5, 0, 2] = float("inf"), float("-inf"), float("inf")
    ctx = []
    for i, length in enumerate(lens):
        k, v = rnd(length, 2.0), rnd(length)
        if where == "own" and i == n // 2:
            v[length // 2, :, 0], v[-1, :, 1], v[0, 1, 2] = float("inf"), float("-inf"), float("inf")
            if length > 2:
                v[1, :, 3], v[2, :, 3] = float("inf"), float("-inf")
        k, v = torch.cat([pk, k]), torch.cat([pv, v])
        row = eng.add_seq(list(range(shared)) + [10_000 * (i + 1) + j for j in range(length)], k, v)
        ctx.insert(row, (k, v))
    q = rnd(n)
    got, want = eng.forward(q).cpu().double(), dense(q, ctx, d ** -0.5)
    finite = torch.isfinite(want)
    assert ((got[finite] - want[finite]).abs() < TOL * want[finite].abs().clamp(min=1)).all()  # values are up to 4
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isposinf(got), torch.isposinf(want)) and torch.equal(torch.isneginf(got), torch.isneginf(want))
    if where == "own":
        assert (~finite.flatten(1).all(1)).sum() == 1


@pytest.mark.parametrize("d,chunk", [(64, 64), (128, 32), (128, 64), (32, 16)])
@pytest.mark.parametrize("rows", [1, 4, 8])
def test_many_small_weights(d, chunk, rows):
    # one token of large weight and no value, 4000 of 2^-26 to 2^-30 of it with values of up to 60000, rows alone and over shared tokens:
    # the small ones are the result.  Values to 1 %: its distance from their weights' last bit is what is looked at
    H, n = 2, 4000
    eng = engine(H, d, chunk, max_chunks=(n + 64) // chunk + 3 * rows + 4)
    k, v = torch.zeros(n, H, d), torch.full((n, H, d), 60000.0)
    k[:, :, 0] = -torch.linspace(0, 2.8, n)[:, None]
    k[7, :, 0], v[7] = 18.0, 0.0
    own = torch.full((1, H, d), -10.0).half()
    ctx = []
    for i in range(rows):
        kk, vv = torch.cat([k.half(), own]), torch.cat([v.half(), own])
        row = eng.add_seq(list(range(n)) + [10_000 * (i + 1)], kk, vv)
        ctx.insert(row, (kk, vv))
    q = torch.zeros(rows, H, d)
    q[:, :, 0] = d ** 0.5
    want = dense(q.half(), ctx, d ** -0.5)
    for mode in (0, 2) if (d, chunk) != (128, 64) else (2,):  # the items' kernels have weights of 11 bits
        eng.ctx.set_option(cabi.CA_OPT_DIRECT, mode)
        eng.valid = False
        got = eng.forward(q.half()).cpu().double()
        assert want.abs().min() > 0.5 and ((got - want).abs() < 0.01 * want.abs()).all(), mode


def test_the_same_as_the_other_kernels():
    # one switch between them, the same tree: results differ by roundings only, and a row without tokens is zero both ways
    for d, chunk in ((128, 64), (80, 32)):
        H, g = 4, torch.Generator().manual_seed(3)
        eng = engine(H, d, chunk, max_chunks=80)
        fill(eng, g, 2 * chunk, [30, 1, 77, 64, 5])
        q = torch.randn(5, H, d, generator=g).half()
        out = {}
        for mode in (0, 1, 2):
            eng.ctx.set_option(cabi.CA_OPT_DIRECT, mode)
            eng.valid = False
            out[mode] = eng.forward(q).float()
        assert (out[0] - out[2]).abs().max() < TOL and (out[0] - out[1]).abs().max() < TOL
        # queries that do not lie on 16 bytes: what was taken before is taken still, by the any-geometry kernel
        if d != 128:
            odd = torch.empty(q.numel() + 1, dtype=torch.float16, device="cuda")[1:].view(q.shape).copy_(q)
            res = torch.empty_like(q, device="cuda")
            eng.ctx.attention(odd, res, 0)
            assert (res.float() - out[0]).abs().max() < TOL


@pytest.mark.parametrize("H,lens,items", [(4, [400], True), (2, [339] * 10, True), (8, [64], False), (32, [400], False)])
def test_host_calls_of_few_rows(H, lens, items):
    # calls on host buffers: few rows that would take clusters of CTAs go by items, bit by bit as with the one-launch kernel off
    g = torch.Generator().manual_seed(H)
    eng = engine(H, 128, 64, max_chunks=sum(n // 64 + 3 for n in lens), mode=1)
    ctx = fill(eng, g, 0, lens)
    q = torch.randn(len(lens), H, 128, generator=g).half()
    out = {}
    for mode in (0, 1, 2):
        eng.ctx.set_option(cabi.CA_OPT_DIRECT, mode)
        eng.valid = False
        eng.refresh()
        out[mode] = torch.empty_like(q)
        eng.ctx.attention_host(q, out[mode])
        assert (out[mode].double() - dense(q, ctx, 128 ** -0.5)).abs().max() < TOL
    assert not torch.equal(out[0], out[2]) and torch.equal(out[1], out[0 if items else 2])


def test_captured_and_replayed():
    H, d, chunk, g = 4, 64, 32, torch.Generator().manual_seed(1)
    eng = engine(H, d, chunk, max_chunks=40)
    ctx = fill(eng, g, 40, [20, 50])
    q = torch.randn(2, H, d, generator=g).half().cuda()
    out = torch.empty_like(q)
    eng.refresh()
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        eng.ctx.attention(q, out, 0)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            eng.ctx.attention(q, out, 0)
    q.copy_(torch.randn(2, H, d, generator=g).half())
    graph.replay()
    torch.cuda.synchronize()
    assert (out.cpu().double() - dense(q.cpu(), ctx, d ** -0.5)).abs().max() < TOL


@pytest.mark.parametrize("heads,kv,d", [(4, 4, 64), (6, 3, 128), (16, 4, 128), (12, 3, 64), (16, 2, 128), (8, 1, 64)])
@pytest.mark.parametrize("sink,scale", [(True, None), (False, -0.07)])
@pytest.mark.parametrize("chunk,lens", [(64, [1, 15, 16, 17, 63, 64, 65, 129]), (32, [700]), (64, [33] * 20), (48, [5, 300])])
def test_grouped_heads(heads, kv, d, sink, scale, chunk, lens):
    # 1 to 8 query heads to a key/value head, with and without the sink, a scale that turns the order of scores round, values turned back;
    # the items' kernels, the rule's choice and this kernel against the oracle
    import chunk_attn
    import gagorax_oracle as oracle
    from chunk_attn import SpanBatch
    from test_gpu_block_ops import close, rnd
    dev, base, eps, dt = torch.device("cuda:0"), 500.0, 1e-5, torch.bfloat16
    scale = d ** -0.5 if scale is None else scale
    cache = chunk_attn.Attention.shaped(n_heads=heads, n_kv_heads=kv, d_key=d, d_value=d, scale=scale, sink=sink, chunk_size=chunk, memory_mb=64, dtype=dt, device=dev)
    qn, kn = rnd(1, d) * 0.2 + 1, rnd(2, d) * 0.2 + 1
    kf = torch.from_numpy((base ** (-2.0 * np.arange(d // 2) / d)).astype(np.float32)).to(dev)
    width, want, last = (heads + 2 * kv) * d, [], []
    for i, n in enumerate(lens):
        x = rnd(10 + i, n + 1, width).to(dt)
        tokens = [10_000 * (i + 1) + j for j in range(n)]
        cache.extend([-1], [tokens])
        cache.store_qkv(x[:n].to(dev), SpanBatch([tokens], [0], [i], dev).positions, qn.to(dev), kn.to(dev), eps, d, kf, kf)
        last.append(x[n:])
        z, pos = x.double().numpy(), np.arange(n + 1)
        q, k, v = (z[:, a:b].reshape(n + 1, -1, d) for a, b in ((0, heads * d), (heads * d, (heads + kv) * d), ((heads + kv) * d, width)))
        q = oracle.rotary(oracle.rms_norm(q, qn.double().numpy(), eps), pos, d, base)[-1]
        k, v = oracle.rotary(oracle.rms_norm(k, kn.double().numpy(), eps), pos, d, base), oracle.rotary(v, pos, d, base)
        s = np.einsum("hd,thd->ht", q, np.repeat(k, heads // kv, 1)) * scale
        top = np.maximum(s.max(1, keepdims=True), 0.0) if sink else s.max(1, keepdims=True)
        p = np.exp(s - top)
        o = np.einsum("ht,thd->hd", p / (p.sum(1, keepdims=True) + (np.exp(-top) if sink else 0.0)), np.repeat(v, heads // kv, 1))
        want.append(oracle.rotary(o[None], np.array([-n]), d, base))
    spans = SpanBatch([[7]] * len(lens), lens, list(range(len(lens))), dev)
    q = cache.store_qkv(torch.cat(last).to(dev), spans.positions, qn.to(dev), kn.to(dev), eps, d, kf, kf, append_tokens=[7] * len(lens))
    for mode in (0, 1, 2):
        cache.set_option(cabi.CA_OPT_DIRECT, mode)
        got = cache.forward_rows(q, spans.positions, kf)
        close(got, np.concatenate(want), dt, "mode %d" % mode)
    assert cache.plan_stats()["kernels_per_step"] == 1 and cache.device_status() == 0


class Shape(C.Structure):
    _fields_ = [(n, C.c_int32) for n in ("n_heads", "n_kv_heads", "d_key", "d_value", "sink")] + [("scale", C.c_float), ("latent", C.c_int32), ("window", C.c_int32)]


class RowsArgs(C.Structure):
    _fields_ = [("q", C.c_void_p), ("out", C.c_void_p), ("n_rows", C.c_int32)] + [(n, C.c_void_p) for n in ("positions", "value_freq", "row_entry", "path_off", "path_chunks", "blocks")] + \
               [("n_blocks", C.c_int32), ("block_rows", C.c_int32)]


def stream_now():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def rewritten_plan(handle, infos, n_seqs, d):
    """A plan built for the context, whose one-launch lists are then cut again, for single rows and heads of d elements."""
    arr, n = cabi.make_infos(infos)
    plan, cluster = C.c_void_p(), C.c_int()
    cabi.check(cabi.lib.ca_plan_build_for_context(handle, C.byref(plan), arr, n, n_seqs))
    cabi.check(cabi.lib.ca_plan_direct(plan, 2, d, 1, C.byref(cluster)))
    assert cluster.value > 0
    cabi.check(cabi.lib.ca_refresh_from_plan(handle, plan, stream_now()))
    cabi.lib.ca_plan_destroy(plan)


@pytest.mark.parametrize("dtype,d,off", [(torch.float32, 64, False), (torch.float16, 64, True), (torch.float16, 128, True)])
def test_lists_that_are_not_this_contexts(dtype, d, off):
    # lists cut for other kernels than a context's (fp32 caches, the option switched off) are left aside; its own way is taken
    g = torch.Generator().manual_seed(2)
    eng = CabiEngine(4, d, 64, dtype, max_chunks=40)
    if off:
        eng.ctx.set_option(cabi.CA_OPT_DIRECT, 0)
    rnd = lambda n: torch.randn(n, 4, d, generator=g).to(dtype)
    ctx = []
    for i, n in enumerate([70, 5, 200]):
        k, v = rnd(n), rnd(n)
        ctx.insert(eng.add_seq([1000 * i + j for j in range(n)], k, v), (k, v))
    q = rnd(3)
    want = eng.forward(q)
    kernels = eng.ctx.stats()["kernels_per_step"]
    rewritten_plan(eng.ctx._h, eng.tree.get_chunks(), 3, d)
    assert torch.equal(eng.forward(q), want) and eng.ctx.stats()["kernels_per_step"] == kernels
    assert (want.cpu().double() - dense(q, ctx, d ** -0.5)).abs().max() < TOL


def test_lists_of_rows_for_grouped_heads():
    # blocks of 8 rows are blocks of 32 columns where four query heads share a key/value head: such lists are left aside
    n, d, heads, kv = 8, 64, 16, 4
    shape = Shape(heads, kv, d, d, 1, 0.1, 0, 0)
    size = cabi.lib.ca_chunk_bytes_shaped(C.byref(shape), 64, cabi.CA_DTYPE_BF16)
    g = torch.Generator(device="cuda").manual_seed(4)
    pool = torch.randn(12 * size // 2, generator=g, device="cuda").bfloat16()
    handle = C.c_void_p()
    cabi.check(cabi.lib.ca_context_create_shaped(C.byref(handle), 0, C.byref(shape), 64, cabi.CA_DTYPE_BF16, C.c_void_p(pool.data_ptr()), C.c_int64(12), 1))
    try:
        infos = [(0, 64, 0, n)] + [(1 + i, 20 + i, i, i + 1) for i in range(n)]
        q = torch.randn(n, heads, d, generator=g, device="cuda").bfloat16()
        positions = torch.tensor([64 + 19 + i for i in range(n)], dtype=torch.int32, device="cuda")
        stats = cabi.PlanStats()

        def run():
            out = torch.empty_like(q)
            args = RowsArgs(q.data_ptr(), out.data_ptr(), n, positions.data_ptr(), None, None, None, None, None, 0, 0)
            cabi.check(cabi.lib.ca_attention_rows(handle, C.byref(args), stream_now()))
            cabi.check(cabi.lib.ca_context_stats(handle, C.byref(stats)))
            torch.cuda.synchronize()
            return out, stats.as_dict()["kernels_per_step"]

        arr, m = cabi.make_infos(infos)
        cabi.check(cabi.lib.ca_context_set_option(handle, cabi.CA_OPT_DIRECT, 0))
        cabi.check(cabi.lib.ca_refresh_kernel_context(handle, arr, m, n, stream_now()))
        want, kernels = run()
        cabi.check(cabi.lib.ca_context_set_option(handle, cabi.CA_OPT_DIRECT, 2))
        rewritten_plan(handle, infos, n, d)
        got, now = run()
        assert torch.equal(got, want) and now == kernels > 1
        status = C.c_int32()
        assert cabi.lib.ca_status_read(handle, stream_now(), C.byref(status)) == 0
    finally:
        cabi.lib.ca_context_destroy(handle)
