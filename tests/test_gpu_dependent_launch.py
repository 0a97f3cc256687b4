"""Which kernels of a step are programmatic dependents of the kernel ahead, as the edges of a captured graph show it."""
import ctypes as C

import pytest
import torch

from chunk_attn import cabi
from gpu_helpers import CabiEngine

pytestmark = pytest.mark.gpu


RELAXED, PROGRAMMATIC = 2, 1   # of the driver's capture modes and types of edges


def programmatic_edges(step):
    """Of two steps captured one behind the other: (kernels, programmatic edges between them)."""
    cuda = C.CDLL("libcuda.so.1")
    step()
    stream, graph, nodes, n = torch.cuda.Stream(), C.c_void_p(), C.c_size_t(), C.c_size_t()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        handle = C.c_void_p(stream.cuda_stream)
        assert cuda.cuStreamBeginCapture_v2(handle, RELAXED) == 0
        try:
            step()
            step()
        finally:
            assert cuda.cuStreamEndCapture(handle, C.byref(graph)) == 0
    assert cuda.cuGraphGetNodes(graph, None, C.byref(nodes)) == 0
    n.value = 64
    ends, data = (C.c_void_p * 128)(), (C.c_uint8 * (8 * 64))()   # an edge's data: ports of its ends, its type, five bytes of nothing
    assert cuda.cuGraphGetEdges_v2(graph, ends, C.byref(ends, 64 * C.sizeof(C.c_void_p)), data, C.byref(n)) == 0 and n.value <= 64
    assert cuda.cuGraphDestroy(graph) == 0
    return nodes.value, sum(data[8 * i + 2] == PROGRAMMATIC for i in range(n.value))


def filled(dtype, d, lens, direct):
    g = torch.Generator().manual_seed(3)
    eng = CabiEngine(4, d, 64, dtype, max_chunks=40)
    eng.ctx.set_option(cabi.CA_OPT_DIRECT, direct)
    for i, n in enumerate(lens):
        eng.add_seq([1000 * i + j for j in range(n)], torch.randn(n, 4, d, generator=g), torch.randn(n, 4, d, generator=g))
    q = torch.randn(len(lens), 4, d, generator=g).to(dtype).cuda()
    out = torch.empty_like(q)
    eng.refresh()
    return eng.ctx.set_option, lambda: eng.ctx.attention(q, out, 0)


def latent(rows, H=32, lens=(70, 130)):
    import chunk_attn
    from chunk_attn import SpanBatch
    from test_gpu_latent_rows import EPS, frequencies
    dev, lens, R, rot = torch.device("cuda:0"), list(lens), 512, 64
    cache = chunk_attn.Attention.latent(n_heads=H, latent=R, rotated=rot, scale=(R + rot) ** -0.5, window=0, chunk_size=64, memory_mb=64, dtype=torch.bfloat16, device=dev)
    cache.set_option(cabi.CA_OPT_LATENT_ROWS, rows)
    freq = frequencies(rot)[1]
    qn, kn = torch.ones(16, device=dev), torch.ones(R, device=dev)
    tokens = [[1000 * i + j for j in range(n)] for i, n in enumerate(lens)]
    cache.extend([-1] * len(lens), tokens)
    rnd = lambda *shape: torch.randn(*shape, device=dev, generator=torch.Generator(device=dev).manual_seed(1)).bfloat16()
    cache.store_latent(rnd(sum(lens), 16 + R + rot), SpanBatch(tokens, [0] * len(lens), list(range(len(lens))), dev).positions, qn, kn, EPS, freq)
    spans = SpanBatch([[7]] * len(lens), lens, list(range(len(lens))), dev)
    cache.store_latent(rnd(len(lens), 16 + R + rot), spans.positions, qn, kn, EPS, freq, append_tokens=[7] * len(lens))
    q_lat, q, sink = rnd(len(lens), H, R), rnd(len(lens), H, 8 + rot), torch.zeros(H, device=dev)
    return cache.set_option, lambda: cache.forward_latent(q_lat, q, spans.positions, freq, sink)


def grouped(direct):
    import chunk_attn
    from chunk_attn import SpanBatch
    dev, lens, H, G, d = torch.device("cuda:0"), [70, 500], 8, 2, 64
    cache = chunk_attn.Attention.shaped(n_heads=H, n_kv_heads=G, d_key=d, d_value=d, scale=0.1, sink=True, chunk_size=64, memory_mb=64, dtype=torch.bfloat16, device=dev)
    cache.set_option(cabi.CA_OPT_DIRECT, direct)
    ones, freq = torch.ones(d, device=dev), torch.full((d // 2,), 0.1, device=dev)
    rnd = lambda *shape: torch.randn(*shape, device=dev, generator=torch.Generator(device=dev).manual_seed(1)).bfloat16()
    tokens = [[1000 * i + j for j in range(n)] for i, n in enumerate(lens)]
    cache.extend([-1] * len(lens), tokens)
    spans = SpanBatch(tokens, [0] * len(lens), list(range(len(lens))), dev)
    cache.store_qkv(rnd(sum(lens), (H + 2 * G) * d), spans.positions, ones, ones, 1e-5, d, freq, freq)
    spans = SpanBatch([[7]] * len(lens), lens, list(range(len(lens))), dev)
    q = cache.store_qkv(rnd(len(lens), (H + 2 * G) * d), spans.positions, ones, ones, 1e-5, d, freq, freq, append_tokens=[7] * len(lens))
    return cache.set_option, lambda: cache.forward_rows(q, spans.positions, freq)


CASES = {
    # kernels of a step, dependent ones of them with the option's bit 1 (attention) and bit 0 (merge)
    "one launch": (lambda: filled(torch.float16, 64, [70, 5], 2), 1, 1, 0),
    "any geometry": (lambda: filled(torch.float32, 64, [70, 5], 0), 1, 1, 0),
    "any geometry, rows of no granules": (lambda: filled(torch.float16, 20, [70, 5], 0), 1, 1, 0),
    "items": (lambda: filled(torch.float16, 128, [70, 500], 0), 2, 1, 1),
    "grouped, one launch": (lambda: grouped(2), 1, 1, 0),
    "grouped, items": (lambda: grouped(0), 2, 0, 1),
    "latent, by sequences": (lambda: latent(2), 1, 1, 0),
    "latent, items": (lambda: latent(0), 2, 1, 1),
}


@pytest.mark.parametrize("name", CASES)
def test_option(name):
    make, kernels, attention, merge = CASES[name]
    set_option, step = make()
    for mask in (3, 2, 1, 0):
        set_option(cabi.CA_OPT_DEPENDENT_LAUNCH, mask)
        count, edges = programmatic_edges(step)
        # the first step's attention kernel has none ahead of it
        want = (attention if mask & 2 else 0) + (2 * merge if mask & 1 else 0)
        assert (count, edges) == (2 * kernels, want), (mask, count, edges)


@pytest.mark.parametrize("heads", [16, 32, 64])
def test_tensor_memory_of_two_kernels(heads):
    # A latent step and, behind it on the stream, one over wide runs, whose kernel holds tensor memory while it waits for the kernel
    # ahead: results are those of steps alone.  (The latent kernel has its own before it lets the next one in.)
    from test_gpu_wide_finish import build
    for rows in (2, 0):
        _, step = latent(rows, heads, [70, 130] * 100)
        eng, _, q = build(4, 130, 8 * 64, [3], 8, 5)
        q, out = q.cuda(), torch.empty_like(q).cuda()
        wide = lambda: eng.ctx.attention(q, out, 0)
        eng.refresh()
        want_latent, _ = step().clone(), wide()
        torch.cuda.synchronize()
        want = out.clone()
        for _ in range(20):
            got = step()
            out.zero_()
            step()
            wide()
            step()
            wide()
        torch.cuda.synchronize()
        assert torch.equal(out, want) and torch.equal(got, want_latent) and eng.ctx.status() == 0
