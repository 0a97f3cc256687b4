"""Kernels at the sizes where their tiles, splits and dispatch rules end, against dense attention in 64 bits."""
import pytest
import torch

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
def test_split_rows(dtype, d, chunk, lens):
    # every lane layout (4 or 8 lanes per token, 1 to 8 granules each; the last two have rows of no whole granules), blocks that
    # end inside a chunk, clusters of 1 to 8 CTAs, warps without a block.  The pool's unused rows hold NaN.
    H, n = 3, len(lens)
    g = torch.Generator().manual_seed(d + chunk)
    eng = CabiEngine(H, d, chunk, dtype, max_chunks=sum(x // chunk + 2 for x in lens))
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
