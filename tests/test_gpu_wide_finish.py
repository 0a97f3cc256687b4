"""The wide-runs kernel as the only kernel of a step (one prompt under many rows, each with a short tail of its own) against
dense attention in 64 bits and against the step in several kernels."""
import pytest
import torch

from chunk_attn import cabi
from gpu_helpers import CabiEngine
from test_gpu_kernel_edges import dense

pytestmark = pytest.mark.gpu
C = 64


def build(H, n, shared, tails, n_ctas, seed, bad=None):
    """n rows over `shared` common tokens (whole chunks), row i with tails[i % len(tails)] tokens of its own.  bad: a row and what is
    wrong with its last token."""
    g = torch.Generator().manual_seed(seed)
    rnd = lambda k: (torch.randn(k, H, 128, generator=g)).half()
    eng = CabiEngine(H, 128, C, torch.float16, max_chunks=shared // C + 2 * n + 4)
    eng.ctx.set_option(cabi.CA_OPT_NUM_CTAS, n_ctas)   # few CTAs by comparison: blocks of rows are cut into few pieces
    eng.ctx.set_option(cabi.CA_OPT_WIDE_RUNS, 2)
    eng.ctx.set_option(cabi.CA_OPT_FINISH_IN_WIDE, 2)
    pk, pv = rnd(shared), rnd(shared)
    ctx = []
    for i in range(n):
        t = tails[i % len(tails)]
        k, v = torch.cat([pk, rnd(t)]), torch.cat([pv, rnd(t)])
        if bad and bad[0] == i:
            side, value = bad[1].split()
            (k if side == "key" else v)[-1, :, 5] = float(value)
        row = eng.add_seq(list(range(shared)) + [10_000 * (i + 1) + j for j in range(t)], k, v)
        ctx.insert(row, (k, v))
    return eng, ctx, rnd(n)


def off(eng, q):
    eng.ctx.set_option(cabi.CA_OPT_FINISH_IN_WIDE, 0)
    out = eng.forward(q)
    eng.ctx.set_option(cabi.CA_OPT_FINISH_IN_WIDE, 2)
    return out


# weights of 11 bits, fp32 sums, results below 2 rounded to fp16: the repository's bar for fp16
TOL = 1e-3


@pytest.mark.parametrize("H,n,pieces,n_ctas", [(2, 17, 1, 2), (3, 128, 1, 4), (2, 129, 1, 4), (4, 300, 1, 8), (3, 130, 2, 12), (2, 33, 2, 4), (5, 256, 2, 20)])
@pytest.mark.parametrize("shared,tails", [(2 * C, [8]), (5 * C, [1, 7, 8, 9, 63, 16, 2]), (32 * C, [3, 30])])
def test_one_kernel(H, n, pieces, n_ctas, shared, tails):
    if shared == 2 * C and pieces == 2:
        pieces = 1   # a piece has two chunks at least
    eng, ctx, q = build(H, n, shared, tails, n_ctas, H * n + shared)
    some = [0, 1, n // 2, n - 2, n - 1]
    for step in range(3):  # the tails grow beyond what the work list says
        got = eng.forward(q)
        st = eng.ctx.stats()
        assert st["n_items_wide"] == (n + 127) // 128 * H * pieces and st["n_items_short"] == n * H and st["kernels_per_step"] == 1
        want = dense(q[some].cuda(), [(ctx[r][0].cuda(), ctx[r][1].cuda()) for r in some], 128 ** -0.5)
        assert (got[some].double() - want).abs().max() < TOL
        assert (got.float() - off(eng, q).float()).abs().max() < TOL  # every row
        g1 = torch.Generator().manual_seed(step)
        k1, v1 = torch.randn(n, H, 128, generator=g1).half(), torch.randn(n, H, 128, generator=g1).half()
        if max(tails) + step >= C - 1:
            break
        eng.append_token([5] * n, k1, v1)
        ctx = [(torch.cat([k, a[None]]), torch.cat([v, b[None]])) for (k, v), a, b in zip(ctx, k1, v1)]
    assert eng.ctx.status() == 0


@pytest.mark.parametrize("n_ctas,pieces", [(4, 1), (8, 2)])
@pytest.mark.parametrize("tails", [[1], [9, 3]])
@pytest.mark.parametrize("what", ["key nan", "key inf", "value nan", "value inf"])
def test_a_row_with_no_number_stays_alone(n_ctas, pieces, tails, what):
    # a row's own token that is not a number, or infinite, shows in that row as it does in dense attention, not in the others (the
    # next row is walked by the same warp)
    H, n, bad = 2, 130, 41
    eng, ctx, q = build(H, n, 8 * C, tails, n_ctas, 7, bad=(bad, what))
    got = eng.forward(q)
    st = eng.ctx.stats()
    assert st["n_items_wide"] == 2 * H * pieces and st["kernels_per_step"] == 1
    want = dense(q.cuda(), [(k.cuda(), v.cuda()) for k, v in ctx], 128 ** -0.5)
    others = [r for r in range(n) if r != bad]
    assert (got[others].double() - want[others]).abs().max() < TOL
    if what.startswith("value"):
        assert torch.equal(got[bad, :, 5].isnan(), want[bad, :, 5].isnan()) and torch.equal(got[bad, :, 5].isinf(), want[bad, :, 5].isinf())
        got[bad, :, 5] = want[bad, :, 5] = 0
    number = ~torch.isnan(want[bad])   # an infinite key is a score of +inf, or one of -inf and then a weight of zero
    assert torch.equal(number, ~torch.isnan(got[bad])) and bool((got[bad].double() - want[bad])[number].abs().lt(TOL).all())
    assert bool(number.all()) == what.startswith("value") and not (what == "key nan" and bool(number.any()))


def test_empty_tails_and_peers():
    # freshly reserved tails hold nothing; the rows of a step may go into every rank's full-width output
    eng, ctx, q = build(2, 40, 4 * C, [0], 4, 1)
    got = eng.forward(q)
    assert eng.ctx.stats()["kernels_per_step"] == 1
    assert (got.cpu().double() - dense(q, ctx, 128 ** -0.5)).abs().max() < TOL
    peers = [torch.full((40, 6, 128), float("nan"), dtype=torch.float16, device="cuda") for _ in range(2)]
    eng.ctx.attention_to_peers(q.cuda().contiguous(), [p.data_ptr() for p in peers], 6, 3)
    torch.cuda.synchronize()
    for p in peers:
        assert torch.equal(p[:, 3:5], got) and torch.isnan(p[:, :3].float()).all()


def test_where_it_is_taken():
    # by default a batch this small goes in several kernels; a switch for the other finishing kernel holds here, too
    eng, _, q = build(2, 129, 8 * C, [8], 4, 2)
    eng.ctx.set_option(cabi.CA_OPT_FINISH_IN_WIDE, 1)
    eng.refresh()
    assert eng.ctx.stats()["kernels_per_step"] > 1
    eng.ctx.set_option(cabi.CA_OPT_FINISH_IN_WIDE, 2)
    assert eng.ctx.stats()["kernels_per_step"] == 1
    eng.ctx.set_option(cabi.CA_OPT_FINISH_IN_TAILS, 0)
    assert eng.ctx.stats()["kernels_per_step"] == 3
    with pytest.raises(cabi.CAError):
        eng.ctx.set_option(cabi.CA_OPT_FINISH_IN_WIDE, 3)


@pytest.mark.parametrize("H,n,shared,own,one", [(16, 856, 1536, 1, False),   # two pieces, 224 CTAs: 29 us in three kernels, 34 in one
                                                (16, 856, 1536, 8, False), (16, 1112, 1536, 8, True),
                                                (32, 600, 3776, 1, False),  # more CTAs than a wave, most of the last one idle: 78 and 85
                                                (32, 984, 1024, 8, True), (32, 856, 1024, 1, False)])
def test_rule(H, n, shared, own, one):
    # the work list alone says which way a step goes: no tokens are stored here
    eng = CabiEngine(H, 128, C, torch.float16, max_chunks=shared // C + n + 4)
    for i in range(n):
        eng.tree.add_seq_detailed(list(range(shared)) + [10_000 * (i + 1) + j for j in range(own)])
    eng.refresh()
    st = eng.ctx.stats()
    assert st["n_items_wide"] > 0 and (st["kernels_per_step"] == 1) == one
