"""The selective scan over its whole range of shapes: every number of states per lane, spans and runs of them, rows that can and
cannot be copied 16 bytes at a time, against the recurrence in 64 bits."""
import ctypes as C

import numpy as np
import pytest
import torch

import gagorax_oracle as oracle
from chunk_attn import SpanBatch, cabi, ops
from test_gpu_block_ops import close, rnd

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
# spans end before, at and behind the groups of 8 tokens and the 32 that are staged together
EDGES = [1, 7, 8, 9, 31, 32, 33, 65]


def scan(lens, channels, states, dtype, A=None):
    n, E = sum(lens), len(lens)
    x, z = rnd(1, n, channels).to(dtype), rnd(2, n, channels).to(dtype)
    dt, bc = rnd(3, n, channels), rnd(4, n, 2 * states)
    A = -torch.exp(rnd(5, channels, states)) if A is None else A
    D, bias = rnd(6, channels), rnd(7, channels) - 2
    state = torch.full((E + 1, channels, states), 7.0, device=DEV)
    spans = SpanBatch([[1] * k for k in lens], [0] * E, list(range(E, 0, -1)), DEV)
    y = ops.selective_scan(x.to(DEV), z.to(DEV), dt.to(DEV), bias.to(DEV), A.to(DEV), bc.to(DEV), D.to(DEV), state, spans)
    at, want, ends = 0, [], []
    num = lambda t: t.double().numpy()
    for k in lens:
        s = slice(at, at + k)
        o, S = oracle.selective_scan(num(x[s]), oracle.softplus(num(dt[s]) + num(bias)), num(A), num(bc[s])[:, :states], num(bc[s])[:, states:], num(D))
        want.append(o * oracle.silu(num(z[s])))
        ends.append(S)
        at += k
    return y, state, want, ends


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lens,channels,states", [
    (EDGES, 40, 3), (EDGES, 33, 6), (EDGES, 136, 8), (EDGES, 72, 16), (EDGES, 72, 18), (EDGES, 40, 64), (EDGES, 17, 129), (EDGES, 24, 256),
    ([40] * 20, 4096, 16), ([33] * 8, 4096, 64), ([300, 257], 200, 4), ([300, 257], 200, 16), ([400], 136, 128), ([400, 31], 130, 160),
    ([33] * 130, 64, 16),  # more spans than are put into order
    ([3, 32, 1, 9] * 60, 1024, 16), ([3, 32, 1, 9] * 60, 264, 100),  # short ones: several by a CTA
    # the kernel of short spans: one to four lanes a channel, some without states, rows that are not read four at a time
    ([1, 7, 8, 2, 9, 1, 17, 3], 40, 5), ([1, 7, 8, 2, 9, 1, 17, 3], 33, 8), ([1, 7, 8, 2, 9, 1, 33, 3], 72, 16), ([1, 7, 8, 2, 9, 1, 33, 3], 36, 13),
    ([1, 7, 8, 2, 9, 1, 17, 3], 72, 18), ([1, 7, 8, 2, 9, 1, 17, 3], 40, 32), ([33, 64, 65, 8] * 16, 4096, 16), ([33, 64, 65, 8] * 8, 1100, 20), ([128] + [1] * 15, 70, 16)])
def test_scan_shapes(lens, channels, states, dtype):
    y, state, want, ends = scan(lens, channels, states, dtype)
    close(y, np.concatenate(want), dtype)
    state = state.cpu()
    for e, S in enumerate(ends):
        close(state[len(lens) - e], S, torch.float32, "state")
    assert bool((state[0] == 7.0).all())


def test_rates_without_bound():
    """A state that is forgotten at once: nothing of it may come back with the tokens that fill up a span's last group."""
    A = -torch.exp(rnd(5, 48, 16))
    A[:, 3] = -float("inf")
    y, state, want, ends = scan([5, 12, 32], 48, 16, torch.float32, A)
    close(y, np.concatenate(want), torch.float32)
    for e, S in enumerate(ends):
        close(state[3 - e], S, torch.float32, "state")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lens", [[5, 33], [1, 1, 1]])
def test_smallest_steps(lens, dtype):
    # steps of exp(-88), which is below 2^-126, are steps: inputs of 1e38 bring them back into sight.  Spans and single tokens
    n, E, channels, states = sum(lens), len(lens), 40, 16
    x, z = torch.full((n, channels), 1e38).to(dtype), torch.ones(n, channels).to(dtype)
    dt, bias, bc = torch.full((n, channels), -88.0), torch.zeros(channels), torch.ones(n, 2 * states)
    state = torch.zeros(E, channels, states, device=DEV)
    spans = SpanBatch([[1] * k for k in lens], [0] * E, list(range(E)), DEV)
    ops.selective_scan(x.to(DEV), z.to(DEV), dt.to(DEV), bias.to(DEV), torch.full((channels, states), -1.0, device=DEV), bc.to(DEV),
                       torch.zeros(channels, device=DEV), state, spans)
    for e, k in enumerate(lens):  # every token adds the same; numbers below 2^-126 have 20 bits there
        want = k * float(np.exp(-88.0)) * x[0, 0].item()
        assert bool((state[e] / want - 1).abs().lt(1e-5).all())


class Spans(C.Structure):
    _fields_ = [(n, C.c_int32) for n in ("n_entries", "n_tokens", "max_tokens", "n_work", "work_len")] + \
               [(n, C.c_void_p) for n in ("cu", "start", "slot", "entry_of", "work", "work_off")]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lens,channels", [([3, 0, 5] * 100, 8192), ([0, 0, 9, 33, 0] * 40, 4096), ([0, 40], 64)])
@pytest.mark.parametrize("N", [16, 64])   # the kernel of short spans, and the one whose CTAs have several
def test_spans_without_tokens(lens, channels, N, dtype):
    # batches that the C interface takes: a CTA that has several spans goes on behind one without tokens, whose state stays (or, at a
    # sequence's beginning, becomes zero).  Compared with the batch without those spans, bit by bit
    E, n = len(lens), sum(lens)
    bf16 = dtype == torch.bfloat16
    x, z, dt, bc = rnd(1, n, channels).to(dtype).to(DEV), rnd(2, n, channels).to(dtype).to(DEV), rnd(3, n, channels).to(DEV), rnd(4, n, 2 * N).to(DEV)
    A, D, bias = (-torch.exp(rnd(5, channels, N))).to(DEV), rnd(6, channels).to(DEV), (rnd(7, channels) - 2).to(DEV)
    state0 = rnd(8, E, channels, N).to(DEV)
    scan = cabi.lib.ca_selective_scan
    scan.argtypes = [C.c_void_p] * 3 + [C.c_int64] + [C.c_void_p] * 4 + [C.c_int64] + [C.c_void_p] * 3 + [C.POINTER(Spans)] + [C.c_int] * 3 + [C.c_void_p]

    def run(entries):
        ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
        length = [lens[e] for e in entries]
        cu = ints([0] + list(np.cumsum(length)))
        pieces = [[i, int(c), int(c) + k, 0] for i, (k, c) in enumerate(zip(length, np.cumsum([0] + length)))]
        starts = ints([e % 2 for e in entries])  # every other one has a past
        slots, of = ints(entries), ints([i for i, k in enumerate(length) for _ in range(k)])
        work, off = ints(pieces), ints(list(range(len(entries) + 1)))
        sp = Spans(len(entries), n, max(lens), len(pieces), 64, cu.data_ptr(), starts.data_ptr(), slots.data_ptr(), of.data_ptr(), work.data_ptr(), off.data_ptr())
        y, state = torch.full((n, channels), float("nan"), dtype=dtype, device=DEV), state0.clone()
        assert scan(y.data_ptr(), x.data_ptr(), z.data_ptr(), channels, dt.data_ptr(), bias.data_ptr(), A.data_ptr(), bc.data_ptr(), 2 * N, D.data_ptr(),
                    state.data_ptr(), None, C.byref(sp), channels, N, cabi.CA_DTYPE_BF16 if bf16 else cabi.CA_DTYPE_F32, None) == 0
        torch.cuda.synchronize()
        return y, state

    y, state = run(list(range(E)))
    want_y, want = run([e for e in range(E) if lens[e]])
    assert bool(torch.isfinite(want_y).all())
    for e in range(E):
        if not lens[e] and e % 2 == 0:
            want[e] = 0
    assert torch.equal(y, want_y) and torch.equal(state, want)
