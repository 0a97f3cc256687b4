"""Decode of latent caches by sequences (a CTA or a cluster of two for each, one launch) against attention in 64 bits, and where it is
taken."""
import ctypes as C

import numpy as np
import pytest
import torch

import chunk_attn
from chunk_attn import SpanBatch, cabi
from test_gpu_latent import DEV, close, rnd

pytestmark = pytest.mark.gpu
EPS = 1e-5


def frequencies(rot):
    f = 10000.0 ** (-2.0 * np.arange(rot // 2) / rot)
    return f, torch.from_numpy(np.stack([f.astype(np.float32), (f - f.astype(np.float32)).astype(np.float32)])).to(DEV)


def turn(x, positions, f):
    a = positions.reshape((-1,) + (1,) * (x.ndim - 1)) * f
    h = x.shape[-1] // 2
    u, w, c, s = x[..., :h], x[..., h:], np.cos(a), np.sin(a)
    return np.concatenate([u * c - w * s, w * c + u * s], -1)


def build(H, R, rot, window, lens, seed):
    """A cache of len(lens) sequences, their entries in 64 bits, and the last tokens' queries."""
    cache = chunk_attn.Attention.latent(n_heads=H, latent=R, rotated=rot, scale=(R + rot) ** -0.5, window=window, chunk_size=64,
                                        memory_mb=64 + sum(lens) * (R + rot + 64) * 2 // 2 ** 20, dtype=torch.bfloat16, device=DEV)
    f, freq = frequencies(rot)
    qn, kn = rnd(seed + 1, 16) * 0.1 + 1, rnd(seed + 2, R) * 0.1 + 1
    entries = []
    last = []
    for i, n in enumerate(lens):
        x = rnd(seed + 10 + i, n, 16 + R + rot).to(torch.bfloat16)
        tokens = [100_000 * (i + 1) + j for j in range(n)]
        cache.extend([-1], [tokens[:-1]])
        cache.store_latent(x[:-1].to(DEV), SpanBatch([tokens[:-1]], [0], [i], DEV).positions, qn.to(DEV), kn.to(DEV), EPS, freq)
        last.append(x[-1:])
        z = x.double().numpy()[:, 16:]
        lat = z[:, :R] / np.sqrt((z[:, :R] ** 2).mean(-1, keepdims=True) + EPS) * kn.double().numpy()
        entries.append((lat, turn(z[:, R:], np.arange(n, dtype=np.float64), f)))
    spans = SpanBatch([[7]] * len(lens), [n - 1 for n in lens], list(range(len(lens))), DEV)
    cache.store_latent(torch.cat(last).to(DEV), spans.positions, qn.to(DEV), kn.to(DEV), EPS, freq, append_tokens=[7] * len(lens))
    q_lat, q = rnd(seed + 3, len(lens), H, R).to(torch.bfloat16), rnd(seed + 4, len(lens), H, 8 + rot).to(torch.bfloat16)
    sink = rnd(seed + 5, H)
    want = []
    for i, (lat, key) in enumerate(entries):
        lo = max(0, lens[i] - window) if window else 0
        s = q_lat[i].double().numpy() @ lat[lo:].T + turn(q[i:i + 1, :, 8:].double().numpy(), np.array([lens[i] - 1.0]), f)[0] @ key[lo:].T
        s = np.concatenate([s * (R + rot) ** -0.5, sink.double().numpy()[:, None]], -1)
        p = np.exp(s - s.max(-1, keepdims=True))
        want.append((p / p.sum(-1, keepdims=True))[:, :-1] @ lat[lo:])
    return cache, lambda: cache.forward_latent(q_lat.to(DEV), q.to(DEV), spans.positions, freq, sink.to(DEV)), np.stack(want)


@pytest.mark.parametrize("H,R,rot", [(1, 64, 8), (16, 512, 64), (17, 192, 64), (32, 512, 64), (24, 44, 12), (40, 256, 32), (72, 128, 64)])
@pytest.mark.parametrize("window,lens", [(0, [2, 3, 63, 64, 65, 128, 129, 700]), (100, [2, 99, 100, 101, 163, 164, 165, 640]), (0, [200] * 80)])
def test_sequences(H, R, rot, window, lens):
    # one and two CTAs a sequence (8 sequences: two, 80: one), tiles that a CTA of two does not get, windows that begin inside a tile,
    # heads that fill a block of rows, a part of one, two; rows of the cache that are not whole lines
    cache, run, want = build(H, R, rot, window, lens, H + len(lens))
    out = {}
    for mode in (0, 1, 2):
        cache.set_option(cabi.CA_OPT_LATENT_ROWS, mode)
        out[mode] = run()
        close(out[mode], want, torch.bfloat16, "mode %d" % mode)
    assert cache.device_status() == 0
    with pytest.raises(RuntimeError):
        cache.set_option(cabi.CA_OPT_LATENT_ROWS, 3)


class Shape(C.Structure):
    _fields_ = [(n, C.c_int32) for n in ("n_heads", "n_kv_heads", "d_key", "d_value", "sink")] + [("scale", C.c_float), ("latent", C.c_int32), ("window", C.c_int32)]


class LatentArgs(C.Structure):
    _fields_ = [("q_lat", C.c_void_p), ("q_rot", C.c_void_p), ("q_rot_row", C.c_int64), ("q_rot_head", C.c_int64), ("out", C.c_void_p), ("n_rows", C.c_int32)] + \
               [(n, C.c_void_p) for n in ("positions", "freq", "sink", "row_entry", "path_off", "path_chunks", "blocks")] + \
               [(n, C.c_int32) for n in ("n_blocks", "block_rows", "delta_tokens")]


@pytest.mark.parametrize("head", [30, 64])
def test_chunks_ahead_of_the_window_that_are_not_full(head):
    # lists that the C interface takes: a sequence begins with a chunk of `head` tokens, which no window reaches any more.  Positions do
    # not follow from the number of chunks then; the step's result is that of its items, whatever the option says
    n, H, R, rot, window = 3, 16, 128, 64, 60
    shape = Shape(H, 1, R + rot, R, 0, 0.1, 1, window)
    size = cabi.lib.ca_chunk_bytes_shaped(C.byref(shape), 64, cabi.CA_DTYPE_BF16)
    g = torch.Generator(device="cuda").manual_seed(4)
    pool = torch.randn(4 * n * size // 2, generator=g, device="cuda").bfloat16()
    handle, stream = C.c_void_p(), C.c_void_p(torch.cuda.current_stream().cuda_stream)
    cabi.check(cabi.lib.ca_context_create_shaped(C.byref(handle), 0, C.byref(shape), 64, cabi.CA_DTYPE_BF16, C.c_void_p(pool.data_ptr()), C.c_int64(4 * n), 1))
    try:
        tokens = [head, 64, 64, 20]
        arr, m = cabi.make_infos([(4 * s + i, t, s, s + 1) for s in range(n) for i, t in enumerate(tokens)])
        q_lat, q_rot = (torch.randn(n, H, w, generator=g, device="cuda").bfloat16() for w in (R, rot))
        positions = torch.full((n,), sum(tokens) - 1, dtype=torch.int32, device="cuda")
        freq = frequencies(rot)[1]
        out = {}
        for mode in (0, 1, 2):
            cabi.check(cabi.lib.ca_context_set_option(handle, cabi.CA_OPT_LATENT_ROWS, mode))
            cabi.check(cabi.lib.ca_refresh_kernel_context(handle, arr, m, n, stream))
            out[mode] = torch.empty_like(q_lat)
            args = LatentArgs(q_lat.data_ptr(), q_rot.data_ptr(), H * rot, rot, out[mode].data_ptr(), n, positions.data_ptr(), freq.data_ptr(), None, None, None, None,
                              None, 0, 0, -1)
            cabi.check(cabi.lib.ca_latent_attention(handle, C.byref(args), stream))
            torch.cuda.synchronize()
        for mode in (1, 2):  # the two ways differ by the rounding of a bf16 result
            assert (out[mode].float() - out[0].float()).norm() < 2 ** -7 * out[0].float().norm()
    finally:
        cabi.lib.ca_context_destroy(handle)
