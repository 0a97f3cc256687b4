"""Decode of latent caches by sequences (a CTA or a cluster of two for each, one launch) against attention in 64 bits, and where it is
taken."""
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
