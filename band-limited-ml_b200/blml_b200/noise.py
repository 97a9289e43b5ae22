"""NumPy's seeded normals, drawn by several threads.

The solver's starts take their noise from default_rng(seed).standard_normal, as the reference draws it
(blml_binned.py:429-436). PCG64 jumps to any place of its raw stream, and a normal takes one raw word, now and then more
(the ziggurat's rejections), so a thread that starts at an arbitrary place may begin inside another draw, but falls into
the true draws' boundaries as soon as the two meet, and stays there. Each thread therefore draws past the next one's
place, and the pieces are joined where four values in a row agree: the very values one thread would draw."""
import os
from concurrent.futures import ThreadPoolExecutor

import numpy as np

_SERIAL = 1 << 17        # below: one thread (1.3 ms; starting the others and joining them costs 0.5)
_LEAD = 64               # draws that a thread gives up to fall into step
_RAW = 1.03              # raw words per draw, with room (1.022 on average)


def _pieces(seed, n, threads):
    """The first n normals of default_rng(seed), as consecutive arrays; None when two threads did not meet."""
    L = int(np.ceil(n * _RAW / threads)) + 4 * _LEAD

    def draw(k):
        g = np.random.Generator(np.random.PCG64(seed).advance(k * L) if k else np.random.PCG64(seed))
        return g, g.standard_normal(L + 4 * _LEAD if k < threads - 1 else L)

    with ThreadPoolExecutor(threads) as pool:
        parts = list(pool.map(draw, range(threads)))
    out, at, total = [], 0, 0
    for k in range(threads):
        a = parts[k][1]
        end = len(a)
        if k < threads - 1:
            nxt = parts[k + 1][1][_LEAD:_LEAD + 4]
            lo = int(len(a) / _RAW) - 8 * _LEAD             # the next thread's place lies past this draw
            hit = np.flatnonzero(a[lo:-4] == nxt[0]) + lo
            if len(hit) != 1 or not np.array_equal(a[hit[0]:hit[0] + 4], nxt):
                return None
            end = int(hit[0])
        piece = a[at:min(end, at + n - total)]
        out.append(piece); total += len(piece)
        if total >= n:
            return out
        at = _LEAD
    out.append(parts[-1][0].standard_normal(n - total))     # the last thread's generator goes on
    return out


def normal_pieces(seed, n, threads=None):
    """np.random.default_rng(seed).standard_normal(n) as a list of arrays to be joined."""
    if threads is None:
        threads = min(8, len(os.sched_getaffinity(0)))
    if n >= _SERIAL and threads > 1 and isinstance(seed, (int, np.integer)):
        out = _pieces(seed, n, threads)
        if out is not None:
            return out
    return [np.random.default_rng(seed).standard_normal(n)]


def seeded_normals(seed, n, device, out=None):
    """default_rng(seed).standard_normal(n) on the device (float64); out: a vector to fill."""
    import torch
    if out is None:
        out = torch.empty(n, dtype=torch.float64, device=device)
    at = 0
    for a in normal_pieces(seed, n):
        out[at:at + len(a)].copy_(torch.from_numpy(a))
        at += len(a)
    return out
