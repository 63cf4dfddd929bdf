"""epi_connect_noalloc's slot search against the rule itself, evaluated pair by
pair in numpy (connect_proc, cell_connection.cpp:70-129): a non-membrane cell
connects to every lower-index particle binned in the 5 x 5 x 5 bins around its
own (wrapped in x, y and z) whose distance satisfies the predicate.

Forms: the smallest grid (5 bins per axis, every window wraps), bin counts
that do and do not fill the scan's passes, dense tissues whose rows exceed a
warp, positions just outside the box, radii that reach across the window.
Lists are whole numbers: equality, no tolerance.
"""
import ctypes

import numpy as np
import pytest

from epi_b200 import capi

pytestmark = pytest.mark.gpu

AG = 2.0 + 1e-7


def pdiff(a, b, L):
    d = a - b
    return np.where(d > 0.5 * L, d - L, np.where(d <= -0.5 * L, d + L, d))


def rule(x, y, z, r, nmemb, nmx, nmy, lx, ly, lz, lt):
    """Rows of connected_cell (sorted), None for particles outside the grid."""
    n = len(x)
    an = (int(lx / 2 + 0.5), int(ly / 2 + 0.5), int(lz / 2))
    bins = np.stack([((0.5 * lx - pdiff(0.5 * lx, x, lx)) / AG).astype(int),
                     ((0.5 * ly - pdiff(0.5 * ly, y, ly)) / AG).astype(int),
                     (np.maximum(z, 0.0) / AG).astype(int)])
    own = np.stack([(x / AG).astype(int), (y / AG).astype(int), (z / AG).astype(int)])
    ok = np.all((bins >= 0) & (bins < np.array(an)[:, None]), axis=0)
    ok[nmemb:] &= np.all((own >= 0) & (own < np.array(an)[:, None]), axis=0)[nmemb:]
    rows = [set() for _ in range(n)]
    for j in range(nmemb):
        c, w = j % nmx, j // nmx
        rows[j] |= {w * nmx + (c - 1) % nmx, w * nmx + (c + 1) % nmx,
                    (w - 1) % nmy * nmx + c, (w + 1) % nmy * nmx + c}
    for c in range(nmemb, n):
        if not ok[c]:
            continue
        o = np.arange(c)
        near = ok[:c].copy()
        for k in range(3):
            d = (bins[k, :c] - own[k, c]) % an[k]
            near &= (d <= 2) | (d >= an[k] - 2)
        dx, dy, dz = pdiff(x[c], x[:c], lx), pdiff(y[c], y[:c], ly), z[c] - z[:c]
        rs = r[c] + r[:c]
        near &= (dx * dx + dy * dy) + dz * dz <= ((lt * lt) * rs) * rs
        for q in o[near]:
            rows[c].add(int(q))
            rows[q].add(c)
    return [sorted(v) if g else None for v, g in zip(rows, ok)]


def call(x, y, z, r, nmemb, nmx, nmy, lx, ly, lz, lt, max_conn):
    import torch
    f = capi.lib().epi_connect_noalloc
    f.argtypes = ([ctypes.c_void_p] * 4 + [ctypes.c_int32] * 4 + [ctypes.c_double] * 4 +
                  [ctypes.c_int32, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p])
    f.restype = ctypes.c_int
    d = [torch.tensor(a, dtype=torch.float64, device="cuda") for a in (x, y, z, r)]
    conn = torch.full((len(x), max_conn), -7, dtype=torch.int32, device="cuda")
    count = torch.full((len(x),), -7, dtype=torch.int32, device="cuda")
    rc = f(*(a.data_ptr() for a in d), len(x), nmemb, nmx, nmy, lx, ly, lz, lt, max_conn,
           conn.data_ptr(), count.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == capi.EPI_OK
    torch.cuda.synchronize()
    return conn.cpu().numpy(), count.cpu().numpy()


@pytest.mark.parametrize("lx,ly,lz,cells,radius,spread", [
    (9.5, 9.0, 10.0, 300, 0.5, 0.0),      # 5 bins per axis: every window wraps
    (9.0, 9.0, 10.0, 700, 1.4, 0.0),      # rows longer than a warp
    (16.0, 18.0, 20.0, 1500, 0.6, 0.3),   # positions just outside the box
    (10.0, 12.0, 64.0, 500, 3.0, 0.0),    # reach beyond the window in x and y
    (64.0, 62.0, 24.0, 900, 1.0, 0.0),    # 31 x 32 x 12 bins: more than one scan pass
])
def test_search_equals_the_rule(built, lx, ly, lz, cells, radius, spread):
    rng = np.random.default_rng(int(cells + 10 * lx))
    nmx, nmy = 7, 5
    nmemb = nmx * nmy
    n = nmemb + cells
    x = rng.uniform(-spread, lx - 0.01, n)
    y = rng.uniform(-spread, ly - 0.01, n)
    z = rng.uniform(-spread, lz - 0.01, n)
    r = radius * rng.uniform(0.6, 1.0, n)
    x[nmemb + 3], y[nmemb + 3] = lx, 0.0        # the box edge itself
    z[nmemb + 7] = lz + 5.0                     # outside the grid
    x[nmemb + 9] = np.nan
    max_conn = 160
    want = rule(np.nan_to_num(x, nan=-99.0), y, z, r, nmemb, nmx, nmy, lx, ly, lz, 1.2)
    conn, count = call(x, y, z, r, nmemb, nmx, nmy, lx, ly, lz, 1.2, max_conn)
    for i in range(n):
        if want[i] is None:
            assert count[i] == -1, i
        else:
            assert count[i] == len(want[i]), i
            assert list(conn[i, :count[i]]) == want[i], i
            assert np.all(conn[i, count[i]:] == -7), i
    assert max(len(w) for w in want if w is not None) <= max_conn
