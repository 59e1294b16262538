"""Field map of a solved BEM problem: the perturbation field as polynomials
over square cells of a quadtree in the (rho, z) half plane, read by the
float64 form of the adaptive far rule (csrc/spt_map.cu, spt_device.cuh).

Away from the surface the field is analytic, so a cell a few half-widths from
it needs 12 x 12 coefficients for 1e-14 of the field.  A cell is kept when
its highest two Chebyshev orders are below TAIL of its largest coefficient
(sampled by the direct sum with tighter thresholds than the adaptive rule's
own), and divided otherwise; near a panel (closer than two of its lengths)
and behind the surface there are no cells, and points there take the direct
sum, with the Gauss-8 panel nodes that are kept beside the map for it.  Not
in the reference.

Sampling the cells takes 10 to 250 ms, so it waits until a geometry has been
asked for about as many points as its direct sums evaluate in that time
(`worth`); until then its map has no cells, only the panel nodes.
"""

import ctypes

import numpy as np

from . import _lib

N = _lib.MAP_N
TAIL = 2e-14         # accepted truncation, of the cell's largest coefficient
KAPPA = 3.0          # half-widths from the surface from which a cell is tried
KAPPA_SURE = 12.0    # ... and taken as it is: (2 KAPPA_SURE)^-N is far below rounding
REACH = 24.0         # half side of the root square, in radii of the profile's bounding sphere
MAX_CELLS = 32768    # 76 MB; the levels nearest the surface are left out beyond it
MAX_LEVEL = 28       # the tables' last level: MAP_ROOT_BITS + 4 MAP_BITS
# points that the direct sums evaluate in the time the cells take: measured 0.9 M
# (39 panels, 10 ms), 2.3 M (600, 56 ms), 13 M (2000, 180 ms), 7 M (3000, 250 ms)
WORTH, WORTH_PER_PANEL = 1_000_000, 3000
GAUSS = {8: np.polynomial.legendre.leggauss(8)}
# thresholds of the samples' sums: Gauss-4 from 16 lengths, Gauss-2 from 1000,
# the run rule from 8 arclengths, cluster expansions from 4 radii
SAMPLE_RULE = dict(ratio4=16.0, ratio2=1000.0, ratio_run=8.0, cluster_kappa=4.0)

NODES = np.cos(np.pi * (np.arange(N) + 0.5) / N)
DCT = 2.0 / N * np.cos(np.outer(np.arange(N), np.pi * (np.arange(N) + 0.5) / N))
DCT[0] *= 0.5
MONO = np.zeros((N, N))
for _k in range(N):
    MONO[_k, : _k + 1] = np.polynomial.chebyshev.cheb2poly(np.eye(N)[_k])[: _k + 1]


def panel_nodes(profile, sigma, n):
    """[3, n_seg * n]: the n-point Gauss rule over each whole segment, as
    (rho_q, z_q, area_q * sigma_q), segment-major."""
    x, w = GAUSS[n] if n in GAUSS else np.polynomial.legendre.leggauss(n)
    t = 0.5 * (x + 1.0)
    p0, tan = profile[:-1], profile[1:] - profile[:-1]
    out = np.empty((3, len(p0), n))
    rho, z, dens = out
    np.add(np.multiply(tan[:, 0:1], t, out=rho), p0[:, 0:1], out=rho)
    np.add(np.multiply(tan[:, 1:2], t, out=z), p0[:, 1:2], out=z)
    np.add(np.multiply(sigma[1:, None] - sigma[:-1, None], t, out=dens), sigma[:-1, None], out=dens)
    area = 2.0 * np.pi * rho
    area *= np.sqrt((tan * tan).sum(axis=-1))[:, None] * 0.5 * w
    dens *= area
    return out.reshape(3, -1)


def link_tables(leaves, divided):
    """Lookup tables of a quadtree, one int32 array: a root table of the first
    MAP_ROOT_BITS levels (4^MAP_ROOT_BITS entries, j-major), then tables of
    MAP_BITS levels each.  leaves: (level, i, j, number) arrays; divided:
    {level: (i, j)} of the divided cells.  An entry: the cell's number, -1 for
    none, -2 - the number of the next table."""
    R, B = _lib.MAP_ROOT_BITS, _lib.MAP_BITS
    root = np.full((1 << R, 1 << R), -1, dtype=np.int32)
    ids, count = {}, 0
    for t in range(R, MAX_LEVEL + 1, B):
        if t not in divided or len(divided[t][0]) == 0:
            break
        key = (divided[t][0].astype(np.int64) << 32) | divided[t][1]
        order = np.argsort(key)
        ids[t] = (key[order], count + order)
        count += len(key)
    tab = np.full((count, 1 << B, 1 << B), -1, dtype=np.int32)
    low = (1 << B) - 1

    def table_of(t, i, j):
        key, num = ids[t]
        return num[np.searchsorted(key, (i.astype(np.int64) << 32) | j)]

    for t in ids:
        i, j = divided[t]
        if t == R:
            root[j, i] = -2 - table_of(t, i, j)
        else:
            tab[table_of(t - B, i >> B, j >> B), j & low, i & low] = -2 - table_of(t, i, j)
    lv, li, lj, num = leaves
    for level in np.unique(lv):
        m = lv == level
        i, j, n = li[m], lj[m], num[m]
        if level <= R:  # few: coarse cells far from the surface
            w = 1 << (R - level)
            for a, b, k in zip(i, j, n):
                root[b * w:(b + 1) * w, a * w:(a + 1) * w] = k
            continue
        t = R + (level - R - 1) // B * B
        up = level - t
        node = table_of(t, i >> up, j >> up)
        rest = B - up
        for dj in range(1 << rest):
            for di in range(1 << rest):
                tab[node, ((j << rest) + dj) & low, ((i << rest) + di) & low] = n
    return np.concatenate([root.reshape(-1), tab.reshape(-1)])


def worth(profile):
    """The number of points from which the cells of a profile pay."""
    return WORTH + WORTH_PER_PANEL * (len(profile) - 1)


def _lay_out(tables, scale, z_lo, tab, records):
    """(doubles tensor that starts with the cluster table, SptBem.reserved) of a
    map on its device.  Synchronises: it may be read on any stream afterwards."""
    import torch

    dev = tables.seg.device
    with torch.cuda.device(dev):
        base, unit = tables.clusters.reshape(-1), _lib.MAP_UNIT
        start = -(-base.numel() // unit) * unit
        rec_at = -(-(_lib.MAP_HEADER + tab.size // 2) // 8) * 8
        p8_at = rec_at + sum(r.numel() for r in records)
        head = np.zeros(rec_at)
        head[:4] = scale, z_lo, rec_at, p8_at
        head[_lib.MAP_HEADER: _lib.MAP_HEADER + tab.size // 2] = tab.view(np.float64)
        p8 = panel_nodes(tables.profile, tables.sigma, 8).ravel()
        small = torch.as_tensor(np.concatenate([np.zeros(start - base.numel()), head, p8]), device=dev)
        gap = start - base.numel() + rec_at
        out = torch.cat([base, small[:gap], *(r.reshape(-1) for r in records), small[gap:]])
        torch.cuda.current_stream(dev).synchronize()
    return out, (_lib.MAP_TAG << 16) | (start // unit)


def bare(tables):
    """The map without cells: a root square of no extent, which holds no point,
    and the panel nodes."""
    return _lay_out(tables, np.inf, 0.0, np.zeros(0, dtype=np.int32), [])


def build(tables):
    """The map of a BemTables with its cells, or None when there is nothing to map."""
    import torch

    dev = tables.seg.device
    lib = _lib.lib()
    view = tables.view("adaptive", field_map=False, **SAMPLE_RULE)
    prof = tables.profile
    zc = 0.5 * (prof[:, 1].min() + prof[:, 1].max())
    half = REACH * float(np.hypot(prof[:, 0], prof[:, 1] - zc).max())
    side, z_lo = 2.0 * half, zc - half
    t64 = lambda a: torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64), device=dev)
    cheb, dct, mono = t64(NODES), t64(DCT), t64(MONO)
    with torch.cuda.device(dev):
        stream = ctypes.c_void_p(torch.cuda.current_stream(dev).cuda_stream)
        i, j = np.zeros(1, dtype=np.int64), np.zeros(1, dtype=np.int64)
        kept, records, divided, n_kept = [], [], {}, 0
        for level in range(MAX_LEVEL + 1):
            h = half / (1 << level)
            cells = t64(np.stack([(2 * i + 1) * h, z_lo + (2 * j + 1) * h, np.full(len(i), h)], 1))
            flag = torch.empty(len(i), dtype=torch.int32, device=dev)
            ratio = torch.empty(len(i), dtype=torch.float64, device=dev)
            _lib.check(lib.spt_map_classify(cells.data_ptr(), len(i), ctypes.byref(view), KAPPA, flag.data_ptr(),
                                            ratio.data_ptr(), stream), "spt_map_classify")
            flag_h, ratio_h = flag.cpu().numpy(), ratio.cpu().numpy()
            split = flag_h == 0
            tried = np.nonzero(flag_h == 1)[0]
            if len(tried):
                sample = cells[torch.as_tensor(tried, device=dev)].contiguous()
                rec = torch.empty((len(tried), _lib.MAP_REC), dtype=torch.float64, device=dev)
                tail = torch.empty(len(tried), dtype=torch.float64, device=dev)
                _lib.check(lib.spt_map_cells(sample.data_ptr(), len(tried), ctypes.byref(view), cheb.data_ptr(),
                                             dct.data_ptr(), mono.data_ptr(), rec.data_ptr(), tail.data_ptr(), stream),
                           "spt_map_cells")
                ok = (tail.cpu().numpy() <= TAIL) | (ratio_h[tried] >= KAPPA_SURE)
                split[tried[~ok]] = True
                take = np.nonzero(ok)[0][: MAX_CELLS - n_kept]
                if len(take):
                    at = tried[take]
                    kept.append((np.full(len(take), level), i[at], j[at], n_kept + np.arange(len(take))))
                    records.append(rec[torch.as_tensor(take, device=dev)])
                    n_kept += len(take)
            i, j = i[split], j[split]
            if len(i) == 0 or n_kept >= MAX_CELLS or level == MAX_LEVEL:
                break
            divided[level] = (i, j)
            i, j = (np.concatenate([2 * i + a for a in (0, 1) for _ in (0, 1)]),
                    np.concatenate([2 * j + b for _ in (0, 1) for b in (0, 1)]))
        if not kept or 0 not in divided:
            return None
        tab = link_tables(tuple(np.concatenate(c) for c in zip(*kept)), divided)
    return _lay_out(tables, 1.0 / side, z_lo, tab, records)
