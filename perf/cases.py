"""The work that users have this framework do, as cases to measure.

Every case goes through the public entry points: ``Interpolator`` with its
device-resident and host calls, and ``autograd.interpolate``.  A case is a
dict of plain values; ``prepare`` makes what a program holds before the call
(a resident mesh, queries, values), ``run`` is one pass.

Kinds of case:

  interp   ``Interpolator.interpolate_device``: values at device queries
  host     ``Interpolator.interpolate``: numpy arrays in and out
  csr      ``Interpolator.get_weights_device``: the weights as a device CSR, kept
           in buffers of the caller's
  train    ``autograd.interpolate`` forward, then backward into queries and values
  fresh    a key set used once: ``Interpolator(keys, constructor='gpu')``, then
           one interpolation

Queries are float32 or float64 (``q``), values too (``v``); ``d`` is the
number of value columns, 0 for a plain vector of values.  ``cloud`` is how
the keys lie: 'uniform' in the unit cube, or 'clusters' (a Gaussian mixture,
whose density varies by orders of magnitude).  ``order`` is how the queries
come: 'random', or 'raster' (the points of a regular grid in raster order,
as when scattered samples are resampled onto voxels).
"""
import math

import numpy as np
import torch

import natinterp3d_b200 as ni
from natinterp3d_b200.autograd import interpolate as interpolate_with_gradients

_DTYPES = {32: torch.float32, 64: torch.float64}


def _case(name, kind, keys, queries, d=0, q=64, v=64, cloud='uniform', order='random',
          predicates='fast'):
    c = {'kind': kind, 'keys': keys, 'queries': queries, 'd': d, 'q': q, 'v': v, 'cloud': cloud,
         'order': order, 'predicates': predicates}
    if name:
        c['name'] = name
    return c


def listed():
    return [
        # a probe inside an interactive loop: the smallest call, all latency
        _case('probe_64', 'interp', 20_000, 64),
        # one frame of a particle or mesh simulation that samples a float32 field
        _case('frame_f32', 'interp', 50_000, 5_003, d=3, q=32, v=32),
        # the small configuration of the parity tests: a scalar at 100k points
        _case('scalar_100k', 'interp', 10_000, 100_000),
        # scattered samples resampled onto a voxel grid, float32 throughout
        _case('raster_f32', 'interp', 200_000, 96 * 101 * 103, d=1, q=32, v=32, order='raster'),
        # the benchmark's plain workload: the largest call
        _case('plain_10m', 'interp', 1_000_000, 10_000_000, d=3, q=64, v=32),
        # wide feature vectors carried by the keys
        _case('features_64', 'interp', 20_000, 30_001, d=64, q=32, v=32),
        # clustered keys with exact predicates: the safe setting for uneven data
        _case('clusters_exact', 'interp', 100_000, 300_007, d=1, cloud='clusters',
              predicates='exact'),
        # the weights themselves, reused for many value sets afterwards
        _case('csr_1m', 'csr', 200_000, 1_000_000),
        # the benchmark's differentiable workload: one training step
        _case('train_1m', 'train', 200_000, 1_000_000, d=16, q=64, v=32),
        # a training step on a small batch of query points
        _case('train_10k', 'train', 10_000, 10_007, d=4),
        # numpy in, numpy out
        _case('host_500k', 'host', 100_000, 500_000, d=2),
        # keys that move from frame to frame: the mesh is built, then used once
        _case('fresh_20k', 'fresh', 20_000, 25_000, d=1),
    ]


def _log(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, n | 1 if rng.random() < 0.7 else n))


def draw(rng):
    """One more case of the listed ones' ranges."""
    kind = rng.choice(['interp', 'interp', 'interp', 'interp', 'csr', 'csr', 'train', 'train', 'host',
                       'fresh'])
    if kind == 'fresh':
        return _case(None, kind, _log(rng, 2_000, 30_000), _log(rng, 1_000, 100_000),
                     d=rng.randint(0, 3))
    q, v = rng.choice([(64, 64), (64, 32), (32, 32), (32, 64)])
    if kind == 'host':
        return _case(None, kind, _log(rng, 5_000, 200_000), _log(rng, 1_000, 1_000_000),
                     d=rng.randint(0, 4), q=q, v=v)
    if kind == 'csr':
        return _case(None, kind, _log(rng, 5_000, 400_000), _log(rng, 64, 1_500_000), q=q, v=v,
                     cloud=rng.choice(['uniform', 'uniform', 'clusters']))
    if kind == 'train':
        return _case(None, kind, _log(rng, 5_000, 300_000), _log(rng, 1_000, 1_000_000),
                     d=rng.choice([0, 1, 3, 4, 8, 16, 32]), q=q, v=v)
    order = rng.choice(['random', 'random', 'raster'])
    if rng.random() < 0.2:
        return _case(None, kind, _log(rng, 10_000, 100_000), _log(rng, 1_000, 200_000),
                     d=_log(rng, 5, 64), q=q, v=v, order=order)
    return _case(None, kind, _log(rng, 5_000, 1_000_000), _log(rng, 64, 5_000_000),
                 d=rng.randint(0, 4), q=q, v=v, order=order,
                 cloud=rng.choice(['uniform', 'uniform', 'clusters']),
                 predicates=rng.choice(['fast', 'fast', 'fast', 'exact']))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _device():
    return torch.device('cuda', torch.cuda.current_device())


def _margin(case):
    """Distance from the cube's faces that queries of a uniform cloud keep: a few key spacings,
    where interpolation is wanted and the convex hull's own effects are gone."""
    return min(0.25, 4.0 * case['keys'] ** (-1.0 / 3.0))


def _inputs(case, seed):
    """(keys numpy [N, 3] float64, queries [M, 3], values [N] or [N, d], cotangent [M] or [M, d]);
    tensors on the GPU."""
    N, M, d = case['keys'], case['queries'], case['d']
    rng = np.random.default_rng(seed)
    dev = _device()
    gen = torch.Generator(device=dev).manual_seed(seed)
    qt, vt = _DTYPES[case['q']], _DTYPES[case['v']]
    if case['cloud'] == 'clusters':
        k = 16
        centre = rng.uniform(0.2, 0.8, (k, 3))
        width = np.exp(rng.uniform(math.log(0.01), math.log(0.1), k))
        member = rng.integers(0, k, N)
        keys = centre[member] + width[member, None] * rng.standard_normal((N, 3))
        # queries beside keys, at the local spacing
        pick = torch.randint(0, N, (M,), generator=gen, device=dev)
        near = torch.from_numpy(keys).to(dev)[pick]
        w = torch.from_numpy(width).to(dev)[torch.from_numpy(member).to(dev)[pick]]
        step = torch.randn((M, 3), generator=gen, device=dev, dtype=torch.float64)
        queries = near + step * (0.5 * w * (N / k) ** (-1.0 / 3.0))[:, None]
    else:
        keys = rng.uniform(0.0, 1.0, (N, 3))
        m = _margin(case)
        if case['order'] == 'raster':
            nx = max(1, round(M ** (1.0 / 3.0)))
            ny = max(1, round((M / nx) ** 0.5))
            nz = -(-M // (nx * ny))
            at = torch.arange(M, device=dev)
            cell = torch.stack([at // (ny * nz), at // nz % ny, at % nz], 1).to(torch.float64)
            n = torch.tensor([nx, ny, nz], device=dev, dtype=torch.float64)
            shift = torch.rand((1, 3), generator=gen, device=dev, dtype=torch.float64)
            queries = m + (1.0 - 2.0 * m) * (cell + shift) / n
        else:
            queries = torch.rand((M, 3), generator=gen, device=dev, dtype=torch.float64)
            queries = m + (1.0 - 2.0 * m) * queries
    values = torch.randn((N, max(d, 1)), generator=gen, device=dev, dtype=torch.float64).to(vt)
    out_t = torch.float32 if qt == vt == torch.float32 else torch.float64
    cotangent = torch.randn((M, max(d, 1)), generator=gen, device=dev, dtype=torch.float64).to(out_t)
    if d == 0:
        values, cotangent = values[:, 0].contiguous(), cotangent[:, 0].contiguous()
    return keys, queries.to(qt).contiguous(), values, cotangent


def _mesh(keys, predicates):
    """An interpolator over the keys' mesh as a saved mesh file gives it: built once on the GPU,
    then its tets put in a fixed order, so that every process holds the same mesh."""
    built = ni.Interpolator(keys, constructor='gpu')
    if built.construction['constructor'] != 'gpu':
        raise RuntimeError('the keys of this case are not in general position')
    vxyz, tv, tn = built.mesh_arrays
    dev = _device()
    p = torch.from_numpy(tv).to(dev).long()
    opp = torch.from_numpy(tn).to(dev).long().flip(1)  # neighbour opposite p[i]
    # the even permutation of each tet that puts its two lowest vertices first
    by = p.argsort(1)
    odd = torch.zeros(len(p), dtype=torch.bool, device=dev)
    for i in range(4):
        for j in range(i + 1, 4):
            odd ^= by[:, i] > by[:, j]
    by[:, 2:] = torch.where(odd[:, None], by[:, 2:].flip(1), by[:, 2:])
    p, opp = p.gather(1, by), opp.gather(1, by)
    # tets in a fixed pseudo-random order (by a hash of their vertices): tets that are near in
    # space are not near in memory, as in a mesh built by inserting keys one by one
    n = len(vxyz)
    code = (p[:, 0] * n + p[:, 1]) * 1_000_003 + p[:, 2] * 7_919 + p[:, 3]
    order = (code * 0x2545F4914F6CDD1D).argsort()
    rank = torch.empty_like(order)
    rank[order] = torch.arange(len(order), device=dev)
    p, opp = p[order], opp[order]
    opp = torch.where(opp >= 0, rank[opp.clamp_min(0)], opp)
    out = ni.Interpolator.from_mesh(built.centroid, vxyz, p.int().cpu().numpy(),
                                    opp.flip(1).int().cpu().numpy(), predicates=predicates)
    out.device_mesh  # resident from here on
    return out


def prepare(case, seed):
    keys, queries, values, cotangent = _inputs(case, seed)
    state = {'case': case}
    if case['kind'] == 'fresh':
        state.update(keys=keys, queries=queries, values=values)
        return state
    state['interp'] = _mesh(keys, case['predicates'])
    if case['kind'] == 'host':
        state.update(queries=queries.cpu().numpy(), values=values.cpu().numpy())
    elif case['kind'] == 'train':
        state.update(queries=queries.requires_grad_(True), values=values.requires_grad_(True),
                     cotangent=cotangent)
    elif case['kind'] == 'csr':
        # the program's own buffers for the weights, with room for 24 a query
        room = 24 * len(queries) + 4096
        state.update(queries=queries,
                     cols=torch.zeros(room, dtype=torch.int32, device=queries.device),
                     vals=torch.zeros(room, dtype=queries.dtype, device=queries.device))
    else:
        state.update(queries=queries, values=values)
    return state


def run(state):
    kind = state['case']['kind']
    if kind == 'interp':
        return state['interp'].interpolate_device(state['queries'], state['values'])
    if kind == 'host':
        return state['interp'].interpolate(state['queries'], state['values'])
    if kind == 'csr':
        rowptr, cols, vals = state['interp'].get_weights_device(state['queries'])
        state['cols'][:len(cols)].copy_(cols)
        state['vals'][:len(vals)].copy_(vals)
        return {'rowptr': rowptr, 'cols': state['cols'], 'vals': state['vals']}
    if kind == 'train':
        q, v = state['queries'], state['values']
        out = interpolate_with_gradients(state['interp'], q, v)
        gq, gv = torch.autograd.grad(out, (q, v), state['cotangent'])
        return {'out': out, 'grad_queries': gq, 'grad_values': gv}
    interp = ni.Interpolator(state['keys'], constructor='gpu')
    return interp.interpolate_device(state['queries'], state['values'])


# ---------------------------------------------------------------------------
# the least work of one pass
# ---------------------------------------------------------------------------
TETS_PER_KEY = 6.75     # Delaunay tets of random points
NEIGHBOURS = 15.5       # natural neighbours of a random point
FACES = 2 * NEIGHBOURS - 4   # boundary faces of its cavity
CAVITY = 18.0           # tets of its cavity


def work(case):
    N, M, d = case['keys'], case['queries'], max(case['d'], 1)
    qs, vs = case['q'] // 8, case['v'] // 8
    os = 4 if qs == vs == 4 else 8
    # the mesh: vertices, tets and their neighbours, as far as the queries reach it
    reach = min(TETS_PER_KEY * N, M * (CAVITY + FACES))
    nbytes = 3 * qs * M + 32 * reach + 24 * min(N, reach)
    # per query: a sphere test of each cavity tet and of the tets around the cavity, a
    # circumcentre per boundary face and per directed boundary edge, a subcell volume per face
    # corner, a sum over the cavity's and the faces' terms
    flops = M * ((CAVITY + FACES) * 10 + FACES * (90 + 3 * (55 + 85)) + 4 * CAVITY + 3 * FACES)
    nnz = NEIGHBOURS * M
    if case['kind'] == 'csr':
        nbytes += nnz * (4 + qs) + 4 * M
    else:
        nbytes += N * d * vs + M * d * os
        flops += 2 * nnz * d
    if case['kind'] == 'train':
        nbytes += M * d * os + 3 * qs * M + N * d * vs
        flops += 4 * nnz * d + M * FACES * 3 * 300
    if case['kind'] == 'fresh':
        nbytes += 24 * N
        flops += N * ((CAVITY + FACES) * 80 + FACES * 20)
    return {'bytes': nbytes, 'flops': flops}


# ---------------------------------------------------------------------------
# the same results in plain 64-bit torch
# ---------------------------------------------------------------------------
def _combinations(n, k, dev):
    return torch.combinations(torch.arange(n, device=dev), k)


def _dot(a, b):
    return (a * b).sum(-1)


def _circumcentre3(a, b, c):
    u, v = b - a, c - a
    n = torch.linalg.cross(u, v)
    num = _dot(u, u)[..., None] * torch.linalg.cross(v, n) + \
        _dot(v, v)[..., None] * torch.linalg.cross(n, u)
    return a + num / (2.0 * _dot(n, n))[..., None]


def _circumcentre4(a, b, c, d):
    u, v, w = b - a, c - a, d - a
    vw = torch.linalg.cross(v, w)
    num = _dot(u, u)[..., None] * vw + _dot(v, v)[..., None] * torch.linalg.cross(w, u) + \
        _dot(w, w)[..., None] * torch.linalg.cross(u, v)
    return a + num / (2.0 * _dot(u, vw))[..., None]


def _corner_volumes(p):
    """p [..., 4, 3]: the signed volume, in the tet p, of the points nearest to each corner
    [..., 4], positive in sum for every tet: six flat-cornered pieces per corner (corner,
    edge midpoint, face circumcentre, tet circumcentre)."""
    centre = _circumcentre4(*(p[..., i, :] for i in range(4)))
    sign = torch.sign(_dot(p[..., 1, :] - p[..., 0, :],
                           torch.linalg.cross(p[..., 2, :] - p[..., 0, :], p[..., 3, :] - p[..., 0, :])))
    out = []
    for k in range(4):
        total = 0.0
        for i in range(4):
            for j in range(4):
                if len({i, j, k}) < 3:
                    continue
                rest = 6 - i - j - k
                # orientation of (edge k-i, face k-i-j, tet) against that of (0, 1, 2, 3)
                perm = [k, i, j, rest]
                flips = sum(perm[x] > perm[y] for x in range(4) for y in range(x + 1, 4))
                mid = 0.5 * (p[..., i, :] - p[..., k, :])
                face = _circumcentre3(p[..., k, :], p[..., i, :], p[..., j, :]) - p[..., k, :]
                piece = _dot(mid, torch.linalg.cross(face, centre - p[..., k, :])) / 6.0
                total = total + (-piece if flips % 2 else piece)
        out.append(total)
    return torch.stack(out, -1) * sign[..., None]


def _natural_neighbours(p):
    """p [B, K, 3], keys relative to their query: [B, F, 3] facets (indices, -1 where unused) of
    the cell around the query.  Under inversion at the query they are the facets of the points'
    convex hull."""
    B, K, _ = p.shape
    s = p / _dot(p, p)[..., None]
    tri = _combinations(K, 3, p.device)
    a, b, c = (s[:, tri[:, i]] for i in range(3))
    n = torch.linalg.cross(b - a, c - a)
    off = _dot(n, a)
    side = torch.bmm(n, s.transpose(1, 2)) - off[..., None]       # [B, T, K]
    for i in range(3):
        side.scatter_(2, tri[None, :, i, None].expand(B, -1, 1), 0.0)
    facet = ((side <= 0).all(2) & (off > 0)) | ((side >= 0).all(2) & (off < 0))
    count = facet.sum(1)
    F = int(count.max())
    at = torch.where(facet, torch.arange(len(tri), device=p.device)[None], len(tri))
    at = at.topk(F, 1, largest=False).values
    out = torch.cat([tri, tri.new_full((1, 3), -1)])[at]
    return out


def _cells(q, keys):
    """The cell of each query q [B, 3]: (keys' indices [B, 56], facets [B, F, 3] into them).  It
    starts from the nearest 56 keys; a further key that cuts the cell (one nearer to a corner of
    it than the query is) takes the place of one that does not touch it, until none is left."""
    far = torch.cdist(q, keys, compute_mode='donot_use_mm_for_euclid_dist')
    near = far.topk(min(400, len(keys)), 1, largest=False).indices
    rel = keys[near] - q[:, None]
    chosen = torch.arange(56, device=q.device).expand(len(q), -1).clone()   # places in near
    facets = _natural_neighbours(rel[:, :56])
    todo = torch.arange(len(q), device=q.device)
    for _ in range(8):
        f, r, c = facets[todo], rel[todo], chosen[todo]
        rows = torch.arange(len(todo), device=q.device)
        live = f[..., 0] >= 0
        corner = r[rows[:, None, None], c[rows[:, None, None], f.clamp_min(0)]]
        centre = _circumcentre4(torch.zeros_like(corner[..., 0, :]), *corner.unbind(2))
        slack = _dot(r, r)[:, None] - 2.0 * torch.bmm(centre, r.transpose(1, 2))
        slack.scatter_(2, c[rows[:, None, None], f.clamp_min(0)], 0.0)
        cuts = (torch.where(live[..., None], slack, 0.0) < 0).any(1)
        more = cuts.any(1)
        if not more.any():
            break
        todo, f, c, cuts = todo[more], f[more], c[more], cuts[more]
        rows = rows[:len(todo)]
        # neighbours so far first, then the keys that cut, then the nearest others
        rank = cuts.to(torch.int64)
        held = torch.zeros(len(todo), 57, dtype=torch.bool, device=q.device)
        held.scatter_(1, torch.where(f < 0, 56, f).flatten(1), True)
        rank.scatter_(1, c, torch.where(held[:, :56], 2, rank.gather(1, c)))
        c = rank.argsort(dim=1, descending=True, stable=True)[:, :56]
        chosen[todo] = c
        f = _natural_neighbours(rel[todo].gather(1, c[..., None].expand(-1, -1, 3)))
        F = max(f.shape[1], facets.shape[1])
        facets = torch.nn.functional.pad(facets, (0, 0, 0, F - facets.shape[1]), value=-1)
        facets[todo] = torch.nn.functional.pad(f, (0, 0, 0, F - f.shape[1]), value=-1)
    return near.gather(1, chosen), facets


def _weights(q, keys):
    """Natural-neighbour weights of queries q [B, 3] (float64, may need gradients) with respect
    to keys [N, 3]: (index [B, K], weight [B, K])."""
    with torch.no_grad():
        idx, facets = _cells(q.detach(), keys)
        # the neighbours first, the others' places unused
        used = torch.zeros(idx.shape[0], idx.shape[1] + 1, dtype=torch.bool, device=q.device)
        used.scatter_(1, torch.where(facets < 0, idx.shape[1], facets).flatten(1), True)
        used = used[:, :-1]
        n = int(used.sum(1).max())
        place = used.long().argsort(dim=1, descending=True, stable=True)
        inverse = place.argsort(1)
        idx = idx.gather(1, place)[:, :n]
        live = used.gather(1, place)[:, :n]
        B, F, _ = facets.shape
        facets = torch.where(facets < 0, -1, inverse.gather(1, facets.clamp_min(0).flatten(1)).view(B, F, 3))
        rel = keys[idx] - q[:, None]
        # the tets of the neighbours' own tetrahedralization whose spheres hold the query
        quad = _combinations(n, 4, q.device)
        centre = _circumcentre4(*(rel[:, quad[:, i]] for i in range(4)))    # [B, Q, 3]
        r2 = _dot(centre - rel[:, quad[:, 0]], centre - rel[:, quad[:, 0]])
        tet = live[:, quad].all(2) & (_dot(centre, centre) < r2)
        hit = tet.nonzero()
        cen, rad = centre[tet], r2[tet]
        gap = rel[hit[:, 0]] - cen[:, None]
        gap = _dot(gap, gap) - rad[:, None]
        gap.scatter_(1, quad[hit[:, 1]], 1.0)
        gap = torch.where(live[hit[:, 0]], gap, 1.0)
        hit = hit[(gap > 0).all(1)]
    p = keys[idx] - q[:, None]
    stolen = torch.zeros(p.shape[:2], dtype=torch.float64, device=q.device)
    row = hit[:, :1].expand(-1, 4)
    corner = quad[hit[:, 1]]
    stolen = stolen.index_put((row, corner), _corner_volumes(p[row, corner]), accumulate=True)
    # less what the tets of query and facet leave to the keys
    fb, ff = (facets[..., 0] >= 0).nonzero(as_tuple=True)
    tri = facets[fb, ff]
    corners = torch.cat([torch.zeros((len(fb), 1, 3), dtype=torch.float64, device=q.device),
                         p[fb[:, None], tri]], 1)
    left = _corner_volumes(corners)[:, 1:]
    stolen = stolen.index_put((fb[:, None].expand(-1, 3), tri), -left, accumulate=True)
    return idx, stolen / stolen.sum(1, keepdim=True)


def exact(case, seed):
    """run()'s outputs in plain float64 torch: each query's natural neighbours among its 400 nearest
    keys by brute force, then the definition of the weights.  Only where that takes seconds, and
    for evenly spread keys, whose neighbours are among those."""
    if case['cloud'] != 'uniform' or case['queries'] > 30_001 or case['kind'] == 'csr':
        return None
    keys, queries, values, cotangent = _inputs(case, seed)
    keys = torch.from_numpy(keys).to(queries.device)
    v = values.double().reshape(case['keys'], -1)
    g = cotangent.double().reshape(case['queries'], -1)
    grad = case['kind'] == 'train'
    out, gq, gv = [], [], torch.zeros_like(v)
    step = 64
    for a in range(0, case['queries'], step):
        q = queries[a:a + step].double().requires_grad_(grad)
        idx, w = _weights(q, keys)
        y = (w[..., None] * v[idx]).sum(1)
        out.append(y.detach())
        if grad:
            gq.append(torch.autograd.grad(y, q, g[a:a + step])[0])
            gv.index_add_(0, idx.flatten(), (w.detach()[..., None] * g[a:a + step, None]).flatten(0, 1))
    out = torch.cat(out).reshape((case['queries'],) + tuple(values.shape[1:]))
    if case['kind'] == 'host':
        out = out.cpu().numpy()
    if not grad:
        return out
    return {'out': out, 'grad_queries': torch.cat(gq), 'grad_values': gv.reshape(values.shape)}
