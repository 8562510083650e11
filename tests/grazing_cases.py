"""Scenes in which the order of visits decides a closest hit.

A box's entry distance is accurate to a few ulps.  A triangle's distance is off
by its conditioning, without bound for a ray along its plane, so a grazed
triangle's computed distance can lie well before the box it is in.  With another
hit between the two, the traversal that meets the other one first prunes the box,
and the one that meets the grazed triangle first keeps it.

Each cell holds one ray, such a triangle, another one across the ray halfway
between the grazed one's distance and its box, and clutter that the ray misses
but whose boxes it enters, which spreads both over nodes of different depth and
order.  Distances are computed in the traversal's single-precision operation
order."""
import numpy as np

from renderingengine_b200 import scenes

F = np.float32
GAP = 2.0 ** -10  # least gap of a cell, of the distance


def _dot(a, b):
    return (a[..., 0] * b[..., 0] + a[..., 1] * b[..., 1]) + a[..., 2] * b[..., 2]


def _cross(a, b):
    return np.stack([a[..., 1] * b[..., 2] - a[..., 2] * b[..., 1], a[..., 2] * b[..., 0] - a[..., 0] * b[..., 2],
                     a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0]], -1)


def triangle_distance(o, d, v):
    """Moller-Trumbore as the traversal computes it: (hit, t)."""
    e1, e2 = v[..., 1, :] - v[..., 0, :], v[..., 2, :] - v[..., 0, :]
    with np.errstate(all="ignore"):
        p = _cross(d, e2)
        det = _dot(e1, p)
        inv = F(1) / det
        s = o - v[..., 0, :]
        u = _dot(s, p) * inv
        q = _cross(s, e1)
        w = _dot(d, q) * inv
        t = _dot(e2, q) * inv
        hit = (det != 0) & np.isfinite(det) & (u >= 0) & (u <= 1) & (w >= 0) & (u + w <= 1) & np.isfinite(t)
    return hit, t


def box_distance(o, d, v):
    """Slab test of the triangle's own box: (entered, near)."""
    lo, hi = v.min(-2), v.max(-2)
    inv = F(1) / d
    back = np.signbit(inv)
    near = ((np.where(back, hi, lo) - o) * inv).max(-1)
    far = ((np.where(back, lo, hi) - o) * inv).min(-1)
    return (far >= near) & (far > 0), near


def _regular(v):
    """The degenerate rule of scene creation."""
    e1, e2 = v[..., 1, :] - v[..., 0, :], v[..., 2, :] - v[..., 0, :]
    c = _cross(e1, e2)
    scale = np.maximum(_dot(e1, e1), _dot(e2, e2))
    return _dot(c, c) > scale * scale * F(1e-13)


def unit(v):
    """normalize3 of the ray generation, single precision."""
    return v / np.sqrt(_dot(v, v))[..., None]


def _across(rng, centre, d, size):
    """A triangle around `centre`, perpendicular to d."""
    a = np.cross(d, rng.normal(size=d.shape))
    a /= np.linalg.norm(a, axis=-1, keepdims=True)
    b = np.cross(d, a)
    ang = np.array([0.3, 2.4, 4.5])
    return (centre[..., None, :] + size[..., None, None] * (np.cos(ang)[:, None] * a[..., None, :]
                                                             + np.sin(ang)[:, None] * b[..., None, :])).astype(F)


def cells(seed, side, clutter):
    """side^3 cells two units apart: (positions (n, 3, 3), origins, forwards,
    directions), direction = unit(forward)."""
    rng = np.random.default_rng(seed)
    count = side ** 3
    home = 2.0 * (np.stack(np.unravel_index(np.arange(count), (side,) * 3), -1) - (side - 1) / 2)
    out = [None] * count
    while any(c is None for c in out):
        n = 20_000
        at = rng.integers(0, count, n)
        o = (home[at] + rng.uniform(-0.1, 0.1, (n, 3))).astype(F)
        forward = unit(rng.normal(size=(n, 3)).astype(F))
        d = unit(forward)
        d64 = d.astype(np.float64)
        w = np.cross(d64, rng.normal(size=(n, 3)))
        w /= np.linalg.norm(w, axis=1, keepdims=True)
        along = d64 + np.cross(d64, w) * (10.0 ** rng.uniform(-6, -3, n) * rng.choice([-1, 1], n))[:, None]
        p = o + d64 * rng.uniform(0.2, 0.6, n)[:, None]
        ab = rng.normal(size=(n, 3, 2))
        ab -= ab.mean(1, keepdims=True) + rng.uniform(-0.3, 0.3, (n, 1, 2))
        size = 10.0 ** rng.uniform(-2, -1, n)
        v = (p[:, None] + size[:, None, None] * (ab[:, :, :1] * along[:, None] + ab[:, :, 1:] * w[:, None])).astype(F)
        hit, t = triangle_distance(o, d, v)
        entered, near = box_distance(o, d, v)
        late = hit & entered & _regular(v) & (t > 0.05) & (t < 0.7) & (near > t * F(1 + GAP)) & (near < t * F(1.2))
        for i in np.flatnonzero(late):
            if out[at[i]] is not None:
                continue
            between, gap = (float(t[i]) + float(near[i])) / 2, float(near[i]) - float(t[i])
            rival = _across(rng, o[i] + d64[i] * between, d64[i], np.array(gap * 0.1))
            ok, tr = triangle_distance(o[i], d[i], rival)
            _, near_r = box_distance(o[i], d[i], rival)
            if not (ok and t[i] < tr < near[i] and near_r <= tr and _regular(rival)):
                continue
            # Beside the ray, most before the grazed triangle, none hit.
            m = 4 * clutter
            size = 10.0 ** rng.uniform(-2.5, -1, m)
            foot = o[i] + d64[i] * (between * rng.uniform(0.5, 1.05, m))[:, None]
            side_step = np.cross(d64[i], rng.normal(size=(m, 3)))
            side_step /= np.linalg.norm(side_step, axis=1, keepdims=True)
            mess = (foot[:, None] + side_step[:, None] * (size * 0.6)[:, None, None]
                    + size[:, None, None] * rng.normal(size=(m, 3, 3)) * 0.5).astype(F)
            missed = ~triangle_distance(o[i][None], d[i][None], mess)[0] & _regular(mess)
            out[at[i]] = (np.concatenate([v[i][None], rival[None], mess[missed][:clutter]]), o[i], forward[i], d[i])
    return (np.concatenate([c[0] for c in out]), np.stack([c[1] for c in out]), np.stack([c[2] for c in out]),
            np.stack([c[3] for c in out]))


def scene(seed, side, clutter):
    """(SceneData of double-sided triangles, origins, forwards, directions)."""
    pos, o, forward, d = cells(seed, side, clutter)
    order = np.random.default_rng(seed + 1).permutation(len(pos))
    data = scenes.triangle_soup(len(pos), seed=seed)
    data.triangles = scenes.canonical_triangles(pos[order], None, np.zeros(len(pos), np.uint32),
                                                np.arange(len(pos), dtype=np.uint32), np.zeros(len(pos), np.uint32))
    return data, o, forward, d
