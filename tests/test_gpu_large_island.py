"""One island of 48 bodies, more than a warp of them: the first search's pairs against a restatement of the search in numpy, in
float32 and the reference's order of operations (World::rebuild_pairs, fast_pairs, near_pairs, world.cpp:1851-2598) - every
node against every triangle, without the reference's hash and grids, so the pairs are compared as a set. Slow and fast
bodies, one-sided and two-sided skins; the slowest bodies' margins depend on the top speed of every slow body."""
import numpy as np
import pytest

from beamlab_b200 import rigs, world_from_rig

pytestmark = pytest.mark.gpu

f32 = np.float32
DIMS, INTERVAL, DT, CRAD, HULL_DEPTH = (3, 2, 2), f32(17.0), f32(0.0005), f32(0.05), f32(0.3)


def large_island(seed, n=48):
    """n lattices of 12 nodes in rows of 8, their faces 0.04 to 0.2 m apart; every fifth faster than 8 m/s."""
    rng, gen = rigs.TRng(seed), np.random.default_rng(seed)
    bodies = []
    for k in range(n):
        speed = float(gen.uniform(9.0, 14.0) if k % 5 == 2 else gen.uniform(0.5, 7.5))
        origin = (0.62 * (k % 8) + float(gen.uniform(0.0, 0.08)), 2.0 + 0.4 * (k // 24), 0.38 * ((k // 8) % 3) + float(gen.uniform(0.0, 0.05)))
        body = rigs.lattice_body(rng, dims=DIMS, origin=origin, velocity=tuple(speed * d for d in (0.8, 0.0, 0.6 * (-1.0) ** k)))
        body["tris"] = rigs.lattice_tris(DIMS)
        body["tri_two_sided"] = np.full(len(body["tris"]), k % 3 != 0, np.uint8)
        bodies.append(body)
    return {"settings": {"gravity": (0.0, -9.81, 0.0), "dt": 0.0005, "sleeping": False},
            "statics": {"terrain": rigs.flat_terrain(), "boxes": [], "build_grid": True}, "bodies": bodies}


def dot(a, b):
    return a[..., 0] * b[..., 0] + a[..., 1] * b[..., 1] + a[..., 2] * b[..., 2]


def cross(a, b):
    return np.stack([a[..., 1] * b[..., 2] - a[..., 2] * b[..., 1], a[..., 2] * b[..., 0] - a[..., 0] * b[..., 2],
                     a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0]], -1)


def closest(p, a, b, c):
    """closest_on_triangle (softbody.h:158-190)"""
    ab, ac, ap, bp, cp = b - a, c - a, p - a, p - b, p - c
    d1, d2, d3, d4, d5, d6 = dot(ab, ap), dot(ac, ap), dot(ab, bp), dot(ac, bp), dot(ab, cp), dot(ac, cp)
    va, vb, vc = d3 * d6 - d5 * d4, d5 * d2 - d1 * d6, d1 * d4 - d3 * d2
    with np.errstate(divide="ignore", invalid="ignore"):
        e_ab, e_ac, e_bc = d1 / (d1 - d3), d2 / (d2 - d6), (d4 - d3) / ((d4 - d3) + (d5 - d6))
        den = f32(1.0) / (va + vb + vc)
        inside = a + ab * (vb * den)[..., None] + ac * (vc * den)[..., None]
        cases = [((d1 <= 0) & (d2 <= 0), a + 0 * p), ((d3 >= 0) & (d4 <= d3), b + 0 * p), ((vc <= 0) & (d1 >= 0) & (d3 <= 0), a + ab * e_ab[..., None]),
                 ((d6 >= 0) & (d5 <= d6), c + 0 * p), ((vb <= 0) & (d2 >= 0) & (d6 <= 0), a + ac * e_ac[..., None]),
                 ((va <= 0) & (d4 - d3 >= 0) & (d5 - d6 >= 0), b + (c - b) * e_bc[..., None])]
    return np.select([m[..., None] & np.ones(3, bool) for m, _ in cases], [v for _, v in cases], inside)


def boxes_hit(amn, amx, bmn, bmx):
    return np.all((amn <= bmx) & (amx >= bmn), -1)


def expected_pairs(rig, nodes):
    B = len(rig["bodies"])
    nb = np.repeat(np.arange(B), [len(x["p"]) for x in nodes])
    first = np.concatenate([[0], np.cumsum([len(x["p"]) for x in nodes])])
    P, V, M = (np.concatenate([np.ascontiguousarray(x[k]) for x in nodes]).astype(f32) for k in ("p", "v", "mass"))
    T = np.concatenate([b["tris"].astype(np.int64) + first[k] for k, b in enumerate(rig["bodies"])])
    tb = np.repeat(np.arange(B), [len(b["tris"]) for b in rig["bodies"]])
    two = np.concatenate([b["tri_two_sided"] for b in rig["bodies"]]).astype(bool)
    of = [slice(first[k], first[k + 1]) for k in range(B)]
    hull = np.array([not b["tri_two_sided"].all() for b in rig["bodies"]])
    # the set-up (world.cpp:1870-1954)
    sp = np.sqrt(np.array([dot(V[s], V[s]).max() for s in of], f32))
    fast = sp > f32(8.0)
    speed = sp[~fast].max() + f32(0.5)
    margin = f32(2.0) * speed * INTERVAL * DT + f32(0.02)
    slow_reach = f32(2.0) * speed * INTERVAL * DT + f32(0.01)
    travel, Tn = f32(1.25) * INTERVAL * DT, INTERVAL * DT
    rms = np.array([f32(np.sqrt((M[s].astype(np.float64) * dot(V[s], V[s])).sum() / M[s].astype(np.float64).sum())) for s in of], f32)
    extra = np.where(fast, np.clip(f32(1.25) * rms, f32(8.0), f32(400.0)) * INTERVAL * DT, f32(0.0)).astype(f32)
    mn, mx = np.array([P[s].min(0) for s in of]), np.array([P[s].max(0) for s in of])
    grow = (CRAD + margin + extra + np.where(hull, HULL_DEPTH, f32(0.0)))[:, None].astype(f32)
    gmn, gmx = mn - grow, mx + grow
    partner = boxes_hit(gmn[:, None], gmx[:, None], gmn[None], gmx[None]) & ~np.eye(B, dtype=bool)
    # every triangle (rows) against every node (columns)
    a, b, c = (P[T[:, q]][:, None] for q in range(3))
    va, vb, vc = (V[T[:, q]][:, None] for q in range(3))
    p, v = P[None], V[None]
    tmn, tmx = np.minimum(a, np.minimum(b, c)), np.maximum(a, np.maximum(b, c))
    tn = cross(b - a, c - a)
    tu = tn * (f32(1.0) / np.sqrt(dot(tn, tn)))[..., None]
    depth, ts = np.where(two, f32(0.0), HULL_DEPTH).astype(f32)[:, None], two[:, None]

    def near_triangle(r):
        s = dot(p - a, tu)
        q = p - tu * s[..., None]
        d2, dq = closest(p, a, b, c) - p, closest(q, a, b, c) - q
        return np.where(ts, (np.abs(s) <= r) & (dot(d2, d2) <= r * r), (s <= r) & (s >= -r - depth) & (dot(dq, dq) <= r * r))

    def in_box(r):
        r = np.broadcast_to(r, (len(T), len(P)))[..., None]
        return np.all((p >= tmn - r) & (p <= tmx + r), -1)

    # near_pairs' filter (world.cpp:2536-2583)
    da, db, dc = v - va, v - vb, v - vc
    reach = (CRAD + depth) + f32(1.25) * np.sqrt(np.maximum(dot(da, da), np.maximum(dot(db, db), dot(dc, dc)))) * Tn + f32(0.02)
    d = p - closest(p, a, b, c)
    keep = dot(d, d) < reach * reach
    n0 = tn / np.sqrt(dot(tn, tn))[..., None]
    s0 = dot(n0, p - a)
    sg = np.where(s0 >= 0, f32(1.0), f32(-1.0))
    close = np.maximum(f32(0.0), np.maximum(-sg * dot(n0, da), np.maximum(-sg * dot(n0, db), -sg * dot(n0, dc))))
    keep &= ~((ts | (s0 > CRAD)) & (np.abs(s0) - f32(1.25) * close * Tn - f32(0.02) >= CRAD))
    other = tb[:, None] != nb[None]
    # the slow bodies' nodes near a partner's box against the triangles near a partner's box (world.cpp:1966-2083)
    near_node = np.array([(partner[nb[i]] & boxes_hit(gmn, gmx, P[i], P[i])).any() for i in range(len(P))]) & ~fast[nb]
    rq = (CRAD + margin + extra[tb] + depth[:, 0])[:, None]
    near_tri = np.array([(partner[tb[t]] & boxes_hit(gmn, gmx, tmn[t, 0] - rq[t], tmx[t, 0] + rq[t])).any() for t in range(len(T))])
    r = (CRAD + margin + extra[tb])[:, None]
    slow = other & near_node[None] & near_tri[:, None] & in_box(r + depth) & near_triangle(r)
    # the fast bodies' nodes against their partners' triangles (world.cpp:2330-2475)
    o_fast = fast[tb]
    rt = np.where(o_fast, (CRAD + f32(0.01)) + travel * np.sqrt(np.maximum(dot(va, va), np.maximum(dot(vb, vb), dot(vc, vc)))[:, 0]), CRAD + slow_reach).astype(f32)
    body_r = CRAD + slow_reach + travel * (sp[None, :] + np.where(o_fast, sp[tb], f32(0.0))[:, None]) + np.where(o_fast, extra[tb], f32(0.0))[:, None]
    in_reach = np.all((tmx >= mn[None] - body_r[..., None]) & (tmn <= mx[None] + body_r[..., None]), -1)  # (triangle, body)
    rn = rt[:, None] + np.sqrt(dot(v, v)) * travel
    quick = other & fast[nb][None] & partner[tb[:, None], nb[None]] & in_reach[:, nb] & in_box(rn + depth) & near_triangle(rn)
    t, i = np.nonzero((slow | quick) & keep)
    tri_first = np.concatenate([[0], np.cumsum([len(b["tris"]) for b in rig["bodies"]])])
    assert slow[t, i].any() and quick[t, i].any() and not (slow & quick).any()
    return {(int(nb[y]), int(y - first[nb[y]]), int(tb[x]), int(x - tri_first[tb[x]])) for x, y in zip(t, i)}


@pytest.mark.parametrize("seed", (1, 2))
def test_island_of_48_bodies_finds_the_pairs(seed):
    rig = large_island(seed)
    w = world_from_rig(rig)
    want = expected_pairs(rig, [h.nodes() for h in w.bodies()])
    w.step_substeps(1)
    got = [tuple(int(x) for x in row) for row in w.pairs()]
    assert len(set(got)) == len(got) and set(got) == want
    st = w.stats()
    assert st["pair_searches"] == 1 and st["device_errors"] == 0  # (one island)
    w.close()
    # its contacts whole and 448 at a time, searches in every frame: the same states bit for bit
    a, b = world_from_rig(rig), world_from_rig(rig, contact_whole_max=0)
    for _ in range(4):
        a.step_substeps(33)
        b.step_substeps(33)
        assert np.array_equal(a.pairs(), b.pairs())
        for x, y in zip(a.bodies(), b.bodies()):
            x, y = x.nodes(), y.nodes()
            assert np.array_equal(x["p"].view(np.uint32), y["p"].view(np.uint32)) and np.array_equal(x["v"].view(np.uint32), y["v"].view(np.uint32))
    assert a.stats()["contacts"] == b.stats()["contacts"] > 0 and a.stats()["device_errors"] == 0
    a.close()
    b.close()
