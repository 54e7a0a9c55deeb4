"""The P2P work plan (fmm/p2p_plan.py) on the CPU: the tasks, entries, slots
and chunks, walked as the kernels walk them, cover every listed triangle pair
exactly once, symmetric and one-sided, whole and as row shards."""
import numpy as np
import pytest

from tectosaur_b200.fmm.p2p_plan import build
from tectosaur_b200.fmm.tree import Tree, interactions, tri_centers_radii

from helpers import bumpy_mesh


def _pairs(lst, obs, src):
    out = set()
    for i, o in enumerate(lst.obs_n_idxs):
        for s in lst.src_n_idxs[lst.obs_src_starts[i]:lst.obs_src_starts[i + 1]]:
            out |= {(a, b) for a in range(obs.start[o], obs.end[o])
                    for b in range(src.start[s], src.end[s])}
    return out


def _walk(plan):
    """{(obs, src): times} as the kernels and the reduction add them up."""
    tasks, entries, chunks = (np.asarray(a) for a in (plan.tasks, plan.entries, plan.chunks))
    slots_in = np.asarray(plan.slots_in)
    got = {}
    task_w, slot_v = [], {}
    for o0, cnt, e0, e1 in tasks:
        assert 0 < cnt <= plan.chunk and 0 < e1 - e0 <= 128
        w = []
        for s0, n, v in entries[e0:e1]:
            w += [(o, s) for o in range(o0, o0 + cnt) for s in range(s0, s0 + n)]
            for k in range(n if v >= 0 else 0):
                assert v + k < plan.n_slots and v + k not in slot_v
                slot_v[v + k] = [(s0 + k, o) for o in range(o0, o0 + cnt)]
        task_w.append(w)
    assert len(slot_v) == plan.n_slots
    for o0, cnt, t0, t1, v0, v1, off in chunks:
        add = [p for t in range(t0, t1) for p in task_w[t]]
        for v in slots_in[v0:v1]:
            for e in range(cnt):
                vs = slot_v[v + off + e]
                assert all(p[0] == o0 + e for p in vs)
                add += vs
        for p in add:
            assert o0 <= p[0] < o0 + cnt
            got[p] = got.get(p, 0) + 1
    return got


@pytest.mark.parametrize("leaf,chunk", [(3, 32), (40, 32), (100, 32), (100, 64), (10 ** 9, 64)])
@pytest.mark.parametrize("mode", ["fmm", "treecode", "two"])
def test_plan_covers_the_list(leaf, chunk, mode):
    pts, tris = bumpy_mesh(13, seed=3, amp=0.3)
    tree = Tree(*tri_centers_radii(pts, tris), leaf, device=False)
    src = tree
    if mode == "two":
        p2, t2 = bumpy_mesh(9, seed=4)
        src = Tree(*tri_centers_radii(p2 + 0.3, t2), leaf, device=False)
    inner = 1.0 if mode == "treecode" else 2.0
    lst = interactions(tree, src, inner, 2.0, 0, mode == "treecode")["p2p"]
    want = _pairs(lst, tree, src)
    sym = build(tree, src, lst, chunk, True, 36, dev="cpu")
    assert sym.sym == (mode == "fmm") or mode == "treecode"
    one = build(tree, src, lst, chunk, False, 36, dev="cpu")
    assert not one.sym and one.n_slots == 0
    for plan in (sym, one):
        got = _walk(plan)
        assert set(got) == want and max(got.values(), default=1) == 1


@pytest.mark.parametrize("want_sym", [True, False])
def test_shard_plans_keep_the_rows(want_sym):
    """A shard's chunks hold the whole plan's terms, task by task."""
    pts, tris = bumpy_mesh(16, seed=5, amp=0.3)
    tree = Tree(*tri_centers_radii(pts, tris), 12, device=False)
    lst = interactions(tree, tree, 2.0, 2.0, 0, False)["p2p"]
    whole = _walk(build(tree, tree, lst, 32, want_sym, 36, dev="cpu"))
    rng = np.random.default_rng(0)
    keep = rng.random(tree.n_nodes) < 0.4
    plan = build(tree, tree, lst, 32, want_sym, 36, keep=keep, dev="cpu")
    got = _walk(plan)
    kept = {t for n in tree.leaves() if keep[n] for t in range(tree.start[n], tree.end[n])}
    assert got == {p: c for p, c in whole.items() if p[0] in kept}


def test_too_many_slots_falls_back():
    pts, tris = bumpy_mesh(10, seed=6)
    tree = Tree(*tri_centers_radii(pts, tris), 8, device=False)
    lst = interactions(tree, tree, 2.0, 2.0, 0, False)["p2p"]
    assert build(tree, tree, lst, 32, True, 36, dev="cpu").sym
    assert not build(tree, tree, lst, 32, True, 1 << 40, dev="cpu").sym
