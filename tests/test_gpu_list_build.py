"""The Verlet-list build over its variants: one and four particles a warp, 16-
and 32-bit ids, boxes of fewer than five cells a side (minimum image), rows
longer than the build keeps in shared memory, bonded exclusions, partial last
chunks.  The list read back has to hold every pair within the list radius that
a brute-force search finds, none twice, no pair beyond it and no excluded one.
Distances within 2e-6 nm of the radius (FP32 coordinates of a box of at most
14 nm round at 1e-6 nm) may fall on either side."""
import numpy as np
import pytest

from quantom_b200 import engine as E
from quantom_b200 import systems as S

pytestmark = pytest.mark.gpu

# box, waters, chains, length, cutoff
CASES = [(2.7, 601, 0, 0, 1.2),        # two cells a side
         (3.0, 879, 0, 0, 1.2),        # four
         (3.3, 1100, 0, 0, 1.2),       # five: the smallest grid that is walked
         (4.0, 1901, 2, 23, 1.2),      # exclusions
         (4.4, 2600, 2, 24, 2.05),     # rows of 1,300 entries, minimum image
         (5.6, 5500, 3, 30, 2.05),     # rows of 1,300 entries in the grid
         (8.1, 16385, 4, 50, 1.0),     # four particles a warp, an odd count
         (8.1, 16385, 4, 50, 2.05),    # the same with long rows
         (13.0, 66003, 2, 64, 1.0)]    # 32-bit ids


@pytest.mark.parametrize("box,waters,chains,length,cutoff", CASES)
def test_list_is_the_brute_force_list(box, waters, chains, length, cutoff):
    import torch
    spec = S.SystemSpec("box", box, waters, cutoff=cutoff, chains=S.ChainSpec(chains, length) if chains else None,
                        mc_sweeps=4)
    s = S.make_system(spec, seed=11)
    skin = 0.05
    p = E.default_params(box_len=box, cutoff=cutoff, dt=spec.dt, semantics=E.SEMANTICS_PHYSICS, skin=skin,
                         switch_on=cutoff - 0.2, nlist_period=0)
    with E.Engine(s, p) as eng:
        off, ids = eng.nlist(E.NL_PAIR)
        fc, fs = eng.positions()
    n_of = s.compounds["n_particles"] if chains else []
    x = np.concatenate([fc[c, :k] for c, k in enumerate(n_of)] + [fs]).astype(np.float64)
    x -= np.floor(x / box) * box
    base = np.concatenate([[0], np.cumsum(n_of)]).astype(int)
    excl = {(base[c] + q, base[ig["compound_ids"][z]] + ig["local_ids"][z])
            for c, k in enumerate(n_of) for q in range(k) for ig in [s.compounds[c]["lj_ignore_list"][q]]
            for z in range(ig["n_ignores"])}
    n, r = len(x), cutoff + skin
    got = np.zeros((2, len(ids)), np.int64)
    got[0], got[1] = np.repeat(np.arange(n), np.diff(off)), ids
    keys = np.sort(got[0] * n + got[1])
    assert (np.diff(keys) > 0).all()
    assert not any(i * n + j in set(keys[np.searchsorted(keys, i * n):np.searchsorted(keys, (i + 1) * n)])
                   for i, j in excl)
    xt = torch.as_tensor(x, device="cuda")
    keys = torch.as_tensor(keys, device="cuda")
    ex = torch.as_tensor(sorted(int(i) * n + int(j) for i, j in excl), dtype=torch.int64, device="cuda")
    for lo in range(0, n, 512):
        d = xt[None, :, :] - xt[lo: lo + 512, None, :]
        d -= box * torch.round(d / box)
        dist = d.norm(dim=-1)
        rows = torch.arange(lo, min(n, lo + 512), device="cuda")
        dist[rows - lo, rows] = 1e9
        a, b = int(torch.searchsorted(keys, lo * n)), int(torch.searchsorted(keys, min(n, lo + 512) * n))
        mine = keys[a:b]
        assert (dist.reshape(-1)[mine - lo * n] < r + 2e-6).all()
        want = torch.nonzero(dist < r - 2e-6)
        want = (want[:, 0] + lo) * n + want[:, 1]
        want = want[~torch.isin(want, ex)]
        assert torch.isin(want, mine).all()


@pytest.mark.parametrize("box,waters", [(4.0, 1901), (8.1, 16385)])   # one and four particles a warp
@pytest.mark.parametrize("axis,value", [(0, np.nan), (1, np.nan), (2, np.nan), (0, np.inf)])
def test_particle_without_candidates(box, waters, axis, value):
    """A particle that is not finite on some axis has an empty candidate stream:
    its row is empty, the others' rows are those of the box without it, the next
    step reports it, and the engine goes on from a finite state."""
    spec = S.SystemSpec("box", box, waters, cutoff=1.0, mc_sweeps=4)
    s = S.make_system(spec, seed=12)
    p = E.default_params(box_len=box, cutoff=1.0, dt=spec.dt, semantics=E.SEMANTICS_PHYSICS, skin=0.05, switch_on=0.8,
                         nlist_period=0)
    lost = waters // 3
    bad = s.solvents.copy()
    bad["pos"][lost, axis] = value
    with E.Engine(s, p) as eng:
        off, ids = (np.asarray(a).copy() for a in eng.nlist(E.NL_PAIR))
        rows = np.repeat(np.arange(waters), np.diff(off))
        eng.set_state(s.states, None, bad)
        boff, bids = eng.nlist(E.NL_PAIR)
        brows = np.repeat(np.arange(waters), np.diff(boff))
        keep = (rows != lost) & (ids != lost)
        assert np.array_equal(brows, rows[keep]) and np.array_equal(bids, ids[keep])
        with pytest.raises(E.LimaError) as ei:
            eng.step(1)
            eng.synchronize()
        assert ei.value.status == E.ERR_NUMERIC
        eng.set_state(s.states, None, s.solvents)
        goff, gids = eng.nlist(E.NL_PAIR)
        assert np.array_equal(goff, off) and np.array_equal(gids, ids)


@pytest.mark.parametrize("apart", [0.001, 0.02, 0.04, 0.06, 0.08, 0.1])
@pytest.mark.parametrize("axis", [0, 2])
def test_rebuild_with_particles_thrown_out_of_the_box(apart, axis):
    """Two waters too close together are thrown up to many box lengths away (or
    to infinity) within a step, which asks for a rebuild at those positions: a
    numeric status or none, and the engine goes on from an ordinary state."""
    box, waters = 4.0, 1900
    spec = S.SystemSpec("box", box, waters, cutoff=1.0, mc_sweeps=4)
    s = S.make_system(spec, seed=13)
    p = E.default_params(box_len=box, cutoff=1.0, dt=spec.dt, semantics=E.SEMANTICS_PHYSICS, skin=0.05, switch_on=0.8,
                         nlist_period=0)
    close = s.solvents.copy()
    close["pos"][1] = close["pos"][0]
    close["pos"][1, axis] += np.float32(apart)
    close["pos_tsub1"][:2] = close["pos"][:2]
    with E.Engine(s, p) as eng:
        off, ids = (np.asarray(a).copy() for a in eng.nlist(E.NL_PAIR))
        eng.set_state(s.states, None, close)
        try:
            for _ in range(6):
                eng.step(1)
                eng.synchronize()
        except E.LimaError as e:
            assert e.status == E.ERR_NUMERIC
        eng.set_state(s.states, None, s.solvents)
        goff, gids = eng.nlist(E.NL_PAIR)
        assert np.array_equal(goff, off) and np.array_equal(gids, ids)


@pytest.mark.parametrize("box,waters", [(10.0, 1000), (20.0, 17000)])   # one and four particles a warp
@pytest.mark.parametrize("beyond", [0, 1])
def test_capacity_counts_rows_without_their_exclusions(box, waters, beyond):
    """A row that fits the list once its bonded exclusions are out of it is
    accepted; one entry more is a capacity status.  A straight chain in the
    middle, its middle particle's neighbours in two clusters of waters that do
    not see each other, the other waters on a sparse lattice."""
    length, mid = 24, 12
    spec = S.SystemSpec("box", box, waters, cutoff=0.9, chains=S.ChainSpec(1, length), mc_sweeps=0)
    s = S.make_system(spec, seed=14)
    skin = 0.1
    n = length + waters
    # the list's capacity (a third more than an even density fills, and 96, in chunks of 32)
    cap = (int(1.6 * (4 / 3 * np.pi * 1.0 ** 3 * n / box ** 3) + 96) + 31) // 32 * 32
    excl = int(s.compounds[0]["lj_ignore_list"][mid]["n_ignores"])
    near = 8                                         # chain particles within 1 nm of the middle one
    assert 1 < excl < near
    in_reach = cap + beyond - (near - excl)          # waters in its list
    c = box / 2
    st, sol = s.states.copy(), s.solvents.copy()
    st["positions"][0, :length] = c
    st["positions"][0, :length, 1] += 0.21 * (np.arange(length) - mid)
    rng = np.random.default_rng(2)
    x = rng.uniform(-0.01, 0.01, (in_reach, 3)) + c
    x[:, 0] += np.where(np.arange(in_reach) % 2, 0.93, -0.93)
    g = (np.stack(np.meshgrid(*[np.arange(int(box / 0.72))] * 3), -1).reshape(-1, 3) + 0.5) * 0.72
    g = g[np.linalg.norm(g - c, axis=1) > 4.0]
    sol["pos"] = np.concatenate([x, g[: waters - in_reach]])
    p = E.default_params(box_len=box, cutoff=0.9, dt=spec.dt, semantics=E.SEMANTICS_PHYSICS, skin=skin, switch_on=0.8,
                         nlist_period=0)
    with E.Engine(s, p) as eng:
        if beyond:
            with pytest.raises(E.LimaError) as ei:
                eng.set_state(st, None, sol)
            assert ei.value.status == E.ERR_CAPACITY
        else:
            eng.set_state(st, None, sol)
            off, ids = eng.nlist(E.NL_PAIR)
            assert off[mid + 1] - off[mid] == cap
            mine = ids[off[mid]:off[mid + 1]]
            assert (mine < length).sum() == near - excl and (mine >= length).sum() == in_reach
